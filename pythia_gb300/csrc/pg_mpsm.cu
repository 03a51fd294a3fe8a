// MPSM / sort-merge join on sm_103a.
//
// Replaces SortMergeJoinOp::BufferAndSort (operators/join.cpp:945-996) and
// the merge loops of OldMPSMJoinOp / MPSMJoinOp (join.cpp:1245-1371,
// 1516-1538; PresortedPrepartitionedMergeJoinOp::getNext, join.cpp:1929-1968),
// which sort per-thread runs of both inputs and merge each build run against
// the probe runs, buffering the build tuples of the current key
// (mostfreqbuildkeyoccurances) and emitting the cartesian product of equal-key
// groups.
//
// Joins whose keys span a compact range count one side's keys in a table and
// look the other side up (mj_dense_join further down), with no sort.
//
// GPU plan otherwise: sort both relations (pg_sort.cu), cut each sorted relation into
// equal-key runs (stream compaction of run heads: run starts and run keys),
// match build runs to probe runs by merging the two sorted run-key arrays, scan the per-run output counts |R_k|*|S_k|, and either fold
// count and sum (no output materialised; a build column sums as
// |S_k| * sum_R_k, a probe column as |R_k| * sum_S_k, wrapping int64 like the
// reference's CtLong +=) or write every pair, each thread producing a
// contiguous slice of output positions (load-balanced over skewed groups).
// The reference's per-key buffer limit does not exist here: any multiplicity
// is joined.
#include "pg_internal.cuh"
#include "pg_sort.cuh"
#include <algorithm>

#define MJ_MAX_COLS 16

struct MjCols {
	int n, ow_words;
	uint8_t side[MJ_MAX_COLS];
	uint16_t off[MJ_MAX_COLS];    // byte offset in the side's tuple
	uint8_t words[MJ_MAX_COLS];
};

struct MjSide {
	const pg_rec* rec;   // sorted records
	const char* rows;    // original tuples
	uint32_t W, koff;
	int mode;            // pg_sort_mode
	const uint64_t* run_start;  // [nruns + 1]
	uint64_t nruns;
};

// Word w of column (off, words) of the tuple behind record r.
__device__ __forceinline__ uint32_t mj_word(const MjSide& sd, const pg_rec& r, uint32_t off, uint32_t w)
{
	if (sd.mode == 2) return reinterpret_cast<const uint32_t*>(sd.rows + r.val * sd.W + off)[w];
	// 16-byte tuple: the key half and the other half.
	uint32_t byte = off + 4 * w;
	bool in_key = (byte >= sd.koff && byte < sd.koff + 8);
	unsigned long long half = in_key ? (unsigned long long) r.key : r.val;
	uint32_t rel = in_key ? byte - sd.koff : (byte >= 8 ? byte - 8 : byte);
	return rel == 0 ? (uint32_t) half : (uint32_t) (half >> 32);
}

__device__ __forceinline__ unsigned long long mj_col64(const MjSide& sd, const pg_rec& r, uint32_t off, uint32_t words)
{
	uint32_t lo = mj_word(sd, r, off, 0);
	if (words == 2) return ((unsigned long long) mj_word(sd, r, off, 1) << 32) | lo;
	return (unsigned long long) (long long) (int32_t) lo;
}

// Equal-key runs of a sorted record array by stream compaction over chunks of
// MJ_RUN_CHUNK records: k_run_count counts run heads per chunk, a scan of the
// chunk counts gives each chunk its first run id, and k_run_write writes, in
// order, every run's first record index and key.
#define MJ_RUN_CHUNK 4096
#define MJ_RUN_THREADS 256

__device__ __forceinline__ bool mj_head(const pg_rec* rec, uint64_t i)
{
	return i == 0 || rec[i].key != rec[i - 1].key;
}

__global__ void __launch_bounds__(MJ_RUN_THREADS)
k_run_count(const pg_rec* __restrict__ rec, uint64_t n, uint64_t* __restrict__ ccount)
{
	__shared__ uint32_t wsum[MJ_RUN_THREADS / 32];
	const uint64_t nchunks = pg_div_up(n, MJ_RUN_CHUNK);
	for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
		const uint64_t lo = c * MJ_RUN_CHUNK, hi = pg_min64(n, lo + MJ_RUN_CHUNK);
		uint32_t cnt = 0;
		for (uint64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) cnt += mj_head(rec, i);
		#pragma unroll
		for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
		if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
		__syncthreads();
		if (threadIdx.x == 0) {
			uint64_t t = 0;
			for (int w = 0; w < MJ_RUN_THREADS / 32; ++w) t += wsum[w];
			ccount[c] = t;
		}
		__syncthreads();
	}
}

__global__ void __launch_bounds__(MJ_RUN_THREADS)
k_run_write(const pg_rec* __restrict__ rec, uint64_t n, const uint64_t* __restrict__ cfirst,
		uint64_t* __restrict__ start, long long* __restrict__ rkey)
{
	__shared__ uint32_t wsum[MJ_RUN_THREADS / 32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const uint64_t nchunks = pg_div_up(n, MJ_RUN_CHUNK);
	for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
		const uint64_t lo = c * MJ_RUN_CHUNK, hi = pg_min64(n, lo + MJ_RUN_CHUNK);
		uint64_t base = cfirst[c];
		for (uint64_t i0 = lo; i0 < hi; i0 += blockDim.x) {
			const uint64_t i = i0 + threadIdx.x;
			const bool h = i < hi && mj_head(rec, i);
			const uint32_t ball = __ballot_sync(0xffffffffu, h);
			if (lane == 0) wsum[warp] = __popc(ball);
			__syncthreads();
			uint32_t before = 0, total = 0;
			#pragma unroll
			for (int w = 0; w < MJ_RUN_THREADS / 32; ++w) { const uint32_t x = wsum[w]; before += w < warp ? x : 0; total += x; }
			if (h) {
				const uint64_t id = base + before + __popc(ball & ((1u << lane) - 1));
				start[id] = i;
				rkey[id] = rec[i].key;
			}
			base += total;
			__syncthreads();
		}
	}
}

// For every build run: matching probe run (or none), output count, and the
// folded count/sum contribution. A warp takes MJ_WARP_RUNS consecutive build
// runs: one lane finds the window of probe runs whose keys lie in the batch's
// key range (two binary searches), then the lanes take consecutive build runs
// (coalesced reads of keys and starts, coalesced count/match writes) and
// binary-search their key inside the window, which stays in L1. The summed
// column of a matched run is added by its lane when the run is short, and by
// the whole warp (strided loads, shuffle reduction) when it is long, so skewed
// keys do not serialise on one lane.
#define MJ_WARP_RUNS 512
#define MJ_SHORT_RUN 64

__device__ __forceinline__ uint64_t mj_lower(const long long* __restrict__ K, uint64_t lo, uint64_t hi, long long k)
{
	while (lo < hi) {
		const uint64_t mid = (lo + hi) >> 1;
		if (K[mid] < k) lo = mid + 1; else hi = mid;
	}
	return lo;
}

__global__ void __launch_bounds__(256)
k_match_runs(MjSide R, MjSide S, const long long* __restrict__ RK, const long long* __restrict__ SK,
		MjCols pc, int sum_col, uint64_t* __restrict__ counts, uint64_t* __restrict__ match,
		unsigned long long* __restrict__ agg)
{
	const int lane = threadIdx.x & 31;
	const uint64_t gwarp = ((uint64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const uint64_t nwarps = ((uint64_t) gridDim.x * blockDim.x) >> 5;
	const bool sum_r = sum_col >= 0 && pc.side[sum_col] == 0, sum_s = sum_col >= 0 && pc.side[sum_col] != 0;
	const uint32_t soff = sum_col >= 0 ? pc.off[sum_col] : 0, swords = sum_col >= 0 ? pc.words[sum_col] : 0;
	unsigned long long sum_acc = 0;
	for (uint64_t u0 = gwarp * MJ_WARP_RUNS; u0 < R.nruns; u0 += nwarps * MJ_WARP_RUNS) {
		const uint64_t u1 = pg_min64(R.nruns, u0 + MJ_WARP_RUNS);
		uint64_t slo = 0, shi = 0;
		if (lane == 0) {
			slo = mj_lower(SK, 0, S.nruns, RK[u0]);
			const long long klast = RK[u1 - 1];
			shi = klast == LLONG_MAX ? S.nruns : mj_lower(SK, slo, S.nruns, klast + 1);
		}
		slo = __shfl_sync(0xffffffffu, slo, 0);
		shi = __shfl_sync(0xffffffffu, shi, 0);
		for (uint64_t j = u0; j < u1; j += 32) {
			const uint64_t u = j + lane;
			const bool valid = u < u1;
			uint64_t c = 0, m = UINT64_MAX, lo_i = 0, hi_i = 0, other = 0;
			if (valid) {
				const long long k = RK[u];
				const uint64_t v = mj_lower(SK, slo, shi, k);
				if (v < shi && SK[v] == k) {
					const uint64_t r0 = R.run_start[u], r1 = R.run_start[u + 1];
					const uint64_t s0 = S.run_start[v], s1 = S.run_start[v + 1];
					c = (r1 - r0) * (s1 - s0);
					m = v;
					if (sum_r) { lo_i = r0; hi_i = r1; other = s1 - s0; }
					else if (sum_s) { lo_i = s0; hi_i = s1; other = r1 - r0; }
				}
				counts[u] = c;
				match[u] = m;
			}
			if (sum_col < 0) continue;
			const MjSide& sd = sum_r ? R : S;
			const bool longrun = hi_i - lo_i > MJ_SHORT_RUN;
			if (!longrun && hi_i > lo_i) {
				unsigned long long part = 0;
				for (uint64_t i = lo_i; i < hi_i; ++i) part += mj_col64(sd, sd.rec[i], soff, swords);
				sum_acc += part * (unsigned long long) other;
			}
			uint32_t longs = __ballot_sync(0xffffffffu, longrun);
			while (longs) {
				const int l = __ffs(longs) - 1;
				longs &= longs - 1;
				const uint64_t a = __shfl_sync(0xffffffffu, lo_i, l), b = __shfl_sync(0xffffffffu, hi_i, l);
				const uint64_t o = __shfl_sync(0xffffffffu, other, l);
				unsigned long long part = 0;
				for (uint64_t i = a + lane; i < b; i += 32) part += mj_col64(sd, sd.rec[i], soff, swords);
				#pragma unroll
				for (int q = 16; q > 0; q >>= 1) part += __shfl_xor_sync(0xffffffffu, part, q);
				if (lane == 0) sum_acc += part * (unsigned long long) o;
			}
		}
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) sum_acc += __shfl_down_sync(0xffffffffu, sum_acc, o);
	if (lane == 0 && sum_acc) atomicAdd(agg, sum_acc);
}

#define MJ_PER_THREAD 8

// Writes output rows [t*8, t*8+8): pair (u, v) of position p is found by a
// binary search over the scanned counts; within a pair, position q maps to
// probe tuple q / |R_u| and build tuple q % |R_u|.
__global__ void k_mj_write(MjSide R, MjSide S, MjCols pc, const uint64_t* __restrict__ offs,
		const uint64_t* __restrict__ match, uint64_t nout, char* __restrict__ out)
{
	const uint64_t ow = (uint64_t) pc.ow_words * 4;
	for (uint64_t t = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; t * MJ_PER_THREAD < nout;
			t += (uint64_t) gridDim.x * blockDim.x) {
		uint64_t p = t * MJ_PER_THREAD;
		const uint64_t pend = pg_min64(nout, p + MJ_PER_THREAD);
		// upper_bound(offs, p) - 1 over runs with offsets
		uint64_t lo = 0, hi = R.nruns;
		while (lo < hi) {
			uint64_t mid = (lo + hi) >> 1;
			if (offs[mid] <= p) lo = mid + 1; else hi = mid;
		}
		uint64_t u = lo - 1;
		while (p < pend) {
			while (offs[u + 1] <= p) ++u;           // skip empty runs
			const uint64_t v = match[u];
			const uint64_t r0 = R.run_start[u], nr = R.run_start[u + 1] - r0;
			const uint64_t s0 = S.run_start[v];
			uint64_t q = p - offs[u];
			const uint64_t stop = pg_min64(pend, offs[u + 1]);
			for (; p < stop; ++p, ++q) {
				const pg_rec& br = R.rec[r0 + q % nr];
				const pg_rec& pr = S.rec[s0 + q / nr];
				uint32_t* o = reinterpret_cast<uint32_t*>(out + p * ow);
				int wo = 0;
				for (int c = 0; c < pc.n; ++c)
					for (int w = 0; w < pc.words[c]; ++w)
						o[wo++] = pc.side[c] ? mj_word(S, pr, pc.off[c], w) : mj_word(R, br, pc.off[c], w);
			}
		}
	}
}

// Runs of both sides (starts and keys in `out`), with one readback of their numbers.
static int mj_runs(pg_ctx* ctx, cudaStream_t s, const pg_rec* const (&rec)[2], const uint64_t (&n)[2], PgScratch& out,
		uint64_t* (&starts)[2], long long* (&keys)[2], uint64_t (&nruns)[2])
{
	int rc;
	PgScratch mem(ctx, s);
	uint64_t *cc[2], *total = nullptr;
	if ((rc = mem.get((void**) &total, 16))) return rc;
	for (int i = 0; i < 2; ++i) {
		const uint64_t nchunks = pg_div_up(n[i], MJ_RUN_CHUNK);
		if ((rc = mem.get((void**) &cc[i], (nchunks + 1) * 8))) return rc;
		k_run_count<<<(int) std::min<uint64_t>(nchunks, (uint64_t) ctx->sm_count * 8), MJ_RUN_THREADS, 0, s>>>(rec[i], n[i], cc[i]);
		PG_LAUNCHED(ctx);
		if ((rc = pg_scan_u64(ctx, s, cc[i], nchunks, total + i))) return rc;
	}
	PG_CUDA(ctx, cudaMemcpyAsync(nruns, total, 16, cudaMemcpyDeviceToHost, s));
	PG_CUDA(ctx, cudaStreamSynchronize(s));
	for (int i = 0; i < 2; ++i) {
		if ((rc = out.get((void**) &starts[i], (nruns[i] + 1) * 8))) return rc;
		if ((rc = out.get((void**) &keys[i], (nruns[i] + 1) * 8))) return rc;
		const uint64_t nchunks = pg_div_up(n[i], MJ_RUN_CHUNK);
		k_run_write<<<(int) std::min<uint64_t>(nchunks, (uint64_t) ctx->sm_count * 8), MJ_RUN_THREADS, 0, s>>>(rec[i], n[i], cc[i],
				starts[i], keys[i]);
		PG_LAUNCHED(ctx);
		PG_CUDA(ctx, cudaMemcpyAsync(starts[i] + nruns[i], &n[i], 8, cudaMemcpyHostToDevice, s));
	}
	return PG_OK;
}

// Key range of tuples 0, step, 2 step, ... (keys ^ 2^63 as unsigned) into mm =
// [~smallest, largest], zero before; with `unsorted` (step 1), also whether some key is greater than
// the next one.
__global__ void k_mj_minmax(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes,
		uint64_t step, unsigned long long* __restrict__ mm, unsigned long long* __restrict__ unsorted)
{
	unsigned long long lo = ~0ull, hi = 0;
	bool down = false;
	for (uint64_t i = (blockIdx.x * (uint64_t) blockDim.x + threadIdx.x) * step; i < n;
			i += (uint64_t) gridDim.x * blockDim.x * step) {
		const long long k = pg_load_key(in + i * W + koff, kbytes);
		const unsigned long long u = (unsigned long long) k ^ (1ull << 63);
		lo = u < lo ? u : lo;
		hi = u > hi ? u : hi;
		if (unsorted && i + 1 < n && k > pg_load_key(in + (i + 1) * W + koff, kbytes)) down = true;
	}
	if (unsorted && __any_sync(0xffffffffu, down) && (threadIdx.x & 31) == 0) *unsorted = 1;
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		const unsigned long long a = __shfl_down_sync(0xffffffffu, lo, o), b = __shfl_down_sync(0xffffffffu, hi, o);
		lo = a < lo ? a : lo;
		hi = b > hi ? b : hi;
	}
	if ((threadIdx.x & 31) == 0) { atomicMax(&mm[0], ~lo); atomicMax(&mm[1], hi); }
}


// ---------------------------------------------------------------------------
// Keys of compact range: a counting sort of one side takes the place of sorting
// both. A table of 4-byte counts over the key window [kmin, kmin + range) is
// filled with one L2 atomic a tuple, and the other side looks its keys up.
//
// - Count/sum: the side without the summed column is counted; a tuple of the
//   other side then adds its count to the rows and count * column to the sum.
// - Rows: the build side is counted, the counts are scanned into run starts,
//   its packed columns are scattered into their runs, and every probe tuple
//   writes one row per value of its key's run.
//
// Both relations are read once or twice and neither is written back sorted,
// which is what the sort-merge of the same join spends its time on.
// ---------------------------------------------------------------------------
#define MJ_ILP 2                    // tuples in flight a thread of the counting and lookup passes
#define MJ_BLOCKS_PER_SM 64         // blocks of those passes: many short ones (64M x 64M: 0.75 ms; 8 and 16: 0.92)
#define MJ_MAX_RANGE (1ull << 30)
#define MJ_MIN_RANGE (1ull << 24)   // window always worth a table (64 MB, kept in L2)
#define MJ_MAX_RUN 16384            // longest build run whose rows one warp writes for a probe tuple

// Key of tuple i; V16: 16-byte tuples with an 8-byte key in either half.
template <bool V16>
__device__ __forceinline__ int64_t mj_key(const char* __restrict__ in, uint64_t i, uint32_t W, uint32_t koff,
		uint32_t kbytes, uint64_t pol, uint4& t)
{
	if (V16) {
		t = pg_ld_hint16(in + i * 16, pol);
		return koff == 0 ? (int64_t) (((uint64_t) t.y << 32) | t.x) : (int64_t) (((uint64_t) t.w << 32) | t.z);
	}
	return pg_load_key(in + i * W + koff, kbytes);
}

// The build-projected words of a row that are not the join key, packed.
struct MjPack {
	int n;
	uint8_t roff[2];             // word offsets in the build tuple
};

__device__ __forceinline__ uint32_t mjw_word(const uint4& t, uint32_t i)
{
	return i == 0 ? t.x : i == 1 ? t.y : i == 2 ? t.z : t.w;
}

__device__ __forceinline__ unsigned long long mj_packed(const uint4& t, const MjPack& bp)
{
	unsigned long long v = 0;
	if (bp.n > 0) v = mjw_word(t, bp.roff[0]);
	if (bp.n > 1) v |= (unsigned long long) mjw_word(t, bp.roff[1]) << 32;
	return v;
}

// Table loads, kept in L2 while the relations stream past.
__device__ __forceinline__ uint32_t mj_ld16(const uint16_t* p, uint64_t pol)
{
	uint16_t v;
	asm("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
	return v;
}

__device__ __forceinline__ uint32_t mj_ld32(const uint32_t* p, uint64_t pol)
{
	uint32_t v;
	asm("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
	return v;
}

__device__ __forceinline__ unsigned long long mj_ld64(const unsigned long long* p, uint64_t pol)
{
	unsigned long long v;
	asm("ld.global.nc.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(pol));
	return v;
}

// cnt[key - kmin] += 1 for every tuple; a key outside the window sets *outside.
// Lanes that hold lane 0's key add once together when there are several of
// them, so that one key with most of the rows does not queue 32 adds a warp.
// SHARED: each block counts in shared memory and adds its counts to the table once.
// Few keys otherwise queue every tuple's add at a few L2 addresses: 64M tuples of 4 to 1024
// keys 13.4 to 4.9 ms, with it 0.24 (sorting the side and matching its few runs: 1.7 to 2.5).
// VALS: also the range of the packed build values, into vmm = [~smallest, largest],
// zero before.
#define MJ_SHARED_RANGE 8192        // counts in shared memory: 32 KB, six blocks on an SM
#define MJ_SHARED_ROWS 8            // tuples a block for each of its counts, which it adds at its end
template <bool V16, bool VALS, bool SHARED>
__global__ void __launch_bounds__(256)
k_mj_count(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes, long long kmin,
		uint32_t range, uint32_t* __restrict__ cnt, unsigned int* __restrict__ outside, MjPack bp,
		unsigned long long* __restrict__ vmm)
{
	extern __shared__ uint32_t mj_counts[];
	if (SHARED) {
		for (uint32_t i = threadIdx.x; i < range; i += blockDim.x) mj_counts[i] = 0;
		__syncthreads();
	}
	unsigned long long vlo = ~0ull, vhi = 0;
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x, pol = pg_policy_evict_first();
	const uint32_t lane = threadIdx.x & 31;
	bool out = false;
	for (uint64_t base = blockIdx.x * (uint64_t) blockDim.x; base < n; base += stride * MJ_ILP) {
		uint32_t d[MJ_ILP];
		#pragma unroll
		for (int j = 0; j < MJ_ILP; ++j) {
			const uint64_t i = base + threadIdx.x + j * stride;
			d[j] = 0xFFFFFFFFu;
			if (i < n) {
				uint4 t;
				const uint64_t x = (uint64_t) mj_key<V16>(in, i, W, koff, kbytes, pol, t) - (uint64_t) kmin;
				if (x < range) d[j] = (uint32_t) x; else out = true;
				if (VALS) {
					const unsigned long long v = mj_packed(t, bp);
					vlo = min(vlo, v);
					vhi = max(vhi, v);
				}
			}
		}
		#pragma unroll
		for (int j = 0; j < MJ_ILP; ++j) {
			const uint32_t same = __ballot_sync(0xffffffffu, d[j] == __shfl_sync(0xffffffffu, d[j], 0));
			const bool many = __popc(same) >= 4;
			if (d[j] == 0xFFFFFFFFu || (many && lane && (same >> lane & 1))) continue;
			atomicAdd(SHARED ? &mj_counts[d[j]] : &cnt[d[j]], many && lane == 0 ? (uint32_t) __popc(same) : 1u);
		}
	}
	if (out) *outside = 1;
	if (SHARED) {
		__syncthreads();
		for (uint32_t i = threadIdx.x; i < range; i += blockDim.x)
			if (mj_counts[i]) atomicAdd(&cnt[i], mj_counts[i]);
	}
	if (VALS) {
		__shared__ unsigned long long red[2][8];
		#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			vlo = min(vlo, __shfl_xor_sync(0xffffffffu, vlo, o));
			vhi = max(vhi, __shfl_xor_sync(0xffffffffu, vhi, o));
		}
		if (lane == 0) { red[0][threadIdx.x >> 5] = vlo; red[1][threadIdx.x >> 5] = vhi; }
		__syncthreads();
		if (threadIdx.x == 0) {
			for (int w = 1; w < 8; ++w) { vlo = min(vlo, red[0][w]); vhi = max(vhi, red[1][w]); }
			atomicMax(&vmm[0], ~vlo);
			atomicMax(&vmm[1], vhi);
		}
	}
}

// agg[0] += the other side's tuples of each key, agg[1] += that many times
// column (soff, swords); swords 0: no sum.
template <bool V16>
__global__ void __launch_bounds__(256)
k_mj_lookup(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes, uint32_t soff,
		uint32_t swords, long long kmin, uint32_t range, const uint32_t* __restrict__ cnt,
		unsigned long long* __restrict__ agg, const int* __restrict__ status)
{
	if (blockIdx.x == 0 && threadIdx.x == 0) pg_collect(agg + 3, nullptr, status);
	__shared__ unsigned long long red[2][8];
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x, pol = pg_policy_evict_first();
	const uint64_t keep = pg_policy_keep(4);
	unsigned long long rows = 0, sum = 0;
	for (uint64_t base = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; base < n; base += stride * MJ_ILP) {
		uint32_t c[MJ_ILP];
		unsigned long long v[MJ_ILP];
		#pragma unroll
		for (int j = 0; j < MJ_ILP; ++j) {
			const uint64_t i = base + j * stride;
			c[j] = 0;
			v[j] = 0;
			if (i < n) {
				uint4 t;
				const uint64_t x = (uint64_t) mj_key<V16>(in, i, W, koff, kbytes, pol, t) - (uint64_t) kmin;
				if (V16) {
					const uint32_t w = soff / 4;
					const uint32_t lo = w == 0 ? t.x : w == 1 ? t.y : w == 2 ? t.z : t.w;
					const uint32_t hi = w == 0 ? t.y : w == 1 ? t.z : t.w;
					v[j] = swords == 2 ? ((unsigned long long) hi << 32) | lo : (unsigned long long) (long long) (int32_t) lo;
				}
				if (x < range) {
					asm("ld.global.nc.L1::evict_last.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(c[j]) : "l"(cnt + x), "l"(keep));
					if (!V16 && swords) {
						const uint32_t* q = reinterpret_cast<const uint32_t*>(in + i * W + soff);
						v[j] = swords == 2 ? ((unsigned long long) q[1] << 32) | q[0] : (unsigned long long) (long long) (int32_t) q[0];
					}
				}
			}
		}
		#pragma unroll
		for (int j = 0; j < MJ_ILP; ++j) { rows += c[j]; sum += v[j] * c[j]; }
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		rows += __shfl_down_sync(0xffffffffu, rows, o);
		sum += __shfl_down_sync(0xffffffffu, sum, o);
	}
	if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = rows; red[1][threadIdx.x >> 5] = sum; }
	__syncthreads();
	if (threadIdx.x < 2) {
		unsigned long long t = 0;
		#pragma unroll
		for (int w = 0; w < 8; ++w) t += red[threadIdx.x][w];
		if (t && (threadIdx.x == 0 || swords)) atomicAdd(&agg[threadIdx.x], t);
	}
}

// Exclusive scan of the counts in place (mod 2^32; a side has fewer than 2^32
// tuples): sums of MJ_SCAN counts, their scan (pg_scan_u64), then each
// block's counts. The largest count goes to *mx.
#define MJ_SCAN 4096
__global__ void __launch_bounds__(256)
k_mj_scan_sums(const uint32_t* __restrict__ cnt, uint32_t range, uint64_t* __restrict__ sums, unsigned int* __restrict__ mx)
{
	__shared__ uint32_t red[2][8];
	const uint64_t lo = (uint64_t) blockIdx.x * MJ_SCAN;
	uint32_t s = 0, m = 0;
	#pragma unroll
	for (int j = 0; j < MJ_SCAN / 256; ++j) {
		const uint64_t i = lo + j * 256 + threadIdx.x;
		const uint32_t c = i < range ? cnt[i] : 0;
		s += c;
		m = max(m, c);
	}
	s = __reduce_add_sync(0xffffffffu, s);
	m = __reduce_max_sync(0xffffffffu, m);
	if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = s; red[1][threadIdx.x >> 5] = m; }
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int w = 1; w < 8; ++w) { s += red[0][w]; m = max(m, red[1][w]); }
		sums[blockIdx.x] = s;
		if (m > *mx) atomicMax(mx, m);
	}
}

__global__ void __launch_bounds__(256)
k_mj_scan_apply(uint32_t* __restrict__ cnt, uint32_t range, const uint64_t* __restrict__ sums)
{
	__shared__ uint32_t wt[8];
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr int PER = MJ_SCAN / 256;
	// Warp w scans its own MJ_SCAN / 8 counts, 32 at a time.
	const uint64_t lo = (uint64_t) blockIdx.x * MJ_SCAN + warp * (MJ_SCAN / 8) + lane;
	uint32_t c[PER], mine = 0;
	#pragma unroll
	for (int j = 0; j < PER; ++j) { c[j] = lo + j * 32 < range ? cnt[lo + j * 32] : 0; mine += c[j]; }
	const uint32_t tot = __reduce_add_sync(0xffffffffu, mine);
	if (lane == 0) wt[warp] = tot;
	__syncthreads();
	uint32_t run = (uint32_t) sums[blockIdx.x];
	for (uint32_t w = 0; w < warp; ++w) run += wt[w];
	#pragma unroll
	for (int j = 0; j < PER; ++j) {
		uint32_t x = c[j];
		#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
			if (lane >= (uint32_t) o) x += y;
		}
		if (lo + j * 32 < range) cnt[lo + j * 32] = run + x - c[j];
		run += __shfl_sync(0xffffffffu, x, 31);
	}
}

// Bytes of a value slot: values that span less than 2^16 or 2^32 are kept as
// differences from the smallest (vmm, from the counting pass). The scattered stores
// and the probe's scattered reads then move fewer bytes and stay in L2 for more
// tuples: 16M x 16M with four duplicates a key and values below 1000, 2 bytes
// against 4: 245 -> 208 us the fill, 562 -> 522 the rows.
__device__ __forceinline__ uint32_t mj_val_bytes(unsigned long long span)
{
	return span < (1u << 16) ? 2 : span < (1ull << 32) ? 4 : 8;
}

// Scatters the packed build columns into their keys' runs: pos[d] is run d's
// first slot before and its end (the next run's start) after. One tuple a thread
// in many blocks: each waits for its returning add (four a thread: 10 us more).
// Nothing is done when a run is longer than MJ_MAX_RUN or a key lay outside the
// window (meta[0], meta[1]).
#define MJ_FILL_BLOCKS_PER_SM 64
__global__ void __launch_bounds__(256)
k_mj_fill(const char* __restrict__ R, uint64_t n, uint32_t koff, long long kmin, uint32_t range, MjPack bp,
		uint32_t* __restrict__ pos, unsigned long long* __restrict__ val, const unsigned int* __restrict__ meta,
		const unsigned long long* __restrict__ vmm)
{
	if (meta[0] > MJ_MAX_RUN || meta[1]) return;
	const unsigned long long vmin = ~vmm[0];
	const uint32_t bytes = mj_val_bytes(vmm[1] - vmin);
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x, pol = pg_policy_evict_first();
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += stride) {
		uint4 t;
		const uint64_t x = (uint64_t) mj_key<true>(R, i, 16, koff, 8, pol, t) - (uint64_t) kmin;
		if (x >= range) continue;
		const uint32_t at = atomicAdd(&pos[x], 1u);
		if (at >= n) continue;
		const unsigned long long v = mj_packed(t, bp);
		if (bytes == 2) reinterpret_cast<uint16_t*>(val)[at] = (uint16_t) (v - vmin);
		else if (bytes == 4) reinterpret_cast<uint32_t*>(val)[at] = (uint32_t) (v - vmin);
		else val[at] = v;
	}
}

// Rows of each probe tuple: one per value of its key's run [ends[d - 1],
// ends[d]). A warp looks up 32 T tuples at once, reserves their rows with one
// add on the cursor, and writes them 32 at a time, each lane finding its row's
// tuple by a search over the lanes' offsets, so that a warp stores consecutive
// rows whatever the runs' lengths. Rows past `cap` are counted only.
// Bound by DRAM: the values' scattered reads miss L2 under the stream of rows
// (16M tuples, 64M rows, 4-byte values: 1.36 GB read and 1.07 written). The whole join
// above with its group-by: no limit on registers 1214 us, with 6 blocks an SM 1160, and
// two tuples a lane instead of four 1105 (1150 with the slices); of keys with one
// row 1484, 1513 and 1590, so those take four.
//
// A warp's tuples may have thousands of rows each. Those of more than MJ_SLICE_MAX rows
// in all go on a list instead, MJ_SLICE rows an entry, and a second launch (SLICE) has a
// warp write an entry's rows. 1000 tuples with 16,000 rows each: 18.97 ms without it,
// 0.47 with (1.45 sorted, where a thread takes eight rows); 64 such tuples among 4M others 8.4,
// 0.27 (1.10). The second launch, empty, takes 2 to 4 us.
#define MJ_ROWS_BLOCKS_PER_SM 24
#define MJ_SLICE 2048u
#define MJ_SLICE_MAX 8192u
// Entries (tuples' first index / 32 T << 16 | slice) that hold the slices of `cap` rows: more
// rows than that do not fit the output.
static uint64_t mj_slices(uint64_t cap) { return cap / (MJ_SLICE / 2) + 16; }

template <int T, bool SLICE>                          // T tuples a lane
__global__ void __launch_bounds__(256, 6)
k_mj_rows(const char* __restrict__ S, uint64_t n, uint32_t koff, long long kmin, uint32_t range,
		const uint32_t* __restrict__ ends, const unsigned long long* __restrict__ val, uint32_t wsel,
		uint4* __restrict__ out, uint64_t cap, unsigned long long* __restrict__ cursor, const unsigned int* __restrict__ meta,
		const unsigned long long* __restrict__ vmm, unsigned long long* __restrict__ list, uint64_t list_cap,
		unsigned long long* __restrict__ listed, const int* __restrict__ status)
{
	if (!SLICE && blockIdx.x == 0 && threadIdx.x == 0) pg_collect(cursor + 3, nullptr, status);
	if (meta[0] > MJ_MAX_RUN || meta[1]) return;
	const unsigned long long vmin = ~vmm[0];
	const uint32_t bytes = mj_val_bytes(vmm[1] - vmin);
	const uint32_t lane = threadIdx.x & 31;
	const uint64_t pol = pg_policy_evict_first(), keep = pg_policy_keep(4);
	const uint64_t nwarps = ((uint64_t) gridDim.x * blockDim.x) >> 5;
	const uint32_t w0 = wsel & 15, w1 = (wsel >> 4) & 15, w2 = (wsel >> 8) & 15, w3 = (wsel >> 12) & 15;
	const uint64_t units = SLICE ? pg_min64(*listed, list_cap) : pg_div_up(n, 32 * T);
	for (uint64_t u = ((uint64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
		const unsigned long long entry = SLICE ? list[u] : u << 16;
		const uint64_t c0 = (entry >> 16) * (32 * T);
		uint4 t[T];
		uint32_t lo[T], m[T];
		#pragma unroll
		for (int j = 0; j < T; ++j) {
			const uint64_t i = c0 + j * 32 + lane;
			lo[j] = 0; m[j] = 0;
			t[j] = make_uint4(0, 0, 0, 0);
			if (i < n) {
				const uint64_t x = (uint64_t) mj_key<true>(S, i, 16, koff, 8, pol, t[j]) - (uint64_t) kmin;
				if (x < range) {
					m[j] = mj_ld32(ends + x, keep);
					if (x) lo[j] = mj_ld32(ends + x - 1, keep);
				}
			}
		}
		uint32_t off[T], total = 0;
		#pragma unroll
		for (int j = 0; j < T; ++j) {
			m[j] -= lo[j];
			uint32_t x = m[j];
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
				if (lane >= (uint32_t) o) x += y;
			}
			off[j] = x - m[j];
			m[j] = __shfl_sync(0xffffffffu, x, 31);       // rows of the 32 tuples
			total += m[j];
		}
		unsigned long long row = 0;
		if (!SLICE && total > MJ_SLICE_MAX) {
			const uint32_t pieces = (total + MJ_SLICE - 1) / MJ_SLICE;
			if (lane == 0) row = atomicAdd(listed, (unsigned long long) pieces);
			row = __shfl_sync(0xffffffffu, row, 0);
			for (uint32_t p = lane; p < pieces; p += 32)
				if (row + p < list_cap) list[row + p] = u << 16 | p;
				else atomicAdd(cursor, (unsigned long long) pg_min32(MJ_SLICE, total - p * MJ_SLICE));
			continue;
		}
		// Rows [first, last) of the warp's tuples.
		const uint32_t first = SLICE ? (uint32_t) (entry & 0xFFFF) * MJ_SLICE : 0;
		const uint32_t last = SLICE ? pg_min32(total, first + MJ_SLICE) : total;
		if (lane == 0 && last > first) row = atomicAdd(cursor, (unsigned long long) (last - first));
		row = __shfl_sync(0xffffffffu, row, 0) - first;
		uint32_t before = 0;                     // rows of the tuples before these 32
		#pragma unroll
		for (int j = 0; j < T; ++j) {
			const uint32_t begin = SLICE && first > before ? first - before : 0;
			const uint32_t end = !SLICE ? m[j] : last > before ? pg_min32(m[j], last - before) : 0;
			for (uint32_t r0 = begin; r0 < end; r0 += 32) {
				const uint32_t r = r0 + lane;
				uint32_t x = 0;                  // the last tuple whose offset is <= r (it has rows)
				#pragma unroll
				for (uint32_t step = 16; step; step >>= 1)
					if (__shfl_sync(0xffffffffu, off[j], x + step) <= r) x += step;
				const uint32_t at = __shfl_sync(0xffffffffu, lo[j], x) + (r - __shfl_sync(0xffffffffu, off[j], x));
				unsigned long long v = 0;
				if (r < end) {
					if (bytes == 2) v = vmin + mj_ld16(reinterpret_cast<const uint16_t*>(val) + at, keep);
					else if (bytes == 4) v = vmin + mj_ld32(reinterpret_cast<const uint32_t*>(val) + at, keep);
					else v = mj_ld64(val + at, keep);
				}
				auto pick = [&](uint32_t w) -> uint32_t {
					return w < 4 ? __shfl_sync(0xffffffffu, mjw_word(t[j], w), x) : w == 4 ? (uint32_t) v : (uint32_t) (v >> 32);
				};
				const uint4 o = make_uint4(pick(w0), pick(w1), pick(w2), pick(w3));
				if (r < end && row + r < cap) pg_st_hint16(out + row + r, o, pol);
			}
			row += m[j];
			if (SLICE) before += m[j];
		}
	}
}

// Word selector (4 bits per output word: 0-3 probe tuple word, 4-5 packed
// build word) and packed build words of the 16-byte output rows of the
// counted materialising join; false when the layout is not one it takes:
// 16-byte tuples with 8-byte keys on both sides, 16-byte rows whose build
// words other than the key (taken from the probe tuple's equal key) fit 8 bytes.
static bool mj_rows_fit(const pg_rel* R, const pg_rel* S, const MjCols& pc, uint32_t* wsel, MjPack* bp)
{
	if (R->width != 16 || S->width != 16 || R->key_bytes != 8 || S->key_bytes != 8 || (R->key_off & 7) ||
			(S->key_off & 7) || pc.ow_words != 4 ||
			(reinterpret_cast<uintptr_t>(R->data) & 15) || (reinterpret_cast<uintptr_t>(S->data) & 15))
		return false;
	bp->n = 0; bp->roff[0] = bp->roff[1] = 0;
	*wsel = 0;
	uint32_t o = 0;
	for (int c = 0; c < pc.n; ++c)
		for (uint32_t j = 0; j < pc.words[c]; ++j, ++o) {
			const uint32_t byte = pc.off[c] + 4 * j;
			uint32_t sel;
			if (pc.side[c]) {
				sel = byte / 4;
			} else if (byte >= R->key_off && byte < R->key_off + 8) {
				sel = (S->key_off + (byte - R->key_off)) / 4;
			} else {
				int p = -1;
				for (int q = 0; q < bp->n; ++q) if (bp->roff[q] == byte / 4) p = q;
				if (p < 0) {
					if (bp->n == 2) return false;
					p = bp->n;
					bp->roff[bp->n++] = (uint8_t) (byte / 4);
				}
				sel = 4 + (uint32_t) p;
			}
			*wsel |= sel << (4 * o);
		}
	return true;
}


static bool mj_v16(const pg_rel* r)
{
	return r->width == 16 && r->key_bytes == 8 && (r->key_off == 0 || r->key_off == 8) &&
		!(reinterpret_cast<uintptr_t>(r->data) & 15);
}

// First and last key into mm = [~first, last] (keys ^ 2^63 as unsigned); zeros when
// they show that the side is not sorted.
__global__ void k_mj_ends(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes,
		unsigned long long* __restrict__ mm)
{
	const unsigned long long a = (unsigned long long) pg_load_key(in + koff, kbytes) ^ (1ull << 63);
	const unsigned long long b = (unsigned long long) pg_load_key(in + (n - 1) * W + koff, kbytes) ^ (1ull << 63);
	mm[0] = a <= b ? ~a : 0;
	mm[1] = a <= b ? b : 0;
}

// The sides' flags, and what the device made of them.
struct MjSorted {
	bool flagged[2], known, sorted[2];
};

// Whether the flagged sides are sorted, in one readback, unless that is known.
static int mj_confirm_sorted(pg_ctx* ctx, cudaStream_t s, const pg_rel* R, const pg_rel* S, MjSorted* f)
{
	if (f->known || !(f->flagged[0] || f->flagged[1])) return PG_OK;
	int rc;
	PgScratch mem(ctx, s);
	unsigned long long* mm = nullptr;             // [key range, unsorted, spare] of each side
	if ((rc = mem.get((void**) &mm, 64))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(mm, 0, 64, s));
	for (int i = 0; i < 2; ++i) {
		if (!f->flagged[i]) continue;
		const pg_rel* r = i ? S : R;
		const int blocks = (int) std::min<uint64_t>(pg_div_up(r->n, 256), (uint64_t) ctx->sm_count * 8);
		k_mj_minmax<<<blocks, 256, 0, s>>>((const char*) r->data, r->n, r->width, r->key_off, r->key_bytes, 1, mm + 4 * i,
				mm + 4 * i + 2);
		PG_LAUNCHED(ctx);
	}
	unsigned long long h[8];
	PG_CUDA(ctx, cudaMemcpyAsync(h, mm, 64, cudaMemcpyDeviceToHost, s));
	PG_CUDA(ctx, cudaStreamSynchronize(s));
	for (int i = 0; i < 2; ++i) f->sorted[i] = f->flagged[i] && !h[4 * i + 2];
	f->known = true;
	return PG_OK;
}

// Rows of more tuples than this partition both sides first: 64M x 64M with four
// duplicates a key 6.83 -> 4.40 ms (4-byte values; by sorting both sides in buckets 5.98),
// 48M with 2-byte values and a group-by 4.76 -> 3.80; 32M 2.33 -> 2.74 with 2-byte values,
// 4.16 -> 3.74 with 4-byte ones (how wide they are is known only after the counting pass,
// which the copies come before).
#define MJ_SPLIT_TUPLES (32ull << 20)

// The join by a table of counts when the counted side's keys span a compact
// range: at most 2^24 values (1000 x 1000: sum 62 us against 161 sorted, rows 122
// against 178), or 16 times its tuples, where the table's random accesses come near the
// cost of sorting both sides (sum and rows: 16M x 16M 2.50 and 2.69 ms against 3.09 and
// 3.28, 64M x 64M over 2^30 8.05 and 8.61 against 10.13 and 10.69).
// The window comes from every 1024th tuple widened by 1/64 a side on large
// inputs, checked by the counting pass, else from every tuple. *handled =
// false (nothing produced): the caller sorts. So it does where the tables do not fit in
// memory; the partitioned copies are the first to be done without.
static int mj_dense_join(pg_ctx* ctx, cudaStream_t s, const pg_rel* R, const pg_rel* S, const MjCols& pc, int sum_col,
		int flags, void* out, uint64_t out_capacity, pg_join_result* res, MjSorted* sorted, bool* handled)
{
	*handled = false;
	const bool materialize = (flags & PG_JOIN_MATERIALIZE) != 0;
	uint32_t wsel = 0;
	MjPack bp = {};
	if (materialize && (!mj_rows_fit(R, S, pc, &wsel, &bp) || (reinterpret_cast<uintptr_t>(out) & 15)))
		return PG_OK;
	if (materialize && sum_col >= 0) {      // the sum as a join of its own, then the rows
		pg_join_result a;
		bool done = false;
		int rs = mj_dense_join(ctx, s, R, S, pc, sum_col, flags & ~PG_JOIN_MATERIALIZE, nullptr, 0, &a, sorted, &done);
		if (rs || !done) return rs;
		if ((rs = mj_dense_join(ctx, s, R, S, pc, -1, flags, out, out_capacity, res, sorted, handled)) || !*handled) return rs;
		res->sum = a.sum;
		return PG_OK;
	}
	// C is counted, P looks up.
	const bool sum_build = sum_col >= 0 && pc.side[sum_col] == 0;
	const bool count_build = materialize || (sum_col >= 0 ? !sum_build : R->n <= S->n);
	const pg_rel *C = count_build ? R : S, *P = count_build ? S : R;
	const int ci = count_build ? 0 : 1, pi = 1 - ci;
	int rc;
	// [~key min, key max], [rows, sum], [largest count, key outside], two words of
	// pg_readback, [~value min, value max], slices listed
	PgScratch mem(ctx, s);
	unsigned long long* mm = nullptr;
	if ((rc = mem.get((void**) &mm, 80))) return rc;
	unsigned long long* agg = mm + 2;
	unsigned int* meta = reinterpret_cast<unsigned int*>(mm + 4);
	unsigned long long* vmm = mm + 7;
	// -1: from a flagged side's ends; 0: from a sample; 1: from every key.
	const int first = C->n >= (1ull << 22) ? 0 : 1;
	for (int attempt = sorted->flagged[ci] ? -1 : first; attempt < 2; attempt = std::max(attempt + 1, first)) {
		const uint64_t step = attempt == 0 ? 1024 : 1;
		PG_CUDA(ctx, cudaMemsetAsync(mm, 0, 80, s));
		if (attempt < 0) {
			k_mj_ends<<<1, 1, 0, s>>>((const char*) C->data, C->n, C->width, C->key_off, C->key_bytes, mm);
		} else {
			const int mblocks = (int) std::min<uint64_t>(pg_div_up(pg_div_up(C->n, step), 256), (uint64_t) ctx->sm_count * 8);
			k_mj_minmax<<<mblocks, 256, 0, s>>>((const char*) C->data, C->n, C->width, C->key_off, C->key_bytes, step, mm, nullptr);
		}
		PG_LAUNCHED(ctx);
		unsigned long long h[2];
		PG_CUDA(ctx, cudaMemcpyAsync(h, mm, 16, cudaMemcpyDeviceToHost, s));
		PG_CUDA(ctx, cudaStreamSynchronize(s));
		h[0] = ~h[0];
		if (h[0] > h[1]) continue;                                        // not sorted
		if (step > 1) {
			const unsigned long long slack = (h[1] - h[0]) / 64 + 64;
			h[0] = h[0] > slack ? h[0] - slack : 0;
			h[1] = ~0ull - h[1] > slack ? h[1] + slack : ~0ull;
		}
		const unsigned long long span = h[1] - h[0];
		// A sample's span is at most the exact one: too wide ends both attempts.
		if (span >= MJ_MAX_RANGE || span >= std::max<unsigned long long>(MJ_MIN_RANGE + (MJ_MIN_RANGE >> 4), 16 * C->n)) break;
		const uint32_t range = (uint32_t) span + 1;
		const long long kmin = (long long) (h[0] ^ (1ull << 63));
		// [counts, sums of MJ_SCAN counts, values, listed slices]
		PgScratch tables(ctx, s), copies(ctx, s);
		uint32_t* cnt = nullptr;
		uint64_t* sums = nullptr;
		unsigned long long* val = nullptr;
		const uint64_t nb = pg_div_up(range, MJ_SCAN);
		if (tables.want((void**) &cnt, (uint64_t) range * 4)) return PG_OK;
		unsigned long long* list = nullptr;
		// (A warp with more rows than an output of at most MJ_SLICE_MAX takes needs no list.)
		const uint64_t slices = materialize && out_capacity > MJ_SLICE_MAX ? mj_slices(out_capacity) : 0;
		if (materialize && (tables.want((void**) &sums, nb * 8) || tables.want((void**) &val, C->n * 8) ||
				(slices && tables.want((void**) &list, slices * 8)))) return PG_OK;
		// Rows of more tuples than L2 holds values of: both sides by the top 8 bits of
		// the window first (without memory for the copies, as they are), then a grid that
		// goes through them once, in order, so that the blocks in flight use the same part of
		// the table (the counting pass two: its threads take two tuples half the input apart;
		// side by side 64M tuples over 2^26 keys took 2% longer).
		char* split[2] = {nullptr, nullptr};
		bool parted = false;
		// A side that is sorted is in pieces as it is.
		const bool part = materialize && C->n > MJ_SPLIT_TUPLES && P->n > MJ_SPLIT_TUPLES / 4;
		if (part && (rc = mj_confirm_sorted(ctx, s, R, S, sorted))) return rc;
		const bool csorted = sorted->sorted[ci], psorted = sorted->sorted[pi];
		if (part && (csorted || !copies.want((void**) &split[0], C->n * 16)) &&
				(psorted || !copies.want((void**) &split[1], P->n * 16))) {
			pg_hashfn f = {};
			f.fn = PG_FN_PARAMMODULO;
			f.nbuckets = 256;
			f.min = kmin;
			f.skipbits = range > 256 ? 24 - __builtin_clz(range - 1) : 0;
			f.k = (int64_t) 255 << f.skipbits;
			rc = csorted ? PG_OK : pg_partition_fn(ctx, s, C, f, split[0], nullptr);
			if (!rc && !psorted) rc = pg_partition_fn(ctx, s, P, f, split[1], nullptr);
			if (rc && rc != PG_ERR_OOM) return rc;
			parted = !rc;
			if (rc) cudaGetLastError();
		}
		const char* const cdata = (const char*) (parted && !csorted ? split[0] : C->data);
		const char* const pdata = (const char*) (parted && !psorted ? split[1] : P->data);
		auto grid = [&](uint64_t n, uint32_t per_block, uint32_t per_sm) -> int {
			const uint64_t b = pg_div_up(n, per_block);
			return (int) (parted ? b : std::min<uint64_t>(b, (uint64_t) ctx->sm_count * per_sm));
		};
		PG_CUDA(ctx, cudaMemsetAsync(cnt, 0, (uint64_t) range * 4, s));
		const int cblocks = grid(C->n, 256 * MJ_ILP, MJ_BLOCKS_PER_SM), pblocks = grid(P->n, 256 * MJ_ILP, MJ_BLOCKS_PER_SM);
		// Counted in shared memory where the blocks' own counts fit there and are few
		// beside their tuples.
		const uint64_t shblocks = std::min<uint64_t>(C->n / ((uint64_t) MJ_SHARED_ROWS * range), (uint64_t) ctx->sm_count * 6);
		const bool sh = range <= MJ_SHARED_RANGE && shblocks >= (uint64_t) ctx->sm_count / 2;
#define MJ_COUNT_AS(V, VALS, SH) k_mj_count<V, VALS, SH><<<SH ? (int) shblocks : cblocks, 256, SH ? range * 4 : 0, s>>>(cdata, \
				C->n, C->width, C->key_off, C->key_bytes, kmin, range, cnt, meta + 1, bp, vmm)
#define MJ_COUNT(V, VALS) do { if (sh) MJ_COUNT_AS(V, VALS, true); else MJ_COUNT_AS(V, VALS, false); } while (0)
		if (materialize) MJ_COUNT(true, true);
		else if (mj_v16(C)) MJ_COUNT(true, false);
		else MJ_COUNT(false, false);
#undef MJ_COUNT
#undef MJ_COUNT_AS
		PG_LAUNCHED(ctx);
		if (!materialize) {
			const uint32_t soff = sum_col >= 0 ? pc.off[sum_col] : 0, swords = sum_col >= 0 ? pc.words[sum_col] : 0;
			if (mj_v16(P)) k_mj_lookup<true><<<pblocks, 256, 0, s>>>((const char*) P->data, P->n, 16, P->key_off, 8, soff,
					swords, kmin, range, cnt, agg, ctx->d_status);
			else k_mj_lookup<false><<<pblocks, 256, 0, s>>>((const char*) P->data, P->n, P->width, P->key_off, P->key_bytes,
					soff, swords, kmin, range, cnt, agg, ctx->d_status);
			PG_LAUNCHED(ctx);
		} else {
			k_mj_scan_sums<<<(unsigned) nb, 256, 0, s>>>(cnt, range, sums, meta);
			PG_LAUNCHED(ctx);
			if ((rc = pg_scan_u64(ctx, s, sums, nb, nullptr))) {
				if (rc != PG_ERR_OOM) return rc;
				cudaGetLastError();
				return PG_OK;
			}
			k_mj_scan_apply<<<(unsigned) nb, 256, 0, s>>>(cnt, range, sums);
			PG_LAUNCHED(ctx);
			const int fblocks = grid(C->n, 256, MJ_FILL_BLOCKS_PER_SM);
			k_mj_fill<<<fblocks, 256, 0, s>>>(cdata, C->n, C->key_off, kmin, range, bp, cnt, val, meta, vmm);
			PG_LAUNCHED(ctx);
#define MJ_ROWS(T, SLICE, blocks) do { k_mj_rows<T, SLICE><<<blocks, 256, 0, s>>>(pdata, P->n, P->key_off, kmin, range, cnt, \
				val, wsel, reinterpret_cast<uint4*>(out), out_capacity, agg, meta, vmm, list, slices, mm + 9, ctx->d_status); \
				PG_LAUNCHED(ctx); } while (0)
			const bool two = !parted && C->n / 2 >= range;
			if (two) MJ_ROWS(2, false, grid(P->n, 256 * 2, MJ_ROWS_BLOCKS_PER_SM));
			else MJ_ROWS(4, false, grid(P->n, 256 * 4, MJ_ROWS_BLOCKS_PER_SM));
			const int sblocks = (int) std::min<uint64_t>(pg_div_up(slices, 8), (uint64_t) ctx->sm_count * 6);
			if (slices && two) MJ_ROWS(2, true, sblocks);
			else if (slices) MJ_ROWS(4, true, sblocks);
#undef MJ_ROWS
		}
		unsigned long long o[4];     // rows, sum, (largest count, key outside)
		rc = pg_readback_collected(ctx, s, agg, 3, o, "pg_mpsm_join");
		if (rc) return rc;
		if (o[2] >> 32) continue;                                         // the sample missed a key
		if (materialize && (uint32_t) o[2] > MJ_MAX_RUN) break;
		res->n_out = o[0];
		res->sum = (int64_t) o[1];
		*handled = true;
		if (materialize && o[0] > out_capacity)
			return pg_fail(ctx, PG_ERR_OUTPUT_FULL, "pg_mpsm_join: output capacity too small");
		break;
	}
	return PG_OK;
}

extern "C" int pg_mpsm_join(pg_ctx* ctx, pg_stream stream, const pg_rel* R, const pg_rel* S,
		const pg_col* proj, int nproj, void* out, uint64_t out_capacity,
		int flags, int sum_col, pg_join_result* res)
{
	if (!ctx || !R || !S || !res) return pg_fail(ctx, PG_ERR_ARG, "pg_mpsm_join: null argument");
	for (const pg_rel* r : {R, S}) {
		if (r->n && !r->data) return pg_fail(ctx, PG_ERR_ARG, "pg_mpsm_join: null data");
		if (r->width == 0 || (r->width & 3) || (r->key_bytes != 4 && r->key_bytes != 8) ||
				(r->key_off & 3) || r->key_off + r->key_bytes > r->width)
			return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_mpsm_join: 4-byte-aligned tuples with an int or long key");
	}
	if (nproj < 0 || nproj > MJ_MAX_COLS) return pg_fail(ctx, PG_ERR_ARG, "pg_mpsm_join: 0..16 columns");
	MjCols pc; pc.n = nproj; pc.ow_words = 0;
	for (int i = 0; i < nproj; ++i) {
		const pg_col& c = proj[i];
		uint32_t w = c.side ? S->width : R->width;
		if (c.side > 1 || (c.bytes != 4 && c.bytes != 8) || (c.off & 3) || c.off + c.bytes > w)
			return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_mpsm_join: projected columns must be 4/8 bytes, aligned");
		pc.side[i] = (uint8_t) c.side; pc.off[i] = (uint16_t) c.off; pc.words[i] = (uint8_t) (c.bytes / 4);
		pc.ow_words += c.bytes / 4;
	}
	if (sum_col >= nproj) return pg_fail(ctx, PG_ERR_ARG, "pg_mpsm_join: sum_col out of range");
	if (!(flags & PG_JOIN_SUM)) sum_col = -1;
	const bool materialize = (flags & PG_JOIN_MATERIALIZE) != 0;
	res->n_out = 0; res->sum = 0;
	if (R->n == 0 || S->n == 0) return PG_OK;
	cudaStream_t s = (cudaStream_t) stream;
	int rc;
	MjSorted sorted = {{(flags & PG_JOIN_BUILD_SORTED) != 0, (flags & PG_JOIN_PROBE_SORTED) != 0}, false, {false, false}};
	if (R->n < (1ull << 32) && S->n < (1ull << 32)) {
		bool handled = false;
		if ((rc = mj_dense_join(ctx, s, R, S, pc, sum_col, flags, out, out_capacity, res, &sorted, &handled))) return rc;
		if (handled) return PG_OK;
		if ((rc = mj_confirm_sorted(ctx, s, R, S, &sorted))) return rc;
	}
	const bool r_sorted = sorted.sorted[0], s_sorted = sorted.sorted[1];
	// A sorted 16-byte tuple keyed at offset 0 is its own sorted record array.
	pg_rec *rr = nullptr, *sr = nullptr;
	const bool r_own = !(r_sorted && pg_sort_mode(R) == 0 && !(reinterpret_cast<uintptr_t>(R->data) & 15));
	const bool s_own = !(s_sorted && pg_sort_mode(S) == 0 && !(reinterpret_cast<uintptr_t>(S->data) & 15));
	PgScratch mem(ctx, s);
	if (r_own) { if ((rc = pg_sort_records(ctx, s, R, &rr))) return rc; mem.own(rr); }
	else rr = (pg_rec*) R->data;
	if (s_own) { if ((rc = pg_sort_records(ctx, s, S, &sr))) return rc; mem.own(sr); }
	else sr = (pg_rec*) S->data;
	MjSide RS{rr, (const char*) R->data, R->width, R->key_off, pg_sort_mode(R), nullptr, 0};
	MjSide SS{sr, (const char*) S->data, S->width, S->key_off, pg_sort_mode(S), nullptr, 0};
	uint64_t* starts[2] = {nullptr, nullptr};
	long long* rkeys[2] = {nullptr, nullptr};
	uint64_t nruns[2];
	if ((rc = mj_runs(ctx, s, {rr, sr}, {R->n, S->n}, mem, starts, rkeys, nruns))) return rc;
	uint64_t *rst = starts[0], *sst = starts[1];
	long long *rk = rkeys[0], *sk = rkeys[1];
	RS.run_start = rst; SS.run_start = sst;
	RS.nruns = nruns[0]; SS.nruns = nruns[1];
	uint64_t *counts = nullptr, *match = nullptr;
	unsigned long long* acc = nullptr;  // [total, sum]
	if ((rc = mem.get((void**) &counts, (RS.nruns + 1) * 8))) return rc;
	if ((rc = mem.get((void**) &match, (RS.nruns + 1) * 8))) return rc;
	if ((rc = mem.get((void**) &acc, 16))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(acc, 0, 16, s));
	// One warp per MJ_WARP_RUNS build runs, 8 warps per CTA.
	int blocks = (int) std::min<uint64_t>(pg_div_up(pg_div_up(RS.nruns, MJ_WARP_RUNS), 8), (uint64_t) ctx->sm_count * 16);
	k_match_runs<<<std::max(blocks, 1), 256, 0, s>>>(RS, SS, rk, sk, pc, sum_col, counts, match, acc + 1);
	PG_LAUNCHED(ctx);
	if ((rc = pg_scan_u64(ctx, s, counts, RS.nruns, (uint64_t*) acc))) return rc;
	unsigned long long h[2];
	PG_CUDA(ctx, cudaMemcpyAsync(h, acc, 16, cudaMemcpyDeviceToHost, s));
	if ((rc = pg_check_status(ctx, s, "pg_mpsm_join"))) return rc;
	res->n_out = h[0];
	res->sum = (int64_t) h[1];
	if (materialize && res->n_out) {
		if (res->n_out > out_capacity) {
			rc = pg_fail(ctx, PG_ERR_OUTPUT_FULL, "pg_mpsm_join: output capacity too small");
		} else {
			PG_CUDA(ctx, cudaMemcpyAsync(counts + RS.nruns, &res->n_out, 8, cudaMemcpyHostToDevice, s));
			int wb = (int) std::min<uint64_t>(pg_div_up(pg_div_up(res->n_out, MJ_PER_THREAD), 256), (uint64_t) ctx->sm_count * 16);
			k_mj_write<<<wb, 256, 0, s>>>(RS, SS, pc, counts, match, res->n_out, (char*) out);
			PG_LAUNCHED(ctx);
			rc = pg_check_status(ctx, s, "pg_mpsm_join");
		}
	}
	return rc;
}
