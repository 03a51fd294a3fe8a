// Page sort on sm_103a: LSD radix passes over key - min.
//
// Replaces TupleBuffer::sort<KeyT> (util/buffer.inl:135-292, std::sort on the
// key at keyoffset, reached through sortAllInPage, operators/join.cpp:893-912)
// and the SSE bitonic block sort (util/bitonicsort.cpp:371-443), which sorts
// 4096-record cache blocks with a bitonic network and then merges blocks
// pairwise.
//
// Up to 2^20 tuples take one cooperative launch (k_sort_small); more take stable
// 256-way passes of the partition, over a key window from a sample that the first
// pass checks (radix_passes). Tuples travel as 16-byte records {int64 key, uint64 val}: a
// 16-byte tuple with an 8-byte key is its own record; any other layout sorts (widened
// key, row index) records and gathers rows at the end. The reference's structure, 4096-tuple
// bitonic pages and log2(n/4096) merge passes, each CTA producing 2048 outputs of a
// run pair located by a merge-path binary search (Odeh et al., "Merge Path", 2012), stays
// behind PG_TUNE_SORT_PATH. Ties are left in unspecified
// order, as std::sort leaves them. Unlike the reference's bitonic path (asserting
// power-of-two sizes above 4096 records, util/buffer.cpp:101-104) any n is accepted,
// including n = 4096.
#include "pg_internal.cuh"
#include "pg_sort.cuh"
#include <algorithm>

#define TS_TILE 4096
#define TS_THREADS 512
#define MG_THREADS 256
#define MG_ITEMS 8
#define MG_CHUNK (MG_THREADS * MG_ITEMS)

// Mode: 0 = 16-byte tuple, key at 0; 1 = 16-byte tuple, key at 8; 2 = index records.
__global__ void __launch_bounds__(TS_THREADS)
k_tile_sort(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes,
		int mode, pg_rec* __restrict__ out, bool bulk_ok, int* __restrict__ status)
{
	extern __shared__ __align__(128) unsigned char sm[];
	pg_rec* rec = reinterpret_cast<pg_rec*>(sm);                        // [TS_TILE]
	long long* key = reinterpret_cast<long long*>(rec + TS_TILE);      // [TS_TILE]
	uint16_t* pos = reinterpret_cast<uint16_t*>(key + TS_TILE);        // [TS_TILE]
	__shared__ __align__(8) uint64_t bar;
	const int tid = threadIdx.x;
	const uint64_t base = (uint64_t) blockIdx.x * TS_TILE;
	const uint32_t rows = (uint32_t) pg_min64(TS_TILE, n - base);

	if (mode != 2) {
		const uint32_t bytes = rows * 16;
		if (bulk_ok) {
			if (tid == 0) {
				pg_mbar_init(&bar, 1);
				pg_fence_mbar_init();
				pg_mbar_expect_tx(&bar, bytes);
				pg_bulk_g2s(rec, in + base * 16, bytes, &bar);
			}
			__syncthreads();
			// A wait past the context's limit records PG_ERR_TIMEOUT and then
			// drains the copy; only a copy that never lands ends the block.
			if (!pg_mbar_wait_timed(&bar, 0, pg_spin_knob(status), status)) return;
		} else {
			const uint4* src = reinterpret_cast<const uint4*>(in + base * 16);
			for (uint32_t i = tid; i < rows; i += blockDim.x) reinterpret_cast<uint4*>(rec)[i] = src[i];
		}
		__syncthreads();
		if (mode == 1)
			for (uint32_t i = tid; i < rows; i += blockDim.x) {
				pg_rec r = rec[i];
				rec[i].key = (long long) r.val; rec[i].val = (unsigned long long) r.key;
			}
	} else {
		for (uint32_t i = tid; i < rows; i += blockDim.x) {
			rec[i].key = pg_load_key(in + (base + i) * W + koff, kbytes);
			rec[i].val = base + i;
		}
	}
	__syncthreads();
	for (uint32_t i = tid; i < TS_TILE; i += blockDim.x) {
		key[i] = i < rows ? rec[i].key : 0;
		pos[i] = (uint16_t) i;
	}
	__syncthreads();
	// Bitonic network over (key, pad) with pad = position >= rows, so padding
	// sorts after every real tuple whatever its key.
	for (uint32_t k = 2; k <= TS_TILE; k <<= 1) {
		for (uint32_t j = k >> 1; j > 0; j >>= 1) {
			for (uint32_t t = tid; t < TS_TILE / 2; t += blockDim.x) {
				uint32_t i = 2 * t - (t & (j - 1));
				uint32_t l = i + j;
				long long ki = key[i], kl = key[l];
				uint16_t pi = pos[i], pl = pos[l];
				bool padi = pi >= rows, padl = pl >= rows;
				bool gt = (padi != padl) ? padi : (ki > kl);
				bool asc = (i & k) == 0;
				if (gt == asc) { key[i] = kl; key[l] = ki; pos[i] = pl; pos[l] = pi; }
			}
			__syncthreads();
		}
	}
	for (uint32_t i = tid; i < rows; i += blockDim.x) out[base + i] = rec[pos[i]];
}

__device__ __forceinline__ uint64_t merge_path(const pg_rec* A, uint64_t la, const pg_rec* B, uint64_t lb, uint64_t d)
{
	uint64_t lo = d > lb ? d - lb : 0, hi = d < la ? d : la;
	while (lo < hi) {
		uint64_t mid = (lo + hi) >> 1;
		if (A[mid].key <= B[d - 1 - mid].key) lo = mid + 1; else hi = mid;
	}
	return lo;
}

__global__ void __launch_bounds__(MG_THREADS)
k_merge_pass(const pg_rec* __restrict__ src, pg_rec* __restrict__ dst, uint64_t n, uint64_t L)
{
	__shared__ pg_rec sA[MG_CHUNK];
	__shared__ uint64_t split[2];
	const uint64_t o0 = (uint64_t) blockIdx.x * MG_CHUNK;
	if (o0 >= n) return;
	const uint64_t p0 = o0 / (2 * L) * (2 * L);
	const pg_rec* A = src + p0;
	const uint64_t la = pg_min64(L, n - p0);
	const pg_rec* B = A + la;
	const uint64_t lb = (n - p0 > L) ? pg_min64(L, n - p0 - L) : 0;
	const uint64_t d0 = o0 - p0, d1 = pg_min64(d0 + MG_CHUNK, la + lb);
	if (threadIdx.x < 2) split[threadIdx.x] = merge_path(A, la, B, lb, threadIdx.x ? d1 : d0);
	__syncthreads();
	const uint64_t a0 = split[0], a1 = split[1];
	const uint64_t b0 = d0 - a0, b1 = d1 - a1;
	const uint32_t na = (uint32_t) (a1 - a0), nb = (uint32_t) (b1 - b0);
	// Stage both slices back to back: [A slice][B slice].
	for (uint32_t i = threadIdx.x; i < na + nb; i += blockDim.x)
		sA[i] = i < na ? A[a0 + i] : B[b0 + i - na];
	__syncthreads();
	const pg_rec* xa = sA;
	const pg_rec* xb = sA + na;
	const uint32_t dt = threadIdx.x * MG_ITEMS;
	const uint32_t total = na + nb;
	if (dt >= total) return;
	// Split of this thread's diagonal inside the staged slices.
	uint32_t lo = dt > nb ? dt - nb : 0, hi = dt < na ? dt : na;
	while (lo < hi) {
		uint32_t mid = (lo + hi) >> 1;
		if (xa[mid].key <= xb[dt - 1 - mid].key) lo = mid + 1; else hi = mid;
	}
	uint32_t i = lo, j = dt - lo;
	const uint32_t cnt = pg_min32(MG_ITEMS, total - dt);
	pg_rec* o = dst + o0 + dt;
	for (uint32_t q = 0; q < cnt; ++q) {
		bool takeA = j >= nb || (i < na && xa[i].key <= xb[j].key);
		o[q] = takeA ? xa[i++] : xb[j++];
	}
}

__global__ void k_records_to_tuples(const pg_rec* __restrict__ rec, uint64_t n, int mode,
		const char* __restrict__ in, uint32_t W, char* __restrict__ out)
{
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n;
			i += (uint64_t) gridDim.x * blockDim.x) {
		pg_rec r = rec[i];
		if (mode == 0) reinterpret_cast<pg_rec*>(out)[i] = r;
		else if (mode == 1) {
			pg_rec t; t.key = (long long) r.val; t.val = (unsigned long long) r.key;
			reinterpret_cast<pg_rec*>(out)[i] = t;
		} else {
			if (((W | reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 7) == 0) {
				const uint2* s = reinterpret_cast<const uint2*>(in + r.val * W);
				uint2* d = reinterpret_cast<uint2*>(out + i * W);
				#pragma unroll 4
				for (uint32_t w = 0; w < W / 8; ++w) d[w] = s[w];
				continue;
			}
			const uint32_t* s = reinterpret_cast<const uint32_t*>(in + r.val * W);
			uint32_t* d = reinterpret_cast<uint32_t*>(out + i * W);
			#pragma unroll 4
			for (uint32_t w = 0; w < W / 4; ++w) d[w] = s[w];
		}
	}
}

// ---------------------------------------------------------------------------
// LSD radix path: ceil(bits / d) stable 2^d-way partitions on successive d-bit
// digits of (key - min), d = 8 or the PG_TUNE_RADIX_BITS knob (4..12), sort the
// tuples (pg_partition.cu; each pass reads them twice and writes them once). This
// is ParameterizedModuloValueHasher::generate's multi-pass radix split
// (hash.cpp:237-267) driven to completion. Ties keep input order.
// ---------------------------------------------------------------------------
__global__ void k_sort_minmax(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff,
		uint32_t kbytes, uint64_t step, unsigned long long* __restrict__ mm)
{
	unsigned long long lo = ~0ull, hi = 0;
	for (uint64_t i = (blockIdx.x * (uint64_t) blockDim.x + threadIdx.x) * step; i < n;
			i += (uint64_t) gridDim.x * blockDim.x * step) {
		const unsigned long long u = (unsigned long long) pg_load_key(in + i * W + koff, kbytes) ^ (1ull << 63);
		lo = u < lo ? u : lo;
		hi = u > hi ? u : hi;
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		const unsigned long long a = __shfl_down_sync(0xffffffffu, lo, o), b = __shfl_down_sync(0xffffffffu, hi, o);
		lo = a < lo ? a : lo;
		hi = b > hi ? b : hi;
	}
	if ((threadIdx.x & 31) == 0) { atomicMax(&mm[0], ~lo); atomicMax(&mm[1], hi); }      // zero before
}

// (key, other half) or (key, row index) records for layouts other than a
// 16-byte tuple keyed at offset 0.
__global__ void k_make_records(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff,
		uint32_t kbytes, int mode, pg_rec* __restrict__ out)
{
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n;
			i += (uint64_t) gridDim.x * blockDim.x) {
		pg_rec r;
		if (mode == 1) {
			const pg_rec t = reinterpret_cast<const pg_rec*>(in)[i];
			r.key = (long long) t.val; r.val = (unsigned long long) t.key;
		} else {
			r.key = pg_load_key(in + i * W + koff, kbytes);
			r.val = i;
		}
		out[i] = r;
	}
}

// Smallest and largest key of rows 0, step, 2 step, ... (step 1: every row),
// sign bit flipped (unsigned order = signed order). One host round trip.
static int sort_key_range(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint64_t step, unsigned long long (&h)[2])
{
	int rc;
	unsigned long long* mm = nullptr;
	if ((rc = pg_alloc_async(ctx, s, (void**) &mm, 16))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(mm, 0, 16, s));
	const int blocks = (int) std::min<uint64_t>(pg_div_up(pg_div_up(in->n, step), 256), (uint64_t) ctx->sm_count * 8);
	k_sort_minmax<<<blocks, 256, 0, s>>>((const char*) in->data, in->n, in->width, in->key_off, in->key_bytes, step, mm);
	PG_LAUNCHED(ctx);
	PG_CUDA(ctx, cudaMemcpyAsync(h, mm, 16, cudaMemcpyDeviceToHost, s));
	PG_CUDA(ctx, cudaStreamSynchronize(s));
	pg_free_async(ctx, s, mm);
	h[0] = ~h[0];
	return PG_OK;
}

static int bits_of(unsigned long long x) { return x == 0 ? 0 : 64 - __builtin_clzll(x); }

// ---------------------------------------------------------------------------
// Up to SS_MAX_ROWS 16-byte tuples in one cooperative launch: key range, then
// as many 8-bit LSD passes as the range needs, with grid barriers where the
// multi-launch form has launches and a host round trip. The rows stay in L2
// between passes; every block holds its rows in registers, ranks them as
// k_part_sweep does, publishes its bucket counts, adds up the other blocks'
// and stores each row at its place. Bound by the barriers and L2 round trips of
// its passes. Whole calls: 5000 rows of 20 bits 92 -> 45 us and 200,000 of 24 bits 140
// -> 56 us (a launch or three a pass before), 200,000 of 50 bits 213 -> 97 us (bitonic
// tiles and merges before). Ties keep input order.
// ---------------------------------------------------------------------------
#define SS_THREADS 1024
#define SS_WARPS (SS_THREADS / 32)
#define SS_MAX_ROWS (1u << 20)

__device__ __forceinline__ unsigned long long ss_key(const uint4& t, uint32_t kw, uint32_t kbytes)
{
	const uint32_t lo = kw == 0 ? t.x : kw == 1 ? t.y : kw == 2 ? t.z : t.w;
	const uint32_t hi = kw == 0 ? t.y : kw == 1 ? t.z : t.w;
	const long long k = kbytes == 4 ? (long long) (int32_t) lo : (long long) (((unsigned long long) hi << 32) | lo);
	return (unsigned long long) k ^ (1ull << 63);             // unsigned order = signed order
}

// mm: [~smallest, largest] key, zero before; counts: [blocks][256].
template <int ITEMS>
__global__ void __launch_bounds__(SS_THREADS, 1)
k_sort_small(const uint4* __restrict__ in, uint32_t n, uint32_t kw, uint32_t kbytes, uint4* out, uint4* tmp,
		unsigned long long* mm, uint32_t* bar, uint32_t* counts, int* __restrict__ status)
{
	__shared__ uint16_t cnt[SS_WARPS][256];        // a warp's rows of a bucket, then its first of the block's
	__shared__ uint32_t part[2][4][256];
	__shared__ uint32_t base[256];
	__shared__ unsigned long long red[2][SS_WARPS];
	__shared__ uint32_t wt[8];
	const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, c = blockIdx.x;
	const uint32_t spin = pg_spin_knob(status);
	uint32_t epoch = 0;
	bool dead = false;
	const uint32_t r0 = c * (SS_THREADS * ITEMS) + warp * (32 * ITEMS) + lane;      // item j: row r0 + 32 j
	uint4 t[ITEMS];
	unsigned long long lo = ~0ull, hi = 0;
	#pragma unroll
	for (int j = 0; j < ITEMS; ++j) {
		if (r0 + j * 32 >= n) continue;
		t[j] = __ldcs(in + r0 + j * 32);
		const unsigned long long u = ss_key(t[j], kw, kbytes);
		lo = min(lo, u);
		hi = max(hi, u);
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
		hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
	}
	if (lane == 0) { red[0][warp] = lo; red[1][warp] = hi; }
	__syncthreads();
	lo = red[0][lane]; hi = red[1][lane];
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
		hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
	}
	if (G > 1) {
		if (tid == 0) { atomicMax(&mm[0], ~lo); atomicMax(&mm[1], hi); }
		pg_grid_sync(bar, epoch, dead, spin, status);
		// One thread's look for the whole block: past a barrier that was given up on the
		// range still changes, and the block's threads must make the same passes.
		if (tid == 0) { red[0][0] = ~pg_ld_relaxed(mm); red[1][0] = pg_ld_relaxed(mm + 1); }
		__syncthreads();
		lo = red[0][0];
		hi = red[1][0];
	}
	const unsigned long long span = hi - lo;
	const int passes = span ? (64 - __clzll((long long) span) + 7) / 8 : 0;
	if (!passes) {
		#pragma unroll
		for (int j = 0; j < ITEMS; ++j)
			if (r0 + j * 32 < n) out[r0 + j * 32] = t[j];
		return;
	}
	for (int p = 0; p < passes; ++p) {
		uint4* const dst = (passes - 1 - p) % 2 == 0 ? out : tmp;
		for (uint32_t i = tid; i < SS_WARPS * 128; i += SS_THREADS) reinterpret_cast<uint32_t*>(cnt)[i] = 0;
		__syncthreads();
		uint32_t br[ITEMS];                        // bucket, rank in the warp's rows of it << 8
		#pragma unroll
		for (int j = 0; j < ITEMS; ++j) {
			const bool mine = r0 + j * 32 < n;
			const uint32_t b = mine ? (uint32_t) ((ss_key(t[j], kw, kbytes) - lo) >> (8 * p)) & 255u : 0;
			uint32_t peers = __ballot_sync(0xffffffffu, mine);
			#pragma unroll
			for (int k = 0; k < 8; ++k) {
				const bool on = (b >> k) & 1u;
				const uint32_t m = __ballot_sync(0xffffffffu, on);
				peers &= on ? m : ~m;
			}
			const uint32_t at = cnt[warp][b], below = __popc(peers & ((1u << lane) - 1));
			__syncwarp();
			if (mine && below == 0) cnt[warp][b] = (uint16_t) (at + __popc(peers));
			__syncwarp();
			br[j] = b | ((at + below) << 8);
		}
		__syncthreads();
		// Four threads a bucket: a quarter of the warps, then of the blocks, each.
		const uint32_t b = tid & 255, q = tid >> 8;
		{
			uint32_t x[SS_WARPS / 4], sum = 0;
			#pragma unroll
			for (int w = 0; w < SS_WARPS / 4; ++w) { x[w] = cnt[q * (SS_WARPS / 4) + w][b]; sum += x[w]; }
			part[0][q][b] = sum;
			__syncthreads();
			uint32_t at = 0;
			for (uint32_t k = 0; k < q; ++k) at += part[0][k][b];
			#pragma unroll
			for (int w = 0; w < SS_WARPS / 4; ++w) { cnt[q * (SS_WARPS / 4) + w][b] = (uint16_t) at; at += x[w]; }
			if (q == 3) {
				if (G > 1) counts[c * 256 + b] = at;
				else part[1][0][b] = at;
			}
		}
		uint32_t total = 0, before = 0;
		if (G > 1) {
			pg_grid_sync(bar, epoch, dead, spin, status);
			#pragma unroll 8
			for (uint32_t k = q; k < G; k += 4) {
				const uint32_t x = __ldcg(counts + k * 256 + b);
				total += x;
				before += k < c ? x : 0;
			}
			part[0][q][b] = total;
			part[1][q][b] = before;
		}
		__syncthreads();
		if (tid < 256) {
			if (G > 1) {
				total = part[0][0][b] + part[0][1][b] + part[0][2][b] + part[0][3][b];
				before = part[1][0][b] + part[1][1][b] + part[1][2][b] + part[1][3][b];
			} else total = part[1][0][b];
			uint32_t inc = total;
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
				if (lane >= (uint32_t) o) inc += y;
			}
			if (lane == 31) wt[warp] = inc;
			asm volatile("bar.sync 1, 256;" ::: "memory");
			for (uint32_t w = 0; w < warp; ++w) inc += wt[w];
			base[b] = inc - total + before;
		}
		__syncthreads();
		#pragma unroll
		for (int j = 0; j < ITEMS; ++j) {
			if (r0 + j * 32 >= n) continue;
			const uint32_t d = br[j] & 255, row = base[d] + cnt[warp][d] + (br[j] >> 8);
			if (row < n) __stcg(dst + row, t[j]);
		}
		if (p + 1 == passes) return;
		pg_grid_sync(bar, epoch, dead, spin, status);
		#pragma unroll
		for (int j = 0; j < ITEMS; ++j)
			if (r0 + j * 32 < n) t[j] = __ldcg(dst + r0 + j * 32);
	}
}

static int sort_small(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, void* out, void* tmp)
{
	const uint32_t n = (uint32_t) in->n;
	const bool four = n <= (uint32_t) ctx->sm_count * SS_THREADS * 4;
	const uint32_t G = (uint32_t) pg_div_up(n, SS_THREADS * (four ? 4 : 8));
	int rc;
	char* mem = nullptr;                   // [smallest, largest, barrier], [G][256] counts
	if ((rc = pg_alloc_async(ctx, s, (void**) &mem, 64 + (size_t) G * 1024))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(mem, 0, 64, s));
	const uint4* src = (const uint4*) in->data;
	uint4 *o = (uint4*) out, *t = (uint4*) tmp;
	uint32_t nn = n, kw = in->key_off / 4, kb = in->key_bytes;
	unsigned long long* mm = reinterpret_cast<unsigned long long*>(mem);
	uint32_t *bar = reinterpret_cast<uint32_t*>(mem + 16), *counts = reinterpret_cast<uint32_t*>(mem + 64);
	void* args[] = {&src, &nn, &kw, &kb, &o, &t, &mm, &bar, &counts, &ctx->d_status};
	PG_CUDA(ctx, cudaLaunchCooperativeKernel(four ? (void*) k_sort_small<4> : (void*) k_sort_small<8>, dim3(G), dim3(SS_THREADS),
			args, 0, s));
	PG_LAUNCHED(ctx);
	pg_free_async(ctx, s, mem);
	return PG_OK;
}

// The passes over the low `bits` bits of key - base, the last into `out`. With
// `refuted`, the first one confirms that no key lies outside.
static int radix_passes(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, int64_t base, int bits, void* out, void* tmp,
		bool* refuted)
{
	const int passes = (bits + 7) / 8;
	pg_rel cur = *in;
	for (int p = 0; p < passes; ++p) {
		void* dst = (passes - 1 - p) % 2 == 0 ? out : tmp;
		if (int rc = pg_radix_pass(ctx, s, &cur, base, p, bits, p == 0 ? refuted : nullptr, dst)) return rc;
		if (p == 0 && refuted && *refuted) return PG_OK;
		cur.data = dst;
	}
	return PG_OK;
}

// Sorts `in` into `out` by radix passes when the key span allows; returns
// PG_OK with *done = false (nothing queued) when it does not. `tmp` holds n
// tuples of scratch; `range`: the key range (sort_key_range), where it is known.
static int radix_sort(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, void* out, void* tmp, const unsigned long long* range,
		bool* done)
{
	*done = false;
	const uint64_t n = in->n;
	if (n == 0 || n >= (1ull << 32)) return PG_OK;
	const int64_t path = ctx->tune[PG_TUNE_SORT_PATH];
	if (path == 2) return PG_OK;
	const int64_t tb = ctx->tune[PG_TUNE_RADIX_BITS];
	const int digit = tb >= 4 && tb <= 12 ? (int) tb : 8;
	const bool sweep = digit == 8 && pg_radix_pass_takes(in, out) && pg_radix_pass_takes(in, tmp);
	if (path == 0 && tb == 0 && sweep && n <= SS_MAX_ROWS && n <= (uint64_t) ctx->sm_count * SS_THREADS * 8) {
		*done = true;
		return sort_small(ctx, s, in, out, tmp);
	}
	int rc;
	unsigned long long h[2];
	if (sweep && n >= (1ull << 22) && !range) {
		// Large inputs: the window of the digits from every 1024th row, checked
		// by the first pass, instead of a pass for the exact
		// range: the aligned power of two around the sample, or the sample
		// widened by 1/256 a side, whichever needs no more passes than the
		// sample's own span.
		if ((rc = sort_key_range(ctx, s, in, 1024, h))) return rc;
		const unsigned long long span = h[1] - h[0], slack = span / 256 + 64;
		const int want = (bits_of(span) + 7) / 8, ab = bits_of(h[0] ^ h[1]);
		const unsigned long long lo = h[0] > slack ? h[0] - slack : 0, hi = ~0ull - h[1] > slack ? h[1] + slack : ~0ull;
		const int wb = bits_of(hi - lo);
		unsigned long long base = 0;
		int bits = 0;
		if ((ab + 7) / 8 == want) { bits = ab; base = ab == 64 ? 0 : h[0] >> ab << ab; }
		else if ((wb + 7) / 8 == want) { bits = wb; base = lo; }
		if (bits) {
			bool refuted = false;
			if ((rc = radix_passes(ctx, s, in, (int64_t) (base ^ (1ull << 63)), bits, out, tmp, &refuted))) return rc;
			if (!refuted) { *done = true; return PG_OK; }
		}
	}
	if (range) { h[0] = range[0]; h[1] = range[1]; }
	else if ((rc = sort_key_range(ctx, s, in, 1, h))) return rc;
	const int bits = bits_of(h[1] - h[0]);
	// Tuples that k_part_sweep does not take (other widths, unaligned, other digits) go
	// by a digit function that masks a signed difference: up to 63 bits. Wider spans go to
	// the bitonic tiles and merge-path merges, and so do up to 2^18 of them whose span needs
	// more than four 8-bit passes: the few merges cost less there.
	if (bits > 63 && !sweep) return PG_OK;
	if (path == 0 && bits > 32 && n <= (1ull << 18)) return PG_OK;
	const long long kmin = (long long) (h[0] ^ (1ull << 63));
	if (bits == 0) {   // one key value: already sorted
		PG_CUDA(ctx, cudaMemcpyAsync(out, in->data, n * in->width, cudaMemcpyDeviceToDevice, s));
		*done = true;
		return PG_OK;
	}
	if (sweep) {
		if ((rc = radix_passes(ctx, s, in, kmin, bits, out, tmp, nullptr))) return rc;
		*done = true;
		return PG_OK;
	}
	const int passes = (bits + digit - 1) / digit;
	pg_rel cur = *in;
	for (int p = 0; p < passes; ++p) {
		pg_hashfn f;
		f.fn = PG_FN_PARAMMODULO;
		f.skipbits = digit * p;
		f.k = (int64_t) ((1u << digit) - 1) << f.skipbits;
		f.min = kmin;
		f.max = 0; f.bucketrange = 0;
		f.nbuckets = 1u << digit;
		void* dst = ((passes - 1 - p) % 2 == 0) ? out : tmp;
		if ((rc = pg_partition_fn(ctx, s, &cur, f, dst, nullptr))) return rc;
		cur.data = dst;
	}
	*done = true;
	return PG_OK;
}

int pg_sort_mode(const pg_rel* r)
{
	if (r->width == 16 && r->key_bytes == 8 && r->key_off == 0) return 0;
	if (r->width == 16 && r->key_bytes == 8 && r->key_off == 8) return 1;
	return 2;
}

// Sorts `in` into records; *recs receives a pool allocation of n records
// (caller frees with pg_free_async on stream s).
static int sort_records(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, const unsigned long long* range, pg_rec** recs)
{
	const uint64_t n = in->n;
	int rc;
	const int mode = pg_sort_mode(in);
	PgScratch mem(ctx, s);
	pg_rec *a = nullptr, *b = nullptr;
	if ((rc = mem.get((void**) &a, n * sizeof(pg_rec)))) return rc;
	if (n == 0) { *recs = (pg_rec*) mem.keep(a); return PG_OK; }
	{
		// Radix path: sort 16-byte records (the tuples themselves when the
		// layout is a 16-byte tuple keyed at 0).
		pg_rec* src = nullptr;
		pg_rel r = *in;
		if (mode != 0) {
			if ((rc = mem.get((void**) &src, n * sizeof(pg_rec)))) return rc;
			const int blocks = (int) std::min<uint64_t>(pg_div_up(n, 256), (uint64_t) ctx->sm_count * 16);
			k_make_records<<<blocks, 256, 0, s>>>((const char*) in->data, n, in->width, in->key_off,
					in->key_bytes, mode, src);
			PG_LAUNCHED(ctx);
			r.data = src; r.width = 16; r.key_off = 0; r.key_bytes = 8;
		}
		if ((rc = mem.get((void**) &b, n * sizeof(pg_rec)))) return rc;
		bool done = false;
		if ((rc = radix_sort(ctx, s, &r, a, b, range, &done))) return rc;
		mem.drop(b);
		b = nullptr;
		mem.drop(src);
		if (done) { *recs = (pg_rec*) mem.keep(a); return PG_OK; }
	}
	const uint64_t tiles = pg_div_up(n, TS_TILE);
	const size_t smem = TS_TILE * (sizeof(pg_rec) + 8 + 2);
	PG_CUDA(ctx, cudaFuncSetAttribute(k_tile_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
	const bool bulk_ok = mode != 2 && (reinterpret_cast<uintptr_t>(in->data) & 15) == 0;
	k_tile_sort<<<(unsigned) tiles, TS_THREADS, smem, s>>>((const char*) in->data, n, in->width, in->key_off,
			in->key_bytes, mode, a, bulk_ok, ctx->d_status);
	PG_LAUNCHED(ctx);
	if (n > TS_TILE) {
		if ((rc = mem.get((void**) &b, n * sizeof(pg_rec)))) return rc;
		const unsigned blocks = (unsigned) pg_div_up(n, MG_CHUNK);
		for (uint64_t L = TS_TILE; L < n; L <<= 1) {
			k_merge_pass<<<blocks, MG_THREADS, 0, s>>>(a, b, n, L);
			PG_LAUNCHED(ctx);
			std::swap(a, b);
		}
	}
	*recs = (pg_rec*) mem.keep(a);
	return PG_OK;
}

int pg_sort_records(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, pg_rec** recs)
{
	return sort_records(ctx, s, in, nullptr, recs);
}

// Passes over the tuples themselves, by their width, that cost no more than sorting
// (key, row) records and gathering the tuples. Both read the exact key range first. A
// pass over 20M tuples takes 290 us (8 bytes), 350 (12), 500 (24) or 700 (40); over the
// records 205 to 270, with 480 to 950 to make them and gather. 20M tuples, tuples against
// records: 8 bytes, 2 and 4 passes 628 against 889 us, 1163 against 1298; 12 bytes, 2: 707
// and 1005; 24 bytes, 1 to 4: 574, 1029, 1481, 1935 and 955, 1210, 1567, 1776; 40 bytes, 3:
// 2136 and 1760; 3M of 200 bytes, 2: 924 and 1156, of 100, 3: 819 and 771. Up to 2^20
// records take one launch, and only the gather of wide tuples costs more: 1M of 100 bytes,
// 1 and 2 passes 166 and 267 against 217 and 240; of 200, 2: 386 each; of 400, 1 and 2: 422
// and 771 against 661 and 678. Below 40 MB the round trip for the range costs more than that.
#define SORT_TUPLE_WIDTH 400        // of which the partition's smallest tiles of 256 fit shared memory
static int sort_tuple_passes(uint32_t width, uint64_t n)
{
	if (n <= SS_MAX_ROWS) return n * width < (40ull << 20) ? -1 : width > 128 && width <= 256 ? 2 : 1;
	return width <= 8 ? 5 : width <= 12 ? 4 : width <= 24 ? 3 : 2;
}

// Radix passes over the tuples. *done = false: not taken (the key span, or no memory).
static int sort_tuples(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, void* out, const unsigned long long* range, bool* done)
{
	PgScratch mem(ctx, s);
	void* tmp = nullptr;
	*done = false;
	if (mem.want(&tmp, in->n * in->width)) return PG_OK;
	const int rc = radix_sort(ctx, s, in, out, tmp, range, done);
	if (rc != PG_ERR_OOM) return rc;
	cudaGetLastError();
	*done = false;
	return PG_OK;
}

extern "C" int pg_sort_pages(pg_ctx* ctx, pg_stream stream, const pg_rel* in, void* out)
{
	if (!ctx || !in) return pg_fail(ctx, PG_ERR_ARG, "pg_sort_pages: null argument");
	if (in->n && (!in->data || !out)) return pg_fail(ctx, PG_ERR_ARG, "pg_sort_pages: null data");
	if (in->width == 0 || (in->width & 3) || (in->key_bytes != 4 && in->key_bytes != 8) ||
			(in->key_off & 3) || in->key_off + in->key_bytes > in->width)
		return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_sort_pages: 4-byte-aligned tuples with an int or long key");
	if (in->data == out && in->n) return pg_fail(ctx, PG_ERR_ARG, "pg_sort_pages: output may not alias input");
	cudaStream_t s = (cudaStream_t) stream;
	if (in->n == 0) return PG_OK;
	pg_rec* recs = nullptr;
	int rc;
	// 16-byte tuples sort themselves; others too where that takes few passes (knob 1:
	// always), else as (key, row) records with the tuples gathered at the end. Up to 2^20
	// records sort in one launch. Without memory for one form the other is tried.
	const int64_t path = ctx->tune[PG_TUNE_SORT_PATH];
	bool tuples = in->width == 16 || path == 1, done = false;
	unsigned long long h[2];
	const unsigned long long* range = nullptr;
	if (!tuples && path == 0 && in->width <= SORT_TUPLE_WIDTH && in->n < (1ull << 32)) {
		const int passes = sort_tuple_passes(in->width, in->n);
		if (passes > 0) {
			if ((rc = sort_key_range(ctx, s, in, 1, h))) return rc;
			range = h;
			tuples = (bits_of(h[1] - h[0]) + 7) / 8 <= passes;
		}
	}
	if (tuples) {
		if ((rc = sort_tuples(ctx, s, in, out, range, &done))) return rc;
		if (done) return pg_check_status(ctx, s, "pg_sort_pages");
	}
	rc = sort_records(ctx, s, in, range, &recs);
	if (rc == PG_ERR_OOM && !tuples && path == 0 && in->width <= SORT_TUPLE_WIDTH) {
		cudaGetLastError();
		int rt = sort_tuples(ctx, s, in, out, range, &done);
		if (rt || done) return rt ? rt : pg_check_status(ctx, s, "pg_sort_pages");
	}
	if (rc) return rc;
	const int mode = pg_sort_mode(in);
	int blocks = (int) std::min<uint64_t>(pg_div_up(in->n, 256), (uint64_t) ctx->sm_count * 16);
	k_records_to_tuples<<<blocks, 256, 0, s>>>(recs, in->n, mode, (const char*) in->data, in->width, (char*) out);
	PG_LAUNCHED(ctx);
	pg_free_async(ctx, s, recs);
	return pg_check_status(ctx, s, "pg_sort_pages");
}

extern "C" int pg_partition_sort(pg_ctx* ctx, pg_stream stream, const pg_rel* data,
		const uint64_t* offsets_host, uint32_t nbuckets, void* scratch_out)
{
	if (!ctx || !data || !offsets_host || !scratch_out)
		return pg_fail(ctx, PG_ERR_ARG, "pg_partition_sort: null argument");
	cudaStream_t s = (cudaStream_t) stream;
	for (uint32_t b = 0; b < nbuckets; ++b) {
		pg_rel part = *data;
		part.data = (const char*) data->data + offsets_host[b] * data->width;
		part.n = offsets_host[b + 1] - offsets_host[b];
		if (part.n == 0) continue;
		int rc = pg_sort_pages(ctx, stream, &part, (char*) scratch_out + offsets_host[b] * data->width);
		if (rc) return rc;
	}
	PG_CUDA(ctx, cudaMemcpyAsync((void*) data->data, scratch_out, data->n * data->width, cudaMemcpyDeviceToDevice, s));
	return pg_check_status(ctx, s, "pg_partition_sort");
}
