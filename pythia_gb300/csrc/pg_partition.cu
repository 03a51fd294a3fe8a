// Stable range/radix partitioning on sm_103a.
//
// Replaces PartitionOp's three phases (operators/partition.cpp:166-359):
// histogram (copySourceIntoPageAndPopulateHistogram, :166-200), per-partition
// prefix over workers (:292-307) and the stable scatter (repartition,
// :250-268). The reference's "workers" become CTAs: CTA c owns a contiguous
// chunk of the input, so the output order within a partition is input order,
// exactly what the reference produces when its threads read consecutive
// slices.
//
// 16-byte tuples and at most 256 buckets (sw_wins): k_chunk_hist counts tuples per (bucket,
// block), an exclusive scan over the bucket-major counts gives every block its first
// output slot per bucket, and k_part_sweep streams the block's tiles again, ranks
// their tuples and stores each bucket's rows of a tile as one run.
//
// Other widths and fan-outs: k_part_hist counts and k_part_scatter moves tiles staged
// in shared memory by bulk copies (cp.async.bulk + mbarrier, double-buffered). It ranks
// tuples within the tile per bucket (per-warp ballots over the bucket bits + per-warp
// counters, which keeps the order stable) and writes each tile out grouped by bucket, so a
// warp's stores go to consecutive addresses of one partition (write-combining through
// shared memory).
#include "pg_internal.cuh"
#include <algorithm>
#include <type_traits>

#define PART_MAX_BUCKETS 4096
#define PART_TILE_BYTES (20 * 1024)     // measured best: 4 CTAs per SM

// Bucket of the key at p: the radix function (parammodulo, the sort's
// digits) inlined when FN says so, else the general bucket function.
#define PART_FN_ANY (-1)
template <int FN>
__device__ __forceinline__ uint32_t part_bucket(const pg_hashfn& f, const char* p, uint32_t kbytes)
{
	if (FN == PG_FN_PARAMMODULO) {
		const int64_t v = pg_load_key(p, kbytes);
		return (uint32_t) (((v - f.min) & f.k) >> f.skipbits);
	}
	if (FN == PG_FN_MIXRADIX) return (uint32_t) (pg_mix64((uint64_t) pg_load_key(p, kbytes)) >> f.skipbits);
	return pg_hash_field(f, p, kbytes);
}

template <int FN>
__global__ void k_part_hist(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff,
		uint32_t kbytes, pg_hashfn f, uint32_t tile, uint64_t tiles_per_cta,
		uint64_t* __restrict__ counts, uint32_t G, int* __restrict__ status)
{
	extern __shared__ uint32_t hist[];
	const uint32_t B = f.nbuckets;
	for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) hist[b] = 0;
	__syncthreads();
	uint64_t lo = (uint64_t) blockIdx.x * tiles_per_cta * tile;
	uint64_t hi = std::min<uint64_t>(n, lo + tiles_per_cta * tile);
	bool bad = false;
	for (uint64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
		uint32_t b = part_bucket<FN>(f, in + i * W + koff, kbytes);
		if (b < B) atomicAdd(&hist[b], 1u); else bad = true;
	}
	if (bad) pg_set_status(status, PG_ERR_ARG);
	__syncthreads();
	for (uint32_t b = threadIdx.x; b < B; b += blockDim.x)
		counts[(uint64_t) b * G + blockIdx.x] = hist[b];
}

// Copies `bytes` from global to shared with 4-byte words (fallback path for
// tiles a bulk copy cannot take: unaligned base or ragged tail).
__device__ __forceinline__ void part_copy_words(uint32_t* dst, const uint32_t* src, uint32_t words)
{
	for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

// NBITS > 0: the bucket index has exactly NBITS bits (ranking loop unrolled).
template <int NW, int FN, int NBITS>
__global__ void __launch_bounds__(NW * 32)
k_part_scatter(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes,
		pg_hashfn f, uint32_t tile, uint64_t tiles_per_cta, const uint64_t* __restrict__ offs,
		uint32_t G, char* __restrict__ out, bool bulk_ok, int* __restrict__ status)
{
	extern __shared__ __align__(128) unsigned char smem[];
	const uint32_t B = f.nbuckets;
	const uint32_t tile_bytes = tile * W;
	unsigned char* buf0 = smem;
	unsigned char* buf1 = smem + tile_bytes;
	uint16_t* cnt = reinterpret_cast<uint16_t*>(smem + 2 * tile_bytes);        // [NW][B]
	uint32_t* tstart = reinterpret_cast<uint32_t*>(cnt + NW * B);               // [B]
	uint32_t* delta = tstart + B;                                                // [B]
	uint32_t* running = delta + B;                                               // [B]
	uint16_t* inv = reinterpret_cast<uint16_t*>(running + B);                   // [tile]
	uint16_t* bkt = inv + tile;                                                  // [tile]
	uint64_t* bar = reinterpret_cast<uint64_t*>(
			(reinterpret_cast<uintptr_t>(bkt + tile) + 15) & ~uintptr_t(15));     // [2]
	__shared__ uint32_t warp_sums[32];
	__shared__ uint32_t carry;

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const uint32_t nbits = NBITS > 0 ? NBITS : (B > 1 ? 32 - __clz(B - 1) : 0);
	const uint64_t first = (uint64_t) blockIdx.x * tiles_per_cta;
	const uint64_t ntiles_total = pg_div_up(n, tile);
	const uint64_t last = std::min<uint64_t>(ntiles_total, first + tiles_per_cta);
	if (first >= last) return;

	for (uint32_t b = tid; b < B; b += blockDim.x) running[b] = (uint32_t) offs[(uint64_t) b * G + blockIdx.x];
	for (uint32_t i = tid; i < NW * B; i += blockDim.x) cnt[i] = 0;
	if (tid == 0) { pg_mbar_init(&bar[0], 1); pg_mbar_init(&bar[1], 1); pg_fence_mbar_init(); }
	__syncthreads();

	// Issue the load of tile t into buffer (t & 1). Bulk copies only for
	// whole, 16-byte multiple tiles; the rest are copied by the threads.
	auto tile_rows = [&](uint64_t t) -> uint32_t {
		return (uint32_t) std::min<uint64_t>(tile, n - t * tile);
	};
	auto issue = [&](uint64_t t) {
		uint32_t rows = tile_rows(t);
		uint32_t bytes = rows * W;
		unsigned char* dst = (t & 1) ? buf1 : buf0;
		const char* src = in + t * (uint64_t) tile * W;
		if (bulk_ok && (bytes & 15) == 0) {
			if (tid == 0) {
				pg_mbar_expect_tx(&bar[t & 1], bytes);
				pg_bulk_g2s(dst, src, bytes, &bar[t & 1]);
			}
			return true;
		}
		return false;
	};
	uint32_t phase[2] = {0, 0};
	const uint32_t spin = pg_spin_knob(status);
	bool bulk_pending = issue(first);

	for (uint64_t t = first; t < last; ++t) {
		const uint32_t rows = tile_rows(t);
		unsigned char* cur = (t & 1) ? buf1 : buf0;
		if (bulk_pending) {
			if (!pg_mbar_wait_timed(&bar[t & 1], phase[t & 1], spin, status)) return;
			phase[t & 1] ^= 1;
		} else {
			part_copy_words(reinterpret_cast<uint32_t*>(cur),
					reinterpret_cast<const uint32_t*>(in + t * (uint64_t) tile * W), rows * W / 4);
		}
		__syncthreads();
		// Prefetch the next tile into the other buffer while this one is ranked.
		bool next_bulk = false;
		if (t + 1 < last) next_bulk = issue(t + 1);

		// (1) rank within the tile: warp w owns rows [w*sub, (w+1)*sub).
		// Lanes with the same bucket are found with one ballot per bucket
		// bit (the bucket index has nbits bits): cheaper than a match over
		// 32-bit values, with the same peer masks.
		const uint32_t sub = tile / NW;
		uint16_t* mycnt = cnt + warp * B;
		for (uint32_t it = 0; it < sub; it += 32) {
			uint32_t p = warp * sub + it + lane;
			bool valid = p < rows;
			uint32_t b = valid ? part_bucket<FN>(f, reinterpret_cast<const char*>(cur) + (uint64_t) p * W + koff, kbytes) : 0u;
			if (valid && b >= B) { pg_set_status(status, PG_ERR_ARG); b = 0; }
			uint32_t peers = __ballot_sync(0xffffffffu, valid);
			#pragma unroll
			for (uint32_t k = 0; k < (NBITS > 0 ? (uint32_t) NBITS : nbits); ++k) {
				const bool on = (b >> k) & 1u;
				const uint32_t m = __ballot_sync(0xffffffffu, on);
				peers &= on ? m : ~m;
			}
			uint32_t leader = __ffs(peers) - 1;
			uint32_t below = peers & ((1u << lane) - 1);
			uint32_t old = 0;
			if (valid && lane == leader) {
				old = mycnt[b];
				mycnt[b] = (uint16_t) (old + __popc(peers));
			}
			old = __shfl_sync(0xffffffffu, old, leader);
			if (valid) {
				bkt[p] = (uint16_t) b;
				inv[p] = (uint16_t) (old + __popc(below));   // rank within warp sub-tile, for now
			}
			__syncwarp();
		}
		__syncthreads();
		// (2) per bucket: warp prefixes, tile totals, and a scan over buckets
		// for each bucket's first row of the grouped tile.
		if (tid == 0) carry = 0;
		__syncthreads();
		for (uint32_t b0 = 0; b0 < B; b0 += blockDim.x) {
			uint32_t b = b0 + tid;
			uint32_t tot = 0;
			if (b < B) {
				#pragma unroll 4
				for (int w = 0; w < NW; ++w) {
					uint32_t c = cnt[w * B + b];
					cnt[w * B + b] = (uint16_t) tot;
					tot += c;
				}
			}
			// block exclusive scan of tot
			uint32_t x = tot;
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
				if (lane >= o) x += y;
			}
			if (lane == 31) warp_sums[warp] = x;
			__syncthreads();
			if (warp == 0) {
				uint32_t v = lane < NW ? warp_sums[lane] : 0, vv = v;
				#pragma unroll
				for (int o = 1; o < 32; o <<= 1) {
					uint32_t y = __shfl_up_sync(0xffffffffu, vv, o);
					if (lane >= o) vv += y;
				}
				if (lane < NW) warp_sums[lane] = vv - v;
				if (lane == NW - 1) warp_sums[31] = vv;
			}
			__syncthreads();
			if (b < B) {
				const uint32_t ts = carry + x - tot + warp_sums[warp];
				tstart[b] = ts;
				// Output row of grouped slot s of bucket b: running[b] + (s - ts),
				// kept as one word mod 2^32 (rows stay below 2^32).
				delta[b] = running[b] - ts;
				running[b] += tot;
			}
			__syncthreads();
			if (tid == 0) carry += warp_sums[31];
			__syncthreads();
		}
		// (3) grouped slot of every row, recorded as the permutation
		// slot -> row.
		uint16_t* perm = reinterpret_cast<uint16_t*>(bar + 2);
		for (uint32_t it = 0; it < sub; it += 32) {
			uint32_t p = warp * sub + it + lane;
			if (p < rows) {
				uint32_t b = bkt[p];
				perm[tstart[b] + cnt[warp * B + b] + inv[p]] = (uint16_t) p;
			}
		}
		__syncthreads();
		// (4) write out: slot s of bucket b goes to row delta[b] + s. Threads
		// walk the tile in grouped order so that neighbouring lanes store to
		// neighbouring rows of one partition.
		{
			if (W == 16) {
				for (uint32_t s = tid; s < rows; s += blockDim.x) {
					uint32_t p = perm[s];
					uint32_t b = bkt[p];
					uint64_t dest = (uint32_t) (delta[b] + s);
					uint4 v = reinterpret_cast<const uint4*>(cur)[p];
					pg_st_stream16(out + dest * 16, v);
				}
			} else {
				const uint32_t words = W / 4;
				for (uint32_t e = tid; e < rows * words; e += blockDim.x) {
					uint32_t s = e / words, wd = e - s * words;
					uint32_t p = perm[s];
					uint32_t b = bkt[p];
					uint64_t dest = (uint32_t) (delta[b] + s);
					reinterpret_cast<uint32_t*>(out + dest * W)[wd] =
						reinterpret_cast<const uint32_t*>(cur + (uint64_t) p * W)[wd];
				}
			}
		}
		// (5) reset the counters: step (2) left warp prefixes in every warp's
		// row of each bucket present in the tile. Small tables are cleared
		// whole, large ones only at the buckets this tile used.
		if (NW * B <= 4 * rows) {
			for (uint32_t i = tid; i < NW * B; i += blockDim.x) cnt[i] = 0;
		} else {
			for (uint32_t p = tid; p < rows; p += blockDim.x) {
				uint32_t b = bkt[p];
				#pragma unroll
				for (int w = 0; w < NW; ++w) cnt[w * B + b] = 0;
			}
		}
		__syncthreads();
		bulk_pending = next_bulk;
	}
}

static size_t part_smem_bytes(uint32_t tile, uint32_t W, uint32_t B, int NW)
{
	size_t s = 2 * (size_t) tile * W;          // tile buffers
	s += (size_t) NW * B * 2;                  // per-warp counters
	s += 3 * (size_t) B * 4;                   // tstart, delta, running
	s += 2 * (size_t) tile * 2;                // inv, bkt
	s = (s + 15) & ~size_t(15);
	s += 16;                                   // mbarriers
	s += (size_t) tile * 2;                    // grouped-slot -> row permutation
	return s;
}

// ---------------------------------------------------------------------------
// 16-byte tuples and at most 256 buckets. k_chunk_hist counts every block's
// chunk of the input per bucket (at the copy rate); a block of k_part_sweep
// adds up the chunks before its own and goes through its chunk in tiles:
//
// - the next tile arrives by a bulk copy while this one is worked on;
// - every warp takes its rows of the tile 32 at a time: lanes of the same bucket
//   are found with one ballot a bucket bit, and a counter per warp and bucket
//   gives each row its rank;
// - a thread a bucket turns the warps' counts into each warp's first slot of the
//   bucket in the grouped tile and the bucket's first output row;
// - the rows, still in registers, go to their slots, over the tile itself;
// - a thread a bucket stores the bucket's rows of the tile with one bulk copy.
//
// Every row keeps its order within its bucket. 100M tuples in 256 buckets:
// counting 230 us (the copy rate), partitioning 660 us, against 909 us with
// 20 KB tiles, a slot -> row permutation and a store a row; two thirds of that
// is the scattered stores (the same rows stored in tile order: 560 us). Tiles of
// 3072 rows, two blocks on an SM: smaller ones cost more in barriers (256 x 8 in
// three blocks 780 us), more threads in registers (512 x 6 670 us, 1024 x 3
// 1030 us). One-sweep forms with a look-back instead of the counting pass took
// as long a pass or longer (DRAM rows are no better used and every tile waits).
// ---------------------------------------------------------------------------
#define SW_BUCKETS 256
#define PG_FN_DIGIT32 66              // PG_FN_DIGIT within the key's low 32 bits
#define SW_CHECKED(FN) ((FN) != PG_FN_DIGIT && (FN) != PG_FN_DIGIT32)   // the bucket may be out of range
#define SW_THREADS 384
#define SW_ITEMS 8
#define SW_BLOCKS_PER_SM 2
#define SW_WARPS (SW_THREADS / 32)
#define SW_TILE (SW_THREADS * SW_ITEMS)
#define SW_HIST_SPLIT 2             // blocks of k_chunk_hist per chunk

// Key of a tuple (4 or 8 bytes at word kw), widened. K0: 8 bytes at word 0.
template <bool K0>
__device__ __forceinline__ int64_t sw_key(const uint4& t, uint32_t kw, uint32_t kbytes)
{
	if (K0) return (int64_t) (((uint64_t) t.y << 32) | t.x);
	const uint32_t lo = kw == 0 ? t.x : kw == 1 ? t.y : kw == 2 ? t.z : t.w;
	const uint32_t hi = kw == 0 ? t.y : kw == 1 ? t.z : t.w;
	return kbytes == 4 ? (int64_t) (int32_t) lo : (int64_t) (((uint64_t) hi << 32) | lo);
}

// Bucket of a key. PG_FN_DIGIT is taken from 32-bit words: only its low bits
// after the shift are kept.
template <int FN>
__device__ __forceinline__ uint32_t sw_bucket(const pg_hashfn& f, int64_t v, uint32_t kbytes)
{
	// All of the digit in the low word: the borrow does not matter.
	if (FN == PG_FN_DIGIT32) return (((uint32_t) v - (uint32_t) f.min) >> f.skipbits) & (uint32_t) f.k;
	if (FN == PG_FN_DIGIT) {
		const uint64_t x = (uint64_t) v - (uint64_t) f.min;
		const bool upper = f.skipbits >= 32;
		return __funnelshift_r(upper ? (uint32_t) (x >> 32) : (uint32_t) x, upper ? 0u : (uint32_t) (x >> 32),
				f.skipbits & 31) & (uint32_t) f.k;
	}
	if (FN == PG_FN_MIXRADIX) return (uint32_t) (pg_mix64((uint64_t) v) >> f.skipbits);
	if (FN == PG_FN_KNUTH) return (uint32_t) ((((uint64_t) v * 2654435761ull) & (uint64_t) f.k) >> f.skipbits);
	return pg_hash_value(f, v, kbytes);
}

// Lanes of the warp whose 8-bit value equals b, among `valid`: a ballot a bit.
__device__ __forceinline__ uint32_t sw_peers(uint32_t b, uint32_t valid)
{
	uint32_t peers = valid;
	#pragma unroll
	for (int k = 0; k < 8; ++k) {
		const bool on = (b >> k) & 1u;
		const uint32_t m = __ballot_sync(0xffffffffu, on);
		peers &= on ? m : ~m;
	}
	return peers;
}

// counts[c][b]: rows of bucket b in chunk c (chunk_rows rows each). With
// `outside`, a key outside [f.min, f.min + 2^window) sets it.
template <int FN, bool K0>
__global__ void __launch_bounds__(512)
k_chunk_hist(const uint4* __restrict__ in, uint32_t n, uint32_t kw, uint32_t kbytes, pg_hashfn f, uint32_t chunk_rows,
		uint32_t* __restrict__ counts, uint32_t window, int* __restrict__ outside, int* __restrict__ status)
{
	__shared__ uint32_t h[SW_BUCKETS];
	if (threadIdx.x < SW_BUCKETS) h[threadIdx.x] = 0;
	__syncthreads();
	const uint32_t lo = blockIdx.x * chunk_rows, hi = (uint32_t) pg_min64(n, (uint64_t) lo + chunk_rows);
	bool bad = false, out = false;
	for (uint64_t i0 = (uint64_t) lo + blockIdx.y * 512 + threadIdx.x; i0 < hi; i0 += 4 * SW_HIST_SPLIT * 512) {
		uint4 t[4];
		#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const uint64_t i = i0 + j * (SW_HIST_SPLIT * 512);
			t[j] = i < hi ? pg_ld_stream16(in + i) : make_uint4(0, 0, 0, 0);
		}
		#pragma unroll
		for (int j = 0; j < 4; ++j) {
			if (i0 + j * (SW_HIST_SPLIT * 512) >= hi) continue;
			const int64_t key = sw_key<K0>(t[j], kw, kbytes);
			const uint32_t b = sw_bucket<FN>(f, key, kbytes);
			if (b < f.nbuckets) atomicAdd(&h[b], 1u); else bad = true;
			if (outside && window < 64 && ((uint64_t) key - (uint64_t) f.min) >> window) out = true;
		}
	}
	if (bad) pg_set_status(status, PG_ERR_ARG);
	if (out) *outside = 1;
	__syncthreads();
	if (threadIdx.x < SW_BUCKETS && h[threadIdx.x]) atomicAdd(&counts[blockIdx.x * SW_BUCKETS + threadIdx.x], h[threadIdx.x]);
}

// Exclusive scan of x over threads 0..255 (the others must not call it). wt: 8
// words of shared memory.
__device__ __forceinline__ uint32_t sw_scan256(uint32_t x, uint32_t* wt)
{
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	uint32_t inc = x;
	#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
		if (lane >= (uint32_t) o) inc += y;
	}
	if (lane == 31) wt[warp] = inc;
	asm volatile("bar.sync 1, 256;" ::: "memory");
	uint32_t before = 0;
	#pragma unroll
	for (int w = 0; w < 8; ++w) before += (uint32_t) w < warp ? wt[w] : 0;
	return before + inc - x;                // the caller's next block barrier frees wt
}

struct SwShared {
	uint4 tile[2][SW_TILE];
	uint16_t slot[SW_WARPS][SW_BUCKETS];    // a warp's count of a bucket, then its first slot
	uint32_t wt[8];
	uint64_t bar[2];
};

template <int FN, bool K0>
__global__ void __launch_bounds__(SW_THREADS, SW_BLOCKS_PER_SM)
k_part_sweep(const uint4* __restrict__ in, uint32_t n, uint32_t kw, uint32_t kbytes, pg_hashfn f, uint32_t chunk_tiles,
		const uint32_t* __restrict__ counts, uint64_t* __restrict__ offsets, uint4* __restrict__ out, int* __restrict__ status)
{
	static_assert(SW_THREADS > SW_BUCKETS, "a thread a bucket, and a warp that waits for the first tile");
	extern __shared__ __align__(128) unsigned char sw_sm[];
	SwShared& sm = *reinterpret_cast<SwShared*>(sw_sm);
	const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, B = f.nbuckets;
	const uint32_t t0 = blockIdx.x * chunk_tiles;
	const uint32_t tiles = (uint32_t) pg_min64(chunk_tiles, pg_div_up(n, SW_TILE) - t0);
	auto rows_of = [&](uint32_t k) -> uint32_t { return pg_min32(SW_TILE, n - (t0 + k) * SW_TILE); };
	auto issue = [&](uint32_t k) {
		const uint32_t bytes = rows_of(k) * 16;
		pg_mbar_expect_tx(&sm.bar[k & 1], bytes);
		pg_bulk_g2s_hint(sm.tile[k & 1], in + (uint64_t) (t0 + k) * SW_TILE, bytes, &sm.bar[k & 1], pg_policy_evict_first());
	};
	if (tid == 0) {
		pg_mbar_init(&sm.bar[0], 1);
		pg_mbar_init(&sm.bar[1], 1);
		pg_fence_mbar_init();
		issue(0);
		if (tiles > 1) issue(1);
	}
	for (uint32_t i = tid; i < SW_WARPS * SW_BUCKETS / 2; i += SW_THREADS) reinterpret_cast<uint32_t*>(sm.slot)[i] = 0;
	__syncthreads();
	const uint32_t spin = pg_spin_knob(status);
	// Thread b keeps bucket b's next output row: the rows of lower buckets and
	// those of earlier chunks come before this chunk's. The other warps wait for
	// the first tile meanwhile.
	uint32_t next = 0;
	if (tid >= SW_BUCKETS) pg_mbar_wait_timed(&sm.bar[0], 0, spin, status);
	else {
		uint32_t total = 0;
		if (tid < B)
			#pragma unroll 8
			for (uint32_t c = 0; c < gridDim.x; ++c) {
				const uint32_t x = __ldg(counts + c * SW_BUCKETS + tid);
				total += x;
				next += c < blockIdx.x ? x : 0;
			}
		const uint32_t first = sw_scan256(total, sm.wt);
		if (offsets && blockIdx.x == 0) {
			if (tid < B) offsets[tid] = first;
			if (tid == 0) offsets[B] = n;
		}
		next += first;
	}
	__syncthreads();
	const uint64_t pol = pg_policy_evict_first();
	uint16_t* const slot = sm.slot[warp];
	const uint32_t r0 = warp * (SW_ITEMS * 32) + lane;      // item j: row r0 + 32 j of the tile
	for (uint32_t k = 0; k < tiles; ++k) {
		const uint32_t rows = rows_of(k);
		uint4* const tile = sm.tile[k & 1];
		// A wait past the context's limit records PG_ERR_TIMEOUT and goes on until
		// the copy lands; the rows are unspecified if it never does.
		pg_mbar_wait_timed(&sm.bar[k & 1], (k >> 1) & 1, spin, status);
		auto work = [&](auto whole) {
			constexpr bool FULL = decltype(whole)::value;
			uint4 t[SW_ITEMS];
			uint32_t br[SW_ITEMS];                       // bucket, rank in the warp's rows of it << 8
			uint32_t first = 0, tot = 0, row = 0;        // thread b: bucket b's first slot, rows, first output row
			#pragma unroll
			for (int j = 0; j < SW_ITEMS; ++j) {
				const bool mine = FULL || r0 + j * 32 < rows;
				t[j] = tile[r0 + j * 32];
				uint32_t b = sw_bucket<FN>(f, sw_key<K0>(t[j], kw, kbytes), kbytes);
				if (SW_CHECKED(FN) && b >= B) b = 0;     // the histogram reported it
				const uint32_t peers = sw_peers(b, FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, mine));
				const uint32_t at = slot[b], below = __popc(peers & ((1u << lane) - 1));
				__syncwarp();
				if (mine && below == 0) slot[b] = (uint16_t) (at + __popc(peers));
				__syncwarp();
				br[j] = b | ((at + below) << 8);
			}
			__syncthreads();
			if (tid < SW_BUCKETS) {
				uint32_t c[SW_WARPS];
				#pragma unroll
				for (int w = 0; w < SW_WARPS; ++w) { c[w] = sm.slot[w][tid]; tot += c[w]; }
				first = sw_scan256(tot, sm.wt);
				row = next;
				next += tot;
				uint32_t at = first;
				#pragma unroll
				for (int w = 0; w < SW_WARPS; ++w) { sm.slot[w][tid] = (uint16_t) at; at += c[w]; }
			}
			__syncthreads();
			#pragma unroll
			for (int j = 0; j < SW_ITEMS; ++j) {
				const uint32_t s = slot[br[j] & 255] + (br[j] >> 8);
				if ((FULL || r0 + j * 32 < rows) && s < SW_TILE) tile[s] = t[j];
			}
			pg_fence_proxy_async_smem();
			__syncthreads();
			// (Past n only when a copy gave up above.)
			if (tot && (uint64_t) row + tot <= n) pg_bulk_s2g_hint(out + row, tile + first, tot * 16, pol);
			// The counters for the next tile.
			#pragma unroll
			for (uint32_t i = tid; i < SW_WARPS * SW_BUCKETS / 2; i += SW_THREADS) reinterpret_cast<uint32_t*>(sm.slot)[i] = 0;
			pg_bulk_wait_read();
		};
		if (rows == SW_TILE) work(std::true_type());
		else work(std::false_type());
		// The buffer's next copy comes after this tile's stores have read it.
		__syncthreads();
		if (tid == 0 && k + 2 < tiles) issue(k + 2);
	}
}

// Whether k_part_sweep can take a partition of `in` into `out`.
static bool sw_takes(const pg_rel* in, const void* out, uint32_t buckets)
{
	return in->width == 16 && (in->key_off & 3) == 0 && buckets <= SW_BUCKETS &&
		!((reinterpret_cast<uintptr_t>(in->data) | reinterpret_cast<uintptr_t>(out)) & 15);
}

// Whether it is the faster one, for the functions and fan-outs where k_part_scatter's
// smaller tiles, more blocks and fewer ballots can win. Scatter against sweep: one bucket
// 64M tuples 438 and 620 us, 3M 63 and 81; two buckets 3M 68 and 77, 500,000 46 and 52, 8M 131
// and 115, 64M 662 and 545. Functions that both compute twice a tuple and that cost more than
// the ranking: exactrange into 3 buckets 1094 and 1151 us (64M), 92 and 114 (3M), into 200
// 1268 and 1214, 111 and 116; bytes into 64 1481 and 1508, 122 and 138, but 500,000 tuples 72
// and 64. Below 400,000 tuples a block has one tile and the fewer launches win (100,000
// in 2 buckets 45 and 40, exactrange into 3 46 and 43).
static bool sw_wins(const pg_hashfn& f, uint64_t n)
{
	if (n < 400000) return true;
	switch (f.fn) {
	case PG_FN_RANGE: case PG_FN_EXACTRANGE: return f.nbuckets > 4;
	case PG_FN_BYTES: return f.nbuckets > 4 && n < 2500000;
	default: return f.nbuckets > 2 || (f.nbuckets == 2 && n >= 4000000);
	}
}

// `check` (pg_radix_pass): the key window is confirmed before the rows move;
// *refuted and nothing written when it is not.
struct SwCheck { uint32_t window; bool* refuted; };

template <int FN, bool K0>
static int sw_partition_as(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, const pg_hashfn& f, void* out, uint64_t* offsets,
		const SwCheck* check)
{
	const uint32_t n = (uint32_t) in->n, ntiles = (uint32_t) pg_div_up(n, SW_TILE);
	const uint32_t chunk = (uint32_t) pg_div_up(ntiles, ctx->sm_count * SW_BLOCKS_PER_SM), G = (uint32_t) pg_div_up(ntiles, chunk);
	int rc;
	uint32_t* counts = nullptr;               // [G][256], then the flag of a key outside the window
	const size_t bytes = (size_t) G * SW_BUCKETS * 4 + 4;
	PgScratch mem(ctx, s);
	if ((rc = mem.get((void**) &counts, bytes))) return rc;
	int* outside = reinterpret_cast<int*>(counts + (size_t) G * SW_BUCKETS);
	PG_CUDA(ctx, cudaMemsetAsync(counts, 0, bytes, s));
	k_chunk_hist<FN, K0><<<dim3(G, SW_HIST_SPLIT), 512, 0, s>>>((const uint4*) in->data, n, in->key_off / 4, in->key_bytes, f,
			chunk * SW_TILE, counts, check ? check->window : 64, check ? outside : nullptr, ctx->d_status);
	PG_LAUNCHED(ctx);
	if (check) {
		int bad = 0;
		PG_CUDA(ctx, cudaMemcpyAsync(&bad, outside, 4, cudaMemcpyDeviceToHost, s));
		PG_CUDA(ctx, cudaStreamSynchronize(s));
		if (bad) { *check->refuted = true; return PG_OK; }
	}
	PG_CUDA(ctx, cudaFuncSetAttribute(k_part_sweep<FN, K0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(SwShared)));
	k_part_sweep<FN, K0><<<G, SW_THREADS, sizeof(SwShared), s>>>((const uint4*) in->data, n, in->key_off / 4, in->key_bytes,
			f, chunk, counts, offsets, (uint4*) out, ctx->d_status);
	PG_LAUNCHED(ctx);
	return PG_OK;
}

static int sw_partition_digit(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, const pg_hashfn& f, uint32_t bits, void* out,
		uint64_t* offsets, const SwCheck* check)
{
	const bool k0 = in->key_off == 0 && in->key_bytes == 8;
	if (f.skipbits + bits <= 32)
		return k0 ? sw_partition_as<PG_FN_DIGIT32, true>(ctx, s, in, f, out, offsets, check)
		          : sw_partition_as<PG_FN_DIGIT32, false>(ctx, s, in, f, out, offsets, check);
	return k0 ? sw_partition_as<PG_FN_DIGIT, true>(ctx, s, in, f, out, offsets, check)
	          : sw_partition_as<PG_FN_DIGIT, false>(ctx, s, in, f, out, offsets, check);
}

// The functions that are one run of bits of key - min (modulo, and
// parammodulo whose bits lie below the sign bit: its signed shift then equals
// the unsigned one) go as PG_FN_DIGIT.
static int sw_partition(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, pg_hashfn f, void* out, uint64_t* offsets)
{
	uint32_t lg = 0;
	while ((1u << lg) < f.nbuckets) ++lg;
	if (f.fn == PG_FN_MODULO) { f.fn = PG_FN_DIGIT; f.min = 0; f.skipbits = 0; }
	else if (f.fn == PG_FN_PARAMMODULO && f.skipbits + lg < 64) f.fn = PG_FN_DIGIT;
	if (f.fn == PG_FN_DIGIT) {
		f.k = f.nbuckets - 1;
		return sw_partition_digit(ctx, s, in, f, lg, out, offsets, nullptr);
	}
	if (f.fn == PG_FN_KNUTH) return sw_partition_as<PG_FN_KNUTH, false>(ctx, s, in, f, out, offsets, nullptr);
	if (f.fn == PG_FN_MIXRADIX) return sw_partition_as<PG_FN_MIXRADIX, false>(ctx, s, in, f, out, offsets, nullptr);
	return sw_partition_as<PART_FN_ANY, false>(ctx, s, in, f, out, offsets, nullptr);
}

bool pg_radix_pass_takes(const pg_rel* in, const void* out) { return sw_takes(in, out, SW_BUCKETS) && in->n < (1ull << 32); }

int pg_radix_pass(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, int64_t base, int pass, int window, bool* refuted, void* out)
{
	pg_hashfn f = {};
	f.fn = PG_FN_DIGIT; f.min = base; f.skipbits = 8 * pass; f.nbuckets = SW_BUCKETS; f.k = SW_BUCKETS - 1;
	const SwCheck check = {(uint32_t) window, refuted};
	return sw_partition_digit(ctx, s, in, f, 8, out, nullptr, refuted ? &check : nullptr);
}

extern "C" int pg_partition(pg_ctx* ctx, pg_stream stream, const pg_rel* in,
		const pg_hashcfg* cfg, void* out, uint64_t* offsets)
{
	if (!ctx || !in || !cfg || !offsets) return pg_fail(ctx, PG_ERR_ARG, "pg_partition: null argument");
	pg_hashfn f;
	if (pg_hashfn_derive(cfg, &f)) return pg_fail(ctx, PG_ERR_ARG, "pg_partition: invalid hash configuration");
	int rc = pg_partition_fn(ctx, (cudaStream_t) stream, in, f, out, offsets);
	if (rc) return rc;
	return pg_check_status(ctx, (cudaStream_t) stream, "pg_partition");
}

// Partition by an already derived bucket function; offsets may be null. Does
// not synchronise (the radix sort chains passes on the stream).
int pg_partition_fn(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, const pg_hashfn& f,
		void* out, uint64_t* offsets)
{
	const uint32_t B = f.nbuckets, W = in->width;
	if (B == 0 || B > PART_MAX_BUCKETS)
		return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_partition: at most 4096 buckets in one pass");
	if (W == 0 || (W & 3) || W > 1024)
		return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_partition: tuple width must be a multiple of 4 bytes, at most 1024");
	if (in->key_off + in->key_bytes > W || (in->key_bytes != 4 && in->key_bytes != 8))
		return pg_fail(ctx, PG_ERR_ARG, "pg_partition: key must be a 4- or 8-byte column inside the tuple");
	if (in->n >= (1ull << 32)) return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_partition: at most 2^32-1 tuples");
	const uint64_t n = in->n;
	if (n == 0) {
		if (offsets) PG_CUDA(ctx, cudaMemsetAsync(offsets, 0, (B + 1) * sizeof(uint64_t), s));
		return PG_OK;
	}
	if (sw_takes(in, out, B) && sw_wins(f, n)) return sw_partition(ctx, s, in, f, out, offsets);
	const int NW = B <= 1024 ? 8 : 4;
	const int64_t tb = ctx->tune[PG_TUNE_PARTITION_TILE];
	uint32_t tile = (uint32_t) (tb > 0 ? std::min<int64_t>(65536, std::max<int64_t>(8192, tb)) : PART_TILE_BYTES) / W;
	tile = std::max<uint32_t>(NW * 32, tile / (NW * 32) * (NW * 32));
	const uint64_t ntiles = pg_div_up(n, tile);
	const size_t smem = part_smem_bytes(tile, W, B, NW);
	if (smem > 220 * 1024) return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_partition: tile does not fit shared memory");
	int per_sm = (int) std::max<size_t>(1, std::min<size_t>(8, (228 * 1024) / (smem + 1024)));
	uint64_t G = std::min<uint64_t>(ntiles, (uint64_t) ctx->sm_count * per_sm);
	uint64_t tpc = pg_div_up(ntiles, G);
	G = pg_div_up(ntiles, tpc);

	int rc;
	uint64_t* counts = nullptr;
	PgScratch mem(ctx, s);
	if ((rc = mem.get((void**) &counts, (size_t) B * G * 8 + 8))) return rc;
	const bool radix = f.fn == PG_FN_PARAMMODULO, mix = f.fn == PG_FN_MIXRADIX;
	if (radix)
		k_part_hist<PG_FN_PARAMMODULO><<<(unsigned) G, 512, B * sizeof(uint32_t), s>>>((const char*) in->data, n, W,
				in->key_off, in->key_bytes, f, tile, tpc, counts, (uint32_t) G, ctx->d_status);
	else if (mix)
		k_part_hist<PG_FN_MIXRADIX><<<(unsigned) G, 512, B * sizeof(uint32_t), s>>>((const char*) in->data, n, W,
				in->key_off, in->key_bytes, f, tile, tpc, counts, (uint32_t) G, ctx->d_status);
	else
		k_part_hist<PART_FN_ANY><<<(unsigned) G, 512, B * sizeof(uint32_t), s>>>((const char*) in->data, n, W,
				in->key_off, in->key_bytes, f, tile, tpc, counts, (uint32_t) G, ctx->d_status);
	PG_LAUNCHED(ctx);
	if ((rc = pg_scan_u64(ctx, s, counts, (uint64_t) B * G, nullptr))) return rc;
	bool bulk_ok = ((reinterpret_cast<uintptr_t>(in->data) & 15) == 0) && (((uint64_t) tile * W) % 16 == 0);
#define PS_LAUNCH(NWv, FNv, NB) do { \
		PG_CUDA(ctx, cudaFuncSetAttribute(k_part_scatter<NWv, FNv, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)); \
		k_part_scatter<NWv, FNv, NB><<<(unsigned) G, NWv * 32, smem, s>>>((const char*) in->data, n, W, in->key_off, \
				in->key_bytes, f, tile, tpc, counts, (uint32_t) G, (char*) out, bulk_ok, ctx->d_status); } while (0)
	// Radix passes (parammodulo) of 256 or 64 buckets and partitions on the
	// top bits of the key hash (mixradix, 32 to 256 buckets) take specialised
	// kernels; everything else the general one.
	if (NW == 8 && radix && B == 256) PS_LAUNCH(8, PG_FN_PARAMMODULO, 8);
	else if (NW == 8 && radix && B == 64) PS_LAUNCH(8, PG_FN_PARAMMODULO, 6);
	else if (NW == 8 && mix && B == 256) PS_LAUNCH(8, PG_FN_MIXRADIX, 8);
	else if (NW == 8 && mix && B == 128) PS_LAUNCH(8, PG_FN_MIXRADIX, 7);
	else if (NW == 8 && mix && B == 64) PS_LAUNCH(8, PG_FN_MIXRADIX, 6);
	else if (NW == 8 && mix && B == 32) PS_LAUNCH(8, PG_FN_MIXRADIX, 5);
	else if (NW == 8) PS_LAUNCH(8, PART_FN_ANY, 0);
	else PS_LAUNCH(4, PART_FN_ANY, 0);
#undef PS_LAUNCH
	PG_LAUNCHED(ctx);
	// offsets[b] = first slot of bucket b = scanned count of (b, CTA 0).
	// Strided copy: counts[b*G] for b < B, then n.
	if (offsets) {
		PG_CUDA(ctx, cudaMemcpy2DAsync(offsets, sizeof(uint64_t), counts, G * sizeof(uint64_t),
				sizeof(uint64_t), B, cudaMemcpyDeviceToDevice, s));
		PG_CUDA(ctx, cudaMemcpyAsync(offsets + B, &in->n, sizeof(uint64_t), cudaMemcpyHostToDevice, s));
	}
	return PG_OK;
}
