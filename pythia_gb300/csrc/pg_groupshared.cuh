// Group tables in shared memory, for the dense group-by and the join that feeds one.
//
// Few groups otherwise put every row's atomic on a handful of L2 lines: each CTA sums
// its rows into a table of its own, then adds each slot it saw into the global table
// once. A slot is 32-bit words, which take native adds where a shared 64-bit one is a
// compare-and-swap loop: a count or an int sum one word, a long sum two, a dec sum its
// t2 word in two and t2's overflows in a third; the chunks of a value far below the
// column's largest, rare, go to the global table's lazy words, or with few groups,
// where those are hot lines too, to lazy words here (LAZY). The first add into a sum's
// slot returns the initial 0 and marks it seen. Copies of the table against equal
// keys: no faster.
#pragma once
#include "pg_internal.cuh"
#include <algorithm>

#define GB_DEC (VT == PG_VAL_DEC && AGG == PG_AGG_SUM)     // inside templates on VT, AGG
#define GBS_THREADS 1024
#define GBS_MAX_BYTES (224 * 1024)
#define GBS_LAZY_BYTES (8 * PG_FX_LAZY)

// v added to a 64-bit word in shared memory by its 32-bit halves: the upper half needs
// an add only for a carry or a large value.
__device__ __forceinline__ void gb_shared_add64(unsigned long long* p, unsigned long long v)
{
	pg_fx_add_halves(reinterpret_cast<uint32_t*>(p), v, [](uint32_t* q, uint32_t x) { return atomicAdd(q, x); });
}

template <int VT, int AGG>
__host__ __device__ constexpr uint32_t gbs_words() { return GB_DEC ? 3 : AGG == PG_AGG_COUNT || VT == PG_VAL_INT ? 1 : 2; }

template <int VT, int AGG, bool LAZY>
struct GbShared {
	static constexpr uint32_t LW = LAZY ? 2 * PG_FX_LAZY : 0, SW = gbs_words<VT, AGG>();
	unsigned long long* sl;      // lazy word c of slot d at sl[d + c range]
	uint32_t* sw;                // word w of slot d at sw[d + w range]
	unsigned char* spres;
	uint32_t range;
	unsigned long long* acc;     // the global table: word w of slot d at acc[d + w range]
	int fs, fb;
	uint32_t fl;                 // a dec sum's flags, gathered

	__device__ __forceinline__ GbShared(unsigned char* mem, uint32_t r, unsigned long long* a, PgFx fx)
	{
		range = r; acc = a; fl = 0;
		fs = GB_DEC ? fx.p[0] : 0;
		fb = GB_DEC ? fx.p[1] : 0;
		sl = reinterpret_cast<unsigned long long*>(mem);
		sw = reinterpret_cast<uint32_t*>(mem) + (size_t) range * LW;
		spres = reinterpret_cast<unsigned char*>(sw + range * SW);
		for (uint32_t d = threadIdx.x; d < range * (LW + SW); d += blockDim.x) reinterpret_cast<uint32_t*>(mem)[d] = 0;
		if (AGG == PG_AGG_SUM) for (uint32_t d = threadIdx.x; d < range; d += blockDim.x) spres[d] = 0;
		__syncthreads();
	}

	// One row of slot d < range: its value's bits (none for a count).
	__device__ __forceinline__ void add(uint32_t d, uint64_t v)
	{
		if (AGG == PG_AGG_COUNT) { atomicAdd(&sw[d], 1u); return; }
		if (GB_DEC) {
			const pg_fx3 f = pg_fx_take(v, fs, fb, fl);
			v = f.w2;
			if (f.w0 | f.w1) {
				#pragma unroll
				for (int c = 0; c < PG_FX_LAZY; ++c) {
					const uint64_t x = pg_fx_chunk(f.w0, f.w1, c);
					if (!x) continue;
					if (LAZY) gb_shared_add64(&sl[d + c * range], x);
					else atomicAdd(&acc[d + (uint64_t) (PG_FX_L0 + c) * range], (unsigned long long) x);
				}
			}
		}
		const uint32_t lo = (uint32_t) v, old = atomicAdd(&sw[d], lo);
		if (old == 0) spres[d] = 1;
		const uint32_t hi = SW == 1 ? 0 : (uint32_t) (v >> 32) + (old + lo < lo);
		if (!hi) return;
		const uint32_t oh = atomicAdd(&sw[d + range], hi);
		if (!GB_DEC) return;
		// A value's part of t2 is within +-2^60: hi did not wrap.
		const int32_t was = (int32_t) oh, is = (int32_t) (oh + hi);
		if ((int32_t) hi > 0 ? is < was : is > was) atomicAdd(&sw[d + 2 * range], (int32_t) hi > 0 ? 1u : ~0u);
	}

	// The CTA's slots into the global table, and a sum's groups marked.
	__device__ __forceinline__ void flush(unsigned char* __restrict__ present)
	{
		__syncthreads();
		for (uint32_t d = threadIdx.x; d < range; d += blockDim.x) {
			if (AGG == PG_AGG_COUNT) {
				if (sw[d]) atomicAdd(&acc[d], (unsigned long long) sw[d]);
				continue;
			}
			if (!spres[d]) continue;
			const unsigned long long v = SW == 1 ? sw[d] : ((unsigned long long) sw[d + range] << 32) | sw[d];
			if (GB_DEC) {
				const uint64_t t3 = (uint64_t) (int64_t) (int32_t) sw[d + 2 * range];
				pg_fx_atomic_add(&acc[d], range, pg_fx4{0, 0, v, t3 - (v >> 63)});
				#pragma unroll
				for (int c = 0; c < (LAZY ? PG_FX_LAZY : 0); ++c)
					if (sl[d + c * range]) atomicAdd(&acc[d + (uint64_t) (PG_FX_L0 + c) * range], sl[d + c * range]);
			} else if (VT == PG_VAL_INT) atomicAdd(reinterpret_cast<unsigned int*>(&acc[d]), (unsigned int) v);
			else atomicAdd(&acc[d], v);
			present[d] = 1;
		}
	}
};

// Launch of a kernel on these tables: shared bytes and blocks for n rows over `range`
// slots, while the flushes are fewer than the rows (1M rows in 4000 groups take 79 us in
// L2, with more slots to flush than rows 90). A table of half the SM's shared memory
// or less lets two CTAs share it; dec sums keep lazy words there when they fit in that
// half.
struct GbsPlan {
	uint64_t bytes;
	bool lazy;
};

template <int VT, int AGG>
static GbsPlan gbs_plan(uint64_t range)
{
	GbsPlan p = {range * (4 * gbs_words<VT, AGG>() + (AGG == PG_AGG_SUM ? 1 : 0)), false};
	p.lazy = GB_DEC && p.bytes + range * GBS_LAZY_BYTES <= GBS_MAX_BYTES / 2;
	if (p.lazy) p.bytes += range * GBS_LAZY_BYTES;
	return p;
}

// *blocks = 0: not with shared tables.
template <class K>
static int gbs_blocks(pg_ctx* ctx, K kernel, const GbsPlan& p, uint64_t range, uint64_t n, int* blocks)
{
	*blocks = 0;
	if (p.bytes > GBS_MAX_BYTES) return PG_OK;
	int per_sm = 0;
	PG_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GBS_MAX_BYTES));
	PG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, GBS_THREADS, p.bytes));
	const uint64_t b = std::min<uint64_t>(pg_div_up(n, GBS_THREADS), (uint64_t) ctx->sm_count * std::max(per_sm, 1));
	if (range * b <= n) *blocks = (int) b;
	return PG_OK;
}
