// Filter and Project on sm_103a.
//
// Replace Filter::map and Project::map (operators/filter.cpp:37-85,
// project.cpp:37-104), which MapWrapper calls tuple by tuple per thread
// (mapwrapper.cpp:38-138), with one launch over the whole relation.
//
// Filter is a stable compaction in one pass: a tile of tuples arrives in shared
// memory by a bulk copy, its predicates are evaluated there, the tile's first
// output row comes from a warp that adds up the tiles' counts as they are
// published, and the survivors are written with consecutive lanes on
// consecutive words: one read of the relation and one write of the survivors.
// Project stages tiles the same way: one read, one write. Tuples wide enough that some of
// their sectors need not be read are not staged. Both are bound by
// HBM; 50M 24-byte tuples, half passing, measured 370 us for the filter (0.72
// of the copy rate; 835 us in two passes with a thread copying each tuple), and
// 25M of them to 16-byte rows 160 us for the projection (378 us with a
// division and a word map in shared memory per output vector).
#include "pg_pred.cuh"
#include <algorithm>
#include <cstring>

#define FL_THREADS 256
// Wider tuples are not staged: their predicates read the columns' sectors and only
// the survivors are read whole, a warp a survivor. 600 MB of tuples of 300, 400 and 1000
// bytes, no survivors: staged 154, 195 and 138 us, unstaged 78, 71 and 51 (131, 115 and 65
// in two passes); a third pass: 192, 218 and 166 against 151, 118 and 118 (572, 349 and 702);
// all pass: 274, 264 and 226 against 336, 238 and 274 (2184, 1005 and 1689). At 240 bytes
// staging is never slower than the two passes were (144 us with no survivors, 153), from
// 300 it was.
#define FL_STAGE_WIDTH 240
#define FL_DIRECT_ROWS 512
#define FL_TILE_BYTES (24 * 1024)     // eight blocks of 256 threads on an SM
#define PJ_TILE_BYTES (24 * 1024)
// A projection of at most a quarter of a wider tuple reads its columns straight from
// memory: 600 MB of 400-byte tuples, 4, 48, 100 and 200 bytes kept: staged 170, 181, 193 and
// 206 us, unstaged 58, 72, 131 and 162 (a thread a tuple 57, 158, 748 and 1647); of 1000-byte
// ones, 8, 248 and 500: 109, 134 and 156 against 33, 95 to 119 and 184; of 136, 32 and 68: 135
// and 156 against 132 and 218. Up to 128 bytes the sectors are all read anyway (100 bytes, 4
// kept: 119 both).
#define PJ_STAGE_WIDTH 128
#define PJ_STAGE_MAX 1024
#define PJ_DIRECT_ROWS 512
#define HJ_PROJ_MAX 16

int pg_pred_prepare(pg_ctx* ctx, const pg_pred* preds, int npred, uint32_t width, PgPredSet* out, bool* has_char)
{
	if (npred < 0 || npred > PG_PRED_MAX || (npred && !preds))
		return pg_fail(ctx, PG_ERR_ARG, "predicates: 0..4 predicates");
	memset(out, 0, sizeof(*out));
	out->n = npred;
	*has_char = false;
	for (int i = 0; i < npred; ++i) {
		const pg_pred& p = preds[i];
		if (p.op > PG_CMP_GE) return pg_fail(ctx, PG_ERR_ARG, "predicates: unknown comparison");
		const bool num = p.type == PG_PRED_INT || p.type == PG_PRED_LONG || p.type == PG_PRED_DEC;
		if (num) {
			const uint32_t want = p.type == PG_PRED_INT ? 4 : 8;
			if (p.bytes != want || (p.off & 3) || p.off + p.bytes > width)
				return pg_fail(ctx, PG_ERR_ARG, "predicates: int 4 bytes, long/dec 8 bytes, 4-byte aligned, inside the tuple");
			uint64_t v = 0;
			memcpy(&v, p.value, p.bytes);
			out->v[i] = v;
		} else if (p.type == PG_PRED_CHAR) {
			if (p.bytes < 1 || p.bytes > 128 || p.off + p.bytes > width)
				return pg_fail(ctx, PG_ERR_ARG, "predicates: char columns of 1..128 bytes inside the tuple");
			*has_char = true;
		} else {
			return pg_fail(ctx, PG_ERR_ARG, "predicates: unknown column type");
		}
		out->type[i] = p.type; out->op[i] = p.op; out->off[i] = p.off; out->bytes[i] = p.bytes;
	}
	return PG_OK;
}

bool pg_pred_as16(const pg_pred* preds, int npred, PgPred16* out)
{
	memset(out, 0, sizeof(*out));
	out->n = npred;
	for (int i = 0; i < npred; ++i) {
		const pg_pred& p = preds[i];
		if (p.type == PG_PRED_CHAR || (p.off & 3) || p.off + p.bytes > 16) return false;
		out->word[i] = (uint8_t) (p.off / 4);
		out->type[i] = (uint8_t) p.type;
		out->op[i] = (uint8_t) p.op;
		uint64_t v = 0;
		memcpy(&v, p.value, p.type == PG_PRED_INT ? 4 : 8);
		out->v[i] = v;
	}
	return true;
}

// Copies `bytes` (a multiple of 4) of a tile into shared memory: a bulk copy of
// the 16-byte multiple when src is 16-byte aligned, the rest by words; ends
// with every thread seeing the tile. A wait past the context's limit records
// PG_ERR_TIMEOUT and goes on until the copy lands; the tile's contents are
// unspecified if it never does.
__device__ __forceinline__ void fl_load_tile(unsigned char* dst, const char* src, uint32_t bytes, uint64_t* bar,
		int* status)
{
	const bool bulk = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && bytes >= 16;
	const uint32_t body = bulk ? bytes & ~15u : 0;
	if (bulk && threadIdx.x == 0) {
		pg_mbar_init(bar, 1);
		pg_fence_mbar_init();
		pg_mbar_expect_tx(bar, body);
		pg_bulk_g2s_hint(dst, src, body, bar, pg_policy_evict_first());
	}
	for (uint32_t i = body / 4 + threadIdx.x; i < bytes / 4; i += blockDim.x)
		reinterpret_cast<uint32_t*>(dst)[i] = __ldcs(reinterpret_cast<const uint32_t*>(src) + i);
	__syncthreads();
	if (bulk) pg_mbar_wait_timed(bar, 0, pg_spin_knob(status), status);
}

// Rows of w bytes in a tile of at most `bytes` bytes: a multiple of 32, so that
// tiles start on 16-byte boundaries.
static uint32_t fl_tile_rows(uint32_t w, uint32_t bytes) { return std::max<uint32_t>(32, bytes / w / 32 * 32); }

// Rows of a tile that is not staged: blocks for every SM before rows for every thread.
static uint32_t fl_direct_rows(const pg_ctx* ctx, uint64_t n, uint32_t most)
{
	return (uint32_t) std::min<uint64_t>(most, std::max<uint64_t>(32, n / ((uint64_t) ctx->sm_count * 8) / 32 * 32));
}

#define FL_READY (1ull << 63)       // of a tile's first output row
#define FL_COUNTED (1u << 31)      // of a tile's count
#define FL_SPIN_LIMIT (1u << 22)
#define FL_LOOK 8                  // counts a lane of the scanning warp reads at once

// The scanning warp of k_filter: adds up the tiles' counts in order as they
// are published and publishes every tile's first output row. One warp keeps up:
// a step of 256 tiles takes one L2 round trip, in which about 100 tiles
// finish. (Tiles that looked back over each other's counts themselves took 500
// us against 360 on 50M 24-byte tuples: a thousand blocks in flight each read
// back over the same few lines to the last known total.)
__device__ __forceinline__ void fl_scan_tiles(const uint32_t* __restrict__ count,
		unsigned long long* __restrict__ first, uint64_t ntiles, unsigned long long* __restrict__ total, int* __restrict__ status)
{
	const uint32_t lane = threadIdx.x & 31, spin = pg_spin_knob(status);
	unsigned long long run = 0;
	uint32_t polls = 0;
	for (uint64_t t = 0; t < ntiles;) {
		uint32_t v[FL_LOOK], done = 32 * FL_LOOK;
		#pragma unroll
		for (int q = 0; q < FL_LOOK; ++q) v[q] = t + q * 32 + lane < ntiles ? pg_ld_relaxed(count + t + q * 32 + lane) : 0;
		#pragma unroll
		for (int q = FL_LOOK - 1; q >= 0; --q) {                 // leading counts that are there
			const uint32_t gap = __ballot_sync(0xffffffffu, !(v[q] & FL_COUNTED));
			if (gap) done = q * 32 + __ffs(gap) - 1;
		}
		uint32_t inc[FL_LOOK];
		#pragma unroll
		for (int q = 0; q < FL_LOOK; ++q) inc[q] = v[q] = q * 32 + lane < done ? v[q] & ~FL_COUNTED : 0;
		#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			#pragma unroll
			for (int q = 0; q < FL_LOOK; ++q) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, inc[q], o);
				if (lane >= (uint32_t) o) inc[q] += y;
			}
		}
		#pragma unroll
		for (int q = 0; q < FL_LOOK; ++q) {
			if (q * 32 + lane < done) pg_st_relaxed(first + t + q * 32 + lane, FL_READY | (run + inc[q] - v[q]));
			run += __shfl_sync(0xffffffffu, inc[q], 31);
		}
		t += done;
		polls = done ? 0 : polls + 1;
		if (polls && (polls == (spin ? spin : FL_SPIN_LIMIT) || polls >= FL_SPIN_LIMIT)) {
			if (lane == 0) pg_set_status(status, PG_ERR_TIMEOUT);
			if (polls >= FL_SPIN_LIMIT) return;
		}
	}
	if (lane == 0) *total = run;
}

// One tile a block, in shared memory (STAGED) or where it is (U = unit of the row
// copies), and one block whose first
// warp scans the tiles' counts: the first to arrive, so it runs whenever a
// tile waits for it, and every tile that it waits for has been taken by a
// running block before any later tile.
template <typename U, bool STAGED>
__global__ void __launch_bounds__(FL_THREADS)
k_filter(const char* __restrict__ in, uint64_t n, uint32_t w, uint32_t tile_rows, const PgPredSet P,
		uint32_t* __restrict__ count, unsigned long long* __restrict__ first, unsigned int* __restrict__ ticket,
		char* __restrict__ out, unsigned long long* __restrict__ total, int* __restrict__ status)
{
	extern __shared__ __align__(128) unsigned char fl_sm[];
	uint32_t* const mask = reinterpret_cast<uint32_t*>(fl_sm + (STAGED ? tile_rows * w : 0));   // [tile_rows / 32]
	uint32_t* const before = mask + tile_rows / 32;                                       // [tile_rows / 32]
	uint16_t* const sel = reinterpret_cast<uint16_t*>(before + tile_rows / 32);           // [tile_rows]
	__shared__ __align__(8) uint64_t bar;
	__shared__ unsigned int s_tile;
	__shared__ unsigned long long s_first;
	__shared__ uint32_t s_count;
	const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (tid == 0) s_tile = atomicAdd(ticket, 1u);
	__syncthreads();
	if (s_tile == 0) {
		if (warp == 0) fl_scan_tiles(count, first, gridDim.x - 1, total, status);
		return;
	}
	const uint64_t t = s_tile - 1;
	const uint32_t rows = (uint32_t) pg_min64(tile_rows, n - t * tile_rows), chunks = (rows + 31) / 32;
	const char* const tile = STAGED ? reinterpret_cast<const char*>(fl_sm) : in + t * tile_rows * w;
	if (STAGED) fl_load_tile(fl_sm, in + t * tile_rows * w, rows * w, &bar, status);
	for (uint32_t c = warp; c < chunks; c += FL_THREADS / 32) {
		const uint32_t i = c * 32 + lane;
		const uint32_t m = __ballot_sync(0xffffffffu, i < rows && pg_pred_eval(P, tile + (STAGED ? i * w : (uint64_t) i * w)));
		if (lane == 0) mask[c] = m;
	}
	__syncthreads();
	if (warp == 0) {
		uint32_t run = 0;
		for (uint32_t c0 = 0; c0 < chunks; c0 += 32) {
			const uint32_t c = c0 + lane, x = c < chunks ? __popc(mask[c]) : 0;
			uint32_t inc = x;
			#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
				if (lane >= (uint32_t) o) inc += y;
			}
			if (c < chunks) before[c] = run + inc - x;
			run += __shfl_sync(0xffffffffu, inc, 31);
		}
		if (lane == 0) {
			pg_st_relaxed(count + t, FL_COUNTED | run);
			unsigned long long v;
			const uint32_t spin = pg_spin_knob(status);
			uint32_t polls = 0;
			while (!((v = pg_ld_relaxed(first + t)) & FL_READY)) {
				++polls;
				if (polls == (spin ? spin : FL_SPIN_LIMIT) || polls >= FL_SPIN_LIMIT) {
					pg_set_status(status, PG_ERR_TIMEOUT);
					if (polls >= FL_SPIN_LIMIT) { v = n; break; }     // nothing is written then
				}
			}
			s_first = v & ~FL_READY;
			s_count = run;
		}
	}
	__syncthreads();
	for (uint32_t i = tid; i < rows; i += FL_THREADS) {
		const uint32_t m = mask[i >> 5];
		if (m >> (i & 31) & 1) sel[before[i >> 5] + __popc(m & ((1u << (i & 31)) - 1))] = (uint16_t) i;
	}
	__syncthreads();
	// Survivor k's units go to row first + k: lanes on consecutive units.
	const uint32_t upt = w / sizeof(U), units = s_count * upt;
	if (s_first + s_count > n) return;                    // the wait gave up
	U* const dst = reinterpret_cast<U*>(out + s_first * w);
	const U* const src = reinterpret_cast<const U*>(tile);
	if (!STAGED) {                                        // a warp Q survivors at once
		constexpr int Q = sizeof(U) == 8 ? 8 : 4;
		const uint32_t count = s_count;
		for (uint32_t k0 = warp; k0 < count; k0 += Q * (FL_THREADS / 32))
			for (uint32_t u = lane; u < upt; u += 32) {
				U v[Q];
				#pragma unroll
				for (int q = 0; q < Q; ++q) {
					const uint32_t k = k0 + q * (FL_THREADS / 32);
					if (k < count) v[q] = __ldcs(src + (uint64_t) sel[k] * upt + u);
				}
				#pragma unroll
				for (int q = 0; q < Q; ++q) {
					const uint32_t k = k0 + q * (FL_THREADS / 32);
					if (k < count) __stcs(dst + (uint64_t) k * upt + u, v[q]);
				}
			}
		return;
	}
	// The loop starts at a 128-byte boundary of the output, so that a warp's
	// store covers whole lines.
	const uint32_t skew = (uint32_t) (reinterpret_cast<uintptr_t>(dst) / sizeof(U)) & (128 / sizeof(U) - 1);
	for (uint32_t i = tid; i < units + skew; i += FL_THREADS) {
		if (i < skew) continue;
		const uint32_t e = i - skew, k = e / upt;
		__stcs(dst + e, src[sel[k] * upt + (e - k * upt)]);
	}
}

extern "C" int pg_filter(pg_ctx* ctx, pg_stream stream, const pg_rel* in, const pg_pred* preds, int npred,
		void* out, uint64_t* n_out)
{
	if (!ctx || !in || !n_out) return pg_fail(ctx, PG_ERR_ARG, "pg_filter: null argument");
	if (in->n && (!in->data || !out)) return pg_fail(ctx, PG_ERR_ARG, "pg_filter: null data");
	if (in->width == 0 || (in->width & 3)) return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_filter: tuple width must be a multiple of 4");
	if (in->n && ((reinterpret_cast<uintptr_t>(in->data) | reinterpret_cast<uintptr_t>(out)) & 3))
		return pg_fail(ctx, PG_ERR_ARG, "pg_filter: data must be 4-byte aligned");
	PgPredSet P;
	bool has_char = false;
	int rc;
	if ((rc = pg_pred_prepare(ctx, preds, npred, in->width, &P, &has_char))) return rc;
	*n_out = 0;
	if (in->n == 0) return PG_OK;
	cudaStream_t s = (cudaStream_t) stream;
	const uint32_t w = in->width;
	uint8_t* chars = nullptr;
	if (has_char) {
		uint8_t host[PG_PRED_MAX * 128];
		memset(host, 0, sizeof host);
		for (int i = 0; i < npred; ++i) memcpy(host + i * 128, preds[i].value, 128);
		if ((rc = pg_alloc_async(ctx, s, (void**) &chars, sizeof host))) return rc;
		PG_CUDA(ctx, cudaMemcpyAsync(chars, host, sizeof host, cudaMemcpyHostToDevice, s));
		PG_CUDA(ctx, cudaStreamSynchronize(s));     // `host` leaves scope
		P.chars = chars;
	}
	uint64_t* scratch = nullptr;
	const bool staged = w <= FL_STAGE_WIDTH;
	const uint32_t rows = staged ? fl_tile_rows(w, FL_TILE_BYTES) : fl_direct_rows(ctx, in->n, FL_DIRECT_ROWS);
	const uint64_t ntiles = pg_div_up(in->n, rows);
	if (ntiles >= (1ull << 31) - 1) {
		pg_free_async(ctx, s, chars);
		return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_filter: too many tuples");
	}
	// [total, two words of pg_readback, ticket, first output row of each tile,
	// survivors of each tile]
	if ((rc = pg_alloc_async(ctx, s, (void**) &scratch, 32 + ntiles * 12))) { pg_free_async(ctx, s, chars); return rc; }
	PG_CUDA(ctx, cudaMemsetAsync(scratch, 0, 32 + ntiles * 12, s));
	unsigned long long* total = reinterpret_cast<unsigned long long*>(scratch);
	const size_t smem = (staged ? (size_t) rows * w : 0) + rows / 32 * 8 + rows * 2;
	const uintptr_t base = reinterpret_cast<uintptr_t>(out) | (staged ? 0 : reinterpret_cast<uintptr_t>(in->data));
#define FL_LAUNCH(U, ST) do { \
		if (ST) PG_CUDA(ctx, cudaFuncSetAttribute(k_filter<U, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)); \
		k_filter<U, ST><<<(unsigned) ntiles + 1, FL_THREADS, smem, s>>>((const char*) in->data, in->n, w, rows, P, \
				reinterpret_cast<uint32_t*>(total + 4 + ntiles), total + 4, reinterpret_cast<unsigned int*>(total + 3), (char*) out, total, ctx->d_status); } while (0)
#define FL_LAUNCH_AS(ST) do { \
		if (!((w | base) & 15)) FL_LAUNCH(uint4, ST); \
		else if (!((w | base) & 7)) FL_LAUNCH(uint2, ST); \
		else FL_LAUNCH(uint32_t, ST); } while (0)
	if (staged) FL_LAUNCH_AS(true);
	else FL_LAUNCH_AS(false);
#undef FL_LAUNCH_AS
#undef FL_LAUNCH
	PG_LAUNCHED(ctx);
	unsigned long long h[2];
	rc = pg_readback(ctx, s, total, 1, nullptr, h, "pg_filter");
	pg_free_async(ctx, s, scratch);
	pg_free_async(ctx, s, chars);
	if (rc) return rc;
	*n_out = h[0];
	return PG_OK;
}

struct ProjCols {
	int n;
	uint16_t src[HJ_PROJ_MAX];    // word offset in the input tuple
	uint8_t words[HJ_PROJ_MAX];
	uint32_t ow;                  // output words
};

// A tile of tuples in shared memory (STAGED) or where it is, then the output rows
// in units of U (1, 2 or 4 words). A thread keeps to one unit of the row, so its source words are
// looked up once; consecutive threads store consecutive units.
template <typename U, bool STAGED>
__global__ void __launch_bounds__(FL_THREADS)
k_project(const char* __restrict__ in, uint64_t n, uint32_t iw, uint32_t tile_rows, const ProjCols pc,
		char* __restrict__ out, int* __restrict__ status)
{
	constexpr uint32_t UW = sizeof(U) / 4;
	extern __shared__ __align__(128) unsigned char pj_sm[];
	__shared__ __align__(8) uint64_t bar;
	const uint64_t t0 = (uint64_t) blockIdx.x * tile_rows;
	const uint32_t rows = (uint32_t) pg_min64(tile_rows, n - t0);
	const uint32_t upt = pc.ow / UW, lanes = FL_THREADS / upt;      // units a row, rows at a time
	const uint32_t r0 = threadIdx.x / upt, u = threadIdx.x - r0 * upt;
	uint32_t src[UW];
	#pragma unroll
	for (uint32_t q = 0; q < UW; ++q) {
		uint32_t k = u * UW + q;
		src[q] = 0;
		#pragma unroll
		for (int c = 0; c < HJ_PROJ_MAX; ++c) {
			if (c >= pc.n) break;
			if (k < pc.words[c]) { src[q] = pc.src[c] + k; break; }
			k -= pc.words[c];
		}
	}
	if (STAGED) fl_load_tile(pj_sm, in + t0 * iw * 4, rows * iw * 4, &bar, status);
	if (r0 >= lanes) return;
	const uint32_t* const tile = reinterpret_cast<const uint32_t*>(STAGED ? reinterpret_cast<const char*>(pj_sm) : in + t0 * iw * 4);
	U* const dst = reinterpret_cast<U*>(out + t0 * pc.ow * 4);
	#pragma unroll 4
	for (uint32_t r = r0; r < rows; r += lanes) {
		const uint32_t* const p = tile + (STAGED ? r * iw : (uint64_t) r * iw);
		U v;
		auto word = [&](uint32_t q) { return STAGED ? p[src[q]] : __ldcs(p + src[q]); };
		if constexpr (UW == 4) v = make_uint4(word(0), word(1), word(2), word(3));
		else if constexpr (UW == 2) v = make_uint2(word(0), word(1));
		else v = word(0);
		__stcs(dst + r * upt + u, v);
	}
}

// Rows wider than a block's units, or of few words of wide tuples: one thread per tuple.
__global__ void k_project_wide(const uint32_t* __restrict__ in, uint64_t n, uint32_t iw, const ProjCols pc,
		uint32_t* __restrict__ out)
{
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t i = (uint64_t) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
		const uint32_t* t = in + i * iw;
		uint32_t* o = out + i * pc.ow;
		uint32_t k = 0;
		#pragma unroll
		for (int c = 0; c < HJ_PROJ_MAX; ++c) {
			if (c >= pc.n) break;
			for (uint32_t q = 0; q < pc.words[c]; ++q) o[k++] = __ldcs(t + pc.src[c] + q);
		}
	}
}

extern "C" int pg_project(pg_ctx* ctx, pg_stream stream, const pg_rel* in, const pg_col* cols, int ncols, void* out)
{
	if (!ctx || !in) return pg_fail(ctx, PG_ERR_ARG, "pg_project: null argument");
	if (ncols < 1 || ncols > HJ_PROJ_MAX || !cols) return pg_fail(ctx, PG_ERR_ARG, "pg_project: 1..16 columns");
	if (in->width == 0 || (in->width & 3)) return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_project: tuple width must be a multiple of 4");
	if (in->n && (!in->data || !out)) return pg_fail(ctx, PG_ERR_ARG, "pg_project: null data");
	if (in->n && ((reinterpret_cast<uintptr_t>(in->data) | reinterpret_cast<uintptr_t>(out)) & 3))
		return pg_fail(ctx, PG_ERR_ARG, "pg_project: data must be 4-byte aligned");
	ProjCols pc;
	pc.n = ncols; pc.ow = 0;
	for (int c = 0; c < ncols; ++c) {
		if ((cols[c].off & 3) || (cols[c].bytes & 3) || cols[c].bytes == 0 || cols[c].off + cols[c].bytes > in->width)
			return pg_fail(ctx, PG_ERR_ARG, "pg_project: columns must be 4-byte multiples inside the tuple");
		pc.src[c] = (uint16_t) (cols[c].off / 4);
		pc.words[c] = (uint8_t) (cols[c].bytes / 4);
		pc.ow += cols[c].bytes / 4;
	}
	if (in->n == 0) return PG_OK;
	cudaStream_t s = (cudaStream_t) stream;
	const uint32_t iw = in->width / 4;
	const uintptr_t o = reinterpret_cast<uintptr_t>(out);
	const uint32_t uw = (pc.ow & 3) == 0 && !(o & 15) ? 4 : (pc.ow & 1) == 0 && !(o & 7) ? 2 : 1;
	const bool staged = in->width <= PJ_STAGE_WIDTH || (in->width <= PJ_STAGE_MAX && 4 * pc.ow > iw);
	const uint32_t rows = staged ? fl_tile_rows(in->width, PJ_TILE_BYTES) : fl_direct_rows(ctx, in->n, PJ_DIRECT_ROWS);
	const uint64_t ntiles = pg_div_up(in->n, rows);
	// Unstaged rows of one word, and of up to four of wide or few tuples: a thread a row,
	// which has all its loads in flight (4 of 136 bytes 99 us against 107 by units, 8: 123 and
	// 110, of 200 and more 83 to 36 either way; 12 of 1000 47 to 56 and 57, of 400 94 and 87;
	// 250,000 tuples, 8 of 400 24 and 31; 50,000, 16 of 400 23 and 32).
	const bool by_row = !staged && (pc.ow == 1 || (pc.ow == 2 && (in->width >= 200 || in->n < 1000000)) ||
			(pc.ow <= 4 && (in->width >= 900 || in->n < 200000)));
	if (!by_row && pc.ow / uw <= FL_THREADS && ntiles < (1ull << 31) - 1) {
		const size_t smem = staged ? (size_t) rows * in->width : 0;
#define PJ_LAUNCH(U, ST) do { \
		if (ST) PG_CUDA(ctx, cudaFuncSetAttribute(k_project<U, ST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)); \
		k_project<U, ST><<<(unsigned) ntiles, FL_THREADS, smem, s>>>((const char*) in->data, in->n, iw, rows, pc, (char*) out, \
				ctx->d_status); } while (0)
#define PJ_LAUNCH_AS(U) do { if (staged) PJ_LAUNCH(U, true); else PJ_LAUNCH(U, false); } while (0)
		if (uw == 4) PJ_LAUNCH_AS(uint4);
		else if (uw == 2) PJ_LAUNCH_AS(uint2);
		else PJ_LAUNCH_AS(uint32_t);
#undef PJ_LAUNCH_AS
#undef PJ_LAUNCH
	} else {
		const int grid = (int) std::min<uint64_t>(pg_div_up(in->n, 256), (uint64_t) ctx->sm_count * 16);
		k_project_wide<<<grid, 256, 0, s>>>((const uint32_t*) in->data, in->n, iw, pc, (uint32_t*) out);
	}
	PG_LAUNCHED(ctx);
	return pg_check_status(ctx, s, "pg_project");
}
