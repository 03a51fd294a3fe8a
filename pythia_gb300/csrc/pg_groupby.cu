// Group-by aggregation (aggregate_sum, aggregate_count) on sm_103a.
//
// Replaces GenericAggregate::remember + fold (operators/genericaggregate.cpp:
// 240-282; aggregatesum.cpp:53-107; aggregatecount.cpp:37-52) and the getNext
// emission of groups (genericaggregate.cpp:419-487). The reference keeps a
// chained table per thread (ThreadLocal) or one locked table (Global); a
// second aggregate over a merge combines thread partials.
//
// Here one open-addressing table per operator holds every group: the key word
// is claimed with atomicCAS, accumulators are updated with atomics. Integer
// sums and counts are exact (wrapping like the reference's CtInt/CtLong +=).
// Dec (double) sums are exact fixed-point integers (pg_fixsum.h): a value
// becomes a count of units 2^s, counts add into seven words per group with
// integer atomics (a value near the column's largest: one returning add, its
// old word giving the rare overflow into another word), and the sum is
// rounded to a double once at emission. Integer adds do not depend on the
// order in which threads arrive, so every run gives the same bits; when all
// values are within 2^135 of the largest, the result is the correctly rounded
// exact sum. The unit comes from the largest exponent of the column (sampled,
// with a margin, on large inputs; a value above the bound makes the operator
// redo the sum with the exact bound). Infinities and NaNs are summed on the
// side and patch their groups' results. Blocks add the rows of groups they
// meet often in shared memory first, which cuts L2 atomics on skewed keys.
#include "pg_groupshared.cuh"

#define GB_THREADS 256

// An open-addressing group table. A group's aggregate is one word of acc (a
// count, a long sum, an int sum in its low 4 bytes) or, for a dec sum, the
// table words of its count of units (pg_fixsum.h) at acc[slot + k * (cap +
// 1)], k < PG_FX_WORDS.
struct GbTable {
	unsigned long long* keys;   // [cap + 1]; slot cap is the group whose key is the empty marker
	unsigned long long* acc;    // [PG_FX_WORDS (cap + 1)]
	int* sentinel_used;
	uint32_t log2cap;
	__device__ __forceinline__ uint64_t wstride() const { return (1ull << log2cap) + 1; }
};

// One row's (or a combined run's) value: an integer, or a dec sum's count.
struct GbVal {
	unsigned long long i;
	pg_fx4 f;
};

// Adds v into the aggregate of slot `slot` (a dec sum's word k at acc[slot +
// k * wstride]).
template <int VT, int AGG>
__device__ __forceinline__ void fold_slot(unsigned long long* acc, uint64_t wstride, uint64_t slot, const GbVal& v)
{
	if (AGG == PG_AGG_COUNT) atomicAdd(&acc[slot], v.i);
	else if (VT == PG_VAL_LONG) atomicAdd(&acc[slot], v.i);
	else if (VT == PG_VAL_INT) atomicAdd(reinterpret_cast<unsigned int*>(&acc[slot]), (unsigned int) v.i);
	else pg_fx_atomic_add(&acc[slot], wstride, v.f);
}

// Adds count a into four chained words t[k * stride] in shared memory. A value near the
// column's largest is two 32-bit adds on t2, where 64-bit ones were compare-and-swap loops:
// 20M rows hashed into 10 groups 403 -> 208 us, into 300 408 -> 387, into 100,000 536 -> 514.
__device__ __forceinline__ void gb_shared_chain_add(unsigned long long* t, uint32_t stride, const pg_fx3& a)
{
	pg_fx_chain_add_halves(reinterpret_cast<uint32_t*>(t), stride, a, [](uint32_t* p, uint32_t v) { return atomicAdd(p, v); });
}

// A dec sum's count from table words acc[slot + k * wstride].
__device__ __forceinline__ pg_fx4 gb_table_count(const unsigned long long* acc, uint64_t wstride, uint64_t slot)
{
	return pg_fx_from_table(reinterpret_cast<const uint64_t*>(acc + slot), wstride);
}

// Loads one row's value (a dec value quantised for unit 2^fs, bound fb).
template <int VT, int AGG>
__device__ __forceinline__ GbVal gb_load_val(const char* r, uint32_t voff, int fs, int fb, uint32_t& fl)
{
	GbVal v = {0, {0, 0, 0, 0}};
	if (AGG == PG_AGG_COUNT) v.i = 1;
	else if (VT == PG_VAL_INT) v.i = (unsigned long long) (long long) *reinterpret_cast<const int32_t*>(r + voff);
	else if (VT == PG_VAL_LONG) v.i = (unsigned long long) pg_load_key(r + voff, 8);
	else v.f = pg_fx_widen(pg_fx_take((uint64_t) pg_load_key(r + voff, 8), fs, fb, fl));
	return v;
}

// Finds or claims the slot of key k. Returns cap (the side slot) for the
// empty-marker key, or UINT64_MAX when the table is full.
__device__ __forceinline__ uint64_t gb_slot(unsigned long long* keys, uint32_t log2cap, int64_t k,
		int* sentinel_used)
{
	const uint64_t cap = 1ull << log2cap, mask = cap - 1;
	if (k == PG_EMPTY_KEY) { if (!*sentinel_used) atomicExch(sentinel_used, 1); return cap; }
	uint64_t s = pg_mix64((uint64_t) k) >> (64 - log2cap);
	for (uint64_t probe = 0; probe < cap; ++probe) {
		unsigned long long cur = keys[s];
		if (cur == (unsigned long long) k) return s;
		if (cur == (unsigned long long) PG_EMPTY_KEY) {
			unsigned long long old = atomicCAS(&keys[s], (unsigned long long) PG_EMPTY_KEY, (unsigned long long) k);
			if (old == (unsigned long long) PG_EMPTY_KEY || old == (unsigned long long) k) return s;
		}
		s = (s + 1) & mask;
	}
	return UINT64_MAX;
}

// Combines the values of lanes in `peers` (same key) at the leader lane:
// integer adds (256-bit for dec sums' counts of units), exact in any order.
template <int VT, int AGG>
__device__ __forceinline__ void warp_combine(uint32_t peers, GbVal& v)
{
	GbVal t = {0, {0, 0, 0, 0}};
	uint32_t m = peers;
	while (m) {
		const int src = __ffs(m) - 1; m &= m - 1;
		if (GB_DEC) {
			const pg_fx4 x = {__shfl_sync(peers, v.f.w0, src), __shfl_sync(peers, v.f.w1, src),
			                  __shfl_sync(peers, v.f.w2, src), __shfl_sync(peers, v.f.w3, src)};
			pg_fx_add4(t.f, x);
		} else {
			t.i += __shfl_sync(peers, v.i, src);
		}
	}
	v = t;
}

// No GROUP BY: one group. Warps fold their rows, then each block adds once.
template <int VT, int AGG>
__global__ void __launch_bounds__(GB_THREADS)
k_gb_single(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t voff, GbTable t, PgFx fx)
{
	__shared__ unsigned long long sacc[PG_FX_WORDS];
	if (threadIdx.x < PG_FX_WORDS) sacc[threadIdx.x] = 0;
	__syncthreads();
	uint32_t fl = 0;
	const int fs = GB_DEC ? fx.p[0] : 0, fb = GB_DEC ? fx.p[1] : 0;
	GbVal v = {0, {0, 0, 0, 0}};
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += stride) {
		const GbVal x = gb_load_val<VT, AGG>(in + i * W, voff, fs, fb, fl);
		if (GB_DEC) pg_fx_add4(v.f, x.f);
		else v.i += x.i;
	}
	warp_combine<VT, AGG>(0xffffffffu, v);
	if ((threadIdx.x & 31) == 0) fold_slot<VT, AGG>(sacc, 1, 0, v);
	if (fl) atomicOr(reinterpret_cast<unsigned int*>(fx.p + 2), fl);
	__syncthreads();
	if (threadIdx.x == 0) {
		GbVal s = {sacc[0], {0, 0, 0, 0}};
		if (GB_DEC) s.f = gb_table_count(sacc, 1, 0);
		fold_slot<VT, AGG>(t.acc, t.wstride(), 0, s);
	}
}

// Writes one group's row: kbytes of key (none for 0), then its aggregate:
// word a, or for a dec sum the count c of units 2^fx_s rounded to a double.
template <int VT, int AGG>
__device__ __forceinline__ void gb_write_agg(char* o, uint32_t kbytes, int64_t k, unsigned long long a,
		const pg_fx4& c, int fx_s)
{
	if (kbytes == 4) *reinterpret_cast<int32_t*>(o) = (int32_t) k;
	else if (kbytes == 8) {
		reinterpret_cast<uint32_t*>(o)[0] = (uint32_t) k;
		reinterpret_cast<uint32_t*>(o)[1] = (uint32_t) ((uint64_t) k >> 32);
	}
	o += kbytes;
	if (AGG == PG_AGG_SUM && VT == PG_VAL_INT) { *reinterpret_cast<uint32_t*>(o) = (uint32_t) a; return; }
	if (GB_DEC) a = (unsigned long long) __double_as_longlong(pg_fx_double4(c, fx_s));
	reinterpret_cast<uint32_t*>(o)[0] = (uint32_t) a;
	reinterpret_cast<uint32_t*>(o)[1] = (uint32_t) (a >> 32);
}

template <int VT, int AGG, bool HASKEY>
__global__ void k_gb_emit(GbTable t, uint32_t kbytes, char* __restrict__ out, uint64_t cap_rows,
		unsigned long long* __restrict__ cursor, uint64_t nonkey_rows, PgFx fx, const int* __restrict__ status)
{
	if (blockIdx.x == 0 && threadIdx.x == 0) pg_collect(cursor + 1, GB_DEC ? fx.p + 2 : nullptr, status);
	const int fx_s = GB_DEC ? fx.p[0] : 0;
	const uint64_t cap = 1ull << t.log2cap;
	const uint32_t aw = (AGG == PG_AGG_SUM && VT == PG_VAL_INT) ? 4 : 8;
	const uint32_t ow = (HASKEY ? kbytes : 0) + aw;
	const uint64_t limit = HASKEY ? cap + 1 : 1;
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < pg_div_up(limit, 32) * 32;
			i += (uint64_t) gridDim.x * blockDim.x) {
		bool used = false;
		if (i < limit) {
			if (!HASKEY) used = nonkey_rows > 0;
			else if (i < cap) used = t.keys[i] != (unsigned long long) PG_EMPTY_KEY;
			else used = *t.sentinel_used != 0;
		}
		uint32_t ball = __ballot_sync(0xffffffffu, used);
		if (!ball) continue;
		int lane = threadIdx.x & 31;
		unsigned long long base = 0;
		if (lane == __ffs(ball) - 1) base = atomicAdd(cursor, (unsigned long long) __popc(ball));
		base = __shfl_sync(0xffffffffu, base, __ffs(ball) - 1);
		if (!used) continue;
		uint64_t pos = base + __popc(ball & ((1u << lane) - 1));
		if (pos >= cap_rows) continue;
		const int64_t k = HASKEY ? (i < cap ? (int64_t) t.keys[i] : PG_EMPTY_KEY) : 0;
		gb_write_agg<VT, AGG>(out + pos * ow, HASKEY ? kbytes : 0, k, t.acc[i],
				GB_DEC ? gb_table_count(t.acc, t.wstride(), i) : pg_fx4{0, 0, 0, 0}, fx_s);
	}
}

// ---------------------------------------------------------------------------
// Dense key domain (keys span at most a few times the group count, e.g.
// group numbers 0..G-1 or surrogate keys): a min/max pass, then the slot of a
// row is key - kmin. No probing and no key words: a row costs its atomics
// (one for a typical dec value, as for the integer aggregates); a sum's first
// add marks the group present. A dec sum's table keeps
// each of its PG_FX_WORDS words in an array of its own (word k of slot i at
// acc[i + k * range]), so the word every row adds into takes 8 bytes a group
// of L2.
// ---------------------------------------------------------------------------
// Min and max key over rows 0, step, 2 step, ... (step 1: every row).
template <bool VEC16>
__global__ void k_gb_key_minmax(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff,
		uint32_t kbytes, unsigned long long* __restrict__ mm, uint64_t step)
{
	unsigned long long lo = ~0ull, hi = 0;
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	const uint64_t ns = pg_div_up(n, step);
	for (uint64_t j = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; j < ns; j += stride) {
		const uint64_t i = j * step;
		int64_t k;
		if (VEC16) {
			const uint4 t = __ldg(reinterpret_cast<const uint4*>(in) + i);
			k = koff == 0 ? (int64_t) (((uint64_t) t.y << 32) | t.x) : (int64_t) (((uint64_t) t.w << 32) | t.z);
		} else {
			k = pg_load_key(in + i * W + koff, kbytes);
		}
		const unsigned long long u = (unsigned long long) k ^ (1ull << 63);
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

// Key and value words of row i: the 8-byte key at koff and the value at voff
// (an int sign-extended), from one 16-byte load when VEC16.
template <int VT, bool VEC16>
__device__ __forceinline__ void gb_row_kv(const char* __restrict__ in, uint64_t i, uint32_t W, uint32_t koff,
		uint32_t kbytes, uint32_t voff, int64_t& k, uint64_t& vbits)
{
	if (VEC16) {
		const uint4 t = __ldg(reinterpret_cast<const uint4*>(in) + i);
		k = koff == 0 ? (int64_t) (((uint64_t) t.y << 32) | t.x) : (int64_t) (((uint64_t) t.w << 32) | t.z);
		vbits = voff == 0 ? (((uint64_t) t.y << 32) | t.x) : voff == 8 ? (((uint64_t) t.w << 32) | t.z)
			: voff == 4 ? t.y : t.w;
		if (VT == PG_VAL_INT) vbits = (uint64_t) (int64_t) (int32_t) (voff == 0 ? t.x : voff == 4 ? t.y : voff == 8 ? t.z : t.w);
	} else {
		const char* r = in + i * W;
		k = pg_load_key(r + koff, kbytes);
		vbits = VT == PG_VAL_INT ? (uint64_t) (int64_t) *reinterpret_cast<const int32_t*>(r + voff)
			: (uint64_t) pg_load_key(r + voff, 8);
	}
}

// ---------------------------------------------------------------------------
// Hashed groups: a table of 4-key buckets, so that one 32-byte load finds a
// row's group (at load 1/2 a key's home bucket overflows for one key in 20;
// slot-by-slot probing made the 32 lanes of a warp wait for the longest of
// their probe sequences), then one atomic. In front of it every block keeps
// the groups it met first in a small direct-mapped table in shared memory and
// adds their rows there: keys that many rows share, which would queue at one
// L2 address, are met early.
//
// Bound by L2 (a random bucket read and an atomic a row). One row in flight a
// thread, six blocks on an SM and about 64 blocks per SM in turn measured
// best: 20M rows in 250,000 groups 320 us, against 530 with six blocks per SM
// and 1010 with four rows a thread in three resident blocks. Partitioning the
// rows first (shared-memory tables per partition) took 850 us, and 9.5 ms for
// 64M rows in 4M groups where this takes 1.6.
// ---------------------------------------------------------------------------
#define GBH_CACHE_LOG2 8                    // groups kept per block: 256 (4 KB, 10 KB for dec)
#define GBH_BLOCKS_PER_SM 64
// Few groups: room for all of them in every block (32 KB, 40 KB for dec), and
// fewer blocks, which each end by adding their groups to the table: eight rows a
// block for every group, unless that would leave an SM without its five blocks (1M rows in
// 300 groups 113 -> 94 us, dec 149 -> 119). 20M rows in 1000 groups: 180 us, 527 with 256
// places.
#define GBH_FEW 1024u
#define GBH_FEW_ROWS 8
#define GBH_FEW_RESIDENT 5
#define GBH_FEW_LOG2 (GB_DEC ? 10 : 11)
#define GBH_FEW_PROBES 4
#define GBH_FEW_BLOCKS_PER_SM 24

// The bucket's keys straight from L2 (other blocks insert concurrently; an
// empty slot seen late only costs the atomicCAS that finds it taken).
__device__ __forceinline__ pg_u64x4 gbh_bucket(const unsigned long long* p)
{
	pg_u64x4 v;
	asm volatile("ld.relaxed.gpu.global.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(v.a), "=l"(v.b), "=l"(v.c), "=l"(v.d) : "l"(p) : "memory");
	return v;
}

// Slot of key k (not the empty marker), whose home bucket b0 was read as v:
// found or claimed there, else in the buckets after it. UINT64_MAX when every
// bucket is full.
__device__ __forceinline__ uint64_t gbh_slot(unsigned long long* keys, uint32_t log2cap, unsigned long long k, uint64_t b,
		pg_u64x4 v)
{
	const uint64_t nb = 1ull << (log2cap - 2);
	for (uint64_t probe = 0; probe < nb; ++probe) {
		if (v.a == k) return 4 * b;
		if (v.b == k) return 4 * b + 1;
		if (v.c == k) return 4 * b + 2;
		if (v.d == k) return 4 * b + 3;
		// Slots fill in order: claim the first empty one, or find there the
		// key that took it meanwhile.
		const unsigned long long empty = (unsigned long long) PG_EMPTY_KEY;
		#pragma unroll
		for (int i = 0; i < 4; ++i) {
			const unsigned long long cur = i == 0 ? v.a : i == 1 ? v.b : i == 2 ? v.c : v.d;
			if (cur != empty) continue;
			const unsigned long long old = atomicCAS(&keys[4 * b + i], empty, k);
			if (old == empty || old == k) return 4 * b + i;
		}
		b = (b + 1) & (nb - 1);
		v = gbh_bucket(keys + 4 * b);
	}
	return UINT64_MAX;
}

template <int VT, int AGG, bool VEC16>
__global__ void __launch_bounds__(GB_THREADS, 6)
k_gb_hash(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes, uint32_t voff,
		GbTable t, uint32_t places, uint32_t probes, PgFx fx, int* __restrict__ status)
{
	extern __shared__ __align__(16) unsigned char gbh_sm[];
	unsigned long long* const skeys = reinterpret_cast<unsigned long long*>(gbh_sm);   // [places], a power of two
	unsigned long long* const sacc = skeys + places;                                  // [places], for dec 4 words places apart
	for (uint32_t i = threadIdx.x; i < places; i += blockDim.x) skeys[i] = (unsigned long long) PG_EMPTY_KEY;
	for (uint32_t i = threadIdx.x; i < (GB_DEC ? 4 : 1) * places; i += blockDim.x) sacc[i] = 0;
	__syncthreads();
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	bool full = false;
	uint32_t fl = 0;
	const int fs = GB_DEC ? fx.p[0] : 0, fb = GB_DEC ? fx.p[1] : 0;
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += stride) {
		int64_t k;
		uint64_t vbits = 0;
		if (AGG == PG_AGG_COUNT && !VEC16) k = pg_load_key(in + i * W + koff, kbytes);
		else gb_row_kv<VT, VEC16>(in, i, W, koff, kbytes, voff, k, vbits);
		GbVal v = {AGG == PG_AGG_COUNT ? 1 : vbits, {0, 0, 0, 0}};
		pg_fx3 f = {0, 0, 0};
		if (GB_DEC) f = pg_fx_take(vbits, fs, fb, fl);
		if (k == PG_EMPTY_KEY) {
			if (!*t.sentinel_used) atomicExch(t.sentinel_used, 1);
			v.f = pg_fx_widen(f);
			fold_slot<VT, AGG>(t.acc, t.wstride(), 1ull << t.log2cap, v);
			continue;
		}
		const uint64_t h = pg_mix64((uint64_t) k);
		uint32_t c = (uint32_t) h & (places - 1);
		bool here = false;
		for (uint32_t p = 0; p < probes; ++p, c = (c + 1) & (places - 1)) {
			unsigned long long cur = *(volatile unsigned long long*) &skeys[c];
			if (cur == (unsigned long long) PG_EMPTY_KEY) {
				cur = atomicCAS(&skeys[c], (unsigned long long) PG_EMPTY_KEY, (unsigned long long) k);
				if (cur == (unsigned long long) PG_EMPTY_KEY) cur = (unsigned long long) k;
			}
			if (cur == (unsigned long long) k) { here = true; break; }
		}
		if (here) {
			if (GB_DEC) gb_shared_chain_add(&sacc[c], places, f);
			else if (VT == PG_VAL_INT && AGG == PG_AGG_SUM) fold_slot<VT, AGG>(sacc, places, c, v);
			else gb_shared_add64(&sacc[c], v.i);
			continue;
		}
		const uint64_t b = h >> (66 - t.log2cap);
		const uint64_t slot = gbh_slot(t.keys, t.log2cap, (unsigned long long) k, b, gbh_bucket(t.keys + 4 * b));
		if (slot == UINT64_MAX) { full = true; continue; }
		if (GB_DEC) {
			const uint64_t at[1] = {slot};
			const bool ok[1] = {true};
			const pg_fx3 x[1] = {f};
			pg_fx_atomic_add_rows<1>(t.acc, t.wstride(), at, 1, ok, x, nullptr);
		} else fold_slot<VT, AGG>(t.acc, t.wstride(), slot, v);
	}
	__syncthreads();
	for (uint32_t i = threadIdx.x; i < places; i += blockDim.x) {
		const unsigned long long k = skeys[i];
		if (k == (unsigned long long) PG_EMPTY_KEY) continue;
		const uint64_t b = pg_mix64(k) >> (66 - t.log2cap);
		const uint64_t slot = gbh_slot(t.keys, t.log2cap, k, b, gbh_bucket(t.keys + 4 * b));
		if (slot == UINT64_MAX) { full = true; continue; }
		GbVal v = {sacc[i], {0, 0, 0, 0}};
		if (GB_DEC) v.f = pg_fx_from_chain(reinterpret_cast<const uint64_t*>(sacc + i), places);
		fold_slot<VT, AGG>(t.acc, t.wstride(), slot, v);
	}
	if (full) pg_set_status(status, PG_ERR_TABLE_FULL);
	if (fl) atomicOr(reinterpret_cast<unsigned int*>(fx.p + 2), fl);
}

#define GBD_ILP 4
// ILP rows per thread in flight (their loads and atomics issued together).
template <int VT, int AGG, bool VEC16, int ILP>
__global__ void __launch_bounds__(GB_THREADS)
k_gb_dense(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes, uint32_t voff,
		long long kmin, uint64_t range, unsigned long long* __restrict__ acc, PgFx fx,
		unsigned char* __restrict__ present, unsigned int* __restrict__ overflow)
{
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	bool outside = false;
	uint32_t fl = 0;
	const int fs = GB_DEC ? fx.p[0] : 0, fb = GB_DEC ? fx.p[1] : 0;
	for (uint64_t base = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; base < n; base += stride * ILP) {
		uint64_t d[ILP];
		unsigned long long iv[ILP];
		pg_fx3 f[ILP];
		bool ok[ILP];
		#pragma unroll
		for (int j = 0; j < ILP; ++j) {
			const uint64_t i = base + j * stride;
			ok[j] = i < n;
			d[j] = 0; iv[j] = 0; f[j] = pg_fx3{0, 0, 0};
			if (!ok[j]) continue;
			int64_t k;
			uint64_t vbits;
			gb_row_kv<VT, VEC16>(in, i, W, koff, kbytes, voff, k, vbits);
			d[j] = (uint64_t) k - (uint64_t) kmin;
			if (d[j] >= range) { ok[j] = false; outside = true; d[j] = 0; continue; }   // key outside the table
			if (AGG == PG_AGG_COUNT) iv[j] = 1;
			else if (GB_DEC) f[j] = pg_fx_take(vbits, fs, fb, fl);
			else iv[j] = vbits;
		}
		if (GB_DEC) {
			pg_fx_atomic_add_rows<ILP>(acc, range, d, 1, ok, f, present);
		} else {
			// A sum's first add returns the initial 0 and marks its group: a
			// byte store a row beside an add that returns nothing took longer
			// (3.10 against 2.50 ms for 256M rows in 1M groups).
			unsigned long long old[ILP];
			#pragma unroll
			for (int j = 0; j < ILP; ++j) {
				old[j] = 1;
				if (!ok[j]) continue;
				if (AGG == PG_AGG_COUNT) atomicAdd(&acc[d[j]], iv[j]);
				else if (VT == PG_VAL_INT)
					old[j] = atomicAdd(reinterpret_cast<unsigned int*>(&acc[d[j]]), (unsigned int) iv[j]);
				else old[j] = atomicAdd(&acc[d[j]], iv[j]);
			}
			if (AGG == PG_AGG_SUM) {
				#pragma unroll
				for (int j = 0; j < ILP; ++j)
					if (old[j] == 0) present[d[j]] = 1;
			}
		}
	}
	if (outside) *overflow = 1;
	if (fl) atomicOr(reinterpret_cast<unsigned int*>(fx.p + 2), fl);
}

// Dense group-by over a window whose table fits in shared memory (GbShared). Int and
// long sums are bound by the read, dec ones by instructions (75% of issue):
// 64M rows in 300 groups 223, 224 and 352 us, as before but for dec's 520; in 3000 (over
// 1500 in L2 before, dec at 57 bytes a slot) 223, 224 and 351 from 1540 to 1750; in
// 12,000, long and dec with one CTA an SM, 230, 328 and 438 from 1550, 1550 and 1000. One
// row a thread, the next one loaded, and 64 warps an SM: dec 352, four rows and 32 warps
// 466.
template <int VT, int AGG, bool VEC16, bool LAZY>
__global__ void __launch_bounds__(GBS_THREADS, 2)
k_gb_dense_smem(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff, uint32_t kbytes, uint32_t voff,
		long long kmin, uint32_t range, unsigned long long* __restrict__ acc, PgFx fx,
		unsigned char* __restrict__ present, unsigned int* __restrict__ overflow)
{
	extern __shared__ __align__(16) unsigned char gsm[];
	GbShared<VT, AGG, LAZY> t(gsm, range, acc, fx);
	const uint64_t stride = (uint64_t) gridDim.x * blockDim.x;
	bool outside = false;
	int64_t k = 0;
	uint64_t vbits = 0;
	uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x;
	if (i < n) gb_row_kv<VT, VEC16>(in, i, W, koff, kbytes, voff, k, vbits);
	for (; i < n; i += stride) {
		const uint64_t d = (uint64_t) k - (uint64_t) kmin, v = vbits;
		if (i + stride < n) gb_row_kv<VT, VEC16>(in, i + stride, W, koff, kbytes, voff, k, vbits);
		if (d < range) t.add((uint32_t) d, v);
		else outside = true;                                // key outside the table
	}
	if (outside) *overflow = 1;
	if (t.fl) atomicOr(reinterpret_cast<unsigned int*>(fx.p + 2), t.fl);
	t.flush(present);
}

template <int VT, int AGG>
__global__ void k_gb_dense_emit(const unsigned long long* __restrict__ acc, PgFx fx,
		const unsigned char* __restrict__ present, uint64_t range, long long kmin, uint32_t kbytes,
		char* __restrict__ out, uint64_t cap_rows, unsigned long long* __restrict__ cursor, unsigned long long* __restrict__ tail,
		const int* __restrict__ status)
{
	if (blockIdx.x == 0 && threadIdx.x == 0) pg_collect(tail, GB_DEC ? fx.p + 2 : nullptr, status);
	const int fx_s = GB_DEC ? fx.p[0] : 0;
	const uint32_t aw = (AGG == PG_AGG_SUM && VT == PG_VAL_INT) ? 4 : 8;
	const uint32_t ow = kbytes + aw;
	const int lane = threadIdx.x & 31;
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < pg_div_up(range, 32) * 32;
			i += (uint64_t) gridDim.x * blockDim.x) {
		const bool used = i < range && (AGG == PG_AGG_COUNT ? acc[i] != 0 : present[i] != 0);
		const uint32_t ball = __ballot_sync(0xffffffffu, used);
		if (!ball) continue;
		unsigned long long base = 0;
		if (lane == 0) base = atomicAdd(cursor, (unsigned long long) __popc(ball));
		base = __shfl_sync(0xffffffffu, base, 0);
		if (!used) continue;
		const uint64_t pos = base + __popc(ball & ((1u << lane) - 1));
		if (pos >= cap_rows) continue;
		const int64_t k = (int64_t) ((uint64_t) kmin + i);
		if (GB_DEC)
			gb_write_agg<VT, AGG>(out + pos * ow, kbytes, k, 0, gb_table_count(acc, range, i), fx_s);
		else gb_write_agg<VT, AGG>(out + pos * ow, kbytes, k, acc[i], pg_fx4{0, 0, 0, 0}, 0);
	}
}

// ---------------------------------------------------------------------------
// Dec sums: the unit, and the groups that met infinities or NaNs
// ---------------------------------------------------------------------------
// Largest finite exponent field of the 8-byte column at voff over rows 0,
// step, 2 step, ... into p[3].
__global__ void k_fx_max_field(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t voff, uint64_t step,
		int* __restrict__ p)
{
	int m = 0;
	const uint64_t ns = pg_div_up(n, step);
	for (uint64_t j = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; j < ns; j += (uint64_t) gridDim.x * blockDim.x) {
		const int e = pg_fx_field((uint64_t) pg_load_key(in + j * step * W + voff, 8));
		if (e != PG_FX_EXP_SPECIAL && e > m) m = e;
	}
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
	if ((threadIdx.x & 31) == 0 && m) atomicMax(&p[3], m);
}

// p[0] unit exponent, p[1] bound, p[2] flags cleared, from the field in p[3].
__global__ void k_fx_finish(int* __restrict__ p, int margin)
{
	const int bound = min(p[3] + margin, PG_FX_EXP_SPECIAL - 1);
	p[0] = pg_fx_unit(bound);
	p[1] = bound;
	p[2] = 0;
}

int pg_fx_prepare(pg_ctx* ctx, cudaStream_t s, const char* data, uint64_t n, uint32_t W, uint32_t voff,
		uint64_t step, int margin, PgFx fx)
{
	PG_CUDA(ctx, cudaMemsetAsync(fx.p, 0, 16, s));
	if (n) {
		const int blocks = (int) std::max<uint64_t>(1, std::min<uint64_t>(pg_div_up(pg_div_up(n, step), 256),
				(uint64_t) ctx->sm_count * 8));
		k_fx_max_field<<<blocks, 256, 0, s>>>(data, n, W, voff, step, fx.p);
		PG_LAUNCHED(ctx);
	}
	k_fx_finish<<<1, 1, 0, s>>>(fx.p, step > 1 ? margin : 0);
	PG_LAUNCHED(ctx);
	return PG_OK;
}

// Rows whose dec value is an infinity or NaN, counted.
__global__ void k_fx_special_count(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t voff,
		unsigned long long* __restrict__ cnt)
{
	unsigned long long c = 0;
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
		c += pg_fx_field((uint64_t) pg_load_key(in + i * W + voff, 8)) == PG_FX_EXP_SPECIAL;
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
	if ((threadIdx.x & 31) == 0 && c) atomicAdd(cnt, c);
}

// The special values of each group that has any, OR-ed into fl[slot] of a
// small table of their keys (all rows key 0 when kbytes is 0).
__global__ void k_fx_special_collect(const char* __restrict__ in, uint64_t n, uint32_t W, uint32_t koff,
		uint32_t kbytes, uint32_t voff, unsigned long long* __restrict__ keys, unsigned int* __restrict__ fl,
		uint32_t log2cap, int* __restrict__ sentinel)
{
	for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x) {
		const uint64_t b = (uint64_t) pg_load_key(in + i * W + voff, 8);
		if (pg_fx_field(b) != PG_FX_EXP_SPECIAL) continue;
		const int64_t k = kbytes ? pg_load_key(in + i * W + koff, kbytes) : 0;
		const uint64_t slot = gb_slot(keys, log2cap, k, sentinel);
		if (slot != UINT64_MAX) atomicOr(&fl[slot], pg_fx_special(b));
	}
}

// Output rows (key of kbytes, then the 8-byte sum) of groups in the table get
// the IEEE result of their special values.
__global__ void k_fx_special_patch(char* __restrict__ out, uint64_t rows, uint32_t kbytes,
		const unsigned long long* __restrict__ keys, const unsigned int* __restrict__ fl, uint32_t log2cap,
		const int* __restrict__ sentinel)
{
	const uint64_t cap = 1ull << log2cap;
	for (uint64_t r = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; r < rows; r += (uint64_t) gridDim.x * blockDim.x) {
		char* o = out + r * (kbytes + 8);
		int64_t k = 0;
		if (kbytes == 4) k = *reinterpret_cast<const int32_t*>(o);
		else if (kbytes == 8)
			k = (int64_t) (((uint64_t) reinterpret_cast<const uint32_t*>(o)[1] << 32) | reinterpret_cast<const uint32_t*>(o)[0]);
		uint64_t slot = UINT64_MAX;
		if (k == PG_EMPTY_KEY) { if (*sentinel) slot = cap; }
		else {
			uint64_t h = pg_mix64((uint64_t) k) >> (64 - log2cap);
			for (uint64_t probe = 0; probe < cap; ++probe, h = (h + 1) & (cap - 1)) {
				if (keys[h] == (unsigned long long) k) { slot = h; break; }
				if (keys[h] == (unsigned long long) PG_EMPTY_KEY) break;
			}
		}
		if (slot == UINT64_MAX || !fl[slot]) continue;
		const uint64_t v = pg_fx_special_bits(fl[slot]);
		reinterpret_cast<uint32_t*>(o + kbytes)[0] = (uint32_t) v;
		reinterpret_cast<uint32_t*>(o + kbytes)[1] = (uint32_t) (v >> 32);
	}
}

int pg_fx_patch_specials(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint32_t voff, char* out, uint64_t ngroups)
{
	int rc;
	unsigned long long* cnt = nullptr;
	if ((rc = pg_alloc_async(ctx, s, (void**) &cnt, 16))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(cnt, 0, 16, s));
	const int blocks = (int) std::max<uint64_t>(1, std::min<uint64_t>(pg_div_up(in->n, 256), (uint64_t) ctx->sm_count * 8));
	k_fx_special_count<<<blocks, 256, 0, s>>>((const char*) in->data, in->n, in->width, voff, cnt);
	PG_LAUNCHED(ctx);
	unsigned long long h = 0;
	PG_CUDA(ctx, cudaMemcpyAsync(&h, cnt, 8, cudaMemcpyDeviceToHost, s));
	PG_CUDA(ctx, cudaStreamSynchronize(s));
	pg_free_async(ctx, s, cnt);
	if (!h || !ngroups) return PG_OK;
	uint32_t lg = 6;
	while ((1ull << lg) < 2 * h) ++lg;
	const uint64_t cap = 1ull << lg;
	char* mem = nullptr;
	if ((rc = pg_alloc_async(ctx, s, (void**) &mem, (cap + 1) * 12 + 16))) return rc;
	unsigned long long* keys = reinterpret_cast<unsigned long long*>(mem);
	unsigned int* fl = reinterpret_cast<unsigned int*>(keys + cap + 1);
	int* sentinel = reinterpret_cast<int*>(fl + cap + 1);
	PG_CUDA(ctx, cudaMemsetAsync(keys, 0xFF, (cap + 1) * 8, s));
	PG_CUDA(ctx, cudaMemsetAsync(fl, 0, (cap + 1) * 4 + 8, s));
	k_fx_special_collect<<<blocks, 256, 0, s>>>((const char*) in->data, in->n, in->width, in->key_off, in->key_bytes,
			voff, keys, fl, lg, sentinel);
	PG_LAUNCHED(ctx);
	const int pblocks = (int) std::max<uint64_t>(1, std::min<uint64_t>(pg_div_up(ngroups, 256), (uint64_t) ctx->sm_count * 8));
	k_fx_special_patch<<<pblocks, 256, 0, s>>>(out, ngroups, in->key_bytes, keys, fl, lg, sentinel);
	PG_LAUNCHED(ctx);
	pg_free_async(ctx, s, mem);
	return PG_OK;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Rows that gb_row_kv reads with one 16-byte load.
template <int VT, int AGG>
static bool gb_vec16(const pg_rel* in, uint32_t voff)
{
	return in->width == 16 && (in->key_off == 0 || in->key_off == 8) && in->key_bytes == 8 &&
		(reinterpret_cast<uintptr_t>(in->data) & 15) == 0 &&
		(AGG == PG_AGG_COUNT || (VT == PG_VAL_INT ? (voff & 3) == 0 : (voff == 0 || voff == 8)));
}

// One dense aggregation over the key window [kmin, kmin + range): table, fill,
// aggregation, emission. *overflow: some key lay outside the window (nothing
// of this run is usable then); *fxfl: the dec sum's flags (fx).
template <int VT, int AGG>
static int gb_dense_window(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint32_t voff, bool vec16, long long kmin,
		uint64_t range, void* out, uint64_t out_cap, uint64_t* ngroups, bool* overflow, PgFx fx, uint32_t* fxfl)
{
	int rc;
	char* mem = nullptr;
	const uint64_t words = range * (GB_DEC ? PG_FX_WORDS : 1);
	const size_t bytes = words * 8 + 32 + range;
	if ((rc = pg_alloc_async(ctx, s, (void**) &mem, bytes))) return rc;
	unsigned long long* acc = reinterpret_cast<unsigned long long*>(mem);      // a dec sum: word k of slot i at acc[i + k range]
	unsigned long long* cursor = acc + words;
	unsigned int* oflag = reinterpret_cast<unsigned int*>(cursor + 1);         // then two words of pg_readback
	unsigned char* present = reinterpret_cast<unsigned char*>(cursor + 4);
	PG_CUDA(ctx, cudaMemsetAsync(mem, 0, bytes, s));
	const GbsPlan plan = gbs_plan<VT, AGG>(range);
	auto* const kernel = vec16
			? plan.lazy ? k_gb_dense_smem<VT, AGG, true, GB_DEC> : k_gb_dense_smem<VT, AGG, true, false>
			: plan.lazy ? k_gb_dense_smem<VT, AGG, false, GB_DEC> : k_gb_dense_smem<VT, AGG, false, false>;
	int sblocks = 0;
	if (ctx->tune[PG_TUNE_GROUPBY_PATH] != 7 && (rc = gbs_blocks(ctx, kernel, plan, range, in->n, &sblocks))) return rc;
	if (sblocks) {
		kernel<<<sblocks, GBS_THREADS, plan.bytes, s>>>((const char*) in->data, in->n, in->width, in->key_off,
				in->key_bytes, voff, kmin, (uint32_t) range, acc, fx, present, oflag);
		PG_LAUNCHED(ctx);
	} else {
		// Four rows in flight a thread and many blocks in turn: 256M rows in 1M
		// groups 2.52 ms (dec) and 2.44 (long), against 2.64 and 2.55 with eight
		// blocks per SM; eight rows hold too many registers for dec sums.
		const int64_t knob = ctx->tune[PG_TUNE_GROUPBY_ILP];
		const int ilp = knob == 8 ? 8 : GBD_ILP;
		const int gblocks = (int) std::min<uint64_t>(pg_div_up(in->n, (uint64_t) GB_THREADS * ilp),
				(uint64_t) ctx->sm_count * 128);
#define GBD_LAUNCH(V, I) k_gb_dense<VT, AGG, V, I><<<gblocks, GB_THREADS, 0, s>>>((const char*) in->data, in->n, \
				in->width, in->key_off, in->key_bytes, voff, kmin, range, acc, fx, present, oflag)
		if (vec16 && ilp == 8) GBD_LAUNCH(true, 8);
		else if (vec16) GBD_LAUNCH(true, GBD_ILP);
		else if (ilp == 8) GBD_LAUNCH(false, 8);
		else GBD_LAUNCH(false, GBD_ILP);
#undef GBD_LAUNCH
		PG_LAUNCHED(ctx);
	}
	const int eblocks = (int) std::min<uint64_t>(pg_div_up(range, 256), (uint64_t) ctx->sm_count * 8);
	k_gb_dense_emit<VT, AGG><<<eblocks, 256, 0, s>>>(acc, fx, present, range, kmin, in->key_bytes, (char*) out,
			out_cap, cursor, cursor + 2, ctx->d_status);
	PG_LAUNCHED(ctx);
	unsigned long long h[3];
	rc = pg_readback_collected(ctx, s, cursor, 2, h, "pg_groupby");
	pg_free_async(ctx, s, mem);
	*ngroups = h[0];
	*overflow = h[1] != 0;
	*fxfl |= (uint32_t) h[2];
	return rc;
}

// Key range of rows 0, step, 2 step, ...: h[0], h[1] = min and max with the
// sign bit flipped (unsigned order = signed order).
static int gb_key_range(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, bool vec16, uint64_t step, unsigned long long* h)
{
	int rc;
	unsigned long long* mm = nullptr;
	if ((rc = pg_alloc_async(ctx, s, (void**) &mm, 32))) return rc;
	PG_CUDA(ctx, cudaMemsetAsync(mm, 0, 16, s));
	const uint64_t ns = pg_div_up(in->n, step);
	const int blocks = (int) std::max<uint64_t>(1, std::min<uint64_t>(pg_div_up(ns, 256), (uint64_t) ctx->sm_count * 8));
	if (vec16) k_gb_key_minmax<true><<<blocks, 256, 0, s>>>((const char*) in->data, in->n, in->width, in->key_off,
			in->key_bytes, mm, step);
	else k_gb_key_minmax<false><<<blocks, 256, 0, s>>>((const char*) in->data, in->n, in->width, in->key_off,
			in->key_bytes, mm, step);
	PG_LAUNCHED(ctx);
	PG_CUDA(ctx, cudaMemcpyAsync(h, mm, 16, cudaMemcpyDeviceToHost, s));
	PG_CUDA(ctx, cudaStreamSynchronize(s));
	pg_free_async(ctx, s, mm);
	h[0] = ~h[0];
	return PG_OK;
}

// Dense keys: slot = key - kmin. Large inputs first try a key window from a
// sample of every 1024th row widened by an eighth on each side (no full
// min/max pass); a key outside it sends the operator to the exact window.
template <int VT, int AGG>
static int gb_dense(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint32_t voff, uint64_t hint,
		void* out, uint64_t out_cap, uint64_t* ngroups, bool* done, PgFx fx, uint32_t* fxfl)
{
	*done = false;
	int rc;
	const bool vec16 = gb_vec16<VT, AGG>(in, voff);
	const uint64_t limit = std::max<uint64_t>(4 * std::max<uint64_t>(hint, 1), std::min<uint64_t>(2 * in->n, 1ull << 22));
	unsigned long long h[2];
	if (in->n >= (1ull << 22)) {
		if ((rc = gb_key_range(ctx, s, in, vec16, 1024, h))) return rc;
		const unsigned long long span = h[1] - h[0];
		const unsigned long long slack = span / 8 + 64;
		const unsigned long long lo_u = h[0] > slack ? h[0] - slack : 0;
		const unsigned long long hi_u = ~0ull - h[1] > slack ? h[1] + slack : ~0ull;
		const uint64_t range = hi_u - lo_u + 1;
		if (range != 0 && range <= limit && range <= (1ull << 28)) {
			bool overflow = false;
			if ((rc = gb_dense_window<VT, AGG>(ctx, s, in, voff, vec16, (long long) (lo_u ^ (1ull << 63)), range,
					out, out_cap, ngroups, &overflow, fx, fxfl))) return rc;
			if (!overflow) {
				*done = true;
				if (*ngroups > out_cap) return pg_fail(ctx, PG_ERR_OUTPUT_FULL, "pg_groupby: output capacity too small");
				return PG_OK;
			}
		}
		// The sampled keys alone span too much: so do all.
		if (span >= limit || span >= (1ull << 28)) return PG_OK;
	}
	if ((rc = gb_key_range(ctx, s, in, vec16, 1, h))) return rc;
	const long long kmin = (long long) (h[0] ^ (1ull << 63)), kmax = (long long) (h[1] ^ (1ull << 63));
	const uint64_t range = (uint64_t) kmax - (uint64_t) kmin + 1;
	if (range == 0 || range > limit || range > (1ull << 28)) return PG_OK;
	bool overflow = false;
	if ((rc = gb_dense_window<VT, AGG>(ctx, s, in, voff, vec16, kmin, range, out, out_cap, ngroups, &overflow,
			fx, fxfl))) return rc;
	*done = true;
	if (*ngroups > out_cap) return pg_fail(ctx, PG_ERR_OUTPUT_FULL, "pg_groupby: output capacity too small");
	return PG_OK;
}

template <int VT, int AGG>
static int gb_run(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint32_t voff, uint64_t hint,
		void* out, uint64_t out_cap, uint64_t* ngroups, PgFx fx, uint32_t* fxfl)
{
	const bool haskey = in->key_bytes != 0;
	const int64_t gpath = ctx->tune[PG_TUNE_GROUPBY_PATH];
	if (haskey && in->n && (gpath == 0 || gpath == 6 || gpath == 7)) {
		bool done = false;
		int rc = gb_dense<VT, AGG>(ctx, s, in, voff, hint, out, out_cap, ngroups, &done, fx, fxfl);
		if (rc || done) return rc;
	}
	uint64_t groups = haskey ? std::max<uint64_t>(1, std::min<uint64_t>(hint ? hint : in->n, in->n ? in->n : 1)) : 1;
	for (int attempt = 0; attempt < 6; ++attempt) {
		uint32_t lg = 10;
		while ((1ull << lg) < 2 * groups) ++lg;
		const uint64_t cap = 1ull << lg;
		GbTable t;
		t.log2cap = lg;
		char* mem = nullptr;
		int rc;
		const uint64_t aw = GB_DEC ? PG_FX_WORDS : 1;                  // accumulator words a slot
		size_t bytes = (cap + 4) * 8 + (cap + 1) * 8 * aw + 64;
		if ((rc = pg_alloc_async(ctx, s, (void**) &mem, bytes))) return rc;
		t.keys = reinterpret_cast<unsigned long long*>(mem);
		t.acc = t.keys + cap + 4;
		t.sentinel_used = reinterpret_cast<int*>(t.acc + aw * (cap + 1));
		unsigned long long* cursor = reinterpret_cast<unsigned long long*>(t.sentinel_used + 2);
		PG_CUDA(ctx, cudaMemsetAsync(t.keys, 0xFF, (cap + 1) * 8, s));
		PG_CUDA(ctx, cudaMemsetAsync(t.acc, 0, (cap + 1) * 8 * aw + 64, s));
		if (in->n && haskey) {
			const bool few = groups <= GBH_FEW;
			const uint32_t places = 1u << (few ? GBH_FEW_LOG2 : GBH_CACHE_LOG2), probes = few ? GBH_FEW_PROBES : 1;
			const size_t smem = (size_t) places * (GB_DEC ? 40 : 16);
			uint64_t most = (uint64_t) ctx->sm_count * (few ? GBH_FEW_BLOCKS_PER_SM : GBH_BLOCKS_PER_SM);
			if (few) most = std::min(most, std::max<uint64_t>(in->n / (GBH_FEW_ROWS * groups), (uint64_t) ctx->sm_count * GBH_FEW_RESIDENT));
			const int blocks = (int) std::min<uint64_t>(pg_div_up(in->n, GB_THREADS), most);
			if (gb_vec16<VT, AGG>(in, voff))
				k_gb_hash<VT, AGG, true><<<blocks, GB_THREADS, smem, s>>>((const char*) in->data, in->n, in->width, in->key_off,
						in->key_bytes, voff, t, places, probes, fx, ctx->d_status);
			else
				k_gb_hash<VT, AGG, false><<<blocks, GB_THREADS, smem, s>>>((const char*) in->data, in->n, in->width, in->key_off,
						in->key_bytes, voff, t, places, probes, fx, ctx->d_status);
			PG_LAUNCHED(ctx);
		} else if (in->n) {
			const int blocks = (int) std::min<uint64_t>(pg_div_up(in->n, GB_THREADS), (uint64_t) ctx->sm_count * 4);
			k_gb_single<VT, AGG><<<blocks, GB_THREADS, 0, s>>>((const char*) in->data, in->n, in->width, voff, t, fx);
			PG_LAUNCHED(ctx);
		}
		// The groups are written out before the table is known to have held them
		// all; one that was full is enlarged and filled again.
		int eblocks = (int) std::min<uint64_t>(pg_div_up(cap + 1, 256), (uint64_t) ctx->sm_count * 8);
		if (haskey) k_gb_emit<VT, AGG, true><<<eblocks, 256, 0, s>>>(t, in->key_bytes, (char*) out, out_cap, cursor, 0, fx, ctx->d_status);
		else k_gb_emit<VT, AGG, false><<<1, 32, 0, s>>>(t, 0, (char*) out, out_cap, cursor, in->n, fx, ctx->d_status);
		PG_LAUNCHED(ctx);
		unsigned long long h[2];
		rc = pg_readback_collected(ctx, s, cursor, 1, h, "pg_groupby");
		pg_free_async(ctx, s, mem);
		if (rc == PG_ERR_TABLE_FULL) { groups *= 4; continue; }
		if (rc) return rc;
		*ngroups = h[0];
		*fxfl |= (uint32_t) h[1];
		if (h[0] > out_cap) return pg_fail(ctx, PG_ERR_OUTPUT_FULL, "pg_groupby: output capacity too small");
		return PG_OK;
	}
	return pg_fail(ctx, PG_ERR_TABLE_FULL, "pg_groupby: group table kept overflowing");
}

// A dec sum: the unit from the column's largest exponent (every 1024th row
// with a margin of 4x on large inputs), the aggregation, a rerun on the exact
// unit if a value lay above the sampled bound, then the groups that met
// infinities or NaNs patched.
static int gb_dec_sum(pg_ctx* ctx, cudaStream_t s, const pg_rel* in, uint32_t voff, uint64_t hint,
		void* out, uint64_t out_cap, uint64_t* ngroups)
{
	int rc;
	PgFx fx;
	if ((rc = pg_alloc_async(ctx, s, (void**) &fx.p, 16))) return rc;
	const bool sampled = in->n >= (1ull << 22);
	uint32_t fl = 0;
	rc = pg_fx_prepare(ctx, s, (const char*) in->data, in->n, in->width, voff, sampled ? 1024 : 1, 2, fx);
	if (!rc) rc = gb_run<PG_VAL_DEC, PG_AGG_SUM>(ctx, s, in, voff, hint, out, out_cap, ngroups, fx, &fl);
	if (!rc && (fl & PG_FX_RANGE)) {
		fl = 0;
		rc = pg_fx_prepare(ctx, s, (const char*) in->data, in->n, in->width, voff, 1, 0, fx);
		if (!rc) rc = gb_run<PG_VAL_DEC, PG_AGG_SUM>(ctx, s, in, voff, hint, out, out_cap, ngroups, fx, &fl);
	}
	if (!rc && (fl & PG_FX_SPECIALS)) rc = pg_fx_patch_specials(ctx, s, in, voff, (char*) out, *ngroups);
	pg_free_async(ctx, s, fx.p);
	return rc;
}

extern "C" int pg_groupby(pg_ctx* ctx, pg_stream stream, const pg_rel* in,
		uint32_t val_off, int val_type, int agg, uint64_t groups_hint,
		void* out, uint64_t out_capacity, uint64_t* ngroups)
{
	if (!ctx || !in || !ngroups) return pg_fail(ctx, PG_ERR_ARG, "pg_groupby: null argument");
	if (in->n && !in->data) return pg_fail(ctx, PG_ERR_ARG, "pg_groupby: null data");
	if (in->width == 0 || (in->width & 3)) return pg_fail(ctx, PG_ERR_UNSUPPORTED, "pg_groupby: tuple width must be a multiple of 4");
	if (in->key_bytes != 0 && ((in->key_bytes != 4 && in->key_bytes != 8) || (in->key_off & 3) ||
			in->key_off + in->key_bytes > in->width))
		return pg_fail(ctx, PG_ERR_ARG, "pg_groupby: key must be a 4-byte-aligned int or long column, or absent");
	if (agg != PG_AGG_SUM && agg != PG_AGG_COUNT) return pg_fail(ctx, PG_ERR_ARG, "pg_groupby: bad aggregate");
	if (agg == PG_AGG_SUM) {
		uint32_t vb = val_type == PG_VAL_INT ? 4 : 8;
		if (val_type < 0 || val_type > 2 || (val_off & 3) || val_off + vb > in->width)
			return pg_fail(ctx, PG_ERR_ARG, "pg_groupby: bad sum column");
	}
	cudaStream_t s = (cudaStream_t) stream;
	const PgFx none = {nullptr};
	uint32_t fl = 0;
	if (agg == PG_AGG_COUNT)
		return gb_run<PG_VAL_LONG, PG_AGG_COUNT>(ctx, s, in, val_off, groups_hint, out, out_capacity, ngroups, none, &fl);
	if (val_type == PG_VAL_INT)
		return gb_run<PG_VAL_INT, PG_AGG_SUM>(ctx, s, in, val_off, groups_hint, out, out_capacity, ngroups, none, &fl);
	if (val_type == PG_VAL_LONG)
		return gb_run<PG_VAL_LONG, PG_AGG_SUM>(ctx, s, in, val_off, groups_hint, out, out_capacity, ngroups, none, &fl);
	return gb_dec_sum(ctx, s, in, val_off, groups_hint, out, out_capacity, ngroups);
}

// Emits the present groups of a dense group table (acc/present over `range`
// slots, group key = kmin + slot) as (key, agg) rows of kbytes + agg bytes,
// appending at *cursor. Used by pg_hashjoin_groupby.
int pg_dense_groups_emit(pg_ctx* ctx, cudaStream_t s, const unsigned long long* acc, PgFx fx,
		const unsigned char* present, uint64_t range, long long kmin, uint32_t kbytes, int val_type, int agg,
		void* out, uint64_t out_cap, unsigned long long* cursor)
{
	const int eblocks = (int) std::min<uint64_t>(pg_div_up(range, 256), (uint64_t) ctx->sm_count * 8);
	if (agg == PG_AGG_COUNT)
		k_gb_dense_emit<PG_VAL_LONG, PG_AGG_COUNT><<<eblocks, 256, 0, s>>>(acc, fx, present, range, kmin, kbytes, (char*) out, out_cap, cursor, cursor + 1, ctx->d_status);
	else if (val_type == PG_VAL_INT)
		k_gb_dense_emit<PG_VAL_INT, PG_AGG_SUM><<<eblocks, 256, 0, s>>>(acc, fx, present, range, kmin, kbytes, (char*) out, out_cap, cursor, cursor + 1, ctx->d_status);
	else if (val_type == PG_VAL_LONG)
		k_gb_dense_emit<PG_VAL_LONG, PG_AGG_SUM><<<eblocks, 256, 0, s>>>(acc, fx, present, range, kmin, kbytes, (char*) out, out_cap, cursor, cursor + 1, ctx->d_status);
	else
		k_gb_dense_emit<PG_VAL_DEC, PG_AGG_SUM><<<eblocks, 256, 0, s>>>(acc, fx, present, range, kmin, kbytes, (char*) out, out_cap, cursor, cursor + 1, ctx->d_status);
	PG_LAUNCHED(ctx);
	return PG_OK;
}
