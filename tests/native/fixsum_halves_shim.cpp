// Host entry points over the 32-bit halves' adds of pythia_gb300/csrc/pg_fixsum.h
// (shared-memory tables of the hashed group-by), with plain adds in place of atomics.
#include "pg_fixsum.h"

static uint32_t plain_add(uint32_t* p, uint32_t v)
{
	const uint32_t old = *p;
	*p = old + v;
	return old;
}

extern "C" uint32_t fx_add_halves(uint32_t* q, uint64_t v) { return pg_fx_add_halves(q, v, plain_add); }

// Adds the signed 192-bit count w[0..3) into the chained words t[k * stride].
extern "C" void fx_chain_add_halves(uint64_t* t, uint64_t stride, const uint64_t* w)
{
	const pg_fx3 a = {w[0], w[1], w[2]};
	pg_fx_chain_add_halves(reinterpret_cast<uint32_t*>(t), stride, a, plain_add);
}

extern "C" void fx_chain_count(const uint64_t* t, uint64_t stride, uint64_t* w)
{
	const pg_fx4 a = pg_fx_from_chain(t, stride);
	w[0] = a.w0; w[1] = a.w1; w[2] = a.w2; w[3] = a.w3;
}
