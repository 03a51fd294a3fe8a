// Settles a fake join table of repeated keys before the k-th read that
// hj_view (pythia_gb300/csrc/pg_tableview.h) makes of it, for the Python test.
#include "pg_tableview.h"

static int g_reads, g_settle_before;
static bool g_unique, g_spec;

static void tick()
{
	if (g_reads++ == g_settle_before) { g_unique = false; g_spec = false; }
}

struct FakeSpec {
	bool load(std::memory_order) const { tick(); return g_spec; }
};

struct FakeBool {
	operator bool() const { tick(); return g_unique; }
};

struct FakeTable {
	FakeSpec spec;
	FakeBool unique;
};

// Bit 0: spec, bit 1: unique; bits 8 on: the reads made.
extern "C" int tableview_settled_before(int k)
{
	g_reads = 0;
	g_settle_before = k;
	g_unique = g_spec = true;
	const FakeTable t = FakeTable();
	const HjView v = hj_view(t);
	return (v.spec ? 1 : 0) | (v.unique ? 2 : 0) | (g_reads << 8);
}
