// What one probe goes by of a join table that another thread may settle
// meanwhile (pg_hashtable.cuh). Host code without CUDA, so that a host test can
// settle a table between any two of the reads.
#ifndef PG_TABLEVIEW_H
#define PG_TABLEVIEW_H

#include <atomic>

struct HjView {
	bool spec;       // only the window's base and the header describe the table
	bool unique;     // no repeated keys (taken for granted, and checked by the header, while spec holds)
};

// `spec` is read first: settling writes every other field and then clears it, so a
// table seen settled is seen whole, and of one that is not no other field is used.
// Read the other way round, a table of repeated keys settled in between looked unique and
// settled, and its probe stopped at each key's first match with no check.
template <class Table>
inline HjView hj_view(const Table& ht)
{
	HjView v;
	v.spec = ht.spec.load(std::memory_order_acquire);
	v.unique = v.spec || ht.unique;
	return v;
}

#endif
