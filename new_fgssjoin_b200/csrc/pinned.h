// pinned.h -- page-locked host memory for what the library returns (pinned.cpp).
#pragma once

#include <stddef.h>

#include "../../include/fgss.h"

namespace fgss {

// A block of at least `bytes` from the process-wide pool, or nullptr.
void* pinned_take(size_t bytes);
// Gives a block of the pool back (true), or returns false for other memory.
bool pinned_give(void* b);

// Does one block of the pool hold the `bytes` bytes from p?
bool pinned_holds(const void* p, size_t bytes);

// Columns of n records and T tokens (freed by fgss_sets_free): one page-locked
// block of 256-byte aligned columns that starts with `id`, so the copies from
// the device, and to it when the sets are joined, run at the link's rate; or
// malloc'd columns where page-locked memory cannot be had.  loc: with the
// token positions.
void alloc_host_sets(fgss_sets* s, uint64_t n, uint64_t T, bool loc);

}  // namespace fgss
