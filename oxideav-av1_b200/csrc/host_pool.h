// host_pool.h — the helper threads that share a call's host preparation
// (validation, dependency analysis, record building) with the calling thread.
#pragma once

#include <cstddef>
#include <functional>

namespace av1g {

// Runs fn(0) .. fn(n - 1), each once, on the calling thread and on idle helper
// threads, and returns when all have finished.  An exception that fn throws is
// rethrown here.  Callers on several threads share the helpers; a call needs
// none of them to finish.  `items`: how much work there is in all; little of it
// stays on the calling thread.
void parallel_for(int n, long long items, const std::function<void(int)>& fn);

// The number of parts to cut `items` pieces of work into, at least `grain` in
// each: 1 (no helpers involved) for small calls.
int parallel_parts(long long items, long long grain);

// Sends the whole cache lines of [p, p + n), which the caller has just written and
// nobody else touches, to memory.  A part of an upload that stays in its thread's
// cache is fetched from there by the copy engine: 6 MB written by eight threads took 696 us
// to copy to the device, against 128 us when one thread had written them.  Does
// nothing on hosts without SSE2: only the copy's time depends on it.
void write_back(void* p, size_t n);

}  // namespace av1g
