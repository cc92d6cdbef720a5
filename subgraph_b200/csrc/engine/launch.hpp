// Dynamic shared memory of kernel launches.
#pragma once
#include <cstddef>

namespace sg {

// CTAs of `threads` threads and `smem` bytes of dynamic shared memory that an
// SM of the current device holds (at least 1).  Called before every launch of
// a kernel that may have more than 48 KB of dynamic shared memory: the first
// call for a kernel raises its limit to all the device allows beside the
// kernel's static part.  The limit is state of the whole process and a kernel
// is launched with several sizes (they follow the template and the graph), so
// it is never set to one launch's size: another thread's launch may come between.
int resident_ctas(const void *kern, int threads, size_t smem);

}  // namespace sg
