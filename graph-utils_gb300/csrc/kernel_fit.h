// kernel_fit.h -- how many CTAs or clusters of a kernel are resident at once.
#pragma once

#include <cstddef>

namespace gu {

// CTAs per SM of a kernel launched with so many threads and bytes of dynamic shared
// memory; with cluster > 1, clusters of that many CTAs on the whole device (0: the kernel
// cannot run so).  A launch above 48 KiB needs the kernel's consent on the device it runs
// on: given here, for up to smem_most bytes, on the kernel's first use there (and for
// clusters of more than eight CTAs).
//
// The calculation costs as much as a small launch, so its answers are kept -- by device
// and kernel as well as by shape: two kernels, or one kernel on two devices, may come with
// equal shapes and need each its own.  `device` is the current one.  Safe from several
// threads.
int kernel_fit(int device, const void *kernel, int threads, size_t smem, size_t smem_most, int cluster = 1);

}  // namespace gu
