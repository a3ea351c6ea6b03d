// Small arithmetic of the kernels that tests compile for the host, without a GPU.
#pragma once

#ifdef __CUDACC__
#define UG_HD __host__ __device__ __forceinline__
#else
#define UG_HD inline
#endif

namespace ug {

// Where a list of noise events (cap entries, the last one kept for its mark) goes on: at its
// start, or, resumed, behind the mark at `at` that its last segment ended with.  A full list has
// that mark in its last entry; it goes on there, where only the next mark is written, over it.
UG_HD int list_start(bool resume, int at, int cap)
{
    return !resume ? 0 : at + 1 < cap ? at + 1 : cap - 1;
}

}  // namespace ug
