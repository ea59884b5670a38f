// Which copies of a two-stage ring are still to be waited for when its producer stops.  Plain C++: the host's test
// includes it too.
#pragma once

#ifdef __CUDACC__
#define AFQ_HD __host__ __device__ __forceinline__
#else
#define AFQ_HD inline
#endif

namespace afq {

// The producer has issued tiles 0 .. n - 1 of every stage before `stages` and, of that one, the first `extra`; stage v
// goes to buffer v & 1.  The last stage whose tile j went to buffer p, or -1: earlier copies of that tile have landed
// (their readers had finished before it was issued).
AFQ_HD int ring_last(unsigned stages, int extra, int j, int p) {
    if ((int)(stages & 1) == p && j < extra) return (int)stages;
    const int v = (int)stages - 1;
    return v < 0 ? -1 : (v & 1) == p ? v : v - 1;
}

}  // namespace afq
