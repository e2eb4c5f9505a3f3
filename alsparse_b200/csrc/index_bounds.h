// Bounds of look-ahead accesses.  A handle may hold up to 2^31 - 33 elements and 2^31 - 1 rows, so the index a kernel is
// about to request (position + look-ahead) need not fit an int although every index it reads does.  It always fits an
// unsigned: the sum is formed and compared there.  (Comparing the look-ahead with what is left, end - position, is as
// right and costs the stream kernel of the dense-block product registers: up to 20 % of its time, B200.)
// Plain C++ as well, so that the arithmetic is tested on the host at the limits.
#pragma once

#ifdef __CUDACC__
#define ASB_HD __host__ __device__ __forceinline__
#else
#define ASB_HD inline
#endif

namespace asb {

// at + ahead < end, for 0 <= at, end and 0 <= ahead <= INT_MAX
ASB_HD bool ahead_inside(int at, int ahead, int end) {
    return (unsigned)at + (unsigned)ahead < (unsigned)end;
}

// at + ahead <= end
ASB_HD bool ahead_complete(int at, int ahead, int end) {
    return (unsigned)at + (unsigned)ahead <= (unsigned)end;
}

// min(at + ahead, end)
ASB_HD int ahead_or_end(int at, int ahead, int end) {
    const unsigned sum = (unsigned)at + (unsigned)ahead;
    return (int)(sum < (unsigned)end ? sum : (unsigned)end);
}

}  // namespace asb
