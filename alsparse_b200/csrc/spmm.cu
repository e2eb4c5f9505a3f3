// CSR x dense SpMM kernels for sm_100a, row-major dense operands.
//
// Y[r, :] = beta * Y[r, :] + sum over stored elements (alpha * a) * X[col, :], the operation
// of the reference's gemm_{s,d}_csr_row (arithmetic defined by
// src/plain/kernel/level3/mm/gemm/gemm_x_csr_row_plain.c:4-23: alpha is folded into the
// element before the accumulation).  The reference's own device build has no row-major SpMM
// (src/kernel/dcu/level3/mm/csrmm/dcu_gemm_x_csr_row.cpp:15-36 returns NOT_SUPPORTED).
//
// A group of lanes spans the dense columns, VEC consecutive columns per lane, so every stored element
// turns into one fully coalesced read of a row of X (64 fp32 columns = 256 bytes = 16 lanes x
// float4).  The group fetches (col, alpha*a) pairs with coalesced loads and hands them round with
// shuffles; several X rows are in flight per group.  Bandwidth-bound: the
// traffic is nnz * columns * sizeof(T) of X rows against 2 flops per element, far below what
// would justify staging tiles for tensor cores.
#include <limits.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "index_bounds.h"
#include "internal.h"

namespace asb {

template <typename T, int VEC>
struct Pack;
template <>
struct Pack<float, 1> { using type = float; };
template <>
struct Pack<float, 2> { using type = float2; };
template <>
struct Pack<float, 4> { using type = float4; };
template <>
struct Pack<double, 1> { using type = double; };
template <>
struct Pack<double, 2> { using type = double2; };

template <typename T, int VEC>
__device__ __forceinline__ void load_vec(const T *__restrict__ p, T (&out)[VEC]) {
    using P = typename Pack<T, VEC>::type;
    const P t = __ldg(reinterpret_cast<const P *>(p));
    const T *s = reinterpret_cast<const T *>(&t);
#pragma unroll
    for (int i = 0; i < VEC; i++) out[i] = s[i];
}

// A group of LPR lanes (a power of two up to 32) owns one sparse row; 32/LPR rows share a warp.
// Lane g of the group holds VEC consecutive dense columns starting at ct + g*VEC, so one step of
// the group reads LPR*VEC*sizeof(T) contiguous bytes of an X row (64 fp32 columns: 16 lanes x
// float4 = 256 bytes, two rows per warp instruction).
// VEC > 1 requires: columns % VEC == 0, ldx % VEC == 0, ldy % VEC == 0 and X, Y aligned to
// VEC * sizeof(T); the launcher checks and otherwise uses VEC == 1.
constexpr int kSpmmUnroll = 4;     // X rows in flight per lane group (8 and 16 were slower on B200)
constexpr int kSpmmMinBlocks = 8;  // full occupancy (32 registers) measured fastest
template <typename T, int VEC, int LPR, bool HAS_BETA>
__global__ void __launch_bounds__(256, kSpmmMinBlocks)
    spmm_row_kernel(int rows, const int *__restrict__ row_lo, const int *__restrict__ row_hi,
                    const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ X, int columns,
                    long long ldx, T *__restrict__ Y, long long ldy, T alpha, T beta) {
    constexpr int UNROLL = kSpmmUnroll;
    constexpr int RPW = 32 / LPR;  // rows per warp
    const int lane = threadIdx.x & 31;
    const int gl = lane % LPR, grp = lane / LPR;
    const unsigned gmask = LPR == 32 ? 0xffffffffu : (((1u << LPR) - 1u) << (grp * LPR));
    const long long row = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * RPW + grp;
    if (row >= rows) return;  // whole groups leave together; shuffles below name only their group
    // [row_lo[row], row_hi[row]) are the stored elements this launch multiplies: the whole row (row_hi = row_lo + 1
    // of the offset array) or the part of it that falls into one column block (see SpmmBlocks)
    const int s = __ldg(row_lo + row), e = __ldg(row_hi + row);

    for (int ct = 0; ct < columns; ct += LPR * VEC) {
        const int c = ct + gl * VEC;
        const bool live = c < columns;
        T acc[VEC];
#pragma unroll
        for (int i = 0; i < VEC; i++) acc[i] = T(0);

        for (int base = s; base < e; base += LPR) {
            const int mine = base + gl;
            int cj = 0;
            T vj = T(0);
            if (mine < e) {
                cj = __ldcs(col + mine);
                vj = alpha * __ldcs(val + mine);
            }
            const int n = min(LPR, e - base);
            int k = 0;
            for (; k + UNROLL <= n; k += UNROLL) {
                T xv[UNROLL][VEC];
                T av[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; u++) {
                    const int cc = __shfl_sync(gmask, cj, k + u, LPR);
                    av[u] = __shfl_sync(gmask, vj, k + u, LPR);
                    if (live) load_vec<T, VEC>(X + (long long)cc * ldx + c, xv[u]);
                }
                if (live) {
#pragma unroll
                    for (int u = 0; u < UNROLL; u++)
#pragma unroll
                        for (int i = 0; i < VEC; i++) acc[i] = fma(av[u], xv[u][i], acc[i]);
                }
            }
            for (; k < n; k++) {
                const int cc = __shfl_sync(gmask, cj, k, LPR);
                const T a = __shfl_sync(gmask, vj, k, LPR);
                if (live) {
                    T xv[VEC];
                    load_vec<T, VEC>(X + (long long)cc * ldx + c, xv);
#pragma unroll
                    for (int i = 0; i < VEC; i++) acc[i] = fma(a, xv[i], acc[i]);
                }
            }
        }

        if (live) {
            T *out = Y + row * ldy + c;
#pragma unroll
            for (int i = 0; i < VEC; i++) {
                T o = acc[i];
                if (HAS_BETA) o = fma(beta, out[i], o);
                acc[i] = o;
            }
            using P = typename Pack<T, VEC>::type;
            P packed;
            T *ps = reinterpret_cast<T *>(&packed);
#pragma unroll
            for (int i = 0; i < VEC; i++) ps[i] = acc[i];
            __stcs(reinterpret_cast<P *>(out), packed);
        }
    }
}

// ---- the stream kernel ---------------------------------------------------------------------------------
//
// What bounds this product is the stream of X rows into the SMs: L2 delivers it at 19-20 TB/s (rows of 128 bytes and
// more; 64-byte rows 17 TB/s, one request per SM and clock below that) when enough loads are in flight, HBM random
// 256-byte rows at 7-10.  The kernel above has 4 rows in flight per lane group, none while a group fetches its next
// elements or offsets, and issues everything once per group.  Here a warp walks a contiguous SEGMENT of the stored
// elements, row boundaries or not: LPR lanes per X row, so 32 / LPR consecutive elements per step; the X rows of the next
// U steps are requested before those of the current U are multiplied, elements are fetched two batches ahead and the
// ends of the next 32 rows wait in registers.  A row that ends is summed over the lane groups and written at once; what a
// segment holds of a row that goes on behind its end is left in `part` for spmm_cross_reduce_kernel.
//
// Measured (B200, us, kernel above -> here): 2^20 rows of 32 elements x 64 fp32 columns 1720 -> 1200 (X = 268 MB), 2^18
// rows 308 -> 193 (11 TB/s), 300,007 rows of 27 x 16 columns 130 -> 92, power-law 400,009 rows x 24 columns 627 -> 188,
// 20,000 rows x 12 columns 423 -> 14.  U = 4 with 3 or 4 blocks per SM: 1270-1335 / 212-245; U = 2 with 5 or 6 blocks
// (spills): 1320-1430.  One segment per lane group instead of per warp: 1660-1900, the groups of a warp run apart.
//
// Segments: `per_warp` whole rows each (even matrices, no table), or the table of spmm_segments_ensure (skewed ones).
constexpr int kStreamUnroll = 2;     // steps per group; two groups are in flight
constexpr int kStreamMinBlocks = 4;  // 64 registers
struct StreamSegments {
    const MergeCoord *seg;  // nseg + 1 starts (null: per_warp rows each)
    const int *slot;        // place in `part` of what a segment leaves unfinished
    int nseg;
    int per_warp;
    int row0, row1;  // the rows to produce (a window of the matrix)
};

template <typename T, int VEC, int LPR, bool HAS_BETA>
__global__ void __launch_bounds__(256, kStreamMinBlocks)
    spmm_stream_kernel(const StreamSegments sg, const int *__restrict__ row_ptr, const int *__restrict__ col,
                       const T *__restrict__ val, const T *__restrict__ X, int c0, int columns, int ldx, T *__restrict__ Y,
                       long long ldy, T *__restrict__ part, T alpha, T beta) {
    constexpr int U = kStreamUnroll;
    constexpr int S = 32 / LPR;                        // elements per step
    constexpr int Q = LPR < 2 * U ? 2 * U / LPR : 1;  // elements a lane holds of one batch
    constexpr int G = LPR * Q / U;                     // groups of U steps per batch: even, for the two buffers
    static_assert(G % 2 == 0, "groups alternate between two buffers");
    const int lane = threadIdx.x & 31, gl = lane % LPR, sub = lane / LPR;
    const int g = blockIdx.x * 8 + (threadIdx.x >> 5);
    int r, r_end, k, k_end, slot = -1;
    if (sg.seg) {
        if (g >= sg.nseg) return;
        const MergeCoord a = sg.seg[g], b = sg.seg[g + 1];
        r = a.row, k = a.nz, r_end = b.row, k_end = b.nz;
        slot = __ldg(sg.slot + g);
        if (r < sg.row0) r = sg.row0, k = __ldg(row_ptr + r);
        if (r_end >= sg.row1) r_end = sg.row1, k_end = __ldg(row_ptr + r_end), slot = -1;
    } else {
        const long long first = sg.row0 + (long long)g * sg.per_warp;
        if (first >= sg.row1) return;
        r = (int)first, r_end = (int)min((long long)sg.row1, first + sg.per_warp);
        k = __ldg(row_ptr + r), k_end = __ldg(row_ptr + r_end);
    }
    const unsigned c = (unsigned)c0 + blockIdx.y * (LPR * VEC) + gl * VEC;
    const bool live = c < (unsigned)columns;
    const T *Xc = X + (live ? c : 0);  // (lanes beyond the last column read the first and drop it)

    // ends of rows r .. r + 31 (lane by lane), and of the 32 rows behind them
    auto load_ends = [&](int ahead) {
        return ahead_inside(r, ahead + lane, r_end) ? __ldg(row_ptr + ((unsigned)r + ahead + lane + 1)) : INT_MAX;
    };
    int ends = load_ends(0), ends_next = load_ends(32), at = 0;
    // Elements of this batch, the next and the one behind it.  Beyond the segment: column 0, which is read and dropped.
    int cj[Q], cn[Q], cm[Q];
    T vj[Q], vn[Q], vm[Q];
    auto load_batch = [&](int from, int ahead, int (&cc)[Q], T (&vv)[Q]) {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            cc[q] = 0, vv[q] = T(0);
            if (ahead_inside(from, ahead + q * 32 + lane, k_end)) {
                const int j = from + ahead + q * 32 + lane;
                cc[q] = __ldcs(col + j), vv[q] = __ldcs(val + j);
            }
        }
    };
    load_batch(k, 0, cj, vj);
    load_batch(k, 32 * Q, cn, vn);
    T xv[2][U][VEC];
    auto load_rows = [&](int buf, int group, const int (&cc)[Q]) {  // X rows of the U steps of a group
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = (group * U + u) * S;
            const int j = __shfl_sync(0xffffffffu, cc[e / 32], e % 32 + sub);
            load_vec<T, VEC>(Xc + (size_t)(unsigned)j * (unsigned)ldx, xv[buf][u]);
        }
    };
    T acc[VEC], old[VEC];
#pragma unroll
    for (int i = 0; i < VEC; i++) acc[i] = T(0), old[i] = T(0);
    using P = typename Pack<T, VEC>::type;
    auto fetch_old = [&] {  // Y of the row in work, long before it is needed
        if (HAS_BETA && live && sub == 0 && r < r_end) {
            const P t = __ldcs(reinterpret_cast<const P *>(Y + r * ldy + c));
            const T *ts = reinterpret_cast<const T *>(&t);
#pragma unroll
            for (int i = 0; i < VEC; i++) old[i] = ts[i];
        }
    };
    fetch_old();
    int row_end = __shfl_sync(0xffffffffu, ends, 0);
    auto sum_groups = [&] {
#pragma unroll
        for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
            for (int i = 0; i < VEC; i++) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    };
    auto finish_row = [&] {
        sum_groups();
        P packed;
        T *ps = reinterpret_cast<T *>(&packed);
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            ps[i] = HAS_BETA ? fma(beta, old[i], acc[i]) : acc[i];
            acc[i] = T(0);
        }
        if (live && sub == 0) __stcs(reinterpret_cast<P *>(Y + r * ldy + c), packed);
        r++;
        if (++at == 32) {
            at = 0, ends = ends_next;
            ends_next = load_ends(32);
        }
        row_end = __shfl_sync(0xffffffffu, ends, at);
        fetch_old();
    };
    while (row_end == k) finish_row();  // empty rows
    if (k < k_end) load_rows(0, 0, cj);
    while (k < k_end) {  // (everything about k is uniform over the warp)
        const int k0 = k;
        load_batch(k0, 64 * Q, cm, vm);
#pragma unroll
        for (int q = 0; q < Q; q++) vj[q] *= alpha;
#pragma unroll
        for (int grp = 0; grp < G; grp++) {
            if (grp + 1 < G) load_rows((grp + 1) & 1, grp + 1, cj);
            else load_rows(0, 0, cn);
            constexpr int GS = U * S;
            if (ahead_complete(k0, (grp + 1) * GS, min(row_end, k_end))) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = (grp * U + u) * S;
                    const T a = __shfl_sync(0xffffffffu, vj[e / 32], e % 32 + sub);
#pragma unroll
                    for (int i = 0; i < VEC; i++) acc[i] = fma(a, xv[grp & 1][u][i], acc[i]);
                }
                k = k0 + (grp + 1) * GS;
                while (row_end == k) finish_row();
            } else {  // row by row through the group
                const int stop = ahead_or_end(k0, (grp + 1) * GS, k_end);
                while (k < stop) {
                    const int hi = min(row_end, stop);
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int e = (grp * U + u) * S;
                        const T a = __shfl_sync(0xffffffffu, vj[e / 32], e % 32 + sub);
                        if (k0 + e + sub >= k && k0 + e + sub < hi) {
#pragma unroll
                            for (int i = 0; i < VEC; i++) acc[i] = fma(a, xv[grp & 1][u][i], acc[i]);
                        }
                    }
                    k = hi;
                    while (row_end == k) finish_row();
                }
            }
        }
#pragma unroll
        for (int q = 0; q < Q; q++) cj[q] = cn[q], vj[q] = vn[q], cn[q] = cm[q], vn[q] = vm[q];
    }
    if (slot >= 0) {
        sum_groups();
        P packed;
        T *ps = reinterpret_cast<T *>(&packed);
#pragma unroll
        for (int i = 0; i < VEC; i++) ps[i] = acc[i];
        if (live && sub == 0) *reinterpret_cast<P *>(part + (size_t)slot * columns + c) = packed;
    }
}

// Start of every segment: the point on the diagonal i * items of the walk through elements and row ends in which a row
// end counts as kStreamRowItems elements (finishing a row costs a group about as much as loading that many).  A start
// inside a row of at most kStreamWhole elements moves back to the row's beginning: short rows are never cut.
constexpr int kStreamRowItems = 8, kStreamWhole = 64;
__global__ void spmm_segments_kernel(int rows, int nnz, const int *__restrict__ row_ptr, int items, int nseg,
                                     MergeCoord *__restrict__ out, int *__restrict__ slot) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nseg) return;
    const long long diag = (long long)i * items;
    int lo = 0, hi = rows;  // rows whose end lies at or before the diagonal
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if ((long long)row_ptr[mid + 1] + (long long)kStreamRowItems * (mid + 1) <= diag) lo = mid + 1;
        else hi = mid;
    }
    int nz = nnz;
    bool cut = false;
    if (lo < rows) {
        const int s = row_ptr[lo], e = row_ptr[lo + 1];
        const long long at = diag - (long long)kStreamRowItems * lo;
        nz = e - s <= kStreamWhole || at < s ? s : at > e ? e : (int)at;
        cut = nz > s;
    }
    out[i].row = lo, out[i].nz = nz;
    if (i > 0) slot[i - 1] = cut ? 0 : -1;  // the segment before leaves a part of row lo behind
}

// Y[row, :] += what the segments before the row's last one hold of it, in order.  One block per such row: the threads
// span the columns; with few columns several runs of segments are summed side by side and then added up in order.
template <typename T>
__global__ void __launch_bounds__(256)
    spmm_cross_reduce_kernel(const int *__restrict__ row_of, const int *__restrict__ first_of, const T *__restrict__ part,
                             int columns, T *__restrict__ Y, long long ldy) {
    __shared__ T s_sum[256];
    const int row = row_of[blockIdx.x], k0 = first_of[blockIdx.x], k1 = first_of[blockIdx.x + 1];
    const int wide = min(columns, (int)blockDim.x), runs = blockDim.x / wide;
    const int run = threadIdx.x / wide, lane = threadIdx.x % wide;
    const int per = (k1 - k0 + runs - 1) / runs;
    for (int c0 = 0; c0 < columns; c0 += wide) {
        const int c = c0 + lane;
        T acc = T(0);
        if (run < runs && c < columns)
            for (int k = k0 + run * per, e = min(k1, k + per); k < e; k++) acc += part[(size_t)k * columns + c];
        __syncthreads();
        s_sum[threadIdx.x] = acc;
        __syncthreads();
        if (run == 0 && c < columns) {
            for (int v = 1; v < runs; v++) acc += s_sum[v * wide + lane];
            Y[(long long)row * ldy + c] += acc;
        }
    }
}

// ---- narrow dense blocks -------------------------------------------------------------------------------
//
// With a handful of dense columns (an X row of at most 32 bytes) the kernel above degenerates: two lanes per row hand
// their elements round two at a time and every round waits for its own X rows (2^21 rows of 32 elements times 1..8
// fp32 columns: 0.68..1.24 ms, where an SpMV of the same matrix takes 0.2 ms).  Here the lanes of a group split the
// ELEMENTS of the row instead, as in the vector SpMV: a lane gathers the whole X row of its element (one or two
// 16-byte loads when the shapes allow, scalars otherwise), carries KC partial sums, two elements in flight, and the
// group reduces them by shuffles.  alpha is folded into the stored value before the sum, as in the kernel above.
template <typename T, int LANES, int KC, bool ALIGNED, bool HAS_BETA>
__global__ void __launch_bounds__(256)
    spmm_row_narrow_kernel(int rows, const int *__restrict__ row_lo, const int *__restrict__ row_hi,
                           const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ X, int columns,
                           long long ldx, T *__restrict__ Y, long long ldy, T alpha, T beta) {
    constexpr int GROUPS = 256 / LANES;
    constexpr int PER16 = 16 / (int)sizeof(T);  // elements per 16-byte load
    const int lane = threadIdx.x % LANES;
    const long long row = (long long)blockIdx.x * GROUPS + threadIdx.x / LANES;
    int s = 0, e = 0;
    if (row < rows) {
        s = __ldg(row_lo + row);
        e = __ldg(row_hi + row);
    }
    T acc[KC];
#pragma unroll
    for (int k = 0; k < KC; k++) acc[k] = T(0);
    auto take = [&](int j) {
        const int cj = __ldcs(col + j);
        const T vj = alpha * __ldcs(val + j);
        const T *xr = X + (long long)cj * ldx;
        T xv[KC];
        if (ALIGNED) {  // columns == KC, rows of X on 16-byte boundaries
#pragma unroll
            for (int k = 0; k < KC; k += PER16) {
                using P = typename Pack<T, PER16>::type;
                const P t = __ldg(reinterpret_cast<const P *>(xr + k));
                const T *sp = reinterpret_cast<const T *>(&t);
#pragma unroll
                for (int i = 0; i < PER16; i++) xv[k + i] = sp[i];
            }
        } else {
#pragma unroll
            for (int k = 0; k < KC; k++) xv[k] = k < columns ? __ldg(xr + k) : T(0);
        }
#pragma unroll
        for (int k = 0; k < KC; k++) acc[k] = fma(vj, xv[k], acc[k]);
    };
    int j = s + lane;
    for (; j + LANES < e; j += 2 * LANES) {
        take(j);
        take(j + LANES);
    }
    if (j < e) take(j);
#pragma unroll
    for (int k = 0; k < KC; k++) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    }
    if (lane == 0 && row < rows) {
        T *out = Y + row * ldy;
#pragma unroll
        for (int k = 0; k < KC; k++)
            if (k < columns) {
                T o = acc[k];
                if (HAS_BETA) o = fma(beta, out[k], o);
                out[k] = o;
            }
    }
}

// ---- column blocks -----------------------------------------------------------------------------------
//
// Every stored element reads one row of X (columns * sizeof(T) bytes).  With unstructured columns and an X far
// larger than L2 nearly all of these reads come from HBM: 64 fp32 columns on 6.7e7 elements move 17 GB for
// 1.6 GB of operands.  Cutting the columns of A into P blocks and running the product block by block makes the
// rows of X a pass touches a slab of 1/P of X that stays in L2, so X crosses HBM about once; the price is that Y
// is written P times and read P - 1 times.  Rows with ascending columns need no copy of A for this: the part of
// a row inside a block is a contiguous run, described by P + 1 offsets per row.  (An experiment kept as an
// option: see spmm_pick_blocks for what it measured.)
__global__ void rows_ascending_kernel(int rows, const int *__restrict__ row_ptr, const int *__restrict__ col,
                                      unsigned long long *__restrict__ bad) {
    unsigned long long n = 0;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (long long)gridDim.x * blockDim.x)
        for (int k = row_ptr[r]; k + 1 < row_ptr[r + 1]; k++) n += col[k] > col[k + 1];
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(bad, n);
}

// split[p * rows + r] = first element of row r whose column is >= p * width (p = 0 .. blocks)
__global__ void spmm_split_kernel(int rows, int blocks, int width, const int *__restrict__ row_ptr,
                                  const int *__restrict__ col, int *__restrict__ split) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)rows * (blocks + 1)) return;
    const int p = (int)(i / rows), r = (int)(i % rows);
    int lo = row_ptr[r], hi = row_ptr[r + 1];
    if (p == 0) hi = lo;
    else if (p == blocks) lo = hi;
    const long long want = (long long)p * width;
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if ((long long)col[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    split[i] = lo;
}

void spmm_blocks_destroy(SpmmBlocks &b) {
    if (b.d_split) cudaFree(b.d_split);  // (even of a null pointer it ends a stream capture)
    b = SpmmBlocks{};
}

// Column-block table for `blocks` blocks, built on first use and kept until another count is asked for.
// Leaves b.blocks == 1 (no blocking) when the rows are not in ascending column order.
alphasparse_status_t col_blocks_ensure(DeviceCtx *ctx, SpmmBlocks &b, int blocks, cudaStream_t st) {
    if (b.blocks == blocks || (b.unsorted && blocks > 1)) return ALPHA_SPARSE_STATUS_SUCCESS;
    const int64_t old_bytes = b.d_split ? (int64_t)sizeof(int) * ctx->rows * (b.blocks + 1) : 0;
    spmm_blocks_destroy(b);
    ctx->device_bytes -= old_bytes;
    b.blocks = 1;
    if (blocks <= 1) return ALPHA_SPARSE_STATUS_SUCCESS;
    unsigned long long *d_bad = nullptr, h_bad = 0;
    ASB_CUDA_OR(device_alloc(&d_bad, sizeof(h_bad)), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    cudaError_t e = cudaMemsetAsync(d_bad, 0, sizeof(h_bad), st);
    if (e == cudaSuccess) {
        rows_ascending_kernel<<<148 * 8, 256, 0, st>>>((int)ctx->rows, ctx->d_row_ptr, ctx->d_col, d_bad);
        count_launch();
        e = cudaMemcpyAsync(&h_bad, d_bad, sizeof(h_bad), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_bad);
    if (e != cudaSuccess) {
        record_cuda_error(e, "column blocks");
        return ALPHA_SPARSE_STATUS_EXECUTION_FAILED;
    }
    if (h_bad) {
        b.unsorted = true;
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    const int width = (int)((ctx->cols + blocks - 1) / blocks);
    const size_t cells = (size_t)ctx->rows * (size_t)(blocks + 1);
    ASB_CUDA_OR(device_alloc(&b.d_split, sizeof(int) * cells), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    spmm_split_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>((int)ctx->rows, blocks, width, ctx->d_row_ptr,
                                                                     ctx->d_col, b.d_split);
    count_launch();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        spmm_blocks_destroy(b);
        b.blocks = 1;
        record_cuda_error(e, "column blocks");
        return ALPHA_SPARSE_STATUS_EXECUTION_FAILED;
    }
    b.blocks = blocks, b.width = width;
    ctx->device_bytes += (int64_t)(sizeof(int) * cells);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// ---- long rows ------------------------------------------------------------------------------------------

void spmm_split_destroy(SpmmSplit &s) {
    cudaFree(s.d_hi_short), cudaFree(s.d_chunk_lo), cudaFree(s.d_chunk_hi), cudaFree(s.d_long_row), cudaFree(s.d_long_first);
    cudaFree(s.d_part);
    free(s.h_long_row), free(s.h_long_first);
    s = SpmmSplit{};
}

// Y[row, :] += the row's partial sums in chunk order.  One block per long row, threads over the dense columns.
template <typename T>
__global__ void spmm_long_reduce_kernel(const int *__restrict__ long_row, const int *__restrict__ long_first,
                                        const T *__restrict__ part, int columns, T *__restrict__ Y, long long ldy) {
    const int row = long_row[blockIdx.x], k0 = long_first[blockIdx.x], k1 = long_first[blockIdx.x + 1];
    for (int c = threadIdx.x; c < columns; c += blockDim.x) {
        T acc = T(0);
        for (int k = k0; k < k1; k++) acc += part[(size_t)k * columns + c];
        Y[(long long)row * ldy + c] += acc;
    }
}

// Rows that one lane group would still be walking long after every other row is done.  (Only where the rows are uneven:
// rows that are all long keep every lane group equally busy as they are.)
static bool spmm_long_rows(const DeviceCtx *ctx) {
    const int64_t min_len = option(kOptSpmmSplitMin);
    return min_len > 0 && ctx->max_row_nnz > min_len && (double)ctx->max_row_nnz > 8.0 * ctx->mean_row_nnz;
}

// Looks at the row lengths once (first row-major product of the handle) and builds the chunk tables when some row
// is longer than spmm_split_min.
static alphasparse_status_t spmm_split_ensure(DeviceCtx *ctx, cudaStream_t st) {
    SpmmSplit &sp = ctx->split;
    if (sp.state != 0) return ALPHA_SPARSE_STATUS_SUCCESS;
    const int64_t min_len = option(kOptSpmmSplitMin), chunk = std::max<int64_t>(64, option(kOptSpmmSplitChunk));
    if (ctx->rows == 0 || !spmm_long_rows(ctx)) {
        sp.state = 1;
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    std::vector<int> ptr, hi, clo, chi, lrow, lfirst;
    try {
        ptr.resize((size_t)ctx->rows + 1);
    } catch (...) {
        return ALPHA_SPARSE_STATUS_ALLOC_FAILED;
    }
    ASB_CUDA_OR(cudaMemcpyAsync(ptr.data(), ctx->d_row_ptr, sizeof(int) * ptr.size(), cudaMemcpyDeviceToHost, st),
                ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    ASB_CUDA_OR(cudaStreamSynchronize(st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    try {
        hi.resize((size_t)ctx->rows);
        for (int64_t r = 0; r < ctx->rows; r++) {
            const int a = ptr[(size_t)r], e = ptr[(size_t)r + 1];
            hi[(size_t)r] = e;
            if ((int64_t)e - a <= min_len) continue;
            hi[(size_t)r] = a;  // nothing of this row in the row pass
            lrow.push_back((int)r);
            lfirst.push_back((int)clo.size());
            for (int64_t k = a; k < e; k += chunk) {
                clo.push_back((int)k);
                chi.push_back((int)std::min<int64_t>(e, k + chunk));
            }
        }
        lfirst.push_back((int)clo.size());
    } catch (...) {
        return ALPHA_SPARSE_STATUS_ALLOC_FAILED;
    }
    SpmmSplit t;
    t.nlong = (int64_t)lrow.size(), t.nchunks = (int64_t)clo.size();
    t.h_long_row = static_cast<int *>(malloc(sizeof(int) * std::max<size_t>(1, lrow.size())));
    t.h_long_first = static_cast<int *>(malloc(sizeof(int) * lfirst.size()));
    cudaError_t e = (t.h_long_row && t.h_long_first) ? cudaSuccess : cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = device_alloc(&t.d_hi_short, sizeof(int) * hi.size());
    if (e == cudaSuccess) e = device_alloc(&t.d_chunk_lo, sizeof(int) * clo.size());
    if (e == cudaSuccess) e = device_alloc(&t.d_chunk_hi, sizeof(int) * chi.size());
    if (e == cudaSuccess) e = device_alloc(&t.d_long_row, sizeof(int) * lrow.size());
    if (e == cudaSuccess) e = device_alloc(&t.d_long_first, sizeof(int) * lfirst.size());
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_hi_short, hi.data(), sizeof(int) * hi.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_chunk_lo, clo.data(), sizeof(int) * clo.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_chunk_hi, chi.data(), sizeof(int) * chi.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_long_row, lrow.data(), sizeof(int) * lrow.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_long_first, lfirst.data(), sizeof(int) * lfirst.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // the vectors go out of scope
    if (e != cudaSuccess) {
        record_cuda_error(e, "long rows of the dense-block product");
        spmm_split_destroy(t);
        return ALPHA_SPARSE_STATUS_ALLOC_FAILED;
    }
    memcpy(t.h_long_row, lrow.data(), sizeof(int) * lrow.size());
    memcpy(t.h_long_first, lfirst.data(), sizeof(int) * lfirst.size());
    t.state = 2;
    sp = t;
    ctx->device_bytes += (int64_t)(sizeof(int) * (hi.size() + clo.size() + chi.size() + lrow.size() + lfirst.size()));
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// The chunk tables (first product of the handle) and room for the partial sums of a product with `columns` columns.
static alphasparse_status_t spmm_split_prepare(DeviceCtx *ctx, size_t tsz, int columns, cudaStream_t st) {
    alphasparse_status_t s = spmm_split_ensure(ctx, st);
    if (s != ALPHA_SPARSE_STATUS_SUCCESS || ctx->split.state != 2) return s;
    SpmmSplit &sp = ctx->split;
    const size_t want = tsz * (size_t)sp.nchunks * (size_t)columns;
    if (sp.part_bytes < want) {
        cudaFree(sp.d_part);
        ctx->device_bytes -= (int64_t)sp.part_bytes;
        sp.d_part = nullptr, sp.part_bytes = 0;
        ASB_CUDA_OR(device_alloc(&sp.d_part, want), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        sp.part_bytes = want;
        ctx->device_bytes += (int64_t)want;
    }
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// ---- segments of a skewed matrix ---------------------------------------------------------------------

void spmm_segments_destroy(SpmmSegments &s) {
    cudaFree(s.d_seg);  // (one block: the other tables lie behind it)
    for (const SpmmSegments::Part &p : s.parts) cudaFree(p.p);
    s = SpmmSegments{};
}

// Rows of such lengths that segments of whole rows would not be of equal work.
static bool spmm_uneven(const DeviceCtx *ctx) {
    return option(kOptSpmmSplitMin) > 0 && ctx->max_row_nnz > kStreamWhole && (double)ctx->max_row_nnz > 8.0 * ctx->mean_row_nnz;
}

// Built at the first product of a handle whose rows are uneven (even rows need no table).
// Segments of 64 to 256 items, enough of them to keep every warp of the chip (about 5,000) busy twice.
static alphasparse_status_t spmm_segments_ensure(DeviceCtx *ctx, cudaStream_t st) {
    SpmmSegments &sp = ctx->segments;
    if (sp.state != 0) return ALPHA_SPARSE_STATUS_SUCCESS;
    const int64_t most = std::max<int64_t>(64, std::min<int64_t>(256, option(kOptSpmmSplitChunk)));
    if (!spmm_uneven(ctx)) {
        sp.state = 1;
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    const int64_t total = ctx->nnz + kStreamRowItems * ctx->rows;
    int64_t items = 64;
    while (items < most && total / items > 2 * 5000) items *= 2;
    items = std::min(items, most);
    SpmmSegments t;
    t.nseg = (int)((total + items - 1) / items);
    auto fail = [&](alphasparse_status_t s) {
        spmm_segments_destroy(t);
        return s;
    };
    std::vector<int> slot, first;
    std::vector<MergeCoord> seg;
    // one block for the four tables (every segment may leave a part of another row: nseg rows at most), since an
    // allocation takes as long as everything else here
    const size_t n = (size_t)t.nseg, table_bytes = sizeof(MergeCoord) * (n + 1) + sizeof(int) * (3 * n + 1);
    cudaError_t e = device_alloc(&t.d_seg, table_bytes);
    if (e != cudaSuccess) {
        record_cuda_error(e, "segments of the dense-block product");
        return fail(ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    }
    t.d_slot = reinterpret_cast<int *>(t.d_seg + n + 1), t.d_row = t.d_slot + n, t.d_first = t.d_row + n;
    spmm_segments_kernel<<<(unsigned)(t.nseg / 256 + 1), 256, 0, st>>>((int)ctx->rows, (int)ctx->nnz, ctx->d_row_ptr, (int)items,
                                                                      t.nseg, t.d_seg, t.d_slot);
    count_launch();
    try {
        seg.resize((size_t)t.nseg + 1), slot.resize((size_t)t.nseg);
        e = cudaMemcpyAsync(seg.data(), t.d_seg, sizeof(MergeCoord) * seg.size(), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(slot.data(), t.d_slot, sizeof(int) * slot.size(), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) {
            t.seg_row.resize(seg.size());
            for (size_t i = 0; i < seg.size(); i++) t.seg_row[i] = seg[i].row;
            for (size_t i = 0; i < slot.size(); i++) {
                if (slot[i] < 0) continue;
                const int row = seg[i + 1].row;  // slots of a row are neighbours: its segments are
                if (t.cross_row.empty() || t.cross_row.back() != row) t.cross_row.push_back(row), t.cross_first.push_back((int)t.nslots);
                slot[i] = (int)t.nslots++;
            }
            t.cross_first.push_back((int)t.nslots);
        }
    } catch (...) {
        return fail(ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    }
    const size_t ncross = t.cross_row.size();
    if (e == cudaSuccess && ncross > 0) {
        e = cudaMemcpyAsync(t.d_row, t.cross_row.data(), sizeof(int) * ncross, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(t.d_first, t.cross_first.data(), sizeof(int) * (ncross + 1), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(t.d_slot, slot.data(), sizeof(int) * slot.size(), cudaMemcpyHostToDevice, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        record_cuda_error(e, "segments of the dense-block product");
        return fail(e == cudaErrorMemoryAllocation ? ALPHA_SPARSE_STATUS_ALLOC_FAILED : ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    }
    t.state = 2;
    sp = std::move(t);
    ctx->device_bytes += (int64_t)table_bytes;
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// The table (made at the first product of the handle) and room for the partial sums of a product with `columns` columns.
// *part: null when the product has to do with whole rows, because rows are even, because memory for the table is
// not to be had, or because the stream is being captured and nothing may be allocated now.
template <typename T>
static alphasparse_status_t spmm_segments_prepare(DeviceCtx *ctx, int columns, cudaStream_t st, T **part) {
    *part = nullptr;
    SpmmSegments &sp = ctx->segments;
    if (sp.state == 1) return ALPHA_SPARSE_STATUS_SUCCESS;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    ASB_CUDA_OR(cudaStreamIsCapturing(st, &capture), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    if (sp.state == 0) {
        if (capture != cudaStreamCaptureStatusNone) return ALPHA_SPARSE_STATUS_SUCCESS;
        const alphasparse_status_t s = spmm_segments_ensure(ctx, st);
        if (s == ALPHA_SPARSE_STATUS_ALLOC_FAILED) return ALPHA_SPARSE_STATUS_SUCCESS;
        if (s != ALPHA_SPARSE_STATUS_SUCCESS || sp.state != 2) return s;
    }
    const size_t want = std::max<size_t>(1, sizeof(T) * (size_t)sp.nslots * (size_t)columns);
    size_t have = 0;
    for (const SpmmSegments::Part &p : sp.parts) {
        if (p.st != st) continue;
        if (p.bytes >= want) {
            *part = static_cast<T *>(p.p);
            return ALPHA_SPARSE_STATUS_SUCCESS;
        }
        have = std::max(have, p.bytes);
    }
    if (capture != cudaStreamCaptureStatusNone) return ALPHA_SPARSE_STATUS_SUCCESS;
    SpmmSegments::Part grown{st, nullptr, std::max(want, 2 * have)};
    try {
        sp.parts.reserve(sp.parts.size() + 1);
    } catch (...) {
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    const cudaError_t e = device_alloc_bytes(&grown.p, grown.bytes);
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    ASB_CUDA_OR(e, ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    sp.parts.push_back(grown);
    ctx->device_bytes += (int64_t)grown.bytes;
    *part = static_cast<T *>(grown.p);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// Column blocks are used only when asked for (option spmm_col_blocks > 1).  Measured on B200 with 64 fp32 columns,
// 2^21 rows of 32 elements and a 537 MB X: 3.51 ms in one pass, 4.08 / 4.60 / 5.16 / 6.37 ms with 4 / 6 / 8 / 12
// blocks.  Blocking does take the reads of X off HBM, but every stored element still pulls a whole row of X from
// L2 into an SM, and that stream (17 GB) already runs at the pace the one-pass kernel reaches from HBM; the
// extra passes over Y and the shorter per-row runs only add to it.
// Rows too long for one lane group come first: with them the product runs in segments, in one pass.
static int spmm_pick_blocks(const DeviceCtx *ctx) {
    const int64_t blocks = spmm_long_rows(ctx) ? 1 : option(kOptSpmmColBlocks);
    return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, 64));
}

// Which of the two kernels multiplies: a lane group per row (spmm_row_kernel: 32 / LPR rows end at once, nothing is
// fetched ahead) or a warp walking the elements (spmm_stream_kernel: ending a row takes the whole warp some 200
// instructions and, with beta != 0, a wait for Y, but X rows are requested ahead).  So rows of few elements go to the
// former, and the more so the fewer lanes a row takes, where Y is read, and where X rows come quickly because neighbouring
// rows share them (`banded`).  Measured (B200, row / stream kernel, us): diagonal of 262,144 rows x 12 fp32 columns, beta
// != 0 12.4 / 53.9; 2^20 rows of 5 x 12 94 / 216, x 64 359 / 384, x 128 718 / 711; 2^20 rows of 12 x 16, banded 122 / 187; 2^19
// rows of 20 x 12 172 / 153, banded 105 / 140; 262,144 rows of 27 x 24 145 / 109, x 64 261 / 219.  The limits below are mean row
// lengths at which the two were level, from 10,900 pairs over 2^10 to 2^22 rows, 1 to 160 elements, 5 to 256 columns and both
// precisions; a rule that always knew would be 1.1 % faster over those.
//
// With fewer rows than fill the chip a few times over, what counts is the longest row: the row kernel walks it four
// elements at a time, 0.24 us each, while the stream kernel takes 6-8 us however long its rows.  (2^13 rows of 8 +- 3 x 12 fp32
// columns 13 / 7, all of 8 7 / 11.)  That also bounds what an uneven matrix may have: its longest row has to be done in the
// time of the others (2^20 rows of 1 and one of 100 x 12 82 / 176, one of 400 186 / 177; 262,144 rows and one of 400 119 / 48),
// and wider blocks are worth it only where the stream kernel would wait for Y (2^20 x 24 and one of 100 130 / 196, beta = 0
// 119 / 113).
//
// An odd number of columns below 32 in single precision fills its one slice of 32 lanes: the limits of {4, 32} are those of
// more columns, whose last slice is nearly empty (2^20 rows of 1 x 31, beta = 0 225 / 114, x 33 275 / 230).
static bool spmm_row_by_row(const DeviceCtx *ctx, int lane_bytes, int lanes, int columns, bool has_beta) {
    struct Limit {
        int lane_bytes, lanes;
        float mean[2][2];  // [banded][beta != 0]
        int longest;       // of up to kRowsFew rows
    };
    static const Limit limits[] = {
        {16, 4, {{9.f, 12.5f}, {15.f, 30.f}}, 11}, {16, 8, {{5.f, 9.f}, {10.f, 15.f}}, 15},
        {16, 16, {{0.7f, 5.f}, {3.f, 10.f}}, 21},  {16, 32, {{0.8f, 5.f}, {0.5f, 0.9f}}, 24},
        {8, 8, {{8.f, 12.f}, {15.f, 40.f}}, 15},   {8, 16, {{0.7f, 10.f}, {7.f, 27.f}}, 21},
        {8, 32, {{0.9f, 28.f}, {0.7f, 0.8f}}, 44}, {4, 16, {{160.f, 40.f}, {30.f, 160.f}}, 24},
        {4, 32, {{7.f, 30.f}, {1.f, 15.f}}, 44},
    };
    constexpr int64_t kRowsOneWave = 148 * 32, kRowsFew = 40000;
    const Limit *l = std::find_if(std::begin(limits), std::end(limits),
                                  [&](const Limit &c) { return c.lane_bytes == lane_bytes && c.lanes == lanes; });
    if (l == std::end(limits)) l = limits;  // (few lanes of few bytes: blocks of at most 32 bytes, asked for by option)
    float mean = l->mean[ctx->shifted_rows >= 0.5][has_beta];
    if (lane_bytes == 4 && columns < 32 && lanes == 32 && !has_beta) mean = std::min(mean, 0.9f);
    if (spmm_uneven(ctx))
        return (has_beta || lanes == 4) && 20000 * ctx->max_row_nnz <= ctx->rows + ctx->nnz && ctx->mean_row_nnz <= 0.5 * mean;
    if (ctx->rows <= kRowsFew) return ctx->max_row_nnz <= (ctx->rows <= kRowsOneWave ? std::max(8, l->longest / 3) : l->longest);
    return ctx->mean_row_nnz <= mean;
}

// spmm_row_kernel over whole rows, or (option spmm_col_blocks) in one pass per column block over the part of every row
// inside the block.
template <typename T, int VEC, int LPR>
static void launch_row_groups(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y,
                              int ldy, cudaStream_t st, const RowWindow *w) {
    constexpr int rows_per_block = 8 * (32 / LPR);
    // A window is the same kernel on a slice: offsets are absolute, so shifting the offset arrays and Y
    // by the first row is all it takes.
    const int64_t first = w ? w->begin : 0, rows = w ? w->count : ctx->rows;
    const unsigned blocks = (unsigned)((rows + rows_per_block - 1) / rows_per_block);
    const T *val = static_cast<const T *>(ctx->d_val);
    Y += first * (int64_t)ldy;
    const int passes = ctx->spmm.d_split ? ctx->spmm.blocks : 1;
    for (int p = 0; p < passes; p++) {
        const int *lo = ctx->spmm.d_split ? ctx->spmm.d_split + (size_t)p * ctx->rows + first : ctx->d_row_ptr + first;
        const int *hi = ctx->spmm.d_split ? lo + ctx->rows : lo + 1;
        // the first pass applies beta, the later ones add to what is there
        const T b = p == 0 ? beta : T(1);
        if (b == T(0))
            spmm_row_kernel<T, VEC, LPR, false><<<blocks, 256, 0, st>>>(
                (int)rows, lo, hi, ctx->d_col, val, X, columns, ldx, Y, ldy, alpha, b);
        else
            spmm_row_kernel<T, VEC, LPR, true><<<blocks, 256, 0, st>>>(
                (int)rows, lo, hi, ctx->d_col, val, X, columns, ldx, Y, ldy, alpha, b);
    }
    count_launch(passes);
}

template <typename T, int VEC, int LPR>
static alphasparse_status_t launch_row(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y,
                                       int ldy, cudaStream_t st, const RowWindow *w) {
    T *part = nullptr;
    if (ctx->spmm.d_split || spmm_row_by_row(ctx, VEC * (int)sizeof(T), LPR, columns, beta != T(0))) {
        if (ctx->profile) cudaEventRecord(ctx->ev_start, st);
        launch_row_groups<T, VEC, LPR>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
        if (ctx->profile) cudaEventRecord(ctx->ev_stop, st);
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    const alphasparse_status_t s = spmm_segments_prepare<T>(ctx, columns, st, &part);
    if (s != ALPHA_SPARSE_STATUS_SUCCESS) return s;
    SpmmSegments &sp = ctx->segments;
    if (ctx->profile) cudaEventRecord(ctx->ev_start, st);
    const int row0 = (int)(w ? w->begin : 0), row1 = (int)(w ? w->begin + w->count : ctx->rows);
    StreamSegments sg{};
    sg.row0 = row0, sg.row1 = row1;
    int64_t groups;
    if (part) {
        // segments that hold anything of the window: the first one that ends at or behind its first row, up to the
        // first one that ends at or behind its end
        const auto b = sp.seg_row.begin() + 1, e = sp.seg_row.end();
        const int64_t s0 = std::lower_bound(b, e, row0) - b, s1 = std::min<int64_t>(sp.nseg, std::lower_bound(b, e, row1) - b + 1);
        sg.seg = sp.d_seg + s0, sg.slot = sp.d_slot + s0, sg.nseg = (int)(s1 - s0);
        groups = s1 - s0;
    } else {
        // whole rows, about 256 elements a warp, but no fewer warps than the chip holds twice
        const int64_t rows = row1 - row0, resident = 148ll * 4 * 8;
        int64_t per = (int64_t)(256.0 / std::max(1.0, ctx->mean_row_nnz));
        per = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(per, 64), rows / (2 * resident)));
        sg.per_warp = (int)per;
        groups = (rows + per - 1) / per;
    }
    const T *val = static_cast<const T *>(ctx->d_val);
    // (one launch for up to 65535 slices of LPR * VEC columns, the most a grid is high)
    for (int64_t c0 = 0; c0 < columns; c0 += 65535ll * (LPR * VEC)) {
        const int64_t slices = std::min<int64_t>(65535, (columns - c0 + LPR * VEC - 1) / (LPR * VEC));
        const dim3 grid((unsigned)((groups + 7) / 8), (unsigned)slices);
        if (beta == T(0))
            spmm_stream_kernel<T, VEC, LPR, false><<<grid, 256, 0, st>>>(sg, ctx->d_row_ptr, ctx->d_col, val, X, (int)c0, columns,
                                                                        ldx, Y, ldy, part, alpha, beta);
        else
            spmm_stream_kernel<T, VEC, LPR, true><<<grid, 256, 0, st>>>(sg, ctx->d_row_ptr, ctx->d_col, val, X, (int)c0, columns,
                                                                       ldx, Y, ldy, part, alpha, beta);
        count_launch();
    }
    if (part) {
        const int64_t l0 = std::lower_bound(sp.cross_row.begin(), sp.cross_row.end(), row0) - sp.cross_row.begin();
        const int64_t l1 = std::lower_bound(sp.cross_row.begin(), sp.cross_row.end(), row1) - sp.cross_row.begin();
        if (l1 > l0) {
            spmm_cross_reduce_kernel<T><<<(unsigned)(l1 - l0), 256, 0, st>>>(sp.d_row + l0, sp.d_first + l0, part, columns, Y, ldy);
            count_launch();
        }
    }
    if (ctx->profile) cudaEventRecord(ctx->ev_stop, st);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

template <typename T, int VEC>
static alphasparse_status_t launch_row_lanes(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y,
                                             int ldy, cudaStream_t st, const RowWindow *w) {
    // smallest group (4 .. 32 lanes) whose lanes cover the dense columns in one pass, if any
    const int need = (columns + VEC - 1) / VEC;
    // An X beyond L2 (126 MB) with unstructured columns is read in slices of 256 bytes a row: the part of X in use is half
    // as large and more of it stays in L2.  Measured (us, 32 -> 16 lanes): 474,552 rows of 27 elements x 128 fp32 / 128 fp64
    // / 64 fp64 columns 796 / 1639 / 917 -> 721 / 1465 / 852, power-law 400,009 rows x 64 fp64 685 -> 615.  Not where X fits
    // (50,000 rows x 128 fp64 columns 139 -> 158), neighbouring rows share X rows (stencil 78^3 x 128 fp64 933 -> 1042) or
    // lanes hold less than 16 bytes (200,000 rows x 127 fp32 columns 603 -> 877).
    const bool sliced = VEC * sizeof(T) == 16 && ctx->shifted_rows < 0.5 && sizeof(T) * (size_t)ctx->cols * columns > (126u << 20);
    if (need <= 4) return launch_row<T, VEC, 4>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
    if (need <= 8) return launch_row<T, VEC, 8>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
    if (need <= 16 || (sliced && !spmm_row_by_row(ctx, VEC * (int)sizeof(T), 32, columns, beta != T(0))))
        return launch_row<T, VEC, 16>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
    return launch_row<T, VEC, 32>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
}

template <typename T, int LANES, int KC, bool ALIGNED>
static void launch_narrow_as(int rows, const int *lo, const int *hi, DeviceCtx *ctx, T alpha, const T *X, int columns,
                             int ldx, T beta, T *Y, long long ldy, cudaStream_t st) {
    const unsigned blocks = (unsigned)(((long long)rows + 256 / LANES - 1) / (256 / LANES));
    const T *val = static_cast<const T *>(ctx->d_val);
    if (beta == T(0))
        spmm_row_narrow_kernel<T, LANES, KC, ALIGNED, false><<<blocks, 256, 0, st>>>(rows, lo, hi, ctx->d_col, val, X, columns,
                                                                                    ldx, Y, ldy, alpha, beta);
    else
        spmm_row_narrow_kernel<T, LANES, KC, ALIGNED, true><<<blocks, 256, 0, st>>>(rows, lo, hi, ctx->d_col, val, X, columns,
                                                                                   ldx, Y, ldy, alpha, beta);
    count_launch();
}

template <typename T, int KC, bool ALIGNED>
static void launch_narrow_lanes(int lanes, int rows, const int *lo, const int *hi, DeviceCtx *ctx, T alpha, const T *X,
                                int columns, int ldx, T beta, T *Y, long long ldy, cudaStream_t st) {
    if (lanes <= 4) launch_narrow_as<T, 4, KC, ALIGNED>(rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (lanes <= 8) launch_narrow_as<T, 8, KC, ALIGNED>(rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (lanes <= 16) launch_narrow_as<T, 16, KC, ALIGNED>(rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else launch_narrow_as<T, 32, KC, ALIGNED>(rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
}

// One launch of the narrow kernel over `rows` rows (or chunks) in the widest form the shapes allow.
template <typename T>
static void launch_narrow_pick(int lanes, int rows, const int *lo, const int *hi, DeviceCtx *ctx, T alpha, const T *X,
                               int columns, int ldx, T beta, T *Y, long long ldy, cudaStream_t st) {
    constexpr int PER16 = 16 / (int)sizeof(T), WIDE = 2 * PER16;
    const bool aligned = ((uintptr_t)X & 15) == 0 && ldx % PER16 == 0;
    if (aligned && columns == WIDE)
        launch_narrow_lanes<T, WIDE, true>(lanes, rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (aligned && columns == PER16)
        launch_narrow_lanes<T, PER16, true>(lanes, rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (columns <= PER16)
        launch_narrow_lanes<T, PER16, false>(lanes, rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else
        launch_narrow_lanes<T, WIDE, false>(lanes, rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
}

// The row-major product with an X row of at most 32 bytes: windows and long rows as in launch_row.
template <typename T>
static void launch_narrow(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y, int ldy, cudaStream_t st,
                          const RowWindow *w) {
    const int64_t first = w ? w->begin : 0, rows = w ? w->count : ctx->rows;
    const SpmmSplit &sp = ctx->split;
    const bool split = sp.state == 2;
    const double m = ctx->mean_row_nnz;
    const int lanes = m <= 8 ? 4 : m <= 16 ? 8 : m <= 32 ? 16 : 32;
    if (ctx->profile) cudaEventRecord(ctx->ev_start, st);
    const int *lo = ctx->d_row_ptr + first, *hi = split ? sp.d_hi_short + first : lo + 1;
    launch_narrow_pick<T>(lanes, (int)rows, lo, hi, ctx, alpha, X, columns, ldx, beta, Y + first * (int64_t)ldy, ldy, st);
    if (split) {
        const int *lb = std::lower_bound(sp.h_long_row, sp.h_long_row + sp.nlong, (int)first);
        const int *le = std::lower_bound(sp.h_long_row, sp.h_long_row + sp.nlong, (int)(first + rows));
        const int64_t l0 = lb - sp.h_long_row, l1 = le - sp.h_long_row;
        const int64_t c0 = sp.h_long_first[l0], c1 = sp.h_long_first[l1];
        if (c1 > c0) {
            T *part = static_cast<T *>(sp.d_part) + (size_t)c0 * columns;
            // the partial sums are a dense block of their own: `columns` wide, rows packed
            launch_narrow_pick<T>(32, (int)(c1 - c0), sp.d_chunk_lo + c0, sp.d_chunk_hi + c0, ctx, alpha, X, columns, ldx, T(0),
                                  part, columns, st);
            spmm_long_reduce_kernel<T><<<(unsigned)(l1 - l0), 32, 0, st>>>(sp.d_long_row + l0, sp.d_long_first + l0,
                                                                         static_cast<const T *>(sp.d_part), columns, Y, ldy);
            count_launch();
        }
    }
    if (ctx->profile) cudaEventRecord(ctx->ev_stop, st);
}

template <typename T>
alphasparse_status_t launch_spmm_row(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx,
                                     T beta, T *Y, int ldy, cudaStream_t st, const RowWindow *w) {
    if (ctx->rows == 0 || columns <= 0 || (w && w->count <= 0)) return ALPHA_SPARSE_STATUS_SUCCESS;
    block_used(ctx, st);
    const bool narrow = (size_t)columns * sizeof(T) <= 32 && option(kOptSpmmNarrow);
    alphasparse_status_t bs;
    if (narrow) {
        bs = spmm_split_prepare(ctx, sizeof(T), columns, st);
        if (bs != ALPHA_SPARSE_STATUS_SUCCESS) return bs;
        launch_narrow<T>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
        ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    bs = col_blocks_ensure(ctx, ctx->spmm, spmm_pick_blocks(ctx), st);
    if (bs != ALPHA_SPARSE_STATUS_SUCCESS) return bs;
    auto fits = [&](int vec) {
        const uintptr_t mask = (uintptr_t)(vec * sizeof(T) - 1);
        return columns % vec == 0 && ldx % vec == 0 && ldy % vec == 0 &&
               ((uintptr_t)X & mask) == 0 && ((uintptr_t)Y & mask) == 0;
    };
    // Widest 16-byte pack the shapes and alignments allow.
    if constexpr (sizeof(T) == 4) {
        if (fits(4)) bs = launch_row_lanes<T, 4>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
        else if (fits(2)) bs = launch_row_lanes<T, 2>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
        else bs = launch_row_lanes<T, 1>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
    } else {
        if (fits(2)) bs = launch_row_lanes<T, 2>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
        else bs = launch_row_lanes<T, 1>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st, w);
    }
    if (bs != ALPHA_SPARSE_STATUS_SUCCESS) return bs;
    ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// ---- column-major dense operands ------------------------------------------------------------------
//
// Y[:, c] = beta * Y[:, c] + alpha * (A * X[:, c]) for every dense column c, element (r, c) of a dense
// operand at [c * ld + r]: the operation of the reference's gemm_{s,d}_csr_col (arithmetic defined by
// src/plain/kernel/level3/mm/gemm/gemm_x_csr_col_plain.c:4-21: a dot product from zero per (row, column),
// then y = y*beta + alpha*dot).  Each dense column is an independent SpMV on the same A, so the kernel
// is the vector SpMV with KC columns carried side by side: a group of LANES lanes owns a sparse row,
// every stored element is loaded once and multiplied into KC accumulators, one gather per column.
// blockIdx.y selects the block of KC columns; A is re-read once per block.
template <typename T, int LANES, int KC, bool HAS_BETA>
__global__ void __launch_bounds__(256)
    spmm_col_kernel(int rows, const int *__restrict__ row_lo, const int *__restrict__ row_hi,
                    const int *__restrict__ col, const T *__restrict__ val, const T *__restrict__ X, int columns,
                    long long ldx, T *__restrict__ Y, long long ldy, T alpha, T beta) {
    constexpr int GROUPS = 256 / LANES;
    const int lane = threadIdx.x % LANES;
    const long long row = (long long)blockIdx.x * GROUPS + threadIdx.x / LANES;
    const int c0 = blockIdx.y * KC;
    int s = 0, e = 0;
    if (row < rows) {  // the whole row, or the chunk of a long row that stands in for a row (see SpmmSplit)
        s = __ldg(row_lo + row);
        e = __ldg(row_hi + row);
    }
    T acc[KC];
#pragma unroll
    for (int k = 0; k < KC; k++) acc[k] = T(0);
    for (int j = s + lane; j < e; j += LANES) {
        const int cj = __ldg(col + j);
        const T vj = __ldg(val + j);
#pragma unroll
        for (int k = 0; k < KC; k++)
            if (c0 + k < columns) acc[k] = fma(vj, __ldg(X + (long long)(c0 + k) * ldx + cj), acc[k]);
    }
#pragma unroll
    for (int k = 0; k < KC; k++) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    }
    if (lane == 0 && row < rows) {
#pragma unroll
        for (int k = 0; k < KC; k++)
            if (c0 + k < columns) {
                T *out = Y + (long long)(c0 + k) * ldy + row;
                T o = alpha * acc[k];
                if (HAS_BETA) o = fma(beta, *out, o);
                *out = o;
            }
    }
}

// Y[c * ldy + row] += the row's partial sums (part[c * nchunks + k]) in chunk order: one thread per (long row, column).
template <typename T>
__global__ void spmm_long_reduce_col_kernel(int nlong, const int *__restrict__ long_row, const int *__restrict__ long_first,
                                            const T *__restrict__ part, long long nchunks, int columns, T *__restrict__ Y,
                                            long long ldy) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nlong * columns) return;
    const int l = (int)(i % nlong), c = (int)(i / nlong);
    T acc = T(0);
    for (int k = long_first[l]; k < long_first[l + 1]; k++) acc += part[(long long)c * nchunks + k];
    Y[(long long)c * ldy + long_row[l]] += acc;
}

template <typename T, int LANES>
static void launch_col(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y, int ldy,
                       cudaStream_t st) {
    constexpr int KC = 4;
    const dim3 grid((unsigned)((ctx->rows + 256 / LANES - 1) / (256 / LANES)), (unsigned)((columns + KC - 1) / KC));
    const T *val = static_cast<const T *>(ctx->d_val);
    const SpmmSplit &sp = ctx->split;
    const bool split = sp.state == 2;
    const int *hi = split ? sp.d_hi_short : ctx->d_row_ptr + 1;
    if (ctx->profile) cudaEventRecord(ctx->ev_start, st);
    if (beta == T(0))
        spmm_col_kernel<T, LANES, KC, false><<<grid, 256, 0, st>>>((int)ctx->rows, ctx->d_row_ptr, hi, ctx->d_col, val, X,
                                                                  columns, ldx, Y, ldy, alpha, beta);
    else
        spmm_col_kernel<T, LANES, KC, true><<<grid, 256, 0, st>>>((int)ctx->rows, ctx->d_row_ptr, hi, ctx->d_col, val, X,
                                                                 columns, ldx, Y, ldy, alpha, beta);
    count_launch();
    if (split && sp.nchunks > 0) {
        // the chunks of the long rows as rows of their own (a warp each) into partial sums, then onto Y
        T *part = static_cast<T *>(sp.d_part);
        const dim3 cgrid((unsigned)((sp.nchunks + 7) / 8), grid.y);
        spmm_col_kernel<T, 32, KC, false><<<cgrid, 256, 0, st>>>((int)sp.nchunks, sp.d_chunk_lo, sp.d_chunk_hi, ctx->d_col, val,
                                                                X, columns, ldx, part, sp.nchunks, alpha, T(0));
        const long long cells = (long long)sp.nlong * columns;
        spmm_long_reduce_col_kernel<T><<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(
            (int)sp.nlong, sp.d_long_row, sp.d_long_first, part, sp.nchunks, columns, Y, ldy);
        count_launch(2);
    }
    if (ctx->profile) cudaEventRecord(ctx->ev_stop, st);
}

// ---- column-major operands, banded matrix ---------------------------------------------------------------
//
// When neighbouring rows hold neighbouring columns (stencils, banded matrices in natural order) a lane per row gathers
// coalesced from every column of X as it is stored, so nothing needs transposing: a warp stages the offsets, columns and
// values of kRowTileSmall rows in shared memory once (as the row-tile SpMV does, spmv.cu) and walks them for KC dense columns
// at a time.  A is read once from HBM, X and Y once each; what bounds it is the latency of the gathers (they come out of
// L2: shared memory leaves L1 little room), so U elements of a row are taken together, U * KC gathers in flight.
// Measured (B200, 27-point stencil 80^3, us, through transposes -> here): fp64 1 / 2 / 4 / 6 / 13 / 32 columns 87 / 115 / 159 /
// 211 / 316 / 569 -> 40 / 42 / 52 / 60 / 118 / 220; fp32 3 / 6 / 32 columns 117 / 173 / 264 -> 33 / 50 / 181; 20^3 fp32 x 32
// columns 25 -> 9.  U = 2 for eight columns took 310 us for 32 (3: 220, 4: 218 in fp64, but 181 -> 218 in fp32); U = 2 / 4
// for six 81 / 73 (6: 60).  Blocks of four warps made no difference, fewer resident warps (more L1) lost 20-80 %.
template <typename T, int KC, bool HAS_BETA>
__global__ void __launch_bounds__(kRowTileSmall)
    spmm_col_tile_kernel(int rows, const int *__restrict__ row_ptr, const int *__restrict__ col, const T *__restrict__ val,
                         const T *__restrict__ X, int columns, long long ldx, T *__restrict__ Y, long long ldy, T alpha,
                         T beta, int cap, int *__restrict__ status) {
    constexpr int U = KC >= 8 ? 3 : KC >= 4 ? 6 : 8;
    extern __shared__ __align__(128) unsigned char smem[];
    T *s_val = reinterpret_cast<T *>(smem);
    int *s_col = reinterpret_cast<int *>(s_val + cap);
    int *s_ptr = s_col + cap;

    const int tid = threadIdx.x;
    const int r0 = blockIdx.x * kRowTileSmall;
    const int nr = min(kRowTileSmall, rows - r0);
    if (!stage_row_tile<T, kRowTileSmall>(r0, nr, row_ptr, col, val, s_val, s_col, s_ptr, cap, status) || tid >= nr) return;

    const int a0 = s_ptr[0] & ~3;
    const int b = s_ptr[tid] - a0, e = s_ptr[tid + 1] - a0;
    const long long r = r0 + tid;
    for (long long c0 = (long long)blockIdx.y * KC; c0 < columns; c0 += (long long)gridDim.y * KC) {
        const int live = (int)min((long long)KC, columns - c0);
        const T *x[KC];  // (beyond the last column: the last one again, dropped below)
        T acc[KC], old[KC];
#pragma unroll
        for (int i = 0; i < KC; i++) {
            x[i] = X + (c0 + min(i, live - 1)) * ldx;
            acc[i] = T(0), old[i] = T(0);
            if (HAS_BETA && i < live) old[i] = __ldcs(Y + (c0 + i) * ldy + r);
        }
        for (int k = b; k < e; k += U) {
            T v[U], xv[U][KC];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (k + u < e) {
                    const int c = s_col[k + u];
                    v[u] = s_val[k + u];
#pragma unroll
                    for (int i = 0; i < KC; i++) xv[u][i] = __ldg(x[i] + c);
                }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (k + u < e) {
#pragma unroll
                    for (int i = 0; i < KC; i++) acc[i] = fma(v[u], xv[u][i], acc[i]);
                }
        }
#pragma unroll
        for (int i = 0; i < KC; i++)
            if (i < live) __stcs(Y + (c0 + i) * ldy + r, HAS_BETA ? fma(beta, old[i], alpha * acc[i]) : alpha * acc[i]);
    }
}

template <typename T, int KC>
static alphasparse_status_t launch_col_tile(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y, int ldy,
                                            cudaStream_t st) {
    auto kernel = beta == T(0) ? spmm_col_tile_kernel<T, KC, false> : spmm_col_tile_kernel<T, KC, true>;
    const size_t smem = rowtile_smem_bytes(ctx, kRowTileSmall);
    static std::atomic<unsigned long long> granted[2];
    ASB_CUDA_OR(allow_tile_smem(reinterpret_cast<const void *>(kernel), smem, ctx->device, &granted[beta == T(0) ? 0 : 1]),
                ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    // A warp does all columns of its rows; where the rows alone do not fill the chip they are shared out.
    const int64_t tiles = (ctx->rows + kRowTileSmall - 1) / kRowTileSmall, chunks = (columns + KC - 1) / KC;
    const int64_t share = std::min(chunks, std::max<int64_t>(1, 148 * 32 / tiles));
    if (ctx->profile) cudaEventRecord(ctx->ev_start, st);
    kernel<<<dim3((unsigned)tiles, (unsigned)share), kRowTileSmall, smem, st>>>(
        (int)ctx->rows, ctx->d_row_ptr, ctx->d_col, static_cast<const T *>(ctx->d_val), X, columns, ldx, Y, ldy, alpha, beta,
        rowtile_cap(ctx, kRowTileSmall), ctx->d_status);
    if (ctx->profile) cudaEventRecord(ctx->ev_stop, st);
    count_launch();
    ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// B[f * ld_b + s] = A[s * ld_a + f] for f < n_fast, s < n_slow: a column-major operand (f = row, s = dense column)
// into a row-major one, or back (f = dense column, s = row).  32 x 32 tiles through shared memory; the tiles along the
// longer of the two extents are numbered by blockIdx.x (`slow_on_x`), whose range is the wide one.
template <typename T>
__global__ void __launch_bounds__(256) dense_transpose_kernel(long long n_fast, long long n_slow, const T *__restrict__ A,
                                                              long long ld_a, T *__restrict__ B, long long ld_b,
                                                              int slow_on_x) {
    __shared__ T tile[32][33];
    const long long f0 = (long long)(slow_on_x ? blockIdx.y : blockIdx.x) * 32;
    const long long s0 = (long long)(slow_on_x ? blockIdx.x : blockIdx.y) * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
        const long long f = f0 + tx, sl = s0 + ty + k;
        if (f < n_fast && sl < n_slow) tile[ty + k][tx] = A[sl * ld_a + f];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
        const long long f = f0 + ty + k, sl = s0 + tx;
        if (f < n_fast && sl < n_slow) B[f * ld_b + sl] = tile[tx][ty + k];
    }
}

template <typename T>
static void dense_transpose(long long n_fast, long long n_slow, const T *A, long long ld_a, T *B, long long ld_b,
                            cudaStream_t st) {
    const long long tf = (n_fast + 31) / 32, ts = (n_slow + 31) / 32;
    const int slow_on_x = ts > tf;
    const dim3 grid((unsigned)(slow_on_x ? ts : tf), (unsigned)(slow_on_x ? tf : ts));
    dense_transpose_kernel<T><<<grid, 256, 0, st>>>(n_fast, n_slow, A, ld_a, B, ld_b, slow_on_x);
    count_launch();
}

static alphasparse_status_t grow_scratch(DeviceCtx *ctx, void **buf, size_t *have, size_t want) {
    if (*have >= want) return ALPHA_SPARSE_STATUS_SUCCESS;
    cudaFree(*buf);
    ctx->device_bytes -= (int64_t)*have;
    *buf = nullptr, *have = 0;
    ASB_CUDA_OR(device_alloc(buf, want), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    *have = want;
    ctx->device_bytes += (int64_t)want;
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

template <typename T>
alphasparse_status_t launch_spmm_col(DeviceCtx *ctx, T alpha, const T *X, int columns, int ldx, T beta, T *Y,
                                     int ldy, cudaStream_t st) {
    if (ctx->rows == 0 || columns <= 0) return ALPHA_SPARSE_STATUS_SUCCESS;
    block_used(ctx, st);
    if (ctx->algorithm == ALPHA_SPARSE_CUDA_ALG_ROWTILE && ctx->shifted_rows >= 0.5 && ctx->nnz > 0 &&
        rowtile_smem_bytes(ctx, kRowTileSmall) <= 48 * 1024) {
        const int passes = (columns + 7) / 8, per = (columns + passes - 1) / passes;  // columns in equal groups of at most 8
        if (per <= 1) return launch_col_tile<T, 1>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
        if (per <= 2) return launch_col_tile<T, 2>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
        if (per <= 3) return launch_col_tile<T, 3>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
        if (per <= 4) return launch_col_tile<T, 4>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
        if (per <= 6) return launch_col_tile<T, 6>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
        return launch_col_tile<T, 8>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    }
    // The kernel below gathers one x element per (stored element, dense column): four L2 requests per element and
    // pass of four columns, where the row-major kernels take a whole X row with one or two (2^21 rows of 32 elements
    // times 8 / 64 fp32 columns: 2.0 / 16.2 ms column-major against 0.6 / 3.5 ms row-major).  From spmm_col_via_row
    // columns on the operands are therefore transposed into row-major copies kept with the handle (X, and Y when
    // beta != 0), multiplied there, and Y is transposed back.
    const int64_t via = option(kOptSpmmColViaRow);
    if (via > 0 && columns >= via && columns <= 32 * 65535) {
        const size_t xb = sizeof(T) * (size_t)ctx->cols * (size_t)columns, yb = sizeof(T) * (size_t)ctx->rows * (size_t)columns;
        alphasparse_status_t s = grow_scratch(ctx, &ctx->d_cm_x, &ctx->cm_x_bytes, xb);
        if (s == ALPHA_SPARSE_STATUS_SUCCESS) s = grow_scratch(ctx, &ctx->d_cm_y, &ctx->cm_y_bytes, yb);
        if (s != ALPHA_SPARSE_STATUS_SUCCESS) return s;
        T *xt = static_cast<T *>(ctx->d_cm_x), *yt = static_cast<T *>(ctx->d_cm_y);
        dense_transpose<T>(ctx->cols, columns, X, ldx, xt, columns, st);
        if (beta != T(0)) dense_transpose<T>(ctx->rows, columns, Y, ldy, yt, columns, st);
        s = launch_spmm_row<T>(ctx, alpha, xt, columns, columns, beta, yt, columns, st, nullptr);
        if (s != ALPHA_SPARSE_STATUS_SUCCESS) return s;
        dense_transpose<T>(columns, ctx->rows, yt, columns, Y, ldy, st);
        ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        return ALPHA_SPARSE_STATUS_SUCCESS;
    }
    if ((columns + 3) / 4 > 65535) return ALPHA_SPARSE_STATUS_NOT_SUPPORTED;
    const alphasparse_status_t ps = spmm_split_prepare(ctx, sizeof(T), columns, st);
    if (ps != ALPHA_SPARSE_STATUS_SUCCESS) return ps;
    const double m = ctx->mean_row_nnz;
    if (m <= 8) launch_col<T, 4>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (m <= 16) launch_col<T, 8>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else if (m <= 32) launch_col<T, 16>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    else launch_col<T, 32>(ctx, alpha, X, columns, ldx, beta, Y, ldy, st);
    ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

template alphasparse_status_t launch_spmm_col<float>(DeviceCtx *, float, const float *, int, int, float, float *,
                                                     int, cudaStream_t);
template alphasparse_status_t launch_spmm_col<double>(DeviceCtx *, double, const double *, int, int, double,
                                                      double *, int, cudaStream_t);

template alphasparse_status_t launch_spmm_row<float>(DeviceCtx *, float, const float *, int, int,
                                                     float, float *, int, cudaStream_t, const RowWindow *);
template alphasparse_status_t launch_spmm_row<double>(DeviceCtx *, double, const double *, int, int,
                                                      double, double *, int, cudaStream_t, const RowWindow *);

}  // namespace asb
