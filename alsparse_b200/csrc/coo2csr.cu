// COO -> CSR on the GPU, for alphasparse_convert_csr on large COO handles, and the matrices derived from a handle's
// device copy (transpose, structured descriptors): everything that sorts stored elements.
//
// The reference sorts (row, column, value) records with a serial qsort and then counts rows
// (src/core/format/convert_csr_x_coo.c:14-81); minutes at 2^28 elements.  Here the same output --
// elements ordered by row then column, duplicates kept, in input order among equals (qsort leaves
// that unspecified) -- comes from a stable least-significant-digit radix sort of keys that hold the row above
// the column in just the bits the dimensions need (32-bit keys when they fit, else 64-bit), carrying the element's
// position, up to 8 bits per pass, followed by one binary search per row for the offsets and one gather of the
// values.  Integer work, HBM-bound: every pass reads the keys twice and writes keys and positions once.
#include <algorithm>
#include <vector>

#include "internal.h"

namespace asb {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;  // elements per thread, 32 apart inside the warp's run of 512: coalesced loads
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortBins = 256;

// key of a (row, column) pair: row << col_bits | column
template <typename K>
__global__ void coo_keys_kernel(long long nnz, const int *__restrict__ ri, const int *__restrict__ ci, int rows,
                                int cols, int col_bits, K *__restrict__ keys, unsigned long long *__restrict__ bad) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnz) return;
    const int r = ri[i], c = ci[i];
    if (r < 0 || r >= rows || c < 0 || c >= cols) atomicAdd(bad, 1ull);
    keys[i] = ((K)(unsigned)r << col_bits) | (K)(unsigned)c;
}

// Per block: how many of its elements fall into each digit value.  hist is digit-major
// (hist[d * blocks + b]) so that one exclusive scan over it yields every block's write offsets.
template <typename K>
__global__ void __launch_bounds__(kSortThreads)
    radix_hist_kernel(long long n, const K *__restrict__ keys, int shift, unsigned mask, unsigned *__restrict__ hist) {
    __shared__ unsigned s_cnt[kSortBins];
    s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const long long base = (long long)blockIdx.x * kSortTile + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const long long i = base + k * kSortThreads;
        if (i < n) atomicAdd(&s_cnt[(unsigned)(keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s_cnt[threadIdx.x];
}

// Exclusive scan of n unsigned values in three steps (block sums, scan of the sums by one block, add).
constexpr int kScanThreads = 256, kScanItems = 16, kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned *total) {
    __shared__ unsigned s_warp[kScanThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    unsigned before = 0, all = 0;
    for (int w = 0; w < kScanThreads / 32; w++) {
        if (w < wid) before += s_warp[w];
        all += s_warp[w];
    }
    __syncthreads();
    if (total) *total = all;
    return before + inc - v;
}

__global__ void __launch_bounds__(kScanThreads)
    scan_sums_kernel(long long n, const unsigned *__restrict__ in, unsigned *__restrict__ sums) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    unsigned s = 0;
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n) s += in[base + k];
    unsigned total;
    block_exclusive_scan(s, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_top_kernel(int nblocks, unsigned *__restrict__ sums) {
    unsigned carry = 0;  // one block walks the block sums, kScanThreads at a time
    for (int base = 0; base < nblocks; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const unsigned v = i < nblocks ? sums[i] : 0;
        unsigned total;
        const unsigned ex = block_exclusive_scan(v, &total);
        if (i < nblocks) sums[i] = carry + ex;
        carry += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads)
    scan_apply_kernel(long long n, unsigned *__restrict__ data, const unsigned *__restrict__ sums) {
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    unsigned v[kScanItems], s = 0;
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? data[base + k] : 0;
        s += v[k];
    }
    unsigned run = sums[blockIdx.x] + block_exclusive_scan(s, nullptr);
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n) {
            data[base + k] = run;
            run += v[k];
        }
}

// Stable scatter of one pass.  A warp owns 512 consecutive elements and takes them 32 at a time; the lanes that hold
// the same digit find each other with one ballot per digit bit, so an element's rank among the warp's elements of its
// digit is (those of earlier steps) + (lower lanes of this step): element order, no atomics.  The tile is put in digit
// order in shared memory first and then written out, so that neighbouring threads write neighbouring addresses (runs of
// 16 elements per digit on average) where scattering straight from registers touches a sector per element: 3.7e6 64-bit
// keys of 36 bits take 10 passes of 60 us with 4-bit digits scattered directly, 5 of 45 us this way.
template <typename K>
__global__ void __launch_bounds__(kSortThreads)
    radix_scatter_kernel(long long n, const K *__restrict__ keys_in, const unsigned *__restrict__ pos_in, int shift,
                         unsigned mask, const unsigned *__restrict__ offs, K *__restrict__ keys_out,
                         unsigned *__restrict__ pos_out) {
    __shared__ K s_buf[kSortTile];  // the keys in digit order, then the positions
    __shared__ unsigned s_warp[kSortWarps][kSortBins];
    __shared__ unsigned s_dst[kSortBins];  // first destination of a digit minus its first place in the tile
    __shared__ unsigned s_sum[kSortWarps];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const long long base = (long long)blockIdx.x * kSortTile;
    const int count = (int)(n - base < kSortTile ? n - base : kSortTile);
    for (int i = t; i < kSortWarps * kSortBins; i += kSortThreads) (&s_warp[0][0])[i] = 0;
    __syncthreads();

    K key[kSortItems];
    unsigned place[kSortItems], pos[kSortItems];
    const int first = w * (32 * kSortItems) + lane;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const int i = first + 32 * k;
        key[k] = i < count ? keys_in[base + i] : (K)0;
        // no positions yet: the element's own place in the input
        pos[k] = i < count ? (pos_in ? pos_in[base + i] : (unsigned)(base + i)) : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        // slots beyond the input come after every element of the tile: counted with the last digit, never written
        const unsigned d = first + 32 * k < count ? (unsigned)(key[k] >> shift) & mask : (unsigned)kSortBins - 1;
        unsigned peers = 0xffffffffu;
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool bit = (d >> b) & 1u;
            const unsigned with = __ballot_sync(0xffffffffu, bit);
            peers &= bit ? with : ~with;
        }
        const unsigned before = s_warp[w][d];
        __syncwarp();
        const unsigned lower = __popc(peers & ((1u << lane) - 1u));
        if (lower == 0) s_warp[w][d] = before + __popc(peers);
        place[k] = before + lower;
        __syncwarp();
    }
    __syncthreads();
    {
        // thread t is digit t: exclusive prefix of its counts over the warps, then over the digits of the tile
        unsigned run = 0;
#pragma unroll
        for (int v = 0; v < kSortWarps; v++) {
            const unsigned c = s_warp[v][t];
            s_warp[v][t] = run;
            run += c;
        }
        unsigned inc = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) s_sum[w] = inc;
        __syncthreads();
        unsigned start = inc - run;
        for (int v = 0; v < w; v++) start += s_sum[v];
#pragma unroll
        for (int v = 0; v < kSortWarps; v++) s_warp[v][t] += start;
        s_dst[t] = offs[(size_t)t * gridDim.x + blockIdx.x] - start;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const unsigned d = first + 32 * k < count ? (unsigned)(key[k] >> shift) & mask : (unsigned)kSortBins - 1;
        place[k] += s_warp[w][d];
        s_buf[place[k]] = key[k];
    }
    __syncthreads();
    unsigned dst[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const int i = t + k * kSortThreads;
        if (i < count) {
            const K v = s_buf[i];
            dst[k] = s_dst[(unsigned)(v >> shift) & mask] + (unsigned)i;
            keys_out[dst[k]] = v;
        }
    }
    __syncthreads();
    unsigned *s_pos = reinterpret_cast<unsigned *>(s_buf);
#pragma unroll
    for (int k = 0; k < kSortItems; k++) s_pos[place[k]] = pos[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const int i = t + k * kSortThreads;
        if (i < count) pos_out[dst[k]] = s_pos[i];
    }
}

// ptr[r] = first sorted element whose row is >= r (r = 0 .. rows); columns in sorted order.
template <typename K>
__global__ void csr_from_sorted_kernel(long long nnz, int rows, int col_bits, const K *__restrict__ keys,
                                       int *__restrict__ ptr, int *__restrict__ col) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= rows) {
        long long lo = 0, hi = nnz;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if ((long long)(keys[mid] >> col_bits) < i) lo = mid + 1;
            else hi = mid;
        }
        ptr[i] = (int)lo;
    }
    if (i < nnz) col[i] = (int)(unsigned)(keys[i] & (((K)1 << col_bits) - 1));
}

template <typename T>
__global__ void gather_values_kernel(long long nnz, const unsigned *__restrict__ pos, const T *__restrict__ in,
                                     T *__restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nnz) out[i] = in[pos[i]];
}

static int bits_for(int64_t n) {
    int b = 1;
    while (b < 31 && (1ll << b) < n) b++;
    return b;
}

static alphasparse_status_t device_exclusive_scan(unsigned *d_data, long long n, unsigned *d_sums, cudaStream_t st) {
    const int nb = (int)((n + kScanTile - 1) / kScanTile);
    scan_sums_kernel<<<nb, kScanThreads, 0, st>>>(n, d_data, d_sums);
    scan_top_kernel<<<1, kScanThreads, 0, st>>>(nb, d_sums);
    scan_apply_kernel<<<nb, kScanThreads, 0, st>>>(n, d_data, d_sums);
    count_launch(3);
    ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// Pieces of one device block, each on a 256-byte boundary.  First pass with a null base: how much is needed.
struct Carve {
    char *base;
    size_t used = 0;
    explicit Carve(void *p) : base(static_cast<char *>(p)) {}
    template <typename P>
    P *take(size_t count) {
        char *p = base ? base + used : nullptr;
        used += (std::max<size_t>(count, 1) * sizeof(P) + 255) & ~(size_t)255;
        return reinterpret_cast<P *>(p);
    }
};

// Scratch of one sort of n keys.
template <typename K>
struct SortScratch {
    K *keys[2];
    unsigned *pos[2], *hist, *sums;
    SortScratch(Carve &c, long long n) {
        const size_t blocks = (size_t)((n + kSortTile - 1) / kSortTile), cells = blocks * kSortBins;
        keys[0] = c.take<K>((size_t)n), keys[1] = c.take<K>((size_t)n);
        pos[0] = c.take<unsigned>((size_t)n), pos[1] = c.take<unsigned>((size_t)n);
        hist = c.take<unsigned>(cells), sums = c.take<unsigned>((cells + kScanTile - 1) / kScanTile + 1);
    }
};

// Stable sort of s.keys[0] by its low `bits` bits; `payload`: s.pos[0] holds the elements' payloads (else they are the
// positions 0 .. n-1).  On return *cur says which of the two buffers holds the result.
template <typename K>
static alphasparse_status_t radix_sort(const SortScratch<K> &s, long long n, int bits, bool payload, int *cur, cudaStream_t st) {
    const unsigned blocks = (unsigned)((n + kSortTile - 1) / kSortTile);
    const int passes = std::max(1, (bits + 7) / 8);
    *cur = 0;
    for (int p = 0, shift = 0; p < passes; p++) {
        const int width = (bits - shift + (passes - p) - 1) / (passes - p);  // the bits left, spread over the passes left
        const unsigned mask = (1u << width) - 1u;
        radix_hist_kernel<K><<<blocks, kSortThreads, 0, st>>>(n, s.keys[*cur], shift, mask, s.hist);
        count_launch();
        alphasparse_status_t status = device_exclusive_scan(s.hist, (long long)blocks * kSortBins, s.sums, st);
        if (status != ALPHA_SPARSE_STATUS_SUCCESS) return status;
        radix_scatter_kernel<K><<<blocks, kSortThreads, 0, st>>>(n, s.keys[*cur], p > 0 || payload ? s.pos[*cur] : nullptr, shift,
                                                                mask, s.hist, s.keys[*cur ^ 1], s.pos[*cur ^ 1]);
        count_launch();
        *cur ^= 1;
        shift += width;
    }
    ASB_CUDA_OR(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// One block of a conversion, used on the library stream alone and given back when it goes out of scope.
struct ScopedBlock {
    DeviceBlock b;
    BlockUse use;
    explicit ScopedBlock(cudaStream_t st) { use.add(st); }
    ~ScopedBlock() { device_block_give(&b, use); }
    void done() { use = BlockUse{}; }  // the stream has been waited for
};

// Host COO arrays in, device CSR (one block, ctx_adopt_block's layout) and HOST 3-array CSR out (caller-provided buffers
// of rows+1 / nnz / nnz elements).  The index arrays go over first and are sorted while the values follow on a stream
// of their own.  (Sending the sorted columns back while the values come in was no faster: with the cores filling and
// emptying the rings both directions of the link slow down by what the overlap gains.)
template <typename T, typename K>
static alphasparse_status_t coo_to_csr_keyed(int64_t rows, int64_t cols, int64_t nnz, const int *ri, const int *ci,
                                             const T *v, int *out_ptr, int *out_col, T *out_val, DeviceBlock *out) {
    cudaStream_t st = current_stream();
    ScopedBlock scratch(st), result(st);
    const size_t n = (size_t)nnz;
#define TRY(expr, code) ASB_CUDA_OR(expr, code)
    auto layout = [&](void *p, int **d_ri, int **d_ci, T **d_v, unsigned long long **d_bad) {
        Carve c(p);
        *d_ri = c.take<int>(n), *d_ci = c.take<int>(n), *d_v = c.take<T>(n), *d_bad = c.take<unsigned long long>(1);
        SortScratch<K> s(c, nnz);
        return std::make_pair(s, c.used);
    };
    int *d_ri, *d_ci;
    T *d_v;
    unsigned long long *d_bad;
    TRY(device_block_take(layout(nullptr, &d_ri, &d_ci, &d_v, &d_bad).second, st, false, &scratch.b), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    const SortScratch<K> sort = layout(scratch.b.p, &d_ri, &d_ci, &d_v, &d_bad).first;
    TRY(device_block_take(adopt_block_bytes(sizeof(T), rows, nnz), st, true, &result.b), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    int *d_ptr, *d_col;
    T *d_val;
    adopt_block_layout(result.b.p, rows, nnz, &d_ptr, &d_col, &d_val);

    TRY(cudaMemsetAsync(d_bad, 0, 8, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(copy_to_device(d_ri, ri, sizeof(int) * n, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(copy_to_device(d_ci, ci, sizeof(int) * n, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    const unsigned blocks = (unsigned)((nnz + 255) / 256);
    const int col_bits = bits_for(cols);
    coo_keys_kernel<K><<<blocks, 256, 0, st>>>(nnz, d_ri, d_ci, (int)rows, (int)cols, col_bits, sort.keys[0], d_bad);
    count_launch();
    int cur = 0;
    alphasparse_status_t status = radix_sort<K>(sort, nnz, col_bits + bits_for(rows), false, &cur, st);
    if (status != ALPHA_SPARSE_STATUS_SUCCESS) return status;
    const long long work = std::max<long long>(nnz, rows + 1);
    csr_from_sorted_kernel<K><<<(unsigned)((work + 255) / 256), 256, 0, st>>>(nnz, (int)rows, col_bits, sort.keys[cur], d_ptr,
                                                                            d_col);
    count_launch();
    TRY(cudaMemsetAsync(d_ptr + rows + 1, 0, sizeof(int) * 4, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(d_col + nnz, 0, sizeof(int) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(d_val + nnz, 0, sizeof(T) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(copy_to_device_beside(d_v, v, sizeof(T) * n, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    gather_values_kernel<T><<<blocks, 256, 0, st>>>(nnz, sort.pos[cur], d_v, d_val);
    count_launch();
    unsigned long long bad = 0;
    Download back({{out_ptr, d_ptr, sizeof(int) * (size_t)(rows + 1)},
                   {out_col, d_col, sizeof(int) * n},
                   {out_val, d_val, sizeof(T) * n},
                   {&bad, d_bad, 8}},
                  st);
    TRY(back.finish(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    scratch.done(), result.done();
    if (bad) return ALPHA_SPARSE_STATUS_INVALID_VALUE;
    *out = result.b;
    result.b = DeviceBlock{};
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

template <typename T>
alphasparse_status_t coo_to_csr_device(int64_t rows, int64_t cols, int64_t nnz, const int *ri, const int *ci,
                                       const T *v, int *out_ptr, int *out_col, T *out_val, DeviceBlock *out) {
    if (bits_for(rows) + bits_for(cols) <= 32)
        return coo_to_csr_keyed<T, unsigned>(rows, cols, nnz, ri, ci, v, out_ptr, out_col, out_val, out);
    return coo_to_csr_keyed<T, unsigned long long>(rows, cols, nnz, ri, ci, v, out_ptr, out_col, out_val, out);
}

// ---- A^T from the device copy of A ------------------------------------------------------------------
//
// The reference materialises the transpose on the host with a counting sort (src/core/format/transpose_x_csr.c:7-62)
// and its transposed gemv adds the elements of a column of A in ascending row order
// (src/plain/kernel/level2/mv/gemv/gemv_x_csr_trans_plain.c:14-25).  Here the same arrays come from the device copy
// without touching the host: the stored elements, taken in storage order (rows ascending), are sorted by column
// with the stable radix sort above (32-bit keys = column, over the bits the column count uses; the payload is the
// element's position), so the elements of a column come out by ascending row; the row of each is found again by a
// binary search in the row offsets, the new offsets by a binary search in the sorted columns.
template <typename T>
__global__ void transpose_fill_kernel(long long nnz, int rows, int cols, const unsigned *__restrict__ keys,
                                      const unsigned *__restrict__ pos, const int *__restrict__ row_ptr,
                                      const T *__restrict__ val, int *__restrict__ tptr, int *__restrict__ tcol,
                                      T *__restrict__ tval) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= cols) {  // first sorted element whose column is >= i
        long long lo = 0, hi = nnz;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if ((long long)keys[mid] < i) lo = mid + 1;
            else hi = mid;
        }
        tptr[i] = (int)lo;
    }
    if (i < nnz) {
        const int k = (int)pos[i];
        int lo = 0, hi = rows;  // last row whose first element is <= k (empty rows share an offset: take the last)
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (row_ptr[mid] <= k) lo = mid;
            else hi = mid;
        }
        tcol[i] = lo;
        tval[i] = val[k];
    }
}

// Device arrays of A^T in the layout ctx_adopt expects (cols + 1 + 4 offsets, nnz + kTailPad columns and values,
// tails zeroed), allocated here and handed to the caller.
template <typename T>
alphasparse_status_t transpose_csr_device(const DeviceCtx *c, int **out_ptr, int **out_col, T **out_val) {
    cudaStream_t st = current_stream();
    const int64_t nnz = c->nnz, rows = c->rows, cols = c->cols;
    ScopedBlock scratch(st);
    int *tptr = nullptr, *tcol = nullptr;
    T *tval = nullptr;
    auto release = [&] { cudaFree(tptr), cudaFree(tcol), cudaFree(tval); };
#undef TRY
#define TRY(expr, code)                   \
    do {                                  \
        cudaError_t _e = (expr);          \
        if (_e != cudaSuccess) {          \
            record_cuda_error(_e, #expr); \
            release();                    \
            return (code);                \
        }                                 \
    } while (0)
    const size_t n = (size_t)nnz, padded = n + kTailPad;
    TRY(device_alloc(&tptr, sizeof(int) * (size_t)(cols + 1 + 4)), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(device_alloc(&tcol, sizeof(int) * padded), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(device_alloc(&tval, sizeof(T) * padded), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(cudaMemsetAsync(tptr, 0, sizeof(int) * (size_t)(cols + 1 + 4), st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(tcol + n, 0, sizeof(int) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(tval + n, 0, sizeof(T) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    if (nnz > 0) {
        Carve need(nullptr);
        (void)SortScratch<unsigned>(need, nnz);
        TRY(device_block_take(need.used, st, false, &scratch.b), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        Carve have(scratch.b.p);
        const SortScratch<unsigned> sort(have, nnz);
        TRY(cudaMemcpyAsync(sort.keys[0], c->d_col, sizeof(int) * n, cudaMemcpyDeviceToDevice, st),
            ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        int cur = 0;
        alphasparse_status_t s = radix_sort<unsigned>(sort, nnz, bits_for(cols), false, &cur, st);
        if (s != ALPHA_SPARSE_STATUS_SUCCESS) {
            release();
            return s;
        }
        const long long work = std::max<long long>(nnz, cols + 1);
        transpose_fill_kernel<T><<<(unsigned)((work + 255) / 256), 256, 0, st>>>(
            nnz, (int)rows, (int)cols, sort.keys[cur], sort.pos[cur], c->d_row_ptr, static_cast<const T *>(c->d_val), tptr, tcol,
            tval);
        count_launch();
        TRY(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    }
    TRY(cudaStreamSynchronize(st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    scratch.done();
#undef TRY
    *out_ptr = tptr, *out_col = tcol, *out_val = tval;
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

// ---- matrices derived from the device copy of A for structured descriptors -----------------------------
//
// What a SYMMETRIC / TRIANGULAR / DIAGONAL descriptor makes of the stored matrix (the reference's symv / trmv /
// diagmv and symm / trmm / diagmm kernels, src/plain/kernel/level2/mv/{symv,trmv,diagmv},
// src/plain/kernel/level3/mm/{symm,trmm,diagmm}) is an ordinary matrix: the kept triangle, its mirror image for
// SYMMETRIC, its transpose for TRIANGULAR with op = TRANSPOSE, an explicit unit diagonal, or only the diagonal.
// Every stored element emits 0, 1 or 2 (row, column) keys, an exclusive scan places them, the stable radix sort
// orders them by (row, column) -- equal pairs keep storage order -- and the values are gathered at the end.
// Payload of a key: the position of the stored element, or kUnitPayload for an explicit 1 on the diagonal.
constexpr unsigned kUnitPayload = 0xffffffffu;

struct DeriveRule {
    int type;       // ALPHA_SPARSE_MATRIX_TYPE_SYMMETRIC / TRIANGULAR / DIAGONAL
    int upper;      // kept triangle
    int unit;       // unit diagonal: stored diagonal entries are ignored
    int flip;       // TRIANGULAR under op = TRANSPOSE: (i, j) becomes (j, i)
    int diag_rule;  // DIAGONAL, rows storing their diagonal more than once: 0 first entry, 1 all, 2 last
};

__device__ __forceinline__ int derive_row_of(const int *__restrict__ row_ptr, int rows, int k) {
    int lo = 0, hi = rows;  // last row whose first element is <= k (empty rows share an offset: take the last)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (row_ptr[mid] <= k) lo = mid;
        else hi = mid;
    }
    return lo;
}

// DIAGONAL with the first / last rule: the smallest / largest position of a stored diagonal entry per row.
__global__ void derive_diag_pick_kernel(long long nnz, int rows, const int *__restrict__ row_ptr,
                                        const int *__restrict__ col, int last, int *__restrict__ pick) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnz) return;
    const int i = derive_row_of(row_ptr, rows, (int)k);
    if (col[k] != i) return;
    if (last) atomicMax(pick + i, (int)k);
    else atomicMin(pick + i, (int)k);
}

__device__ __forceinline__ unsigned derive_emits(const DeriveRule &r, int i, int j, int k, const int *__restrict__ pick) {
    if (r.type == ALPHA_SPARSE_MATRIX_TYPE_DIAGONAL) {
        if (r.unit || j != i) return 0;
        return r.diag_rule == 1 || pick[i] == k ? 1u : 0u;
    }
    const bool off = r.upper ? j > i : j < i;
    if (off) return r.type == ALPHA_SPARSE_MATRIX_TYPE_SYMMETRIC ? 2u : 1u;
    return j == i && !r.unit ? 1u : 0u;
}

__global__ void derive_count_kernel(long long nnz, int rows, const int *__restrict__ row_ptr, const int *__restrict__ col,
                                    DeriveRule rule, const int *__restrict__ pick, unsigned *__restrict__ count) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnz) return;
    const int i = derive_row_of(row_ptr, rows, (int)k);
    count[k] = derive_emits(rule, i, col[k], (int)k, pick);
}

// `offset` holds the exclusive scan of the counts; the explicit unit diagonal takes the first `rows` places.
__global__ void derive_emit_kernel(long long nnz, int rows, const int *__restrict__ row_ptr, const int *__restrict__ col,
                                   DeriveRule rule, const int *__restrict__ pick, const unsigned *__restrict__ offset,
                                   int bits, unsigned long long *__restrict__ keys, unsigned *__restrict__ pos) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned first = rule.unit ? (unsigned)rows : 0u;
    if (rule.unit && t < rows) {
        keys[t] = ((unsigned long long)(unsigned)t << bits) | (unsigned)t;
        pos[t] = kUnitPayload;
    }
    if (t >= nnz) return;
    const int k = (int)t, i = derive_row_of(row_ptr, rows, k), j = col[k];
    const unsigned n = derive_emits(rule, i, j, k, pick);
    if (n == 0) return;
    const unsigned o = first + offset[k];
    const bool flip = rule.flip && j != i;
    keys[o] = flip ? ((unsigned long long)(unsigned)j << bits) | (unsigned)i
                   : ((unsigned long long)(unsigned)i << bits) | (unsigned)j;
    pos[o] = (unsigned)k;
    if (n == 2) {
        keys[o + 1] = ((unsigned long long)(unsigned)j << bits) | (unsigned)i;
        pos[o + 1] = (unsigned)k;
    }
}

template <typename T>
__global__ void derive_fill_kernel(long long m, int rows, int bits, const unsigned long long *__restrict__ keys,
                                   const unsigned *__restrict__ pos, const T *__restrict__ val, int *__restrict__ ptr,
                                   int *__restrict__ col_out, T *__restrict__ val_out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= rows) {  // first sorted key whose row is >= i
        long long lo = 0, hi = m;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if ((long long)(keys[mid] >> bits) < i) lo = mid + 1;
            else hi = mid;
        }
        ptr[i] = (int)lo;
    }
    if (i < m) {
        col_out[i] = (int)(unsigned)(keys[i] & ((1ull << bits) - 1));
        val_out[i] = pos[i] == kUnitPayload ? T(1) : val[pos[i]];
    }
}

// Device arrays of the derived square matrix in the layout ctx_adopt expects, allocated here and handed to the
// caller with the number of stored elements.
template <typename T>
alphasparse_status_t derive_csr_device(const DeviceCtx *c, int type, int upper, int unit, int flip, int diag_rule,
                                       int **out_ptr, int **out_col, T **out_val, int64_t *out_nnz) {
    cudaStream_t st = current_stream();
    const int64_t nnz = c->nnz, rows = c->rows;
    const DeriveRule rule{type, upper, unit, flip, diag_rule};
    ScopedBlock scratch(st);
    unsigned *d_sums = nullptr, *d_count = nullptr;
    int *d_pick = nullptr, *dptr = nullptr, *dcol = nullptr;
    T *dval = nullptr;
    auto release = [&](bool all) {
        cudaFree(d_sums), cudaFree(d_count), cudaFree(d_pick);
        if (all) cudaFree(dptr), cudaFree(dcol), cudaFree(dval);
    };
#define TRY(expr, code)                   \
    do {                                  \
        cudaError_t _e = (expr);          \
        if (_e != cudaSuccess) {          \
            record_cuda_error(_e, #expr); \
            release(true);                \
            return (code);                \
        }                                 \
    } while (0)
    const unsigned eblocks = (unsigned)((std::max<int64_t>(nnz, 1) + 255) / 256);
    const bool picks = type == ALPHA_SPARSE_MATRIX_TYPE_DIAGONAL && !unit && diag_rule != 1 && nnz > 0;
    if (picks) {
        TRY(device_alloc(&d_pick, sizeof(int) * (size_t)rows), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        // bytes 0x7f.. = a large positive int for the minimum, 0xff.. = -1 for the maximum
        TRY(cudaMemsetAsync(d_pick, diag_rule == 2 ? 0xff : 0x7f, sizeof(int) * (size_t)rows, st),
            ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        derive_diag_pick_kernel<<<eblocks, 256, 0, st>>>(nnz, (int)rows, c->d_row_ptr, c->d_col, diag_rule == 2, d_pick);
        count_launch();
    }
    // how many keys every stored element emits, and where
    unsigned long long emitted = 0;
    if (nnz > 0) {
        const int scan_blocks = (int)((nnz + kScanTile - 1) / kScanTile);
        unsigned last_count = 0, last_offset = 0;
        TRY(device_alloc(&d_count, sizeof(unsigned) * (size_t)nnz), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        TRY(device_alloc(&d_sums, sizeof(unsigned) * (size_t)(scan_blocks + 1)), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        derive_count_kernel<<<eblocks, 256, 0, st>>>(nnz, (int)rows, c->d_row_ptr, c->d_col, rule, d_pick, d_count);
        count_launch();
        TRY(cudaMemcpyAsync(&last_count, d_count + nnz - 1, 4, cudaMemcpyDeviceToHost, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        alphasparse_status_t s = device_exclusive_scan(d_count, nnz, d_sums, st);
        if (s != ALPHA_SPARSE_STATUS_SUCCESS) {
            release(true);
            return s;
        }
        TRY(cudaMemcpyAsync(&last_offset, d_count + nnz - 1, 4, cudaMemcpyDeviceToHost, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        TRY(cudaStreamSynchronize(st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
        emitted = (unsigned long long)last_offset + last_count;  // at most 2 * nnz < 2^32: the 32-bit scan is exact
        cudaFree(d_sums), d_sums = nullptr;
    }
    // 32-bit offsets, as for every handle; a symmetric matrix may double its stored elements
    if (emitted + (unit ? (unsigned long long)rows : 0ull) > (unsigned long long)(INT32_MAX - 64)) {
        release(true);
        record_error("the matrix derived for this descriptor would hold more than 2^31 - 65 elements");
        return ALPHA_SPARSE_STATUS_NOT_SUPPORTED;
    }
    const int64_t m = (int64_t)emitted + (unit ? rows : 0);
    const size_t n = (size_t)m, padded = n + kTailPad;
    TRY(device_alloc(&dptr, sizeof(int) * (size_t)(rows + 1 + 4)), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(device_alloc(&dcol, sizeof(int) * padded), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(device_alloc(&dval, sizeof(T) * padded), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
    TRY(cudaMemsetAsync(dptr, 0, sizeof(int) * (size_t)(rows + 1 + 4), st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(dcol + n, 0, sizeof(int) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    TRY(cudaMemsetAsync(dval + n, 0, sizeof(T) * kTailPad, st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    if (m > 0) {
        Carve need(nullptr);
        (void)SortScratch<unsigned long long>(need, m);
        TRY(device_block_take(need.used, st, false, &scratch.b), ALPHA_SPARSE_STATUS_ALLOC_FAILED);
        Carve have(scratch.b.p);
        const SortScratch<unsigned long long> sort(have, m);
        const int bits = bits_for(rows);  // square: rows == cols
        const long long work = std::max<long long>(nnz, unit ? rows : 0);
        derive_emit_kernel<<<(unsigned)((work + 255) / 256), 256, 0, st>>>(nnz, (int)rows, c->d_row_ptr, c->d_col, rule,
                                                                          d_pick, d_count, bits, sort.keys[0], sort.pos[0]);
        count_launch();
        int cur = 0;
        alphasparse_status_t s = radix_sort<unsigned long long>(sort, m, 2 * bits, true, &cur, st);
        if (s != ALPHA_SPARSE_STATUS_SUCCESS) {
            release(true);
            return s;
        }
        const long long fill = std::max<long long>(m, rows + 1);
        derive_fill_kernel<T><<<(unsigned)((fill + 255) / 256), 256, 0, st>>>(
            m, (int)rows, bits, sort.keys[cur], sort.pos[cur], static_cast<const T *>(c->d_val), dptr, dcol, dval);
        count_launch();
        TRY(cudaGetLastError(), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    }
    TRY(cudaStreamSynchronize(st), ALPHA_SPARSE_STATUS_EXECUTION_FAILED);
    scratch.done();
#undef TRY
    release(false);
    *out_ptr = dptr, *out_col = dcol, *out_val = dval, *out_nnz = m;
    return ALPHA_SPARSE_STATUS_SUCCESS;
}

template alphasparse_status_t derive_csr_device<float>(const DeviceCtx *, int, int, int, int, int, int **, int **, float **,
                                                       int64_t *);
template alphasparse_status_t derive_csr_device<double>(const DeviceCtx *, int, int, int, int, int, int **, int **, double **,
                                                        int64_t *);

template alphasparse_status_t transpose_csr_device<float>(const DeviceCtx *, int **, int **, float **);
template alphasparse_status_t transpose_csr_device<double>(const DeviceCtx *, int **, int **, double **);

template alphasparse_status_t coo_to_csr_device<float>(int64_t, int64_t, int64_t, const int *, const int *,
                                                       const float *, int *, int *, float *, DeviceBlock *);
template alphasparse_status_t coo_to_csr_device<double>(int64_t, int64_t, int64_t, const int *, const int *,
                                                        const double *, int *, int *, double *, DeviceBlock *);

}  // namespace asb
