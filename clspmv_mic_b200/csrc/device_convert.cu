// device_convert.cu — COO -> format converters that run on the device.
//
// clspmv_device_coo2<fmt>_f32 takes a COO whose arrays are in device memory
// and writes a device copy of the format struct holding, array for array and
// byte for byte, what the host converter clspmv_coo2<fmt>_f32 (the templates
// of matrix_storage.h, restating include/matrix_storage.h:936-2409 of
// clSpMV) makes from the same COO, with the same statuses: the same argument
// checks, the same refusals, and CLSPMV_ERR_NOT_SORTED where the host
// converter wants a (row, col)-sorted COO (every format but DIA / BDIA, which
// keep the last value of a repeated (row, col) in COO order).
// clspmv_device_sort_coo_f32 sorts a device COO in place, stably, as
// clspmv_sort_coo_f32 does on the host.
//
// Output arrays come from device_alloc and are released with
// clspmv_device_free_<fmt> (an empty array still gets an allocation, so no
// pointer is NULL after a success). Every call synchronises `stream`: sizes
// are read back to size the outputs, once per call where the format allows.
//
// The work is integer index arithmetic over the COO, bound by HBM. One pass
// (k_front) checks ids and order, builds the row pointer, and makes CSR's
// copies or marks the diagonals on the way. Each padded layout is then
// written once, every byte of it coalesced: ELL and SELL by quads of rows,
// DIA by rows whose entries are staged in shared memory, whole or by windows, and the 4-wide block
// formats by merging the sorted rows of a block row (k_blocks), without
// sorting. Entries a row holds twice keep the last value in COO order, as in
// the host loops. The generic BCSR / BELL of any block shape group their
// entries by a stable radix sort (CUB) on (block row, block column).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "api_internal.h"
#include "clspmv_b200.h"

using clspmv::cuda_status;

namespace {

constexpr int kT = 256;

int grid_for(long long n)
{
    const long long b = (n + kT - 1) / kT;
    return (int)std::max(1LL, std::min(b, 148LL * 32));
}

#define GRID_STRIDE(i, n) \
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

long long aligned_len(long long n, long long a) { return n % a == 0 ? n : n + (a - n % a); }

int bits_for(long long n)   // bits of the largest value in [0, n)
{
    int b = 0;
    while (b < 62 && (1LL << b) < n) b++;
    return b;
}

// Device arrays of one call on one stream, released at scope exit unless kept.
struct Allocs {
    cudaStream_t st;
    std::vector<void*> ptrs;
    int rc = CLSPMV_OK;
    bool keep = false;
    explicit Allocs(cudaStream_t s) : st(s) {}
    template <class T>
    T* get(size_t n)
    {
        if (rc) return nullptr;
        void* p = nullptr;
        if ((rc = clspmv::device_alloc(&p, std::max<size_t>(n, 1) * sizeof(T)))) return nullptr;
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    ~Allocs()
    {
        if (keep || ptrs.empty()) return;
        const bool idle = cudaStreamSynchronize(st) == cudaSuccess;   // the arrays were used on `st` alone
        int idle_on = idle ? clspmv::kIdleAll : clspmv::kIdleNone;
        for (void* p : ptrs) idle_on = clspmv::device_release(p, idle_on);
    }
};

template <class T>
int read_back(const T* dev, T* host, cudaStream_t st)
{
    int rc = cuda_status(cudaMemcpyAsync(host, dev, sizeof(T), cudaMemcpyDeviceToHost, st));
    if (!rc) rc = cuda_status(cudaStreamSynchronize(st));
    return rc;
}

int launched(cudaStream_t st, int n = 1)
{
    (void)st;
    return clspmv::after_launch(n);
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// What one conversion reads back from the device.
struct Info {
    int flags;         // bit 0: a neighbour pair is out of (row, col) order; 1: an id is outside the matrix; 2: a row is at or past `len`
    int most;          // longest row / block row
    long long total;   // slots, blocks or diagonals
    int small, big;    // entries of the gap lists
    int pad[2];
};
constexpr int kBad = 3;

__device__ __forceinline__ bool bad_input(const Info* info) { return __ldcg(&info->flags) & kBad; }

// Runs of rows without entries: k_front writes runs of up to kGap row
// pointers itself and lists the others, up to kBigGap rows for one warp of
// k_gaps, longer ones for all of its grid.
constexpr int kGap = 32, kBigGap = 4096;
struct GapLists {
    int4* small;   // (first row, end row, value)
    int4* big;
    int nsmall, nbig;
};

__device__ __noinline__ void fill_gap(int* rp, int r0, int r1, int v, const GapLists& gl, Info* info)   // rp[r0 .. r1) = v
{
    if (r1 - r0 <= kGap) {
        for (int r = r0; r < r1; r++) rp[r] = v;
    } else if (r1 - r0 <= kBigGap) {
        const int at = atomicAdd(&info->small, 1);
        if (at < gl.nsmall) gl.small[at] = make_int4(r0, r1, v, 0);
    } else {
        const int at = atomicAdd(&info->big, 1);
        if (at < gl.nbig) gl.big[at] = make_int4(r0, r1, v, 0);
    }
}

// One pass over the COO, 4 consecutive entries per lane (128-bit loads with
// VEC): id range and order into info->flags, row pointer rp[r] = first entry
// of a row >= r (r in [0, h]) where rp is given, CSR's copies (COPY), the bit
// of every diagonal that holds an entry (MARK) and whether a row is at or
// past `lim`. Bound by HBM with the row pointer's part confined to lanes whose
// 4 entries start a row (instruction bound at 173 us without that): 64M
// entries in 88 us on B200 (5.8 TB/s), where a check of one entry per thread
// took 142 us and the search of each block row's start another 20 us.
template <bool VEC, bool COPY, bool MARK>
__global__ void __launch_bounds__(kT) k_front(const int* __restrict__ row, const int* __restrict__ col,
                                              const float* __restrict__ val, long long n, int h, int w, int* rp,
                                              GapLists gl, int* ocol, float* oval, unsigned* mark, int lim, Info* info)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * (kT / 32);
    bool unsorted = false, outside = false, past = false;
    for (long long base = ((long long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5)) * 128; base < n; base += nwarps * 128) {
        const long long i0 = base + lane * 4;
        int pr0 = -1, pc0 = -1;
        if (lane == 0 && base > 0) {
            pr0 = __ldg(row + base - 1);
            pc0 = __ldg(col + base - 1);
        }
        int r[4], c[4];
        int m = 4;   // entries of this lane
        if (VEC && i0 + 3 < n) {
            const int4 rv = __ldg(reinterpret_cast<const int4*>(row + i0)), cv = __ldg(reinterpret_cast<const int4*>(col + i0));
            r[0] = rv.x; r[1] = rv.y; r[2] = rv.z; r[3] = rv.w;
            c[0] = cv.x; c[1] = cv.y; c[2] = cv.z; c[3] = cv.w;
            if (COPY) {
                *reinterpret_cast<int4*>(ocol + i0) = cv;
                *reinterpret_cast<float4*>(oval + i0) = __ldg(reinterpret_cast<const float4*>(val + i0));
            }
        } else {   // past the end: the last entry again, which breaks no order and starts no row
            m = (int)max(0LL, min(4LL, n - i0));
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const long long i = min(i0 + j, n - 1);
                r[j] = __ldg(row + i);
                c[j] = __ldg(col + i);
                if (COPY && j < m) {
                    ocol[i] = c[j];
                    oval[i] = __ldg(val + i);
                }
            }
        }
        int pr = __shfl_up_sync(0xffffffffu, r[3], 1), pc = __shfl_up_sync(0xffffffffu, c[3], 1);
        if (lane == 0) {
            pr = pr0;
            pc = pc0;
        }
        // 64-bit keys compare rows, then columns (ids past the sign bit are outside anyway)
        unsigned long long k = pr < 0 ? 0 : ((unsigned long long)(unsigned)pr << 32) | (unsigned)pc;
        bool in = pr >= -1 && pr < h;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            in = in && (unsigned)r[j] < (unsigned)h && (unsigned)c[j] < (unsigned)w;
            const unsigned long long kj = ((unsigned long long)(unsigned)r[j] << 32) | (unsigned)c[j];
            unsorted = unsorted || k > kj;
            k = kj;
        }
        outside = outside || !in;
        past = past || max(max(r[0], r[1]), max(r[2], r[3])) >= lim;
        if (rp && in && !unsorted && r[3] != pr) {   // no row pointer of an unsorted COO is used
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = (int)(i0 + j);
                if (r[j] == pr + 1) rp[r[j]] = i;
                else if (r[j] > pr) fill_gap(rp, pr + 1, r[j] + 1, i, gl, info);
                pr = r[j];
            }
        }
        if (MARK && in) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const long long p = (long long)c[j] - r[j] + h - 1;
                const unsigned bit = 1u << (p & 31);
                if (!(__ldcg(mark + (p >> 5)) & bit)) atomicOr(mark + (p >> 5), bit);
            }
        }
    }
    if (rp && blockIdx.x == 0 && threadIdx.x == 0) {   // rows after the last entry
        const int last = __ldg(row + n - 1);
        if (last >= 0 && last < h) fill_gap(rp, last + 1, h + 1, (int)n, gl, info);
    }
    const int f = __reduce_or_sync(0xffffffffu, (unsorted ? 1 : 0) | (outside ? 2 : 0) | (past ? 4 : 0));
    if (lane == 0 && f) atomicOr(&info->flags, f);
}

// An unsorted COO lists runs that overlap, of up to all rows each: they are
// not filled (1M entries over 20M rows: 21 ms).
__global__ void __launch_bounds__(kT) k_gaps(int* rp, GapLists gl, const Info* info)
{
    if (bad_input(info)) return;
    const int lane = threadIdx.x & 31;
    const int ns = min(info->small, gl.nsmall), nb = min(info->big, gl.nbig);
    for (int g = blockIdx.x * (kT / 32) + (threadIdx.x >> 5); g < ns; g += gridDim.x * (kT / 32)) {
        const int4 v = gl.small[g];
        for (int r = v.x + lane; r < v.y; r += 32) rp[r] = v.z;
    }
    for (int g = 0; g < nb; g++) {
        const int4 v = gl.big[g];
        for (long long r = v.x + (long long)blockIdx.x * kT + threadIdx.x; r < v.y; r += (long long)gridDim.x * kT) rp[r] = v.z;
    }
}

__global__ void k_coo_keys(const int* __restrict__ row, const int* __restrict__ col, long long n, int colbits,
                           unsigned long long* keys, int* idx)
{
    GRID_STRIDE(i, n)
    {
        keys[i] = ((unsigned long long)(unsigned)row[i] << colbits) | (unsigned)col[i];
        idx[i] = (int)i;
    }
}

__global__ void k_block_keys(const int* __restrict__ row, const int* __restrict__ col, long long n, int bw, int bh,
                             int colbits, unsigned long long* keys, int* idx)
{
    GRID_STRIDE(i, n)
    {
        keys[i] = ((unsigned long long)(unsigned)(row[i] / bh) << colbits) | (unsigned)(col[i] / bw);
        idx[i] = (int)i;
    }
}

template <class T>
__global__ void k_gather(const int* __restrict__ idx, const T* __restrict__ src, long long n, T* dst)
{
    GRID_STRIDE(i, n) dst[i] = src[idx[i]];
}

// rp[r] = first position whose sorted id is >= r, for r in [0, nrows].
__global__ void k_lower_bounds(const int* __restrict__ ids, long long n, int nrows, int* rp)
{
    GRID_STRIDE(r, (long long)nrows + 1)
    {
        long long lo = 0, hi = n;
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (ids[mid] < r) lo = mid + 1;
            else hi = mid;
        }
        rp[r] = (int)lo;
    }
}

__global__ void k_max_len(const int* __restrict__ rp, int nrows, int* out, const Info* info)
{
    if (info && bad_input(info)) return;
    int m = 0;
    GRID_STRIDE(r, nrows) m = max(m, rp[r + 1] - rp[r]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m > __ldcg(out)) atomicMax(out, m);
}

// wsh[s] = (longest row of slice s) * sh; wsh[ns] = 0.
__global__ void k_slice_slots(const int* __restrict__ rp, int nrows, int sh, int ns, long long* wsh, const Info* info)
{
    if (bad_input(info)) return;   // rp is unfinished
    GRID_STRIDE(s, (long long)ns + 1)
    {
        int m = 0;
        if (s < ns) {
            const long long r1 = min((long long)nrows, (s + 1) * (long long)sh);
            for (long long r = s * (long long)sh; r < r1; r++) m = max(m, rp[r + 1] - rp[r]);
        }
        wsh[s] = (long long)m * sh;
    }
}

__global__ void k_to_int(const long long* __restrict__ a, long long n, int* b, Info* info)
{
    GRID_STRIDE(i, n)
    {
        b[i] = (int)a[i];
        if (i == n - 1) info->total = a[i];
    }
}

// Largest s in [0, ns) with ptr[s] <= t: the slice holding slot t (a
// zero-width slice shares its start with the next one and is never chosen).
__device__ __forceinline__ int slice_of(const int* __restrict__ ptr, int ns, long long t)
{
    int lo = 0, hi = ns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((long long)ptr[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ELL slot (k, r) = t: entry k of row r, else the row's last column (0 for
// an empty row) with value 0; rows past the height are all zero
// (include/matrix_storage.h:1385-1389).
__global__ void k_ell_fill(const int* __restrict__ rp, const int* __restrict__ col, const float* __restrict__ val,
                           int h, long long len, long long total, int* ocol, float* oval)
{
    GRID_STRIDE(t, total)
    {
        const long long k = t / len, r = t - k * len;
        int c = 0;
        float v = 0.f;
        if (r < h) {
            const int a = rp[r], b = rp[r + 1];
            if (k < b - a) {
                c = col[a + k];
                v = val[a + k];
            } else if (b > a) {
                c = col[b - 1];
            }
        }
        ocol[t] = c;
        oval[t] = v;
    }
}

// SELL slot t: entry k of row r of its slice, else padding that copies the
// slot to its left (the row's last column), and for an empty row (or a row
// past the height) slot 0 of the slice, itself 0 when the slice's first row
// is empty (include/matrix_storage.h:1466-1496).
__global__ void k_sell_fill(const int* __restrict__ ptr, int ns, const int* __restrict__ rp,
                            const int* __restrict__ col, const float* __restrict__ val, int h, int sh, long long total,
                            int* ocol, float* oval)
{
    GRID_STRIDE(t, total)
    {
        const int s = slice_of(ptr, ns, t);
        const long long off = t - ptr[s];
        const long long k = off / sh;
        const long long r = (long long)s * sh + (off - k * sh);
        int c;
        float v = 0.f;
        const int a = r < h ? rp[r] : 0, b = r < h ? rp[r + 1] : 0;
        if (k < b - a) {
            c = col[a + k];
            v = val[a + k];
        } else if (b > a) {
            c = col[b - 1];
        } else {
            const long long r0 = (long long)s * sh;
            c = rp[r0 + 1] > rp[r0] ? col[rp[r0]] : 0;
        }
        ocol[t] = c;
        oval[t] = v;
    }
}

// The 4 rows row0 .. row0+3 of one lane of the quad fills: first entry,
// length, padding column.
struct Quad {
    int a[4], n[4], pad[4];
    __device__ void load(const int* __restrict__ rp, const int* __restrict__ col, long long row0, int h, int empty)
    {
        int e[5];
#pragma unroll
        for (int i = 0; i < 5; i++) e[i] = row0 + i <= h ? __ldg(rp + row0 + i) : 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            a[i] = e[i];
            n[i] = row0 + i < h ? e[i + 1] - e[i] : 0;
            pad[i] = n[i] > 0 ? __ldg(col + e[i + 1] - 1) : empty;
        }
    }
    // slot column k of the 4 rows, at dst (a multiple of 4)
    __device__ void store(const int* __restrict__ col, const float* __restrict__ val, int k, size_t dst, int* ocol, float* oval) const
    {
        int c[4];
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            c[i] = k < n[i] ? __ldg(col + a[i] + k) : pad[i];
            v[i] = k < n[i] ? __ldg(val + a[i] + k) : 0.f;
        }
        *reinterpret_cast<int4*>(ocol + dst) = make_int4(c[0], c[1], c[2], c[3]);
        *reinterpret_cast<float4*>(oval + dst) = make_float4(v[0], v[1], v[2], v[3]);
    }
};

// Slot columns per warp of the quad fills: one search or row setup per run,
// while one wide slice is still shared between warps.
constexpr int kFillCols = 64;

// SELL with slice heights of 4 Q rows: a lane writes 4 rows of a slot column
// with one 128-bit store per array, Q lanes a column, 32 / Q columns a warp
// step. Warps take equal runs of the columns of all slices, so the slice is
// searched once per run and a row's entries are read from consecutive words:
// 0.286 ms (4.9 TB/s) for the 160M slots of the power-law matrix of 700k rows
// on B200, against 2.86 ms for k_sell_fill, which searches once per slot.
// Other slice heights keep that kernel.
template <int Q>
__global__ void __launch_bounds__(kT) k_sell_fill_quads(const int* __restrict__ ptr, int ns, const int* __restrict__ rp,
                                                        const int* __restrict__ col, const float* __restrict__ val, int h,
                                                        long long cols, int* ocol, float* oval)
{
    constexpr int sh = 4 * Q, G = 32 / Q;
    const int lane = threadIdx.x & 31, g = lane / Q, q = lane % Q;
    const long long nwarps = (long long)gridDim.x * (kT / 32);
    for (long long c0 = ((long long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5)) * kFillCols; c0 < cols; c0 += nwarps * kFillCols) {
        const long long c1 = min(c0 + kFillCols, cols);
        long long c = c0;
        int s = slice_of(ptr, ns, c * sh);
        while (c < c1) {
            const long long sb = ptr[s] / sh, se = ptr[s + 1] / sh;
            if (se <= c) {   // slices without columns
                s = slice_of(ptr, ns, c * sh);
                continue;
            }
            const long long ce = min(c1, se), r0 = (long long)s * sh;
            const int first = __ldg(rp + r0), next = __ldg(rp + r0 + 1);
            Quad qd;
            qd.load(rp, col, r0 + 4 * q, h, next > first ? __ldg(col + first) : 0);
#pragma unroll 2
            for (long long cc = c + g; cc < ce; cc += G) qd.store(col, val, (int)(cc - sb), (size_t)cc * sh + 4 * q, ocol, oval);
            c = ce;
            s++;
        }
    }
}

// ELL (len a multiple of 4) the same way: a warp takes 32 rows and
// kFillCols slot columns.
__global__ void __launch_bounds__(kT) k_ell_fill_quads(const int* __restrict__ rp, const int* __restrict__ col,
                                                       const float* __restrict__ val, int h, long long len, int num,
                                                       int* ocol, float* oval)
{
    const int lane = threadIdx.x & 31, g = lane >> 3, q = lane & 7;
    const long long groups = (len + 31) / 32, runs = (num + kFillCols - 1) / kFillCols;
    const long long nwarps = (long long)gridDim.x * (kT / 32);
    for (long long t = (long long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5); t < groups * runs; t += nwarps) {
        const long long run = t / groups, row0 = (t - run * groups) * 32 + 4 * q;
        if (row0 >= len) continue;
        Quad qd;
        qd.load(rp, col, row0, h, 0);
        const int k1 = (int)min((long long)num, (run + 1) * kFillCols);
#pragma unroll 2
        for (int k = (int)run * kFillCols + g; k < k1; k += 4) qd.store(col, val, k, (size_t)k * len + row0, ocol, oval);
    }
}

// Columns (and values) of a contiguous COO range, copied by a warp into its
// part of shared memory with one word of skew per 32, so that lanes walking
// rows of equal length meet different banks. The copies are asynchronous:
// the whole range is in flight at once.
__device__ __forceinline__ int skewed(int i) { return i + (i >> 5); }
__device__ __forceinline__ void copy_word(void* dst, const void* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}
struct InSmem {    // entry p of the range staged from lo on
    const int* cols;
    const float* vals;
    int lo;
    __device__ int at(int p) const { return skewed(p - lo); }
    __device__ int col(int i) const { return cols[i]; }
    __device__ float val(int i) const { return vals[i]; }
};
struct InPlace {
    const int* __restrict__ cols;
    const float* __restrict__ vals;
    __device__ int at(int p) const { return p; }
    __device__ int col(int i) const { return __ldg(cols + i); }
    __device__ float val(int i) const { return __ldg(vals + i); }
};
template <bool VALS>
__device__ __forceinline__ InSmem stage(const int* __restrict__ col, const float* __restrict__ val, int lo, int hi, int cap, int* smem)
{
    float* sv = reinterpret_cast<float*>(smem + skewed(cap));
    __syncwarp();   // the last range has been read
#pragma unroll 4
    for (int i = threadIdx.x & 31; i < hi - lo; i += 32) {
        copy_word(smem + skewed(i), col + lo + i);
        if (VALS) copy_word(sv + skewed(i), val + lo + i);
    }
    copies_done();
    return InSmem{smem, sv, lo};
}

// Diagonals of the marked bits: their number into info->total, the offsets.
__global__ void k_mark_counts(const unsigned* __restrict__ mark, long long words, int* cnt)
{
    GRID_STRIDE(i, words + 1) cnt[i] = i < words ? __popc(mark[i]) : 0;
}
__global__ void k_publish(const int* src, Info* info) { info->total = *src; }
__device__ __forceinline__ long long diag_rank(const unsigned* __restrict__ mark, const int* __restrict__ first, long long p)
{
    return first[p >> 5] + __popc(mark[p >> 5] & ((1u << (p & 31)) - 1));
}
__global__ void k_dia_offsets(const unsigned* __restrict__ mark, const int* __restrict__ first, long long words, int h, int* off)
{
    GRID_STRIDE(i, words)
    {
        int at = first[i];
        for (unsigned m = mark[i]; m; m &= m - 1) off[at++] = (int)(i * 32 + (__ffs(m) - 1) - (h - 1));
    }
}

// Sorted input, DIA: a lane walks its row's entries along the diagonals,
// whose offsets ascend as the row's columns do, and writes a slot of every
// diagonal (zero where the row has none there), so a warp stores 32
// consecutive slots at a time and no slot is cleared first. Its 32 rows are
// one contiguous range of the COO, staged in shared memory. The scatter by
// entries it replaces cleared the array and wrote one sector per entry.
// A repeated (row, col) keeps its last value.
constexpr int kRowWarps = 4;   // warps per CTA of the staged kernels

template <class E>
__device__ __forceinline__ void dia_row(const E& x, int p, int e, long long r, long long len, const int* __restrict__ off, int nd,
                                        float* out)
{
    // INT_MIN is below every r + off
    int i = p < e ? x.at(p) : 0;
    int c = p < e ? x.col(i) : INT_MIN;
    for (int d = 0; d < nd; d++, out += len) {
        const long long want = r + __ldg(off + d);
        float v = 0.f;
        while (c == want) {
            v = x.val(i);
            p++;
            i = p < e ? x.at(p) : 0;
            c = p < e ? x.col(i) : INT_MIN;
        }
        if (r < len) *out = v;
    }
}

// The same for 32 rows of more entries than are staged at once: each lane has a
// window of up to W entries of its row, filled by the whole warp from
// consecutive words when it is used up, which rows of a band are at the same
// diagonal. Rows walked in place, a lane each, took longer than the scatter by
// entries (100k rows of 301 diagonals 2.38 against 2.05 ms in all, 10k of 3,001 3.64
// against 1.89; here 0.64 and 1.18).
__device__ __forceinline__ void dia_rows_by_windows(const int* __restrict__ col, const float* __restrict__ val, int p, int e,
                                                    long long r, long long len, const int* __restrict__ off, int nd, int W,
                                                    int* smem, float* out)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, stride = W + 1;   // lanes at the same place of their windows meet different banks
    int* const cols = smem + lane * stride;
    float* const vals = reinterpret_cast<float*>(smem + 32 * stride) + lane * stride;
    int at = 0, have = 0, c = INT_MIN;   // place in the window, its entries, the column there (INT_MIN is below every r + off)
    auto refill = [&]() {                // p: first entry past the window
        if (!__any_sync(kAll, at == have && p < e)) return false;
        // with the lanes that have used half of theirs, or rows that start a diagonal apart would wait for one each
        const unsigned need = __ballot_sync(kAll, 2 * at >= have && p < e);
        if (need >> lane & 1) p -= have - at;
        __syncwarp();   // the windows have been read
        for (unsigned m = need; m; m &= m - 1) {
            const int l = __ffs(m) - 1, q = __shfl_sync(kAll, p, l), n = __shfl_sync(kAll, e, l) - q;
            if (lane < min(n, W)) {
                copy_word(smem + l * stride + lane, col + q + lane);
                copy_word(smem + (32 + l) * stride + lane, val + q + lane);
            }
        }
        copies_done();
        if (need >> lane & 1) {
            have = min(e - p, W);
            p += have;
            at = 0;
            c = cols[0];
        }
        return true;
    };
    refill();
    for (int d = 0; d < nd; d++, out += len) {
        const long long want = r + __ldg(off + d);
        float v = 0.f;
        do {
            while (c == want) {
                v = vals[at++];
                c = at < have ? cols[at] : INT_MIN;
            }
        } while (refill());
        if (r < len) *out = v;
    }
}

__global__ void __launch_bounds__(kRowWarps * 32) k_dia_rows(const int* __restrict__ rp, const int* __restrict__ col,
                                                             const float* __restrict__ val, int h, long long len,
                                                             const int* __restrict__ off, int nd, int cap, float* data)
{
    extern __shared__ int dsm[];
    int* smem = dsm + (threadIdx.x >> 5) * 2 * skewed(cap);
    const int lane = threadIdx.x & 31, window = min(32, 2 * skewed(cap) / 64 - 1);   // 32 from 1,024 entries on, 3 of the least
    const long long nwarps = (long long)gridDim.x * kRowWarps;
    for (long long r0 = ((long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5)) * 32; r0 < len; r0 += nwarps * 32) {
        const long long r = r0 + lane;
        const int p = __ldg(rp + min(r, (long long)h)), e = __ldg(rp + min(r + 1, (long long)h));
        const int lo = __shfl_sync(0xffffffffu, p, 0), hi = __shfl_sync(0xffffffffu, e, 31);
        if (hi - lo <= cap) dia_row(stage<true>(col, val, lo, hi, cap, smem), p, e, r, len, off, nd, data + r);
        else if (window >= 8) dia_rows_by_windows(col, val, p, e, r, len, off, nd, window, smem, data + r);
        else dia_row(InPlace{col, val}, p, e, r, len, off, nd, data + r);
    }
}

// Unsorted input: each slot keeps the value of its highest COO position.
__global__ void k_dia_claim(const int* __restrict__ row, const int* __restrict__ col, long long n, int h,
                            const unsigned* __restrict__ mark, const int* __restrict__ first, long long len, int* owner)
{
    GRID_STRIDE(i, n)
    {
        const int r = row[i], c = col[i];
        atomicMax(owner + diag_rank(mark, first, (long long)c - r + h - 1) * len + r, (int)i);
    }
}

__global__ void k_dia_scatter_owned(const int* __restrict__ row, const int* __restrict__ col,
                                    const float* __restrict__ val, long long n, int h, const unsigned* __restrict__ mark,
                                    const int* __restrict__ first, long long len, const int* __restrict__ owner, float* data)
{
    GRID_STRIDE(i, n)
    {
        const int r = row[i], c = col[i];
        const long long slot = diag_rank(mark, first, (long long)c - r + h - 1) * len + r;
        if (owner[slot] == (int)i) data[slot] = val[i];
    }
}

__global__ void k_block_heads(const unsigned long long* __restrict__ keys, long long n, int* head)
{
    GRID_STRIDE(i, n) head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// For each block (in (block row, block column) order): its block row and
// block column.
__global__ void k_block_list(const unsigned long long* __restrict__ keys, const int* __restrict__ head,
                             const int* __restrict__ bid, long long n, int colbits, int* brow, int* bcol)
{
    GRID_STRIDE(i, n)
    if (head[i]) {
        const int b = bid[i] - 1;
        brow[b] = (int)(keys[i] >> colbits);
        bcol[b] = (int)(keys[i] & ((1ULL << colbits) - 1));
    }
}

// col_id of block b: its first column
__global__ void k_bcsr_colid(const int* __restrict__ bcol, long long nb, int bw, int* out)
{
    GRID_STRIDE(b, nb) out[b] = bcol[b] * bw;
}

// Block formats: where an entry of block b lands. inner row hh, column
// w4 * 4 + w of the block.
struct BcsrPlace {    // data[k*len + b], k = inner row * bw + inner column (include/matrix_storage.h:1728)
    long long len;
    int bw;
    __device__ long long operator()(int, int, long long b, int hh, int w4, int w) const
    {
        return ((long long)hh * bw + w4 * 4 + w) * len + b;
    }
};
struct BellPlace {    // data[r + k*len + j*colsz] (include/matrix_storage.h:1992)
    long long len, colsz;
    int bw;
    __device__ long long operator()(int r, int j, long long, int hh, int w4, int w) const
    {
        return (long long)r + ((long long)hh * bw + w4 * 4 + w) * len + j * colsz;
    }
};
template <class Place>
__global__ void k_block_scatter(const int* __restrict__ idx, const int* __restrict__ bid, const int* __restrict__ row,
                                const int* __restrict__ col, const float* __restrict__ val, long long n, int bw, int bh,
                                const int* __restrict__ brow, const int* __restrict__ bcol, const int* __restrict__ brp,
                                Place place, float* data)
{
    GRID_STRIDE(i, n)
    {
        const int e = idx[i];
        const int r = row[e], c = col[e];
        if (i + 1 < n) {
            const int e2 = idx[i + 1];
            if (row[e2] == r && col[e2] == c) continue;
        }
        const long long b = bid[i] - 1;
        const int br = brow[b];
        const int cc = c - bcol[b] * bw;
        data[place(br, (int)(b - brp[br]), b, r % bh, cc >> 2, cc & 3)] = val[e];
    }
}

// bell col ids, slot (j, r): the first column of block j of block row r,
// else the row's last (0 for an empty or missing row).
__global__ void k_bell_cols(const int* __restrict__ brp, const int* __restrict__ bcol, int nbr, int bw, long long len,
                            long long total, int* out)
{
    GRID_STRIDE(t, total)
    {
        const long long j = t / len, r = t - j * len;
        int c = 0;
        if (r < nbr) {
            const int a = brp[r], e = brp[r + 1];
            if (j < e - a) c = bcol[a + j] * bw;
            else if (e > a) c = bcol[e - 1] * bw;
        }
        out[t] = c;
    }
}

// ---------------------------------------------------------------------------
// The 4-wide block formats (BW in {4, 8}, BH in {1, 2, 4, 8}). The rows of a
// sorted COO are sorted by column, so the blocks of a block row are a merge
// of its BH rows: BH lanes hold one row each, the least block column among
// the lanes' next entries is the next block, and every lane takes its
// entries of that block. A warp merges 32 / BH block rows side by side, whose
// 32 rows are one contiguous range of the COO, staged in shared memory. One
// pass counts the blocks, a second writes them, each lane its row's 4 values
// per strip with one 128-bit store. Block rows of more than kItemNnz entries are cut into
// items of about that many, at block columns of their longest row, so that
// one long row does not keep a warp to itself.
//
// Against sorting all entries by (block row, block column) with 64-bit keys
// (five radix passes, 3.6 ms for 64M entries, after 0.5 ms of keys, heads and
// scans and before a 0.6 ms scatter): the two passes read 4 and 8 bytes per
// entry and write the result, in 68 and 194 us for the 4x4 SBELL of 64M
// entries on B200 (3.8 and 4.0 TB/s; instructions of the merge bound both).
// The conversion's kernels went from 5.2 to 0.43 ms.
// ---------------------------------------------------------------------------
constexpr int kItemNnz = 512;

__global__ void k_item_counts(const int* __restrict__ rp, int h, int bh, int nbr, int item_nnz, int* cnt, const Info* info)
{
    if (bad_input(info)) return;
    GRID_STRIDE(b, (long long)nbr + 1)
    {
        const long long n = b < nbr ? rp[min((long long)h, (b + 1) * bh)] - rp[b * bh] : 0;
        cnt[b] = b < nbr ? (int)max(1LL, (n + item_nnz - 1) / item_nnz) : 0;
    }
}

__global__ void k_item_rows(const int* __restrict__ first, int nbr, int* brow, const Info* info)
{
    if (bad_input(info)) return;
    GRID_STRIDE(b, nbr)
    for (int i = first[b]; i < first[b + 1]; i++) brow[i] = (int)b;
}

// brp[b] = blocks before block row b; the longest block row and the number of blocks into info.
__global__ void k_block_ptr(const int* __restrict__ first, const int* __restrict__ before, int nbr, int* brp, Info* info)
{
    if (bad_input(info)) return;
    int m = 0;
    GRID_STRIDE(b, (long long)nbr + 1)
    {
        const int v = before[first[b]];
        brp[b] = v;
        if (b < nbr) m = max(m, before[first[b + 1]] - v);
        else info->total = v;
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m > __ldcg(&info->most)) atomicMax(&info->most, m);
}

struct BlockJob {
    const int* rp;      // row pointer, h + 1
    const int* col;
    const float* val;
    int h, nbr;
    const int* first;   // first item of each block row, nbr + 1
    const int* brow;    // block row of each item
    int cap;            // entries staged per warp
    const Info* info;
    int* count;         // counting pass: blocks per item
    const int* before;  // writing pass: blocks before each item
    const int* brp;     // blocks before each block row
};

// First entry of row [p, e) whose column is at or past c.
__device__ __forceinline__ int lower_col(const int* __restrict__ col, int p, int e, long long c)
{
    while (p < e) {
        const int mid = p + ((e - p) >> 1);
        if (__ldg(col + mid) < c) p = mid + 1;
        else e = mid;
    }
    return p;
}

template <int BH>
__device__ __forceinline__ int group_min(int v)
{
#pragma unroll
    for (int o = 1; o < BH; o <<= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <int BH>
__device__ __forceinline__ int group_max(int v)
{
#pragma unroll
    for (int o = 1; o < BH; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Where a lane's strips go: row hh of its block row's blocks, one block after
// another. V4: strips start at multiples of 4 values (128-bit stores).
template <bool V4>
struct Strips {
    float* data;         // strip 0 of the next block
    long long next, w4;  // to the next block's, to the next strip's
    int* col;            // its column id, 4-wide units
    long long cnext;
    template <int BW>
    __device__ void put(const float* v, bool id, int bc)
    {
#pragma unroll
        for (int w = 0; w < BW / 4; w++) {
            float* p = data + w * w4;
            if (V4) {
                *reinterpret_cast<float4*>(p) = make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] = v[4 * w + i];
            }
        }
        if (id) *col = bc * (BW / 4);
        data += next;
        col += cnext;
    }
};

// The merge of the entries [p, e) of a group's BH rows; returns the number
// of blocks, written through `out` with WRITE. Every lane of the warp takes
// part until the last group is done.
template <int BH, int BW, bool WRITE, class E, class Out>
__device__ __forceinline__ int merge_rows(const E& x, int p, int e, bool id, Out out)
{
    constexpr unsigned kAll = 0xffffffffu;
    int bc = p < e ? x.col(x.at(p)) / BW : INT_MAX;
    int n = 0;
    while (true) {
        const int m = group_min<BH>(bc);
        if (__all_sync(kAll, m == INT_MAX)) break;
        if (m == INT_MAX) continue;
        float v[BW];
        if (WRITE) {
#pragma unroll
            for (int t = 0; t < BW; t++) v[t] = 0.f;
        }
        if (bc == m) {
            const int c0 = m * BW;
            if (p + BW <= e) {   // the whole row of the block at once
                if (WRITE) {
                    int i[BW];
                    bool full = true;
#pragma unroll
                    for (int t = 0; t < BW; t++) {
                        i[t] = x.at(p + t);
                        full = full && x.col(i[t]) == c0 + t;
                    }
                    if (full) {
#pragma unroll
                        for (int t = 0; t < BW; t++) v[t] = x.val(i[t]);
                        p += BW;
                    }
                } else if (x.col(x.at(p + BW - 1)) < c0 + BW) {
                    p += BW;
                }
            }
            bc = INT_MAX;
            while (p < e) {      // a part of it, or repeats: the last value stays
                const int i = x.at(p), c = x.col(i);
                if (c - c0 >= BW) {
                    bc = c / BW;
                    break;
                }
                if (WRITE) {
                    const float y = x.val(i);
#pragma unroll
                    for (int t = 0; t < BW; t++) v[t] = c - c0 == t ? y : v[t];
                }
                p++;
            }
        }
        if constexpr (WRITE) out.template put<BW>(v, id, m);
        n++;
    }
    return n;
}

template <int BH, int BW, bool WRITE, class Place>
__global__ void __launch_bounds__(kRowWarps * 32) k_blocks(BlockJob J, Place place)
{
    extern __shared__ int dsm[];
    int* smem = dsm + (threadIdx.x >> 5) * (WRITE ? 2 : 1) * skewed(J.cap);
    constexpr int G = 32 / BH;   // items per warp
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, hh = lane % BH;
    if (bad_input(J.info)) return;
    const int nitems = J.first[J.nbr];
    const long long nwarps = (long long)gridDim.x * kRowWarps;
    for (long long w0 = ((long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5)) * G; w0 < nitems; w0 += nwarps * G) {
        const long long item = w0 + lane / BH;
        const bool on = item < nitems;
        const int br = on ? __ldg(J.brow + item) : J.nbr;
        const long long r = (long long)br * BH + hh;
        int p = __ldg(J.rp + min(r, (long long)J.h)), e = __ldg(J.rp + min(r + 1, (long long)J.h));
        const int i0 = on ? __ldg(J.first + br) : 0, pieces = on ? __ldg(J.first + br + 1) - i0 : 1;
        const bool whole = __all_sync(kAll, pieces == 1);
        const int lo = __shfl_sync(kAll, p, 0), hi = __shfl_sync(kAll, e, 31);
        if (!whole) {   // a piece: block columns [from, to), cut at block columns of the longest row
            const int most = group_max<BH>(e - p);
            const int owner = group_min<BH>(e - p == most ? lane : 32);
            const int op = __shfl_sync(kAll, p, owner);
            if (pieces > 1) {
                const int k = (int)(item - i0);
                const long long a = op + (long long)most * k / pieces, b = op + (long long)most * (k + 1) / pieces;
                const long long from = k ? (long long)__ldg(J.col + a) / BW * BW : 0;
                const long long to = k + 1 < pieces ? (long long)__ldg(J.col + b) / BW * BW : LLONG_MAX;
                p = lower_col(J.col, p, e, from);
                e = lower_col(J.col, p, e, to);
            }
        }
        const bool id = on && hh == 0;
        auto walk = [&](const auto& x) {
            if constexpr (WRITE) {
                const int before = on ? __ldg(J.before + item) : 0;
                const int j0 = on ? before - __ldg(J.brp + br) : 0;
                merge_rows<BH, BW, true>(x, p, e, id, place.template start<BH, BW>(on ? br : 0, j0, before, hh));
            } else {
                const int n = merge_rows<BH, BW, false>(x, p, e, id, 0);
                if (id) J.count[item] = n;
            }
        };
        if (whole && hi - lo <= J.cap) walk(stage<WRITE>(J.col, J.val, lo, hi, J.cap, smem));
        else walk(InPlace{J.col, J.val});
    }
}

struct NoPlace {};
template <bool V4>
struct PutB4csr {   // planes (w4, h) of 4 values per block
    long long len, plane;
    int* colid;
    float* data;
    template <int BH, int BW>
    __device__ Strips<V4> start(int, int, long long b, int hh) const
    {
        return Strips<V4>{data + hh * len + b * 4, 4, plane, colid + b, 1};
    }
};
template <bool V4>
struct PutB4ell {   // data[j*colsz + hh*f4 + w4*w4sz + r*4 + w] (include/matrix_storage.h:2178)
    long long len, f4, colsz, w4sz;
    int* colid;
    float* data;
    template <int BH, int BW>
    __device__ Strips<V4> start(int r, int j, long long, int hh) const
    {
        return Strips<V4>{data + j * colsz + hh * f4 + (long long)r * 4, colsz, w4sz, colid + j * len + r, len};
    }
};
struct PutSbell {   // include/matrix_storage.h:2387
    const int* ptr;
    int sh;
    int* colid;
    float* data;
    template <int BH, int BW>
    __device__ Strips<true> start(int r, int j, long long, int hh) const
    {
        const int s = r / sh, lr = r - s * sh;
        const long long hsz = (long long)sh * 4, first = __ldg(ptr + s), colsz = hsz * (BW / 4) * BH;
        return Strips<true>{data + first * (BW * BH) + j * colsz + hh * hsz + (long long)lr * 4, colsz, hsz * BH,
                            colid + first + (long long)j * sh + lr, sh};
    }
};

// Padding of b4ell, slots (j, r) past block row r's last block: its last
// column id (0 for an empty or missing row, already written) and, with CLEAR,
// zero strips (rows up to f4 / 4).
template <bool CLEAR>
__global__ void k_b4ell_pad(const int* __restrict__ brp, int nbr, int num, long long len, long long f4, int strips, int* colid,
                            float* data)
{
    const long long rows = max(len, f4 / 4), total = rows * num;
    GRID_STRIDE(t, total)
    {
        const long long j = t / rows, r = t - j * rows;
        const int n = r < nbr ? brp[r + 1] - brp[r] : 0;
        if (j < n) continue;
        if (r < len) colid[j * len + r] = n > 0 ? colid[(n - 1) * len + r] : 0;
        if (CLEAR && r < f4 / 4)
            for (int i = 0; i < strips; i++)
                *reinterpret_cast<float4*>(data + (j * strips + i) * f4 + r * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Padding of SBELL in the same sense; a warp takes kFillCols slot columns of
// all slices at a time, a lane a block row of a column.
__global__ void __launch_bounds__(kT) k_sbell_pad(const int* __restrict__ ptr, int ns, const int* __restrict__ brp, int nbr,
                                                  int sh, int strips, long long cols, int* colid, float* data)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * (kT / 32);
    for (long long c0 = ((long long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5)) * kFillCols; c0 < cols; c0 += nwarps * kFillCols) {
        const long long c1 = min(c0 + kFillCols, cols);
        long long c = c0;
        int s = slice_of(ptr, ns, c * sh);
        while (c < c1) {
            const long long start = ptr[s], sb = start / sh, se = ptr[s + 1] / sh;
            if (se <= c) {
                s = slice_of(ptr, ns, c * sh);
                continue;
            }
            const long long ce = min(c1, se);
            for (int lr = lane; lr < sh; lr += 32) {
                const long long r = (long long)s * sh + lr;
                const int n = r < nbr ? __ldg(brp + r + 1) - __ldg(brp + r) : 0;
                if (n >= ce - sb) continue;
                const int last = n > 0 ? colid[start + (long long)(n - 1) * sh + lr] : 0;
                for (long long j = max(c - sb, (long long)n); j < ce - sb; j++) {
                    colid[start + j * sh + lr] = last;
                    float* d = data + (start + j * sh) * strips * 4 + (long long)lr * 4;
                    for (int i = 0; i < strips; i++) *reinterpret_cast<float4*>(d + (long long)i * sh * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            c = ce;
            s++;
        }
    }
}

// The values past the last block of every b4csr plane.
__global__ void k_b4csr_tail(long long from, long long len, int planes, float* data)
{
    const long long per = len - from;
    GRID_STRIDE(t, per * planes) data[t / per * len + from + t % per] = 0.f;
}

// ---------------------------------------------------------------------------
// Host steps
// ---------------------------------------------------------------------------

struct Coo {
    int h, w;
    long long n;
    const int* row;
    const int* col;
    const float* val;
};

bool coo_args_ok(const clspmv_coo_f32* m)
{
    if (!m || m->matinfo.width < 0 || m->matinfo.height < 0 || m->matinfo.nnz < 0) return false;
    if (m->matinfo.nnz > 0 && (!m->coo_row_id || !m->coo_col_id || !m->coo_data)) return false;
    return true;
}

bool block_shape_ok(unsigned int bw, unsigned int bh)
{
    return (bw == 4 || bw == 8) && (bh == 1 || bh == 2 || bh == 4 || bh == 8);
}

inline bool at16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int new_info(cudaStream_t st, Allocs& S, Info** info)
{
    *info = S.get<Info>(1);
    if (S.rc) return S.rc;
    return cuda_status(cudaMemsetAsync(*info, 0, sizeof(Info), st));
}

// k_front over the COO (see there for rp, ocol / oval, mark and lim), and the
// gaps it left in rp.
int front(const Coo& c, cudaStream_t st, Allocs& S, Info* info, int* rp, int* ocol = nullptr, float* oval = nullptr,
          unsigned* mark = nullptr, long long lim = LLONG_MAX)
{
    int rc;
    if (c.n == 0) return rp ? cuda_status(cudaMemsetAsync(rp, 0, sizeof(int) * ((size_t)c.h + 1), st)) : CLSPMV_OK;
    // row pointers past INT_MAX - 1 do not fit the gap lists' ints: those are searched
    const bool search = rp && c.h > INT_MAX - kGap;
    GapLists gl{nullptr, nullptr, 0, 0};
    const bool gaps = rp && !search && c.h >= kGap;
    if (gaps) {   // a listed run has more than kGap (kBigGap) rows, and runs are disjoint
        gl.nsmall = (int)(((long long)c.h + 1) / kGap) + 2;
        gl.nbig = (int)(((long long)c.h + 1) / kBigGap) + 2;
        gl.small = S.get<int4>((size_t)gl.nsmall + gl.nbig);
        if (S.rc) return S.rc;
        gl.big = gl.small + gl.nsmall;
    }
    const bool vec = at16(c.row) && at16(c.col) && (!ocol || at16(c.val));
    int* frp = search ? nullptr : rp;
    const int grid = grid_for((c.n + 3) / 4);
    const int past = (int)std::min(lim, (long long)INT_MAX);
#define FRONT(V, C, M) k_front<V, C, M><<<grid, kT, 0, st>>>(c.row, c.col, c.val, c.n, c.h, c.w, frp, gl, ocol, oval, mark, past, info)
    if (ocol) {
        if (vec) FRONT(true, true, false);
        else FRONT(false, true, false);
    } else if (mark) {
        if (vec) FRONT(true, false, true);
        else FRONT(false, false, true);
    } else {
        if (vec) FRONT(true, false, false);
        else FRONT(false, false, false);
    }
#undef FRONT
    if ((rc = launched(st))) return rc;
    if (gaps) {
        k_gaps<<<148, kT, 0, st>>>(rp, gl, info);
        if ((rc = launched(st))) return rc;
    }
    if (search) {
        k_lower_bounds<<<grid_for((long long)c.h + 1), kT, 0, st>>>(c.row, c.n, c.h, rp);
        rc = launched(st);
    }
    return rc;
}

// Status of a conversion that wants a sorted COO, in the host converters' order of checks.
int front_status(int flags, bool shape_ok)
{
    if (flags & 2) return CLSPMV_ERR_ARG;
    if (!shape_ok) return CLSPMV_ERR_UNSUPPORTED;
    if (flags & 1) return CLSPMV_ERR_NOT_SORTED;
    return CLSPMV_OK;
}

// The checks alone: the status of a call that does no work (or could not
// allocate it: `otherwise`).
int checks_only(const Coo& c, cudaStream_t st, bool shape_ok, int otherwise)
{
    Allocs S(st);
    Info *info, host{};
    int rc = new_info(st, S, &info);
    if (!rc) rc = front(c, st, S, info, nullptr);
    if (!rc) rc = read_back(info, &host, st);
    if (!rc) rc = front_status(host.flags, shape_ok);
    return rc ? rc : otherwise;
}

// Entries of 32 rows that the staged kernels hold per warp: a quarter more
// than the mean, within 48 KB for the 4 warps of a CTA; a longer range is
// read in place.
int stage_cap(const Coo& c)
{
    const double mean = c.h > 0 ? 32.0 * (double)c.n / c.h : 0.0;
    return (int)std::min(1344.0, std::max(128.0, (double)(((long long)(mean * 1.25) + 64 + 31) / 32 * 32)));
}
size_t stage_bytes(int cap, bool vals) { return sizeof(int) * (size_t)kRowWarps * (vals ? 2 : 1) * (cap + (cap >> 5)); }
// CTAs of a warp-strided staged kernel over `rows` rows
int stage_grid(long long warps) { return (int)std::max(1LL, std::min((warps + kRowWarps - 1) / kRowWarps, 148LL * 64)); }

// Stable radix sort of (key, position) pairs; on return *idx_out holds the
// positions in key order, and *keys_out the sorted keys.
int sort_pairs(unsigned long long* k0, unsigned long long* k1, int* v0, int* v1, long long n, int end_bit,
               cudaStream_t st, Allocs& S, unsigned long long** keys_out, int** idx_out)
{
    *keys_out = k0;
    *idx_out = v0;
    if (n <= 1 || end_bit == 0) return CLSPMV_OK;
    size_t tb = 0;
    int rc = cuda_status(cub::DeviceRadixSort::SortPairs(nullptr, tb, k0, k1, v0, v1, (int)n, 0, end_bit, st));
    if (rc) return rc;
    void* tmp = S.get<char>(tb);
    if (S.rc) return S.rc;
    rc = cuda_status(cub::DeviceRadixSort::SortPairs(tmp, tb, k0, k1, v0, v1, (int)n, 0, end_bit, st));
    if (rc) return rc;
    *keys_out = k1;
    *idx_out = v1;
    return CLSPMV_OK;
}

template <class T>
int exclusive_sum(const T* in, T* out, long long n, cudaStream_t st, Allocs& S)
{
    size_t tb = 0;
    const bool wide = n > INT_MAX;
    int rc = cuda_status(wide ? cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, n, st)
                              : cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, (int)n, st));
    if (rc) return rc;
    void* tmp = S.get<char>(tb);
    if (S.rc) return S.rc;
    return cuda_status(wide ? cub::DeviceScan::ExclusiveSum(tmp, tb, in, out, n, st)
                            : cub::DeviceScan::ExclusiveSum(tmp, tb, in, out, (int)n, st));
}

template <class T>
int inclusive_sum(const T* in, T* out, long long n, cudaStream_t st, Allocs& S)
{
    size_t tb = 0;
    int rc = cuda_status(cub::DeviceScan::InclusiveSum(nullptr, tb, in, out, (int)n, st));
    if (rc) return rc;
    void* tmp = S.get<char>(tb);
    if (S.rc) return S.rc;
    return cuda_status(cub::DeviceScan::InclusiveSum(tmp, tb, in, out, (int)n, st));
}

int max_len(const int* rp, int nrows, cudaStream_t st, Allocs& S, int* out)
{
    *out = 0;
    if (nrows <= 0) return CLSPMV_OK;
    int* d = S.get<int>(1);
    if (S.rc) return S.rc;
    int rc = cuda_status(cudaMemsetAsync(d, 0, sizeof(int), st));
    if (rc) return rc;
    k_max_len<<<grid_for(nrows), kT, 0, st>>>(rp, nrows, d, nullptr);
    if ((rc = launched(st))) return rc;
    return read_back(d, out, st);
}

// Slice pointer of slices of `sh` rows over row pointer rp (nrows rows):
// ptr[s + 1] = ptr[s] + longest row of slice s * sh; info->total = ptr[ns]
// (past INT_MAX the int pointer has overflowed: the caller checks).
int slice_ptr(const int* rp, int nrows, int sh, int ns, cudaStream_t st, Allocs& S, Allocs& O, Info* info, int** ptr)
{
    long long* w = S.get<long long>((size_t)ns + 1);
    long long* p64 = S.get<long long>((size_t)ns + 1);
    *ptr = O.get<int>((size_t)ns + 1);
    if (S.rc) return S.rc;
    if (O.rc) return O.rc;
    k_slice_slots<<<grid_for(ns + 1), kT, 0, st>>>(rp, nrows, sh, ns, w, info);
    int rc = launched(st);
    if (!rc) rc = exclusive_sum(w, p64, (long long)ns + 1, st, S);
    if (rc) return rc;
    k_to_int<<<grid_for(ns + 1), kT, 0, st>>>(p64, (long long)ns + 1, *ptr, info);
    return launched(st);
}

int row_ptr(const int* ids, long long n, int nrows, cudaStream_t st, int* rp)
{
    k_lower_bounds<<<grid_for((long long)nrows + 1), kT, 0, st>>>(ids, n, nrows, rp);
    return launched(st);
}

Coo view(const clspmv_coo_f32* m)
{
    return Coo{m->matinfo.height, m->matinfo.width, (long long)m->matinfo.nnz, m->coo_row_id, m->coo_col_id,
               m->coo_data};
}

int finish(cudaStream_t st) { return cuda_status(cudaStreamSynchronize(st)); }

// Block rows of a sorted COO for bw x bh blocks: blocks in (block row, block
// column) order with their block row / column, the block row pointer, and
// for each entry in that order its COO position and 1-based block id.
struct Blocks {
    int nbr = 0;
    long long nb = 0;
    int* idx = nullptr;    // COO positions in block order
    int* bid = nullptr;    // 1-based block of each position
    int* brow = nullptr;   // per block
    int* bcol = nullptr;   // per block (block column index)
    int* brp = nullptr;    // nbr + 1
};

int make_blocks(const Coo& c, int bw, int bh, cudaStream_t st, Allocs& S, Blocks& B)
{
    B.nbr = (int)(c.h / bh + (c.h % bh ? 1 : 0));
    const long long nbc = c.w / bw + (c.w % bw ? 1 : 0);
    const int colbits = bits_for(nbc), rowbits = bits_for(B.nbr);
    B.brp = S.get<int>((size_t)B.nbr + 1);
    if (S.rc) return S.rc;
    int rc;
    if (c.n == 0) {
        rc = cuda_status(cudaMemsetAsync(B.brp, 0, sizeof(int) * ((size_t)B.nbr + 1), st));
        return rc;
    }
    unsigned long long* k0 = S.get<unsigned long long>(c.n);
    unsigned long long* k1 = S.get<unsigned long long>(c.n);
    int* v0 = S.get<int>(c.n);
    int* v1 = S.get<int>(c.n);
    int* head = S.get<int>(c.n);
    B.bid = S.get<int>(c.n);
    if (S.rc) return S.rc;
    k_block_keys<<<grid_for(c.n), kT, 0, st>>>(c.row, c.col, c.n, bw, bh, colbits, k0, v0);
    if ((rc = launched(st))) return rc;
    unsigned long long* keys;
    if ((rc = sort_pairs(k0, k1, v0, v1, c.n, colbits + rowbits, st, S, &keys, &B.idx))) return rc;
    k_block_heads<<<grid_for(c.n), kT, 0, st>>>(keys, c.n, head);
    if ((rc = launched(st))) return rc;
    if ((rc = inclusive_sum(head, B.bid, c.n, st, S))) return rc;
    int nb = 0;
    if ((rc = read_back(B.bid + (c.n - 1), &nb, st))) return rc;
    B.nb = nb;
    B.brow = S.get<int>((size_t)nb);
    B.bcol = S.get<int>((size_t)nb);
    if (S.rc) return S.rc;
    k_block_list<<<grid_for(c.n), kT, 0, st>>>(keys, head, B.bid, c.n, colbits, B.brow, B.bcol);
    if ((rc = launched(st))) return rc;
    return row_ptr(B.brow, B.nb, B.nbr, st, B.brp);
}

template <class Place>
int scatter_blocks(const Coo& c, const Blocks& B, int bw, int bh, Place place, float* data, cudaStream_t st)
{
    if (c.n == 0) return CLSPMV_OK;
    k_block_scatter<<<grid_for(c.n), kT, 0, st>>>(B.idx, B.bid, c.row, c.col, c.val, c.n, bw, bh, B.brow, B.bcol,
                                                  B.brp, place, data);
    return launched(st);
}

// Checks of the generic block converters, with the host converters' statuses.
int sorted_front(const Coo& c, cudaStream_t st) { return checks_only(c, st, true, CLSPMV_OK); }

int dia_core(const clspmv_coo_f32* src, clspmv_dia_f32* dst, int alignment, cudaStream_t st, Allocs& O)
{
    if (!coo_args_ok(src) || !dst || alignment <= 0) return CLSPMV_ERR_ARG;
    const Coo c = view(src);
    Allocs S(st);
    const long long len = aligned_len(std::min(c.w, c.h), alignment);
    const long long nd = c.h > 0 ? (long long)c.w + c.h - 1 : 0, words = (nd + 31) / 32;
    int* rp = S.get<int>((size_t)c.h + 1);
    unsigned* mark = S.get<unsigned>((size_t)words + 1);
    int* cnt = S.get<int>((size_t)words + 1);
    int* first = S.get<int>((size_t)words + 1);
    if (S.rc) return checks_only(c, st, true, S.rc);
    Info *info, host{};
    int rc = new_info(st, S, &info);
    if (rc) return rc;
    if ((rc = cuda_status(cudaMemsetAsync(mark, 0, sizeof(unsigned) * ((size_t)words + 1), st)))) return rc;
    if ((rc = front(c, st, S, info, rp, nullptr, nullptr, mark, len))) return rc;
    k_mark_counts<<<grid_for(words + 1), kT, 0, st>>>(mark, words, cnt);
    if ((rc = launched(st))) return rc;
    if ((rc = exclusive_sum(cnt, first, words + 1, st, S))) return rc;
    k_publish<<<1, 1, 0, st>>>(first + words, info);
    if ((rc = launched(st))) return rc;
    if ((rc = read_back(info, &host, st))) return rc;
    if (host.flags & 2) return CLSPMV_ERR_ARG;
    // dia_data[row] with row < aligned(min(w, h)): a taller-than-wide matrix
    // converts while every entry sits above that row, and is rejected when one
    // does not (as by clspmv_coo2dia_f32: the reference writes past its arrays)
    if (c.h > c.w && (host.flags & 4)) return CLSPMV_ERR_ARG;
    dst->matinfo = src->matinfo;
    dst->dia_length = std::min(c.w, c.h);
    dst->dia_length_aligned = (int)len;
    dst->dia_num = 0;
    dst->dia_offsets = nullptr;
    dst->dia_data = nullptr;
    const int D = (int)host.total;
    // The reference refuses at the discovery of a new diagonal when the count
    // found so far times the aligned length reaches 2 nnz
    // (include/matrix_storage.h:972): with D diagonals in all, iff
    // (D - 1) * len >= 2 nnz, leaving dia_num = the least k with k * len >= 2 nnz.
    if (D >= 1 && len > 0 && (long long)(D - 1) * len >= 2LL * c.n) {
        dst->dia_num = (int)((2LL * c.n + len - 1) / len);
        return CLSPMV_ERR_REFUSED;
    }
    int* off = O.get<int>((size_t)D);
    float* data = O.get<float>((size_t)D * (size_t)len);
    if (O.rc) return O.rc;
    if (words > 0) {
        k_dia_offsets<<<grid_for(words), kT, 0, st>>>(mark, first, words, c.h, off);
        if ((rc = launched(st))) return rc;
    }
    if (!(host.flags & 1)) {
        if (D > 0 && len > 0) {
            const int cap = stage_cap(c);
            k_dia_rows<<<stage_grid((len + 31) / 32), kRowWarps * 32, stage_bytes(cap, true), st>>>(rp, c.col, c.val, c.h, len,
                                                                                                  off, D, cap, data);
            if ((rc = launched(st))) return rc;
        }
    } else {
        if ((rc = cuda_status(cudaMemsetAsync(data, 0, sizeof(float) * (size_t)D * (size_t)len, st)))) return rc;
        int* owner = S.get<int>((size_t)D * (size_t)len);
        if (S.rc) return S.rc;
        if ((rc = cuda_status(cudaMemsetAsync(owner, 0xff, sizeof(int) * (size_t)D * (size_t)len, st)))) return rc;
        k_dia_claim<<<grid_for(c.n), kT, 0, st>>>(c.row, c.col, c.n, c.h, mark, first, len, owner);
        if ((rc = launched(st))) return rc;
        k_dia_scatter_owned<<<grid_for(c.n), kT, 0, st>>>(c.row, c.col, c.val, c.n, c.h, mark, first, len, owner, data);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    dst->dia_num = D;
    dst->dia_offsets = off;
    dst->dia_data = data;
    return CLSPMV_OK;
}

// A 4-wide block format between its counting and its writing pass.
struct Merge {
    BlockJob J{};
    int* brp = nullptr;   // blocks before each block row, nbr + 1
    long long max_items = 0;
};

// Calls f(ic<BH>, ic<BW>) for a block shape that block_shape_ok accepts.
template <int V> using ic = std::integral_constant<int, V>;
template <class F>
void with_shape(int bw, int bh, F&& f)
{
#define SHAPE(H)                      \
    if (bh == H) {                    \
        if (bw == 4) f(ic<H>{}, ic<4>{}); \
        else f(ic<H>{}, ic<8>{});     \
    }
    SHAPE(1)
    SHAPE(2)
    SHAPE(4)
    SHAPE(8)
#undef SHAPE
}

template <bool WRITE, class Place>
int merge_pass(const BlockJob& J, long long max_items, int bw, int bh, Place place, cudaStream_t st)
{
    const int grid = stage_grid((max_items * bh + 31) / 32);
    with_shape(bw, bh, [&](auto H, auto W) {
        k_blocks<decltype(H)::value, decltype(W)::value, WRITE, Place>
            <<<grid, kRowWarps * 32, stage_bytes(J.cap, WRITE), st>>>(J, place);
    });
    return launched(st);
}

// Checks, row pointer and block counts: M.brp, info->total (blocks) and
// info->most (longest block row), all on the stream. nbr >= 1.
int count_blocks(const Coo& c, int bw, int bh, cudaStream_t st, Allocs& S, Allocs& O, Info* info, bool brp_is_output, Merge& M)
{
    BlockJob& J = M.J;
    J.col = c.col;
    J.val = c.val;
    J.h = c.h;
    J.nbr = (int)(c.h / bh + (c.h % bh ? 1 : 0));
    J.cap = stage_cap(c);
    J.info = info;
    // cut block rows come to at most one item more per kItemNnz entries; whole ones alone where an int could not count them
    const int item_nnz = J.nbr + c.n / kItemNnz < INT_MAX ? kItemNnz : INT_MAX;
    M.max_items = J.nbr + c.n / item_nnz;
    int* rp = S.get<int>((size_t)c.h + 1);
    int* cnt = S.get<int>((size_t)J.nbr + 1);
    int* first = S.get<int>((size_t)J.nbr + 1);
    int* brow = S.get<int>((size_t)M.max_items);
    int* count = S.get<int>((size_t)M.max_items + 1);
    int* before = S.get<int>((size_t)M.max_items + 1);
    M.brp = (brp_is_output ? O : S).get<int>((size_t)J.nbr + 1);
    if (S.rc || O.rc) return CLSPMV_ERR_ALLOC;
    int rc;
    if ((rc = front(c, st, S, info, rp))) return rc;
    k_item_counts<<<grid_for(J.nbr + 1LL), kT, 0, st>>>(rp, c.h, bh, J.nbr, item_nnz, cnt, info);
    if ((rc = launched(st))) return rc;
    if ((rc = exclusive_sum(cnt, first, J.nbr + 1LL, st, S))) return rc;
    k_item_rows<<<grid_for(J.nbr), kT, 0, st>>>(first, J.nbr, brow, info);
    if ((rc = launched(st))) return rc;
    J.rp = rp;
    J.first = first;
    J.brow = brow;
    J.count = count;
    J.before = before;
    J.brp = M.brp;
    if ((rc = merge_pass<false>(J, M.max_items, bw, bh, NoPlace{}, st))) return rc;
    if ((rc = exclusive_sum(count, before, M.max_items + 1, st, S))) return rc;
    k_block_ptr<<<grid_for(J.nbr + 1LL), kT, 0, st>>>(first, before, J.nbr, M.brp, info);
    return launched(st);
}

// Front of a block converter: the counts and `more` (launches that go with
// them), one read back, the statuses. A matrix without rows has no blocks.
template <class More>
int block_front(const Coo& c, int bw, int bh, bool shape_ok, cudaStream_t st, Allocs& S, Allocs& O, bool brp_is_output,
                Merge& M, Info* host, More&& more)
{
    if (!shape_ok) return checks_only(c, st, false, CLSPMV_ERR_UNSUPPORTED);
    Info* info;
    int rc = new_info(st, S, &info);
    if (rc) return rc;
    if (c.h == 0) {   // an entry would be outside the matrix
        if (c.n > 0) return CLSPMV_ERR_ARG;
        M.brp = (brp_is_output ? O : S).get<int>(1);
        if (S.rc || O.rc) return CLSPMV_ERR_ALLOC;
        rc = cuda_status(cudaMemsetAsync(M.brp, 0, sizeof(int), st));
    } else {
        rc = count_blocks(c, bw, bh, st, S, O, info, brp_is_output, M);
    }
    if (!rc) rc = more(info);
    if (rc == CLSPMV_ERR_ALLOC) return checks_only(c, st, true, rc);
    if (rc) return rc;
    if ((rc = read_back(info, host, st))) return rc;
    return front_status(host->flags, true);
}

}  // namespace

extern "C" {

int clspmv_device_sort_coo_f32(clspmv_coo_f32* mat, clspmv_stream_t stream)
{
    if (!coo_args_ok(mat)) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(mat);
    Allocs S(st);
    int rc = checks_only(c, st, true, CLSPMV_OK);
    if (rc != CLSPMV_ERR_NOT_SORTED) return rc;
    const int colbits = bits_for(c.w), rowbits = bits_for(c.h);
    unsigned long long* k0 = S.get<unsigned long long>(c.n);
    unsigned long long* k1 = S.get<unsigned long long>(c.n);
    int* v0 = S.get<int>(c.n);
    int* v1 = S.get<int>(c.n);
    int* ti = S.get<int>(c.n);
    float* tf = S.get<float>(c.n);
    if (S.rc) return S.rc;
    k_coo_keys<<<grid_for(c.n), kT, 0, st>>>(c.row, c.col, c.n, colbits, k0, v0);
    if ((rc = launched(st))) return rc;
    unsigned long long* keys;
    int* idx;
    if ((rc = sort_pairs(k0, k1, v0, v1, c.n, colbits + rowbits, st, S, &keys, &idx))) return rc;
    k_gather<int><<<grid_for(c.n), kT, 0, st>>>(idx, mat->coo_row_id, c.n, ti);
    if ((rc = launched(st))) return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(mat->coo_row_id, ti, sizeof(int) * c.n, cudaMemcpyDeviceToDevice, st)))) return rc;
    k_gather<int><<<grid_for(c.n), kT, 0, st>>>(idx, mat->coo_col_id, c.n, ti);
    if ((rc = launched(st))) return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(mat->coo_col_id, ti, sizeof(int) * c.n, cudaMemcpyDeviceToDevice, st)))) return rc;
    k_gather<float><<<grid_for(c.n), kT, 0, st>>>(idx, mat->coo_data, c.n, tf);
    if ((rc = launched(st))) return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(mat->coo_data, tf, sizeof(float) * c.n, cudaMemcpyDeviceToDevice, st)))) return rc;
    return finish(st);
}

int clspmv_device_coo2csr_f32(const clspmv_coo_f32* src, clspmv_csr_f32* dst, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    int* rp = O.get<int>((size_t)c.h + 1);
    int* col = O.get<int>((size_t)c.n);
    float* val = O.get<float>((size_t)c.n);
    if (O.rc) return checks_only(c, st, true, O.rc);
    Info *info, host{};
    int rc = new_info(st, S, &info);
    if (!rc) rc = front(c, st, S, info, rp, col, val);
    if (!rc) rc = read_back(info, &host, st);
    if (!rc) rc = front_status(host.flags, true);
    if (rc) return rc;
    O.keep = true;
    dst->matinfo = src->matinfo;
    dst->csr_row_ptr = rp;
    dst->csr_col_id = col;
    dst->csr_data = val;
    return CLSPMV_OK;
}

int clspmv_device_coo2dia_f32(const clspmv_coo_f32* src, clspmv_dia_f32* dst, int alignment, clspmv_stream_t stream)
{
    Allocs O((cudaStream_t)stream);
    const int rc = dia_core(src, dst, alignment, (cudaStream_t)stream, O);
    if (!rc) O.keep = true;
    return rc;
}

int clspmv_device_coo2bdia_f32(const clspmv_coo_f32* src, clspmv_bdia_f32* dst, int alignment, clspmv_stream_t stream)
{
    if (!dst) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    Allocs O(st);
    clspmv_dia_f32 dia;
    int rc = dia_core(src, &dia, alignment, st, O);
    if (rc) return rc;
    // Bands are maximal runs of consecutive offsets (include/matrix_storage.h:
    // 1184-1236); the offsets are few, so the bands are found on the host.
    std::vector<int> offs((size_t)dia.dia_num);
    if (dia.dia_num > 0 &&
        (rc = cuda_status(cudaMemcpy(offs.data(), dia.dia_offsets, sizeof(int) * offs.size(), cudaMemcpyDeviceToHost))))
        return rc;
    std::vector<int> first, bptr(1, 0);
    for (size_t d = 0; d < offs.size(); d++) {
        if (d > 0 && offs[d] - offs[d - 1] == 1) bptr.back()++;
        else {
            first.push_back(offs[d]);
            bptr.push_back(bptr.back() + 1);
        }
    }
    int* boff = O.get<int>(first.size());
    int* bp = O.get<int>(bptr.size());
    if (O.rc) return O.rc;
    if (!first.empty() &&
        (rc = cuda_status(cudaMemcpy(boff, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice))))
        return rc;
    if ((rc = cuda_status(cudaMemcpy(bp, bptr.data(), sizeof(int) * bptr.size(), cudaMemcpyHostToDevice)))) return rc;
    O.keep = true;
    clspmv::device_release(dia.dia_offsets, clspmv::kIdleAll);   // the DIA data array becomes the BDIA one
    dst->matinfo = dia.matinfo;
    dst->bdia_band_num = (int)first.size();
    dst->bdia_length = dia.dia_length;
    dst->bdia_length_aligned = dia.dia_length_aligned;
    dst->bdia_offsets = boff;
    dst->bdia_bptr = bp;
    dst->bdia_data = dia.dia_data;
    return CLSPMV_OK;
}

int clspmv_device_coo2ell_f32(const clspmv_coo_f32* src, clspmv_ell_f32* dst, int alignment, int ellnum,
                              clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || alignment <= 0 || ellnum < 0) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    int* rp = S.get<int>((size_t)c.h + 1);
    if (S.rc) return checks_only(c, st, true, S.rc);
    Info *info, host{};
    int rc = new_info(st, S, &info);
    if (!rc) rc = front(c, st, S, info, rp);
    if (rc) return rc;
    if (c.h > 0) {
        k_max_len<<<grid_for(c.h), kT, 0, st>>>(rp, c.h, &info->most, info);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = read_back(info, &host, st))) return rc;
    if ((rc = front_status(host.flags, true))) return rc;
    const int maxlen = host.most;
    // include/matrix_storage.h:1339-1394: ellnum 0 selects the longest row
    const int num = ellnum == 0 ? maxlen : ellnum;
    const long long len = aligned_len(c.h, alignment);
    dst->matinfo = src->matinfo;
    dst->ell_num = num;
    dst->ell_height_aligned = (int)len;
    dst->ell_col_id = nullptr;
    dst->ell_data = nullptr;
    if (maxlen > num) return ellnum > 0 ? CLSPMV_ERR_ARG : CLSPMV_ERR_REFUSED;
    if (len * num > (long long)INT_MAX) return CLSPMV_ERR_REFUSED;
    const long long total = len * num;
    int* col = O.get<int>((size_t)total);
    float* val = O.get<float>((size_t)total);
    if (O.rc) return O.rc;
    if (total > 0) {
        if (len % 4 == 0) {
            const long long warps = (len + 31) / 32 * ((num + kFillCols - 1) / kFillCols);
            k_ell_fill_quads<<<grid_for(warps * 32), kT, 0, st>>>(rp, c.col, c.val, c.h, len, num, col, val);
        } else {
            k_ell_fill<<<grid_for(total), kT, 0, st>>>(rp, c.col, c.val, c.h, len, total, col, val);
        }
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->ell_col_id = col;
    dst->ell_data = val;
    return CLSPMV_OK;
}

int clspmv_device_coo2sell_f32(const clspmv_coo_f32* src, clspmv_sell_f32* dst, unsigned int slice_height,
                               clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || slice_height == 0 || slice_height > (unsigned)INT_MAX) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    const int sh = (int)slice_height;
    const int ns = c.h / sh + (c.h % sh ? 1 : 0);
    int* rp = S.get<int>((size_t)c.h + 1);
    if (S.rc) return checks_only(c, st, true, S.rc);
    Info *info, host{};
    int* ptr = nullptr;
    int rc = new_info(st, S, &info);
    if (!rc) rc = front(c, st, S, info, rp);
    if (!rc) rc = slice_ptr(rp, c.h, sh, ns, st, S, O, info, &ptr);
    if (rc == CLSPMV_ERR_ALLOC) return checks_only(c, st, true, rc);
    if (rc) return rc;
    if ((rc = read_back(info, &host, st))) return rc;
    if ((rc = front_status(host.flags, true))) return rc;
    const long long total = host.total;
    if (total > INT_MAX) return CLSPMV_ERR_UNSUPPORTED;   // the int slice pointer would overflow
    int* col = O.get<int>((size_t)total);
    float* val = O.get<float>((size_t)total);
    if (O.rc) return O.rc;
    if (total > 0) {
        const long long cols = total / sh;
        const int grid = grid_for((cols + kFillCols - 1) / kFillCols * 32);
#define QUADS(H) \
    case H: k_sell_fill_quads<H / 4><<<grid, kT, 0, st>>>(ptr, ns, rp, c.col, c.val, c.h, cols, col, val); break;
        switch (sh) {
            QUADS(4)
            QUADS(8)
            QUADS(16)
            QUADS(32)
            QUADS(64)
            QUADS(128)
            default: k_sell_fill<<<grid_for(total), kT, 0, st>>>(ptr, ns, rp, c.col, c.val, c.h, sh, total, col, val);
        }
#undef QUADS
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->matinfo = src->matinfo;
    dst->sell_slice_height = slice_height;
    dst->sell_slice_num = ns;
    dst->sell_slice_ptr = ptr;
    dst->sell_col_id = col;
    dst->sell_data = val;
    return CLSPMV_OK;
}

int clspmv_device_coo2b4csr_f32(const clspmv_coo_f32* src, clspmv_b4csr_f32* dst, unsigned int bwidth,
                                unsigned int bheight, int alignment, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || alignment <= 0) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    const int bw = (int)bwidth, bh = (int)bheight;
    Merge M;
    Info host{};
    int rc = block_front(c, bw, bh, block_shape_ok(bwidth, bheight), st, S, O, true, M, &host, [](Info*) { return CLSPMV_OK; });
    if (rc) return rc;
    dst->matinfo = src->matinfo;
    dst->b4csr_bwidth = bwidth;
    dst->b4csr_bheight = bheight;
    const long long nb = host.total;
    // include/matrix_storage.h:1863: block count cap
    if ((size_t)nb > (size_t)CLSPMV_MAX_MEM_OBJ / ((size_t)bw * bh * sizeof(float))) return CLSPMV_ERR_REFUSED;
    const long long len = aligned_len(nb * 4, alignment);
    const int planes = bh * (bw / 4);
    int* colid = O.get<int>((size_t)nb);
    float* data = O.get<float>((size_t)len * planes);
    if (O.rc) return O.rc;
    if (nb > 0) {
        rc = len % 4 == 0 ? merge_pass<true>(M.J, M.max_items, bw, bh, PutB4csr<true>{len, len * bh, colid, data}, st)
                          : merge_pass<true>(M.J, M.max_items, bw, bh, PutB4csr<false>{len, len * bh, colid, data}, st);
        if (rc) return rc;
    }
    if (len > nb * 4) {
        k_b4csr_tail<<<grid_for((len - nb * 4) * planes), kT, 0, st>>>(nb * 4, len, planes, data);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->b4csr_row_num = M.J.nbr;
    dst->b4csr_aligned_size = (int)len;
    dst->b4csr_block_num = (int)nb;
    dst->b4csr_row_ptr = M.brp;
    dst->b4csr_col_id = colid;
    dst->b4csr_data = data;
    return CLSPMV_OK;
}

int clspmv_device_coo2bcsr_f32(const clspmv_coo_f32* src, clspmv_bcsr_f32* dst, unsigned int bwidth,
                               unsigned int bheight, int alignment, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || bwidth == 0 || bheight == 0 || bwidth > (unsigned)INT_MAX ||
        bheight > (unsigned)INT_MAX || alignment <= 0)
        return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    int rc = sorted_front(c, st);
    if (rc) return rc;
    const int bw = (int)bwidth, bh = (int)bheight;
    const size_t bs = (size_t)bw * bh;
    dst->matinfo = src->matinfo;
    dst->bcsr_bwidth = bwidth;
    dst->bcsr_bheight = bheight;
    Blocks B;
    if ((rc = make_blocks(c, bw, bh, st, S, B))) return rc;
    const long long len = aligned_len(B.nb, alignment);
    const size_t ndata = (size_t)len * bs;
    int* rp = O.get<int>((size_t)B.nbr + 1);
    int* colid = O.get<int>((size_t)B.nb);
    float* data = O.get<float>(ndata);
    if (O.rc) return O.rc;
    if ((rc = cuda_status(cudaMemcpyAsync(rp, B.brp, sizeof(int) * ((size_t)B.nbr + 1), cudaMemcpyDeviceToDevice, st))))
        return rc;
    if (ndata && (rc = cuda_status(cudaMemsetAsync(data, 0, sizeof(float) * ndata, st)))) return rc;
    if (B.nb > 0) {
        k_bcsr_colid<<<grid_for(B.nb), kT, 0, st>>>(B.bcol, B.nb, bw, colid);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = scatter_blocks(c, B, bw, bh, BcsrPlace{len, bw}, data, st))) return rc;
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->bcsr_row_num = B.nbr;
    dst->bcsr_aligned_size = (int)len;
    dst->bcsr_block_num = (int)B.nb;
    dst->bcsr_row_ptr = rp;
    dst->bcsr_col_id = colid;
    dst->bcsr_data = data;
    return CLSPMV_OK;
}

int clspmv_device_coo2bell_f32(const clspmv_coo_f32* src, clspmv_bell_f32* dst, unsigned int bwidth,
                               unsigned int bheight, int alignment, int ellnum, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || bwidth == 0 || bheight == 0 || bwidth > (unsigned)INT_MAX ||
        bheight > (unsigned)INT_MAX || alignment <= 0 || ellnum < 0)
        return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    int rc = sorted_front(c, st);
    if (rc) return rc;
    const int bw = (int)bwidth, bh = (int)bheight;
    const size_t bs = (size_t)bw * bh;
    dst->matinfo = src->matinfo;
    dst->bell_bwidth = bwidth;
    dst->bell_bheight = bheight;
    dst->bell_float4_aligned = 0;
    dst->bell_col_id = nullptr;
    dst->bell_data = nullptr;
    Blocks B;
    if ((rc = make_blocks(c, bw, bh, st, S, B))) return rc;
    int maxw = 0;
    if ((rc = max_len(B.brp, B.nbr, st, S, &maxw))) return rc;
    const int num = ellnum == 0 ? maxw : ellnum;
    const long long len = aligned_len(B.nbr, alignment);
    dst->bell_block_num = num;
    dst->bell_row_num = B.nbr;
    dst->bell_height_aligned = (int)len;
    if (maxw > num) return CLSPMV_ERR_ARG;   // a block row longer than ellnum (include/matrix_storage.h:1975)
    const size_t ncol = (size_t)len * num, colsz = (size_t)len * bs, ndata = colsz * num;
    int* col = O.get<int>(ncol);
    float* data = O.get<float>(ndata);
    if (O.rc) return O.rc;
    if (ndata && (rc = cuda_status(cudaMemsetAsync(data, 0, sizeof(float) * ndata, st)))) return rc;
    if (ncol > 0) {
        k_bell_cols<<<grid_for((long long)ncol), kT, 0, st>>>(B.brp, B.bcol, B.nbr, bw, len, (long long)ncol, col);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = scatter_blocks(c, B, bw, bh, BellPlace{len, (long long)colsz, bw}, data, st))) return rc;
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->bell_col_id = col;
    dst->bell_data = data;
    return CLSPMV_OK;
}

int clspmv_device_coo2b4ell_f32(const clspmv_coo_f32* src, clspmv_b4ell_f32* dst, unsigned int bwidth,
                                unsigned int bheight, int alignment, int ellnum, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || alignment <= 0 || ellnum < 0) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    const int bw = (int)bwidth, bh = (int)bheight, bs = bw * bh;
    Merge M;
    Info host{};
    int rc = block_front(c, bw, bh, block_shape_ok(bwidth, bheight), st, S, O, false, M, &host, [](Info*) { return CLSPMV_OK; });
    if (rc) return rc;
    dst->matinfo = src->matinfo;
    dst->b4ell_bwidth = bwidth;
    dst->b4ell_bheight = bheight;
    const int nbr = M.J.nbr, maxw = host.most;
    const int num = ellnum == 0 ? maxw : ellnum;
    // include/matrix_storage.h:2141: padded block count cap
    if ((size_t)nbr * (size_t)num > (size_t)CLSPMV_MAX_MEM_OBJ / ((size_t)bs * sizeof(float))) return CLSPMV_ERR_REFUSED;
    if (maxw > num) return CLSPMV_ERR_REFUSED;
    const long long len = aligned_len(nbr, alignment), f4 = aligned_len(4LL * nbr, alignment);
    const int strips = bh * (bw / 4);
    const size_t ncol = (size_t)len * num, ndata = (size_t)f4 * strips * num;
    int* col = O.get<int>(ncol);
    float* data = O.get<float>(ndata);
    if (O.rc) return O.rc;
    const bool v4 = f4 % 4 == 0;
    if (!v4 && ndata && (rc = cuda_status(cudaMemsetAsync(data, 0, sizeof(float) * ndata, st)))) return rc;
    if (host.total > 0) {
        rc = v4 ? merge_pass<true>(M.J, M.max_items, bw, bh, PutB4ell<true>{len, f4, f4 * strips, f4 * bh, col, data}, st)
                : merge_pass<true>(M.J, M.max_items, bw, bh, PutB4ell<false>{len, f4, f4 * strips, f4 * bh, col, data}, st);
        if (rc) return rc;
    }
    if (num > 0 && std::max(len, f4 / 4) > 0) {
        const int grid = grid_for(std::max(len, f4 / 4) * num);
        if (v4) k_b4ell_pad<true><<<grid, kT, 0, st>>>(M.brp, nbr, num, len, f4, strips, col, data);
        else k_b4ell_pad<false><<<grid, kT, 0, st>>>(M.brp, nbr, num, len, f4, strips, col, data);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->b4ell_row_num = nbr;
    dst->b4ell_block_num = num;
    dst->b4ell_height_aligned = (int)len;
    dst->b4ell_float4_aligned = (int)f4;
    dst->b4ell_col_id = col;
    dst->b4ell_data = data;
    return CLSPMV_OK;
}

int clspmv_device_coo2sbell_f32(const clspmv_coo_f32* src, clspmv_sbell_f32* dst, unsigned int bwidth,
                                unsigned int bheight, unsigned int slice_height, clspmv_stream_t stream)
{
    if (!coo_args_ok(src) || !dst || slice_height == 0 || slice_height > (unsigned)INT_MAX) return CLSPMV_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    const Coo c = view(src);
    Allocs S(st), O(st);
    const int bw = (int)bwidth, bh = (int)bheight, bs = bw * bh, sh = (int)slice_height;
    Merge M;
    Info host{};
    int* ptr = nullptr;
    int ns = 0;
    const bool shape_ok = block_shape_ok(bwidth, bheight);
    int rc = block_front(c, bw, bh, shape_ok, st, S, O, false, M, &host, [&](Info* info) {
        ns = M.J.nbr / sh + (M.J.nbr % sh ? 1 : 0);
        return slice_ptr(M.brp, M.J.nbr, sh, ns, st, S, O, info, &ptr);
    });
    if (rc) return rc;
    dst->matinfo = src->matinfo;
    dst->sbell_bwidth = bwidth;
    dst->sbell_bheight = bheight;
    dst->sbell_slice_num = ns;
    dst->sbell_row_num = M.J.nbr;
    dst->sbell_slice_height = slice_height;
    dst->sbell_slice_ptr = nullptr;
    dst->sbell_col_id = nullptr;
    dst->sbell_data = nullptr;
    const long long total = host.total;
    if (total > INT_MAX) return CLSPMV_ERR_UNSUPPORTED;   // the int slice pointer would overflow
    // include/matrix_storage.h:2350: padded block count cap
    if ((size_t)total > (size_t)CLSPMV_MAX_MEM_OBJ / ((size_t)bs * sizeof(float))) return CLSPMV_ERR_REFUSED;
    int* col = O.get<int>((size_t)total);
    float* data = O.get<float>((size_t)total * bs);
    if (O.rc) return O.rc;
    if (total > 0) {
        if ((rc = merge_pass<true>(M.J, M.max_items, bw, bh, PutSbell{ptr, sh, col, data}, st))) return rc;
        const long long cols = total / sh;
        k_sbell_pad<<<grid_for((cols + kFillCols - 1) / kFillCols * 32), kT, 0, st>>>(ptr, ns, M.brp, M.J.nbr, sh, bs / 4, cols,
                                                                                     col, data);
        if ((rc = launched(st))) return rc;
    }
    if ((rc = finish(st))) return rc;
    O.keep = true;
    dst->sbell_slice_ptr = ptr;
    dst->sbell_col_id = col;
    dst->sbell_data = data;
    return CLSPMV_OK;
}

}  // extern "C"
