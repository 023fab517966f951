// iterate_resident.cu — steps of y <- alpha*A*x + beta*y; x <- y (the
// reference's A^k x loop, src/eval.cpp:19-72) of one DIA, BDIA, COO or CSR matrix that
// fits the shared memory of a thread-block cluster, all in one launch.
//
// A step on a small matrix costs its launch: 65,536 rows of 5 diagonals are
// 1.3 MB, 0.2 us of HBM time, but a graph-replayed kernel takes 4 us. Here
// the cluster's CTAs each keep a run of rows: their entries and the vector's
// part, twice (the last result and the next one). A row's entries that lie in
// another run are read from its owner's shared memory (ld.shared::cluster),
// and one cluster barrier ends a step: all reads of the old vector are done
// before anybody writes over it in the next step. Rows are summed
// by one thread each, in stored order.
//
// 40 steps on one B200, a copy and a launch per step / a launch per step /
// resident: 5-point Laplacian of 65,536 rows (DIA) 228 / 159 / 105 us, of
// 16,384 rows 164 / 118 / 64; of 4,096 rows (COO, two launches a step) 187 / 182 / 60.
#include <cooperative_groups.h>
#include <algorithm>
#include <cstdint>
#include <memory>
#include <new>
#include "api_internal.h"
#include "clspmv_b200.h"

namespace cg = cooperative_groups;

namespace clspmv {
namespace {

constexpr int kThreads = 1024;
constexpr int kMaxCtas = 16;       // a cluster above 8 CTAs is opt-in
constexpr int kMaxDiags = 128;

struct Args {
    int rows, cols, ndiag, per;    // per: rows of a CTA
    long long len;
    const int* offsets;            // DIA: ndiag; BDIA: first offset of each band
    const int* bptr;               // BDIA: diagonals before each band, nband + 1
    int nband;
    const float* data;
    float* x;
    float* y;
    float alpha, beta;
    int steps;
};

__global__ void __launch_bounds__(kThreads) k_dia_resident(Args a)
{
    extern __shared__ float sm[];
    __shared__ int off[kMaxDiags];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), per = a.per;
    const int base = rank * per, n = max(0, min(per, a.rows - base));
    float* const vec[2] = {sm, sm + per};
    float* const val = sm + 2 * per;
    if (a.bptr) {
        for (int b = threadIdx.x; b < a.nband; b += kThreads)
            for (int i = a.bptr[b]; i < a.bptr[b + 1]; i++) off[i] = a.offsets[b] + (i - a.bptr[b]);
    } else {
        for (int i = threadIdx.x; i < a.ndiag; i += kThreads) off[i] = a.offsets[i];
    }
    for (int i = threadIdx.x; i < n; i += kThreads) vec[0][i] = a.x[base + i];
    for (int d = 0; d < a.ndiag; d++)
        for (int i = threadIdx.x; i < n; i += kThreads) val[d * per + i] = a.data[d * a.len + base + i];
    cluster.sync();
    // rows i0 .. i0+31 whose entries all lie in this CTA's run take the short loop
    int lowest = 0, highest = 0;
    for (int d = 0; d < a.ndiag; d++) {
        lowest = min(lowest, off[d]);
        highest = max(highest, off[d]);
    }
    const int lane = threadIdx.x & 31;
    for (int s = 0; s < a.steps; s++) {
        const float* in = vec[s & 1];
        float* out = vec[(s & 1) ^ 1];
        auto put = [&](int i, float acc) {
            const float v = a.alpha * acc;
            out[i] = a.beta == 0.f ? v : fmaf(a.beta, s == 0 ? a.y[base + i] : in[i], v);
        };
        auto inside = [&](int i0) { return i0 + lowest >= 0 && i0 + 32 + highest <= n; };
        int i0 = threadIdx.x - lane;
        while (i0 < n) {
            const int i = i0 + lane;
            if (inside(i0) && inside(i0 + kThreads)) {           // two rows share the offsets
                const float* vp = val + i;
                const float* xp = in + i;
                float p = 0.f, q = 0.f;
#pragma unroll 4
                for (int d = 0; d < a.ndiag; d++, vp += per) {
                    const int o = off[d];
                    p = fmaf(vp[0], xp[o], p);
                    q = fmaf(vp[kThreads], xp[o + kThreads], q);
                }
                put(i, p);
                put(i + kThreads, q);
                i0 += 2 * kThreads;
                continue;
            }
            float acc = 0.f;
            if (inside(i0)) {
                const float* vp = val + i;
#pragma unroll 4
                for (int d = 0; d < a.ndiag; d++, vp += per) acc = fmaf(*vp, in[i + off[d]], acc);
            } else if (i < n) {
                for (int d = 0; d < a.ndiag; d++) {
                    const int l = i + off[d], c = base + l;
                    float xv = 0.f;                              // a diagonal's part outside the matrix multiplies zero
                    if ((unsigned)l < (unsigned)n) {
                        xv = in[l];
                    } else if (c >= 0 && c < a.rows) {
                        const int owner = c / per;
                        xv = cluster.map_shared_rank(in, owner)[c - owner * per];
                    } else if (c >= a.rows && c < a.cols) {
                        xv = a.x[c];                             // past the result's length x stays as it is
                    }
                    acc = fmaf(val[d * per + i], xv, acc);
                }
            }
            if (i < n) put(i, acc);
            i0 += kThreads;
        }
        cluster.sync();
    }
    const float* last = vec[a.steps & 1];
    for (int i = threadIdx.x; i < n; i += kThreads) a.x[base + i] = a.y[base + i] = last[i];
}

// Rows of a COO (row ids) or CSR (row pointer) matrix.
struct RowArgs {
    int rows, cols, nnz, per, cap;   // cap: entries a CTA has room for
    const int* row_id;               // COO, sorted; null: CSR
    const int* row_ptr;
    const int* col;
    const float* val;
    float* x;
    float* y;
    float alpha, beta;
    int steps;
};

__global__ void __launch_bounds__(kThreads) k_rows_resident(RowArgs a)
{
    extern __shared__ float sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), per = a.per;
    const int base = min(a.rows, rank * per), n = min(per, a.rows - base);
    float* const vec[2] = {sm, sm + per};
    int* const start = reinterpret_cast<int*>(sm + 2 * per);     // per + 1, from the CTA's first entry
    int* const where = start + per + 1;                          // per entry: owner << 16 | place in its run, -1 - column past the rows
    float* const val = reinterpret_cast<float*>(where + a.cap);
    auto first_of = [&](int r) {                                 // first entry of a row >= r
        if (!a.row_id) return a.row_ptr[r];
        int lo = 0, hi = a.nnz;
        while (lo < hi) {
            const int mid = lo + ((hi - lo) >> 1);
            if (a.row_id[mid] < r) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    const int e0 = first_of(base);
    for (int i = threadIdx.x; i <= n; i += kThreads) start[i] = min(a.cap, first_of(base + i) - e0);
    for (int i = threadIdx.x; i < n; i += kThreads) vec[0][i] = a.x[base + i];
    __syncthreads();
    for (int j = threadIdx.x; j < start[n]; j += kThreads) {
        const int c = a.col[e0 + j], owner = c / per;
        where[j] = c < a.rows ? owner << 16 | (c - owner * per) : -1 - c;
        val[j] = a.val[e0 + j];
    }
    cluster.sync();
    for (int s = 0; s < a.steps; s++) {
        const float* in = vec[s & 1];
        float* out = vec[(s & 1) ^ 1];
        for (int i = threadIdx.x; i < n; i += kThreads) {
            float acc = 0.f;
            const int e = start[i + 1];
            for (int j = start[i]; j < e; j++) {
                const int w = where[j];
                const float xv = (w >> 16) == rank ? in[w & 0xffff]
                                 : w >= 0          ? cluster.map_shared_rank(in, w >> 16)[w & 0xffff]
                                                   : a.x[-1 - w];   // past the result's length x stays as it is
                acc = fmaf(val[j], xv, acc);
            }
            const float v = a.alpha * acc;
            out[i] = a.beta == 0.f ? v : fmaf(a.beta, s == 0 ? a.y[base + i] : in[i], v);
        }
        cluster.sync();
    }
    const float* last = vec[a.steps & 1];
    for (int i = threadIdx.x; i < n; i += kThreads) a.x[base + i] = a.y[base + i] = last[i];
}

size_t smem_of(int per, int ndiag) { return sizeof(float) * (size_t)per * (ndiag + 2); }

size_t smem_of_rows(int per, int cap) { return sizeof(float) * ((size_t)3 * per + 1 + 2 * (size_t)cap); }

// Shared memory a CTA of these kernels may ask for and its largest cluster on the current device; 0 CTAs: not
// available. Asked, with the kernels' limits raised, for each uploaded matrix (a device reset takes the raised limits back).
struct Limits {
    size_t smem = 0;
    int ctas = 0;
};
Limits raised_limits()
{
    Limits l;
    int device = 0, optin = 0;
    cudaFuncAttributes at{}, at_rows{};
    if (cudaGetDevice(&device) == cudaSuccess &&
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) == cudaSuccess &&
        cudaFuncGetAttributes(&at, k_dia_resident) == cudaSuccess && cudaFuncGetAttributes(&at_rows, k_rows_resident) == cudaSuccess &&
        optin > (int)std::max(at.sharedSizeBytes, at_rows.sharedSizeBytes)) {
        l.smem = (size_t)optin - std::max(at.sharedSizeBytes, at_rows.sharedSizeBytes);
        auto allow = [&](auto k) {
            return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.smem) == cudaSuccess &&
                   cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        };
        if (allow(k_dia_resident) && allow(k_rows_resident)) {
            for (int c = kMaxCtas; c >= 1 && !l.ctas; c /= 2) {
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = c;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3(c);
                cfg.blockDim = dim3(kThreads);
                cfg.dynamicSmemBytes = l.smem;
                cfg.attrs = attr;
                cfg.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, k_dia_resident, &cfg) == cudaSuccess && clusters > 0) l.ctas = c;
            }
        }
    }
    cudaGetLastError();
    return l;
}

// Entries that a CTA holds at most. The cluster has as few CTAs as give each
// one row per thread, more where the values need the room. A step took
// 1.4 us with 1 row per thread and 2.7 with 4 (5 diagonals, 16 CTAs), against 4.0 for a
// launch, and 4.1 with 6: past kEntriesPerCta the launches are the faster way.
constexpr int kEntriesPerCta = 24 * 1024;

template <class K, class A>
int launch_cluster(K kernel, const A& a, int ctas, size_t smem, cudaStream_t st)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int rc = cuda_status(cudaLaunchKernelEx(&cfg, kernel, a));
    return rc ? rc : after_launch(1);
}

int launch(const Args& a, int ctas, cudaStream_t st)
{
    return launch_cluster(k_dia_resident, a, ctas, smem_of(a.per, a.ndiag), st);
}

}  // namespace

// A resident step takes 1.2 us and 0.15 us a diagonal (a run's edge reads it
// from another CTA), a launch's 3.3 us and 0.18 us a diagonal for DIA, 0.31
// us per 4 diagonals of a band for BDIA. So DIA stays to kMaxDiags (150
// diagonals at 2,000 rows, 4 / 40 steps: 33.2 / 31.3 us a step by launches, 33.5 / 23.0
// resident; 250 at 1,200 rows 49 / 48 and 69 / 52), BDIA while diagonals are few for
// their bands (one band of 24, 31, 64 at 2,000 rows, 16 steps: 5.1, 5.7, 8.6
// and 5.1, 6.0, 11.1; nine bands of 3 at 8,000 rows 6.6 and 6.5).
ResidentPlan resident_bdia_plan(int rows, const int* bptr, int nband)
{
    long long quads = 0;
    for (int b = 0; b < nband; b++) quads += (bptr[b + 1] - bptr[b] + 3) / 4;
    const int ndiag = nband > 0 ? bptr[nband] : 0;
    return ndiag <= 11 + 2 * quads ? resident_dia_plan(rows, ndiag) : ResidentPlan{};
}

ResidentPlan resident_dia_plan(int rows, int ndiag)
{
    ResidentPlan p;
    if (rows <= 0 || ndiag < 0 || ndiag > kMaxDiags) return p;
    const Limits l = raised_limits();
    for (int c = 1; c <= l.ctas; c *= 2) {
        const int per = (rows + c - 1) / c;
        if ((per <= kThreads || c == l.ctas) && smem_of(per, ndiag) <= l.smem && (long long)per * ndiag <= kEntriesPerCta) {
            p.ctas = c;
            p.per = per;
            return p;
        }
    }
    return p;
}

int resident_iterate_dia(const clspmv_dia_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st)
{
    return launch(Args{m->matinfo.height, m->matinfo.width, m->dia_num, p.per, m->dia_length_aligned, m->dia_offsets, nullptr, 0,
                       m->dia_data, x, y, alpha, beta, steps}, p.ctas, st);
}

int resident_iterate_bdia(const clspmv_bdia_f32* m, int ndiag, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps,
                          cudaStream_t st)
{
    return launch(Args{m->matinfo.height, m->matinfo.width, ndiag, p.per, m->bdia_length_aligned, m->bdia_offsets, m->bdia_bptr,
                       m->bdia_band_num, m->bdia_data, x, y, alpha, beta, steps}, p.ctas, st);
}

// Rows longer than this keep one thread too long; they stay with the launches.
constexpr int kLongestRow = 64;

// us of a step of one CTA's rows [b, b + n): the barrier, the accesses to its
// own shared memory (a warp's lanes start at their rows' first entries: g of
// them in one bank take g turns), the chain of the longest row of each pass,
// and the reads of other CTAs, whose time goes with the CTAs that a warp's
// lanes read from at once. Fitted to 246 matrices of 200 to 46,000 rows
// (stencils, bands, rows of up to 60 columns near the diagonal or anywhere)
// at 40 steps on B200, 9 % off on average; the chain's share is then taken a
// third higher, which keeps rows of over 30 entries, the ones off by more
// (up to 28 %), on the safe side. CTAs of several passes are estimated from
// every fourth warp, 0.2 ms of an upload of 330k entries.
double rows_step_us(const int* ptr, const int* col, int rows, int per, int b)
{
    const int n = std::min(per, rows - b), skip = n > kThreads ? 4 : 1;
    double turns = 0, slots = 0, chain = 0, others = 0;
    for (int p0 = 0; p0 < n; p0 += kThreads) {
        int pass = 0;
        for (int w0 = p0; w0 < std::min(n, p0 + kThreads); w0 += 32 * skip) {
            const int lanes = std::min(32, n - w0);
            int bank[32] = {}, g = 0, longest = 0;
            unsigned owners[kLongestRow] = {};   // CTAs that the lanes read entry j from; bit 16: past the rows, in global memory
            for (int r = b + w0; r < b + w0 + lanes; r++) {
                const int first = ptr[r], len = ptr[r + 1] - first;
                g = std::max(g, ++bank[(first - ptr[b]) & 31]);
                longest = std::max(longest, len);
                for (int j = 0; j < len; j++) {
                    const int c = col[first + j];
                    if ((unsigned)(c - b) >= (unsigned)per) owners[j] |= 1u << (c < rows ? c / per : kMaxCtas);
                }
            }
            for (int j = 0; j < longest; j++) others += __builtin_popcount(owners[j]);
            turns += (double)longest * g;
            slots += longest;
            pass = std::max(pass, longest);
        }
        chain += pass;
    }
    return 0.7 + 0.055 * chain + skip * (0.0008 * turns + 0.0016 * slots + 0.0065 * others);
}

// A little under what a step by launches takes, replayed: COO's two 4.2-5.8 us, CSR's 5.6-8.3.
constexpr double kCooStep = 4.0, kCsrStep = 5.0;

ResidentPlan resident_rows_plan(int rows, int nnz, const int* row_id, const int* row_ptr, const int* col)
{
    ResidentPlan p;
    if (rows <= 0 || nnz < 0 || (nnz > 0 && ((!row_id && !row_ptr) || !col)) || nnz > kMaxCtas * kEntriesPerCta || rows > kMaxCtas * kEntriesPerCta)
        return p;
    const std::unique_ptr<int[]> ptr(new (std::nothrow) int[(size_t)rows + 1]());
    if (!ptr) return p;
    if (row_id) {
        for (int i = 0; i < nnz; i++) {
            if (row_id[i] < 0 || row_id[i] >= rows || (i > 0 && row_id[i] < row_id[i - 1])) return p;
            ptr[(size_t)row_id[i] + 1]++;
        }
        for (int r = 0; r < rows; r++) ptr[(size_t)r + 1] += ptr[(size_t)r];
    } else {
        std::copy(row_ptr, row_ptr + rows + 1, ptr.get());
    }
    int sign = 0;
    for (int i = 0; i < nnz; i++) sign |= col[i];
    if (sign < 0 || ptr[0] != 0 || ptr[(size_t)rows] > nnz) return p;
    for (int r = 0; r < rows; r++)
        if (ptr[(size_t)r + 1] < ptr[(size_t)r] || ptr[(size_t)r + 1] - ptr[(size_t)r] > kLongestRow) return p;
    const Limits l = raised_limits();
    for (int c = 1; c <= l.ctas; c *= 2) {
        const int per = (rows + c - 1) / c;
        int cap = 0;
        for (int b = 0; b < rows; b += per) cap = std::max(cap, ptr[(size_t)std::min(rows, b + per)] - ptr[(size_t)b]);
        if ((per <= kThreads || c == l.ctas) && per <= 0xffff && smem_of_rows(per, cap) <= l.smem && cap <= kEntriesPerCta) {
            for (int b = 0; b < rows; b += per)
                if (rows_step_us(ptr.get(), col, rows, per, b) > (row_id ? kCooStep : kCsrStep)) return p;
            p.ctas = c;
            p.per = per;
            p.cap = cap;
            return p;
        }
    }
    return p;
}

int resident_iterate_coo(const clspmv_coo_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st)
{
    return launch_cluster(k_rows_resident, RowArgs{m->matinfo.height, m->matinfo.width, m->matinfo.nnz, p.per, p.cap, m->coo_row_id, nullptr,
                                                   m->coo_col_id, m->coo_data, x, y, alpha, beta, steps}, p.ctas, smem_of_rows(p.per, p.cap), st);
}

int resident_iterate_csr(const clspmv_csr_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st)
{
    return launch_cluster(k_rows_resident, RowArgs{m->matinfo.height, m->matinfo.width, m->matinfo.nnz, p.per, p.cap, nullptr, m->csr_row_ptr,
                                                   m->csr_col_id, m->csr_data, x, y, alpha, beta, steps}, p.ctas, smem_of_rows(p.per, p.cap), st);
}

}  // namespace clspmv
