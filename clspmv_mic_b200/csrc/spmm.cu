// spmm.cu — several right-hand sides at once, Y <- alpha * A * X + beta * Y,
// for every device format, with FP32 values or values stored as BF16 / FP16
// (indices untouched, per-row power-of-two scale, FP32 accumulation).
//
// The reference multiplies one vector per call (its kernels read `vec` and
// `result`, e.g. kernels/spmv_ell.cl:4-30). Here X is n x k and Y is m x k,
// both row major with leading dimensions ldx / ldy, k <= 128. Each row of A
// is handled by a group of G lanes that split the k columns between them
// (VEC = 4 columns per lane with 128-bit loads when X / Y rows are 16-byte
// aligned, else 1), so every stored element of A is read once per group and
// multiplies one contiguous row of X. The regular formats (DIA, BDIA, ELL,
// SELL, b4csr, b4ell, SBELL) walk their own layout row by row; CSR and COO
// split the nonzeros into equal runs per warp (power-law rows cost the same
// as short ones; k_spmm_runs).
//
// Reduced-precision storage: clspmv_pack_values converts a device matrix's
// FP32 values in place of a caller-supplied 16-bit array: every value of row
// r is divided by s_r = 2^ceil(log2(max_j |a_rj|)) (exact) before rounding,
// so FP16 keeps its full precision whatever the row's magnitude, and the
// kernels multiply the row sum by s_r.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <cstdlib>
#include <type_traits>
#include <new>
#include "clspmv_b200.h"
#include "api_internal.h"
#include "common.cuh"

using namespace clspmv;

namespace {

constexpr int kSpmmBlock = 256;
constexpr int kSpmmMaxK = 128;

template <class T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }

template <class T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

template <class T> __device__ __forceinline__ T ld_val(const T* p) { return __ldg(p); }

// ---------------------------------------------------------------------------
// Row walks: for_row(m, r, f) calls f(col, idx) for every stored element of
// row r whose column lies inside the matrix, idx indexing the value array.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void for_row(const clspmv_dia_f32& m, int r, F&& f)
{
    const size_t len = (size_t)m.dia_length_aligned;
    for (int d = 0; d < m.dia_num; d++) {
        const int col = r + __ldg(m.dia_offsets + d);
        if (col >= 0 && col < m.matinfo.width) f(col, (size_t)d * len + r);
    }
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_bdia_f32& m, int r, F&& f)
{
    const size_t len = (size_t)m.bdia_length_aligned;
    for (int b = 0; b < m.bdia_band_num; b++) {
        const int i0 = __ldg(m.bdia_bptr + b), i1 = __ldg(m.bdia_bptr + b + 1);
        int col = r + __ldg(m.bdia_offsets + b);
        for (int i = i0; i < i1; i++, col++)
            if (col >= 0 && col < m.matinfo.width) f(col, (size_t)i * len + r);
    }
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_ell_f32& m, int r, F&& f)
{
    const size_t len = (size_t)m.ell_height_aligned;
    for (int s = 0; s < m.ell_num; s++) {
        const size_t idx = (size_t)s * len + r;
        f(__ldg(m.ell_col_id + idx), idx);
    }
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_sell_f32& m, int r, F&& f)
{
    const int sh = (int)m.sell_slice_height;
    const int sl = r / sh;
    const int start = __ldg(m.sell_slice_ptr + sl);
    const int width = (__ldg(m.sell_slice_ptr + sl + 1) - start) / sh;
    for (int s = 0; s < width; s++) {
        const size_t idx = (size_t)start + (size_t)s * sh + (r - sl * sh);
        f(__ldg(m.sell_col_id + idx), idx);
    }
}

// CSR rows for the batched kernel (one group per row; the single-matrix
// path splits CSR by nonzeros instead).
template <class F>
__device__ __forceinline__ void for_row(const clspmv_csr_f32& m, int r, F&& f)
{
    const int j1 = __ldg(m.csr_row_ptr + r + 1);
    for (int j = __ldg(m.csr_row_ptr + r); j < j1; j++) f(__ldg(m.csr_col_id + j), (size_t)j);
}

// Four consecutive columns of one float4 strip of a block (col0 .. col0+3),
// stopping at the matrix width like the reference's serial sbell_spmv.
template <class F>
__device__ __forceinline__ void strip(int col0, size_t idx0, int width, F&& f)
{
#pragma unroll
    for (int w = 0; w < 4; w++)
        if (col0 + w < width) f(col0 + w, idx0 + w);
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_b4csr_f32& m, int r, F&& f)
{
    const int bh = (int)m.b4csr_bheight, bw4 = (int)m.b4csr_bwidth / 4;
    const int br = r / bh, h = r - br * bh;
    const size_t len = (size_t)m.b4csr_aligned_size;
    const int i0 = __ldg(m.b4csr_row_ptr + br), i1 = __ldg(m.b4csr_row_ptr + br + 1);
    for (int i = i0; i < i1; i++) {
        const int c4 = __ldg(m.b4csr_col_id + i);
        for (int w4 = 0; w4 < bw4; w4++)
            strip((c4 + w4) * 4, (size_t)w4 * len * bh + (size_t)h * len + (size_t)i * 4, m.matinfo.width, f);
    }
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_b4ell_f32& m, int r, F&& f)
{
    const int bh = (int)m.b4ell_bheight, bw4 = (int)m.b4ell_bwidth / 4;
    const int br = r / bh, h = r - br * bh;
    const size_t len = (size_t)m.b4ell_height_aligned, f4 = (size_t)m.b4ell_float4_aligned;
    for (int j = 0; j < m.b4ell_block_num; j++) {
        const int c4 = __ldg(m.b4ell_col_id + (size_t)j * len + br);
        for (int w4 = 0; w4 < bw4; w4++)
            strip((c4 + w4) * 4, (size_t)j * f4 * bw4 * bh + (size_t)w4 * f4 * bh + (size_t)h * f4 + (size_t)br * 4,
                  m.matinfo.width, f);
    }
}

template <class F>
__device__ __forceinline__ void for_row(const clspmv_sbell_f32& m, int r, F&& f)
{
    const int bh = (int)m.sbell_bheight, bw4 = (int)m.sbell_bwidth / 4, sh = (int)m.sbell_slice_height;
    const int br = r / bh, h = r - br * bh;
    const int sl = br / sh, s = br - sl * sh;
    const int start = __ldg(m.sbell_slice_ptr + sl);
    const int width = (__ldg(m.sbell_slice_ptr + sl + 1) - start) / sh;
    const size_t base = (size_t)start * bw4 * 4 * bh + (size_t)s * 4;
    for (int j = 0; j < width; j++) {
        const int c4 = __ldg(m.sbell_col_id + (size_t)start + s + (size_t)j * sh);
        for (int w4 = 0; w4 < bw4; w4++)
            strip((c4 + w4) * 4, base + ((size_t)(j * bw4 + w4) * bh + h) * sh * 4, m.matinfo.width, f);
    }
}

// ---------------------------------------------------------------------------
// Lane helpers: a lane owns VEC consecutive columns c0 .. c0+VEC-1 of X / Y.
// ---------------------------------------------------------------------------
template <int VEC> struct Acc;
template <> struct Acc<1> {
    using X = float;
    float v = 0.0f;
    __device__ static X load(const float* x) { return __ldg(x); }
    __device__ static X zero() { return 0.0f; }
    __device__ void fma_v(float a, X xv) { v = fmaf(a, xv, v); }
    __device__ void fma(float a, const float* x) { v = fmaf(a, __ldg(x), v); }
    __device__ void store(float* y, float alpha, float beta) const
    {
        *y = beta == 0.0f ? alpha * v : fmaf(beta, *y, alpha * v);
    }
    __device__ void add(float* y, float alpha) const { *y += alpha * v; }
    __device__ void store_cs(float* y, float alpha, float beta) const
    {
        __stcs(y, beta == 0.0f ? alpha * v : fmaf(beta, *y, alpha * v));
    }
    __device__ void atomic(float* y, float alpha) const { atomicAdd(y, alpha * v); }
};
template <> struct Acc<4> {
    using X = float4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    __device__ static X load(const float* x) { return __ldg(reinterpret_cast<const float4*>(x)); }
    __device__ static X zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ void fma_v(float a, X xv)
    {
        v.x = fmaf(a, xv.x, v.x);
        v.y = fmaf(a, xv.y, v.y);
        v.z = fmaf(a, xv.z, v.z);
        v.w = fmaf(a, xv.w, v.w);
    }
    __device__ void fma(float a, const float* x)
    {
        const float4 xv = __ldg(reinterpret_cast<const float4*>(x));
        v.x = fmaf(a, xv.x, v.x);
        v.y = fmaf(a, xv.y, v.y);
        v.z = fmaf(a, xv.z, v.z);
        v.w = fmaf(a, xv.w, v.w);
    }
    __device__ void store(float* y, float alpha, float beta) const
    {
        float4 o = make_float4(alpha * v.x, alpha * v.y, alpha * v.z, alpha * v.w);
        if (beta != 0.0f) {
            const float4 p = *reinterpret_cast<const float4*>(y);
            o.x = fmaf(beta, p.x, o.x);
            o.y = fmaf(beta, p.y, o.y);
            o.z = fmaf(beta, p.z, o.z);
            o.w = fmaf(beta, p.w, o.w);
        }
        *reinterpret_cast<float4*>(y) = o;
    }
    __device__ void add(float* y, float alpha) const
    {
        float4 p = *reinterpret_cast<float4*>(y);
        p.x += alpha * v.x;
        p.y += alpha * v.y;
        p.z += alpha * v.z;
        p.w += alpha * v.w;
        *reinterpret_cast<float4*>(y) = p;
    }
    __device__ void store_cs(float* y, float alpha, float beta) const { store(y, alpha, beta); }
    __device__ void atomic(float* y, float alpha) const
    {
        atomicAdd(reinterpret_cast<float4*>(y), make_float4(alpha * v.x, alpha * v.y, alpha * v.z, alpha * v.w));
    }
};

struct Dense {
    int k;
    const float* X;
    int ldx;
    float* Y;
    int ldy;
    float alpha, beta;
    const float* scale;   // per-row scale of packed values, or nullptr
    int lshift;           // log2 of lanes per row group
    int x_form;           // block-row kernel: X rows through L1 (0), with an L2 evict-last hint (1), past L1 (2)
};

// Row-walk kernel: one group of 2^lshift lanes per row, grid-stride over rows.
template <int VEC, class T, class M>
__global__ void __launch_bounds__(kSpmmBlock) k_spmm_rows(M m, const T* __restrict__ vals, Dense d)
{
    const int G = 1 << d.lshift;
    const long long t = (long long)blockIdx.x * kSpmmBlock + threadIdx.x;
    const int lane = (int)(t & (G - 1));
    const int c0 = lane * VEC;
    if (c0 >= d.k) return;                      // lanes past k have no columns
    const long long groups = ((long long)gridDim.x * kSpmmBlock) >> d.lshift;
    for (long long r = t >> d.lshift; r < m.matinfo.height; r += groups) {
        Acc<VEC> acc;
        for_row(m, (int)r, [&](int col, size_t idx) { acc.fma(to_f(ld_val(vals + idx)), d.X + (size_t)col * d.ldx + c0); });
        const float a = d.scale ? d.alpha * d.scale[r] : d.alpha;
        acc.store(d.Y + (size_t)r * d.ldy + c0, a, d.beta);
    }
}

// Row r of ELL and SELL: where its slot 0 lies, the step to the next, their number.
__device__ __forceinline__ void slot_row(const clspmv_ell_f32& m, long long r, size_t& at, int& step, int& n)
{
    at = (size_t)r;
    step = m.ell_height_aligned;
    n = m.ell_num;
}
__device__ __forceinline__ void slot_row(const clspmv_sell_f32& m, long long r, size_t& at, int& step, int& n)
{
    const int sh = (int)m.sell_slice_height, sl = (int)r / sh, start = __ldg(m.sell_slice_ptr + sl);
    at = (size_t)start + (r - (long long)sl * sh);
    step = sh;
    n = (__ldg(m.sell_slice_ptr + sl + 1) - start) / sh;
}
__device__ __forceinline__ const int* cols_of(const clspmv_ell_f32& m) { return m.ell_col_id; }
__device__ __forceinline__ const int* cols_of(const clspmv_sell_f32& m) { return m.sell_col_id; }

// SELL and 16-bit ELL rows of kSlotLoads slots and more: a group per row as in
// the row walk, with the column ids, values and X rows of kSlotLoads slots in
// flight together. The time follows the X loads in flight per SM: 8 a lane at
// 32 warps. The row walk has 4 a lane at 64 warps for FP32 ELL, which keeps
// it, but fewer for 16-bit values and one for SELL, whose slot count the
// compiler does not see; short rows keep it too. Slots are summed in the same order.
// B200, 27-point stencil of 101^3, us at k = 8 / 16 / 64: SELL 184 / 329 /
// 1180 -> 95 / 170 / 613, ELL with BF16 values 120 / 218 / 795 -> 92 / 166 /
// 597; SELL of the power law of 2^20 rows at k = 8 7.2 -> 2.1 ms.
constexpr int kSlotLoads = 8;
template <int VEC, class T, class M>
__global__ void __launch_bounds__(kSpmmBlock, 4) k_spmm_slots(M m, const T* __restrict__ vals, Dense d)
{
    constexpr int U = kSlotLoads;
    const int G = 1 << d.lshift;
    const long long t = (long long)blockIdx.x * kSpmmBlock + threadIdx.x;
    const int c0 = (int)(t & (G - 1)) * VEC;
    if (c0 >= d.k) return;
    const float* __restrict__ X = d.X + c0;
    const long long groups = ((long long)gridDim.x * kSpmmBlock) >> d.lshift;
    for (long long r = t >> d.lshift; r < m.matinfo.height; r += groups) {
        size_t at;
        int step, n;
        slot_row(m, r, at, step, n);
        const int* cp = cols_of(m) + at;
        const T* vp = vals + at;
        Acc<VEC> acc;
        int i = 0;
        auto batch = [&](auto count) {
            constexpr int N = decltype(count)::value;
            int c[N];
            float v[N];
            typename Acc<VEC>::X x[N];
#pragma unroll
            for (int u = 0; u < N; u++, cp += step, vp += step) {
                c[u] = __ldg(cp);
                v[u] = to_f(__ldg(vp));
            }
#pragma unroll
            for (int u = 0; u < N; u++) x[u] = Acc<VEC>::load(X + (size_t)c[u] * d.ldx);
#pragma unroll
            for (int u = 0; u < N; u++) acc.fma_v(v[u], x[u]);
            i += N;
        };
        while (i + U <= n) batch(std::integral_constant<int, U>{});
        if (i + U / 2 <= n) batch(std::integral_constant<int, U / 2>{});
        while (i < n) batch(std::integral_constant<int, 1>{});
        acc.store(d.Y + (size_t)r * d.ldy + c0, d.scale ? d.alpha * d.scale[r] : d.alpha, d.beta);
    }
}

// ---------------------------------------------------------------------------
// Block walks: for_block(m, br, f) calls f(c4, base, s4, sh) for every stored
// block of block row br. The block's first column is 4 * c4; the value of its
// row h, column 4 * w4 + w sits at base + w4 * s4 + h * sh + w, so each
// (w4, h) strip is 4 consecutive values. Same addressing as for_row.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ void for_block(const clspmv_b4csr_f32& m, int br, F&& f)
{
    const size_t len = (size_t)m.b4csr_aligned_size, bh = m.b4csr_bheight;
    const int i1 = __ldg(m.b4csr_row_ptr + br + 1);
    for (int i = __ldg(m.b4csr_row_ptr + br); i < i1; i++) f(__ldg(m.b4csr_col_id + i), (size_t)i * 4, len * bh, len);
}

template <class F>
__device__ __forceinline__ void for_block(const clspmv_b4ell_f32& m, int br, F&& f)
{
    const size_t len = (size_t)m.b4ell_height_aligned, f4 = (size_t)m.b4ell_float4_aligned;
    const size_t bh = m.b4ell_bheight, bw4 = m.b4ell_bwidth / 4;
    for (int j = 0; j < m.b4ell_block_num; j++)
        f(__ldg(m.b4ell_col_id + (size_t)j * len + br), (size_t)j * f4 * bw4 * bh + (size_t)br * 4, f4 * bh, f4);
}

template <class F>
__device__ __forceinline__ void for_block(const clspmv_sbell_f32& m, int br, F&& f)
{
    const size_t bh = m.sbell_bheight, bw4 = m.sbell_bwidth / 4, sh = m.sbell_slice_height;
    const int sl = (int)(br / sh), s = br - sl * (int)sh;
    const int start = __ldg(m.sbell_slice_ptr + sl);
    const int width = (__ldg(m.sbell_slice_ptr + sl + 1) - start) / (int)sh;
    const size_t base = (size_t)start * bw4 * 4 * bh + (size_t)s * 4;
    for (int j = 0; j < width; j++)
        f(__ldg(m.sbell_col_id + (size_t)start + s + (size_t)j * sh), base + (size_t)j * bw4 * bh * sh * 4, bh * sh * 4,
          sh * 4);
}

// 4 consecutive values of a block strip. b4csr keeps a block row's blocks
// side by side (block i at 4 * i in each (w4, h) plane), so a group's next
// blocks share the line of this one: those loads allocate in L1 and carry no
// evict-first hint, so that the line is still in L2 when L1 has lost it. In
// b4ell and SBELL the neighbouring groups (block rows) read the rest of the
// line in the same instruction, and the loads stream past L1.
template <class M> struct StripsInL1 { static constexpr bool value = false; };
__device__ __forceinline__ float4 ld_x4_na(const float* p)
{
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
template <> struct StripsInL1<clspmv_b4csr_f32> { static constexpr bool value = true; };

__device__ __forceinline__ uint2 ld_l1_u2(const void* p) { return __ldg(reinterpret_cast<const uint2*>(p)); }
template <bool L1> __device__ __forceinline__ float4 strip4(const float* p, uint64_t pol)
{
    return L1 ? __ldg(reinterpret_cast<const float4*>(p)) : ld_stream_f4(p, pol);
}
template <bool L1> __device__ __forceinline__ float4 strip4(const __nv_bfloat16* p, uint64_t pol)
{
    const uint2 u = L1 ? ld_l1_u2(p) : ld_stream_u2(p, pol);
    return make_float4(bf16_lo(u.x), bf16_hi(u.x), bf16_lo(u.y), bf16_hi(u.y));
}
template <bool L1> __device__ __forceinline__ float4 strip4(const __half* p, uint64_t pol)
{
    const uint2 u = L1 ? ld_l1_u2(p) : ld_stream_u2(p, pol);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ float4 load_x(const float* p, int form, uint64_t pol)
{
    return form == 0 ? __ldg(reinterpret_cast<const float4*>(p)) : form == 1 ? ld_x4(p, pol) : ld_x4_na(p);
}

// One block row of the block-row kernel: the group's lane holds columns
// c0 .. c0+3 of all BH rows of Y. A block's 4 x 4 slice of X is loaded once
// (the 4 X rows in flight together) and multiplies its BH rows from registers
// (the row walk loads it once per row), and each (w4, h) strip of values is
// one 4-value load. Every row accumulates in the same order as the row walk
// (block, strip, column), so the two give the same bits.
template <int BH, int BW4, class T, class M>
__device__ __forceinline__ void block_row(const M& m, const T* __restrict__ vals, int br, int c0, const float* __restrict__ X,
                                          int ldx, float* __restrict__ Y, int ldy, float alpha, float beta,
                                          const float* __restrict__ scale, int x_form)
{
    const int height = m.matinfo.height, width = m.matinfo.width;
    const uint64_t pol = policy_evict_first(), xpol = policy_evict_last();
    Acc<4> acc[BH];
    for_block(m, br, [&](int c4, size_t base, size_t s4, size_t sh) {
#pragma unroll
        for (int w4 = 0; w4 < BW4; w4++) {
            float4 a[BH];
#pragma unroll
            for (int h = 0; h < BH; h++)
                a[h] = strip4<StripsInL1<M>::value>(vals + base + (size_t)w4 * s4 + (size_t)h * sh, pol);
            const int col0 = (c4 + w4) * 4;
            const int ncol = min(4, width - col0);   // the reference stops a block at the matrix width
            float4 xv[4];
            if (ncol == 4) {                         // the 4 X rows in flight together
#pragma unroll
                for (int w = 0; w < 4; w++) xv[w] = load_x(X + (size_t)(col0 + w) * ldx + c0, x_form, xpol);
            } else {
#pragma unroll
                for (int w = 0; w < 4; w++)
                    xv[w] = w < ncol ? load_x(X + (size_t)(col0 + w) * ldx + c0, x_form, xpol) : Acc<4>::zero();
            }
#pragma unroll
            for (int w = 0; w < 4; w++) {
                if (w >= ncol) break;
#pragma unroll
                for (int h = 0; h < BH; h++) {
                    const float av = w == 0 ? a[h].x : w == 1 ? a[h].y : w == 2 ? a[h].z : a[h].w;
                    acc[h].fma_v(av, xv[w]);
                }
            }
        }
    });
#pragma unroll
    for (int h = 0; h < BH; h++) {
        const long long r = (long long)br * BH + h;
        if (r >= height) break;
        const float al = scale ? alpha * scale[r] : alpha;
        acc[h].store(Y + (size_t)r * ldy + c0, al, beta);
    }
}

// Block-row kernel for the 4-wide block formats: one group of 2^lshift lanes
// per BH-high block row (block_row), grid-stride over block rows.
template <int BH, int BW4, class T, class M>
__global__ void __launch_bounds__(kSpmmBlock, BH >= 8 ? 1 : 4) k_spmm_blocks(M m, const T* __restrict__ vals, Dense d)
{
    const long long t = (long long)blockIdx.x * kSpmmBlock + threadIdx.x;
    const int c0 = (int)(t & ((1 << d.lshift) - 1)) * 4;
    if (c0 >= d.k) return;
    const long long groups = ((long long)gridDim.x * kSpmmBlock) >> d.lshift;
    const long long nbr = ((long long)m.matinfo.height + BH - 1) / BH;
    for (long long br = t >> d.lshift; br < nbr; br += groups)
        block_row<BH, BW4>(m, vals, (int)br, c0, d.X, d.ldx, d.Y, d.ldy, d.alpha, d.beta, d.scale, d.x_form);
}

constexpr unsigned kWarpAll = 0xffffffffu;
constexpr int kSegNoRow = 0x7fffffff;

__device__ __forceinline__ float4 f4add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 f4up(float4 v, int off)
{
    return make_float4(__shfl_up_sync(kWarpAll, v.x, off), __shfl_up_sync(kWarpAll, v.y, off),
                       __shfl_up_sync(kWarpAll, v.z, off), __shfl_up_sync(kWarpAll, v.w, off));
}
// Largest r in [0, rows) with row_ptr[r] <= q (q < nnz), by the whole warp:
// each round the 32 lanes probe 32 evenly spaced rows of the interval.
__device__ __forceinline__ int warp_row_of(const int* __restrict__ row_ptr, int rows, long long q, int lane)
{
    int lo = 0, hi = rows - 1;   // invariant: row_ptr[lo] <= q
    while (hi - lo >= 32) {
        const long long span = (long long)hi - lo;
        const int p = lo + (int)(span * lane / 32);
        const unsigned m = __ballot_sync(kWarpAll, __ldg(row_ptr + p) <= q);
        const int j = 31 - __clz(m);
        const int nlo = __shfl_sync(kWarpAll, p, j);
        const int next = __shfl_sync(kWarpAll, p, j < 31 ? j + 1 : 31);
        hi = j < 31 ? next - 1 : hi;
        lo = nlo;
    }
    const int p = lo + lane;
    const unsigned m = __ballot_sync(kWarpAll, p <= hi && __ldg(row_ptr + min(p, hi)) <= q);
    return lo + (31 - __clz(m));
}

// ---------------------------------------------------------------------------
// Long CSR rows at k a multiple of 4: a warp per row. The warp's lanes form
// 32 / G nonzero slots of G = k / 4 lanes (4 columns each); a step covers
// 32 / G consecutive nonzeros of the row with coalesced col_id / value loads
// and one float4 X load per lane, and the slots' partial sums are combined
// once per row by shuffles. The row is owned by its warp, so Y is written
// directly (alpha, beta applied there). Used when rows average
// kWarpRowMin nonzeros or more.
// ---------------------------------------------------------------------------
constexpr int kWarpRowMin = 128;

template <class T>
__global__ void __launch_bounds__(kSpmmBlock) k_spmm_warp_rows(int rows, const int* __restrict__ row_ptr,
                                                               const int* __restrict__ col_id, const T* __restrict__ vals,
                                                               Dense d)
{
    const int lane = threadIdx.x & 31;
    const int G = d.k >> 2;                     // lanes per nonzero slot, 1..32 (k <= 128)
    const int lg = 31 - __clz(G);               // G is a power of two (checked by the launcher)
    const int slots = 32 >> lg;
    const int slot = lane >> lg, c0 = (lane & (G - 1)) * 4;
    const long long nwarps = (long long)gridDim.x * (kSpmmBlock / 32);
    for (long long r = (long long)blockIdx.x * (kSpmmBlock / 32) + (threadIdx.x >> 5); r < rows; r += nwarps) {
        const int j0 = __ldg(row_ptr + r), j1 = __ldg(row_ptr + r + 1);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        int j = j0 + slot;
        // two nonzeros per slot in flight
        for (; j + slots < j1; j += 2 * slots) {
            const int ca = __ldg(col_id + j), cb = __ldg(col_id + j + slots);
            const float va = to_f(ld_val(vals + j)), vb = to_f(ld_val(vals + j + slots));
            const float4 xa = __ldg(reinterpret_cast<const float4*>(d.X + (size_t)ca * d.ldx + c0));
            const float4 xb = __ldg(reinterpret_cast<const float4*>(d.X + (size_t)cb * d.ldx + c0));
            acc.x = fmaf(va, xa.x, acc.x); acc.y = fmaf(va, xa.y, acc.y);
            acc.z = fmaf(va, xa.z, acc.z); acc.w = fmaf(va, xa.w, acc.w);
            acc.x = fmaf(vb, xb.x, acc.x); acc.y = fmaf(vb, xb.y, acc.y);
            acc.z = fmaf(vb, xb.z, acc.z); acc.w = fmaf(vb, xb.w, acc.w);
        }
        if (j < j1) {
            const int ca = __ldg(col_id + j);
            const float va = to_f(ld_val(vals + j));
            const float4 xa = __ldg(reinterpret_cast<const float4*>(d.X + (size_t)ca * d.ldx + c0));
            acc.x = fmaf(va, xa.x, acc.x); acc.y = fmaf(va, xa.y, acc.y);
            acc.z = fmaf(va, xa.z, acc.z); acc.w = fmaf(va, xa.w, acc.w);
        }
        for (int off = 16; off >= G; off >>= 1) {
            acc.x += __shfl_xor_sync(kWarpAll, acc.x, off);
            acc.y += __shfl_xor_sync(kWarpAll, acc.y, off);
            acc.z += __shfl_xor_sync(kWarpAll, acc.z, off);
            acc.w += __shfl_xor_sync(kWarpAll, acc.w, off);
        }
        if (slot == 0) {
            const float a = d.scale ? d.alpha * d.scale[r] : d.alpha;
            float4* y = reinterpret_cast<float4*>(d.Y + (size_t)r * d.ldy + c0);
            float4 o = make_float4(a * acc.x, a * acc.y, a * acc.z, a * acc.w);
            if (d.beta != 0.0f) {
                const float4 p = *y;
                o.x = fmaf(d.beta, p.x, o.x); o.y = fmaf(d.beta, p.y, o.y);
                o.z = fmaf(d.beta, p.z, o.z); o.w = fmaf(d.beta, p.w, o.w);
            }
            *y = o;
        }
    }
}

// ---------------------------------------------------------------------------
// CSR / COO by warp runs. A warp takes 32 P consecutive nonzeros, P per lane
// with 128-bit loads, finds the row of each (CSR: from row_ptr), and splits
// its lanes into slots of G = 2^LG lanes that share the k columns of X and Y
// (VEC columns a lane), or those of the block's panel (blockIdx.y) where few
// nonzeros are worth more warps than that. A slot owns the P G nonzeros that
// its lanes loaded and hands them round by shuffles, with kRunLoads X rows in
// flight: ids, values and rows are read once, coalesced, and no lane waits for
// row_ptr between two nonzeros.
//
// A CSR row that starts and ends in its warp's run is written directly
// (alpha, beta), its pieces in several slots summed by a segmented scan, so
// Y gets no scaling pass of its own. Only rows cut by an edge between warps
// are added atomically, after k_scale_cut has applied beta to those and to
// the rows without entries. With ADD (beta = 1, or Y scaled before) every row
// is added: a row that reads its Y would wait for it. COO has no row pointer to tell them by: beta is
// applied to all of Y first and every row is added, by red.global.add, which
// a slot does not wait for.
//
// Measured on B200 (us, CSR, FP32; before: 16 nonzeros per lane group, a
// search of row_ptr for each, Y zeroed first and every row read, added and
// written): power law of 2^20 rows, k = 4 / 16 / 32: 187 / 327 / 568 -> 103 /
// 198 / 344; 27-point stencil of 100^3: 268 / 378 / 623 -> 122 / 253 / 424.
// At k = 16 on the power law it moves its 1.04 GB of X rows at 5.3 TB/s (X is
// 64 MB: L2 hits 58 %), at k = 64 DRAM carries 3.5 GB at 0.87 of the copy rate. Also measured, not
// kept: rows walked within equal ranges of nonzeros, several slots a row
// (358 us at k = 16 on the power law), ends of rows written without a branch
// (280), evict-last X or streaming Y (within 3 %), 3 CTAs per SM (198).
// ---------------------------------------------------------------------------
constexpr int kRunLoads = 4;

// beta to the rows that an edge between warp runs of 2^lrun nonzeros cuts, and to rows without entries: a warp looks at
// 32 rows, a lane each, and groups of 2^lshift lanes write the ones that need it. A thread per row at every k wrote 32
// lines a store: with 9 of 10 of 2^20 rows empty 872 us of a product at k = 128, 433 at k = 64, 100 at k = 16 (beta 0),
// against 178, 104 and 48. It stays for fewer than 8 single columns (lshift 0: 4M rows, 1 of 50 with entries, k = 5: 61
// us, 70 with 8 lanes a row).
template <int VEC>
__global__ void __launch_bounds__(kSpmmBlock) k_scale_cut(int rows, const int* __restrict__ row_ptr, int lrun, int lshift, Dense d)
{
    const int lane = threadIdx.x & 31, G = 1 << lshift, slot = lane >> lshift, c0 = (lane & (G - 1)) * VEC;
    const unsigned slots = lshift == 0 ? kWarpAll : (1u << (32 >> lshift)) - 1;
    const long long nwarps = (long long)gridDim.x * (kSpmmBlock / 32);
    for (long long r0 = ((long long)blockIdx.x * (kSpmmBlock / 32) + (threadIdx.x >> 5)) * 32; r0 < rows; r0 += nwarps * 32) {
        bool need = false;
        if (r0 + lane < rows) {
            const int s = __ldg(row_ptr + r0 + lane), e = __ldg(row_ptr + r0 + lane + 1);
            need = s >= e || s >> lrun != (e - 1) >> lrun;
        }
        if (VEC == 1 && lshift == 0) {
            float* y = d.Y + (size_t)(r0 + lane) * d.ldy;
            if (need)
                for (int j = 0; j < d.k; j++) y[j] = d.beta == 0.0f ? 0.0f : d.beta * y[j];
            continue;
        }
        const unsigned mask = __ballot_sync(kWarpAll, need);
        if (!mask) continue;
#pragma unroll 4
        for (int i = 0; i < 32; i += 32 >> lshift) {
            if (!(mask >> i & slots)) continue;
            if (!(mask >> (i + slot) & 1)) continue;
            float* y = d.Y + (size_t)(r0 + i + slot) * d.ldy;
            for (int c = c0; c < d.k; c += G * VEC) {
                if (VEC == 4) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (d.beta != 0.0f) {
                        v = *reinterpret_cast<const float4*>(y + c);
                        v = make_float4(d.beta * v.x, d.beta * v.y, d.beta * v.z, d.beta * v.w);
                    }
                    *reinterpret_cast<float4*>(y + c) = v;
                } else {
                    y[c] = d.beta == 0.0f ? 0.0f : d.beta * y[c];
                }
            }
        }
    }
}

// The row that holds nonzero e, the current row having ended at or before it.
__device__ __forceinline__ int next_row(const int* __restrict__ row_ptr, int rows, int row, int e)
{
    for (int i = 0; i < 8; i++) {
        row++;
        if (__ldg(row_ptr + row + 1) > e) return row;
    }
    int lo = row + 1, hi = rows - 1;   // many rows without entries: the largest row that starts at or before e
    while (lo < hi) {
        const int mid = lo + ((hi - lo + 1) >> 1);
        if (__ldg(row_ptr + mid) <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Rows of a lane's P nonzeros from q0 on (kSegNoRow past the last one), q0 in [base, ...), ra the
// row of base. The rows of most runs lie within 256 of ra: every eighth of
// those row pointers is held by one lane, so a lane searches by shuffles and
// then among 8. Otherwise it searches up to the last row.
template <int P>
__device__ __forceinline__ void rows_of(const int* __restrict__ row_ptr, int rows, int ra, long long q0, int end, int lane, int (&r)[P])
{
    const int probe = min((long long)ra + 8 * lane, (long long)rows);   // row_ptr[rows] = nnz is past every q
    const int pv = __ldg(row_ptr + probe);
    const bool near = __shfl_sync(kWarpAll, pv, 31) >= end;   // the rows of the run end before the last probe
    const long long q = min(q0, (long long)end - 1);
    int lo, hi;
    if (near) {
        int j = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const int v = __shfl_sync(kWarpAll, pv, j + s);
            if (v <= q) j += s;
        }
        lo = ra + 8 * j;
        hi = min(lo + 7, rows - 1);
    } else {
        lo = ra;
        hi = rows - 1;
    }
    while (lo < hi) {
        const int mid = lo + ((hi - lo + 1) >> 1);
        if (__ldg(row_ptr + mid) <= q) lo = mid;
        else hi = mid - 1;
    }
    int row = lo, next = __ldg(row_ptr + row + 1);
#pragma unroll
    for (int j = 0; j < P; j++) {
        const long long e = q0 + j;
        if (e < end) {
            if (e >= next) {
                row = next_row(row_ptr, rows, row, (int)e);
                next = __ldg(row_ptr + row + 1);
            }
            r[j] = row;
        } else {
            r[j] = kSegNoRow;
        }
    }
}

template <class T, int P>
__device__ __forceinline__ void load_run(const T* __restrict__ p, long long i, int nnz, bool vec, float (&v)[P])
{
    if (vec && i + P <= nnz) {
        if constexpr (std::is_same<T, float>::value) {
#pragma unroll
            for (int j = 0; j < P; j += 4) {
                const float4 f = __ldcs(reinterpret_cast<const float4*>(p + i + j));
                v[j] = f.x; v[j + 1] = f.y; v[j + 2] = f.z; v[j + 3] = f.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < P; j += 4) {
                const uint2 u = __ldcs(reinterpret_cast<const uint2*>(p + i + j));
                const T* t = reinterpret_cast<const T*>(&u);
#pragma unroll
                for (int q = 0; q < 4; q++) v[j + q] = to_f(t[q]);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < P; j++) v[j] = i + j < nnz ? to_f(ld_val(p + i + j)) : 0.f;
    }
}
template <int P>
__device__ __forceinline__ void load_ids(const int* __restrict__ p, long long i, int nnz, bool vec, int (&c)[P])
{
    if (vec && i + P <= nnz) {
#pragma unroll
        for (int j = 0; j < P; j += 4) {
            const int4 f = __ldcs(reinterpret_cast<const int4*>(p + i + j));
            c[j] = f.x; c[j + 1] = f.y; c[j + 2] = f.z; c[j + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < P; j++) c[j] = i + j < nnz ? __ldg(p + i + j) : 0;
    }
}

__device__ __forceinline__ float shfl_up_x(float v, int o) { return __shfl_up_sync(kWarpAll, v, o); }
__device__ __forceinline__ float4 shfl_up_x(float4 v, int o) { return f4up(v, o); }
__device__ __forceinline__ float x_add(float a, float b) { return a + b; }
__device__ __forceinline__ float4 x_add(float4 a, float4 b) { return f4add(a, b); }

template <int LG, int VEC, int P, class T, bool IS_CSR, bool ADD>
__global__ void __launch_bounds__(kSpmmBlock, 4) k_spmm_runs(int rows, int nnz, const int* __restrict__ row_ptr,
                                                             const int* __restrict__ row_id, const int* __restrict__ col_id,
                                                             const T* __restrict__ vals, bool vec, int per, Dense d)
{
    constexpr int G = 1 << LG, kRun = 32 * P, U = kRunLoads;
    static_assert(P % U == 0, "a batch of X rows stays within a lane's nonzeros");
    using XT = typename Acc<VEC>::X;
    const int lane = threadIdx.x & 31, slot = lane >> LG;
    const int c0 = ((P == 4 ? (int)blockIdx.y * G : 0) + (lane & (G - 1))) * VEC;   // panels only for few nonzeros (P = 4)
    const bool cols = c0 < d.k;
    const float* __restrict__ X = d.X + (cols ? c0 : 0);
    float* const Y = d.Y + c0;
    // `per` consecutive runs per warp: the row of the next run's start is found from this one's
    const long long w0 = ((long long)blockIdx.x * (kSpmmBlock / 32) + (threadIdx.x >> 5)) * per;
    int ra = 0;
    if (IS_CSR && w0 * kRun < nnz) ra = warp_row_of(row_ptr, rows, w0 * kRun, lane);
    for (long long w = w0; w < w0 + per && w * kRun < nnz; w++) {
        const int base = (int)(w * kRun), end = (int)min((long long)nnz, (w + 1) * kRun);
        const long long q0 = base + (long long)lane * P;
        int cc[P], rr[P];
        float vv[P];
        load_ids<P>(col_id, q0, nnz, vec, cc);
        load_run<T, P>(vals, q0, nnz, vec, vv);
        if (IS_CSR) {
            rows_of<P>(row_ptr, rows, ra, q0, end, lane, rr);
        } else {
            load_ids<P>(row_id, q0, nnz, vec, rr);
#pragma unroll
            for (int j = 0; j < P; j++)
                if (q0 + j >= nnz) rr[j] = kSegNoRow;
        }
        // the rows of the nonzeros before and after the slot's
        int before = __shfl_up_sync(kWarpAll, rr[P - 1], 1), after = __shfl_down_sync(kWarpAll, rr[0], 1);
        if (IS_CSR) {
            if (lane == 0) before = __ldg(row_ptr + ra) < base ? ra : -1;
            if (lane == 31) after = rr[P - 1] != kSegNoRow && __ldg(row_ptr + rr[P - 1] + 1) > end ? rr[P - 1] : kSegNoRow;
        } else {
            if (lane == 0) before = base > 0 ? __ldg(row_id + base - 1) : -1;
            if (lane == 31) after = end < nnz ? __ldg(row_id + end) : kSegNoRow;
        }
        const int base_row = __shfl_sync(kWarpAll, before, 0);   // the row that came from before the warp, if any
        before = __shfl_sync(kWarpAll, before, 0, G);
        after = __shfl_sync(kWarpAll, after, G - 1, G);
        int row = __shfl_sync(kWarpAll, rr[0], 0, G);
        bool cut = row == before;    // the current row's sum is a piece
        int head_row = -1;
        Acc<VEC> acc, first;         // first: the piece of the row that the slot starts in, once that row has ended
        auto put = [&](const Acc<VEC>& s, int r, bool whole) {
            float a = d.alpha;
            if (!std::is_same<T, float>::value) a *= d.scale[r];
            float* y = Y + (size_t)r * d.ldy;
            if (ADD || !whole) s.atomic(y, a);
            else if (VEC == 1) s.store_cs(y, a, d.beta);
            else s.store(y, a, d.beta);
        };
        auto row_done = [&]() {
            if (cut) {
                first = acc;
                head_row = row;
                cut = false;
            } else if (cols) {
                put(acc, row, true);
            }
            acc = Acc<VEC>();
        };
#pragma unroll 1
        for (int src = 0; src < G; src++) {
#pragma unroll
            for (int h = 0; h < P; h += U) {
                float av[U];
                int rv[U];
                XT xv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int c = G == 1 ? cc[h + u] : __shfl_sync(kWarpAll, cc[h + u], src, G);
                    av[u] = G == 1 ? vv[h + u] : __shfl_sync(kWarpAll, vv[h + u], src, G);
                    rv[u] = G == 1 ? rr[h + u] : __shfl_sync(kWarpAll, rr[h + u], src, G);
                    xv[u] = cols && rv[u] != kSegNoRow ? Acc<VEC>::load(X + (size_t)c * d.ldx) : Acc<VEC>::zero();
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (rv[u] != row) {
                        row_done();
                        row = rv[u];
                        if (row == kSegNoRow) cut = true;   // past the last nonzero: nothing is written from here on
                    }
                    acc.fma_v(av[u], xv[u]);
                }
            }
        }
        // the slot's last row: done here, or continued in the next slot
        const bool live = row != kSegNoRow, more = live && row == after;
        if (live && !more) row_done();
        // pieces, in slot order: a slot inside one row hands the sum on (through), others start a new one with their last row's piece
        const bool through = more && cut;
        XT v = more ? acc.v : Acc<VEC>::zero();
        const unsigned upto = __ballot_sync(kWarpAll, !through) & (0xffffffffu >> (31 - lane));
        const int seg0 = upto ? (31 - __clz(upto)) & ~(G - 1) : 0;   // first lane of the slot where this slot's sum starts
#pragma unroll
        for (int o = G; o < 32; o <<= 1) {
            const XT t = shfl_up_x(v, o);
            if (lane - o >= seg0) v = x_add(v, t);
        }
        XT pv = v;
        if (G < 32) pv = shfl_up_x(v, G);
        if (head_row >= 0 && head_row != kSegNoRow && cols) {   // a row that came from before ends in this slot
            if (slot > 0) first.v = x_add(first.v, pv);
            put(first, head_row, head_row != base_row);
        }
        if (more && lane >= 32 - G && cols) {                   // a row that goes on in the next warp's run
            acc.v = v;
            put(acc, row, false);
        }
        if (IS_CSR) ra = __shfl_sync(kWarpAll, after != kSegNoRow ? after : row, 31);
        if (IS_CSR && end < nnz && __shfl_sync(kWarpAll, after, 31) == kSegNoRow) ra = next_row(row_ptr, rows, ra, end);
    }
}

__global__ void k_scale_rows(float* Y, int rows, int k, int ldy, float beta)
{
    const long long n = (long long)rows * k;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / k, c = i - r * k;
        float* p = Y + r * ldy + c;
        *p = beta == 0.0f ? 0.0f : beta * *p;
    }
}

// Packing: per-row scale (pass 1), then the scaled 16-bit values (pass 2).
__device__ __forceinline__ float pow2_at_least(float s)
{
    if (!(s > 0.0f) || isinf(s)) return 1.0f;
    int e;
    const float f = frexpf(s, &e);   // s = f * 2^e, f in [0.5, 1)
    (void)f;
    return ldexpf(1.0f, e);
}

template <class T, class M>
__global__ void k_pack_rows(M m, const float* __restrict__ src, T* __restrict__ dst, float* __restrict__ scale)
{
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < m.matinfo.height;
         r += (long long)gridDim.x * blockDim.x) {
        float mx = 0.0f;
        for_row(m, (int)r, [&](int, size_t idx) { mx = fmaxf(mx, fabsf(src[idx])); });
        const float s = pow2_at_least(mx), inv = 1.0f / s;   // exact: s is a power of two
        scale[r] = s;
        for_row(m, (int)r, [&](int, size_t idx) { dst[idx] = from_f<T>(src[idx] * inv); });
    }
}

template <class T>
__global__ void k_pack_csr(int rows, const int* __restrict__ row_ptr, const float* __restrict__ src, T* __restrict__ dst,
                           float* __restrict__ scale)
{
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (long long)gridDim.x * blockDim.x) {
        const int a = row_ptr[r], b = row_ptr[r + 1];
        float mx = 0.0f;
        for (int j = a; j < b; j++) mx = fmaxf(mx, fabsf(src[j]));
        const float s = pow2_at_least(mx), inv = 1.0f / s;
        scale[r] = s;
        for (int j = a; j < b; j++) dst[j] = from_f<T>(src[j] * inv);
    }
}

// COO rows are runs of equal row ids: the thread at the start of a run packs it.
template <class T>
__global__ void k_pack_coo(int nnz, const int* __restrict__ row_id, const float* __restrict__ src, T* __restrict__ dst,
                           float* __restrict__ scale)
{
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (long long)gridDim.x * blockDim.x) {
        const int r = row_id[e];
        if (e > 0 && row_id[e - 1] == r) continue;
        long long f = e;
        float mx = 0.0f;
        for (; f < nnz && row_id[f] == r; f++) mx = fmaxf(mx, fabsf(src[f]));
        const float s = pow2_at_least(mx), inv = 1.0f / s;
        scale[r] = s;
        for (long long j = e; j < f; j++) dst[j] = from_f<T>(src[j] * inv);
    }
}

__global__ void k_fill(float* p, int n, float v)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) p[i] = v;
}

int grid_of(long long threads, int block = kSpmmBlock)
{
    long long g = (threads + block - 1) / block;
    if (g < 1) g = 1;
    if (g > 148LL * 64) g = 148LL * 64;
    return (int)g;
}

int log2_ceil(int v)
{
    int s = 0;
    while ((1 << s) < v) s++;
    return s;
}

// Lanes per row group and the vector width for k, X and Y.
int plan_lanes(int k, const float* X, int ldx, const float* Y, int ldy, int* vec, int* lshift)
{
    if (k < 1 || k > kSpmmMaxK || ldx < k || ldy < k) return CLSPMV_ERR_ARG;
    const bool v4 = k % 4 == 0 && ldx % 4 == 0 && ldy % 4 == 0 && ((uintptr_t)X & 15) == 0 && ((uintptr_t)Y & 15) == 0;
    if (!v4 && k > 32) return CLSPMV_ERR_ALIGN;   // more than 32 lanes per row otherwise
    *vec = v4 ? 4 : 1;
    *lshift = log2_ceil(v4 ? k / 4 : k);
    return CLSPMV_OK;
}

template <class M> const float* values_of(const M& m);
template <> const float* values_of(const clspmv_dia_f32& m) { return m.dia_data; }
template <> const float* values_of(const clspmv_bdia_f32& m) { return m.bdia_data; }
template <> const float* values_of(const clspmv_ell_f32& m) { return m.ell_data; }
template <> const float* values_of(const clspmv_sell_f32& m) { return m.sell_data; }
template <> const float* values_of(const clspmv_b4csr_f32& m) { return m.b4csr_data; }
template <> const float* values_of(const clspmv_b4ell_f32& m) { return m.b4ell_data; }
template <> const float* values_of(const clspmv_sbell_f32& m) { return m.sbell_data; }

template <class T, class M>
int launch_rows(const M& m, const void* vals, Dense d, int vec, cudaStream_t st)
{
    const long long threads = (long long)m.matinfo.height << d.lshift;
    const int grid = grid_of(threads);
    const T* v = static_cast<const T*>(vals);
    if (vec == 4) k_spmm_rows<4, T, M><<<grid, kSpmmBlock, 0, st>>>(m, v, d);
    else k_spmm_rows<1, T, M><<<grid, kSpmmBlock, 0, st>>>(m, v, d);
    return after_launch(1);
}

// Slots per row that the host can tell: ELL's width; for SELL the mean, its slices hold at least that
template <class T> inline bool long_slots(const clspmv_ell_f32& m) { return !std::is_same<T, float>::value && m.ell_num >= kSlotLoads; }
template <class T> inline bool long_slots(const clspmv_sell_f32& m) { return (long long)m.matinfo.nnz >= (long long)kSlotLoads * m.matinfo.height; }

template <class T, class M>
int launch_slots(const M& m, const void* vals, Dense d, int vec, cudaStream_t st)
{
    if (!long_slots<T>(m)) return launch_rows<T>(m, vals, d, vec, st);
    const int grid = grid_of((long long)m.matinfo.height << d.lshift);
    const T* v = static_cast<const T*>(vals);
    if (vec == 4) k_spmm_slots<4, T, M><<<grid, kSpmmBlock, 0, st>>>(m, v, d);
    else k_spmm_slots<1, T, M><<<grid, kSpmmBlock, 0, st>>>(m, v, d);
    return after_launch(1);
}

// CLSPMV_SPMM_BLOCK_ROWS=0 keeps the row walk for the block formats (measurements).
bool block_rows_enabled()
{
    static const bool on = [] {
        const char* e = getenv("CLSPMV_SPMM_BLOCK_ROWS");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

inline int bheight_of(const clspmv_b4csr_f32& m) { return (int)m.b4csr_bheight; }
inline int bheight_of(const clspmv_b4ell_f32& m) { return (int)m.b4ell_bheight; }
inline int bheight_of(const clspmv_sbell_f32& m) { return (int)m.sbell_bheight; }
inline int bwidth_of(const clspmv_b4csr_f32& m) { return (int)m.b4csr_bwidth; }
inline int bwidth_of(const clspmv_b4ell_f32& m) { return (int)m.b4ell_bwidth; }
inline int bwidth_of(const clspmv_sbell_f32& m) { return (int)m.sbell_bwidth; }
// strides of for_block in values, which 4-value loads need to be multiples of 4
inline bool strips_aligned(const clspmv_b4csr_f32& m) { return m.b4csr_aligned_size % 4 == 0; }
inline bool strips_aligned(const clspmv_b4ell_f32& m) { return m.b4ell_float4_aligned % 4 == 0; }
inline bool strips_aligned(const clspmv_sbell_f32&) { return true; }

// CLSPMV_SPMM_X_FORM: how the block-row kernel reads X rows (Dense::x_form; measurements)
int x_form()
{
    static const int f = [] {
        const char* e = getenv("CLSPMV_SPMM_X_FORM");
        return e ? atoi(e) : 0;
    }();
    return f;
}

template <int BH, int BW4, class T, class M>
void launch_block_kernel(const M& m, const T* v, Dense d, cudaStream_t st)
{
    d.x_form = x_form();
    const long long nbr = ((long long)m.matinfo.height + BH - 1) / BH;
    k_spmm_blocks<BH, BW4, T, M><<<grid_of(nbr << d.lshift), kSpmmBlock, 0, st>>>(m, v, d);
}

// Block formats with 128-bit X rows: the block-row kernel; otherwise (X rows
// of single columns, or strips off a 4-value boundary) the row walk.
template <class T, class M>
int launch_blocks(const M& m, const void* vals, Dense d, int vec, cudaStream_t st)
{
    const T* v = static_cast<const T*>(vals);
    const int bh = bheight_of(m), bw4 = bwidth_of(m) / 4;
    if (vec != 4 || !block_rows_enabled() || !strips_aligned(m) || ((uintptr_t)v % (4 * sizeof(T))) != 0 ||
        (bw4 != 1 && bw4 != 2))
        return launch_rows<T>(m, vals, d, vec, st);
    if (m.matinfo.height <= 0) return CLSPMV_OK;
#define BLK(BH)                                                        \
    case BH:                                                           \
        if (bw4 == 1) launch_block_kernel<BH, 1, T>(m, v, d, st);      \
        else launch_block_kernel<BH, 2, T>(m, v, d, st);               \
        break;
    switch (bh) {
        BLK(1)
        BLK(2)
        BLK(4)
        BLK(8)
        default: return launch_rows<T>(m, vals, d, vec, st);
    }
#undef BLK
    return after_launch(1);
}

// CLSPMV_SPMM_WARP_ROWS=0 takes long CSR rows by warp runs too (measurements).
bool warp_rows_enabled()
{
    static const bool on = [] {
        const char* e = getenv("CLSPMV_SPMM_WARP_ROWS");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

template <int LG, int VEC, int P, class T, bool IS_CSR>
void launch_runs(int rows, int nnz, const int* row_ptr, const int* row_id, const int* col_id, const T* v, bool vec, bool add,
                 Dense d, cudaStream_t st)
{
    const long long runs = ((long long)nnz + 32 * P - 1) / (32 * P), wpb = kSpmmBlock / 32;
    const long long resident = 148LL * 4 * wpb;
    const long long per = (runs + resident - 1) / resident;   // 1 while the runs do not fill the device
    const dim3 grid((unsigned)((runs + per * wpb - 1) / (per * wpb)), (unsigned)((d.k + (VEC << LG) - 1) / (VEC << LG)));
    if (!IS_CSR || add) k_spmm_runs<LG, VEC, P, T, IS_CSR, true><<<grid, kSpmmBlock, 0, st>>>(rows, nnz, row_ptr, row_id, col_id, v, vec, (int)per, d);
    else k_spmm_runs<LG, VEC, P, T, IS_CSR, !IS_CSR><<<grid, kSpmmBlock, 0, st>>>(rows, nnz, row_ptr, row_id, col_id, v, vec, (int)per, d);
}

template <class T, bool IS_CSR>
int launch_chunks(int rows, int nnz, const int* row_ptr, const int* row_id, const int* col_id, const void* vals, Dense d,
                  int vec, cudaStream_t st)
{
    // 8 nonzeros per lane once their runs are a third more than the device's warps (1.6M nonzeros): 4 costs 5-10 % at
    // k < 8 from there on (more searches and scans a nonzero); before, where most warps would take 2 runs of 8 and half of
    // them none, it takes 1.2-1.4M nonzeros at k = 7 / 32 / 128 from 46 / 54 / 155 to 40 / 45 / 134 us (300,000 rows, 3 of 10
    // filled), 28 / 36 / 83 to 25 / 29 / 65 (62,000 uneven rows)
    const bool few = nnz < 148 * 32 * 256 / 3 * 4;
    // Few nonzeros leave warps idle while a slot of G lanes walks its 4 G nonzeros: G is halved, down to 4 lanes, until the
    // panels of G lanes' columns make 3/8 of the device's warps (all of them: 20,000 rows of 9 at k = 64 17 -> 19 us; down to 2
    // lanes: 3,000 rows of 4 at k = 12 15 -> 21). beta 0, us: 5,000 rows of 3 at k = 36 / 128 19 / 23 -> 13 / 13 (at beta 1
    // 14 / 19 -> 8 / 8), 60,000 rows of 2 17 / 23 -> 15 / 19, 20,000 rows of 9 19 / 25 -> 17 / 21.
    int lg = d.lshift;
    if (few)
        while (lg > 2 && ((long long)nnz + 127) / 128 * ((d.k + (vec << lg) - 1) / (vec << lg)) < 148 * 12) lg--;
    // A CSR row is added, not written, where Y holds beta * Y already: a row that reads its Y first waits for it, one
    // row after another in a slot. beta = 1, us written / added: 5,000 rows of 3 at k = 36 27 / 14, 2^20 rows of 2 at
    // k = 5 / 36 / 128 45 / 33, 157 / 125, 355 / 343. Other beta than 0 take a pass over Y for that, which pays for a
    // small Y: up to 4 MB for single columns (k < 8 or rows off 16 bytes; 20,000 rows of 9 at k = 5 18 / 15 us) and, where
    // rows hold 3 entries and more on average, 10 MB for those (300,000 rows of 4.5 at k = 7 53 / 48) and 4 MB for
    // others (30,000 rows of 47 at k = 12 / 28 44 / 28, 58 / 43), but 60,000 rows of 2 at k = 16 12.8 / 16.9.
    const long long floats = (long long)rows * d.k;
    const bool filled = nnz >= 3LL * rows;
    const bool add = d.beta == 1.0f || (d.beta != 0.0f && floats <= (vec == 1 && filled ? 5 << 19 : vec == 1 || filled ? 1 << 20 : 0));
    if (d.beta != 1.0f) {
        if (IS_CSR && nnz > 0 && !add)
            (vec == 4 ? k_scale_cut<4> : k_scale_cut<1>)<<<grid_of(rows), kSpmmBlock, 0, st>>>(
                rows, row_ptr, few ? 7 : 8, vec == 1 && d.k < 8 ? 0 : d.lshift, d);
        else
            k_scale_rows<<<grid_of((long long)rows * d.k), kSpmmBlock, 0, st>>>(d.Y, rows, d.k, d.ldy, d.beta);
        int rc = after_launch(1);
        if (rc) return rc;
    }
    if (nnz <= 0) return CLSPMV_OK;
    const T* v = static_cast<const T*>(vals);
    const bool al = ((uintptr_t)col_id & 15) == 0 && (IS_CSR || ((uintptr_t)row_id & 15) == 0) && ((uintptr_t)v & (4 * sizeof(T) - 1)) == 0;
#define RUNS(LG, VEC)                                                                                            \
    case LG:                                                                                                     \
        if (few) launch_runs<LG, VEC, 4, T, IS_CSR>(rows, nnz, row_ptr, row_id, col_id, v, al, add, d, st);           \
        else launch_runs<LG, VEC, 8, T, IS_CSR>(rows, nnz, row_ptr, row_id, col_id, v, al, add, d, st);               \
        break;
    if (vec == 4) {
        switch (lg) {
            RUNS(0, 4) RUNS(1, 4) RUNS(2, 4) RUNS(3, 4) RUNS(4, 4) RUNS(5, 4)
        }
    } else {
        switch (lg) {
            RUNS(0, 1) RUNS(1, 1) RUNS(2, 1) RUNS(3, 1) RUNS(4, 1) RUNS(5, 1)
        }
    }
#undef RUNS
    return after_launch(1);
}

template <class T>
int spmm_typed(int format, const void* dev, const void* vals, Dense d, int vec, cudaStream_t st)
{
    switch (format) {
        case CLSPMV_FORMAT_CSR: {
            const auto& m = *static_cast<const clspmv_csr_f32*>(dev);
            if (!m.csr_row_ptr) return CLSPMV_ERR_ARG;
            const int G = d.k / 4;
            if (vec == 4 && (G & (G - 1)) == 0 && m.matinfo.height > 0 &&
                (long long)m.matinfo.nnz >= (long long)kWarpRowMin * m.matinfo.height && warp_rows_enabled()) {
                const long long warps = m.matinfo.height;
                const int grid = (int)std::min<long long>((warps + kSpmmBlock / 32 - 1) / (kSpmmBlock / 32), 148LL * 16);
                k_spmm_warp_rows<T><<<grid, kSpmmBlock, 0, st>>>(m.matinfo.height, m.csr_row_ptr, m.csr_col_id,
                                                                 static_cast<const T*>(vals ? vals : m.csr_data), d);
                return after_launch(1);
            }
            return launch_chunks<T, true>(m.matinfo.height, m.matinfo.nnz, m.csr_row_ptr, nullptr, m.csr_col_id,
                                          vals ? vals : m.csr_data, d, vec, st);
        }
        case CLSPMV_FORMAT_COO: {
            const auto& m = *static_cast<const clspmv_coo_f32*>(dev);
            return launch_chunks<T, false>(m.matinfo.height, m.matinfo.nnz, nullptr, m.coo_row_id, m.coo_col_id,
                                           vals ? vals : m.coo_data, d, vec, st);
        }
#define ROWS(FMT, TYPE, LAUNCH)                                                      \
    case FMT: {                                                                      \
        const auto& m = *static_cast<const TYPE*>(dev);                              \
        return LAUNCH<T>(m, vals ? vals : values_of(m), d, vec, st);                 \
    }
        ROWS(CLSPMV_FORMAT_DIA, clspmv_dia_f32, launch_rows)
        ROWS(CLSPMV_FORMAT_BDIA, clspmv_bdia_f32, launch_rows)
        ROWS(CLSPMV_FORMAT_ELL, clspmv_ell_f32, launch_slots)
        ROWS(CLSPMV_FORMAT_SELL, clspmv_sell_f32, launch_slots)
#undef ROWS
#define BLOCKS(FMT, TYPE)                                                            \
    case FMT: {                                                                      \
        const auto& m = *static_cast<const TYPE*>(dev);                              \
        return launch_blocks<T>(m, vals ? vals : values_of(m), d, vec, st);          \
    }
        BLOCKS(CLSPMV_FORMAT_B4CSR, clspmv_b4csr_f32)
        BLOCKS(CLSPMV_FORMAT_B4ELL, clspmv_b4ell_f32)
        BLOCKS(CLSPMV_FORMAT_SBELL, clspmv_sbell_f32)
#undef BLOCKS
    }
    return CLSPMV_ERR_ARG;
}

int read_int(const int* dev_ptr, int* out)
{
    return cuda_status(cudaMemcpy(out, dev_ptr, sizeof(int), cudaMemcpyDeviceToHost));
}

bool block_ok(unsigned bw, unsigned bh) { return (bw == 4 || bw == 8) && (bh == 1 || bh == 2 || bh == 4 || bh == 8); }

template <class T>
int pack_typed(int format, const void* dev, T* dst, float* scale, cudaStream_t st)
{
    switch (format) {
        case CLSPMV_FORMAT_CSR: {
            const auto& m = *static_cast<const clspmv_csr_f32*>(dev);
            k_pack_csr<T><<<grid_of(m.matinfo.height), kSpmmBlock, 0, st>>>(m.matinfo.height, m.csr_row_ptr, m.csr_data,
                                                                           dst, scale);
            return after_launch(1);
        }
        case CLSPMV_FORMAT_COO: {
            const auto& m = *static_cast<const clspmv_coo_f32*>(dev);
            k_fill<<<grid_of(m.matinfo.height), kSpmmBlock, 0, st>>>(scale, m.matinfo.height, 1.0f);
            int rc = after_launch(1);
            if (rc || m.matinfo.nnz <= 0) return rc;
            k_pack_coo<T><<<grid_of(m.matinfo.nnz), kSpmmBlock, 0, st>>>(m.matinfo.nnz, m.coo_row_id, m.coo_data, dst, scale);
            return after_launch(1);
        }
#define PACK(FMT, TYPE)                                                                       \
    case FMT: {                                                                               \
        const auto& m = *static_cast<const TYPE*>(dev);                                       \
        k_pack_rows<T, TYPE><<<grid_of(m.matinfo.height), kSpmmBlock, 0, st>>>(m, values_of(m), dst, scale); \
        return after_launch(1);                                                               \
    }
        PACK(CLSPMV_FORMAT_DIA, clspmv_dia_f32)
        PACK(CLSPMV_FORMAT_BDIA, clspmv_bdia_f32)
        PACK(CLSPMV_FORMAT_ELL, clspmv_ell_f32)
        PACK(CLSPMV_FORMAT_SELL, clspmv_sell_f32)
        PACK(CLSPMV_FORMAT_B4CSR, clspmv_b4csr_f32)
        PACK(CLSPMV_FORMAT_B4ELL, clspmv_b4ell_f32)
        PACK(CLSPMV_FORMAT_SBELL, clspmv_sbell_f32)
#undef PACK
    }
    return CLSPMV_ERR_ARG;
}

int check_struct(int format, const void* dev)
{
    if (!dev) return CLSPMV_ERR_ARG;
    switch (format) {
        case CLSPMV_FORMAT_B4CSR: {
            const auto& m = *static_cast<const clspmv_b4csr_f32*>(dev);
            return block_ok(m.b4csr_bwidth, m.b4csr_bheight) ? CLSPMV_OK : CLSPMV_ERR_UNSUPPORTED;
        }
        case CLSPMV_FORMAT_B4ELL: {
            const auto& m = *static_cast<const clspmv_b4ell_f32*>(dev);
            return block_ok(m.b4ell_bwidth, m.b4ell_bheight) ? CLSPMV_OK : CLSPMV_ERR_UNSUPPORTED;
        }
        case CLSPMV_FORMAT_SBELL: {
            const auto& m = *static_cast<const clspmv_sbell_f32*>(dev);
            return block_ok(m.sbell_bwidth, m.sbell_bheight) && m.sbell_slice_height > 0 ? CLSPMV_OK : CLSPMV_ERR_UNSUPPORTED;
        }
        case CLSPMV_FORMAT_SELL:
            return static_cast<const clspmv_sell_f32*>(dev)->sell_slice_height > 0 ? CLSPMV_OK : CLSPMV_ERR_UNSUPPORTED;
        case CLSPMV_FORMAT_CSR:
        case CLSPMV_FORMAT_COO:
        case CLSPMV_FORMAT_DIA:
        case CLSPMV_FORMAT_BDIA:
        case CLSPMV_FORMAT_ELL:
            return CLSPMV_OK;
    }
    return CLSPMV_ERR_ARG;
}

// every format struct starts with its matinfo
int matrix_rows(const void* dev) { return static_cast<const clspmv_matinfo*>(dev)->height; }


// ---------------------------------------------------------------------------
// Batches: many (matrix, X, Y) jobs in one persistent launch. Each job is cut
// into warp tasks of 32 / G rows (G lanes per row for its k) -- or, for a CSR
// job that adds into Y (beta 1), of 32 / G equal chunks of nonzeros, so that
// rows of thousands of entries are shared between groups; the tasks of all
// jobs form one index space that every warp strides through, finding its job
// by binary search over the jobs' first task numbers.
// ---------------------------------------------------------------------------
constexpr int kBatchLongRow = 256;

struct BatchJob {
    int format, value_type, k, lshift, vec, rows;
    int bh;                    // 4: a 4x4-block job, one lane group per block row (block_row); 0: rows
    int chunk, nnz;            // CSR accumulating into Y (beta 1): nonzeros per lane group, else 0 (row mode)
    long long task_begin;
    int ldx, ldy;
    float alpha, beta;
    const void* values;
    const float* scale;
    const float* X;
    float* Y;
    union {
        clspmv_csr_f32 csr;
        clspmv_dia_f32 dia;
        clspmv_bdia_f32 bdia;
        clspmv_ell_f32 ell;
        clspmv_sell_f32 sell;
        clspmv_b4csr_f32 b4csr;
        clspmv_b4ell_f32 b4ell;
        clspmv_sbell_f32 sbell;
    } m;
};

template <int VEC, class T, class M>
__device__ __forceinline__ void batch_row(const M& m, const BatchJob& J, int r, int c0)
{
    const T* vals = static_cast<const T*>(J.values);
    Acc<VEC> acc;
    for_row(m, r, [&](int col, size_t idx) { acc.fma(to_f(ld_val(vals + idx)), J.X + (size_t)col * J.ldx + c0); });
    const float a = J.scale ? J.alpha * J.scale[r] : J.alpha;
    acc.store(J.Y + (size_t)r * J.ldy + c0, a, J.beta);
}

template <int VEC, class T>
__device__ __forceinline__ void batch_dispatch(const BatchJob& J, int r, int c0)
{
    switch (J.format) {
        case CLSPMV_FORMAT_CSR: batch_row<VEC, T>(J.m.csr, J, r, c0); break;
        case CLSPMV_FORMAT_DIA: batch_row<VEC, T>(J.m.dia, J, r, c0); break;
        case CLSPMV_FORMAT_BDIA: batch_row<VEC, T>(J.m.bdia, J, r, c0); break;
        case CLSPMV_FORMAT_ELL: batch_row<VEC, T>(J.m.ell, J, r, c0); break;
        case CLSPMV_FORMAT_SELL: batch_row<VEC, T>(J.m.sell, J, r, c0); break;
        case CLSPMV_FORMAT_B4CSR: batch_row<VEC, T>(J.m.b4csr, J, r, c0); break;
        case CLSPMV_FORMAT_B4ELL: batch_row<VEC, T>(J.m.b4ell, J, r, c0); break;
        case CLSPMV_FORMAT_SBELL: batch_row<VEC, T>(J.m.sbell, J, r, c0); break;
    }
}

template <class T>
__device__ __forceinline__ void batch_blocks(const BatchJob& J, int br, int c0)
{
    const T* v = static_cast<const T*>(J.values);
    switch (J.format) {
        case CLSPMV_FORMAT_B4CSR: block_row<4, 1>(J.m.b4csr, v, br, c0, J.X, J.ldx, J.Y, J.ldy, J.alpha, J.beta, J.scale, 0); break;
        case CLSPMV_FORMAT_B4ELL: block_row<4, 1>(J.m.b4ell, v, br, c0, J.X, J.ldx, J.Y, J.ldy, J.alpha, J.beta, J.scale, 0); break;
        case CLSPMV_FORMAT_SBELL: block_row<4, 1>(J.m.sbell, v, br, c0, J.X, J.ldx, J.Y, J.ldy, J.alpha, J.beta, J.scale, 0); break;
    }
}

// CSR job accumulating into Y: the group owns nonzeros [e0, e0 + chunk); rows
// cut by the chunk's edges are added atomically, the others with a plain add
// (Y already holds beta * Y = Y).
template <int VEC, class T>
__device__ __forceinline__ void batch_chunk(const BatchJob& J, int e0, int c0)
{
    const clspmv_csr_f32& m = J.m.csr;
    const T* vals = static_cast<const T*>(J.values);
    const int e1 = min(J.nnz, e0 + J.chunk);
    int lo = 0, hi = J.rows;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(m.csr_row_ptr + mid) <= e0) lo = mid;
        else hi = mid - 1;
    }
    int row = lo, row_end = __ldg(m.csr_row_ptr + row + 1);
    bool first = true;
    Acc<VEC> acc;
    auto flush = [&](bool last) {
        const float a = J.scale ? J.alpha * J.scale[row] : J.alpha;
        float* y = J.Y + (size_t)row * J.ldy + c0;
        bool cut = first && __ldg(m.csr_row_ptr + row) < e0;
        if (last) cut = cut || row_end > e1;
        if (cut) acc.atomic(y, a);
        else acc.add(y, a);
    };
    for (int e = e0; e < e1; e++) {
        if (e >= row_end) {
            flush(false);
            first = false;
            acc = Acc<VEC>();
            do {
                row++;
                row_end = __ldg(m.csr_row_ptr + row + 1);
            } while (e >= row_end);
        }
        acc.fma(to_f(ld_val(vals + e)), J.X + (size_t)__ldg(m.csr_col_id + e) * J.ldx + c0);
    }
    flush(true);
}

// 4 CTAs per SM, at 64 registers: without the bound a lane group takes 1.2 times as long over a long row (ten rows of
// 20,000 at k = 4: 1.70 against 1.39 ms). 6 CTAs, at 40, leave one lookup in flight: SELL rows of 20,000 at k = 1 1.2
// against 2.7 ms, at k = 32 2.1 against 3.3, for 4 to 13 % in batches of even rows at k = 1, 16 and 32.
__global__ void __launch_bounds__(kSpmmBlock, 4) k_batch(const BatchJob* __restrict__ jobs, int njobs, long long tasks)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * kSpmmBlock) >> 5;
    for (long long t = ((long long)blockIdx.x * kSpmmBlock + threadIdx.x) >> 5; t < tasks; t += nwarps) {
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].task_begin <= t) lo = mid;
            else hi = mid - 1;
        }
        const BatchJob& J = jobs[lo];
        const long long r = (t - J.task_begin) * (32 >> J.lshift) + (lane >> J.lshift);
        const int c0 = (lane & ((1 << J.lshift) - 1)) * J.vec;
        if (J.chunk > 0) {   // r counts chunks of nonzeros here
            const long long e0 = r * J.chunk;
            if (e0 >= J.nnz || c0 >= J.k) continue;
            if (J.vec == 4) {
                if (J.value_type == CLSPMV_VALUES_F32) batch_chunk<4, float>(J, (int)e0, c0);
                else if (J.value_type == CLSPMV_VALUES_BF16) batch_chunk<4, __nv_bfloat16>(J, (int)e0, c0);
                else batch_chunk<4, __half>(J, (int)e0, c0);
            } else {
                if (J.value_type == CLSPMV_VALUES_F32) batch_chunk<1, float>(J, (int)e0, c0);
                else if (J.value_type == CLSPMV_VALUES_BF16) batch_chunk<1, __nv_bfloat16>(J, (int)e0, c0);
                else batch_chunk<1, __half>(J, (int)e0, c0);
            }
            continue;
        }
        if (r >= J.rows || c0 >= J.k) continue;
        if (J.vec == 4) {
            if (J.value_type == CLSPMV_VALUES_F32) batch_dispatch<4, float>(J, (int)r, c0);
            else if (J.value_type == CLSPMV_VALUES_BF16) batch_dispatch<4, __nv_bfloat16>(J, (int)r, c0);
            else batch_dispatch<4, __half>(J, (int)r, c0);
        } else {
            if (J.value_type == CLSPMV_VALUES_F32) batch_dispatch<1, float>(J, (int)r, c0);
            else if (J.value_type == CLSPMV_VALUES_BF16) batch_dispatch<1, __nv_bfloat16>(J, (int)r, c0);
            else batch_dispatch<1, __half>(J, (int)r, c0);
        }
    }
}

// The 4x4-block jobs of a batch (bh = 4) in their own persistent launch: warp
// tasks of 32 / G block rows, one lane group per block row (block_row). Kept
// apart from k_batch, whose other jobs would otherwise run at this path's
// register count.
__global__ void __launch_bounds__(kSpmmBlock, 3) k_batch_blocks(const BatchJob* __restrict__ jobs, int njobs, long long tasks)
{
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * kSpmmBlock) >> 5;
    for (long long t = ((long long)blockIdx.x * kSpmmBlock + threadIdx.x) >> 5; t < tasks; t += nwarps) {
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].task_begin <= t) lo = mid;
            else hi = mid - 1;
        }
        const BatchJob& J = jobs[lo];
        const long long br = (t - J.task_begin) * (32 >> J.lshift) + (lane >> J.lshift);
        const int c0 = (lane & ((1 << J.lshift) - 1)) * 4;
        if (br >= (J.rows + 3) / 4 || c0 >= J.k) continue;
        if (J.value_type == CLSPMV_VALUES_F32) batch_blocks<float>(J, (int)br, c0);
        else if (J.value_type == CLSPMV_VALUES_BF16) batch_blocks<__nv_bfloat16>(J, (int)br, c0);
        else batch_blocks<__half>(J, (int)br, c0);
    }
}

int persistent_grid(const void* kernel, int* cache)
{
    if (!*cache) {
        int dev = 0, nsm = 148, per = 1;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kSpmmBlock, 0) != cudaSuccess || per < 1) {
            cudaGetLastError();
            per = 1;
        }
        *cache = nsm * per;
    }
    return *cache;
}

int batch_blocks_grid()
{
    static int grid = 0;
    return persistent_grid((const void*)k_batch_blocks, &grid);
}

int batch_grid()
{
    static int grid = 0;
    return persistent_grid((const void*)k_batch, &grid);
}

// Fills one device job from a caller's job description.
int make_job(const clspmv_spmm_job& in, BatchJob& out)
{
    int rc = check_struct(in.format, in.dev);
    if (rc) return rc;
    if (in.format == CLSPMV_FORMAT_COO) return CLSPMV_ERR_UNSUPPORTED;   // no row starts to walk
    if (!in.X || !in.Y) return CLSPMV_ERR_ARG;
    if (in.value_type != CLSPMV_VALUES_F32 && in.value_type != CLSPMV_VALUES_BF16 && in.value_type != CLSPMV_VALUES_F16)
        return CLSPMV_ERR_ARG;
    if (in.value_type != CLSPMV_VALUES_F32 && (!in.values || !in.row_scale)) return CLSPMV_ERR_ARG;
    memset(&out, 0, sizeof(out));
    if ((rc = plan_lanes(in.k, in.X, in.ldx, in.Y, in.ldy, &out.vec, &out.lshift))) return rc;
    out.format = in.format;
    out.value_type = in.value_type;
    out.k = in.k;
    out.rows = matrix_rows(in.dev);
    out.ldx = in.ldx;
    out.ldy = in.ldy;
    out.alpha = in.alpha;
    out.beta = in.beta;
    out.scale = in.value_type == CLSPMV_VALUES_F32 ? nullptr : in.row_scale;
    out.X = in.X;
    out.Y = in.Y;
    switch (in.format) {
        case CLSPMV_FORMAT_CSR: out.m.csr = *static_cast<const clspmv_csr_f32*>(in.dev); out.values = out.m.csr.csr_data; break;
        case CLSPMV_FORMAT_DIA: out.m.dia = *static_cast<const clspmv_dia_f32*>(in.dev); out.values = out.m.dia.dia_data; break;
        case CLSPMV_FORMAT_BDIA: out.m.bdia = *static_cast<const clspmv_bdia_f32*>(in.dev); out.values = out.m.bdia.bdia_data; break;
        case CLSPMV_FORMAT_ELL: out.m.ell = *static_cast<const clspmv_ell_f32*>(in.dev); out.values = out.m.ell.ell_data; break;
        case CLSPMV_FORMAT_SELL: out.m.sell = *static_cast<const clspmv_sell_f32*>(in.dev); out.values = out.m.sell.sell_data; break;
        case CLSPMV_FORMAT_B4CSR: out.m.b4csr = *static_cast<const clspmv_b4csr_f32*>(in.dev); out.values = out.m.b4csr.b4csr_data; break;
        case CLSPMV_FORMAT_B4ELL: out.m.b4ell = *static_cast<const clspmv_b4ell_f32*>(in.dev); out.values = out.m.b4ell.b4ell_data; break;
        case CLSPMV_FORMAT_SBELL: out.m.sbell = *static_cast<const clspmv_sbell_f32*>(in.dev); out.values = out.m.sbell.sbell_data; break;
    }
    if (in.value_type != CLSPMV_VALUES_F32) out.values = in.values;
    if (out.format == CLSPMV_FORMAT_CSR && !out.m.csr.csr_row_ptr) return CLSPMV_ERR_ARG;
    // 4x4 blocks with 128-bit X rows: one lane group per block row, as clspmv_spmm does
    const size_t vsize = in.value_type == CLSPMV_VALUES_F32 ? 4 : 2;
    if (out.vec == 4 && block_rows_enabled() && ((uintptr_t)out.values % (4 * vsize)) == 0) {
        bool four = false;
        switch (out.format) {
            case CLSPMV_FORMAT_B4CSR: four = bheight_of(out.m.b4csr) == 4 && bwidth_of(out.m.b4csr) == 4 && strips_aligned(out.m.b4csr); break;
            case CLSPMV_FORMAT_B4ELL: four = bheight_of(out.m.b4ell) == 4 && bwidth_of(out.m.b4ell) == 4 && strips_aligned(out.m.b4ell); break;
            case CLSPMV_FORMAT_SBELL: four = bheight_of(out.m.sbell) == 4 && bwidth_of(out.m.sbell) == 4; break;
        }
        if (four) out.bh = 4;
    }
    // CSR adding into Y with long rows (mean >= kBatchLongRow entries): equal chunks of
    // nonzeros, so long rows are shared between groups (shorter rows: one group per row
    // is faster, measured on B200)
    if (out.format == CLSPMV_FORMAT_CSR && in.beta == 1.0f && out.m.csr.matinfo.nnz > 0 &&
        (long long)out.m.csr.matinfo.nnz >= (long long)kBatchLongRow * out.rows) {
        out.chunk = in.k <= 4 ? 64 : 32;
        out.nnz = out.m.csr.matinfo.nnz;
    }
    return CLSPMV_OK;
}

}  // namespace

struct clspmv_batch {
    int capacity = 0;
    int njobs = 0;
    int nrow_jobs = 0;            // jobs [0, nrow_jobs) run in k_batch, the rest (4x4 blocks) in k_batch_blocks
    long long tasks = 0;
    long long block_tasks = 0;
    BatchJob* host = nullptr;     // pinned staging of the job table
    BatchJob* dev = nullptr;
    cudaEvent_t copied = nullptr; // the last table upload has left `host`
};

namespace {
}  // namespace

extern "C" {

int clspmv_stored_values(int format, const void* dev, size_t* count)
{
    int rc = check_struct(format, dev);
    if (rc) return rc;
    if (!count) return CLSPMV_ERR_ARG;
    int last = 0;
    switch (format) {
        case CLSPMV_FORMAT_CSR: *count = (size_t)static_cast<const clspmv_csr_f32*>(dev)->matinfo.nnz; return CLSPMV_OK;
        case CLSPMV_FORMAT_COO: *count = (size_t)static_cast<const clspmv_coo_f32*>(dev)->matinfo.nnz; return CLSPMV_OK;
        case CLSPMV_FORMAT_DIA: {
            const auto& m = *static_cast<const clspmv_dia_f32*>(dev);
            *count = (size_t)m.dia_num * m.dia_length_aligned;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_BDIA: {
            const auto& m = *static_cast<const clspmv_bdia_f32*>(dev);
            if (m.bdia_band_num > 0 && (rc = read_int(m.bdia_bptr + m.bdia_band_num, &last))) return rc;
            *count = (size_t)last * m.bdia_length_aligned;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_ELL: {
            const auto& m = *static_cast<const clspmv_ell_f32*>(dev);
            *count = (size_t)m.ell_num * m.ell_height_aligned;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_SELL: {
            const auto& m = *static_cast<const clspmv_sell_f32*>(dev);
            if ((rc = read_int(m.sell_slice_ptr + m.sell_slice_num, &last))) return rc;
            *count = (size_t)last;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_B4CSR: {
            const auto& m = *static_cast<const clspmv_b4csr_f32*>(dev);
            *count = (size_t)m.b4csr_aligned_size * m.b4csr_bwidth * m.b4csr_bheight / 4;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_B4ELL: {
            const auto& m = *static_cast<const clspmv_b4ell_f32*>(dev);
            *count = (size_t)m.b4ell_block_num * m.b4ell_float4_aligned * (m.b4ell_bwidth / 4) * m.b4ell_bheight;
            return CLSPMV_OK;
        }
        case CLSPMV_FORMAT_SBELL: {
            const auto& m = *static_cast<const clspmv_sbell_f32*>(dev);
            if ((rc = read_int(m.sbell_slice_ptr + m.sbell_slice_num, &last))) return rc;
            *count = (size_t)last * m.sbell_bwidth * m.sbell_bheight;
            return CLSPMV_OK;
        }
    }
    return CLSPMV_ERR_ARG;
}

int clspmv_pack_values(int format, const void* dev, int value_type, void* values, float* row_scale,
                       clspmv_stream_t stream)
{
    int rc = check_struct(format, dev);
    if (rc) return rc;
    if (!values || !row_scale) return CLSPMV_ERR_ARG;
    size_t count = 0;
    if ((rc = clspmv_stored_values(format, dev, &count))) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // entries no row walk reaches (padding rows, out-of-range diagonals) stay 0
    if ((rc = cuda_status(cudaMemsetAsync(values, 0, count * 2, st)))) return rc;
    if (matrix_rows(dev) <= 0) return CLSPMV_OK;
    if (value_type == CLSPMV_VALUES_BF16) return pack_typed(format, dev, static_cast<__nv_bfloat16*>(values), row_scale, st);
    if (value_type == CLSPMV_VALUES_F16) return pack_typed(format, dev, static_cast<__half*>(values), row_scale, st);
    return CLSPMV_ERR_ARG;
}

int clspmv_spmm(int format, const void* dev, int value_type, const void* values, const float* row_scale, int k,
                const float* X, int ldx, float* Y, int ldy, float alpha, float beta, clspmv_stream_t stream)
{
    int rc = check_struct(format, dev);
    if (rc) return rc;
    if (!X || !Y) return CLSPMV_ERR_ARG;
    if (value_type != CLSPMV_VALUES_F32 && (!values || !row_scale)) return CLSPMV_ERR_ARG;
    int vec = 1, lshift = 0;
    if ((rc = plan_lanes(k, X, ldx, Y, ldy, &vec, &lshift))) return rc;
    if (matrix_rows(dev) <= 0) return CLSPMV_OK;
    Dense d{k, X, ldx, Y, ldy, alpha, beta, value_type == CLSPMV_VALUES_F32 ? nullptr : row_scale, lshift};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // one contiguous vector: the format's own single-vector kernel (CSR's needs a merge plan)
    if (k == 1 && ldx == 1 && ldy == 1 && format != CLSPMV_FORMAT_CSR) {
        rc = launch_packed(format, dev, value_type, values, row_scale, nullptr, X, Y, alpha, beta, st, false);
        if (rc != CLSPMV_ERR_ALIGN) return rc;
    }
    switch (value_type) {
        case CLSPMV_VALUES_F32: return spmm_typed<float>(format, dev, nullptr, d, vec, st);
        case CLSPMV_VALUES_BF16: return spmm_typed<__nv_bfloat16>(format, dev, values, d, vec, st);
        case CLSPMV_VALUES_F16: return spmm_typed<__half>(format, dev, values, d, vec, st);
    }
    return CLSPMV_ERR_ARG;
}

int clspmv_batch_create(int max_jobs, clspmv_batch** out)
{
    if (!out || max_jobs < 1) return CLSPMV_ERR_ARG;
    *out = nullptr;
    clspmv_batch* b = new (std::nothrow) clspmv_batch();
    if (!b) return CLSPMV_ERR_ALLOC;
    b->capacity = max_jobs;
    int rc = cuda_status(cudaMallocHost(&b->host, sizeof(BatchJob) * max_jobs));
    if (!rc) rc = cuda_status(cudaMalloc(&b->dev, sizeof(BatchJob) * max_jobs));
    if (!rc) rc = cuda_status(cudaEventCreateWithFlags(&b->copied, cudaEventDisableTiming));
    if (rc) {
        clspmv_batch_free(b);
        return rc;
    }
    *out = b;
    return CLSPMV_OK;
}

int clspmv_batch_set(clspmv_batch* b, const clspmv_spmm_job* jobs, int njobs, clspmv_stream_t stream, int* bad_job)
{
    if (bad_job) *bad_job = -1;
    if (!b || (!jobs && njobs > 0) || njobs < 0) return CLSPMV_ERR_ARG;
    if (njobs > b->capacity) return CLSPMV_ERR_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int rc = cuda_status(cudaEventSynchronize(b->copied));   // staging free again
    if (rc) return rc;
    // row jobs first (k_batch), then the 4x4-block jobs (k_batch_blocks), each
    // with its own task numbering; a job's place in the table changes nothing
    // in its Y
    b->njobs = 0;
    b->tasks = b->block_tasks = 0;
    b->nrow_jobs = 0;
    int nblock = 0;
    for (int i = 0; i < njobs; i++) {
        BatchJob J;
        if ((rc = make_job(jobs[i], J))) {
            if (bad_job) *bad_job = i;
            return rc;
        }
        if (J.bh) b->host[njobs - 1 - nblock++] = J;   // filled from the end, reversed below
        else b->host[b->nrow_jobs++] = J;
    }
    std::reverse(b->host + b->nrow_jobs, b->host + njobs);
    long long tasks = 0, block_tasks = 0;
    for (int i = 0; i < njobs; i++) {
        BatchJob& J = b->host[i];
        long long& t = J.bh ? block_tasks : tasks;
        J.task_begin = t;
        const long long units = J.chunk > 0 ? ((long long)J.nnz + J.chunk - 1) / J.chunk
                                : J.bh ? ((long long)J.rows + J.bh - 1) / J.bh : J.rows;
        t += (units + (32 >> J.lshift) - 1) / (32 >> J.lshift);
    }
    b->njobs = njobs;
    b->tasks = tasks;
    b->block_tasks = block_tasks;
    if (njobs == 0) return CLSPMV_OK;
    rc = cuda_status(cudaMemcpyAsync(b->dev, b->host, sizeof(BatchJob) * njobs, cudaMemcpyHostToDevice, st));
    if (!rc) rc = cuda_status(cudaEventRecord(b->copied, st));
    return rc;
}

int clspmv_batch_run(clspmv_batch* b, clspmv_stream_t stream)
{
    if (!b) return CLSPMV_ERR_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int n = 0;
    if (b->tasks > 0) {
        const long long grid = std::min<long long>(batch_grid(), (b->tasks + 7) / 8);
        k_batch<<<(int)grid, kSpmmBlock, 0, st>>>(b->dev, b->nrow_jobs, b->tasks);
        n++;
    }
    if (b->block_tasks > 0) {
        const long long grid = std::min<long long>(batch_blocks_grid(), (b->block_tasks + 7) / 8);
        k_batch_blocks<<<(int)grid, kSpmmBlock, 0, st>>>(b->dev + b->nrow_jobs, b->njobs - b->nrow_jobs, b->block_tasks);
        n++;
    }
    return n ? after_launch(n) : CLSPMV_OK;
}

int clspmv_batch_free(clspmv_batch* b)
{
    if (!b) return CLSPMV_ERR_ARG;
    if (b->copied) {
        cudaEventSynchronize(b->copied);
        cudaEventDestroy(b->copied);
    }
    if (b->host) cudaFreeHost(b->host);
    if (b->dev) cudaFree(b->dev);
    delete b;
    return CLSPMV_OK;
}

#define SPMM_ENTRY(name, FMT, TYPE)                                                                        \
    int clspmv_##name##_spmm_f32(const TYPE* dev, int k, const float* X, int ldx, float* Y, int ldy, float alpha, \
                                 float beta, clspmv_stream_t stream)                                              \
    {                                                                                                             \
        return clspmv_spmm(FMT, dev, CLSPMV_VALUES_F32, nullptr, nullptr, k, X, ldx, Y, ldy, alpha, beta, stream); \
    }
SPMM_ENTRY(csr, CLSPMV_FORMAT_CSR, clspmv_csr_f32)
SPMM_ENTRY(coo, CLSPMV_FORMAT_COO, clspmv_coo_f32)
SPMM_ENTRY(dia, CLSPMV_FORMAT_DIA, clspmv_dia_f32)
SPMM_ENTRY(bdia, CLSPMV_FORMAT_BDIA, clspmv_bdia_f32)
SPMM_ENTRY(ell, CLSPMV_FORMAT_ELL, clspmv_ell_f32)
SPMM_ENTRY(sell, CLSPMV_FORMAT_SELL, clspmv_sell_f32)
SPMM_ENTRY(b4csr, CLSPMV_FORMAT_B4CSR, clspmv_b4csr_f32)
SPMM_ENTRY(b4ell, CLSPMV_FORMAT_B4ELL, clspmv_b4ell_f32)
SPMM_ENTRY(sbell, CLSPMV_FORMAT_SBELL, clspmv_sbell_f32)
#undef SPMM_ENTRY

}  // extern "C"
