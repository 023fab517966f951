// Calls of the library on both sides of a device reset of this program's own
// context. argv[1]: the library; argv[2]: "upload" (arrays released before the
// reset are not handed out after it) or "iterate" (steps of A^k x in one launch).
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "clspmv_b200.h"

static void* so;
template <class F>
static F fn(const char* name) { return reinterpret_cast<F>(dlsym(so, name)); }

static int failures = 0;
#define CHECK(c) \
    do { if (!(c)) { failures++; printf("pass %d, line %d: %s\n", pass, __LINE__, #c); } } while (0)

static constexpr int N = 16000;   // a cluster of 16 blocks, more than a kernel may have by default

static void upload(int pass)   // twice the identity, its arrays over 2 MB so that they have pages of their own
{
    const int n = 1 << 20;
    std::vector<int> rp(n + 1), col(n);
    std::vector<float> val(n, 2.0f), x(n), y(n);
    for (int i = 0; i < n; i++) { rp[i] = col[i] = i; x[i] = (float)(i % 97); }
    rp[n] = n;
    clspmv_csr_f32 h{}, d{};
    h.matinfo.width = h.matinfo.height = h.matinfo.nnz = n;
    h.csr_row_ptr = rp.data();
    h.csr_col_id = col.data();
    h.csr_data = val.data();
    float *dx = nullptr, *dy = nullptr, *mine[4];
    for (float*& p : mine) {   // the caller's own, which may lie where the last pass's arrays lay
        CHECK(cudaMalloc(&p, 4 * n) == cudaSuccess);
        CHECK(cudaMemcpy(p, x.data(), 4 * n, cudaMemcpyHostToDevice) == cudaSuccess);
    }
    CHECK(fn<decltype(&clspmv_upload_csr_f32)>("clspmv_upload_csr_f32")(&h, &d) == CLSPMV_OK);
    CHECK(cudaMalloc(&dx, 4 * n) == cudaSuccess && cudaMalloc(&dy, 4 * n) == cudaSuccess);
    CHECK(cudaMemcpy(dx, x.data(), 4 * n, cudaMemcpyHostToDevice) == cudaSuccess);
    CHECK(fn<decltype(&clspmv_csr_scalar_spmv_f32)>("clspmv_csr_scalar_spmv_f32")(&d, dx, dy, 1.0f, 0.0f, nullptr) == CLSPMV_OK);
    CHECK(cudaMemcpy(y.data(), dy, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess);
    int wrong = 0;
    for (int i = 0; i < n; i++) wrong += y[i] != 2 * x[i];
    CHECK(wrong == 0);
    for (float* p : mine) {
        CHECK(cudaMemcpy(y.data(), p, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess);
        CHECK(memcmp(y.data(), x.data(), 4 * n) == 0);
    }
    CHECK(fn<decltype(&clspmv_device_free_csr_f32)>("clspmv_device_free_csr_f32")(&d) == CLSPMV_OK);
}

static void iterate(int pass)   // 8 steps of x <- A x, A the permutation that shifts by one row
{
    int off = 1;
    const int len = (N + 31) / 32 * 32;
    std::vector<float> data(len, 1.0f), x(N), y(N);
    data[N - 1] = 0.0f;
    for (int i = 0; i < N; i++) x[i] = (float)(i % 89);
    clspmv_cocktail_f32 c{};
    c.mat_width = c.mat_height = N;
    c.mat_nnz = N - 1;
    c.ifusedia = true;
    c.dia.matinfo.width = c.dia.matinfo.height = N;
    c.dia.matinfo.nnz = N - 1;
    c.dia.dia_num = 1;
    c.dia.dia_length = N;
    c.dia.dia_length_aligned = len;
    c.dia.dia_offsets = &off;
    c.dia.dia_data = data.data();
    clspmv_cocktail_handle* h = nullptr;
    CHECK(fn<decltype(&clspmv_cocktail_upload_f32)>("clspmv_cocktail_upload_f32")(&c, &h) == CLSPMV_OK);
    if (!h) return;
    float *dx = nullptr, *dy = nullptr;
    CHECK(cudaMalloc(&dx, 4 * N) == cudaSuccess && cudaMalloc(&dy, 4 * N) == cudaSuccess);
    CHECK(cudaMemcpy(dx, x.data(), 4 * N, cudaMemcpyHostToDevice) == cudaSuccess);
    const auto count = fn<decltype(&clspmv_launch_count)>("clspmv_launch_count");
    const auto before = count();
    CHECK(fn<decltype(&clspmv_cocktail_iterate_f32)>("clspmv_cocktail_iterate_f32")(h, dx, dy, 1.0f, 0.0f, 8, nullptr) == CLSPMV_OK);
    CHECK(count() == before + 1);
    CHECK(cudaMemcpy(y.data(), dy, 4 * N, cudaMemcpyDeviceToHost) == cudaSuccess);
    int wrong = 0;
    for (int i = 0; i < N; i++) wrong += y[i] != (i + 8 < N ? x[i + 8] : 0.0f);
    CHECK(wrong == 0);
    fn<decltype(&clspmv_cocktail_free)>("clspmv_cocktail_free")(h);
    CHECK(fn<decltype(&clspmv_device_trim)>("clspmv_device_trim")() == CLSPMV_OK);
}

int main(int argc, char** argv)
{
    if (argc < 3 || !(so = dlopen(argv[1], RTLD_NOW))) return 99;
    for (int pass = 0; pass < 3; pass++) {
        if (std::string(argv[2]) == "iterate") iterate(pass);
        else upload(pass);
        if (failures) break;
        CHECK(cudaDeviceReset() == cudaSuccess);
    }
    return failures;
}
