// api_internal.h — helpers shared by the .cu files of libclspmv_b200.so.
#pragma once
#include <cuda_runtime.h>
#include "clspmv_b200.h"

namespace clspmv {
// Maps a CUDA error to a clspmv_status, remembering its text per thread.
int cuda_status(cudaError_t e);
// Counts `n` kernel launches and returns the status of the last launch.
int after_launch(int n);

// Device arrays that outlast a call, from the bounded list of released ones or cudaMalloc (device_pool.cu).
// device_release waits for the array's device unless `idle_on` names it (or says kIdleAll): no work on the array is
// pending there. It returns what the next array released with this one may name.
constexpr int kIdleNone = -1, kIdleAll = -2;
int device_alloc(void** out, size_t bytes);
int device_release(void* p, int idle_on);

// Format launchers (spmv_api.cu). With `atomic`, alpha*A*x is added into y
// with red.global.add and beta is ignored (apply it first with
// launch_prescale); several launches may then target one y concurrently.
int launch_prescale(float* y, int n, float beta, cudaStream_t st);
int launch_dia(const clspmv_dia_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_bdia(const clspmv_bdia_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_ell(const clspmv_ell_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_sell(const clspmv_sell_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_sell_plan(const clspmv_sell_f32* m, const clspmv_sell_plan* plan, const float* x, float* y, float alpha,
                     float beta, cudaStream_t st, bool atomic);
int launch_csr_scalar(const clspmv_csr_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_csr_vector(const clspmv_csr_f32* m, const float* x, float* y, float alpha, float beta, int tpr, cudaStream_t st, bool atomic);
int launch_csr_merge(const clspmv_csr_f32* m, const int* tc, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_csr_merge_plan(const clspmv_csr_f32* m, int* tc, cudaStream_t st);
int launch_csr_chunk(const clspmv_csr_f32* m, const int* chunk_row, const float* x, float* y, float alpha, float beta,
                     cudaStream_t st, bool atomic);
int launch_csr_chunk_plan(const clspmv_csr_f32* m, int* chunk_row, cudaStream_t st);
int launch_coo(const clspmv_coo_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_b4ell(const clspmv_b4ell_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_sbell(const clspmv_sbell_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_packed(int format, const void* dev, int value_type, const void* values, const float* scale, const int* tc,
                  const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);
int launch_b4csr(const clspmv_b4csr_f32* m, const float* x, float* y, float alpha, float beta, cudaStream_t st, bool atomic);

// DIA / BDIA with the diagonals staged in shared memory by bulk copies
// (diag_bulk.cu); BDIA passes its bptr (the diagonal count is read on the
// device), DIA bptr = nullptr and its ndiag.
bool diag_bulk_supported(int len, const void* data);
int launch_diag_bulk(int rows, int cols, int ndiag, int len, const int* offsets, const int* bptr, int nband,
                     const float* data, const float* x, float* y, float alpha, float beta, cudaStream_t st);

// Steps of y <- alpha*A*x + beta*y; x <- y of a DIA / BDIA matrix of `ndiag` diagonals held by one cluster's shared
// memory, in one launch (iterate_resident.cu); x holds at least as many entries as y.
// The plans are made where the matrix is uploaded, with its device current.
struct ResidentPlan {
    int ctas = 0, per = 0, cap = 0;   // CTAs of the cluster (0: the matrix does not fit, or gains nothing), rows and most entries of one (COO, CSR)
};
ResidentPlan resident_dia_plan(int rows, int ndiag);
ResidentPlan resident_bdia_plan(int rows, const int* bptr, int nband);
// COO (sorted row ids) or CSR (row pointer), from the host arrays.
ResidentPlan resident_rows_plan(int rows, int nnz, const int* row_id, const int* row_ptr, const int* col);
int resident_iterate_dia(const clspmv_dia_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st);
int resident_iterate_bdia(const clspmv_bdia_f32* m, int ndiag, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps,
                          cudaStream_t st);
int resident_iterate_coo(const clspmv_coo_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st);
int resident_iterate_csr(const clspmv_csr_f32* m, const ResidentPlan& p, float* x, float* y, float alpha, float beta, int steps, cudaStream_t st);

// Fused Cocktail SpMV (cocktail_fused.cu): the parts of a partitioned matrix
// (device struct) cut into tiles, interleaved into one work list and run by
// one persistent launch. fused_plan_create returns CLSPMV_ERR_UNSUPPORTED
// when a part's layout is outside what the fused kernel covers.
struct FusedPlan;
int fused_plan_create(const clspmv_cocktail_f32* dev, const int* chunk_plan, FusedPlan** out);
int fused_spmv(const FusedPlan* plan, const float* x, float* y, float alpha, float beta, cudaStream_t st);
void fused_plan_free(FusedPlan* plan);
int fused_plan_items(const FusedPlan* plan);
}  // namespace clspmv
