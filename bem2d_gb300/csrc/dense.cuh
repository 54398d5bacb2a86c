// Launch interfaces of dense.cu (dense operators and Lanczos helpers).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace bem2d_gpu {

void launch_change_basis(int n, const double2* K, long long ldk, const int* bstart_of,
                         const int* bsize_of, const double2* uinv, double2* out, long long ldo,
                         cudaStream_t s);
void launch_gather_blocks(int n, const double2* M, long long ldm, const int* bstart_of,
                          const int* bsize_of, double2* blk, cudaStream_t s);
size_t mv_part_bytes(int n);
void launch_mv(const double2* A, long long lda, int n, const double2* x, double2* y,
               double2* part, cudaStream_t s);
void launch_mvh(const double2* A, long long lda, int n, const double2* x, double2* y,
                cudaStream_t s);
// complex64 versions (part: mv_part_bytes(n) bytes suffice)
void launch_mv(const float2* A, long long lda, int n, const float2* x, float2* y, float2* part,
               cudaStream_t s);
void launch_mvh(const float2* A, long long lda, int n, const float2* x, float2* y,
                cudaStream_t s);
// C (n x m, ldc) = op(A) B, op = A or A^H (herm).  work: room for the K-split
// partial products (zgemm_work_bytes); with less, one pass over K.
void launch_zgemm(bool herm, const double2* A, long long lda, int n, const double2* B,
                  long long ldb, int m, double2* C, long long ldc, void* work,
                  size_t work_bytes, cudaStream_t s);
void launch_zgemm(bool herm, const float2* A, long long lda, int n, const float2* B,
                  long long ldb, int m, float2* C, long long ldc, void* work,
                  size_t work_bytes, cudaStream_t s);
size_t zgemm_work_bytes(int n, int m, size_t elem);
// y = A x or A^H x (herm) in float-float on the FP32 pipe (~1e-13 relative to
// |A| |x|): A (n x n) given as hi = fl32(A), lo = fl32(A - hi), ld n; part:
// mv_part_bytes(n) bytes.  launch_split_ff makes the split.
void launch_mv_ff(bool herm, const float2* Ahi, const float2* Alo, int n, const double2* x,
                  double2* y, double2* part, cudaStream_t s);
void launch_split_ff(const double2* A, long long lda, int n, float2* hi, float2* lo,
                     cudaStream_t s);

// Products with an n x n matrix through exact digit products on the tensor
// cores (oz_gemm.cu): S digits, 8 or 7 for complex128 (FP64 and better than
// float-float accuracy), 4 for complex64 (FP32).  launch_oz_pack packs `rows`
// rows from r0 of A or A^H (herm) into oz_gemm_a_bytes(rows, n, S).
// launch_oz_gemm_pair forms C1 = A B and C2 = A^H B (B n x m, ldb) with
// oz_gemm_work_bytes(rows, n, m, S, sizeof(T)) of work: rows >= n: Apk holds all of
// A packed, then all of A^H; otherwise `rows` rows (a multiple of 64) are packed
// into Apk at a time.  Sets *status on a device-side wait timeout.
size_t oz_gemm_a_bytes(int rows, int n, int S);
size_t oz_gemm_work_bytes(int rows, int n, int m, int S, size_t elem);
template <typename T>
void launch_oz_pack(bool herm, int S, const T* A, long long lda, int r0, int rows, int n, void* dst,
                    cudaStream_t s);
template <typename T>
int launch_oz_gemm_pair(int S, const T* A, long long lda, int rows, void* Apk, int n, const T* B,
                        long long ldb, int m, T* C1, T* C2, long long ldc, void* work, int* status,
                        cudaStream_t s, long long* launches);
// C (rows x m, ldc) = A (rows x k, lda) B (k x m, ldb), complex128
void launch_zgemm_rect(const double2* A, long long lda, int rows, int k, const double2* B,
                       long long ldb, int m, double2* C, long long ldc, cudaStream_t s);
#define BEM2D_BATCHED_DECLS(T)                                                                \
  void launch_batched_dots(const T* Q, long long qstride, int n, int j, const T* W,           \
                           long long wstride, T* h, int ldh, int nb, cudaStream_t s);         \
  void launch_batched_sub(const T* Q, long long qstride, int n, int j, T* W, long long wstride, \
                          const T* h, int ldh, int nb, cudaStream_t s);                       \
  void launch_batched_norm2(int n, const T* W, long long wstride, double* out, int nb,        \
                            cudaStream_t s);                                                  \
  void launch_batched_scale(int n, const T* src, long long sstride, const double* scale,      \
                            T* dst, long long dstride, int nb, cudaStream_t s);               \
  void launch_herm_combine(int n, const T* Y1, const T* Y2, long long stride,                 \
                           const double* theta, T* W, long long wstride, int nb, cudaStream_t s); \
  /* dst slot i (stride dstride) = the first len entries of src slot map[i] */               \
  void launch_gather_slots(const T* src, long long sstride, T* dst, long long dstride,        \
                           long long len, const int* map, int nmap, cudaStream_t s);          \
  /* dst slot map[i] = the first len entries of src slot i */                                \
  void launch_scatter_slots(const T* src, long long sstride, T* dst, long long dstride,       \
                            long long len, const int* map, int nmap, cudaStream_t s);
BEM2D_BATCHED_DECLS(double2)
BEM2D_BATCHED_DECLS(float2)
#undef BEM2D_BATCHED_DECLS
// dst (complex128) = src (complex64), nb columns of n
void launch_widen(int n, const float2* src, long long sstride, double2* dst, long long dstride,
                  int nb, cudaStream_t s);
void launch_axpy_real(int n, double a, const double2* x, double2* y, cudaStream_t s);
bool tridiag_eigenvalues(std::vector<double> d, std::vector<double> e, std::vector<double>* ev);
// Largest eigenvalue of the symmetric tridiagonal (d, e) (e: n-1 entries).
double tridiag_lmax(const std::vector<double>& d, const std::vector<double>& e);
// Largest eigenvalue given a lower bound lo (for a Lanczos tridiagonal, the
// previous step's value: Ritz values interlace) and a guess of the distance
// to it: the step grows fourfold until lo + step bounds the spectrum, then
// bisection to max(atol, 2.2e-16 times the Gershgorin bound); returns the
// lower end of the final bracket, so a result is again a valid lower bound
// (a value above the true one would stall the next calls at itself).  Far
// fewer Sturm sweeps than bisection from the Gershgorin interval once the
// value has settled.
double tridiag_lmax_from(const std::vector<double>& d, const std::vector<double>& e, double lo,
                         double step, double atol);
// k-th largest eigenvalue (k = 1: the largest) by Sturm bisection, to rel
// times the Gershgorin bound of the spectrum.
double tridiag_kth_largest(const std::vector<double>& d, const std::vector<double>& e, int k,
                           double rel);
// Unit eigenvector of the symmetric tridiagonal (d, e) for its eigenvalue
// lambda (inverse iteration).
std::vector<double> tridiag_eigenvector(const std::vector<double>& d, const std::vector<double>& e,
                                        double lambda);

}  // namespace bem2d_gpu
