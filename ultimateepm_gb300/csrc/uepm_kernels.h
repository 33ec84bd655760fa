// uepm_kernels.h -- host-side launch wrappers of the device kernels (one declaration per kernel).
// Scalar type S is double / float (real symmetric H) or cx<double> / cx<float> (complex Hermitian H).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "uepm_common.cuh"

namespace uepm {

// For a launcher that returns false with nothing launched: takes back the error of the call that failed, so that
// the caller's other kernel does not answer for it. An error that was pending before is left for the caller.
struct Refusal {
    bool clean = cudaPeekAtLastError() == cudaSuccess;
    bool operator()() const {
        if (clean) cudaGetLastError();
        return false;
    }
};

// The dynamic shared memory that a CTA may take: 227 KB, less what the kernels hold as static shared memory (800 bytes
// at most; k_refine_y_tc, 2 KB, and k_tridiag_blocked name limits of their own).
constexpr size_t kMaxDynamicSmem = 226 * 1024;
// Lets a kernel be launched with smem bytes of dynamic shared memory, most at the most. Without asking it gets 48 KB
// together with its static shared memory. The limit belongs to the kernel in the whole process, and another thread
// may be about to launch it at another size: every call sets the same one, so that none takes from another what it
// relies on.
template <typename K>
cudaError_t allow_smem(K kern, size_t smem, size_t most = kMaxDynamicSmem) {
    if (smem <= 47 * 1024) return cudaSuccess;
    if (smem > most) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

void count_launch(int n = 1);

// assemble.cu: H(k) in FULL column-major storage (both triangles). SO = double (real H) or
// cx<double>; H32 (optional) receives the FP32 copy for the mixed path (float or cx<float>).
void launch_rows(const DevParams& P, const double* d_k, const int* d_G, double* d_rows, int batch, cudaStream_t s,
                 float2* d_rows32 = nullptr);
// Mixed path, no spin-orbit, square nonlocal wells: the assembly in double-single arithmetic on the
// FP32 pipe (SO = ds2 or ds4), from the k-independent tables in FP32 pairs and d_rows32 (written by
// launch_rows when given).
// The same with spin-orbit coupling (SO = ds4): the scalar part and the spin-orbit blocks in
// double-single, the FP64 element where the nonlocal part needs it.
template <typename SO>
void launch_assemble_soc_ds(const DevParams& P, const DevParamsDS& Q, const float4* Vloc32, const float4* phNL32,
                            const float4* phSO32, const float2* rows32, const cx<double>* Vloc, const double2* phNL,
                            const double2* phSO, const double* rows, SO* H, int ld, size_t mstride,
                            typename Lower<SO>::type* H32, size_t mstride32, int batch, cudaStream_t s,
                            qt<float>* HQ = nullptr, size_t mstrideq = 0);
// Quaternionic H (order N): HQ above receives its FP32 lower triangle; this forms the full FP64 matrix.
void launch_assemble_quat(const DevParams& P, const cx<double>* Vloc, const double2* phNL, const double2* phSO,
                          const double* rows, qt<double>* HQ, size_t mstrideq, int batch, cudaStream_t s);
template <typename SO>
void launch_assemble_ds(const DevParams& P, const DevParamsDS& Q, const float4* Vloc32, const float4* phNL32,
                        const float2* rows32, const cx<double>* Vloc, const double2* phNL, const double* rows, SO* H,
                        int ld, size_t mstride, typename Lower<SO>::type* H32, size_t mstride32, int batch,
                        cudaStream_t s);
template <typename SO>
void launch_assemble(const DevParams& P, const cx<double>* Vloc, const double2* phNL, const double2* phSO, const double* rows,
                     SO* H, int ld, size_t mstride, typename Lower<SO>::type* H32, size_t mstride32, int batch,
                     cudaStream_t s);

// tridiag.cu: Householder reduction in place. d, e: [batch][n]; tq: [batch][n] reflector scalars;
// status: [batch] (ORed with UEPM_K_NONFINITE on NaN/Inf).
// variant: 0 automatic, 1 register-resident (FP32 real, n <= tridiag_reg_max_n()), 2 one CTA per
// matrix (shared memory where the matrix fits, else global memory with a persistent grid), 3 one
// thread-block cluster per matrix (tridiag_cluster.cu), 4 one CTA per matrix in global memory with
// each step's update fused into the next step's product (FP32, n <= 512), 5 the same with every
// other update deferred to the next pass, 6 blocked (panels of 16 columns, lower triangle only, one
// matrix per SM, tridiag_blocked.cu; FP32, n <= 512). Automatic: FP32 in registers to
// tridiag_reg_max_n(complex), for complex orders 175..230 the triangular kernel (tridiag_tri.cu) and from 231
// 6, for real orders from 300 6, else 5; FP64 2, with a cluster of CTAs per matrix for few matrices
// (tridiag_wide.cu).
// ctas_per_sm (0: automatic) caps the persistent grid of the global-memory kernels (tridiag_takes_ctas); cluster
// (0: automatic) is the cluster size of variant 3.
template <typename S>
void launch_tridiag(S* H, int n, int ld, size_t mstride, typename ST<S>::R* d, typename ST<S>::R* e, S* tq, int* status,
                    int batch, cudaStream_t s, int variant = 0, int ctas_per_sm = 0, int cluster = 0,
                    bool tensor_cores = true);
// Whether launch_tridiag's choice takes ctas_per_sm.
bool tridiag_takes_ctas(bool f32, bool cplx, int n, int variant);
// tridiag_wide.cu: the FP64 reduction with a cluster of CTAs per matrix, for few matrices (false, with nothing
// launched, where that does not pay).
template <typename S>
bool launch_tridiag_wide(S* H, int n, int ld, size_t mstride, double* d, double* e, S* tq, int* status, int batch,
                         cudaStream_t s);
// The FP64 reduction of quaternion matrices (order n <= 256; tridiag.cu).
void launch_tridiag_quat(qt<double>* H, int n, int ld, size_t mstride, double* d, double* e, qt<double>* tq, int* status,
                         int batch, cudaStream_t s, int ctas_per_sm);
// tridiag_cluster.cu: cluster size for order n (want = 0: automatic; 0 returned when it cannot fit)
// and the launch (false when the cluster kernel cannot run this case).
template <typename S>
int tridiag_cluster_size(int n, int want);
template <typename S>
bool launch_tridiag_cluster(S* H, int n, int ld, size_t mstride, typename ST<S>::R* d, typename ST<S>::R* e, S* tq,
                            int* status, int batch, cudaStream_t s, int want_c);
// tridiag_blocked.cu: the blocked reduction (false when it cannot run this order); tensor_cores puts
// the complex trailing updates on tcgen05 (where the operand staging fits shared memory).
int tridiag_blocked_max_n();
template <typename S>
bool launch_tridiag_blocked(S* H, int n, int ld, size_t mstride, typename ST<S>::R* d, typename ST<S>::R* e, S* tq,
                            int* status, int batch, cudaStream_t s, bool tensor_cores);
// tridiag_tri.cu: the reduction of quaternion (order 1..256) and complex matrices (order kTriMinCplx..kTriMaxCplx)
// with the lower triangle in shared memory (H: at least the lower triangle, column-major; false when it cannot run).
constexpr int kTriMinCplx = 175, kTriMaxCplx = 230;
template <typename S>
bool launch_tridiag_tri(S* H, int n, int ld, size_t mstride, float* d, float* e, S* tq, int* status, int batch,
                        cudaStream_t s);
// tridiag_reg.cu: the same reduction for FP32 matrices with n <= tridiag_reg_max_n(complex), held in
// registers (launch_tridiag dispatches to it; complex ones in the automatic choice only).
int  tridiag_reg_max_n(bool cplx = false);
void launch_tridiag_reg(float* H, int n, int ld, size_t mstride, float* d, float* e, float* tq, int* status, int batch,
                        cudaStream_t s);
void launch_tridiag_reg(cx<float>* H, int n, int ld, size_t mstride, float* d, float* e, cx<float>* tq, int* status,
                        int batch, cudaStream_t s);
// The same for real local-potential matrices formed in the kernel from the k-independent local V
// ([N][N], N = n: its FP32 rounding V32 off the diagonal, FP64 Vloc plus the rows table's kinetic term
// on it), bit-identical to reducing the assembly's FP32 copy; H receives only the reflector tails.
void launch_tridiag_reg_local(const float* V32, const cx<double>* Vloc, const double* rows, float* H, int n, int ld,
                              size_t mstride, float* d, float* e, float* tq, int* status, int batch, cudaStream_t s);

// tridiag_eig.cu (false, with nothing launched, for orders beyond 512)
template <typename T>
bool launch_bisect(const T* d, const T* e, int n, int nb, T* ev, int ev_ld, int batch, cudaStream_t s, int cap = 0,
                   int* status = nullptr);
template <typename T>
void launch_invit(const T* d, const T* e, const T* ev, int ev_ld, int n, int nb, T* work, T* z, int* status, int batch,
                  cudaStream_t s, int cap = 0);
// Inverse-iteration workspace per matrix (used where the arrays exceed shared memory): U0, U1, the
// multipliers and Z, each n x 32 interleaved by lane, and the row-interchange bits.
template <typename T>
__host__ __device__ inline size_t invit_work_elems(int n) {
    return (size_t)5 * n * 32;
}

// backtransform.cu: X = Q Z for nb real tridiagonal eigenvectors z ([batch][nb][n]); X is written as
// complex ([batch][nb][n]) when Xout is given; optional Hellmann-Feynman gradients ([batch][nb][3]).
template <typename S>
void launch_backtransform(const S* H, int n, int ld, size_t mstride, const S* tq, const typename ST<S>::R* z, int nb,
                          cx<typename ST<S>::R>* Xout, const DevParams& P, const double* d_k, const int* d_G, double* grad,
                          int batch, cudaStream_t s, int lanes = 0);

// The same for a quaternion matrix of order n = N from nz real vectors z ([batch][nz][N]): quaternion
// vector a + b j gives the spinor eigenvectors (a, -conj b) and (b, conj a), written as vectors 2 q and
// 2 q + 1 of [batch][nb][2 N] (nb = 2 nz or 2 nz - 1), with their gradients.
template <typename T>
void launch_backtransform_quat(const qt<T>* H, int n, int ld, size_t mstride, const qt<T>* tq, const T* z, int nz, int nb,
                               cx<T>* Xout, const DevParams& P, const double* d_k, const int* d_G, double* grad,
                               int batch, cudaStream_t s, int lanes = 0);
// Rows per lane that the register budget allows: a requested lane count is honoured where its rows fit.
constexpr int kBtRealRows = 32, kBtCplxRows = 24, kBtQuatRows = 12;
// The nf scalar levels, vectors ([batch][nf][N]) and gradients of H = diag(h, h) as nb bands for both spins:
// band 2 q is level q with spin up (x, 0), band 2 q + 1 with spin down (0, x). X, g and their outputs may be null.
void launch_spin_pairs(const double* E, const cx<double>* X, const double* g, int N, int nf, int nb, int batch, double* Eo,
                       cx<double>* Xo, double* go, cudaStream_t s);
// E[b][i] = ev[b][i / 2], i < nb: the doubly degenerate values of a quaternion matrix (backtransform.cu)
void launch_pair_values(const double* ev, int nz, double* E, int nb, int batch, cudaStream_t s);

// refine.cu: FP64 Rayleigh-Ritz in the m-dimensional subspace of FP32 vectors X32 ([batch][m][n]);
// the nb lowest Ritz values go to Eout, optionally vectors / gradients.
constexpr int kRefineMaxSubspace = 40;
// Y's vectors are padded to a multiple of four, which 2 m covers but for m = 1
__host__ __device__ inline size_t refine_work_elems(int n, int m) { return (size_t)n * (m > 1 ? 2 * m : 4); }
// small-solve scratch per matrix, contiguous: S (m x m), A (m x m), then the m x nb (<= m x m) Ritz
// coefficients W at offset 2 m^2
__host__ __device__ inline size_t refine_small_elems(int m, int) { return (size_t)3 * m * m; }
// H is the FP32-pair copy the mixed-path assembly writes (Split<S>); work holds Y = H X. With a
// local potential only (sv.on), H is not formed: H X = V X + diag(kinetic) X from the resident CSR
// of V (every row lists its diagonal, whose FP64 value V_ii + kinetic is split per k as the
// assembly would), summed in the same column order, so Y is the same as from the dense pairs.
// V without its diagonal in transposed ELL form: slot e of row r at [e * N + r], padded with zero
// values (column r) to the widest row, so that threads on consecutive rows load consecutive words.
struct SparseV {
    bool              on;
    int               W;     // slots per row
    const int*        col;   // [W][N]
    const float2*     re;    // [W][N] (hi, lo) of Re V
    const float2*     im;    // [W][N] (hi, lo) of Im V
    const cx<double>* Vloc;  // N x N column-major, for the diagonal
    const double*     rows;  // [batch][N][ROW_STRIDE], for the kinetic term
    int               N;
};
// half > 0: H is quaternionic, only its first half = n / 2 rows are formed, and the vectors come in pairs
// (launch_backtransform_quat's); the other rows of Y follow from those.
// tensor_cores: a complex dense H takes Y = H X on the tensor cores (refine_tc.cu) where refine_tc_pays; status
// gets UEPM_K_NOCONVERGE there if a bounded wait gives up.
//
// A 128-row tile takes the tensor-core kernel the same time whatever the number of vectors (slicing H binds it): a fixed
// part and one that grows with the order n. The FP32-pipe form's time goes with the rows nr, the padded vectors mp
// and n. Projection of 1000 matrices, FP32 pipe against tensor cores, ms: n = 113 mp = 12 0.33 / 0.39, 16 0.41 / 0.41, 20
// 0.51 / 0.44; 137 20 0.70 / 0.79; 181 12 0.76 / 0.89, 20 1.17 / 0.98; 229 12 1.10 / 1.13, 20 1.79 / 1.24; 338 12 2.24 /
// 2.11; quaternionic (nr = n / 2) 274 12 0.88 / 1.26, 20 1.40 / 1.40; 362 12 1.54 / 1.61, 16 1.85 / 1.73.
inline bool refine_tc_pays(int n, int nr, int mp) {
    return 2ll * nr * mp * n >= 128ll * ((nr + 127) / 128) * (17ll * n + 1200);
}
template <typename S>
void launch_refine_project(const typename Split<S>::type* H, int n, int ld, size_t mstride, const cx<float>* X32, int m,
                           S* work, S* small, int batch, cudaStream_t s, const SparseV& sv, int* status = nullptr,
                           bool tensor_cores = true, int half = 0);
// refine_tc.cu: Y (double-single, [r][mp] per matrix, ystride float4 apart) = H X for complex H on
// the tensor cores; false when it does not apply (nothing launched).
bool launch_refine_y_tc(const ds4* H, int n, int ld, size_t mstride, const cx<float>* X32, int m, int mp, void* work,
                        size_t ystride, int* status, int batch, cudaStream_t s, int half = 0);
template <typename S>
void launch_small_eigh(S* small, int m, int nb, double* Eout, S* W, int* status, int batch, cudaStream_t s, int cap = 0);
template <typename S>
void launch_refine_vectors(int n, int m, int nb, const cx<float>* X32, const S* W, cx<double>* Xout, double* grad,
                           const DevParams& P, const double* d_k, const int* d_G, int batch, cudaStream_t s);

}  // namespace uepm
