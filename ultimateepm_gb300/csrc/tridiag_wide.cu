// tridiag_wide.cu -- the FP64 reduction (k_tridiag, tridiag_kernel.cuh) with a cluster of 2, 4 or 8 CTAs per
// matrix, for batches of at most half as many matrices as SMs (one k-point, a short band path), whose
// one-CTA-per-matrix reduction leaves the other SMs' FP64 pipes idle. Same bits as with one CTA.
#include <algorithm>

#include "tridiag_kernel.cuh"
#include "uepm_common.cuh"
#include "uepm_kernels.h"

namespace uepm {
namespace {

template <typename S, int MAXT, int CL>
bool wide_launch(S* H, int n, int ld, size_t mstride, double* d, double* e, S* tq, int* status, int batch, cudaStream_t s) {
    constexpr int NT   = 256;
    const size_t  smem = sizeof(S) * (size_t)(3 + NT / 32) * n;
    const Refusal refuse;
    auto          kern = k_tridiag<S, NT, MAXT, false, CL>;
    if (allow_smem(kern, smem) != cudaSuccess) return refuse();
    cudaLaunchConfig_t  cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id               = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim            = dim3(CL * batch);
    cfg.blockDim           = dim3(NT);
    cfg.dynamicSmemBytes   = smem;
    cfg.stream             = s;
    cfg.attrs              = at;
    cfg.numAttrs           = 1;
    if (cudaLaunchKernelEx(&cfg, kern, H, n, ld, mstride, d, e, tq, status, batch) != cudaSuccess) return refuse();
    count_launch();
    return true;
}

// The largest cluster that gives each matrix SMs of its own: a GPC has room for two clusters of 8 (16 in all
// on 152 SMs), four of 4 and nine of 2.
template <typename S, int MAXT>
bool wide_pick(S* H, int n, int ld, size_t mstride, double* d, double* e, S* tq, int* status, int batch, cudaStream_t s,
               int sms) {
    if (batch * 8 <= sms * 6 / 7) return wide_launch<S, MAXT, 8>(H, n, ld, mstride, d, e, tq, status, batch, s);
    if (batch * 4 <= sms * 6 / 7) return wide_launch<S, MAXT, 4>(H, n, ld, mstride, d, e, tq, status, batch, s);
    return wide_launch<S, MAXT, 2>(H, n, ld, mstride, d, e, tq, status, batch, s);
}

}  // namespace

template <typename S>
bool launch_tridiag_wide(S* H, int n, int ld, size_t mstride, double* d, double* e, S* tq, int* status, int batch,
                         cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // multiply-adds of the first column's product: a cluster of 4 or 8 pays from 7500 of them, one of 2 from 14000
    // (below, the two cluster barriers cost more than the shared work saves)
    constexpr long long C    = sizeof(S) / sizeof(double);
    const long long     cost = C * C * n * n;
    if (batch * 2 > sms || n > 512 || cost < (batch * 4 <= sms * 6 / 7 ? 7500 : 14000)) return false;
    if (n <= 257) return wide_pick<S, 8>(H, n, ld, mstride, d, e, tq, status, batch, s, sms);
    if constexpr (is_quat<S>::value) return false;  // order 256 at most
    else return wide_pick<S, 16>(H, n, ld, mstride, d, e, tq, status, batch, s, sms);
}
template bool launch_tridiag_wide<double>(double*, int, int, size_t, double*, double*, double*, int*, int, cudaStream_t);
template bool launch_tridiag_wide<cx<double>>(cx<double>*, int, int, size_t, double*, double*, cx<double>*, int*, int,
                                              cudaStream_t);
template bool launch_tridiag_wide<qt<double>>(qt<double>*, int, int, size_t, double*, double*, qt<double>*, int*, int,
                                              cudaStream_t);

}  // namespace uepm
