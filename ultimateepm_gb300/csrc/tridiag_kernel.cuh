// tridiag_kernel.cuh -- k_tridiag, the Householder reduction with one CTA (tridiag.cu) or one cluster of CTAs
// (tridiag_wide.cu) per matrix.
#pragma once

#include <cooperative_groups.h>

#include "uepm_common.cuh"

namespace uepm {

namespace cg = cooperative_groups;

constexpr int kUpd = 4;  // elements per thread per round of the rank-2 update

// SMEM = true: the matrix is copied into shared memory (leading dimension n | 1, odd, so that the
// mirrored row-wise stores do not collide on banks), reduced there, and its reflector columns are
// written back. Used where n x n fits (the FP32 reductions of the mixed path), because those are
// bound by memory latency rather than by arithmetic.
// Global-memory variant: CTAs per SM that must fit the register file (the persistent grid relies on
// several to hide L2/DRAM latency): 5 for the real and complex-FP32 matrices up to n = 161, 4 above,
// fewer for complex FP64 with many row chunks (whose accumulators alone take 4 MAXT registers).
template <typename S, int MAXT>
constexpr int tridiag_min_blocks() {
    return is_quat<S>::value ? 2 : sizeof(S) * MAXT <= 8 * 5 ? 5 : (sizeof(S) <= 8 || MAXT <= 5 ? 4 : (MAXT <= 8 ? 3 : 2));
}

// Column c and row r of element e of the lower triangle of order m, numbered down the columns: column c starts
// at c m - c (c - 1) / 2. The root in FP32 (its argument is exact below 2^24) and at most a step from there;
// walking there column by column took the update of n = 137 most of its time with few elements per thread.
__device__ __forceinline__ void tri_element(int e, int m, int& c, int& r) {
    const float q = 2.f * m + 1.f;
    c             = (int)(0.5f * (q - sqrtf(fmaxf(q * q - 8.f * e, 0.f))));
    int s         = c * m - c * (c - 1) / 2;
    if (s > e) {
        --c;
        s -= m - c;
    } else if (e >= s + m - c) {
        s += m - c;
        ++c;
    }
    r = c + e - s;
}

template <typename T>
__device__ __forceinline__ T shfl_xor(T a, int o) {
    return __shfl_xor_sync(0xffffffffu, a, o);
}
template <typename T>
__device__ __forceinline__ cx<T> shfl_xor(cx<T> a, int o) {
    return mk(shfl_xor(a.x, o), shfl_xor(a.y, o));
}
template <typename T>
__device__ __forceinline__ qt<T> shfl_xor(qt<T> a, int o) {
    return mkq(shfl_xor(a.w, o), shfl_xor(a.x, o), shfl_xor(a.y, o), shfl_xor(a.z, o));
}

// The tests of the reflector's serial chain by bit pattern: a dependent FP64 compare costs it ~110 clocks.
__device__ __forceinline__ bool tiny_or_less(double x) {  // 0 <= x <= the smallest normal number; false for NaN
    return (unsigned long long)__double_as_longlong(x) <= 0x0010000000000000ull;
}
__device__ __forceinline__ bool tiny_or_less(float x) { return x <= num<float>::tiny(); }
__device__ __forceinline__ bool non_negative(double x) { return __double2hiint(x) >= 0; }  // -0 counts as negative
__device__ __forceinline__ bool non_negative(float x) { return x >= 0.f; }
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool finite_bits(float x) { return isfinite(x); }

// zlarfg's scalars of the column (c0; tail), tail2 = |tail|^2: beta real, th = (beta - c0) / beta,
// sc = 1 / (c0 - beta). False where the column is its own (th = 0).
template <typename S>
__device__ __forceinline__ bool reflector_scalars(S c0, typename ST<S>::R tail2, typename ST<S>::R& beta, S& th, S& sc) {
    using R = typename ST<S>::R;
    if constexpr (is_quat<S>::value) {
        quat_reflector(c0, tail2, num<R>::tiny(), beta, th, sc);
        return ST<S>::norm(th) != R(0);
    } else {
        const R c0r = ST<S>::re(c0), c0i = ST<S>::im(c0);
        if (tiny_or_less(tail2) && (!ST<S>::cplx || tiny_or_less(c0i * c0i))) {
            th   = ST<S>::zero();
            sc   = ST<S>::zero();
            beta = c0r;
            return false;
        }
        R ib;
        sqrt_pair(fma(c0r, c0r, ST<S>::cplx ? fma(c0i, c0i, tail2) : tail2), beta, ib);
        if (non_negative(c0r)) {
            beta = -beta;
            ib   = -ib;
        }
        const R ar = c0r - beta;
        th         = ST<S>::make((beta - c0r) * ib, -c0i * ib);
        if constexpr (ST<S>::cplx) {
            const R den = recip(fma(ar, ar, c0i * c0i));
            sc          = ST<S>::make(ar * den, -c0i * den);
        } else {
            sc = recip(ar);
        }
        return true;
    }
}

// Warp vw's part of (A v)_r over its columns c = vw mod NW, A full, m x m, lanes own rows; put(r, value)
// receives it. TF full 32-row chunks; the remaining rows take one instruction for 1, 2 or 4 columns (a lane
// group of 32, 16 or 8 lanes each). The chunk count is a template parameter, so that no dead chunk is issued:
// predicated off they still took the FP64 pipe (91 k instructions per matrix at n = 137, 71 k so).
// P > 1: the work of a virtual warp vw is shared by P warps, sub = 0..P-1: chunks sub, sub + P, ..., and the
// remaining rows with the next chunk's warp. Each row's chain of FMAs is the same.
template <typename S, int NW, int TF, int P, typename Put>
__device__ __forceinline__ void product_t(const S* __restrict__ A, int ld, int m, const S* v, int vw, int sub, int lane, Put put) {
    const int tf = m >> 5;
    if constexpr (TF > 0) {
        S acc[TF];
#pragma unroll
        for (int t = 0; t < TF; ++t) acc[t] = ST<S>::zero();
        constexpr bool kExact = TF <= 8;  // TF is the warp's chunk count, else an upper bound of it
        // U columns' loads in flight: a warp alone on its scheduler otherwise waits out the L2 latency per column
        constexpr int U = P > 1 ? (TF * sizeof(S) <= 16 ? 8 : 4) : 1;
        int           c = vw;
        for (; U > 1 && c + (U - 1) * NW < m; c += U * NW) {
            S a[U][TF];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int t = 0; t < TF; ++t)
                    a[u][t] = kExact || sub + P * t < tf
                                  ? ldc(A + (size_t)(c + u * NW) * ld + lane + 32 * (sub + P * t)) : ST<S>::zero();
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int t = 0; t < TF; ++t) acc[t] = cfma(a[u][t], v[c + u * NW], acc[t]);
        }
        for (; c < m; c += NW) {
            const S* ac = A + (size_t)c * ld + lane + 32 * sub;
            const S  vc = v[c];
            S        a[TF];
#pragma unroll
            for (int t = 0; t < TF; ++t) a[t] = kExact || sub + P * t < tf ? ldc(ac + 32 * P * t) : ST<S>::zero();
#pragma unroll
            for (int t = 0; t < TF; ++t) acc[t] = cfma(a[t], vc, acc[t]);
        }
#pragma unroll
        for (int t = 0; t < TF; ++t)
            if (kExact || sub + P * t < tf) put(lane + 32 * (sub + P * t), acc[t]);
    }
    const int rem = m & 31;
    if (rem && (P == 1 || tf % P == sub)) {
        const int lg = rem <= 8 ? 3 : rem <= 16 ? 4 : 5, g = 32 >> lg;  // 2^lg lanes per column
        const int cs = lane >> lg, rr = (m & ~31) + (lane & ((1 << lg) - 1));
        const S*  ar = A + rr;
        S         at = ST<S>::zero();
        int       c0 = vw * g;
        for (; c0 + 3 * NW * g + g <= m; c0 += 4 * NW * g) {
            S a[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) a[q] = rr < m ? ldc(ar + (size_t)(c0 + q * NW * g + cs) * ld) : ST<S>::zero();
#pragma unroll
            for (int q = 0; q < 4; ++q) at = cfma(a[q], v[c0 + q * NW * g + cs], at);
        }
        for (; c0 < m; c0 += NW * g) {
            const int c = c0 + cs;
            if (c0 + g <= m || c < m) at = cfma(rr < m ? ldc(ar + (size_t)c * ld) : ST<S>::zero(), v[c], at);
        }
        for (int q = 16; q >= (1 << lg); q >>= 1) at = cadd(at, shfl_xor(at, q));
        if (cs == 0 && rr < m) put(rr, at);
    }
}
template <typename S, int NW, int MAXT, int P, typename Put>
__device__ __forceinline__ void product(const S* A, int ld, int m, const S* v, int vw, int sub, int lane, Put put) {
    constexpr int M  = (MAXT + P - 1) / P;
    const int     tf = m >> 5;
#define UEPM_PR(TF_) product_t<S, NW, TF_, P>(A, ld, m, v, vw, sub, lane, put)
    switch (P == 1 ? tf : tf > sub ? (tf - sub + P - 1) / P : 0) {
        case 0: UEPM_PR(0); break;
        case 1: UEPM_PR(1); break;
        case 2: if constexpr (M >= 2) UEPM_PR(2); break;
        case 3: if constexpr (M >= 3) UEPM_PR(3); break;
        case 4: if constexpr (M >= 4) UEPM_PR(4); break;
        case 5: if constexpr (M >= 5) UEPM_PR(5); break;
        case 6: if constexpr (M >= 6) UEPM_PR(6); break;
        case 7: if constexpr (M >= 7) UEPM_PR(7); break;
        case 8: if constexpr (M >= 8) UEPM_PR(8); break;
        case 9: case 10: case 11:
        case 12: if constexpr (M >= 12) UEPM_PR(12); break;
        default: if constexpr (M >= 16) UEPM_PR(16); break;
    }
#undef UEPM_PR
}

// CL > 1 (launched as clusters of CL CTAs): each matrix is reduced by a cluster, for batches that leave most
// SMs idle. The product's NW virtual warps and the update's elements are dealt out over the cluster, the
// partial products and the next column go to every CTA's shared memory (distributed shared memory), and the
// rest is done by every CTA for itself; rank 0 writes the outputs. Every sum keeps its order, so the results
// are the same bits for every CL. Two cluster barriers per column, and one before the first.
template <typename S, int NT, int MAXT, bool SMEM, int CL = 1>
__global__ void __launch_bounds__(NT, SMEM || CL > 1 ? 1 : tridiag_min_blocks<S, MAXT>()) k_tridiag(S* __restrict__ H, int n, int ldg, size_t mstride,
                                                typename ST<S>::R* __restrict__ dOut, typename ST<S>::R* __restrict__ eOut,
                                                S* __restrict__ tqOut, int* __restrict__ status, int batch) {
    using R       = typename ST<S>::R;
    constexpr int NW = NT / 32;
    const int lds = n | 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    S*        As   = reinterpret_cast<S*>(smraw);  // SMEM: n x lds
    S*        v    = SMEM ? As + (size_t)n * lds : As;  // n
    S*        w    = v + n;                        // n
    S*        pacc = w + n;                        // NW * n
    S*        xs   = pacc + NW * n;                // CL > 1: n, the next column
    const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0;
    auto      sync_cluster = [&]() {
        if constexpr (CL > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    auto to_all = [&](S* p, S val) {  // the same place in every CTA of the cluster
        if constexpr (CL > 1) {
#pragma unroll
            for (int q = 0; q < CL; ++q) stc(cg::this_cluster().map_shared_rank(p, q), val);
        } else {
            *p = val;
        }
    };
    __shared__ S   s_th, s_sc, red2[NW];
    __shared__ R   red[NW];
    __shared__ int s_skip;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // The grid may be smaller than the batch: each CTA reduces matrices b, b + gridDim.x, ... so the
    // number of matrices in flight (and their L2 working set) is set by the launch, not the batch.
    for (int b = blockIdx.x / CL; b < batch; b += gridDim.x / CL) {
    S*        Ag  = H + (size_t)b * mstride;
    bool      bad = false;
    S*        A   = SMEM ? As : Ag;
    const int ld  = SMEM ? lds : ldg;
    if (SMEM) {
        for (int q = tid; q < n * n; q += NT) {
            const int c = q / n, r = q - c * n;
            As[(size_t)c * lds + r] = Ag[(size_t)c * ldg + r];
        }
        __syncthreads();
    }

    // xc: this thread's rows (tid, tid + NT) of the column to reduce next, and ss their norm's sum over
    // the tail; from the matrix for column 0, from the previous column's update afterwards
    S xc[2];
    R ss = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int r = tid + k * NT;  // row o + r - 1 of column 0: r = 0 is the diagonal
        xc[k]       = r < n ? ldc(A + r) : ST<S>::zero();
        if (r >= 2 && r < n) ss += ST<S>::norm(xc[k]);
    }
    // Every CTA of the cluster has read column 0 before rank 0 writes its reflector there, and has started before
    // a peer's to_all writes into its shared memory.
    if constexpr (CL > 1) sync_cluster();
    for (int i = 0; i < n - 1; ++i) {
        const int o = i + 1, m = n - o;
        S*        col = A + (size_t)i * ld + o;
        if constexpr (CL > 1) {
            if (i > 0) {
                ss = 0;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int r = tid + k * NT;
                    xc[k]       = r <= m ? ldc(xs + r) : ST<S>::zero();
                    if (r >= 2 && r <= m) ss += ST<S>::norm(xc[k]);
                }
            }
        }

        // ---- Householder vector of A[o:, i] -------------------------------------------------
        // The column's rows are in the registers of the threads that updated it (thread r: row i + r),
        // so nothing is read back, and each warp that holds some sums its squares.
        if (32 * warp <= m) {
            ss = warp_sum(ss);
            if (lane == 0) red[warp] = ss;
        }
        if (tid == 1) s_sc = xc[0];  // c0
        __syncthreads();
        if (warp == 0) {
            R tail2 = red[0];
            for (int q = 1; q < NW && 32 * q <= m; ++q) tail2 += red[q];
            R beta;
            S th, sc;
            const bool reflect = reflector_scalars(s_sc, tail2, beta, th, sc);
            __syncwarp();
            if (lane == 0) {
                const R di = ST<S>::re(xc[0]);
                s_th   = th;
                s_sc   = sc;
                s_skip = !reflect;
                if (rank == 0) {
                    dOut[(size_t)b * n + i]  = di;
                    eOut[(size_t)b * n + i]  = beta;
                    tqOut[(size_t)b * n + i] = th;
                    stc(col, ST<S>::make(beta, R(0)));
                }
                if (!finite_bits(beta) || !finite_bits(di)) bad = true;
            }
        }
        __syncthreads();
        const S th = s_th, sc = s_sc;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int r = tid + k * NT - 1;
            if (r >= 0 && r < m) {
                const S vr = r == 0 ? ST<S>::one() : cmul(xc[k], sc);
                v[r]       = vr;
                if (r > 0 && rank == 0) stc(col + r, vr);
            }
        }
        __syncthreads();
        ss = 0;
        if (s_skip) {  // the next column as it stands
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int r = tid + k * NT;
                xc[k]       = r < m ? ldc(A + (size_t)o * ld + o + r) : ST<S>::zero();
                if (r >= 2 && r < m) ss += ST<S>::norm(xc[k]);
                if (CL > 1 && r < m) stc(xs + r, xc[k]);  // every CTA has it; its own copy
            }
            sync_cluster();
            continue;
        }

        // ---- p = A22 v (full storage): warps own columns, lanes own rows ----------------------
        {
            const int vw = CL > 1 ? rank * (NW / CL) + warp / CL : warp;
            product<S, NW, MAXT, CL>(A + (size_t)o * ld + o, ld, m, v, vw, warp % CL, lane,
                                     [&](int r, S val) { to_all(pacc + vw * n + r, val); });
        }
        sync_cluster();

        // ---- w = tau p; alpha = -tau/2 (w^H v) -------------------------------------------------
        S wr[2], part2 = ST<S>::zero();
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int r = tid + k * NT;
            wr[k]       = ST<S>::zero();
            if (r < m) {
                static_assert(NW == 8, "the tree below");
                const S* pr = pacc + r;
                const S  p  = cadd(cadd(cadd(pr[0], pr[n]), cadd(pr[2 * n], pr[3 * n])),
                                   cadd(cadd(pr[4 * n], pr[5 * n]), cadd(pr[6 * n], pr[7 * n])));
                if constexpr (is_quat<S>::value) {  // w = p tau, and Re(v^H p)
                    wr[k] = cmul(p, th);
                    part2.w += re_dot(v[r], p);
                } else {
                    wr[k] = cmul(th, p);
                    part2 = cfmac(wr[k], v[r], part2);
                }
            }
        }
        if (32 * warp < m) {
            if constexpr (ST<S>::cplx) {
                part2 = warp_sum(part2);
            } else {
                part2 = ST<S>::make(warp_sum(ST<S>::re(part2)), R(0));
            }
            if (lane == 0) red2[warp] = part2;
        }
        __syncthreads();
        if (32 * warp < m) {
            S wv = red2[0];
            for (int q = 1; q < NW && 32 * q < m; ++q) {
                if constexpr (is_quat<S>::value) wv.w += red2[q].w;
                else wv = cadd(wv, red2[q]);
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int r = tid + k * NT;
                if (r < m) {
                    if constexpr (is_quat<S>::value)  // v^H A v is real: -|tau|^2 (v^H p) / 2
                        w[r] = cadd(wr[k], cscale(v[r], R(-0.5) * wv.w * ST<S>::norm(th)));
                    else w[r] = cfma(cscale(cmul(th, wv), R(-0.5)), v[r], wr[k]);
                }
            }
        }
        __syncthreads();

        // ---- A22 -= v w^H + w v^H: lower triangle computed, upper mirrored -------------------
        // The m (m + 1) / 2 lower elements in column-major order, element e to thread e mod NT:
        // consecutive threads take consecutive rows of a column (coalesced), and only the last
        // round has idle lanes (per-column 32-row chunks left ~16 idle lanes in every column).
        // Each thread takes its elements kUpd at a time, all loads first, so that kUpd loads per
        // thread are in flight (one at a time left every element waiting a full L2/DRAM latency).
        // The first m elements are the next column to reduce: they stay in xc.
        {
            const int tot = m * (m + 1) / 2;
            xc[0] = xc[1] = ST<S>::zero();
            for (int e0 = tid + rank * NT; e0 < tot; e0 += kUpd * CL * NT) {
                int cq[kUpd], rq[kUpd];
                S   aq[kUpd];
#pragma unroll
                for (int q = 0; q < kUpd; ++q) tri_element(min(e0 + q * CL * NT, tot - 1), m, cq[q], rq[q]);
#pragma unroll
                for (int q = 0; q < kUpd; ++q)
                    if (e0 + q * CL * NT < tot) aq[q] = ldc(A + (size_t)(o + cq[q]) * ld + o + rq[q]);
#pragma unroll
                for (int q = 0; q < kUpd; ++q) {
                    if (e0 + q * CL * NT >= tot) break;
                    const int cc = cq[q], rr = rq[q];
                    S         a  = cfms_conjb(v[rr], w[cc], aq[q]);
                    a            = cfms_conjb(w[rr], v[cc], a);
                    if (rr == cc) {
                        a = ST<S>::make(ST<S>::re(a), R(0));
                    } else {
                        stc(A + (size_t)(o + rr) * ld + (o + cc), ST<S>::conj(a));
                    }
                    stc(A + (size_t)(o + cc) * ld + o + rr, a);
                    if constexpr (CL > 1) {
                        if (cc == 0) to_all(xs + rr, a);
                    } else if (q < 2 && cc == 0) {  // e0 = tid: rows tid and tid + NT of the next column
                        xc[q] = a;
                        if (rr >= 2) ss += ST<S>::norm(a);
                    }
                }
            }
        }
        sync_cluster();
    }
    if (tid == 0 && rank == 0) {
        const R dl = ST<S>::re(CL > 1 && n > 1 ? xs[0] : xc[0]);
        dOut[(size_t)b * n + n - 1] = dl;
        eOut[(size_t)b * n + n - 1] = R(0);
        tqOut[(size_t)b * n + n - 1] = ST<S>::zero();
        if (!isfinite(dl)) bad = true;
        if (bad && status) atomicOr(status + b, 2);  // UEPM_K_NONFINITE
    }
    if (SMEM) {
        // reflector tails (column i, rows i+2..n-1) for the back-transformation
        __syncthreads();
        for (int q = tid; q < n * n; q += NT) {
            const int c = q / n, r = q - c * n;
            if (r > c + 1) Ag[(size_t)c * ldg + r] = As[(size_t)c * lds + r];
        }
    }
    __syncthreads();  // shared memory is reused by the CTA's next matrix
    }
}

}  // namespace uepm
