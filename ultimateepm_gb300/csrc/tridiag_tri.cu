// tridiag_tri.cu -- Householder reduction of FP32 quaternion or complex Hermitian matrices to real
// symmetric tridiagonal form with the lower triangle resident in shared memory: the first half of Eigen's
// SelfAdjointEigenSolver called by Hamiltonian::Diagonalize (src/EPP/Hamiltonian.cpp:125-134), for the
// mixed path's spin-orbit matrices of inversion-symmetric crystals (quaternion) and its complex matrices
// of order 175 to 230.
//
// Why quaternions. There H(k) = [[UU, UD], [-conj UD, conj UU]], i.e. the quaternion matrix UU + UD j of
// half the order (time reversal times inversion): 64 / 3 N^3 flops instead of 128 / 3 N^3, a quarter
// of the elements at twice the size, half the columns to reduce one after the other, and each Kramers pair
// once, so that its two levels cannot split. Reduction of 1500 Ge matrices (N = 181): 31.6 ms for the
// blocked complex kernel at order 362, 12.4 ms here; whole mixed solve 42.4 -> 20.3 ms.
//
// One CTA per matrix, a persistent grid over the batch. Only the lower triangle is stored (packed by
// columns). Column jn of the reduction:
//   (a) p = A v of the previous reflector v, summed from the pass's partial sums; mu = Re(v^H p);
//       w = p tau - (mu |tau|^2 / 2) v
//   (b) column jn alone takes the previous reflector's update x = a - v w^H - w v^H, and gives the
//       next reflector: beta real, tau = (beta - alpha) / beta, v' = x (alpha - beta)^-1, v'_{jn+1} = 1
//   (c) ONE pass over the trailing triangle: each element takes the update by (v, w), enters both of
//       its products with v' (y_r += a v'_c, y_c += conj(a) v'_r) and is stored back.
// So each element is read and written once per column, for 2 update and 2 product multiply-adds (of 16
// FMAs each for quaternions, 4 for complex numbers). The operand order is kept throughout (H = I - v tau
// v^H with tau between the vectors; v^H A v and d, e are real), so one code serves both.
//
// The pass. A warp takes units of 32 rows x 8 columns (16 complex): lanes own rows (consecutive lanes read
// consecutive elements of a packed column, so no bank conflicts), the columns' operands are broadcast
// 16-byte loads, row sums stay in registers while the warp's units share a row tile, and the columns'
// 32 real sums are reduced over the lanes by one transposing butterfly per unit. Units are dealt out
// in equal contiguous runs; each run's row sums and each unit's column sums have a slot of their own
// and are added in a fixed order, a strip of columns per warp and one float per lane, so results do not
// depend on scheduling. Per column at N = 137 (quaternion; FMA-bound it would take 1.6 k clocks): the pass
// 8.4 k, issue-bound (60 % of the slots; ~750 instructions per unit for 544 FMA-pipe ones, and few units per
// warp in the later columns), the serial chain of (a) and (b) 2.3 k.
//
// Where the triangle does not fit (N > 159), the first columns run the same pass on the matrix in
// global memory (L2), and the trailing triangle is then copied to shared memory.
#include <algorithm>

#include "uepm_common.cuh"
#include "uepm_kernels.h"

namespace uepm {
namespace {

template <typename S>
struct TriShape {  // columns per unit: their sums are 32 floats, one per lane after the butterfly
    static constexpr int CW = 128 / sizeof(S);
};

constexpr size_t kTriSmem = 227 * 1024;

__host__ __device__ inline int tri_up(int x, int a) { return (x + a - 1) / a * a; }

// Shared-memory layout (in elements of S after the packed triangle) for order n, resident order nres.
template <typename S>
struct TriLayout {
    int np, tiles, units, nw;
    size_t tri, vec, rowp, colp, total;  // bytes
    __host__ __device__ TriLayout(int n, int nres, int nt) {
        constexpr int CW = TriShape<S>::CW, TR = 32, SPT = TR / CW;
        nw    = nt / 32;
        np    = tri_up(n, TR);
        tiles = np / TR;
        // the widest pass starts at row 1: every strip of every tile
        units = SPT * tiles * (tiles + 1) / 2;
        tri   = ((size_t)nres * (nres + 1) / 2 * sizeof(S) + 15) / 16 * 16;
        vec   = (size_t)np * sizeof(S);
        rowp  = (size_t)(nw + tiles) * TR * sizeof(S);
        colp  = (size_t)units * CW * sizeof(S);
        total = tri + 3 * vec + rowp + colp;
    }
};

template <typename S>
struct __align__(16) Pack {
    S e[16 / sizeof(S)];
};

__device__ __forceinline__ float comp_of(cx<float> a, int k) { return k ? a.y : a.x; }
__device__ __forceinline__ float comp_of(qt<float> a, int k) { return k == 0 ? a.w : k == 1 ? a.x : k == 2 ? a.y : a.z; }
__device__ __forceinline__ cx<float> real_only(cx<float> a) { return mk(a.x, 0.f); }
__device__ __forceinline__ qt<float> real_only(qt<float> a) { return mkq(a.w, 0.f, 0.f, 0.f); }

// v conj(w) + w' conj(v'): the whole rank-2 term is formed before it meets the matrix element, so the
// element is rounded once per column instead of once per product (the mixed path's eigenvalue error
// follows the square of the reduction's).
__device__ __forceinline__ cx<float> rank2_term(cx<float> v, cx<float> w, cx<float> w2, cx<float> v2) {
    return mk(fmaf(w2.x, v2.x, fmaf(w2.y, v2.y, fmaf(v.x, w.x, v.y * w.y))),
              fmaf(w2.y, v2.x, fmaf(-w2.x, v2.y, fmaf(v.y, w.x, -v.x * w.y))));
}
__device__ __forceinline__ qt<float> rank2_term(qt<float> v, qt<float> w, qt<float> w2, qt<float> v2) {
    const qt<float> t = mkq(fmaf(v.x, w.x, fmaf(v.y, w.y, fmaf(v.z, w.z, v.w * w.w))),
                            fmaf(v.x, w.w, fmaf(-v.y, w.z, fmaf(v.z, w.y, -v.w * w.x))),
                            fmaf(v.x, w.z, fmaf(v.y, w.w, fmaf(-v.z, w.x, -v.w * w.y))),
                            fmaf(-v.x, w.y, fmaf(v.y, w.x, fmaf(v.z, w.w, -v.w * w.z))));
    return cfma(w2, ST<qt<float>>::conj(v2), t);
}

template <int B>
__device__ __forceinline__ void cp_async_b(void* dst, const void* src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(src), "n"(B) : "memory");
}

// The sums over the 32 lanes of q[0..NV-1]: the lane returns value `lane` (NV = 32) or lane / 2
// (NV = 16, both lanes of a pair).
template <int NV>
__device__ __forceinline__ float lane_transpose_sum(float (&q)[NV], int lane) {
    int h = NV / 2;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (h >= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < NV / 2; ++i) {
                if (i < h) {
                    const float send = up ? q[i] : q[i + h];
                    const float keep = up ? q[i + h] : q[i];
                    q[i]             = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            h >>= 1;
        } else {
            q[0] += __shfl_xor_sync(0xffffffffu, q[0], o);
        }
    }
    return q[0];
}

template <int N>
__device__ __forceinline__ float sum_tree(const float* p) {  // N = 4, 8 or 16 values, 16-byte aligned
    float s[N / 4];
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
        const float4 q = reinterpret_cast<const float4*>(p)[i];
        s[i]           = (q.x + q.y) + (q.z + q.w);
    }
#pragma unroll
    for (int h = N / 8; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) s[i] += s[i + h];
    return s[0];
}

// One unit: row `row` (a lane's), columns c0..c0+CW-1. GEN: the unit meets the diagonal, columns before o
// or rows or columns from n on, so that elements are live or not by lane and column; else all are, and no
// instruction is spent on masks. colp receives the columns' sums.
template <typename S, bool RES, bool GEN>
__device__ __forceinline__ void tri_unit(S* __restrict__ A, int stride, int c0, int o, int n, int row, S vr, S wr, S xr, S& y,
                                         const S* __restrict__ v, const S* __restrict__ w, const S* __restrict__ x,
                                         float* __restrict__ colp, int lane) {
    constexpr int CW = TriShape<S>::CW, C = sizeof(S) / 4, GC = 16 / sizeof(S);
    float f[32];
    S     pre[RES ? 1 : CW];
    if constexpr (!RES) {  // global memory: every load of the unit before its first use
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            const int c = c0 + i;
            pre[i]      = !GEN || (row >= c && row < n && c >= o) ? ldc(A + (size_t)c * stride + row) : ST<S>::zero();
        }
    }
    // cptr[row] is element (row, c); packed columns get shorter by one each
    S*  cptr = RES ? A : A + (size_t)c0 * stride;
    int step = stride - 1;
#pragma unroll
    for (int g = 0; g < CW / GC; ++g) {
        const Pack<S> pv = *reinterpret_cast<const Pack<S>*>(v + c0 + g * GC);
        const Pack<S> pw = *reinterpret_cast<const Pack<S>*>(w + c0 + g * GC);
        const Pack<S> px = *reinterpret_cast<const Pack<S>*>(x + c0 + g * GC);
#pragma unroll
        for (int h = 0; h < GC; ++h) {
            const int  i = g * GC + h, c = c0 + i;
            const bool live = !GEN || (row >= c && row < n && c >= o);
            S          q = ST<S>::zero(), a = q;
            if (live) {
                if constexpr (RES) a = ldc(cptr + row);
                else a = pre[i];
                a = csub(a, rank2_term(vr, pw.e[h], wr, pv.e[h]));
                if constexpr (GEN) {
                    if (row == c) a = real_only(a);
                }
                stc(cptr + row, a);
                y = cfma(a, px.e[h], y);
                if (!GEN || row != c) q = cfmac(a, xr, q);
            }
#pragma unroll
            for (int k = 0; k < C; ++k) f[i * C + k] = comp_of(q, k);
            if constexpr (RES) {
                cptr += step;
                --step;
            } else {
                cptr += stride;
            }
        }
    }
    colp[lane] = lane_transpose_sum<32>(f, lane);
}

// A warp's run of units in the pass over rows and columns o..: the first unit u and the end u1, the row
// tile t of u, the tile's first unit and its number of units.
struct TriRun {
    int u, u1, t, base, cnt;
};
template <typename S, int NW>
__device__ __forceinline__ int tri_units(int o, int n, int tiles, int t) {  // units of row tile t
    constexpr int CW = TriShape<S>::CW, SPT = 32 / CW;
    const int     st0 = o / CW;
    return t == tiles - 1 ? min(SPT * tiles, (n + CW - 1) / CW) - st0 : SPT * (t + 1) - st0;
}
template <typename S, int NW>
__device__ __forceinline__ TriRun tri_run(int o, int n, int tiles, int warp) {
    constexpr int CW = TriShape<S>::CW, SPT = 32 / CW;
    const int     T0 = o / 32, st0 = o / CW;
    // units of tile t < tiles - 1: SPT (t + 1) - st0; the last tile's strips end at column n - 1
    const int U = SPT * ((tiles - 1) * tiles / 2 - T0 * (T0 + 1) / 2) - st0 * (tiles - 1 - T0) +
                  tri_units<S, NW>(o, n, tiles, tiles - 1);
    TriRun r;
    // equal runs; with fewer units than warps one each to the first U (no run between is empty)
    r.u    = U >= NW ? U * warp / NW : min(warp, U);
    r.u1   = U >= NW ? U * (warp + 1) / NW : min(warp + 1, U);
    r.t    = T0;
    r.base = 0;
    r.cnt  = tri_units<S, NW>(o, n, tiles, T0);
    while (r.u >= r.base + r.cnt && r.t < tiles - 1) {
        r.base += r.cnt;
        ++r.t;
        r.cnt = tri_units<S, NW>(o, n, tiles, r.t);
    }
    return r;
}

template <typename S, int NT, int MINB, bool SPLIT>
__global__ void __launch_bounds__(NT, MINB)
    k_tridiag_tri(S* __restrict__ H, int n, int nres, int ld, size_t mstride, float* __restrict__ dOut,
                  float* __restrict__ eOut, S* __restrict__ tqOut, int* __restrict__ status, int batch) {
    constexpr int C = sizeof(S) / 4, CW = TriShape<S>::CW, TR = 32, SPT = TR / CW, NW = NT / 32;
    static_assert(CW * C == 32, "a strip's sums are one float per lane");
    constexpr int RT = NT >= 512 ? 1 : 2;  // rows per thread in (b): n <= RT NT
    constexpr int MAXT = 16;
    extern __shared__ __align__(16) unsigned char smraw[];
    const TriLayout<S> L(n, nres, NT);
    S* tri  = reinterpret_cast<S*>(smraw);
    S* vec  = reinterpret_cast<S*>(smraw + L.tri);
    S* wv   = vec + 2 * L.np;
    S* rowp = reinterpret_cast<S*>(smraw + L.tri + 3 * L.vec);
    S* colp = reinterpret_cast<S*>(smraw + L.tri + 3 * L.vec + L.rowp);
    __shared__ __align__(16) float s_mu[NW], s_ss[NW];
    __shared__ S             s_alpha, s_p0;
    __shared__ unsigned char s_run[2 * MAXT];  // first and last warp of each tile's runs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int R0 = SPLIT ? n - nres : 0;  // first resident row and column
    const int tiles = L.tiles, strips = (n + CW - 1) / CW;

    for (int b = blockIdx.x; b < batch; b += gridDim.x) {
        S*     Ag = H + (size_t)b * mstride;
        float* dB = dOut + (size_t)b * n;
        float* eB = eOut + (size_t)b * n;
        S*     tB = tqOut + (size_t)b * n;
        bool   bad = false;
        for (int i = tid; i < 3 * L.np; i += NT) vec[i] = ST<S>::zero();
        S      tau = ST<S>::zero();
        int    cur = 0;  // v is vec + cur np, the next reflector goes to the other half
        TriRun run = tri_run<S, NW>(1, n, tiles, warp);
        for (int jn = 0; jn < n; ++jn) {
            if (jn == R0) {  // the trailing triangle to shared memory
                __syncthreads();
                for (int c = R0 + warp; c < n; c += NW) {
                    const int cl = c - R0;
                    S*        dst = tri + (size_t)cl * nres - cl * (cl + 1) / 2 - R0;
                    for (int r = c + lane; r < n; r += 32) cp_async_b<sizeof(S)>(dst + r, Ag + (size_t)c * ld + r);
                }
                cp_async_wait_all();
                __syncthreads();
            }
            S*        v  = vec + cur * L.np;
            S*        vn = vec + (cur ^ 1) * L.np;
            // ---- (a) p = A v from the partial sums, a strip of CW rows (one float per lane) at a time --
            if (jn > 0) {
                float     mu = 0.f;
                const int T0 = jn / TR, st0 = jn / CW;
                for (int st = st0 + warp; st < strips; st += NW) {
                    const int    t = st / SPT, q1 = s_run[t + MAXT];
                    const float* pr = reinterpret_cast<const float*>(rowp + t * TR + (st - t * SPT) * CW) + lane;
                    const float* pc = reinterpret_cast<const float*>(colp) + lane;
                    float        a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
                    for (int q = s_run[t]; q <= q1; q += 4) {  // the tile's runs, four loads in flight
                        a0 += pr[q * TR * C];
                        if (q + 1 <= q1) a1 += pr[(q + 1) * TR * C];
                        if (q + 2 <= q1) a2 += pr[(q + 2) * TR * C];
                        if (q + 3 <= q1) a3 += pr[(q + 3) * TR * C];
                    }
                    // units (tt, st) of the column's strip, tt = t .. tiles - 1
                    int u = SPT * (t * (t + 1) / 2 - T0 * (T0 + 1) / 2) - st0 * (t - T0) + (st - st0);
                    for (int tt = t; tt < tiles; tt += 4) {
                        const int d1 = SPT * (tt + 1) - st0;
                        a0 += pc[u * 32];
                        if (tt + 1 < tiles) a1 += pc[(u + d1) * 32];
                        if (tt + 2 < tiles) a2 += pc[(u + 2 * d1 + SPT) * 32];
                        if (tt + 3 < tiles) a3 += pc[(u + 3 * d1 + 3 * SPT) * 32];
                        u += 4 * d1 + 6 * SPT;
                    }
                    const float a = (a0 + a1) + (a2 + a3);
                    const int   r = st * CW + lane / C;
                    if (r >= jn) {  // Re(conj(v) p) is the sum over components
                        mu = fmaf(reinterpret_cast<const float*>(v)[st * 32 + lane], a, mu);
                        reinterpret_cast<float*>(wv)[st * 32 + lane] = a;
                        if (r == jn) reinterpret_cast<float*>(&s_p0)[lane & (C - 1)] = a;
                    }
                }
                mu = warp_sum(mu);
                if (lane == 0) s_mu[warp] = mu;
                __syncthreads();
            }
            // ---- (b) w, column jn and its reflector: a row per thread; warps past their last row wait ---
            const bool live = warp * 32 + 31 + (RT - 1) * NT >= jn && warp * 32 < n;
            S          x[RT];
            float      ss = 0.f;
            if (live) {
                const int cj   = jn - R0;
                const S*  acol = !SPLIT || jn >= R0 ? tri + (size_t)cj * nres - cj * (cj + 1) / 2 - R0 : Ag + (size_t)jn * ld;
                float     g = 0.f;
                S         w0 = ST<S>::zero();
                if (jn > 0) {
                    g  = -0.5f * sum_tree<NW>(s_mu) * ST<S>::norm(tau);
                    w0 = cadd(cmul(s_p0, tau), cscale(ST<S>::one(), g));  // v_jn = 1
                }
#pragma unroll
                for (int k = 0; k < RT; ++k) {
                    const int r = tid + k * NT;
                    x[k]        = ST<S>::zero();
                    if (r < jn || r >= n) continue;
                    x[k] = ldc(acol + r);
                    if (jn > 0) {
                        const S vr = ldc(v + r), wr = cadd(cmul(ldc(wv + r), tau), cscale(vr, g));
                        stc(wv + r, wr);
                        x[k] = csub(cfms_conjb(vr, w0, x[k]), wr);
                    }
                    if (r == jn) {
                        dB[jn] = ST<S>::re(x[k]);
                        if (!isfinite(ST<S>::re(x[k]))) bad = true;
                        stc(vn + r, ST<S>::zero());
                    } else if (r == jn + 1) {
                        s_alpha = x[k];
                    } else {
                        ss += ST<S>::norm(x[k]);
                    }
                }
                ss = warp_sum(ss);
            }
            if (jn == n - 1) {
                if (tid == 0) {
                    eB[jn] = 0.f;
                    stc(tB + jn, ST<S>::zero());
                }
                break;
            }
            if (lane == 0) s_ss[warp] = ss;
            __syncthreads();
            if (live) {
                ss = sum_tree<NW>(s_ss);
                const S     al = s_alpha;
                const float im = imag_norm(al), ar = ST<S>::re(al);
                float       beta = ar;
                S           sc = ST<S>::zero();
                tau            = ST<S>::zero();
                if (ss > num<float>::tiny() || im > num<float>::tiny()) {
                    beta = sqrtf(fmaf(ar, ar, ss + im));
                    if (ar >= 0.f) beta = -beta;
                    const S     df = csub(al, cscale(ST<S>::one(), beta));  // alpha - beta
                    tau            = cscale(df, -1.f / beta);
                    sc             = cscale(ST<S>::conj(df), 1.f / ST<S>::norm(df));
                }
#pragma unroll
                for (int k = 0; k < RT; ++k) {
                    const int r = tid + k * NT;
                    if (r == jn + 1) {
                        eB[jn] = beta;
                        stc(tB + jn, tau);
                        if (!isfinite(beta)) bad = true;
                        stc(vn + r, ST<S>::one());
                    }
                    if (r > jn + 1 && r < n) {
                        const S vr = cmul(x[k], sc);
                        stc(vn + r, vr);
                        stc(Ag + (size_t)jn * ld + r, vr);
                    }
                }
            }
            __syncthreads();
            // ---- (c) the pass over rows and columns o.. --------------------------------------------
            const int o = jn + 1, st0 = o / CW;
            while (run.u < run.u1) {
                const int row = run.t * TR + lane;
                const S   vr = ldc(v + row), wr = ldc(wv + row), xr = ldc(vn + row);
                S         y  = ST<S>::zero();
                const int ue = min(run.u1, run.base + run.cnt);
                if (lane == 0) {
                    if (run.u == run.base) s_run[run.t] = (unsigned char)warp;
                    if (ue == run.base + run.cnt) s_run[run.t + MAXT] = (unsigned char)warp;
                }
                const bool ragged = run.t == tiles - 1 && n < L.np;
                for (; run.u < ue; ++run.u) {
                    const int  c0  = (st0 + run.u - run.base) * CW;
                    const bool gen = c0 + CW > run.t * TR || c0 < o || ragged;
                    float*     cp  = reinterpret_cast<float*>(colp + run.u * CW);
                    if (!SPLIT || jn >= R0) {
                        // c0 may lie before the first resident column: those columns are not live
                        const int cl = c0 - R0;
                        S*        tc = tri + (cl * nres - cl * (cl + 1) / 2 - R0);
                        if (gen) tri_unit<S, true, true>(tc, nres - cl, c0, o, n, row, vr, wr, xr, y, v, wv, vn, cp, lane);
                        else tri_unit<S, true, false>(tc, nres - cl, c0, o, n, row, vr, wr, xr, y, v, wv, vn, cp, lane);
                    } else if constexpr (SPLIT) {
                        if (gen) tri_unit<S, false, true>(Ag, ld, c0, o, n, row, vr, wr, xr, y, v, wv, vn, cp, lane);
                        else tri_unit<S, false, false>(Ag, ld, c0, o, n, row, vr, wr, xr, y, v, wv, vn, cp, lane);
                    }
                }
                stc(rowp + (warp + run.t) * TR + lane, y);
                if (run.u < run.u1) {
                    run.base += run.cnt;
                    ++run.t;
                    run.cnt = tri_units<S, NW>(o, n, tiles, run.t);
                }
            }
            if (o + 1 < n) run = tri_run<S, NW>(o + 1, n, tiles, warp);  // the next pass, while others finish
            __syncthreads();
            cur ^= 1;
        }
        bad = __syncthreads_or(bad);
        if (tid == 0 && bad && status) atomicOr(status + b, 2);  // UEPM_K_NONFINITE
    }
}

template <typename S, int NT, int MINB>
bool tri_launch(S* H, int n, int ld, size_t mstride, float* d, float* e, S* tq, int* status, int batch, cudaStream_t s) {
    int nres = n;
    while (nres > 2 && TriLayout<S>(n, nres, NT).total > kMaxDynamicSmem) --nres;
    const size_t smem = TriLayout<S>(n, nres, NT).total;
    auto         kern = k_tridiag_tri<S, NT, MINB, false>;
    if constexpr (MINB == 1) {  // where more CTAs share an SM their triangles fit as they are
        if (nres < n) kern = k_tridiag_tri<S, NT, MINB, true>;
    }
    const Refusal refuse;
    if (allow_smem(kern, smem) != cudaSuccess) return refuse();
    int dev = 0, sms = 0, fit = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, NT, smem) != cudaSuccess || fit < 1) return refuse();
    const int grid = std::min(batch, std::max(1, sms) * fit);
    kern<<<grid, NT, smem, s>>>(H, n, nres, ld, mstride, d, e, tq, status, batch);
    count_launch();
    return true;
}

}  // namespace

// 16 warps per SM at the kernel's 128 registers: CTAs of 128 threads where four fit an SM's shared memory
// (N <= 74), of 256 where two do (N <= 109), else one of 512. Complex matrices come at orders that fill an SM
// (launch_tridiag says why those): CTAs of 512 alone.
template <typename S>
bool launch_tridiag_tri(S* H, int n, int ld, size_t mstride, float* d, float* e, S* tq, int* status, int batch,
                        cudaStream_t s) {
    if constexpr (is_quat<S>::value) {
        if (n < 1 || n > 256) return false;
        if (4 * (TriLayout<S>(n, n, 128).total + 2048) <= kTriSmem)
            return tri_launch<S, 128, 4>(H, n, ld, mstride, d, e, tq, status, batch, s);
        if (2 * (TriLayout<S>(n, n, 256).total + 2048) <= kTriSmem)
            return tri_launch<S, 256, 2>(H, n, ld, mstride, d, e, tq, status, batch, s);
    } else {
        if (n < kTriMinCplx || n > kTriMaxCplx) return false;
    }
    return tri_launch<S, 512, 1>(H, n, ld, mstride, d, e, tq, status, batch, s);
}
template bool launch_tridiag_tri<cx<float>>(cx<float>*, int, int, size_t, float*, float*, cx<float>*, int*, int,
                                            cudaStream_t);
template bool launch_tridiag_tri<qt<float>>(qt<float>*, int, int, size_t, float*, float*, qt<float>*, int*, int,
                                            cudaStream_t);

}  // namespace uepm
