// Density-fitted ERI producer of the (T) inputs and its VJP, float64 on the
// tensor pipe (DMMA, mma.sync m8n8k4 .f64).
//
// pyscfad's DF-CCSD forms ovoo = Lov^T Loo, ovov = Lov^T Lov and
// ovvv = Lov^T Lvv from the three-index factors (pyscfad/cc/dfccsd.py:73-88);
// the (T) driver then transposes them into the kernel layouts vooo and vvop
// (pyscfad/cc/ccsd_t.py:88-106).  Here the kernel layouts come straight from
// the factors, with the transposes folded into the GEMMs' addressing:
//   vvop[a,y,i,p] = sum_P Lov[P,i,a] R[P,p,y],   R = [Lov ; Lvv] (naux, nmo, nvir)
//   vooo[a,i,k,j] = sum_P Lov[P,i,a] Loo[P,j,k]
// so neither ovvv nor any intermediate of vvop's size is formed.  The VJP
// pulls kernel-layout gradients back onto the factors by the transposed
// contractions (dLov, dLoo, and dR in the transposed order Rt = (naux, nvir, nmo)).
//
// All of these are one GEMM shape C = alpha A B (+ C) whose operands are
// addressed through two-level index maps: an index x of a row or column is
// split as (x / div, x % div) and weighted by two strides, which covers every
// permuted layout above.
#include <cuda_runtime.h>
#include <cooperative_groups.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include "ct_common.cuh"
#include "ct_internal.h"
#include "../../include/pyscfad_b200.h"

namespace ctb {
namespace df {

struct Ix {          // x -> (x / div) * s1 + (x % div) * s0
    int div;
    long long s1, s0;
};
struct Opd {
    const double *p;
    Ix r, c;         // row and column index maps
};

__host__ __device__ inline Ix ix_plain(long long s) { return Ix{INT_MAX, 0, s}; }
__host__ __device__ inline Ix ix_two(int div, long long s1, long long s0) { return Ix{div, s1, s0}; }

constexpr int BN = 64, BK = 16, NTHR = 256, STAGES = 3;
constexpr int LDC = BN + 2;                  // a part's sums, read by the other CTAs of its cluster
constexpr int kFold = 32;                    // K steps after which the sums fold
// the ring, 4 mod 16 doubles per row (conflict-free fragments), and the sums behind it
constexpr int ring_doubles(int bm) { return STAGES * BK * (bm + 4 + BN + 4); }
constexpr size_t smem_bytes(int bm, bool sums) { return sizeof(double) * (size_t)(ring_doubles(bm) + (sums ? bm * LDC : 0)); }

// One operand's slice of a K step: W x BK elements, NL per thread.  MF:
// consecutive threads take consecutive rows (m or n) of one k, so a thread's
// loads share the row and differ in k; else consecutive k, one k per thread and
// several rows.  The k part of an address is kept as (quotient, remainder) and
// advanced by BK without divisions.
template <int W, bool MF> struct Loader {
    static constexpr int NL = W * BK / NTHR, NB = MF ? 1 : NL, NK = MF ? NL : 1;
    long long base[NB];   // address part of the m (or n) index; -1 when out of range
    int kq[NK], kr[NK];   // k = kq * div + kr
    int off, k0;          // first position in the staged tile and its k within the step
    __device__ __forceinline__ void init(const Ix &mix, const Ix &kix, int m0, int M, int kb) {
        const int t = threadIdx.x, m = MF ? t % W : t / BK;
        k0 = MF ? t / W : t % BK;
        off = k0 * (W + 4) + m;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int gm = m0 + m + NTHR / BK * j;
            base[j] = gm < M ? (long long)(gm / mix.div) * mix.s1 + (long long)(gm % mix.div) * mix.s0 : -1;
        }
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            const int k = kb + k0 + NTHR / W * j;
            kq[j] = k / kix.div;
            kr[j] = k % kix.div;
        }
    }
    // copies the step at kb and moves on to the next one
    __device__ __forceinline__ void copy(double *dst, const double *p, const Ix &kix, int kb, int K) {
#pragma unroll
        for (int j = 0; j < NL; ++j) {
            const int jb = MF ? 0 : j, jk = MF ? j : 0;
            const bool ok = base[jb] >= 0 && kb + k0 + (MF ? NTHR / W * j : 0) < K;
            const long long a = base[jb] + (long long)kq[jk] * kix.s1 + (long long)kr[jk] * kix.s0;
            cp_async8(dst + off + (MF ? NTHR / W * (W + 4) : NTHR / BK) * j, ok ? p + a : p, ok);
        }
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            kr[j] += BK;
            while (kr[j] >= kix.div) { kr[j] -= kix.div; ++kq[j]; }
        }
    }
};

// C[m,n] = alpha sum_k A[m,k] B[k,n] (+ C[m,n] when acc); BM x 64 tiles, 8 warps
// of 32 x (BM / 4), K steps of 16 in a three-stage cp.async ring.  BM = 64 for
// few tiles and for sums in parts, 128 for many (launch_cost below).  Few tiles
// are bound by the latency of a K step: one step of a lone CTA takes 1.1 us with
// 64 rows and 1.8 with 128 (K steps of 8 with 128 rows, in four stages, 0.9 for
// half the K).  Many are bound by the DMMA pipe: the vvop product of
// nocc=16/nvir=120/naux=360 takes 0.96 ms with 128 rows (23 of 37 TFLOP/s), 1.03
// with 64 and 0.99 with 128 and steps of 8; a 64 x 64 tile with one shared buffer
// took 1.04.
// The sums of the 64-row build fold and may run in parts.
template <int BM, bool AMF, bool BNF>
__global__ void __launch_bounds__(NTHR, 2) gemm_strided_kernel(int M, int N, int K, Opd A, Opd B, double *C, Ix cr,
                                                               Ix cc, double alpha, int acc) {
    constexpr int LDA = BM + 4, LDB = BN + 4, WN = BM / 4, NT = WN / 8;
    constexpr bool SUMS = BM == 64;
    extern __shared__ __align__(16) double dsm[];
    double *As = dsm, *Bs = dsm + STAGES * BK * LDA, *Cs = dsm + ring_doubles(BM);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int wm = (warp / (BN / WN)) * 32, wn = (warp % (BN / WN)) * WN;
    Loader<BM, AMF> la;
    Loader<BN, BNF> lb;
    // gridDim.z parts of K (whole steps), one CTA of a cluster each
    const int steps = (K + BK - 1) / BK;
    const int sb = (int)((long long)steps * blockIdx.z / gridDim.z);
    const int nk = (int)((long long)steps * (blockIdx.z + 1) / gridDim.z) - sb;
    la.init(A.r, A.c, m0, M, sb * BK);
    lb.init(B.c, B.r, n0, N, sb * BK);
    double d[4][NT][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) d[i][j][0] = d[i][j][1] = 0.0;
    auto issue = [&](int s) {
        if (s < nk) {
            la.copy(As + (s % STAGES) * BK * LDA, A.p, A.c, (sb + s) * BK, K);
            lb.copy(Bs + (s % STAGES) * BK * LDB, B.p, B.r, (sb + s) * BK, K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue(s);
    // the accumulators are folded into this thread's elements of Cs every kFold
    // steps: a chain of K / 4 additions loses up to sqrt(K / 512) more (dLov of
    // nocc=16/nvir=120/naux=360, K 16,320: 7e-16 of the norm against 4.4e-15 in one
    // chain), for 1% of the time
    bool folded = false;
    auto each = [&](auto f) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
                f(*reinterpret_cast<double2 *>(Cs + (wm + 8 * i + g) * LDC + wn + 8 * j + 2 * c), d[i][j]);
    };
    for (int s = 0; s < nk; ++s) {
        if (SUMS && s > 0 && s % kFold == 0) {
            each([&](double2 &x, double (&y)[2]) {
                x = folded ? make_double2(x.x + y[0], x.y + y[1]) : make_double2(y[0], y[1]);
                y[0] = y[1] = 0.0;
            });
            folded = true;
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();   // step s landed for every thread; step s - 1's buffer is free
        issue(s + STAGES - 1);
        const double *a_ = As + (s % STAGES) * BK * LDA + c * LDA + wm + g;
        const double *b_ = Bs + (s % STAGES) * BK * LDB + c * LDB + wn + g;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            double a[4], b[NT];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = a_[kk * LDA + 8 * i];
#pragma unroll
            for (int j = 0; j < NT; ++j) b[j] = b_[kk * LDB + 8 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma(d[i][j], a[i], b[j]);
        }
    }
    if (SUMS && folded)
        each([&](double2 &x, double (&y)[2]) { y[0] += x.x; y[1] += x.y; });
    if (SUMS && gridDim.z > 1) {
        // the parts' sums meet in the order of the parts, so that the result does
        // not depend on which CTA ends first: each CTA leaves its tile in shared
        // memory and adds up its share of the elements
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        const int parts = gridDim.z;
        each([&](double2 &x, double (&y)[2]) { x = make_double2(y[0], y[1]); });
        cl.sync();
        for (int e = blockIdx.z * NTHR + threadIdx.x; e < BM * BN; e += parts * NTHR) {
            const int ml = e / BN, nl = e % BN, m = m0 + ml, n = n0 + nl;
            if (m >= M || n >= N) continue;
            double s = 0.0;
            for (int q = 0; q < parts; ++q) s += cl.map_shared_rank(Cs, q)[ml * LDC + nl];
            double *dst = C + (long long)(m / cr.div) * cr.s1 + (long long)(m % cr.div) * cr.s0 +
                          (long long)(n / cc.div) * cc.s1 + (long long)(n % cc.div) * cc.s0;
            *dst = acc ? *dst + alpha * s : alpha * s;
        }
        cl.sync();   // no CTA leaves while another reads its tile
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + wm + 8 * i + g;
        if (m >= M) continue;
        const long long rm = (long long)(m / cr.div) * cr.s1 + (long long)(m % cr.div) * cr.s0;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n = n0 + wn + 8 * j + 2 * c + h;
                if (n >= N) continue;
                double *dst = C + rm + (long long)(n / cc.div) * cc.s1 + (long long)(n % cc.div) * cc.s0;
                *dst = acc ? *dst + alpha * d[i][j][h] : alpha * d[i][j][h];
            }
    }
}

// Time of CTAs on `slots` single places (two a place share its SM's DMMA pipe) in
// units of one CTA's: a pair takes 2, a last one alone 1.4.
static double launch_cost(double ctas, double slots) {
    const int n = (int)std::ceil(ctas / slots);
    return 2.0 * (n / 2) + (n % 2 ? 1.4 : 0.0);
}

// The numbers of parts of a K sum, and the CTAs that are resident in clusters of so
// many, of all (cudaOccupancyMaxActiveClusters on 148 SMs: a cluster stays within a
// GPC, whose SMs do not divide by every size; 35 tiles of K 10,400 take 221 us
// in eight parts and 163 in seven).
constexpr int kNumParts = 6, kParts[kNumParts] = {1, 2, 3, 4, 6, 8};
constexpr double kResident[kNumParts] = {1.0, 1.0, 279.0 / 296, 284.0 / 296, 270.0 / 296, 264.0 / 296};

template <int BM>
static cudaError_t launch(int M, int N, int K, const Opd &A, const Opd &B, double *C, Ix cr, Ix cc, double alpha,
                          bool acc, int parts, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, parts);
    if (cfg.gridDim.y > 65535) return cudaErrorInvalidValue;
    cfg.blockDim = dim3(NTHR);
    // short sums need no room behind the ring
    cfg.dynamicSmemBytes = smem_bytes(BM, BM == 64 && (parts > 1 || K > kFold * BK));
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = at.val.clusterDim.y = 1;
    at.val.clusterDim.z = parts;
    cfg.attrs = &at;
    cfg.numAttrs = parts > 1 ? 1 : 0;
    auto go = [&](auto kern) {
        const cudaError_t ce = smem_optin(reinterpret_cast<const void *>(kern), (int)cfg.dynamicSmemBytes);
        return ce != cudaSuccess ? ce : cudaLaunchKernelEx(&cfg, kern, M, N, K, A, B, C, cr, cc, alpha, acc ? 1 : 0);
    };
    // consecutive threads along the operand's contiguous index
    if (A.r.s0 == 1)
        return B.c.s0 == 1 ? go(gemm_strided_kernel<BM, true, true>) : go(gemm_strided_kernel<BM, true, false>);
    return B.c.s0 == 1 ? go(gemm_strided_kernel<BM, false, true>) : go(gemm_strided_kernel<BM, false, false>);
}

static cudaError_t gemm(int M, int N, int K, const Opd &A, const Opd &B, double *C, Ix cr, Ix cc, double alpha,
                        bool acc, cudaStream_t st) {
    if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (ce != cudaSuccess) return ce;
    const long long nt = (N + BN - 1) / BN, t64 = nt * ((M + 63) / 64), t128 = nt * ((M + 127) / 128);
    // An accumulating product (the factor gradients: naux rows, long K) takes the
    // number of K parts with the least launch cost x K per part, where a part's
    // start and its share of the sum cost as much as 64 rows of K.  Over 148 products
    // of nocc 2-48 / nvir 20-250 the choice is 2% behind the best number of parts on
    // average (25% at most, below 20 us) and at no size behind one 64 x 64 tile with
    // one shared buffer.  E.g. dLov of nocc=8/nvir=60/naux=204 (32 tiles, K 4080):
    // 62 us in eight parts, 292 in one, 314 with the shared buffer.
    int parts = 1;
    if (acc) {
        double best = 0.0;
        for (int i = 0; i < kNumParts; ++i) {
            const int z = kParts[i], rows = (K + BK * z - 1) / (BK * z) * BK + 64;
            const double cost = launch_cost((double)t64 * z, sms * kResident[i]) * rows;
            if (i == 0 || cost < best) { best = cost; parts = z; }
        }
    }
    // 128-row tiles do a tile pair's work in 1.85 of one tile's time, where they fill the rounds of the GPU
    if (parts == 1 && 1.85 * launch_cost((double)t128, sms) < launch_cost((double)t64, sms))
        return launch<128>(M, N, K, A, B, C, cr, cc, alpha, acc, 1, st);
    return launch<64>(M, N, K, A, B, C, cr, cc, alpha, acc, parts, st);
}

}  // namespace df
}  // namespace ctb

using namespace ctb::df;

extern "C" {

int ct_df_layouts(int nocc, int nvir, int naux, const double *Loo, const double *Lov, const double *R, double *vooo,
                  double *vvop, void *stream) {
    if (!Loo || !Lov || !R || !vooo || !vvop) return CT_ERR_NULL;
    if (nocc < 1 || nvir < 1 || naux < 1 || nocc > 255 || nvir > 1024) return CT_ERR_SHAPE;
    const long long o = nocc, v = nvir, n = o + v;
    cudaStream_t st = (cudaStream_t)stream;
    // rows m = (i, a) = i v + a: Lov[P, i, a] at P o v + m
    const Opd Alov{Lov, ix_plain(1), ix_plain(o * v)};
    // vvop[a, y, i, p]: columns (p, y) = p v + y of R[P, p, y]
    const Opd Br{R, ix_plain(n * v), ix_plain(1)};
    cudaError_t e = gemm((int)(o * v), (int)(n * v), naux, Alov, Br, vvop, ix_two((int)v, n, v * o * n),
                         ix_two((int)v, 1, o * n), 1.0, false, st);
    if (e != cudaSuccess) return CT_ERR_CUDA;
    // vooo[a, i, k, j]: columns (j, k) = j o + k of Loo[P, j, k]
    const Opd Bloo{Loo, ix_plain(o * o), ix_plain(1)};
    e = gemm((int)(o * v), (int)(o * o), naux, Alov, Bloo, vooo, ix_two((int)v, o * o, o * o * o),
             ix_two((int)o, 1, o), 1.0, false, st);
    return e == cudaSuccess ? CT_OK : CT_ERR_CUDA;
}

int ct_df_factor_bar(int nocc, int nvir, int naux, const double *Loo, const double *Lov, const double *Rt,
                     const double *vooo_bar, const double *vvop_bar, double *dLoo, double *dLov, double *dRt,
                     void *stream) {
    if (!Loo || !Lov || !Rt || !vooo_bar || !vvop_bar || !dLoo || !dLov || !dRt) return CT_ERR_NULL;
    if (nocc < 1 || nvir < 1 || naux < 1 || nocc > 255 || nvir > 1024) return CT_ERR_SHAPE;
    const long long o = nocc, v = nvir, n = o + v;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e;
    // dLov[P, (i,a)] += sum_{(y,p)} Rt[P, y, p] vvop_bar[a, y, i, p]
    {
        const Opd A{Rt, ix_plain(v * n), ix_plain(1)};
        const Opd B{vvop_bar, ix_two((int)n, o * n, 1), ix_two((int)v, n, v * o * n)};
        e = gemm(naux, (int)(o * v), (int)(v * n), A, B, dLov, ix_plain(o * v), ix_plain(1), 1.0, true, st);
        if (e != cudaSuccess) return CT_ERR_CUDA;
    }
    // dRt[P, (y,p)] += sum_{(i,a)} Lov[P, i, a] vvop_bar[a, y, i, p]
    {
        const Opd A{Lov, ix_plain(o * v), ix_plain(1)};
        const Opd B{vvop_bar, ix_two((int)v, n, v * o * n), ix_two((int)n, o * n, 1)};
        e = gemm(naux, (int)(v * n), (int)(o * v), A, B, dRt, ix_plain(v * n), ix_plain(1), 1.0, true, st);
        if (e != cudaSuccess) return CT_ERR_CUDA;
    }
    // dLov[P, (i,a)] += sum_{(j,k)} Loo[P, j, k] vooo_bar[a, i, k, j]
    {
        const Opd A{Loo, ix_plain(o * o), ix_plain(1)};
        const Opd B{vooo_bar, ix_two((int)o, 1, o), ix_two((int)v, o * o, o * o * o)};
        e = gemm(naux, (int)(o * v), (int)(o * o), A, B, dLov, ix_plain(o * v), ix_plain(1), 1.0, true, st);
        if (e != cudaSuccess) return CT_ERR_CUDA;
    }
    // dLoo[P, (j,k)] += sum_{(i,a)} Lov[P, i, a] vooo_bar[a, i, k, j]
    {
        const Opd A{Lov, ix_plain(o * v), ix_plain(1)};
        const Opd B{vooo_bar, ix_two((int)v, o * o, o * o * o), ix_two((int)o, 1, o)};
        e = gemm(naux, (int)(o * o), (int)(o * v), A, B, dLoo, ix_plain(o * o), ix_plain(1), 1.0, true, st);
        if (e != cudaSuccess) return CT_ERR_CUDA;
    }
    return CT_OK;
}

}  // extern "C"
