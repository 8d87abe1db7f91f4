// Iterative (T) on the full 6-D triples amplitudes (pyscfad/cc/ccsd_t_slow.py:
// 128-293): the update step of update_amps (:188-208) and the energy of
// energy (:210-220), on (v, v, v, o, o, o) arrays [a][b][c][i][j][k].
//
// The seed (t3_c = P6(W + V) / d3, t3_x = r3(P6(W)) / 3) comes from the
// F1/F2 GEMMs and the orbit epilogue (ct_t3_init in ct_host.cu).  A step is
//   t3_new = (P6(W + V) + P3(fvv' t3) - P3(foo' t3)) / d3
//          = t3_c + (P3(tvv) - P3(too)) / d3,
// P3(x)[abc][ijk] = x[abc][ijk] + x[bac][jik] + x[cba][kji] (:174-176), with
// fvv', foo' the Fock blocks without their diagonals.  The caller forms
// tvv = fvv' t3 on the first virtual index of the [a][b][c][i][j][k] array as a
// plain GEMM.  Two kernels apply P3, divide by d3 and form, in a fixed order,
// |t3_new - t3|^2 and the energy sum t3_new t3_x:
//   step_kernel    forms the foo' products itself from t3's cubes (ct_t3_step);
//                  the faster one up to nocc = 9 and at even nocc <= 20
//   update_kernel  takes too = foo' t3 on the first occupied index of an
//                  occupied-major copy [i][a][b][c][j][k], formed by the caller
//                  as a second GEMM, and writes that copy for the next step
//                  (ct_t3_update)
#include <cuda_runtime.h>
#include <algorithm>
#include "ct_common.cuh"
#include "ct_internal.h"
#include "ct_epi.cuh"
#include "../../include/pyscfad_b200.h"

namespace ctb {
namespace t3it {

constexpr int kThreads = 256, kBlocks = 1024;

__global__ void __launch_bounds__(kThreads) update_kernel(int o, int v, const double *__restrict__ e,
                                                           const double *__restrict__ t3c,
                                                           const double *__restrict__ tvv,
                                                           const double *__restrict__ toom,
                                                           const double *__restrict__ t3,
                                                           const double *__restrict__ t3x,
                                                           double *__restrict__ t3n, double *__restrict__ t3nm,
                                                           double *__restrict__ part) {
    const long long o2 = (long long)o * o, o3 = o2 * o, v2 = (long long)v * v;
    const long long N = v2 * v * o3, mrow = v2 * v * o2;   // occupied-major row: [abc][jk]
    double s0 = 0.0, s1 = 0.0;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < N;
         idx += (long long)kBlocks * kThreads) {
        const long long abc = idx / o3, ijk = idx - abc * o3;
        const int a = (int)(abc / v2), b = (int)((abc / v) % v), c = (int)(abc % v);
        const int i = (int)(ijk / o2), j = (int)((ijk / o) % o), k = (int)(ijk % o);
        const long long bac = ((long long)b * v + a) * v + c, jik = ((long long)j * o + i) * o + k;
        const long long cba = ((long long)c * v + b) * v + a, kji = ((long long)k * o + j) * o + i;
        // too at (abc, ijk), (bac, jik), (cba, kji) in the [i][abc][jk] layout
        const double p3 = (tvv[idx] + tvv[bac * o3 + jik] + tvv[cba * o3 + kji]) -
                          (toom[i * mrow + abc * o2 + j * o + k] + toom[j * mrow + bac * o2 + i * o + k] +
                           toom[k * mrow + cba * o2 + j * o + i]);
        const double d3 = e[i] + e[j] + e[k] - e[o + a] - e[o + b] - e[o + c];
        const double x = t3c[idx] + p3 / d3;
        t3n[idx] = x;
        if (t3nm) t3nm[i * mrow + abc * o2 + j * o + k] = x;
        const double d = x - t3[idx];
        s0 = fma(d, d, s0);
        s1 = fma(x, t3x[idx], s1);
    }
    // fixed-order block sum
    __shared__ double r0[kThreads], r1[kThreads];
    r0[threadIdx.x] = s0;
    r1[threadIdx.x] = s1;
    __syncthreads();
    for (int m = kThreads / 2; m >= 1; m >>= 1) {
        if ((int)threadIdx.x < m) {
            r0[threadIdx.x] += r0[threadIdx.x + m];
            r1[threadIdx.x] += r1[threadIdx.x + m];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = r0[0];
        part[2 * blockIdx.x + 1] = r1[0];
    }
}

__global__ void sum_kernel(const double *__restrict__ part, double *__restrict__ sums, int blocks) {
    __shared__ double r0[kThreads], r1[kThreads];
    double s0 = 0.0, s1 = 0.0;
    for (int b = threadIdx.x; b < blocks; b += kThreads) {
        s0 += part[2 * b];
        s1 += part[2 * b + 1];
    }
    r0[threadIdx.x] = s0;
    r1[threadIdx.x] = s1;
    __syncthreads();
    for (int m = kThreads / 2; m >= 1; m >>= 1) {
        if ((int)threadIdx.x < m) {
            r0[threadIdx.x] += r0[threadIdx.x + m];
            r1[threadIdx.x] += r1[threadIdx.x + m];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        sums[0] = r0[0];
        sums[1] = r1[0];
    }
}

// One step from t3 itself.  foo' t3 needs only the cube t3[abc][...], so its
// three P3 terms are formed here from the cubes of (a,b,c), (b,a,c) and
// (c,b,a) instead of from a product over the whole array:
//   P3(too)[abc][ijk] = sum_m foo'[i,m] t3[abc][mjk] + foo'[j,m] t3[bac][mik] + foo'[k,m] t3[cba][mji]
// which drops the occupied-major copy (written each step and read as four more
// arrays).  A CTA takes a sorted triple a >= b >= c at a time and its up to six
// orderings one after the other, so that the cubes of tvv and t3 that P3 pairs
// are re-read from L2.  The floor is memory: 5 arrays (t3, tvv, t3_c, t3_x in,
// t3_new out) of v^3 o^3 doubles, 202 us at the copy rate at nocc=8/nvir=40.
// With nocc even and <= kStepMaxO (PAIRED) the ordering's three t3 cubes are
// staged in shared memory and a thread owns a 2 x 2 x 2 block of (i, j, k): per m
// nine 16-byte shared loads feed 24 multiply-adds.  Bound by L1/TEX (81% in ncu,
// DRAM 39%): 466 us at nocc=8/nvir=40; one element a thread takes six 8-byte
// loads for 3 multiply-adds, 768 us.  Two CTAs of 256 threads' registers: more
// resident warps or fewer registers measured slower (499 us unbounded, 625 us at
// three).
// Otherwise one element a thread, t3 read through L1: 2 nocc loads of three cubes
// an element, so that from nocc = 11 (for large arrays) a GEMM and update_kernel
// are faster (nocc=24/nvir=16 4.5 ms a cycle against 2.2); the caller chooses.
constexpr int kStepMaxO = 20, kStepThreads = 256, kStepBlocks = CT_T3_STEP_WORK / 2;

struct StepSums {
    double s0 = 0.0, s1 = 0.0;
    __device__ __forceinline__ void add(double xn, double old, double tx) {
        const double d = xn - old;
        s0 = fma(d, d, s0);
        s1 = fma(xn, tx, s1);
    }
};

template <bool PAIRED>
__global__ void __launch_bounds__(kStepThreads, 2) step_kernel(int o, int v, const double *__restrict__ e,
                                                            const double *__restrict__ foo,
                                                            const double *__restrict__ t3c,
                                                            const double *__restrict__ tvv,
                                                            const double *__restrict__ t3,
                                                            const double *__restrict__ t3x,
                                                            double *__restrict__ t3n, double *__restrict__ part) {
    extern __shared__ __align__(16) double ssm[];
    const int o2 = o * o, o3 = o2 * o, tid = threadIdx.x, nthr = blockDim.x;
    double *cs = ssm, *ft = cs + (PAIRED ? 3 * o3 : 0), *eo = ft + o2;   // staged cubes, foo'^T, occupied energies
    const unsigned magic = o > 1 ? (unsigned)(((1ull << 32) + o - 1) / o) : 0u;   // x / o by multiply-high
    auto divo = [&](int x) { return o > 1 ? (int)__umulhi((unsigned)x, magic) : x; };
    for (int q = tid; q < o2; q += nthr) {
        const int m = divo(q), i = q - m * o;
        ft[q] = i == m ? 0.0 : foo[i * o + m];
    }
    for (int i = tid; i < o; i += nthr) eo[i] = e[i];
    __syncthreads();
    const long long ntri = (long long)v * (v + 1) * (v + 2) / 6;
    StepSums S;
    for (long long J = blockIdx.x; J < ntri; J += gridDim.x) {
        int abc[3];
        {
            int a = (int)cbrt(6.0 * (double)J);
            while ((long long)(a + 1) * (a + 2) * (a + 3) / 6 <= J) ++a;
            while ((long long)a * (a + 1) * (a + 2) / 6 > J) --a;
            const int r = (int)(J - (long long)a * (a + 1) * (a + 2) / 6);
            int b = (int)((sqrt(8.0 * r + 1.0) - 1.0) * 0.5);
            while ((b + 1) * (b + 2) / 2 <= r) ++b;
            while (b * (b + 1) / 2 > r) --b;
            abc[0] = a; abc[1] = b; abc[2] = r - b * (b + 1) / 2;
        }
        const double eabc = e[o + abc[0]] + e[o + abc[1]] + e[o + abc[2]];
#pragma unroll
        for (int pi = 0; pi < 6; ++pi) {
            const int x = abc[kR(pi, 0)], y = abc[kR(pi, 1)], z = abc[kR(pi, 2)];
            bool seen = false;   // an ordering equal to an earlier one (repeated indices)
#pragma unroll
            for (int q = 0; q < pi; ++q) seen = seen || (x == abc[kR(q, 0)] && y == abc[kR(q, 1)] && z == abc[kR(q, 2)]);
            if (seen) continue;
            const long long xyz = (((long long)x * v + y) * v + z) * o3, yxz = (((long long)y * v + x) * v + z) * o3,
                            zyx = (((long long)z * v + y) * v + x) * o3;
            if (PAIRED) {
                __syncthreads();   // the previous ordering's cubes are no longer read
                for (int q = 2 * tid; q < o3; q += 2 * nthr) {
                    cp_async16(cs + q, t3 + xyz + q);
                    cp_async16(cs + o3 + q, t3 + yxz + q);
                    cp_async16(cs + 2 * o3 + q, t3 + zyx + q);
                }
                cp_async_wait_all();
                __syncthreads();
                const int h = o / 2;
                for (int q = tid; q < h * h * h; q += nthr) {
                    const int IJ = q / h, K = q - IJ * h, I = IJ / h, Jb = IJ - I * h;
                    const int i = 2 * I, j = 2 * Jb, k = 2 * K;
                    double u[2][2][2];
#pragma unroll
                    for (int t = 0; t < 8; ++t) u[t >> 2][t >> 1 & 1][t & 1] = 0.0;
                    const double *p0 = cs + j * o + k, *p1 = cs + o3 + i * o + k, *p2 = cs + 2 * o3 + j * o + i;
#pragma unroll 2
                    for (int m = 0; m < o; ++m) {
                        const double2 fi = *reinterpret_cast<const double2 *>(ft + m * o + i);
                        const double2 fj = *reinterpret_cast<const double2 *>(ft + m * o + j);
                        const double2 fk = *reinterpret_cast<const double2 *>(ft + m * o + k);
                        double2 a0[2], a1[2], a2[2];
#pragma unroll
                        for (int d = 0; d < 2; ++d) {
                            a0[d] = *reinterpret_cast<const double2 *>(p0 + m * o2 + d * o);   // [j+d][k, k+1]
                            a1[d] = *reinterpret_cast<const double2 *>(p1 + m * o2 + d * o);   // [i+d][k, k+1]
                            a2[d] = *reinterpret_cast<const double2 *>(p2 + m * o2 + d * o);   // [j+d][i, i+1]
                        }
#pragma unroll
                        for (int di = 0; di < 2; ++di)
#pragma unroll
                            for (int dj = 0; dj < 2; ++dj) {
                                const double gi = di ? fi.y : fi.x, gj = dj ? fj.y : fj.x;
                                const double c2 = di ? a2[dj].y : a2[dj].x;
                                u[di][dj][0] = fma(fk.x, c2, fma(gj, a1[di].x, fma(gi, a0[dj].x, u[di][dj][0])));
                                u[di][dj][1] = fma(fk.y, c2, fma(gj, a1[di].y, fma(gi, a0[dj].y, u[di][dj][1])));
                            }
                    }
                    double2 tz[2][2];   // tvv[zyx][k+dk][j+dj][i, i+1]
#pragma unroll
                    for (int dk = 0; dk < 2; ++dk)
#pragma unroll
                        for (int dj = 0; dj < 2; ++dj)
                            tz[dk][dj] = *reinterpret_cast<const double2 *>(tvv + zyx + (k + dk) * o2 + (j + dj) * o + i);
#pragma unroll
                    for (int di = 0; di < 2; ++di)
#pragma unroll
                        for (int dj = 0; dj < 2; ++dj) {
                            const int pos = (i + di) * o2 + (j + dj) * o + k;
                            const double2 tx_ = *reinterpret_cast<const double2 *>(tvv + xyz + pos);
                            const double2 ty_ =
                                *reinterpret_cast<const double2 *>(tvv + yxz + (j + dj) * o2 + (i + di) * o + k);
                            const double2 tc = *reinterpret_cast<const double2 *>(t3c + xyz + pos);
                            const double2 wx = *reinterpret_cast<const double2 *>(t3x + xyz + pos);
                            const double2 old = *reinterpret_cast<const double2 *>(cs + pos);
                            const double eij = eo[i + di] + eo[j + dj] - eabc;
                            double2 xn;
                            xn.x = tc.x + (tx_.x + ty_.x + (di ? tz[0][dj].y : tz[0][dj].x) - u[di][dj][0]) / (eij + eo[k]);
                            xn.y = tc.y + (tx_.y + ty_.y + (di ? tz[1][dj].y : tz[1][dj].x) - u[di][dj][1]) / (eij + eo[k + 1]);
                            *reinterpret_cast<double2 *>(t3n + xyz + pos) = xn;
                            S.add(xn.x, old.x, wx.x);
                            S.add(xn.y, old.y, wx.y);
                        }
                }
            } else {
                const double *c0 = t3 + xyz, *c1 = t3 + yxz, *c2 = t3 + zyx;
                for (int ijk = tid; ijk < o3; ijk += nthr) {
                    const int ij = divo(ijk), k = ijk - ij * o, i = divo(ij), j = ij - i * o;
                    const double tv = tvv[xyz + ijk] + tvv[yxz + j * o2 + i * o + k] + tvv[zyx + k * o2 + j * o + i];
                    double u0 = 0.0, u1 = 0.0, u2 = 0.0;
#pragma unroll 4
                    for (int m = 0; m < o; ++m) {
                        u0 = fma(ft[m * o + i], c0[m * o2 + j * o + k], u0);
                        u1 = fma(ft[m * o + j], c1[m * o2 + i * o + k], u1);
                        u2 = fma(ft[m * o + k], c2[m * o2 + j * o + i], u2);
                    }
                    const double xn = t3c[xyz + ijk] + (tv - (u0 + u1 + u2)) / (eo[i] + eo[j] + eo[k] - eabc);
                    t3n[xyz + ijk] = xn;
                    S.add(xn, c0[ijk], t3x[xyz + ijk]);
                }
            }
        }
    }
    // fixed-order block sum (every CTA's triples and threads are fixed)
    __shared__ double r0[kStepThreads], r1[kStepThreads];
    r0[tid] = S.s0;
    r1[tid] = S.s1;
    __syncthreads();
    for (int m = kStepThreads / 2; m >= 1; m >>= 1) {
        if (tid < m && tid + m < nthr) {
            r0[tid] += r0[tid + m];
            r1[tid] += r1[tid + m];
        }
        __syncthreads();
    }
    if (tid == 0) {
        part[2 * blockIdx.x] = r0[0];
        part[2 * blockIdx.x + 1] = r1[0];
    }
}

}  // namespace t3it
}  // namespace ctb

using namespace ctb;

extern "C" int ct_t3_update(int nocc, int nvir, const double *mo_energy, const double *t3_c, const double *tvv,
                            const double *too_m, const double *t3, const double *t3_x, double *t3_new,
                            double *t3_new_m, double *sums, void *stream) {
    if (nocc < 1 || nocc > 255 || nvir < 1 || nvir > 1024) return CT_ERR_SHAPE;
    if (!mo_energy || !t3_c || !tvv || !too_m || !t3 || !t3_x || !t3_new || !sums) return CT_ERR_NULL;
    // P3 reads other elements of tvv and too_m than the one written
    const double *ins[4] = {t3, tvv, too_m, t3_c};
    for (const double *q : ins)
        if (q == t3_new || (t3_new_m && q == t3_new_m)) return CT_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    double *part = nullptr;
    if (cudaMallocAsync(&part, sizeof(double) * 2 * t3it::kBlocks, st) != cudaSuccess) return CT_ERR_NOMEM;
    t3it::update_kernel<<<t3it::kBlocks, t3it::kThreads, 0, st>>>(nocc, nvir, mo_energy, t3_c, tvv, too_m, t3, t3_x,
                                                                   t3_new, t3_new_m, part);
    t3it::sum_kernel<<<1, t3it::kThreads, 0, st>>>(part, sums, t3it::kBlocks);
    const cudaError_t ce = cudaGetLastError();
    cudaFreeAsync(part, st);
    return ce == cudaSuccess ? CT_OK : CT_ERR_CUDA;
}

extern "C" int ct_t3_step(int nocc, int nvir, const double *mo_energy, const double *foo, const double *t3_c,
                          const double *tvv, const double *t3, const double *t3_x, double *t3_new, double *sums,
                          double *work, void *stream) {
    if (nocc < 1 || nocc > 64 || nvir < 1 || nvir > 1024) return CT_ERR_SHAPE;
    if (!mo_energy || !foo || !t3_c || !tvv || !t3 || !t3_x || !t3_new || !sums || !work) return CT_ERR_NULL;
    // P3 reads other elements of tvv and t3 than the one written
    if (t3 == t3_new || tvv == t3_new || t3_c == t3_new || t3_x == t3_new) return CT_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    const long long ntri = (long long)nvir * (nvir + 1) * (nvir + 2) / 6;
    const int blocks = (int)(ntri < t3it::kStepBlocks ? ntri : t3it::kStepBlocks);
    // 16-byte accesses: even nocc, aligned arrays
    bool paired = nocc % 2 == 0 && nocc <= t3it::kStepMaxO;
    const void *arrays[5] = {t3_c, tvv, t3, t3_x, t3_new};
    for (const void *q : arrays) paired = paired && reinterpret_cast<uintptr_t>(q) % 16 == 0;
    const int o2 = nocc * nocc, o3 = o2 * nocc;
    const size_t smem = sizeof(double) * (size_t)(o2 + nocc + (paired ? 3 * o3 : 0));
    cudaError_t ce = cudaSuccess;
    if (paired) {
        const int thr = std::min(t3it::kStepThreads, (o3 / 8 + 31) / 32 * 32);
        ce = smem_optin(reinterpret_cast<const void *>(t3it::step_kernel<true>), (int)smem);
        if (ce == cudaSuccess)
            t3it::step_kernel<true><<<blocks, thr, smem, st>>>(nocc, nvir, mo_energy, foo, t3_c, tvv, t3, t3_x, t3_new,
                                                              work);
    } else {
        t3it::step_kernel<false><<<blocks, t3it::kStepThreads, smem, st>>>(nocc, nvir, mo_energy, foo, t3_c, tvv, t3,
                                                                          t3_x, t3_new, work);
    }
    if (ce == cudaSuccess) {
        t3it::sum_kernel<<<1, t3it::kThreads, 0, st>>>(work, sums, blocks);
        ce = cudaGetLastError();
    }
    return ce == cudaSuccess ? CT_OK : CT_ERR_CUDA;
}
