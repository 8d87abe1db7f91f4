// Float64 orbit epilogue and V-term bars, the mixed path's V-term bars and the
// energy reduction.  Per wave of sorted jobs (a>=b>=c) the float64 slot path runs:
//   W   G_sigma[p,qr]   = sum_f vvop[x,y,p,o+f] t2T[z,f,qr] - sum_l vooo[x,pq,l] t2T[z,y,l,r]   (ct_pair.cu)
//   EPI orbit epilogue: W, V, r3, D, energy, zbar/d3bar/wbar/vbar, mo_energy_bar
//                                                                   (ccsd_t_vjp.c:9-117, lno_ccsd_t.c:6-29)
//   VT  V-term bars of t1T, fvo, vvop[:,:,:,:o], t2T                (ccsd_t_vjp.c:171-246 gemv parts)
//   VB, TB, OB1, OB2  the bars of the two products                  (ct_pair.cu)
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cstdio>
#include "ct_common.cuh"
#include "ct_internal.h"
#include "ct_epi.cuh"

namespace ctb {

// ---------------------------------------------------------------------------
// Orbit epilogue.  One CTA per job; a thread owns whole element orbits
// {perm(i,j,k)}, so W, V, r3, the denominator and the backward quantities never
// leave registers and nobody else touches an orbit's elements: they are read
// from the six G slots and written back in place, no shared memory and no
// barrier between orbits.  A warp takes half a block-orbit at a time: the
// orbits i >= j >= k of a 2 x 4 x 4 block (I, J, K), whose accesses in every
// permuted order run along 32-byte pieces.  It is bound by the latency of those
// loads: staging the blocks in shared memory (64-thread CTAs, 36 tiles of 4^3)
// spent 4000 instructions per block-orbit on addresses, copies and barriers and
// wrote six W-bar cubes: 50 -> 31 ms over the 6,213 jobs of a nocc=48/nvir=300
// slab block, 307 -> 94 ms for all jobs of nocc=33/nvir=64 with fvo.  w-bar goes
// to slots 0-2 as three copies of one cube, [i][j][k], [i][k][j] and [j][k][i]:
// each W-bar_sigma is one of them with r contiguous (ct_pair.cu).
// ---------------------------------------------------------------------------
enum EpiMode { E_ENERGY, E_VJP, E_LNO_FWD, E_LNO_BWD, E_T3 };
constexpr int kEpiThreads = 256, kEpiWarps = kEpiThreads / 32;

template <int MODE>
__global__ void __launch_bounds__(kEpiThreads, 2) epi_kernel(const WaveView w, const EpiArgs e, double *scratch) {
    constexpr bool BAR = MODE == E_VJP || MODE == E_LNO_BWD;
    __shared__ double U[3][64], F[3][64], eocc[64], occ[kEpiWarps][64], wred[3][kEpiWarps];
    __shared__ const double *va[6], *vb[6];   // vvop[x,y] and t2T[y,x] of the six terms
    const int o = e.o, v = e.v, n = e.n;
    const long long o3 = (long long)o * o * o;
    const int jl = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int a, b, c;
    unpack_job(w.jobs[jl], a, b, c);
    double *S = scratch + (long long)jl * kSlots * o3;
    const double fac = job_fac(a, b, c), eb = e.et_bar;
    const double eabc = e.mo_energy[o + a] + e.mo_energy[o + b] + e.mo_energy[o + c];
    if (tid < 6) {
        int x, y, z;
        term_xyz(tid, a, b, c, x, y, z);
        va[tid] = e.vvop + ((long long)(x * v + y) * o) * n;
        vb[tid] = e.t2T + ((long long)(y * v + x) * o) * o;
    }
    int fnz = 0;
    for (int i = tid; i < 3 * 64; i += kEpiThreads) {
        const int m = i >> 6, r = i & 63, z = m == 0 ? a : (m == 1 ? b : c);
        const double f = r < o ? e.fvo[z * o + r] : 0.0;
        U[m][r] = r < o ? e.t1T[z * o + r] : 0.0;
        F[m][r] = f;
        fnz |= f != 0.0;
    }
    for (int i = tid; i < o; i += kEpiThreads) eocc[i] = e.mo_energy[i];
    for (int i = tid; i < kEpiWarps * 64; i += kEpiThreads) occ[i >> 6][i & 63] = 0.0;
    // with zero fvo rows the fvo part of V adds zeros: skipped
    const bool with_fvo = __syncthreads_or(fnz) != 0;

    KSum eacc;
    double vir = 0.0;
    const int half = warp & 1, nb = (o + 3) / 4, nbo = nb * (nb + 1) * (nb + 2) / 6;
    int BI = 0, BJ = 0, BK = 0;
    auto next = [&](int steps) {   // sorted block triples I >= J >= K, K fastest
        for (int q = 0; q < steps; ++q) {
            if (BK < BJ) ++BK;
            else if (BJ < BI) { ++BJ; BK = 0; }
            else { ++BI; BJ = 0; BK = 0; }
        }
    };
    next(warp >> 1);
    for (int bo = warp >> 1; bo < nbo; bo += kEpiWarps / 2, next(kEpiWarps / 2)) {
        const int ijk[3] = {4 * BI + 2 * half + (lane >> 4), 4 * BJ + ((lane >> 2) & 3), 4 * BK + (lane & 3)};
        const bool mine = ijk[0] < o && ijk[0] >= ijk[1] && ijk[1] >= ijk[2];
        if (!__any_sync(0xffffffffu, mine)) continue;
        double tmp = 0.0;
        if (mine) {
            int pos[6];
            bool first[6];
#pragma unroll
            for (int s = 0; s < 6; ++s) {
                pos[s] = (ijk[kR(s, 0)] * o + ijk[kR(s, 1)]) * o + ijk[kR(s, 2)];
                bool f = true;
#pragma unroll
                for (int t = 0; t < s; ++t) f = f && pos[t] != pos[s];
                first[s] = f;
            }
            const double rden = 1.0 / (eocc[ijk[0]] + eocc[ijk[1]] + eocc[ijk[2]] - eabc);
            double yb[6], wb[6];
            if (MODE == E_LNO_BWD) {
                // (lno_ccsd_t_vjp.c:73-140 on the sorted job's cubes) q = z/D from slot 1,
                // A and B in two parts from slots 2, 4 and 3, 5: the energy is sum A q,
                // z_bar = eb A / D, w_bar = eb B + r3(z_bar), v_bar = r3(z_bar)
                double zb[6], aq = 0.0;
#pragma unroll
                for (int s = 0; s < 6; ++s) {
                    const double q = S[o3 + pos[s]], Ax = S[2 * o3 + pos[s]] + S[4 * o3 + pos[s]];
                    const double Bx = S[3 * o3 + pos[s]] + S[5 * o3 + pos[s]];
                    zb[s] = eb * Ax * rden;
                    wb[s] = eb * Bx;
                    if (first[s]) aq += Ax * q;
                }
                tmp = eb * rden * aq;
                r3_orbit<double>(zb, yb);
#pragma unroll
                for (int s = 0; s < 6; ++s) wb[s] += yb[s];
            } else {
                double w6[6], y6[6], z6[6];
#pragma unroll
                for (int s = 0; s < 6; ++s) w6[s] = y6[s] = 0.0;
#pragma unroll
                for (int sg = 0; sg < 6; ++sg) {
                    const double *G = S + sg * o3;
                    double x[6];
#pragma unroll
                    for (int q = 0; q < 6; ++q) x[q] = G[pos[q]];
#pragma unroll
                    for (int s = 0; s < 6; ++s) w6[s] += x[kComp(s, sg)];
                }
                auto add_v = [&](const double (&L)[3][64], const double *const (&base)[6], int ld) {
                    double u[3][3];
                    int at[6];
#pragma unroll
                    for (int m = 0; m < 3; ++m)
#pragma unroll
                        for (int q = 0; q < 3; ++q) u[m][q] = L[m][ijk[q]];
#pragma unroll
                    for (int q = 0; q < 6; ++q) at[q] = ijk[kR(q, 0)] * ld + ijk[kR(q, 1)];
#pragma unroll
                    for (int sg = 0; sg < 6; ++sg) {
                        const double *A = base[sg];
                        double x[6];
#pragma unroll
                        for (int q = 0; q < 6; ++q) x[q] = __ldg(A + at[q]);
#pragma unroll
                        for (int s = 0; s < 6; ++s) {
                            const int cs = kComp(s, sg);
                            y6[s] += x[cs] * u[kR(sg, 2)][kR(cs, 2)];
                        }
                    }
                };
                add_v(U, va, n);
                if (with_fvo) add_v(F, vb, o);
#pragma unroll
                for (int s = 0; s < 6; ++s) y6[s] = w6[s] + 0.5 * y6[s];
                if (MODE == E_T3) {
                    // the iterative solver's seed (pyscfad/cc/ccsd_t_slow.py:188-220 on the 6-D
                    // amplitudes): W and W + V are P6(w)[., a, b, c] and P6(w + v)[., a, b, c];
                    // P6 makes the 6-D arrays invariant under a simultaneous permutation of
                    // (i, j, k) and (a, b, c), and D under any permutation of either, so
                    // t3_c[pi(a,b,c)][pi(pos)] = (W + V) / D and t3_x[...] = r3(W) / 3 (the energy
                    // is sum t3 t3_x, :210-220) for each permutation pi
                    r3_orbit<double>(w6, z6);
                    const int abc[3] = {a, b, c};
                    // one cube's six elements at a time, as streaming stores: element by
                    // element over the cubes the seed took 28.7 ms at nocc=32/nvir=32 and
                    // 51.1 at nocc=48/nvir=24, so 26.7 and 48.7
#pragma unroll
                    for (int s = 0; s < 6; ++s) {
                        y6[s] *= rden;
                        z6[s] *= 1.0 / 3.0;
                    }
#pragma unroll
                    for (int pi = 0; pi < 6; ++pi) {
                        const long long ia = ((long long)abc[kR(pi, 0)] * v + abc[kR(pi, 1)]) * v + abc[kR(pi, 2)];
                        double *tc = e.t3_c + ia * o3, *tx = e.t3_x + ia * o3;
#pragma unroll
                        for (int s = 0; s < 6; ++s) __stcs(tc + pos[kComp(s, pi)], y6[s]);
#pragma unroll
                        for (int s = 0; s < 6; ++s) __stcs(tx + pos[kComp(s, pi)], z6[s]);
                    }
                    continue;
                }
                r3_orbit<double>(y6, z6);
                // one reciprocal per orbit: d3 = fac / D; its distinct W.Z products share d3,
                // so they are summed before the compensated add, and the mo_energy-bar
                // partial eb d3^2 / fac = eb fac / D^2 reuses 1/D
                const double d3 = fac * rden;
                double wz = 0.0;
#pragma unroll
                for (int s = 0; s < 6; ++s)
                    if (first[s]) wz += w6[s] * z6[s];
                eacc.add(wz * d3);
                if (MODE == E_LNO_FWD) {
#pragma unroll
                    for (int s = 0; s < 6; ++s) {
                        S[pos[s]] = w6[s];
                        S[o3 + pos[s]] = z6[s] * rden;
                    }
                }
                if (MODE == E_VJP) {
                    const double ebd3 = eb * d3;
                    tmp = eb * d3 * rden * wz;
                    double zb[6];
#pragma unroll
                    for (int s = 0; s < 6; ++s) zb[s] = ebd3 * w6[s];
                    r3_orbit<double>(zb, yb);
#pragma unroll
                    for (int s = 0; s < 6; ++s) wb[s] = ebd3 * z6[s] + yb[s];
                }
            }
            if (BAR) {
                vir += tmp;
#pragma unroll
                for (int s = 0; s < 6; ++s)
                    if (first[s]) {
                        S[pos[s]] = wb[s];
                        S[o3 + pos[s]] = wb[kComp(s, 1)];
                        S[2 * o3 + pos[s]] = wb[kComp(s, 4)];
                        S[6 * o3 + pos[s]] = yb[s];
                    }
            }
        }
        if (BAR) {
            // occupied mo_energy bar: sums over two of the block's axes (lane bits 0-1 are
            // k's, 2-3 j's, 4 i's), one axis after the other (blocks may coincide)
            double s2 = tmp, s1 = tmp, s0;
            s2 += __shfl_xor_sync(0xffffffffu, s2, 4);
            s2 += __shfl_xor_sync(0xffffffffu, s2, 8);
            s2 += __shfl_xor_sync(0xffffffffu, s2, 16);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
            s0 = s1;
            s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
            s0 += __shfl_xor_sync(0xffffffffu, s0, 4);
            s0 += __shfl_xor_sync(0xffffffffu, s0, 8);
            if (lane < 4) occ[warp][4 * BK + lane] += s2;
            __syncwarp();
            if (lane < 16 && (lane & 3) == 0) occ[warp][4 * BJ + (lane >> 2)] += s1;
            __syncwarp();
            if ((lane & 15) == 0) occ[warp][4 * BI + 2 * half + (lane >> 4)] += s0;
            __syncwarp();
        }
    }
    if (MODE == E_T3) return;
    // job energy and the virtual mo_energy bar: a fixed shuffle tree per warp, then over the warps
    ksum_tree(eacc, vir);
    if (lane == 0) { wred[0][warp] = eacc.s; wred[1][warp] = eacc.c; wred[2][warp] = vir; }
    __syncthreads();
    if (warp == 0) {
        KSum k;
        k.s = lane < kEpiWarps ? wred[0][lane] : 0.0;
        k.c = lane < kEpiWarps ? wred[1][lane] : 0.0;
        double vt = lane < kEpiWarps ? wred[2][lane] : 0.0;
        ksum_tree(k, vt);
        if (lane == 0) {
            const long long amaj = (long long)a * (a + 1) * (a + 2) / 6 + (long long)b * (b + 1) / 2 + c;
            if (MODE != E_LNO_BWD) e.job_e[amaj] = 2.0 * k.value();   // there the projection kernel's energy stands
            if (BAR) {
                atomicAdd(&e.mo_energy_bar[o + a], vt);
                atomicAdd(&e.mo_energy_bar[o + b], vt);
                atomicAdd(&e.mo_energy_bar[o + c], vt);
            }
        }
    }
    if (BAR && tid < o) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < kEpiWarps; ++q) s += occ[q][tid];
        atomicAdd(&e.mo_energy_bar[tid], -s);
    }
}

// V-term bars of one job.  With Vbar_sigma[p,q,r] = ybar[idx_sigma(p,q,r)]:
//   vvop_bar[x,y,p,q] += 1/2 sum_r Vbar t1T[z,r]     (get_vvoo_bar, ccsd_t_vjp.c:171-186)
//   t2T_bar[y,x,p,q]  += 1/2 sum_r Vbar fvo[z,r]     (get_t2T_bar gemv, :228-230)
//   t1T_bar[z,r]      += 1/2 sum_pq Vbar vvop[x,y,p,q]   (get_t1T_bar, :188-204)
//   fvo_bar[z,r]      += 1/2 sum_pq Vbar t2T[y,x,p,q]    (get_fvo_bar, :233-246)
// For each term the index r sits on one axis of ybar (two terms per axis), so
// the CTA makes one coalesced pass per axis: ybar contracted along that axis
// with the two terms' t1/fvo vectors, and along the other two with their
// vvop/t2T matrices.
__device__ __forceinline__ double ldg_st(const double *p) { return __ldg(p); }
__device__ __forceinline__ float ldg_st(const float *p) { return __ldg(p); }

struct VtTerm {
    int x, y, z, mp, mq;
};

__device__ __forceinline__ VtTerm vt_term(int sg, int a, int b, int c) {
    VtTerm t;
    term_xyz(sg, a, b, c, t.x, t.y, t.z);
    const int ri = kInv(sg);
    t.mp = kR(ri, 0) == 0 ? 0 : (kR(ri, 1) == 0 ? 1 : 2);
    t.mq = kR(ri, 0) == 1 ? 0 : (kR(ri, 1) == 1 ? 1 : 2);
    return t;
}

// One axis pass per CTA (blockIdx.x = 3 * job + axis).  The o^2 pairs of the
// two other axes are processed in chunks of VT_CH: the chunk's ybar values
// (all r) are staged in shared memory as Ys[r][pair]; then each thread
// contracts one pair along r with the two terms' t1/fvo rows (vvop-bar and
// t2T-bar updates), and 4 * o threads contract one r along the chunk's pairs
// with the terms' vvop/t2T values (t1T-bar / fvo-bar partials, kept in
// registers across chunks).  No warp shuffles.
constexpr int VT_CH = 256;

// QRT: ybar (slot 6) is qr-tiled (the mixed path's slot layout): element
// (i,j,k) at i o^2 + (j/8) 8o + (k/8) 64 + (j%8) 8 + k%8
template <typename ST, bool QRT>
__global__ void __launch_bounds__(VT_CH) vterm_kernel(const WaveView w, const EpiArgs e, const ST *scratch) {
    constexpr int NTHR = VT_CH, LD = VT_CH + 1;
    extern __shared__ __align__(16) uint8_t vsm[];
    ST *Ys = reinterpret_cast<ST *>(vsm);                                 // [o][LD]
    double *AB = reinterpret_cast<double *>(vsm + sizeof(ST) * 64 * LD);  // [4][VT_CH]: A_t0, A_t1, B_t0, B_t1
    double *UW = AB + 4 * VT_CH;                                         // [4][64]: u_t0, u_t1, w_t0, w_t1
    const int o = e.o, v = e.v, n = e.n, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int jl = blockIdx.x / 3, ax = blockIdx.x - 3 * (blockIdx.x / 3), tid = threadIdx.x;
    int a, b, c;
    unpack_job(w.jobs[jl], a, b, c);
    const ST *Yb = scratch + ((long long)jl * kSlots + 6) * o3;
    // terms per axis of r: axis 0 -> sigma 3,5; axis 1 -> sigma 1,4; axis 2 -> sigma 0,2
    const int s0 = ax == 0 ? 3 : (ax == 1 ? 1 : 0), s1 = ax == 0 ? 5 : (ax == 1 ? 4 : 2);
    const VtTerm T0 = vt_term(s0, a, b, c), T1 = vt_term(s1, a, b, c);
    // coordinate m of pair (f0, f1) with r's axis set to 0, without indexed arrays
    auto coord = [&](int m, int f0, int f1) {
        const int c0 = ax == 0 ? 0 : f0, c1 = ax == 0 ? f0 : (ax == 1 ? 0 : f1), c2 = ax == 2 ? 0 : f1;
        return m == 0 ? c0 : (m == 1 ? c1 : c2);
    };
    const long long rstep = ax == 0 ? (long long)oo : (ax == 1 ? (long long)o : 1LL);
    // x / o by multiply-high with ceil(2^32 / o): exact for x < 2^32 / o^2 (x < o^2 * 4 here)
    const unsigned omag = (unsigned)(((1ull << 32) + o - 1) / o);
    auto divo = [&](int x) { return (int)__umulhi((unsigned)x, omag); };
    int fvo_nz = 0;
    for (int i = tid; i < 2 * o; i += NTHR) {
        const int t = i / o, r = i - t * o;
        const int z = t ? T1.z : T0.z;
        UW[t * 64 + r] = e.t1T[z * o + r];
        const double f = e.fvo[z * o + r];
        UW[(2 + t) * 64 + r] = f;
        fvo_nz |= (f != 0.0);
    }
    // with both terms' fvo rows zero the t2T-bar updates of this pass add zeros: skipped
    const bool with_fvo = __syncthreads_or(fvo_nz) != 0;
    // (r, q4) of this thread's r-contraction: q4 = 0,1 -> A of term 0,1; 2,3 -> B
    const int rr = tid % 64, q4 = tid / 64;
    const bool rowner = rr < o && q4 < 4;
    double racc = 0.0;
    for (int base = 0; base < oo; base += VT_CH) {
        const int cnt = min(VT_CH, oo - base);
        __syncthreads();  // previous chunk consumed
        // stage ybar: Ys[r][j] = ybar(pair base + j, r); consecutive threads take
        // consecutive memory (pairs for axes 0/1, r for axis 2)
        auto tile = [&](int j, int k) { return (j >> 3) * 8 * o + (k >> 3) * 64 + (j & 7) * 8 + (k & 7); };
        if (ax < 2) {
            if (tid < cnt) {
                const int pr = base + tid, f0 = divo(pr), f1 = pr - f0 * o;
                if (QRT) {
                    if (ax == 0) {
                        const ST *src = Yb + tile(f0, f1);
#pragma unroll 8
                        for (int r = 0; r < o; ++r) Ys[r * LD + tid] = src[(long long)r * oo];
                    } else {
                        const ST *src = Yb + (long long)f0 * oo;
#pragma unroll 8
                        for (int r = 0; r < o; ++r) Ys[r * LD + tid] = src[tile(r, f1)];
                    }
                } else {
                    const ST *src = Yb + (ax == 0 ? (long long)pr : (long long)f0 * oo + f1);
#pragma unroll 8
                    for (int r = 0; r < o; ++r) Ys[r * LD + tid] = src[r * rstep];
                }
            }
        } else {
            for (int i = tid; i < cnt * o; i += NTHR) {
                const int j = divo(i), r = i - j * o;
                if (QRT) {
                    const int pr = base + j, f0 = divo(pr), f1 = pr - f0 * o;
                    Ys[r * LD + j] = Yb[(long long)f0 * oo + tile(f1, r)];
                } else {
                    Ys[r * LD + j] = Yb[(long long)(base + j) * o + r];
                }
            }
        }
        // the chunk's vvop / t2T values of both terms at (P, Q) of each pair
        for (int i = tid; i < cnt * 2; i += NTHR) {
            const int t = i >= cnt ? 1 : 0, j = i - t * cnt;
            const int pr = base + j, f0 = divo(pr), f1 = pr - f0 * o;
            const int tx = t ? T1.x : T0.x, ty = t ? T1.y : T0.y;
            const int P = coord(t ? T1.mp : T0.mp, f0, f1), Q = coord(t ? T1.mq : T0.mq, f0, f1);
            AB[t * VT_CH + j] = e.vvop[((long long)(tx * v + ty) * o + P) * n + Q];
            AB[(2 + t) * VT_CH + j] = e.t2T[((long long)(ty * v + tx) * o + P) * o + Q];
        }
        __syncthreads();
        // pair contraction along r -> vvop-bar / t2T-bar
        if (tid < cnt) {
            double su0 = 0, su1 = 0, sw0 = 0, sw1 = 0;
            for (int r = 0; r < o; ++r) {
                const double val = (double)Ys[r * LD + tid];
                su0 += val * UW[r]; su1 += val * UW[64 + r];
                sw0 += val * UW[128 + r]; sw1 += val * UW[192 + r];
            }
            const int pr = base + tid, f0 = divo(pr), f1 = pr - f0 * o;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int tx = t ? T1.x : T0.x, ty = t ? T1.y : T0.y;
                const int P = coord(t ? T1.mp : T0.mp, f0, f1), Q = coord(t ? T1.mq : T0.mq, f0, f1);
                atomicAdd(e.vvop_bar + ((long long)(tx * v + ty) * o + P) * n + Q, 0.5 * (t ? su1 : su0));
                if (with_fvo) atomicAdd(e.t2T_bar + ((long long)(ty * v + tx) * o + P) * o + Q, 0.5 * (t ? sw1 : sw0));
            }
        }
        // r contraction along the chunk's pairs -> t1T-bar / fvo-bar partials
        // (four independent partial sums hide the add latency)
        if (rowner) {
            const ST *row = Ys + rr * LD;
            const double *vec = AB + q4 * VT_CH;
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
            int j = 0;
            for (; j + 4 <= cnt; j += 4) {
                a0 += (double)row[j] * vec[j];
                a1 += (double)row[j + 1] * vec[j + 1];
                a2 += (double)row[j + 2] * vec[j + 2];
                a3 += (double)row[j + 3] * vec[j + 3];
            }
            for (; j < cnt; ++j) a0 += (double)row[j] * vec[j];
            racc += (a0 + a1) + (a2 + a3);
        }
    }
    if (rowner) {
        const int z = (q4 & 1) ? T1.z : T0.z;
        double *dst = (q4 < 2 ? e.t1T_bar : e.fvo_bar) + z * o + rr;
        atomicAdd(dst, 0.5 * racc);
    }
}

template <typename ST>
static size_t vterm_smem() {
    return sizeof(ST) * 64 * (VT_CH + 1) + sizeof(double) * (4 * VT_CH + 4 * 64);
}

template <typename ST, bool QRT>
static cudaError_t launch_vterm(const WaveView &w, const EpiArgs &e, const ST *scratch, cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    if (e.o > 64) return cudaErrorInvalidValue;
    {
        cudaError_t ce = smem_optin(reinterpret_cast<const void *>(vterm_kernel<ST, QRT>), (int)vterm_smem<ST>());
        if (ce != cudaSuccess) return ce;
    }
    vterm_kernel<ST, QRT><<<w.n_jobs * 3, VT_CH, vterm_smem<ST>(), st>>>(w, e, scratch);
    return cudaGetLastError();
}

cudaError_t f64_epilogue(const WaveView &w, const EpiArgs &e, double *scratch, cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    if (e.o > 64) return cudaErrorInvalidValue;
    const dim3 grid(w.n_jobs), block(kEpiThreads);
    if (e.t3_c) {
        if (!e.t3_x || e.with_vjp) return cudaErrorInvalidValue;
        epi_kernel<E_T3><<<grid, block, 0, st>>>(w, e, scratch);
    } else if (e.with_vjp) {
        if (e.lno_phase == 2) epi_kernel<E_LNO_BWD><<<grid, block, 0, st>>>(w, e, scratch);
        else epi_kernel<E_VJP><<<grid, block, 0, st>>>(w, e, scratch);
    } else if (e.lno_phase == 1) {
        epi_kernel<E_LNO_FWD><<<grid, block, 0, st>>>(w, e, scratch);
    } else {
        epi_kernel<E_ENERGY><<<grid, block, 0, st>>>(w, e, scratch);
    }
    return cudaGetLastError();
}

cudaError_t f64_vterm(const WaveView &w, const EpiArgs &e, const double *scratch, cudaStream_t st) {
    return launch_vterm<double, false>(w, e, scratch, st);
}

// V-term bars of the mixed path (float ybar, qr-tiled slots): the same four
// contractions as vterm_kernel, one CTA per (job, axis), restructured for
// shared-memory throughput.  A chunk of 256 pairs (pair index f0*o + f1 of
// the two axes other than r's) is staged r-major as Ys[r][j] (row stride
// 260 floats: 16-byte rows, and 65 16-byte units per row so that 8 threads
// reading 8 consecutive rows hit 8 distinct bank groups): with 16-byte
// cp.async pieces of 4 pairs for axes 0 and 1 (4 consecutive f1 lie in one
// 8-run of the tiled slot), and through registers for axis 2, whose runs
// are along r.  Then
//   U: one thread per pair: sum_r Ys[r][j] * (t1_z0, t1_z1, fvo_z0, fvo_z1)[r]
//      (one float4 broadcast per r) -> vvop_bar / t2T_bar;
//   B: thread (r, quarter): sum over its 64 pairs of Ys[r][j..j+3] (float4)
//      times the pair's (vvop_t0, vvop_t1, t2T_t0, t2T_t1) (float4 broadcast),
//      float partials per chunk added into float64 -> t1T_bar / fvo_bar.
// Products and per-chunk sums are float (the ybar operand is float on this
// path), chunk sums and the output reductions float64.
constexpr int V2_NT = 256, V2_CH = 256, V2_LD = V2_CH + 4;

static size_t vterm2_smem(int o) {
    return sizeof(float) * (size_t)o * V2_LD + sizeof(float4) * (V2_CH + 64) + sizeof(double) * 4 * 4 * 64;
}

template <int AX>
__device__ __forceinline__ void vterm2_axis(const WaveView &w, const EpiArgs &e, const float *Yb, int a, int b,
                                            int c, uint8_t *sm) {
    const int o = e.o, v = e.v, n = e.n, oo = o * o, tid = threadIdx.x;
    float *Ys = reinterpret_cast<float *>(sm);                  // [o][V2_LD]
    float4 *AB = reinterpret_cast<float4 *>(Ys + o * V2_LD);     // [V2_CH]
    float4 *UW = AB + V2_CH;                                     // [64]
    double *Bq = reinterpret_cast<double *>(UW + 64);            // [4 quarters][4 combos][64]
    // terms per axis of r: axis 0 -> sigma 3,5; axis 1 -> sigma 1,4; axis 2 -> sigma 0,2
    constexpr int S0 = AX == 0 ? 3 : (AX == 1 ? 1 : 0), S1 = AX == 0 ? 5 : (AX == 1 ? 4 : 2);
    const VtTerm T0 = vt_term(S0, a, b, c), T1 = vt_term(S1, a, b, c);
    auto coord = [](int m, int f0, int f1) {
        const int c0 = AX == 0 ? 0 : f0, c1 = AX == 0 ? f0 : (AX == 1 ? 0 : f1), c2 = AX == 2 ? 0 : f1;
        return m == 0 ? c0 : (m == 1 ? c1 : c2);
    };
    auto tile = [o](int j, int k) { return (j >> 3) * 8 * o + (k >> 3) * 64 + (j & 7) * 8 + (k & 7); };
    const unsigned omag = (unsigned)(((1ull << 32) + o - 1) / o);
    auto divo = [omag](int x) { return (int)__umulhi((unsigned)x, omag); };
    int fvo_nz = 0;
    if (tid < o) {
        const int r = tid;
        const float f0 = (float)e.fvo[T0.z * o + r], f1 = (float)e.fvo[T1.z * o + r];
        UW[r] = make_float4((float)e.t1T[T0.z * o + r], (float)e.t1T[T1.z * o + r], f0, f1);
        fvo_nz = (e.fvo[T0.z * o + r] != 0.0) || (e.fvo[T1.z * o + r] != 0.0);
    }
    // with both terms' fvo rows zero the t2T-bar updates of this pass add zeros: skipped
    const bool with_fvo = __syncthreads_or(fvo_nz) != 0;
    const int br = tid & 63, qd = tid >> 6;   // B role: row r, quarter of the chunk's pairs
    double bacc0 = 0.0, bacc1 = 0.0, bacc2 = 0.0, bacc3 = 0.0;
    for (int base = 0; base < oo; base += V2_CH) {
        const int cnt = min(V2_CH, oo - base);   // a multiple of 4 (o % 8 == 0)
        __syncthreads();                         // previous chunk consumed
        if (AX != 2) {
            const int npc = cnt >> 2;
            for (int i = tid; i < o * npc; i += V2_NT) {
                const int r = i / npc, q4 = i - r * npc;
                const int pr = base + 4 * q4, f0 = divo(pr), f1 = pr - f0 * o;
                const float *src = AX == 0 ? Yb + (long long)r * oo + tile(f0, f1) : Yb + (long long)f0 * oo + tile(r, f1);
                cp_async16(Ys + r * V2_LD + 4 * q4, src);
            }
            cp_async_commit();
        } else if (tid < cnt) {
            const int pr = base + tid, f0 = divo(pr), f1 = pr - f0 * o;
            const float *src = Yb + (long long)f0 * oo + tile(f1, 0);
#pragma unroll 4
            for (int r0 = 0; r0 < o; r0 += 8) {
                const float4 y0 = __ldg(reinterpret_cast<const float4 *>(src + r0 * 8));
                const float4 y1 = __ldg(reinterpret_cast<const float4 *>(src + r0 * 8 + 4));
                float *d = Ys + r0 * V2_LD + tid;
                d[0] = y0.x; d[V2_LD] = y0.y; d[2 * V2_LD] = y0.z; d[3 * V2_LD] = y0.w;
                d[4 * V2_LD] = y1.x; d[5 * V2_LD] = y1.y; d[6 * V2_LD] = y1.z; d[7 * V2_LD] = y1.w;
            }
        }
        // the chunk's vvop / t2T values of both terms at (P, Q) of each pair
        if (tid < cnt) {
            const int pr = base + tid, f0 = divo(pr), f1 = pr - f0 * o;
            const int P0 = coord(T0.mp, f0, f1), Q0 = coord(T0.mq, f0, f1);
            const int P1 = coord(T1.mp, f0, f1), Q1 = coord(T1.mq, f0, f1);
            AB[tid] = make_float4((float)e.vvop[((long long)(T0.x * v + T0.y) * o + P0) * n + Q0],
                                  (float)e.vvop[((long long)(T1.x * v + T1.y) * o + P1) * n + Q1],
                                  (float)e.t2T[((long long)(T0.y * v + T0.x) * o + P0) * o + Q0],
                                  (float)e.t2T[((long long)(T1.y * v + T1.x) * o + P1) * o + Q1]);
        }
        if (AX != 2) cp_async_wait_all();
        __syncthreads();
        // U: pair contraction along r -> vvop-bar / t2T-bar
        if (tid < cnt) {
            float su0 = 0.f, su1 = 0.f, sw0 = 0.f, sw1 = 0.f;
#pragma unroll 8
            for (int r = 0; r < o; ++r) {
                const float y = Ys[r * V2_LD + tid];
                const float4 u = UW[r];
                su0 = fmaf(y, u.x, su0); su1 = fmaf(y, u.y, su1);
                sw0 = fmaf(y, u.z, sw0); sw1 = fmaf(y, u.w, sw1);
            }
            const int pr = base + tid, f0 = divo(pr), f1 = pr - f0 * o;
            const int P0 = coord(T0.mp, f0, f1), Q0 = coord(T0.mq, f0, f1);
            const int P1 = coord(T1.mp, f0, f1), Q1 = coord(T1.mq, f0, f1);
            atomicAdd(e.vvop_bar + ((long long)(T0.x * v + T0.y) * o + P0) * n + Q0, 0.5 * (double)su0);
            atomicAdd(e.vvop_bar + ((long long)(T1.x * v + T1.y) * o + P1) * n + Q1, 0.5 * (double)su1);
            if (with_fvo) {
                atomicAdd(e.t2T_bar + ((long long)(T0.y * v + T0.x) * o + P0) * o + Q0, 0.5 * (double)sw0);
                atomicAdd(e.t2T_bar + ((long long)(T1.y * v + T1.x) * o + P1) * o + Q1, 0.5 * (double)sw1);
            }
        }
        // B: r contraction along the quarter's pairs -> t1T-bar / fvo-bar partials
        if (br < o) {
            float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
            const int j1 = min(qd * (V2_CH / 4) + V2_CH / 4, cnt);
            const float *row = Ys + br * V2_LD;
            for (int j = qd * (V2_CH / 4); j < j1; j += 4) {
                const float4 y4 = *reinterpret_cast<const float4 *>(row + j);
                const float yy[4] = {y4.x, y4.y, y4.z, y4.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 m = AB[j + u];
                    p0 = fmaf(yy[u], m.x, p0); p1 = fmaf(yy[u], m.y, p1);
                    p2 = fmaf(yy[u], m.z, p2); p3 = fmaf(yy[u], m.w, p3);
                }
            }
            bacc0 += p0; bacc1 += p1; bacc2 += p2; bacc3 += p3;
        }
    }
    if (br < o) {
        Bq[(qd * 4 + 0) * 64 + br] = bacc0;
        Bq[(qd * 4 + 1) * 64 + br] = bacc1;
        Bq[(qd * 4 + 2) * 64 + br] = bacc2;
        Bq[(qd * 4 + 3) * 64 + br] = bacc3;
    }
    __syncthreads();
    {
        // combo k = tid / 64: 0, 1 -> t1T-bar of term 0, 1; 2, 3 -> fvo-bar of term 0, 1
        const int k = tid >> 6, r = tid & 63;
        if (r < o) {
            const double s = Bq[k * 64 + r] + Bq[(4 + k) * 64 + r] + Bq[(8 + k) * 64 + r] + Bq[(12 + k) * 64 + r];
            const int z = (k & 1) ? T1.z : T0.z;
            atomicAdd((k < 2 ? e.t1T_bar : e.fvo_bar) + z * o + r, 0.5 * s);
        }
    }
}

__global__ void __launch_bounds__(V2_NT) vterm2_kernel(const WaveView w, const EpiArgs e, const float *scratch) {
    extern __shared__ __align__(16) uint8_t vsm2[];
    const int o = e.o;
    const long long o3 = (long long)o * o * o;
    const int jl = blockIdx.x / 3, ax = blockIdx.x - 3 * (blockIdx.x / 3);
    int a, b, c;
    unpack_job(w.jobs[jl], a, b, c);
    const float *Yb = scratch + ((long long)jl * kSlots + 6) * o3;
    if (ax == 0) vterm2_axis<0>(w, e, Yb, a, b, c, vsm2);
    else if (ax == 1) vterm2_axis<1>(w, e, Yb, a, b, c, vsm2);
    else vterm2_axis<2>(w, e, Yb, a, b, c, vsm2);
}

cudaError_t f32_vterm(const WaveView &w, const EpiArgs &e, const float *scratch, cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    if (e.o > 64 || e.o % 8 != 0) return cudaErrorInvalidValue;
    const size_t smem = vterm2_smem(e.o);
    {
        cudaError_t ce = smem_optin(reinterpret_cast<const void *>(vterm2_kernel), (int)vterm2_smem(64));
        if (ce != cudaSuccess) return ce;
    }
    vterm2_kernel<<<w.n_jobs * 3, V2_NT, smem, st>>>(w, e, scratch);
    return cudaGetLastError();
}

// Deterministic compensated sum of the per-job energies, fixed order: each
// CTA sums a fixed contiguous chunk (Neumaier pairs, merged down fixed shuffle
// trees), then one CTA merges the partials the same way.  A single thread
// merging the 2048 values of its CTA, and one more the 256 partials, took 57 us
// whatever n was; the trees take 6 us at n = 220 and 9 us at n = 295,240.  Past a
// million values the adds of a thread are the time: 1024 threads a CTA there
// (n = 1.67e8, nvir = 1000: 251 us against 574 with 256, and 295 of the serial merge).
constexpr int kRedThreads = 256, kRedThreadsLong = 1024;

// the pair (s, c) of a CTA's threads merged in a fixed order; valid in thread 0
__device__ __forceinline__ KSum block_ksum(KSum k) {
    __shared__ double ws[32], wc[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    auto tree = [](KSum &x, int top) {
        for (int m = top; m >= 1; m >>= 1) {
            const double s2 = __shfl_down_sync(0xffffffffu, x.s, m), c2 = __shfl_down_sync(0xffffffffu, x.c, m);
            x.c += c2;
            x.add(s2);
        }
    };
    tree(k, 16);
    if (lane == 0) { ws[warp] = k.s; wc[warp] = k.c; }
    __syncthreads();
    if (warp == 0) {
        k.s = lane < nw ? ws[lane] : 0.0;
        k.c = lane < nw ? wc[lane] : 0.0;
        tree(k, 16);
    }
    return k;
}

// out: nullable; with it (a single CTA) the sum itself, else this CTA's pair into part
__global__ void __launch_bounds__(kRedThreadsLong) reduce_energy_part_kernel(const double *job_e, long long n,
                                                                         double *part, double *out) {
    const long long chunk = (n + gridDim.x - 1) / gridDim.x;
    const long long lo = blockIdx.x * chunk, hi = lo + chunk < n ? lo + chunk : n;
    KSum k;
#pragma unroll 4
    for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) k.add(job_e[i]);
    k = block_ksum(k);
    if (threadIdx.x == 0) {
        if (out) {
            out[0] = k.value();
        } else {
            part[2 * blockIdx.x] = k.s;
            part[2 * blockIdx.x + 1] = k.c;
        }
    }
}

__global__ void __launch_bounds__(kRedThreads) reduce_energy_final_kernel(const double *part, int nparts,
                                                                          double *out) {
    KSum k;
    for (int i = threadIdx.x; i < nparts; i += kRedThreads) {
        k.add(part[2 * i]);
        k.c += part[2 * i + 1];
    }
    k = block_ksum(k);
    if (threadIdx.x == 0) out[0] = k.value();
}

// single-CTA variant (no work buffer)
__global__ void __launch_bounds__(1024) reduce_energy_kernel(const double *job_e, long long n, double *out) {
    KSum k;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) k.add(job_e[i]);
    k = block_ksum(k);
    if (threadIdx.x == 0) out[0] = k.value();
}

cudaError_t reduce_energy_1cta(const double *job_e, long long n, double *e_out, cudaStream_t st) {
    reduce_energy_kernel<<<1, 1024, 0, st>>>(job_e, n, e_out);
    return cudaGetLastError();
}

cudaError_t reduce_energy(const double *job_e, long long n, double *e_out, double *work, cudaStream_t st) {
    // one CTA up to 8 values a thread (the second launch costs more than it saves)
    const int parts = n <= 8 * kRedThreads ? 1 : (int)(n / kRedThreads < kReduceParts ? n / kRedThreads : kReduceParts);
    const int threads = n > (1LL << 20) ? kRedThreadsLong : kRedThreads;
    reduce_energy_part_kernel<<<parts, threads, 0, st>>>(job_e, n, work, parts == 1 ? e_out : nullptr);
    if (parts > 1) reduce_energy_final_kernel<<<1, kRedThreads, 0, st>>>(work, parts, e_out);
    return cudaGetLastError();
}

}  // namespace ctb
