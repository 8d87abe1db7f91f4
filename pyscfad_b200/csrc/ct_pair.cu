// Float64 GEMMs of the slot path (nocc > 24, nocc = 1; the W build also for the
// iterative solver's seed, the allocation-free energy and energies over few jobs at
// every nocc) on the float64 tensor pipe.  The operations per term t = (job, sigma)
// with (x, y, z) as in ct_common.cuh:
//   W    G_t[p,qr]  = sum_f vvop[x,y,p,o+f] t2T[z,f,qr] - sum_l vooo[x,pq,l] t2T[z,y,l,r]
//                                                     (get_wv, ccsd_t.c:98-152)
//   VB   vvop_bar[x,y,p,o+f] += sum_qr t2T[z,f,qr] Wbar_t[p,qr]   (get_vvov_bar, ccsd_t_vjp.c:139-152)
//   TB   t2T_bar[z,f,qr]     += sum_{t: z} sum_p vvop[x,y,p,o+f] Wbar_t[p,qr]   (get_t2T_bar dgemm 1)
//   OB1  vooo_bar[x,pq,l]    -= sum_{t: x} sum_r t2T[z,y,l,r] Wbar_t[pq,r]      (get_vooo_bar, :154-169)
//   OB2  t2T_bar[z,y,l,r]    -= sum_pq vooo[x,pq,l] Wbar_t[pq,r]                (get_t2T_bar dgemm 2)
// A job's two terms with the same z (W, VB) or x (OB2) share the large operand,
// so one CTA takes both: 2 o rows against one tile of it.  TB and OB1 sum over
// a wave's terms with that z or x, so an output tile is added to memory once
// per part of the list.  All kernels: 256 threads, operands in a ring of
// kStages shared-memory stages filled by cp.async (16-byte pieces when the sizes
// are even and the arrays aligned, else 8), row strides of 4 or 12 mod 16 doubles so
// that fragment loads touch every bank once.
// Against 64 x 48 tiles of one term with a register prefetch and F2 as a pass of
// its own (slab block of 6,213 jobs, nocc=48/nvir=300, ms; in brackets the time of
// the flops at 37 TFLOP/s): W 127 -> 91 (78), VB 87 -> 81 (67), TB 100 -> 82 (67),
// OB1 27 -> 13 (11), OB2 19 -> 12 (11).  nocc=33/nvir=64, all jobs: W 225 -> 146,
// VB 61 -> 60, TB 92 -> 50, OB1 88 -> 39, OB2 67 -> 42 (odd sizes copy 8 bytes at a
// time, and 33 takes five tiles of 8).
#include <cuda_runtime.h>
#include <algorithm>
#include "ct_common.cuh"
#include "ct_internal.h"

namespace ctb {
namespace pairk {

constexpr int kThreads = 256, kStages = 3, kKC = 16, kLD = kKC + 4;

struct Args {
    const double *t2T, *vooo, *vvop;
    double *S;                         // the wave's slots: G in 0-5, later w-bar in 0-2 (wbar_cube)
    double *t2T_bar, *vooo_bar, *vvop_bar;
    const int *jobs, *entries, *parts;
    int o, v, n;
    int cols;                          // VB: columns of a CTA
    unsigned magic;                    // ceil(2^32 / o)
};

// terms of a job that share z = c, b, a / x = a, b, c
__device__ __forceinline__ int term_of_z(int i, int h) { return (0x534120 >> (4 * (2 * i + h))) & 15; }
__device__ __forceinline__ int term_of_x(int i, int h) { return 2 * i + h; }

template <int VEC> __device__ __forceinline__ void cp_piece(double *dst, const double *src, bool ok) {
    if (VEC == 2) cp_async16z(dst, src, ok);
    else cp_async8(dst, src, ok);
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest kStages - 2 groups have landed
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory"); }

// the loop every kernel runs: stage(it, buf) requests iteration it's operands, mma(it, buf) uses them
template <class Stage, class Mma> __device__ __forceinline__ void ring(int n_it, Stage stage, Mma mma) {
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < n_it) stage(s, s);
        cp_commit();
    }
    int buf = 0, nbuf = kStages - 1;
    for (int it = 0; it < n_it; ++it) {
        cp_wait();
        __syncthreads();   // iteration it has landed for all; its successor's buffer is free
        if (it + kStages - 1 < n_it) stage(it + kStages - 1, nbuf);
        cp_commit();
        mma(it, buf);
        buf = buf + 1 == kStages ? 0 : buf + 1;
        nbuf = nbuf + 1 == kStages ? 0 : nbuf + 1;
    }
}

// Sizes for nocc <= 8 TT: a term's rows are two halves of MP tiles of 8 (one per
// warp), a (p or r) index as columns takes TT tiles
template <int TT> struct Dim {
    static constexpr int MP = (TT + 1) / 2, RP = 16 * MP, CT = 8 * TT;
};

// ---------------------------------------------------------------- W
// 2 o rows (h, p) x the columns (q, r) of NQ q: two, of which a warp takes one,
// or (past nocc = 48, where a warp's accumulators would leave one CTA per SM) one,
// of which a warp takes half of r.  F2 couples q with its A operand, so a column
// tile of whole q takes F2 as further K iterations into the same accumulators:
// a second pass over the G slots (a read and a write of 5.3 MB per job at
// nocc = 48) is not needed.
template <int TT> constexpr int w_nq() { return TT <= 6 ? 2 : 1; }
template <int TT> constexpr int w_stage() {
    using D = Dim<TT>;
    constexpr int NQ = w_nq<TT>();
    const int f1 = 2 * D::RP * kLD + kKC * (NQ * D::CT + 4), f2 = 2 * NQ * D::RP * 12 + 16 * (D::CT + 4);
    return f1 > f2 ? f1 : f2;
}

template <int TT, int VEC>
__global__ void __launch_bounds__(kThreads, 2) w_kernel(const Args A) {
    using D = Dim<TT>;
    constexpr int MP = D::MP, RP = D::RP, CT = D::CT, NQ = w_nq<TT>(), NT = NQ == 2 ? TT : MP;
    constexpr int BS = NQ * CT + 4, SZ = w_stage<TT>();
    constexpr int KL = 8, A2 = KL + 4, B2 = CT + 4;   // F2: K chunks of 8
    extern __shared__ __align__(16) double sm[];
    const int o = A.o, v = A.v, n = A.n, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int jl = blockIdx.x / 3, zi = blockIdx.x - 3 * jl, q0 = NQ * blockIdx.y;
    int a, b, c, x0, y0, x1, y1, z;
    unpack_job(A.jobs[jl], a, b, c);
    term_xyz(term_of_z(zi, 0), a, b, c, x0, y0, z);
    term_xyz(term_of_z(zi, 1), a, b, c, x1, y1, z);
    const double *v0 = A.vvop + ((long long)x0 * v + y0) * o * n + o, *v1 = A.vvop + ((long long)x1 * v + y1) * o * n + o;
    const double *tz = A.t2T + (long long)z * v * oo + (long long)q0 * o;
    const double *w0 = A.vooo + x0 * o3 + (long long)q0 * o, *w1 = A.vooo + x1 * o3 + (long long)q0 * o;
    const double *t0 = A.t2T + ((long long)z * v + y0) * oo, *t1 = A.t2T + ((long long)z * v + y1) * oo;
    const int n1 = (v + kKC - 1) / kKC, n2 = (o + KL - 1) / KL;
    const bool two = NQ == 2 && q0 + 1 < o;

    auto stage = [&](int it, int buf) {
        double *As = sm + buf * SZ;
        if (it < n1) {
            double *Bs = As + 2 * RP * kLD;
            const int k0 = it * kKC;
            constexpr int PC = kKC / VEC, RW = kThreads / PC;
            const int kc = (tid % PC) * VEC;
            const bool kok = k0 + kc < v;
#pragma unroll
            for (int i = 0; i < 2 * RP / RW; ++i) {
                const int row = i * RW + tid / PC, p = row < RP ? row : row - RP;
                cp_piece<VEC>(As + row * kLD + kc, (row < RP ? v0 : v1) + (long long)p * n + k0 + kc, kok && p < o);
            }
            const int kr = tid >> 4;
            const double *src = tz + (long long)(k0 + kr) * oo;
#pragma unroll
            for (int j = 0; j < (NQ * TT + 2 * VEC - 1) / (2 * VEC); ++j) {
                const int cl = ((tid & 15) + 16 * j) * VEC, qi = cl >= CT, r = cl - qi * CT;
                if (cl < NQ * CT)
                    cp_piece<VEC>(Bs + kr * BS + cl, src + qi * o + r, r < o && (!qi || two) && k0 + kr < v);
            }
        } else {
            double *Bs = As + 2 * NQ * RP * A2;
            const int k0 = (it - n1) * KL;
            constexpr int PC = KL / VEC, RW = kThreads / PC;
            const int kc = (tid % PC) * VEC;
            const bool kok = k0 + kc < o;
#pragma unroll
            for (int i = 0; i < (2 * NQ * RP + RW - 1) / RW; ++i) {
                const int row = i * RW + tid / PC, hq = row / RP, p = row - hq * RP, qi = NQ == 2 ? hq & 1 : 0;   // row = (h, q, p)
                if (2 * NQ * RP % RW == 0 || row < 2 * NQ * RP)
                    cp_piece<VEC>(As + row * A2 + kc, (hq < NQ ? w0 : w1) + (long long)p * oo + qi * o + k0 + kc,
                              kok && p < o && (!qi || two));
            }
            const int kr = tid >> 4, h = kr >> 3, l = kr & 7;
            const double *src = (h ? t1 : t0) + (k0 + l) * o;
#pragma unroll
            for (int j = 0; j < (TT + 2 * VEC - 1) / (2 * VEC); ++j) {
                const int r = ((tid & 15) + 16 * j) * VEC;
                if (r < CT) cp_piece<VEC>(Bs + kr * B2 + r, src + r, r < o && k0 + l < o);
            }
        }
    };
    // warps (h, half of p, q or half of r); with an odd TT the second half is a tile
    // short, and the halves are swapped for h = 1 so that each scheduler has as many tiles
    const int h = warp >> 2, wc = (warp & 1) ^ (NQ == 1 ? h : 0), half = ((warp >> 1) & 1) ^ h;
    const int qi = NQ == 2 ? wc : 0, r0 = NQ == 2 ? 0 : wc * MP * 8;
    const bool last = TT % 2 == 0 || half == 0, lastc = NQ == 2 || TT % 2 == 0 || wc == 0;
    double acc[MP][NT][2];
#pragma unroll
    for (int m = 0; m < MP; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    auto step = [&](const double *ap, int as, const double *bp) {
        double af[MP];
#pragma unroll
        for (int m = 0; m < MP; ++m) af[m] = ap[m * 8 * as];
#pragma unroll
        for (int t = 0; t < NT; ++t)
            if (t + 1 < NT || lastc) {
                const double bf = bp[8 * t];
#pragma unroll
                for (int m = 0; m < MP; ++m)
                    if (m + 1 < MP || last) dmma(acc[m][t], af[m], bf);
            }
    };
    auto mma = [&](int it, int buf) {
        const double *As = sm + buf * SZ;
        if (it == n1) {
#pragma unroll
            for (int m = 0; m < MP; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) { acc[m][t][0] = -acc[m][t][0]; acc[m][t][1] = -acc[m][t][1]; }
        }
        if (it < n1) {
            const double *ap = As + (h * RP + half * MP * 8 + g) * kLD + c4;
            const double *bp = As + 2 * RP * kLD + c4 * BS + qi * CT + r0 + g;
#pragma unroll
            for (int ks = 0; ks < kKC / 4; ++ks) step(ap + 4 * ks, kLD, bp + 4 * ks * BS);
        } else {
            const double *ap = As + ((NQ * h + qi) * RP + half * MP * 8 + g) * A2 + c4;
            const double *bp = As + 2 * NQ * RP * A2 + (h * KL + c4) * B2 + r0 + g;
#pragma unroll
            for (int ks = 0; ks < KL / 4; ++ks) step(ap + 4 * ks, A2, bp + 4 * ks * B2);
        }
    };
    ring(n1 + n2, stage, mma);

    if (qi && !two) return;
    double *dst = A.S + ((long long)jl * kSlots + term_of_z(zi, h)) * o3 + (q0 + qi) * o;
#pragma unroll
    for (int m = 0; m < MP; ++m) {
        const int p = (half * MP + m) * 8 + g;
        if (p >= o || !(m + 1 < MP || last)) continue;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int r = r0 + 8 * t + 2 * c4;
            double *d = dst + (long long)p * oo + r;
            if (VEC == 2) {
                if (r < o) *reinterpret_cast<double2 *>(d) = make_double2(-acc[m][t][0], -acc[m][t][1]);
            } else {
                if (r < o) d[0] = -acc[m][t][0];
                if (r + 1 < o) d[1] = -acc[m][t][1];
            }
        }
    }
}

// ---------------------------------------------------------------- VB
// 2 o rows (h, p) x up to 64 virtuals f, K = qr; both operands run along K (the
// w-bar rows in pieces of o)
template <int TT, int VEC>
__global__ void __launch_bounds__(kThreads, 2) vb_kernel(const Args A) {
    using D = Dim<TT>;
    constexpr int MP = D::MP, RP = D::RP, NT = 4, SZ = (2 * RP + 64) * kLD;
    extern __shared__ __align__(16) double sm[];
    const int o = A.o, v = A.v, n = A.n, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int jl = blockIdx.x / 3, zi = blockIdx.x - 3 * jl, f0 = A.cols * blockIdx.y, fn = min(A.cols, v - f0);
    int a, b, c, x0, y0, x1, y1, z;
    unpack_job(A.jobs[jl], a, b, c);
    term_xyz(term_of_z(zi, 0), a, b, c, x0, y0, z);
    term_xyz(term_of_z(zi, 1), a, b, c, x1, y1, z);
    const int t0 = term_of_z(zi, 0), t1 = term_of_z(zi, 1);
    const double *s0 = A.S + ((long long)jl * kSlots + wbar_cube(t0)) * o3;
    const double *s1 = A.S + ((long long)jl * kSlots + wbar_cube(t1)) * o3;
    const bool p0 = wbar_first(t0), p1 = wbar_first(t1);
    const double *tz = A.t2T + ((long long)z * v + f0) * oo;

    auto stage = [&](int it, int buf) {
        double *As = sm + buf * SZ;
        constexpr int PC = kKC / VEC, RW = kThreads / PC;
        const int kc = (tid % PC) * VEC, k = it * kKC + kc;
        const bool kok = k < oo;
        const int q = (int)__umulhi((unsigned)k, A.magic), k1 = k + q * (oo - o);   // k as q o^2 + r
        const double *a0 = s0 + (p0 ? k : k1), *a1 = s1 + (p1 ? k : k1);
        const int d0 = p0 ? oo : o, d1 = p1 ? oo : o;
#pragma unroll
        for (int i = 0; i < (2 * RP + 64) / RW; ++i) {
            const int row = i * RW + tid / PC, p = row < RP ? row : row - RP;
            const double *src = row < 2 * RP ? (row < RP ? a0 + p * d0 : a1 + p * d1)
                                             : tz + (long long)(row - 2 * RP) * oo + k;
            cp_piece<VEC>(As + row * kLD + kc, src, kok && (row < 2 * RP ? p < o : row - 2 * RP < fn));
        }
    };
    const int h = warp >> 2, ci = warp & 1, half = ((warp >> 1) & 1) ^ h;
    const bool last = TT % 2 == 0 || half == 0;
    const int nt = min(NT, (fn - 32 * ci + 7) >> 3);   // column tiles of this warp
    double acc[MP][NT][2];
#pragma unroll
    for (int m = 0; m < MP; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    auto mma = [&](int, int buf) {
        const double *ap = sm + buf * SZ + (h * RP + half * MP * 8 + g) * kLD + c4;
        const double *bp = sm + buf * SZ + (2 * RP + 32 * ci + g) * kLD + c4;
#pragma unroll
        for (int ks = 0; ks < kKC / 4; ++ks) {
            double af[MP];
#pragma unroll
            for (int m = 0; m < MP; ++m) af[m] = ap[m * 8 * kLD + 4 * ks];
#pragma unroll
            for (int t = 0; t < NT; ++t)
                if (t < nt) {
                    const double bf = bp[t * 8 * kLD + 4 * ks];
#pragma unroll
                    for (int m = 0; m < MP; ++m)
                        if (m + 1 < MP || last) dmma(acc[m][t], af[m], bf);
                }
        }
    };
    ring((oo + kKC - 1) / kKC, stage, mma);

    double *dst = A.vvop_bar + ((long long)(h ? x1 : x0) * v + (h ? y1 : y0)) * o * n + o + f0 + 32 * ci;
#pragma unroll
    for (int m = 0; m < MP; ++m) {
        const int p = (half * MP + m) * 8 + g;
        if (p >= o || !(m + 1 < MP || last)) continue;
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int f = 8 * t + 2 * c4 + e;
                if (32 * ci + f < fn) atomicAdd(dst + (long long)p * n + f, acc[m][t][e]);
            }
    }
}

// ---------------------------------------------------------------- OB2
// l x (h, r) of the two terms with that x, K = pq; both operands run along the
// columns, vooo is read once for both terms
template <int TT, int VEC>
__global__ void __launch_bounds__(kThreads, 2) ob2_kernel(const Args A) {
    using D = Dim<TT>;
    constexpr int MP = D::MP, CT = D::CT, LD = CT + 4, SZ = 3 * kKC * LD;
    extern __shared__ __align__(16) double sm[];
    const int o = A.o, v = A.v, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int jl = blockIdx.x / 3, xi = blockIdx.x - 3 * jl;
    int a, b, c, x, y0, z0, y1, z1;
    unpack_job(A.jobs[jl], a, b, c);
    term_xyz(term_of_x(xi, 0), a, b, c, x, y0, z0);
    term_xyz(term_of_x(xi, 1), a, b, c, x, y1, z1);
    const double *src0 = A.vooo + x * o3;
    const int s1 = term_of_x(xi, 0), s2 = term_of_x(xi, 1);
    const double *src1 = A.S + ((long long)jl * kSlots + wbar_cube(s1)) * o3;
    const double *src2 = A.S + ((long long)jl * kSlots + wbar_cube(s2)) * o3;
    const bool p1 = wbar_first(s1), p2 = wbar_first(s2);

    auto stage = [&](int it, int buf) {
        const int kr = tid >> 4, k = it * kKC + kr;
        const int p = (int)__umulhi((unsigned)k, A.magic), kt = (k - p * o) * o + p;   // k = (p, q), kt = (q, p)
        double *dst = sm + buf * SZ + kr * LD;
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const double *src = u == 0 ? src0 + k * o : (u == 1 ? src1 + (p1 ? k : kt) * o : src2 + (p2 ? k : kt) * o);
#pragma unroll
            for (int j = 0; j < (TT + 2 * VEC - 1) / (2 * VEC); ++j) {
                const int r = ((tid & 15) + 16 * j) * VEC;
                if (r < CT) cp_piece<VEC>(dst + u * kKC * LD + r, src + r, r < o && k < oo);
            }
        }
    };
    // warps (term, half of l, half of r); with an odd TT a half may be a tile short
    const int h = warp >> 2, hl = ((warp >> 1) & 1) ^ h, hr = (warp & 1) ^ h;
    const bool ml = TT % 2 == 0 || hl == 0, mr = TT % 2 == 0 || hr == 0;
    double acc[MP][MP][2];
#pragma unroll
    for (int m = 0; m < MP; ++m)
#pragma unroll
        for (int t = 0; t < MP; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    auto mma = [&](int, int buf) {
        const double *ap = sm + buf * SZ + c4 * LD + hl * MP * 8 + g;
        const double *bp = sm + buf * SZ + ((1 + h) * kKC + c4) * LD + hr * MP * 8 + g;
#pragma unroll
        for (int ks = 0; ks < kKC / 4; ++ks) {
            double af[MP];
#pragma unroll
            for (int m = 0; m < MP; ++m) af[m] = m + 1 < MP || ml ? ap[4 * ks * LD + 8 * m] : 0.0;
#pragma unroll
            for (int t = 0; t < MP; ++t)
                if (t + 1 < MP || mr) {
                    const double bf = bp[4 * ks * LD + 8 * t];
#pragma unroll
                    for (int m = 0; m < MP; ++m)
                        if (m + 1 < MP || ml) dmma(acc[m][t], af[m], bf);
                }
        }
    };
    ring((oo + kKC - 1) / kKC, stage, mma);

    double *dst = A.t2T_bar + ((long long)(h ? z1 : z0) * v + (h ? y1 : y0)) * oo;
#pragma unroll
    for (int m = 0; m < MP; ++m) {
        const int l = (hl * MP + m) * 8 + g;
        if (l >= o) continue;
#pragma unroll
        for (int t = 0; t < MP; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = (hr * MP + t) * 8 + 2 * c4 + e;
                if (r < o) atomicAdd(dst + l * o + r, -acc[m][t][e]);
            }
    }
}

// ---------------------------------------------------------------- TB, OB1
// One part of the terms with a z or x (cut by the plan into parts of about equal
// length): their descriptors in shared memory, kTerms at a time (two blocks, so
// that the ring may run ahead into the next one)
constexpr int kTerms = 64;
struct Terms {
    int js[2 * kTerms];   // 8 jl + sigma
    int pr[2 * kTerms];   // TB: x v + y; OB1: z v + y
};

struct Part {
    int key, e0, nt;      // z or x, first entry, terms
};
__device__ __forceinline__ Part part_of(const Args &A) {
    const int *q = A.parts + 3 * blockIdx.x;
    return {q[0], q[1], q[2] - q[1]};
}

// descriptors of terms [base, base + kTerms) of the part; visible after the next barrier
template <bool TB> __device__ __forceinline__ void load_terms(const Args &A, const Part &P, int base, Terms &T) {
    const int i = base + threadIdx.x;
    if (threadIdx.x < kTerms && i < P.nt) {
        const int id = A.entries[P.e0 + i], jl = id / 6, s = id - 6 * jl;
        int a, b, c, x, y, z;
        unpack_job(A.jobs[jl], a, b, c);
        term_xyz(s, a, b, c, x, y, z);
        T.js[i & (2 * kTerms - 1)] = 8 * jl + s;
        T.pr[i & (2 * kTerms - 1)] = (TB ? x : z) * A.v + y;
    }
}

// TB: 64 virtuals f x 128 columns qr, K = p of each term in chunks of 16; both
// operands run along the columns.  8 warps of 32 x 32.
template <int VEC>
__global__ void __launch_bounds__(kThreads, 2) tb_kernel(const Args A) {
    constexpr int LA = 64 + 4, LB = 128 + 4, SZ = kKC * (LA + LB);
    extern __shared__ __align__(16) double sm[];
    __shared__ Terms T;
    const int o = A.o, v = A.v, n = A.n, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const Part P = part_of(A);
    const int tn = (oo + 127) / 128, f0 = (blockIdx.y / tn) * 64, n0 = (blockIdx.y % tn) * 128;
    const int per = (o + kKC - 1) / kKC, op = (o + 3) & ~3;   // chunks of a term, its rows as MMA steps
    int st_t = 0, st_c = 0, mm_c = 0;                          // positions of the request and of the product
    load_terms<true>(A, P, 0, T);
    __syncthreads();
    int ct[8 / VEC];   // this thread's w-bar columns (q, r) as q o^2 + r
#pragma unroll
    for (int j = 0; j < 8 / VEC; ++j) {
        const int cl = n0 + ((tid & 15) + 16 * j) * VEC;
        ct[j] = cl + (int)__umulhi((unsigned)cl, A.magic) * (oo - o);
    }
    auto stage = [&](int, int buf) {
        double *As = sm + buf * SZ, *Bs = As + kKC * LA;
        const int js = T.js[st_t & (2 * kTerms - 1)], xy = T.pr[st_t & (2 * kTerms - 1)], k0 = st_c * kKC;
        const double *va = A.vvop + (long long)xy * o * n + o + f0;
        const bool first = wbar_first(js & 7);
        const double *wb = A.S + ((long long)(js >> 3) * kSlots + wbar_cube(js & 7)) * o3;
        const int kr = tid >> 4, p = k0 + kr;
        const bool pok = p < o;
#pragma unroll
        for (int j = 0; j < 4 / VEC; ++j) {
            const int cl = ((tid & 15) + 16 * j) * VEC;
            cp_piece<VEC>(As + kr * LA + cl, va + (long long)p * n + cl, pok && f0 + cl < v);
        }
#pragma unroll
        for (int j = 0; j < 8 / VEC; ++j) {
            const int cl = ((tid & 15) + 16 * j) * VEC;
            cp_piece<VEC>(Bs + kr * LB + cl, wb + (first ? p * oo + n0 + cl : p * o + ct[j]), pok && n0 + cl < oo);
        }
        if (++st_c == per) {
            st_c = 0;
            // halfway into a block, the next one's descriptors (its previous content has been requested)
            if ((++st_t & (kTerms - 1)) == kTerms / 2) load_terms<true>(A, P, (st_t & ~(kTerms - 1)) + kTerms, T);
        }
    };
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto mma = [&](int, int buf) {
        const double *ap = sm + buf * SZ + c4 * LA + wm + g, *bp = sm + buf * SZ + kKC * LA + c4 * LB + wn + g;
        const int rows = min(kKC, op - mm_c * kKC);
        if (++mm_c == per) mm_c = 0;
#pragma unroll
        for (int ks = 0; ks < kKC / 4; ++ks) {
            if (4 * ks >= rows) break;
            double af[4], bf[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { af[i] = ap[4 * ks * LA + 8 * i]; bf[i] = bp[4 * ks * LB + 8 * i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
    };
    ring(P.nt * per, stage, mma);

    double *dst = A.t2T_bar + (long long)P.key * v * oo;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int f = f0 + wm + 8 * i + g;
        if (f >= v) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int cl = n0 + wn + 8 * j + 2 * c4 + e;
                if (cl < oo) atomicAdd(dst + (long long)f * oo + cl, acc[i][j][e]);
            }
    }
}

// OB1: 128 rows pq x l, K = r of each term in chunks of 16; both operands run along K
template <int TT, int VEC>
__global__ void __launch_bounds__(kThreads, 2) ob1_kernel(const Args A) {
    using D = Dim<TT>;
    constexpr int MP = D::MP, RP = D::RP, SZ = (128 + RP) * kLD;
    extern __shared__ __align__(16) double sm[];
    __shared__ Terms T;
    const int o = A.o, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const Part P = part_of(A);
    const int m0 = blockIdx.y * 128;
    const int per = (o + kKC - 1) / kKC, op = (o + 3) & ~3;
    int st_t = 0, st_c = 0, mm_c = 0;
    load_terms<false>(A, P, 0, T);
    __syncthreads();
    constexpr int PC = kKC / VEC, RW = kThreads / PC;
    int rt[128 / RW];   // this thread's rows (p, q) as q o + p
#pragma unroll
    for (int i = 0; i < 128 / RW; ++i) {
        const int row = m0 + i * RW + tid / PC, p = (int)__umulhi((unsigned)row, A.magic);
        rt[i] = (row - p * o) * o + p;
    }
    auto stage = [&](int, int buf) {
        double *As = sm + buf * SZ;
        const int js = T.js[st_t & (2 * kTerms - 1)], zy = T.pr[st_t & (2 * kTerms - 1)];
        const bool first = wbar_first(js & 7);
        const int kc = (tid % PC) * VEC, k = st_c * kKC + kc;
        const double *wb = A.S + ((long long)(js >> 3) * kSlots + wbar_cube(js & 7)) * o3 + k;
        const double *tt = A.t2T + (long long)zy * oo + k;
        const bool kok = k < o;
#pragma unroll
        for (int i = 0; i < 128 / RW; ++i) {
            const int row = i * RW + tid / PC;
            cp_piece<VEC>(As + row * kLD + kc, wb + (first ? m0 + row : rt[i]) * o, kok && m0 + row < oo);
        }
#pragma unroll
        for (int i = 0; i < (RP + RW - 1) / RW; ++i) {
            const int l = i * RW + tid / PC;
            if (RP % RW == 0 || l < RP) cp_piece<VEC>(As + (128 + l) * kLD + kc, tt + l * o, kok && l < o);
        }
        if (++st_c == per) {
            st_c = 0;
            if ((++st_t & (kTerms - 1)) == kTerms / 2) load_terms<false>(A, P, (st_t & ~(kTerms - 1)) + kTerms, T);
        }
    };
    const int wm = (warp >> 1) * 32, half = (warp & 1) ^ ((warp >> 2) & 1);
    const bool last = TT % 2 == 0 || half == 0;
    double acc[4][MP][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int t = 0; t < MP; ++t) acc[i][t][0] = acc[i][t][1] = 0.0;
    auto mma = [&](int, int buf) {
        const double *ap = sm + buf * SZ + (wm + g) * kLD + c4, *bp = sm + buf * SZ + (128 + half * MP * 8 + g) * kLD + c4;
        const int rows = min(kKC, op - mm_c * kKC);
        if (++mm_c == per) mm_c = 0;
#pragma unroll
        for (int ks = 0; ks < kKC / 4; ++ks) {
            if (4 * ks >= rows) break;
            double af[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) af[i] = ap[8 * i * kLD + 4 * ks];
#pragma unroll
            for (int t = 0; t < MP; ++t)
                if (t + 1 < MP || last) {
                    const double bf = bp[8 * t * kLD + 4 * ks];
#pragma unroll
                    for (int i = 0; i < 4; ++i) dmma(acc[i][t], af[i], bf);
                }
        }
    };
    ring(P.nt * per, stage, mma);

    double *dst = A.vooo_bar + P.key * o3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int pq = m0 + wm + 8 * i + g;
        if (pq >= oo) continue;
#pragma unroll
        for (int t = 0; t < MP; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int l = (half * MP + t) * 8 + 2 * c4 + e;
                if (l < o) atomicAdd(dst + (long long)pq * o + l, -acc[i][t][e]);
            }
    }
}

template <class K> static cudaError_t run(K kernel, dim3 grid, int stage_doubles, const Args &A, cudaStream_t st) {
    const int smem = kStages * stage_doubles * (int)sizeof(double);
    cudaError_t e = smem_optin(reinterpret_cast<const void *>(kernel), smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, kThreads, smem, st>>>(A);
    return cudaGetLastError();
}

template <int TT, int VEC>
static cudaError_t launch(GemmKind kind, const WaveView &w, Args &A, cudaStream_t st) {
    using D = Dim<TT>;
    const int o = A.o, v = A.v, oo = o * o, pairs = 3 * w.n_jobs;
    if (kind == K_W) return run(w_kernel<TT, VEC>, dim3(pairs, (o + w_nq<TT>() - 1) / w_nq<TT>()), w_stage<TT>(), A, st);
    // the bars of nocc 2-24 are ct_cube.cu's
    if constexpr (TT == 2 || TT == 3) return cudaErrorInvalidValue;
    else switch (kind) {
    case K_VB: {
        const int ng = (v + 63) / 64;
        A.cols = ((v + ng - 1) / ng + 15) / 16 * 16;
        return run(vb_kernel<TT, VEC>, dim3(pairs, (v + A.cols - 1) / A.cols), (2 * D::RP + 64) * kLD, A, st);
    }
    case K_TB: {
        if (w.n_zparts <= 0) return cudaSuccess;
        A.entries = w.tb_entries;
        A.parts = w.zparts;
        return run(tb_kernel<VEC>, dim3(w.n_zparts, ((v + 63) / 64) * ((oo + 127) / 128)), kKC * (64 + 128 + 8), A, st);
    }
    case K_OB1: {
        if (w.n_xparts <= 0) return cudaSuccess;
        A.entries = w.x_entries;
        A.parts = w.xparts;
        return run(ob1_kernel<TT, VEC>, dim3(w.n_xparts, (oo + 127) / 128), (128 + D::RP) * kLD, A, st);
    }
    default: return run(ob2_kernel<TT, VEC>, dim3(pairs, 1), 3 * kKC * (D::CT + 4), A, st);
    }
}

template <int VEC>
static cudaError_t launch_o(GemmKind kind, const WaveView &w, Args &A, cudaStream_t st) {
    switch ((A.o + 7) / 8) {
    case 1: return launch<1, VEC>(kind, w, A, st);
    case 2: return launch<2, VEC>(kind, w, A, st);
    case 3: return launch<3, VEC>(kind, w, A, st);
    case 4: return launch<4, VEC>(kind, w, A, st);
    case 5: return launch<5, VEC>(kind, w, A, st);
    case 6: return launch<6, VEC>(kind, w, A, st);
    case 7: return launch<7, VEC>(kind, w, A, st);
    case 8: return launch<8, VEC>(kind, w, A, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pairk

cudaError_t f64_gemm(GemmKind kind, const WaveView &w, const double *t2T, const double *vooo, const double *vvop,
                     double *slots, double *out, cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    pairk::Args A{};
    A.t2T = t2T;
    A.vooo = vooo;
    A.vvop = vvop;
    A.S = slots;
    A.t2T_bar = A.vooo_bar = A.vvop_bar = out;   // each kind adds into one of them
    A.jobs = w.jobs;
    A.o = w.o; A.v = w.v; A.n = w.n;
    A.magic = (unsigned)(((1ull << 32) + w.o - 1) / w.o);
    const bool even = w.o % 2 == 0 && w.v % 2 == 0;
    auto aligned = [](const double *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    return even && aligned(t2T) && aligned(vooo) && aligned(vvop) && aligned(slots)
               ? pairk::launch_o<2>(kind, w, A, st)
               : pairk::launch_o<1>(kind, w, A, st);
}

}  // namespace ctb
