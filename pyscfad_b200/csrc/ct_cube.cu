// Float64 path for small nocc (o <= kCubeMaxO): one CTA keeps a sorted job's
// o^3 cube in shared memory from the W build to the last gradient.
//
// The slot path (ct_fp64.cu) writes the six G_sigma cubes of a job to memory,
// reads them in the orbit epilogue and writes six W-bar cubes back; at small
// nocc its GEMM tiles are o columns wide and bound by operand traffic (3.2
// flop/byte at nocc = 16).  Here (job a >= b >= c, terms as in ct_common.cuh):
//   F1  for each z the two terms with that z form one GEMM
//         D[(h,p), qr] = sum_f vvop[x_h,y_h,p,o+f] t2T[z,f,qr]   (2o x o^2 x v)
//       t2T[z] is read once for 2o rows, straight into B fragments; D is
//       added into the cube W through each term's index permutation
//   F2  for each x: D[(h,r), pq] = sum_l t2T[z_h,y_h,l,r] vooo[x,pq,l], subtracted
//   EPI element orbits from the cube: V, r3, energy, mo_energy bars; ybar
//       replaces W in place, w-bar (one cube: the six W-bar_sigma are its index
//       permutations) goes to the job's scratch
//   VT  V-term bars from the ybar cube; then w-bar is read back in its place
//   VB  vvop_bar[x_h,y_h,p,o+f] += sum_qr Wbar_h[p,qr] t2T[z,f,qr]   (2o x v x o^2)
//   OB2 t2T_bar[z_h,y_h,l,r] -= sum_pq Wbar_h[pq,r] vooo[x,pq,l]
//   OB1 vooo_bar[x,pq,l] -= sum_(h,r) t2T[z_h,y_h,l,r] Wbar_h[pq,r]
// and a second kernel, grouped by z over a wave's terms as on the slot path:
//   TB  t2T_bar[z,f,qr] += sum_t sum_p vvop[x,y,p,o+f] Wbar_t[p,qr]
// (the same arithmetic as ccsd_t.c:98-152, ccsd_t_vjp.c:9-246; file and line
// per step in ct_fp64.cu).  All products run on the float64 tensor pipe.
#include <cuda_runtime.h>
#include <algorithm>
#include "ct_common.cuh"
#include "ct_internal.h"
#include "ct_epi.cuh"

namespace ctb {
namespace cube {

// what a launch does
enum Mode { M_ENERGY = 0, M_VJP = 1, M_LNO_FWD = 2, M_LNO_BWD = 3 };

struct Args {
    EpiArgs e;
    const int *jobs;
    const double *vooo;
    double *vooo_bar;
    double *cubes;        // per-job scratch: w-bar cube (canonical) or the LNO slots
    long long stride;     // doubles per job
    int sj, si;           // padded strides of the shared cube (k has stride 1)
    int cube_sz, stage_sz, tmp_sz;   // doubles
    int passes;           // column passes of F1/F2
    int kc, nch;          // K chunk of F1's staged operand (a multiple of 16) and their count
    int vb_groups, vb_ks; // VB: column groups of 8 VbNT virtuals, K splits
    int ob2_ks;
    unsigned magic;       // ceil(2^32 / o)
};

constexpr int VbNT = 2;   // 8-column tiles a warp takes per VB unit
// a staged row is the K chunk + 4 (4 mod 16 doubles: conflict-free fragments);
// a V-term tile row has an odd stride (its column reads walk all banks)
__host__ __device__ constexpr int tile_ld(int o) { return o | 1; }

// terms by shared index: F1/VB pair the terms with z = c, b, a; F2/OB the terms with x = a, b, c
__host__ __device__ constexpr int term_z(int i, int h) { return (0x534120 >> (4 * (2 * i + h))) & 15; }
__host__ __device__ constexpr int term_x(int i, int h) { return 2 * i + h; }
// term whose staged t2T[y,x] tile is t2T[z,y] of term s: 3, 5, 1, 4, 0, 2
__host__ __device__ constexpr int tile_zy(int s) { return (0x204153 >> (4 * s)) & 15; }
// (a, b, c) positions of x, y, z of term s: R_s
__device__ __forceinline__ int pick(int m, int a, int b, int c) { return m == 0 ? a : (m == 1 ? b : c); }
// runtime R_s(m), 2 bits each
__device__ __forceinline__ int rtR(int s, int m) {
    // rows (0,1,2) (0,2,1) (1,0,2) (1,2,0) (2,0,1) (2,1,0)
    constexpr unsigned long long P =
        (0ull | 1ull << 2 | 2ull << 4) | (0ull | 2ull << 2 | 1ull << 4) << 6 | (1ull | 0ull << 2 | 2ull << 4) << 12 |
        (1ull | 2ull << 2 | 0ull << 4) << 18 | (2ull | 0ull << 2 | 1ull << 4) << 24 |
        (2ull | 1ull << 2 | 0ull << 4) << 30;
    return (int)((P >> (6 * s + 2 * m)) & 3);
}

template <int MT, int NT, int MODE, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) job_kernel(const Args A) {
    extern __shared__ __align__(16) double sm[];
    const EpiArgs &e = A.e;
    const int o = e.o, v = e.v, n = e.n, oo = o * o;
    const long long o3 = (long long)oo * o;
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
    const int g = lane >> 2, c4 = lane & 3;
    const int sj = A.sj, si = A.si;
    constexpr int HR = 4 * MT;   // F1/F2 rows of a term (o <= HR)
    // k-steps of B requested ahead: one is enough with two CTAs per SM (two spill more;
    // nocc=16/nvir=120 energy 84 against 89 ms), two with one (31.5 against 33.0 ms).
    // With one, eight of the builds in use spill 4 to 28 bytes.
    constexpr int PF = MT == 6 ? 2 : 1;
    double *W = sm;                          // the cube, (i, j, k) at i si + j sj + k
    double *St = W + A.cube_sz;              // GEMM staging, later the V-term tiles
    double *Tm = St + A.stage_sz;            // per-orbit partials / reductions
    double *U = Tm + A.tmp_sz;               // t1T rows a, b, c
    double *F = U + 3 * o;                   // fvo rows a, b, c
    double *eocc = F + 3 * o;
    const int tl = tile_ld(o), tsz = o * tl;
    double *VA = St, *VB = St + 6 * tsz;     // vvop[x,y,:,:o] and t2T[y,x] tiles of the six terms
    __shared__ double wred[3][MAXT / 32];

    int a, jb, c;
    unpack_job(A.jobs[blockIdx.x], a, jb, c);
    double *Sj = A.cubes + (long long)blockIdx.x * A.stride;
    auto S = [&](int m) { return m == 0 ? si : (m == 1 ? sj : 1); };
    auto divo = [&](int x) { return (int)__umulhi((unsigned)x, A.magic); };
    auto xyz = [&](int s, int &x, int &y, int &z) {
        x = pick(rtR(s, 0), a, jb, c);
        y = pick(rtR(s, 1), a, jb, c);
        z = pick(rtR(s, 2), a, jb, c);
    };

    int fnz = 0;
    for (int i = tid; i < 3 * o; i += nthr) {
        const int w = divo(i), r = i - w * o, z = pick(w, a, jb, c);
        U[i] = e.t1T[z * o + r];
        const double f = e.fvo[z * o + r];
        F[i] = f;
        fnz |= f != 0.0;
    }
    for (int i = tid; i < o; i += nthr) eocc[i] = e.mo_energy[i];
    // with zero fvo rows the fvo part of V and the t2T part of its bar add zeros: skipped
    const bool with_fvo = __syncthreads_or(fnz) != 0;

    if (MODE != M_LNO_BWD) {
        // with one column pass the first term's sums initialise the cube; with
        // more, a later pass's would overwrite what the second term has added
        const bool fresh = A.passes == 1;
        if (!fresh)
            for (int i = tid; i < A.cube_sz; i += nthr) W[i] = 0.0;
        // ---- F1 (phases 0-2) and F2 (3-5): iterations (phase, pass, K chunk),
        // the A operand of the next iteration copied while this one runs
        const int nch = A.nch, KC = A.kc, AS = KC + 4, per = A.passes * nch, n_it = 3 * per + 3 * A.passes;
        // position of an iteration, stepped rather than divided out
        struct Pos {
            int ph = 0, pass = 0, ch = 0;
            __device__ __forceinline__ void next(int passes, int nch) {
                if (ph < 3 && ch + 1 < nch) { ++ch; return; }
                ch = 0;
                if (++pass == passes) { pass = 0; ++ph; }
            }
        };
        auto stage = [&](const Pos &q, int buf) {
            double *dst = St + buf * (8 * MT * AS);
            if (q.ph < 3) {
                const int k0 = q.ch * KC, kw = min(KC, (v - k0 + 3) & ~3);
                int x0, y0, z0, x1, y1, z1;
                xyz(term_z(q.ph, 0), x0, y0, z0);
                xyz(term_z(q.ph, 1), x1, y1, z1);
                const double *r0 = e.vvop + ((long long)x0 * v + y0) * o * n + o + k0;
                const double *r1 = e.vvop + ((long long)x1 * v + y1) * o * n + o + k0;
                for (int m = warp; m < 8 * MT; m += nw) {
                    const int p = m < HR ? m : m - HR;
                    const double *src = (m < HR ? r0 : r1) + (long long)p * n;
                    for (int k = lane; k < kw; k += 32) {
                        const bool ok = p < o && k0 + k < v;
                        cp_async8(dst + m * AS + k, src + k, ok);
                    }
                }
            } else {
                int x0, y0, z0, x1, y1, z1;
                xyz(term_x(q.ph - 3, 0), x0, y0, z0);
                xyz(term_x(q.ph - 3, 1), x1, y1, z1);
                const double *r0 = e.t2T + ((long long)z0 * v + y0) * oo, *r1 = e.t2T + ((long long)z1 * v + y1) * oo;
                const int kw = (o + 3) & ~3;
                for (int k = warp; k < kw; k += nw)
                    for (int m = lane; m < 8 * MT; m += 32) {
                        const int r = m < HR ? m : m - HR;
                        const bool ok = r < o && k < o;
                        const double *src = (m < HR ? r0 : r1) + k * o + r;
                        cp_async8(dst + m * AS + k, src, ok);
                    }
            }
            cp_async_commit();
        };
        // B fragments of an iteration: lane (k = c4, column g) of each 8-column
        // tile, PF k-steps in flight in registers.  The first ones are requested
        // as soon as the previous iteration's products are done, under its adds
        // into the cube.
        const double *rp = nullptr;
        int off[NT], full = 0, rem = 0;
        long long kst = 0;
        bool on = false;
        double b[PF][NT], acc[MT][NT][2];
        auto load_b = [&](int q, double (&d)[NT]) {
            if (q < full) {
#pragma unroll
                for (int t = 0; t < NT; ++t) d[t] = __ldg(rp + off[t]);
            } else {
                const bool in = q == full && c4 < rem;
#pragma unroll
                for (int t = 0; t < NT; ++t) d[t] = in ? __ldg(rp + off[t]) : 0.0;
            }
            rp += kst;
        };
        auto prep = [&](const Pos &q) {
            const bool f1 = q.ph < 3;
            const int n0 = (q.pass * nw + warp) * (8 * NT);
            on = n0 < oo;
            const int m = f1 ? 2 - q.ph : q.ph - 3, xz = pick(m, a, jb, c);   // z of F1 phases c, b, a; x of F2 phases
            rp = f1 ? e.t2T + (long long)xz * v * oo + ((long long)q.ch * KC + c4) * oo : A.vooo + xz * o3 + c4;
            kst = f1 ? 4LL * oo : 4;
            const int K = f1 ? min(KC, v - q.ch * KC) : o;
            full = K >> 2;
            rem = K & 3;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int col = min(n0 + 8 * t + g, oo - 1);
                off[t] = f1 ? col : col * o;
            }
            if (on) {
#pragma unroll
                for (int u = 0; u < PF; ++u) load_b(u, b[u]);
            }
        };
        Pos cur, nxt;
        stage(cur, 0);
        prep(cur);
        nxt.next(A.passes, nch);
        for (int it = 0; it < n_it; ++it, cur = nxt, nxt.next(A.passes, nch)) {
            const int ph = cur.ph;
            const bool f1 = ph < 3;
            if (cur.ch == 0) {
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
            }
            cp_async_wait_all();
            __syncthreads();   // this iteration's A operand; the other buffer and the last scatter are done
            if (it + 1 < n_it) stage(nxt, (it + 1) & 1);
            const bool mine = on;
            if (mine) {
                const int ks = full + (rem != 0);
                const double *As = St + (it & 1) * (8 * MT * AS) + g * AS + c4;
                for (int s = 0; s < ks; s += PF) {
#pragma unroll
                    for (int u = 0; u < PF; ++u) {
                        if (s + u < ks) {
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                const double af = As[m * 8 * AS + 4 * (s + u)];
#pragma unroll
                                for (int t = 0; t < NT; ++t) dmma(acc[m][t], af, b[u][t]);
                            }
                            load_b(s + u + PF, b[u]);
                        }
                    }
                }
            }
            if (it + 1 < n_it) prep(nxt);
            if (f1 && cur.ch + 1 < nch) continue;
            // add into the cube: the two terms one after the other (they may
            // meet at the same element), different columns never meet.  A
            // column's loads go out before its stores.  No product runs meanwhile,
            // so the instructions count: term h's rows are h HR + p with HR = 4 MT
            // >= o, so only its first (odd MT) and last row tile are predicated,
            // and columns only in the last group (energy at nocc=16/nvir=120
            // 112 -> 87 ms against a predicate per element).
            const int n0 = (cur.pass * nw + warp) * (8 * NT);
            const double sgn = f1 ? 1.0 : -1.0;
            const bool tail = n0 + 8 * NT > oo;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = f1 ? term_z(ph, h) : term_x(ph - 3, h);
                // row index p (F1) or r (F2); column (q, r) or (p, q)
                const int sr = S(rtR(s, f1 ? 0 : 2)), s1 = S(rtR(s, f1 ? 1 : 0)), s2 = S(rtR(s, f1 ? 2 : 1));
                const bool set = fresh && ph == 0 && h == 0;
                if (mine) {
                    constexpr int MH = (MT + 1) / 2;           // row tiles of a term
                    const int m0 = h * (MT / 2);               // its first tile
                    const int p0 = 8 * m0 + g - h * HR;        // row of the first tile
                    const bool lo = MT % 2 == 0 || h == 0 || g >= 4, hi = p0 + 8 * (MH - 1) < o;
                    double *wr = W + p0 * sr;
#pragma unroll
                    for (int t = 0; t < NT; ++t)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int col = n0 + 8 * t + 2 * c4 + q, i1 = divo(col), i2 = col - i1 * o;
                            if (tail && col >= oo) continue;
                            double *d = wr + i1 * s1 + i2 * s2;
                            double x[MH];
#pragma unroll
                            for (int m = 0; m < MH; ++m)
                                x[m] = !set && (m > 0 || lo) && (m < MH - 1 || hi) ? d[m * 8 * sr] : 0.0;
#pragma unroll
                            for (int m = 0; m < MH; ++m)
                                if ((m > 0 || lo) && (m < MH - 1 || hi))
                                    d[m * 8 * sr] = fma(sgn, acc[h * (MT / 2) + m][t][q], x[m]);
                        }
                }
                if (h == 0) __syncthreads();
            }
        }
        __syncthreads();   // W complete, staging free
    }

    // ---- V-term tiles of the six terms
    if (MODE == M_LNO_FWD) {
        // the W cube to slot 0
        for (int i = tid; i < (int)o3; i += nthr) {
            const int ij = divo(i), k = i - ij * o, ii = divo(ij), j = ij - ii * o;
            Sj[i] = W[ii * si + j * sj + k];
        }
    }
    {
        constexpr bool need_t2 = MODE == M_VJP || MODE == M_LNO_BWD;
        for (int s = 0; s < 6; ++s) {
            int x, y, z;
            xyz(s, x, y, z);
            const double *sv = e.vvop + ((long long)x * v + y) * o * n, *st = e.t2T + ((long long)y * v + x) * oo;
            for (int pq = tid; pq < oo; pq += nthr) {
                const int p = divo(pq), q = pq - p * o, d = s * tsz + p * tl + q;
                cp_async8(VA + d, sv + p * n + q, true);
                if (need_t2 || with_fvo) cp_async8(VB + d, st + pq, true);
            }
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
    }

    // ---- orbit epilogue (ccsd_t_vjp.c:9-117 per element; lno_ccsd_t.c:6-29)
    const double fac = job_fac(a, jb, c), eb = e.et_bar;
    const double eabc = e.mo_energy[o + a] + e.mo_energy[o + jb] + e.mo_energy[o + c];
    KSum eacc;
    double vir = 0.0;
    for (int t = tid; t < e.n_orb; t += nthr) {
        const int pk = __ldg(e.orbits + t);
        const int ijk[3] = {pk & 255, (pk >> 8) & 255, (pk >> 16) & 255};
        int pos[6];
        bool first[6];
#pragma unroll
        for (int s = 0; s < 6; ++s) {
            pos[s] = ijk[kR(s, 0)] * si + ijk[kR(s, 1)] * sj + ijk[kR(s, 2)];
            bool f = true;
#pragma unroll
            for (int u = 0; u < s; ++u) f = f && pos[u] != pos[s];
            first[s] = f;
        }
        const double rden = 1.0 / (eocc[ijk[0]] + eocc[ijk[1]] + eocc[ijk[2]] - eabc);
        double yb[6], wb[6], tmp;
        if (MODE == M_LNO_BWD) {
            double zb[6], aq = 0.0;
#pragma unroll
            for (int s = 0; s < 6; ++s) {
                const long long gp = ((long long)ijk[kR(s, 0)] * o + ijk[kR(s, 1)]) * o + ijk[kR(s, 2)];
                const double q = Sj[o3 + gp], Ax = Sj[2 * o3 + gp] + Sj[4 * o3 + gp], Bx = Sj[3 * o3 + gp] + Sj[5 * o3 + gp];
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
            for (int s = 0; s < 6; ++s) w6[s] = W[pos[s]];
            {
                // V[s] = sum over terms of A_t[P,Q] u_z(t)[R] at the slot's rearranged position
                double u[3][3];
#pragma unroll
                for (int w = 0; w < 3; ++w)
#pragma unroll
                    for (int m = 0; m < 3; ++m) u[w][m] = U[w * o + ijk[m]];
#pragma unroll
                for (int s = 0; s < 6; ++s) {
                    double vs = 0.0;
#pragma unroll
                    for (int t6 = 0; t6 < 6; ++t6) {
                        const int cs = kComp(s, t6);
                        vs += VA[t6 * tsz + ijk[kR(cs, 0)] * tl + ijk[kR(cs, 1)]] * u[kR(t6, 2)][kR(cs, 2)];
                    }
                    y6[s] = w6[s] + 0.5 * vs;
                }
                if (with_fvo) {
#pragma unroll
                    for (int w = 0; w < 3; ++w)
#pragma unroll
                        for (int m = 0; m < 3; ++m) u[w][m] = F[w * o + ijk[m]];
#pragma unroll
                    for (int s = 0; s < 6; ++s) {
                        double vs = 0.0;
#pragma unroll
                        for (int t6 = 0; t6 < 6; ++t6) {
                            const int cs = kComp(s, t6);
                            vs += VB[t6 * tsz + ijk[kR(cs, 0)] * tl + ijk[kR(cs, 1)]] * u[kR(t6, 2)][kR(cs, 2)];
                        }
                        y6[s] += 0.5 * vs;
                    }
                }
            }
            r3_orbit<double>(y6, z6);
            const double d3 = fac * rden;
            double wz = 0.0;
#pragma unroll
            for (int s = 0; s < 6; ++s)
                if (first[s]) wz += w6[s] * z6[s];
            eacc.add(wz * d3);
            if (MODE == M_LNO_FWD) {
#pragma unroll
                for (int s = 0; s < 6; ++s) W[pos[s]] = z6[s] * rden;
            }
            if (MODE == M_VJP) {
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
        if (MODE == M_VJP || MODE == M_LNO_BWD) {
            vir += tmp;
            Tm[t] = tmp;
#pragma unroll
            for (int s = 0; s < 6; ++s)
                if (first[s]) {
                    W[pos[s]] = yb[s];
                    Sj[((long long)ijk[kR(s, 0)] * o + ijk[kR(s, 1)]) * o + ijk[kR(s, 2)]] = wb[s];
                }
        }
    }
    // job energy and the virtual mo_energy bar: a fixed shuffle tree per warp, then over the warps
    {
        double vt = vir;
        ksum_tree(eacc, vt);
        if (lane == 0) { wred[0][warp] = eacc.s; wred[1][warp] = eacc.c; wred[2][warp] = vt; }
    }
    __syncthreads();   // wred, Tm, the ybar cube and w-bar are complete
    if (warp == 0) {
        KSum k;
        k.s = lane < nw ? wred[0][lane] : 0.0;
        k.c = lane < nw ? wred[1][lane] : 0.0;
        double vt = lane < nw ? wred[2][lane] : 0.0;
        ksum_tree(k, vt);
        if (lane == 0) {
            const long long amaj = (long long)a * (a + 1) * (a + 2) / 6 + (long long)jb * (jb + 1) / 2 + c;
            if (MODE == M_ENERGY || MODE == M_VJP) e.job_e[amaj] = 2.0 * k.value();
            if (MODE == M_VJP || MODE == M_LNO_BWD) {
                atomicAdd(&e.mo_energy_bar[o + a], vt);
                atomicAdd(&e.mo_energy_bar[o + jb], vt);
                atomicAdd(&e.mo_energy_bar[o + c], vt);
            }
        }
    }
    if (MODE == M_LNO_FWD) {
        for (int i = tid; i < (int)o3; i += nthr) {
            const int ij = divo(i), k = i - ij * o, ii = divo(ij), j = ij - ii * o;
            Sj[o3 + i] = W[ii * si + j * sj + k];
        }
    }
    if (MODE == M_ENERGY || MODE == M_LNO_FWD) return;

    // ---- occupied mo_energy bar: a warp takes pairs i >= j, lane k its orbit
    // (i, j, k); lane x collects index x's sum (o <= 32)
    {
        double mine = 0.0;
        int i = 0, j = warp;   // pair warp, warp + nw, ... in the order (i, j <= i)
        for (;;) {
            while (j > i) { ++i; j -= i; }
            if (i >= o) break;
            const double t = lane <= j ? Tm[i * (i + 1) * (i + 2) / 6 + j * (j + 1) / 2 + lane] : 0.0;
            double s = t;
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            mine += t + (lane == i ? s : 0.0) + (lane == j ? s : 0.0);
            j += nw;
        }
        __syncthreads();   // Tm read by every warp
        Tm[warp * 32 + lane] = mine;
        __syncthreads();
        if (tid < o) {
            double s = 0.0;
            for (int w = 0; w < nw; ++w) s += Tm[w * 32 + tid];
            atomicAdd(&e.mo_energy_bar[tid], -s);
        }
        __syncthreads();
    }
    // ---- VT, pair part: contraction of ybar along r
    for (int s = 0; s < 6; ++s) {
        int x, y, z;
        xyz(s, x, y, z);
        const int zr = rtR(s, 2), st = S(zr), sp = S(rtR(s, 0)), sq = S(rtR(s, 1));
        const double *u = U + zr * o, *f = F + zr * o;
        double *dv = e.vvop_bar + ((long long)x * v + y) * o * n, *dt = e.t2T_bar + ((long long)y * v + x) * oo;
        for (int pq = tid; pq < oo; pq += nthr) {
            const int p = divo(pq), q = pq - p * o;
            const double *yp = W + p * sp + q * sq;
            double su = 0.0, sw = 0.0;
            if (with_fvo) {
                for (int r = 0; r < o; ++r) {
                    const double yv = yp[r * st];
                    su += yv * u[r];
                    sw += yv * f[r];
                }
                atomicAdd(dt + pq, 0.5 * sw);
            } else {
                for (int r = 0; r < o; ++r) su += yp[r * st] * u[r];
            }
            atomicAdd(dv + p * n + q, 0.5 * su);
        }
    }
    // ---- VT, r part: contraction of ybar along (p, q), split over the threads
    {
        const int parts = nthr / o, part = tid / o, r = tid - part * o;
        if (part < parts) {
#pragma unroll
            for (int zi = 0; zi < 3; ++zi) {
                double a1 = 0.0, a2 = 0.0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int s = term_z(zi, h);
                    const int s0 = S(kR(s, 0)), s1 = S(kR(s, 1));
                    const double *yp = W + r * S(kR(s, 2)), *va = VA + s * tsz, *vb = VB + s * tsz;
                    for (int pq = part; pq < oo; pq += parts) {
                        const int p = divo(pq), q = pq - p * o;
                        const double yv = yp[p * s0 + q * s1];
                        a1 += yv * va[p * tl + q];
                        a2 += yv * vb[p * tl + q];
                    }
                }
                Tm[(zi * 2 * parts + part) * o + r] = a1;
                Tm[((zi * 2 + 1) * parts + part) * o + r] = a2;
            }
        }
        __syncthreads();
        for (int i = tid; i < 6 * o; i += nthr) {
            const int w = divo(i), rr = i - w * o, zi = w >> 1;
            double s = 0.0;
            for (int q = 0; q < parts; ++q) s += Tm[(w * parts + q) * o + rr];
            const int z = pick(2 - zi, a, jb, c);
            atomicAdd(((w & 1) ? e.fvo_bar : e.t1T_bar) + z * o + rr, 0.5 * s);
        }
    }
    // ---- w-bar back in the place of ybar (every warp is past its reads: the
    // barrier above follows them), then its copies with j and with i contiguous,
    // [i][k][j] and [j][k][i], so that the t2-bar GEMM reads every term along r
    for (int i = tid; i < (int)o3; i += nthr) {
        const int ij = divo(i), k = i - ij * o, ii = divo(ij), j = ij - ii * o;
        W[ii * si + j * sj + k] = Sj[i];
    }
    __syncthreads();
    for (int i = tid; i < (int)o3; i += nthr) {
        const int xy = divo(i), z = i - xy * o, x = divo(xy), y = xy - x * o;
        Sj[o3 + i] = W[x * si + z * sj + y];
        Sj[2 * o3 + i] = W[z * si + x * sj + y];
    }

    // A operand of VB and OB2, straight from the cube: row tile m of term h holds
    // rows h HR + p; the address of (row, k) is its row part plus the k part of its
    // term, stepped along k (k = 4 ks + c4 is a pair (k1, k2 < o) of the cube's axes)
    struct KStep {
        int k2, f0, f1;            // k2 and both terms' k parts
        int d0, d1, w0, w1;        // steps of 4 along k2, and at a wrap to the next k1
        __device__ __forceinline__ void init(int k, int k1, int o, int a0, int b0, int a1, int b1) {
            k2 = k - k1 * o;
            f0 = k1 * a0 + k2 * b0;
            f1 = k1 * a1 + k2 * b1;
            d0 = 4 * b0; d1 = 4 * b1;
            w0 = a0 - o * b0; w1 = a1 - o * b1;
        }
        __device__ __forceinline__ void next(int o) {
            k2 += 4; f0 += d0; f1 += d1;
            while (k2 >= o) { k2 -= o; f0 += w0; f1 += w1; }
        }
    };
    const bool second = MT % 2 == 1 && g >= 4;   // this lane's rows of the middle tile are term 1's
    auto row_parts = [&](int sr0, int sr1, int (&ra)[MT]) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int row = m * 8 + g, p = row < HR ? row : row - HR;
            ra[m] = p < o ? p * (row < HR ? sr0 : sr1) : 0;   // rows past o: any element, not stored
        }
    };
    auto load_a = [&](const KStep &K, const int (&ra)[MT], double (&af)[MT]) {
        const int fm = second ? K.f1 : K.f0;
#pragma unroll
        for (int m = 0; m < MT; ++m)
            af[m] = W[ra[m] + (2 * m + 1 < MT ? K.f0 : (2 * m + 1 == MT ? fm : K.f1))];
    };

    // ---- VB: units (z, column group, K split) over the warps
    {
        const int k4 = (oo + 3) >> 2, units = 3 * A.vb_groups * A.vb_ks;
        for (int un = warp; un < units; un += nw) {
            const int zi = un / (A.vb_groups * A.vb_ks), rem = un - zi * (A.vb_groups * A.vb_ks);
            const int gr = rem / A.vb_ks, sp = rem - gr * A.vb_ks;
            const int ka = k4 * sp / A.vb_ks, kb = k4 * (sp + 1) / A.vb_ks, kf = min(kb, oo >> 2);
            const int s0 = term_z(zi, 0), s1 = term_z(zi, 1);
            const int z = pick(2 - zi, a, jb, c);
            int ra[MT];
            row_parts(S(rtR(s0, 0)), S(rtR(s1, 0)), ra);
            KStep K;
            const int kk = 4 * ka + c4;
            K.init(kk, divo(kk), o, S(rtR(s0, 1)), S(rtR(s0, 2)), S(rtR(s1, 1)), S(rtR(s1, 2)));
            const double *bp[VbNT];
#pragma unroll
            for (int t = 0; t < VbNT; ++t)
                bp[t] = e.t2T + ((long long)z * v + min((gr * VbNT + t) * 8 + g, v - 1)) * oo + kk;
            double acc[MT][VbNT][2];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < VbNT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
            double b[VbNT], af[MT];
            if (ka < kf)
#pragma unroll
                for (int t = 0; t < VbNT; ++t) b[t] = __ldg(bp[t]);
#pragma unroll 4
            for (int ks = ka; ks < kf; ++ks) {
                double nb[VbNT];
#pragma unroll
                for (int t = 0; t < VbNT; ++t) {
                    bp[t] += 4;
                    nb[t] = ks + 1 < kf ? __ldg(bp[t]) : 0.0;
                }
                load_a(K, ra, af);
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < VbNT; ++t) dmma(acc[m][t], af[m], b[t]);
                K.next(o);
#pragma unroll
                for (int t = 0; t < VbNT; ++t) b[t] = nb[t];
            }
            if (kf < kb) {   // the last k-step, part past o^2
                const bool in = c4 < (oo & 3);
                if (!in) K.f0 = K.f1 = 0;
                load_a(K, ra, af);
#pragma unroll
                for (int t = 0; t < VbNT; ++t) b[t] = in ? __ldg(bp[t]) : 0.0;
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < VbNT; ++t) dmma(acc[m][t], in ? af[m] : 0.0, b[t]);
            }
            int x0, y0, zz, x1, y1;
            xyz(s0, x0, y0, zz);
            xyz(s1, x1, y1, zz);
            double *d0 = e.vvop_bar + ((long long)x0 * v + y0) * o * n + o;
            double *d1 = e.vvop_bar + ((long long)x1 * v + y1) * o * n + o;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int row = m * 8 + g, pr = row < HR ? row : row - HR;
                if (pr >= o) continue;
                double *d = (row < HR ? d0 : d1) + (long long)pr * n;
#pragma unroll
                for (int t = 0; t < VbNT; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int f = (gr * VbNT + t) * 8 + 2 * c4 + h;
                        if (f < v) atomicAdd(d + f, acc[m][t][h]);
                    }
            }
        }
    }
    // ---- OB2: units (x, 8 N2 columns l, K split): D[(h,r), l] = sum_pq Wbar_h[pq,r] vooo[x,pq,l]
    {
        constexpr int N2 = MT <= 2 ? 1 : 2;
        const int ln = (o + 8 * N2 - 1) / (8 * N2), k4 = (oo + 3) >> 2, units = 3 * ln * A.ob2_ks;
        for (int un = warp; un < units; un += nw) {
            const int xi = un / (ln * A.ob2_ks), rem = un - xi * (ln * A.ob2_ks);
            const int lt = rem / A.ob2_ks, sp = rem - lt * A.ob2_ks;
            const int ka = k4 * sp / A.ob2_ks, kb = k4 * (sp + 1) / A.ob2_ks, kf = min(kb, oo >> 2);
            const int s0 = 2 * xi, s1 = 2 * xi + 1;
            int x, y0, z0, x1, y1, z1;
            xyz(s0, x, y0, z0);
            xyz(s1, x1, y1, z1);
            int ra[MT];
            row_parts(S(rtR(s0, 2)), S(rtR(s1, 2)), ra);
            KStep K;
            const int kk = 4 * ka + c4;
            K.init(kk, divo(kk), o, S(rtR(s0, 0)), S(rtR(s0, 1)), S(rtR(s1, 0)), S(rtR(s1, 1)));
            const double *bp[N2];
#pragma unroll
            for (int t = 0; t < N2; ++t)
                bp[t] = A.vooo + x * o3 + (long long)kk * o + min((lt * N2 + t) * 8 + g, o - 1);
            double acc[MT][N2][2];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < N2; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
            double b[N2], af[MT];
            if (ka < kf)
#pragma unroll
                for (int t = 0; t < N2; ++t) b[t] = __ldg(bp[t]);
#pragma unroll 2
            for (int ks = ka; ks < kf; ++ks) {
                double nb[N2];
#pragma unroll
                for (int t = 0; t < N2; ++t) {
                    bp[t] += 4 * o;
                    nb[t] = ks + 1 < kf ? __ldg(bp[t]) : 0.0;
                }
                load_a(K, ra, af);
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < N2; ++t) dmma(acc[m][t], af[m], b[t]);
                K.next(o);
#pragma unroll
                for (int t = 0; t < N2; ++t) b[t] = nb[t];
            }
            if (kf < kb) {
                const bool in = c4 < (oo & 3);
                if (!in) K.f0 = K.f1 = 0;
                load_a(K, ra, af);
#pragma unroll
                for (int t = 0; t < N2; ++t) b[t] = in ? __ldg(bp[t]) : 0.0;
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int t = 0; t < N2; ++t) dmma(acc[m][t], in ? af[m] : 0.0, b[t]);
            }
            double *d0 = e.t2T_bar + ((long long)z0 * v + y0) * oo, *d1 = e.t2T_bar + ((long long)z1 * v + y1) * oo;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int row = m * 8 + g, pr = row < HR ? row : row - HR;
                if (pr >= o) continue;
                double *d = (row < HR ? d0 : d1) + pr;
#pragma unroll
                for (int t = 0; t < N2; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int l = (lt * N2 + t) * 8 + 2 * c4 + h;
                        if (l < o) atomicAdd(d + l * o, -acc[m][t][h]);
                    }
            }
        }
    }
    // ---- OB1: units (x, 32 columns pq): D[l, pq] = sum_(h,r) t2T[z_h,y_h,l,r] Wbar_h[pq,r]
    {
        constexpr int ML = (MT + 1) / 2, N1 = 4;
        const int ng = (oo + 8 * N1 - 1) / (8 * N1), units = 3 * ng;
        for (int un = warp; un < units; un += nw) {
            const int xi = un / ng, n0 = (un - xi * ng) * (8 * N1);
            const int x = pick(xi, a, jb, c);
            double acc[ML][N1][2];
#pragma unroll
            for (int m = 0; m < ML; ++m)
#pragma unroll
                for (int t = 0; t < N1; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = term_x(xi, h);
                const double *T = VB + tile_zy(s) * tsz;
                const int sp = S(rtR(s, 0)), sq = S(rtR(s, 1)), sr = S(rtR(s, 2));
                int cb[N1];
#pragma unroll
                for (int t = 0; t < N1; ++t) {
                    const int pq = min(n0 + 8 * t + g, oo - 1), p = divo(pq), q = pq - p * o;
                    cb[t] = p * sp + q * sq;
                }
                for (int k = 0; k < o; k += 4) {
                    const int r = k + c4;
                    const bool in = r < o;
                    double bf[N1];
#pragma unroll
                    for (int t = 0; t < N1; ++t) bf[t] = in ? W[cb[t] + r * sr] : 0.0;
#pragma unroll
                    for (int m = 0; m < ML; ++m) {
                        const int l = m * 8 + g;
                        const double af = in && l < o ? T[l * tl + r] : 0.0;
#pragma unroll
                        for (int t = 0; t < N1; ++t) dmma(acc[m][t], af, bf[t]);
                    }
                }
            }
            double *d = A.vooo_bar + x * o3;
#pragma unroll
            for (int m = 0; m < ML; ++m) {
                const int l = m * 8 + g;
                if (l >= o) continue;
#pragma unroll
                for (int t = 0; t < N1; ++t)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int pq = n0 + 8 * t + 2 * c4 + h;
                        if (pq < oo) atomicAdd(d + (long long)pq * o + l, -acc[m][t][h]);
                    }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// TB: t2T_bar[z,f,qr] += sum_t sum_p vvop[x,y,p,o+f] Wbar_t[p,qr] over the
// wave's terms with that z.  64 (f) x 64 (qr) tiles, 4 warps of 32 x 32, one
// stage = `tps` terms of op rows (o rounded up to the MMA's K); one CTA per tile
// and part of a z's term list (the parts add into t2T_bar).  Each job's w-bar comes as three cubes,
// the contiguous axis that of c, b or a: a term reads the one of its z, where
// its r runs along memory (from one cube, a third of the terms were gathered
// along p and a third along q in 8-byte pieces).  Even sizes copy 16 bytes.
// ---------------------------------------------------------------------------
struct TbArgs {
    const double *vvop, *cubes;
    double *t2T_bar;
    long long stride;
    int o, v, n, op, tps, tiles_n;
    int vec_a, vec_b;     // 16-byte copies of the vvop rows / the cubes
    unsigned magic;
    const int *jobs, *entries, *parts;
};
constexpr int kTbLD = 68, kTbTerms = 128;

__global__ void __launch_bounds__(128, 4) tb_kernel(const TbArgs P) {
    extern __shared__ __align__(16) double tsm[];
    __shared__ int t_xy[kTbTerms], t_js[kTbTerms];
    const int o = P.o, v = P.v, n = P.n, oo = o * o, op = P.op;
    const int rows = op * P.tps, buf = rows * kTbLD;
    double *As = tsm, *Bs = tsm + 2 * buf;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    const int tm = blockIdx.y / P.tiles_n, tn = blockIdx.y - tm * P.tiles_n;
    const int f0 = tm * 64, n0 = tn * 64;
    const int z = P.parts[3 * blockIdx.x], e0 = P.parts[3 * blockIdx.x + 1];
    const int nt = P.parts[3 * blockIdx.x + 2] - e0, nst = (nt + P.tps - 1) / P.tps;
    // this thread's column of the A and B copies and its first row (of every 2, or 4)
    const int ca = P.vec_a ? 2 * (tid & 31) : tid & 63, ra = P.vec_a ? tid >> 5 : tid >> 6, da = P.vec_a ? 4 : 2;
    const int cb = P.vec_b ? 2 * (tid & 31) : tid & 63, rb = P.vec_b ? tid >> 5 : tid >> 6, db = P.vec_b ? 4 : 2;
    const int col = n0 + cb, cq = (int)__umulhi((unsigned)col, P.magic), cr = col - cq * o;
    const bool f_ok = f0 + ca < v, c_ok = col < oo;
    auto load_terms = [&](int base) {
        const int i = base + tid;
        if (tid < kTbTerms && i < nt) {
            const int id = P.entries[e0 + i], jl = id / 6, s = id - 6 * jl;
            int a, b, c;
            unpack_job(P.jobs[jl], a, b, c);
            t_xy[tid] = pick(rtR(s, 0), a, b, c) * v + pick(rtR(s, 1), a, b, c);
            t_js[tid] = jl * 8 + s;
        }
    };
    auto stage = [&](int st) {
        double *a_ = As + (st & 1) * buf + ca, *b_ = Bs + (st & 1) * buf + cb;
        for (int u = 0; u < P.tps; ++u) {
            const int t = st * P.tps + u;
            const bool t_ok = t < nt;
            const int xy = t_ok ? t_xy[t & (kTbTerms - 1)] : 0, js = t_ok ? t_js[t & (kTbTerms - 1)] : 0;
            const double *src = P.vvop + (long long)xy * o * n + o + f0 + ca;
            for (int p = ra; p < op; p += da) {
                const bool ok = t_ok && f_ok && p < o;
                if (P.vec_a) cp_async16z(a_ + (u * op + p) * kTbLD, src + p * n, ok);
                else cp_async8(a_ + (u * op + p) * kTbLD, src + p * n, ok);
            }
            const int s = js & 7, cube = wbar_cube(s);
            const bool first = wbar_first(s);
            const int sp0 = first ? oo : o, sq = first ? o : oo;
            const double *q = P.cubes + (long long)(js >> 3) * P.stride + (long long)cube * oo * o + cq * sq + cr;
            for (int p = rb; p < op; p += db) {
                const bool ok = t_ok && c_ok && p < o;
                if (P.vec_b) cp_async16z(b_ + (u * op + p) * kTbLD, q + p * sp0, ok);
                else cp_async8(b_ + (u * op + p) * kTbLD, q + p * sp0, ok);
            }
        }
        cp_async_commit();
    };
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    load_terms(0);
    __syncthreads();
    stage(0);
    const int per = kTbTerms / P.tps;   // stages per block of term descriptors
    for (int st = 0; st < nst; ++st) {
        cp_async_wait_all();
        __syncthreads();
        if (st + 1 < nst) {
            if ((st + 1) % per == 0) {
                load_terms((st + 1) * P.tps);
                __syncthreads();
            }
            stage(st + 1);
        }
        const double *a_ = As + (st & 1) * buf + wm + g + c4 * kTbLD, *b_ = Bs + (st & 1) * buf + wn + g + c4 * kTbLD;
        for (int k = 0; k < rows; k += 4, a_ += 4 * kTbLD, b_ += 4 * kTbLD) {
            double af[4], bf[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { af[i] = a_[8 * i]; bf[i] = b_[8 * i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
    }
    double *dst = P.t2T_bar + (long long)z * v * oo;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int f = f0 + wm + 8 * i + g;
        if (f >= v) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int cl = n0 + wn + 8 * j + 2 * c4 + h;
                if (cl < oo) atomicAdd(dst + (long long)f * oo + cl, acc[i][j][h]);
            }
    }
}

// Strides (sj, si) of the shared cube: the smallest cost over a few paddings,
// cost = worst bank multiplicity of the fragment patterns (4 rows of one index
// x 4 consecutive of another) over every pair of axes.
static void pick_strides(int o, int &sj, int &si) {
    int best = 1 << 30;
    for (int pj = 0; pj < 4; ++pj)
        for (int pi = 0; pi < 8; ++pi) {
            const int j = o + pj, i = o * j + pi, s[3] = {i, j, 1};
            int cost = 0;
            for (int x = 0; x < 3; ++x)
                for (int y = 0; y < 3; ++y) {
                    if (x == y) continue;
                    int cnt[16] = {}, worst = 0;
                    for (int u = 0; u < 4; ++u)
                        for (int w = 0; w < 4; ++w) worst = std::max(worst, ++cnt[(u * s[x] + w * s[y]) % 16]);
                    cost += worst;
                }
            cost = cost * 64 + pj * 8 + pi;   // least padding among equals
            if (cost < best) { best = cost; sj = j; si = i; }
        }
}

template <int MT, int NT, int MODE, int MAXT, int MINB>
static cudaError_t launch(Args &A, int n_jobs, cudaStream_t st) {
    const int o = A.e.o, oo = o * o;
    const int groups = ((oo + 7) / 8 + NT - 1) / NT;
    A.passes = (groups + MAXT / 32 - 1) / (MAXT / 32);
    const int nw = (groups + A.passes - 1) / A.passes;
    pick_strides(o, A.sj, A.si);
    A.cube_sz = (o * A.si + 1) & ~1;
    const int tiles_sz = 12 * o * tile_ld(o);
    A.tmp_sz = (MODE == M_VJP || MODE == M_LNO_BWD) ? std::max(A.e.n_orb, 6 * nw * 32) : 0;
    // the longest K chunk that still lets MINB CTAs share the SM (fewer, longer
    // chunks: fewer barriers), split evenly over the virtuals
    const int room = (228 * 1024 / MINB - 2048) / 8 - A.cube_sz - A.tmp_sz - 7 * o;
    const int cap = std::max(32, std::min(128, (room / (2 * 8 * MT) - 4) / 16 * 16));
    A.nch = (A.e.v + cap - 1) / cap;
    A.kc = std::max(32, ((A.e.v + A.nch - 1) / A.nch + 15) / 16 * 16);
    A.stage_sz = std::max(2 * 8 * MT * (A.kc + 4), tiles_sz);
    A.magic = (unsigned)(((1ull << 32) + o - 1) / o);
    A.vb_groups = (A.e.v + 8 * VbNT - 1) / (8 * VbNT);
    // K splits: units to fill the rounds of warps to 70% (shorter units pay more
    // for their start and their atomics than a fuller last round gains)
    auto splits = [&](int units, int kmax) {
        int ks = 1;
        while (ks < 8 && 2 * ks <= kmax) {
            const int u = units * ks, rounds = (u + nw - 1) / nw;
            if (u * 10 >= rounds * nw * 7) break;
            ks *= 2;
        }
        return ks;
    };
    A.vb_ks = splits(3 * A.vb_groups, oo / 32);
    constexpr int N2 = MT <= 2 ? 1 : 2;   // job_kernel's OB2 tile
    A.ob2_ks = splits(3 * ((o + 8 * N2 - 1) / (8 * N2)), oo / 32);
    const size_t smem = sizeof(double) * (size_t)(A.cube_sz + A.stage_sz + A.tmp_sz + 7 * o);
    const void *fn = reinterpret_cast<const void *>(job_kernel<MT, NT, MODE, MAXT, MINB>);
    cudaError_t ce = smem_optin(fn, (int)smem);
    if (ce != cudaSuccess) return ce;
    job_kernel<MT, NT, MODE, MAXT, MINB><<<n_jobs, nw * 32, smem, st>>>(A);
    return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_o(Args &A, int n_jobs, cudaStream_t st) {
    switch ((A.e.o + 3) / 4) {   // tiles of 8 over the 2 o rows
    case 1: return launch<1, 2, MODE, 32, 16>(A, n_jobs, st);
    case 2: return launch<2, 2, MODE, 128, 5>(A, n_jobs, st);
    case 3: return launch<3, 3, MODE, 192, 3>(A, n_jobs, st);
    case 4: return launch<4, 4, MODE, 256, 2>(A, n_jobs, st);
    // nocc = 20 with the gradients' partials leaves room for one CTA per SM
    case 5: return A.e.o == 20 && MODE != M_ENERGY ? launch<5, 2, MODE, 512, 1>(A, n_jobs, st)
                                                   : launch<5, 3, MODE, 256, 2>(A, n_jobs, st);
    case 6: return launch<6, 3, MODE, 512, 1>(A, n_jobs, st);
    default: return cudaErrorInvalidValue;
    }
}

static Args make_args(const int *jobs, const EpiArgs &e, const double *vooo, double *vooo_bar, double *cubes,
                      long long stride) {
    Args A{};
    A.e = e;
    A.jobs = jobs;
    A.vooo = vooo;
    A.vooo_bar = vooo_bar;
    A.cubes = cubes;
    A.stride = stride;
    return A;
}

}  // namespace cube

cudaError_t cube_energy(const int *jobs, int n_jobs, const EpiArgs &e, const double *vooo, cudaStream_t st) {
    if (n_jobs <= 0) return cudaSuccess;
    cube::Args A = cube::make_args(jobs, e, vooo, nullptr, nullptr, 0);
    return cube::launch_o<cube::M_ENERGY>(A, n_jobs, st);
}

cudaError_t cube_vjp(const WaveView &w, const EpiArgs &e, const double *vooo, double *vooo_bar, double *cubes,
                     cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    cube::Args A = cube::make_args(w.jobs, e, vooo, vooo_bar, cubes, 3LL * e.o * e.o * e.o);
    return cube::launch_o<cube::M_VJP>(A, w.n_jobs, st);
}

cudaError_t cube_lno_forward(const WaveView &w, const EpiArgs &e, const double *vooo, double *slots,
                             cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    cube::Args A = cube::make_args(w.jobs, e, vooo, nullptr, slots, (long long)kSlots * e.o * e.o * e.o);
    return cube::launch_o<cube::M_LNO_FWD>(A, w.n_jobs, st);
}

cudaError_t cube_lno_backward(const WaveView &w, const EpiArgs &e, const double *vooo, double *vooo_bar,
                              double *slots, cudaStream_t st) {
    if (w.n_jobs <= 0) return cudaSuccess;
    cube::Args A = cube::make_args(w.jobs, e, vooo, vooo_bar, slots, (long long)kSlots * e.o * e.o * e.o);
    return cube::launch_o<cube::M_LNO_BWD>(A, w.n_jobs, st);
}

cudaError_t cube_tb(const WaveView &w, const EpiArgs &e, const double *cubes, long long stride, cudaStream_t st) {
    if (w.n_zparts <= 0) return cudaSuccess;
    cube::TbArgs P{};
    P.vvop = e.vvop;
    P.cubes = cubes;
    P.t2T_bar = e.t2T_bar;
    P.stride = stride;
    P.o = e.o; P.v = e.v; P.n = e.n;
    P.op = (e.o + 3) & ~3;
    P.tps = std::max(1, 16 / P.op);
    if (P.tps == 3) P.tps = 2;   // a power of two divides the descriptor block
    P.tiles_n = (e.o * e.o + 63) / 64;
    P.magic = (unsigned)(((1ull << 32) + e.o - 1) / e.o);
    P.vec_a = e.o % 2 == 0 && e.n % 2 == 0 && reinterpret_cast<uintptr_t>(e.vvop) % 16 == 0;
    P.vec_b = e.o % 2 == 0 && stride % 2 == 0 && reinterpret_cast<uintptr_t>(cubes) % 16 == 0;
    P.jobs = w.jobs;
    P.entries = w.tb_entries;
    P.parts = w.zparts;
    const int tiles = ((e.v + 63) / 64) * P.tiles_n;
    const size_t smem = sizeof(double) * 4 * (size_t)P.op * P.tps * cube::kTbLD;
    cudaError_t ce = smem_optin(reinterpret_cast<const void *>(cube::tb_kernel), (int)smem);
    if (ce != cudaSuccess) return ce;
    cube::tb_kernel<<<dim3(w.n_zparts, tiles), 128, smem, st>>>(P);
    return cudaGetLastError();
}

}  // namespace ctb
