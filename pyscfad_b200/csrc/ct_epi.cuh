// Device helpers shared by the orbit epilogue kernels (float64 path in
// ct_fp64.cu, pipelined float path in ct_epi_f32.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "ct_common.cuh"

namespace ctb {

// 16-byte asynchronous global -> shared copy (no register round-trip)
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// W-bar as staged by the mixed path's epilogue: WB 1 = float rounded to the
// nearest tf32 (it feeds tf32 tensor-core GEMMs, whose MMA would otherwise
// truncate); 0 = float kept whole (BF16x3 splits it on the way out).
template <int WB> __device__ __forceinline__ float wbar_store(float x) {
    if (WB == 1) {
        uint32_t r;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
        return __uint_as_float(r);
    }
    return x;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// r3 over the six slots of an element orbit, y[s] = sum_t kR3C(t) x[kComp(s,t)]
// (weights 4 for the identity, -2 for the transpositions, 1 for the 3-cycles;
// add_and_permute, ccsd_t.c:98-119).  Row s of kComp is a permutation of the
// six slots, so with S = sum(x) this is 6 x[s] + 3 (x[kComp(s,3)] +
// x[kComp(s,4)]) - 2 S: three operations per slot after the shared sum instead
// of six multiply-adds.
template <typename AT> __device__ __forceinline__ void r3_orbit(const AT (&x)[6], AT (&y)[6]) {
    const AT tot = ((x[0] + x[1]) + (x[2] + x[3])) + (x[4] + x[5]);
    const AT m2s = (AT)-2 * tot;
#pragma unroll
    for (int s = 0; s < 6; ++s) y[s] = (AT)6 * x[s] + ((AT)3 * (x[kComp(s, 3)] + x[kComp(s, 4)]) + m2s);
}

// Neumaier pairs and a plain partial summed down a warp in a fixed order; valid in lane 0
__device__ __forceinline__ void ksum_tree(KSum &k, double &v) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        const double s2 = __shfl_down_sync(0xffffffffu, k.s, m), c2 = __shfl_down_sync(0xffffffffu, k.c, m);
        v += __shfl_down_sync(0xffffffffu, v, m);
        k.c += c2;
        k.add(s2);
    }
}

// One element orbit {perm(i,j,k)} of a staged block-orbit (I,J,K) = (BI,BJ,BK)
// of the mixed path: W, V, r3, the denominator, the job-energy contribution and
// (vjp) the backward quantities, all in registers (ccsd_t_vjp.c:9-117 per
// element; lno_ccsd_t.c:6-29).  Staged tiles: Gs[sigma][buffer d] blocks of BLK
// elements with u-stride TP, V tiles VA/VB[sigma][slot][T^2], t1/fvo rows
// Us/Ws[3][64] of a, b, c.  Writes W-bar in place into Gs, ybar to the staging
// buffer Yg laid out like the G tiles (the caller flushes both) and this
// element's mo_energy-bar partial to tmp.  W, V, r3 and the bars are float; the
// denominator, the energy terms and the mo_energy-bar partials are float64.
template <int T, int TP, int BLK, int WB>
__device__ __forceinline__ void orbit_element(const int (&loc)[3], int BI, int BJ, int BK, const int (&dmap)[6],
                                              float *Gs, const float *VA, const float *VB, const float *Us,
                                              const float *Ws, const double *eocc, float *Yg, int o, double fac,
                                              double eabc, double eb, bool vjp, KSum &eacc, double &vir_acc,
                                              bool with_fvo, double &tmp, bool lno) {
    constexpr int T2 = T * T;
    tmp = 0.0;
    const int ijk[3] = {BI * T + loc[0], BJ * T + loc[1], BK * T + loc[2]};
    if (ijk[0] >= o || ijk[1] >= o || ijk[2] >= o) return;
    if ((BI == BJ && loc[0] < loc[1]) || (BJ == BK && loc[1] < loc[2])) return;
    int off[6], vp[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        off[s] = dmap[s] * BLK + loc[kR(s, 0)] * TP + loc[kR(s, 1)] * T + loc[kR(s, 2)];
        vp[s] = loc[kR(s, 0)] * T + loc[kR(s, 1)];
    }
    bool first[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        bool f = true;
#pragma unroll
        for (int t = 0; t < s; ++t) f = f && (off[t] != off[s]);
        first[s] = f;
    }
    // t1 and fvo of the three virtuals at the three occupieds: nine values each
    float u[3][3], fv[3][3];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            u[m][q] = Us[m * 64 + ijk[q]];
            fv[m][q] = with_fvo ? Ws[m * 64 + ijk[q]] : 0.f;
        }
    float W[6], Y[6], Z[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        float ws = 0, vs = 0;
#pragma unroll
        for (int sg = 0; sg < 6; ++sg) {
            const int cs = kComp(s, sg);
            ws += Gs[sg * 6 * BLK + off[cs]];
            const int vi = (sg * 6 + cs) * T2 + vp[cs];
            vs += VA[vi] * u[kR(sg, 2)][kR(cs, 2)];
            if (with_fvo) vs += VB[vi] * fv[kR(sg, 2)][kR(cs, 2)];
        }
        W[s] = ws;
        Y[s] = ws + 0.5f * vs;
    }
    r3_orbit<float>(Y, Z);
    // one reciprocal per element: d3 = fac / D; the orbit's distinct W.Z
    // products share d3, so they are summed before the compensated add, and
    // the mo_energy-bar partial eb d3^2 / fac = eb fac / D^2 reuses 1/D
    const double rden = 1.0 / (eocc[ijk[0]] + eocc[ijk[1]] + eocc[ijk[2]] - eabc);
    const double d3 = fac * rden;
    double wz = 0.0;
#pragma unroll
    for (int s = 0; s < 6; ++s)
        if (first[s]) wz += (double)W[s] * (double)Z[s];
    eacc.add(wz * d3);
    if (lno) {
        // LNO energy (no VJP): the W cube into slot 0 and z/D into slot 1 of
        // the staged tiles, at the orbit's own positions (read above by this
        // thread only); the projection follows in a separate kernel
#pragma unroll
        for (int s = 0; s < 6; ++s) {
            Gs[off[s]] = W[s];
            Gs[6 * BLK + off[s]] = (float)((double)Z[s] * rden);
        }
        return;
    }
    if (vjp) {
        const float ebd3 = (float)(eb * d3);
        float zb[6], wb[6];
        tmp = eb * d3 * rden * wz;
#pragma unroll
        for (int s = 0; s < 6; ++s) {
            zb[s] = ebd3 * W[s];
            wb[s] = ebd3 * Z[s];
        }
        float yb[6];
        r3_orbit<float>(zb, yb);
#pragma unroll
        for (int s = 0; s < 6; ++s) wb[s] = wbar_store<WB>(wb[s] + yb[s]);
        vir_acc += tmp;
#pragma unroll
        for (int sg = 0; sg < 6; ++sg)
#pragma unroll
            for (int s = 0; s < 6; ++s) Gs[sg * 6 * BLK + off[s]] = wb[kComp(s, kInv(sg))];
#pragma unroll
        for (int s = 0; s < 6; ++s)
            if (first[s]) Yg[off[s]] = yb[s];
    }
}

// LNO backward for one element orbit (lno_ccsd_t_vjp.c:73-140 on the sorted
// job's cubes).  Tile groups 0-4 hold q = z/D and the two parts (axes 1-2,
// axis 0) of A = sum_t wt_t M_t(w) and B = sum_t wt_t M_t^T(q) at the orbit's
// slot positions (groups 1 + 3 and 2 + 4); the energy is
// sum A q, so z_bar = eb A / D, w_bar = eb B + r3(z_bar), v_bar = r3(z_bar)
// (the canonical chain of orbit_element with those two products replaced)
// and the mo_energy-bar partial is eb A q / D.  W-bar goes in place into
// groups 0-5, ybar to its staging buffer.  Arithmetic in float64 (there is no V
// term to form here).
template <int T, int TP, int BLK, int WB>
__device__ __forceinline__ void orbit_lno_bar(const int (&loc)[3], int BI, int BJ, int BK, const int (&dmap)[6],
                                              float *Gs, const double *eocc, float *Yg, int o, double eabc, double eb,
                                              double &vir_acc, double &tmp) {
    tmp = 0.0;
    const int ijk[3] = {BI * T + loc[0], BJ * T + loc[1], BK * T + loc[2]};
    if (ijk[0] >= o || ijk[1] >= o || ijk[2] >= o) return;
    if ((BI == BJ && loc[0] < loc[1]) || (BJ == BK && loc[1] < loc[2])) return;
    int off[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) off[s] = dmap[s] * BLK + loc[kR(s, 0)] * TP + loc[kR(s, 1)] * T + loc[kR(s, 2)];
    bool first[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        bool f = true;
#pragma unroll
        for (int t = 0; t < s; ++t) f = f && (off[t] != off[s]);
        first[s] = f;
    }
    const double rden = 1.0 / (eocc[ijk[0]] + eocc[ijk[1]] + eocc[ijk[2]] - eabc);
    double zb[6], wb[6], aq = 0.0;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        const double q = Gs[off[s]];
        const double A = (double)Gs[6 * BLK + off[s]] + (double)Gs[18 * BLK + off[s]];
        const double B = (double)Gs[12 * BLK + off[s]] + (double)Gs[24 * BLK + off[s]];
        zb[s] = eb * A * rden;
        wb[s] = eb * B;
        if (first[s]) aq += A * q;
    }
    tmp = eb * rden * aq;
    double yb[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < 6; ++u) t += kR3C(u) * zb[kComp(s, u)];
        yb[s] = t;
        wb[s] += t;
    }
    vir_acc += tmp;
    float w[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) w[s] = wbar_store<WB>((float)wb[s]);
#pragma unroll
    for (int sg = 0; sg < 6; ++sg)
#pragma unroll
        for (int s = 0; s < 6; ++s) Gs[sg * 6 * BLK + off[s]] = w[kComp(s, kInv(sg))];
#pragma unroll
    for (int s = 0; s < 6; ++s)
        if (first[s]) Yg[off[s]] = (float)yb[s];
}

}  // namespace ctb
