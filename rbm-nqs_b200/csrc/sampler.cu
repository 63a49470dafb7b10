// sampler.cu -- fused Metropolis sweep -> E_loc -> O_k kernel for the complex
// RBM (rbm_base / rbm_symmetry), plus the batched evaluation kernels used by
// the parity entry points.
//
// Layout: one warp owns one Markov chain.  The chain's theta table
// (theta[k + nh*s], T = nh*S entries, machine/rbm_symmetry.cpp:48-61) is
// spread over the 32 lanes, E = ceil(T/32) entries per lane, kept in
// registers; a flip of site f adds -2 sigma_f W[P_s(f), k] to entry (k, s)
// (rbm_symmetry.cpp:63-95), gathered from the FP32 copy of W in shared
// memory through the per-site permutation table.  psi ratios reduce over the
// lanes with warp shuffles; every lane holds the same configuration bits and
// takes the same accept/reject branch.  theta is recomputed in FP64 from the
// configuration after every sweep (mixed-precision scheme), so FP32
// drift never outlives one sweep.  With the Pfaffian factor (sites <= 32) the
// warp also holds X^{-1} in shared memory (pfaffian.cuh).  FP64 sweeps, and FP32
// sweeps of 16 entries per lane in launches of enough chains and sweeps
// (screen_pays), screen the proposals by products (sampler_screen.cuh), whose drift
// the screen's margin allows for.
#include <algorithm>
#include <map>
#include <mutex>

#include "common.cuh"
#include "sampler.cuh"
#include "sweep_common.cuh"

namespace rbmnqs {

template <typename R> struct Wsel;
template <> struct Wsel<float> {
    static __device__ __forceinline__ const float2* get(const MachineDev& m, const float2* sW) { return sW; }
};
template <> struct Wsel<double> {
    static __device__ __forceinline__ const double2* get(const MachineDev& m, const float2*) { return m.W64; }
};

// Lane `lane` owns theta entries t = lane + 32 e (e < E), t = k + nh*s.
__device__ __forceinline__ bool slot_valid(int lane, int e, int T) { return lane + 32 * e < T; }

template <typename R>
__device__ __forceinline__ int urow(const MachineDev& m, const uint8_t* sPerm, int f, int s) {
    return m.symmetric ? (int)sPerm[f * m.S + s] : f;
}

__device__ __forceinline__ int smem_bit(const uint32_t* wsp, int i) { return (wsp[i >> 5] >> (i & 31)) & 1; }

// theta = b + W^T(P_s sigma) in FP64, rounded to R (rbm_base.cpp:161-172).
template <int E, typename R>
__device__ __forceinline__ void theta_fp64(const MachineDev& m, const double2* W64, const uint8_t* sPerm, int lane,
                           const uint32_t sp[4], C2<R> th[E]) {
    double2 acc[E];
    int kk[E], ss[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int t = slot_valid(lane, e, m.T) ? lane + 32 * e : 0;
        kk[e] = t % m.nh;
        ss[e] = t / m.nh;
        acc[e] = slot_valid(lane, e, m.T) ? m.hb[kk[e]] : make_double2(0, 0);
    }
    for (int i = 0; i < m.n; i++) {
        const double sg = spin_bit(sp, i) ? -1.0 : 1.0;
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (!slot_valid(lane, e, m.T)) continue;
            const double2 w = W64[urow<R>(m, sPerm, i, ss[e]) * m.nh + kk[e]];
            acc[e].x = fma(sg, w.x, acc[e].x);
            acc[e].y = fma(sg, w.y, acc[e].y);
        }
    }
#pragma unroll
    for (int e = 0; e < E; e++) th[e] = mk<R>((R)acc[e].x, (R)acc[e].y);
}

// Bias part of log(psi'/psi): sum_f -2 sigma_f v[f mod n_vb]
// (rbm_base.cpp:306-318), for configuration bits in registers or in the
// warp's scratch.
__device__ __forceinline__ double2 bias_delta(const MachineDev& m, const uint32_t sp[4], const int* fl, int nf) {
    double2 b = make_double2(0, 0);
    for (int q = 0; q < nf; q++) {
        const double sg = spin_bit(sp, fl[q]) ? -1.0 : 1.0;
        const double2 v = m.vb[fl[q] % m.n_vb];
        b.x -= 2.0 * sg * v.x;
        b.y -= 2.0 * sg * v.y;
    }
    return b;
}

// Visible-bias index f mod n_vb of site 0 <= f < n, without an integer
// division for one bias per site (n_vb = n) and for a power-of-two basis
// (one bias for all sites, one per sublattice, ...).
__device__ __forceinline__ int vb_index(int f, int n_vb, int n) {
    return n_vb == n ? f : ((n_vb & (n_vb - 1)) == 0 ? (f & (n_vb - 1)) : f % n_vb);
}

// The bias sizes passed in registers (the machine descriptor is in global
// memory and the term loop of evaluate() calls this once per term).
__device__ __forceinline__ double2 bias_delta_smem(const double2* vb, int n_vb, int n, const uint32_t* wsp,
                                                   const int* fl, int nf) {
    double2 b = make_double2(0, 0);
    for (int q = 0; q < nf; q++) {
        const double sg = smem_bit(wsp, fl[q]) ? -1.0 : 1.0;
        const double2 v = vb[vb_index(fl[q], n_vb, n)];
        b.x -= 2.0 * sg * v.x;
        b.y -= 2.0 * sg * v.y;
    }
    return b;
}
__device__ __forceinline__ double2 bias_delta_smem(const MachineDev& m, const uint32_t* wsp, const int* fl, int nf) {
    return bias_delta_smem(m.vb, m.n_vb, m.n, wsp, fl, nf);
}

// psi(sigma with flips)/psi(sigma) for the RBM part from the warp's theta
// (wth) and the per-entry ln cosh cache (cre, cu) of the current theta, all
// in the warp's shared scratch.  Returns the real log-magnitude sum (without
// bias) and the phase product.
// Entry e of this lane is theta[k + nh s] with t = lane + 32 e; the pair
// (k, s) is packed as (s << 16) | k once per sample (no division per term).
template <int E>
__device__ __forceinline__ void entry_index(const MachineDev& m, int lane, uint32_t (&ks)[E]) {
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int t = lane + 32 * e;
        ks[e] = t < m.T ? ((uint32_t)(t / m.nh) << 16) | (uint32_t)(t % m.nh) : 0u;
    }
}

// The machine sizes the ratio loop reads, held in registers (the machine
// descriptor itself is in global memory).
struct RatioDims {
    int T, nh, S, symmetric;
};
__device__ __forceinline__ RatioDims ratio_dims(const MachineDev& m) { return RatioDims{m.T, m.nh, m.S, m.symmetric}; }

// NF > 0: a compile-time flip count (the flips and their signs stay in
// registers); NF = 0: nf flips at run time.
// WS (FP32): W and the symmetry table are in shared memory, read by shared
// addresses.
// FP32 (R = float): the lane's entries go through lnc_lane and the cache is
// the lane aggregate (cl.re, cl.u) of the current theta; FP64: one ln cosh
// per entry against the per-entry cache (cre, cu).
template <typename R> struct LaneCache {
    R re;
    C2<R> u;
};
__device__ __forceinline__ int lane_entries(int lane, int T, int E) {
    const int v = (T - lane + 31) >> 5;
    return v < 0 ? 0 : (v > E ? E : v);
}
template <int E>
__device__ __forceinline__ LaneCache<float> lane_cache(const float2* wth, int lane, int T) {
    float2 x[E];
#pragma unroll
    for (int e = 0; e < E; e++) x[e] = slot_valid(lane, e, T) ? wth[lane + 32 * e] : make_float2(0.f, 0.f);
    LaneCache<float> c;
    lnc_lane<E>(x, lane_entries(lane, T, E), c.re, c.u);
    return c;
}

template <int E, typename R, int NF = 0, bool WS = false>
__device__ __forceinline__ void ratio_terms(const RatioDims m, const uint8_t* sPerm, const C2<R>* W,
                                            const C2<R>* wth, const uint32_t* wsp, const int* fl, int nf_,
                                            const R* cre, const C2<R>* cu, const LaneCache<R> cl, int lane,
                                            R& dre, C2<R>& ph, const uint32_t (&ks)[E]) {
    const int nf = NF > 0 ? NF : nf_;
    R sgn2[NF > 0 ? NF : 6];
#pragma unroll
    for (int q = 0; q < (NF > 0 ? NF : 6); q++)
        if (q < nf) sgn2[q] = smem_bit(wsp, fl[q]) ? (R)2 : (R)-2;  // -2 sigma_f
    dre = 0;
    ph = mk<R>(1, 0);
    C2<R> xs[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        xs[e] = mk<R>(0, 0);
        if (!slot_valid(lane, e, m.T)) continue;
        const int t = lane + 32 * e, k = ks[e] & 0xffffu, s = ks[e] >> 16;
        C2<R> x = wth[t];
#pragma unroll
        for (int q = 0; q < (NF > 0 ? NF : 6); q++) {
            if (q >= nf) break;
            C2<R> u;
            if constexpr (WS && sizeof(R) == 4) {
                const int row = m.symmetric ? (int)lds_u8(smem_addr(sPerm) + (uint32_t)(fl[q] * m.S + s)) : fl[q];
                const float2 v = lds_f2(smem_addr(W) + 8u * (uint32_t)(row * m.nh + k));
                u = mk<R>(v.x, v.y);
            } else {
                const int row = m.symmetric ? (int)sPerm[fl[q] * m.S + s] : fl[q];
                u = W[row * m.nh + k];
            }
            x.x = fma(sgn2[q], u.x, x.x);
            x.y = fma(sgn2[q], u.y, x.y);
        }
        if constexpr (sizeof(R) == 4) {
            xs[e] = x;
        } else {
            R re, ux, uy;
            lnc_full<R>(x.x, x.y, re, ux, uy);
            dre += re - cre[t];
            ph = cmul(ph, cmulc(mk<R>(ux, uy), cu[t]));
        }
    }
    if constexpr (sizeof(R) == 4) {
        float re;
        float2 u;
        lnc_lane<E>(xs, lane_entries(lane, m.T, E), re, u);
        dre = re - cl.re;
        ph = cmulc(u, cl.u);
    }
    dre = warp_sum(dre);
    ph = warp_cprod(ph);
}

// E_loc and O_k of the configuration in the warp's scratch (wsp bits, wth
// theta): local_op.cpp:31-60, rbm_base.cpp:194-217, rbm_symmetry.cpp:97-130.
// Pfaffian factor (PF): term ratios multiply by the rank-2m ratio from the
// warp's X^{-1} in shared memory (pA, leading dimension kPfLd), the O_k of
// the pair parameters are gathered from it.
template <int NF>
__device__ __forceinline__ double2 pf_ratio_smem(const PfDev& p, uint32_t bits, const int* fl, int lane, PfStage& st,
                                                 const double2* pA) {
    double2 ib[2 * kPfMaxFlips];
    auto xi = [&](int t) { return pA[lane * kPfLd + t]; };
    auto xcol = [&](int f) { return pA[lane * kPfLd + f]; };
    return pf_ratio<NF>(p, bits, fl, lane, st, xi, xcol, ib);
}

__device__ __noinline__ double2 pf_ratio_any(const PfDev& p, uint32_t bits, const int* fl, int nf, int lane,
                                             PfStage& st, const double2* pA) {
    switch (nf) {
        case 1: return pf_ratio_smem<1>(p, bits, fl, lane, st, pA);
        case 2: return pf_ratio_smem<2>(p, bits, fl, lane, st, pA);
        case 3: return pf_ratio_smem<3>(p, bits, fl, lane, st, pA);
        case 4: return pf_ratio_smem<4>(p, bits, fl, lane, st, pA);
        default: return make_double2(nan(""), nan(""));  // more flips than the staging holds
    }
}

template <int E, typename R, bool PF, bool WS>
__device__ __forceinline__ void evaluate(const MachineDev* __restrict__ mp, const HamDev H,
                                      const uint8_t* sPerm, const uint8_t* sInv, const C2<R>* W, const C2<R>* wth,
                                      const uint32_t* wsp, R* cre, C2<R>* cu, const C2<R>* tn, int lane,
                                      double2* Eout, C2<R>* Orow, PfStage* pst, const double2* pA) {
    const MachineDev& m = *mp;
    const RatioDims rd = ratio_dims(m);
    uint32_t ks[E];
    entry_index<E>(m, lane, ks);
    // ln cosh cache of the current theta
    LaneCache<R> cl{};
    if constexpr (sizeof(R) == 4) {
        cl = lane_cache<E>(wth, lane, m.T);
    } else {
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (!slot_valid(lane, e, m.T)) continue;
            const int t = lane + 32 * e;
            R re, ux, uy;
            lnc_full<R>(wth[t].x, wth[t].y, re, ux, uy);
            cre[t] = re;
            cu[t] = mk<R>(ux, uy);
        }
        __syncwarp();
    }
    if (Eout) {
        double ex = 0, ey = 0;
        const double2* vb = m.vb;
        const int nvb = m.n_vb, nsites = m.n;
        for (int o = 0; o < H.n_ops; o++) {
            const OpDev* op = H.ops + o;
            const int k = op->k;
            int loc = 0;
            for (int i = 0; i < k; i++) loc |= smem_bit(wsp, op->sites[i]) << i;
            const int q0 = H.rowptr[op->rp + loc], q1 = H.rowptr[op->rp + loc + 1];
            for (int q = q0; q < q1; q++) {
                const uint32_t mask = H.ent_mask[q];
                const double2 val = H.ent_val[q];
                if (mask == 0) {
                    ex += val.x;
                    ey += val.y;
                    continue;
                }
                const int nf = __popc(mask);
                int fl[6];
                // one- and two-site flips (every bond operator) with the flips
                // in registers; larger flips with run-time loops
                R dre;
                C2<R> ph;
                if (nf <= 2) {
                    const int i0 = __ffs(mask) - 1;
                    const int i1 = nf == 2 ? __ffs(mask & (mask - 1)) - 1 : i0;
                    fl[0] = op->sites[i0];
                    fl[1] = op->sites[i1];
                    if (nf == 2) {
                        const int f2[2] = {fl[0], fl[1]};
                        ratio_terms<E, R, 2, WS>(rd, sPerm, W, wth, wsp, f2, 2, cre, cu, cl, lane, dre, ph, ks);
                    } else {
                        const int f1[1] = {fl[0]};
                        ratio_terms<E, R, 1, WS>(rd, sPerm, W, wth, wsp, f1, 1, cre, cu, cl, lane, dre, ph, ks);
                    }
                } else {
                    uint32_t mm = mask;
                    for (int j = 0; j < nf; j++) {
                        fl[j] = op->sites[__ffs(mm) - 1];
                        mm &= mm - 1;
                    }
                    ratio_terms<E, R, 0, WS>(rd, sPerm, W, wth, wsp, fl, nf, cre, cu, cl, lane, dre, ph, ks);
                }
                const double2 b = bias_delta_smem(vb, nvb, nsites, wsp, fl, nf);
                double rx, ry;
                const double lm = (double)dre + b.x;  // ln|psi'/psi| of the RBM part
                if (sizeof(R) == 4 && fabs(lm) < 80.0) {
                    // FP32 path: the ratio to FP32 accuracy in FP32 arithmetic
                    // (its inputs carry FP32 rounding already)
                    const float mag = exp_r((float)lm);
                    float sb, cb;
                    sincos_r((float)b.y, &sb, &cb);
                    rx = (double)(mag * ((float)ph.x * cb - (float)ph.y * sb));
                    ry = (double)(mag * ((float)ph.x * sb + (float)ph.y * cb));
                } else {
                    const double mag = exp(lm);
                    double sb, cb;
                    sincos(b.y, &sb, &cb);
                    rx = mag * ((double)ph.x * cb - (double)ph.y * sb);
                    ry = mag * ((double)ph.x * sb + (double)ph.y * cb);
                }
                if constexpr (PF) {
                    const double2 c2 = pf_ratio_any(m.pf, wsp[0], fl, nf, lane, *pst, pA);
                    const double2 r = zmul(make_double2(rx, ry), c2);
                    rx = r.x;
                    ry = r.y;
                }
                ex += val.x * rx - val.y * ry;
                ey += val.x * ry + val.y * rx;
            }
        }
        if (lane == 0) *Eout = make_double2(ex, ey);
    }
    if (Orow) {
        // tanh(theta) from the warp's scratch (tn)
        __syncwarp();
        const int n = m.n, nh = m.nh, S = m.S, nvb = m.n_vb;
        auto sg = [&](int i) -> R { return smem_bit(wsp, i) ? (R)-1 : (R)1; };
        if (!m.symmetric) {
            for (int q = lane; q < nvb; q += 32) Orow[q] = mk<R>(sg(q), 0);
            for (int q = lane; q < nh; q += 32) Orow[nvb + q] = tn[q];
            for (int k = 0; k < nh; k++) {
                const C2<R> t = tn[k];
                for (int j = lane; j < n; j += 32) {
                    const R s = sg(j);
                    Orow[nvb + nh + j + n * k] = mk<R>(s * t.x, s * t.y);
                }
            }
        } else {
            for (int q = lane; q < nvb; q += 32) {
                R acc = 0;
                for (int s = 0; s < S; s++) acc += sg(m.orbit[q * S + s]);
                Orow[q] = mk<R>(acc, 0);
            }
            for (int q = lane; q < nh; q += 32) {
                C2<R> acc = mk<R>(0, 0);
                for (int s = 0; s < S; s++) {
                    acc.x += tn[q + nh * s].x;
                    acc.y += tn[q + nh * s].y;
                }
                Orow[nvb + q] = acc;
            }
            for (int k = 0; k < nh; k++) {
                for (int j = lane; j < n; j += 32) {
                    C2<R> acc = mk<R>(0, 0);
                    for (int s = 0; s < S; s++) {
                        const R sv = sg(sInv[s * n + j]);
                        const C2<R> t = tn[k + nh * s];
                        acc.x = fma(sv, t.x, acc.x);
                        acc.y = fma(sv, t.y, acc.y);
                    }
                    Orow[nvb + nh + j + n * k] = acc;
                }
            }
        }
    }
    __syncwarp();
}

// Publish the warp's configuration and theta to its scratch for evaluate().
template <int E, typename R>
__device__ __forceinline__ void stage(const MachineDev& m, const uint32_t sp[4], const C2<R> th[E], uint32_t* wsp,
                                      C2<R>* wth, int lane) {
    if (lane < 4) wsp[lane] = spin_word(sp, lane);
#pragma unroll
    for (int e = 0; e < E; e++)
        if (slot_valid(lane, e, m.T)) wth[lane + 32 * e] = th[e];
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Shared-memory carve-up.  Block-wide tables (shared by every chain of the
// block) followed by one scratch area per warp.  The same byte arithmetic
// runs on host (launch sizing) and device (carving).  Expanded tables are
// padded to TP = 32 E columns (zero beyond T) so the FP32 sweep needs no
// per-entry bounds test: a zero column leaves its theta entry, and so its
// ln cosh, unchanged.
struct Smem {
    float2* U;      // [n+1][TP] U[f*TP + t] = W[P_s(f), k], row n = 0
    double2* U64;   // [n][TP] FP64 copy for the theta recompute
    float2* W32;    // FP32 W, site-major
    double2* W64;   // FP64 W, site-major (theta recompute, gather path)
    uint8_t* perm;  // [n][S]
    uint8_t* inv;   // [S][n]
    float* bre;     // [n+1] Re v[f mod n_vb] (Metropolis bias term), [n] = 0
    int2* bonds;    // proposal bonds
    float2* Wg;     // gather path: [n+1][nh] FP32 W, row n = 0 (shared or global)
    uint8_t* Pg;    // gather path, symmetric: [n+1][S] P_s(f), row n = n; with
                    // lane_rows in lane order: [n+1][32 / nh][E], entry
                    // [f][g][e] = P_{g + e 32 / nh}(f) (the rows of the
                    // entries e of the lanes l with l / nh = g)
    unsigned char* ham;  // evaluation: staged Hamiltonian tables
    double2* base64;     // [TP] hb + sum_f W[P_s(f), k]: theta of the all-up configuration (FP64)
    unsigned char* warp0;
    int warp_bytes;
};

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }
// Row length of the per-entry tables: 32 lanes x the entries per lane that
// the kernels use (elements_per_lane: 1, 2, 4, 8 or 16), so that the tables'
// layout and the kernels' indexing t = lane + 32 e agree for every T.
__host__ __device__ inline int padded_T(int T) {
    const int e = (T + 31) / 32;
    return 32 * (e <= 1 ? 1 : e <= 2 ? 2 : e <= 4 ? 4 : e <= 8 ? 8 : 16);
}

// per-warp scratch.  Evaluation: spins (16 B) | theta [T] | ln cosh re [T] |
// phase [T] | tanh theta [T] (evaluated in FP64 from the FP64 theta, so
// O_k keep FP32 accuracy next to the poles of tanh).  Sweeps: proposal ln|cosh| [TP].
// With the Pfaffian factor: evaluation + the PfStage staging, the n x n FP64
// matrix X^{-1} and its unscramble buffer; sweeps: the PfSweepStage staging
// and X^{-1} as its circulant half only (the proposal ln cosh values stay in
// registers, the fresh inverse runs in global scratch), so that the 14
// chains per SM of 2048 chains on 148 SMs fit the 164 KB carve-out and
// leave 92 KB of L1.
__host__ __device__ inline int eval_rbm_bytes(int T, int rsize) { return align16(16 + T * 7 * rsize); }
__host__ __device__ inline int sweep_rbm_bytes(int T, int rsize) { return align16(padded_T(T) * rsize); }
__host__ __device__ inline int eval_warp_bytes(int T, int rsize, int pf) {
    return eval_rbm_bytes(T, rsize) + (pf ? (int)sizeof(PfStage) + 2 * kPfMatBytes : 0);
}
__host__ __device__ inline int sweep_warp_bytes(int T, int rsize, int pf) {
    return pf ? (int)sizeof(PfSweepStage) + kPfCircBytes : sweep_rbm_bytes(T, rsize);
}

__host__ __device__ inline int table_bytes(const MachineDev& m, int fp64, const SmemPlan& pl, int n_bonds) {
    const int TP = padded_T(m.T);
    int b = 0;
    if (pl.use_u) b += align16((m.n + 1) * TP * 8);
    if (pl.u64) b += align16(m.n * TP * 16);
    if (!fp64 && pl.w32) b += align16(m.n * m.nh * 8);
    if (pl.w64) b += align16(m.n * m.nh * 16);
    if (m.symmetric) b += align16(m.n * m.S) * 2;
    b += align16((m.n + 1) * 4);
    if (pl.bonds) b += align16(n_bonds * 8);
    if (pl.gather && pl.wg) b += align16((m.n + 1) * m.nh * 8);
    if (pl.gather && m.symmetric) b += align16((m.n + 1) * m.S);
    b += align16(pl.ham);
    if (pl.u64 || pl.gather) b += align16(TP * 16);
    return b;
}

__device__ inline Smem carve(unsigned char* base, const MachineDev& m, int fp64, const SmemPlan& pl, int n_bonds,
                             int warp_bytes) {
    const int TP = padded_T(m.T);
    Smem s{};
    int off = 0;
    if (pl.use_u) {
        s.U = reinterpret_cast<float2*>(base + off);
        off += align16((m.n + 1) * TP * 8);
    }
    if (pl.u64) {
        s.U64 = reinterpret_cast<double2*>(base + off);
        off += align16(m.n * TP * 16);
    }
    if (!fp64 && pl.w32) {
        s.W32 = reinterpret_cast<float2*>(base + off);
        off += align16(m.n * m.nh * 8);
    }
    if (pl.w64) {
        s.W64 = reinterpret_cast<double2*>(base + off);
        off += align16(m.n * m.nh * 16);
    }
    if (m.symmetric) {
        s.perm = base + off;
        off += align16(m.n * m.S);
        s.inv = base + off;
        off += align16(m.n * m.S);
    }
    s.bre = reinterpret_cast<float*>(base + off);
    off += align16((m.n + 1) * 4);
    if (pl.bonds) {
        s.bonds = reinterpret_cast<int2*>(base + off);
        off += align16(n_bonds * 8);
    }
    if (pl.gather) {
        if (pl.wg) {
            s.Wg = reinterpret_cast<float2*>(base + off);
            off += align16((m.n + 1) * m.nh * 8);
        } else {
            s.Wg = const_cast<float2*>(m.W32);  // [n+1][nh] in global memory
        }
        if (m.symmetric) {
            s.Pg = base + off;
            off += align16((m.n + 1) * m.S);
        }
    }
    s.ham = base + off;
    off += align16(pl.ham);
    if (pl.u64 || pl.gather) {
        s.base64 = reinterpret_cast<double2*>(base + off);
        off += align16(TP * 16);
    }
    s.warp0 = base + off;
    s.warp_bytes = warp_bytes;
    return s;
}

__device__ inline void load_tables(const MachineDev& m, const Smem& s, int fp64, const SmemPlan& pl,
                                   const int2* bonds, int n_bonds) {
    const int tid = threadIdx.x, nt = blockDim.x;
    const int TP = padded_T(m.T);
    if (!fp64 && pl.w32)
        for (int i = tid; i < m.n * m.nh; i += nt) s.W32[i] = m.W32[i];
    if (pl.w64)
        for (int i = tid; i < m.n * m.nh; i += nt) s.W64[i] = m.W64[i];
    if (m.symmetric)
        for (int i = tid; i < m.n * m.S; i += nt) {
            s.perm[i] = m.perm[i];
            s.inv[i] = m.inv[i];
        }
    for (int i = tid; i <= m.n; i += nt) s.bre[i] = i < m.n ? (float)m.vb[i % m.n_vb].x : 0.f;
    if (pl.bonds)
        for (int i = tid; i < n_bonds; i += nt) s.bonds[i] = bonds[i];
    if (pl.gather && pl.wg)
        for (int i = tid; i < (m.n + 1) * m.nh; i += nt) s.Wg[i] = i < m.n * m.nh ? m.W32[i] : make_float2(0.f, 0.f);
    if (pl.gather && m.symmetric) {
        if (pl.lane_rows) {
            const int G = 32 / m.nh, E = m.T / 32;
            for (int i = tid; i < (m.n + 1) * m.S; i += nt) {
                const int f = i / m.S, j = i % m.S, g = j / E, e = j % E;
                s.Pg[i] = f < m.n ? m.perm[f * m.S + g + e * G] : (uint8_t)m.n;
            }
        } else {
            for (int i = tid; i < (m.n + 1) * m.S; i += nt) s.Pg[i] = i < m.n * m.S ? m.perm[i] : (uint8_t)m.n;
        }
    }
    if (pl.use_u || pl.u64)
        for (int i = tid; i < (m.n + 1) * TP; i += nt) {
            const int f = i / TP, t = i % TP;
            double2 w = make_double2(0, 0);
            if (f < m.n && t < m.T) {
                const int k = t % m.nh, sy = t / m.nh;
                const int row = m.symmetric ? (int)m.perm[f * m.S + sy] : f;
                w = m.W64[row * m.nh + k];
            }
            if (pl.use_u) s.U[i] = make_float2((float)w.x, (float)w.y);
            if (pl.u64 && f < m.n) s.U64[i] = w;
        }
    __syncthreads();
    // theta of the all-up configuration per entry; a recompute then subtracts
    // 2 W over the down spins only: theta = base - 2 sum_{f down} W[P_s(f), k]
    if (pl.u64 || pl.gather) {
        const double2* W64 = pl.w64 ? s.W64 : m.W64;
        for (int t = tid; t < TP; t += nt) {
            double2 acc = make_double2(0, 0);
            if (t < m.T) {
                const int k = t % m.nh, sy = t / m.nh;
                acc = m.hb[k];
                for (int f = 0; f < m.n; f++) {
                    const double2 w = pl.u64 ? s.U64[f * TP + t]
                                             : W64[(m.symmetric ? (int)s.perm[f * m.S + sy] : f) * m.nh + k];
                    acc.x += w.x;
                    acc.y += w.y;
                }
            }
            s.base64[t] = acc;
        }
    }
    __syncthreads();
}

// theta_out[chain][lane + 32 e] = th[e] (coalesced per e)
template <int E>
__device__ __forceinline__ void store_theta(float2* out, int chain, int lane, const float2 (&th)[E]) {
    float2* dst = out + (size_t)chain * (32 * E) + lane;
#pragma unroll
    for (int e = 0; e < E; e++) dst[32 * e] = th[e];
}

// One chain: metropolis_sampler::sample_chain (metropolis_sampler.cpp:118-273)
// for the warp's chain, general path (FP64 parity mode, and FP32 when the
// expanded flip table does not fit in shared memory).  Sampled
// configurations (16 bytes each) are recorded and evaluated afterwards by
// eval_kernel, one warp per sample: calling the evaluation from inside the
// sweep loop would make the call's register saves push the loop's live state
// (theta, ln cosh, bits) to local memory.  Randomness: Philox4x32-10 with
// counter {proposal, epoch, chain, 0}; lane j draws proposal (base + j), so
// one Philox call per lane serves 32 proposals.
//
// PF: the Pfaffian factor rides along (pfaffian.cuh): fresh X^{-1} at chain
// start, ratio of every proposal by the rank-2m formula, X^{-1} updated on
// acceptance and rebuilt every pf.refresh accepted moves
// (abstract_sampler.cpp:103-113).  pst / Cx: the warp's staging and X^{-1}
// (circulant half) in shared memory; pscr: its Gauss-Jordan workspace in
// global memory.  With PF the proposal's ln cosh values stay in registers
// (wlp unused).
template <int E, typename R, bool PF>
__device__ __forceinline__ void run_chain(const SamplerArgs& a, const Smem& sm, int chain, int lane, R* wlp,
                                          PfSweepStage* pst, double2* Cx, double2* pscr) {
    const MachineDev& m = a.m;
    const C2<R>* W = Wsel<R>::get(m, sm.W32 ? sm.W32 : m.W32);
    const double2* W64 = sm.W64 ? sm.W64 : m.W64;
    const int2* bonds = sm.bonds ? sm.bonds : a.prop_bonds;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    uint32_t sp[4];
    chain_start(a, chain, key, epoch, sp);

    C2<R> th[E];
    R L[E], lpn[E];  // lpn: the proposal's ln|cosh| (PF; else in wlp)
    theta_fp64<E, R>(m, W64, sm.perm, lane, sp, th);
#pragma unroll
    for (int e = 0; e < E; e++) L[e] = slot_valid(lane, e, m.T) ? lnc_re<R>(th[e].x, th[e].y) : (R)0;

    // Pfaffian context (pfaffian.cpp:284-297)
    double2 ib1[2], ib2[4];
    PfPairs<1> cp1;
    PfPairs<2> cp2;
    int ar = 0;  // accepted moves since the chain start (refresh counter)
    // the fresh context is built before the next proposal (one inlined copy
    // for the chain start and every refresh; a refresh due after the chain's
    // last proposal changes nothing that the chain outputs)
    bool fresh = true;

    // U(f, e): the flip row of site f for this lane's entry e
    auto U = [&](int f, int e) -> C2<R> {
        const int t = lane + 32 * e;
        return W[urow<R>(m, sm.perm, f, t / m.nh) * m.nh + t % m.nh];
    };

    const int n = m.n;
    // warm-up sweeps run every epoch, as in the reference; persistent chains
    // only differ in starting from the previous epoch's configuration
    const int total = segment_sweeps(a);
    uint32_t prop = prop_base(a), nacc = 0;
    uint32_t rr0 = 0, rr1 = 0, rr2 = 0;
    const uint32_t thr = a.bond_thr24;  // bond proposal iff (r0 >> 8) < thr
    for (int st = 0; st < total; st++) {
        int slot = 0;
        while (slot < n) {
            if ((prop & 31u) == 0) {
                const uint4 r = philox4x32(make_uint4(prop + lane, epoch, (uint32_t)chain, 0), key);
                rr0 = r.x;
                rr1 = r.y;
                rr2 = r.z;
            }
            const int src = prop & 31u;
            const uint32_t r0 = __shfl_sync(kFull, rr0, src);
            const uint32_t r1 = __shfl_sync(kFull, rr1, src);
            const uint32_t r2 = __shfl_sync(kFull, rr2, src);
            prop++;
            int f0, f1 = -1;
            if ((r0 >> 8) < thr) {
                const int2 b = bonds[pick(r1, (uint32_t)a.n_prop_bonds)];
                f0 = b.x;
                f1 = b.y;
                slot += 2;
            } else {
                f0 = (int)pick(r1, (uint32_t)n);
                slot += 1;
            }
            if constexpr (PF)
                if (fresh) {
                    pf_fresh_circ(m.pf, sp[0], lane, Cx, *pst, pscr);
                    fresh = false;
                }
            const bool s0 = spin_bit(sp, f0), s1 = f1 >= 0 && spin_bit(sp, f1);
            const R g0 = s0 ? (R)2 : (R)-2;  // -2 sigma_f
            const R g1 = s1 ? (R)2 : (R)-2;
            R d = 0;
#pragma unroll
            for (int e = 0; e < E; e++) {
                if (!slot_valid(lane, e, m.T)) continue;
                C2<R> t = th[e];
                const C2<R> u0 = U(f0, e);
                t.x = fma(g0, u0.x, t.x);
                t.y = fma(g0, u0.y, t.y);
                if (f1 >= 0) {
                    const C2<R> u1 = U(f1, e);
                    t.x = fma(g1, u1.x, t.x);
                    t.y = fma(g1, u1.y, t.y);
                }
                const R lp = lnc_re<R>(t.x, t.y);
                if constexpr (PF)
                    lpn[e] = lp;
                else
                    wlp[lane + 32 * e] = lp;  // read back only if accepted
                d += lp - L[e];
            }
            d = warp_sum(d);
            // bias: -2 sigma_f Re v[f mod n_vb] (rbm_base.cpp:306-318)
            {
                const int fl[2] = {f0, f1};
                d += (R)bias_delta(m, sp, fl, f1 >= 0 ? 2 : 1).x;
            }
            // accept with min(1, |psi'/psi|^2) (metropolis_sampler.cpp:223-243);
            // with the Pfaffian factor |psi'/psi|^2 = e^{2d} |Pf ratio|^2
            bool accept;
            if constexpr (PF) {
                const int fl[2] = {f0, f1};
                const double2 c2 = f1 >= 0 ? pf_ratio_circ<2>(m.pf, sp[0], fl, lane, *pst, Cx, ib2, cp2)
                                           : pf_ratio_circ<1>(m.pf, sp[0], fl, lane, *pst, Cx, ib1, cp1);
                accept = (double)unit24<R>(r2) < exp(2.0 * (double)d) * zabs2(c2);
            } else {
                accept = unit24<R>(r2) < exp_r((R)2 * d);
            }
            if (accept) {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    if (!slot_valid(lane, e, m.T)) continue;
                    const C2<R> u0 = U(f0, e);
                    th[e].x = fma(g0, u0.x, th[e].x);
                    th[e].y = fma(g0, u0.y, th[e].y);
                    if (f1 >= 0) {
                        const C2<R> u1 = U(f1, e);
                        th[e].x = fma(g1, u1.x, th[e].x);
                        th[e].y = fma(g1, u1.y, th[e].y);
                    }
                    L[e] = PF ? lpn[e] : wlp[lane + 32 * e];
                }
                flip_bit(sp, f0);
                if (f1 >= 0) flip_bit(sp, f1);
                nacc++;
                if constexpr (PF) {
                    ar++;
                    if (m.pf.refresh && ar % m.pf.refresh == 0)
                        fresh = true;
                    else if (f1 >= 0)
                        pf_accept_circ<2>(lane, *pst, ib2, cp2, Cx, m.pf.n);
                    else
                        pf_accept_circ<1>(lane, *pst, ib1, cp1, Cx, m.pf.n);
                }
            }
        }
        // FP64 recompute of theta once per sweep
        theta_fp64<E, R>(m, W64, sm.perm, lane, sp, th);
#pragma unroll
        for (int e = 0; e < E; e++) L[e] = slot_valid(lane, e, m.T) ? lnc_re<R>(th[e].x, th[e].y) : (R)0;
        if (const int j = sample_slot(a, st); j >= 0) {
            const size_t idx = (size_t)chain * a.spc + j;
            if (lane < 4) a.samples[4 * idx + lane] = spin_word(sp, lane);
        }
    }
    chain_finish(a, chain, lane, sp, nacc, prop);
}

// ln|cosh(a + ib)| without the constant -ln 2, FP32 sweep form.  With
// z = exp(-2|a|):  4 e^{-2|a|} |cosh x|^2 = 1 + z^2 + 2 z cos 2b, so
//   ln|cosh x| = |a| - ln 2 + 0.5 ln(1 + z^2 + 2 z cos 2b):
// one ex2, one cos, one lg2.  The sum of squares form used by lnc_re avoids
// the cancellation at the zeros of cosh (a = 0, b = pi/2 + k pi); this form
// only loses digits there, which leaves the Metropolis decision unchanged
// except for transitions at configurations of vanishing amplitude.  The
// hardware cosine takes the argument in revolutions, so 2b needs no
// separate range reduction for the accuracy the acceptance test needs.
//
// The three MUFU operations are issued in their flush-to-zero forms: the
// non-flushing forms add a denormal test and rescale around each one.  A
// flushed z (|a| > 43) leaves m2 = 1, the exact limit; a flushed m2 (a zero
// of cosh to FP32 precision) gives ln|cosh| = -inf, i.e. a proposal of
// vanishing amplitude that is rejected either way.
// Sum of ln|cosh| (the form above) over a lane's E entries: the |a| terms
// add up and the factors 1 + z^2 + 2 z cos 2b (each in [0, 4]) multiply in
// groups of four, one lg2 per group instead of one per entry.  A group's
// product stays within FP32 range unless its states have vanishing
// amplitude (then ln|cosh| is -inf either way).  Same order of operations
// for a given group of entries wherever it is formed.
template <int E> __device__ __forceinline__ float lnc_sweep_sum(const float2 (&t)[E]) {
    float sa = 0.f, lg = 0.f;
#pragma unroll
    for (int g = 0; g < E; g += 4) {
        float pm = 1.f;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (g + q >= E) break;
            const float2 x = t[g + q];
            const float aa = fabsf(x.x);
            const float z = ex2_ftz(aa * -2.88539008177792681f);
            const float c2 = cos_ftz(2.f * x.y);
            pm *= fmaf(z, fmaf(2.f, c2, z), 1.f);
            sa += aa;
        }
        lg += lg2_ftz(pm);
    }
    return fmaf(0.346573590279972655f, lg, sa);
}

// FP32 sweep path with the expanded flip table in shared memory.  Proposals
// are decoded lane-parallel: with each Philox batch, lane j turns its draw
// into a packed (f0, f1, bond) code and 0.5 ln u, so a proposal costs two
// shuffles; a single-site proposal uses the all-zero pad row n as its second
// flip, which keeps the update branch-free; acceptance compares
// 0.5 ln u < log|psi'/psi| (the same test as u < |psi'/psi|^2).  NW = 1
// when all sites fit in the first configuration word (n <= 32): the bit
// lookups then need no word selection.
template <int E, int NW>
__device__ __forceinline__ void run_chain_fast(const SamplerArgs& a, const Smem& sm, int chain, int lane) {
    const MachineDev& m = a.m;
    const int n = m.n, TP = 32 * E;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    uint32_t sp[4];
    chain_start(a, chain, key, epoch, sp);
    auto sbit = [&](int i) -> bool {
        if constexpr (NW == 1)
            return (sp[0] >> i) & 1u;
        else
            return spin_bit(sp, i);
    };
    auto sflip = [&](int i) {
        if constexpr (NW == 1)
            sp[0] ^= 1u << i;
        else
            flip_bit(sp, i);
    };

    float2 th[E];
    float SL = 0.f;  // this lane's sum of ln|cosh theta_e| (current state)
    auto recompute = [&]() {
        if (sm.U64) {
            double2 acc[E];
#pragma unroll
            for (int e = 0; e < E; e++) acc[e] = sm.base64[lane + 32 * e];
            // down spins in increasing order
#pragma unroll
            for (int wd = 0; wd < NW; wd++) {
                uint32_t bits = spin_word(sp, wd);
                while (bits) {
                    const int f = 32 * wd + __ffs(bits) - 1;
                    bits &= bits - 1;
                    const double2* col = sm.U64 + f * TP + lane;
#pragma unroll
                    for (int e = 0; e < E; e++) {
                        const double2 w = col[32 * e];
                        acc[e].x = fma(-2.0, w.x, acc[e].x);
                        acc[e].y = fma(-2.0, w.y, acc[e].y);
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < E; e++) th[e] = make_float2((float)acc[e].x, (float)acc[e].y);
        } else {
            theta_fp64<E, float>(m, sm.W64 ? sm.W64 : m.W64, sm.perm, lane, sp, th);
        }
        SL = lnc_sweep_sum<E>(th);
    };
    recompute();

    const int2* bonds = sm.bonds ? sm.bonds : a.prop_bonds;
    const int total = segment_sweeps(a);
    const uint32_t thr = a.bond_thr24;
    uint32_t prop = prop_base(a), nacc = 0, pcode = 0;
    float plu = 0.f;
    for (int st = 0; st < total; st++) {
        int slot = 0;
        while (slot < n) {
            if ((prop & 31u) == 0) {
                const uint4 r = philox4x32(make_uint4(prop + lane, epoch, (uint32_t)chain, 0), key);
                uint32_t f0, f1, bond;
                if ((r.x >> 8) < thr) {
                    const int2 b = bonds[pick(r.y, (uint32_t)a.n_prop_bonds)];
                    f0 = (uint32_t)b.x;
                    f1 = (uint32_t)b.y;
                    bond = 1;
                } else {
                    f0 = pick(r.y, (uint32_t)n);
                    f1 = (uint32_t)n;
                    bond = 0;
                }
                pcode = f0 | (f1 << 8) | (bond << 16);
                plu = 0.346573590279972655f * lg2_ftz(unit24<float>(r.z));  // 0.5 ln u
            }
            const int src = prop & 31u;
            const uint32_t code = __shfl_sync(kFull, pcode, src);
            const float lu = __shfl_sync(kFull, plu, src);
            prop++;
            const int f0 = code & 255u, f1 = (code >> 8) & 255u;
            const bool bond = (code >> 16) != 0;
            slot += bond ? 2 : 1;
            const float g0 = sbit(f0) ? 2.f : -2.f;  // -2 sigma_f
            const float g1 = (bond && sbit(f1)) ? 2.f : -2.f;
            const float2 G0 = make_float2(g0, g0), G1 = make_float2(g1, g1);
            const float2* u0 = sm.U + f0 * TP + lane;
            const float2* u1 = sm.U + f1 * TP + lane;
            float2 tq[E];
            if (bond) {
#pragma unroll
                for (int e = 0; e < E; e++) tq[e] = __ffma2_rn(G1, u1[32 * e], __ffma2_rn(G0, u0[32 * e], th[e]));
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) tq[e] = __ffma2_rn(G0, u0[32 * e], th[e]);
            }
            const float sp_new = lnc_sweep_sum<E>(tq);
            float d = sweep_sum(sp_new - SL);
            d = fmaf(g0, sm.bre[f0], d);
            d = fmaf(g1, sm.bre[f1], d);
            if (lu < d) {
#pragma unroll
                for (int e = 0; e < E; e++) th[e] = tq[e];
                SL = sp_new;
                sflip(f0);
                if (bond) sflip(f1);
                nacc++;
            }
        }
        recompute();  // FP64 recompute of theta once per sweep
        if (const int j = sample_slot(a, st); j >= 0) {
            const size_t idx = (size_t)chain * a.spc + j;
            if (lane < 4) a.samples[4 * idx + lane] = spin_word(sp, lane);
        }
    }
    if (a.theta_out) store_theta<E>(a.theta_out, chain, lane, th);
    chain_finish(a, chain, lane, sp, nacc, prop);
}

// Two chains per warp (FP32 expanded-table path, n <= 32, theta tables of
// at most 32 E entries): lanes 0-15 run chain 2 pair, lanes 16-31 chain
// 2 pair + 1.  Lane h of a half holds the entries that lanes h and h + 16
// hold in run_chain_fast, t = h + 16 j + 32 k (j = 0, 1; k < E), and keeps
// their two ln|cosh| sums apart, so that adding them reproduces the first
// level of run_chain_fast's butterfly and the remaining 16-lane reduction
// its other levels: every sum, decision and configuration is bit-identical
// to the one-chain-per-warp sweep.  The per-proposal work that does not
// scale with the entries (decoding, bias, acceptance, bit updates, loop
// control) is issued once for both chains.  Each chain keeps its proposal
// counter and slot count; a chain whose sweep is complete waits (its lanes
// compute but apply nothing) until the other's is, and both then take the
// FP64 recompute.  Proposals are drawn 16 at a time (lane j of the half
// draws proposal prop + j): the same Philox counters as 32 at a time.
template <int E>
__device__ __forceinline__ void run_chain_pair(const SamplerArgs& a, const Smem& sm, int pair, int lane) {
    const MachineDev& m = a.m;
    const int n = m.n, TP = 32 * E;
    const int half = lane >> 4, hl = lane & 15;
    const int chain = 2 * pair + half;
    const bool live = chain < a.n_chains;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    uint32_t sp[4];
    chain_start(a, live ? chain : 2 * pair, key, epoch, sp);
    uint32_t s0 = sp[0];  // n <= 32: the whole configuration

    float2 th[2 * E];  // entry 2 k + j is t = hl + 16 j + 32 k
    float SA = 0.f, SB = 0.f;  // sums over j = 0 and j = 1 (current state)
    auto recompute = [&]() {
        double2 acc[2 * E];
#pragma unroll
        for (int e = 0; e < 2 * E; e++) acc[e] = sm.base64[hl + 16 * (e & 1) + 32 * (e >> 1)];
        for (uint32_t bits = s0; bits; bits &= bits - 1) {  // down spins in increasing order
            const double2* col = sm.U64 + (__ffs(bits) - 1) * TP + hl;
#pragma unroll
            for (int e = 0; e < 2 * E; e++) {
                const double2 w = col[16 * (e & 1) + 32 * (e >> 1)];
                acc[e].x = fma(-2.0, w.x, acc[e].x);
                acc[e].y = fma(-2.0, w.y, acc[e].y);
            }
        }
        float2 tA[E], tB[E];
#pragma unroll
        for (int k = 0; k < E; k++) {
            th[2 * k] = make_float2((float)acc[2 * k].x, (float)acc[2 * k].y);
            th[2 * k + 1] = make_float2((float)acc[2 * k + 1].x, (float)acc[2 * k + 1].y);
            tA[k] = th[2 * k];
            tB[k] = th[2 * k + 1];
        }
        SA = lnc_sweep_sum<E>(tA);
        SB = lnc_sweep_sum<E>(tB);
    };
    recompute();

    const int2* bonds = sm.bonds ? sm.bonds : a.prop_bonds;
    const int total = segment_sweeps(a);
    const uint32_t thr = a.bond_thr24;
    uint32_t prop = prop_base(a), nacc = 0, pcode = 0;
    float plu = 0.f;
    for (int st = 0; st < total; st++) {
        int slot = live ? 0 : n;
        while (__any_sync(kFull, slot < n)) {
            const bool on = slot < n;
            if (on && (prop & 15u) == 0) {
                const uint4 r = philox4x32(make_uint4(prop + hl, epoch, (uint32_t)chain, 0), key);
                uint32_t f0, f1, bond;
                if ((r.x >> 8) < thr) {
                    const int2 b = bonds[pick(r.y, (uint32_t)a.n_prop_bonds)];
                    f0 = (uint32_t)b.x;
                    f1 = (uint32_t)b.y;
                    bond = 1;
                } else {
                    f0 = pick(r.y, (uint32_t)n);
                    f1 = (uint32_t)n;
                    bond = 0;
                }
                pcode = f0 | (f1 << 8) | (bond << 16);
                plu = 0.346573590279972655f * lg2_ftz(unit24<float>(r.z));  // 0.5 ln u
            }
            const int src = prop & 15u;
            const uint32_t code = __shfl_sync(kFull, pcode, src, 16);
            const float lu = __shfl_sync(kFull, plu, src, 16);
            const int f0 = code & 255u, f1 = (code >> 8) & 255u;
            const bool bond = (code >> 16) != 0;
            const float g0 = (s0 >> f0) & 1u ? 2.f : -2.f;  // -2 sigma_f
            const float g1 = (bond && ((s0 >> f1) & 1u)) ? 2.f : -2.f;
            const float2 G0 = make_float2(g0, g0), G1 = make_float2(g1, g1);
            const float2* u0 = sm.U + f0 * TP + hl;
            const float2* u1 = sm.U + f1 * TP + hl;
            float2 tn[2 * E], tA[E], tB[E];
#pragma unroll
            for (int k = 0; k < E; k++) {
                tn[2 * k] = __ffma2_rn(G1, u1[32 * k], __ffma2_rn(G0, u0[32 * k], th[2 * k]));
                tn[2 * k + 1] = __ffma2_rn(G1, u1[16 + 32 * k], __ffma2_rn(G0, u0[16 + 32 * k], th[2 * k + 1]));
                tA[k] = tn[2 * k];
                tB[k] = tn[2 * k + 1];
            }
            const float nA = lnc_sweep_sum<E>(tA), nB = lnc_sweep_sum<E>(tB);
            // the one-chain sweep's sum: lanes h and h + 16 of it are this
            // lane's two partials (integer sums are exact in any order)
            const float vA = nA - SA, vB = nB - SB;
            const int iv = fix22(vA) + fix22(vB);
            const int ilo = __reduce_add_sync(kFull, hl == lane ? iv : 0);
            const int ihi = __reduce_add_sync(kFull, hl == lane ? 0 : iv);
            const bool big = !(fabsf(vA) < 16.f) || !(fabsf(vB) < 16.f);
            const unsigned bigm = __ballot_sync(kFull, big);
            float d;
            if (bigm & (half ? 0xffff0000u : 0x0000ffffu)) {
                d = vA + vB;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(kFull, d, o);
            } else {
                d = (float)(half ? ihi : ilo) * (1.f / kFixScale);
            }
            d = fmaf(g0, sm.bre[f0], d);
            d = fmaf(g1, sm.bre[f1], d);
            if (on) {
                prop++;
                slot += bond ? 2 : 1;
                if (lu < d) {
#pragma unroll
                    for (int e = 0; e < 2 * E; e++) th[e] = tn[e];
                    SA = nA;
                    SB = nB;
                    s0 ^= 1u << f0;
                    if (bond) s0 ^= 1u << f1;
                    nacc++;
                }
            }
        }
        recompute();  // FP64 recompute of theta once per sweep
        if (const int j = sample_slot(a, st); live && j >= 0) {
            const size_t idx = (size_t)chain * a.spc + j;
            if (hl < 4) a.samples[4 * idx + hl] = hl == 0 ? s0 : 0u;
        }
    }
    if (live) {
        if (hl < 4) a.spins[4 * chain + hl] = hl == 0 ? s0 : 0u;
        if (hl == 0) {
            const uint32_t made = prop - prop_base(a);
            a.n_acc[chain] = (a.sweep0 ? a.n_acc[chain] : 0u) + nacc;
            a.n_prop[chain] = (a.sweep0 ? a.n_prop[chain] : 0u) + made;
        }
    }
}

// FP32 sweep path with gathered flip rows, for theta tables whose expanded
// flip table does not fit in shared memory (e.g. 128 sites x 512 entries):
// entry e of this lane is (k_e, s_e) = ((lane + 32 e) mod nh, (lane + 32 e) /
// nh), computed once per chain; the flip row of site f is
// W[P_{s_e}(f), k_e], two dependent shared-memory loads (the symmetry table
// byte, then the FP32 W element).  Site n is the all-zero pad row (single-
// site proposals use it as their second flip).  The proposal's theta' is
// kept in registers and becomes theta on acceptance.  Otherwise the same
// proposal decoding, running ln|cosh| sum and FP64 recompute per sweep as
// run_chain_fast.
// WS: the FP32 flip rows (with their zero pad row) are in shared memory.
template <int E, bool SYM, bool WS>
__device__ __forceinline__ void run_chain_gather(const SamplerArgs& a, const Smem& sm, int chain, int lane) {
    const MachineDev& m = a.m;
    const int n = m.n, nh = m.nh, S = m.S;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    uint32_t sp[4];
    chain_start(a, chain, key, epoch, sp);

    uint32_t ent[E];   // (s_e << 16) | k_e
    uint32_t vmask = 0;
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int t = lane + 32 * e;
        const bool ok = t < m.T;
        const int k = ok ? t % nh : 0, s = ok ? t / nh : 0;
        ent[e] = ((uint32_t)s << 16) | (uint32_t)k;
        vmask |= ok ? 1u << e : 0u;
    }
    const float2* Wg = sm.Wg;
    const uint8_t* Pg = sm.Pg;
    const uint32_t wsa = WS ? smem_addr(Wg) : 0u, psa = SYM ? smem_addr(Pg) : 0u;
    auto row = [&](int f, uint32_t en) -> int { return SYM ? (int)Pg[f * S + (en >> 16)] : f; };
    auto urd = [&](int f, int e) -> float2 {
        const uint32_t en = ent[e];
        float2 u;
        if constexpr (WS) {
            const int r = SYM ? (int)lds_u8(psa + (uint32_t)(f * S + (en >> 16))) : f;
            u = lds_f2(wsa + 8u * (uint32_t)(r * nh + (en & 0xffffu)));
        } else {
            u = Wg[row(f, en) * nh + (en & 0xffffu)];
        }
        return ((vmask >> e) & 1u) ? u : make_float2(0.f, 0.f);
    };

    float2 th[E];
    float SL = 0.f;
    const double2* W64 = sm.W64 ? sm.W64 : m.W64;
    auto recompute = [&]() {
        // FP64 theta = b + sum_f sigma_f W[P_s(f), k], four entries at a time
#pragma unroll
        for (int c = 0; c < E; c += 4) {
            double2 acc[4];
#pragma unroll
            for (int q = 0; q < 4; q++)
                acc[q] = (c + q < E && ((vmask >> (c + q)) & 1u)) ? sm.base64[lane + 32 * (c + q)]
                                                                   : make_double2(0, 0);
#pragma unroll
            for (int wd = 0; wd < 4; wd++) {  // down spins in increasing order
                uint32_t bits = spin_word(sp, wd);
                while (bits) {
                    const int f = 32 * wd + __ffs(bits) - 1;
                    bits &= bits - 1;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (c + q >= E || !((vmask >> (c + q)) & 1u)) continue;
                        const uint32_t en = ent[c + q];
                        const double2 w = W64[row(f, en) * nh + (en & 0xffffu)];
                        acc[q].x = fma(-2.0, w.x, acc[q].x);
                        acc[q].y = fma(-2.0, w.y, acc[q].y);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (c + q < E) th[c + q] = make_float2((float)acc[q].x, (float)acc[q].y);
        }
        SL = lnc_sweep_sum<E>(th);
    };
    recompute();

    const int2* bonds = sm.bonds ? sm.bonds : a.prop_bonds;
    const int total = segment_sweeps(a);
    const uint32_t thr = a.bond_thr24;
    uint32_t prop = prop_base(a), nacc = 0, pcode = 0;
    float plu = 0.f;
    for (int st = 0; st < total; st++) {
        int slot = 0;
        while (slot < n) {
            if ((prop & 31u) == 0) {
                const uint4 r = philox4x32(make_uint4(prop + lane, epoch, (uint32_t)chain, 0), key);
                uint32_t f0, f1, bond;
                if ((r.x >> 8) < thr) {
                    const int2 b = bonds[pick(r.y, (uint32_t)a.n_prop_bonds)];
                    f0 = (uint32_t)b.x;
                    f1 = (uint32_t)b.y;
                    bond = 1;
                } else {
                    f0 = pick(r.y, (uint32_t)n);
                    f1 = (uint32_t)n;
                    bond = 0;
                }
                pcode = f0 | (f1 << 8) | (bond << 16);
                plu = 0.346573590279972655f * lg2_ftz(unit24<float>(r.z));  // 0.5 ln u
            }
            const int src = prop & 31u;
            const uint32_t code = __shfl_sync(kFull, pcode, src);
            const float lu = __shfl_sync(kFull, plu, src);
            prop++;
            const int f0 = code & 255u, f1 = (code >> 8) & 255u;
            const bool bond = (code >> 16) != 0;
            slot += bond ? 2 : 1;
            const float g0 = spin_bit(sp, f0) ? 2.f : -2.f;  // -2 sigma_f
            const float g1 = (bond && spin_bit(sp, f1)) ? 2.f : -2.f;
            const float2 G0 = make_float2(g0, g0), G1 = make_float2(g1, g1);
            float2 tn[E];
            if (bond) {
#pragma unroll
                for (int e = 0; e < E; e++) tn[e] = __ffma2_rn(G1, urd(f1, e), __ffma2_rn(G0, urd(f0, e), th[e]));
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) tn[e] = __ffma2_rn(G0, urd(f0, e), th[e]);
            }
            const float sp_new = lnc_sweep_sum<E>(tn);
            float d = sweep_sum(sp_new - SL);
            d = fmaf(g0, sm.bre[f0], d);
            d = fmaf(g1, sm.bre[f1], d);
            if (lu < d) {
#pragma unroll
                for (int e = 0; e < E; e++) th[e] = tn[e];
                SL = sp_new;
                flip_bit(sp, f0);
                if (bond) flip_bit(sp, f1);
                nacc++;
            }
        }
        recompute();  // FP64 recompute of theta once per sweep
        if (const int j = sample_slot(a, st); j >= 0) {
            const size_t idx = (size_t)chain * a.spc + j;
            if (lane < 4) a.samples[4 * idx + lane] = spin_word(sp, lane);
        }
    }
    if (a.theta_out) store_theta<E>(a.theta_out, chain, lane, th);
    chain_finish(a, chain, lane, sp, nacc, prop);
}

// The gather sweep for symmetric machines whose theta fills every lane
// entry (T = 32 E) with nh | 32: lane l holds the entries (k, s) = (l mod
// nh, l / nh + e 32 / nh), so the rows P_s(f) of its E entries are E
// consecutive bytes of the lane-ordered symmetry table; a flip costs one
// E-byte shared load, then per entry a byte extract and the W element load
// (no per-entry index arithmetic or validity selects).  The arithmetic is
// run_chain_gather's, operation for operation.
template <int E>
__device__ __forceinline__ void run_chain_lanerows(const SamplerArgs& a, const Smem& sm, int chain, int lane) {
    const MachineDev& m = a.m;
    const int n = m.n, nh = m.nh;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    uint32_t sp[4];
    chain_start(a, chain, key, epoch, sp);

    const int k = lane % nh, g = lane / nh;
    const uint32_t wk = smem_addr(sm.Wg) + 8u * (uint32_t)k;       // FP32 W row r: wk + 8 nh r
    const uint32_t rowb = 8u * (uint32_t)nh;
    const uint32_t pta = smem_addr(sm.Pg) + (uint32_t)(g * E);    // this lane group's rows of flip 0
    const uint32_t fstride = (uint32_t)m.S;                        // bytes per flip
    auto rowof = [](const uint32_t (&pw)[E / 4], int e) -> uint32_t { return (pw[e >> 2] >> (8 * (e & 3))) & 0xffu; };
    const double2* W64 = sm.W64 ? sm.W64 : m.W64;

    float2 th[E];
    float SL = 0.f;
    auto recompute = [&]() {
        // FP64 theta = b + sum_f sigma_f W[P_s(f), k], four entries at a time
#pragma unroll
        for (int c = 0; c < E; c += 4) {
            double2 acc[4];
#pragma unroll
            for (int q = 0; q < 4; q++) acc[q] = sm.base64[lane + 32 * (c + q)];
#pragma unroll
            for (int wd = 0; wd < 4; wd++) {  // down spins in increasing order
                uint32_t bits = spin_word(sp, wd);
                while (bits) {
                    const int f = 32 * wd + __ffs(bits) - 1;
                    bits &= bits - 1;
                    uint32_t pw[1];
                    lds_words<4>(pta + (uint32_t)f * fstride + (uint32_t)c, pw);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const uint32_t r = (pw[0] >> (8 * q)) & 0xffu;
                        const double2 w = W64[r * nh + k];
                        acc[q].x = fma(-2.0, w.x, acc[q].x);
                        acc[q].y = fma(-2.0, w.y, acc[q].y);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) th[c + q] = make_float2((float)acc[q].x, (float)acc[q].y);
        }
        SL = lnc_sweep_sum<E>(th);
    };
    if (a.theta_in) {
        const float2* src = a.theta_in + (size_t)chain * (32 * E) + lane;
#pragma unroll
        for (int e = 0; e < E; e++) th[e] = src[32 * e];
        SL = lnc_sweep_sum<E>(th);
    } else {
        recompute();
    }

    const int2* bonds = sm.bonds ? sm.bonds : a.prop_bonds;
    const int total = segment_sweeps(a);
    const uint32_t thr = a.bond_thr24;
    uint32_t prop = prop_base(a), nacc = 0, pcode = 0;
    float plu = 0.f;
    for (int st = 0; st < total; st++) {
        int slot = 0;
        while (slot < n) {
            if ((prop & 31u) == 0) {
                const uint4 r = philox4x32(make_uint4(prop + lane, epoch, (uint32_t)chain, 0), key);
                uint32_t f0, f1, bond;
                if ((r.x >> 8) < thr) {
                    const int2 b = bonds[pick(r.y, (uint32_t)a.n_prop_bonds)];
                    f0 = (uint32_t)b.x;
                    f1 = (uint32_t)b.y;
                    bond = 1;
                } else {
                    f0 = pick(r.y, (uint32_t)n);
                    f1 = (uint32_t)n;
                    bond = 0;
                }
                pcode = f0 | (f1 << 8) | (bond << 16);
                plu = 0.346573590279972655f * lg2_ftz(unit24<float>(r.z));  // 0.5 ln u
            }
            const int src = prop & 31u;
            const uint32_t code = __shfl_sync(kFull, pcode, src);
            const float lu = __shfl_sync(kFull, plu, src);
            prop++;
            const int f0 = code & 255u, f1 = (code >> 8) & 255u;
            const bool bond = (code >> 16) != 0;
            slot += bond ? 2 : 1;
            const float g0 = spin_bit(sp, f0) ? 2.f : -2.f;  // -2 sigma_f
            const float g1 = (bond && spin_bit(sp, f1)) ? 2.f : -2.f;
            const float2 G0 = make_float2(g0, g0), G1 = make_float2(g1, g1);
            uint32_t p0[E / 4];
            lds_words<E>(pta + (uint32_t)f0 * fstride, p0);
            float2 tn[E];
            if (bond) {
                uint32_t p1[E / 4];
                lds_words<E>(pta + (uint32_t)f1 * fstride, p1);
#pragma unroll
                for (int e = 0; e < E; e++)
                    tn[e] = __ffma2_rn(G1, lds_f2(wk + rowof(p1, e) * rowb),
                                       __ffma2_rn(G0, lds_f2(wk + rowof(p0, e) * rowb), th[e]));
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) tn[e] = __ffma2_rn(G0, lds_f2(wk + rowof(p0, e) * rowb), th[e]);
            }
            const float sp_new = lnc_sweep_sum<E>(tn);
            float d = sweep_sum(sp_new - SL);
            d = fmaf(g0, sm.bre[f0], d);
            d = fmaf(g1, sm.bre[f1], d);
            if (lu < d) {
#pragma unroll
                for (int e = 0; e < E; e++) th[e] = tn[e];
                SL = sp_new;
                flip_bit(sp, f0);
                if (bond) flip_bit(sp, f1);
                nacc++;
            }
        }
        recompute();  // FP64 recompute of theta once per sweep
        if (const int j = sample_slot(a, st); j >= 0) {
            const size_t idx = (size_t)chain * a.spc + j;
            if (lane < 4) a.samples[4 * idx + lane] = spin_word(sp, lane);
        }
    }
    if (a.theta_out) store_theta<E>(a.theta_out, chain, lane, th);
    chain_finish(a, chain, lane, sp, nacc, prop);
}

// ---------------------------------------------------------------------------
// The sweeps of several sessions (independent trainings of a batch) in one
// launch.  Every problem gets a contiguous range of blocks; a block stages
// its problem's tables (the problem's own shared-memory plan for the
// launch's warps per block) and its warps take the problem's chains,
// chain = warp * blocks + local block (one chain per warp and pass).  The
// per-chain sweep is the per-session kernel's function for the problem's
// entries per lane and path, so every chain's samples, counters and final
// configuration are bit-identical to the session's own launch.
template <int E>
__device__ __forceinline__ void batch_chain(const SamplerArgs& a, const Smem& sm, int chain, int lane, int path) {
    if (path == 0) {  // expanded flip table
        if (a.m.n <= 32)
            run_chain_fast<E, 1>(a, sm, chain, lane);
        else
            run_chain_fast<E, 4>(a, sm, chain, lane);
        return;
    }
    if constexpr (E >= 4) {
        if (a.plan.lane_rows) {
            run_chain_lanerows<E>(a, sm, chain, lane);
            return;
        }
    }
    if (a.m.symmetric) {
        if (a.plan.wg)
            run_chain_gather<E, true, true>(a, sm, chain, lane);
        else
            run_chain_gather<E, true, false>(a, sm, chain, lane);
    } else {
        if (a.plan.wg)
            run_chain_gather<E, false, true>(a, sm, chain, lane);
        else
            run_chain_gather<E, false, false>(a, sm, chain, lane);
    }
}

template <int E>
__global__ void __launch_bounds__(32 * kBatchSweepWarps)
    sampler_batch_kernel(const BatchSweepDesc* __restrict__ desc, int nprob) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(16) unsigned char sa_raw[sizeof(SamplerArgs)];
    __shared__ int pidx;
    if (threadIdx.x == 0) {
        int i = 0;
        while (i + 1 < nprob && desc[i + 1].block0 <= (int)blockIdx.x) i++;
        pidx = i;
    }
    __syncthreads();
    {  // the problem's arguments into shared memory, word by word
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&desc[pidx].a);
        uint32_t* dst = reinterpret_cast<uint32_t*>(sa_raw);
        for (int w = threadIdx.x; w < (int)(sizeof(SamplerArgs) / 4); w += blockDim.x) dst[w] = src[w];
    }
    __syncthreads();
    const SamplerArgs& a = *reinterpret_cast<const SamplerArgs*>(sa_raw);
    const int lb = blockIdx.x - desc[pidx].block0, nb = desc[pidx].blocks;
    const int path = desc[pidx].path;
    Smem sm = carve(smem, a.m, 0, a.plan, a.n_prop_bonds, sweep_warp_bytes(a.m.T, 4, 0));
    load_tables(a.m, sm, 0, a.plan, a.prop_bonds, a.n_prop_bonds);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int chain = warp * nb + lb; chain < a.n_chains; chain += kBatchSweepWarps * nb)
        batch_chain<E>(a, sm, chain, lane, path);
}

// Thread bound per entries-per-lane: 28 warps (896 threads, 72 registers)
// keep 4096 chains resident on 148 SMs for E <= 4.
template <int E, bool PF = false> struct MaxThreads {
    static constexpr int v = PF ? 512 : (E <= 2 ? 1024 : (E <= 4 ? 896 : (E <= 8 ? 512 : 256)));
    static constexpr int gather = E <= 4 ? 896 : (E <= 8 ? 640 : 384);
    static constexpr int pair = E <= 1 ? 1024 : (E <= 2 ? 768 : 512);  // 2 E entries per lane
};

// All chains at once, persistent warps: global warp g = warp * gridDim.x +
// blockIdx.x takes chains g, g + total_warps, ... so consecutive chains land
// on different SMs and every block holds the tables once.  FAST selects the
// FP32 expanded-table path.
template <int E, typename R, int FAST, bool PF>
__global__ void __launch_bounds__(FAST == 2 ? MaxThreads<E, PF>::gather
                                            : (FAST == 3 ? MaxThreads<E, PF>::pair : MaxThreads<E, PF>::v),
                                  1) sampler_kernel(const SamplerArgs a) {
    if constexpr (!PF && FAST != 3)  // behind a screened sweep
        if (a.gate && !*a.gate) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int fp64 = sizeof(R) == 8;
    Smem sm = carve(smem, a.m, fp64, a.plan, a.n_prop_bonds, sweep_warp_bytes(a.m.T, sizeof(R), PF));
    load_tables(a.m, sm, fp64, a.plan, a.prop_bonds, a.n_prop_bonds);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    R* wlp = reinterpret_cast<R*>(sm.warp0 + warp * sm.warp_bytes);
    PfSweepStage* pst = reinterpret_cast<PfSweepStage*>(sm.warp0 + warp * sm.warp_bytes);
    double2* Cx = reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(pst) + sizeof(PfSweepStage));
    double2* pscr = PF ? a.m.pf.scratch + (size_t)(blockIdx.x * (blockDim.x >> 5) + warp) * kPfMaxSites * kPfMaxSites
                       : nullptr;
    const int total_warps = (blockDim.x >> 5) * gridDim.x;
    if constexpr (FAST == 3) {
        // two chains per warp (the chain-pair loop bound is warp-uniform)
        const int pairs = (a.n_chains + 1) / 2;
        for (int pair = warp * gridDim.x + blockIdx.x; pair < pairs; pair += total_warps)
            run_chain_pair<E>(a, sm, pair, lane);
    } else
    for (int chain = warp * gridDim.x + blockIdx.x; chain < a.n_chains; chain += total_warps) {
        if constexpr (FAST == 1)
            if (a.m.n <= 32)
                run_chain_fast<E, 1>(a, sm, chain, lane);
            else
                run_chain_fast<E, 4>(a, sm, chain, lane);
        else if constexpr (FAST == 2) {
            if constexpr (E >= 4) {
                if (a.plan.lane_rows) {
                    run_chain_lanerows<E>(a, sm, chain, lane);
                    continue;
                }
            }
            if (a.m.symmetric) {
                if (a.plan.wg)
                    run_chain_gather<E, true, true>(a, sm, chain, lane);
                else
                    run_chain_gather<E, true, false>(a, sm, chain, lane);
            } else {
                if (a.plan.wg)
                    run_chain_gather<E, false, true>(a, sm, chain, lane);
                else
                    run_chain_gather<E, false, false>(a, sm, chain, lane);
            }
        } else
            run_chain<E, R, PF>(a, sm, chain, lane, wlp, pst, Cx, pscr);
    }
}

// ---------------------------------------------------------------------------
// Batched evaluation at given configurations: log psi, E_loc, O_k, or the
// log psi ratio for given flips (parity entry points).
template <int E, typename R, bool PF>
__global__ void __launch_bounds__(256, E <= 4 ? 4 : 2) eval_kernel(const EvalArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const MachineDev& m = a.m;
    const int fp64 = sizeof(R) == 8;
    Smem sm = carve(smem, m, fp64, a.plan, 0, eval_warp_bytes(m.T, sizeof(R), PF));
    load_tables(m, sm, fp64, a.plan, nullptr, 0);
    // the operator tables in shared memory: every term of E_loc walks them
    // in a chain of dependent loads
    HamDev H = a.H;
    if (a.plan.ham) {
        unsigned char* hb = sm.ham;
        OpDev* sops = reinterpret_cast<OpDev*>(hb);
        hb += align16(H.n_ops * (int)sizeof(OpDev));
        int* srow = reinterpret_cast<int*>(hb);
        hb += align16(H.n_rows * 4);
        uint32_t* smask = reinterpret_cast<uint32_t*>(hb);
        hb += align16(H.n_ents * 4);
        double2* sval = reinterpret_cast<double2*>(hb);
        const int ow = H.n_ops * (int)(sizeof(OpDev) / 4);
        for (int i = threadIdx.x; i < ow; i += blockDim.x)
            reinterpret_cast<int*>(sops)[i] = reinterpret_cast<const int*>(H.ops)[i];
        for (int i = threadIdx.x; i < H.n_rows; i += blockDim.x) srow[i] = H.rowptr[i];
        for (int i = threadIdx.x; i < H.n_ents; i += blockDim.x) {
            smask[i] = H.ent_mask[i];
            sval[i] = H.ent_val[i];
        }
        __syncthreads();
        H.ops = sops;
        H.rowptr = srow;
        H.ent_mask = smask;
        H.ent_val = sval;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * (blockDim.x >> 5) + warp;
    if (b >= a.B) return;
    unsigned char* wbase = sm.warp0 + warp * sm.warp_bytes;
    uint32_t* wsp = reinterpret_cast<uint32_t*>(wbase);
    C2<R>* wth = reinterpret_cast<C2<R>*>(wbase + 16);
    R* cre = reinterpret_cast<R*>(wbase + 16 + m.T * 2 * sizeof(R));
    C2<R>* cu = reinterpret_cast<C2<R>*>(wbase + 16 + m.T * 3 * sizeof(R));
    C2<R>* tn = reinterpret_cast<C2<R>*>(wbase + 16 + m.T * 5 * sizeof(R));
    PfStage* pst = reinterpret_cast<PfStage*>(wbase + eval_rbm_bytes(m.T, sizeof(R)));
    double2* pA = reinterpret_cast<double2*>(wbase + eval_rbm_bytes(m.T, sizeof(R)) + sizeof(PfStage));
    const C2<R>* W = Wsel<R>::get(m, sm.W32 ? sm.W32 : m.W32);
    uint32_t sp[4];
#pragma unroll
    for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * b + w];
    C2<double> th64[E];
    theta_fp64<E, double>(m, m.W64, sm.perm, lane, sp, th64);
    C2<R> th[E];
#pragma unroll
    for (int e = 0; e < E; e++) th[e] = mk<R>((R)th64[e].x, (R)th64[e].y);
    if (a.O) {
#pragma unroll
        for (int e = 0; e < E; e++)
            if (slot_valid(lane, e, m.T)) {
                const C2<double> t = ctanh_r<double>(th64[e].x, th64[e].y);
                tn[lane + 32 * e] = mk<R>((R)t.x, (R)t.y);
            }
    }
    stage<E, R>(m, sp, th, wsp, wth, lane);

    if (a.logpsi) {
        // log psi = bias + sum ln cosh theta (rbm_base.cpp:294-304,
        // rbm_symmetry.cpp:138-147)
        R re = 0, im = 0;
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (!slot_valid(lane, e, m.T)) continue;
            R r, ux, uy;
            lnc_full<R>(th[e].x, th[e].y, r, ux, uy);
            re += r;
            im += atan2(uy, ux);
        }
        re = warp_sum(re);
        im = warp_sum(im);
        double2 lpf = make_double2(0.0, 0.0);
        if constexpr (PF) lpf = pf_log_pfaffian(m.pf, sp[0], lane, pA);  // pfaffian.hpp:73-75
        if (lane == 0) {
            double bx = 0, by = 0;
            for (int i = 0; i < m.n_vb; i++) {
                double ssum = 0;
                if (m.symmetric) {
                    for (int s = 0; s < m.S; s++) ssum += spin_bit(sp, m.orbit[i * m.S + s]) ? -1.0 : 1.0;
                } else {
                    ssum = spin_bit(sp, i) ? -1.0 : 1.0;
                }
                bx += m.vb[i].x * ssum;
                by += m.vb[i].y * ssum;
            }
            a.logpsi[b] = make_double2(bx + (double)re - 0.69314718055994531 * m.T + lpf.x, by + (double)im + lpf.y);
        }
    }
    if constexpr (PF) {
        // X^{-1} of this configuration into the warp's matrix
        if (a.ratio || a.eloc || a.O) pf_fresh(m.pf, sp[0], lane, pA, *pst, pA + kPfMaxSites * kPfLd, kPfLd);
    }
    if (a.ratio) {
        LaneCache<R> cl{};
        if constexpr (sizeof(R) == 4) {
            cl = lane_cache<E>(wth, lane, m.T);
        } else {
#pragma unroll
            for (int e = 0; e < E; e++) {
                if (!slot_valid(lane, e, m.T)) continue;
                R r, ux, uy;
                lnc_full<R>(th[e].x, th[e].y, r, ux, uy);
                cre[lane + 32 * e] = r;
                cu[lane + 32 * e] = mk<R>(ux, uy);
            }
            __syncwarp();
        }
        int fl[6];
        const int nf = a.n_flips;
        for (int q = 0; q < nf; q++) fl[q] = a.flips[b * nf + q];
        R dre;
        C2<R> ph;
        uint32_t ks[E];
        entry_index<E>(m, lane, ks);
        ratio_terms<E, R>(ratio_dims(m), sm.perm, W, wth, wsp, fl, nf, cre, cu, cl, lane, dre, ph, ks);
        double2 lr = make_double2(0.0, 0.0);
        if constexpr (PF) {
            const double2 c2 = pf_ratio_any(m.pf, sp[0], fl, nf, lane, *pst, pA);
            lr = make_double2(0.5 * log(zabs2(c2)), atan2(c2.y, c2.x));
        }
        if (lane == 0) {
            const double2 bd = bias_delta_smem(m, wsp, fl, nf);
            a.ratio[b] = make_double2((double)dre + bd.x + lr.x, atan2((double)ph.y, (double)ph.x) + bd.y + lr.y);
        }
        __syncwarp();
    }
    if (a.eloc || a.O) {
        C2<R>* Orow = a.O ? reinterpret_cast<C2<R>*>(a.O) + (size_t)b * m.P : nullptr;
        if (sizeof(R) == 4 && sm.W32)
            evaluate<E, R, PF, true>(a.md, H, sm.perm, sm.inv, W, wth, wsp, cre, cu, tn, lane,
                               a.eloc ? a.eloc + b : nullptr, Orow, pst, pA);
        else
            evaluate<E, R, PF, false>(a.md, H, sm.perm, sm.inv, W, wth, wsp, cre, cu, tn, lane,
                               a.eloc ? a.eloc + b : nullptr, Orow, pst, pA);
        if constexpr (PF)
            if (Orow) pf_derivative(m.pf, sp[0], lane, pA, Orow + m.P_neural);
    }
}

// ---------------------------------------------------------------------------
// Learned proposals (learned-proposal extension; no reference counterpart).
// A move is one entry m of a dictionary of flip sets (every single site and
// every off-diagonal flip set of the Hamiltonian: x / y bonds of the Kitaev
// model, stars of the toric code).  The network maps the current
// configuration s to logits over the dictionary; the proposal is
// q(m|s) = (1 - eps) softmax(logits(s))_m + eps / D, and s' = s with m's
// sites flipped.  Every move is its own inverse, so the Metropolis-Hastings
// ratio is |psi(s')/psi(s)|^2 q(m|s') / q(m|s), q(m|s') from the network at
// s'.  The uniform part eps / D keeps every single-site flip possible
// (irreducible chain).  Random streams: Philox {128 move + 2 lane + k,
// epoch, chain, 3} for the Gumbel draws, {128 move + 64, ...} for the
// mixture draw and {move, epoch, chain, 4} for the acceptance.

// The proposal's log probability from a logits row: lanes hold m = lane +
// 32 i; returns log q(m) for the given m on every lane and log-sum-exp.
__device__ __forceinline__ float logq_of(const float* row, int D, int m, float eps, int lane) {
    float mx = -INFINITY;
    for (int i = lane; i < D; i += 32) mx = fmaxf(mx, row[i]);
    mx = warp_max(mx);
    float se = 0.f;
    for (int i = lane; i < D; i += 32) se += __expf(row[i] - mx);
    se = warp_sum(se);
    const float p = __expf(row[m] - mx) / se;
    return __logf((1.f - eps) * p + eps / (float)D);
}

// one warp per chain: draw m ~ q(.|s), record it, log q(m|s) and s'
__global__ void learned_propose(const LearnedArgs a) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    const int D = a.n_moves;
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < a.n_chains; c += nw) {
        const float* row = a.logits + (size_t)c * a.ldl;
        // Gumbel-max over the softmax part: argmax_m logit_m - ln(-ln u_m)
        float best = -INFINITY;
        int bm = 0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint4 r = philox4x32(make_uint4(128u * a.move + 2u * lane + k, epoch, (uint32_t)c, 3), key);
            const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int m = lane + 32 * (4 * k + q);
                if (m >= D) break;
                const float u = ((float)(rr[q] >> 8) + 0.5f) * (1.f / 16777216.f);
                const float g = row[m] - __logf(-__logf(u));
                if (g > best) {
                    best = g;
                    bm = m;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(kFull, best, o);
            const int om = __shfl_xor_sync(kFull, bm, o);
            if (ob > best || (ob == best && om < bm)) {
                best = ob;
                bm = om;
            }
        }
        // the uniform part of the mixture
        const uint4 r = philox4x32(make_uint4(128u * a.move + 64u, epoch, (uint32_t)c, 3), key);
        if (unit24<float>(r.x) < a.eps) bm = (int)pick(r.y, (uint32_t)D);
        const float lq = logq_of(row, D, bm, a.eps, lane);
        if (lane < 4) a.prop[4 * c + lane] = a.spins[4 * c + lane] ^ a.mmask[4 * bm + lane];
        if (lane == 0) {
            a.mv[c] = bm;
            a.qfw[c] = lq;
        }
    }
}

// Shared tables of the learned kernels: FP64 W, the symmetry table and the
// all-up theta (theta recomputed from the configuration), FP32 W with its
// zero row (flip rows of the ratio); each from global memory when the
// shared copies do not fit (smem_w 0).
struct LearnTabs {
    const double2* W64;
    const float2* W32;
    const uint8_t* perm;
    const double2* base;
    const float* bre;  // Re v[f mod n_vb], [n] = 0
};
__host__ __device__ inline int learned_smem_bytes(const MachineDev& m, int smem_w) {
    const int TP = padded_T(m.T);
    int b = align16(TP * 16) + align16((m.n + 1) * 4);
    if (smem_w) b += align16(m.n * m.nh * 16) + align16((m.n + 1) * m.nh * 8) + (m.symmetric ? align16(m.n * m.S) : 0);
    return b;
}
__device__ LearnTabs learned_tables(const MachineDev& m, unsigned char* smem, int smem_w) {
    const int TP = padded_T(m.T), tid = threadIdx.x, nt = blockDim.x;
    LearnTabs L{m.W64, m.W32, m.perm, nullptr, nullptr};
    int off = 0;
    double2* base = reinterpret_cast<double2*>(smem + off);
    off += align16(TP * 16);
    float* bre = reinterpret_cast<float*>(smem + off);
    off += align16((m.n + 1) * 4);
    if (smem_w) {
        double2* w64 = reinterpret_cast<double2*>(smem + off);
        off += align16(m.n * m.nh * 16);
        float2* w32 = reinterpret_cast<float2*>(smem + off);
        off += align16((m.n + 1) * m.nh * 8);
        for (int i = tid; i < m.n * m.nh; i += nt) w64[i] = m.W64[i];
        for (int i = tid; i < (m.n + 1) * m.nh; i += nt) w32[i] = i < m.n * m.nh ? m.W32[i] : make_float2(0.f, 0.f);
        L.W64 = w64;
        L.W32 = w32;
        if (m.symmetric) {
            uint8_t* p = smem + off;
            for (int i = tid; i < m.n * m.S; i += nt) p[i] = m.perm[i];
            L.perm = p;
        }
    }
    for (int i = tid; i <= m.n; i += nt) bre[i] = i < m.n ? (float)m.vb[i % m.n_vb].x : 0.f;
    __syncthreads();
    for (int t = tid; t < TP; t += nt) {
        double2 acc = make_double2(0, 0);
        if (t < m.T) {
            const int k = t % m.nh, sy = t / m.nh;
            acc = m.hb[k];
            for (int f = 0; f < m.n; f++) {
                const double2 w = L.W64[(m.symmetric ? (int)L.perm[f * m.S + sy] : f) * m.nh + k];
                acc.x += w.x;
                acc.y += w.y;
            }
        }
        base[t] = acc;
    }
    __syncthreads();
    L.base = base;
    L.bre = bre;
    return L;
}

// FP32 theta of a configuration (lane entries t = lane + 32 e, zero beyond
// T), recomputed in FP64 as the all-up table minus 2 W over the down spins.
// The lane's entries (k, s) of theta, t = lane + 32 e; -1 beyond T.
template <int E> struct LaneEnt {
    int k[E], s[E];
    __device__ LaneEnt(const MachineDev& m, int lane) {
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int t = lane + 32 * e;
            k[e] = t < m.T ? t % m.nh : -1;
            s[e] = t < m.T ? t / m.nh : 0;
        }
    }
};

template <int E>
__device__ __forceinline__ void learned_theta(const MachineDev& m, const LearnTabs& L, const LaneEnt<E>& le,
                                              const uint32_t (&sp)[4], int lane, float2 (&th)[E]) {
    // one pass over the down spins, every entry of the lane per spin
    double2 acc[E];
    int ro[E];  // row offset of the lane's entries in the symmetry table
#pragma unroll
    for (int e = 0; e < E; e++) {
        acc[e] = le.k[e] >= 0 ? L.base[lane + 32 * e] : make_double2(0, 0);
        ro[e] = m.symmetric ? le.s[e] : 0;
    }
#pragma unroll
    for (int wd = 0; wd < 4; wd++) {
        uint32_t bits = sp[wd];
        while (bits) {
            const int f = 32 * wd + __ffs(bits) - 1;
            bits &= bits - 1;
            const int fS = f * m.S;
#pragma unroll
            for (int e = 0; e < E; e++) {
                if (le.k[e] < 0) continue;
                const int row = m.symmetric ? (int)L.perm[fS + ro[e]] : f;
                const double2 w = L.W64[row * m.nh + le.k[e]];
                acc[e].x = fma(-2.0, w.x, acc[e].x);
                acc[e].y = fma(-2.0, w.y, acc[e].y);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < E; e++) th[e] = make_float2((float)acc[e].x, (float)acc[e].y);
}

// Re log psi(s with the move's flips)/psi(s): lane partial of the ln|cosh|
// difference (sum with sweep_sum) plus, on lane 0, the visible bias; tp
// receives theta of the moved configuration.
template <int E>
__device__ __forceinline__ float move_partial(const MachineDev& m, const LearnTabs& L, const LaneEnt<E>& le,
                                              const float2 (&th)[E], float s0, const uint32_t (&sp)[4], uint32_t fw0,
                                              uint32_t fw1, int lane, float2 (&tp)[E]) {
    const int nf = (fw1 >> 16) & 0xff;
#pragma unroll
    for (int e = 0; e < E; e++) tp[e] = th[e];
    float bias = 0.f;
    for (int q = 0; q < nf; q++) {
        const int f = q < 4 ? (fw0 >> (8 * q)) & 0xff : (fw1 >> (8 * (q - 4))) & 0xff;
        const float g = spin_bit(sp, f) ? 2.f : -2.f;  // -2 sigma_f
        bias = fmaf(g, L.bre[f], bias);
        const float2 G2 = make_float2(g, g);
#pragma unroll
        for (int e = 0; e < E; e++) {
            if (le.k[e] < 0) continue;
            const float2 w = L.W32[(m.symmetric ? (int)L.perm[f * m.S + le.s[e]] : f) * m.nh + le.k[e]];
            tp[e] = __ffma2_rn(G2, w, tp[e]);
        }
    }
    return lnc_sweep_sum<E>(tp) - s0 + (lane == 0 ? bias : 0.f);
}

// one warp per chain: log q(m|s') from the network at s', |psi'/psi|^2 in
// FP32 from the FP64-recomputed theta, Metropolis-Hastings test
template <int E>
__global__ void __launch_bounds__(256) learned_accept(const LearnedArgs a, int smem_w) {
    extern __shared__ __align__(16) unsigned char smem[];
    const LearnTabs L = learned_tables(a.m, smem, smem_w);
    const int lane = threadIdx.x & 31;
    const LaneEnt<E> le(a.m, lane);
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < a.n_chains; c += nw) {
        const int mv = a.mv[c];
        const float qrev = logq_of(a.logits + (size_t)c * a.ldl, a.n_moves, mv, a.eps, lane);
        uint32_t sp[4];
#pragma unroll
        for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * c + w];
        float2 th[E], tp[E];
        float2* tc = a.theta ? a.theta + (size_t)c * (32 * E) + lane : nullptr;
        if (tc) {
#pragma unroll
            for (int e = 0; e < E; e++) th[e] = tc[32 * e];
        } else {
            learned_theta<E>(a.m, L, le, sp, lane, th);
        }
        const float s0 = lnc_sweep_sum<E>(th);
        const float d =
            sweep_sum(move_partial<E>(a.m, L, le, th, s0, sp, a.mflip[2 * mv], a.mflip[2 * mv + 1], lane, tp));
        const uint4 r = philox4x32(make_uint4(a.move, epoch, (uint32_t)c, 4), key);
        // accept with min(1, |psi'/psi|^2 q(m|s') / q(m|s))
        const bool acc = __logf(unit24<float>(r.x) + 0x1p-25f) < 2.f * d + qrev - a.qfw[c];
        if (lane < 4 && acc) a.spins[4 * c + lane] = a.prop[4 * c + lane];
        if (tc && acc) {
#pragma unroll
            for (int e = 0; e < E; e++) tc[32 * e] = tp[e];
        }
        if (lane == 0) {
            a.n_acc[c] += acc ? 1u : 0u;
            a.n_try[c] += 1u;
        }
    }
}

// Training targets of the proposal network at configurations spins[0..B):
// t_m proportional to min(1, |psi(s with move m)/psi(s)|^2), a locally
// balanced choice (g(r) = min(1, r) satisfies g(r) = r g(1/r)), so that
// moves likely to be accepted get most of the proposal probability.
template <int E>
__global__ void __launch_bounds__(256) learned_targets(const LearnedArgs a, int smem_w) {
    extern __shared__ __align__(16) unsigned char smem[];
    const LearnTabs L = learned_tables(a.m, smem, smem_w);
    const int lane = threadIdx.x & 31;
    const LaneEnt<E> le(a.m, lane);
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int D = a.n_moves;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < a.B; b += nw) {
        uint32_t sp[4];
#pragma unroll
        for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * b + w];
        float2 th[E];
        learned_theta<E>(a.m, L, le, sp, lane, th);
        const float s0 = lnc_sweep_sum<E>(th);
        float lg[8];  // min(0, 2 ln|psi'/psi|) of moves lane + 32 i
#pragma unroll
        for (int i = 0; i < 8; i++) lg[i] = -INFINITY;
        // moves in groups of MG: their partial sums are independent, so the
        // transcendentals and the warp reductions of a group overlap (the
        // same per-move arithmetic and reduction)
        constexpr int MG = 4;
        for (int mv0 = 0; mv0 < D; mv0 += MG) {
            float d[MG];
#pragma unroll
            for (int g = 0; g < MG; g++) {
                const int mv = min(mv0 + g, D - 1);
                float2 tp[E];
                d[g] = move_partial<E>(a.m, L, le, th, s0, sp, a.mflip[2 * mv], a.mflip[2 * mv + 1], lane, tp);
            }
#pragma unroll
            for (int g = 0; g < MG; g++) {
                const float dg = sweep_sum(d[g]);
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (mv0 + g == lane + 32 * i) lg[i] = fminf(0.f, 2.f * dg);
            }
        }
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 8; i++) mx = fmaxf(mx, lg[i]);
        mx = warp_max(mx);
        float se = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) se += lane + 32 * i < D ? __expf(lg[i] - mx) : 0.f;
        se = warp_sum(se);
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (lane + 32 * i < D) a.targets[(size_t)b * D + lane + 32 * i] = __expf(lg[i] - mx) / se;
    }
}

// theta of every chain's configuration into a.theta (FP64 recompute,
// rounded to FP32): the starting point of learned moves that run without a
// sweep before them.
template <int E>
__global__ void __launch_bounds__(256) learned_theta_init(const LearnedArgs a, int smem_w) {
    extern __shared__ __align__(16) unsigned char smem[];
    const LearnTabs L = learned_tables(a.m, smem, smem_w);
    const int lane = threadIdx.x & 31;
    const LaneEnt<E> le(a.m, lane);
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < a.n_chains; c += nw) {
        uint32_t sp[4];
#pragma unroll
        for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * c + w];
        float2 th[E];
        learned_theta<E>(a.m, L, le, sp, lane, th);
        float2* tc = a.theta + (size_t)c * (32 * E) + lane;
#pragma unroll
        for (int e = 0; e < E; e++) tc[32 * e] = th[e];
    }
}

// Fresh chains (Philox stream 1, as chain_start) when the control word asks
// for initialisation: for epochs whose moves run without a sweep kernel.
__global__ void init_chains(uint32_t* spins, int n, int n_chains, const uint32_t* ctl, uint64_t seed) {
    if (!ctl[1]) return;
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_chains; c += gridDim.x * blockDim.x) {
        const uint4 r = philox4x32(make_uint4(0, ctl[0], (uint32_t)c, 1), key);
        const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int lo = 32 * w;
            const uint32_t mask = n >= lo + 32 ? 0xffffffffu : (n > lo ? ((1u << (n - lo)) - 1) : 0u);
            spins[4 * c + w] = rw[w] & mask;
        }
    }
}

cudaError_t launch_init_chains(uint32_t* spins, int n, int n_chains, const uint32_t* ctl, uint64_t seed,
                               cudaStream_t st) {
    init_chains<<<std::min(148 * 4, (n_chains + 255) / 256), 256, 0, st>>>(spins, n, n_chains, ctl, seed);
    return cudaGetLastError();
}

__global__ void record_kernel(const uint32_t* spins, int n_chains, int spc, int j, uint32_t* samples) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 4 * n_chains; t += gridDim.x * blockDim.x) {
        const int c = t >> 2, w = t & 3;
        samples[4 * ((size_t)c * spc + j) + w] = spins[t];
    }
}

__global__ void learned_rate(const uint32_t* n_acc, const uint32_t* n_try, int n, double* out) {
    __shared__ double ra[32], rt[32];
    double sa = 0, st = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        sa += n_acc[i];
        st += n_try[i];
    }
    sa = warp_sum(sa);
    st = warp_sum(st);
    if ((threadIdx.x & 31) == 0) {
        ra[threadIdx.x >> 5] = sa;
        rt[threadIdx.x >> 5] = st;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double A = 0, Tt = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            A += ra[w];
            Tt += rt[w];
        }
        *out = Tt > 0 ? A / Tt : 0.0;
    }
}

cudaError_t launch_learned_propose(const LearnedArgs& a, cudaStream_t st) {
    learned_propose<<<std::min(148 * 8, (a.n_chains + 7) / 8), 256, 0, st>>>(a);
    return cudaGetLastError();
}

static cudaError_t launch_learned_kernel(const LearnedArgs& a, int which, int rows, cudaStream_t st) {
    const int full = learned_smem_bytes(a.m, 1);
    const int smem_w = full <= 160 * 1024;
    const int smem = learned_smem_bytes(a.m, smem_w);
    const void* fn = nullptr;
#define RBMNQS_LK(E)                                                                                 \
    fn = which == 0   ? reinterpret_cast<const void*>(learned_accept<E>)                          \
         : which == 1 ? reinterpret_cast<const void*>(learned_targets<E>)                         \
                      : reinterpret_cast<const void*>(learned_theta_init<E>);
    switch (elements_per_lane(a.m.T)) {
        case 1: RBMNQS_LK(1) break;
        case 2: RBMNQS_LK(2) break;
        case 4: RBMNQS_LK(4) break;
        case 8: RBMNQS_LK(8) break;
        case 16: RBMNQS_LK(16) break;
        default: return cudaErrorInvalidValue;
    }
#undef RBMNQS_LK
    cudaError_t e = ensure_dynamic_smem(fn, smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int blocks = std::max(1, std::min((rows + 7) / 8, 2 * sms));
    LearnedArgs aa = a;
    int flag = smem_w;
    void* args[] = {&aa, &flag};
    return cudaLaunchKernel(fn, dim3(blocks), dim3(256), args, smem, st);
}

cudaError_t launch_learned_accept(const LearnedArgs& a, cudaStream_t st) {
    return launch_learned_kernel(a, 0, a.n_chains, st);
}

cudaError_t launch_learned_targets(const LearnedArgs& a, cudaStream_t st) {
    if (a.B <= 0) return cudaSuccess;
    if (a.n_moves > 256) return cudaErrorInvalidValue;
    return launch_learned_kernel(a, 1, a.B, st);
}

cudaError_t launch_learned_theta(const LearnedArgs& a, cudaStream_t st) {
    if (!a.theta) return cudaErrorInvalidValue;
    return launch_learned_kernel(a, 2, a.n_chains, st);
}

cudaError_t launch_record(const uint32_t* spins, int n_chains, int spc, int j, uint32_t* samples, cudaStream_t st) {
    record_kernel<<<std::min(148 * 4, (4 * n_chains + 255) / 256), 256, 0, st>>>(spins, n_chains, spc, j, samples);
    return cudaGetLastError();
}

cudaError_t launch_learned_rate(const uint32_t* n_acc, const uint32_t* n_try, int n_chains, double* out,
                                cudaStream_t st) {
    learned_rate<<<1, 1024, 0, st>>>(n_acc, n_try, n_chains, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Special-function-unit throughput probe: each thread runs `iters` rounds of
// four independent ex2/lg2/sin/cos chains.  Used as the measured peak for
// the sampler's roofline (its ln cosh work is MUFU-bound, not HBM/tensor).
__global__ void mufu_probe(float* out, int iters) {
    float a = threadIdx.x * 1e-3f, b = 0.5f + blockIdx.x * 1e-4f, c = 0.25f, d = 0.75f;
    for (int i = 0; i < iters; i++) {
        a = __expf(-a) + 0.1f;
        b = __logf(b + 1.0f);
        c = __sinf(c) + 0.2f;
        d = __cosf(d);
    }
    if (a + b + c + d == 12345.0f) out[0] = a;  // keeps the chains live
}

cudaError_t launch_mufu_probe(float* out, int iters, int blocks, cudaStream_t st) {
    mufu_probe<<<blocks, 256, 0, st>>>(out, iters);
    return cudaGetLastError();
}

// Next epoch: counter + 1, chains re-initialised only in reference mode.
__global__ void advance_ctl(uint32_t* ctl, int reinit) {
    ctl[0] += 1;
    ctl[1] = reinit ? 1u : 0u;
}

cudaError_t launch_advance(uint32_t* ctl, int reinit, cudaStream_t st) {
    advance_ctl<<<1, 1, 0, st>>>(ctl, reinit);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
int elements_per_lane(int T) {
    const int e = (T + 31) / 32;
    if (e <= 1) return 1;
    if (e <= 2) return 2;
    if (e <= 4) return 4;
    if (e <= 8) return 8;
    if (e <= 16) return 16;
    return -1;
}

int sampler_smem_bytes(const MachineDev& m, int fp64, int warps, const SmemPlan& plan, int n_bonds) {
    return table_bytes(m, fp64, plan, n_bonds) + warps * sweep_warp_bytes(m.T, fp64 ? 8 : 4, m.pf.n > 0);
}

int ham_stage_bytes(const HamDev& H) {
    if (H.n_rows <= 0) return 0;
    const int b = align16(H.n_ops * (int)sizeof(OpDev)) + align16(H.n_rows * 4) + align16(H.n_ents * 4) +
                  align16(H.n_ents * 16);
    return b <= 48 * 1024 ? b : 0;
}

int eval_smem_bytes(const MachineDev& m, int fp64, int warps, const SmemPlan& plan) {
    return table_bytes(m, fp64, plan, 0) + warps * eval_warp_bytes(m.T, fp64 ? 8 : 4, m.pf.n > 0);
}

template <int E, typename R, int FAST, bool PF> static const void* sampler_fn() {
    return reinterpret_cast<const void*>(sampler_kernel<E, R, FAST, PF>);
}

// The Pfaffian variants exist for theta tables up to 128 entries (32 sites,
// alpha <= 4); they take the general (non-table) sweep.
static const void* pick_sampler(int E, int fp64, int exp_table, int pf, int gather, int pair) {
    if (pair && !fp64 && !pf && exp_table) {
        if (E == 1) return sampler_fn<1, float, 3, false>();
        if (E == 2) return sampler_fn<2, float, 3, false>();
        if (E == 4) return sampler_fn<4, float, 3, false>();
        return nullptr;
    }
    if (pf) {
#define RBMNQS_PICK_PF(EE) \
    if (E == EE) return fp64 ? sampler_fn<EE, double, 0, true>() : sampler_fn<EE, float, 0, true>();
        RBMNQS_PICK_PF(1) RBMNQS_PICK_PF(2) RBMNQS_PICK_PF(4)
#undef RBMNQS_PICK_PF
        return nullptr;
    }
#define RBMNQS_PICK(EE)                                                   \
    if (E == EE) {                                                        \
        if (fp64) return sampler_fn<EE, double, 0, false>();              \
        if (exp_table) return sampler_fn<EE, float, 1, false>();          \
        return gather ? sampler_fn<EE, float, 2, false>() : sampler_fn<EE, float, 0, false>(); \
    }
    RBMNQS_PICK(1) RBMNQS_PICK(2) RBMNQS_PICK(4) RBMNQS_PICK(8) RBMNQS_PICK(16)
#undef RBMNQS_PICK
    return nullptr;
}

static cudaError_t plan_sampler_impl(const MachineDev& m, int fp64, int n_chains, int n_bonds, SamplerShape* out,
                                     int max_wpb, int pair_mode) {
    const int E = elements_per_lane(m.T);
    if (E < 0) return cudaErrorInvalidValue;
    int dev = 0, sms = 0, smem_max = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int budget = smem_max - 8 * 1024;
    const int TP = 32 * E;
    SmemPlan pl{};
    pl.lane_entries = E;
    // FP32 expanded-table path when the table fits; its theta recompute uses
    // the FP64 expanded table when that fits too, else FP64 W
    const int pf = m.pf.n > 0;
    pl.use_u = !fp64 && !pf && (m.n + 1) * TP * 8 <= 64 * 1024;
    // FP32 without the expanded table: gathered flip rows (W32 with its pad
    // row in shared memory when it fits, else from L2)
    pl.gather = !fp64 && !pf && !pl.use_u;
    pl.wg = pl.gather && (m.n + 1) * m.nh * 8 <= 64 * 1024;
    pl.lane_rows = pl.gather && pl.wg && m.symmetric && 32 % m.nh == 0 && m.T == TP && E >= 4;
    pl.u64 = pl.use_u && m.n * TP * 16 <= 96 * 1024;
    pl.w32 = !fp64 && !pl.use_u && !pl.gather && m.n * m.nh * 8 <= 64 * 1024;
    pl.w64 = m.n * m.nh * 16 <= 32 * 1024;
    pl.bonds = n_bonds > 0 && n_bonds * 8 <= 8 * 1024;
    // two chains per warp for small configurations with both expanded
    // tables (entries per lane 2 E <= 8): fewer instructions per chain but
    // half the resident warps and more registers per thread, which measured
    // slower on the 32-spin alpha = 4 shape at 4096 and 16384 chains; so
    // only on request (pair_mode 1, e.g. by the autotuner)
    pl.pair = pl.use_u && pl.u64 && m.n <= 32 && E <= 4 && pair_mode == 1;
    const void* fn = pick_sampler(E, fp64, pl.use_u, pf, pl.gather, pl.pair);
    if (!fn) return cudaErrorInvalidValue;
    cudaFuncAttributes fa;
    err = cudaFuncGetAttributes(&fa, fn);
    if (err != cudaSuccess) return err;
    // warps per block: enough for one block per SM to hold every chain,
    // limited by the kernel's thread bound, registers and shared memory
    const int units = pl.pair ? (n_chains + 1) / 2 : n_chains;  // warps' work items
    const int want = (units + sms - 1) / sms;
    int wpb = fa.maxThreadsPerBlock / 32;
    const int regs = fa.numRegs > 0 ? fa.numRegs : 64;
    const int reg_warps = 65536 / (regs * 32);
    if (wpb > reg_warps) wpb = reg_warps;
    if (wpb > want) wpb = want;
    if (max_wpb > 0 && wpb > max_wpb) wpb = max_wpb;
    if (wpb < 1) wpb = 1;
    if (pl.u64 && sampler_smem_bytes(m, fp64, wpb, pl, n_bonds) > budget) {
        if (pl.pair) return plan_sampler_impl(m, fp64, n_chains, n_bonds, out, max_wpb, 0);
        pl.u64 = 0;
    }
    while (wpb > 1 && sampler_smem_bytes(m, fp64, wpb, pl, n_bonds) > budget) wpb--;
    const int smem = sampler_smem_bytes(m, fp64, wpb, pl, n_bonds);
    if (smem > budget) return cudaErrorInvalidValue;
    err = ensure_dynamic_smem(fn, smem);
    if (err != cudaSuccess) return err;
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * wpb, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    long blocks = ((long)units + wpb - 1) / wpb;
    if (blocks > (long)sms * per_sm) blocks = (long)sms * per_sm;
    if (pf) {
        // the Pfaffian sweep's Gauss-Jordan scratch, tables and spills live
        // in L1: ask for no more shared memory than the resident blocks use
        // (1 KB reserved per block), the rest of the SM's 256 KB stays L1.
        // The hint is a whole percentage, rounded down: the driver raises it
        // to the smallest carve-out that the launch needs (rounding up can
        // step past a carve-out that fits, e.g. 164 KB at 72 %).
        int sm_max = 0;
        cudaDeviceGetAttribute(&sm_max, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        const long resident = std::min<long>(per_sm, (blocks + sms - 1) / sms);
        const long need = resident * (smem + 1024);
        if (sm_max > 0) {
            const int pct = (int)std::min<long>(100, need * 100 / sm_max);
            err = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
            if (err != cudaSuccess) return err;
        }
    }
    out->plan = pl;
    out->warps_per_block = wpb;
    out->blocks = (int)blocks;
    out->smem = smem;
    return cudaSuccess;
}

// Does the screened sweep pay for a launch of `sweeps` sweeps?  Its start (tables, z
// of every entry) costs 0.2 to 0.7 ms at 512 entries, and its warps are 16 per SM
// where the sums have up to 28, so it needs chains and sweeps to earn that back.
// FP32, time over the sums' kernel, 512 entries of 128 spins, Kitaev / toric code /
// basic machine.  First line: weights of spread 0.035 (5, 30, 15 % accepted), by which
// the lines are drawn, second: 0.02, untrained (70 % accepted, the screen's worst).
//   chains per SM, sweeps  64, 1            14, 1            14, 4            7, 16
//                    0.67 1.08  -     0.80 1.25 0.64   0.54 0.81 0.52   0.68 0.97 0.77
//                    0.93 1.43  -     1.09 1.58 0.72   0.82 1.22 0.62   1.03 1.38 0.91
//   and basic machines at 7, 8: 0.83 / 1.04, at 1, 16: 0.90 / 1.02; symmetric ones at
//   1, 16: 0.93 1.15 / 1.23 1.65.
// FP64: 0.02 to 0.7, one sweep included, but for the smallest machines' single
// sweep (8 sites: 1.0 to 1.4).
static bool screen_pays(const MachineDev& m, int fp64, int n_chains, int sms, int sweeps) {
    if (fp64) return sweeps > 1 || m.T > 32;
    const int per_sm = (n_chains + sms - 1) / sms;
    const int least = per_sm >= 64   ? 1
                      : per_sm >= 14 ? (m.symmetric ? 4 : 1)
                      : per_sm >= 4  ? (m.symmetric ? 16 : 8)
                                     : (m.symmetric ? 32 : 16);
    return sweeps >= least;
}

cudaError_t plan_sampler(const MachineDev& m, int fp64, int n_chains, int n_bonds, SamplerShape* out, int max_wpb,
                         int pair_mode, int sweeps) {
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (m.pf.n == 0 && (fp64 || pair_mode != 1) && screen_pays(m, fp64, n_chains, sms, sweeps) &&
        plan_screen(m, fp64, n_chains, n_bonds, max_wpb, out, &err)) {
        if (err != cudaSuccess) return err;
        SamplerShape ex{};
        err = plan_sampler_impl(m, fp64, n_chains, n_bonds, &ex, max_wpb, 0);
        out->exact = ex;
        return err;
    }
    return plan_sampler_impl(m, fp64, n_chains, n_bonds, out, max_wpb, pair_mode);
}

cudaError_t ensure_dynamic_smem(const void* fn, int bytes) {
    // the attribute belongs to the kernel on the current device: cache it per
    // (device, kernel) so that a second device gets its own setting
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> set;
    std::lock_guard<std::mutex> lk(mu);
    int dev = 0;
    const cudaError_t de = cudaGetDevice(&dev);
    if (de != cudaSuccess) return de;
    int& cur = set[{dev, fn}];
    if (bytes <= cur) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

// The FP32 expanded-table (one chain per warp) and gather paths store
// theta_out; the FP64, screened, Pfaffian and two-chain paths do not.
bool sampler_writes_theta(const MachineDev& m, int fp64, const SamplerShape& sh) {
    return !fp64 && m.pf.n == 0 && !sh.plan.pair && !sh.plan.screen && (sh.plan.use_u || sh.plan.gather);
}

cudaError_t launch_sampler(const SamplerArgs& a0, int fp64, const SamplerShape& sh, cudaStream_t st) {
    SamplerArgs a = a0;
    a.plan = sh.plan;
    SweepShape ex = sh;
    if (sh.plan.screen) {
        const cudaError_t e = launch_screen(a, fp64, sh, st);
        if (e != cudaSuccess) return e;
        ex = sh.exact;
        a.plan = ex.plan;
        a.gate = a.screen_off;
    }
    const int E = elements_per_lane(a.m.T);
    const void* fn = pick_sampler(E, fp64, ex.plan.use_u, a.m.pf.n > 0, ex.plan.gather, ex.plan.pair);
    if (!fn) return cudaErrorInvalidValue;
    const cudaError_t e = ensure_dynamic_smem(fn, ex.smem);
    if (e != cudaSuccess) return e;
    void* args[] = {&a};
    return cudaLaunchKernel(fn, dim3(ex.blocks), dim3(32 * ex.warps_per_block), args, ex.smem, st);
}

template <int E, typename R, bool PF>
static cudaError_t launch_e2(const EvalArgs& a, int wpb, cudaStream_t st) {
    const int smem = eval_smem_bytes(a.m, sizeof(R) == 8, wpb, a.plan);
    cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(eval_kernel<E, R, PF>), smem);
    if (err != cudaSuccess) return err;
    const int blocks = (a.B + wpb - 1) / wpb;
    eval_kernel<E, R, PF><<<blocks, 32 * wpb, smem, st>>>(a);
    return cudaGetLastError();
}

template <int E, typename R>
static cudaError_t launch_e(const EvalArgs& a, int wpb, cudaStream_t st) {
    if (a.m.pf.n > 0) {
        if constexpr (E <= 4) return launch_e2<E, R, true>(a, wpb, st);
        return cudaErrorInvalidValue;
    }
    return launch_e2<E, R, false>(a, wpb, st);
}

#define RBMNQS_DISPATCH(FN, ARGS)                                            \
    switch (elements_per_lane(ARGS.m.T)) {                                   \
        case 1: return fp64 ? FN<1, double>(ARGS, wpb, st) : FN<1, float>(ARGS, wpb, st);   \
        case 2: return fp64 ? FN<2, double>(ARGS, wpb, st) : FN<2, float>(ARGS, wpb, st);   \
        case 4: return fp64 ? FN<4, double>(ARGS, wpb, st) : FN<4, float>(ARGS, wpb, st);   \
        case 8: return fp64 ? FN<8, double>(ARGS, wpb, st) : FN<8, float>(ARGS, wpb, st);   \
        case 16: return fp64 ? FN<16, double>(ARGS, wpb, st) : FN<16, float>(ARGS, wpb, st); \
        default: return cudaErrorInvalidValue;                               \
    }

static cudaError_t launch_eval_warp(const EvalArgs& a, int fp64, int wpb, cudaStream_t st) {
    RBMNQS_DISPATCH(launch_e, a)
}

// FP32 E_loc, O_k and log psi of symmetric machines go to the product kernel
// (eloc_sym.cu), E_loc and O_k of the others to the term-table kernel (eloc.cu) when
// it supports the machine; ratios, FP64, the Pfaffian factor and the other log
// psi to eval_kernel.
cudaError_t launch_eval(const EvalArgs& a, int fp64, int wpb, cudaStream_t st) {
    if (!fp64 && !a.ratio && a.tt.terms && a.m.pf.n == 0) {
        const cudaError_t es = a.B == 0 ? cudaSuccess : launch_eloc_sym(a, st);
        if (es != cudaErrorNotSupported) return es;
    }
    if (!fp64 && (a.eloc || a.O) && !a.ratio && a.tt.terms && a.m.pf.n == 0) {
        EvalArgs f = a;
        f.logpsi = nullptr;
        const cudaError_t e = launch_eloc_fast(f, st);
        if (e == cudaSuccess) {
            if (!a.logpsi) return cudaSuccess;
            EvalArgs r = a;
            r.eloc = nullptr;
            r.O = nullptr;
            return launch_eval_warp(r, fp64, wpb, st);
        }
        if (e != cudaErrorNotSupported) return e;
    }
    return launch_eval_warp(a, fp64, wpb, st);
}


// ---------------------------------------------------------------------------
// Batch sweep (several sessions, one launch)
bool sampler_batch_plan(const MachineDev& m, int fp64, int n_chains, int n_bonds, BatchSweepDesc* d, int* smem) {
    const int E = elements_per_lane(m.T);
    if (fp64 || m.pf.n > 0 || E > 8) return false;
    SamplerShape sh{};
    if (plan_sampler(m, 0, n_chains, n_bonds, &sh, kBatchSweepWarps, 0, 0) != cudaSuccess) return false;
    SmemPlan pl = sh.plan;
    pl.pair = 0;
    if (!pl.use_u && !pl.gather) return false;
    int dev = 0, smem_max = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int budget = smem_max - 8 * 1024 - (int)sizeof(SamplerArgs);
    int bytes = sampler_smem_bytes(m, 0, kBatchSweepWarps, pl, n_bonds);
    if (bytes > budget && pl.u64) {  // without the FP64 expanded table
        pl.u64 = 0;
        bytes = sampler_smem_bytes(m, 0, kBatchSweepWarps, pl, n_bonds);
    }
    if (bytes > budget) return false;
    d->a.plan = pl;
    d->E = E;
    d->path = pl.use_u ? 0 : 1;
    d->blocks = (n_chains + kBatchSweepWarps - 1) / kBatchSweepWarps;
    *smem = bytes;
    return true;
}

cudaError_t launch_sampler_batch(int E, const BatchSweepDesc* desc_dev, int nprob, int blocks, int smem,
                                 cudaStream_t st) {
    if (nprob < 1 || blocks < 1) return cudaErrorInvalidValue;
    const void* fn = nullptr;
    switch (E) {
        case 1: fn = reinterpret_cast<const void*>(sampler_batch_kernel<1>); break;
        case 2: fn = reinterpret_cast<const void*>(sampler_batch_kernel<2>); break;
        case 4: fn = reinterpret_cast<const void*>(sampler_batch_kernel<4>); break;
        case 8: fn = reinterpret_cast<const void*>(sampler_batch_kernel<8>); break;
        default: return cudaErrorInvalidValue;
    }
    cudaError_t e = ensure_dynamic_smem(fn, smem);
    if (e != cudaSuccess) return e;
    const BatchSweepDesc* d = desc_dev;
    int np = nprob;
    void* args[] = {&d, &np};
    return cudaLaunchKernel(fn, dim3(blocks), dim3(32 * kBatchSweepWarps), args, smem, st);
}

}  // namespace rbmnqs
