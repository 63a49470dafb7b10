// eloc_sym.cu -- local energy, log-derivatives and log psi of symmetric machines
// in FP32 (local_op.cpp:31-60, rbm_base.cpp:194-217, rbm_symmetry.cpp:97-147), one
// warp per configuration, psi ratios as products without transcendentals.
// log psi is summed in FP64 from the terms of tanh theta.
//
// With z = exp(-2 theta) and delta = -2 sum_f sigma_f W[P_s(f), k] over a term's
// flips, cosh(theta + delta) / cosh(theta) = exp(-delta) (z + q) / (1 + z),
// q = exp(2 delta).  So
//   psi'/psi = [prod_e 1 / (1 + z_e)] [prod_e (z_e + q_e)]
//              exp(sum_f sigma_f (2 sum_e W_fe - 2 v_f)):
// the first product is formed once per configuration (FP64), the last factor
// from one number per site, and a term costs one complex addition and one
// complex multiplication per theta entry (six FMA-pipe operations, packed in
// pairs) instead of an ex2, a sine and a cosine.  q depends on the spins of
// the flipped sites (2^nf patterns), the hidden unit k and the tuple of W
// rows (P_s(f_0), P_s(f_1), ...); under the lattice symmetries the terms share
// few distinct tuples (the 128-spin Kitaev lattice: 256 for 128 terms x 128
// symmetries), so every block holds the whole table q[pattern][tuple][k] in
// shared memory.
//
// The products carry their exponents as integers: a lane's product over its
// entries is scaled to a leading one, mantissas multiply and exponents add in
// the warp's butterfly, and exp() joins them in FP64, 32 terms at a time.
// Configurations with Re sum theta < 0 take -theta (cosh is even), which keeps
// |z| below one on average.
//
// Range.  z and q are each rounded once from FP64, over their whole range (where |Re
// theta| > 7, z is exp(-2 theta) itself, not 1 - (1 - z): a flip that cancels a
// saturated theta leaves z + q as small as z).  A lane multiplies its entries in two chains of E /
// 2; a chain that ends above 2^-116 F^(E/2 - 1), F a bound on |z + q| over the
// configuration's entries and the block's table, has not been below 2^-116 on its
// way, and one that overflowed ends as infinity or NaN.  A configuration with a
// chain outside that range takes term_product_scaled() from that term on, which
// scales after every factor.  Factors that FP32 does not hold, or that are zero
// (|z| > e^68, |4 W| > 60 in a row, q outside 2^+-86, non-finite weights) send
// the configuration to ratio_slow(), the ln cosh sums in FP64.
//
// Layout as in eloc.cuh: groups of KB hidden units with one symmetry index s,
// lane l owns the groups l + 32 j; entries in pairs, real and imaginary parts
// apart.  Bound: shared-memory wavefronts (ncu: 82 % of peak, 86 % with O_k; 10.9
// thousand per configuration of 128 spins and 512 entries, 4.9 of them the q rows,
// 4.3 the FP64 recompute of theta, and 2.5 for O_k), the FMA pipe at 35 %, issue
// 53 %.  Measured on 262144 configurations of 128 spins, 512 entries, with O_k: 29.3
// ms by ln cosh sums (eloc.cuh, which stays for basic machines, whose flipped rows
// are not shared, and for tables beyond shared memory), 13.9 ms here; 4096 of 32
// spins, 128 entries: 0.061 and 0.055 ms.  8192 of 128 spins whose products are all
// rescaled (weights of spread 0.3) 1.03 ms, as by ln cosh sums; all in ratio_slow()
// 10 ms.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "eloc.cuh"

namespace rbmnqs {
namespace {

using namespace eloc;

struct SymLayout {
    int w64, perm, inv, cls, q, base, terms, diag, vals, vb, site, qmax, warp0, warp_bytes, total;
    int ws64;    // row stride of the FP64 W copy (double2)
    int qs, qp;  // row and pattern strides of q (bytes)
};

// Shared-memory carve-up, the same arithmetic on host and device.  The warps'
// scratch (configuration, tanh theta [T], spins as +-1 [n]) first holds the
// single-site factors exp(-+4 W) from which q is built.
__host__ __device__ inline SymLayout sym_layout(const MachineDev& m, const TermTable& tt, int kb, int warps,
                                                bool with_O) {
    SymLayout L{};
    L.ws64 = w64_stride(m.nh);
    L.qs = 4 * w32_stride(m.nh, kb, true);
    L.qp = (tt.n_cls + 1) * L.qs;
    L.warp_bytes = a16(16 + m.T * 8 + m.n * 4);
    int off = 0;
    auto take = [&](int bytes) {
        const int at = off;
        off += a16(bytes);
        return at;
    };
    L.w64 = take(m.n * L.ws64 * 16);
    L.q = take(L.qp << tt.nf_max);
    L.cls = take(2 * tt.n_terms * (m.S + 1));
    L.perm = take(m.n * m.S);
    L.inv = take(with_O ? m.n * m.S : 0);
    L.base = take(m.T * 16);
    L.terms = take((tt.n_terms + tt.n_diag) * (int)sizeof(TermDev));
    L.diag = L.terms + tt.n_terms * (int)sizeof(TermDev);
    L.vals = take(tt.n_vals * 16);
    L.vb = take(m.n_vb * 16);
    L.site = take((m.n + 1) * 16);
    L.qmax = take(4);
    L.warp0 = off;
    const int scratch = warps * L.warp_bytes, factors = m.n * m.nh * 32;
    off += a16(scratch > factors ? scratch : factors);
    L.total = off;
    return L;
}

struct SymTabs {
    const double2 *W64, *base, *vals, *vb;
    const uint8_t* perm;
    const TermDev* terms;
    int ws64;
};

// E_loc's off-diagonal part by ln cosh sums in FP64 from the weights, for
// configurations outside the range of the products.  th: the warp's scratch,
// left holding theta (FP32).
__device__ __noinline__ double2 ratio_slow(const MachineDev* __restrict__ md, int n_terms, const SymTabs& t,
                                           uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, float2* th, int lane) {
    const MachineDev& m = *md;
    const uint32_t sp[4] = {s0, s1, s2, s3};
    double cre = 0;
    double2 cu = make_double2(1, 0);
    for (int e = lane; e < m.T; e += 32) {
        const int k = e % m.nh, s = e / m.nh;
        double2 x = t.base[e];
        for (int f = 0; f < m.n; f++)
            if (sbit(sp, f)) {
                const double2 w = t.W64[t.perm[f * m.S + s] * t.ws64 + k];
                x.x = fma(-2.0, w.x, x.x);
                x.y = fma(-2.0, w.y, x.y);
            }
        th[e] = make_float2((float)x.x, (float)x.y);
        double re, ux, uy;
        lnc_full<double>(th[e].x, th[e].y, re, ux, uy);
        cre += re;
        cu = cmul(cu, make_double2(ux, uy));
    }
    double ex = 0, ey = 0;
    for (int ti = 0; ti < n_terms; ti++) {
        const TermDev tm = t.terms[ti];
        const int nf = term_nf(tm);
        const double2 val = t.vals[tm.voff + term_loc(tm, sp)];
        if (val.x == 0.0 && val.y == 0.0) continue;  // uniform
        double re = -cre;
        double2 u = make_double2(cu.x, -cu.y);
        for (int e = lane; e < m.T; e += 32) {
            const int k = e % m.nh, s = e / m.nh;
            double x = th[e].x, y = th[e].y;
            for (int q = 0; q < nf; q++) {
                const int f = term_flip(tm, q);
                const double g = sbit(sp, f) ? 2.0 : -2.0;
                const double2 w = t.W64[t.perm[f * m.S + s] * t.ws64 + k];
                x = fma(g, w.x, x);
                y = fma(g, w.y, y);
            }
            double r1, ux, uy;
            lnc_full<double>(x, y, r1, ux, uy);
            re += r1;
            u = cmul(u, make_double2(ux, uy));
        }
        re = warp_sum(re);
        u = warp_cprod(u);
        double bx = 0, by = 0;
        for (int q = 0; q < nf; q++) {
            const int f = term_flip(tm, q);
            const double sg = sbit(sp, f) ? -1.0 : 1.0;
            const double2 v = t.vb[vbi(f, m.n_vb, m.n)];
            bx -= 2.0 * sg * v.x;
            by -= 2.0 * sg * v.y;
        }
        const double mag = exp(re + bx);
        double sb, cb;
        sincos(by, &sb, &cb);
        const double rx = mag * (u.x * cb - u.y * sb), ry = mag * (u.x * sb + u.y * cb);
        if (lane == 0) {
            ex += val.x * rx - val.y * ry;
            ey += val.x * ry + val.y * rx;
        }
    }
    return make_double2(ex, ey);
}

// The factors (z + q) of the lane's entries, in pairs, to mul(pair, real parts,
// imaginary parts): zr, zi pairs; qb the pattern's table (byte address), cb the
// term's row of the tuple table.
template <int KB, int NG, typename F>
__device__ __forceinline__ void term_factors(const float2 (&zr)[KB * NG / 2], const float2 (&zi)[KB * NG / 2],
                                             uint32_t qb, uint32_t cb, const uint32_t (&s2)[NG],
                                             const uint32_t (&ko)[NG], F&& factor) {
    auto mul = [&](int p, float2 qr, float2 qi) { factor(p, __fadd2_rn(zr[p], qr), __fadd2_rn(zi[p], qi)); };
    if constexpr (KB == 4) {
#pragma unroll
        for (int j = 0; j < NG; j++) {
            const uint32_t at = qb + lds16(cb + s2[j]) + ko[j];
            const float4 v0 = lds128(at), v1 = lds128(at + 16);
            mul(2 * j, make_float2(v0.x, v0.y), make_float2(v0.z, v0.w));
            mul(2 * j + 1, make_float2(v1.x, v1.y), make_float2(v1.z, v1.w));
        }
    } else if constexpr (KB == 2) {
#pragma unroll
        for (int j = 0; j < NG; j++) {
            const float4 v = lds128(qb + lds16(cb + s2[j]) + ko[j]);
            mul(j, make_float2(v.x, v.y), make_float2(v.z, v.w));
        }
    } else {
#pragma unroll
        for (int j = 0; j < NG; j += 2) {
            const float2 v0 = lds64(qb + lds16(cb + s2[j]) + ko[j]);
            const float2 v1 = lds64(qb + lds16(cb + s2[j + 1]) + ko[j + 1]);
            mul(j / 2, make_float2(v0.x, v1.x), make_float2(v0.y, v1.y));
        }
    }
}

// Scale p to a leading one: p 2^-e, e its exponent.  False outside 2^-116 ..
// 2^116 (and for NaN).
__device__ __forceinline__ bool split(float2& p, int& e) {
    const float mx = fmaxf(fabsf(p.x), fabsf(p.y));
    const uint32_t b = __float_as_uint(mx) & 0x7f800000u;
    e = (int)(b >> 23) - 127;
    const float sc = __uint_as_float(0x7f000000u - b);
    p.x *= sc;
    p.y *= sc;
    return mx >= 1.2037062e-35f && mx <= 8.3076750e34f && p.x == p.x && p.y == p.y;
}

// Product over the lane's entries of (z + q), scaled to a leading one.  False
// where a chain ends below `low` or the product leaves the range of split().
template <int KB, int NG>
__device__ __forceinline__ bool term_product(const float2 (&zr)[KB * NG / 2], const float2 (&zi)[KB * NG / 2],
                                             uint32_t qb, uint32_t cb, const uint32_t (&s2)[NG],
                                             const uint32_t (&ko)[NG], float low, float2& u, int& e) {
    float2 Px, Py;
    term_factors<KB, NG>(zr, zi, qb, cb, s2, ko, [&](int p, float2 fr, float2 fi) {
        if (p == 0) {
            Px = fr;
            Py = fi;
        } else {
            const float2 nx = __ffma2_rn(Px, fr, __fmul2_rn(make_float2(-Py.x, -Py.y), fi));
            Py = __ffma2_rn(Px, fi, __fmul2_rn(Py, fr));
            Px = nx;
        }
    });
    u = make_float2(Px.x * Px.y - Py.x * Py.y, Px.x * Py.y + Py.x * Px.y);
    const float lo = fminf(fmaxf(fabsf(Px.x), fabsf(Py.x)), fmaxf(fabsf(Px.y), fabsf(Py.y)));
    return split(u, e) & (lo >= low);
}

// The same, scaled after every factor: false only where a factor is zero or
// outside split()'s range.
template <int KB, int NG>
__device__ __forceinline__ bool term_product_scaled(const float2 (&zr)[KB * NG / 2], const float2 (&zi)[KB * NG / 2],
                                                    uint32_t qb, uint32_t cb, const uint32_t (&s2)[NG],
                                                    const uint32_t (&ko)[NG], float2& u, int& e) {
    bool ok = true;
    u = make_float2(1.f, 0.f);
    e = 0;
    term_factors<KB, NG>(zr, zi, qb, cb, s2, ko, [&](int, float2 fr, float2 fi) {
        float2 f[2] = {make_float2(fr.x, fi.x), make_float2(fr.y, fi.y)};
#pragma unroll
        for (int i = 0; i < 2; i++) {
            int ef, eu;
            ok &= split(f[i], ef);
            u = cmul(u, f[i]);
            ok &= split(u, eu);
            e += ef + eu;
        }
    });
    return ok;
}

// Butterfly reduce-scatter of KT per-lane partials (mantissas multiply,
// exponents add): afterwards every lane holds the total of term
// (lane >> (5 - log2 KT)).
template <int KT>
__device__ __forceinline__ void reduce_products(int (&e)[KT], float2 (&u)[KT], int lane, int& R, float2& U) {
#pragma unroll
    for (int stage = 0; stage < (KT == 8 ? 3 : 2); stage++) {
        const int off = 16 >> stage, half = (KT >> stage) >> 1;
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < KT / 2; i++) {
            if (i >= half) break;
            const int ke = up ? e[half + i] : e[i], se = up ? e[i] : e[half + i];
            const float2 ku = up ? u[half + i] : u[i], su = up ? u[i] : u[half + i];
            float2 ru;
            ru.x = __shfl_xor_sync(kFull, su.x, off);
            ru.y = __shfl_xor_sync(kFull, su.y, off);
            e[i] = ke + __shfl_xor_sync(kFull, se, off);
            u[i] = cmul(ku, ru);
        }
    }
    int r = e[0];
    float2 v = u[0];
#pragma unroll
    for (int off = (KT == 8 ? 2 : 4); off >= 1; off >>= 1) {
        float2 w;
        w.x = __shfl_xor_sync(kFull, v.x, off);
        w.y = __shfl_xor_sync(kFull, v.y, off);
        r += __shfl_xor_sync(kFull, r, off);
        v = cmul(v, w);
    }
    R = r;
    U = v;
}

// LP: log psi as well (its FP64 sums cost the kernel without them 9 % when they
// are compiled into it).
template <int KB, int NG, bool LP>
__global__ void __launch_bounds__(32 * eloc_warps(KB* NG), eloc_min_blocks(KB* NG))
    eloc_sym_kernel(const EvalArgs a, const SymLayout L) {
    constexpr int E = KB * NG, NP = E / 2;
    constexpr int KT = E >= 16 ? 4 : 8;  // terms per reduction round
    static_assert(E % 2 == 0, "entries per lane come in pairs");
    extern __shared__ __align__(16) unsigned char smem[];
    const MachineDev& m = a.m;
    const int n = m.n, nh = m.nh, S = m.S, T = m.T, n_vb = m.n_vb, SP = S + 1;
    const int tid = threadIdx.x, nthr = blockDim.x, warps = nthr >> 5;
    const int n_terms = a.tt.n_terms, n_diag = a.tt.n_diag, n_cls = a.tt.n_cls, npat = 1 << a.tt.nf_max;

    double2* sW64 = reinterpret_cast<double2*>(smem + L.w64);
    uint8_t* sPerm = smem + L.perm;
    uint8_t* sInv = smem + L.inv;
    uint16_t* sCls = reinterpret_cast<uint16_t*>(smem + L.cls);
    double2* sBase = reinterpret_cast<double2*>(smem + L.base);
    TermDev* sTerms = reinterpret_cast<TermDev*>(smem + L.terms);
    TermDev* sDiag = reinterpret_cast<TermDev*>(smem + L.diag);
    double2* sVals = reinterpret_cast<double2*>(smem + L.vals);
    double2* sVb = reinterpret_cast<double2*>(smem + L.vb);
    double2* sSite = reinterpret_cast<double2*>(smem + L.site);  // 2 sum_e W_fe; entry n: sum_e hb_e
    unsigned* sQmax = reinterpret_cast<unsigned*>(smem + L.qmax);  // largest |q| component, a float's bits
    double2* fac = reinterpret_cast<double2*>(smem + L.warp0);   // exp(-4 W), exp(4 W) per (row, k)
    auto rk = [&](int r) { return a.wrank ? (int)a.wrank[r] : r; };
    for (int i = tid; i < n * nh; i += nthr) {
        const double2 w = m.W64[i];
        sW64[rk(i / nh) * L.ws64 + i % nh] = w;
        // rows beyond |4 Re W| = 60 have no FP32 factor: NaN sends their
        // terms to ratio_slow
        double s, c;
        sincos(4.0 * w.y, &s, &c);
        const double g = exp(4.0 * w.x), gi = 1.0 / g;
        const bool ok = fabs(4.0 * w.x) <= 60.0;
        const double bad = __longlong_as_double(0x7ff8000000000000ll);
        fac[2 * i] = ok ? make_double2(gi * c, -gi * s) : make_double2(bad, bad);
        fac[2 * i + 1] = ok ? make_double2(g * c, g * s) : make_double2(bad, bad);
    }
    for (int i = tid; i < n * S; i += nthr) {
        sPerm[i] = (uint8_t)rk(m.perm[i]);
        if (a.O) sInv[i] = m.inv[i];
    }
    // tuple offsets per (term, symmetry); column S: the tuple n_cls, q = 1
    for (int i = tid; i < n_terms * SP; i += nthr) {
        const int t = i / SP, s = i - t * SP;
        sCls[i] = (uint16_t)((s < S ? (int)a.tt.cls[t * S + s] : n_cls) * L.qs);
    }
    for (int i = tid; i < n_terms; i += nthr) sTerms[i] = a.tt.terms[i];
    for (int i = tid; i < n_diag; i += nthr) sDiag[i] = a.tt.diag[i];
    for (int i = tid; i < a.tt.n_vals; i += nthr) sVals[i] = a.tt.vals[i];
    for (int i = tid; i < n_vb; i += nthr) sVb[i] = m.vb[i];
    if (tid == 0) *sQmax = 0;
    __syncthreads();
    // q of every tuple, hidden unit and spin pattern (bit set: spin down)
    float qmax = 0.f;
    for (int i = tid; i < (n_cls + 1) * nh; i += nthr) {
        const int c = i / nh, k = i - c * nh, kk = k % KB, k0 = k - kk;
        const uint8_t* tup = a.tt.tup + 8 * c;
        const int nf = c < n_cls ? tup[6] : 0;
        const int at = 8 * k0 + (KB == 1 ? 0 : 16 * (kk >> 1) + 4 * (kk & 1));
        for (int p = 0; p < npat; p++) {
            double2 v = make_double2(1, 0);
            for (int q = 0; q < nf; q++) v = cmul(v, fac[2 * (tup[q] * nh + k) + ((p >> q) & 1)]);
            unsigned char* row = smem + L.q + p * L.qp + c * L.qs + at;
            // beyond 2^+-86: out of the products' range
            const double mx = fmax(fabs(v.x), fabs(v.y));
            const bool ok = mx < 7.7e25 && mx > 1.3e-26;
            const float bad = __int_as_float(0x7fc00000);
            if (ok) qmax = fmaxf(qmax, (float)mx);
            *reinterpret_cast<float*>(row) = ok ? (float)v.x : bad;
            *reinterpret_cast<float*>(row + (KB == 1 ? 4 : 8)) = ok ? (float)v.y : bad;
        }
    }
    const unsigned qw = __reduce_max_sync(kFull, __float_as_uint(qmax));
    if ((tid & 31) == 0) atomicMax(sQmax, qw);
    for (int t = tid; t < T; t += nthr) {
        const int k = t % nh, s = t / nh;
        double2 acc = m.hb[k];
        for (int f = 0; f < n; f++) {
            const double2 w = sW64[sPerm[f * S + s] * L.ws64 + k];
            acc.x += w.x;
            acc.y += w.y;
        }
        sBase[t] = acc;
    }
    for (int f = tid >> 5; f <= n; f += warps) {  // a warp per site
        double2 acc = make_double2(0, 0);
        if (f < n) {
            for (int e = tid & 31; e < T; e += 32) {
                const int k = e % nh, s = e / nh;
                const double2 w = sW64[sPerm[f * S + s] * L.ws64 + k];
                acc.x += 2.0 * w.x;
                acc.y += 2.0 * w.y;
            }
        } else {
            for (int k = tid & 31; k < nh; k += 32) acc.x += m.hb[k].x * S;
        }
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if ((tid & 31) == 0) sSite[f] = acc;
    }
    __syncthreads();  // fac is done: the region becomes the warps' scratch

    const int warp = tid >> 5, lane = tid & 31;
    unsigned char* wbase = smem + L.warp0 + warp * L.warp_bytes;
    float2* tn = reinterpret_cast<float2*>(wbase + 16);
    float* sgn = reinterpret_cast<float*>(wbase + 16 + T * 8);
    const int G = T / KB, NGK = nh / KB;
    uint32_t s2[NG], ko[NG];  // byte offsets of the group's symmetry index and first hidden unit
    uint32_t vmask = 0;
#pragma unroll
    for (int j = 0; j < NG; j++) {
        const int g = lane + 32 * j;
        const bool ok = g < G;
        s2[j] = 2u * (uint32_t)(ok ? g / NGK : S);
        ko[j] = 8u * (uint32_t)(ok ? (g % NGK) * KB : 0);
        vmask |= ok ? 1u << j : 0u;
    }
    const uint32_t qa = (uint32_t)__cvta_generic_to_shared(smem + L.q);
    const uint32_t ca = (uint32_t)__cvta_generic_to_shared(sCls);

    for (int b = blockIdx.x * warps + warp; b < a.B; b += gridDim.x * warps) {
        uint32_t sp[4];
#pragma unroll
        for (int w = 0; w < 4; w++) sp[w] = a.spins[4 * b + w];
        if (a.O)
            for (int i = lane; i < n; i += 32) sgn[i] = sbit(sp, i) ? -1.f : 1.f;
        // orientation: -theta when Re sum theta < 0
        double rs = 0;
        for (int f = lane; f < n; f += 32) rs += sbit(sp, f) ? -sSite[f].x : sSite[f].x;
        const bool neg = warp_sum(rs) + 2.0 * sSite[n].x < 0;

        // theta in FP64 (down spins subtracted from the all-up table), tanh
        // theta in FP64 into the warp's scratch, z = exp(-+2 theta) to FP32
        // pairs, and the lane's product of 1 + z
        float2 zr[NP], zi[NP];
        float zmax = 0.f;
        double2 D = make_double2(1, 0);
        int ec = 0;  // the product's exponent, apart from D
        auto lead = [&]() {  // D to a leading one
            const int hi = (__double2hiint(fmax(fabs(D.x), fabs(D.y))) >> 20) & 0x7ff;
            const double sc = __hiloint2double((min(max(2046 - hi, 1), 2046)) << 20, 0);
            D.x *= sc;
            D.y *= sc;
            ec += hi - 1023;
        };
        double lre = 0, lim = 0;  // sum ln cosh theta (principal values), ln 2 per entry left out
#pragma unroll
        for (int j = 0; j < NG; j++) {
            double2 acc[KB];
            const bool ok = (vmask >> j) & 1u;
            const int gs = (int)(s2[j] >> 1), gk = (int)(ko[j] >> 3);
            const int t0 = gk + nh * gs;
#pragma unroll
            for (int i = 0; i < KB; i++) acc[i] = ok ? sBase[t0 + i] : make_double2(0, 0);
            if (ok) {
#pragma unroll
                for (int wd = 0; wd < 4; wd++) {
                    uint32_t bits = sp[wd];
                    while (bits) {
                        const int f = 32 * wd + __ffs(bits) - 1;
                        bits &= bits - 1;
                        const double2* wr = sW64 + sPerm[f * S + gs] * L.ws64 + gk;
#pragma unroll
                        for (int i = 0; i < KB; i++) {
                            const double2 w = wr[i];
                            acc[i].x = fma(-2.0, w.x, acc[i].x);
                            acc[i].y = fma(-2.0, w.y, acc[i].y);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < KB; i++) {
                const int e = j * KB + i;
                double zx = 0, zy = 0;
                if (ok) {
                    const double x = acc[i].x, aa = fabs(x);
                    double s, c, w = 0;
                    sincos(acc[i].y, &s, &c);
                    if (LP || a.O) {  // the terms of ctanh_r
                        const double omz = -expm1(-2.0 * aa);
                        w = 1.0 - omz;
                        const double X = (1.0 + w) * c, Y = omz * s;
                        if constexpr (LP) {
                            lre += aa + 0.5 * log(X * X + Y * Y);
                            lim += atan2(copysign(omz, x) * s, X);
                        }
                        if (a.O) {
                            const double inv = 1.0 / (X * X + Y * Y);
                            tn[t0 + i] = make_float2((float)(copysign(omz * (1.0 + w), x) * inv),
                                                     (float)(4.0 * w * s * c * inv));
                        }
                    }
                    // |z|; where log psi needs w anyway, from w up to |x| = 7 (good
                    // to 1e-10 there; 262144 configurations of 128 spins with O_k
                    // 14.15 ms that way, 13.95 by exp).  Beyond e^68, where a
                    // factor's product may leave FP32, NaN
                    const double v = neg ? 2.0 * x : -2.0 * x;
                    double r;
                    if (LP && aa <= 7.0)
                        r = v > 0 ? 1.0 / w : w;
                    else
                        r = v <= 68.0 ? exp(v) : __longlong_as_double(0x7ff8000000000000ll);
                    zx = r * (c * c - s * s);
                    zy = (neg ? 2.0 : -2.0) * r * s * c;
                    zmax = fmaxf(zmax, (float)r);
                    D = cmul(D, make_double2(1.0 + zx, zy));
                    if (e % 8 == 7) lead();
                }
                if (e & 1) {
                    zr[e >> 1].y = (float)zx;
                    zi[e >> 1].y = (float)zy;
                } else {
                    zr[e >> 1].x = (float)zx;
                    zi[e >> 1].x = (float)zy;
                }
            }
        }

        if constexpr (LP) {
            lre = warp_sum(lre);
            lim = warp_sum(lim);
            double bx = 0, by = 0;
            for (int q = 0; q < n_vb; q++) {
                double acc = 0;
                for (int s = lane; s < S; s += 32) acc += sbit(sp, m.orbit[q * S + s]) ? -1.0 : 1.0;
                acc = warp_sum(acc);
                bx += sVb[q].x * acc;
                by += sVb[q].y * acc;
            }
            if (lane == 0) a.logpsi[b] = make_double2(bx + lre - 0.69314718055994531 * T, by + lim);
        }
        if (a.eloc) {
            double ex = 0.0, ey = 0.0;
            // prod 1 / (1 + z) = D 2^-ec
            bool safe;
            {
                lead();
                safe = __all_sync(kFull, D.x != 0.0 || D.y != 0.0);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    double2 w;
                    w.x = __shfl_xor_sync(kFull, D.x, o);
                    w.y = __shfl_xor_sync(kFull, D.y, o);
                    ec += __shfl_xor_sync(kFull, ec, o);
                    D = cmul(D, w);
                }
                const double inv = 1.0 / (D.x * D.x + D.y * D.y);
                D.x *= inv;
                D.y *= -inv;
            }
            // the lowest end of a chain that has stayed in range (NaN in z: any)
            const uint32_t fb = __float_as_uint(2.83f * (__uint_as_float(*sQmax) +
                                                         __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(zmax)))));
            const int lexp = (NP - 1) * ((int)(fb >> 23) - 126) - 116;
            bool scaled = lexp > 8;
            const float low = __uint_as_float((uint32_t)(max(min(lexp, 8), -116) + 127) << 23);
            for (int c0 = 0; c0 < n_terms && safe; c0 += 32) {
                // the lane's term: its pattern table and exponent
                const int tl = min(c0 + lane, n_terms - 1);
                const TermDev tm = sTerms[tl];
                const int nf = term_nf(tm);
                int pat = 0;
                double lx = 0, ly = 0;
                for (int q = 0; q < nf; q++) {
                    const int f = term_flip(tm, q), d = sbit(sp, f);
                    pat |= d << q;
                    const double sg = d ? -1.0 : 1.0, so = neg ? -sg : sg;
                    const double2 v = sVb[vbi(f, n_vb, n)];
                    lx += so * sSite[f].x - 2.0 * sg * v.x;
                    ly += so * sSite[f].y - 2.0 * sg * v.y;
                }
                if (neg) pat ^= npat - 1;
                const uint32_t pb = qa + (uint32_t)(pat * L.qp);
                int Re = 0;
                float2 U = make_float2(0.f, 0.f);
                for (int r = 0; r < 32 / KT && c0 + r * KT < n_terms && !scaled; r++) {
                    int pe[KT];
                    float2 pu[KT];
                    bool ok = true;
#pragma unroll
                    for (int q = 0; q < KT; q++) {
                        const uint32_t qb = __shfl_sync(kFull, pb, r * KT + q);
                        const int ti = min(c0 + r * KT + q, n_terms - 1);
                        ok &= term_product<KB, NG>(zr, zi, qb, ca + 2u * (uint32_t)(ti * SP), s2, ko, low, pu[q], pe[q]);
                    }
                    if (!__all_sync(kFull, ok)) {
                        scaled = true;
                        break;
                    }
                    int R;
                    float2 V;
                    reduce_products<KT>(pe, pu, lane, R, V);
                    // to the lane of the term
                    const int src = (lane & (KT - 1)) * (32 / KT);
                    const int er = __shfl_sync(kFull, R, src);
                    const float vx = __shfl_sync(kFull, V.x, src), vy = __shfl_sync(kFull, V.y, src);
                    if (lane / KT == r) {
                        Re = er;
                        U = make_float2(vx, vy);
                    }
                }
                if (scaled) {  // one term at a time
#pragma unroll 1
                    for (int t = c0; t < min(c0 + 32, n_terms) && safe; t++) {
                        const uint32_t qb = __shfl_sync(kFull, pb, t - c0);
                        float2 V;
                        int R;
                        const bool ok = term_product_scaled<KB, NG>(zr, zi, qb, ca + 2u * (uint32_t)(t * SP), s2, ko, V, R);
                        safe = __all_sync(kFull, ok);
                        R = __reduce_add_sync(kFull, R);
                        V = warp_cprod(V);
                        if (lane == t - c0) {
                            Re = R;
                            U = V;
                        }
                    }
                }
                if (safe && c0 + lane < n_terms) {
                    const double2 val = sVals[tm.voff + term_loc(tm, sp)];
                    if (val.x != 0.0 || val.y != 0.0) {
                        const double mag = exp(lx + (double)(Re - ec) * 0.693147180559945309);
                        double sb, cb;
                        sincos(ly, &sb, &cb);
                        const double2 u = cmul(cmul(make_double2(U.x, U.y), D), make_double2(mag * cb, mag * sb));
                        ex += val.x * u.x - val.y * u.y;
                        ey += val.x * u.y + val.y * u.x;
                    }
                }
            }
            if (!safe) {
                __syncwarp();
                const SymTabs tabs{sW64, sBase, sVals, sVb, sPerm, sTerms, L.ws64};
                // ratio_slow leaves theta in the scratch; tanh theta is formed
                // again for O_k
                const double2 e = ratio_slow(a.md, n_terms, tabs, sp[0], sp[1], sp[2], sp[3], tn, lane);
                ex = e.x;
                ey = e.y;
                if (a.O)
                    for (int t = lane; t < T; t += 32) {
                        const int k = t % nh, s = t / nh;
                        double2 x = sBase[t];
                        for (int f = 0; f < n; f++)
                            if (sbit(sp, f)) {
                                const double2 w = sW64[sPerm[f * S + s] * L.ws64 + k];
                                x.x = fma(-2.0, w.x, x.x);
                                x.y = fma(-2.0, w.y, x.y);
                            }
                        const double2 tt = ctanh_r<double>(x.x, x.y);
                        tn[t] = make_float2((float)tt.x, (float)tt.y);
                    }
            }
            // diagonal matrix elements, one operator per lane
            for (int d = lane; d < n_diag; d += 32) {
                const TermDev td = sDiag[d];
                const double2 v = sVals[td.voff + term_loc(td, sp)];
                ex += v.x;
                ey += v.y;
            }
            ex = warp_sum(ex);
            ey = warp_sum(ey);
            if (lane == 0) a.eloc[b] = make_double2(ex, ey);
        }
        if (a.O) {
            __syncwarp();
            write_O_sym(m, sp, tn, sgn, sInv, reinterpret_cast<float2*>(a.O) + (size_t)b * m.P, lane);
        }
        __syncwarp();
    }
}

template <int KB, int NG, bool LP> const void* fn() {
    return reinterpret_cast<const void*>(eloc_sym_kernel<KB, NG, LP>);
}

template <bool LP> const void* pick_sym(int kb, int ng) {
    switch (100 * kb + ng) {
        case 401: return fn<4, 1, LP>();
        case 402: return fn<4, 2, LP>();
        case 404: return fn<4, 4, LP>();
        case 201: return fn<2, 1, LP>();
        case 202: return fn<2, 2, LP>();
        case 204: return fn<2, 4, LP>();
        case 208: return fn<2, 8, LP>();
        case 102: return fn<1, 2, LP>();
        case 104: return fn<1, 4, LP>();
        case 108: return fn<1, 8, LP>();
        case 116: return fn<1, 16, LP>();
    }
    return nullptr;
}

}  // namespace

cudaError_t launch_eloc_sym(const EvalArgs& a, cudaStream_t st) {
    const MachineDev& m = a.m;
    // with few terms and entries the block's tables cost more than they save
    // (8 sites, 16 entries, 256 configurations: 19 us here, 17 us by ln cosh
    // sums; 32 sites, 128 entries, 4096 configurations: 53 and 61 us)
    if (!m.symmetric || !a.tt.cls || a.tt.n_terms * m.T <= 256) return cudaErrorNotSupported;
    const int kb = m.nh % 4 == 0 ? 4 : (m.nh % 2 == 0 ? 2 : 1);
    const int G = m.T / kb;
    int ng = kb == 1 ? 2 : 1;  // entries come in pairs
    while (32 * ng < G) ng *= 2;
    const void* f = a.logpsi ? pick_sym<true>(kb, ng) : pick_sym<false>(kb, ng);
    if (!f) return cudaErrorNotSupported;
    int dev = 0, budget = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&budget, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // as many warps as the tables leave room for, at least half a block
    int warps = eloc_warps(kb * ng);
    SymLayout L = sym_layout(m, a.tt, kb, warps, a.O != nullptr);
    while (L.total > budget && warps > 8) {
        warps -= 2;
        L = sym_layout(m, a.tt, kb, warps, a.O != nullptr);
    }
    if (L.total > budget || L.qp > 0xffff) return cudaErrorNotSupported;
    if ((e = ensure_dynamic_smem(f, L.total)) != cudaSuccess) return e;
    // resident blocks per SM, per (device, kernel, threads, shared memory)
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, int>, int> cache;
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        int& c = cache[std::make_tuple(dev, f, warps, L.total)];
        if (!c && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, f, 32 * warps, L.total) != cudaSuccess || c < 1))
            c = 1;
        per_sm = c;
    }
    const int blocks = std::max(1, std::min((a.B + warps - 1) / warps, sms * per_sm));
    EvalArgs aa = a;
    void* args[] = {&aa, &L};
    return cudaLaunchKernel(f, dim3(blocks), dim3(32 * warps), args, (size_t)L.total, st);
}

}  // namespace rbmnqs
