// sampler_screen.cuh -- FP32 Metropolis sweep (metropolis_sampler.cpp:118-273)
// whose proposals are screened by products and decided by the ln|cosh| sums
// only where the screen cannot tell.
//
// The decision of a proposal is  0.5 ln u < d,  d = sum_e ln|cosh theta'_e| -
// sum_e ln|cosh theta_e| + bias, the sums in the fixed order and arithmetic of
// lnc_sweep_sum on the chain's FP32 theta (decide_exact below: one ex2 and one
// cosine per entry, for theta and for theta').  The screen computes the same
// number from z = exp(-2 theta), held in registers: a flip of site f multiplies
// z by p = exp(4 sigma_f W[P_s(f), k], a table entry, and
//   ln|cosh theta'| - ln|cosh theta| = ln|1 + z p| - ln|1 + z| - 2 sigma_f Re W,
// four FMA-pipe operations for the product, three for |1 + z p|^2, one to
// multiply them up, one lg2 per four entries and no other transcendental.  When
// |d - 0.5 ln u| exceeds a margin for what the two computations can differ by, the
// screen decides; otherwise theta at the start of the sweep is formed from its
// configuration in FP64, the sweep's accepted flips are applied to it in FP32, in
// order, and decide_exact decides.
//
// Sessions in FP64 use the same screen; what it cannot tell is decided by the
// ln|cosh| sums in FP64 (decide_fp64) on theta kept in FP64 in the same way.
//
// The sums ln|1 + z| are kept as integers (2^-16 steps of lg2 a lane), so that the
// difference of two of them is exact: in FP32 a sum of 1e4 is good to 1e-3.
//
// Margin, FP64 sessions.  A worst case, every rounding at its bound and all of one
// sign: what the screen decides is what the sums in FP64 would, up to their own ties
// of 1e-13.  In u = 2^-24 (set_margin):
//  - z carries a relative error eps = u (6 max |Re theta| + 2 max |Im theta| + 24 + 3
//    k) after k site flips: theta rounded, ex2 (2.5 u), the sine and cosine after
//    their reduction (11 u; both measured over all floats), then per flip the
//    rounding of p (u) and of a complex product with FMA (2 u; Jeannerod, Kornerup,
//    Louvet, Muller, Math. Comp. 86, 2017).  An error common to z and w = z p moves
//    d by eps |w - z| / (|1 + w| |1 + z|) per entry.  With a^2 and b^2 the largest 1 /
//    |1 + z|^2 and 1 / |1 + w|^2 that is below |p - 1| (1 + a) b <= |p - 1| t with t =
//    (1 + a^2) / 2 + b^2, and below 6 t however large p: the sum over the entries is S
//    t eps, S the largest row's sum of min(exp(4 |W|) - 1, 6).
//  - The products' own rounding of w, 3 u a site: |w / (1 + w)| <= 1 + b an entry.
//  - The sums of ln|1 + z|: 2 u an entry for the squared moduli and their products, 2.6
//    u + 2 u |lg2| a group (lg2, measured over all floats), the additions, and half a
//    step a lane.
// The first-order terms carry a factor 1.15 for the second order, which holds while
// eps (1 + a) < 1/16; closer to a zero of cosh the margin is infinite, as where a
// lane's sum leaves the integers' range (or is NaN).  It grows with the accepted
// flips: z is refreshed from theta every four sweeps (FP32 sessions: eight).
//
// Margin, FP32 sessions.  The screen has to agree with the FP32 sums as they are
// computed, and the worst cases of these (cosine and additions of |Re theta|, 1e-2
// at 512 entries) exceed what they err by a hundredfold.  So the margin is an
// estimate, m0 + coef (a^2 + b^2) with m0 = 8e-4 + 1e-4 max |Re theta| and coef = 2e-6
// + 5e-7 max |Im theta|.  Over 5e7 proposals of machines of 384 and 512 entries
// (weights of spread 0.005 to 0.1, hidden biases of either sign, near the zeros of
// cosh, all entries of a unit equal) the largest difference was 0.29 of it.  Against
// 64 bits the screen was off by 2.4e-4 at most, so what it decides is right by them
// too; chains, samples and counters are those of the FP32 sums, bit for bit, in every
// test.
//
// Weights that leave too many proposals open (kOff: the FP64 margin at mean counts
// and |1 + z| = 1), that reach |Re theta| > 40, that mostly overflow a product of four
// |1 + z|^2 (a sum of -Re theta of 22; 512 entries of 128 spins: spread of the weights
// 0.2 0.2 % of the proposals, 0.25 48 %, 0.3 94 %), or that FP32 factors do not hold,
// turn the launch over to the sums' kernel (sampler.cu), which is launched behind
// this one and returns at once otherwise (2 us).  At a spread of 0.3, 16384 chains x 4
// sweeps: 17.9 ms screened, 5.0 by the sums.
//
// Layout: groups of KB consecutive hidden units with one symmetry index, lane l
// owns the groups l + 32 j, entries in pairs (packed FP32x2).  Symmetric machines
// keep p and W of every row in shared memory and find the row of (site, symmetry)
// in a 16-bit table; basic machines read row f directly, from shared memory or,
// where p does not fit, from L2.  The loop is bound by issue and latency (ncu, 512
// entries: 327 warp instructions a proposal, issue 62 % of active cycles, LSU 42 %,
// FMA pipe 34 %, FP64 1.5 %; 16 warps at 128 registers: with 20 at 96 the loop
// spills, 15.8 ms below).  Measured: 16384 chains x 16 sweeps of 128 spins, 512
// entries, FP32: 19.7 ms by the exact sums, 14.1 screened, 0.17 % of the proposals
// decided exactly (28 ms with a worst case of the FP32 sums' rounding in the margin);
// FP64 sessions, 500 chains x 19 sweeps of 32 spins, 96 entries: 1.33 ms by the sums,
// 0.25 screened (0.22 with FP32's margin), 0.8 % decided exactly.
#pragma once

#include <type_traits>

#include "eloc.cuh"
#include "sweep_common.cuh"

namespace rbmnqs {
namespace screen {

// sweeps between refreshes of z
__host__ __device__ constexpr int refresh_of(bool fp64) { return fp64 ? 4 : 8; }

// A chain's state between the sweep loop and its services, in the warp's scratch
// (z and z p of the last proposal: in local memory).  The loop keeps everything
// in registers and leaves through this state where a proposal needs the exact
// sums or theta is wanted: what the services use, the loop then neither saves nor
// shares registers with.
struct State {
    uint32_t start[4];  // configuration at the start of the sweep
    uint32_t sp[4];     // current configuration
    int LS;             // sum ln|1 + z|, in log_sum's steps
    float inv;          // 1 / min |1 + z|^2
    int st, slot, np, applied;
    uint32_t prop, nacc;
    int k;  // site flips since the refresh of z
    uint32_t code;      // the open proposal: sites, bond flag (bit 16), spins (bits 17, 18)
    float lu;
    int LSn;
    float inv_n;
    int accept;
    int sum_np;  // FP64 sessions: the sum of ln|cosh theta| after the sweep's first sum_np flips
    double sum;
};
constexpr int kStateBytes = 112;

// The margin of a proposal.  FP64: (fac (eps0 + eps1 k) + R1) t + R0 + R2 |LS| with
// t = (1 + a^2) / 2 + b^2, k the site flips since the refresh of z and fac = 1, or fac2
// for two sites; FP32: m0 + coef (a^2 + b^2).
struct Margin {
    float eps0, eps1, R0, R1, R2, fac2, mn_min;
    float m0, coef;
    int off;  // the launch is left to the sums' kernel
    // machine bounds (as uints, for atomicMax): max |Re theta|, max |Im theta|, S,
    // max 4 |W|, max |sum_e Re W_fe + Re v|, and what -Re theta of four entries may add
    // up to: their hidden biases' part and eight times theta's spread
    unsigned bre, bim, S, xmax, smax, sat;
};
constexpr float kOff = 0.3f, kSat32 = 21.f, kSat64 = 30.f;

// Hidden units per group: as the row loads can be widest for symmetric machines;
// pairs for basic machines, whose lanes then read consecutive 16 bytes.
__host__ __device__ inline int group_width(const MachineDev& m) {
    if (!m.symmetric) return 2;
    return m.nh % 4 == 0 ? 4 : (m.nh % 2 == 0 ? 2 : 1);
}

// Shared-memory carve-up, the same arithmetic on host (sizing) and device.
struct Layout {
    int p, w, off, row, w64, base, site, bonds, mar, warp0, warp_bytes, total;
    int list;  // the sweep's accepted flips in a warp's scratch, behind theta
    int qs;    // row stride of p and W in shared memory (bytes)
    int ws64;  // row stride of the FP64 W (double2), shared or global
    int p_smem, w64_smem, bonds_smem;
};
// p_budget: bytes that the p table of a basic machine may take in shared memory
__host__ __device__ inline Layout make_layout(const MachineDev& m, int n_bonds, int warps, int p_budget, int fp64) {
    Layout L{};
    const int n = m.n, nh = m.nh, kb = group_width(m);
    const bool sym = m.symmetric != 0;
    L.qs = sym ? 4 * eloc::w32_stride(nh, kb, true) : 8 * nh;
    L.p_smem = sym || 3 * n * L.qs <= p_budget;
    L.w64_smem = sym && n * nh * 16 <= 32 * 1024;
    L.ws64 = L.w64_smem ? eloc::w64_stride(nh) : nh;
    L.bonds_smem = n_bonds * 8 <= 8 * 1024;
    L.list = kStateBytes + eloc::a16(m.T * (fp64 ? 16 : 8));
    L.warp_bytes = L.list + eloc::a16(n * 4);
    int at = 0;
    auto take = [&](int bytes) {
        const int o = at;
        at += eloc::a16(bytes);
        return o;
    };
    // symmetric: two signs of n + 1 rows (row n, read by groups beyond T: p = 1)
    L.p = take(L.p_smem ? 2 * (n + 1) * L.qs : 0);
    L.w = take(L.p_smem ? (n + 1) * L.qs : 0);
    L.off = take(sym ? 2 * n * (m.S + 1) : 0);
    L.row = take(sym ? n * (m.S + 1) : 0);
    L.w64 = take(L.w64_smem ? n * L.ws64 * 16 : 0);
    L.base = take(m.T * 16);
    L.site = take((n + 1) * 8);
    L.bonds = take(L.bonds_smem ? n_bonds * 8 : 0);
    L.mar = take((int)sizeof(Margin));
    L.warp0 = at;
    L.total = at + warps * L.warp_bytes;
    return L;
}

// The margin's coefficients from the machine's bounds (see the top of the file).
// E: entries per lane; with two, the products are of two.
__device__ inline void set_margin(Margin& g, int n, int T, int E, bool fp64, bool bonds) {
    constexpr float u = 5.9604645e-8f, c = 1.15f;
    const float bre = __uint_as_float(g.bre) * 1.001f, bim = __uint_as_float(g.bim) * 1.001f;
    const float x = __uint_as_float(g.xmax) * 1.001f, sm = __uint_as_float(g.smax) * 1.001f;
    float typ = 0.f;
    if (fp64) {
        // S of two rows: (e^x - 1)(e^y - 1) <= (their sum) max / 2, or both at their bound
        const float t = (float)T, S = __uint_as_float(g.S) * 1.001f + 4.f * u * t;
        const float e0 = 6.f * bre + 2.f * bim + 24.f, uu = u * 1.002f;
        g.fac2 = 2.f * (1.f + fminf(0.5f * expm1f(x), 0.83f));
        // common error of z; 3 u (1 + b) an entry and site: 1 + b <= 3 (1/2 + b^2)
        g.eps0 = uu * c * (S * e0 + 9.f * t);
        g.eps1 = uu * c * 3.f * S;
        g.R0 = uu * (2840.f + 4.5f * t + 44.f * sm + 170.f);
        g.R1 = uu * 3.68f * t;
        g.R2 = uu * 10.5f;
        const float eps = uu * (e0 + 3.f * (float)(refresh_of(true) * (n + 1) + 2));
        g.mn_min = 400.f * eps * eps;
        typ = g.R0 + g.R2 * t + 2.f * ((bonds ? g.fac2 : 1.f) * (g.eps0 + g.eps1 * n) + g.R1);
    }
    g.m0 = 8e-4f + 1e-4f * bre;
    g.coef = 2e-6f + 5e-7f * bim;
    g.off = !(typ < kOff) || !(bre < 40.f) || !(x < 84.f) || !(bim < 900.f) ||
            !(__uint_as_float(g.sat) < (fp64 ? kSat64 : kSat32) * (E > 2 ? 1.f : 2.f));
}

__device__ inline void load_tables(const SamplerArgs& a, const Layout& L, unsigned char* smem, bool fp64) {
    const MachineDev& m = a.m;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int n = m.n, nh = m.nh, S = m.S, SP = S + 1;
    const bool sym = m.symmetric != 0;
    float* site = reinterpret_cast<float*>(smem + L.site);
    Margin* mar = reinterpret_cast<Margin*>(smem + L.mar);
    if (L.p_smem) {
        const int per = L.qs / 8;  // 8-byte slots a row, the padding zero
        float2* P = reinterpret_cast<float2*>(smem + L.p);
        float2* W = reinterpret_cast<float2*>(smem + L.w);
        for (int i = tid; i < 2 * (n + 1) * per; i += nt) {
            const int sg = i / ((n + 1) * per), r = i / per - sg * (n + 1), k = i % per;
            float2 v = make_float2(0.f, 0.f);
            if (k < nh) {
                if (r < n)
                    v = reinterpret_cast<const float2*>(m.P32)[(sg * n + r) * nh + k];
                else if (sym)  // pairs of parts, or one entry's
                    v = (nh & 1) ? make_float2(1.f, 0.f) : ((k & 1) ? v : make_float2(1.f, 1.f));
            }
            P[i] = v;
        }
        for (int i = tid; i < (n + 1) * per; i += nt) {
            const int r = i / per, k = i % per;
            W[i] = r < n && k < nh ? m.W32[r * nh + k] : make_float2(0.f, 0.f);
        }
    }
    if (sym) {
        uint16_t* off = reinterpret_cast<uint16_t*>(smem + L.off);
        uint8_t* row = smem + L.row;
        for (int i = tid; i < n * SP; i += nt) {
            const int f = i / SP, s = i - f * SP, r = s < S ? (int)m.perm[f * S + s] : n;
            off[i] = (uint16_t)(r * L.qs);
            row[i] = (uint8_t)r;
        }
    }
    if (L.w64_smem) {
        double2* W = reinterpret_cast<double2*>(smem + L.w64);
        for (int i = tid; i < n * nh; i += nt) W[i / nh * L.ws64 + i % nh] = m.W64[i];
    }
    if (L.bonds_smem) {
        int2* b = reinterpret_cast<int2*>(smem + L.bonds);
        for (int i = tid; i < a.n_prop_bonds; i += nt) b[i] = a.prop_bonds[i];
    }
    // Re v (bias term of the exact sum) beside sum_e Re W_fe + Re v
    if (tid == 0) mar->bre = mar->bim = mar->S = mar->xmax = mar->smax = mar->sat = 0;
    __syncthreads();
    const double2* W64 = L.w64_smem ? reinterpret_cast<const double2*>(smem + L.w64) : m.W64;
    // theta of the all-up configuration, the bounds |b| + sum_f |W|, and per group
    // of hidden units sum -Re b and theta's variance
    double2* base = reinterpret_cast<double2*>(smem + L.base);
    const int kb = group_width(m);
    for (int t0 = 0; t0 < m.T; t0 += nt) {
        const int t = t0 + tid, k = t % nh, s = t / nh;
        float b = 0.f, v = 0.f;
        if (t < m.T) {
            double2 acc = m.hb[k];
            float bx = fabsf((float)acc.x), by = fabsf((float)acc.y);
            b = fmaxf(-(float)acc.x, 0.f);
            for (int f = 0; f < n; f++) {
                const double2 w = W64[(sym ? (int)smem[L.row + f * SP + s] : f) * L.ws64 + k];
                acc.x += w.x;
                acc.y += w.y;
                const float wx = (float)w.x;
                bx += fabsf(wx);
                by += fabsf((float)w.y);
                v = fmaf(wx, wx, v);
            }
            base[t] = acc;
            // non-finite weights give bounds above any limit
            atomicMax(&mar->bre, __float_as_uint(bx == bx ? bx : 1e30f));
            atomicMax(&mar->bim, __float_as_uint(by == by ? by : 1e30f));
        }
        for (int o = 1; o < kb; o <<= 1) {
            b += __shfl_xor_sync(kFull, b, o);
            v += __shfl_xor_sync(kFull, v, o);
        }
        const float w = (float)kb, sat = b * (4.f / w) + 8.f * sqrtf(v / w);
        atomicMax(&mar->sat, __float_as_uint(sat == sat ? sat : 1e30f));
    }
    for (int f = tid >> 5; f <= n; f += nt >> 5) {  // a warp per site
        double acc = 0;
        float S = 0.f, xm = 0.f;
        if (f < n)
            for (int t = tid & 31; t < m.T; t += 32) {
                const double2 w = W64[(sym ? (int)smem[L.row + f * SP + t / nh] : f) * L.ws64 + t % nh];
                acc += w.x;
                const float wx = (float)w.x, wy = (float)w.y, x = 4.f * sqrtf(wx * wx + wy * wy);
                S += fminf(ex2_ftz(1.442696f * x) - 1.f, 6.f);  // NaN: bre, bim
                xm = fmaxf(xm, x);
            }
        acc = warp_sum(acc);
        S = warp_sum(S);
        xm = warp_max(xm);
        if ((tid & 31) == 0) {
            const float v = f < n ? (float)m.vb[f % m.n_vb].x : 0.f;
            const float s = f < n ? (float)(acc + m.vb[f % m.n_vb].x) : 0.f;
            site[2 * f] = v;
            site[2 * f + 1] = s;
            const float sm = fabsf(s) + fabsf(v);
            atomicMax(&mar->S, __float_as_uint(fmaxf(S, 0.f)));
            atomicMax(&mar->xmax, __float_as_uint(xm));
            atomicMax(&mar->smax, __float_as_uint(sm == sm ? sm : 1e30f));
        }
    }
    __syncthreads();
    if (tid == 0) {
        set_margin(*mar, n, m.T, a.plan.lane_entries, fp64, a.bond_thr24 != 0);
        if (blockIdx.x == 0) *a.screen_off = mar->off;
    }
    __syncthreads();
}

// One chain.  wscr: the warp's scratch (state, theta [T] in the session's precision,
// the sweep's accepted flips [n]).  PS: p and W rows in shared memory (always for symmetric machines).
template <int KB, int NG, bool SYM, bool PS, bool F64>
__device__ __forceinline__ void run_chain(const SamplerArgs& a, const Layout& L, unsigned char* smem,
                                          unsigned char* wscr, int chain, int lane) {
    constexpr int E = KB * NG, NP = E / 2;
    static_assert(E % 2 == 0 && (SYM ? PS : KB == 2), "entries in pairs; basic machines in groups of two");
    const MachineDev& m = a.m;
    const int n = m.n, nh = m.nh, T = m.T, SP = m.S + 1;
    const uint2 key = make_uint2((uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t epoch = a.ctl[0];
    State* S = reinterpret_cast<State*>(wscr);
    using TH = std::conditional_t<F64, double2, float2>;
    TH* th = reinterpret_cast<TH*>(wscr + kStateBytes);
    uint32_t* plist = reinterpret_cast<uint32_t*>(wscr + L.list);
    {
        uint32_t sp[4];
        chain_start(a, chain, key, epoch, sp);
        if (lane < 4) S->sp[lane] = spin_word(sp, lane);
        if (lane == 0) {
            S->st = S->np = S->slot = 0;
            S->prop = prop_base(a);
            S->nacc = 0;
        }
        __syncwarp();
    }
    const double2* base = reinterpret_cast<const double2*>(smem + L.base);
    const double2* W64 = L.w64_smem ? reinterpret_cast<const double2*>(smem + L.w64) : m.W64;
    const uint8_t* rows = smem + L.row;
    const uint32_t wa = smem_addr(smem + L.w);
    const uint32_t sa = smem_addr(smem + L.site);
    const uint32_t pa = smem_addr(smem + L.p), oa = smem_addr(smem + L.off);
    const uint32_t psign = (uint32_t)((n + 1) * L.qs);
    const int G = T / KB, NGK = nh / KB;
    // per group: symmetric, the byte offset of its symmetry index in a row of
    // the offset table; basic, unused.  ko: byte offset of its first entry in a row
    uint32_t s2[NG], ko[NG];
#pragma unroll
    for (int j = 0; j < NG; j++) {
        const int g = lane + 32 * j;
        const bool ok = g < G;
        s2[j] = 2u * (uint32_t)(SYM ? (ok ? g / NGK : m.S) : 0);
        ko[j] = 8u * (uint32_t)(SYM ? (ok ? (g % NGK) * KB : 0) : (ok ? g * KB : 0));
    }

    // theta of configuration S->start (FP64, down spins in increasing order)
    // into the scratch, two groups at a time
    auto theta_of = [&]() {
        constexpr int NJ = NG >= 2 ? 2 : 1;
#pragma unroll 1
        for (int j0 = 0; j0 < NG; j0 += NJ) {
            double2 acc[NJ * KB];
            int gs[NJ], gk[NJ];
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int g = min(lane + 32 * (j0 + j), G - 1);  // beyond T: computed, not stored
                gs[j] = SYM ? g / NGK : 0;
                gk[j] = SYM ? (g - gs[j] * NGK) * KB : g * KB;
#pragma unroll
                for (int i = 0; i < KB; i++) acc[KB * j + i] = base[KB * g + i];
            }
#pragma unroll 1
            for (int wd = 0; wd < 4; wd++) {
                uint32_t bits = S->start[wd];
                while (bits) {
                    const int f = 32 * wd + __ffs(bits) - 1;
                    bits &= bits - 1;
#pragma unroll
                    for (int j = 0; j < NJ; j++) {
                        const double2* w = W64 + (SYM ? (int)rows[f * SP + gs[j]] : f) * L.ws64 + gk[j];
#pragma unroll
                        for (int i = 0; i < KB; i++) {
                            const double2 v = w[i];
                            acc[KB * j + i].x = fma(-2.0, v.x, acc[KB * j + i].x);
                            acc[KB * j + i].y = fma(-2.0, v.y, acc[KB * j + i].y);
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int g = lane + 32 * (j0 + j);
                if (g < G)
#pragma unroll
                    for (int i = 0; i < KB; i++) {
                        if constexpr (F64)
                            th[KB * g + i] = acc[KB * j + i];
                        else
                            th[KB * g + i] = make_float2((float)acc[KB * j + i].x, (float)acc[KB * j + i].y);
                    }
            }
        }
        __syncwarp();
    };
    // W entry t of site f
    auto wrow = [&](int f, int t) -> float2 {
        if constexpr (SYM) {
            const int g = t / KB, q = NGK == 1 ? g : g / NGK, k = (g - q * NGK) * KB + t % KB;
            return lds_f2(wa + (uint32_t)(rows[f * SP + q] * L.qs) + 8u * k);
        } else if constexpr (PS) {
            return lds_f2(wa + (uint32_t)(f * L.qs) + 8u * t);
        } else {
            return __ldg(m.W32 + f * nh + t);
        }
    };
    // The FP64 sessions' decision: u < |psi'/psi|^2 by the ln|cosh| sums in FP64, after
    // the accepted flips from `applied` on have been applied to theta in the
    // scratch.  The sum at theta is kept for the next open proposal (S->sum, of
    // the sweep's first S->sum_np flips).
    auto decide_fp64 = [&](uint32_t code, uint32_t prop, int applied, int np) -> bool {
        auto w64 = [&](int f, int q, int k) -> double2 {
            return W64[(SYM ? (int)rows[f * SP + q] : f) * L.ws64 + k];
        };
        const int f0 = code & 255u, f1 = (code >> 8) & 255u;
        const bool bond = (code >> 16) & 1u, kept = S->sum_np == np;
        const double g0 = (code >> 17) & 1u ? 2.0 : -2.0, g1 = (code >> 18) & 1u ? 2.0 : -2.0;
        double sx = 0, sy = 0;
#pragma unroll 1
        for (int t = lane; t < T; t += 32) {
            const int q = SYM ? t / nh : 0, k = SYM ? t - q * nh : t;
            double2 x;
            if constexpr (F64) x = th[t];
#pragma unroll 1
            for (int i = applied; i < np; i++) {
                const uint32_t c = plist[i];
                const double h0 = (c >> 17) & 1u ? 2.0 : -2.0, h1 = (c >> 18) & 1u ? 2.0 : -2.0;
                double2 w = w64(c & 255u, q, k);
                x.x = fma(h0, w.x, x.x);
                x.y = fma(h0, w.y, x.y);
                if ((c >> 16) & 1u) {
                    w = w64((c >> 8) & 255u, q, k);
                    x.x = fma(h1, w.x, x.x);
                    x.y = fma(h1, w.y, x.y);
                }
            }
            if constexpr (F64) th[t] = x;
            if (!kept) sx += lnc_re<double>(x.x, x.y);
            double2 w = w64(f0, q, k);
            double2 y = make_double2(fma(g0, w.x, x.x), fma(g0, w.y, x.y));
            if (bond) {
                w = w64(f1, q, k);
                y = make_double2(fma(g1, w.x, y.x), fma(g1, w.y, y.y));
            }
            sy += lnc_re<double>(y.x, y.y);
        }
        sx = kept ? S->sum : warp_sum(sx);
        sy = warp_sum(sy);
        double d = sy - sx + g0 * m.vb[f0 % m.n_vb].x;
        if (bond) d += g1 * m.vb[f1 % m.n_vb].x;
        const uint4 r = philox4x32(make_uint4(prop, epoch, (uint32_t)chain, 0), key);
        const bool accept = unit24<double>(r.z) < exp(2.0 * d);
        __syncwarp();
        if (lane == 0) {
            S->sum = accept ? sy : sx;
            S->sum_np = accept ? np + 1 : np;
        }
        return accept;
    };
    // d of a proposal (code: sites, bond flag in bit 16, spins of the sites in
    // bits 17 and 18) by the ln|cosh| sums of theta and theta' over the entries
    // lane + 32 e, in the arithmetic of lnc_sweep_sum and sweep_sum, after the
    // accepted flips from `applied` on have been applied to theta in the scratch
    float2* th32 = reinterpret_cast<float2*>(th);
    auto decide_exact = [&](uint32_t code, int applied, int np) -> float {
#pragma unroll 1
        for (; applied < np; applied++) {
            const uint32_t c = plist[applied];
            const int q0 = c & 255u, q1 = (c >> 8) & 255u;
            const float h0 = (c >> 17) & 1u ? 2.f : -2.f, h1 = (c >> 18) & 1u ? 2.f : -2.f;
            const bool two = (c >> 16) & 1u;
#pragma unroll 4
            for (int t = lane; t < T; t += 32) {
                float2 v = __ffma2_rn(make_float2(h0, h0), wrow(q0, t), th32[t]);
                if (two) v = __ffma2_rn(make_float2(h1, h1), wrow(q1, t), v);
                th32[t] = v;
            }
        }
        const int f0 = code & 255u, f1 = (code >> 8) & 255u;
        const bool bond = (code >> 16) & 1u;
        const float g0 = (code >> 17) & 1u ? 2.f : -2.f, g1 = (code >> 18) & 1u ? 2.f : -2.f;
        float sa0 = 0.f, lg0 = 0.f, sa1 = 0.f, lg1 = 0.f;
#pragma unroll 1
        for (int e0 = 0; e0 < a.plan.lane_entries; e0 += 4) {
            float pm0 = 1.f, pm1 = 1.f;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (e0 + q >= a.plan.lane_entries) break;
                const int t = lane + 32 * (e0 + q);
                float2 x = make_float2(0.f, 0.f), y = x;
                if (t < T) {
                    x = th32[t];
                    y = __ffma2_rn(make_float2(g0, g0), wrow(f0, t), x);
                    if (bond) y = __ffma2_rn(make_float2(g1, g1), wrow(f1, t), y);
                }
                const float ax = fabsf(x.x), ay = fabsf(y.x);
                const float zx = ex2_ftz(ax * -2.88539008177792681f), zy = ex2_ftz(ay * -2.88539008177792681f);
                const float cx = cos_ftz(2.f * x.y), cy = cos_ftz(2.f * y.y);
                pm0 *= fmaf(zx, fmaf(2.f, cx, zx), 1.f);
                pm1 *= fmaf(zy, fmaf(2.f, cy, zy), 1.f);
                sa0 += ax;
                sa1 += ay;
            }
            lg0 += lg2_ftz(pm0);
            lg1 += lg2_ftz(pm1);
        }
        const float s0 = fmaf(0.346573590279972655f, lg0, sa0), s1 = fmaf(0.346573590279972655f, lg1, sa1);
        float d = sweep_sum(s1 - s0);
        d = fmaf(g0, lds_f2(sa + 8u * f0).x, d);
        return fmaf(g1, lds_f2(sa + 8u * f1).x, d);
    };

    // squared moduli of 1 + z over the lane's entries: the sum of their lg2 in
    // 2^-16 steps over the warp (times ln 2 / 2: sum ln|1 + z|) and one over their
    // minimum
    const Margin& mar = *reinterpret_cast<const Margin*>(smem + L.mar);
    constexpr float kStep = 0.346573590279972655f / 65536.f;
    auto log_sum = [&](const float2 (&xr)[NP], const float2 (&xi)[NP], float& inv) -> int {
        float lg = 0.f, lo = 1e30f;
        const float2 one = make_float2(1.f, 1.f);
#pragma unroll
        for (int p = 0; p < NP; p += 2) {
            const float2 u = __fadd2_rn(xr[p], one);
            float2 q = __ffma2_rn(u, u, __fmul2_rn(xi[p], xi[p]));
            lo = fminf(lo, fminf(q.x, q.y));
            if (p + 1 < NP) {
                const float2 v = __fadd2_rn(xr[p + 1], one);
                const float2 r = __ffma2_rn(v, v, __fmul2_rn(xi[p + 1], xi[p + 1]));
                lo = fminf(lo, fminf(r.x, r.y));
                q = __fmul2_rn(q, r);
            }
            lg += lg2_ftz(q.x * q.y);
        }
        // outside +-511 (or NaN): a minimum of 0, an infinite margin.  Inside, two
        // totals differ by less than 2^31 steps
        const float mn = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(fabsf(lg) < 511.f ? lo : 0.f)));
        inv = __fdividef(1.f, mn);
        if constexpr (F64)
            if (!(mn > mar.mn_min)) inv = __int_as_float(0x7f800000);
        return __reduce_add_sync(kFull, __float2int_rn(lg * 65536.f));
    };
    const float m0 = mar.m0, coef = mar.coef;
    // FP64 margin's part that accepted proposals change
    auto margin = [&](int LS, int k, float& eps) -> float {
        eps = fmaf(mar.eps1, (float)k, mar.eps0);
        return fmaf(mar.R2 * kStep, fabsf((float)LS), mar.R0);
    };
    // w = x p(f, spin sg)
    auto times_p = [&](int f, int sg, const float2 (&xr)[NP], const float2 (&xi)[NP], float2 (&wr)[NP],
                       float2 (&wi)[NP]) {
        auto mul = [&](int p, float2 pr, float2 pi) {
            const float2 yr = xr[p], yi = xi[p];
            wr[p] = __ffma2_rn(yr, pr, __fmul2_rn(make_float2(-yi.x, -yi.y), pi));
            wi[p] = __ffma2_rn(yr, pi, __fmul2_rn(yi, pr));
        };
        if constexpr (PS) {
            const uint32_t pb = pa + (sg ? psign : 0u) + (SYM ? 0u : (uint32_t)(f * L.qs));
            const uint32_t ob = oa + 2u * (uint32_t)(f * SP);
            if constexpr (KB == 4) {
#pragma unroll
                for (int j = 0; j < NG; j++) {
                    const uint32_t at = pb + eloc::lds16(ob + s2[j]) + ko[j];
                    const float4 v0 = eloc::lds128(at), v1 = eloc::lds128(at + 16);
                    mul(2 * j, make_float2(v0.x, v0.y), make_float2(v0.z, v0.w));
                    mul(2 * j + 1, make_float2(v1.x, v1.y), make_float2(v1.z, v1.w));
                }
            } else if constexpr (KB == 2) {
#pragma unroll
                for (int j = 0; j < NG; j++) {
                    const float4 v = eloc::lds128(pb + (SYM ? eloc::lds16(ob + s2[j]) : 0u) + ko[j]);
                    mul(j, make_float2(v.x, v.y), make_float2(v.z, v.w));
                }
            } else {
#pragma unroll
                for (int j = 0; j < NG; j += 2) {
                    const float2 v0 = eloc::lds64(pb + eloc::lds16(ob + s2[j]) + ko[j]);
                    const float2 v1 = eloc::lds64(pb + eloc::lds16(ob + s2[j + 1]) + ko[j + 1]);
                    mul(j / 2, make_float2(v0.x, v1.x), make_float2(v0.y, v1.y));
                }
            }
        } else {
            const char* pb = reinterpret_cast<const char*>(m.P32) + (size_t)(sg * n + f) * (8 * nh);
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(pb + ko[j]));
                mul(j, make_float2(v.x, v.y), make_float2(v.z, v.w));
            }
        }
    };

    const int2* bonds = L.bonds_smem ? reinterpret_cast<const int2*>(smem + L.bonds) : a.prop_bonds;
    const int total = segment_sweeps(a);
    const uint32_t thr = a.bond_thr24;
    volatile float hold[8 * NP];  // z, then z p of the open proposal
    bool open = false;            // the loop left at a proposal that needs the exact sums
    for (;;) {
        if (!open) {
            // z from theta at the start of the sweep
            const int st = S->st;
            if (lane < 4) S->start[lane] = S->sp[lane];
            __syncwarp();
            theta_of();
            if (st >= total) break;  // a launch of no sweeps
            float2 zr[NP], zi[NP];
#pragma unroll
            for (int j = 0; j < NG; j++) {
                const int g = lane + 32 * j;
#pragma unroll
                for (int i = 0; i < KB; i++) {
                    // beyond T: 1 (p = 1), whose |1 + z|^2 is never the smallest for
                    // long; basic machines 0, since their p is another group's
                    float2 z = make_float2(SYM ? 1.f : 0.f, 0.f);
                    if (g < G) {
                        const float2 t = make_float2((float)th[KB * g + i].x, (float)th[KB * g + i].y);
                        const float r = ex2_ftz(t.x * -2.88539008177792681f);
                        float s, c;
                        sincos_r(2.f * t.y, &s, &c);
                        z = make_float2(r * c, -r * s);
                    }
                    const int e = j * KB + i;
                    if (e & 1) {
                        zr[e >> 1].y = z.x;
                        zi[e >> 1].y = z.y;
                    } else {
                        zr[e >> 1].x = z.x;
                        zi[e >> 1].x = z.y;
                    }
                }
            }
            float inv;
            const int ls = log_sum(zr, zi, inv);
#pragma unroll
            for (int p = 0; p < NP; p++) {
                hold[4 * p] = zr[p].x;
                hold[4 * p + 1] = zr[p].y;
                hold[4 * p + 2] = zi[p].x;
                hold[4 * p + 3] = zi[p].y;
            }
            if (lane == 0) {
                S->LS = ls;
                S->inv = inv;
                S->k = 0;
                S->applied = 0;
                S->sum_np = -1;
                S->accept = 0;
            }
            __syncwarp();
        } else {
            const int np = S->np;
            int applied = S->applied;
            if (applied < 0) {
                theta_of();
                applied = 0;
                if (lane == 0) S->sum_np = -1;
                __syncwarp();
            }
            bool accept;
            if constexpr (F64)
                accept = decide_fp64(S->code, S->prop - 1, applied, np);
            else
                accept = S->lu < decide_exact(S->code, applied, np);
            __syncwarp();
            if (lane == 0) {
                S->applied = np;
                S->accept = accept;
                if (accept) {
                    const uint32_t c = S->code;
                    S->LS = S->LSn;
                    S->inv = S->inv_n;
                    plist[np] = c;
                    S->np = np + 1;
                    S->nacc++;
                    S->k += (c >> 16) & 1u ? 2 : 1;
                    S->sp[(c & 255u) >> 5] ^= 1u << (c & 31u);
                    if ((c >> 16) & 1u) S->sp[((c >> 8) & 255u) >> 5] ^= 1u << ((c >> 8) & 31u);
                }
            }
            __syncwarp();
        }
        // ---- the sweep loop, from the state
        float2 zr[NP], zi[NP];
        {
            const int o = S->accept ? 4 * NP : 0;
#pragma unroll
            for (int p = 0; p < NP; p++) {
                zr[p] = make_float2(hold[o + 4 * p], hold[o + 4 * p + 1]);
                zi[p] = make_float2(hold[o + 4 * p + 2], hold[o + 4 * p + 3]);
            }
        }
        const uint32_t spa = smem_addr(S->sp);  // the configuration stays in the scratch
        int LS = S->LS;
        float inv = S->inv;
        int st = S->st, slot = S->slot, np = S->np, applied = S->applied;
        uint32_t prop = S->prop, nacc = S->nacc, pcode = 0;
        float plu = 0.f, eps = 0.f, rest = 0.f;
        int k = S->k;
        if constexpr (F64) rest = margin(LS, k, eps);
        auto draw = [&]() {  // this lane's proposal of the batch of 32
            const uint4 r = philox4x32(make_uint4((prop & ~31u) + lane, epoch, (uint32_t)chain, 0), key);
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
        };
        if (prop & 31u) draw();
        open = false;
        for (;;) {
            if (slot >= n) {  // the sweep is done
                if (const int j = sample_slot(a, st); j >= 0) {
                    const size_t idx = (size_t)chain * a.spc + j;
                    __syncwarp();
                    if (lane < 4) a.samples[4 * idx + lane] = S->sp[lane];
                }
                st++;
                slot = np = 0;
                applied = -1;
                if (st == total || st % refresh_of(F64) == 0) break;
                if (lane < 4) S->start[lane] = S->sp[lane];
            }
            if ((prop & 31u) == 0) draw();
            const int src = prop & 31u;
            const uint32_t code = __shfl_sync(kFull, pcode, src);
            const float lu = __shfl_sync(kFull, plu, src);
            prop++;
            const int f0 = code & 255u, f1 = (code >> 8) & 255u;
            const bool bond = (code >> 16) != 0;
            slot += bond ? 2 : 1;
            const uint32_t b0 = (lds_u32(spa + ((f0 >> 5) << 2)) >> (f0 & 31)) & 1u;
            const uint32_t b1 = bond ? (lds_u32(spa + ((f1 >> 5) << 2)) >> (f1 & 31)) & 1u : 0u;
            const float g0 = b0 ? 2.f : -2.f;  // -2 sigma_f
            const float g1 = b1 ? 2.f : -2.f;
            float2 wr[NP], wi[NP];
            times_p(f0, b0, zr, zi, wr, wi);
            if (bond) times_p(f1, b1, wr, wi, wr, wi);
            float inv_n;
            const int LSn = log_sum(wr, wi, inv_n);
            const float D = fmaf(g1, lds_f2(sa + 8u * f1).y, fmaf(g0, lds_f2(sa + 8u * f0).y, (float)(int)((unsigned)LSn - (unsigned)LS) * kStep));
            const uint32_t full = code | (b0 << 17) | (b1 << 18);
            float mg;
            if constexpr (F64)
                mg = fmaf(fmaf(bond ? mar.fac2 : 1.f, eps, mar.R1), fmaf(0.5f, inv + 1.f, inv_n), rest);
            else
                mg = fmaf(coef, inv_n + inv, m0);
            if (!(fabsf(D - lu) > mg)) {
#pragma unroll
                for (int p = 0; p < NP; p++) {
                    hold[4 * (NP + p)] = wr[p].x;
                    hold[4 * (NP + p) + 1] = wr[p].y;
                    hold[4 * (NP + p) + 2] = wi[p].x;
                    hold[4 * (NP + p) + 3] = wi[p].y;
                }
                if (lane == 0) {
                    S->code = full;
                    S->lu = lu;
                    S->LSn = LSn;
                    S->inv_n = inv_n;
                }
                open = true;
                break;
            }
            if (lu < D) {
#pragma unroll
                for (int p = 0; p < NP; p++) {
                    zr[p] = wr[p];
                    zi[p] = wi[p];
                }
                LS = LSn;
                inv = inv_n;
                if (lane == 0) {
                    plist[np] = full;
                    S->sp[f0 >> 5] ^= 1u << (f0 & 31);
                    if (bond) S->sp[f1 >> 5] ^= 1u << (f1 & 31);
                }
                __syncwarp();
                np++;
                nacc++;
                if constexpr (F64) {
                    k += bond ? 2 : 1;
                    rest = margin(LS, k, eps);
                }
            }
        }
        // ---- back to the state
        if (open) {
#pragma unroll
            for (int p = 0; p < NP; p++) {
                hold[4 * p] = zr[p].x;
                hold[4 * p + 1] = zr[p].y;
                hold[4 * p + 2] = zi[p].x;
                hold[4 * p + 3] = zi[p].y;
            }
        }
        if (lane == 0) {
            S->LS = LS;
            S->inv = inv;
            S->st = st;
            S->slot = slot;
            S->np = np;
            S->applied = applied;
            S->prop = prop;
            S->nacc = nacc;
            S->k = k;
        }
        __syncwarp();
        if (!open && st == total) break;
    }
    const uint32_t sp[4] = {S->sp[0], S->sp[1], S->sp[2], S->sp[3]};
    chain_finish(a, chain, lane, sp, S->nacc, S->prop);
    __syncwarp();
}

// Threads per block by entries per lane: z and z p of the entries in registers
// (16 entries: 128 registers; with 640 threads and 96 the loop spills).
__host__ __device__ constexpr int max_threads(int E) { return E >= 16 ? 512 : (E >= 8 ? 768 : 896); }

template <int KB, int NG, bool SYM, bool PS, bool F64>
__global__ void __launch_bounds__(max_threads(KB* NG), 1) screen_kernel(const SamplerArgs a, const Layout L) {
    extern __shared__ __align__(16) unsigned char smem[];
    load_tables(a, L, smem, F64);
    if (reinterpret_cast<const Margin*>(smem + L.mar)->off) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_warps = (blockDim.x >> 5) * gridDim.x;
    // consecutive chains on different SMs
    for (int chain = warp * gridDim.x + blockIdx.x; chain < a.n_chains; chain += total_warps)
        run_chain<KB, NG, SYM, PS, F64>(a, L, smem, smem + L.warp0 + warp * L.warp_bytes, chain, lane);
}

template <int KB, int NG, bool SYM, bool PS, bool F64> const void* fn() {
    return reinterpret_cast<const void*>(screen_kernel<KB, NG, SYM, PS, F64>);
}

// groups per lane
inline int groups(const MachineDev& m) {
    const int kb = group_width(m), G = m.T / kb;
    int ng = kb == 1 ? 2 : 1;  // entries come in pairs
    while (32 * ng < G) ng *= 2;
    return ng;
}

// kernel of a machine; the instantiations are split over two files that compile
// in parallel (null: none)
const void* pick_fp32(const MachineDev& m, bool p_smem);
const void* pick_fp64(const MachineDev& m, bool p_smem);

}  // namespace screen
}  // namespace rbmnqs
