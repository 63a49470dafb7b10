// cg_factored.cu -- matrix-free SR conjugate gradients (cg_solver.cpp:260-334,
// cg1 semantics) of basic RBMs, one or many systems in one cooperative
// persistent launch, on the factors of O instead of O itself.
//
// A sample's log-derivatives of a basic RBM are the outer product of its
// spins and its hidden activations (rbm_base.cpp:194-217): with s = (sigma, 1)
// and t = (tanh theta, 1), O[v_j] = sigma_j, O[h_k] = t_k, O[W_jk] = sigma_j t_k.
// The operator of cg_solver.cpp aprod,
//   A b = (1/N) O^H (O b) - conj(d) (d . b) + f o b,
//   f_p = diag_p (r1 (+ rd for non-neural p)) + r2 max(diag),
// then needs the N x (n + nh) factors only:
//   u_n   = sum_k t_nk (b_hk + sum_j sigma_nj B_jk) + sum_j sigma_nj b_vj,
//   Y_jk  = sum_n sigma_nj conj(t_nk) (u_n - d . b),   A b = Y / N + f o b
// (d = <O>, so the mean's share is taken out of u before the second product),
// two FP64 contractions of 2 N n nh multiply-adds each.  sigma comes from the
// samples' bits, t from the first n + nh entries of the stored O rows: per
// system 2 MB instead of the 271 MB of O (128 spins, alpha = 2, 1024 samples),
// so the factors stay in L2 and the bound is the FP64 tensor pipe
// (mma.sync m16n8k8.f64) instead of HBM; what is left above it is the
// latency of three grid barriers and of staging through L2.  Measured against
// O streamed twice per iteration (cg_multi.cu, which stays for the systems
// without this structure: symmetric machines, the Pfaffian factor, full
// enumeration): twelve toric-code problems, L = 3..8 and 1024 samples, 100
// iterations 58 -> 7.5 ms; one system of 98 spins, 19502 parameters and 1000
// samples, 60 iterations 6.8 -> 1.6 ms.
//
// Three phases per iteration, a grid barrier after each, all systems of the
// launch in lockstep:
//   A  units of 64 samples x 32 hidden units: B_jk of the unit's columns in
//      shared memory (kept while the block's next unit has the same
//      columns), partial u per column tile, one more partial for the visible
//      biases; d . b and sum f |b|^2 per tile of 128 parameters;
//   B  units of 64 sites x 16 hidden units x one sample chunk (at most
//      kMaxChunks per system): conj(t) u in shared memory, partial Y per chunk,
//      sum |u - d . b|^2 per chunk;
//   C  p^H A p = sum |u - d . b|^2 / N + sum f |p|^2, then p, x, r and
//      ||r||^2 per tile of 128 parameters.
// Units go to blocks as contiguous ranges of equal cost.  Tiles, chunks and
// the order of every sum depend only on the system's sizes, so a system's
// result depends neither on the grid nor on the launch's other systems.
// Barriers are bounded (coop.cuh): a timeout marks every system's result
// with status -2 and the kernel returns.
#include <algorithm>

#include "common.cuh"
#include "coop.cuh"
#include "sr.cuh"

namespace rbmnqs {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsA = 64;    // samples per phase-A unit
constexpr int kHidA = 32;     // hidden units per phase-A unit
constexpr int kSitesB = 64;   // sites per phase-B unit
constexpr int kHidB = 16;     // hidden units per phase-B unit
constexpr int kStep = 256;    // samples staged at a time in phase B
constexpr int kMaxChunks = 8;
constexpr int kTile = 128;    // parameters per phase-C tile (four tiles per pass of the block)
constexpr int kMaxSites = 128;
constexpr int kCostV = 24;    // cost of a visible row unit (phase A), in the units of Shape's costs
// Row strides (doubles) of the staged operands: 4 mod 16, so that the 16
// lanes of a half warp (four rows, four columns) read distinct bank pairs.
constexpr int kStrideA = 2 * kHidA + 4;
constexpr int kStrideB = 2 * kHidB + 4;
constexpr int kStageBytes = kStep * kStrideB * 8;
static_assert(kMaxSites * kStrideA * 8 <= kStageBytes, "phase-A operand fits the stage");
constexpr int kOffV = kStageBytes;                 // u of the staged samples
constexpr int kOffW = kOffV + kStep * 16;          // their spins
constexpr int kOffBv = kOffW + kStep * 16;         // b of the visible biases
constexpr int kOffRed = kOffBv + kMaxSites * 16;   // reductions
constexpr int kSmemBytes = kOffRed + (kWarps / 2) * 32 * 8 * 8;

struct SysState {
    double rsold, beta, db_x, db_y, pap, rs;
    int itn, done;
};

// D += A B, A 16 x 8 (rows of +-1), B 8 x 8, FP64
__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4], double b0, double b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
// +1.0, or -1.0 where bit s of w is set
__device__ __forceinline__ double sign_of(uint32_t w, int s) {
    return __hiloint2double((int)(0x3ff00000u | ((w << (31 - s)) & 0x80000000u)), 0);
}

// [lo, hi): the units of a system whose start cost lies in [c0, c1)
__device__ __forceinline__ void owned(long long c0, long long c1, long long cost0, long long unit_cost, int units,
                                      int& lo, int& hi) {
    auto first_at = [&](long long c) -> long long {
        return c <= cost0 ? 0 : (c - cost0 + unit_cost - 1) / unit_cost;
    };
    lo = (int)min(first_at(c0), (long long)units);
    hi = (int)min(first_at(c1), (long long)units);
}

struct Shape {
    int kta, rta, ktb, jtb, js, chunk, nch, tiles;
    long long cost_a, cost_b, cost_t;
};
__host__ __device__ inline Shape shape_of(const CgFactProb& p) {
    Shape s;
    s.kta = (p.nh + kHidA - 1) / kHidA;
    s.rta = (p.N + kRowsA - 1) / kRowsA;
    s.ktb = (p.nh + kHidB - 1) / kHidB;
    s.jtb = (p.n + kSitesB - 1) / kSitesB;
    s.js = 16 * ((((p.n + 15) / 16) + s.jtb - 1) / s.jtb);  // sites per unit: equal shares of 16-site groups
    s.chunk = kStep * ((p.N + kStep * kMaxChunks - 1) / (kStep * kMaxChunks));
    s.nch = (p.N + s.chunk - 1) / s.chunk;
    s.tiles = (p.P + kTile - 1) / kTile;
    // a unit's time: its products plus a fixed part (staging, reductions)
    // worth about 20 sites (A) or 128 samples of 64 sites (B)
    s.cost_a = p.n + 20;
    s.cost_b = (long long)(s.chunk < p.N ? s.chunk : p.N) * ((p.n + 15) / 16) / (8 * s.jtb) + 64 * (s.chunk / kStep);
    s.cost_t = 6;
    return s;
}

// A block's share of a system, fixed for the launch: phase-A units, visible
// row units and tiles (phase A, one cost line), phase-B units, phase-C tiles.
struct Share {
    int kta, rta, ktb, jtb, js, chunk, nch, tiles;
    int a0, a1, v0, v1, ta0, ta1, b0, b1, tc0, tc1;
    double r1, r1d, mx;  // regularisation: f_p = diag_p r1 (r1d) + mx
};

template <typename TO>
__global__ void __launch_bounds__(kThreads, 1)
    cg_factored_kernel(const CgFactProb* __restrict__ probs, int nprob, CgFactScratch s) {
    __shared__ CgFactProb pr[kCgMultiMax];
    __shared__ SysState ss[kCgMultiMax];
    __shared__ Share sp[kCgMultiMax];
    __shared__ double2 tred[kWarps];
    __shared__ double tred_f[kWarps];
    __shared__ int any_active;
    extern __shared__ __align__(16) unsigned char smem[];
    double* stage = reinterpret_cast<double*>(smem);
    double2* sV = reinterpret_cast<double2*>(smem + kOffV);
    uint32_t* sW = reinterpret_cast<uint32_t*>(smem + kOffW);
    double2* sBv = reinterpret_cast<double2*>(smem + kOffBv);
    double* red = reinterpret_cast<double*>(smem + kOffRed);
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int lr = lane >> 2, lc = lane & 3;  // row / column of the lane in an mma fragment
    const int G = gridDim.x, blk = blockIdx.x;
    for (int i = tid; i < nprob; i += kThreads) {
        pr[i] = probs[i];
        ss[i] = SysState{};
    }
    __syncthreads();
    if (tid < nprob) {
        const long long ac0 = s.a_cost * blk / G, ac1 = s.a_cost * (blk + 1) / G;
        const long long bc0 = s.b_cost * blk / G, bc1 = s.b_cost * (blk + 1) / G;
        const long long tc0 = s.t_cost * blk / G, tc1 = s.t_cost * (blk + 1) / G;
        const CgFactProb& p = pr[tid];
        const Shape h = shape_of(p);
        Share& o = sp[tid];
        o.kta = h.kta;
        o.rta = h.rta;
        o.ktb = h.ktb;
        o.jtb = h.jtb;
        o.js = h.js;
        o.chunk = h.chunk;
        o.nch = h.nch;
        o.tiles = h.tiles;
        long long at = p.a_cost0;
        owned(ac0, ac1, at, h.cost_a, h.kta * h.rta, o.a0, o.a1);
        at += h.cost_a * h.kta * h.rta;
        owned(ac0, ac1, at, kCostV, h.rta, o.v0, o.v1);
        at += (long long)kCostV * h.rta;
        owned(ac0, ac1, at, h.cost_t, h.tiles, o.ta0, o.ta1);
        owned(bc0, bc1, p.b_cost0, h.cost_b, h.nch * h.ktb * h.jtb, o.b0, o.b1);
        owned(tc0, tc1, p.t_cost0, h.cost_t, h.tiles, o.tc0, o.tc1);
        o.r1 = p.sch->value[1];
        o.r1d = o.r1 + p.sch->value[3];
        o.mx = *p.max_diag * p.sch->value[2];
    }
    __syncthreads();

    // the vector that A multiplies: x (init), else the direction r + beta p
    auto bval = [&](const CgFactProb& p, double beta, bool init, int q) -> double2 {
        if (init) return __ldcg(p.x + q);
        const double2 r = __ldcg(p.r + q);
        if (beta == 0.0) return r;
        const double2 pp = __ldcg(p.p + q);
        return make_double2(fma(beta, pp.x, r.x), fma(beta, pp.y, r.y));
    };
    auto freg = [&](const CgFactProb& p, const Share& sh, int q) -> double {
        return p.diag[q] * (q < p.n_neural ? sh.r1 : sh.r1d) + sh.mx;
    };

    auto phase_a = [&](bool init) {
        int have_i = -1, have_kt = -1;  // columns staged in shared memory
        for (int i = 0; i < nprob; i++) {
            const CgFactProb& p = pr[i];
            if (ss[i].done) continue;
            const double beta = ss[i].beta;
            const Share& sh = sp[i];
            const int n = p.n, nh = p.nh, N = p.N, P = p.P, np = (n + 7) & ~7;
            const TO* O = reinterpret_cast<const TO*>(p.O);
            double2* ru = reinterpret_cast<double2*>(red);
            // warp (wr, wc): 16 samples x 8 hidden units (16 real columns).
            // A unit's spins and activations are loaded while the unit
            // before it is computed
            const int wr = wib & 3, wc = wib >> 2;
            uint4 wa, wb;
            TO ta[2], tb[2];
            auto fetch = [&](int u) {
                const int kt = u / sh.rta, ra = (u - kt * sh.rta) * kRowsA + wr * 16 + lr, rb = ra + 8;
                wa = wb = make_uint4(0, 0, 0, 0);
                if (ra < N) wa = *reinterpret_cast<const uint4*>(p.spins + 4 * (size_t)ra);
                if (rb < N) wb = *reinterpret_cast<const uint4*>(p.spins + 4 * (size_t)rb);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const int k = kt * kHidA + wc * 8 + t * 4 + lc;
                    ta[t] = tb[t] = TO{};
                    if (k < nh && ra < N) ta[t] = O[(size_t)ra * P + n + k];
                    if (k < nh && rb < N) tb[t] = O[(size_t)rb * P + n + k];
                }
            };
            if (sh.a0 < sh.a1) fetch(sh.a0);
            double2 bh[2];
            for (int u = sh.a0; u < sh.a1; u++) {
                const int kt = u / sh.rta, n0 = (u - kt * sh.rta) * kRowsA, k0 = kt * kHidA;
                if (have_i != i || have_kt != kt) {
                    // a warp takes the hidden units wi and wi + 16, its
                    // lanes the sites; all loads in flight before the
                    // stores
                    double2 v[8], vp[8];
                    const double2* b1 = (init ? p.x : p.r) + n + nh;
                    const bool two = !init && beta != 0.0;
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int k = k0 + wib + 16 * (q >> 2), j = lane + 32 * (q & 3);
                        v[q] = vp[q] = make_double2(0, 0);
                        if (j < n && k < nh) v[q] = __ldcg(b1 + j + n * k);
                    }
                    if (two) {
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int k = k0 + wib + 16 * (q >> 2), j = lane + 32 * (q & 3);
                            if (j < n && k < nh) vp[q] = __ldcg(p.p + n + nh + j + n * k);
                        }
                    }
                    __syncthreads();  // the previous unit is done with the stage
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int kk = wib + 16 * (q >> 2), j = lane + 32 * (q & 3);
                        if (j < np)
                            *reinterpret_cast<double2*>(stage + j * kStrideA + 2 * kk) =
                                two ? make_double2(fma(beta, vp[q].x, v[q].x), fma(beta, vp[q].y, v[q].y)) : v[q];
                    }
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const int k = k0 + wc * 8 + t * 4 + lc;
                        bh[t] = k < nh ? bval(p, beta, init, n + k) : make_double2(0, 0);
                    }
                    have_i = i;
                    have_kt = kt;
                    __syncthreads();
                }
                double c[2][4];
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    c[t][0] = c[t][2] = bh[t].x;
                    c[t][1] = c[t][3] = bh[t].y;
                }
                const uint4 xwa = wa, xwb = wb;
                const TO xa2[2] = {ta[0], ta[1]}, xb2[2] = {tb[0], tb[1]};
                if (u + 1 < sh.a1) fetch(u + 1);
                const double* sb = stage + lc * kStrideA + wc * 16 + lr;
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    const uint32_t xa = w == 0 ? xwa.x : (w == 1 ? xwa.y : (w == 2 ? xwa.z : xwa.w));
                    const uint32_t xb = w == 0 ? xwb.x : (w == 1 ? xwb.y : (w == 2 ? xwb.z : xwb.w));
                    const int je = min(np - 32 * w, 32);
                    for (int j = 0; j < je; j += 8) {
                        const double a[4] = {sign_of(xa, j + lc), sign_of(xb, j + lc), sign_of(xa, j + 4 + lc),
                                             sign_of(xb, j + 4 + lc)};
                        const double* bj = sb + (32 * w + j) * kStrideA;
#pragma unroll
                        for (int t = 0; t < 2; t++) mma_f64(c[t], a, bj[8 * t], bj[4 * kStrideA + 8 * t]);
                    }
                }
                // u of the unit's columns: over the lane's hidden units, the
                // four lanes of a row, then the four column warps in order
                double2 ua = make_double2(0, 0), ub = ua;
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    ua.x += xa2[t].x * c[t][0] - xa2[t].y * c[t][1];
                    ua.y += xa2[t].x * c[t][1] + xa2[t].y * c[t][0];
                    ub.x += xb2[t].x * c[t][2] - xb2[t].y * c[t][3];
                    ub.y += xb2[t].x * c[t][3] + xb2[t].y * c[t][2];
                }
#pragma unroll
                for (int o = 1; o <= 2; o <<= 1) {
                    ua.x += __shfl_xor_sync(kFull, ua.x, o);
                    ua.y += __shfl_xor_sync(kFull, ua.y, o);
                    ub.x += __shfl_xor_sync(kFull, ub.x, o);
                    ub.y += __shfl_xor_sync(kFull, ub.y, o);
                }
                if (lc == 0) {
                    ru[wc * kRowsA + wr * 16 + lr] = ua;
                    ru[wc * kRowsA + wr * 16 + lr + 8] = ub;
                }
                __syncthreads();
                if (tid < kRowsA && n0 + tid < N) {
                    double2 t = ru[tid];
                    for (int q = 1; q < 4; q++) {
                        t.x += ru[q * kRowsA + tid].x;
                        t.y += ru[q * kRowsA + tid].y;
                    }
                    p.upart[(size_t)kt * N + n0 + tid] = t;
                }
                __syncthreads();
            }
            // visible biases of 64 samples, eight lanes per sample: the last
            // partial of u
            for (int u = sh.v0; u < sh.v1; u++) {
                const int row = u * kRowsA + (tid >> 3);
                uint4 w = make_uint4(0, 0, 0, 0);
                if (row < N) w = *reinterpret_cast<const uint4*>(p.spins + 4 * (size_t)row);
                if (tid < n) sBv[tid] = bval(p, beta, init, tid);
                __syncthreads();
                double2 v = make_double2(0, 0);
#pragma unroll
                for (int q = 0; q < kMaxSites / 8; q++) {
                    const int j = (tid & 7) + 8 * q;
                    if (j >= n) break;
                    const uint32_t x = q < 4 ? w.x : (q < 8 ? w.y : (q < 12 ? w.z : w.w));
                    const double sg = sign_of(x, j & 31);
                    v.x = fma(sg, sBv[j].x, v.x);
                    v.y = fma(sg, sBv[j].y, v.y);
                }
#pragma unroll
                for (int o = 1; o <= 4; o <<= 1) {
                    v.x += __shfl_xor_sync(kFull, v.x, o);
                    v.y += __shfl_xor_sync(kFull, v.y, o);
                }
                if ((tid & 7) == 0 && row < N) p.upart[(size_t)sh.kta * N + row] = v;
                __syncthreads();
            }
            // d . b and sum f |b|^2 of the owned tiles, four tiles per pass
            const int t1 = sh.ta1;
            for (int t = sh.ta0; t < t1; t += kThreads / kTile) {
                const int tt = t + tid / kTile, q = tt * kTile + tid % kTile;
                double2 db = make_double2(0, 0);
                double fb = 0;
                if (tt < t1 && q < P) {
                    const double2 dq = p.d[q], v = bval(p, beta, init, q);
                    db.x = dq.x * v.x - dq.y * v.y;
                    db.y = dq.x * v.y + dq.y * v.x;
                    fb = freg(p, sh, q) * (v.x * v.x + v.y * v.y);
                }
                db.x = warp_sum(db.x);
                db.y = warp_sum(db.y);
                fb = warp_sum(fb);
                if (lane == 0) {
                    tred[wib] = db;
                    tred_f[wib] = fb;
                }
                __syncthreads();
                if (tid % kTile == 0 && tt < t1) {
                    for (int w = 1; w < kTile / 32; w++) {
                        db.x += tred[wib + w].x;
                        db.y += tred[wib + w].y;
                        fb += tred_f[wib + w];
                    }
                    s.tdb[p.tile0 + tt] = db;
                    s.tfb[p.tile0 + tt] = fb;
                }
                __syncthreads();
            }
        }
    };

    auto phase_b = [&]() {
        int have_i = -1, have_c = -1, have_ch = -1;  // (chunk, hidden tile) and chunk staged in shared memory
        for (int i = 0; i < nprob; i++) {
            const CgFactProb& p = pr[i];
            if (ss[i].done) continue;
            const double dbx = ss[i].db_x, dby = ss[i].db_y;
            const Share& sh = sp[i];
            const int n = p.n, nh = p.nh, N = p.N, P = p.P;
            const TO* O = reinterpret_cast<const TO*>(p.O);
            // the activations of a stage, loaded while the stage before it
            // is computed: hidden unit kk of the samples r0, r0 + 32, ...
            constexpr int RT = kStep / (kThreads / kHidB), RS = kThreads / kHidB;
            const int kk = tid % kHidB, r0 = tid / kHidB;
            const bool one = sh.chunk <= kStep;  // a chunk is one stage, kept from unit to unit
            TO t[RT];
            auto fetch = [&](int u, int m0) {
                const int ck = u / sh.jtb, k = (ck % sh.ktb) * kHidB + kk;
#pragma unroll
                for (int q = 0; q < RT; q++) {
                    const int row = m0 + r0 + q * RS;
                    t[q] = TO{};
                    if (row < N && k < nh) t[q] = O[(size_t)row * P + n + k];
                }
            };
            if (sh.b0 < sh.b1) fetch(sh.b0, sh.b0 / sh.jtb / sh.ktb * sh.chunk);
            for (int u = sh.b0; u < sh.b1; u++) {
                const int ck = u / sh.jtb, jt = u - ck * sh.jtb, ch = ck / sh.ktb, kt = ck - ch * sh.ktb;
                const int j0 = jt * sh.js, j1 = min(n, j0 + sh.js), k0 = kt * kHidB;
                const int s0 = ch * sh.chunk, s1 = min(N, s0 + sh.chunk);
                double2* y = p.ypart + (size_t)ch * P;
                // warp (wj, wc, wk): 16 sites x 8 hidden units x half of the
                // staged samples; a scheduler's four warps have the four wj,
                // so that a short site tile idles none of them
                const int wj = wib >> 2, wc = wib & 1, wk = (wib >> 1) & 1;
                const bool live = j0 + 16 * wj < j1;
                double c[2][4] = {};
                double hs = 0, vv = 0;            // hidden-bias column sum, |u|^2
                double2 vs = make_double2(0, 0);  // visible-bias row sum
                for (int m0 = s0; m0 < s1; m0 += kStep) {
                    const bool fresh = have_i != i || have_c != ck || !one;
                    const bool fresh_v = have_i != i || have_ch != ch || !one;
                    __syncthreads();  // everyone is done with the stage
                    if (fresh_v) {
                        if (tid < kStep) {
                            const int row = m0 + tid;
                            double2 v = make_double2(0, 0);
                            uint4 w = make_uint4(0, 0, 0, 0);
                            if (row < N) {
                                w = *reinterpret_cast<const uint4*>(p.spins + 4 * (size_t)row);
                                for (int q0 = 0; q0 <= sh.kta; q0 += 9) {  // nine loads in flight
                                    double2 x[9];
#pragma unroll
                                    for (int q = 0; q < 9; q++) {
                                        x[q] = make_double2(0, 0);
                                        if (q0 + q <= sh.kta) x[q] = __ldcg(p.upart + (size_t)(q0 + q) * N + row);
                                    }
#pragma unroll
                                    for (int q = 0; q < 9; q++) {
                                        v.x += x[q].x;
                                        v.y += x[q].y;
                                    }
                                }
                                v.x -= dbx;
                                v.y -= dby;
                            }
                            sV[tid] = v;
                            *reinterpret_cast<uint4*>(sW + 4 * tid) = w;
                        }
                        have_ch = ch;
                        __syncthreads();
                    }
                    if (fresh) {
                        // conj(t) u
#pragma unroll
                        for (int q = 0; q < RT; q++) {
                            const int r = r0 + q * RS;
                            const double2 v = sV[r];
                            *reinterpret_cast<double2*>(stage + r * kStrideB + 2 * kk) =
                                make_double2(t[q].x * v.x + t[q].y * v.y, t[q].x * v.y - t[q].y * v.x);
                        }
                        have_i = i;
                        have_c = ck;
                        __syncthreads();
                        if (!one && m0 + kStep < s1)
                            fetch(u, m0 + kStep);
                        else if (!one && u + 1 < sh.b1)
                            fetch(u + 1, (u + 1) / sh.jtb / sh.ktb * sh.chunk);
                        else if (one && (ck + 1) * sh.jtb < sh.b1)  // the next unit with other columns
                            fetch((ck + 1) * sh.jtb, (ck + 1) / sh.ktb * sh.chunk);
                    }
                    if (live) {
                        const int rb = wk * (kStep / 2);
                        const double* sc = stage + (rb + lc) * kStrideB + wc * 16 + lr;
                        const uint32_t* sw = sW + 4 * (rb + lc) + ((j0 + 16 * wj) >> 5);
                        const int sh0 = ((j0 + 16 * wj) & 31) + lr;
                        const int re = min(kStep / 2, s1 - m0 - rb);
#pragma unroll 4
                        for (int r = 0; r < re; r += 8) {
                            const uint32_t x0 = sw[4 * r], x1 = sw[4 * (r + 4)];
                            const double a[4] = {sign_of(x0, sh0), sign_of(x0, sh0 + 8), sign_of(x1, sh0),
                                                 sign_of(x1, sh0 + 8)};
                            const double* br = sc + r * kStrideB;
#pragma unroll
                            for (int t = 0; t < 2; t++) mma_f64(c[t], a, br[8 * t], br[4 * kStrideB + 8 * t]);
                        }
                    }
                    if (jt == 0) {  // hidden biases: 32 real columns x 16 sample groups
                        const double* sc = stage + (tid >> 5) * (kStep / kWarps) * kStrideB + lane;
                        for (int r = 0; r < kStep / kWarps; r++) hs += sc[r * kStrideB];
                        if (kt == 0 && tid < kStep) {
                            const double2 v = sV[tid];
                            vv += v.x * v.x + v.y * v.y;
                        }
                    }
                    if (kt == 0) {  // visible biases: 64 sites x 8 sample groups
                        const int j = j0 + (tid & 63);
                        if (j < j1)
                            for (int r = (tid >> 6) * (kStep / 8); r < ((tid >> 6) + 1) * (kStep / 8); r++) {
                                const double sg = sign_of(sW[4 * r + (j >> 5)], j & 31);
                                vs.x = fma(sg, sV[r].x, vs.x);
                                vs.y = fma(sg, sV[r].y, vs.y);
                            }
                    }
                }
                // the two sample halves, then the rare bias sums, in order
                double* mine = red + ((2 * wj + wc) * 32 + lane) * 8;
                if (wk == 1) {
#pragma unroll
                    for (int t = 0; t < 2; t++)
#pragma unroll
                        for (int e = 0; e < 4; e++) mine[4 * t + e] = c[t][e];
                }
                __syncthreads();
                if (wk == 0) {
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const int k = k0 + wc * 8 + t * 4 + lc, j = j0 + 16 * wj + lr;
                        double2* yk = y + n + nh + (size_t)n * k;
                        if (k < nh && j < j1) yk[j] = make_double2(c[t][0] + mine[4 * t], c[t][1] + mine[4 * t + 1]);
                        if (k < nh && j + 8 < j1)
                            yk[j + 8] = make_double2(c[t][2] + mine[4 * t + 2], c[t][3] + mine[4 * t + 3]);
                    }
                }
                if (jt == 0) {
                    __syncthreads();
                    red[wib * 32 + lane] = hs;
                    __syncthreads();
                    if (tid < 32) {
                        double t = red[tid];
                        for (int w = 1; w < kWarps; w++) t += red[w * 32 + tid];
                        if (k0 + tid / 2 < nh) reinterpret_cast<double*>(y + n + k0)[tid] = t;
                    }
                    if (kt == 0) {
                        const double t = warp_sum(vv);
                        if (lane == 0) tred_f[wib] = t;
                        __syncthreads();
                        if (tid == 0) {
                            double a = tred_f[0];
                            for (int w = 1; w < kStep / 32; w++) a += tred_f[w];
                            p.vv[ch] = a;
                        }
                    }
                }
                if (kt == 0) {
                    __syncthreads();
                    double2* rv = reinterpret_cast<double2*>(red);
                    rv[tid] = vs;
                    __syncthreads();
                    if (tid < 64 && j0 + tid < j1) {
                        double2 t = rv[tid];
                        for (int g = 1; g < 8; g++) {
                            t.x += rv[64 * g + tid].x;
                            t.y += rv[64 * g + tid].y;
                        }
                        y[j0 + tid] = t;
                    }
                }
            }
        }
        __syncthreads();
    };

    auto phase_c = [&](bool init) {
        for (int i = 0; i < nprob; i++) {
            const CgFactProb& p = pr[i];
            const SysState st = ss[i];
            if (st.done) continue;
            const Share& sh = sp[i];
            const int P = p.P;
            const double alpha = init ? 0.0 : st.rsold / st.pap;
            const int t1 = sh.tc1;
            for (int t = sh.tc0; t < t1; t += kThreads / kTile) {
                const int tt = t + tid / kTile, q = tt * kTile + tid % kTile;
                double rl = 0;
                if (tt < t1 && q < P) {
                    double2 y = make_double2(0, 0), yc[kMaxChunks];
#pragma unroll
                    for (int c = 0; c < kMaxChunks; c++) {
                        yc[c] = make_double2(0, 0);
                        if (c < sh.nch) yc[c] = __ldcg(p.ypart + (size_t)c * P + q);
                    }
#pragma unroll
                    for (int c = 0; c < kMaxChunks; c++) {
                        y.x += yc[c].x;
                        y.y += yc[c].y;
                    }
                    const double2 b = bval(p, st.beta, init, q);
                    const double f = freg(p, sh, q);
                    const double ax = fma(f, b.x, y.x / p.norm), ay = fma(f, b.y, y.y / p.norm);
                    double2 r;
                    if (init) {
                        const double2 fq = p.F[q];
                        r = make_double2(fq.x - ax, fq.y - ay);
                    } else {
                        r = __ldcg(p.r + q);
                        double2 x = __ldcg(p.x + q);
                        x.x = fma(alpha, b.x, x.x);
                        x.y = fma(alpha, b.y, x.y);
                        r.x = fma(-alpha, ax, r.x);
                        r.y = fma(-alpha, ay, r.y);
                        p.x[q] = x;
                        p.p[q] = b;
                    }
                    p.r[q] = r;
                    rl = r.x * r.x + r.y * r.y;
                }
                rl = warp_sum(rl);
                if (lane == 0) tred_f[wib] = rl;
                __syncthreads();
                if (tid % kTile == 0 && tt < t1) {
                    for (int w = 1; w < kTile / 32; w++) rl += tred_f[wib + w];
                    s.trs[p.tile0 + tt] = rl;
                }
                __syncthreads();
            }
        }
    };

    // per-system totals of the tile partials, one warp per system
    auto total = [&](const double* part, const CgFactProb& p) -> double {
        const int nt = (p.P + kTile - 1) / kTile;
        double v = 0;
        for (int t0 = lane; t0 < nt; t0 += 9 * 32) {  // nine loads in flight (33152 parameters: 259 tiles)
            double x[9];
#pragma unroll
            for (int q = 0; q < 9; q++) x[q] = t0 + 32 * q < nt ? __ldcg(part + p.tile0 + t0 + 32 * q) : 0.0;
#pragma unroll
            for (int q = 0; q < 9; q++) v += x[q];
        }
        return warp_sum(v);
    };
    auto reduce_db = [&]() {
        for (int i = wib; i < nprob; i += kWarps) {
            const CgFactProb& p = pr[i];
            if (ss[i].done) continue;
            const int nt = (p.P + kTile - 1) / kTile;
            double sx = 0, sy = 0;
            for (int t0 = lane; t0 < nt; t0 += 9 * 32) {
                double2 x[9];
#pragma unroll
                for (int q = 0; q < 9; q++) {
                    x[q] = make_double2(0, 0);
                    if (t0 + 32 * q < nt) x[q] = __ldcg(s.tdb + p.tile0 + t0 + 32 * q);
                }
#pragma unroll
                for (int q = 0; q < 9; q++) {
                    sx += x[q].x;
                    sy += x[q].y;
                }
            }
            sx = warp_sum(sx);
            sy = warp_sum(sy);
            if (lane == 0) {
                ss[i].db_x = sx;
                ss[i].db_y = sy;
            }
        }
        __syncthreads();
    };
    auto reduce_pap = [&]() {
        for (int i = wib; i < nprob; i += kWarps) {
            const CgFactProb& p = pr[i];
            if (ss[i].done) continue;
            const double v0 = lane < sp[i].nch ? __ldcg(p.vv + lane) : 0.0;
            const double fb = total(s.tfb, p), v = warp_sum(v0);
            if (lane == 0) ss[i].pap = v / p.norm + fb;
        }
        __syncthreads();
    };
    auto reduce_rs = [&]() {
        for (int i = wib; i < nprob; i += kWarps) {
            if (ss[i].done) continue;
            const double rs = total(s.trs, pr[i]);
            if (lane == 0) ss[i].rs = rs;
        }
        __syncthreads();
    };
    auto product = [&](bool init) -> bool {
        phase_a(init);
        if (!grid_barrier(s.sync, G)) return false;
        reduce_db();
        phase_b();
        if (!grid_barrier(s.sync, G)) return false;
        reduce_pap();
        phase_c(init);
        if (!grid_barrier(s.sync, G)) return false;
        reduce_rs();
        return true;
    };

    // r = F - A x0, p = r
    bool ok = product(true);
    if (ok) {
        if (tid < nprob) {
            SysState& st = ss[tid];
            st.rsold = st.rs;
            st.beta = 0.0;
            st.itn = 0;
            st.done = pr[tid].max_it <= 0;
        }
        __syncthreads();
    }
    while (ok) {
        if (tid == 0) {
            int a = 0;
            for (int i = 0; i < nprob; i++) a |= !ss[i].done;
            any_active = a;
        }
        __syncthreads();
        if (!any_active) break;
        if (!(ok = product(false))) break;
        if (tid < nprob) {
            SysState& st = ss[tid];
            if (!st.done) {
                if (st.rs < pr[tid].rtol) {
                    st.done = 1;  // cg1: stop before the direction update, itn not advanced
                } else {
                    st.beta = st.rs / st.rsold;
                    st.rsold = st.rs;
                    st.itn++;
                    if (st.itn >= pr[tid].max_it) st.done = 1;
                }
            }
        }
        __syncthreads();
    }
    if (blk == 0 && tid < nprob) {
        CgResultDev* res = pr[tid].res;
        res->status = ok ? 0 : -2;
        res->istop = 0;
        res->qlp_iterations = 0;
        res->acond = 0;
        res->iterations = ss[tid].itn;
        res->residual = ss[tid].rs;
    }
}

const void* kernel_of(int fp64) {
    return fp64 ? reinterpret_cast<const void*>(cg_factored_kernel<double2>)
                : reinterpret_cast<const void*>(cg_factored_kernel<float2>);
}

}  // namespace

size_t cg_fact_work_bytes(int N, int n, int nh) {
    CgFactProb p{};
    p.N = N;
    p.n = n;
    p.nh = nh;
    p.P = n + nh + n * nh;
    const Shape s = shape_of(p);
    return ((size_t)(s.kta + 1) * N + (size_t)s.nch * p.P) * sizeof(double2) + kMaxChunks * sizeof(double);
}

void cg_fact_carve(CgFactProb* p, void* base) {
    const Shape s = shape_of(*p);
    p->upart = reinterpret_cast<double2*>(base);
    p->ypart = p->upart + (size_t)(s.kta + 1) * p->N;
    p->vv = reinterpret_cast<double*>(p->ypart + (size_t)s.nch * p->P);
}

int cg_fact_units(CgFactProb* probs, int nprob, CgFactScratch* sc) {
    long long a = 0, b = 0, t = 0;
    int tiles = 0;
    for (int i = 0; i < nprob; i++) {
        CgFactProb& p = probs[i];
        const Shape s = shape_of(p);
        p.a_cost0 = a;
        p.b_cost0 = b;
        p.t_cost0 = t;
        p.tile0 = tiles;
        a += s.cost_a * s.kta * s.rta + (long long)kCostV * s.rta + s.cost_t * s.tiles;
        b += s.cost_b * s.nch * s.ktb * s.jtb;
        t += s.cost_t * s.tiles;
        tiles += s.tiles;
    }
    sc->a_cost = a;
    sc->b_cost = b;
    sc->t_cost = t;
    return tiles;
}

cudaError_t cg_fact_blocks(int* blocks) {
    int dev = 0, sms = 148, coop = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return cudaErrorNotSupported;
    for (int fp64 = 0; fp64 < 2; fp64++) {
        if ((e = ensure_dynamic_smem(kernel_of(fp64), kSmemBytes)) != cudaSuccess) return e;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_of(fp64), kThreads, kSmemBytes)) !=
            cudaSuccess)
            return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
    }
    *blocks = sms;  // one block per SM
    return cudaSuccess;
}

cudaError_t launch_cg_fact(const CgFactProb* probs_dev, int nprob, int fp64, const CgFactScratch& s, int blocks,
                           cudaStream_t st) {
    if (nprob < 1 || nprob > kCgMultiMax || blocks < 1) return cudaErrorInvalidValue;
    cudaError_t e = launch_init_sync(s.sync, st);
    if (e != cudaSuccess) return e;
    CgFactScratch sc = s;
    const CgFactProb* p = probs_dev;
    int np = nprob;
    void* args[] = {&p, &np, &sc};
    if ((e = ensure_dynamic_smem(kernel_of(fp64), kSmemBytes)) != cudaSuccess) return e;
    return cudaLaunchCooperativeKernel(kernel_of(fp64), dim3(blocks), dim3(kThreads), args, kSmemBytes, st);
}

}  // namespace rbmnqs
