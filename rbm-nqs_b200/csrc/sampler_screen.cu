// sampler_screen.cu -- plan and launch of the screened sweep (sampler_screen.cuh),
// one session per launch, persistent warps; its FP32 kernels.
#include <algorithm>

#include "sampler_screen.cuh"

namespace rbmnqs {
namespace screen {

// FP32: 16 entries per lane.  With fewer the exact sums alone are as fast (they
// need 3 special functions an entry; the screen's fixed cost per proposal is
// about 60 instructions): 32 spins, 128 entries, 4096 chains x 64 sweeps: 0.98 ms
// screened, 0.95 ms by the sums; 98 spins, 196 entries, 1000 chains x 31 sweeps:
// 2.1 and 2.0 ms.
const void* pick_fp32(const MachineDev& m, bool p_smem) {
    const int kb = group_width(m), ng = groups(m);
    if (!m.symmetric) return ng != 8 ? nullptr : (p_smem ? fn<2, 8, false, true, false>() : fn<2, 8, false, false, false>());
    switch (100 * kb + ng) {
        case 404: return fn<4, 4, true, true, false>();
        case 208: return fn<2, 8, true, true, false>();
        case 116: return fn<1, 16, true, true, false>();
    }
    return nullptr;
}

}  // namespace screen

namespace {

// a basic machine's p and W rows stay in shared memory up to this size (one
// copy per block of up to 32 warps), else p is read from L2
constexpr int kBasicRows = 120 * 1024;

}  // namespace

bool plan_screen(const MachineDev& m, int fp64, int n_chains, int n_bonds, int max_wpb, SamplerShape* out, cudaError_t* err) {
    if (!m.symmetric && (m.nh & 1)) return false;
    int dev = 0, sms = 0, smem_max = 0;
    if ((*err = cudaGetDevice(&dev)) != cudaSuccess) return true;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int budget = smem_max - 8 * 1024;
    screen::Layout L = screen::make_layout(m, n_bonds, 1, kBasicRows, fp64);
    if (m.symmetric && (m.n + 1) * L.qs > 0xffff) return false;  // 16-bit row offsets
    const void* f = fp64 ? screen::pick_fp64(m, L.p_smem) : screen::pick_fp32(m, L.p_smem);
    if (!f) return false;
    cudaFuncAttributes fa;
    if ((*err = cudaFuncGetAttributes(&fa, f)) != cudaSuccess) return true;
    // one block per SM with enough warps to hold every chain, limited by
    // the kernel's thread bound, registers and shared memory
    const int regs = fa.numRegs > 0 ? fa.numRegs : 64;
    int wpb = std::min(fa.maxThreadsPerBlock / 32, 65536 / (regs * 32));
    wpb = std::min(wpb, (n_chains + sms - 1) / sms);
    if (max_wpb > 0) wpb = std::min(wpb, max_wpb);
    wpb = std::max(wpb, 1);
    while (wpb > 1 && screen::make_layout(m, n_bonds, wpb, kBasicRows, fp64).total > budget) wpb--;
    L = screen::make_layout(m, n_bonds, wpb, kBasicRows, fp64);
    if (L.total > budget) return false;
    if ((*err = ensure_dynamic_smem(f, L.total)) != cudaSuccess) return true;
    int per_sm = 0;
    if ((*err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, 32 * wpb, L.total)) != cudaSuccess) return true;
    const long blocks = std::min<long>(((long)n_chains + wpb - 1) / wpb, (long)sms * std::max(per_sm, 1));
    SmemPlan pl{};
    pl.screen = 1;
    pl.lane_entries = elements_per_lane(m.T);
    pl.p_budget = kBasicRows;
    out->plan = pl;
    out->warps_per_block = wpb;
    out->blocks = (int)blocks;
    out->smem = L.total;
    return true;
}

cudaError_t launch_screen(const SamplerArgs& a0, int fp64, const SamplerShape& sh, cudaStream_t st) {
    SamplerArgs a = a0;
    screen::Layout L = screen::make_layout(a.m, a.n_prop_bonds, sh.warps_per_block, sh.plan.p_budget, fp64);
    const void* f = fp64 ? screen::pick_fp64(a.m, L.p_smem) : screen::pick_fp32(a.m, L.p_smem);
    if (!f || L.total != sh.smem || !a.m.P32 || !a.screen_off) return cudaErrorInvalidValue;
    const cudaError_t e = ensure_dynamic_smem(f, L.total);
    if (e != cudaSuccess) return e;
    void* args[] = {&a, &L};
    return cudaLaunchKernel(f, dim3(sh.blocks), dim3(32 * sh.warps_per_block), args, (size_t)L.total, st);
}

}  // namespace rbmnqs
