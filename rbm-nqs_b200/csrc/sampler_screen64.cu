// sampler_screen64.cu -- the screened sweep's kernels for FP64 sessions
// (sampler_screen.cuh): every size, since the exact FP64 sums cost an exponential,
// a sine, a cosine and a logarithm in FP64 per entry and proposal.
#include "sampler_screen.cuh"

namespace rbmnqs {
namespace screen {

const void* pick_fp64(const MachineDev& m, bool p_smem) {
    const int kb = group_width(m), ng = groups(m);
    if (!m.symmetric) {
        switch (ng) {
            case 1: return p_smem ? fn<2, 1, false, true, true>() : fn<2, 1, false, false, true>();
            case 2: return p_smem ? fn<2, 2, false, true, true>() : fn<2, 2, false, false, true>();
            case 4: return p_smem ? fn<2, 4, false, true, true>() : fn<2, 4, false, false, true>();
            case 8: return p_smem ? fn<2, 8, false, true, true>() : fn<2, 8, false, false, true>();
        }
        return nullptr;
    }
    switch (100 * kb + ng) {
        case 401: return fn<4, 1, true, true, true>();
        case 402: return fn<4, 2, true, true, true>();
        case 404: return fn<4, 4, true, true, true>();
        case 201: return fn<2, 1, true, true, true>();
        case 202: return fn<2, 2, true, true, true>();
        case 204: return fn<2, 4, true, true, true>();
        case 208: return fn<2, 8, true, true, true>();
        case 102: return fn<1, 2, true, true, true>();
        case 104: return fn<1, 4, true, true, true>();
        case 108: return fn<1, 8, true, true, true>();
        case 116: return fn<1, 16, true, true, true>();
    }
    return nullptr;
}

}  // namespace screen
}  // namespace rbmnqs
