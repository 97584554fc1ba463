// Mixed FP32/FP64 instantiation of the trace kernels (fused multiply-add allowed).
#include "st_launch.h"
#include "st_trace_impl.cuh"

namespace stb {
// element tests of the grid probe's candidates
template <int FLAT>
static void resolve(const SceneDev &S, uint64_t s0, const ProbeOut &o, const RunState *rs, cudaStream_t st) {
    // persistent grid: every resident block on every SM
    constexpr int kBlocks = FLAT ? kResolveFlatMinBlocks : kResolveMinBlocks;
    static const int per_sm = resident_blocks(k_sun_resolve<1, kBlocks, FLAT>, kResolveBlock);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_sun_resolve<1, kBlocks, FLAT><<<sms * per_sm, kResolveBlock, 0, st>>>(S, s0, o, rs);
}
int launch_probe_mixed(const SceneDev &S, uint64_t s0, uint32_t n, const ProbeOut &o, const RunState *rs,
                      cudaStream_t st) {
    if (S.sun.grid_on && !S.explicit_rays && !S.sun.point_source) {
        if (launch_sun_probe_flat(S, s0, n, o, rs, st)) {
            int dev = 0, sms = 148;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            k_sun_resolve_amb<1><<<sms, kResolveBlock, 0, st>>>(S, s0, o);
            return 2;
        }
        launch_sun_candidates(S, s0, n, o, rs, st);
        // first stages of flat elements only take the flat-only variant
        if (S.stages[0].flat_only)
            resolve<1>(S, s0, o, rs, st);
        else
            resolve<0>(S, s0, o, rs, st);
        return 2;
    }
    launch_k_probe<1>(S, s0, n, o, rs, st);
    return 1;
}

int launch_trace_mixed(bool records, const SceneDev &S, const HitRec *hits, const uint32_t *total,
                      const RunState *rs, const TraceOut &O, const WfState &W, const WfQueues &Q,
                      const ReplayIn *replay, cudaStream_t st) {
    return records ? wf_launch<1, 1>(S, hits, total, rs, O, W, Q, replay, st)
                   : wf_launch<1, 0>(S, hits, total, rs, O, W, Q, replay, st);
}
// finite-element queries of this precision's kernels that found too few nodes since the
// last call (the flag is cleared)
unsigned take_fe_failures_mixed() {
    unsigned v = 0;
    if (cudaMemcpyFromSymbol(&v, g_fe_fail, sizeof v) != cudaSuccess) return 0;
    if (v) {
        const unsigned z = 0;
        cudaMemcpyToSymbol(g_fe_fail, &z, sizeof z);
    }
    return v;
}
}  // namespace stb
