// The parameters of a wave's kernels as fake_cudart.cpp logs them (WaveParams needs nvcc).
#include "../skirt7_b200/csrc/skg_scene.cuh"

#include <cstdio>
#include <cstring>

size_t fake_params_size() { return sizeof(skg::WaveParams); }

void fake_params(const void* params, char* out, size_t n) {
    skg::WaveParams W;
    memcpy(&W, params, sizeof(W));
    snprintf(out, n, "wave %d npool %d path_tau %d ordered %d max_scatt %d refill %d", W.wave, W.npool, W.path_tau,
             W.hist != nullptr, W.R.max_scatt, W.R.refill);
}

void fake_launch_pass(const void* params, int busy, int jobs) {
    skg::WaveParams W;
    memcpy(&W, params, sizeof(W));
    if (W.wave < busy) W.jcount[skg::J_PATH] = (unsigned)jobs;
}
