// The megakernel integrator's record mode (sm_103a): per-sample radiance and event hashes, one thread per
// pixel (k_pathtrace, megakernel.cuh).  A translation unit of its own, compiled with the
// double-precision math of libm_double in line: out of line, as the other kernels have it, this kernel's calls
// cost it 5 % (box scene, 128 x 128, 4 spp recorded: 1.34 ms on the device in line, 1.40 out of line;
// k_mega the other way round, 4.74 out of line and 4.80 in line on the instanced stress scene).
#define LTS_LIBM_CALL __forceinline__
#include <cuda_runtime.h>

#include <string>

#include "dev_common.cuh"
#include "dev_math.cuh"
#include "once_per_device.hpp"
#include "tracer.cuh"
#include "tracer_dev.cuh"
#include "megakernel.cuh"

namespace lts {

#define TRY(call)                                                                       \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
    } while (0)

std::string pathtrace_init() {
    static OncePerDevice once;
    int dev = 0;
    TRY(cudaGetDevice(&dev));
    return once.run(dev, []() -> std::string {
        unsigned char p2[512];
        const float* mc = nullptr;
        texture_tables(p2, &mc);
        TRY(cudaMemcpyToSymbol(c_perm, p2, 512));
        TRY(cudaMemcpyToSymbol(c_marble, mc, 30 * sizeof(float)));
        return "";
    });
}

std::string pathtrace_set_libm_double(int on) {
    const int v = on ? 1 : 0;
    TRY(cudaMemcpyToSymbol(c_libm_double, &v, sizeof v));
    return "";
}

std::string pathtrace_record_launch(const SceneView& sv, const RenderParams& rp, int nleaf, cudaStream_t s) {
    const dim3 block(kBX, kBY);
    const dim3 grid((rp.x1 - rp.x0 + kBX - 1) / kBX, (rp.y1 - rp.y0 + kBY - 1) / kBY);
    k_pathtrace<true><<<grid, block, 0, s>>>(sv, rp, nleaf);
    TRY(cudaGetLastError());
    return "";
}

}  // namespace lts
