// Per-world free-body control-step kernel, the heterogeneous batch's
// free-body family kernels, and their host launchers; the device code lives
// in scene_step.cuh.
#include "mix.h"
#include "scene_step.cuh"

#include <algorithm>
#include <cstdlib>

namespace numi {
namespace {

// 128 registers: 16 warps per SM, i.e. four environments of four warps.  At
// 96 registers (20 warps) the spills cost more than the warps gave: 36-body
// piles 10.3 against 9.8 ms.
template <bool kComp, bool kConvex>
__global__ void __launch_bounds__(32 * kSceneMaxWarps, 16 / kSceneMaxWarps) scene_step_kernel(const __grid_constant__ SceneParams p) {
    extern __shared__ float4 smem4[];
    const int item = blockIdx.x;
    const int env = p.env_index != nullptr ? p.env_index[item] : item;
    scene_step_item<kComp, kConvex>(p, reinterpret_cast<float*>(smem4), item, env);
}

// The batch's free-body family (mix_step.cu): the claim loop over free-body
// items, one CTA per item.  It sits in this translation unit so that it and
// the per-world kernel call one compiled copy of the control step: a batch
// reproduces each world alone bit for bit.
template <bool kConvex>
__global__ void __launch_bounds__(32 * kSceneMaxWarps, 16 / kSceneMaxWarps)
    mix_scene_kernel(const MixWorld* __restrict__ worlds, int world_count, int steps, const std::uint32_t* __restrict__ items,
                     int item_count, unsigned* next_item) {
    extern __shared__ float4 smem4[];
    __shared__ unsigned next;
    for (;;) {
        if (threadIdx.x == 0) next = atomicAdd(next_item, 1u);
        __syncthreads();
        const unsigned claimed = next;
        __syncthreads();
        if (claimed >= static_cast<unsigned>(item_count)) break;
        const std::uint32_t code = items[claimed];
        const int world = static_cast<int>(code >> kMixWorldShift);
        const int env = static_cast<int>(code & kMixEnvMask);
        for (int k = 0; k < steps; ++k) {
            const SceneParams& sp = worlds[static_cast<size_t>(k) * world_count + world].scene;
            if (kConvex && sp.support_mapped)
                scene_step_item<false, true>(sp, reinterpret_cast<float*>(smem4), env, env);
            else
                scene_step_item<false, false>(sp, reinterpret_cast<float*>(smem4), env, env);
            __syncthreads();
        }
    }
}

// The FP64 audit of the bodies each environment committed in the launch with
// the same parameters.
__global__ void __launch_bounds__(32) scene_audit_kernel(SceneParams p) {
    const int item = blockIdx.x;
    if (item >= p.env_count || p.audit == nullptr) return;
    const int env = p.env_index != nullptr ? p.env_index[item] : item;
    const SceneModel& M = *p.model;
    const bool reset = p.reset_masks != nullptr && p.reset_masks[item] != 0u;
    audit_scene(M, p.q + static_cast<size_t>(env) * M.nb * 7, p.v + static_cast<size_t>(env) * M.nb * 6,
                p.audit + static_cast<size_t>(env) * kAuditWords, reset, static_cast<int>(threadIdx.x));
}

}  // namespace

namespace {

// Resident environments per SM of the per-world launch (0: as many as the
// registers allow).  NUMI_B200_SCENE_RESIDENT, read once, overrides it; a
// lower count is reached by asking each CTA for more shared memory.
int scene_resident_limit() {
    static const int limit = [] {
        const char* env = std::getenv("NUMI_B200_SCENE_RESIDENT");
        const int v = env ? std::atoi(env) : 0;
        return v > 0 && v <= 32 ? v : 0;
    }();
    return limit;
}

// SMs of the current device (0 when it cannot be asked).
int device_sms() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
}

// Warps and shared memory (floats) of a launch over `envs` environments of
// `nb` bodies.  The registers hold 16 warps per SM.  Four warps per
// environment finish one soonest, so that is the shape while every
// environment is resident at once (4 per SM, 592 on 148 SMs); past that,
// fewer warps waste less on barriers and idle lanes, and small worlds do best
// with one.  us per control step of 1 / 2 / 4 warps (3370, 3370, 7000 floats
// up to 28 bodies, 7000 above):
//   pile    9 bodies:  592 envs 224 / 210 / 203;  4000 envs  610 /  983 / 1234
//   pile   20 bodies:  592 envs 316 / 233 / 213;  4000 envs  841 / 1129 / 1377
//   pile   28 bodies:  592 envs 426 / 311 / 222;  4000 envs 1228 / 1616 / 1450
//   pile   36 bodies:  592 envs 533 / 351 / 246;  4000 envs 2201 / 1568 / 1599
//   pile   61 bodies:  592 envs 807 / 501 / 371;  4000 envs 3285 / 2176 / 2286
// Support-mapped worlds keep per-thread polytopes in local memory, which
// wants the L1 more than residency, so above 28 bodies they keep four warps
// at any environment count and below, with one warp, 2800 floats:
//   hulls  35 bodies:  592 envs 282 / 216 / 136;  4000 envs 1028 /  740 /  705
//   hulls  61 bodies:  592 envs 488 / 373 / 225;  4000 envs 2177 / 1671 / 1668
//   capsule-box pairs through GJK, 35 bodies:     4000 envs 2862 / 2072 / 1817
//   hulls   9 bodies, 4000 envs, one warp in 2800 / 3370 floats 447 / 463
//   cylinders 14 bodies, 3000 envs,                             751 / 913
//   cylinders 23 bodies, 3000 envs,                            1914 / 2119
// Where the line costs most: 20 to 28 support-mapped bodies just past eight
// environments per SM, where two warps are up to a fifth faster than one
// (cylinders 23 bodies, 1500 envs 1366 / 1115; hulls 28 bodies 534 / 444).
// Shared memory: no more than a shape uses, because what it leaves is L1.
SceneShape scene_shape(int nb, int envs, bool compensated, bool convex) {
    SceneShape shape{};
    constexpr int kSmall = 28;   // bodies
    const int sms = device_sms();
    int total = 7000;
    if (envs <= 4 * sms || (convex && nb > kSmall)) {
        shape.warps = 4;
    } else if (nb > kSmall) {
        shape.warps = 2;
    } else {
        shape.warps = envs <= 8 * sms ? 2 : 1;
        total = convex && shape.warps == 1 ? 2800 : 3370;
    }
    const int words = std::max(kUnionLeast, std::min(kUnionMost, total - scene_smem_words(nb, 0, compensated)));
    shape.smem = static_cast<size_t>(scene_smem_words(nb, words, compensated)) * sizeof(float);
    if (const int limit = scene_resident_limit()) {
        int dev = 0, per_sm = 0, per_block = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess && per_sm > 0 &&
            cudaDeviceGetAttribute(&per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess) {
            // 1 KB reserved per CTA
            const size_t padded = std::min(static_cast<size_t>(per_sm / limit) - 1024, static_cast<size_t>(per_block));
            if (padded > shape.smem) shape.smem = padded;
        }
    }
    return shape;
}

}  // namespace
size_t scene_workspace_words() { return static_cast<size_t>(kWsWords); }

namespace {

template <typename F>
cudaError_t for_scene_kernel(bool compensated, bool convex, F&& f) {
    if (compensated) return convex ? f(scene_step_kernel<true, true>) : f(scene_step_kernel<true, false>);
    return convex ? f(scene_step_kernel<false, true>) : f(scene_step_kernel<false, false>);
}

}  // namespace

cudaError_t configure_scene_step_kernel() {
    // The driver's default carveout keeps the rest of the unified L1 as
    // cache, which the manifold tables rely on.
    cudaError_t e = cudaSuccess;
    for (const bool compensated : {false, true})
        for (const bool convex : {false, true})
            if (e == cudaSuccess)
                e = for_scene_kernel(compensated, convex, [&](auto kernel) {
                    int dev = 0, per_block = 0;
                    cudaError_t q = cudaGetDevice(&dev);
                    if (q == cudaSuccess) q = cudaDeviceGetAttribute(&per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
                    return q != cudaSuccess ? q : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, per_block);
                });
    return e;
}

cudaError_t configure_mix_scene_kernel(bool convex, size_t max_dynamic_smem) {
    const int bytes = static_cast<int>(max_dynamic_smem);
    return convex ? cudaFuncSetAttribute(mix_scene_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)
                  : cudaFuncSetAttribute(mix_scene_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// A batch ends with its longest environments, so it takes the shape that
// finishes one soonest; room for a full block of pairs at any body count.
// 4000-environment mix: 7633 us with one warp, 5715 with two, 5143 with four
// (5329 in 7000 floats).
int mix_scene_warps() { return kSceneMaxWarps; }
size_t mix_scene_smem_bytes() { return size_t(10200) * sizeof(float); }

cudaError_t mix_scene_occupancy(bool convex, size_t smem_per_block, int* blocks_per_sm) {
    const int threads = 32 * mix_scene_warps();
    return convex ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, mix_scene_kernel<true>, threads, smem_per_block)
                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, mix_scene_kernel<false>, threads, smem_per_block);
}

cudaError_t launch_mix_scene(bool convex, const MixWorld* worlds, int world_count, int steps, const std::uint32_t* items,
                             int item_count, unsigned* next_item, size_t smem_per_block, int grid, cudaStream_t stream) {
    if (smem_per_block < mix_scene_smem_bytes()) return cudaErrorInvalidValue;
    const int threads = 32 * mix_scene_warps();
    if (convex)
        mix_scene_kernel<true><<<grid, threads, smem_per_block, stream>>>(worlds, world_count, steps, items, item_count, next_item);
    else
        mix_scene_kernel<false><<<grid, threads, smem_per_block, stream>>>(worlds, world_count, steps, items, item_count, next_item);
    return cudaGetLastError();
}

cudaError_t launch_scene_audit(const SceneParams& p, cudaStream_t stream) {
    scene_audit_kernel<<<p.env_count, 32, 0, stream>>>(p);
    return cudaGetLastError();
}

int scene_step_warps(const SceneParams& p) { return scene_shape(p.bodies, p.env_count, p.q_comp != nullptr, p.support_mapped != 0).warps; }

cudaError_t launch_scene_step(const SceneParams& p, cudaStream_t stream) {
    const bool compensated = p.q_comp != nullptr;
    if (p.bodies < 1 || p.bodies > kSceneMaxBodies) return cudaErrorInvalidValue;
    const SceneShape shape = scene_shape(p.bodies, p.env_count, compensated, p.support_mapped != 0);
    return for_scene_kernel(compensated, p.support_mapped != 0, [&](auto kernel) {
        kernel<<<p.env_count, 32 * shape.warps, shape.smem, stream>>>(p);
        return cudaGetLastError();
    });
}

}  // namespace numi
