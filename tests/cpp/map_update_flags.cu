// The update kernel of a mapping step under each error flag that a binning can
// raise: prints the flag and the number of bytes of the map and its optimiser
// state that the step changed.
#include <cstdio>
#include <cstring>
#include <vector>

#include "fvgs_device.cuh"
#include "fvgs_launch.h"

using namespace fvgs;

template <typename T>
T* upload(const std::vector<T>& v) {
    T* p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * v.size()) != cudaSuccess) return nullptr;
    cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
    return p;
}

int main() {
    const int n = 1000;
    std::vector<float4> plane[5];  // position, scale, rotation, colour and opacity, nine state planes
    for (int i = 0; i < n; ++i) {
        plane[0].push_back(make_float4(0.01f * (i % 7), 0.02f * (i % 5), 2.0f + 0.001f * i, 0.f));
        plane[1].push_back(make_float4(0.05f, 0.04f, 0.03f, 0.f));
        plane[2].push_back(make_float4(0.f, 0.f, 0.f, 1.f));
        plane[3].push_back(make_float4(0.2f, 0.4f, 0.6f, 0.5f));
    }
    plane[4].assign(9 * n, make_float4(0.f, 0.f, 0.f, 0.f));
    std::vector<float> delta(16 * n, 0.01f);
    const uint32_t pixels = 3;
    for (int i = 0; i < n; ++i) std::memcpy(&delta[16 * i + 12], &pixels, 4);
    DevPose pose{};
    pose.q[3] = 1.f;
    pose.qd[3] = 1.0;
    MapUpdateArgs a{};
    float4** dst[5] = {&a.pos, &a.scale, &a.rot, &a.col, &a.adam};
    for (int k = 0; k < 5; ++k) *dst[k] = upload(plane[k]);
    a.cap = n;
    a.n = n;
    a.delta2d = upload(delta);
    a.counts = upload(std::vector<uint32_t>(n, 1u));
    a.pose = upload(std::vector<DevPose>(1, pose));
    a.K = {100.f, 100.f, 50.f, 50.f};
    a.eta = 0.01f;
    a.beta1 = 0.9f;
    a.beta2 = 0.999f;
    a.eps = 1e-8f;
    for (uint32_t flags : {kErrOverflow, kErrTimeout, kErrBounds, 0u}) {
        DevStatus st{};
        st.flags = flags;
        const DevStatus* d_st = upload(std::vector<DevStatus>(1, st));
        if (launch_map_update(a, d_st, 8, nullptr) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return 1;
        size_t changed = 0;
        for (int k = 0; k < 5; ++k) {
            std::vector<float4> now(plane[k].size());
            if (cudaMemcpy(now.data(), *dst[k], sizeof(float4) * now.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
                return 1;
            const auto *x = reinterpret_cast<const char*>(now.data()),
                       *y = reinterpret_cast<const char*>(plane[k].data());
            for (size_t b = 0; b < sizeof(float4) * now.size(); ++b) changed += x[b] != y[b];
        }
        std::printf("%u %zu\n", flags, changed);
    }
    return 0;
}
