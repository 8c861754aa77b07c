// Test harness: functions that stand in for a library call or a division, on the GPU.
// Built by tests/test_gpu_short_forms.py with the FP64 unit's flags.
#include <cuda_runtime.h>

#include <type_traits>

#include "phx.h"
#include "../../photon_gb300/csrc/step_kernels.cuh"
#include "../../photon_gb300/csrc/radiation.cuh"
#include "../../photon_gb300/csrc/volume.cuh"

__global__ void k_temps(const double* x, long long n, double* p08, double* p17) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    p08[i] = phx::powTemp08(x[i]);
    p17[i] = phx::powTemp17(x[i]);
}
__global__ void k_decay(const double* x, long long n, const double* exp2T, double* out) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) out[i] = phx::radDecay(x[i], exp2T);
}
__global__ void k_div(const float* x, const float* d, long long n, float* fast, float* ref) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    fast[i] = phx::vDivBy(x[i], d[i], 1.0f / d[i]);
    ref[i] = x[i] / d[i];
}

namespace {
struct Buf {
    void* p = nullptr;
    explicit Buf(size_t bytes) { cudaMalloc(&p, bytes); }
    ~Buf() { cudaFree(p); }
    template <class T> T* as() { return static_cast<T*>(p); }
};
unsigned blocks(long long n) { return (unsigned)((n + 255) / 256); }
}  // namespace

extern "C" int temps(const double* hx, long long n, double* h08, double* h17) {
    const size_t b = (size_t)n * 8;
    Buf x(b), a(b), c(b);
    cudaMemcpy(x.p, hx, b, cudaMemcpyHostToDevice);
    k_temps<<<blocks(n), 256>>>(x.as<double>(), n, a.as<double>(), c.as<double>());
    cudaMemcpy(h08, a.p, b, cudaMemcpyDeviceToHost);
    cudaMemcpy(h17, c.p, b, cudaMemcpyDeviceToHost);
    return (int)cudaGetLastError();
}
extern "C" int decay(const double* hx, long long n, double* h) {
    const size_t b = (size_t)n * 8;
    Buf x(b), o(b), k(sizeof(phx::RadConst<double>));
    cudaMemcpy(x.p, hx, b, cudaMemcpyHostToDevice);
    phx::k_rad_setup<double><<<1, phx::RAD_EXP_N>>>(k.as<phx::RadConst<double>>());
    k_decay<<<blocks(n), 256>>>(x.as<double>(), n, k.as<phx::RadConst<double>>()->exp2T, o.as<double>());
    cudaMemcpy(h, o.p, b, cudaMemcpyDeviceToHost);
    return (int)cudaGetLastError();
}
extern "C" int div_by(const float* hx, const float* hd, long long n, float* hf, float* hr) {
    const size_t b = (size_t)n * 4;
    Buf x(b), d(b), f(b), r(b);
    cudaMemcpy(x.p, hx, b, cudaMemcpyHostToDevice);
    cudaMemcpy(d.p, hd, b, cudaMemcpyHostToDevice);
    k_div<<<blocks(n), 256>>>(x.as<float>(), d.as<float>(), n, f.as<float>(), r.as<float>());
    cudaMemcpy(hf, f.p, b, cudaMemcpyDeviceToHost);
    cudaMemcpy(hr, r.p, b, cudaMemcpyDeviceToHost);
    return (int)cudaGetLastError();
}
