// common.cuh -- shared types for the maxLq B200 engine.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include "../../include/maxlq.h"

namespace mlq {

// ----------------------------------------------------------------------------
// Complex arithmetic on float2 / double2 storage.
// ----------------------------------------------------------------------------
template <typename T>
struct cpx {
    T x, y;
};
template <>
struct __align__(8) cpx<float> {
    float x, y;
};
template <>
struct __align__(16) cpx<double> {
    double x, y;
};

template <typename T>
__host__ __device__ __forceinline__ cpx<T> mk(T a, T b) {
    cpx<T> r;
    r.x = a;
    r.y = b;
    return r;
}
template <typename T>
__host__ __device__ __forceinline__ cpx<T> operator+(cpx<T> a, cpx<T> b) { return mk(a.x + b.x, a.y + b.y); }
template <typename T>
__host__ __device__ __forceinline__ cpx<T> operator-(cpx<T> a, cpx<T> b) { return mk(a.x - b.x, a.y - b.y); }
template <typename T>
__host__ __device__ __forceinline__ cpx<T> operator*(cpx<T> a, cpx<T> b) {
    return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T>
__host__ __device__ __forceinline__ cpx<T> operator*(cpx<T> a, T s) { return mk(a.x * s, a.y * s); }
template <typename T>
__host__ __device__ __forceinline__ cpx<T> conj(cpx<T> a) { return mk(a.x, -a.y); }
// multiply by -i (sign < 0) or +i (sign > 0)
template <int SIGN, typename T>
__host__ __device__ __forceinline__ cpx<T> rot90(cpx<T> a) {
    return SIGN < 0 ? mk(a.y, -a.x) : mk(-a.y, a.x);
}
template <typename T>
__host__ __device__ __forceinline__ cpx<T> czero() { return mk(T(0), T(0)); }

template <typename TO, typename TI>
__host__ __device__ __forceinline__ cpx<TO> ccast(cpx<TI> a) { return mk((TO)a.x, (TO)a.y); }

// ----------------------------------------------------------------------------
// A spectral band: the modes kept by a dealiasing cube cut.  cut = largest
// |j| kept on every axis; full = no cut (cut >= N/2).  Arrays in a band are
// stored "pruned": kx in [0, nx), ky/kz compact index in [0, nb) ordered
// 0..cut, -cut..-1 (or natural FFT order when full).
// ----------------------------------------------------------------------------
struct Band {
    int n;     // grid size
    int cut;   // largest |j| kept
    int nx;    // kx extent (cut+1, or n/2+1 when full)
    int nb;    // ky/kz extent (2cut+1, or n when full)
    int full;  // 1 when no mode is removed
};

__host__ __device__ __forceinline__ int band_fft_index(const Band& b, int ci) {
    return ci <= b.cut ? ci : b.n - b.nb + ci;
}
__host__ __device__ __forceinline__ int band_compact_index(const Band& b, int fi) {
    // returns -1 when the FFT index is outside the band
    if (b.full) return fi;
    if (fi <= b.cut) return fi;
    if (fi >= b.n - b.cut) return fi - (b.n - b.nb);
    return -1;
}
// signed wavenumber index j of an FFT index
__host__ __device__ __forceinline__ int signed_j(int n, int fi) { return fi <= n / 2 ? fi : fi - n; }

constexpr double MACH_EPSILON = 2.0e-16;  // global_variables.f90:28

struct CudaError : std::runtime_error {
    int status;
    CudaError(const std::string& m, int s) : std::runtime_error(m), status(s) {}
};

// Programmatic dependent launch.  A kernel launched with launch_pdl may start
// while its predecessor in the stream still drains: everything before
// pdl_begin (twiddle and wavenumber tables, index arithmetic) overlaps the
// predecessor's last blocks and the launch gap; pdl_begin waits until the
// predecessor has completed and its writes are visible.  A kernel calls it
// once, in every thread, before it touches memory that another kernel of the
// stream reads or writes.  A CG iteration at q = 4: 64^3 FP64 0.474 -> 0.385
// ms, 32^3 0.84 -> 0.73, 128^3 FP64 1.59 -> 1.49, 192^3 mixed 3.16 -> 3.03, 256^3 FP64
// 8.97 -> 8.86, 512^3 mixed unchanged (35.3).
// EARLY lets the successor start as soon as this kernel's blocks run, instead
// of as they exit.  64^3 gains from it (0.398 -> 0.380 ms); from 128^3 on it
// gains nothing and then costs (256^3 FP64 8.86 -> 9.45, 512^3 mixed 35.3 ->
// 43.5 ms), so the pass kernels take it up to N = 64 and the one-block
// finalize always.
template <bool EARLY = false>
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_pdl(bool on, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = on ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

#define MLQ_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            throw ::mlq::CudaError(std::string(#call) + ": " + cudaGetErrorString(e_),          \
                                   e_ == cudaErrorMemoryAllocation ? MLQ_ERR_OOM : MLQ_ERR_CUDA); \
    } while (0)

}  // namespace mlq
