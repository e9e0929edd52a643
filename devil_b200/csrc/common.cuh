// Device helpers shared by every kernel of the devil B200 path.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define DEV __device__ __forceinline__

namespace devil {

// Programmatic dependent launch between the kernels of an iteration: a kernel
// launched by launch_dependent (internal.h) may become resident while the one
// before it still runs and waits here, before its first access to global memory,
// until that one has ended and its writes are visible; grid_trigger says that the
// kernel's own follower may be made resident.  Data of the kernel before it are
// read by plain or .cg loads, not __ldg.  The loops of a fit are chains of kernels
// of 5 to 30 us: with the launches overlapped, and slices staged before the wait,
// IRLS takes 2.3 ms instead of 2.9 on 200 x 2,000 (p = 4, per cell), 3.6 instead of
// 4.8 on 2,000 x 5,000 and 24.0 instead of 25.3 on 4,000 x 1 M (p = 2, grouped).
DEV void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
DEV void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

constexpr float kLog2e = 1.4426950408889634f;

// MUFU.EX2 / MUFU.RCP through PTX (approximate, ~1-2 ulp; FTZ).
DEV float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
DEV float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
DEV float fast_exp(float x) { return ex2_approx(x * kLog2e); }

template <class T>
DEV T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <class T>
DEV T warp_max(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// value loaders for the two CSR value types
DEV float load_val(const uint16_t* v, int64_t e) { return (float)__ldg(v + e); }
DEV float load_val(const float* v, int64_t e) { return __ldg(v + e); }

// ---------------------------------------------------------------------
// solution of a p x p system by one thread, column-major, from its LU
// factors with partial pivoting (row swaps piv), the factorisation Eigen's
// MatrixXd::inverse() uses for dynamic sizes
// ---------------------------------------------------------------------
DEV void lu_solve(int p, const double* LU, const int* piv, double* x) {
    for (int k = 0; k < p; ++k)
        if (piv[k] != k) { double t = x[k]; x[k] = x[piv[k]]; x[piv[k]] = t; }
    for (int i = 0; i < p; ++i) {
        double s = x[i];
        for (int j = 0; j < i; ++j) s -= LU[j * p + i] * x[j];
        x[i] = s;
    }
    for (int i = p - 1; i >= 0; --i) {
        double s = x[i];
        for (int j = i + 1; j < p; ++j) s -= LU[j * p + i] * x[j];
        x[i] = s / LU[i * p + i];
    }
}

// index of (i, j), i <= j, in packed upper-triangular storage by rows of j:
// pairs are enumerated (0,0),(0,1),(1,1),(0,2),(1,2),(2,2),...
DEV constexpr int tri_index(int i, int j) { return j * (j + 1) / 2 + i; }

}  // namespace devil
