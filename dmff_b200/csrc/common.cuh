// Shared device helpers for the ADMP / PME engine (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>

#define DMFFB_DIELECTRIC 1389.35455846  // dmff/common/constants.py:3
#define DMFFB_SQRT3 1.7320508075688772
#define DMFFB_RT3_REF 1.73205080757      // dmff/admp/multipole.py:13 (truncated, used in C2_gl)
#define DMFFB_TWO_OVER_SQRTPI 1.1283791670955126

namespace dmffb {

// ------------------------------------------------------------------ math wrappers
__device__ __forceinline__ float d_erfc(float x) { return erfcf(x); }
__device__ __forceinline__ double d_erfc(double x) { return erfc(x); }
__device__ __forceinline__ float d_erf(float x) { return erff(x); }
__device__ __forceinline__ double d_erf(double x) { return erf(x); }
__device__ __forceinline__ float d_exp(float x) { return expf(x); }
__device__ __forceinline__ double d_exp(double x) { return exp(x); }
__device__ __forceinline__ float d_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double d_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float d_rsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double d_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float d_floor(float x) { return floorf(x); }
__device__ __forceinline__ double d_floor(double x) { return floor(x); }

// value + derivative with respect to the pair distance r
template <typename T>
struct Dl {
    T v, d;
    __device__ __forceinline__ Dl() {}
    __device__ __forceinline__ Dl(T v_, T d_) : v(v_), d(d_) {}
};
template <typename T> __device__ __forceinline__ Dl<T> operator+(Dl<T> a, Dl<T> b) { return Dl<T>(a.v + b.v, a.d + b.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator-(Dl<T> a, Dl<T> b) { return Dl<T>(a.v - b.v, a.d - b.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator*(Dl<T> a, Dl<T> b) { return Dl<T>(a.v * b.v, a.d * b.v + a.v * b.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator*(T s, Dl<T> a) { return Dl<T>(s * a.v, s * a.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator+(T s, Dl<T> a) { return Dl<T>(s + a.v, a.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator-(Dl<T> a) { return Dl<T>(-a.v, -a.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator*(Dl<T> a, T s) { return Dl<T>(a.v * s, a.d * s); }
template <typename T> __device__ __forceinline__ Dl<T> operator+(Dl<T> a, T s) { return Dl<T>(a.v + s, a.d); }
template <typename T> __device__ __forceinline__ Dl<T> operator-(Dl<T> a, T s) { return Dl<T>(a.v - s, a.d); }

// ------------------------------------------------------------------ vectors
template <typename T>
struct __align__(4 * sizeof(T)) Vec4 {
    T x, y, z, w;
};

// g[0..2] += (x, y, z) for a 4-element slot: one 16-byte reduction in FP32
__device__ __forceinline__ void add3(float* g, float x, float y, float z) {
    atomicAdd((float4*)g, make_float4(x, y, z, 0.f));
}
__device__ __forceinline__ void add3(double* g, double x, double y, double z) {
    atomicAdd(g, x);
    atomicAdd(g + 1, y);
    atomicAdd(g + 2, z);
}

// ------------------------------------------------------------------ warp helpers
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Segmented sums over runs of equal keys in a warp.  A key may appear in several runs (rows
// skipped by a launch sit between rows of the same atom), so runs are identified by a run id:
// the number of run heads up to and including the lane.  After seg_sum, the head lane of each
// run holds that run's total.
__device__ __forceinline__ bool seg_head(int key) {
    const int lane = threadIdx.x & 31;
    int prev = __shfl_up_sync(0xffffffffu, key, 1);
    return lane == 0 || prev != key;
}
__device__ __forceinline__ int seg_run_id(int key) {
    const int lane = threadIdx.x & 31;
    const unsigned heads = __ballot_sync(0xffffffffu, seg_head(key));
    return __popc(heads & (0xffffffffu >> (31 - lane)));
}
// seg_sum takes the lanes' run relations from seg_reach: bit k set where lane + 2^k belongs to the run
__device__ __forceinline__ unsigned seg_reach(int run) {
    const int lane = threadIdx.x & 31;
    unsigned m = 0u;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int o = 1 << k, other = __shfl_down_sync(0xffffffffu, run, o);
        if (lane + o < 32 && other == run) m |= 1u << k;
    }
    return m;
}
template <typename T>
__device__ __forceinline__ T seg_sum(T v, unsigned reach) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const T ov = __shfl_down_sync(0xffffffffu, v, 1 << k);
        if ((reach >> k) & 1u) v += ov;
    }
    return v;
}

// Sums NS values over the warp by recursive halving: at each of the five steps a lane hands one half
// of what it holds to its partner and keeps the other, so 20 values take 21 exchanges where a
// butterfly per value takes 100.  The lanes that end up holding a sum write it to out[0 .. NS).
template <typename T, int NS>
__device__ __forceinline__ void warp_sums(T (&v)[NS], T* out, int lane) {
    int idx = 0, sz = NS;
    constexpr int H[5] = {(NS + 1) / 2, ((NS + 1) / 2 + 1) / 2, (((NS + 1) / 2 + 1) / 2 + 1) / 2,
                          ((((NS + 1) / 2 + 1) / 2 + 1) / 2 + 1) / 2,
                          (((((NS + 1) / 2 + 1) / 2 + 1) / 2 + 1) / 2 + 1) / 2};
#pragma unroll
    for (int step = 0; step < 5; ++step) {
        const int n = step == 0 ? NS : H[step - 1], h = H[step], o = 16 >> step;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            if (k >= h) break;
            const T lo = v[k], hi = k + h < n ? v[k + h < NS ? k + h : 0] : T(0);
            v[k] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
        }
        if (up) {
            idx += h;
            sz = max(sz - h, 0);
        } else {
            sz = min(sz, h);
        }
    }
    if (sz >= 1) out[idx] = v[0];
}

// block-wide reduction of NV doubles into dst[] with one atomicAdd per value per block
template <int NV>
__device__ __forceinline__ void block_reduce_add(double (&v)[NV], double* dst) {
    __shared__ double sh[32][NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (NV == 1) {
        const double t = warp_sum(v[0]);
        if (lane == 0) sh[wid][0] = t;
    } else {
        warp_sums<double, NV>(v, sh[wid], lane);
    }
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    if (wid == 0) {
        if (NV == 1) {
            double t = lane < nw ? sh[lane][0] : 0.0;
            t = warp_sum(t);
            if (lane == 0 && t != 0.0) atomicAdd(dst, t);
        } else if (lane < NV) {
            double t = 0.0;
            for (int w = 0; w < nw; ++w) t += sh[w][lane];
            if (t != 0.0) atomicAdd(dst + lane, t);
        }
    }
    __syncthreads();  // the shared buffer may be reused by the next call
}

// ------------------------------------------------------------------ clearing
// Arrays an evaluation starts from zero, cleared by its first kernel (k_prepare, or k_clear where there
// is none) instead of a memset each: a memset is a launch, 2 to 4 us of a small system's step.
struct ClearList {
    static constexpr int kMax = 8;
    int32_t* p[kMax];
    int64_t words[kMax];
    int count = 0;
    __host__ void add(void* ptr, size_t bytes) {  // bytes a multiple of 4
        if (!ptr || !bytes) return;
        p[count] = (int32_t*)ptr;
        words[count++] = (int64_t)(bytes / 4);
    }
};

__device__ __forceinline__ void clear_all(const ClearList& c, int64_t i, int64_t step) {
    for (int a = 0; a < c.count; ++a)
        for (int64_t k = i; k < c.words[a]; k += step) c.p[a][k] = 0;
}

static __global__ void __launch_bounds__(256) k_clear(ClearList c) {
    clear_all(c, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------ box
struct Box {
    double h[9];     // rows = lattice vectors
    double hinv[9];  // inverse
};

template <typename T>
struct BoxT {
    T h[9], hinv[9];
};

// minimum image as the reference's pbc_shift (spatial.py:14-32): ds = dr hinv; n = floor(ds+1/2);
// dr = (ds - n) h.  Returns n through nout.
template <typename T>
__device__ __forceinline__ void pbc_shift(const BoxT<T>& b, T& x, T& y, T& z, T* nout) {
    T s0 = x * b.hinv[0] + y * b.hinv[3] + z * b.hinv[6];
    T s1 = x * b.hinv[1] + y * b.hinv[4] + z * b.hinv[7];
    T s2 = x * b.hinv[2] + y * b.hinv[5] + z * b.hinv[8];
    T n0 = d_floor(s0 + T(0.5)), n1 = d_floor(s1 + T(0.5)), n2 = d_floor(s2 + T(0.5));
    s0 -= n0; s1 -= n1; s2 -= n2;
    x = s0 * b.h[0] + s1 * b.h[3] + s2 * b.h[6];
    y = s0 * b.h[1] + s1 * b.h[4] + s2 * b.h[7];
    z = s0 * b.h[2] + s1 * b.h[5] + s2 * b.h[8];
    if (nout) { nout[0] = n0; nout[1] = n1; nout[2] = n2; }
}

}  // namespace dmffb
