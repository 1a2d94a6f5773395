// Reciprocal convolution of a mesh that fits in L2 by direct DFTs: real mesh -> forward 3-D DFT ->
// multiply by the influence function (recip.py:438-466) -> inverse 3-D DFT -> real mesh, in three
// kernels, for any extents (primes included) of up to kDftMaxK points per axis, FP32 and FP64.
//
//   k_dft_fwd      (x-plane, chunk of kz) per CTA: real DFT along z of the chunk's kz, DFT along y
//   k_dft_columns  block of (ky, kz) columns per CTA: DFT along x, times G, inverse DFT along x;
//                  with want_energy also the energy and the k-space tensor of the box gradient
//   k_dft_inv      (x-plane, chunk of y pairs) per CTA: inverse DFT along y, then along z
//
// Why direct sums: at these sizes a transform is bound by latency, not by arithmetic.  Folding the
// input (x_n + x_{K-n} against cosines, x_n - x_{K-n} against sines) and computing outputs k and
// K - k from the same two sums leaves 3 K^4 multiply-adds for the whole convolution: 0.019 G at 50^3,
// 0.5 us of the FP32 pipes.  Each pass is two shared-memory contractions between two barriers,
// whatever the factors of K, where an FFT line of 50 points needs a barrier per radix and cuFFT one
// kernel per axis.  Every plane is read by several CTAs (one per chunk), so that about 300 CTAs share
// a 50^3 mesh instead of 50.
//
// Transforms are unnormalised in both directions (the convention the gather expects).  The DFT
// matrices hold cos and sin of 2 pi a b / K, a, b = 0 .. K/2, rounded from FP64; G is multiplied in FP64.
#pragma once
#include "admp_recip.cuh"
#include "common.cuh"

namespace dmffb {

constexpr int kDftMaxK = 128;
constexpr int kDftThreads = 512;  // largest block of the three kernels

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

// operand of the folded sums: c0, c1 go with the cosine, s0, s1 with the sine
template <typename T> struct alignas(16) Cpair { T c0, c1, s0, s1; };

template <typename T>
struct DftConvArgs {
    using T2 = typename Vec2<T>::type;
    int K[3], H[3];       // extents and K / 2
    const T* grid_in;     // [K0*K1*K2] spread mesh
    T* grid_out;          // [K0*K1*K2] convolved mesh
    T2* spec;             // [K0][K1][H2 + 1] half spectrum between the passes
    const T2* W[3];       // [H + 1][dft_stride(H)] (cos, sin) of 2 pi a b / K per axis
    const double* G;      // [K0*K1*(H2 + 1)] influence function, or null: computed here
    int fwd_chunk;        // kz per CTA of the forward pass, a multiple of the tile's TW
    int inv_chunk;        // y pairs per CTA of the inverse pass, likewise
    int cols;             // columns per CTA of the column pass
    // influence function and energy (ConvArgs' conventions)
    const double* bmod;
    double hinv[9];
    double V, kappa, escale;
    int kind;
    int want_energy;
    double* scal;         // [0] energy, [1..6] k-space tensor
    T* zero_real;         // mesh of K0*K1*K2 elements the column pass sets to 0 (may be null)
};

// work items of each pass
template <typename T> __host__ __device__ inline int dft_fwd_items(const DftConvArgs<T>& a) {
    return a.K[0] * ((a.H[2] + a.fwd_chunk) / a.fwd_chunk);
}
template <typename T> __host__ __device__ inline int dft_inv_items(const DftConvArgs<T>& a) {
    return a.K[0] * ((a.H[1] + a.inv_chunk) / a.inv_chunk);
}
template <typename T> __host__ __device__ inline int dft_col_items(const DftConvArgs<T>& a) {
    return (a.K[1] * (a.H[2] + 1) + a.cols - 1) / a.cols;
}

// row stride of the matrices: H + 1 columns padded with zeros to a multiple of 4
__host__ __device__ inline int dft_stride(int H) { return (H + 4) & ~3; }
// elements of one axis's matrix
__host__ __device__ inline size_t dft_mat_elems(int H) { return (size_t)2 * (H + 1) * dft_stride(H); }

// shared memory (elements of T) of each pass, without the DFT matrices
template <typename T> __host__ __device__ inline size_t dft_fwd_elems(const DftConvArgs<T>& a) {
    return 4 * (size_t)(a.H[1] + 1) * ((a.fwd_chunk + 4) + (a.H[2] + 1)) + 16;
}
template <typename T> __host__ __device__ inline size_t dft_col_elems(const DftConvArgs<T>& a) {
    return 8 * (size_t)(a.H[0] + 1) * (a.cols + 4) + 16;
}
template <typename T> __host__ __device__ inline size_t dft_inv_elems(const DftConvArgs<T>& a) {
    return 4 * (size_t)(a.H[2] + 4) * ((a.H[1] + 1) + (a.inv_chunk + 4)) + 16;
}

// copies an axis's matrix to shared memory without waiting for it (dft_wait does)
template <typename T>
__device__ __forceinline__ void dft_load_mat(const DftConvArgs<T>& a, int axis, T* dst) {
    const int chunks = (int)(dft_mat_elems(a.H[axis]) * sizeof(T) / 16);
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const char* src = (const char*)a.W[axis];
    for (int t = threadIdx.x; t < chunks; t += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * t), "l"(src + 16 * (size_t)t) : "memory");
}
__device__ __forceinline__ void dft_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// a / b for 0 <= a < 2^22, 1 <= b < 2^11, with rcp = 1.f / b
__device__ __forceinline__ int dft_div(int a, float rcp) { return __float2int_rd(((float)a + 0.5f) * rcp); }

// two matrix entries (cos, sin), (cos, sin)
__device__ __forceinline__ void dft_w2(const float2* w, float2& u, float2& v) {
    const float4 f = *(const float4*)w;
    u = make_float2(f.x, f.y);
    v = make_float2(f.z, f.w);
}
__device__ __forceinline__ void dft_w2(const double2* w, double2& u, double2& v) {
    u = w[0];
    v = w[1];
}

// acc[i][j] = sum over k < m of (c0 cos, c1 cos, s0 sin, s1 sin) with Cpair V[k vk + j vc] and matrix
// entry w[k wk + i]: a TW x TV tile of outputs per thread.  Shared-memory reads bound these sums (a
// 128-bit read takes four cycles of the SM whatever the lanes share): a 1 x 1 tile reads 6 cycles
// per 4 multiply-adds and warp, 2 x 2 reads 12 per 16 and 4 x 2 16 per 32.
// One running sum over all m products would round at the size of what it holds, and left the convolution of an
// FP32 mesh 1.1 to 1.6 times the rounding error of an FFT at 17 to 61 points and 1.9 at 85.  Single outputs keep
// four running sums that meet at the end (0.8 to 0.95 times an FFT's error); the wide tiles, which have no
// registers for that, add up eight products at a time: 0.8 to 1.1 times at 59 to 97 points.  Evaluations of 900
// polarizable atoms took 534 us at 50^3 with one sum and take 525, at 61^3 561 and 565.  FP64 keeps the one
// sum: its rounding is far below that of the sums over sites, and four or eight cost 1 to 7 % of an evaluation.
template <typename T, int TW, int TV>
__device__ __forceinline__ void dft_tile(const Cpair<T>* V, int vk, int vc, const typename Vec2<T>::type* w, int wk, int m,
                                         T (&acc)[TW][TV][4]) {
    using T2 = typename Vec2<T>::type;
    const auto add = [&](int k, T (&a)[TW][TV][4]) {
        Cpair<T> v[TV];
        T2 c[TW];
#pragma unroll
        for (int j = 0; j < TV; ++j) v[j] = V[k * vk + j * vc];
        if constexpr (TW == 1) {
            c[0] = w[k * wk];
        } else {
#pragma unroll
            for (int i = 0; i < TW; i += 2) dft_w2(w + k * wk + i, c[i], c[i + 1]);
        }
#pragma unroll
        for (int i = 0; i < TW; ++i)
#pragma unroll
            for (int j = 0; j < TV; ++j) {
                a[i][j][0] += v[j].c0 * c[i].x;
                a[i][j][1] += v[j].c1 * c[i].x;
                a[i][j][2] += v[j].s0 * c[i].y;
                a[i][j][3] += v[j].s1 * c[i].y;
            }
    };
    // b = a + b (each time the sums of a part meet the others), or b = 0
    const auto join = [](T (&b)[TW][TV][4], const T (*a)[TV][4]) {
#pragma unroll
        for (int i = 0; i < TW; ++i)
#pragma unroll
            for (int j = 0; j < TV; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) b[i][j][q] = a ? b[i][j][q] + a[i][j][q] : T(0);
    };
    int k = 0;
    join(acc, nullptr);
    if constexpr (sizeof(T) == 8) {
#pragma unroll (TW * TV == 1 ? 8 : 4)
        for (; k < m; ++k) add(k, acc);
    } else if constexpr (TW * TV == 1) {
        T s[3][TW][TV][4];
#pragma unroll
        for (int n = 0; n < 3; ++n) join(s[n], nullptr);
#pragma unroll 2
        for (; k + 4 <= m; k += 4) {
            add(k, acc);
            add(k + 1, s[0]);
            add(k + 2, s[1]);
            add(k + 3, s[2]);
        }
        if (k < m) add(k, acc);
        if (k + 1 < m) add(k + 1, s[0]);
        if (k + 2 < m) add(k + 2, s[1]);
        join(acc, s[0]);
        join(s[1], s[2]);
        join(acc, s[1]);
    } else {
        while (k < m) {
            T s[TW][TV][4];
            join(s, nullptr);
            if (k + 8 <= m) {
#pragma unroll
                for (int n = 0; n < 8; ++n) add(k + n, s);
                k += 8;
            } else {
                for (; k < m; ++k) add(k, s);
            }
            join(acc, s);
        }
    }
}

constexpr int kDftBatch = 2;  // folded elements (4 global reads each) in flight per thread

// forward z and y transforms of plane x for kz in [k0, k0 + chunk); wys, wzs: matrices in shared
// memory (their copies may still be in flight)
template <typename T, int TW, int TV>
__device__ inline void dft_fwd_item(const DftConvArgs<T>& a, int item, T* sm, const T* wys, const T* wzs) {
    using T2 = typename Vec2<T>::type;
    const int tid = threadIdx.x, nth = blockDim.x;
    const int Ky = a.K[1], Kz = a.K[2], hz = a.H[2] + 1, hy = a.H[1] + 1;
    const int sy = dft_stride(a.H[1]), sz = dft_stride(a.H[2]);
    const int nchunk = (a.H[2] + a.fwd_chunk) / a.fwd_chunk;
    const int x = item / nchunk, k0 = (item - x * nchunk) * a.fwd_chunk;
    const int C = min(a.fwd_chunk, hz - k0), CS = (a.fwd_chunk + 3) & ~3;
    Cpair<T>* EO = (Cpair<T>*)sm;    // [hy][CS] z transforms, folded along y
    Cpair<T>* RZ = EO + hy * CS;     // [hy][hz] input folded along y and z
    const T2 *wy = (const T2*)wys, *wz = (const T2*)wzs + k0;
    const T* plane = a.grid_in + (size_t)x * Ky * Kz;
    const float rz = 1.f / (float)hz;
    for (int t0 = tid; t0 < hy * hz; t0 += kDftBatch * nth) {
        T u[kDftBatch][4];
        bool sy_[kDftBatch], sz_[kDftBatch];
#pragma unroll
        for (int q = 0; q < kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hy * hz) {
                const int y = dft_div(t, rz), z = t - y * hz;
                const int y2 = y == 0 ? 0 : Ky - y, z2 = z == 0 ? 0 : Kz - z;
                sy_[q] = y2 == y;
                sz_[q] = z2 == z;
                u[q][0] = plane[y * Kz + z];
                u[q][1] = plane[y * Kz + z2];
                u[q][2] = plane[y2 * Kz + z];
                u[q][3] = plane[y2 * Kz + z2];
            }
        }
#pragma unroll
        for (int q = 0; q < kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hy * hz) {
                const T e1 = sz_[q] ? u[q][0] : u[q][0] + u[q][1], o1 = sz_[q] ? T(0) : u[q][0] - u[q][1];
                const T e2 = sz_[q] ? u[q][2] : u[q][2] + u[q][3], o2 = sz_[q] ? T(0) : u[q][2] - u[q][3];
                Cpair<T> p;
                if (sy_[q]) p = {e1, T(0), o1, T(0)};
                else p = {e1 + e2, e1 - e2, o1 + o2, o1 - o2};
                RZ[t] = p;
            }
        }
    }
    dft_wait();
    __syncthreads();
    {  // z transform of (row y) +- (row Ky - y)
        const int nk = (C + TW - 1) / TW, ny = (hy + TV - 1) / TV;
        const float rk = 1.f / (float)nk;
        for (int t = tid; t < nk * ny; t += nth) {
            const int yt = dft_div(t, rk), k = (t - yt * nk) * TW, y = min(yt * TV, hy - TV);
            T s[TW][TV][4];
            dft_tile<T, TW, TV>(RZ + y * hz, 1, hz, wz + k, sz, hz, s);
#pragma unroll
            for (int j = 0; j < TV; ++j)
#pragma unroll
                for (int i = 0; i < TW; ++i)
                    if (k + i < C) {
                        Cpair<T> p = {s[i][j][0], -s[i][j][2], s[i][j][1], -s[i][j][3]};
                        EO[(y + j) * CS + k + i] = p;
                    }
        }
    }
    __syncthreads();
    T2* out = a.spec + (size_t)x * Ky * hz + k0;
    const int nc = (C + TV - 1) / TV, nw = (hy + TW - 1) / TW;
    const float rc = 1.f / (float)nc;
    for (int t = tid; t < nc * nw; t += nth) {
        const int wt = dft_div(t, rc), k = (t - wt * nc) * TV;
        T s[TW][TV][4];
        dft_tile<T, TW, TV>(EO + k, CS, 1, wy + wt * TW, sy, hy, s);
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int ky = wt * TW + i;
            if (ky >= hy) break;
#pragma unroll
            for (int j = 0; j < TV; ++j) {
                if (k + j >= C) break;
                T2 o;
                o.x = s[i][j][0] + s[i][j][3];
                o.y = s[i][j][1] - s[i][j][2];
                out[ky * hz + k + j] = o;
                if (ky != 0 && 2 * ky != Ky) {
                    o.x = s[i][j][0] - s[i][j][3];
                    o.y = s[i][j][1] + s[i][j][2];
                    out[(Ky - ky) * hz + k + j] = o;
                }
            }
        }
    }
}

// G of mesh point (kx, column c) and, with the energy, its terms added to red
template <typename T>
__device__ __forceinline__ double dft_influence(const DftConvArgs<T>& a, int kx, int c, T re, T im, double (&red)[7]) {
    const int hz = a.H[2] + 1;
    const int ky = c / hz, kz = c - ky * hz;
    const int m1 = kx < (a.K[0] + 1) / 2 ? kx : kx - a.K[0];
    const int m2 = ky < (a.K[1] + 1) / 2 ? ky : ky - a.K[1];
    const int m3 = kz < (a.K[2] + 1) / 2 ? kz : kz - a.K[2];
    double kv[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) kv[q] = 6.283185307179586 * (a.hinv[3 * q] * m1 + a.hinv[3 * q + 1] * m2 + a.hinv[3 * q + 2] * m3);
    const double ksq = kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2];
    const double th = a.bmod[kx] * a.bmod[a.K[0] + ky] * a.bmod[a.K[0] + a.K[1] + kz];
    if (m1 == 0 && m2 == 0 && m3 == 0 && a.kind == CK_COUL) return 0.0;
    double Cv, dlnC;
    influence(a.kind, ksq, a.kappa, a.V, Cv, dlnC);
    const double G = Cv / (th * th);
    if (a.want_energy) {
        const double w = (kz == 0 || 2 * kz == a.K[2]) ? 1.0 : 2.0;
        const double Ek = a.escale * w * G * ((double)re * re + (double)im * im);
        const double f = Ek * dlnC;
        red[0] += Ek;
        red[1] += f * kv[0] * kv[0];
        red[2] += f * kv[1] * kv[1];
        red[3] += f * kv[2] * kv[2];
        red[4] += f * kv[0] * kv[1];
        red[5] += f * kv[0] * kv[2];
        red[6] += f * kv[1] * kv[2];
    }
    return G;
}

// x transform, influence function and inverse x transform of one block of columns; TABLE: G comes
// from a.G and no energy is summed
template <typename T, int TW, int TV, bool TABLE>
__device__ inline void dft_col_item(const DftConvArgs<T>& a, int item, T* sm, const T* wxs, double (&red)[7]) {
    using T2 = typename Vec2<T>::type;
    const int tid = threadIdx.x, nth = blockDim.x;
    const int Kx = a.K[0], hx = a.H[0] + 1, sx = dft_stride(a.H[0]);
    const int ncol = a.K[1] * (a.H[2] + 1);
    const int c0 = item * a.cols, C = min(a.cols, ncol - c0), CS = (a.cols + 3) & ~3;
    Cpair<T>* EO = (Cpair<T>*)sm;   // [hx][CS] folded input
    Cpair<T>* PM = EO + hx * CS;    // [hx][CS] folded spectrum
    const T2* wx = (const T2*)wxs;
    const float rc = 1.f / (float)C;
    T2* S = a.spec + c0;
    const double* G = a.G + c0;
    for (int t0 = tid; t0 < hx * C; t0 += kDftBatch * nth) {
        T2 u[kDftBatch], v[kDftBatch];
        bool self[kDftBatch];
#pragma unroll
        for (int q = 0; q < kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hx * C) {
                const int x = dft_div(t, rc), c = t - x * C, x2 = x == 0 ? 0 : Kx - x;
                self[q] = x == x2;
                u[q] = S[x * ncol + c];
                v[q] = S[x2 * ncol + c];
            }
        }
#pragma unroll
        for (int q = 0; q < kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hx * C) {
                const int x = dft_div(t, rc), c = t - x * C;
                Cpair<T> p;
                if (self[q]) p = {u[q].x, u[q].y, T(0), T(0)};
                else p = {u[q].x + v[q].x, u[q].y + v[q].y, u[q].x - v[q].x, u[q].y - v[q].y};
                EO[x * CS + c] = p;
            }
        }
    }
    const int nc = (C + TV - 1) / TV, nw = (hx + TW - 1) / TW;
    const float rt = 1.f / (float)nc;
    dft_wait();
    __syncthreads();
    for (int t = tid; t < nc * nw; t += nth) {
        const int wt = dft_div(t, rt), c = (t - wt * nc) * TV;
        double g[TW][TV][2];
        if (TABLE) {
#pragma unroll
            for (int i = 0; i < TW; ++i)
#pragma unroll
                for (int j = 0; j < TV; ++j) {
                    const int k = min(wt * TW + i, hx - 1), cc = min(c + j, C - 1);
                    g[i][j][0] = G[k * ncol + cc];
                    g[i][j][1] = G[(k == 0 ? 0 : Kx - k) * ncol + cc];
                }
        }
        T s[TW][TV][4];
        dft_tile<T, TW, TV>(EO + c, CS, 1, wx + wt * TW, sx, hx, s);
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int k = wt * TW + i;
            if (k >= hx) break;
#pragma unroll
            for (int j = 0; j < TV; ++j) {
                if (c + j >= C) break;
                T ur = s[i][j][0] + s[i][j][3], ui = s[i][j][1] - s[i][j][2];
                const double g1 = TABLE ? g[i][j][0] : dft_influence(a, k, c0 + c + j, ur, ui, red);
                ur = (T)((double)ur * g1);
                ui = (T)((double)ui * g1);
                Cpair<T> p;
                if (k == 0 || 2 * k == Kx) {
                    p = {ur, ui, T(0), T(0)};
                } else {
                    T vr = s[i][j][0] - s[i][j][3], vi = s[i][j][1] + s[i][j][2];
                    const double g2 = TABLE ? g[i][j][1] : dft_influence(a, Kx - k, c0 + c + j, vr, vi, red);
                    vr = (T)((double)vr * g2);
                    vi = (T)((double)vi * g2);
                    p = {ur + vr, ui + vi, ur - vr, ui - vi};
                }
                PM[k * CS + c + j] = p;
            }
        }
    }
    __syncthreads();
    for (int t = tid; t < nc * nw; t += nth) {
        const int wt = dft_div(t, rt), c = (t - wt * nc) * TV;
        T s[TW][TV][4];
        dft_tile<T, TW, TV>(PM + c, CS, 1, wx + wt * TW, sx, hx, s);
#pragma unroll
        for (int i = 0; i < TW; ++i) {
            const int x = wt * TW + i;
            if (x >= hx) break;
#pragma unroll
            for (int j = 0; j < TV; ++j) {
                if (c + j >= C) break;
                T2 o;
                o.x = s[i][j][0] - s[i][j][3];
                o.y = s[i][j][1] + s[i][j][2];
                S[x * ncol + c + j] = o;
                if (x != 0 && 2 * x != Kx) {
                    o.x = s[i][j][0] + s[i][j][3];
                    o.y = s[i][j][1] - s[i][j][2];
                    S[(Kx - x) * ncol + c + j] = o;
                }
            }
        }
    }
}

// inverse y and z transforms of plane x for the y pairs (y, Ky - y), y in [y0, y0 + chunk)
template <typename T, int TW, int TV>
__device__ inline void dft_inv_item(const DftConvArgs<T>& a, int item, T* sm, const T* wys, const T* wzs) {
    using T2 = typename Vec2<T>::type;
    const int tid = threadIdx.x, nth = blockDim.x;
    const int Ky = a.K[1], Kz = a.K[2], hz = a.H[2] + 1, hy = a.H[1] + 1;
    const int sy = dft_stride(a.H[1]), sz = dft_stride(a.H[2]), ZS = (hz + 3) & ~3;
    const int nchunk = (a.H[1] + a.inv_chunk) / a.inv_chunk;
    const int x = item / nchunk, y0 = (item - x * nchunk) * a.inv_chunk;
    const int C = min(a.inv_chunk, hy - y0);
    Cpair<T>* EO = (Cpair<T>*)sm;  // [hy][ZS] folded spectrum
    Cpair<T>* F = EO + hy * ZS;    // [C rounded up to TW][ZS] rows y and Ky - y
    const T2 *wy = (const T2*)wys + y0, *wz = (const T2*)wzs;
    const T2* S = a.spec + (size_t)x * Ky * hz;
    const float rz = 1.f / (float)hz;
    for (int t0 = tid; t0 < hy * hz; t0 += 2 * kDftBatch * nth) {
        T2 u[2 * kDftBatch], v[2 * kDftBatch];
        bool self[2 * kDftBatch];
#pragma unroll
        for (int q = 0; q < 2 * kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hy * hz) {
                const int ky = dft_div(t, rz), k = t - ky * hz, ky2 = ky == 0 ? 0 : Ky - ky;
                self[q] = ky == ky2;
                u[q] = S[t];
                v[q] = S[ky2 * hz + k];
            }
        }
#pragma unroll
        for (int q = 0; q < 2 * kDftBatch; ++q) {
            const int t = t0 + q * nth;
            if (t < hy * hz) {
                const int ky = dft_div(t, rz), k = t - ky * hz;
                Cpair<T> p;
                if (self[q]) p = {u[q].x, u[q].y, T(0), T(0)};
                else p = {u[q].x + v[q].x, u[q].y + v[q].y, u[q].x - v[q].x, u[q].y - v[q].y};
                EO[ky * ZS + k] = p;
            }
        }
    }
    dft_wait();
    __syncthreads();
    {
        const int nk = (hz + TV - 1) / TV, nw = (C + TW - 1) / TW;
        const float rk = 1.f / (float)nk;
        for (int t = tid; t < nk * nw; t += nth) {
            const int wt = dft_div(t, rk), k = (t - wt * nk) * TV;
            T s[TW][TV][4];
            dft_tile<T, TW, TV>(EO + k, ZS, 1, wy + wt * TW, sy, hy, s);
#pragma unroll
            for (int i = 0; i < TW; ++i)
#pragma unroll
                for (int j = 0; j < TV; ++j) {
                    if (k + j >= hz) break;
                    // kz and Kz - kz are complex conjugates: interior columns count twice
                    const T f = (k + j == 0 || 2 * (k + j) == Kz) ? T(1) : T(2);
                    Cpair<T> p = {f * (s[i][j][0] - s[i][j][3]), f * (s[i][j][0] + s[i][j][3]),
                                  f * (s[i][j][1] + s[i][j][2]), f * (s[i][j][1] - s[i][j][2])};
                    F[(wt * TW + i) * ZS + k + j] = p;
                }
        }
    }
    __syncthreads();
    T* plane = a.grid_out + (size_t)x * Ky * Kz;
    const int nz = (hz + TW - 1) / TW, ny = (C + TV - 1) / TV;
    const float rn = 1.f / (float)nz;
    for (int t = tid; t < nz * ny; t += nth) {
        const int yt = dft_div(t, rn), z0 = (t - yt * nz) * TW, yp = yt * TV;
        T s[TW][TV][4];
        dft_tile<T, TW, TV>(F + yp * ZS, 1, ZS, wz + z0, sz, hz, s);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (yp + j >= C) break;
            const int y = y0 + yp + j;
            const bool other = y != 0 && 2 * y != Ky;
#pragma unroll
            for (int i = 0; i < TW; ++i) {
                const int z = z0 + i;
                if (z >= hz) break;
                const bool both = z != 0 && 2 * z != Kz;
                plane[y * Kz + z] = s[i][j][0] - s[i][j][2];
                if (both) plane[y * Kz + Kz - z] = s[i][j][0] + s[i][j][2];
                if (other) {
                    plane[(Ky - y) * Kz + z] = s[i][j][1] - s[i][j][3];
                    if (both) plane[(Ky - y) * Kz + Kz - z] = s[i][j][1] + s[i][j][3];
                }
            }
        }
    }
}

template <typename T, int TW, int TV>
__global__ void __launch_bounds__(kDftThreads) k_dft_fwd(DftConvArgs<T> a) {
    extern __shared__ __align__(16) unsigned char dft_sm[];
    T* sm = (T*)dft_sm;
    T *wy = sm + ((dft_fwd_elems(a) + 3) & ~(size_t)3), *wz = wy + dft_mat_elems(a.H[1]);
    dft_load_mat(a, 1, wy);
    dft_load_mat(a, 2, wz);
    dft_fwd_item<T, TW, TV>(a, blockIdx.x, sm, wy, wz);
}

template <typename T, int TW, int TV, bool TABLE>
__global__ void __launch_bounds__(kDftThreads) k_dft_columns(DftConvArgs<T> a) {
    extern __shared__ __align__(16) unsigned char dft_sm[];
    T* sm = (T*)dft_sm;
    T* wx = sm + ((dft_col_elems(a) + 3) & ~(size_t)3);
    dft_load_mat(a, 0, wx);
    double red[7] = {0, 0, 0, 0, 0, 0, 0};
    dft_col_item<T, TW, TV, TABLE>(a, blockIdx.x, sm, wx, red);
    if (a.zero_real) {
        const int64_t m = (int64_t)a.K[0] * a.K[1] * a.K[2];
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
            a.zero_real[i] = T(0);
    }
    if (!TABLE && a.want_energy) block_reduce_add<7>(red, a.scal);
}

template <typename T, int TW, int TV>
__global__ void __launch_bounds__(kDftThreads) k_dft_inv(DftConvArgs<T> a) {
    extern __shared__ __align__(16) unsigned char dft_sm[];
    T* sm = (T*)dft_sm;
    T *wy = sm + ((dft_inv_elems(a) + 3) & ~(size_t)3), *wz = wy + dft_mat_elems(a.H[1]);
    dft_load_mat(a, 1, wy);
    dft_load_mat(a, 2, wz);
    dft_inv_item<T, TW, TV>(a, blockIdx.x, sm, wy, wz);
}

// shared memory of the three kernels (bytes)
template <typename T> __host__ inline size_t dft_fwd_smem(const DftConvArgs<T>& a) {
    return sizeof(T) * (((dft_fwd_elems(a) + 3) & ~(size_t)3) + dft_mat_elems(a.H[1]) + dft_mat_elems(a.H[2]));
}
template <typename T> __host__ inline size_t dft_col_smem(const DftConvArgs<T>& a) {
    return sizeof(T) * (((dft_col_elems(a) + 3) & ~(size_t)3) + dft_mat_elems(a.H[0]));
}
template <typename T> __host__ inline size_t dft_inv_smem(const DftConvArgs<T>& a) {
    return sizeof(T) * (((dft_inv_elems(a) + 3) & ~(size_t)3) + dft_mat_elems(a.H[1]) + dft_mat_elems(a.H[2]));
}

// influence function of the half spectrum (k = 0: 0), for the passes of a dipole solve
static __global__ void k_dft_gtable(int K0, int K1, int K2, Box b, const double* bmod, double kappa, double V, double* G) {
    const int hz = K2 / 2 + 1;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)K0 * K1 * hz) return;
    const int k3 = (int)(idx % hz), k2 = (int)((idx / hz) % K1), k1 = (int)(idx / ((int64_t)hz * K1));
    const int m1 = k1 < (K0 + 1) / 2 ? k1 : k1 - K0;
    const int m2 = k2 < (K1 + 1) / 2 ? k2 : k2 - K1;
    const int m3 = k3 < (K2 + 1) / 2 ? k3 : k3 - K2;
    double g = 0.0;
    if (m1 != 0 || m2 != 0 || m3 != 0) {
        double ksq = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double kc = 6.283185307179586 * (b.hinv[3 * c] * m1 + b.hinv[3 * c + 1] * m2 + b.hinv[3 * c + 2] * m3);
            ksq += kc * kc;
        }
        double C, dln;
        influence(CK_COUL, ksq, kappa, V, C, dln);
        const double th = bmod[k1] * bmod[K0 + k2] * bmod[K0 + K1 + k3];
        g = C / (th * th);
    }
    G[idx] = g;
}

}  // namespace dmffb
