// Reciprocal-space smooth PME for multipoles up to quadrupoles (sm_100a).
//
// Follows dmff/admp/recip.py:9-471: order-6 cardinal B-splines on a K1 x K2 x K3 mesh, the
// multipole "gradient operator" spread (recip.py:254-349), an FFT, the influence function
// C_k / theta_k^2 (recip.py:438-466, Ck_1 at :474) and the energy sum.  The reference gets
// forces by autodiff; here the gather is explicit: the convolved mesh phi is interpolated
// with B-spline derivatives up to third order (20 sums per atom), giving dE/dpos, dE/dQ,
// torques and the box gradient in one pass.
//
// Layout: each atom's 6x6x6 stencil is 36 (x, y) columns of 6 contiguous z points; one warp owns one
// atom, its lanes cover whole columns in runs of six consecutive addresses.  The multipole is first
// mapped to mesh-derivative coefficients c_abc (mu^u = -B mu, Theta^u = B Theta B^T with B the
// reference's derivative operator, recip.py:213/251), so the per-point work is a 3-term dot product.
// Spreading uses FP32/FP64 atomics on the mesh (it lives in L2); the gather is atomics-free.
#pragma once
#include "common.cuh"

namespace dmffb {

struct MeshGeom {
    double NA[9];   // grid coordinates x_j = sum_c NA[j][c] R_c  (NA = diag(K) h^-T)
    double B[9];    // derivative operator used by the reference: B = NA^T
    int K[3];
};

// order-6 B-spline values and derivatives at u = w + j, j = 0..5, w in [0, 1]
template <typename T>
__device__ __forceinline__ void bspline6(T w, T M0[6], T M1[6], T M2[6], T M3[6]) {
    T m2[2] = {w, T(1) - w};
    T m3[3], m4[4], m5[5];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        T a = j < 2 ? m2[j] : T(0);
        T b = j > 0 ? m2[j - 1] : T(0);
        m3[j] = ((w + T(j)) * a + (T(3) - w - T(j)) * b) * T(0.5);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        T a = j < 3 ? m3[j] : T(0);
        T b = j > 0 ? m3[j - 1] : T(0);
        m4[j] = ((w + T(j)) * a + (T(4) - w - T(j)) * b) * T(1.0 / 3.0);
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        T a = j < 4 ? m4[j] : T(0);
        T b = j > 0 ? m4[j - 1] : T(0);
        m5[j] = ((w + T(j)) * a + (T(5) - w - T(j)) * b) * T(0.25);
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        T a = j < 5 ? m5[j] : T(0);
        T b = j > 0 ? m5[j - 1] : T(0);
        M0[j] = ((w + T(j)) * a + (T(6) - w - T(j)) * b) * T(0.2);
        M1[j] = a - b;
        T c0 = j < 4 ? m4[j] : T(0), c1 = (j >= 1 && j - 1 < 4) ? m4[j - 1] : T(0), c2 = j >= 2 ? m4[j - 2] : T(0);
        M2[j] = c0 - T(2) * c1 + c2;
        T e0 = j < 3 ? m3[j] : T(0), e1 = (j >= 1 && j - 1 < 3) ? m3[j - 1] : T(0);
        T e2 = (j >= 2 && j - 2 < 3) ? m3[j - 2] : T(0), e3 = j >= 3 ? m3[j - 3] : T(0);
        M3[j] = e0 - T(3) * e1 + T(3) * e2 - e3;
    }
}

__device__ __forceinline__ int wrapi(int g, int K) {
    g %= K;
    return g < 0 ? g + K : g;
}

// mesh-derivative coefficients of one site: c[0]=000, 1..3 = e_x,e_y,e_z, 4..9 = xx,yy,zz,xy,xz,yz
// (second-order entries hold Theta^u_jk summed over both orders for j != k).
template <typename T>
__device__ __forceinline__ void site_coefs(const double* B, T q, const T mu[3], const T Th[3][3], T c[10]) {
    c[0] = q;
#pragma unroll
    for (int j = 0; j < 3; ++j) c[1 + j] = -(T(B[3 * j]) * mu[0] + T(B[3 * j + 1]) * mu[1] + T(B[3 * j + 2]) * mu[2]);
    T BT[3][3];  // (B Theta)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int d = 0; d < 3; ++d) BT[j][d] = T(B[3 * j]) * Th[0][d] + T(B[3 * j + 1]) * Th[1][d] + T(B[3 * j + 2]) * Th[2][d];
    T Tu[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) Tu[j][k] = BT[j][0] * T(B[3 * k]) + BT[j][1] * T(B[3 * k + 1]) + BT[j][2] * T(B[3 * k + 2]);
    c[4] = Tu[0][0];
    c[5] = Tu[1][1];
    c[6] = Tu[2][2];
    c[7] = Tu[0][1] + Tu[1][0];
    c[8] = Tu[0][2] + Tu[2][0];
    c[9] = Tu[1][2] + Tu[2][1];
}

// harmonic quadrupole (Q4..Q8, recip.py:317-349 with the /3) -> Cartesian coefficient matrix
template <typename T>
__device__ __forceinline__ void quad_cart(const T* Qq, T Th[3][3]) {
    const T s = T(DMFFB_SQRT3 / 6.0);
    Th[2][2] = Qq[0] * T(1.0 / 3.0);
    Th[0][0] = -Qq[0] * T(1.0 / 6.0) + Qq[3] * s;
    Th[1][1] = -Qq[0] * T(1.0 / 6.0) - Qq[3] * s;
    Th[0][2] = Th[2][0] = Qq[1] * s;
    Th[1][2] = Th[2][1] = Qq[2] * s;
    Th[0][1] = Th[1][0] = Qq[4] * s;
}

template <typename T>
struct SpreadArgs {
    int n;
    const double* pos;  // [n*3]
    const T* Qg;        // [n*9] permanent (may be null)
    const double* U;    // [n*3] Cartesian dipoles (may be null)
    const T* q1;        // [n] plain charges for charge-only channels (may be null)
    int lmax;           // 0: charge only, 1: up to dipole, 2: up to quadrupole
    MeshGeom g;
    T* grid;
    int perm_mul;  // warps visit atoms in the order (w * perm_mul) mod n, gcd(perm_mul, n) = 1
};

template <typename T>
__device__ __forceinline__ void site_multipole(const SpreadArgs<T>& a, int at, T& q, T mu[3], T Th[3][3]) {
    q = T(0);
    mu[0] = mu[1] = mu[2] = T(0);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) Th[r][c] = T(0);
    if (a.q1) q = a.q1[at];
    if (a.Qg) {
        const T* Q = a.Qg + 9 * at;
        q += Q[0];
        if (a.lmax >= 1) { mu[0] = Q[2]; mu[1] = Q[3]; mu[2] = Q[1]; }
        if (a.lmax >= 2) quad_cart(Q + 4, Th);
    }
    if (a.U) {
        mu[0] += (T)a.U[3 * at];
        mu[1] += (T)a.U[3 * at + 1];
        mu[2] += (T)a.U[3 * at + 2];
    }
}

// A CTA of the spread and the gather takes `apc` sites (at most kSiteAtoms).  What one site needs once
// is computed once, by one thread each, into shared memory: the splines of a site and axis (up to
// derivative ORD, interleaved so that the orders of one point are one vector load), its wrapped first
// stencil point, and for the spread its coefficients.
constexpr int kSiteThreads = 256, kSiteAtoms = 32;

// Sites per CTA.  One per warp while that leaves the SMs fewer than eight CTAs (450 sites: 57 CTAs
// instead of 15), more once the chip is full, where the per-CTA work is shared by more sites.
inline int sites_per_cta(int n) { return n <= 8 * 8 * 148 ? 8 : (n <= 16 * 8 * 148 ? 16 : kSiteAtoms); }

template <typename T, int ORD>
struct SiteStencils {
    static constexpr int NV = ORD <= 1 ? 2 : 4;  // orders stored per point
    __align__(16) T w[kSiteAtoms][3][6][NV];
    int org[kSiteAtoms][3];

    __device__ __forceinline__ void set(const MeshGeom& g, const double* pos, int at, int m, int d) {
        const double x = g.NA[3 * d] * pos[3 * at] + g.NA[3 * d + 1] * pos[3 * at + 1] + g.NA[3 * d + 2] * pos[3 * at + 2];
        const double c = ceil(x);
        org[m][d] = wrapi((int)c - 3, g.K[d]);
        T M[4][6];
        bspline6<T>((T)(c - x), M[0], M[1], M[2], M[3]);
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
            for (int o = 0; o < NV; ++o) w[m][d][t][o] = o <= ORD ? M[o][t] : T(0);
    }
};

// g + d wrapped into [0, K) for g in [0, K), d >= 0
__device__ __forceinline__ int wrap_up(int g, int K) {
    while (g >= K) g -= K;
    return g;
}

// Spread of the sites' multipoles (CH: charges alone) onto the mesh.  A warp takes a site, first its 36
// columns' weights (lanes own columns, results through shared memory), then its 216 points 32 at a
// time: seven atomics per lane whose addresses are runs of six.  Bound by the L2 atomics: 21 M in
// 36 us for 99000 charges, 23 us for 30000 multipoles.  With lanes owning whole columns and every lane
// evaluating all splines these took 168 and 56 us.
template <typename T, bool CH>
__global__ void __launch_bounds__(kSiteThreads) k_spread(SpreadArgs<T> a, int apc) {
    constexpr int ORD = CH ? 0 : 2, NW = kSiteThreads / 32;
    __shared__ SiteStencils<T, ORD> st;
    __shared__ T s_c[kSiteAtoms][CH ? 1 : 10];
    __shared__ T s_col[NW][36][CH ? 1 : 3];
    __shared__ int s_base[NW][36];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int first = blockIdx.x * apc, m1 = min(apc, a.n - first);
    // concurrently running warps take atoms far apart in the box, which keeps them off the same
    // mesh addresses (atoms are usually stored in spatial order)
    auto site = [&](int m) { return (int)(((int64_t)(first + m) * a.perm_mul) % a.n); };
    for (int k = tid; k < 4 * m1; k += kSiteThreads) {
        const int m = k >> 2, d = k & 3;
        const int at = site(m);
        if (d < 3) {
            st.set(a.g, a.pos, at, m, d);
        } else if (CH) {
            s_c[m][0] = a.q1[at];
        } else {
            T q, mu[3], Th[3][3], c[10];
            site_multipole(a, at, q, mu, Th);
            site_coefs<T>(a.g.B, q, mu, Th, c);
#pragma unroll
            for (int j = 0; j < 10; ++j) s_c[m][CH ? 0 : j] = c[j];
        }
    }
    __syncthreads();
    const int K0 = a.g.K[0], K1 = a.g.K[1], K2 = a.g.K[2];
    for (int m = wl; m < m1; m += NW) {
        const int ox = st.org[m][0], oy = st.org[m][1], oz = st.org[m][2];
        for (int L = lane; L < 36; L += 32) {
            const int ix = L / 6, iy = L - 6 * ix;
            s_base[wl][L] = wrap_up(ox + ix, K0) * K1 + wrap_up(oy + iy, K1);
            const T* X = st.w[m][0][ix];
            const T* Y = st.w[m][1][iy];
            const T* c = s_c[m];
            if (CH) {
                s_col[wl][L][0] = c[0] * (X[0] * Y[0]);
            } else {
                constexpr int o1 = CH ? 0 : 1, o2 = CH ? 0 : 2;  // in range for the CH instantiation too
                const T x0 = X[0], x1 = X[1], x2 = X[o2], y0 = Y[0], y1 = Y[1], y2 = Y[o2];
                const T xy = x0 * y0, x1y = x1 * y0, xy1 = x0 * y1;
                s_col[wl][L][0] = c[0] * xy + c[1] * x1y + c[2] * xy1 + c[4] * x2 * y0 + c[5] * x0 * y2 + c[7] * x1 * y1;
                s_col[wl][L][o1] = c[3] * xy + c[8] * x1y + c[9] * xy1;
                s_col[wl][L][o2] = c[6] * xy;
            }
        }
        __syncwarp();
#pragma unroll
        for (int pass = 0; pass < 7; ++pass) {
            const int p = lane + 32 * pass;
            if (p < 216) {
                const int col = p / 6, iz = p - 6 * col;
                const T* Z = st.w[m][2][iz];
                const T* sc = s_col[wl][col];
                const T v = CH ? sc[0] * Z[0] : sc[0] * Z[0] + sc[CH ? 0 : 1] * Z[1] + sc[CH ? 0 : 2] * Z[CH ? 0 : 2];
                atomicAdd(a.grid + (size_t)s_base[wl][col] * K2 + wrap_up(oz + iz, K2), v);
            }
        }
        __syncwarp();
    }
}

enum { CK_COUL = 0, CK_DISP6 = 1, CK_DISP8 = 2, CK_DISP10 = 3 };

template <typename T>
struct ConvArgs {
    int K[3];
    int Kh;              // K3/2 + 1
    T* S;                // [K1*K2*Kh] interleaved complex (re, im), overwritten by G*S
    const double* bmod;  // [K1 + K2 + K3] per-dimension B-spline moduli (recip.py:440-448)
    double hinv[9];
    double V;
    double kappa;
    double escale;       // DIELECTRIC for Coulomb, 1 for dispersion
    int kind;
    double* scal;        // [0] energy, [1..6] sum E_k (dlnC/dk2) k k  (xx,yy,zz,xy,xz,yz)
    int want_energy;
    T* zero_real = nullptr;  // real grid of nzero elements the kernel sets to 0 (may be null)
    int64_t nzero = 0;
};

// influence function C(k^2) and d ln C / d k^2
__device__ __forceinline__ void influence(int kind, double ksq, double kappa, double V, double& C, double& dlnC) {
    const double SQRT_PI = 1.7724538509055159;
    const double PI = 3.141592653589793;
    if (kind == CK_COUL) {
        C = 2.0 * PI / V / ksq * exp(-ksq / 4.0 / (kappa * kappa));
        dlnC = -1.0 / ksq - 1.0 / (4.0 * kappa * kappa);
        return;
    }
    // dispersion (recip.py:477-508): ksq thresholded at 1e-16
    const double ks = ksq < 1e-16 ? 1e-16 : ksq;
    const double x2 = ks / 4.0 / (kappa * kappa);
    const double x = sqrt(x2);
    const double ex = exp(-x2);
    const double ec = erfc(x);
    double f, dfdx, pref;
    if (kind == CK_DISP6) {
        const double x3 = x2 * x;
        f = (1 - 2 * x2) * ex + 2 * x3 * SQRT_PI * ec;
        // d/dx: (-4x)e + (1-2x^2)(-2x)e + 6x^2 sqrt(pi) erfc - 2x^3 * 2 e
        dfdx = -4 * x * ex - 2 * x * (1 - 2 * x2) * ex + 6 * x2 * SQRT_PI * ec - 4 * x3 * ex;
        pref = SQRT_PI * PI / 2 / V * kappa * kappa * kappa / 3;
    } else if (kind == CK_DISP8) {
        const double x4 = x2 * x2, x5 = x4 * x;
        f = (3 - 2 * x2 + 4 * x4) * ex - 4 * x5 * SQRT_PI * ec;
        dfdx = (-4 * x + 16 * x2 * x) * ex - 2 * x * (3 - 2 * x2 + 4 * x4) * ex - 20 * x4 * SQRT_PI * ec + 8 * x5 * ex;
        pref = SQRT_PI * PI / 2 / V * pow(kappa, 5) / 45;
    } else {
        const double x4 = x2 * x2, x6 = x4 * x2, x7 = x6 * x;
        f = (15 - 6 * x2 + 4 * x4 - 8 * x6) * ex + 8 * x7 * SQRT_PI * ec;
        dfdx = (-12 * x + 16 * x2 * x - 48 * x4 * x) * ex - 2 * x * (15 - 6 * x2 + 4 * x4 - 8 * x6) * ex + 56 * x6 * SQRT_PI * ec - 16 * x7 * ex;
        pref = SQRT_PI * PI / 2 / V * pow(kappa, 7) / 1260;
    }
    C = pref * f;
    // d/dk2 = dx/dk2 d/dx, x = sqrt(k2)/(2 kappa) -> dx/dk2 = 1/(8 kappa^2 x)
    dlnC = (ksq < 1e-16) ? 0.0 : dfdx / f / (8.0 * kappa * kappa * x);
}

// Influence function, energy and k-space tensor over the half spectrum.  A warp takes rows (k1, k2) in
// turn, lanes the k3 of a row; the sums stay in registers until the end, so a launch issues seven
// atomics per CTA of a grid that fills the chip once (kConvCtas).  With one element per thread and
// a CTA per 256 of them, the atomics of 22 000 CTAs on the same seven words bounded it: 180 us at
// 225^3, now 57 (FP64 exponentials and quotients, 92 MB moved).
constexpr int kConvCtas = 8 * 148;

template <typename T, bool COUL>
__global__ void __launch_bounds__(256) k_conv(ConvArgs<T> a) {
    const int lane = threadIdx.x & 31;
    const int rows = a.K[0] * a.K[1], Kh = a.Kh;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const double TWO_PI = 6.283185307179586;
    const double c0 = TWO_PI * a.hinv[2], c1 = TWO_PI * a.hinv[5], c2 = TWO_PI * a.hinv[8];
    const double ik = 1.0 / (4.0 * a.kappa * a.kappa), pref = TWO_PI / a.V;
    double red[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int row = gw; row < rows; row += nw) {
        const int k1 = row / a.K[1], k2 = row - k1 * a.K[1];
        const int m1 = k1 < (a.K[0] + 1) / 2 ? k1 : k1 - a.K[0];
        const int m2 = k2 < (a.K[1] + 1) / 2 ? k2 : k2 - a.K[1];
        const double b0 = TWO_PI * (a.hinv[0] * m1 + a.hinv[1] * m2), b1 = TWO_PI * (a.hinv[3] * m1 + a.hinv[4] * m2),
                     b2 = TWO_PI * (a.hinv[6] * m1 + a.hinv[7] * m2);
        const double th12 = a.bmod[k1] * a.bmod[a.K[0] + k2];
        for (int k3 = lane; k3 < Kh; k3 += 32) {
            const int m3 = k3 < (a.K[2] + 1) / 2 ? k3 : k3 - a.K[2];
            const double kv[3] = {b0 + c0 * m3, b1 + c1 * m3, b2 + c2 * m3};
            const double ksq = kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2];
            const double th = th12 * a.bmod[a.K[0] + a.K[1] + k3], th2 = th * th;
            double G = 0.0, dlnC = 0.0;
            const bool zero = m1 == 0 && m2 == 0 && m3 == 0;
            if (COUL) {
                if (!zero) {  // influence() with its quotients brought over one denominator
                    const double d = 1.0 / (ksq * th2);
                    G = pref * exp(-ksq * ik) * d;
                    dlnC = -d * th2 - ik;
                }
            } else {
                double C;
                influence(a.kind, ksq, a.kappa, a.V, C, dlnC);
                G = C / th2;
            }
            T* s = a.S + 2 * ((size_t)row * Kh + k3);
            const double re = (double)s[0], im = (double)s[1];
            if (a.want_energy) {
                const bool self_conj = (k3 == 0) || ((a.K[2] % 2 == 0) && k3 == a.K[2] / 2);
                const double w = self_conj ? 1.0 : 2.0;
                const double Ek = a.escale * w * G * (re * re + im * im);
                red[0] += Ek;
                const double f = Ek * dlnC, fx = f * kv[0], fy = f * kv[1];
                red[1] += fx * kv[0];
                red[2] += fy * kv[1];
                red[3] += f * kv[2] * kv[2];
                red[4] += fx * kv[1];
                red[5] += fx * kv[2];
                red[6] += fy * kv[2];
            }
            s[0] = (T)(re * G);
            s[1] = (T)(im * G);
        }
    }
    // the spread input of this pass has been transformed: clear it for the next spread
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.nzero; i += (int64_t)gridDim.x * blockDim.x)
        a.zero_real[i] = T(0);
    if (a.want_energy) block_reduce_add<7>(red, a.scal);
}

enum { GATHER_FULL = 0, GATHER_FIELD = 1 };

template <typename T>
struct GatherArgs {
    int n;
    const double* pos;
    const T* Qg;          // permanent multipoles (torque and coefficients), may be null
    const double* U;      // induced dipoles added to the spread multipole, may be null
    const T* q1;          // plain charges (charge-only channel), may be null
    int lmax;
    MeshGeom g;
    const T* phi;         // convolved mesh (real)
    double scale;         // dE/dmesh = scale * phi   (2*DIELECTRIC or 2)
    double* grad;         // [n*3] += dE/dpos
    T* torque;            // [n*4] += torque of permanent multipoles (may be null)
    double* gQ;           // [n*9] += dE/dQ_global (may be null)
    double* dq1;          // [n] += dE/dq for the charge channel (may be null)
    double* scal;         // [0] energy (1/2 sum c P), [1..9] X_NA
};

// Interpolation of the convolved mesh and its derivatives at the sites (CH: charges alone, value and
// first derivatives), then dE/dpos, dE/dQ, torques and the box term.  A warp takes a site: lanes
// 0..29 read five columns' six points per pass (runs of six addresses) and keep the sums over the columns
// at their own z, contract them with the z splines and add them over the warp.  The rest, a few
// hundred FP64 operations per site, runs with one thread per site.  Latency-bound (L2 reads): 55 us
// for 99000 charges, 44 us for 30000 multipoles.  With lane 0 of each warp doing that rest for its one
// site, ten atomics per eight sites and all 20 sums also for charges these took 336 and 110 us.
template <typename T, bool CH>
__global__ void __launch_bounds__(kSiteThreads) k_gather(GatherArgs<T> a, int apc) {
    constexpr int ORD = CH ? 1 : 3, NS = CH ? 4 : 20, NW = kSiteThreads / 32;
    __shared__ SiteStencils<T, ORD> st;
    __shared__ T s_P[kSiteAtoms][NS + 1];  // odd stride: the sites' threads read it side by side
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int first = blockIdx.x * apc, m1 = min(apc, a.n - first);
    for (int k = tid; k < 3 * m1; k += kSiteThreads) st.set(a.g, a.pos, first + k / 3, k / 3, k % 3);
    __syncthreads();
    const int K0 = a.g.K[0], K1 = a.g.K[1], K2 = a.g.K[2];
    const int grp = lane / 6, iz = lane - 6 * grp;
    for (int m = wl; m < m1; m += NW) {
        const int ox = st.org[m][0], oy = st.org[m][1], gz = wrap_up(st.org[m][2] + iz, K2);
        T v[8];
#pragma unroll
        for (int pass = 0; pass < 8; ++pass) {
            const int col = grp + 5 * pass, ix = col / 6, iy = col - 6 * ix;
            v[pass] = grp < 5 && col < 36
                          ? a.phi[((size_t)wrap_up(ox + ix, K0) * K1 + wrap_up(oy + iy, K1)) * K2 + gz]
                          : T(0);
        }
        // partial sums P_abc, a+b+c <= 3, order:
        // 0:000 1:100 2:010 3:001 4:200 5:020 6:002 7:110 8:101 9:011
        // 10:300 11:030 12:003 13:210 14:201 15:120 16:021 17:102 18:012 19:111
        T P[NS];
        const T* Z = st.w[m][2][iz];
        if constexpr (CH) {
            T A00 = T(0), A10 = T(0), A01 = T(0);
#pragma unroll
            for (int pass = 0; pass < 8; ++pass) {
                const int col = min(grp + 5 * pass, 35), ix = col / 6, iy = col - 6 * ix;
                const T* X = st.w[m][0][ix];
                const T* Y = st.w[m][1][iy];
                const T t0 = v[pass] * Y[0], t1 = v[pass] * Y[1];
                A00 += X[0] * t0;
                A10 += X[1] * t0;
                A01 += X[0] * t1;
            }
            P[0] = A00 * Z[0];
            P[1] = A10 * Z[0];
            P[2] = A01 * Z[0];
            P[3] = A00 * Z[1];
        } else {
            T A00 = T(0), A10 = T(0), A01 = T(0), A20 = T(0), A11 = T(0), A02 = T(0), A30 = T(0), A21 = T(0),
              A12 = T(0), A03 = T(0);
#pragma unroll
            for (int pass = 0; pass < 8; ++pass) {
                const int col = min(grp + 5 * pass, 35), ix = col / 6, iy = col - 6 * ix;
                const T* X = st.w[m][0][ix];
                const T* Y = st.w[m][1][iy];
                const T t0 = v[pass] * Y[0], t1 = v[pass] * Y[1], t2 = v[pass] * Y[2], t3 = v[pass] * Y[3];
                A00 += X[0] * t0;
                A10 += X[1] * t0;
                A20 += X[2] * t0;
                A30 += X[3] * t0;
                A01 += X[0] * t1;
                A11 += X[1] * t1;
                A21 += X[2] * t1;
                A02 += X[0] * t2;
                A12 += X[1] * t2;
                A03 += X[0] * t3;
            }
            const T z0 = Z[0], z1 = Z[1], z2 = Z[2], z3 = Z[3];
            P[0] = A00 * z0;
            P[1] = A10 * z0;
            P[2] = A01 * z0;
            P[3] = A00 * z1;
            P[4] = A20 * z0;
            P[5] = A02 * z0;
            P[6] = A00 * z2;
            P[7] = A11 * z0;
            P[8] = A10 * z1;
            P[9] = A01 * z1;
            P[10] = A30 * z0;
            P[11] = A03 * z0;
            P[12] = A00 * z3;
            P[13] = A21 * z0;
            P[14] = A20 * z1;
            P[15] = A12 * z0;
            P[16] = A02 * z1;
            P[17] = A10 * z2;
            P[18] = A01 * z2;
            P[19] = A11 * z1;
        }
        warp_sums<T, NS>(P, s_P[m], lane);
    }
    __syncthreads();
    if (wl) return;  // one thread per site from here on
    double red[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) red[k] = 0.0;
    if (CH && lane < m1) {
        // c = {q}: energy q P_000 / 2, dE/dx = -q (P_100, P_010, P_001)
        const int at = first + lane;
        const double q = (double)a.q1[at], P0 = a.scale * (double)s_P[lane][0];
        double Y[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) Y[j] = -q * (a.scale * (double)s_P[lane][1 + j]);
        const double* NA = a.g.NA;
        double* gr = a.grad + 3 * at;
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) gr[cc] += NA[cc] * Y[0] + NA[3 + cc] * Y[1] + NA[6 + cc] * Y[2];
        red[0] = 0.5 * (q * P0);
        if (a.dq1) a.dq1[at] += P0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) red[1 + 3 * j + cc] = Y[j] * a.pos[3 * at + cc];
    }
    if (!CH && lane < m1) {
        const int at = first + lane;
        const double sc = a.scale;
        double Pd[20];
#pragma unroll
        for (int k = 0; k < 20; ++k) Pd[k] = sc * (double)s_P[lane][k < NS ? k : 0];
        // site multipole (the one that was spread)
        SpreadArgs<T> sa;
        sa.Qg = a.Qg; sa.U = a.U; sa.q1 = a.q1; sa.lmax = a.lmax;
        T q, mu[3], Th[3][3];
        site_multipole(sa, at, q, mu, Th);
        T cT[10];
        site_coefs<T>(a.g.B, q, mu, Th, cT);
        double c[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) c[k] = (double)cT[k];
        const double* B = a.g.B;
        // dE/dmu^u_j and dE/dTheta^u_jk
        const double Pu[3] = {Pd[1], Pd[2], Pd[3]};
        const double P2[3][3] = {{Pd[4], Pd[7], Pd[8]}, {Pd[7], Pd[5], Pd[9]}, {Pd[8], Pd[9], Pd[6]}};
        double dmu[3];
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) dmu[cc] = -(Pu[0] * B[cc] + Pu[1] * B[3 + cc] + Pu[2] * B[6 + cc]);
        {
            // dE/dx_j = -sum_abc c_abc P_{abc + e_j}
            // coefficient -> (a,b,c) exponents; index of abc+e_j in P
            const int up[10][3] = {{1, 2, 3},   {4, 7, 8},   {7, 5, 9},   {8, 9, 6},    {10, 13, 14},
                                   {15, 11, 16}, {17, 18, 12}, {13, 15, 19}, {14, 19, 17}, {19, 16, 18}};
            double Y[3] = {0, 0, 0};
#pragma unroll
            for (int k = 0; k < 10; ++k)
#pragma unroll
                for (int j = 0; j < 3; ++j) Y[j] -= c[k] * Pd[up[k][j]];
            double* gr = a.grad + 3 * at;
            const double* NA = a.g.NA;
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) gr[cc] += NA[cc] * Y[0] + NA[3 + cc] * Y[1] + NA[6 + cc] * Y[2];
            double e = 0.0;
#pragma unroll
            for (int k = 0; k < 10; ++k) e += c[k] * Pd[k];
            red[0] = 0.5 * e;
            // dE/dTheta (Cartesian) = B^T P2 B
            double BP[3][3];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
#pragma unroll
                for (int k = 0; k < 3; ++k) BP[cc][k] = B[cc] * P2[0][k] + B[3 + cc] * P2[1][k] + B[6 + cc] * P2[2][k];
            double dTh[3][3];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
#pragma unroll
                for (int d = 0; d < 3; ++d) dTh[cc][d] = BP[cc][0] * B[d] + BP[cc][1] * B[3 + d] + BP[cc][2] * B[6 + d];
            double g[9];
            g[0] = Pd[0];
            g[1] = dmu[2];
            g[2] = dmu[0];
            g[3] = dmu[1];
            const double s6 = DMFFB_SQRT3 / 6.0;
            g[4] = dTh[2][2] / 3.0 - dTh[0][0] / 6.0 - dTh[1][1] / 6.0;
            g[5] = (dTh[0][2] + dTh[2][0]) * s6;
            g[6] = (dTh[1][2] + dTh[2][1]) * s6;
            g[7] = (dTh[0][0] - dTh[1][1]) * s6;
            g[8] = (dTh[0][1] + dTh[1][0]) * s6;
            if (a.gQ) {
#pragma unroll
                for (int k = 0; k < 9; ++k) a.gQ[9 * at + k] += g[k];
            }
            if (a.dq1) a.dq1[at] += g[0];
            if (a.torque && a.Qg) {
                T qp[9], gT[9], t[3];
#pragma unroll
                for (int k = 0; k < 9; ++k) { qp[k] = a.Qg[9 * at + k]; gT[k] = (T)g[k]; }
                if (a.lmax < 2) { for (int k = 4; k < 9; ++k) qp[k] = T(0); }
                if (a.lmax < 1) { qp[1] = qp[2] = qp[3] = T(0); }
                torque9(qp, gT, t);
                // atomics: the real-space FULL pass may add to the same torques concurrently
                add3(a.torque + 4 * at, t[0], t[1], t[2]);
            }
            {
                // X_NA = Y (x) R + (dE/dB)^T,  dE/dB = -Pu (x) mu + 2 P2 B Theta
                const double R[3] = {a.pos[3 * at], a.pos[3 * at + 1], a.pos[3 * at + 2]};
                double PB[3][3];
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int k = 0; k < 3; ++k) PB[j][k] = P2[j][0] * B[k] + P2[j][1] * B[3 + k] + P2[j][2] * B[6 + k];
#pragma unroll
                for (int j = 0; j < 3; ++j)
#pragma unroll
                    for (int cc = 0; cc < 3; ++cc) {
                        double dB = -Pu[j] * (double)mu[cc];
                        dB += 2.0 * (PB[j][0] * (double)Th[0][cc] + PB[j][1] * (double)Th[1][cc] + PB[j][2] * (double)Th[2][cc]);
                        // (dE/dB)^T[cc][j] adds to X_NA[cc][j]; Y (x) R adds to X_NA[j][cc]
                        red[1 + 3 * cc + j] += dB;
                        red[1 + 3 * j + cc] += Y[j] * R[cc];
                    }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        const double v = warp_sum(red[k]);
        if (lane == 0 && v != 0.0) atomicAdd(a.scal + k, v);
    }
}


// ---------------------------------------------------------------------------------------------
// Lean kernels for the CG loop, where only induced dipoles are spread and only the first
// derivatives of the convolved mesh are gathered: value + first-derivative splines, 3 mesh
// coefficients, 3 sums; small register footprint for occupancy.
template <typename T>
__device__ __forceinline__ void bspline6_01(T w, T M0[6], T M1[6]) {
    T m2[2] = {w, T(1) - w};
    T m3[3], m4[4], m5[5];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        m3[j] = ((w + T(j)) * (j < 2 ? m2[j] : T(0)) + (T(3) - w - T(j)) * (j > 0 ? m2[j - 1] : T(0))) * T(0.5);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        m4[j] = ((w + T(j)) * (j < 3 ? m3[j] : T(0)) + (T(4) - w - T(j)) * (j > 0 ? m3[j - 1] : T(0))) * T(1.0 / 3.0);
#pragma unroll
    for (int j = 0; j < 5; ++j)
        m5[j] = ((w + T(j)) * (j < 4 ? m4[j] : T(0)) + (T(5) - w - T(j)) * (j > 0 ? m4[j - 1] : T(0))) * T(0.25);
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const T a = j < 5 ? m5[j] : T(0), b = j > 0 ? m5[j - 1] : T(0);
        M0[j] = ((w + T(j)) * a + (T(6) - w - T(j)) * b) * T(0.2);
        M1[j] = a - b;
    }
}

template <typename T>
__device__ __forceinline__ void stencil01(const MeshGeom& g, const double* pos, int at, int m0[3], T Mx[2][6],
                                          T My[2][6], T Mz[2][6]) {
    const double R0 = pos[3 * at], R1 = pos[3 * at + 1], R2 = pos[3 * at + 2];
    T (*Ms[3])[6] = {Mx, My, Mz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double x = g.NA[3 * d] * R0 + g.NA[3 * d + 1] * R1 + g.NA[3 * d + 2] * R2;
        const double c = ceil(x);
        m0[d] = (int)c;
        bspline6_01<T>((T)(c - x), Ms[d][0], Ms[d][1]);
    }
}

// v[k] for a runtime k in 0..5 without indexing a register array (a select chain keeps the
// stencil in registers instead of the stack)
template <typename T>
__device__ __forceinline__ T sel6(const T v[6], int k) {
    T r = v[0];
#pragma unroll
    for (int t = 1; t < 6; ++t) r = (k == t) ? v[t] : r;
    return r;
}

// dE/dmu (Cartesian) of every site from the convolved mesh: out = scale * (-B^T grad_u phi).
// Lanes take whole (x, y) stencil columns and read their six z points in sequence (one cache
// line, L1 hits after the first); sel6 keeps the column weights in registers.
template <typename T>
__global__ void __launch_bounds__(256) k_gather_field(int n, const double* pos, MeshGeom g, const T* phi, double scale,
                                                      double* out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= n) return;
    const int at = warp;
    int m0[3];
    T Mx[2][6], My[2][6], Mz[2][6];
    stencil01<T>(g, pos, at, m0, Mx, My, Mz);
    const int K0 = g.K[0], K1 = g.K[1], K2 = g.K[2];
    T p1 = T(0), p2 = T(0), p3 = T(0);
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const int L = lane + 32 * pass;
        if (L < 36) {
            const int ix = L / 6, iy = L - 6 * ix;
            const int gx = wrapi(m0[0] - 3 + ix, K0), gy = wrapi(m0[1] - 3 + iy, K1);
            const T* line = phi + ((size_t)gx * K1 + gy) * K2;
            int gz = wrapi(m0[2] - 3, K2);
            T s0 = T(0), s1 = T(0);
#pragma unroll
            for (int t = 0; t < 6; ++t) {
                const T v = __ldg(line + gz);
                s0 += v * Mz[0][t];
                s1 += v * Mz[1][t];
                gz = (gz + 1 == K2) ? 0 : gz + 1;
            }
            const T mx0 = sel6(Mx[0], ix), mx1 = sel6(Mx[1], ix), my0 = sel6(My[0], iy), my1 = sel6(My[1], iy);
            p1 += mx1 * my0 * s0;
            p2 += mx0 * my1 * s0;
            p3 += mx0 * my0 * s1;
        }
    }
    p1 = warp_sum(p1);
    p2 = warp_sum(p2);
    p3 = warp_sum(p3);
    if (lane == 0) {
        const double* B = g.B;
        const double P1 = scale * (double)p1, P2 = scale * (double)p2, P3 = scale * (double)p3;
#pragma unroll
        for (int c = 0; c < 3; ++c) out[3 * at + c] = -(P1 * B[c] + P2 * B[3 + c] + P3 * B[6 + c]);
    }
}

// ---------------------------------------------------------------------------------------------
// Stencil cache for the CG loop.  Positions are fixed during the dipole solve, so the wrapped
// first stencil point (m0 - 3 per dimension) and the value / first-derivative B-spline weights
// of every atom are computed once per evaluation (k_stencil_prep, with the same arithmetic as
// stencil01) and read by the cached dipole spread and field gather, instead of every lane
// recomputing three spline sets and two integer wraps per pass in every iteration.
// Weights per atom: value and derivative of each point side by side, x then y then z.
template <typename T>
struct StencilCache {
    const int4* org;  // wrapped first stencil point per dimension (w unused)
    const T* w;       // [n * 36]
};

template <typename T>
__global__ void __launch_bounds__(256) k_stencil_prep(int n, const double* pos, MeshGeom g, int4* org, T* w) {
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= n) return;
    int m0[3];
    T Mx[2][6], My[2][6], Mz[2][6];
    stencil01<T>(g, pos, at, m0, Mx, My, Mz);
    org[at] = make_int4(wrapi(m0[0] - 3, g.K[0]), wrapi(m0[1] - 3, g.K[1]), wrapi(m0[2] - 3, g.K[2]), 0);
    T* o = w + 36 * (size_t)at;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        o[2 * j] = Mx[0][j];
        o[2 * j + 1] = Mx[1][j];
        o[12 + 2 * j] = My[0][j];
        o[13 + 2 * j] = My[1][j];
        o[24 + 2 * j] = Mz[0][j];
        o[25 + 2 * j] = Mz[1][j];
    }
}

// One warp's place in a six-point stencil: lanes 0..29 form five groups of six consecutive z points of
// one (x, y) column, the 36 columns take eight passes, so that the mesh addresses of a pass are five
// runs of six.  The atom's 36 weights sit in the lanes (w[0..31] in wl, w[32..35] in wh of lanes 0..3)
// and the wrapped mesh bases in lanes 0..5 (x rows times K1) and 6..11 (y columns); the passes take
// them by shuffles.  Loading a column's weights and wrapping its indices in each pass instead made
// the spread of 30000 dipoles 18.2 us against 15.5 and the gather 22.7 against 21.
template <typename T>
struct StencilLanes {
    T wl, wh, z0, z1;  // z0, z1: value and derivative at the lane's z point
    int base, grp, gz;

    __device__ __forceinline__ StencilLanes(const StencilCache<T>& st, const MeshGeom& g, int at, int lane) {
        grp = lane / 6;
        const int iz = lane - 6 * grp;
        const int4 o = st.org[at];
        const T* w = st.w + 36 * (size_t)at;
        wl = __ldg(w + lane);
        wh = lane < 4 ? __ldg(w + 32 + lane) : T(0);
        base = 0;
        if (lane < 6) base = wrap_up(o.x + lane, g.K[0]) * g.K[1];
        else if (lane < 12) base = wrap_up(o.y + lane - 6, g.K[1]);
        const T a0 = __shfl_sync(0xffffffffu, wl, (24 + 2 * iz) & 31), a1 = __shfl_sync(0xffffffffu, wl, (25 + 2 * iz) & 31);
        const T b0 = __shfl_sync(0xffffffffu, wh, (2 * iz - 8) & 31), b1 = __shfl_sync(0xffffffffu, wh, (2 * iz - 7) & 31);
        z0 = iz < 4 ? a0 : b0;
        z1 = iz < 4 ? a1 : b1;
        gz = wrap_up(o.z + iz, g.K[2]);
    }
    // the lane's column of a pass (the last one where there is none), its weights and mesh point: every
    // lane of the warp takes part
    __device__ __forceinline__ int column(int pass) const { return min(grp + 5 * pass, 35); }
    __device__ __forceinline__ bool has(int pass) const { return grp < 5 && grp + 5 * pass < 36; }
    __device__ __forceinline__ void weights(int col, T& x0, T& x1, T& y0, T& y1) const {
        const int ix = col / 6, iy = col - 6 * ix;
        x0 = __shfl_sync(0xffffffffu, wl, 2 * ix);
        x1 = __shfl_sync(0xffffffffu, wl, 2 * ix + 1);
        y0 = __shfl_sync(0xffffffffu, wl, 12 + 2 * iy);
        y1 = __shfl_sync(0xffffffffu, wl, 13 + 2 * iy);
    }
    __device__ __forceinline__ size_t point(const MeshGeom& g, int col) const {
        const int ix = col / 6, iy = col - 6 * ix;
        return (size_t)(__shfl_sync(0xffffffffu, base, ix) + __shfl_sync(0xffffffffu, base, 6 + iy)) * g.K[2] + gz;
    }
};

// dipole (mu0, mu1, mu2) of atom `at` onto the mesh from the cached stencil, one warp
template <typename T>
__device__ __forceinline__ void spread_dip_atom(const MeshGeom& g, T* grid, const StencilCache<T>& st, int at, int lane,
                                                T mu0, T mu1, T mu2) {
    const double* B = g.B;
    const T c1 = -(T(B[0]) * mu0 + T(B[1]) * mu1 + T(B[2]) * mu2);
    const T c2 = -(T(B[3]) * mu0 + T(B[4]) * mu1 + T(B[5]) * mu2);
    const T c3 = -(T(B[6]) * mu0 + T(B[7]) * mu1 + T(B[8]) * mu2);
    const StencilLanes<T> sl(st, g, at, lane);
#pragma unroll
    for (int pass = 0; pass < 8; ++pass) {
        const int col = sl.column(pass);
        T x0, x1, y0, y1;
        sl.weights(col, x0, x1, y0, y1);
        const size_t k = sl.point(g, col);
        const T v = (c1 * x1 * y0 + c2 * x0 * y1) * sl.z0 + c3 * x0 * y0 * sl.z1;
        if (sl.has(pass)) atomicAdd(grid + k, v);
    }
}

// Scalars of the per-pass solve: r.u, its previous value, u.w, r.r, b.b, alpha, its previous value and
// the r.u that an update is adding up; behind them the solve's schedule: the steps begun, the next step
// before which the residual is read, the last one and its residual, whether the solve has stopped, and at
// which step.
enum { CGS_RU = 0, CGS_RU_PREV = 1, CGS_UW = 2, CGS_RR = 3, CGS_BB = 4, CGS_ALPHA = 5, CGS_ALPHA_PREV = 6, CGS_RU_NEW = 7,
       CGS_COUNT = 8, CGS_STEP = 8, CGS_NEXT = 9, CGS_LAST = 10, CGS_LAST_RMS = 11, CGS_DONE = 12, CGS_STOP = 13,
       CGS_WORDS = 14 };
constexpr int kCgCheckEvery = 4;  // steps between two reads of the residual, at most
constexpr int kCgHead = 31;       // steps queued before a solve's first read, at most

// steps from a read at `step`, with residual rms, to the next: kCgCheckEvery, or fewer where the decay since the
// last read (rms 0: none yet) says that the solve will have converged by then
__host__ __device__ inline int cg_segment(int step, double rms, int last, double last_rms, double goal) {
    if (!(last_rms > 0.0 && rms < last_rms && step > last)) return kCgCheckEvery;
    const double rate = pow(rms / last_rms, 1.0 / (double)(step - last));
    const double need = log(goal / rms) / log(rate);
    if (!(need > 0.0 && need < (double)kCgCheckEvery)) return kCgCheckEvery;
    const int k = (int)ceil(need);
    return k > 1 ? k : 1;
}

// What a step of the per-pass solve goes by: the scalars, the number of components and the relative
// tolerance.  every: the solve stops at the first step that has converged (as the persistent solve does), else at
// the first read that finds it converged.
struct CgSchedule {
    double* sc;
    double n3, tol;
    int every;
};

// A step begins (one thread, in the spread): the residual the last one left is read where a read is due, and
// the sums move on.  A solve that has converged stops here: r.u of 0 makes alpha and beta of its later steps 0
// (cg_coefs), which leave x, r and u as they are, so that steps queued without a read in between leave what a
// solve with every read leaves.
__device__ __noinline__ void cg_next(const CgSchedule& g) {
    double* sc = g.sc;
    const int step = (int)sc[CGS_STEP];
    const double rms = sqrt(sc[CGS_RR] / g.n3), goal = g.tol * sqrt(sc[CGS_BB] / g.n3);
    const bool read = step == (int)sc[CGS_NEXT];
    if (sc[CGS_DONE] != 0.0 || ((read || g.every) && rms <= goal)) {
        if (sc[CGS_DONE] == 0.0) sc[CGS_STOP] = step;
        sc[CGS_DONE] = 1.0;
        sc[CGS_RU] = 0.0;
    } else {
        if (read) {
            sc[CGS_NEXT] = step + cg_segment(step, rms, (int)sc[CGS_LAST], sc[CGS_LAST_RMS], goal);
            sc[CGS_LAST] = step;
            sc[CGS_LAST_RMS] = rms;
        }
        sc[CGS_STEP] = step + 1;
        sc[CGS_RU_PREV] = sc[CGS_RU];
        sc[CGS_RU] = sc[CGS_RU_NEW];
        sc[CGS_ALPHA_PREV] = sc[CGS_ALPHA];
    }
    sc[CGS_RU_NEW] = sc[CGS_RR] = sc[CGS_UW] = 0.0;
}

// sched: the solve whose step this spread begins (sc null: none); a CTA of its own in front does that
template <typename T>
__global__ void __launch_bounds__(256) k_spread_dip_cached(SpreadArgs<T> a, StencilCache<T> st, CgSchedule sched) {
    int cta = blockIdx.x;
    if (sched.sc && cta-- == 0) {
        if (threadIdx.x == 0) cg_next(sched);
        return;
    }
    const int warp = (cta * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= a.n) return;  // whole warps: every lane takes part in the shuffles
    const int at = (int)(((int64_t)warp * a.perm_mul) % a.n);
    spread_dip_atom<T>(a.g, a.grid, st, at, lane, (T)a.U[3 * at], (T)a.U[3 * at + 1], (T)a.U[3 * at + 2]);
}

// Field terms folded into the gather: out = recip [+ mv] [+ (1/pol + self1) U]; with dot_out, sum U . out
// is reduced into *dot_out.
struct FieldCombine {
    const double* mv = nullptr;  // real-space matvec field (may be null)
    const double* U = nullptr;  // dipoles of the diagonal term (null: no diagonal term)
    const double* pol = nullptr;
    double self1 = 0.0;
    double* dot_out = nullptr;
};

// k_gather_field with the cached stencil: one warp per atom, eight mesh loads per lane in flight, lanes
// 0..2 finish one component each.  Returns the lane's part of U_at . out_at when cmb.U is set.
template <typename T>
__device__ __forceinline__ double gather_field_atom(const StencilCache<T>& st, const MeshGeom& g, const T* phi,
                                                    double scale, double* out, const FieldCombine& cmb, int at,
                                                    int lane) {
    const StencilLanes<T> sl(st, g, at, lane);
    double u = 0.0, pp = 1.0, mv = 0.0;
    if (cmb.U && lane < 3) {  // read beside the mesh
        u = cmb.U[3 * at + lane];
        pp = cmb.pol[at];
        if (cmb.mv) mv = cmb.mv[3 * at + lane];
    }
    T v[8];
#pragma unroll
    for (int pass = 0; pass < 8; ++pass) {
        const int col = sl.column(pass);
        const size_t k = sl.point(g, col);
        v[pass] = sl.has(pass) ? phi[k] : T(0);
    }
    T s00 = T(0), s10 = T(0), s01 = T(0);
#pragma unroll
    for (int pass = 0; pass < 8; ++pass) {
        T x0, x1, y0, y1;
        sl.weights(sl.column(pass), x0, x1, y0, y1);
        const T t0 = v[pass] * y0, t1 = v[pass] * y1;
        s00 += x0 * t0;
        s10 += x1 * t0;
        s01 += x0 * t1;
    }
    T p1 = s10 * sl.z0, p2 = s01 * sl.z0, p3 = s00 * sl.z1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        p1 += __shfl_xor_sync(0xffffffffu, p1, o);
        p2 += __shfl_xor_sync(0xffffffffu, p2, o);
        p3 += __shfl_xor_sync(0xffffffffu, p3, o);
    }
    if (lane >= 3) return 0.0;
    const double* B = g.B;
    const double b1 = lane == 0 ? B[0] : (lane == 1 ? B[1] : B[2]), b2 = lane == 0 ? B[3] : (lane == 1 ? B[4] : B[5]),
                 b3 = lane == 0 ? B[6] : (lane == 1 ? B[7] : B[8]);
    double r = -(scale * (double)p1 * b1 + scale * (double)p2 * b2 + scale * (double)p3 * b3), d = 0.0;
    if (cmb.U) {
        pp = pp < 1e-8 ? 1e-8 : pp;
        r += (DMFFB_DIELECTRIC / pp + cmb.self1) * u + mv;
        d = u * r;
    }
    out[3 * at + lane] = r;
    return d;
}

// CTAs of a warp-per-atom kernel that ends in a block reduction: as many as fit the chip at `per_sm`,
// each warp taking the same number of atoms, so that a launch sends that many atomics to the sum
// instead of one per eight atoms (at 30000 atoms 3750 on one word).
inline unsigned atom_ctas(int n, int per_sm) {
    const int warps = 8 * 148 * per_sm, rounds = (n + warps - 1) / warps;
    return (unsigned)((n + 8 * rounds - 1) / (8 * rounds));
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 3) k_gather_field_cached(int n, StencilCache<T> st, MeshGeom g, const T* phi,
                                                             double scale, double* out, FieldCombine cmb) {
    const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
    double d[1] = {0.0};
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += nw)
        d[0] += gather_field_atom<T>(st, g, phi, scale, out, cmb, w, lane);
    if (cmb.dot_out) block_reduce_add<1>(d, cmb.dot_out);
}

}  // namespace dmffb
