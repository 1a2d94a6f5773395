// The whole induced-dipole CG solve in one persistent cooperative launch (FP32 engines, meshes that
// the direct DFT convolution serves).
//
// The dipole solve of the reference (pme.py:342-423 solves A U = -E_perm by fixed-point steps;
// the engine uses preconditioned CG on the same linear system) repeats, per iteration, a chain of
// dependent passes on data that sits in L2: vector update and dipole spread, 3-D transform, influence
// multiply, inverse transform, field gather, with the real-space matvec beside them.  CG is taken in
// its form with one synchronisation per iteration (Chronopoulos and Gear 1989: w = A u of the
// preconditioned residual u gives gamma = r.u and delta = u.w, from which alpha and beta follow, and
// s = A p is carried along as s = w + beta s), so that the update of an atom's vectors is local to the
// warp that spreads it and the real-space matvec can share the pass of the gather.  Launched one
// kernel per pass, a small box spends most of an iteration in launch gaps and host round trips.
// Here one cooperative grid runs every iteration and decides convergence on the device; the passes
// are separated by a grid barrier:
//   B  p = u + beta p, s = w + beta s, x += alpha p, r -= alpha s, u = M r, u onto the mesh; r.u, r.r
//   C  forward x-plane DFT passes        D  spectrum columns (x DFT, * G, inverse x DFT)
//   E  inverse x-plane DFT passes        F  real-space matvec, field gather and diagonal (w = A u), u.w
// (with phase_ns set, block 0 adds the device-clock time of each pass, barrier included)
// Measured per iteration at 450 / 3999 / 12288 atoms, seven passes and classic CG before: 26 / 35 / 62 us,
// these five passes 22 / 32 / 61.
//
// The three sums of iteration k (u.w, r.u, r.r) accumulate in slot k mod 4 of acc[4][4] and are read
// after the barriers of iteration k; slot k + 1 is cleared in pass C of iteration k, three
// iterations after its last reads.
//
// The grid barrier is an arrival counter and a generation word (release on arrival, acquire on
// the wait).  Every wait is bounded by the device clock: past `wait_ns` the CTA records
// DMFFB_CG_TIMEOUT in the status word and leaves; the others leave at their next barrier (which
// can no longer complete, so their own waits run out as well), and the host reads the status.
#pragma once
#include <cuda/atomic>

#include "admp_dftconv.cuh"
#include "admp_real.cuh"
#include "admp_recip.cuh"
#include "common.cuh"

namespace dmffb {

constexpr int kCgThreads = 512;  // 1024 (64 registers, spills) takes 28 us per iteration at 450 atoms against 22
constexpr int DMFFB_CG_TIMEOUT = 1;    // a grid barrier wait ran out
constexpr int DMFFB_CG_NONFINITE = 2;  // non-finite residual

struct CgBarrier {
    unsigned* count;  // arrivals of the current generation
    unsigned* gen;    // generation
    int* status;      // 0, or DMFFB_CG_* of the first failure
    long long wait_ns;
    unsigned phantom;  // arrivals expected beyond the grid's CTAs (0; a test sets 1 to make waits run out)
};

struct CgStatus {
    int iters;
    int converged;
    int status;
    int pad;
    double rr;  // r . r at exit
};

__device__ __forceinline__ long long cg_clock_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// grid-wide barrier of nblocks co-resident CTAs; false when this CTA must leave (a wait ran out
// here or a failure was recorded anywhere)
__device__ inline bool cg_grid_sync(const CgBarrier& b, unsigned nblocks) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> cnt(*b.count), gen(*b.gen);
        cuda::atomic_ref<int, cuda::thread_scope_device> st(*b.status);
        const unsigned g = gen.load(cuda::memory_order_relaxed);
        int ok = 1;
        if (cnt.fetch_add(1u, cuda::memory_order_acq_rel) == nblocks + b.phantom - 1) {
            cnt.store(0u, cuda::memory_order_relaxed);
            gen.store(g + 1u, cuda::memory_order_release);
        } else {
            long long t0 = 0;
            for (unsigned poll = 1; gen.load(cuda::memory_order_acquire) == g; ++poll) {
                if (poll & 63u) continue;
                const long long now = cg_clock_ns();
                if (t0 == 0) t0 = now;
                if (st.load(cuda::memory_order_relaxed) != 0 || now - t0 > b.wait_ns) {
                    int expect = 0;
                    st.compare_exchange_strong(expect, DMFFB_CG_TIMEOUT, cuda::memory_order_relaxed);
                    ok = 0;
                    break;
                }
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// The vectors of the single-synchronisation CG, FP64 [3n]: solution, residual, u = M r, direction p and
// s = A p; w = A u, in two parts (reciprocal + diagonal, real space) or whole in Ap (fmv null).
struct CgVectors {
    double *x, *r, *u, *p, *s;
    const double *Ap, *fmv;
    const double* pol;  // [n]
};

// alpha and beta of an iteration from its sums and the previous ones (0: first iteration)
__device__ __forceinline__ void cg_coefs(double gamma, double gamma_prev, double delta, double alpha_prev, double& alpha,
                                         double& beta) {
    beta = gamma_prev != 0.0 ? gamma / gamma_prev : 0.0;
    const double den = delta - (alpha_prev != 0.0 ? beta * gamma / alpha_prev : 0.0);
    alpha = den != 0.0 ? gamma / den : 0.0;
}

// The vector update of component c of atom `at`: leaves u and its copy in kernel precision, adds to the
// sums r.u and r.r, returns u.  The first iteration (beta 0) does not read p and s.
template <typename T>
__device__ __forceinline__ double cg_update(const CgVectors& v, Vec4<T>* p4, double alpha, double beta, int at, int c,
                                            double& ru, double& rr) {
    const int k = 3 * at + c;
    double pp = v.pol[at];
    pp = pp < 1e-8 ? 1e-8 : pp;
    const double w = v.fmv ? v.Ap[k] + v.fmv[k] : v.Ap[k];
    const double p = beta != 0.0 ? v.u[k] + beta * v.p[k] : v.u[k];
    const double s = beta != 0.0 ? w + beta * v.s[k] : w;
    const double r = v.r[k] - alpha * s, u = r * pp / DMFFB_DIELECTRIC;
    v.p[k] = p;
    v.s[k] = s;
    v.x[k] += alpha * p;
    v.r[k] = r;
    v.u[k] = u;
    ((T*)(p4 + at))[c] = (T)u;
    ru += r * u;
    rr += r * r;
    return u;
}

// The per-pass solve's vector update, one thread per component.  Folding the next spread into it, a warp
// per atom, took 16 us at 12288 atoms and 30 at 30000 against 3 + 7.5 and 3.5 + 15.5 for the two
// launches: three lanes of a warp wait for the vectors where here all threads do.
template <typename T>
__global__ void __launch_bounds__(256) k_cg_update1(int n, CgVectors v, Vec4<T>* p4, double* sc) {
    double alpha, beta;
    cg_coefs(sc[CGS_RU], sc[CGS_RU_PREV], sc[CGS_UW], sc[CGS_ALPHA_PREV], alpha, beta);
    double sum[2] = {0.0, 0.0}, rr[1];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < 3 * n) cg_update<T>(v, p4, alpha, beta, k / 3, k % 3, sum[0], sum[1]);
    if (k == 0) sc[CGS_ALPHA] = alpha;
    rr[0] = sum[1];
    double ru[1] = {sum[0]};
    block_reduce_add<1>(ru, sc + CGS_RU_NEW);
    block_reduce_add<1>(rr, sc + CGS_RR);
}

struct CgSolveArgs {
    int n;
    CgVectors v;
    double *Ap, *fmv;  // the two parts of w
    // real-space matvec
    CsrArgs csr;
    const MvCoef<float>* coef;
    Vec4<float>* p4;  // [n] u in FP32
    // spread / gather
    StencilCache<float> st;
    MeshGeom g;
    int perm_mul;
    double gscale;  // 2 * DIELECTRIC
    double self1;
    // convolution (grid_in: the spread mesh, grid_out: the convolved mesh)
    DftConvArgs<float> fc;
    // scalars
    double* acc;         // [4][4] {u.w, r.u, r.r, -}, zero at launch
    const double* init;  // CGS_RU_NEW, CGS_RR and CGS_BB of the initial residual
    double tol;
    int max_iter;
    CgBarrier bar;
    CgStatus* out;
    unsigned long long* phase_ns;  // [8] time per pass summed over the iterations (block 0), or null
};

// elements of the largest working area of the convolution passes
__host__ __device__ inline size_t cg_work_elems(const DftConvArgs<float>& a) {
    const size_t f = dft_fwd_elems(a), c = dft_col_elems(a), i = dft_inv_elems(a);
    const size_t m = f > c ? (f > i ? f : i) : (c > i ? c : i);
    return (m + 3) & ~(size_t)3;
}

__global__ void __launch_bounds__(kCgThreads) k_cg_solve(CgSolveArgs a) {
    extern __shared__ __align__(16) unsigned char dft_sm[];
    float* const sm = (float*)dft_sm;
    // the DFT matrices stay in shared memory for the whole solve
    float* const wx = sm + cg_work_elems(a.fc);
    float* const wy = wx + dft_mat_elems(a.fc.H[0]);
    float* const wz = wy + dft_mat_elems(a.fc.H[1]);
    dft_load_mat(a.fc, 0, wx);
    dft_load_mat(a.fc, 1, wy);
    dft_load_mat(a.fc, 2, wz);
    const unsigned nb = gridDim.x;
    const int tid = threadIdx.x, nth = blockDim.x;
    const int lane = tid & 31;
    const int warps_cta = nth >> 5;
    const int gwarp = blockIdx.x * warps_cta + (tid >> 5), nwarps = nb * warps_cta;
    const int m3 = 3 * a.n;
    FieldCombine cmb;
    cmb.U = a.v.u;
    cmb.pol = a.v.pol;
    cmb.self1 = a.self1;
    const double rms_b = sqrt(a.init[CGS_BB] / (double)m3);
    double rr = a.init[CGS_RR];
    int it = 0, conv = 0, status = 0;
    double ru = a.init[CGS_RU_NEW], ru_prev = 0.0, alpha_prev = 0.0;
    const int nfwd = dft_fwd_items(a.fc), ncol = dft_col_items(a.fc), ninv = dft_inv_items(a.fc);
    const int K3 = a.fc.K[0] * a.fc.K[1] * a.fc.K[2];
    // pass timing on block 0 (device clock at each barrier exit)
    const bool timed = a.phase_ns && blockIdx.x == 0 && tid == 0;
    long long tp = timed ? cg_clock_ns() : 0;
    auto mark = [&](int ph) {
        if (timed) {
            const long long t = cg_clock_ns();
            a.phase_ns[ph] += (unsigned long long)(t - tp);
            tp = t;
        }
    };
    // the initial u onto the mesh
    for (int w = gwarp; w < a.n; w += nwarps) {
        const int at = (int)(((int64_t)w * a.perm_mul) % a.n);
        spread_dip_atom<float>(a.g, a.fc.zero_real, a.st, at, lane, (float)a.v.u[3 * at], (float)a.v.u[3 * at + 1],
                               (float)a.v.u[3 * at + 2]);
    }
    bool ok = cg_grid_sync(a.bar, nb);
    mark(1);
    while (ok) {
        const double rms = sqrt(rr / (double)m3);
        if (!isfinite(rms)) {
            status = DMFFB_CG_NONFINITE;
            break;
        }
        if (rms <= a.tol * rms_b) {
            conv = 1;
            break;
        }
        if (it >= a.max_iter) break;
        double* acc = a.acc + 4 * (it & 3);
        if (blockIdx.x == 0 && tid < 4) a.acc[4 * ((it + 1) & 3) + tid] = 0.0;
        // C, D, E: the convolution
        for (int w = blockIdx.x; w < nfwd; w += nb) {
            dft_fwd_item<float, 1, 1>(a.fc, w, sm, wy, wz);
            __syncthreads();
        }
        if (!cg_grid_sync(a.bar, nb)) break;
        mark(2);
        {
            double none[7];  // no energy sums in the solve
            for (int w = blockIdx.x; w < ncol; w += nb) {
                dft_col_item<float, 1, 1, true>(a.fc, w, sm, wx, none);
                __syncthreads();
            }
            for (int k = blockIdx.x * nth + tid; k < K3; k += nb * nth) a.fc.zero_real[k] = 0.f;
        }
        if (!cg_grid_sync(a.bar, nb)) break;
        mark(3);
        for (int w = blockIdx.x; w < ninv; w += nb) {
            dft_inv_item<float, 1, 1>(a.fc, w, sm, wy, wz);
            __syncthreads();
        }
        if (!cg_grid_sync(a.bar, nb)) break;
        mark(4);
        // F: real-space matvec and field gather, Ap = recip field of u + (1/pol + self) u
        {
            double uw[1] = {0.0};
            for (int w = gwarp; w < 2 * a.n; w += nwarps)
                uw[0] += w < a.n ? matvec_atom<float>(a.csr, a.coef, a.p4, a.v.u, a.fmv, w, lane)
                                 : gather_field_atom<float>(a.st, a.g, a.fc.grid_out, a.gscale, a.Ap, cmb, w - a.n, lane);
            block_reduce_add<1>(uw, acc);
        }
        if (!cg_grid_sync(a.bar, nb)) break;
        mark(5);
        // B: update and spread
        double alpha, beta;
        cg_coefs(ru, ru_prev, acc[0], alpha_prev, alpha, beta);
        {
            double sum[2] = {0.0, 0.0};
            for (int w = gwarp; w < a.n; w += nwarps) {
                const int at = (int)(((int64_t)w * a.perm_mul) % a.n);
                const float u =
                    lane < 3 ? (float)cg_update<float>(a.v, a.p4, alpha, beta, at, lane, sum[0], sum[1]) : 0.f;
                spread_dip_atom<float>(a.g, a.fc.zero_real, a.st, at, lane, __shfl_sync(0xffffffffu, u, 0),
                                       __shfl_sync(0xffffffffu, u, 1), __shfl_sync(0xffffffffu, u, 2));
            }
            block_reduce_add<2>(sum, acc + 1);
        }
        if (!cg_grid_sync(a.bar, nb)) break;
        mark(1);
        ru_prev = ru;
        alpha_prev = alpha;
        ru = acc[1];
        rr = acc[2];
        ++it;
    }
    if (blockIdx.x == 0 && tid == 0) {
        cuda::atomic_ref<int, cuda::thread_scope_device> st(*a.bar.status);
        const int bst = st.load(cuda::memory_order_acquire);
        a.out->iters = it;
        a.out->converged = conv;
        a.out->status = bst != 0 ? bst : status;
        a.out->rr = rr;
    }
}

// dynamic shared memory of k_cg_solve: the convolution passes' working area and the DFT matrices
__host__ inline size_t cg_solve_smem(const DftConvArgs<float>& a) {
    return sizeof(float) * (cg_work_elems(a) + dft_mat_elems(a.H[0]) + dft_mat_elems(a.H[1]) + dft_mat_elems(a.H[2]));
}

}  // namespace dmffb
