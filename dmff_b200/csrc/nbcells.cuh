// Lennard-Jones + point-charge Coulomb over the cell grid, without a pair list.
//
// The engine's own neighbour list (dmff/common/nblist.py:27-55 semantics: every i < j whose
// minimum-image distance is < rc, nbond from the covalent map) is, for the classical terms,
// written once per step and read once by the pair kernel: at 100 000 atoms and rc 10 A that is
// 61 M rows, 0.74 GB out and back, plus j-side force atomics.  This pass evaluates the same pair
// set straight from the cell binning of the step's positions:
//   * one warp per atom i walks the forward half of the 5^3 stencil of half-width cells (the 62
//     offsets after (0, 0, 0) in lexicographic order, and in its own cell the atoms after it in
//     cell order), so every unordered pair is met once, as one concatenated candidate list, 32
//     candidates per batch, reading a cell-ordered float4 copy of the positions (contiguous runs
//     per cell, the atom index in the w slot); atoms are taken in cell order, so the warps of a
//     block share their candidates through L1 (with at least 5 cells per axis the 5 offsets of an
//     axis are distinct cells, and a box of at least 2.5 rc has one image of a pair within rc);
//   * stencil cells with no point within rc of the atom are skipped (per atom, from its position
//     in its cell);
//   * FP32 prefilter on float positions, the exact FP64 test of the list build (within_rc on the
//     lower/higher orientation) inside a 2e-3 A band around rc, so the kept set is the list's
//     set bit for bit;
//   * pairs with a topological scale (nbond != 0, a covalent partner whose index lies in the
//     atom's [cov_lo, cov_hi] range) are skipped here: an FP64 pass over the covalent rows
//     within rc evaluates them (k_nb_pair with a cut-off test);
//   * every other kept pair is queued in shared memory and evaluated 32 at a time (every lane
//     busy): nb_eval in kernel precision on the FP64 minimum-image vector and distance of
//     k_nb_pair; the force on i accumulates in lane registers (one warp sum and one reduction per
//     atom), the force on the partner goes out as one 16-byte reduction into its cell slot;
//   * the count of kept pairs (scaled ones included) is the list's row count.
// Energies and the box gradient accumulate per lane (about 20 pairs each) and meet in an FP64 block
// reduction.
#pragma once
#include "classical.cuh"
#include "nblist.cuh"

namespace dmffb {

// What a pair reads of a partner, one 32-byte load: the position as the caller gave it and, in w, the
// charge (FP32 engines: the float charge and the LJ type; FP64 engines: the charge).
struct __align__(32) NbRec {
    double x, y, z, w;
};

template <typename T>
struct NbCellArgs {
    int n;
    const double* pos;        // [3n] FP64 (borderline distance tests)
    const float4* posc;       // [n] FP32 x, y, z inside the box and the atom index (int bits), cell order
    Box boxd;
    double rc;
    int nc[3];                // half-width cells per axis (>= 5)
    double width[3];          // perpendicular widths of the box (the distance between the faces
                              // of constant fractional coordinate k)
    const int32_t* cell_start;
    const int32_t* atom_cell;  // [n]
    NbArgs cov;               // covalent-map lookup (cov_ptr / cov_j / cov_nb over i < j)
    const int32_t* cov_lo;    // [n] smallest / largest covalent partner index (lo > hi: none)
    const int32_t* cov_hi;
    const NbRec* rec;         // [n] in cell order: FP64 position, charge and (FP32) LJ type
    const int32_t* type;      // [n] LJ type or null
    int ntypes;
    const T* sig_tt;
    const T* eps_tt;
    T mc, ml;                 // scales of nbond 0 (the trailing 1.0 entries)
    T kappa, krf, crf;
    int coul;
    T* gcell;                 // [n][4] dE/dpos in cell order
    double* scal;             // [0] E_coul, [1] E_lj, [2..10] box gradient, [11] pairs i < j within rc
};

__device__ __forceinline__ void nb_rec_get(const NbRec& r, float& q, int& type) {
    const long long b = __double_as_longlong(r.w);
    q = __int_as_float((int)b);
    type = (int)(b >> 32);
}
__device__ __forceinline__ void nb_rec_get(const NbRec& r, double& q, int&) { q = r.w; }

// the records of the cell order, and the cell-ordered gradients cleared
template <typename T>
__global__ void k_nb_records(int n, const float4* posc, const double* pos, const T* qT, const int32_t* type, NbRec* rec,
                             T* gcell) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = __float_as_int(posc[k].w);
    NbRec r;
    r.x = pos[3 * i];
    r.y = pos[3 * i + 1];
    r.z = pos[3 * i + 2];
    if (sizeof(T) == 4)
        r.w = __longlong_as_double((long long)(unsigned)__float_as_int((float)qT[i]) |
                                   ((long long)(type ? type[i] : 0) << 32));
    else
        r.w = (double)qT[i];
    rec[k] = r;
#pragma unroll
    for (int c = 0; c < 4; ++c) gcell[4 * (int64_t)k + c] = T(0);
}

// forces of the cell pass: -(reciprocal and bonded + scaled rows + cell order)
template <typename T>
__global__ void k_nb_forces(int n, const T* glr, const double* gd, const T* gcell, const int32_t* cell_start,
                            const int32_t* atom_cell, const int32_t* rank, double* forces) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T* g = gcell + 4 * (int64_t)(cell_start[atom_cell[i]] + rank[i]);
#pragma unroll
    for (int c = 0; c < 3; ++c) forces[3 * i + c] = -((double)glr[3 * i + c] + (double)g[c] + gd[3 * i + c]);
}

// distance of an FP64 square in kernel precision: FP32 from the hardware's reciprocal square root and
// one FP64 Newton step (error 1e-14, so it rounds to the same float as the FP64 root all but always)
__device__ __forceinline__ void nb_root(double r2, double& r) { r = sqrt(r2); }
__device__ __forceinline__ void nb_root(double r2, float& r) {
    const double y = (double)rsqrtf((float)r2);
    const double q = r2 * y;
    r = (float)fma(0.5 * y, fma(-q, q, r2), q);
}

// One kept pair (i, the atom in cell slot k), met once: energy, box gradient, the force on i
// (registers) and on the partner (a reduction into its slot).
template <typename T, bool ORTHO>
__device__ __forceinline__ void nb_cell_pair(const NbCellArgs<T>& a, int k, double xi, double yi, double zi, bool lj,
                                             int ti, T qi, T& g0, T& g1, T& g2, T (&acc)[11]) {
    const NbRec rj = a.rec[k];
    // the pair geometry of k_nb_pair: FP64 minimum image, then kernel precision
    T e[3], r;
    double dr[3] = {rj.x - xi, rj.y - yi, rj.z - zi}, nd[3];
    if (ORTHO) {  // pbc_shift without the products with zero
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double t = dr[c] * a.boxd.hinv[4 * c];
            nd[c] = floor(t + 0.5);
            dr[c] = (t - nd[c]) * a.boxd.h[4 * c];
        }
    } else {
        BoxT<double> bx;
#pragma unroll
        for (int c = 0; c < 9; ++c) { bx.h[c] = a.boxd.h[c]; bx.hinv[c] = a.boxd.hinv[c]; }
        pbc_shift(bx, dr[0], dr[1], dr[2], nd);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) e[c] = (T)dr[c];
    nb_root(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2], r);
    T qj;
    int tj = 0;
    nb_rec_get(rj, qj, tj);
    int tp = 0;
    if (lj) {
        if (sizeof(T) == 8) tj = a.type[__float_as_int(a.posc[k].w)];
        tp = ti * a.ntypes + tj;
    }
    T ec, dec, phi, el, del, ds, dp;
    nb_eval<T>(r, qi * qj, a.mc, a.ml, lj ? a.sig_tt[tp] : T(0), lj ? a.eps_tt[tp] : T(0), lj, a.coul, a.kappa,
               a.krf, a.crf, ec, dec, phi, el, del, ds, dp);
    // e = r_j - r_i (minimum image); dE/dr_i = -(dE/dr / r) e; image counts of r_i - r_j are -nd
    const T s = (dec + del) / r;
    const T f0 = s * e[0], f1 = s * e[1], f2 = s * e[2];
    g0 -= f0;
    g1 -= f1;
    g2 -= f2;
    add3(a.gcell + 4 * (int64_t)k, f0, f1, f2);
    acc[0] += ec;
    acc[1] += el;
    if (nd[0] != 0.0 || nd[1] != 0.0 || nd[2] != 0.0) {  // most pairs meet inside the box
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const T nn = (T)nd[q];
            acc[2 + 3 * q] -= nn * f0;
            acc[3 + 3 * q] -= nn * f1;
            acc[4 + 3 * q] -= nn * f2;
        }
    }
}

// Bound by instruction issue (FP64 minimum image, erfc / exp, the candidate test): 607 us for the 20.8 M
// pairs of 99000 atoms at rc 10 A.  Scalar reductions into [3n], three FP64 gathers plus charge
// and type per partner, FP64 division in the cell pruning and a full FP64 root took it to 822 us.
template <typename T, bool ORTHO>
__global__ void __launch_bounds__(32 * kNbWarps, sizeof(T) == 4 ? 4 : 0) k_nb_cells(NbCellArgs<T> a) {
    constexpr int S = 2, W = 2 * S + 1, NQ = (W * W * W + 1) / 2;  // offsets q0 = 62 .. 124 of the 5^3 stencil
    __shared__ int s_beg[kNbWarps][NQ];
    __shared__ int s_off[kNbWarps][NQ + 1];
    __shared__ int s_q[kNbWarps][64];  // kept candidates (cell slots) waiting for a full 32-lane batch
    const int wl = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // warps take the atoms in cell order: the warps of a block share one stencil, so their
    // candidate reads (contiguous runs of the cell-ordered copy) hit L1 after the first
    const int ks = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const bool live = ks < a.n;  // warps past the end still take part in the block reduction
    double red[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) red[k] = 0.0;
    if (live) {
        const float4 p4 = a.posc[ks];
        const int i = __float_as_int(p4.w);
        const NbRec ri = a.rec[ks];
        float hf[9], hif[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) { hf[k] = (float)a.boxd.h[k]; hif[k] = (float)a.boxd.hinv[k]; }
        const float rlo = (float)(a.rc - 2e-3), rhi = (float)(a.rc + 2e-3);
        const float rlo2 = rlo * rlo, rhi2 = rhi * rhi;
        // The atom's cell (from the binning) and its position in it, in cell units.  A stencil cell none of
        // whose points lies within rc + 0.01 A of the atom is skipped (about a third of the forward
        // half for half-width cells).  Orthorhombic boxes: the exact distance to the cell's box;
        // others the lower bound max_k gap_k width_k (gap_k the fractional gap along k).  The margin
        // covers the FP32 prefilter band (rc +- 2e-3 A) and the rounding of the binning and of
        // the FP32 gaps, so the kept pairs are unchanged.
        const int ac = a.atom_cell[i];
        const int c3[3] = {ac / (a.nc[2] * a.nc[1]), (ac / a.nc[2]) % a.nc[1], ac % a.nc[2]};
        float u[3], cw[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double v = ri.x * a.boxd.hinv[k] + ri.y * a.boxd.hinv[3 + k] + ri.z * a.boxd.hinv[6 + k];
            v = (v - floor(v)) * a.nc[k];
            u[k] = (float)(v - c3[k]);
            cw[k] = (float)(a.width[k] / a.nc[k]);
        }
        const float rprune = (float)(a.rc + 0.01);
        int carry = 0;
        if (lane == 0) s_off[wl][0] = 0;
        for (int q0 = 0; q0 < NQ; q0 += 32) {
            const int q = q0 + lane;
            int cnt = 0;
            if (q < NQ) {
                const int qq = q + NQ - 1;  // (0, 0, 0) and the offsets after it
                const int dd[3] = {qq / (W * W) - S, (qq / W) % W - S, qq % W - S};
                int cc = 0;
                float d2 = 0.f, dmax = 0.f;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    int ck = c3[k] + dd[k];
                    ck += ck < 0 ? a.nc[k] : (ck >= a.nc[k] ? -a.nc[k] : 0);
                    cc = cc * a.nc[k] + ck;
                    const float gap = fmaxf(0.f, fmaxf(dd[k] - u[k], u[k] - (dd[k] + 1))) * cw[k];
                    d2 += gap * gap;
                    dmax = fmaxf(dmax, gap);
                }
                int cs = a.cell_start[cc];
                const int ce = a.cell_start[cc + 1];
                if (q == 0) cs = max(cs, ks + 1);  // own cell: the atoms after i in cell order
                cnt = max(ce - cs, 0);
                if (q > 0 && (ORTHO ? d2 > rprune * rprune : dmax > rprune)) cnt = 0;
                s_beg[wl][q] = cs;
            }
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (q < NQ) s_off[wl][q + 1] = carry + incl;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        const int total = carry;
        const int lo = a.cov_lo[i], hi = a.cov_hi[i];
        const bool lj = a.type != nullptr;
        T qi;
        int ti = 0;
        nb_rec_get(ri, qi, ti);
        if (sizeof(T) == 8 && lj) ti = a.type[i];
        T g0 = T(0), g1 = T(0), g2 = T(0);
        T acc[11];  // per-lane sums of about 40 pairs, in kernel precision
#pragma unroll
        for (int k = 0; k < 11; ++k) acc[k] = T(0);
        int npair = 0;
        const unsigned lt = (1u << lane) - 1u;
        int qn = 0;  // queued kept candidates (warp-uniform)
        int qc = 0;
        for (int base = 0; base < total; base += 32) {
            const int t = base + lane;
            bool keep = false;
            int slot = 0, j = -1;
            if (t < total) {
                while (t >= s_off[wl][qc + 1]) ++qc;
                slot = s_beg[wl][qc] + (t - s_off[wl][qc]);
                const float4 pj = a.posc[slot];
                j = __float_as_int(pj.w);
                const float d0 = pj.x - p4.x, d1 = pj.y - p4.y, d2 = pj.z - p4.z;
                bool amb = false;
                float r2;
                if (ORTHO) {
                    const float dd[3] = {d0, d1, d2};
                    r2 = 0.f;
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        const float tt = dd[q] * hif[4 * q];
                        const float sq = tt - floorf(tt + 0.5f);
                        amb |= fabsf(sq) > 0.4999f;
                        const float ev = sq * hf[4 * q];
                        r2 = fmaf(ev, ev, r2);
                    }
                } else {
                    float sf[3];
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        const float tt = d0 * hif[q] + d1 * hif[3 + q] + d2 * hif[6 + q];
                        sf[q] = tt - floorf(tt + 0.5f);
                        amb |= fabsf(sf[q]) > 0.4999f;
                    }
                    const float e0 = sf[0] * hf[0] + sf[1] * hf[3] + sf[2] * hf[6];
                    const float e1 = sf[0] * hf[1] + sf[1] * hf[4] + sf[2] * hf[7];
                    const float e2 = sf[0] * hf[2] + sf[1] * hf[5] + sf[2] * hf[8];
                    r2 = e0 * e0 + e1 * e1 + e2 * e2;
                }
                if (!amb && r2 < rlo2) keep = true;
                else if (!amb && r2 > rhi2) keep = false;
                else keep = j > i ? within_rc(a.boxd, a.pos + 3 * i, a.pos + 3 * j, a.rc)
                                  : within_rc(a.boxd, a.pos + 3 * j, a.pos + 3 * i, a.rc);
            }
            if (keep) ++npair;
            // topologically scaled pairs belong to the FP64 covalent pass
            if (keep && j >= lo && j <= hi) {
                const int nbd = j > i ? lookup_nbond(a.cov, i, j) : lookup_nbond(a.cov, j, i);
                if (nbd != 0) keep = false;
            }
            // queue the kept candidates; evaluate them 32 at a time with every lane busy
            const unsigned mk = __ballot_sync(0xffffffffu, keep);
            if (keep) s_q[wl][qn + __popc(mk & lt)] = slot;
            qn += __popc(mk);
            __syncwarp();
            if (qn >= 32) {
                nb_cell_pair<T, ORTHO>(a, s_q[wl][lane], ri.x, ri.y, ri.z, lj, ti, qi, g0, g1, g2, acc);
                __syncwarp();
                if (lane < qn - 32) s_q[wl][lane] = s_q[wl][32 + lane];
                qn -= 32;
                __syncwarp();
            }
        }
        if (lane < qn)
            nb_cell_pair<T, ORTHO>(a, s_q[wl][lane], ri.x, ri.y, ri.z, lj, ti, qi, g0, g1, g2, acc);
#pragma unroll
        for (int k = 0; k < 11; ++k) red[k] = (double)acc[k];
        red[11] = (double)npair;
        __syncwarp();
        g0 = warp_sum(g0);
        g1 = warp_sum(g1);
        g2 = warp_sum(g2);
        if (lane == 0) add3(a.gcell + 4 * (int64_t)ks, g0, g1, g2);
    }
    block_reduce_add<12>(red, a.scal);
}

}  // namespace dmffb
