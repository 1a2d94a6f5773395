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
//     candidates per batch, reading a cell-ordered float4 copy of the positions (a contiguous run
//     per z column of cells, two where it wraps, seen from the image the column wraps to, which is the
//     nearest one for every pair within rc; the atom index in the w slot); atoms are taken in cell order, so the warps of a
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
// Energies accumulate per lane (about seven pairs each), the box gradient per lane in FP64; they meet in
// an FP64 block reduction.
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

// One kept pair (i, the atom in cell slot k), met once: energy, box gradient (the lane's FP64 sums
// box[0], box[32], ...), the force on i (registers) and on the partner (a reduction into its slot).
template <typename T, bool ORTHO>
__device__ __forceinline__ void nb_cell_pair(const NbCellArgs<T>& a, int k, double xi, double yi, double zi, bool lj,
                                             int ti, T qi, T& g0, T& g1, T& g2, T (&acc)[2], double* box) {
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
    r = (T)sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
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
            box[32 * (3 * q)] -= nd[q] * (double)f0;
            box[32 * (3 * q + 1)] -= nd[q] * (double)f1;
            box[32 * (3 * q + 2)] -= nd[q] * (double)f2;
        }
    }
}

// Bound by instruction issue (FP64 minimum image, erf / exp; 73 % of the issue slots): 486 us for
// the 20.8 M pairs of 99000 atoms at rc 10 A, FP64 root included (479 with a reciprocal root and one Newton
// step, good to 1e-14, in its place).  Before: with a minimum image per candidate, 63 cells per
// atom searched and pruned one by one and FP32 box sums in registers 563; with scalar reductions into
// [3n], three FP64 gathers plus charge and type per partner and FP64 division in the pruning 822.
template <typename T, bool ORTHO>
__global__ void __launch_bounds__(32 * kNbWarps, sizeof(T) == 4 ? 4 : 0) k_nb_cells(NbCellArgs<T> a) {
    constexpr int NC = 13, NR = 2 * NC;  // forward columns of the 5^3 stencil, runs
    __shared__ int s_beg[kNbWarps][NR], s_off[kNbWarps][NR + 1], s_img[kNbWarps][NR];
    __shared__ float s_shift[18][3];  // lattice vectors a column can wrap by: 9 nx + 3 (ny + 1) + nz + 1
    __shared__ double s_box[kNbWarps][9][32];  // the lanes' box gradients: in FP64, and few pairs cross the box
    __shared__ int s_q[kNbWarps][64];  // kept candidates (cell slots) waiting for a full 32-lane batch
    const int wl = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    // warps take the atoms in cell order: the warps of a block share one stencil, so their
    // candidate reads (contiguous runs of the cell-ordered copy) hit L1 after the first
    const int ks = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const bool live = ks < a.n;  // warps past the end still take part in the block reduction
    if (threadIdx.x < 18) {
        const int t = threadIdx.x, nx = t / 9, ny = (t / 3) % 3 - 1, nz = t % 3 - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            s_shift[t][c] = (float)(nx * a.boxd.h[c] + ny * a.boxd.h[3 + c] + nz * a.boxd.h[6 + c]);
    }
    __syncthreads();
    double red[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) red[k] = 0.0;
    if (live) {
        const float4 p4 = a.posc[ks];
        const int i = __float_as_int(p4.w);
        const NbRec ri = a.rec[ks];
        const NbFilter f(a.cov);
        // The atom's cell (from the binning) and its position in it, in cell units.  A lane takes one of
        // the 13 columns (dx, dy) whose cells follow the atom's in lexicographic order and cuts its z range
        // to the cells with a point within rc + 0.01 A of the atom.  Orthorhombic boxes: by the exact
        // distance to the cell's box; others by the lower bound max_k gap_k width_k (gap_k the
        // fractional gap along k).  The margin covers the FP32 prefilter band and the rounding of the
        // binning and of the FP32 gaps, so the kept pairs are unchanged.
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
        int cnt[2] = {0, 0}, beg[2] = {0, 0}, img = 0, nz = 0;
        if (lane < NC) {
            const int dx = lane < 3 ? 0 : 1 + (lane - 3) / 5, dy = lane < 3 ? lane : (lane - 3) % 5 - 2;
            const float gx = fmaxf(0.f, dx - u[0]) * cw[0];
            const float gy = fmaxf(0.f, fmaxf(dy - u[1], u[1] - (dy + 1))) * cw[1];
            const float rest = ORTHO ? rprune * rprune - gx * gx - gy * gy : rprune - fmaxf(gx, gy);
            if (rest >= 0.f) {
                const float reach = (ORTHO ? sqrtf(rest) : rprune) / cw[2];  // in cells
                const int up = min(2, (int)floorf(u[2] + reach));
                const int dn = lane == 0 ? 0 : max(-2, (int)ceilf(u[2] - 1.f - reach));
                int x = c3[0] + dx, y = c3[1] + dy;
                const int nx = x >= a.nc[0] ? 1 : 0, ny = y < 0 ? -1 : (y >= a.nc[1] ? 1 : 0);
                x -= nx * a.nc[0];
                y -= ny * a.nc[1];
                const int* col = a.cell_start + (x * a.nc[1] + y) * a.nc[2];
                const int zb = c3[2] + dn, ze = c3[2] + up;
                const int z0 = max(zb, 0), z1 = min(ze, a.nc[2] - 1);
                nz = zb < 0 ? -1 : (ze >= a.nc[2] ? 1 : 0);
                beg[0] = lane == 0 ? ks + 1 : col[z0];  // own column: the atoms after i in cell order
                cnt[0] = max(col[z1 + 1] - beg[0], 0);
                if (nz) {
                    const int w0 = nz < 0 ? zb + a.nc[2] : 0, w1 = nz < 0 ? a.nc[2] - 1 : ze - a.nc[2];
                    beg[1] = col[w0];
                    cnt[1] = col[w1 + 1] - beg[1];
                }
                img = 9 * nx + 3 * (ny + 1) + 1;
            }
        }
        int incl = cnt[0] + cnt[1];
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane < NC) {
            s_beg[wl][2 * lane] = beg[0];
            s_beg[wl][2 * lane + 1] = beg[1];
            s_img[wl][2 * lane] = img;
            s_img[wl][2 * lane + 1] = img + nz;
            s_off[wl][2 * lane] = incl - cnt[0] - cnt[1];
            s_off[wl][2 * lane + 1] = incl - cnt[1];
            if (lane == NC - 1) s_off[wl][NR] = incl;
        }
        __syncwarp();
        const int total = s_off[wl][NR];
        const int lo = a.cov_lo[i], hi = a.cov_hi[i];
        const bool lj = a.type != nullptr;
        T qi;
        int ti = 0;
        nb_rec_get(ri, qi, ti);
        if (sizeof(T) == 8 && lj) ti = a.type[i];
        T g0 = T(0), g1 = T(0), g2 = T(0);
        T acc[2] = {T(0), T(0)};  // per-lane energies of about seven pairs, in kernel precision
        double* const box = &s_box[wl][0][lane];
#pragma unroll
        for (int k = 0; k < 9; ++k) box[32 * k] = 0.0;
        int npair = 0;
        const unsigned lt = (1u << lane) - 1u;
        int qn = 0;  // queued kept candidates (warp-uniform)
        // the lane's run: its end, the slot of candidate 0 and the atom seen from the run's image
        int run = -1, end = 0, first = 0;
        float bx = 0.f, by = 0.f, bz = 0.f;
        for (int base = 0; base < total; base += 32) {
            const int t = base + lane;
            bool keep = false;
            int slot = 0, j = -1;
            if (t < total) {
                if (t >= end) {
                    do end = s_off[wl][++run + 1];
                    while (t >= end);
                    first = s_beg[wl][run] - s_off[wl][run];
                    const float* sh = s_shift[s_img[wl][run]];
                    bx = p4.x - sh[0];
                    by = p4.y - sh[1];
                    bz = p4.z - sh[2];
                }
                slot = first + t;
                const float4 pj = a.posc[slot];
                j = __float_as_int(pj.w);
                const float dx = pj.x - bx, dy = pj.y - by, dz = pj.z - bz;
                const float r2 = dx * dx + dy * dy + dz * dz;
                if (r2 < f.rlo2) keep = true;
                else if (r2 <= f.rhi2) keep = j > i ? within_rc(a.boxd, a.pos + 3 * i, a.pos + 3 * j, a.rc)
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
                nb_cell_pair<T, ORTHO>(a, s_q[wl][lane], ri.x, ri.y, ri.z, lj, ti, qi, g0, g1, g2, acc, box);
                __syncwarp();
                if (lane < qn - 32) s_q[wl][lane] = s_q[wl][32 + lane];
                qn -= 32;
                __syncwarp();
            }
        }
        if (lane < qn)
            nb_cell_pair<T, ORTHO>(a, s_q[wl][lane], ri.x, ri.y, ri.z, lj, ti, qi, g0, g1, g2, acc, box);
#pragma unroll
        for (int k = 0; k < 9; ++k) red[2 + k] = box[32 * k];
        red[0] = (double)acc[0];
        red[1] = (double)acc[1];
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
