// Cell-list neighbour build (sm_100a), replacing the freud AABB query behind
// NeighborList.allocate (dmff/common/nblist.py:27-55).
//
// Output rows (i, j, nbond), i < j, sorted by i: exactly the pairs whose minimum-image distance
// (the reference's pbc_shift, spatial.py:14-32) is < rc, with nbond read from a sparse
// covalent map (the reference reads a dense N x N map, nblist.py:22-25).  The distance test
// runs in FP64 with every product and sum rounded separately in a fixed order, so the pair set
// is reproducible bit for bit by an elementwise float64 computation on the host.
//
// The engine's builds: k_bin_count (+ k_bin_scan) + k_bin_fill sort the atoms into half-width cells, one pass of
// k_pairs_cell (k_pairs_flat in boxes below five such cells) runs the distance tests and leaves each
// atom's rows in its slots, and k_nb_place scans the counts and copies the slots to their final
// places.  The kernels before those (k_cell_count .. k_pairs_warp: cells at least rc wide, 27-cell
// scan, count and write passes) serve the build that allocates no memory.
#pragma once
#include "common.cuh"

namespace dmffb {

struct NbArgs {
    int n;
    const double* pos;
    Box box;
    double rc;
    int nc[3];
    const int32_t* cell_start;  // [ncell+1]
    const int32_t* cell_atoms;  // [n]
    const int32_t* cov_ptr;     // [n+1] rows of j > i
    const int32_t* cov_j;
    const int32_t* cov_nb;
    const int32_t* cov_lo = nullptr;  // [n] smallest / largest covalent partner (either direction) or null
    const int32_t* cov_hi = nullptr;
    int32_t* count;             // [n] (pass 0) per-atom pair counts
    const int64_t* offset;      // [n+1] (pass 1)
    int32_t* pairs;             // [cap*3]
    int64_t cap;
};

// exact, non-contracted FP64 minimum-image distance test (order: x, y, z; left to right)
__device__ __forceinline__ bool within_rc(const Box& b, const double* pi, const double* pj, double rc) {
    const double d0 = __dsub_rn(pj[0], pi[0]);
    const double d1 = __dsub_rn(pj[1], pi[1]);
    const double d2 = __dsub_rn(pj[2], pi[2]);
    double s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double t = __dadd_rn(__dadd_rn(__dmul_rn(d0, b.hinv[k]), __dmul_rn(d1, b.hinv[3 + k])), __dmul_rn(d2, b.hinv[6 + k]));
        s[k] = __dsub_rn(t, floor(__dadd_rn(t, 0.5)));
    }
    double e[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        e[c] = __dadd_rn(__dadd_rn(__dmul_rn(s[0], b.h[c]), __dmul_rn(s[1], b.h[3 + c])), __dmul_rn(s[2], b.h[6 + c]));
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(e[0], e[0]), __dmul_rn(e[1], e[1])), __dmul_rn(e[2], e[2]));
    return __dsqrt_rn(r2) < rc;
}

__device__ __forceinline__ int cell_of(const Box& b, const int nc[3], const double* p, int c3[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double s = p[0] * b.hinv[k] + p[1] * b.hinv[3 + k] + p[2] * b.hinv[6 + k];
        s -= floor(s);
        int c = (int)(s * nc[k]);
        c = c < 0 ? 0 : (c >= nc[k] ? nc[k] - 1 : c);
        c3[k] = c;
    }
    return (c3[0] * nc[1] + c3[1]) * nc[2] + c3[2];
}

static __global__ void k_cell_count(int n, const double* pos, Box b, int nc0, int nc1, int nc2, int32_t* atom_cell,
                             int32_t* cell_count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int nc[3] = {nc0, nc1, nc2};
    int c3[3];
    const int c = cell_of(b, nc, pos + 3 * i, c3);
    atom_cell[i] = c;
    atomicAdd(cell_count + c, 1);
}

static __global__ void k_cell_fill(int n, const int32_t* atom_cell, const int32_t* cell_start, int32_t* cursor,
                            int32_t* cell_atoms) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = atom_cell[i];
    const int k = atomicAdd(cursor + c, 1);
    cell_atoms[cell_start[c] + k] = i;
}

__device__ __forceinline__ int lookup_nbond(const NbArgs& a, int i, int j) {
    for (int k = a.cov_ptr[i]; k < a.cov_ptr[i + 1]; ++k)
        if (a.cov_j[k] == j) return a.cov_nb[k];
    return 0;
}

// small boxes (fewer than 3 cells on an axis): every j > i is a candidate.  Pass 0 counts the pairs
// of each atom, pass 1 writes the rows at offset[i]
template <int PASS>
__global__ void __launch_bounds__(128) k_pairs_all(NbArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const double* pi = a.pos + 3 * i;
    int cnt = 0;
    int64_t out = (PASS == 1) ? a.offset[i] : 0;
    for (int j = i + 1; j < a.n; ++j) {
        if (!within_rc(a.box, pi, a.pos + 3 * j, a.rc)) continue;
        if (PASS == 1) {
            if (out < a.cap) {
                a.pairs[3 * out] = i;
                a.pairs[3 * out + 1] = j;
                a.pairs[3 * out + 2] = lookup_nbond(a, i, j);
            }
            ++out;
        } else {
            ++cnt;
        }
    }
    if (PASS == 0) a.count[i] = cnt;
}


// Warp-per-atom variant: lanes stride over the candidates of each of the 27 cells; a FP32
// distance decides every candidate farther than 1e-3 A from the cutoff (and away from a
// half-box image ambiguity), the exact FP64 test decides the rest, so the pair set is the one
// of within_rc.  Output order: ballot prefix within each chunk keeps rows sorted by i.
template <int PASS>
__global__ void __launch_bounds__(256) k_pairs_warp(NbArgs a) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= a.n) return;
    const double* pi = a.pos + 3 * i;
    const double pix = pi[0], piy = pi[1], piz = pi[2];
    float hf[9], hif[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) { hf[k] = (float)a.box.h[k]; hif[k] = (float)a.box.hinv[k]; }
    const float rlo = (float)(a.rc - 1e-3), rhi = (float)(a.rc + 1e-3);
    const float rlo2 = rlo * rlo, rhi2 = rhi * rhi;
    int c3[3];
    cell_of(a.box, a.nc, pi, c3);
    int64_t out = (PASS == 1) ? a.offset[i] : 0;
    int cnt = 0;
    const unsigned lt = (1u << lane) - 1u;
    for (int dx = -1; dx <= 1; ++dx) {
        const int cx = (c3[0] + dx + a.nc[0]) % a.nc[0];
        for (int dy = -1; dy <= 1; ++dy) {
            const int cy = (c3[1] + dy + a.nc[1]) % a.nc[1];
            for (int dz = -1; dz <= 1; ++dz) {
                const int cz = (c3[2] + dz + a.nc[2]) % a.nc[2];
                const int c = (cx * a.nc[1] + cy) * a.nc[2] + cz;
                const int cs = a.cell_start[c], ce = a.cell_start[c + 1];
                for (int base = cs; base < ce; base += 32) {
                    const int k = base + lane;
                    bool keep = false;
                    int j = -1;
                    if (k < ce) {
                        j = a.cell_atoms[k];
                        if (j > i) {
                            const double* pj = a.pos + 3 * j;
                            const float d0 = (float)(pj[0] - pix), d1 = (float)(pj[1] - piy), d2 = (float)(pj[2] - piz);
                            bool amb = false;
                            float sf[3];
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                float t = d0 * hif[q] + d1 * hif[3 + q] + d2 * hif[6 + q];
                                float nn = floorf(t + 0.5f);
                                sf[q] = t - nn;
                                amb |= fabsf(sf[q]) > 0.4999f;
                            }
                            const float e0 = sf[0] * hf[0] + sf[1] * hf[3] + sf[2] * hf[6];
                            const float e1 = sf[0] * hf[1] + sf[1] * hf[4] + sf[2] * hf[7];
                            const float e2 = sf[0] * hf[2] + sf[1] * hf[5] + sf[2] * hf[8];
                            const float r2 = e0 * e0 + e1 * e1 + e2 * e2;
                            if (!amb && r2 < rlo2) keep = true;
                            else if (!amb && r2 > rhi2) keep = false;
                            else keep = within_rc(a.box, pi, pj, a.rc);
                        }
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, keep);
                    if (PASS == 1) {
                        if (keep) {
                            const int64_t slot = out + __popc(m & lt);
                            if (slot < a.cap) {
                                a.pairs[3 * slot] = i;
                                a.pairs[3 * slot + 1] = j;
                                a.pairs[3 * slot + 2] = lookup_nbond(a, i, j);
                            }
                        }
                        out += __popc(m);
                    } else {
                        cnt += __popc(m);
                    }
                }
            }
        }
    }
    if (PASS == 0 && lane == 0) a.count[i] = cnt;
}


// ------------------------------------------------------------------ the engine's builds
//
// Counting sort of the atoms into the cells, in two launches (three for many cells).  k_bin_count takes each atom's cell
// and its arrival rank there; the last CTA to finish scans the counts into cell_start and clears
// them for the next call (they are zero between calls), so no memset, no library scan and no
// cursor array.  k_bin_fill writes the cell-ordered float4 positions (x, y, z, atom index as int
// bits), all that the pair passes read.  `zero` is cleared on the way (the build's sums and totals).
// Launch-bound at liquid sizes: the seven launches this replaces (FP32 copy, two memsets, count,
// two-kernel scan, fill) took 13.5 us of device time at 12288 atoms, these two 7.  The last CTA takes 3 us for
// a tile of 4096 cells: boxes of more than two (atoms in a vacuum) leave the scan to k_bin_scan, a CTA per
// tile, which starts from sums that k_bin_count left per tile (125000 cells: 4 + 5.5 us against 96).
constexpr int kBinThreads = 512;
constexpr int kBinItems = 8;  // counts per thread and tile of a scan
constexpr int kBinTile = kBinThreads * kBinItems, kBinTiles = 64 * 64 * 64 / kBinTile;  // at most 64 cells an axis

struct BinArgs {
    int n;
    const double* pos;
    Box box;
    int nc[3];
    int32_t* atom_cell;   // [n]
    int32_t* rank;        // [n]
    int32_t* cell_count;  // [ncell rounded up to kBinItems], zero between calls
    int32_t* cell_start;  // [ncell + 1]
    unsigned* done;       // CTAs that have finished, zero between calls
    int32_t* tiles;       // [kBinTiles] atoms per tile of cells, zero between calls; null: the last CTA scans
    int32_t* zero;        // words to clear, or null
    int nzero;
    float4* posc;         // [n]
    int32_t* cell_atoms;  // [n] the atom indices of posc by themselves, or null
};

// cell_start of the tile of counts from cell t0 on, whose atoms come after `before` others, and the counts cleared;
// returns the tile's atoms (whole CTA)
__device__ __forceinline__ int bin_tile(const BinArgs& a, int ncell, int t0, int before, int* s_warp) {
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int c0 = t0 + kBinItems * threadIdx.x;
    int v[kBinItems];
#pragma unroll
    for (int k = 0; k < kBinItems; ++k) v[k] = 0;
    if (c0 < ncell) {
        int4* src = (int4*)(a.cell_count + c0);
        *(int4*)v = __ldcg(src);
        *(int4*)(v + 4) = __ldcg(src + 1);
        src[0] = make_int4(0, 0, 0, 0);
        src[1] = make_int4(0, 0, 0, 0);
    }
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kBinItems; ++k) sum += v[k];
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[wl] = incl;
    __syncthreads();
    int total = 0;
    for (int w = 0; w < kBinThreads / 32; ++w) {
        if (w < wl) before += s_warp[w];
        total += s_warp[w];
    }
    int at = before + incl - sum;
#pragma unroll
    for (int k = 0; k < kBinItems; ++k) {
        if (c0 + k < ncell) a.cell_start[c0 + k] = at;
        at += v[k];
    }
    __syncthreads();
    return total;
}

static __global__ void __launch_bounds__(kBinThreads) k_bin_count(BinArgs a) {
    __shared__ bool s_last;
    __shared__ int s_warp[kBinThreads / 32], s_tile[kBinTiles];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (a.tiles) {
        if (threadIdx.x < kBinTiles) s_tile[threadIdx.x] = 0;
        __syncthreads();
    }
    if (i < a.n) {
        int c3[3];
        const int c = cell_of(a.box, a.nc, a.pos + 3 * i, c3);
        a.atom_cell[i] = c;
        a.rank[i] = atomicAdd(a.cell_count + c, 1);
        if (a.tiles) atomicAdd(s_tile + c / kBinTile, 1);
    }
    for (int k = i; k < a.nzero; k += gridDim.x * blockDim.x) a.zero[k] = 0;
    if (a.tiles) {
        __syncthreads();
        if (threadIdx.x < kBinTiles && s_tile[threadIdx.x]) atomicAdd(a.tiles + threadIdx.x, s_tile[threadIdx.x]);
        return;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int ncell = a.nc[0] * a.nc[1] * a.nc[2];
    int before = 0;
    for (int t0 = 0; t0 < ncell; t0 += kBinTile) before += bin_tile(a, ncell, t0, before, s_warp);
    if (threadIdx.x == 0) {
        a.cell_start[ncell] = a.n;
        *a.done = 0u;
    }
}

static __global__ void __launch_bounds__(kBinThreads) k_bin_scan(BinArgs a) {
    __shared__ int s_warp[kBinThreads / 32];
    static_assert(kBinTiles <= 64, "two tiles a lane");
    const int ncell = a.nc[0] * a.nc[1] * a.nc[2], t = blockIdx.x, lane = threadIdx.x & 31;
    const int before = __reduce_add_sync(0xffffffffu, (lane < t ? a.tiles[lane] : 0) + (lane + 32 < t ? a.tiles[lane + 32] : 0));
    bin_tile(a, ncell, t * kBinTile, before, s_warp);
    if (t == 0 && threadIdx.x == 0) a.cell_start[ncell] = a.n;
}

static __global__ void k_bin_fill(BinArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (a.tiles && i < kBinTiles) a.tiles[i] = 0;
    if (i >= a.n) return;
    // the image inside the box: FP32 then resolves a distance to about 1e-7 of the box, however far
    // the caller's coordinates have drifted
    const double* p = a.pos + 3 * i;
    double s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = p[0] * a.box.hinv[k] + p[1] * a.box.hinv[3 + k] + p[2] * a.box.hinv[6 + k];
        s[k] -= floor(s[k]);
    }
    float w[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) w[c] = (float)(s[0] * a.box.h[c] + s[1] * a.box.h[3 + c] + s[2] * a.box.h[6 + c]);
    const int k = a.cell_start[a.atom_cell[i]] + a.rank[i];
    a.posc[k] = make_float4(w[0], w[1], w[2], __int_as_float(i));
    if (a.cell_atoms) a.cell_atoms[k] = i;
}

// Totals of a build (read back by the host) and, behind them in the same array, the sums of the
// counts over runs of kNbRun atoms (half rows, full-list entries, scaled rows): the pair passes add
// into the run sums, k_nb_place turns them into offsets.
constexpr int kNbRun = 1024;
struct NbTotals {
    long long rows, entries, scaled;
    int max_h, max_f;  // largest half-row and full-list count of an atom
};
__host__ __device__ inline int nb_runs(int n) { return (n + kNbRun - 1) / kNbRun; }
__host__ __device__ inline int nb_sum_words(int n) { return (int)(sizeof(NbTotals) / 4) + 3 * nb_runs(n); }

// Both layouts the engine uses: half rows (i, j, nbond), j > i, sorted by i (pair kernels), and the
// full neighbour CSR (j != i, packed j | scale index << 28) for the atomics-free CG matvec.  FP32
// positions prefilter the candidates; those within about 2e-3 A of rc take the exact FP64 test on pos.
struct Nb2Args {
    NbArgs a;
    const float4* posc;       // [n] cell order
    int32_t* count_f;         // [n] full-list counts (null: half rows only, no CSR)
    int32_t* count_s;         // [n] half rows with nbond != 0
    int32_t* sums;            // [3][runs]
    const int64_t* off_f;     // [n+1] pass 1 of k_pairs_warp3
    int32_t* ent;             // [cap_f]
    int64_t cap_f;
    int32_t* srows;           // [cap_s] pass 1: indices of the half rows with nbond != 0
    const int32_t* off_s;     // [n]
    int64_t cap_s;
    // keep masks of the candidate batches (k_pairs_warp3): pass 0 stores one word per batch of 32
    // candidates at mask[i * mask_stride + batch] when the atom's batches fit the stride; pass 1
    // reads them instead of repeating the distance tests (null: no masks)
    uint32_t* mask = nullptr;
    int mask_stride = 0;
    // slots of the single-pass kernels: each atom's entries (all its neighbours, or those j > i where no
    // CSR is wanted) go to slots[i * slot_cap + k] as j | min(nbond, 7) << 28, which k_nb_place turns into
    // rows and CSR entries at the offsets of the counts; slots past the capacity are dropped (the
    // totals' maxima tell)
    int32_t* slots = nullptr;
    int slot_cap = 0;
};

// the FP32 box and prefilter bounds of a pair pass
struct NbFilter {
    float h[9], hi[9], rlo2, rhi2;
    float far[3];  // fractional differences (by the sum of their terms' sizes) that FP32 resolves to the band
    __device__ __forceinline__ explicit NbFilter(const NbArgs& a) {
#pragma unroll
        for (int k = 0; k < 9; ++k) { h[k] = (float)a.box.h[k]; hi[k] = (float)a.box.hinv[k]; }
        // the band around rc covers the FP32 rounding of in-box positions and their images
        double size = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) size += fabs(a.box.h[k]);
        const double band = 2e-3 + 1e-6 * size;
        const float rlo = (float)fmax(a.rc - band, 0.0), rhi = (float)(a.rc + band);
        rlo2 = rlo * rlo;
        rhi2 = rhi * rhi;
        // a fractional difference of size t is rounded by at most 2.4e-7 t (three roundings a term and two
        // sums), its image vector by that times |h_k| for each axis k: two thirds of the band over the three axes
        // (the vector's own rounding has the rest), and less than half the margin of the image test
#pragma unroll
        for (int k = 0; k < 3; ++k)
            far[k] = (float)fmin(band / (1.1e-6 * (fabs(a.box.h[3 * k]) + fabs(a.box.h[3 * k + 1]) + fabs(a.box.h[3 * k + 2]))),
                                 200.0);
    }
};

// Is the pair (i, j), j != i, within rc?  d0, d1, d2: the FP32 difference r_j - r_i.  ORTHO: the box
// is orthorhombic and the prefilter's minimum image is three multiplies per axis.  Coordinates that have
// drifted so far apart that FP32 does not resolve the band take the exact test.
template <bool ORTHO>
__device__ __forceinline__ bool nb_keep(const NbArgs& a, const NbFilter& f, int i, int j, float d0, float d1, float d2) {
    bool amb = false;
    float r2;
    if (ORTHO) {
        const float dd[3] = {d0, d1, d2};
        r2 = 0.f;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float tt = dd[q] * f.hi[4 * q];
            const float sq = tt - floorf(tt + 0.5f);
            amb |= fabsf(sq) > 0.4999f || !(fabsf(tt) <= f.far[q]);
            const float e = sq * f.h[4 * q];
            r2 = fmaf(e, e, r2);
        }
    } else {
        float sf[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float t0 = d0 * f.hi[q], t1 = d1 * f.hi[3 + q], t2 = d2 * f.hi[6 + q], tt = t0 + t1 + t2;
            sf[q] = tt - floorf(tt + 0.5f);
            amb |= fabsf(sf[q]) > 0.4999f || !(fabsf(t0) + fabsf(t1) + fabsf(t2) <= f.far[q]);
        }
        const float e0 = sf[0] * f.h[0] + sf[1] * f.h[3] + sf[2] * f.h[6];
        const float e1 = sf[0] * f.h[1] + sf[1] * f.h[4] + sf[2] * f.h[7];
        const float e2 = sf[0] * f.h[2] + sf[1] * f.h[5] + sf[2] * f.h[8];
        r2 = e0 * e0 + e1 * e1 + e2 * e2;
    }
    if (!amb && r2 < f.rlo2) return true;
    if (!amb && r2 > f.rhi2) return false;
    return j > i ? within_rc(a.box, a.pos + 3 * i, a.pos + 3 * j, a.rc)
                 : within_rc(a.box, a.pos + 3 * j, a.pos + 3 * i, a.rc);
}

// nbond of a pair; the covalent map is read only for partners inside the atom's range [plo, phi]
__device__ __forceinline__ int nb_bond(const NbArgs& a, int i, int j, int plo, int phi) {
    return (j < plo || j > phi) ? 0 : (j > i ? lookup_nbond(a, i, j) : lookup_nbond(a, j, i));
}

// The lane's part of an atom's pairs j > i within rc with nbond != 0, from the few rows of its covalent map: the
// count pass then looks up no candidate (30000 atoms at rc 12 A: 623 us with a lookup of each kept one, 475 without).
__device__ __forceinline__ int nb_scaled(const NbArgs& a, int i, int lane) {
    int cnt = 0;
    const int beg = a.cov_ptr[i], end = a.cov_ptr[i + 1];
    for (int k = beg + lane; k < end; k += 32) {
        const int j = a.cov_j[k];
        int first = beg;  // a partner given twice counts once, with its first nbond (lookup_nbond)
        while (a.cov_j[first] != j) ++first;
        if (first == k && a.cov_nb[k] != 0 && within_rc(a.box, a.pos + 3 * i, a.pos + 3 * j, a.rc)) ++cnt;
    }
    return cnt;
}

// the counts of one atom (lane 0 of its warp)
__device__ __forceinline__ void nb_counts(const Nb2Args& b, int i, int nh, int nf, int ns) {
    const int runs = nb_runs(b.a.n), run = i / kNbRun;
    b.a.count[i] = nh;
    b.count_s[i] = ns;
    if (nh) atomicAdd(b.sums + run, nh);
    if (ns) atomicAdd(b.sums + 2 * runs + run, ns);
    if (b.count_f) {
        b.count_f[i] = nf;
        if (nf) atomicAdd(b.sums + runs + run, nf);
    }
}

// One atom's slots: the warp appends up to 32 neighbours (keep: the lane holds one) to the slots of
// atom i and advances its counts.
struct NbSlots {
    int32_t* slots;
    int cap, nh = 0, nf = 0, ns = 0;
    int i, plo, phi;
    bool all;  // both directions (CSR wanted)
    __device__ __forceinline__ NbSlots(const Nb2Args& b, int i_)
        : slots(b.slots + (int64_t)i_ * b.slot_cap), cap(b.slot_cap), i(i_), plo(b.a.cov_lo ? b.a.cov_lo[i_] : 0),
          phi(b.a.cov_hi ? b.a.cov_hi[i_] : b.a.n), all(b.count_f != nullptr) {}
    __device__ __forceinline__ void add(const Nb2Args& b, bool keep, int j, unsigned lt) {
        const bool up = keep && j > i;
        const unsigned mf = __ballot_sync(0xffffffffu, keep), mh = __ballot_sync(0xffffffffu, up);
        int nbd = 0;
        if (all ? keep : up) {
            nbd = nb_bond(b.a, i, j, plo, phi);
            const int k = all ? nf + __popc(mf & lt) : nh + __popc(mh & lt);
            if (k < cap) slots[k] = j | (min(nbd, 7) << 28);
        }
        nf += __popc(mf);
        nh += __popc(mh);
        ns += __popc(__ballot_sync(0xffffffffu, up && nbd != 0));
    }
};

// Kept candidates wait in shared memory until 32 of them fill the lanes: about a quarter of a batch of
// candidates is kept, and everything past the distance test runs once per 32 neighbours.
struct NbQueue {
    int* q;  // [64] of the warp
    int n = 0;
    __device__ __forceinline__ explicit NbQueue(int* q_) : q(q_) {}
    __device__ __forceinline__ void push(NbSlots& out, const Nb2Args& b, bool keep, int j, int lane, unsigned lt) {
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) q[n + __popc(m & lt)] = j;
        n += __popc(m);
        if (n < 32) return;
        __syncwarp();
        out.add(b, true, q[lane], lt);
        const int tail = q[32 + lane];
        __syncwarp();
        n -= 32;
        if (lane < n) q[lane] = tail;
        __syncwarp();
    }
    __device__ __forceinline__ void flush(NbSlots& out, const Nb2Args& b, int lane, unsigned lt) {
        __syncwarp();
        if (n) out.add(b, lane < n, q[lane], lt);
        __syncwarp();
        n = 0;
    }
};

// Boxes of fewer than five half-width cells on an axis: one warp per atom, every other atom is a
// candidate.  Latency-bound (450 atoms: 14 batches per warp, 450 warps): 10 us at 450 atoms, where
// the thread-per-atom count and write passes it replaces took 95 + 201 us and the CSR needed two
// more kernels over the rows.
template <bool ORTHO>
__global__ void __launch_bounds__(128) k_pairs_flat(Nb2Args b) {
    __shared__ int s_q[4][64];
    const NbArgs& a = b.a;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= a.n) return;
    const NbFilter f(a);
    const unsigned lt = (1u << lane) - 1u;
    const double pix = a.pos[3 * i], piy = a.pos[3 * i + 1], piz = a.pos[3 * i + 2];
    NbSlots out(b, i);
    NbQueue queue(s_q[threadIdx.x >> 5]);
    for (int j0 = 0; j0 < a.n; j0 += 32) {
        const int j = j0 + lane;
        bool keep = false;
        if (j < a.n && j != i)
            keep = nb_keep<ORTHO>(a, f, i, j, (float)(a.pos[3 * j] - pix), (float)(a.pos[3 * j + 1] - piy),
                                  (float)(a.pos[3 * j + 2] - piz));
        queue.push(out, b, keep, j, lane, lt);
    }
    queue.flush(out, b, lane, lt);
    if (lane == 0) nb_counts(b, i, out.nh, out.nf, out.ns);
}

// Cells at least rc / S wide and a (2S + 1)^3 stencil (S = 2: 125 cells of half width, about 0.58 of
// the 27-cell search volume), one warp per atom in cell order.  The warp first
// lays the stencil's cells out as one concatenated candidate list (cell starts and a prefix sum of
// their counts in shared memory, in the dx, dy, dz order of the 27-cell scan), then walks it in
// full 32-lane batches; each lane finds its candidate's cell by advancing a cursor (lanes move
// forward monotonically), seen from the image that the cell wraps to, as in k_pairs_cell.  Count pass and fill
// pass: it serves neighbourhoods too large to stage.  30000 atoms at rc 12 A, a whole build: 642 us (683 in a
// triclinic box); with a minimum image per candidate and its covalent partners looked up in the count pass
// too 1090 (1173).
constexpr int kNbWarps = 8;  // warps per block of k_pairs_warp3
constexpr size_t kNbStageBytes = 44u << 10;  // largest candidate stage of k_pairs_cell: with its static
                                              // shared arrays it stays under the 48 KB default

template <int PASS, int S>
__global__ void __launch_bounds__(32 * kNbWarps) k_pairs_warp3(Nb2Args b) {
    constexpr int W = 2 * S + 1, NQ = W * W * W;
    __shared__ int s_beg[kNbWarps][NQ];
    __shared__ int s_off[kNbWarps][NQ + 1];
    __shared__ float s_sh[kNbWarps][NQ][3];  // lattice vectors that the cell wraps by
    const NbArgs& a = b.a;
    const int wl = threadIdx.x >> 5;
    const int ks = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (ks >= a.n) return;  // whole warps leave together
    const float4 p4 = b.posc[ks];
    const int i = __float_as_int(p4.w);
    const NbFilter f(a);
    int c3[3];
    cell_of(a.box, a.nc, a.pos + 3 * i, c3);
    // stencil cells -> (start, count), prefix-summed in q order
    int carry = 0;
    if (lane == 0) s_off[wl][0] = 0;
    for (int q0 = 0; q0 < NQ; q0 += 32) {
        const int q = q0 + lane;
        int cnt = 0;
        if (q < NQ) {
            int c[3] = {c3[0] + q / (W * W) - S, c3[1] + (q / W) % W - S, c3[2] + q % W - S}, wrap[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                wrap[k] = c[k] < 0 ? -1 : (c[k] >= a.nc[k] ? 1 : 0);
                c[k] -= wrap[k] * a.nc[k];
            }
            const int cc = (c[0] * a.nc[1] + c[1]) * a.nc[2] + c[2];
            const int cs = a.cell_start[cc];
            cnt = a.cell_start[cc + 1] - cs;
            s_beg[wl][q] = cs;
#pragma unroll
            for (int k = 0; k < 3; ++k)
                s_sh[wl][q][k] = (float)(wrap[0] * a.box.h[k] + wrap[1] * a.box.h[3 + k] + wrap[2] * a.box.h[6 + k]);
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
    int64_t out_h = (PASS == 1) ? a.offset[i] : 0, out_f = (PASS == 1 && b.off_f) ? b.off_f[i] : 0;
    int64_t out_s = (PASS == 1 && b.srows) ? b.off_s[i] : 0;
    int cnt_h = 0, cnt_f = 0;
    const int plo = a.cov_lo ? a.cov_lo[i] : 0, phi = a.cov_hi ? a.cov_hi[i] : a.n;
    const unsigned lt = (1u << lane) - 1u;
    int qc = 0;
    // both passes see the same candidate list, so the masks are complete exactly when it fits
    const bool use_mask = b.mask && (total + 31) / 32 <= b.mask_stride;
    uint32_t* mrow = use_mask ? b.mask + (size_t)i * b.mask_stride : nullptr;
    for (int base = 0; base < total; base += 32) {
        const int t = base + lane;
        bool keep = false;
        int j = -1;
        if (PASS == 1 && use_mask) {
            const uint32_t mk = mrow[base >> 5];
            if (mk == 0u) continue;  // warp-uniform: no candidate of this batch is kept
            if ((mk >> lane) & 1u) {
                while (t >= s_off[wl][qc + 1]) ++qc;
                j = a.cell_atoms[s_beg[wl][qc] + (t - s_off[wl][qc])];
                keep = true;
            }
        } else if (t < total) {
            while (t >= s_off[wl][qc + 1]) ++qc;
            const float4 pj = b.posc[s_beg[wl][qc] + (t - s_off[wl][qc])];
            j = __float_as_int(pj.w);
            const float dx = pj.x + s_sh[wl][qc][0] - p4.x, dy = pj.y + s_sh[wl][qc][1] - p4.y, dz = pj.z + s_sh[wl][qc][2] - p4.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 < f.rlo2) keep = j != i;
            else if (r2 <= f.rhi2 && j != i) keep = j > i ? within_rc(a.box, a.pos + 3 * i, a.pos + 3 * j, a.rc)
                                                          : within_rc(a.box, a.pos + 3 * j, a.pos + 3 * i, a.rc);
        }
        const bool up = keep && j > i;
        const unsigned mf = __ballot_sync(0xffffffffu, keep);
        const unsigned mh = __ballot_sync(0xffffffffu, up);
        if (PASS == 0 && use_mask && lane == 0) mrow[base >> 5] = mf;
        if (PASS == 1) {
            const int nbd = keep ? nb_bond(a, i, j, plo, phi) : 0;
            const unsigned ms = __ballot_sync(0xffffffffu, up && nbd != 0);
            if (keep) {
                int sidx = nbd - 1;
                if (sidx < 0) sidx += 6;
                const int64_t sf_ = out_f + __popc(mf & lt);
                if (b.ent && sf_ < b.cap_f) b.ent[sf_] = j | (sidx << 28);
                if (up) {
                    const int64_t sh = out_h + __popc(mh & lt);
                    if (sh < a.cap) {
                        a.pairs[3 * sh] = i;
                        a.pairs[3 * sh + 1] = j;
                        a.pairs[3 * sh + 2] = nbd;
                    }
                    const int64_t ss = out_s + __popc(ms & lt);
                    if (nbd != 0 && b.srows && ss < b.cap_s) b.srows[ss] = (int32_t)sh;
                }
            }
            out_f += __popc(mf);
            out_h += __popc(mh);
            out_s += __popc(ms);
        } else {
            cnt_f += __popc(mf);
            cnt_h += __popc(mh);
        }
    }
    if (PASS == 0) {
        const int cnt_s = __reduce_add_sync(0xffffffffu, nb_scaled(a, i, lane));
        if (lane == 0) nb_counts(b, i, cnt_h, cnt_f, cnt_s);
    }
}

// Block-per-cell single pass over the (2S + 1)^3 stencil: one CTA takes every atom of one cell.  Cells of
// a z column are contiguous in cell order, so the stencil is (2S + 1)^2 columns of one run of atoms, two
// where the column wraps.  The runs are staged in shared memory as (x, y, z, j) float4s, shifted by the
// lattice vectors their column wraps by: with in-box positions that is the image nearest to the cell's
// atoms for every pair within rc (the box holds at least 2S + 1 cells of rc / S per axis), so a
// candidate's test is one difference and one comparison for any box, candidates near rc taking the
// exact FP64 test.  The NW warps of the CTA take the cell's atoms in turn.  Neighbourhoods larger than
// `chmax` entries are read from global memory instead.
// Bound by instruction issue: 49 us at 12288 atoms and rc 8 A, 101 at 30000.  With a minimum image per
// candidate, the emission run once per batch of candidates, a cell search per staged entry and rows
// and CSR entries in slots of their own it took 81 and 170.
template <int S, int NW>
__global__ void __launch_bounds__(32 * NW) k_pairs_cell(Nb2Args b, int chmax) {
    constexpr int W = 2 * S + 1, NC = W * W;
    static_assert(NC <= 32, "a lane per column");
    __shared__ int s_beg[2 * NC], s_off[2 * NC + 1];
    __shared__ float s_sh[2 * NC][3];
    __shared__ int s_q[NW][64];
    extern __shared__ __align__(16) float4 s_cand[];
    const NbArgs& a = b.a;
    const int c = blockIdx.x;
    const int cs0 = a.cell_start[c], m = a.cell_start[c + 1] - cs0;
    if (m == 0) return;  // whole CTA
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (wl == 0) {
        const int c2 = c % a.nc[2], c1 = (c / a.nc[2]) % a.nc[1], c0 = c / (a.nc[2] * a.nc[1]);
        int cnt[2] = {0, 0};
        if (lane < NC) {
            int x = c0 + lane / W - S, y = c1 + lane % W - S;
            const int nx = x < 0 ? -1 : (x >= a.nc[0] ? 1 : 0), ny = y < 0 ? -1 : (y >= a.nc[1] ? 1 : 0);
            x -= nx * a.nc[0];
            y -= ny * a.nc[1];
            const int* col = a.cell_start + (x * a.nc[1] + y) * a.nc[2];
            // [z0, z1] inside the box and, wrapped by nz, the rest
            const int z0 = max(c2 - S, 0), z1 = min(c2 + S, a.nc[2] - 1);
            const int nz = c2 - S < 0 ? -1 : (c2 + S >= a.nc[2] ? 1 : 0);
            const int w0 = nz < 0 ? c2 - S + a.nc[2] : 0, w1 = nz < 0 ? a.nc[2] - 1 : c2 + S - a.nc[2];
            s_beg[2 * lane] = col[z0];
            cnt[0] = col[z1 + 1] - col[z0];
            s_beg[2 * lane + 1] = nz ? col[w0] : 0;
            cnt[1] = nz ? col[w1 + 1] - col[w0] : 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double sh = nx * a.box.h[k] + ny * a.box.h[3 + k];
                s_sh[2 * lane][k] = (float)sh;
                s_sh[2 * lane + 1][k] = (float)(sh + nz * a.box.h[6 + k]);
            }
        }
        int incl = cnt[0] + cnt[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane < NC) {
            s_off[2 * lane] = incl - cnt[0] - cnt[1];
            s_off[2 * lane + 1] = incl - cnt[1];
            if (lane == NC - 1) s_off[2 * NC] = incl;
        }
    }
    __syncthreads();
    const int total = s_off[2 * NC];
    const bool staged = total <= chmax;
    auto candidate = [&](int run, int k) {
        float4 p = b.posc[s_beg[run] + k];
        p.x += s_sh[run][0];
        p.y += s_sh[run][1];
        p.z += s_sh[run][2];
        return p;
    };
    if (staged)
        for (int run = wl; run < 2 * NC; run += NW) {
            const int off = s_off[run], cnt = s_off[run + 1] - off;
            for (int k = lane; k < cnt; k += 32) s_cand[off + k] = candidate(run, k);
        }
    __syncthreads();
    const NbFilter f(a);
    const unsigned lt = (1u << lane) - 1u;
    for (int ai = wl; ai < m; ai += NW) {
        const float4 p4 = b.posc[cs0 + ai];
        const int i = __float_as_int(p4.w);
        NbSlots out(b, i);
        NbQueue queue(s_q[wl]);
        auto test = [&](const float4& pj) {
            const float dx = pj.x - p4.x, dy = pj.y - p4.y, dz = pj.z - p4.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            const int j = __float_as_int(pj.w);
            if (r2 > f.rhi2 || j == i) return false;
            if (r2 < f.rlo2) return true;
            return j > i ? within_rc(a.box, a.pos + 3 * i, a.pos + 3 * j, a.rc)
                         : within_rc(a.box, a.pos + 3 * j, a.pos + 3 * i, a.rc);
        };
        if (staged) {
            for (int base = 0; base < total; base += 32) {
                const int t = base + lane;
                bool keep = false;
                int j = -1;
                if (t < total) {
                    const float4 pj = s_cand[t];
                    j = __float_as_int(pj.w);
                    keep = test(pj);
                }
                queue.push(out, b, keep, j, lane, lt);
            }
        } else {
            for (int run = 0; run < 2 * NC; ++run) {
                const int cnt = s_off[run + 1] - s_off[run];
                for (int base = 0; base < cnt; base += 32) {
                    const int k = base + lane;
                    bool keep = false;
                    int j = -1;
                    if (k < cnt) {
                        const float4 pj = candidate(run, k);
                        j = __float_as_int(pj.w);
                        keep = test(pj);
                    }
                    queue.push(out, b, keep, j, lane, lt);
                }
            }
        }
        queue.flush(out, b, lane, lt);
        if (lane == 0) nb_counts(b, i, out.nh, out.nf, out.ns);
    }
}

// Offsets from the counts, and the slots turned into rows and CSR entries there.  A CTA takes kPlaceAtoms
// atoms, a warp each: it sums the run sums before their run and the counts of the run's earlier atoms,
// scans its own, and writes each atom's rows, CSR entries and the indices of its rows with nbond != 0,
// all in atom order; the CTA of the last atom writes the totals.  Nothing is written past a capacity: the
// caller compares the totals before it uses the lists.  Bound by latency and the writes: 18 us at 12288
// atoms (22 copying rows and entries from slots of their own), for two memsets, two two-kernel scans, a copy kernel and a library selection over all rows that took 47 us and
// two more host round trips.
constexpr int kPlaceAtoms = 8, kPlaceThreads = 32 * kPlaceAtoms;
static_assert(kNbRun % kPlaceAtoms == 0, "a CTA's atoms lie in one run");

struct PlaceArgs {
    int n;
    NbArgs cov;                                  // the covalent map (nbond past a slot's three bits)
    const int32_t *count_h, *count_f, *count_s;  // count_f null: no CSR, the slots hold j > i alone
    const int32_t* sums;                         // [3][runs]
    NbTotals* tot;                               // max_h, max_f zero on entry
    int64_t *off_h, *off_f;                      // [n+1]; off_f null: no CSR
    int32_t* off_s;                              // [n]
    const int32_t* slots;                        // null: offsets and totals only
    int slot_cap;
    int32_t* rows;
    int64_t rows_cap;
    int32_t* ent;
    int64_t ent_cap;
    int32_t* srows;  // null: not wanted
    int64_t srows_cap;
};

static __global__ void __launch_bounds__(kPlaceThreads) k_nb_place(PlaceArgs a) {
    constexpr int NW = kPlaceThreads / 32;
    __shared__ long long s_part[NW][3], s_off[3][kPlaceAtoms];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5;
    const int a0 = blockIdx.x * kPlaceAtoms, run = a0 / kNbRun, runs = nb_runs(a.n);
    const int32_t* const cnt[3] = {a.count_h, a.count_f, a.count_s};
    long long base[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (!cnt[k]) continue;
        for (int r = tid; r < run; r += kPlaceThreads) base[k] += a.sums[k * runs + r];
        for (int i = run * kNbRun + tid; i < a0; i += kPlaceThreads) base[k] += cnt[k][i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) base[k] += __shfl_down_sync(0xffffffffu, base[k], o);
        if (lane == 0) s_part[wl][k] = base[k];
    }
    __syncthreads();
    if (wl < 3 && cnt[wl]) {  // one warp per count: the atoms of the CTA
        const int k = wl, i = a0 + lane;
        const bool mine = lane < kPlaceAtoms && i < a.n;
        const int c = mine ? cnt[k][i] : 0;
        long long before = 0;
        for (int w = 0; w < NW; ++w) before += s_part[w][k];
        int incl = c, mx = c;
#pragma unroll
        for (int o = 1; o < kPlaceAtoms; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        const long long off = before + incl - c;
        if (lane < kPlaceAtoms) s_off[k][lane] = off;
        if (mine) {
            if (k == 0 && a.off_h) a.off_h[i] = off;
            if (k == 1) a.off_f[i] = off;
            if (k == 2 && a.off_s) a.off_s[i] = (int32_t)off;
        }
        if (mine && i == a.n - 1) {
            const long long total = off + c;
            if (k == 0) {
                a.tot->rows = total;
                if (a.off_h) a.off_h[a.n] = total;
            } else if (k == 1) {
                a.tot->entries = total;
                a.off_f[a.n] = total;
            } else {
                a.tot->scaled = total;
            }
        }
        if (lane == 0 && k == 0) atomicMax(&a.tot->max_h, mx);
        if (lane == 0 && k == 1) atomicMax(&a.tot->max_f, mx);
    }
    if (!a.slots) return;  // whole grid
    __syncthreads();
    const int i = a0 + wl;
    if (i >= a.n) return;
    const int32_t* const src = a.slots + (int64_t)i * a.slot_cap;
    const int ns = min(a.count_f ? a.count_f[i] : a.count_h[i], a.slot_cap);
    int64_t bh = s_off[0][wl], bs = s_off[2][wl];
    const int64_t bf = a.count_f ? s_off[1][wl] : 0;
    const unsigned lt = (1u << lane) - 1u;
    constexpr int U = 4;  // slot loads in flight per lane
    for (int k0 = 0; k0 < ns; k0 += 32 * U) {
        int32_t v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + 32 * u + lane;
            v[u] = k < ns ? src[k] : -1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + 32 * u + lane;
            const bool ok = k < ns;
            const int j = v[u] & 0x0FFFFFFF;
            int nbd = (v[u] >> 28) & 7;
            if (ok && nbd == 7) nbd = j > i ? lookup_nbond(a.cov, i, j) : lookup_nbond(a.cov, j, i);
            int sidx = nbd - 1;
            if (sidx < 0) sidx += 6;
            if (ok && a.ent && bf + k < a.ent_cap) a.ent[bf + k] = j | (sidx << 28);
            const bool up = ok && j > i;
            const unsigned mh = __ballot_sync(0xffffffffu, up), ms = __ballot_sync(0xffffffffu, up && nbd != 0);
            if (up) {
                const int64_t r = bh + __popc(mh & lt);
                if (a.rows && r < a.rows_cap) {
                    a.rows[3 * r] = i;
                    a.rows[3 * r + 1] = j;
                    a.rows[3 * r + 2] = nbd;
                }
                const int64_t p = bs + __popc(ms & lt);
                if (nbd != 0 && a.srows && p < a.srows_cap) a.srows[p] = (int32_t)r;
            }
            bh += __popc(mh);
            bs += __popc(ms);
        }
    }
}

}  // namespace dmffb
