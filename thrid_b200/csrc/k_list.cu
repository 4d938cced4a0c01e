// k_list.cu -- bookkeeping pair list (mklist_cell.F90:8-352 / mklist.F90:8-234)
// and molecule wrap (transcor.F90) on the device.
//
// Layout.  Atoms are counting-sorted into the reference's cells
// (cellcount = INT(L/rcut_book), cell = MOD(INT((x+L)/cellsize), n),
// mklist_cell.F90:114-180); inside a cell by (4x4x4 sub-cell, atom index), and
// each cell's segment is padded with dummy slots (perm = -1) to a multiple of
// 8, so every 8-slot CLUSTER lies inside one cell.
//
// List.  For every i-cluster the row holds each atom slot t of a cluster that
// it owns (owns) that is a partner of at least one of its atoms, as
// (mask << 24 | t): bit b of the mask says that (8*cluster + b, t) is a list
// pair.  Every pair is stored once.
// Membership is the reference test pair for pair: exact FP64
// r^2 < rcut_book^2 (no FMA, Fortran dnint minimum image) minus the mkexcl
// exclusions; pgk_get_nblist() writes the pairs back in the reference CSR
// layout and row order.  When the reference would
// refuse the cell index (rdscript.F90:1595-1610) the same cells are scanned
// as distinct neighbour cells, which covers every pair of the all-pair
// mklist2a test because cellsize >= rcut_book.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "pgk_ctx.cuh"

#define MAX_CELL_ATOMS 4096
#define SUBKEY_SHIFT 25

// transcor.F90: wrap each molecule by its first atom into [0, L)
__global__ void k_transcor(double* __restrict__ pos, const int* __restrict__ mol_idx,
                           const int* __restrict__ mol_list, int nmole, const DynState* __restrict__ dyn) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmole) return;
    int b = mol_idx[m], e = mol_idx[m + 1];
    int a0 = mol_list[b];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double L = dyn->box[d];
        double x = pos[3 * a0 + d];
        double sh = 0.0;
        if (x < 0.0) sh = L;
        else if (x > L) sh = -L;
        if (sh != 0.0)
            for (int q = b; q < e; ++q) {
                int k = mol_list[q];
                pos[3 * k + d] = __dadd_rn(pos[3 * k + d], sh);
            }
    }
}

__device__ __forceinline__ int cell_coord(double x, double L, double cs, int nc) {
    int c = (int)__ddiv_rn(__dadd_rn(x, L), cs);
    c %= nc;
    return c < 0 ? c + nc : c;
}

// cell of each atom (reference rule) and its sort key inside the cell: the
// 4x4x4 sub-cell (Morton order) above the atom index
__global__ void k_cell_assign(const double* __restrict__ pos, int n, const DynState* __restrict__ dyn,
                              int* __restrict__ cell_of, int* __restrict__ cell_cnt, int* __restrict__ subkey) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c[3], sc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double L = dyn->box[d], cs = dyn->cellsize[d];
        c[d] = cell_coord(pos[3 * i + d], L, cs, dyn->ncell[d]);
        double u = __ddiv_rn(__dadd_rn(pos[3 * i + d], L), cs);
        double fr = u - floor(u);
        int q = (int)(fr * 4.0);
        sc[d] = q < 0 ? 0 : (q > 3 ? 3 : q);
    }
    int key = c[0] + dyn->ncell[0] * (c[1] + dyn->ncell[1] * c[2]);
    cell_of[i] = key;
    int morton = 0;
#pragma unroll
    for (int b = 0; b < 2; ++b)
        morton |= (((sc[0] >> b) & 1) << (3 * b)) | (((sc[1] >> b) & 1) << (3 * b + 1)) |
                  (((sc[2] >> b) & 1) << (3 * b + 2));
    subkey[i] = (morton << SUBKEY_SHIFT) | i;
    atomicAdd(&cell_cnt[key], 1);
}

// exclusive scan of the padded cell sizes (one CTA; ncells <= a few 10^4)
__global__ void k_cell_scan(const int* __restrict__ cnt, int* __restrict__ start, int* __restrict__ fill,
                            int ncells, unsigned* status) {
    __shared__ int part[1024];
    int t = threadIdx.x, nt = blockDim.x;
    int per = (ncells + nt - 1) / nt;
    int b = t * per, e = min(ncells, b + per);
    int s = 0, mx = 0;
    for (int k = b; k < e; ++k) { s += (cnt[k] + 7) & ~7; mx = max(mx, cnt[k]); }
    part[t] = s;
    if (mx > MAX_CELL_ATOMS) atomicOr(status, ST_CELL_OVERFLOW);
    __syncthreads();
    if (t == 0) {
        int run = 0;
        for (int k = 0; k < nt; ++k) { int v = part[k]; part[k] = run; run += v; }
        start[ncells] = run;
    }
    __syncthreads();
    int run = part[t];
    for (int k = b; k < e; ++k) { start[k] = run; fill[k] = run; run += (cnt[k] + 7) & ~7; }
}

__global__ void k_cell_place(const int* __restrict__ cell_of, int n, int* __restrict__ fill, int* __restrict__ perm) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = atomicAdd(&fill[cell_of[i]], 1);
    perm[p] = i;
}

// deterministic order inside each cell: ascending (sub-cell, atom index);
// the padding slots at the end of the segment get perm = -1
__global__ void k_cell_sort(int* __restrict__ perm, const int* __restrict__ start, const int* __restrict__ cnt,
                            const int* __restrict__ subkey, int ncells) {
    __shared__ int v[MAX_CELL_ATOMS];
    int cell = blockIdx.x;
    if (cell >= ncells) return;
    int b = start[cell], n = cnt[cell], npad = start[cell + 1] - b;
    for (int k = n + threadIdx.x; k < npad; k += blockDim.x) perm[b + k] = -1;
    if (n <= 0 || n > MAX_CELL_ATOMS) return;
    int np = 1;
    while (np < n) np <<= 1;
    for (int k = threadIdx.x; k < np; k += blockDim.x) v[k] = k < n ? subkey[perm[b + k]] : 0x7fffffff;
    __syncthreads();
    for (int size = 2; size <= np; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int k = threadIdx.x; k < np; k += blockDim.x) {
                int p = k ^ stride;
                if (p > k) {
                    bool up = (k & size) == 0;
                    int a = v[k], c = v[p];
                    if ((a > c) == up) { v[k] = c; v[p] = a; }
                }
            }
            __syncthreads();
        }
    for (int k = threadIdx.x; k < n; k += blockDim.x) perm[b + k] = v[k] & ((1 << SUBKEY_SHIFT) - 1);
}

// Sorted copies of the build: FP64 positions, types, FP32 positions wrapped
// into the box (the screening tests) and, per cluster, the centre and half
// widths of its bounding box (minimum image relative to its first atom).
// Eight consecutive lanes hold one cluster.
__global__ void k_sorted_gather(const int* __restrict__ perm, int npad, const double* __restrict__ pos,
                                const int* __restrict__ typ, const DynState* __restrict__ dyn,
                                int* __restrict__ iperm, double* __restrict__ pos_s, int* __restrict__ typ_s,
                                float4* __restrict__ pf, float4* __restrict__ cbox) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = s < npad ? perm[s] : -1;
    double x[3] = {0.0, 0.0, 0.0};
    int ty = 0;
    if (i >= 0) {
        iperm[i] = s;
        ty = typ[i];
        for (int d = 0; d < 3; ++d) x[d] = pos[3 * (size_t)i + d];
    }
    float w[3], lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double L = dyn->box[d];
        const double xw = x[d] - L * floor(x[d] / L);
        w[d] = (float)xw;
        // extent relative to the cluster's first atom (slots of a cluster are real from the front)
        const double x0 = __shfl_sync(0xffffffffu, xw, threadIdx.x & 24);
        double r = xw - x0;
        r -= L * rint(r / L);
        lo[d] = i >= 0 ? (float)r : 0.f;
        hi[d] = lo[d];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    }
    if (s >= npad) return;
    for (int d = 0; d < 3; ++d) pos_s[3 * (size_t)s + d] = x[d];
    typ_s[s] = ty;
    pf[s] = make_float4(w[0], w[1], w[2], __int_as_float(i));
    if ((s & 7) == 0) {
        cbox[s >> 2] = make_float4(w[0] + 0.5f * (lo[0] + hi[0]), w[1] + 0.5f * (lo[1] + hi[1]),
                                   w[2] + 0.5f * (lo[2] + hi[2]), 0.f);
        cbox[(s >> 2) + 1] = make_float4(0.5f * (hi[0] - lo[0]), 0.5f * (hi[1] - lo[1]), 0.5f * (hi[2] - lo[2]), 0.f);
    }
}

__device__ __forceinline__ bool is_excluded(const int* __restrict__ exs_idx, const int* __restrict__ exs_list,
                                            int io, int jo) {
    int b = exs_idx[io], e = exs_idx[io + 1];
    for (int k = b; k < e; ++k) {
        int v = exs_list[k];
        if (v == jo) return true;
        if (v > jo) return false;
    }
    return false;
}

// A pair of clusters I != J is kept in the row of the lower one when I + J is
// odd and of the higher one when it is even: every cluster then owns about
// half of its neighbours.  (All pairs in the lower cluster's row made the rows
// of the first cell layers about twice, those of the last a third of the mean,
// and the pair kernel's blocks as uneven.)  LOWER: all pairs in the lower
// cluster's row (pgk_ctx::plain_order).
template <bool LOWER>
__device__ __forceinline__ bool owns(int I, int J) { return LOWER || ((I + J) & 1) ? I < J : I > J; }

// nearest integer of a moderate x (adding 1.5 2^23 rounds to one)
__device__ __forceinline__ float rnd_int(float x) { return __fadd_rn(__fadd_rn(x, 12582912.f), -12582912.f); }

// One block of four warps per i-cluster:
//  1. bounding boxes: the clusters J of the distinct neighbour cells that the
//     cluster owns (owns) and whose box comes within rcut_book (a warp takes
//     a quarter of the cells, a lane a cluster);
//  2. the eight atoms of each such J against the eight cluster atoms in FP32
//     (two cluster atoms per packed operation); FRAME boxes (at least four
//     cells a side) use coordinates relative to the cluster's centre, others
//     the image of every pair.  r^2 below sqlo (above sqhi) is inside
//     (outside) rcut_book whatever the rounding; between the two the
//     reference's exact FP64 test decides.  Exclusions are looked up when j's
//     block of atom indices is one of the cluster's excluded partners;
//  3. the entries (mask << 24 | t) grouped by mask by a stable counting sort
//     (bins of mask_bin), each warp ranking a quarter of the candidates, and
//     written to the row: 32 consecutive entries then mostly share their mask
//     bits, which keeps the pair kernel's warps uniform.
// Every step keeps the candidates' order (LOWER: cells in scan order, slots
// ascending), so a build of the same positions gives the same rows.  A row of
// more than CL_CCAP candidates is sorted piece by piece (LOWER: k_sort_rows joins
// the pieces).  nlistnball (the reference's row count, one sentinel per empty
// row) is the number of pairs plus the atoms i < n-1 without a partner of higher
// index; hasup[slot] = 1 marks the atoms that have one.
// Bound by issue (63 % busy), the barriers between the steps and the latency of
// the candidate loads (fetched one iteration ahead).  Measured: 200,004 atoms
// 1.78 ms (one warp per cluster, a bounding-box test per atom, FP64-to-FP32
// conversions per pair) -> 0.82; 12,000 atoms 0.311 -> 0.093; 1,536 atoms 0.104
// -> 0.030 ms.
#define CL_JCAP (MAX_CELL_ATOMS / 8)   // clusters that a warp can queue
// candidates sorted at a time (multiple of 128).  LOWER: the first layers' rows are twice the mean, and 4,096 take
// them in one piece but for a few
#define CL_CCAP(LOWER) ((LOWER) ? 4096 : 2048)
#define ROW_PIECES ((int)0x80000000)   // ClistArgs::mark
#define CL_EXCAP 32          // excluded partners of an atom staged in shared memory (longer lists: global)
struct ClistArgs {
    const float4* pf; const float4* cbox; const double* pos_s;
    const int* cell_of; const int* cell_start; const int* cell_cnt;
    const int* exs_idx; const int* exs_list; const int2* exs_rng;
    int ncl, ccap;
    int mark;                      // bit that a row sorted in pieces sets in its count (for k_sort_rows), or 0
    double sqcut;
    float rbox, sqlo, sqhi;
    int* clist; int* ccnt; unsigned char* hasup; unsigned long long* counters; unsigned* status;
};

template <bool FRAME, bool LOWER>
__global__ void __launch_bounds__(128, LOWER ? 6 : 0) k_build_clist(ClistArgs a, const DynState* __restrict__ dyn) {
    __shared__ int sJ[4][CL_JCAP];
    constexpr int ccap = CL_CCAP(LOWER);
    __shared__ unsigned cand[ccap];
    __shared__ int hist[4][256];
    __shared__ int soff[5], sne[4], swarp[4], smaxj;
    __shared__ float4 sxy[4], sz[4];               // cluster atoms 2p, 2p+1: (x0, x1, y0, y1), (z0, z1, -, -)
    __shared__ int sio[8];
    __shared__ int2 srng[8];
    __shared__ int2 scell[27];
    __shared__ unsigned sbloom[64];
    __shared__ unsigned char sbin[256];            // mask_bin of every mask
    __shared__ int sexc[8][CL_EXCAP], snex[8];     // excluded partners of the cluster atoms
    __shared__ double sbox[6];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int cl = blockIdx.x, s0 = 8 * cl;
    const float L0 = (float)dyn->box[0], L1 = (float)dyn->box[1], L2 = (float)dyn->box[2];
    const float B0 = 1.f / L0, B1 = 1.f / L1, B2 = 1.f / L2;
    const int nc0 = dyn->ncell[0], nc1 = dyn->ncell[1], nc2 = dyn->ncell[2];
    const float4 ctr = a.cbox[2 * cl], hw = a.cbox[2 * cl + 1];
    if (tid < 8) {
        const float4 p = a.pf[s0 + tid];
        const int io = __float_as_int(p.w);
        sio[tid] = io;
        srng[tid] = io >= 0 ? a.exs_rng[io] : make_int2(INT_MAX, -1);
        float x = p.x, y = p.y, z = p.z;
        if (FRAME) {
            x -= ctr.x; y -= ctr.y; z -= ctr.z;
            x = fmaf(-L0, rnd_int(x * B0), x); y = fmaf(-L1, rnd_int(y * B1), y); z = fmaf(-L2, rnd_int(z * B2), z);
        }
        ((float*)&sxy[tid >> 1])[tid & 1] = x;
        ((float*)&sxy[tid >> 1])[2 + (tid & 1)] = y;
        ((float*)&sz[tid >> 1])[tid & 1] = z;
    }
    if (tid == 0) smaxj = 1;
    if (tid >= 64) sbloom[tid - 64] = 0u;
    if (tid >= 32 && tid < 35) { sbox[tid - 32] = dyn->box[tid - 32]; sbox[tid - 29] = 1.0 / dyn->box[tid - 32]; }
    sbin[tid] = (unsigned char)mask_bin(tid);
    sbin[tid + 128] = (unsigned char)mask_bin(tid + 128);
    __syncthreads();
    const int key = a.cell_of[sio[0]];
    const int cx = key % nc0, cy = (key / nc0) % nc1, cz = key / (nc0 * nc1);
    const int nz = nc2 >= 3 ? 3 : nc2, ny = nc1 >= 3 ? 3 : nc1, nx = nc0 >= 3 ? 3 : nc0;
    const int ncel = nx * ny * nz;
    if (tid < ncel) {             // the distinct neighbour cells' clusters
        const int c = tid % nx, b = (tid / nx) % ny, e = tid / (nx * ny);
        const int x = nc0 >= 3 ? (cx + c - 1 + nc0) % nc0 : c;
        const int y = nc1 >= 3 ? (cy + b - 1 + nc1) % nc1 : b;
        const int z = nc2 >= 3 ? (cz + e - 1 + nc2) % nc2 : e;
        const int cell = x + nc0 * (y + nc1 * z);
        const int J0 = a.cell_start[cell] >> 3, nj = (a.cell_cnt[cell] + 7) >> 3;
        scell[tid] = make_int2(J0, J0 + nj);
        atomicMax(&smaxj, nj);
    }
    {                             // 16 threads a cluster atom
        const int ii = tid >> 4, io = sio[ii];
        int b = 0, n = 0;
        if (io >= 0) { b = a.exs_idx[io]; n = a.exs_idx[io + 1] - b; }
        for (int q = tid & 15; q < min(n, CL_EXCAP); q += 16) sexc[ii][q] = a.exs_list[b + q];
        if ((tid & 15) == 0) snex[ii] = n;
    }
    // filter of the excluded partners: blocks of 16 atom indices, hashed
    if (tid >= 32 && tid < 40) {
        const int2 rg = srng[tid - 32];
        if (rg.y >= rg.x) {
            const int b0 = rg.x >> 4, b1 = rg.y >> 4;
            if (b1 - b0 >= 256) for (int q = 0; q < 64; ++q) sbloom[q] = 0xffffffffu;
            else for (int q = b0; q <= b1; ++q) atomicOr(&sbloom[(q >> 5) & 63], 1u << (q & 31));
        }
    }
    unsigned vmask = 0;                                  // real cluster atoms
#pragma unroll
    for (int ii = 0; ii < 8; ++ii) vmask |= sio[ii] >= 0 ? 1u << ii : 0u;
    __syncthreads();
    if (smaxj > CL_JCAP) {       // a cell beyond MAX_CELL_ATOMS: k_cell_scan has set the status, the host stops
        if (tid == 0) a.ccnt[cl] = 0;
        return;
    }
    int bw = max(1, CL_JCAP / smaxj);                    // a warp's cells in one round of step 1
    if (LOWER) bw = min(bw, (ncel + 3) >> 2);
    const int batch = 4 * bw;
    const float rb2 = a.rbox * a.rbox;
    int* __restrict__ row = a.clist + (size_t)cl * a.ccap;
    const float mid = 0.5f * (a.sqlo + a.sqhi), band = 0.5f * (a.sqhi - a.sqlo) * 1.0001f;
    int npair = 0;
    unsigned up = 0;
    int count = 0;                                       // row entries so far (uniform)
    int pieces = 0;                                      // sorted pieces of the row
    for (int q0 = 0; q0 < ncel; q0 += batch) {
        // 1: owned clusters near the bounding box
        int nj = 0;
        // LOWER: a warp's cells consecutive, so that the candidates come in scan order; else every fourth cell, which
        // spreads the near cells, and with them the entries, over the warps
        const int qs = LOWER ? 1 : 4, qb = LOWER ? q0 + w * bw : q0 + w, qe = min(ncel, LOWER ? qb + bw : q0 + batch);
        for (int q = qb; q < qe; q += qs) {
            const int J1 = scell[q].y;
            for (int jb = scell[q].x; jb < J1; jb += 32) {
                const int J = jb + lane;
                bool ok = J < J1 && (J == cl || owns<LOWER>(cl, J));
                if (ok) {
                    const float4 c = a.cbox[2 * J], h = a.cbox[2 * J + 1];
                    float dx = c.x - ctr.x, dy = c.y - ctr.y, dz = c.z - ctr.z;
                    dx = fmaf(-L0, rnd_int(dx * B0), dx);
                    dy = fmaf(-L1, rnd_int(dy * B1), dy);
                    dz = fmaf(-L2, rnd_int(dz * B2), dz);
                    const float ex = fmaxf(fabsf(dx) - hw.x - h.x, 0.f), ey = fmaxf(fabsf(dy) - hw.y - h.y, 0.f);
                    const float ez = fmaxf(fabsf(dz) - hw.z - h.z, 0.f);
                    ok = ex * ex + ey * ey + ez * ez <= rb2;
                }
                const unsigned b = __ballot_sync(0xffffffffu, ok);
                if (ok) sJ[w][nj + __popc(b & ((1u << lane) - 1u))] = J;
                nj += __popc(b);
            }
        }
        if (lane == 0) swarp[w] = nj;
        __syncthreads();
        if (tid == 0) {
            int o = 0;
            for (int q = 0; q < 4; ++q) { soff[q] = o; o += swarp[q]; }
            soff[4] = o;
        }
        __syncthreads();
        const int ntot = 8 * soff[4];                    // candidate atoms
        for (int c0 = 0; c0 < ntot; c0 += ccap) {
            if (LOWER) ++pieces;
            const int nc = min(ccap, ntot - c0);
            const int part = ((nc + 127) >> 7) << 5;     // a warp's share, a multiple of 32
            const int lo = w * part, hi = min(nc, lo + part);
            for (int q = tid; q < 4 * 256; q += 128) (&hist[0][0])[q] = 0;
            __syncthreads();
            // 2: masks of this warp's candidates, compacted in order
            int ne = 0;
            unsigned known = __reduce_or_sync(0xffffffffu, up);
            // slot, position and flag of a candidate, loaded one iteration ahead
            auto fetch = [&](int k, int& t, float4& p, bool& hj) {
                t = 0;
                p.w = __int_as_float(-1);
                hj = true;
                if (k < hi) {
                    const int g = (c0 + k) >> 3;
                    const int q = (g >= soff[1]) + (g >= soff[2]) + (g >= soff[3]);
                    t = 8 * sJ[q][g - soff[q]] + (k & 7);
                    p = a.pf[t];
                    hj = a.hasup[t] != 0;
                }
            };
            int tn;
            float4 pn;
            bool hn;
            fetch(lo + lane, tn, pn, hn);
            for (int k0 = lo; k0 < hi; k0 += 32) {
                const int t = tn;
                const float4 pj = pn;
                const bool hj = hn;
                fetch(k0 + 32 + lane, tn, pn, hn);
                unsigned mask = 0;
                {
                    const int jo = __float_as_int(pj.w);
                    if (jo >= 0) {
                        float near = 1e30f;              // smallest | r^2 - mid |
                        float jx = pj.x, jy = pj.y, jz = pj.z;
                        if (FRAME) {
                            jx -= ctr.x; jy -= ctr.y; jz -= ctr.z;
                            jx = fmaf(-L0, rnd_int(jx * B0), jx);
                            jy = fmaf(-L1, rnd_int(jy * B1), jy);
                            jz = fmaf(-L2, rnd_int(jz * B2), jz);
                        }
                        const float2 nx2 = make_float2(-jx, -jx), ny2 = make_float2(-jy, -jy), nz2 = make_float2(-jz, -jz);
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            const float4 xy = sxy[p], zz = sz[p];
                            float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), nx2);
                            float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), ny2);
                            float2 dz = __fadd2_rn(make_float2(zz.x, zz.y), nz2);
                            if (!FRAME) {
                                dx.x = fmaf(-L0, rnd_int(dx.x * B0), dx.x); dx.y = fmaf(-L0, rnd_int(dx.y * B0), dx.y);
                                dy.x = fmaf(-L1, rnd_int(dy.x * B1), dy.x); dy.y = fmaf(-L1, rnd_int(dy.y * B1), dy.y);
                                dz.x = fmaf(-L2, rnd_int(dz.x * B2), dz.x); dz.y = fmaf(-L2, rnd_int(dz.y * B2), dz.y);
                            }
                            const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
                            const float2 off = __fadd2_rn(r2, make_float2(-mid, -mid));
                            if (off.x < 0.f) mask |= 1u << (2 * p);
                            if (off.y < 0.f) mask |= 2u << (2 * p);
                            near = fminf(near, fminf(fabsf(off.x), fabsf(off.y)));
                        }
                        unsigned valid = vmask;
                        if ((t >> 3) == cl) valid &= (1u << (t & 7)) - 1u;   // each pair once: t above the atom
                        mask &= valid;
                        if (!(near > band)) {     // near rcut_book: the reference's exact FP64 test decides
                            const double* pt = a.pos_s + 3 * (size_t)t;
                            const double x = pt[0], y = pt[1], z = pt[2];
#pragma unroll
                            for (int ii = 0; ii < 8; ++ii) {
                                const double* pi = a.pos_s + 3 * (size_t)(s0 + ii);
                                const double r0 = mi_exact(__dsub_rn(pi[0], x), sbox[0], sbox[3]);
                                const double r1 = mi_exact(__dsub_rn(pi[1], y), sbox[1], sbox[4]);
                                const double r2 = mi_exact(__dsub_rn(pi[2], z), sbox[2], sbox[5]);
                                const double dr = __dadd_rn(__dadd_rn(__dmul_rn(r0, r0), __dmul_rn(r1, r1)),
                                                            __dmul_rn(r2, r2));
                                mask = (mask & ~(1u << ii)) | (dr < a.sqcut ? 1u << ii : 0u);
                            }
                            mask &= valid;
                        }
                        if (mask && ((sbloom[(jo >> 9) & 63] >> ((jo >> 4) & 31)) & 1u)) {
                            unsigned m = mask;
                            while (m) {
                                const int ii = __ffs(m) - 1;
                                m &= m - 1;
                                const int2 rg = srng[ii];
                                if (jo < rg.x || jo > rg.y) continue;
                                bool ex = false;
                                if (snex[ii] <= CL_EXCAP)
                                    for (int q = 0; q < snex[ii]; ++q) ex = ex || sexc[ii][q] == jo;
                                else ex = is_excluded(a.exs_idx, a.exs_list, sio[ii], jo);
                                if (ex) mask &= ~(1u << ii);
                            }
                        }
                        // atoms with a partner of higher index, until all are known
                        if (mask) {
                            if (!hj || (mask & ~known)) {
                                unsigned gt = 0;
#pragma unroll
                                for (int ii = 0; ii < 8; ++ii) gt |= (jo > sio[ii] ? 1u : 0u) << ii;
                                up |= gt & mask;
                                if (!hj && (mask & ~gt)) a.hasup[t] = 1;
                            }
                            npair += __popc(mask);
                        }
                    }
                }
                known |= __reduce_or_sync(0xffffffffu, up);
                const unsigned b = __ballot_sync(0xffffffffu, mask != 0);
                if (mask) {
                    cand[lo + ne + __popc(b & ((1u << lane) - 1u))] = (mask << 24) | (unsigned)t;
                    atomicAdd(&hist[w][sbin[mask]], 1);
                }
                ne += __popc(b);
            }
            if (lane == 0) sne[w] = ne;
            __syncthreads();
            // 3: first position of every (bin, warp), then the ranks
            int v[2][4], tot = 0;
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int q = 0; q < 4; ++q) { v[e][q] = hist[q][2 * tid + e]; tot += v[e][q]; }
            int inc = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) swarp[w] = inc;
            __syncthreads();
            int run = count + inc - tot;
            for (int q = 0; q < w; ++q) run += swarp[q];
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int q = 0; q < 4; ++q) { hist[q][2 * tid + e] = run; run += v[e][q]; }
            __syncthreads();
            int* __restrict__ bin = hist[w];
            for (int k0 = 0; k0 < ne; k0 += 32) {
                const int k = k0 + lane;
                const bool ok = k < ne;
                const unsigned e = ok ? cand[lo + k] : 0u;
                const unsigned kb = ok ? sbin[e >> 24] : 256u + lane;
                const unsigned grp = __match_any_sync(0xffffffffu, kb);
                const int rank = __popc(grp & ((1u << lane) - 1u));
                const int base = ok ? bin[kb] : 0;
                __syncwarp();
                if (ok) {
                    if (base + rank < a.ccap) row[base + rank] = (int)e;
                    if (rank == 0) bin[kb] = base + __popc(grp);
                }
                __syncwarp();
            }
            count += sne[0] + sne[1] + sne[2] + sne[3];
            __syncthreads();                             // cand, hist, sne are reused
        }
        __syncthreads();                                 // sJ, soff are reused
    }
    up = __reduce_or_sync(0xffffffffu, up);
    npair = warp_sum(npair);
    if (lane < 8 && ((up >> lane) & 1u)) a.hasup[s0 + lane] = 1;
    if (lane == 0 && npair) atomicAdd(&a.counters[0], (unsigned long long)npair);
    if (tid == 0) {
        a.ccnt[cl] = min(count, a.ccap) | (LOWER && pieces > 1 ? a.mark : 0);
        if (count > a.ccap) atomicOr(a.status, ST_LIST_OVERFLOW);
        atomicMax(&a.counters[1], (unsigned long long)count);
    }
}

// Rows that k_build_clist sorted in pieces: one stable sort over the whole row
// (a warp per row; rows that are not marked are left alone).
__global__ void __launch_bounds__(128) k_sort_rows(int* __restrict__ clist, int* __restrict__ ccnt, int ncl, int ccap) {
    extern __shared__ int srow[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, cl = blockIdx.x * 4 + w;
    if (cl >= ncl || ccnt[cl] >= 0) return;
    int* buf = srow + (size_t)w * (ccap + 256);
    int* bin = buf + ccap;
    int* row = clist + (size_t)cl * ccap;
    const int n = ccnt[cl] & ~ROW_PIECES;
    for (int q = lane; q < 256; q += 32) bin[q] = 0;
    __syncwarp();
    if (lane == 0) ccnt[cl] = n;
    for (int k = lane; k < n; k += 32) {
        const int e = row[k];
        buf[k] = e;
        atomicAdd(&bin[mask_bin((unsigned)e >> 24)], 1);
    }
    __syncwarp();
    int v[8], tot = 0;                               // exclusive prefix sums of the bins, 8 a lane
#pragma unroll
    for (int q = 0; q < 8; ++q) { v[q] = bin[8 * lane + q]; tot += v[q]; }
    int run = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
    }
    run -= tot;
#pragma unroll
    for (int q = 0; q < 8; ++q) { bin[8 * lane + q] = run; run += v[q]; }
    __syncwarp();
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        const bool in = k < n;
        const int e = in ? buf[k] : 0;
        const unsigned kb = in ? mask_bin((unsigned)e >> 24) : 256u + lane;
        const unsigned grp = __match_any_sync(0xffffffffu, kb);
        const int rank = __popc(grp & ((1u << lane) - 1u));
        const int base = in ? bin[kb] : 0;
        __syncwarp();
        if (in) {
            row[base + rank] = e;
            if (rank == 0) bin[kb] = base + __popc(grp);
        }
        __syncwarp();
    }
}

// atoms i < n-1 without a partner of higher index (one sentinel row each)
__global__ void k_count_noup(const unsigned char* __restrict__ hasup, const int* __restrict__ iperm, int m,
                             unsigned long long* counters) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned v = (i < m && !hasup[iperm[i]]) ? 1u : 0u;
    unsigned w = __popc(__ballot_sync(0xffffffffu, v));
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(&counters[2], (unsigned long long)w);
}

pgk_status launch_transcor(pgk_ctx* c) {
    if (c->nmole == 0) return PGK_OK;
    k_transcor<<<(c->nmole + 255) / 256, 256, 0, c->st>>>(c->pos, c->mol_idx, c->mol_list, c->nmole, c->dyn);
    PGK_LAUNCHED(c);
    PGK_CUDA(c, cudaGetLastError());
    return PGK_OK;
}

// list-mode rule of rdscript.F90:1595-1610
static int list_mode_for(const pgk_ctx* c, const double* box, int* nc) {
    for (int d = 0; d < 3; ++d) nc[d] = (int)(box[d] / c->prm.rcut_book);
    if (c->prm.list_mode == PGK_LIST_CELL) return PGK_LIST_CELL;
    if (c->prm.list_mode == PGK_LIST_ALLPAIR) return PGK_LIST_ALLPAIR;
    if (nc[0] < 3 || nc[1] < 3 || nc[2] < 3 || (long long)nc[0] * nc[1] * nc[2] <= 27) return PGK_LIST_ALLPAIR;
    return PGK_LIST_CELL;
}

// (re)allocate the sorted/padded arrays for up to npad_cap slots
// cluster rows (book and pruned) for npad_cap/8 clusters of ccap entries
static pgk_status alloc_rows(pgk_ctx* c) {
    pgk_dfree(c, c->clist); pgk_dfree(c, c->plist);
    c->clist = nullptr; c->plist = nullptr;
    const size_t bytes = sizeof(int) * (size_t)(c->npad_cap / 8) * c->ccap;
    if (pgk_dmalloc(c, &c->clist, bytes) != cudaSuccess) {
        c->clist = nullptr;
        return pgk_fail(c, PGK_E_NOMEM, "cluster pair list exceeds device memory");
    }
    c->pcap = ((c->ccap + c->pseg - 1) / c->pseg + 31) / 32 * 32;
    const size_t pbytes = sizeof(int) * (size_t)(c->npad_cap / 8) * c->pseg * c->pcap;
    if (c->prune_buffer > 0.f && pgk_dmalloc(c, &c->plist, pbytes) != cudaSuccess) {
        c->plist = nullptr;
        return pgk_fail(c, PGK_E_NOMEM, "pruned pair list exceeds device memory");
    }
    return PGK_OK;
}

static pgk_status ensure_sorted_capacity(pgk_ctx* c, int npad_cap) {
    if (npad_cap <= c->npad_cap) return PGK_OK;
    pgk_dfree(c, c->perm); pgk_dfree(c, c->pos_s); pgk_dfree(c, c->typ_s); pgk_dfree(c, c->xq); pgk_dfree(c, c->xq64);
    pgk_dfree(c, c->pf_s); pgk_dfree(c, c->cbox); pgk_dfree(c, c->hasup);
    c->hasup = nullptr; c->pf_s = nullptr; c->cbox = nullptr;
    pgk_dfree(c, c->ccnt); pgk_dfree(c, c->clist); pgk_dfree(c, c->fsort); pgk_dfree(c, c->plist); pgk_dfree(c, c->pcnt);
    pgk_dfree(c, c->xq_prune);
    c->perm = nullptr; c->pos_s = nullptr; c->typ_s = nullptr; c->xq = nullptr; c->xq64 = nullptr;
    c->ccnt = nullptr; c->clist = nullptr; c->fsort = nullptr; c->plist = nullptr; c->pcnt = nullptr;
    c->xq_prune = nullptr;
    int ncl = npad_cap / 8;
    PGK_CUDA(c, pgk_dmalloc(c, &c->perm, sizeof(int) * npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->pos_s, sizeof(double) * 3 * npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->typ_s, sizeof(int) * npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->pf_s, sizeof(float4) * npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->hasup, npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->cbox, sizeof(float4) * 2 * ncl));
    PGK_CUDA(c, pgk_dmalloc(c, &c->fsort, sizeof(long long) * 3 * (size_t)npad_cap));
    PGK_CUDA(c, cudaMemsetAsync(c->fsort, 0, sizeof(long long) * 3 * (size_t)npad_cap, c->st));
    if (c->mixed()) PGK_CUDA(c, pgk_dmalloc(c, &c->xq, sizeof(int4) * npad_cap));
    else PGK_CUDA(c, pgk_dmalloc(c, &c->xq64, sizeof(double4) * npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->ccnt, sizeof(int) * ncl));
    if (c->prune_buffer > 0.f) {
        const size_t xb = (c->mixed() ? sizeof(int4) : sizeof(double4)) * (size_t)npad_cap;
        PGK_CUDA(c, pgk_dmalloc(c, &c->pcnt, sizeof(int) * ncl * c->pseg));
        PGK_CUDA(c, pgk_dmalloc(c, &c->xq_prune, xb));
        PGK_CUDA(c, cudaMemsetAsync(c->xq_prune, 0, xb, c->st));
    }
    c->npad_cap = npad_cap;
    return alloc_rows(c);
}

// pgk_ctx::plain_order from here on
pgk_status keep_plain_order(pgk_ctx* c) {
    if (!c->mixed() || c->plain_order) return PGK_OK;
    c->plain_order = true;
    c->pseg = 1;                            // the allocated segments of a row hold the whole of it (alloc_rows)
    c->pcap = c->ccap;
    if (c->prune_buffer > 0.f) PGK_CUDA(c, cudaMemsetAsync(&c->prune->force, 1, 1, c->st));   // re-prune
    ++c->list_epoch;                        // captured steps hold the segments
    return PGK_OK;
}

pgk_status launch_mklist(pgk_ctx* c) {
    int n = c->natom;
    // the box may have changed on the device (MTK): read it back
    PGK_CUDA(c, cudaMemcpyAsync(&c->hdyn, c->dyn, sizeof(DynState), cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaStreamSynchronize(c->st));
    int nc[3];
    int mode = list_mode_for(c, c->hdyn.box, nc);
    if (mode == PGK_LIST_CELL && (nc[0] < 3 || nc[1] < 3 || nc[2] < 3))
        return pgk_fail(c, PGK_E_CELL_OVERFLOW, "mklist_cell needs at least 3 cells per direction");
    for (int d = 0; d < 3; ++d) nc[d] = std::max(1, nc[d]);
    long long ncells = (long long)nc[0] * nc[1] * nc[2];
    if (ncells > c->maxcells) {
        pgk_dfree(c, c->cell_cnt); pgk_dfree(c, c->cell_start); pgk_dfree(c, c->cell_fill);
        c->maxcells = (int)ncells;
        PGK_CUDA(c, pgk_dmalloc(c, &c->cell_cnt, sizeof(int) * (ncells + 1)));
        PGK_CUDA(c, pgk_dmalloc(c, &c->cell_start, sizeof(int) * (ncells + 1)));
        PGK_CUDA(c, pgk_dmalloc(c, &c->cell_fill, sizeof(int) * (ncells + 1)));
    }
    long long npad_max = (long long)n + 7 * ncells;
    if (npad_max >= (1 << 24)) return pgk_fail(c, PGK_E_UNSUPPORTED, "more than 2^24 padded atom slots");
    pgk_status s;
    if ((npad_max + 7) / 8 * 8 > c->npad_cap) {
        if ((s = ensure_sorted_capacity(c, (int)((npad_max + 7) / 8 * 8)))) return s;
    }
    DynState& h = c->hdyn;
    for (int d = 0; d < 3; ++d) { h.ncell[d] = nc[d]; h.cellsize[d] = h.box[d] / (double)nc[d]; }
    h.list_mode_used = mode;
    PGK_CUDA(c, cudaMemcpyAsync(c->dyn, &h, sizeof(DynState), cudaMemcpyHostToDevice, c->st));
    for (int attempt = 0; attempt < 3; ++attempt) {
        PGK_CUDA(c, cudaMemsetAsync(c->cell_cnt, 0, sizeof(int) * (ncells + 1), c->st));
        PGK_CUDA(c, cudaMemsetAsync(c->counters, 0, 4 * sizeof(unsigned long long), c->st));
        int tb = 256, nb = (n + tb - 1) / tb;
        k_cell_assign<<<nb, tb, 0, c->st>>>(c->pos, n, c->dyn, c->cell_of, c->cell_cnt, c->subkey);
        k_cell_scan<<<1, 1024, 0, c->st>>>(c->cell_cnt, c->cell_start, c->cell_fill, (int)ncells, c->status);
        k_cell_place<<<nb, tb, 0, c->st>>>(c->cell_of, n, c->cell_fill, c->perm);
        k_cell_sort<<<(int)ncells, 512, 0, c->st>>>(c->perm, c->cell_start, c->cell_cnt, c->subkey, (int)ncells);
        int npad = 0;
        PGK_CUDA(c, cudaMemcpyAsync(&npad, c->cell_start + ncells, sizeof(int), cudaMemcpyDeviceToHost, c->st));
        PGK_CUDA(c, cudaStreamSynchronize(c->st));
        c->npad = npad;
        c->ncl = npad / 8;
        k_sorted_gather<<<(npad + 255) / 256, 256, 0, c->st>>>(c->perm, npad, c->pos, c->typ, c->dyn, c->iperm,
                                                               c->pos_s, c->typ_s, c->pf_s, c->cbox);
        double sq = c->prm.rcut_book * c->prm.rcut_book;
        // screening margin on r^2: FP32 coordinates (up to twice the box) carry
        // 2^-24 relative error each, a distance component up to 4x that
        const double lmax = std::max(h.box[0], std::max(h.box[1], h.box[2]));
        const double eps_pos = 4.0 * 5.96e-8 * 2.0 * lmax;
        const double scr = std::max(0.01, 2.0 * 2.0 * c->prm.rcut_book * 1.7321 * eps_pos + 1.0e-3);
        PGK_CUDA(c, cudaMemsetAsync(c->hasup, 0, (size_t)npad, c->st));
        ClistArgs a;
        a.pf = c->pf_s; a.cbox = c->cbox; a.pos_s = c->pos_s;
        a.cell_of = c->cell_of; a.cell_start = c->cell_start; a.cell_cnt = c->cell_cnt;
        a.exs_idx = c->exs_idx; a.exs_list = c->exs_list; a.exs_rng = c->exs_rng;
        const size_t ssm = (size_t)4 * (c->ccap + 256) * sizeof(int);      // k_sort_rows
        const bool sort = c->plain_order && ssm <= 160 * 1024;
        a.ncl = c->ncl; a.ccap = c->ccap; a.mark = sort ? ROW_PIECES : 0;
        a.sqcut = sq; a.rbox = (float)(c->prm.rcut_book + 0.05);
        a.sqlo = (float)(sq * (1.0 - 1.0e-5) - scr); a.sqhi = (float)(sq * (1.0 + 1.0e-5) + scr);
        a.clist = c->clist; a.ccnt = c->ccnt; a.hasup = c->hasup; a.counters = c->counters; a.status = c->status;
        // the cluster frame is exact when rcut_book plus half a cell stays below half the box
        bool frame = true;
        for (int d = 0; d < 3; ++d)
            frame = frame && nc[d] >= 4 && c->prm.rcut_book + 0.5 * h.cellsize[d] + 0.1 < 0.5 * h.box[d];
        auto* build = c->plain_order ? (frame ? k_build_clist<true, true> : k_build_clist<false, true>)
                                     : (frame ? k_build_clist<true, false> : k_build_clist<false, false>);
        build<<<c->ncl, 128, 0, c->st>>>(a, c->dyn);
        if (sort) {
            PGK_CUDA(c, smem_limit(k_sort_rows, ssm));
            k_sort_rows<<<(c->ncl + 3) / 4, 128, ssm, c->st>>>(c->clist, c->ccnt, c->ncl, c->ccap);
            PGK_LAUNCHED(c);
        }
        if (n > 1) k_count_noup<<<(n - 1 + 255) / 256, 256, 0, c->st>>>(c->hasup, c->iperm, n - 1, c->counters);
        c->launches += 7;
        PGK_CUDA(c, cudaGetLastError());
        unsigned long long cnt[4];
        unsigned st;
        PGK_CUDA(c, cudaMemcpyAsync(cnt, c->counters, sizeof(cnt), cudaMemcpyDeviceToHost, c->st));
        PGK_CUDA(c, cudaMemcpyAsync(&st, c->status, sizeof(st), cudaMemcpyDeviceToHost, c->st));
        PGK_CUDA(c, cudaStreamSynchronize(c->st));
        if (st & ST_CELL_OVERFLOW)
            return pgk_fail(c, PGK_E_CELL_OVERFLOW, "number of atoms in a cell exceeds the device maximum");
        if (st & ST_LIST_OVERFLOW) {
            // grow the cluster rows and rebuild (the reference STOPs here)
            unsigned zero = 0;
            PGK_CUDA(c, cudaMemsetAsync(c->status, 0, sizeof(zero), c->st));
            // a quarter of headroom above the longest row, so the rows of
            // later builds (density fluctuations) rarely force another regrowth
            c->ccap = (int)(((long long)cnt[1] * 5 / 4 + 32 + 31) / 32 * 32);
            if ((s = alloc_rows(c))) return s;
            continue;
        }
        h.nlistnball = (long long)(cnt[0] + cnt[2]);
        h.nmaxrow = (int)cnt[1];
        PGK_CUDA(c, cudaMemcpyAsync(&c->dyn->nlistnball, &h.nlistnball, sizeof(long long),
                                    cudaMemcpyHostToDevice, c->st));
        c->list_valid = true;
        ++c->list_epoch;
        if (c->prune_buffer > 0.f) PGK_CUDA(c, cudaMemsetAsync(&c->prune->force, 1, 1, c->st));   // re-prune
        return pair_autotune(c);      // once per context
    }
    return pgk_fail(c, PGK_E_LIST_OVERFLOW, "pair list overflow after regrowth");
}

// Reference CSR (nb_indexall / nb_listall) from the device cluster rows:
// every stored pair goes to the row of its lower original index, then each
// row is ordered like the reference (27-cell z-y-x scan or ascending j).
pgk_status export_nblist(pgk_ctx* c, int32_t* nb_index, int32_t* nb_list, int64_t cap, int64_t* nl) {
    if (!c->list_valid) return pgk_fail(c, PGK_E_INVALID, "no pair list has been built");
    int n = c->natom, npad = c->npad, ncl = c->ncl;
    std::vector<int> ccnt(ncl), perm(npad), cell_of(n);
    std::vector<int> rows((size_t)ncl * c->ccap);
    PGK_CUDA(c, cudaMemcpyAsync(ccnt.data(), c->ccnt, sizeof(int) * ncl, cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaMemcpyAsync(perm.data(), c->perm, sizeof(int) * npad, cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaMemcpyAsync(cell_of.data(), c->cell_of, sizeof(int) * n, cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaMemcpyAsync(rows.data(), c->clist, sizeof(int) * rows.size(), cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaMemcpyAsync(&c->hdyn, c->dyn, sizeof(DynState), cudaMemcpyDeviceToHost, c->st));
    PGK_CUDA(c, cudaStreamSynchronize(c->st));
    const DynState& h = c->hdyn;
    int nc0 = h.ncell[0], nc1 = h.ncell[1], nc2 = h.ncell[2];
    bool cellmode = h.list_mode_used == PGK_LIST_CELL;
    std::vector<std::vector<int>> part(n);
    for (int cl = 0; cl < ncl; ++cl)
        for (int k = 0; k < ccnt[cl]; ++k) {
            unsigned e = (unsigned)rows[(size_t)cl * c->ccap + k];
            int j = perm[e & 0xFFFFFFu];
            for (int b = 0; b < 8; ++b) {
                if (!((e >> (24 + b)) & 1u)) continue;
                int i = perm[8 * cl + b];
                if (i < j) part[i].push_back(j); else part[j].push_back(i);
            }
        }
    long long pos = 0;
    std::vector<std::pair<long long, int>> tmp;
    for (int i = 0; i < n - 1; ++i) {
        tmp.clear();
        int ki = cell_of[i];
        int ix = ki % nc0, iy = (ki / nc0) % nc1, iz = ki / (nc0 * nc1);
        for (int j : part[i]) {
            long long ord = j;
            if (cellmode) {   // 27-cell scan order z, y, x (mklist_cell.F90:218-273)
                int kj = cell_of[j];
                int jx = kj % nc0, jy = (kj / nc0) % nc1, jz = kj / (nc0 * nc1);
                int dx = ((jx - ix) % nc0 + nc0) % nc0; if (dx == nc0 - 1) dx = -1;
                int dy = ((jy - iy) % nc1 + nc1) % nc1; if (dy == nc1 - 1) dy = -1;
                int dz = ((jz - iz) % nc2 + nc2) % nc2; if (dz == nc2 - 1) dz = -1;
                long long slot = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
                ord = slot * (long long)n + j;
            }
            tmp.push_back({ord, j});
        }
        std::sort(tmp.begin(), tmp.end());
        if (nb_index) nb_index[i] = (int32_t)(pos + 1);
        if (tmp.empty()) {
            if (nb_list && pos < cap) nb_list[pos] = 0;
            ++pos;
        } else {
            for (auto& p : tmp) {
                if (nb_list && pos < cap) nb_list[pos] = p.second + 1;
                ++pos;
            }
        }
    }
    if (nb_index && n >= 1) nb_index[n - 1] = (int32_t)(pos + 1);
    *nl = pos;
    if (nb_list && pos > cap) return pgk_fail(c, PGK_E_INVALID, "nb_listall capacity too small");
    return PGK_OK;
}
