// k_heatf.cu -- heat flux of the -DHF build and the region Langevin thermostat.
//
//   calcom.F90                  molecule centres of mass, velocities (k_calcom)
//   ewaldr_hf.F90:213-520       per-atom pair potentials and the calvirihf
//                               virial of every list pair (k_hf_pair)
//   cal*_hf.F90                 bonded parts (k_bonded.cu, launch_bonded_hf)
//   calheatf.F90:365-1466       region sums of the kinetic, potential and
//                               virial transport terms (k_flux_*)
//   langevin_regist.F90         region of each atom (k_lt_regist)
//   langevin_region.F90         half steps with random and friction terms
//                               (k_langevin)
//
// The per-atom arrays stay on the device in original atom order:
// pot[8][N] and the z column of the per-atom virial W[8][nreg][3][N]
// (category-major).  They are written for the last heat-flux evaluation of a
// call; the records come from region sums formed term by term (k_flux_*).
//
// k_hf_pair walks the same 8-atom cluster rows as the pair kernel, twice: lanes
// own entries and sum the neighbour's shares, then lanes own cluster atoms and
// sum theirs.
// Pair distances and scalar factors are FP32 in mixed precision and FP64
// otherwise; velocities, region geometry and the sums in memory are FP64.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "pgk_ctx.cuh"
#include "pgk_hf.cuh"

// ---- calcom.F90 / molecule velocities of calheatf.F90:556-607 -------------------
__device__ __forceinline__ void mole_mean(const double* __restrict__ x, const double* __restrict__ mass,
                                          const int* __restrict__ mol_list, int b, int e, double* c) {
    if (e - b == 1) {
        int i = mol_list[b];
        c[0] = x[3 * i]; c[1] = x[3 * i + 1]; c[2] = x[3 * i + 2];
    } else {
        double ms = 0.0;
        c[0] = c[1] = c[2] = 0.0;
        for (int q = b; q < e; ++q) {
            int i = mol_list[q];
            double mi = mass[i];
            ms = ms + mi;
            c[0] = c[0] + mi * x[3 * i]; c[1] = c[1] + mi * x[3 * i + 1]; c[2] = c[2] + mi * x[3 * i + 2];
        }
        double inv = 1.0 / ms;
        c[0] = c[0] * inv; c[1] = c[1] * inv; c[2] = c[2] * inv;
    }
}
// vel null: the centres only
__global__ void k_calcom(const double* __restrict__ pos, const double* __restrict__ vel,
                          const double* __restrict__ mass, const int* __restrict__ mol_idx,
                          const int* __restrict__ mol_list, int nmole, const DynState* __restrict__ dyn,
                          double* __restrict__ com, double* __restrict__ cvel) {
    pdl_enter();
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmole) return;
    const int b = mol_idx[m], e = mol_idx[m + 1];
    double c[3];
    mole_mean(pos, mass, mol_list, b, e, c);
    for (int d = 0; d < 3; ++d) com[3 * m + d] = hf_wrap1(c[d], dyn->box[d]);
    if (!vel) return;
    mole_mean(vel, mass, mol_list, b, e, c);
    for (int d = 0; d < 3; ++d) cvel[3 * m + d] = c[d];
}

// molecule tag of a sorted slot: molecule number, and whether the heat-flux z
// is the molecule's (the sign bit) and lies exactly on a region's plane
#define HF_MS_ID 0x3fffffff
#define HF_MS_PLANE 0x40000000
__device__ __forceinline__ int hf_tag(const HfDev& h, int i, unsigned planes) {
    return h.mol_of[i] | (planes ? HF_MS_PLANE : 0) | (h.hftyp[i] == PGK_HFTYP_MOLE ? (int)0x80000000 : 0);
}

// heat-flux z, molecule tag and region bits of every sorted slot
__global__ void k_hf_slots(const int* __restrict__ perm, int npad, const double* __restrict__ pos, HfDev h,
                           const DynState* __restrict__ dyn, double* __restrict__ zs, int* __restrict__ ms,
                           uint4* __restrict__ bs) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= npad) return;
    int i = perm[s];
    if (i < 0) { zs[s] = 0.0; ms[s] = HF_MS_ID; bs[s] = make_uint4(0u, 0u, 0u, 0u); return; }
    const double z = hf_z(h, pos, i, dyn->box[2]);
    const uint4 b = flux_bits(h, i, z, dyn->box[2]);
    zs[s] = z;
    bs[s] = b;
    ms[s] = hf_tag(h, i, b.w);
}

// ---- calheatf.F90, volume-based, z components --------------------------------
// A record needs the region sums only, and they are linear in the terms
// (FluxDev), so they are formed pair by pair and bonded term by bonded term
// from the velocities; the per-atom arrays (190 MB for 43,200 atoms and 23
// regions, FP64 atomics per pair, category, region and axis) are written for
// the evaluation that pgk_get_hf_atm can read, not for every record.

// Per atom: heat-flux z, molecule tag, velocities and region bits into the
// sorted slots (iperm; null: no pair list), kinetic transport into the sums.
__global__ void __launch_bounds__(256) k_flux_atoms(const double* __restrict__ pos, const double* __restrict__ mass,
                                                    const int* __restrict__ iperm, FluxDev f,
                                                    const DynState* __restrict__ dyn, double* __restrict__ zs,
                                                    int* __restrict__ ms, double4* __restrict__ vs,
                                                    uint4* __restrict__ bs) {
    pdl_enter();
    __shared__ double sk[PGK_HF_MAX_REGIONS];
    const int nreg = f.h.nreg;
    if (threadIdx.x < PGK_HF_MAX_REGIONS) sk[threadIdx.x] = 0.0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double kz = 0.0;
    unsigned in = 0u;
    if (i < f.h.natom) {
        const double vx = f.vel[3 * i], vy = f.vel[3 * i + 1], vz = f.vel[3 * i + 2];
        const double z = hf_z(f.h, pos, i, dyn->box[2]), pvz = flux_vz(f, i);
        const uint4 m = flux_bits(f.h, i, z, dyn->box[2]);
        in = m.z;
        kz = 0.5 * mass[i] * (vx * vx + vy * vy + vz * vz) * pvz;
        if (iperm) {
            const int s = iperm[i];
            zs[s] = z;
            ms[s] = hf_tag(f.h, i, m.w);
            bs[s] = m;
            for (int q = 0; q < FLUX_SUMS; ++q) f.sum[(size_t)FLUX_SUMS * s + q] = 0.0;
            vs[s] = make_double4(vx, vy, vz, pvz);
        }
    }
    unsigned any = __reduce_or_sync(0xffffffffu, in);
    while (any) {
        const int r = __ffs(any) - 1;
        any &= any - 1;
        const double s = warp_sum((in >> r) & 1u ? kz : 0.0);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sk[r], s);
    }
    __syncthreads();
    double* acc = f.acc + (size_t)(blockIdx.x % FLUX_COPIES) * nreg * FLUX_COLS;
    if (threadIdx.x < nreg && sk[threadIdx.x] != 0.0) atomicAdd(acc + threadIdx.x * FLUX_COLS, sk[threadIdx.x]);
}

// Pair part of the region sums over the cluster rows (the book rows, or the
// pruned rows while they are current): one warp per (cluster, row segment),
// one lane per entry, a loop over the entry's mask bits.  A pair's share of
// region r is s (C_r(z_i) - C_r(z_j)) / 2 with s = f_ij . (v_i + v_j) and
// C_r(z) = z clamped to the slab -- the plane-crossing cases of calvirihf as
// one difference.  It is linear in s, so the pairs only add s to one atom and
// take it from the other, next to their energies (FluxDev.sum), and the
// regions are a sum over the atoms (k_flux_regions).  The cluster atoms' sums
// stay in registers until the end of the row; an entry's go out once per
// entry, those of a pair inside one molecule at once (they are a class of
// their own).  An atom exactly on a plane has hf_frag's own cases: the virial
// part of its pairs goes to the regions directly.
// A pair's distance and scalar factors are T (FP32 in mixed precision), and so
// are a lane's partial sums of the cluster atoms' energies (at most a row's
// entries / 32 terms; FP64 there changes no digit of the error and costs 5 %);
// velocities, f . v, the entries' sums and all sums over lanes, rows, atoms and
// regions are FP64.  Error of the records against FP64 as with the divided 1/r
// and per-atom FP64 virials: 2,592 atoms of propanol, LJ virials 9e-7 and 4e-7
// of the largest region.
// Bound by latency at 16 warps per SM (128 registers): issue 49 % busy, stalls on
// the entries' records and fixed latencies.  Measured, mixed: 43,200-atom slab,
// 23 regions: 0.177 ms and 0.012 ms for the regions (0.33 ms with the regions
// inside the pair loop, four a walk); 8,232-atom water box, one region: 0.045 ms.  (Velocities and f . v in FP32: 0.165 and 0.042 ms, and 1.2 to 1.5 times
// the error.)
// Rows are cut into segments until 16 warps per SM have work (small boxes).
struct FluxPairArgs {
    const int* rows; const int* cnt; int ccap; int ncl; int nseg;
    int cut;                     // rows, cnt: nseg segments of ccap entries per cluster, else whole rows
    const int* typ_s; const int* perm; int ntyp;
    const double* zs; const int* ms; const double4* vs; const uint4* bs;
    double rr2, rl2, rmax2;      // rr2: sqrt_le_limit(rrcut) in FP64
};

template <bool MIXED> struct FluxT { typedef float T; };
template <> struct FluxT<false> { typedef double T; };

// 1/r and 1/r^2.  FP32: the approximate root (2^-22.9) and one Newton step
// y (1 + e/2) with e = 1 - r^2 y^2 exact to 2^-47 (the product's rounding is
// taken back), so 1/r is off by its last rounding, and one residual step for
// the square: no less than a divided root and a division, in half as many
// instructions.
__device__ __forceinline__ void flux_rinv(float r2, float& rinv, float& rinv2) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
    const float h = r2 * y, hl = fmaf(r2, y, -h);
    const float e = fmaf(-hl, y, fmaf(-h, y, 1.f));
    rinv = fmaf(0.5f * y, e, y);
    const float q = rinv * rinv;
    rinv2 = fmaf(fmaf(-r2, q, 1.f), q, q);
}
__device__ __forceinline__ void flux_rinv(double r2, double& rinv, double& rinv2) {
    rinv = rsqrt(r2);
    rinv2 = rinv * rinv;
}

// One pair's terms of the per-atom arrays (categories Coulomb, LJ): energies
// and half forces; false beyond both cutoffs.
template <bool MIXED> struct HfTerm {
    typename FluxT<MIXED>::T pc, pl, fc[3], fl[3];
};
struct HfBox { double L0, L1, L2, B0, B1, B2; };
template <bool MIXED>
__device__ __forceinline__ bool hf_term(const int4& qi, const double4& pi, const int4& qj, const double4& pj,
                                        const FluxPairArgs& a, const HfBox& b, int lj, const float2* lj32,
                                        const double2* lj64, HfTerm<MIXED>& o) {
    typedef typename FluxT<MIXED>::T T;
    T dx, dy, dz, qq;
    if (MIXED) {
        dx = (T)(qi.x - qj.x) * (T)(b.L0 * (1.0 / 4294967296.0));
        dy = (T)(qi.y - qj.y) * (T)(b.L1 * (1.0 / 4294967296.0));
        dz = (T)(qi.z - qj.z) * (T)(b.L2 * (1.0 / 4294967296.0));
        qq = (T)(__int_as_float(qi.w) * __int_as_float(qj.w));
    } else {
        const double x = pi.x - pj.x, y = pi.y - pj.y, z = pi.z - pj.z;
        dx = (T)(x - b.L0 * round(x * b.B0));
        dy = (T)(y - b.L1 * round(y * b.B1));
        dz = (T)(z - b.L2 * round(z * b.B2));
        qq = (T)(pi.w * pj.w);
    }
    const T r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > (T)a.rmax2) return false;
    T rinv, rinv2;
    flux_rinv(r2, rinv, rinv2);
    const T phc = r2 <= (T)a.rr2 ? qq * rinv : (T)0;               // ewaldr_hf.F90:336-371, bare 1/r
    T phl = (T)0, ftl = (T)0;
    if (r2 <= (T)a.rl2) {                                // ewaldr_hf.F90:376-470
        T R2, E;
        if (MIXED) { const float2 lp = lj32[lj]; R2 = lp.x; E = lp.y; }
        else { const double2 lp = lj64[lj]; R2 = lp.x; E = lp.y; }
        const T t2 = rinv2 * R2, t6 = t2 * t2 * t2, t12 = t6 * t6;
        phl = E * (t12 - (T)2 * t6);
        ftl = (T)6 * E * (t12 - t6) * rinv2;
    }
    const T ftc = (T)0.5 * phc * rinv2;
    o.pc = (T)0.5 * phc;
    o.pl = (T)0.5 * phl;
    o.fc[0] = ftc * dx; o.fc[1] = ftc * dy; o.fc[2] = ftc * dz;
    o.fl[0] = ftl * dx; o.fl[1] = ftl * dy; o.fl[2] = ftl * dz;
    return true;
}

// Per-atom arrays of the pair categories: both atoms of a pair receive its
// energy shares and f_ij times the signed length of (zi, zj) inside each
// region, which is C_i - C_j with C the z clamped to the region (see
// k_flux_pair).  A warp takes a cluster's row (segment) twice per window of KW
// regions that the row touches: with one entry per lane, for the shares of the
// entries' atoms (one FP64 atomic per atom, category, region and axis instead
// of one per pair), and with 8 cluster atoms x 4 entries, for the cluster
// atoms', added over the four lanes and flushed once.  Pairs of the class
// (same molecule / different) that the row has fewer of, and atoms exactly on
// a plane, add to both atoms directly.
// Bound by latency at 16 warps per SM (issue 43 % busy; the pair arithmetic is
// done twice, and the entries' records are loaded for each window).  Measured,
// mixed: 43,200-atom slab, 23 regions 0.79 ms (4.86 ms with one lane's atomics
// for every pair, into shared memory for the cluster atom and global memory for
// the entry's); 8,232-atom water box, one region 0.114 ms (1.27 ms).  Three blocks per SM without spills, or six regions a walk, were
// no faster (slab, call of 10 steps: 7.92, 8.04 ms against 7.87).
template <bool MIXED, int KW>
__global__ void __launch_bounds__(128, MIXED ? 4 : 3)
k_hf_pair(const int4* __restrict__ xq, const double4* __restrict__ xq64, FluxPairArgs a,
          const float2* __restrict__ lj32, const double2* __restrict__ lj64, HfDev h,
          const DynState* __restrict__ dyn) {
    __shared__ double sz1[PGK_HF_MAX_REGIONS], sz2[PGK_HF_MAX_REGIONS];
    __shared__ int4 sxq[4][8];
    __shared__ double4 sx64[MIXED ? 1 : 4][8];
    __shared__ double szi[4][8], sC[4][8][KW];
    __shared__ uint4 sbi[4][8];
    __shared__ int smi[4][8], sti[4][8], soi[4][8];
    const int nreg = h.nreg;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < nreg) { sz1[threadIdx.x] = h.z1[threadIdx.x]; sz2[threadIdx.x] = h.z2[threadIdx.x]; }
    __syncthreads();
    const unsigned all = nreg >= 32 ? 0xffffffffu : (1u << nreg) - 1u;
    HfBox bx;
    bx.L0 = dyn->box[0]; bx.L1 = dyn->box[1]; bx.L2 = dyn->box[2];
    bx.B0 = 1.0 / bx.L0; bx.B1 = 1.0 / bx.L1; bx.B2 = 1.0 / bx.L2;
    const size_t N = (size_t)h.natom;
    double* const pot0 = h.pot + (size_t)PGK_HF_ELIN * N;
    double* const W0 = h.W + (size_t)PGK_HF_ELIN * nreg * 3 * N;
    const long long nunit = (long long)a.ncl * a.nseg;
    for (long long u = blockIdx.x * 4 + w; u < nunit; u += gridDim.x * 4) {
        const int cl = (int)(u / a.nseg), seg = (int)(u - (long long)cl * a.nseg);
        const int cnt = a.cnt[a.cut ? u : cl];
        const int chunk = a.cut ? cnt : ((cnt + a.nseg - 1) / a.nseg + 31) & ~31;
        const int k_lo = a.cut ? 0 : seg * chunk, k_hi = min(cnt, k_lo + chunk);
        if (k_lo >= k_hi) continue;                       // warp-uniform
        const int* __restrict__ row = a.rows + (size_t)(a.cut ? u : cl) * a.ccap;
        __syncwarp();
        if (lane < 8) {
            const int s = 8 * cl + lane;
            if (MIXED) sxq[w][lane] = xq[s]; else sx64[MIXED ? 0 : w][lane] = xq64[s];
            szi[w][lane] = a.zs[s];
            sbi[w][lane] = a.bs[s];
            smi[w][lane] = a.ms[s];
            sti[w][lane] = a.typ_s[s] * a.ntyp;
            soi[w][lane] = a.perm[s];
        }
        __syncwarp();
        // regions that a pair of this row segment can touch; the larger class
        unsigned todo = 0u;
        int nsame = 0, npair = 0;
        for (int k = k_lo + lane; k < k_hi; k += 32) {
            const unsigned e = (unsigned)row[k];
            const uint4 bj = a.bs[e & 0xFFFFFFu];
            const int mj = a.ms[e & 0xFFFFFFu];
            npair += __popc(e >> 24);
#pragma unroll
            for (int ii = 0; ii < 8; ++ii)
                if ((e >> (24 + ii)) & 1u) {
                    const uint4 bi = sbi[w][ii];
                    todo |= ~((bi.x & bj.x) | (bi.y & bj.y));
                    nsame += !((smi[w][ii] ^ mj) & HF_MS_ID);
                }
        }
        todo = __reduce_or_sync(0xffffffffu, todo) & all;
        const bool maj = 2 * __reduce_add_sync(0xffffffffu, nsame) > __reduce_add_sync(0xffffffffu, npair);
        const int cc = maj ? 0 : 2;                       // PGK_HF_ELIN + cc: Coulomb, + 1: LJ
        double* const Wc = W0 + (size_t)cc * nreg * 3 * N;
        const size_t ljo = (size_t)nreg * 3 * N;
        bool w0 = true;                                   // energies with the first window
        do {
            int rk[KW];
            unsigned win = 0u;
#pragma unroll
            for (int q = 0; q < KW; ++q) {
                rk[q] = todo ? __ffs(todo) - 1 : -1;
                if (todo) { win |= 1u << rk[q]; todo &= todo - 1; }
            }
            __syncwarp();
            if (lane < 8) {
                const double z = szi[w][lane];
                const uint4 b = sbi[w][lane];
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    const int r = max(rk[q], 0);
                    sC[w][lane][q] = (b.x >> r) & 1u ? sz1[r] : ((b.y >> r) & 1u ? sz2[r] : z);
                }
            }
            __syncwarp();
            // ---- the entries' atoms: lane = entry
            for (int k = k_lo + lane; k < k_hi; k += 32) {
                const unsigned e = (unsigned)row[k];
                const int j = (int)(e & 0xFFFFFFu);
                const unsigned m = e >> 24;
                const double zj = a.zs[j];
                const int mj = a.ms[j], tj = a.typ_s[j], oj = a.perm[j];
                const uint4 bj = a.bs[j];
                int4 qj = make_int4(0, 0, 0, 0);
                double4 pj = make_double4(0, 0, 0, 0);
                if (MIXED) qj = xq[j]; else pj = xq64[j];
                double Cj[KW], ac[KW][3], al[KW][3], pc = 0.0, pl = 0.0;
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    const int r = max(rk[q], 0);
                    Cj[q] = (bj.x >> r) & 1u ? sz1[r] : ((bj.y >> r) & 1u ? sz2[r] : zj);
#pragma unroll
                    for (int d = 0; d < 3; ++d) { ac[q][d] = 0.0; al[q][d] = 0.0; }
                }
#pragma unroll 1
                for (unsigned mm = m; mm; mm &= mm - 1) {
                    const int ii = __ffs(mm) - 1;
                    HfTerm<MIXED> t;
                    if (!hf_term<MIXED>(sxq[w][ii], sx64[MIXED ? 0 : w][ii], qj, pj, a, bx, sti[w][ii] + tj, lj32, lj64, t))
                        continue;
                    const int mi = smi[w][ii];
                    const bool same = !((mi ^ mj) & HF_MS_ID);
                    const uint4 bi = sbi[w][ii];
                    const double zi = szi[w][ii], az = fabs(zi - zj);
                    const bool vir = !((mi < 0) && (mj < 0) && same) && az * bx.B2 < 0.5;
                    if (same != maj || (vir && ((bi.w | bj.w) & win))) {
                        const int oi = soi[w][ii], c0 = same ? 0 : 2;
                        if (same != maj && w0) {
                            double* p = pot0 + (size_t)c0 * N;
                            atomicAdd(p + oi, (double)t.pc); atomicAdd(p + oj, (double)t.pc);
                            atomicAdd(p + N + oi, (double)t.pl); atomicAdd(p + N + oj, (double)t.pl);
                        }
                        // the lower atom index first: the reference's i
                        const double za = oi < oj ? zi : zj, zb = oi < oj ? zj : zi;
#pragma unroll 1
                        for (unsigned rm = vir ? win & ~((bi.x & bj.x) | (bi.y & bj.y)) : 0u; rm; rm &= rm - 1) {
                            const int r = __ffs(rm) - 1;
                            double frag;
                            if (!hf_frag(za, zb, sz1[r], sz2[r], az, frag)) continue;
                            const double D = zi - zj >= 0.0 ? frag : -frag;
                            double* p = W0 + ((size_t)c0 * nreg + r) * 3 * N;
#pragma unroll
                            for (int d = 0; d < 3; ++d) {
                                const double vc = (double)t.fc[d] * D, vl = (double)t.fl[d] * D;
                                if (vc != 0.0) { atomicAdd(p + d * N + oi, vc); atomicAdd(p + d * N + oj, vc); }
                                if (vl != 0.0) { atomicAdd(p + ljo + d * N + oi, vl); atomicAdd(p + ljo + d * N + oj, vl); }
                            }
                        }
                        if (same == maj) { pc += (double)t.pc; pl += (double)t.pl; }
                        continue;
                    }
                    pc += (double)t.pc;
                    pl += (double)t.pl;
                    if (!vir) continue;
#pragma unroll
                    for (int q = 0; q < KW; ++q) {
                        const double D = sC[w][ii][q] - Cj[q];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            ac[q][d] = fma((double)t.fc[d], D, ac[q][d]);
                            al[q][d] = fma((double)t.fl[d], D, al[q][d]);
                        }
                    }
                }
                if (w0) {
                    double* p = pot0 + (size_t)cc * N + oj;
                    if (pc != 0.0) atomicAdd(p, pc);
                    if (pl != 0.0) atomicAdd(p + N, pl);
                }
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    if (rk[q] < 0) continue;
                    double* p = Wc + (size_t)rk[q] * 3 * N + oj;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        if (ac[q][d] != 0.0) atomicAdd(p + d * N, ac[q][d]);
                        if (al[q][d] != 0.0) atomicAdd(p + ljo + d * N, al[q][d]);
                    }
                }
            }
            // ---- the cluster atoms: lane = 8 atoms x 4 entries
            {
                const int ii = lane & 7, sub = lane >> 3;
                const int4 qi = sxq[w][ii];
                const double4 pi = sx64[MIXED ? 0 : w][ii];
                const int mi = smi[w][ii], ti = sti[w][ii];
                const uint4 bi = sbi[w][ii];
                const double zi = szi[w][ii];
                double Ci[KW], ac[KW][3], al[KW][3], pc = 0.0, pl = 0.0;
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    Ci[q] = sC[w][ii][q];
#pragma unroll
                    for (int d = 0; d < 3; ++d) { ac[q][d] = 0.0; al[q][d] = 0.0; }
                }
#pragma unroll 1
                for (int k = k_lo + sub; k < k_hi; k += 4) {
                    const unsigned e = (unsigned)row[k];
                    if (!((e >> (24 + ii)) & 1u)) continue;
                    const int j = (int)(e & 0xFFFFFFu);
                    int4 qj = make_int4(0, 0, 0, 0);
                    double4 pj = make_double4(0, 0, 0, 0);
                    if (MIXED) qj = xq[j]; else pj = xq64[j];
                    HfTerm<MIXED> t;
                    if (!hf_term<MIXED>(qi, pi, qj, pj, a, bx, ti + a.typ_s[j], lj32, lj64, t)) continue;
                    const int mj = a.ms[j];
                    const bool same = !((mi ^ mj) & HF_MS_ID);
                    if (same != maj) continue;
                    pc += (double)t.pc;
                    pl += (double)t.pl;
                    const double zj = a.zs[j];
                    const uint4 bj = a.bs[j];
                    if (((mi < 0) && (mj < 0) && same) || fabs(zi - zj) * bx.B2 >= 0.5 || ((bi.w | bj.w) & win)) continue;
#pragma unroll
                    for (int q = 0; q < KW; ++q) {
                        const int r = max(rk[q], 0);
                        const double D = Ci[q] - ((bj.x >> r) & 1u ? sz1[r] : ((bj.y >> r) & 1u ? sz2[r] : zj));
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            ac[q][d] = fma((double)t.fc[d], D, ac[q][d]);
                            al[q][d] = fma((double)t.fl[d], D, al[q][d]);
                        }
                    }
                }
                __syncwarp();
                const int oi = soi[w][ii];
                auto four = [](double v) {
                    v += __shfl_xor_sync(0xffffffffu, v, 8);
                    return v + __shfl_xor_sync(0xffffffffu, v, 16);
                };
                if (w0) {
                    pc = four(pc);
                    pl = four(pl);
                    double* p = pot0 + (size_t)cc * N;
                    if (sub == 0 && pc != 0.0) atomicAdd(p + oi, pc);
                    if (sub == 1 && pl != 0.0) atomicAdd(p + N + oi, pl);
                }
#pragma unroll
                for (int q = 0; q < KW; ++q) {
                    if (rk[q] < 0) continue;               // warp-uniform
                    double* p = Wc + (size_t)rk[q] * 3 * N;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const double vc = four(ac[q][d]), vl = four(al[q][d]);
                        if (sub == (d & 1) && vc != 0.0) atomicAdd(p + d * N + oi, vc);
                        if (sub == 2 + (d & 1) && vl != 0.0) atomicAdd(p + ljo + d * N + oi, vl);
                    }
                }
            }
            w0 = false;
        } while (todo);
    }
}

template <bool MIXED>
__global__ void __launch_bounds__(128, MIXED ? 4 : 3)
k_flux_pair(const int4* __restrict__ xq, const double4* __restrict__ xq64, FluxPairArgs a,
            const float2* __restrict__ lj32, const double2* __restrict__ lj64, FluxDev f,
            const DynState* __restrict__ dyn) {
    pdl_enter();
    typedef typename FluxT<MIXED>::T T;
    __shared__ int4 sxq[4][8];
    __shared__ double4 sx64[MIXED ? 1 : 4][8];
    __shared__ double4 sv[4][8];
    __shared__ double szi[4][8];
    __shared__ int smi[4][8], sti[4][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double L0 = dyn->box[0], L1 = dyn->box[1], Lz = dyn->box[2];
    const double B0 = 1.0 / L0, B1 = 1.0 / L1, B2 = 1.0 / Lz;
    const T sx = (T)(L0 * (1.0 / 4294967296.0)), sy = (T)(L1 * (1.0 / 4294967296.0)), sz = (T)(Lz * (1.0 / 4294967296.0));
    const T rr2 = (T)a.rr2, rl2 = (T)a.rl2, rmax2 = (T)a.rmax2;
    const double4* __restrict__ vs = a.vs;
    const long long nunit = (long long)a.ncl * a.nseg;
    for (long long u = blockIdx.x * 4 + w; u < nunit; u += gridDim.x * 4) {
        const int cl = (int)(u / a.nseg), seg = (int)(u - (long long)cl * a.nseg);
        const int cnt = a.cnt[a.cut ? u : cl];
        const int chunk = a.cut ? cnt : ((cnt + a.nseg - 1) / a.nseg + 31) & ~31;
        const int k_lo = a.cut ? 0 : seg * chunk, k_hi = min(cnt, k_lo + chunk);
        if (k_lo >= k_hi) continue;                       // warp-uniform
        const int* __restrict__ row = a.rows + (size_t)(a.cut ? u : cl) * a.ccap;
        __syncwarp();
        if (lane < 8) {
            const int s = 8 * cl + lane;
            if (MIXED) sxq[w][lane] = xq[s]; else sx64[MIXED ? 0 : w][lane] = xq64[s];
            sv[w][lane] = vs[s];
            szi[w][lane] = a.zs[s];
            smi[w][lane] = a.ms[s];
            sti[w][lane] = a.typ_s[s] * a.ntyp;
        }
        __syncwarp();
        T pic[8], pil[8];
        double sic[8], sil[8];
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) { pic[ii] = (T)0; pil[ii] = (T)0; sic[ii] = 0.0; sil[ii] = 0.0; }
        for (int k = k_lo + lane; k < k_hi; k += 32) {
            const unsigned e = (unsigned)row[k];
            const int j = (int)(e & 0xFFFFFFu);
            const unsigned m = e >> 24;
            const double zj = a.zs[j];
            const int mj = a.ms[j], tj = a.typ_s[j];
            const double4 vj = vs[j];
            int4 qj = make_int4(0, 0, 0, 0);
            double4 pj = make_double4(0, 0, 0, 0);
            if (MIXED) qj = xq[j]; else pj = xq64[j];
            double pjc = 0.0, pjl = 0.0, sjc = 0.0, sjl = 0.0;
#pragma unroll
            for (int ii = 0; ii < 8; ++ii) {
                if (!((m >> ii) & 1u)) continue;
                T dx, dy, dz, qq;
                if (MIXED) {
                    const int4 qi = sxq[w][ii];
                    dx = (T)(qi.x - qj.x) * sx; dy = (T)(qi.y - qj.y) * sy; dz = (T)(qi.z - qj.z) * sz;
                    qq = (T)(__int_as_float(qi.w) * __int_as_float(qj.w));
                } else {
                    const double4 pi = sx64[MIXED ? 0 : w][ii];
                    const double wx = pi.x - pj.x, wy = pi.y - pj.y, wz = pi.z - pj.z;
                    dx = (T)(wx - L0 * round(wx * B0));
                    dy = (T)(wy - L1 * round(wy * B1));
                    dz = (T)(wz - Lz * round(wz * B2));
                    qq = (T)(pi.w * pj.w);
                }
                const T r2 = dx * dx + dy * dy + dz * dz;
                if (r2 > rmax2) continue;
                T rinv, rinv2;
                flux_rinv(r2, rinv, rinv2);
                const T phc = r2 <= rr2 ? qq * rinv : (T)0;              // ewaldr_hf.F90:336-371, bare 1/r
                T phl = (T)0, ftl = (T)0;
                if (r2 <= rl2) {                                         // ewaldr_hf.F90:376-470
                    T R2, E;
                    if (MIXED) { const float2 lp = lj32[sti[w][ii] + tj]; R2 = lp.x; E = lp.y; }
                    else { const double2 lp = lj64[sti[w][ii] + tj]; R2 = lp.x; E = lp.y; }
                    const T t2 = rinv2 * R2, t6 = t2 * t2 * t2, t12 = t6 * t6;
                    phl = E * (t12 - (T)2 * t6);
                    ftl = (T)12 * E * (t12 - t6) * rinv2;
                }
                const double4 vi = sv[w][ii];
                const double fv = (double)dx * (vi.x + vj.x) + (double)dy * (vi.y + vj.y) + (double)dz * (vi.z + vj.z);
                const int mi = smi[w][ii];
                const bool same = !((mi ^ mj) & HF_MS_ID);
                const double zi = szi[w][ii], az = fabs(zi - zj);
                const bool vir = !((mi < 0) && (mj < 0) && same) && az * B2 < 0.5;
                double sc = vir ? 0.5 * (double)(phc * rinv2) * fv : 0.0;
                double sl = vir ? 0.5 * (double)ftl * fv : 0.0;
                if (same || ((mi | mj) & HF_MS_PLANE)) {
                    const int s = 8 * cl + ii;
                    if (vir && ((mi | mj) & HF_MS_PLANE)) {
                        // the lower atom index first: the reference's i
                        const bool first = a.perm[s] < a.perm[j];
                        const uint4 bi = a.bs[s], bj = a.bs[j];
                        double* acc = f.acc + (size_t)(blockIdx.x % FLUX_COPIES) * f.h.nreg * FLUX_COLS + 9 +
                                      PGK_HF_ELIN + (same ? 0 : 2);
#pragma unroll 1
                        for (int r = 0; r < f.h.nreg; ++r) {
                            double frag;
                            if (((bi.x & bj.x) | (bi.y & bj.y)) >> r & 1u) continue;
                            if (!hf_frag(first ? zi : zj, first ? zj : zi, f.h.z1[r], f.h.z2[r], az, frag)) continue;
                            const double d = zi - zj >= 0.0 ? frag : -frag;
                            atomicAdd(acc + r * FLUX_COLS, sc * d);
                            atomicAdd(acc + r * FLUX_COLS + 1, sl * d);
                        }
                        sc = 0.0;
                        sl = 0.0;
                    }
                    if (same) {
                        double* si = f.sum + (size_t)FLUX_SUMS * s;
                        double* sj = f.sum + (size_t)FLUX_SUMS * j;
                        atomicAdd(si, (double)phc); atomicAdd(sj, (double)phc);
                        atomicAdd(si + 1, (double)phl); atomicAdd(sj + 1, (double)phl);
                        if (sc != 0.0) { atomicAdd(si + 2, sc); atomicAdd(sj + 2, -sc); }
                        if (sl != 0.0) { atomicAdd(si + 3, sl); atomicAdd(sj + 3, -sl); }
                        continue;
                    }
                }
                pic[ii] += phc; pil[ii] += phl; pjc += (double)phc; pjl += (double)phl;
                sic[ii] += sc; sil[ii] += sl; sjc += sc; sjl += sl;
            }
            double* sj = f.sum + (size_t)FLUX_SUMS * j + 4;
            if (pjc != 0.0) atomicAdd(sj, pjc);
            if (pjl != 0.0) atomicAdd(sj + 1, pjl);
            if (sjc != 0.0) atomicAdd(sj + 2, -sjc);
            if (sjl != 0.0) atomicAdd(sj + 3, -sjl);
        }
        // the cluster atoms' 32 sums: halves exchanged until lane l holds the
        // total of value l = 4 atom + sum
        double v[32];
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) {
            v[4 * ii] = (double)pic[ii]; v[4 * ii + 1] = (double)pil[ii];
            v[4 * ii + 2] = sic[ii]; v[4 * ii + 3] = sil[ii];
        }
#pragma unroll
        for (int h = 16; h > 0; h >>= 1) {
            const bool up = lane & h;
#pragma unroll
            for (int q = 0; q < h; ++q) {
                const double keep = up ? v[q + h] : v[q], send = up ? v[q] : v[q + h];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, send, h);
            }
        }
        if (v[0] != 0.0) atomicAdd(f.sum + (size_t)FLUX_SUMS * (8 * cl + (lane >> 2)) + 4 + (lane & 3), v[0]);
    }
}

// Region sums of the atoms' pair sums: a warp takes 32 slots, its lanes one
// region and every (32 / PR)-th slot each, PR the power of two that holds the
// regions (C_r(z) - z1_r: the pairs' differences stay).  Each slot's 8 sums are
// one 64-byte line.
__global__ void __launch_bounds__(256) k_flux_regions(const int* __restrict__ perm, int npad,
                                                      const double* __restrict__ zs, const double4* __restrict__ vs,
                                                      const uint4* __restrict__ bs, FluxDev f) {
    pdl_enter();
    __shared__ double st[8][32][FLUX_SUMS + 2];
    __shared__ unsigned si[8][32];
    __shared__ double sb[8 * PGK_HF_MAX_REGIONS];
    const int nreg = f.h.nreg, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int q = threadIdx.x; q < 8 * nreg; q += 256) sb[q] = 0.0;
    __syncthreads();
    const int s = blockIdx.x * 256 + threadIdx.x;
    const bool has = s < npad && perm[s] >= 0;
    if (has) {
        st[w][lane][0] = zs[s];
        st[w][lane][1] = 0.5 * vs[s].w;
        si[w][lane] = bs[s].z;
#pragma unroll
        for (int q = 0; q < FLUX_SUMS; ++q) st[w][lane][2 + q] = f.sum[(size_t)FLUX_SUMS * s + q];
    }
    const unsigned has_m = __ballot_sync(0xffffffffu, has);      // the slots of st and si that were written
    __syncwarp();
    int pr = 1;
    while (pr < nreg) pr <<= 1;
    const int r = lane & (pr - 1), part = lane / pr, nq = 32 / pr;
    const double z1 = r < nreg ? f.h.z1[r] : 0.0, z2 = r < nreg ? f.h.z2[r] : 0.0;
    double o[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) o[q] = 0.0;
    if (r < nreg)
        for (int k = part; k < 32; k += nq) {
            if (!((has_m >> k) & 1u)) continue;
            const double* p = st[w][k];
            const double D = fmin(fmax(p[0], z1), z2) - z1;
            const double tv = (si[w][k] >> r) & 1u ? p[1] : 0.0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {        // pairs inside one molecule, between two
                o[4 * c] = fma(p[2 + 4 * c], tv, o[4 * c]);
                o[4 * c + 1] = fma(p[3 + 4 * c], tv, o[4 * c + 1]);
                o[4 * c + 2] = fma(p[4 + 4 * c], D, o[4 * c + 2]);
                o[4 * c + 3] = fma(p[5 + 4 * c], D, o[4 * c + 3]);
            }
        }
    __syncwarp();
    for (int h = pr; h < 32; h <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] += __shfl_xor_sync(0xffffffffu, o[q], h);
    if (part == 0 && r < nreg) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (o[q] != 0.0) atomicAdd(sb + 8 * r + q, o[q]);
    }
    __syncthreads();
    double* acc = f.acc + (size_t)(blockIdx.x % FLUX_COPIES) * nreg * FLUX_COLS;
    for (int q = threadIdx.x; q < 8 * nreg; q += 256) {
        const int c = (q >> 2) & 1, v = q & 3;                   // class; energies, virials
        if (sb[q] != 0.0) atomicAdd(acc + (q >> 3) * FLUX_COLS + (v < 2 ? 1 : 9 - 2) + PGK_HF_ELIN + 2 * c + v, sb[q]);
    }
}

// Per-atom reciprocal terms (pgk_set_hf_kspace): the energy is transported in
// the atom's region, the (a, z) column of the tensor counts in region 1.
__global__ void __launch_bounds__(256) k_flux_kspace(const double* __restrict__ pos, const double* __restrict__ pot,
                                                     const double* __restrict__ vir, FluxDev f,
                                                     const DynState* __restrict__ dyn) {
    __shared__ double sp[PGK_HF_MAX_REGIONS + 1];
    const int nreg = f.h.nreg;
    if (threadIdx.x <= PGK_HF_MAX_REGIONS) sp[threadIdx.x] = 0.0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double p = 0.0, v = 0.0;
    unsigned in = 0u;
    if (i < f.h.natom) {
        in = flux_bits(f.h, i, hf_z(f.h, pos, i, dyn->box[2]), dyn->box[2]).z;
        p = pot[i] * flux_vz(f, i);
        const double* t = vir + (size_t)9 * i + 6;
        v = t[0] * f.vel[3 * i] + t[1] * f.vel[3 * i + 1] + t[2] * f.vel[3 * i + 2];
    }
    unsigned any = __reduce_or_sync(0xffffffffu, in);
    while (any) {
        const int r = __ffs(any) - 1;
        any &= any - 1;
        const double s = warp_sum((in >> r) & 1u ? p : 0.0);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sp[r], s);
    }
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sp[PGK_HF_MAX_REGIONS], v);
    __syncthreads();
    double* acc = f.acc + (size_t)(blockIdx.x % FLUX_COPIES) * nreg * FLUX_COLS;
    if (threadIdx.x < nreg && sp[threadIdx.x] != 0.0)
        atomicAdd(acc + threadIdx.x * FLUX_COLS + 1 + PGK_HF_ELC, sp[threadIdx.x]);
    if (threadIdx.x == 0) atomicAdd(acc + 9 + PGK_HF_ELC, sp[PGK_HF_MAX_REGIONS]);
}

// volume normalisation and hftot; leaves the sums zero (one warp per region)
__global__ void k_flux_final(FluxDev f, const DynState* __restrict__ dyn, double* __restrict__ rec) {
    pdl_enter();
    const int r = blockIdx.x, c = threadIdx.x;
    double s = 0.0;
    if (c < FLUX_COLS) {
        for (int k = 0; k < FLUX_COPIES; ++k) {
            double* p = f.acc + ((size_t)k * f.h.nreg + r) * FLUX_COLS + c;
            s += *p;
            *p = 0.0;
        }
        const double area_inv = (1.0 / dyn->box[0]) * (1.0 / dyn->box[1]);
        s *= area_inv / (f.h.z2[r] - f.h.z1[r]);
        rec[r * PGK_HF_NCOL + c] = s;
    }
    const double tot = warp_sum(s);
    if (c == 0) rec[r * PGK_HF_NCOL + 17] = tot;
}

// ---- region Langevin thermostat ----------------------------------------------
struct LtDev {
    int nlt;
    double x1[PGK_LT_MAX_REGIONS], x2[PGK_LT_MAX_REGIONS], y1[PGK_LT_MAX_REGIONS], y2[PGK_LT_MAX_REGIONS];
    double z1[PGK_LT_MAX_REGIONS], z2[PGK_LT_MAX_REGIONS], temp[PGK_LT_MAX_REGIONS], damp[PGK_LT_MAX_REGIONS];
    unsigned long long seed;
};

__device__ __forceinline__ bool lt_in(double lo, double hi, double x, double L) {
    return (lo <= x && x < hi) || (lo <= x - L && x - L < hi);
}
__device__ __forceinline__ int lt_region(const LtDev& l, const double* g, const double* box) {
    for (int r = 0; r < l.nlt; ++r)
        if (lt_in(l.x1[r], l.x2[r], g[0], box[0]) && lt_in(l.y1[r], l.y2[r], g[1], box[1]) &&
            lt_in(l.z1[r], l.z2[r], g[2], box[2]))
            return r;
    return -1;
}

// langevin_regist.F90:86-360 (one thread per molecule)
__global__ void k_lt_regist(const double* __restrict__ pos, const double* __restrict__ mass,
                            const int* __restrict__ mol_idx, const int* __restrict__ mol_list, int nmole,
                            const int* __restrict__ lt_mole, LtDev l, const DynState* __restrict__ dyn,
                            int* __restrict__ reg) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nmole) return;
    const int b = mol_idx[m], e = mol_idx[m + 1];
    const double* box = dyn->box;
    if (lt_mole[m] && e - b > 1) {
        double ms = 0.0, g[3] = {0.0, 0.0, 0.0};
        for (int q = b; q < e; ++q) {
            int i = mol_list[q];
            ms = ms + mass[i];
            for (int d = 0; d < 3; ++d) g[d] = g[d] + mass[i] * pos[3 * i + d];
        }
        for (int d = 0; d < 3; ++d) g[d] = hf_wrap1(g[d] / ms, box[d]);
        const int r = lt_region(l, g, box);
        for (int q = b; q < e; ++q) reg[mol_list[q]] = r;
    } else {
        for (int q = b; q < e; ++q) {
            int i = mol_list[q];
            double g[3];
            for (int d = 0; d < 3; ++d) g[d] = hf_wrap1(pos[3 * i + d], box[d]);
            reg[i] = lt_region(l, g, box);
        }
    }
}

// langevin_region.F90:88-180: former half draws the random accelerations
// (Box-Muller as the reference), kick then friction; latter half friction
// then kick with the stored accelerations.  dekin (if non-null) collects
// sum m v^2 per region before (slot r) and after (slot 8 + r).
__global__ void k_langevin(double* __restrict__ vel, const double* __restrict__ mass, int n,
                           const int* __restrict__ reg, double* __restrict__ frand, LtDev l, double dt,
                           long long step, int former, double* __restrict__ dekin) {
    __shared__ double ek[2 * PGK_LT_MAX_REGIONS];
    if (dekin) {
        for (int q = threadIdx.x; q < 2 * PGK_LT_MAX_REGIONS; q += blockDim.x) ek[q] = 0.0;
        __syncthreads();
    }
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int r = i < n ? reg[i] : -1;
    if (i < n && former) {
        double f[3] = {0.0, 0.0, 0.0};
        if (r >= 0) {
            const double var = 2.0 * l.damp[r] * l.temp[r] / dt * mass[i];
            double u[4];
            lt_draw(l.seed, step, i, u);
            const double twopi = 2.0 * 3.14159265358979323846;
            const double a = sqrt(-2.0 * log(u[0]) * var);
            f[0] = a * cos(twopi * u[1]) / mass[i];
            f[1] = a * sin(twopi * u[1]) / mass[i];
            f[2] = sqrt(-2.0 * log(u[2]) * var) * cos(twopi * u[3]) / mass[i];
        }
        frand[3 * i] = f[0]; frand[3 * i + 1] = f[1]; frand[3 * i + 2] = f[2];
    }
    if (r >= 0) {
        double* v = vel + 3 * i;
        const double m = mass[i];
        if (dekin) atomicAdd(&ek[r], m * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]));
        const double ex = exp(-0.5 * dt * l.damp[r]);
        for (int d = 0; d < 3; ++d) {
            if (former) { v[d] = v[d] + 0.5 * dt * frand[3 * i + d]; v[d] = v[d] * ex; }
            else { v[d] = v[d] * ex; v[d] = v[d] + 0.5 * dt * frand[3 * i + d]; }
        }
        if (dekin) atomicAdd(&ek[PGK_LT_MAX_REGIONS + r], m * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]));
    }
    if (dekin) {
        __syncthreads();
        for (int q = threadIdx.x; q < l.nlt; q += blockDim.x)
            atomicAdd(&dekin[q], 0.5 * (ek[PGK_LT_MAX_REGIONS + q] - ek[q]));
    }
}

// ---- host side -----------------------------------------------------------------
static HfDev hf_dev(pgk_ctx* c) {
    HfDev h;
    h.nreg = c->hfp.nhfregion;
    h.natom = c->natom;
    for (int r = 0; r < PGK_HF_MAX_REGIONS; ++r) { h.z1[r] = c->hfp.hfzpos1[r]; h.z2[r] = c->hfp.hfzpos2[r]; }
    h.hftyp = c->hftyp; h.mol_of = c->mol_of; h.molecom = c->molecom;
    h.pot = c->hf_pot; h.W = c->hf_W;
    return h;
}
static LtDev lt_dev(const pgk_ctx* c) {
    LtDev l;
    const pgk_hfparams& p = c->hfp;
    l.nlt = p.nlangeregion;
    for (int r = 0; r < PGK_LT_MAX_REGIONS; ++r) {
        l.x1[r] = p.ltxpos1[r]; l.x2[r] = p.ltxpos2[r]; l.y1[r] = p.ltypos1[r]; l.y2[r] = p.ltypos2[r];
        l.z1[r] = p.ltzpos1[r]; l.z2[r] = p.ltzpos2[r]; l.temp[r] = p.r_ltemp[r]; l.damp[r] = p.r_ltdamp[r];
    }
    l.seed = p.seed;
    return l;
}

template <typename T>
static pgk_status upload_vec(pgk_ctx* c, T** dst, const std::vector<T>& v) {
    if (*dst) { pgk_dfree(c, *dst); *dst = nullptr; }
    if (v.empty()) return PGK_OK;
    PGK_CUDA(c, pgk_dmalloc(c, dst, sizeof(T) * v.size()));
    PGK_CUDA(c, cudaMemcpyAsync(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, c->st));
    return PGK_OK;
}

pgk_status hf_setup(pgk_ctx* c, const pgk_hfparams* p) {
    if (p->nhfregion < 0 || p->nhfregion > PGK_HF_MAX_REGIONS || p->nlangeregion < 0 ||
        p->nlangeregion > PGK_LT_MAX_REGIONS)
        return pgk_fail(c, PGK_E_INVALID, "region count out of range");
    if (p->nhfregion > 0 && p->ifhfvol != 1)
        return pgk_fail(c, PGK_E_UNSUPPORTED, "only the local volume-based heat flux (ifhfvol) is built");
    for (int r = 0; r < p->nhfregion; ++r)
        if (!(p->hfzpos2[r] > p->hfzpos1[r])) return pgk_fail(c, PGK_E_INVALID, "hfzpos2 must exceed hfzpos1");
    pgk_status s;
    PGK_CUDA(c, cudaStreamSynchronize(c->st));
    int n = c->natom;
    c->hfp = *p;
    c->hfp.hftyp_atm = nullptr;
    c->hfp.lt_mole_based = nullptr;
    if (c->hfp.heatfinterval < 1) c->hfp.heatfinterval = 1;
    std::vector<int> molidx(c->nmole + 1), mollist, molof(n, 0), hftyp(n, PGK_HFTYP_ATOM), ltm(c->nmole, 0);
    if (c->nmole > 0) {
        PGK_CUDA(c, cudaMemcpy(molidx.data(), c->mol_idx, sizeof(int) * (c->nmole + 1), cudaMemcpyDeviceToHost));
        mollist.resize(molidx[c->nmole]);
        PGK_CUDA(c, cudaMemcpy(mollist.data(), c->mol_list, sizeof(int) * mollist.size(), cudaMemcpyDeviceToHost));
    }
    for (int m = 0; m < c->nmole; ++m)
        for (int q = molidx[m]; q < molidx[m + 1]; ++q) molof[mollist[q]] = m;
    if (p->hftyp_atm)
        for (int i = 0; i < n; ++i) {
            if (p->hftyp_atm[i] != PGK_HFTYP_ATOM && p->hftyp_atm[i] != PGK_HFTYP_MOLE)
                return pgk_fail(c, PGK_E_INVALID, "hftyp_atm must be 1 (atom) or 2 (molecule)");
            hftyp[i] = p->hftyp_atm[i];
        }
    if (p->lt_mole_based) for (int m = 0; m < c->nmole; ++m) ltm[m] = p->lt_mole_based[m] ? 1 : 0;
    if ((s = upload_vec(c, &c->mol_of, molof)) || (s = upload_vec(c, &c->hftyp, hftyp)) ||
        (s = upload_vec(c, &c->lt_mole, ltm)))
        return s;
    auto realloc = [&](double** b, size_t cnt) -> pgk_status {
        if (*b) { pgk_dfree(c, *b); *b = nullptr; }
        if (cnt == 0) return PGK_OK;
        if (pgk_dmalloc(c, b, cnt * sizeof(double)) != cudaSuccess) return pgk_fail(c, PGK_E_NOMEM, "heat-flux arrays");
        PGK_CUDA(c, cudaMemsetAsync(*b, 0, cnt * sizeof(double), c->st));
        return PGK_OK;
    };
    const int nreg = c->hfp.nhfregion;
    if ((s = realloc(&c->molecom, (size_t)3 * std::max(1, c->nmole))) ||
        (s = realloc(&c->molevel, (size_t)3 * std::max(1, c->nmole))) ||
        (s = realloc(&c->hf_pot, (size_t)8 * n)) || (s = realloc(&c->hf_W, (size_t)8 * nreg * 3 * n)) ||
        (s = realloc(&c->hf_acc, (size_t)FLUX_COPIES * nreg * FLUX_COLS)) ||
        (s = realloc(&c->hf_rec, (size_t)std::max(1, nreg) * PGK_HF_NCOL)) ||   // one record
        (s = realloc(&c->lt_frand, (size_t)3 * n)) || (s = realloc(&c->lt_dekin, PGK_LT_MAX_REGIONS)))
        return s;
    c->hf_rec_cap = 1;
    c->hf_k_terms = nullptr;
    if (c->lt_reg) pgk_dfree(c, c->lt_reg);
    c->lt_reg = nullptr;
    PGK_CUDA(c, pgk_dmalloc(c, &c->lt_reg, sizeof(int) * n));
    PGK_CUDA(c, cudaMemsetAsync(c->lt_reg, 0xff, sizeof(int) * n, c->st));
    c->hf_set = true;
    if (nreg > 0 && (s = keep_plain_order(c))) return s;
    if (c->hfp.nlangeregion > 0 && (s = launch_lt_regist(c))) return s;
    PGK_CUDA(c, cudaStreamSynchronize(c->st));
    return PGK_OK;
}

static pgk_status ensure_hf_slots(pgk_ctx* c) {
    if (c->hf_slots_cap >= c->npad_cap) return PGK_OK;
    pgk_dfree(c, c->hf_zs); pgk_dfree(c, c->hf_ms); pgk_dfree(c, c->hf_vs); pgk_dfree(c, c->hf_bs); pgk_dfree(c, c->hf_sum);
    c->hf_zs = nullptr; c->hf_ms = nullptr; c->hf_vs = nullptr; c->hf_bs = nullptr; c->hf_sum = nullptr;
    c->hf_slots_cap = 0;
    PGK_CUDA(c, pgk_dmalloc(c, &c->hf_zs, sizeof(double) * c->npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->hf_ms, sizeof(int) * c->npad_cap));
    const size_t vb = sizeof(double4) * (size_t)c->npad_cap;
    PGK_CUDA(c, pgk_dmalloc(c, &c->hf_vs, vb));
    PGK_CUDA(c, pgk_dmalloc(c, &c->hf_bs, sizeof(uint4) * c->npad_cap));
    PGK_CUDA(c, pgk_dmalloc(c, &c->hf_sum, sizeof(double) * FLUX_SUMS * c->npad_cap));
    // padding slots take part in no pair, but a cluster stages them
    PGK_CUDA(c, cudaMemsetAsync(c->hf_zs, 0, sizeof(double) * c->npad_cap, c->st));
    PGK_CUDA(c, cudaMemsetAsync(c->hf_ms, 0, sizeof(int) * c->npad_cap, c->st));
    PGK_CUDA(c, cudaMemsetAsync(c->hf_vs, 0, vb, c->st));
    PGK_CUDA(c, cudaMemsetAsync(c->hf_bs, 0, sizeof(uint4) * c->npad_cap, c->st));
    c->hf_slots_cap = c->npad_cap;
    return PGK_OK;
}

// calforce_hf's per-atom quantities at the current positions (list and the
// pair kernel's packed coordinates must be current)
// Per-atom reciprocal terms of the bulk heat flux (pgk_set_hf_kspace) into
// the intermolecular Coulomb category: each atom's energy, and the (a, z)
// column of its tensor into region 1 -- ewaldk_hf.F90:212-230 writes
// virielct_atm(:, :, i, 1), the single region of the bulk builds.
__global__ void k_hf_kspace_add(const double* __restrict__ pot, const double* __restrict__ vir, int n, int nreg,
                                double* __restrict__ hf_pot, double* __restrict__ hf_W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    hf_pot[(size_t)PGK_HF_ELC * n + i] += pot[i];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        hf_W[((size_t)PGK_HF_ELC * nreg * 3 + a) * n + i] += vir[(size_t)9 * i + a + 6];
}

// the per-atom reciprocal terms at the current positions (energies [N] |
// tensors [9N]; null: the option is off), evaluated once per heat-flux step
static pgk_status hf_kspace_terms(pgk_ctx* c, const double** pot) {
    *pot = nullptr;
    const int n = c->natom;
    if (!c->hf_k_terms) {
        if (c->hf_kspace == PGK_HF_KSPACE_SPME) {
            pgk_status s = launch_spme_hf_atm(c);
            if (s) return s;
            c->hf_k_terms = c->hfk_out;
        } else if (c->hf_kspace == PGK_HF_KSPACE_EWK) {
            if (!c->hf_ewk_fresh) {   // not yet evaluated at these positions by the force evaluation
                int nw = 0;
                pgk_status s = launch_ewk_hf(c, c->hf_kmax, &nw);
                if (s) return s;
            }
            c->hf_k_terms = c->ewk_out + 3 * (size_t)n;
        }
        c->hf_ewk_fresh = false;
    }
    *pot = c->hf_k_terms;
    return PGK_OK;
}

static pgk_status launch_hf_kspace(pgk_ctx* c) {
    const int n = c->natom;
    const double* pot;
    pgk_status s = hf_kspace_terms(c, &pot);
    if (s || !pot) return s;
    k_hf_kspace_add<<<(n + 255) / 256, 256, 0, c->st>>>(pot, pot + n, n, c->hfp.nhfregion, c->hf_pot, c->hf_W);
    PGK_LAUNCHED(c);
    PGK_CUDA(c, cudaGetLastError());
    return PGK_OK;
}

static bool flux_pair_on(const pgk_ctx* c) {
    return (c->prm.mts_vdw == PGK_MTS_LONG || c->prm.mts_vdw == PGK_MTS_SHORT) && c->ncl > 0;
}
// pruned: this step's pair kernel has left its rows (c->plist)
static FluxPairArgs flux_pair_args(pgk_ctx* c, bool pruned) {
    FluxPairArgs a;
    pruned = pruned && c->prune_buffer > 0.f;
    a.cut = pruned && c->pseg > 1;
    a.rows = pruned ? c->plist : c->clist; a.cnt = pruned ? c->pcnt : c->ccnt;
    a.ccap = pruned ? c->pcap : c->ccap; a.ncl = c->ncl;
    a.typ_s = c->typ_s; a.perm = c->perm; a.ntyp = c->ntyp;
    a.zs = c->hf_zs; a.ms = c->hf_ms; a.vs = c->hf_vs; a.bs = c->hf_bs;
    const double rr2 = c->prm.rrcut * c->prm.rrcut;
    a.rr2 = c->mixed() ? rr2 : sqrt_le_limit(c->prm.rrcut);
    a.rl2 = c->prm.rcut * c->prm.rcut;
    a.rmax2 = std::max(rr2, a.rl2);
    // about 16 warps per SM, in row segments where the clusters alone are fewer
    a.nseg = a.cut ? c->pseg : std::max(1, std::min(8, c->nsm * 16 / std::max(a.ncl, 1)));
    return a;
}
static int flux_pair_grid(const pgk_ctx* c, const FluxPairArgs& a) {
    const long long units = (long long)a.ncl * a.nseg;
    return (int)std::max(1LL, std::min((units + 3) / 4, (long long)c->nsm * 16));
}

// pruned: this step's pair kernel has left its rows
pgk_status launch_hf_atm(pgk_ctx* c, bool pruned) {
    if (!c->hf_set || c->hfp.nhfregion < 1) return pgk_fail(c, PGK_E_INVALID, "no heat-flux regions set");
    pgk_status s;
    const int n = c->natom, nreg = c->hfp.nhfregion;
    if (c->nmole > 0) {
        launch_pdl(k_calcom, (c->nmole + 127) / 128, 128, 0, c->st, c->pos, (const double*)nullptr, c->mass, c->mol_idx,
                   c->mol_list, c->nmole, c->dyn, c->molecom, (double*)nullptr);
        PGK_LAUNCHED(c);
    }
    PGK_CUDA(c, cudaMemsetAsync(c->hf_pot, 0, sizeof(double) * 8 * n, c->st));
    PGK_CUDA(c, cudaMemsetAsync(c->hf_W, 0, sizeof(double) * 8 * nreg * 3 * (size_t)n, c->st));
    HfDev h = hf_dev(c);
    if (flux_pair_on(c)) {
        if ((s = ensure_hf_slots(c))) return s;
        k_hf_slots<<<(c->npad + 255) / 256, 256, 0, c->st>>>(c->perm, c->npad, c->pos, h, c->dyn, c->hf_zs,
                                                              c->hf_ms, c->hf_bs);
        PGK_LAUNCHED(c);
        FluxPairArgs a = flux_pair_args(c, pruned);
        const int blocks = flux_pair_grid(c, a);
#define PGK_HFP(M, KW) k_hf_pair<M, KW><<<blocks, 128, 0, c->st>>>(c->xq, c->xq64, a, c->lj32, c->lj64, h, c->dyn)
        if (c->mixed()) { if (nreg == 1) PGK_HFP(true, 1); else PGK_HFP(true, 4); }
        else { if (nreg == 1) PGK_HFP(false, 1); else PGK_HFP(false, 4); }
#undef PGK_HFP
        PGK_LAUNCHED(c);
        PGK_CUDA(c, cudaGetLastError());
    }
    if ((s = launch_bonded_hf(c, h))) return s;
    return launch_hf_kspace(c);
}

template <bool MIXED>
static void flux_pair_launch(pgk_ctx* c, const FluxPairArgs& a, const FluxDev& f) {
    launch_pdl(k_flux_pair<MIXED>, flux_pair_grid(c, a), 128, 0, c->st, c->xq, c->xq64, a, c->lj32, c->lj64, f, c->dyn);
    PGK_LAUNCHED(c);
    launch_pdl(k_flux_regions, (c->npad + 255) / 256, 256, 0, c->st, c->perm, c->npad, c->hf_zs, c->hf_vs, c->hf_bs,
               f);
    PGK_LAUNCHED(c);
}

pgk_status launch_heatf(pgk_ctx* c, double* dst, bool pruned) {
    const int nreg = c->hfp.nhfregion, n = c->natom;
    pgk_status s;
    FluxDev f;
    f.h = hf_dev(c);
    f.vel = c->vel; f.molevel = c->molevel; f.acc = c->hf_acc;
    if (c->nmole > 0) {
        launch_pdl(k_calcom, (c->nmole + 127) / 128, 128, 0, c->st, c->pos, c->vel, c->mass, c->mol_idx, c->mol_list,
                   c->nmole, c->dyn, c->molecom, c->molevel);
        PGK_LAUNCHED(c);
    }
    const bool pair_on = flux_pair_on(c);
    if (pair_on && (s = ensure_hf_slots(c))) return s;
    f.sum = c->hf_sum;
    const int* ip = pair_on ? c->iperm : nullptr;
    launch_pdl(k_flux_atoms, (n + 255) / 256, 256, 0, c->st, c->pos, c->mass, ip,
               f, c->dyn, c->hf_zs, c->hf_ms, c->hf_vs, c->hf_bs);
    PGK_LAUNCHED(c);
    if (pair_on) {
        const FluxPairArgs a = flux_pair_args(c, pruned);
        if (c->mixed()) flux_pair_launch<true>(c, a, f);
        else flux_pair_launch<false>(c, a, f);
    }
    if ((s = launch_bonded_flux(c, f))) return s;
    const double* pot;
    if ((s = hf_kspace_terms(c, &pot))) return s;
    c->hf_k_terms = nullptr;
    if (pot) {
        k_flux_kspace<<<(n + 255) / 256, 256, 0, c->st>>>(c->pos, pot, pot + n, f, c->dyn);
        PGK_LAUNCHED(c);
    }
    launch_pdl(k_flux_final, nreg, 32, 0, c->st, f, c->dyn, dst);
    PGK_LAUNCHED(c);
    PGK_CUDA(c, cudaGetLastError());
    return PGK_OK;
}

pgk_status launch_lt_regist(pgk_ctx* c) {
    if (c->nmole <= 0) return PGK_OK;
    k_lt_regist<<<(c->nmole + 127) / 128, 128, 0, c->st>>>(c->pos, c->mass, c->mol_idx, c->mol_list, c->nmole,
                                                            c->lt_mole, lt_dev(c), c->dyn, c->lt_reg);
    PGK_LAUNCHED(c);
    PGK_CUDA(c, cudaGetLastError());
    return PGK_OK;
}

pgk_status launch_langevin(pgk_ctx* c, double dt, long long step, bool former) {
    const int n = c->natom;
    k_langevin<<<(n + 255) / 256, 256, 0, c->st>>>(c->vel, c->mass, n, c->lt_reg, c->lt_frand, lt_dev(c), dt, step,
                                                    former ? 1 : 0, c->hfp.ifoutthc ? c->lt_dekin : nullptr);
    PGK_LAUNCHED(c);
    PGK_CUDA(c, cudaGetLastError());
    return PGK_OK;
}
