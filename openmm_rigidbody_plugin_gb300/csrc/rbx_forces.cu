// rbx_forces.cu -- cutoff Lennard-Jones + reaction-field forces for many independent periodic
// systems, by cell lists (the force provider of the batched and served forms; the drop-in takes
// its forces from the OpenMM Context instead).
//
// Functional form: OpenMM NonbondedForce, CutoffPeriodic method, as documented by OpenMM
//   E = K q_i q_j (1/r + k_rf r^2 - c_rf) + 4 eps_ij ((sig_ij/r)^12 - (sig_ij/r)^6),  r < rc,
// Lorentz-Berthelot combination, minimum image in a cubic box, pairs of one rigid body excluded.
//
// The interacting atoms of one rigid body (or one free atom) form a group; groups are cut into units
// of at most four atoms (a water is one unit). Forces come from neighbour lists of units: a unit's
// list holds every unit of another group whose centroid lies within cutoff + skin (0.12 nm) + both
// radii. A rigid unit's atoms stay within its radius of its centroid however the body turns, so a
// list ages only as the centroids move: each system rebuilds its lists when one of its centroids has
// moved half the skin since its last build, and every list is rebuilt for the state a call starts or
// ends in (so the forces there depend only on the positions, never on when earlier calls rebuilt).
// One evaluation, all systems at once:
//   1. ff_check    one thread per unit: its centroid and radius, the centroid's displacement since
//                  the last build (flags the system's rebuild) and, for lists that stay, its atoms'
//                  records at its place in cell order
//   then, for the flagged systems only (the kernels return at once for the others):
//   2. ff_bin      cell of each unit's centroid and cell counts, cells of at least cutoff + skin
//                  + twice the largest radius per edge
//   3. ff_scan     one block per system: exclusive scan of its cells' counts (and count reset)
//   4. ff_scatter  slot in its cell (single-cell systems keep their unit order, no atomics)
//   5. ff_sort     one warp per cell of a multi-cell box: sorts the cell by unit index
//   6. ff_place    every unit's place, and its records there
//   7. ff_build    one warp per unit: the units in range among the 27 cells around it (or, in a
//                  single-cell box, all units by minimum image), in place order, into its list
//   8. ff_force    one warp per unit (all systems): the unit's atoms in registers, each lane taking
//                  one listed unit at a time; per-lane partial sums joined by a fixed butterfly, no
//                  atomics; forces written as OpenMM fixed point (2^32) to the slots
//   9. ff_energy   (energy evaluations only) one block per 2048 units of a system, joined per
//                  system: fixed-order FP64 sum of its units' pair energies.
// The atoms of one group never meet in a list: pairs of one rigid body are excluded, as the
// plugin's ForceField helper removes them (python/forcefield.py:131-138).
#include <cuda_runtime.h>

#include <cstdint>

#include "rbx_internal.h"

namespace rbx {

namespace {

__device__ __forceinline__ float3 atom_position(const DevBuf& B, int prec, int slot) {
    if (prec == PREC_DOUBLE) {
        const double* p = (const double*)B.posq + 4 * (size_t)slot;
        return make_float3((float)p[0], (float)p[1], (float)p[2]);
    }
    const float4 p = ((const float4*)B.posq)[slot];
    if (prec == PREC_MIXED) {
        const float4 c = ((const float4*)B.corr)[slot];
        return make_float3(p.x + c.x, p.y + c.y, p.z + c.z);
    }
    return make_float3(p.x, p.y, p.z);
}

__device__ __forceinline__ int wrap_cell(float x, float invL, int nc) {
    float f = x * invL;
    f -= floorf(f);
    int c = (int)(f * (float)nc);
    return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

// Position of an interacting atom wrapped into [0, L) and its minimum-image displacement.
__device__ __forceinline__ float3 wrap_box(float3 x, const FFSys& S) {
    x.x -= S.L * floorf(x.x * S.invL);
    x.y -= S.L * floorf(x.y * S.invL);
    x.z -= S.L * floorf(x.z * S.invL);
    return x;
}
__device__ __forceinline__ float3 min_image(float dx, float dy, float dz, const FFSys& S) {
    return make_float3(dx - S.L * rintf(dx * S.invL), dy - S.L * rintf(dy * S.invL), dz - S.L * rintf(dz * S.invL));
}

// Coordinate of the unused atom records of a place: outside every cutoff, its square finite.
constexpr float kFar = 1e10f;

// Centroid of a unit (the mean of its atoms' minimum-image displacements from the first, wrapped
// into the box) and its radius.
__device__ __forceinline__ float4 unit_centroid(const FFDev& D, const DevBuf& B, int prec, const FFSys& S, int k0, int n,
                                                float3 (&x)[kMaxUnit]) {
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++)
        if (a < n) x[a] = atom_position(B, prec, D.iatom[k0 + a]);
    float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
    for (int a = 1; a < kMaxUnit; a++) {
        if (a >= n) break;
        const float3 d = min_image(x[a].x - x[0].x, x[a].y - x[0].y, x[a].z - x[0].z, S);
        sx += d.x;
        sy += d.y;
        sz += d.z;
    }
    const float inv = 1.0f / (float)n;
    const float3 c = wrap_box(make_float3(x[0].x + sx * inv, x[0].y + sy * inv, x[0].z + sz * inv), S);
    float rho2 = 0.f;
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++) {
        if (a >= n) break;
        const float3 d = min_image(x[a].x - c.x, x[a].y - c.y, x[a].z - c.z, S);
        rho2 = fmaxf(rho2, fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)));
        x[a] = make_float3(c.x + d.x, c.y + d.y, c.z + d.z);  // at the image nearest the centroid
    }
    return make_float4(c.x, c.y, c.z, sqrtf(rho2));
}

// A unit's records at place p: centroid, and its atoms (at their images nearest the centroid, so that
// one periodic shift moves a whole unit) with their types.
__device__ __forceinline__ void write_place(const FFDev& D, int p, int k0, int n, float4 c, const float3 (&x)[kMaxUnit]) {
    D.scen[p] = c;
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++) {
        if (a >= D.slots) break;
        D.spos[a][p] = a < n ? make_float4(x[a].x, x[a].y, x[a].z, D.ntypes ? __int_as_float(D.atype[k0 + a]) : 0.0f)
                     : make_float4(kFar, kFar, kFar, 0.0f);
    }
}

// 1. Per unit: centroid, radius and the rebuild test. A system that the host has marked gets its
// records with its new places (ff_place).
__global__ void ff_check(FFDev D, DevBuf B, int prec) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    const FFSys S = D.sys[s];
    const int2 kn = D.unit[u];
    const int k0 = kn.x, n = kn.y & 0xff;
    float3 x[kMaxUnit];
    const float4 c = unit_centroid(D, B, prec, S, k0, n, x);
    D.ucen[u] = c;
    if (D.rebuild[s] == 1) return;
    write_place(D, D.place[u], k0, n, c, x);
    const float4 r = D.uref[u];
    const float3 d = min_image(c.x - r.x, c.y - r.y, c.z - r.z, S);
    if (fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)) > S.half_skin2) D.rebuild[s] = 2;
}

__global__ void ff_bin(FFDev D) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    if (!D.rebuild[s]) return;
    const FFSys S = D.sys[s];
    if (S.nc == 1) {
        D.cell_of[u] = S.c0;
        return;
    }
    const float4 c = D.ucen[u];
    const int cx = wrap_cell(c.x, S.invL, S.nc), cy = wrap_cell(c.y, S.invL, S.nc), cz = wrap_cell(c.z, S.invL, S.nc);
    const int cell = S.c0 + (cz * S.nc + cy) * S.nc + cx;
    D.cell_of[u] = cell;
    atomicAdd(D.cell_count + cell, 1);
}

// Exclusive scan of one system's cell counts, in chunks of blockDim.x; the counts are reset.
__global__ void ff_scan(FFDev D) {
    __shared__ int s[256];
    if (!D.rebuild[blockIdx.x]) return;
    if (threadIdx.x == 0) D.rebuilds[blockIdx.x]++;
    const FFSys S = D.sys[blockIdx.x];
    const int ncell = S.nc * S.nc * S.nc;
    if (S.nc == 1) {
        if (threadIdx.x == 0) {
            D.cell_start[S.c0] = S.u0;
            D.cell_start[S.c0 + 1] = S.u1;
        }
        return;
    }
    int base = S.u0;
    for (int c0 = 0; c0 < ncell; c0 += blockDim.x) {
        const int c = c0 + threadIdx.x;
        const int v = c < ncell ? D.cell_count[S.c0 + c] : 0;
        s[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < (int)blockDim.x; o <<= 1) {  // Hillis-Steele inclusive scan
            const int t = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0;
            __syncthreads();
            s[threadIdx.x] += t;
            __syncthreads();
        }
        if (c < ncell) {
            const int start = base + s[threadIdx.x] - v;
            D.cell_start[S.c0 + c] = start;
            D.cell_cursor[S.c0 + c] = start;
            D.cell_count[S.c0 + c] = 0;
        }
        base += s[blockDim.x - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) D.cell_start[S.c0 + ncell] = base;  // equals S.u1
}

// Key of a unit in the order within its cell: its place on a 4 x 4 x 4 grid of the cell in Z-order,
// then its index, so that the units a list takes of one cell lie in short runs of places and a run of
// places is compact.
__device__ __forceinline__ unsigned int cell_key(const FFDev& D, const FFSys& S, int u) {
    const float4 c = D.ucen[u];
    const float x[3] = {c.x, c.y, c.z};
    unsigned int z = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int g = (int)(x[k] * S.invL * (float)(4 * S.nc)) & 3;
        z |= (unsigned int)((g & 1) << k | (g >> 1) << (3 + k));
    }
    return z << 26 | (unsigned int)(u - S.u0);
}

__global__ void ff_scatter(FFDev D) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    if (!D.rebuild[s]) return;
    if (D.sys[s].nc == 1) {
        D.unit_at[u] = u;  // one cell: unit order
        return;
    }
    const int p = atomicAdd(D.cell_cursor + D.cell_of[u], 1);
    D.unit_at[p] = (int)cell_key(D, D.sys[s], u);
}

// Sort each cell of a multi-cell box by its units' keys, so that every cell, and so every list, is in
// a fixed order. One warp per cell: the cell is staged in shared memory and each lane ranks its
// entries against all of them (the entries are distinct, so the ranks are a permutation); a cell
// larger than the stage falls back to an insertion sort by one lane.
constexpr int kSortWarps = 4, kSortStage = 512;
constexpr unsigned int kKeyUnit = (1u << 26) - 1;
__global__ void __launch_bounds__(32 * kSortWarps) ff_sort(FFDev D) {
    __shared__ unsigned int stage[kSortWarps][kSortStage];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * kSortWarps + warp;
    if (w >= D.n_mc) return;
    const int sy = D.mc_sys[w];
    if (!D.rebuild[sy]) return;
    const int c = D.mc_cell[w], u0 = D.sys[sy].u0;
    const int b = D.cell_start[c], e = D.cell_start[c + 1], n = e - b;
    unsigned int* key = (unsigned int*)D.unit_at + b;
    unsigned int* s = stage[warp];
    if (n <= kSortStage) {
        for (int i = lane; i < n; i += 32) s[i] = key[i];
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            const unsigned int v = s[i];
            int rank = 0;
            for (int j = 0; j < n; j++) rank += s[j] < v;
            key[rank] = u0 + (v & kKeyUnit);
        }
    } else if (lane == 0) {
        for (int i = 1; i < n; i++) {
            const unsigned int v = key[i];
            int j = i - 1;
            while (j >= 0 && key[j] > v) {
                key[j + 1] = key[j];
                j--;
            }
            key[j + 1] = v;
        }
        for (int i = 0; i < n; i++) key[i] = u0 + (key[i] & kKeyUnit);
    }
}

// 6. The units of the rebuilt systems at their new places: records, group, build centroid.
__global__ void ff_place(FFDev D, DevBuf B, int prec) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D.n_units) return;
    const int s = D.usys[p];  // places [u0, u1) belong to the system of unit p
    if (!D.rebuild[s]) return;
    const int u = D.unit_at[p];
    const FFSys S = D.sys[s];
    const int2 kn = D.unit[u];
    const int k0 = kn.x, n = kn.y & 0xff;
    float3 x[kMaxUnit];
    const float4 c = unit_centroid(D, B, prec, S, k0, n, x);
    write_place(D, p, k0, n, c, x);
    if (!D.ntypes)
        for (int a = 0; a < D.slots; a++)
            D.spar[a][p] = a < n ? D.param[k0 + a] : make_float4(0.f, 0.f, 0.f, 0.f);
    D.place[u] = p;
    D.sgrp[p] = D.ugrp[u];
    D.uref[u] = c;
}

// 7. Lists, one warp per unit: the lanes test 32 candidates at a time (their centroids and groups lie
// in place order, so a row of neighbour cells is one contiguous run) and append the ones in range in
// order, a ballot giving each its slot. Against one thread per unit of a cell walking the 27 cells
// staged in shared memory, no lane idles (a cell holds about 48 units of 128 threads) and the list is
// written coalesced. A full list marks the system as failed (the capacity is sized from the densest
// system with a wide margin, so this does not happen in a liquid).
template <bool IMAGE>
__device__ __forceinline__ void scan_run(const FFDev& D, const FFSys& S, unsigned int* __restrict__ list, float4 c, int grp,
                                         float3 shift, int q0, int q1, int lane, int& n) {
    for (int qb = q0; qb < q1; qb += 32) {
        const int q = qb + lane;
        bool hit = false;
        if (q < q1) {
            const float4 cq = D.scen[q];
            const int gq = D.sgrp[q];
            float3 d = make_float3(c.x - (cq.x + shift.x), c.y - (cq.y + shift.y), c.z - (cq.z + shift.z));
            if (IMAGE) d = min_image(d.x, d.y, d.z, S);
            const float lim = S.rl + c.w + cq.w;
            hit = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)) < lim * lim && gq != grp;
        }
        const unsigned int m = __ballot_sync(0xffffffffu, hit);
        const int at = n + __popc(m & ((1u << lane) - 1u));
        if (hit && at < D.cap) list[at] = (unsigned int)(q - S.u0);
        n += __popc(m);
    }
}

constexpr int kBuildUnits = 8;  // units per warp of the list build
__global__ void __launch_bounds__(256) ff_build(FFDev D) {
    const int warps = (int)blockDim.x >> 5, warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    for (int k = 0; k < kBuildUnits; k++) {
        const int p = (blockIdx.x * kBuildUnits + k) * warps + warp;
        if (p >= D.n_units) return;
        const int s = D.usys[p];
        if (!D.rebuild[s]) continue;
        const FFSys S = D.sys[s];
        const float4 c = D.scen[p];
        const int grp = D.sgrp[p];
        unsigned int* list = D.nbr + (size_t)p * D.cap;
        int n = 0;
        if (S.nc == 1) {
            scan_run<true>(D, S, list, c, grp, make_float3(0.f, 0.f, 0.f), S.u0, S.u1, lane, n);
        } else {
            // the cells around the unit's own, one contiguous run of places per row (two where the row
            // wraps), with the row's periodic image shift (exact for units in range: a cell edge is at
            // least cutoff + skin + twice the largest radius, and there are at least three per edge)
            const int nc = S.nc, local = D.cell_of[D.unit_at[p]] - S.c0;
            const int cx = local % nc, cy = (local / nc) % nc, cz = local / (nc * nc);
            for (int oz = -1; oz <= 1; oz++) {
                int z = cz + oz;
                const float shz = z < 0 ? -S.L : (z >= nc ? S.L : 0.f);
                z = z < 0 ? z + nc : (z >= nc ? z - nc : z);
                for (int oy = -1; oy <= 1; oy++) {
                    int y = cy + oy;
                    const float shy = y < 0 ? -S.L : (y >= nc ? S.L : 0.f);
                    y = y < 0 ? y + nc : (y >= nc ? y - nc : y);
                    const int* row = D.cell_start + S.c0 + (z * nc + y) * nc;
                    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, nc - 1);
                    if (cx == 0)
                        scan_run<false>(D, S, list, c, grp, make_float3(-S.L, shy, shz), row[nc - 1], row[nc], lane, n);
                    scan_run<false>(D, S, list, c, grp, make_float3(0.f, shy, shz), row[x0], row[x1 + 1], lane, n);
                    if (cx == nc - 1)
                        scan_run<false>(D, S, list, c, grp, make_float3(S.L, shy, shz), row[0], row[1], lane, n);
                }
            }
        }
        if (lane == 0) {
            D.ncnt[p] = min(n, D.cap);
            if (n > D.cap && D.sys_status) atomicOr(D.sys_status + s, 2u);
        }
    }
}

// Compensated FP32 accumulator (Knuth's two-sum): the running sum keeps its rounding error in `lo`.
struct ESum {
    float hi = 0.0f, lo = 0.0f;
    __device__ __forceinline__ void add(float x) {
        const float s = hi + x, bp = s - hi;
        lo += (hi - (s - bp)) + (x - bp);
        hi = s;
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Relaxation: the factor that caps an atom's force.
__device__ __forceinline__ float force_scale(const FFDev& D, float fx, float fy, float fz) {
    const float f2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
    return D.fcap > 0.0f && f2 > D.fcap * D.fcap ? D.fcap * rsqrtf(f2) : 1.0f;
}

// A force component as OpenMM fixed point (2^32) in its place of the force array. Components are kept
// inside the fixed-point range (|F| < 2^31 kJ/mol/nm); a non-finite one, or one beyond the range
// (atoms on top of each other), marks its system as failed.
__device__ __forceinline__ void store_force(const FFDev& D, long long* __restrict__ to, float f, int si) {
    const float kMaxF = 2.0e9f;
    if (D.fcap <= 0.0f && !(fabsf(f) < kMaxF) && D.sys_status) atomicOr(D.sys_status + si, 1u);
    *to = __float2ll_rn(fminf(fmaxf(f, -kMaxF), kMaxF) * 0x1p32f);
}

// 8. Forces from the lists: one warp per unit, the unit's atoms in registers. The lanes take the list
// entries 32 at a time: each finds its listed unit's periodic shift (the minimum image of the
// centroids) and drops the entry when the centroids lie farther apart than cutoff + both radii (no
// pair of the two is then within the cutoff); a ballot packs the others into a per-warp ring. From
// the ring every lane takes one listed unit and pairs its atoms, one after another, with the atoms in
// registers. Each lane keeps partial sums per atom; a fixed butterfly of shuffles joins the lanes, so
// every force is a sum in a fixed order, with no atomics. A pair beyond the cutoff adds exactly
// nothing (its term is selected to zero, never multiplied), and neither does an unused record.
// Atoms sit at their images nearest their own unit's centroid, so the unit shift gives the minimum
// image of every pair within the cutoff when cutoff + two radii < L/2; systems of smaller boxes
// (FFSys::pair_image) take the minimum image per pair as well.
// With at most kMaxTypes atom types (PT) each pair's (K q_i q_j, 12 C12, 6 C6) comes from a type-pair
// table in shared memory, else from the atoms' own parameters by Lorentz-Berthelot.
// The pair term is OpenMM's CutoffPeriodic form: reaction-field Coulomb and unshifted LJ.
//
// Bound: instruction issue (64 % of the slots used), the L1 data pipe (67 %) and load latency, not HBM
// (6 %). Measured on 256 boxes of 64 to 4096 bodies of the water/tetrahedron/ring mix (1.07e6 atoms):
// 0.82 ms per step with list builds and integrator, against 1.22 for one warp per rigid body with its
// atoms in shared memory, neighbours expanded atom by atom through a queue, and the neighbours'
// records in list order. What made the difference: the unit's atoms in registers (no shared-memory
// load per pair), one listed unit per lane instead of one atom (a third of the entry work), records in
// cell order and by atom slot (contiguous lanes read contiguous records: a quarter fewer L1
// wavefronts), and no Lennard-Jones term for the atoms that have none. Not kept, all within 3 %: 80
// registers and 24 warps per SM, blocks of 4, 16 or 32 warps, two atoms at a time in packed FP32
// instructions (the FMA pipe takes as long; 5 % slower).
constexpr int kFW = 8;    // warps (units) per block
constexpr int kRing = 64;  // packed list entries per warp

struct UnitTask {
    int p, s, n, lane;        // place, system, list entries
    float4 c;                 // centroid and radius
    float4* ring;
};

// NI atoms of the unit, the first NL with Lennard-Jones (the others Coulomb only: their pairs skip it,
// and the unit's charge is applied once, to the sum). JS: atom records per place. RELAX: coincident
// atoms have no direction and add nothing. PI: the minimum image per pair.
template <int JS, int NI, int NL, bool ENERGY, bool PT, bool RELAX, bool PI>
__device__ __forceinline__ void unit_forces(const FFDev& D, const FFSys& S, const UnitTask& T, long long* __restrict__ force,
                                            int stride) {
    constexpr unsigned int kAll = 0xffffffffu;
    extern __shared__ float4 stab[];  // PT: the type-pair table
    const int lane = T.lane, nt = D.ntypes;
    const unsigned int* __restrict__ nb = D.nbr + (size_t)T.p * D.cap;
    const int u0 = S.u0;
    const float4 c = T.c;
    const float two_krf = 2.0f * S.krf, rc2 = S.rc2;
    float xi[NI][3], f[NI][3], qi[NI];
    const float4* row[NI];  // the atom's row of the type-pair table
    float4 pi[NI];
#pragma unroll
    for (int a = 0; a < NI; a++) {
        const float4 x = D.spos[a][T.p];
        xi[a][0] = x.x;
        xi[a][1] = x.y;
        xi[a][2] = x.z;
        f[a][0] = f[a][1] = f[a][2] = 0.0f;
        if (PT) {
            row[a] = stab + __float_as_int(x.w) * nt;
            qi[a] = stab[__float_as_int(x.w)].w;
        } else {
            pi[a] = D.spar[a][T.p];
        }
    }
    ESum en;
    // the atoms of one listed unit (place q, shift sh) against the unit's own
    auto stream = [&](float4 e, bool full) {
        const int q = __float_as_int(e.w);
        float4 xq[JS];
#pragma unroll
        for (int b = 0; b < JS; b++) xq[b] = full ? D.spos[b][q] : make_float4(kFar, kFar, kFar, 0.0f);
#pragma unroll
        for (int b = 0; b < JS; b++) {
            const float xj = xq[b].x + e.x, yj = xq[b].y + e.y, zj = xq[b].z + e.z;
            const int tj = __float_as_int(xq[b].w);
            float4 pj = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!PT && full) pj = D.spar[b][q];
            float qj = 0.0f;
            // K q_i q_j, 12 C12, 6 C6 of the pair (and, from the table, the streamed atom's charge)
            auto coefficients = [&](int a) {
                float4 t;
                if (PT) {
                    t = row[a][tj];
                    qj = t.w;
                } else {
                    const float sig = pi[a].y + pj.y, sig2 = sig * sig, sig6 = sig2 * sig2 * sig2;
                    const float c6 = 4.0f * (pi[a].z * pj.z) * sig6;
                    t = make_float4(pi[a].x * pj.x, 12.0f * c6 * sig6, 6.0f * c6, 0.0f);
                }
                return t;
            };
#pragma unroll
            for (int a = 0; a < NI; a++) {
                float3 d = make_float3(xi[a][0] - xj, xi[a][1] - yj, xi[a][2] - zj);
                if (PI) d = min_image(d.x, d.y, d.z, S);
                const float r2 = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
                const bool in = r2 < rc2 && !(PI && xq[b].x >= 0.5f * kFar) && !(RELAX && r2 < 1e-8f);
                const float inv_r = rsqrtf(r2), inv_r2 = inv_r * inv_r;
                const float rf = fmaf(inv_r, inv_r2, -two_krf);
                float gf;
                if (a < NL) {
                    const float4 t = coefficients(a);
                    const float inv_r6 = inv_r2 * inv_r2 * inv_r2;
                    const float lj = inv_r6 * fmaf(t.y, inv_r6, -t.z);  // 12 C12 r^-12 - 6 C6 r^-6
                    gf = fmaf(t.x, rf, lj * inv_r2);
                    if (ENERGY && in)
                        en.add(t.x * (inv_r + S.krf * r2 - S.crf) +
                               inv_r6 * (t.y * (1.0f / 12.0f) * inv_r6 - t.z * (1.0f / 6.0f)));
                } else {
                    gf = qj * rf;
                    if (ENERGY && in) en.add(qi[a] * qj * (inv_r + S.krf * r2 - S.crf));
                }
                gf = in ? gf : 0.0f;
                f[a][0] = fmaf(gf, d.x, f[a][0]);
                f[a][1] = fmaf(gf, d.y, f[a][1]);
                f[a][2] = fmaf(gf, d.z, f[a][2]);
            }
        }
    };
    const float reach = sqrtf(rc2) + c.w + 1e-6f;
    int head = 0, held = 0;  // the ring's first entry and length
    // list entries and their centroids are fetched a batch ahead of their use
    const int last = max(T.n - 1, 0);
    int q0 = T.n ? u0 + (int)nb[min(lane, last)] : u0, q1 = T.n ? u0 + (int)nb[min(32 + lane, last)] : u0;
    float4 c0 = D.scen[q0];
    for (int e0 = 0; e0 < T.n; e0 += 32) {
        const int q = q0;
        const float4 cj = c0;
        q0 = q1;
        c0 = D.scen[q1];
        q1 = u0 + (int)nb[min(e0 + 64 + lane, last)];
        const float dx = cj.x - c.x, dy = cj.y - c.y, dz = cj.z - c.z;
        const float4 e = make_float4(-S.L * rintf(dx * S.invL), -S.L * rintf(dy * S.invL), -S.L * rintf(dz * S.invL),
                                     __int_as_float(q));
        const float ex = dx + e.x, ey = dy + e.y, ez = dz + e.z;
        const float lim = reach + cj.w;
        const bool keep = e0 + lane < T.n && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < lim * lim;
        const unsigned int m = __ballot_sync(kAll, keep);
        if (keep) T.ring[(head + held + __popc(m & ((1u << lane) - 1u))) & (kRing - 1)] = e;
        held += __popc(m);
        __syncwarp();
        if (held >= 32) {
            stream(T.ring[(head + lane) & (kRing - 1)], true);
            head += 32;
            held -= 32;
            __syncwarp();
        }
    }
    if (held) stream(lane < held ? T.ring[(head + lane) & (kRing - 1)] : make_float4(0.f, 0.f, 0.f, 0.f), lane < held);
    // join the lanes (every lane ends with the same sums); lane 3 a + c stores component c of atom a
    const int u = D.unit_at[T.p];
    const int k0 = D.unit[u].x;
    float mine = 0.0f;
#pragma unroll
    for (int a = 0; a < NI; a++) {
        const float w = a < NL ? 1.0f : qi[a];
#pragma unroll
        for (int k = 0; k < 3; k++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) f[a][k] += __shfl_xor_sync(kAll, f[a][k], o);
            f[a][k] *= w;
        }
        const float cap = force_scale(D, f[a][0], f[a][1], f[a][2]);
#pragma unroll
        for (int k = 0; k < 3; k++)
            if (lane == 3 * a + k) mine = f[a][k] * cap;
    }
    if (lane < 3 * NI) store_force(D, force + D.iatom[k0 + lane / 3] + (size_t)(lane % 3) * stride, mine, T.s);
    if (ENERGY) {
        double e = en.value();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(kAll, e, o);
        if (lane == 0) D.e_unit[u] = 0.5 * e;
    }
}

// The unit's exact size (the same choice for every lane): 3 atoms of which one has LJ is a 3-site
// water; other units take the full term for every atom.
template <int JS, bool ENERGY, bool PT, bool RELAX, bool PI>
__device__ __forceinline__ void unit_dispatch(const FFDev& D, const FFSys& S, const UnitTask& T, int ni, int nl,
                                              long long* force, int stride) {
    if (JS >= 4 && ni == 4) return unit_forces<JS, JS >= 4 ? 4 : 1, JS >= 4 ? 4 : 1, ENERGY, PT, RELAX, PI>(D, S, T, force, stride);
    if (JS >= 3 && ni == 3) {
        if (PT && nl <= 1) return unit_forces<JS, JS >= 3 ? 3 : 1, 1, ENERGY, PT, RELAX, PI>(D, S, T, force, stride);
        return unit_forces<JS, JS >= 3 ? 3 : 1, JS >= 3 ? 3 : 1, ENERGY, PT, RELAX, PI>(D, S, T, force, stride);
    }
    if (JS >= 2 && ni == 2) return unit_forces<JS, JS >= 2 ? 2 : 1, JS >= 2 ? 2 : 1, ENERGY, PT, RELAX, PI>(D, S, T, force, stride);
    unit_forces<JS, 1, 1, ENERGY, PT, RELAX, PI>(D, S, T, force, stride);
}

// Blocks per SM: 64 registers for the pass of every step, more where a variant would spill.
template <int JS, bool ENERGY, bool PT> constexpr int force_blocks() {
    return JS <= 2 || (JS == 3 && PT && !ENERGY) ? 4 : PT || !ENERGY ? 3 : 2;
}

template <int JS, bool ENERGY, bool PT, bool RELAX>
__global__ void __launch_bounds__(32 * kFW, (force_blocks<JS, ENERGY, PT>())) ff_force(FFDev D, long long* __restrict__ force, int stride) {
    extern __shared__ float4 stab[];  // PT: the type-pair table
    __shared__ float4 ring[kFW][kRing];
    const int nt = D.ntypes;
    if (PT) {
        for (int t = threadIdx.x; t < nt * nt; t += blockDim.x) stab[t] = D.types[t];
        __syncthreads();
    }
    const int warp = (int)threadIdx.x >> 5;
    UnitTask T;
    T.p = blockIdx.x * kFW + warp;
    if (T.p >= D.n_units) return;
    T.lane = (int)threadIdx.x & 31;
    T.s = D.usys[T.p];
    T.n = D.ncnt[T.p];
    T.c = D.scen[T.p];
    T.ring = ring[warp];
    const FFSys S = D.sys[T.s];
    const int nn = D.unit[D.unit_at[T.p]].y, ni = nn & 0xff, nl = nn >> 8;
    if (S.pair_image)
        unit_dispatch<JS, ENERGY, PT, RELAX, true>(D, S, T, ni, nl, force, stride);
    else
        unit_dispatch<JS, ENERGY, PT, RELAX, false>(D, S, T, ni, nl, force, stride);
}

template <int JS, bool ENERGY, bool RELAX>
void launch_force_kernel(const FFDev& D, long long* f, int stride, cudaStream_t st) {
    const int grid = (D.n_units + kFW - 1) / kFW;
    if (D.ntypes)
        ff_force<JS, ENERGY, true, RELAX><<<grid, 32 * kFW, sizeof(float4) * D.ntypes * D.ntypes, st>>>(D, f, stride);
    else
        ff_force<JS, ENERGY, false, RELAX><<<grid, 32 * kFW, 0, st>>>(D, f, stride);
}

// A capped relaxation forms no energies.
template <int JS> void launch_force_pass(const FFDev& D, bool energy, long long* f, int stride, cudaStream_t st) {
    if (D.fcap > 0.0f) launch_force_kernel<JS, false, true>(D, f, stride, st);
    else if (energy) launch_force_kernel<JS, true, false>(D, f, stride, st);
    else launch_force_kernel<JS, false, false>(D, f, stride, st);
}

// One block per chunk of a system's units.
__global__ void ff_energy(FFDev D, double* part) {
    __shared__ double s[256];
    const int2 c = D.e_chunks.chunk[blockIdx.x];
    const int u0 = D.sys[c.x].u0 + c.y, u1 = min(u0 + kEnergyChunk, D.sys[c.x].u1);
    double e = 0.0;
    for (int u = u0 + (int)threadIdx.x; u < u1; u += blockDim.x) e += D.e_unit[u];
    s[threadIdx.x] = e;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

__global__ void forces_to_user(const long long* __restrict__ f, int stride, int n, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int c = 0; c < 3; c++) out[3 * i + c] = (double)f[i + c * stride] * 0x1p-32;
}

}  // namespace

int launch_forces_to_user(const long long* force, int stride, int natoms, double* out, void* stream) {
    if (natoms == 0) return 0;
    forces_to_user<<<(natoms + 255) / 256, 256, 0, (cudaStream_t)stream>>>(force, stride, natoms, out);
    return cudaPeekAtLastError() == cudaSuccess ? 1 : -1;
}

int launch_forces(const FFDev& D, int prec, const DevBuf& B, bool energy, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (D.n_int == 0) return 0;
    const int t = 256, gg = (D.n_units + t - 1) / t;
    int n = 0;
    ff_check<<<gg, t, 0, st>>>(D, B, prec);
    ff_bin<<<gg, t, 0, st>>>(D);
    ff_scan<<<D.S, 256, 0, st>>>(D);
    ff_scatter<<<gg, t, 0, st>>>(D);
    n += 4;
    if (D.n_mc) {
        ff_sort<<<(D.n_mc + kSortWarps - 1) / kSortWarps, 32 * kSortWarps, 0, st>>>(D);
        n++;
    }
    ff_place<<<gg, t, 0, st>>>(D, B, prec);
    // block size chosen by the autotuner (results do not depend on it: a warp builds each list)
    const int per_block = D.build_threads / 32 * kBuildUnits;
    ff_build<<<(D.n_units + per_block - 1) / per_block, D.build_threads, 0, st>>>(D);
    n += 2;
    if (cudaMemsetAsync(D.rebuild, 0, (size_t)D.S, st) != cudaSuccess) return -1;
    long long* f = const_cast<long long*>(B.force);
    switch (D.slots) {
        case 1: launch_force_pass<1>(D, energy, f, B.stride, st); break;
        case 2: launch_force_pass<2>(D, energy, f, B.stride, st); break;
        case 3: launch_force_pass<3>(D, energy, f, B.stride, st); break;
        default: launch_force_pass<4>(D, energy, f, B.stride, st);
    }
    n++;
    if (energy) {
        const SystemChunks& c = D.e_chunks;
        double* part = c.n == D.S ? D.energy : c.part;  // every system one chunk: its sum is the result
        ff_energy<<<c.n, 256, 0, st>>>(D, part);
        n++;
        if (part != D.energy) {
            if (launch_join_chunks(part, c.chunk0, D.S, 1, D.energy, stream) < 0) return -1;
            n++;
        }
    }
    return cudaPeekAtLastError() == cudaSuccess ? n : -1;
}

}  // namespace rbx
