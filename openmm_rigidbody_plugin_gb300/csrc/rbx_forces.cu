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
// One evaluation, all systems at once. Batches whose systems are all small (prep_limit) take
//   ff_prep     one block per system: each unit's centroid, radius and displacement since the last
//               build; lists that stay get their atoms' records at their places in cell order, the
//               others a new cell order first (cells of at least the reach, cutoff + skin + twice the
//               largest radius, or of half of it; counted, scanned and sorted in shared memory)
// and the others the same in kernels over all units (ff_check, ff_bin, ff_scan, ff_scatter,
// ff_place; those after ff_check return at once for systems whose lists stay). Then
//   ff_force    one warp per unit (all systems). Where the lists are to be rebuilt the warp first
//               builds its own: the units in range among the cells within one cell (of the reach) or
//               two (of half of it) of its own, rows of cells trimmed to the chord of the reach (in a
//               single-cell box: all units by minimum image), row by row. Then the forces: the
//               unit's atoms in registers, each lane taking one listed unit at a time; per-lane
//               partial sums joined by a fixed butterfly, no atomics; forces written as OpenMM fixed
//               point (2^32) to the slots
//   ff_energy   (energy evaluations only) one block per 2048 units of a system, joined per system:
//               fixed-order FP64 sum of its units' pair energies.
// All are launched as a chain (rbx_launch.cuh).
// The atoms of one group never meet in a list: pairs of one rigid body are excluded, as the
// plugin's ForceField helper removes them (python/forcefield.py:131-138).
#include <cuda_runtime.h>

#include <cstdint>

#include "rbx_cells.h"
#include "rbx_internal.h"
#include "rbx_launch.cuh"

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

// Minimum-image displacement.
__device__ __forceinline__ float3 min_image(float dx, float dy, float dz, const FFSys& S) {
    return make_float3(dx - S.L * rintf(dx * S.invL), dy - S.L * rintf(dy * S.invL), dz - S.L * rintf(dz * S.invL));
}

// Coordinate of the unused atom records of a place: outside every cutoff, its square finite.
constexpr float kFar = 1e10f;

// The unit's atoms at their images nearest its centroid c; returns the largest squared distance from it.
__device__ __forceinline__ float atoms_about(const FFSys& S, int n, float4 c, float3 (&x)[kMaxUnit]) {
    float rho2 = 0.f;
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++) {
        if (a >= n) break;
        const float3 d = min_image(x[a].x - c.x, x[a].y - c.y, x[a].z - c.z, S);
        rho2 = fmaxf(rho2, fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)));
        x[a] = make_float3(c.x + d.x, c.y + d.y, c.z + d.z);
    }
    return rho2;
}

// Positions of a unit's atoms.
__device__ __forceinline__ void unit_positions(const FFDev& D, const DevBuf& B, int prec, int k0, int n,
                                               float3 (&x)[kMaxUnit]) {
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++)
        if (a < n) x[a] = atom_position(B, prec, D.iatom[k0 + a]);
}

// Centroid of a unit (the mean of its atoms' minimum-image displacements from the first, wrapped
// into the box) and its radius; x: its atoms about it.
__device__ __forceinline__ float4 unit_centroid(const FFDev& D, const DevBuf& B, int prec, const FFSys& S, int k0, int n,
                                                float3 (&x)[kMaxUnit]) {
    unit_positions(D, B, prec, k0, n, x);
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
    float4 c = make_float4(wrap_coordinate(fmaf(sx, inv, x[0].x), S.L, S.invL),
                           wrap_coordinate(fmaf(sy, inv, x[0].y), S.L, S.invL),
                           wrap_coordinate(fmaf(sz, inv, x[0].z), S.L, S.invL), 0.0f);
    c.w = sqrtf(atoms_about(S, n, c, x));
    return c;
}

// A unit's records at place p: centroid, and its atoms (at their images nearest the centroid, so that
// one periodic shift moves a whole unit) with their types.
__device__ __forceinline__ void write_place(const FFDev& D, int p, int k0, int n, float4 c, const float3 (&x)[kMaxUnit]) {
    D.scen[p] = c;
#pragma unroll
    for (int a = 0; a < kMaxUnit; a++) {
        if (a >= D.slots) break;
        D.spos[a][p] = a < n ? make_float4(x[a].x, x[a].y, x[a].z, D.atype ? __int_as_float(D.atype[k0 + a]) : 0.0f)
                     : make_float4(kFar, kFar, kFar, 0.0f);
    }
}

// Cell of a centroid in its system.
__device__ __forceinline__ int cell_index(const FFSys& S, float4 c) {
    return (cell_of(c.z, S.invL, S.nc) * S.nc + cell_of(c.y, S.invL, S.nc)) * S.nc + cell_of(c.x, S.invL, S.nc);
}

// Key of a unit in the order within its cell: its place on a 4 x 4 x 4 grid of the cell in Z-order,
// then its index, so that the units a list takes of one cell lie in short runs of places and a run of
// places is compact.
constexpr unsigned int kKeyUnit = (1u << 26) - 1;
__device__ __forceinline__ unsigned int cell_key(const FFSys& S, float4 c, int u) {
    const float x[3] = {c.x, c.y, c.z};
    unsigned int z = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int g = (int)(x[k] * S.invL * (float)(4 * S.nc)) & 3;
        z |= (unsigned int)((g & 1) << k | (g >> 1) << (3 + k));
    }
    return z << 26 | (unsigned int)(u - S.u0);
}

__device__ __forceinline__ bool moved_too_far(const FFDev& D, const FFSys& S, int u, float4 c) {
    const float4 r = D.uref[u];
    const float3 d = min_image(c.x - r.x, c.y - r.y, c.z - r.z, S);
    return fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)) > D.half_skin2;
}

// Unit u at its new place p: records, group, build centroid (the one that its cell was taken from).
__device__ __forceinline__ void settle(const FFDev& D, const DevBuf& B, int prec, const FFSys& S, int u, int p) {
    const int2 kn = D.unit[u];
    const int k0 = kn.x, n = kn.y & 0xff;
    float3 x[kMaxUnit];
    const float4 c = D.ucen[u];
    unit_positions(D, B, prec, k0, n, x);
    atoms_about(S, n, c, x);
    write_place(D, p, k0, n, c, x);
    if (D.spar[0])
        for (int a = 0; a < D.slots; a++) D.spar[a][p] = a < n ? D.param[k0 + a] : make_float4(0.f, 0.f, 0.f, 0.f);
    D.place[u] = p;
    D.unit_at[p] = u;
    D.sgrp[p] = D.ugrp[u];
    D.sunit[p] = kn;
    D.uref[u] = c;
}

// Exclusive scan of n counts by a block: each thread a run of them, the runs' sums by warp shuffles.
// put(i, start) receives every start. Each count is read twice, by the same thread and last before its put, which
// may so overwrite it. Ends without a barrier.
template <class Count, class Put>
__device__ __forceinline__ void block_scan(int n, int* wsum, const Count& count, const Put& put) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int per = (n + nthr - 1) / nthr, i0 = min(tid * per, n), i1 = min(i0 + per, n);
    int sum = 0;
    for (int i = i0; i < i1; i++) sum += count(i);
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += v;
    }
    if ((tid & 31) == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    int at = incl - sum;
    for (int w = 0; w < (tid >> 5); w++) at += wsum[w];
    for (int i = i0; i < i1; i++) {
        const int c = count(i);
        put(i, at);
        at += c;
    }
}

// Everything before the force pass for one system, in one block. The cell counts and the keys of the
// system's units, in cell order, are in shared memory. Within a cell units are ranked by key (all
// different), so the order does not depend on the order of the atomics.
// Bound: latency (a chain of dependent loads, and in rebuilds a dozen barriers), so one launch in place
// of six. Per 20 steps with energies and a frame: 512 waters 539 against 623 us in separate kernels, 24
// boxes of 64 to 190 bodies 708 against 832.
__global__ void __launch_bounds__(1024) ff_prep(FFDev D, DevBuf B, int prec) {
    extern __shared__ unsigned int keys[];  // prep_units
    __shared__ int wsum[32];
    int* cell = (int*)(keys + D.prep_units);  // prep_cells
    const int s = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    chain_release();
    const FFSys S = D.sys[s];
    chain_wait();
    bool build = D.force_all;
    for (int u = S.u0 + tid; u < S.u1; u += nthr) {
        const int2 kn = D.unit[u];
        const int k0 = kn.x, n = kn.y & 0xff;
        float3 x[kMaxUnit];
        const float4 c = unit_centroid(D, B, prec, S, k0, n, x);
        D.ucen[u] = c;
        if (D.force_all) continue;
        write_place(D, D.place[u], k0, n, c, x);
        build |= moved_too_far(D, S, u, c);
    }
    build = __syncthreads_or(build);
    if (tid == 0) {
        D.build[s] = build;
        if (build) D.rebuilds[s]++;
    }
    if (!build) return;
    if (S.nc == 1) {  // one cell: unit order
        for (int u = S.u0 + tid; u < S.u1; u += nthr) settle(D, B, prec, S, u, u);
        return;
    }
    const int ncell = S.nc * S.nc * S.nc, units = S.u1 - S.u0;
    for (int i = tid; i < ncell; i += nthr) cell[i] = 0;
    __syncthreads();
    for (int u = S.u0 + tid; u < S.u1; u += nthr) atomicAdd(cell + cell_index(S, D.ucen[u]), 1);
    __syncthreads();
    block_scan(ncell, wsum, [&](int i) { return cell[i]; },
               [&](int i, int at) {
                   cell[i] = at;
                   D.cell_start[S.c0 + i] = S.u0 + at;
               });
    if (tid == 0) D.cell_start[S.c0 + ncell] = S.u1;
    __syncthreads();
    for (int u = S.u0 + tid; u < S.u1; u += nthr) {
        const float4 c = D.ucen[u];
        keys[atomicAdd(cell + cell_index(S, c), 1)] = cell_key(S, c, u);
    }
    __syncthreads();  // cell[i] is now the end of cell i
    for (int i = tid; i < units; i += nthr) {
        const unsigned int key = keys[i];
        const int u = S.u0 + (int)(key & kKeyUnit), c = cell_index(S, D.ucen[u]);
        const int b = c ? cell[c - 1] : 0, e = cell[c];
        int rank = 0;
        for (int j = b; j < e; j++) rank += keys[j] < key;
        settle(D, B, prec, S, u, S.u0 + b + rank);
    }
}

// The same for batches with larger systems, in kernels over all units.
// Per unit: centroid, radius and the rebuild test.
__global__ void ff_check(FFDev D, DevBuf B, int prec) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    chain_release();
    chain_wait();
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    const FFSys S = D.sys[s];
    const int2 kn = D.unit[u];
    const int k0 = kn.x, n = kn.y & 0xff;
    float3 x[kMaxUnit];
    const float4 c = unit_centroid(D, B, prec, S, k0, n, x);
    D.ucen[u] = c;
    if (D.force_all) return;
    write_place(D, D.place[u], k0, n, c, x);
    if (moved_too_far(D, S, u, c)) D.moved[s] = 1;
}

// Whether a system's lists are rebuilt in this evaluation (after ff_check).
__device__ __forceinline__ bool rebuilding(const FFDev& D, int s) { return D.force_all || D.moved[s]; }

__global__ void ff_bin(FFDev D) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    chain_release();
    chain_wait();
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    if (!rebuilding(D, s)) return;
    const FFSys S = D.sys[s];
    if (S.nc > 1) atomicAdd(D.cell_count + S.c0 + cell_index(S, D.ucen[u]), 1);
}

// One block per system: its cells' starts, the counts reset, and whether its lists are rebuilt.
__global__ void __launch_bounds__(1024) ff_scan(FFDev D) {
    __shared__ int wsum[32];
    chain_release();
    chain_wait();
    const int s = blockIdx.x;
    const bool build = rebuilding(D, s);
    if (threadIdx.x == 0) {
        D.build[s] = build;
        if (build) D.rebuilds[s]++;
    }
    if (!build) return;
    const FFSys S = D.sys[s];
    if (S.nc == 1) return;
    const int ncell = S.nc * S.nc * S.nc;
    int* count = D.cell_count + S.c0;
    block_scan(ncell, wsum, [&](int i) { return count[i]; },
               [&](int i, int at) {
                   D.cell_start[S.c0 + i] = S.u0 + at;
                   D.cell_cursor[S.c0 + i] = S.u0 + at;
                   count[i] = 0;
               });
    if (threadIdx.x == 0) D.cell_start[S.c0 + ncell] = S.u1;
}

// Keys of the units of multi-cell boxes, cell by cell (in the order of the atomics).
__global__ void ff_scatter(FFDev D) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    chain_release();
    chain_wait();
    if (u >= D.n_units) return;
    const int s = D.usys[u];
    if (!rebuilding(D, s)) return;
    const FFSys S = D.sys[s];
    if (S.nc == 1) return;
    const float4 c = D.ucen[u];
    D.skey[atomicAdd(D.cell_cursor + S.c0 + cell_index(S, c), 1)] = cell_key(S, c, u);
}

// Every unit of the rebuilt systems at its place: in its cell, by rank of its key (single-cell boxes:
// unit order).
__global__ void ff_place(FFDev D, DevBuf B, int prec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    chain_release();
    chain_wait();
    if (i >= D.n_units) return;
    const int s = D.usys[i];  // places [u0, u1) belong to the system of unit i
    if (!rebuilding(D, s)) return;
    const FFSys S = D.sys[s];
    if (S.nc == 1) return settle(D, B, prec, S, i, i);
    const unsigned int key = D.skey[i];
    const int u = S.u0 + (int)(key & kKeyUnit);
    const int* start = D.cell_start + S.c0 + cell_index(S, D.ucen[u]);
    const int b = start[0], e = start[1];
    int rank = 0;
    for (int j = b; j < e; j++) rank += D.skey[j] < key;
    settle(D, B, prec, S, u, b + rank);
}

// The list of the unit at place p starts at entry 32 list_row.
__device__ __forceinline__ int list_row(const FFSys& S, int p) { return S.list0 + (p - S.u0) * (S.cap >> 5); }

// Lists, a warp per unit: the lanes test 32 candidates at a time and append the ones in range in order,
// a ballot giving each its slot (coalesced). The candidates are the units of the cells within reach,
// row of cells by row: in place order a row is one contiguous run (two where it crosses the box's
// edge), trimmed to the chord of the reach through the row, and the runs are taken as one sequence, so
// that the lanes stay full however short they are. Entries past the list's capacity are counted, not stored
// (the force pass then takes every unit of the system instead of the list).
// Bound: load latency and issue. Cells of half the reach, trimmed, leave about 650 candidates of a
// water's 214 entries; cells of the whole reach (27 of them, untrimmed) had 1600. 20 steps with energies
// and a frame: 66,666 waters 5.0 -> 4.4 ms, 256 boxes of the mix 16.3 -> 14.7; forces of 15,001 bodies
// 0.32 -> 0.26. kAhead chunks of
// candidates are in flight. Built by the force pass itself: a kernel of its own, which has nothing to do
// in most steps, cost 588 against 531 us per 20 steps of 512 waters.
// Returns the length of the list of the unit at place p with centroid c; runs: scratch of 32 records. STORE:
// the list and its length are stored.
template <bool STORE>
__device__ __forceinline__ int build_list(const FFDev& D, const FFSys& S, int p, float4 c, int lane, float4* runs) {
    constexpr unsigned int kAll = 0xffffffffu;
    constexpr int kAhead = 2;
    const int grp = D.sgrp[p];
    unsigned int* list = STORE ? D.nbr + (size_t)32 * list_row(S, p) : nullptr;
    const bool image = S.nc == 1;  // one run, the whole box: minimum image per pair
    const int nc = S.nc, w = S.win, side = 2 * w + 1;
    const int cx = cell_of(c.x, S.invL, nc), cy = cell_of(c.y, S.invL, nc), cz = cell_of(c.z, S.invL, nc);
    // the lane's row of cells and those of it within reach, in an unwrapped count
    CellRange within = {0, -1};
    const int* row = nullptr;
    float sy = 0.f, sz = 0.f;
    if (!image && lane < side * side) {
        int z = cz + lane / side - w, y = cy + lane % side - w;
        const float e = S.L / (float)nc, ie = S.invL * (float)nc, reach = S.reach + c.w;
        const float tz = fmaxf(fmaxf((float)z * e - c.z, c.z - (float)(z + 1) * e), 0.0f);
        const float ty = fmaxf(fmaxf((float)y * e - c.y, c.y - (float)(y + 1) * e), 0.0f);
        const float h2 = reach * reach - fmaf(ty, ty, tz * tz);
        if (h2 > 0.0f) within = cells_within(c.x, sqrtf(h2), ie, cx, w);
        sz = z < 0 ? -S.L : (z >= nc ? S.L : 0.f);
        z = z < 0 ? z + nc : (z >= nc ? z - nc : z);
        sy = y < 0 ? -S.L : (y >= nc ? S.L : 0.f);
        y = y < 0 ? y + nc : (y >= nc ? y - nc : y);
        row = D.cell_start + S.c0 + (z * nc + y) * nc;
    }
    int n = 0;
    // the parts of the rows inside the box, then the parts across its edge. The periodic shifts are exact
    // for units in range: there are at least 2 w + 1 cells per edge.
    const int parts = !image && (cx < w || cx >= nc - w) ? 2 : 1;
    for (int part = 0; part < parts; part++) {
        int r0 = 0, r1 = 0;
        float sx = 0.f;
        if (image) {
            if (lane == 0) {
                r0 = S.u0;
                r1 = S.u1;
            }
        } else {
            const CellRange in = range_part(within, part, cx, w, nc);
            if (part == 1) sx = cx < w ? -S.L : S.L;
            if (in.a <= in.b) {
                r0 = row[in.a];
                r1 = row[in.b + 1];
            }
        }
        // the runs that hold anything, packed: run k covers the sequence from first[k] on
        int first = r1 - r0;
        const bool any = first > 0;
        const int len = first;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kAll, first, o);
            if (lane >= o) first += v;
        }
        const int total = __shfl_sync(kAll, first, 31);
        first -= len;
        const unsigned int held = __ballot_sync(kAll, any);
        __syncwarp();
        if (any) runs[__popc(held & ((1u << lane) - 1u))] = make_float4(__int_as_float(r0 - first), sy, sz, 0.0f);
        __syncwarp();
        int before = 0;  // runs that begin before the chunk
        for (int f0 = 0; f0 < total; f0 += 32 * kAhead) {
            int q[kAhead], gq[kAhead];
            float4 cq[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; k++) {
                const int f = f0 + 32 * k, at = first - f;
                const unsigned int begins = __reduce_or_sync(kAll, any && at >= 0 && at < 32 ? 1u << at : 0u);
                const int r = before + __popc(begins & (0xffffffffu >> (31 - lane))) - 1;
                before += __popc(begins);
                const float4 run = runs[max(r, 0)];
                const bool on = f + lane < total;
                q[k] = on ? __float_as_int(run.x) + f + lane : S.u0;
                cq[k] = D.scen[q[k]];
                gq[k] = on ? D.sgrp[q[k]] : grp;
                cq[k].x += sx;
                cq[k].y += run.y;
                cq[k].z += run.z;
            }
#pragma unroll
            for (int k = 0; k < kAhead; k++) {
                float3 d = make_float3(c.x - cq[k].x, c.y - cq[k].y, c.z - cq[k].z);
                if (image) d = min_image(d.x, d.y, d.z, S);
                const float lim = S.rl + c.w + cq[k].w;
                const bool hit = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z)) < lim * lim && gq[k] != grp;
                const unsigned int m = __ballot_sync(kAll, hit);
                const int at = n + __popc(m & ((1u << lane) - 1u));
                if (STORE && hit && at < S.cap) list[at] = (unsigned int)(q[k] - S.u0);
                n += __popc(m);
            }
        }
    }
    if (STORE && lane == 0) D.ncnt[p] = n;
    __syncwarp();  // the lanes read each other's entries
    return n;
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

// The longest list of each system (most, zero before), a warp per unit.
__global__ void __launch_bounds__(128) ff_list_lengths(FFDev D, int* most) {
    __shared__ float4 runs[4][32];
    chain_release();
    chain_wait();
    const int warp = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31, p = blockIdx.x * 4 + warp;
    if (p >= D.n_units) return;
    const int s = D.usys[p];
    const FFSys S = D.sys[s];
    const int n = build_list<false>(D, S, p, D.scen[p], lane, runs[warp]);
    if (lane == 0) atomicMax(most + s, n);
}

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

// Forces from the lists: one warp per unit, the unit's atoms in registers. The lanes take the list
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
// In systems of at most kMaxTypes atom types each pair's (K q_i q_j, 12 C12, 6 C6) comes from a type-pair table, else
// from the atoms' own parameters by Lorentz-Berthelot (the two round differently, so the form follows from the
// system alone). The table is in shared memory where one holds the types of the whole batch, else the system's
// own is read through L1.
// The pair term is OpenMM's CutoffPeriodic form: reaction-field Coulomb and unshifted LJ.
//
// Bound: instruction issue (62 % of the slots used), the L1 data pipe (53 to 67 %) and load latency, not
// HBM (6 %). Measured per step of 256 boxes of 64 to 4096 bodies of the water/tetrahedron/ring mix
// (1.07e6 atoms), list builds and integrator included: 0.73 ms, against 1.22 for one warp per rigid
// body with its atoms in shared memory, neighbours expanded atom by atom through a queue, and the
// neighbours' records in list order. What made the difference: the unit's atoms in registers (no
// shared-memory load per pair), one listed unit per lane instead of one atom (a third of the entry
// work), records in cell order and by atom slot (contiguous lanes read contiguous records: a quarter
// fewer L1 wavefronts), no Lennard-Jones term for the atoms that have none; then (17.5 -> 16.3 ms per
// 20 steps) all that a place names fetched at once, predicated sums, halving sums over the lanes and
// blocks of 4 warps (8: 16.7). Every pair's energy is added to the compensated sum on its own, without
// branches; the pairs of one streamed atom added up first, in plain FP32, were narrower and no faster (forces
// of 40 boxes with solutes 739 us, now 728). Not kept: 40 warps per SM at 48 registers
// (19.2 ms); 24 at 80, with (20.5) or without (equal) the next atoms fetched before these are paired;
// two atoms at a time in packed FP32 instructions (the FMA pipe takes as long; 5 % slower).
constexpr int kFW = 4;    // warps (units) per block
constexpr int kRing = 64;  // packed list entries per warp

enum PairForm { kAtomParams, kSharedTable, kSystemTable };

struct UnitTask {
    int p, s, n, lane;        // place, system, list entries
    int row;                  // the unit's list (list_row), or where more units are in range than it holds
                              // -1 - its group: every place of the system (the list at row 0) but the group's
    int k0;                   // the unit's first interacting atom
    int q0, q1;               // the lane's first two list entries (before clamping to n)
    int2 types;               // kSystemTable: FFDev::sys_types of the system
    float4 c;                 // centroid and radius
    float4* ring;
};

// Sums of N values over the warp, each in one lane: at every step a lane hands half of its values to its
// partner and takes the partner's share of the other half, so the work halves (N = 9: 12 shuffles
// instead of 45). Returns the index of the value that the lane ends with, in v[0], or -1. Lanes that
// differ in bit 0 end with the same value; the even one has it.
template <int M, int O, int N> __device__ __forceinline__ void join_step(float (&v)[N], int lane, int& first, int& count) {
    if constexpr (O > 0) {
        constexpr int K = (M + 1) / 2;
        if constexpr (M == 1) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            if (lane & O) count = 0;
        } else {
            const bool up = (lane & O) != 0;
#pragma unroll
            for (int i = 0; i < K; i++) {
                const float hi = i + K < M ? v[i + K] : 0.0f;
                const float give = up ? v[i] : hi, keep = up ? hi : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
            }
            first += up ? K : 0;
            count = up ? count - K : min(count, K);
        }
        join_step<K, O / 2>(v, lane, first, count);
    }
}
template <int N> __device__ __forceinline__ int join_lanes(float (&v)[N], int lane) {
    int first = 0, count = N;
    join_step<N, 16>(v, lane, first, count);
    return count > 0 ? first : -1;
}

// NI atoms of the unit, the first NL with Lennard-Jones (the others Coulomb only: their pairs skip it,
// and the unit's charge is applied once, to the sum). JS: atom records per place. RELAX: coincident
// atoms have no direction and add nothing. PI: the minimum image per pair.
template <int JS, int NI, int NL, bool ENERGY, PairForm PF, bool RELAX, bool PI>
__device__ __forceinline__ void unit_forces(const FFDev& D, const FFSys& S, const UnitTask& T, long long* __restrict__ force,
                                            int stride) {
    constexpr unsigned int kAll = 0xffffffffu;
    constexpr bool PT = PF != kAtomParams;
    extern __shared__ float4 stab[];  // kSharedTable: the type-pair table
    const float4* const table = PF == kSharedTable ? stab : D.types + T.types.x;
    const int lane = T.lane, nt = PF == kSharedTable ? D.ntypes : T.types.y;
    const unsigned int* nb = D.nbr + (size_t)32 * max(T.row, 0);
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
            row[a] = table + __float_as_int(x.w) * nt;
            qi[a] = table[__float_as_int(x.w)].w;
        } else {
            pi[a] = D.spar[a][T.p];
            qi[a] = pi[a].x;
        }
    }
    ESum en;
    // the atoms xq of one listed unit (place and shift e) against the unit's own
    auto pairs = [&](const float4 (&xq)[JS], float4 e) {
#pragma unroll
        for (int b = 0; b < JS; b++) {
            const float xj = xq[b].x + e.x, yj = xq[b].y + e.y, zj = xq[b].z + e.z;
            const int tj = __float_as_int(xq[b].w);
            float4 pj;
            if (!PT) pj = D.spar[b][__float_as_int(e.w)];
            float qj = PT ? 0.0f : pj.x;
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
                // (energies with their roundings written out: the same in every form of the kernel)
                const float coulomb_energy = __fadd_rn(__fmaf_rn(S.krf, r2, inv_r), -S.crf);
                float gf;
                if (a < NL) {
                    const float4 t = coefficients(a);
                    const float inv_r6 = inv_r2 * inv_r2 * inv_r2;
                    const float lj = inv_r6 * fmaf(t.y, inv_r6, -t.z);  // 12 C12 r^-12 - 6 C6 r^-6
                    gf = fmaf(t.x, rf, lj * inv_r2);
                    if (ENERGY) {
                        const float lj_energy = __fmaf_rn(__fmul_rn(t.y, 1.0f / 12.0f), inv_r6, -__fmul_rn(t.z, 1.0f / 6.0f));
                        en.add(in ? __fmaf_rn(t.x, coulomb_energy, __fmul_rn(inv_r6, lj_energy)) : 0.0f);
                    }
                } else {
                    gf = qj * rf;
                    if (ENERGY) en.add(in ? __fmul_rn(__fmul_rn(qi[a], qj), coulomb_energy) : 0.0f);
                }
                if (in) {
                    f[a][0] = fmaf(gf, d.x, f[a][0]);
                    f[a][1] = fmaf(gf, d.y, f[a][1]);
                    f[a][2] = fmaf(gf, d.z, f[a][2]);
                }
            }
        }
    };
    const float reach = S.rc + c.w + 1e-6f;
    const int slot = D.iatom[T.k0 + min(lane / 3, NI - 1)];
    int head = 0, held = 0;  // the ring's first entry and length
    // list entries and their centroids are fetched a batch ahead of their use
    // (entries past the list's end, whatever the memory holds, become the system's first place)
    const int last = max(T.n - 1, 0);
    int q0 = u0 + (lane < T.n ? T.q0 : 0), q1 = u0 + (lane + 32 < T.n ? T.q1 : 0);
    float4 c0 = D.scen[q0];
    for (int e0 = 0;;) {
        while (held < 32 && e0 < T.n) {
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
            bool keep = e0 + lane < T.n && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) < lim * lim;
            if (T.row < 0) keep = keep && D.sgrp[q] != -1 - T.row;  // (a branch: as one condition 1.5 % slower)
            const unsigned int m = __ballot_sync(kAll, keep);
            if (keep) T.ring[(head + held + __popc(m & ((1u << lane) - 1u))) & (kRing - 1)] = e;
            held += __popc(m);
            e0 += 32;
            __syncwarp();
        }
        if (held == 0) break;
        float4 x[JS], e = make_float4(0.f, 0.f, 0.f, __int_as_float(u0));
        if (lane < held) {
            e = T.ring[(head + lane) & (kRing - 1)];
#pragma unroll
            for (int b = 0; b < JS; b++) x[b] = D.spos[b][__float_as_int(e.w)];
        } else {
#pragma unroll
            for (int b = 0; b < JS; b++) x[b] = make_float4(kFar, kFar, kFar, 0.0f);
        }
        head += 32;
        held = max(held - 32, 0);
        pairs(x, e);
        __syncwarp();
    }
    // join the lanes; every component of every atom's force is stored by one lane
#pragma unroll
    for (int a = NL; a < NI; a++)
#pragma unroll
        for (int k = 0; k < 3; k++) f[a][k] *= qi[a];
    float v[3 * NI];
    if (RELAX) {  // every lane ends with all sums, for the cap on an atom's force
        float mine = 0.0f;
#pragma unroll
        for (int a = 0; a < NI; a++) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) f[a][k] += __shfl_xor_sync(kAll, f[a][k], o);
            }
            const float cap = force_scale(D, f[a][0], f[a][1], f[a][2]);
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (lane == 3 * a + k) mine = f[a][k] * cap;
        }
        if (lane < 3 * NI) store_force(D, force + slot + (size_t)(lane % 3) * stride, mine, T.s);
    } else {
#pragma unroll
        for (int a = 0; a < NI; a++)
#pragma unroll
            for (int k = 0; k < 3; k++) v[3 * a + k] = f[a][k];
        const int at = join_lanes(v, lane);
        const int to = __shfl_sync(kAll, slot, max(at, 0) / 3 * 3);
        if (at >= 0) store_force(D, force + to + (size_t)(at % 3) * stride, v[0], T.s);
    }
    if (ENERGY) {
        double e = en.value();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(kAll, e, o);
        if (lane == 0) D.e_unit[D.unit_at[T.p]] = 0.5 * e;
    }
}

// The unit's exact size (the same choice for every lane): 3 atoms of which one has LJ is a 3-site
// water, with a pair table or without (20 steps of 40 boxes of 700 to 3100 waters around 64-type solutes
// 5.95 -> 5.57 ms for the latter); other units take the full term for every atom.
template <int JS, bool ENERGY, PairForm PF, bool RELAX, bool PI>
__device__ __forceinline__ void unit_dispatch(const FFDev& D, const FFSys& S, const UnitTask& T, int ni, int nl,
                                              long long* force, int stride) {
    if (JS >= 4 && ni == 4) return unit_forces<JS, JS >= 4 ? 4 : 1, JS >= 4 ? 4 : 1, ENERGY, PF, RELAX, PI>(D, S, T, force, stride);
    if (JS >= 3 && ni == 3) {
        if (nl <= 1) return unit_forces<JS, JS >= 3 ? 3 : 1, 1, ENERGY, PF, RELAX, PI>(D, S, T, force, stride);
        return unit_forces<JS, JS >= 3 ? 3 : 1, JS >= 3 ? 3 : 1, ENERGY, PF, RELAX, PI>(D, S, T, force, stride);
    }
    if (JS >= 2 && ni == 2) return unit_forces<JS, JS >= 2 ? 2 : 1, JS >= 2 ? 2 : 1, ENERGY, PF, RELAX, PI>(D, S, T, force, stride);
    unit_forces<JS, 1, 1, ENERGY, PF, RELAX, PI>(D, S, T, force, stride);
}

// Blocks per SM: 64 registers a thread (32 warps per SM); 80 for units of four atoms. The larger variants
// then spill a little and still gain: forces of 40 boxes with 64-type solutes take 1.09 ms at 128
// registers, 0.98 at 80 and 0.97 at 64 (later, with the list build's code, 0.75 at 80 and 0.77 at 64: the
// form without the type-pair table takes 80, and so does the one with tables per system: 20 steps of 20 boxes
// of waters beside 20 with solutes 4.95 ms, at 64 registers 5.16, at 96 4.93, at 128 5.46; now 4.85, and 4.87
// without any table, as such batches once were).
constexpr int force_blocks(int records) { return records <= 3 ? 8 : 6; }
constexpr int kUntypedBlocks = 6;
// Batches of at most kFewUnits units (two warps per scheduler) leave the SMs nearly empty: a warp's own
// chain of instructions is then the time, and 128 registers let more of it overlap (512 waters, 20 steps
// with energies and a frame: 475 against 537 us; at 2600 units, 683 against 662). With tables per system, whose
// kernel is the larger, up to a wave of such blocks, twice that (1770 units in four boxes of the mix beside two
// with solutes, 20 steps: 0.50 against 0.62 ms).
constexpr int kFewUnits = 8 * kSMs, kFewBlocks = 4;

// PF: kSharedTable, one table for the batch; kSystemTable, a table for some of its systems; kAtomParams, for none.
template <int JS, bool ENERGY, PairForm PF, bool RELAX, int BLOCKS>
__global__ void __launch_bounds__(32 * kFW, BLOCKS) ff_force(FFDev D, long long* __restrict__ force, int stride) {
    extern __shared__ float4 stab[];  // kSharedTable: the type-pair table
    __shared__ float4 ring[kFW][kRing];
    chain_release();
    const int nt = D.ntypes;
    if (PF == kSharedTable) {
        for (int t = threadIdx.x; t < nt * nt; t += blockDim.x) stab[t] = D.types[t];
        __syncthreads();
    }
    const int warp = (int)threadIdx.x >> 5;
    UnitTask T;
    T.p = blockIdx.x * kFW + warp;
    const bool on = T.p < D.n_units;
    T.lane = (int)threadIdx.x & 31;
    T.s = on ? D.usys[T.p] : 0;
    const FFSys S = D.sys[T.s];
    if (PF == kSystemTable) T.types = D.sys_types[T.s];
    chain_wait();
    if (!on) return;
    T.ring = ring[warp];
    // all that the place names is fetched at once: a warp's chain of dependent loads is short
    T.c = D.scen[T.p];
    T.n = D.ncnt[T.p];
    const int2 kn = D.sunit[T.p];
    T.row = list_row(S, T.p);
    const unsigned int* nb = D.nbr + (size_t)32 * T.row;
    T.q0 = (int)nb[T.lane];
    T.q1 = (int)nb[min(32 + T.lane, S.cap - 1)];
    if (D.build[T.s]) {
        T.n = build_list<true>(D, S, T.p, T.c, T.lane, T.ring);
        T.q0 = (int)nb[T.lane];
        T.q1 = (int)nb[min(32 + T.lane, S.cap - 1)];
    }
    if (T.n > S.cap) {
        T.n = S.u1 - S.u0;
        T.row = -1 - D.sgrp[T.p];
        T.q0 = T.lane;
        T.q1 = 32 + T.lane;
    }
    if (T.p == S.u0 && T.lane == 0) D.moved[T.s] = 0;  // for the next evaluation's ff_check
    T.k0 = kn.x;
    const int ni = kn.y & 0xff, nl = kn.y >> 8;
    if (PF == kSystemTable && T.types.y == 0) {
        if (S.pair_image) return unit_dispatch<JS, ENERGY, kAtomParams, RELAX, true>(D, S, T, ni, nl, force, stride);
        return unit_dispatch<JS, ENERGY, kAtomParams, RELAX, false>(D, S, T, ni, nl, force, stride);
    }
    if (S.pair_image) return unit_dispatch<JS, ENERGY, PF, RELAX, true>(D, S, T, ni, nl, force, stride);
    unit_dispatch<JS, ENERGY, PF, RELAX, false>(D, S, T, ni, nl, force, stride);
}

// Shared memory is set aside for the resident blocks only (each its ring, its table and 1 KB of the
// system's), so that L1 has the rest: left to itself the driver took 100 KB where 8 blocks hold 42. Per 20
// steps: 256 boxes of the mix 14.72 -> 14.54 ms, 60 boxes 3.94 -> 3.89, 66,666 waters 4.42 -> 4.37.
template <int JS, bool ENERGY, bool RELAX>
cudaError_t launch_force_kernel(const FFDev& D, long long* f, int stride, cudaStream_t st) {
    const int grid = (D.n_units + kFW - 1) / kFW;
    const size_t table = sizeof(float4) * D.ntypes * D.ntypes;
    auto launch = [&](int blocks, void (*kernel)(FFDev, long long*, int)) {
        const size_t block_shared = sizeof(float4) * kFW * kRing + table + 1024;
        return launch_chained_l1<FFDev, long long*, int>(blocks * block_shared, kernel, grid, 32 * kFW, table, st, D, f, stride);
    };
    if constexpr (!RELAX) {
        if (D.sys_types && D.n_units <= 2 * kFewUnits)
            return launch(kFewBlocks, ff_force<JS, ENERGY, kSystemTable, RELAX, kFewBlocks>);
        if (D.ntypes && D.n_units <= kFewUnits)
            return launch(kFewBlocks, ff_force<JS, ENERGY, kSharedTable, RELAX, kFewBlocks>);
    }
    if (D.sys_types) return launch(kUntypedBlocks, ff_force<JS, ENERGY, kSystemTable, RELAX, kUntypedBlocks>);
    if (!D.ntypes) return launch(kUntypedBlocks, ff_force<JS, ENERGY, kAtomParams, RELAX, kUntypedBlocks>);
    return launch(force_blocks(JS), ff_force<JS, ENERGY, kSharedTable, RELAX, force_blocks(JS)>);
}

// A capped relaxation forms no energies.
template <int JS> cudaError_t launch_force_pass(const FFDev& D, bool energy, long long* f, int stride, cudaStream_t st) {
    if (D.fcap > 0.0f) return launch_force_kernel<JS, false, true>(D, f, stride, st);
    return energy ? launch_force_kernel<JS, true, false>(D, f, stride, st) : launch_force_kernel<JS, false, false>(D, f, stride, st);
}

// One block per chunk of a system's units.
__global__ void ff_energy(FFDev D, double* part) {
    __shared__ double s[256];
    chain_release();
    const int2 c = D.e_chunks.chunk[blockIdx.x];
    chain_wait();
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

namespace {

// The launches of an evaluation; after an error the others are left out of the result, not undone.
struct Chain {
    int n = 0;
    cudaError_t e = cudaSuccess;
    void put(cudaError_t r) {
        if (e == cudaSuccess) e = r;
        n++;
    }
};

// Everything before the force pass.
void put_prep(Chain& chain, const FFDev& D, int prec, const DevBuf& B, cudaStream_t st) {
    const int t = 256, gg = (D.n_units + t - 1) / t;
    if (D.prep_units) {
        const int threads = D.prep_units >= 1024 ? 1024 : (D.prep_units + 31) / 32 * 32;
        chain.put(launch_chained(ff_prep, D.S, threads, sizeof(int) * (D.prep_units + D.prep_cells), st, D, B, prec));
    } else {
        chain.put(launch_chained(ff_check, gg, t, 0, st, D, B, prec));
        chain.put(launch_chained(ff_bin, gg, t, 0, st, D));
        chain.put(launch_chained(ff_scan, D.S, 1024, 0, st, D));
        chain.put(launch_chained(ff_scatter, gg, t, 0, st, D));
        chain.put(launch_chained(ff_place, gg, t, 0, st, D, B, prec));
    }
}

}  // namespace

int launch_list_lengths(const FFDev& D, int prec, const DevBuf& B, int* most, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    Chain chain;
    chain.put(cudaMemsetAsync(most, 0, sizeof(int) * (size_t)D.S, st));
    if (D.n_units) {
        FFDev all = D;
        all.force_all = 1;
        put_prep(chain, all, prec, B, st);
        chain.put(launch_chained(ff_list_lengths, (D.n_units + 3) / 4, 128, 0, st, all, most));
    }
    return chain.e == cudaSuccess ? chain.n : -1;
}

int launch_forces(const FFDev& D, int prec, const DevBuf& B, bool energy, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (D.n_int == 0) return 0;
    Chain chain;
    put_prep(chain, D, prec, B, st);
    long long* f = const_cast<long long*>(B.force);
    switch (D.slots) {
        case 1: chain.put(launch_force_pass<1>(D, energy, f, B.stride, st)); break;
        case 2: chain.put(launch_force_pass<2>(D, energy, f, B.stride, st)); break;
        case 3: chain.put(launch_force_pass<3>(D, energy, f, B.stride, st)); break;
        default: chain.put(launch_force_pass<4>(D, energy, f, B.stride, st));
    }
    if (energy) {
        const SystemChunks& c = D.e_chunks;
        double* part = c.n == D.S ? D.energy : c.part;  // every system one chunk: its sum is the result
        chain.put(launch_chained(ff_energy, c.n, 256, 0, st, D, part));
        if (part != D.energy) {
            if (launch_join_chunks(part, c.chunk0, D.S, 1, D.energy, stream) < 0) return -1;
            chain.n++;
        }
    }
    return chain.e == cudaSuccess ? chain.n : -1;
}

}  // namespace rbx
