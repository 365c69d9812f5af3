// rbx_batch.cpp -- batched systems: one integrator over the atoms of many independent periodic
// systems, forces from the library's cell-list LJ + reaction-field kernels, and runs of steps
// replayed from a captured CUDA graph. The C ABI is declared in include/rbx.h.
//
// Every system keeps a contiguous range of device slots, so the integrator's library order (bodies
// by lowest slot) keeps each system's bodies and free atoms contiguous as well, which the
// per-system kinetic-energy reduction relies on.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <map>
#include <new>
#include <numeric>
#include <thread>
#include <vector>

#include "../../include/rbx.h"
#include "rbx_devarray.h"
#include "rbx_internal.h"

using namespace rbx;

namespace {

constexpr double kOne4PiEps0 = 138.935456;  // kJ nm / (mol e^2)
// Neighbour-list skin (nm, of unit centroids). A longer list costs the force pass one distance test
// per entry, a shorter one more builds. 20 steps at 0.06, 0.08, 0.10, 0.12 and 0.14 nm: 256 boxes of the
// mix at 750 K 15.1, 15.0, 15.0, 14.7 and 14.7 ms, 66,666 waters at 1100 K 4.62, 4.55, 4.52, 4.41 and 4.46.
constexpr double kSkin = 0.12;

#define BATCH_TRY(call)                                                                             \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess) return set_error(RBX_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// body(s) for every system s, the systems split into contiguous ranges of about equal unit counts
// over the host's cores. Each call writes only its own system's outputs, so the results do not
// depend on the split; a thread that cannot be started leaves its range to the calling thread.
template <class F> void for_each_system(const std::vector<FFSys>& sys, F&& body) {
    const int S = (int)sys.size();
    const long long units = S ? (long long)sys[S - 1].u1 - sys[0].u0 : 0;
    const int nt = (int)std::min<long long>({(long long)std::max(1u, std::thread::hardware_concurrency()), 32LL,
                                             std::max(1LL, units / 20000)});
    std::vector<int> lo(nt + 1, S);
    lo[0] = 0;
    for (int t = 1, s = 0; t < nt; t++) {
        while (s < S && (long long)(sys[s].u0 - sys[0].u0) * nt < units * t) s++;
        lo[t] = s;
    }
    auto run = [&](int t) {
        for (int s = lo[t]; s < lo[t + 1]; s++) body(s);
    };
    std::vector<std::thread> pool;
    std::vector<int> inline_ranges;
    for (int t = 1; t < nt; t++) {
        try {
            pool.emplace_back(run, t);
        } catch (...) {
            inline_ranges.push_back(t);
        }
    }
    run(0);
    for (int t : inline_ranges) run(t);
    for (std::thread& th : pool) th.join();
}

template <class T> int upload_vec(DevArray<T>& a, const std::vector<T>& h) {
    if (a.alloc(h.size()) != cudaSuccess) return set_error(RBX_ERR_CUDA, "cudaMalloc of %zu bytes failed", h.size() * sizeof(T));
    if (!h.empty()) BATCH_TRY(cudaMemcpy(a.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return RBX_OK;
}

// Device storage of SystemChunks: systems of the given item counts in chunks of `size` (at least one
// chunk each), `width` partial sums per chunk.
struct ChunkStore {
    DevArray<int2> chunk;
    DevArray<int> chunk0;
    DevArray<double> part;
    int set(const std::vector<int>& items, int size, int width) {
        std::vector<int2> c;
        std::vector<int> c0;
        for (int s = 0; s < (int)items.size(); s++) {
            c0.push_back((int)c.size());
            for (int i = 0; i == 0 || i < items[s]; i += size) c.push_back(make_int2(s, i));
        }
        c0.push_back((int)c.size());
        int rc = upload_vec(chunk, c);
        if (!rc) rc = upload_vec(chunk0, c0);
        if (!rc && part.alloc(c.size() * width) != cudaSuccess) rc = set_error(RBX_ERR_CUDA, "cudaMalloc of partial sums failed");
        return rc;
    }
    SystemChunks view() const { return SystemChunks{(int)chunk.n, chunk.p, chunk0.p, part.p}; }
    size_t bytes() const { return chunk.bytes() + chunk0.bytes() + part.bytes(); }
};

}  // namespace

struct rbx_batch {
    rbx_integrator* integ = nullptr;
    int S = 0, natoms = 0, prec = PREC_MIXED, device = 0;
    std::vector<int> offsets;
    // force field
    DevArray<FFSys> d_sys;
    DevArray<int> d_iatom, d_ugrp, d_usys, d_place, d_unit_at, d_cell_count, d_cell_start, d_cell_cursor;
    DevArray<int> d_sgrp, d_ncnt, d_atype;
    DevArray<int2> d_unit, d_sunit, d_sys_types;
    DevArray<float4> d_param, d_ucen, d_uref, d_scen, d_spos, d_spar, d_types;
    DevArray<unsigned char> d_moved, d_build;
    DevArray<unsigned int> d_skey;      // FFDev::skey
    DevArray<unsigned int> d_nbr;       // neighbour lists of units (FFDev::nbr)
    DevArray<unsigned int> d_rebuilds;  // list builds per system (FFDev::rebuilds)
    DevArray<int> d_most;               // longest list per system, and builds that are not the user's
    // host copies for the set-up with a state: systems, cells allocated per system, unit layout
    std::vector<FFSys> sys_h;
    std::vector<int> cells_alloc, iatom_h;
    std::vector<int2> unit_h;
    std::vector<double> box_h, list_expect;  // list_expect: list lengths at the mean density
    DevArray<double> d_e_unit, d_energy;
    FFDev ff{};
    // per-system reductions
    DevArray<int> d_body0, d_free0;
    ChunkStore ke_chunks, e_chunks;  // of bodies and free atoms, of units
    std::vector<int> body0_h, free0_h;  // host copies: library-order body / free-atom ranges per system
    DevArray<unsigned int> d_sys_status;  // [S] force-kernel failures (FFDev::sys_status)
    DevArray<double> d_ke, d_user;
    std::vector<int> dof;
    double* h_out = nullptr;  // pinned [3*S]
    int last_launches = 0;
    bool u_valid = false;  // d_energy holds the potential energy of the current positions
    // the force buffer holds the forces of the current positions, formed (with their energy) from
    // lists built at those positions: a step call then starts without a force evaluation
    bool f_valid = false;
    // captured runs of (forces, fused step)
    // optional event timing of the force and integrator launch groups (direct launches only)
    bool timing = false;
    std::vector<cudaEvent_t> ev_pool;
    std::vector<std::pair<int, int>> ev_marks;  // (start event, end event) per group
    std::vector<int> ev_kind;                   // 0 = forces, 1 = integrator
    int ev_used = 0;
    int list_threads = 128;  // rbx_batch_set_tuning's block size: lists are built by the force pass now
    int graph_k = 0;
    int graph_launches = 0;  // kernels in one replay of the graph
    double graph_dt = 0.0;
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t graph = nullptr;

    void drop_graph() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
    }
    cudaEvent_t event() {
        if (ev_used == (int)ev_pool.size()) {
            cudaEvent_t e = nullptr;
            if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
            ev_pool.push_back(e);
        }
        return ev_pool[ev_used++];
    }
    ~rbx_batch() {
        for (cudaEvent_t e : ev_pool) cudaEventDestroy(e);
        drop_graph();
        if (cap_stream) cudaStreamDestroy(cap_stream);
        if (h_out) cudaFreeHost(h_out);
        if (integ) rbx_destroy(integ);
    }
};

namespace {

int check(const rbx_batch* b) { return b ? RBX_OK : set_error(RBX_ERR_INVALID_ARGUMENT, "null batch handle"); }

// Cells of at least `edge` per box edge L, at most 256 and at most `most` in the box.
int cells_per_edge(double L, double edge, int most) {
    int nc = (int)std::min(256.0, std::floor(L / edge));
    while (nc > 1 && (long long)nc * nc * nc > most) nc--;
    return nc;
}

// Neighbour-list geometry for a state (host positions, user order): each unit's radius about its
// centroid (constant for a rigid body), and from the largest radius of each system its list cells
// (at least cutoff + skin + two radii per edge, or half of that). The lists themselves are sized by
// size_lists, once the state is on the device.
int setup_lists(rbx_batch* b, void* stream, const double* x) {
    const int S = b->S;
    std::vector<FFSys> sys = b->sys_h;
    std::vector<double> rho(S, 0.0);  // largest atom distance from a unit centroid
    for_each_system(sys, [&](int s) {
        const FFSys& f = sys[s];
        const double L = b->box_h[s];
        auto img = [L](double d) { return d - L * std::nearbyint(d / L); };
        double rho_max = 0.0;
        for (int u = f.u0; u < f.u1; u++) {
            const int k0 = b->unit_h[u].x, n = b->unit_h[u].y & 0xff;
            const double* x0 = x + 3 * (size_t)b->iatom_h[k0];
            double c[3] = {0.0, 0.0, 0.0};
            for (int a = 1; a < n; a++)
                for (int d = 0; d < 3; d++) c[d] += img(x[3 * (size_t)b->iatom_h[k0 + a] + d] - x0[d]);
            for (int d = 0; d < 3; d++) c[d] = x0[d] + c[d] / n;
            for (int a = 0; a < n; a++) {
                double r2 = 0.0;
                for (int d = 0; d < 3; d++) {
                    const double v = img(x[3 * (size_t)b->iatom_h[k0 + a] + d] - c[d]);
                    r2 += v * v;
                }
                rho_max = std::max(rho_max, r2);
            }
        }
        rho[s] = std::sqrt(rho_max);
    });
    b->list_expect.assign(S, 0.0);
    long long most_units = 0, most_cells = 0;
    for (int s = 0; s < S; s++) {
        FFSys& f = sys[s];
        const double L = b->box_h[s], rho_max = rho[s];
        // the device forms the radii in FP32: a margin of 1e-3 nm keeps its ones within the cells
        const double edge = (double)f.rl + 2.0 * rho_max + 1e-3;
        f.pair_image = std::sqrt((double)f.rc2) + 2.0 * rho_max + 1e-3 >= 0.5 * L ? 1 : 0;
        const int U = f.u1 - f.u0;
        // cells of half the reach where the box has five of them and they are not mostly empty, else of
        // the whole reach, else one cell
        const int half = cells_per_edge(L, 0.5 * edge, b->cells_alloc[s]), whole = cells_per_edge(L, edge, b->cells_alloc[s]);
        const bool fine = half >= 5 && (long long)half * half * half <= 2LL * U;
        const int nc = fine ? half : whole >= 3 ? whole : 1;
        f.nc = nc;
        f.win = fine ? 2 : 1;
        f.reach = (float)((double)f.rl + rho_max + 1e-3);
        most_units = std::max<long long>(most_units, U);
        most_cells = std::max<long long>(most_cells, (long long)nc * nc * nc);
        const double reach = (double)f.rl + 2.0 * rho_max;
        b->list_expect[s] = 4.18879 * reach * reach * reach * (double)U / (L * L * L);
    }
    b->sys_h = sys;
    // (on the state's stream: the kernels that read it follow there)
    BATCH_TRY(cudaMemcpyAsync(b->d_sys.p, b->sys_h.data(), sizeof(FFSys) * (size_t)S, cudaMemcpyHostToDevice,
                              (cudaStream_t)stream));
    FFDev& D = b->ff;
    const bool small = prep_limit(most_units, most_cells);
    D.prep_units = small ? (int)most_units : 0;
    D.prep_cells = small ? (int)most_cells : 0;
    return RBX_OK;
}

// Most atoms per unit of a system, from its group sizes: the size with the least pair work, as the
// force pass costs it (per unit pair 28 instructions to find and fetch the listed unit, per atom of
// it 11, per atom pair 17; an atom record is paid for whether it holds an atom or not). Each group is
// cut evenly.
int unit_atoms(const std::vector<int>& group_sizes) {
    double best_cost = 0.0;
    int best = 1;
    for (int m = 1; m <= kMaxUnit; m++) {
        double units = 0.0, atoms = 0.0;
        for (int n : group_sizes) {
            units += (n + m - 1) / m;
            atoms += n;
        }
        const double cost = units * (units * (28.0 + 11.0 * m) + 17.0 * m * atoms);
        if (m == 1 || cost < best_cost) {
            best_cost = cost;
            best = m;
        }
    }
    return best;
}

// The types of atoms [k0, k1): the distinct triples in order of appearance and each atom's index among them;
// false (and no atom of a type) when there are more than kMaxTypes.
bool atom_types(const std::vector<float4>& param, size_t k0, size_t k1, std::vector<float4>& types, std::vector<int>& type_of) {
    std::map<std::array<float, 3>, int> seen;
    types.clear();
    for (size_t k = k0; k < k1; k++) {
        const auto it = seen.emplace(std::array<float, 3>{param[k].x, param[k].y, param[k].z}, (int)types.size()).first;
        if (it->second == (int)types.size()) {
            if (it->second == kMaxTypes) {
                std::fill(type_of.begin() + k0, type_of.begin() + k, 0);
                return false;
            }
            types.push_back(param[k]);
        }
        type_of[k] = it->second;
    }
    return true;
}

// Type-pair table: (K q_i q_j, 12 C12, 6 C6, sqrt(K) q_j) with C12 = 4 eps sig^12, C6 = 4 eps sig^6 and
// Lorentz-Berthelot sig = (sig_i + sig_j)/2, eps = sqrt(eps_i eps_j), formed in FP64 from the
// FP32 type values (the force is (12 C12 r^-6 - 6 C6) r^-8 r).
void append_pair_table(const std::vector<float4>& types, std::vector<float4>& table) {
    for (const float4& i : types)
        for (const float4& j : types) {
            const double sig = (double)i.y + (double)j.y, eps = (double)i.z * (double)j.z;
            const double s6 = sig * sig * sig * sig * sig * sig;
            table.push_back(make_float4((float)((double)i.x * (double)j.x), (float)(48.0 * eps * s6 * s6),
                                        (float)(24.0 * eps * s6), j.x));
        }
}

DevBuf buffers(rbx_batch* b) {
    rbx_buffers rb;
    rbx_context_buffers(b->integ, &rb);
    DevBuf d;
    d.posq = rb.posq;
    d.corr = rb.posq_correction;
    d.velm = rb.velm;
    d.force = rb.force;
    d.stride = rb.stride;
    return d;
}

// List memory for the state on the device. The longest list of each system is counted there, not estimated
// from the mean density: bodies cut into units, clusters and droplets make lists many times longer than that.
// A fifth and 32 entries are left for what the motion adds, and no system gets less than its mean density
// asks for. A list that outgrows its room all the same costs time, not pairs (FFDev::ncnt).
// Every system has a capacity of its own, so that its results do not depend on the others.
int size_lists(rbx_batch* b, void* stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int S = b->S;
    std::vector<int> most(S, 0);
    FFDev D = b->ff;
    D.rebuilds = (unsigned int*)(b->d_most.p + S);  // these are no builds of the user's steps
    if (launch_list_lengths(D, b->prec, buffers(b), b->d_most.p, stream) < 0)
        return set_error(RBX_ERR_CUDA, "list length kernels failed: %s", cudaGetErrorString(cudaGetLastError()));
    BATCH_TRY(cudaMemcpyAsync(most.data(), b->d_most.p, sizeof(int) * (size_t)S, cudaMemcpyDeviceToHost, st));
    BATCH_TRY(cudaStreamSynchronize(st));
    int most_units = 1;
    for (const FFSys& f : b->sys_h) most_units = std::max(most_units, f.u1 - f.u0);
    std::vector<unsigned int> every((most_units + 31) / 32 * 32);
    std::iota(every.begin(), every.end(), 0u);
    long long rows = (long long)every.size() / 32;  // of 32 entries
    for (int s = 0; s < S; s++) {
        FFSys& f = b->sys_h[s];
        const int U = f.u1 - f.u0;
        const double need = std::max(1.35 * b->list_expect[s], 1.2 * most[s]) + 32.0;
        f.cap = ((int)std::ceil(std::min((double)std::max(U - 1, 1), need)) + 31) / 32 * 32;
        f.list0 = (int)rows;
        rows += (long long)U * (f.cap / 32);
        if (rows > INT_MAX) return set_error(RBX_ERR_CUDA, "neighbour lists of more than 2^36 entries");
    }
    const size_t entries = 32 * (size_t)rows;
    if (b->d_nbr.n < entries && b->d_nbr.alloc(entries) != cudaSuccess)
        return set_error(RBX_ERR_CUDA, "cudaMalloc of the neighbour lists failed (%zu entries)", entries);
    b->ff.nbr = b->d_nbr.p;
    BATCH_TRY(cudaMemcpyAsync(b->d_nbr.p, every.data(), sizeof(unsigned int) * every.size(), cudaMemcpyHostToDevice, st));
    BATCH_TRY(cudaMemcpyAsync(b->d_sys.p, b->sys_h.data(), sizeof(FFSys) * (size_t)S, cudaMemcpyHostToDevice, st));
    BATCH_TRY(cudaStreamSynchronize(st));
    return RBX_OK;
}

// Event pair around one launch group when timing is on (never inside a stream capture).
struct Timed {
    rbx_batch* b;
    void* stream;
    int kind, start = -1;
    Timed(rbx_batch* b_, void* s, int k) : b(b_), stream(s), kind(k) {
        if (b->timing) {
            start = b->ev_used;
            cudaEvent_t e = b->event();
            if (e) cudaEventRecord(e, (cudaStream_t)stream); else start = -1;
        }
    }
    ~Timed() {
        if (start < 0) return;
        const int end = b->ev_used;
        cudaEvent_t e = b->event();
        if (!e) return;
        cudaEventRecord(e, (cudaStream_t)stream);
        b->ev_marks.push_back({start, end});
        b->ev_kind.push_back(kind);
    }
};

// One force evaluation. `rebuild` rebuilds every system's lists at the current positions: forces and
// energies at the state a call starts or ends in are formed so, as a function of the positions alone
// (not of when earlier calls last rebuilt); the evaluations in between rebuild a system's lists when
// one of its units has moved half the skin.
int forces(rbx_batch* b, void* stream, bool energy, bool rebuild) {
    Timed t(b, stream, 0);
    FFDev D = b->ff;
    D.force_all = rebuild;
    const int n = launch_forces(D, b->prec, buffers(b), energy, stream);
    if (n < 0) return set_error(RBX_ERR_CUDA, "force kernels failed: %s", cudaGetErrorString(cudaGetLastError()));
    b->last_launches += n;
    return RBX_OK;
}

int integrate(rbx_batch* b, void* stream, int kind, double dt) {
    Timed t(b, stream, 1);
    rbx_buffers rb;
    rbx_context_buffers(b->integ, &rb);
    int rc = kind == STEP_PART1 ? rbx_integrate_part1(b->integ, stream, &rb, dt)
             : kind == STEP_PART2 ? rbx_integrate_part2(b->integ, stream, &rb, dt)
                                  : rbx_integrate_fused(b->integ, stream, &rb, dt);
    if (!rc) b->last_launches += 1;
    return rc;
}

int fused(rbx_batch* b, void* stream, double dt) { return integrate(b, stream, STEP_FUSED, dt); }

int capture(rbx_batch* b, double dt) {
    b->drop_graph();
    const bool timing = b->timing;
    b->timing = false;  // no event records inside the capture
    if (!b->cap_stream) BATCH_TRY(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));
    BATCH_TRY(cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeRelaxed));
    int rc = RBX_OK;
    const int before = b->last_launches;
    for (int i = 0; i < b->graph_k && !rc; i++) {
        rc = forces(b, b->cap_stream, false, false);
        if (!rc) rc = fused(b, b->cap_stream, dt);
    }
    b->graph_launches = b->last_launches - before;
    b->last_launches = before;
    b->timing = timing;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(b->cap_stream, &g);
    if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
    }
    if (e != cudaSuccess) return set_error(RBX_ERR_CUDA, "stream capture failed: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        b->graph = nullptr;
        return set_error(RBX_ERR_CUDA, "graph instantiation failed: %s", cudaGetErrorString(e));
    }
    b->graph_dt = dt;
    return RBX_OK;
}

}  // namespace

extern "C" {

int rbx_batch_create(rbx_batch** out, int num_systems, const int* atom_offsets, const double* box_edges,
                     const double* cutoffs, const int* body_indices, const double* masses, const double* charges,
                     const double* sigmas, const double* epsilons, double eps_solvent, int rotation_mode,
                     int precision, int device) {
    if (!out) return set_error(RBX_ERR_INVALID_ARGUMENT, "null output pointer");
    *out = nullptr;
    if (num_systems <= 0 || !atom_offsets || !box_edges || !cutoffs || !body_indices || !masses || !charges ||
        !sigmas || !epsilons)
        return set_error(RBX_ERR_INVALID_ARGUMENT, "need num_systems > 0 and every per-system and per-atom array");
    if (atom_offsets[0] != 0) return set_error(RBX_ERR_INVALID_ARGUMENT, "atom_offsets[0] must be 0");
    for (int s = 0; s < num_systems; s++) {
        if (atom_offsets[s + 1] <= atom_offsets[s]) return set_error(RBX_ERR_INVALID_ARGUMENT, "system %d has no atoms", s);
        if (!(box_edges[s] > 0.0)) return set_error(RBX_ERR_INVALID_ARGUMENT, "system %d: box edge must be positive", s);
        if (!(cutoffs[s] > 0.0) || !(cutoffs[s] < 0.5 * box_edges[s]))
            return set_error(RBX_ERR_INVALID_ARGUMENT, "system %d: the cutoff must lie in (0, box/2)", s);
    }
    if (!(eps_solvent >= 1.0)) return set_error(RBX_ERR_INVALID_ARGUMENT, "reaction-field dielectric must be >= 1");
    const int N = atom_offsets[num_systems];
    rbx_batch* b = new (std::nothrow) rbx_batch();
    if (!b) return set_error(RBX_ERR_INVALID_ARGUMENT, "out of host memory");
    b->S = num_systems;
    b->natoms = N;
    b->prec = precision;
    b->device = device;
    b->offsets.assign(atom_offsets, atom_offsets + num_systems + 1);

    // one integrator over all systems: per-system body ids made unique
    std::vector<int> ids(N, 0);
    long base = 0;
    for (int s = 0; s < num_systems; s++) {
        int mx = 0;
        for (int i = atom_offsets[s]; i < atom_offsets[s + 1]; i++) {
            if (body_indices[i] > 0) {
                ids[i] = (int)(base + body_indices[i]);
                mx = std::max(mx, body_indices[i]);
            }
        }
        base += mx;
        if (base > 2000000000L) { delete b; return set_error(RBX_ERR_INVALID_ARGUMENT, "too many bodies"); }
    }
    int rc = rbx_create(&b->integ, N, ids.data(), masses, rotation_mode, precision, device);
    if (rc) { delete b; return rc; }

    // force field tables: interacting atoms (charge or LJ) system by system and, within a system,
    // body by body (ascending id; each free atom a group of its own), each group cut into units with
    // their Lennard-Jones atoms first
    std::vector<FFSys> sys(num_systems);
    std::vector<int> iatom, usys, ugrp;
    std::vector<int2> unit;
    std::vector<float4> param;
    int cells = 0, groups = 0, slots = 1;
    for (int s = 0; s < num_systems; s++) {
        FFSys& f = sys[s];
        const size_t i0 = iatom.size();
        f.u0 = (int)unit.size();
        std::map<int, std::vector<int>> bodies;
        std::vector<int> free_atoms;
        for (int i = atom_offsets[s]; i < atom_offsets[s + 1]; i++) {
            if (charges[i] == 0.0 && epsilons[i] == 0.0) continue;
            if (body_indices[i] > 0) bodies[body_indices[i]].push_back(i);
            else free_atoms.push_back(i);
        }
        std::vector<int> sizes(free_atoms.size(), 1);
        for (auto& kv : bodies) sizes.push_back((int)kv.second.size());
        const int most = unit_atoms(sizes);
        auto add_group = [&](const int* atoms, int n) {
            const int m = (n + most - 1) / most;
            for (int k = 0; k < m; k++) {
                const int lo = (int)((long long)n * k / m), hi = (int)((long long)n * (k + 1) / m);
                int lj = 0;
                const int k0 = (int)iatom.size();
                for (int pass = 0; pass < 2; pass++)
                    for (int a = lo; a < hi; a++) {
                        const int i = atoms[a];
                        const float root = (float)std::sqrt(std::max(epsilons[i], 0.0));
                        if ((root != 0.0f) != (pass == 0)) continue;
                        lj += pass == 0;
                        iatom.push_back(i);
                        param.push_back(make_float4((float)(std::sqrt(kOne4PiEps0) * charges[i]), (float)(0.5 * sigmas[i]),
                                                    root, 0.0f));
                    }
                unit.push_back(make_int2(k0, (hi - lo) | lj << 8));
                usys.push_back(s);
                ugrp.push_back(groups);
                slots = std::max(slots, hi - lo);
            }
            groups++;
        };
        for (auto& kv : bodies) add_group(kv.second.data(), (int)kv.second.size());
        for (int i : free_atoms) add_group(&i, 1);
        f.u1 = (int)unit.size();
        if (iatom.size() - i0 >= (size_t)kMaxSystemAtoms) {
            delete b;
            return set_error(RBX_ERR_UNSUPPORTED, "system %d: %zu interacting atoms (at most %d)", s, iatom.size() - i0,
                             kMaxSystemAtoms - 1);
        }
        const double L = box_edges[s], rc_s = cutoffs[s];
        // Pairs are tested by minimum image when the lists are built (and, where cutoff + two radii
        // may reach half the box, when forces are formed), so cutoff + skin + radii may exceed half
        // the box: an image within the cutoff (below half the box) is always the minimum image, and
        // its unit pair is always listed.
        f.rl = (float)(rc_s + kSkin);
        f.cap = 32;  // until the lists are sized (rbx_batch_set_state)
        f.list0 = 0;
        f.pair_image = 1;  // until the radii are known (rbx_batch_set_state)
        // cells for the largest grid any set of radii allows (the radii, known with the positions,
        // can only make the cells larger and fewer): of the whole reach, or of half of it while there
        // are at most two per unit
        const long long units_s = f.u1 - f.u0;
        const int whole = cells_per_edge(L, rc_s + kSkin, 1 << 24), half = cells_per_edge(L, 0.5 * (rc_s + kSkin), 1 << 24);
        const long long room = std::max<long long>((long long)whole * whole * whole,
                                                   std::min((long long)half * half * half, 2 * units_s));
        b->cells_alloc.push_back((int)std::max(1LL, room));
        f.c0 = cells;
        f.nc = 1;
        cells += b->cells_alloc[s];
        f.L = (float)L;
        f.invL = (float)(1.0 / L);
        f.rc = (float)rc_s;
        f.rc2 = (float)(rc_s * rc_s);
        const double krf = (eps_solvent - 1.0) / ((2.0 * eps_solvent + 1.0) * rc_s * rc_s * rc_s);
        f.krf = (float)krf;
        f.crf = (float)(1.0 / rc_s + krf * rc_s * rc_s);
    }
    b->sys_h = sys;
    b->iatom_h = iatom;
    b->unit_h = unit;
    b->box_h.assign(box_edges, box_edges + num_systems);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) { delete b; return set_error(RBX_ERR_CUDA, "cudaSetDevice(%d): %s", device, cudaGetErrorString(e)); }
    const int nint = (int)iatom.size(), nunit = (int)unit.size();
    rc = upload_vec(b->d_sys, sys);
    if (!rc) rc = upload_vec(b->d_iatom, iatom);
    if (!rc) rc = upload_vec(b->d_param, param);
    if (!rc) rc = upload_vec(b->d_unit, unit);
    if (!rc) rc = upload_vec(b->d_usys, usys);
    if (!rc) rc = upload_vec(b->d_ugrp, ugrp);
    std::vector<int> units_of(num_systems);
    for (int s = 0; s < num_systems; s++) units_of[s] = sys[s].u1 - sys[s].u0;
    if (!rc) rc = b->e_chunks.set(units_of, kEnergyChunk, 1);
    // atom types: the distinct (scaled charge, sigma/2, sqrt(epsilon)) triples. A system of at most kMaxTypes
    // types takes each pair's coefficients from a table of type pairs, whatever the systems beside it: one table
    // for the batch where its types fit one together, else a table per such system
    std::vector<float4> pair_table;
    std::vector<int> type_of(param.size(), 0);
    std::vector<int2> sys_types;
    int nt = 0;
    if (!param.empty()) {
        std::vector<float4> types;
        if (atom_types(param, 0, param.size(), types, type_of)) {
            nt = (int)types.size();
            append_pair_table(types, pair_table);
        } else {
            bool any = false;
            auto first_atom = [&](int u) { return u < nunit ? (size_t)unit[u].x : param.size(); };
            for (int s = 0; s < num_systems; s++) {
                const bool typed = atom_types(param, first_atom(sys[s].u0), first_atom(sys[s].u1), types, type_of);
                sys_types.push_back(typed ? make_int2((int)pair_table.size(), (int)types.size()) : make_int2(0, 0));
                if (typed) append_pair_table(types, pair_table);
                any = any || typed;
            }
            if (!any) sys_types.clear();
        }
    }
    if (pair_table.empty()) type_of.clear();
    if (!rc) rc = upload_vec(b->d_types, pair_table);
    if (!rc) rc = upload_vec(b->d_atype, type_of);
    if (!rc) rc = upload_vec(b->d_sys_types, sys_types);
    const size_t u1 = std::max(nunit, 1), records = u1 * slots;
    if (!rc && (b->d_place.alloc(u1) != cudaSuccess || b->d_unit_at.alloc(u1) != cudaSuccess ||
                b->d_ucen.alloc(u1) != cudaSuccess ||
                b->d_uref.alloc(u1) != cudaSuccess || b->d_scen.alloc(u1) != cudaSuccess ||
                b->d_sgrp.alloc(u1) != cudaSuccess || b->d_sunit.alloc(u1) != cudaSuccess || b->d_ncnt.alloc(u1) != cudaSuccess ||
                b->d_spos.alloc(records) != cudaSuccess || b->d_spar.alloc(nt ? 0 : records) != cudaSuccess ||
                b->d_cell_count.alloc(cells) != cudaSuccess || b->d_cell_start.alloc(cells + 1) != cudaSuccess ||
                b->d_cell_cursor.alloc(cells) != cudaSuccess || b->d_e_unit.alloc(u1) != cudaSuccess ||
                b->d_skey.alloc(u1) != cudaSuccess ||
                b->d_energy.alloc(num_systems) != cudaSuccess || b->d_ke.alloc(2 * (size_t)num_systems) != cudaSuccess ||
                b->d_user.alloc(3 * (size_t)N) != cudaSuccess || b->d_sys_status.alloc(num_systems) != cudaSuccess ||
                b->d_moved.alloc(num_systems) != cudaSuccess || b->d_build.alloc(num_systems) != cudaSuccess ||
                b->d_rebuilds.alloc(num_systems) != cudaSuccess || b->d_most.alloc(2 * (size_t)num_systems) != cudaSuccess))
        rc = set_error(RBX_ERR_CUDA, "cudaMalloc of force-field arrays failed");
    if (!rc && (cudaMemset(b->d_sys_status.p, 0, sizeof(unsigned int) * (size_t)num_systems) != cudaSuccess ||
                // (a batch without interacting atoms has no force evaluation to write its energies)
                cudaMemset(b->d_energy.p, 0, sizeof(double) * (size_t)num_systems) != cudaSuccess ||
                cudaMemset(b->d_cell_count.p, 0, sizeof(int) * (size_t)cells) != cudaSuccess ||
                cudaMemset(b->d_moved.p, 0, (size_t)num_systems) != cudaSuccess ||
                cudaMemset(b->d_build.p, 0, (size_t)num_systems) != cudaSuccess ||
                cudaMemset(b->d_rebuilds.p, 0, sizeof(unsigned int) * (size_t)num_systems) != cudaSuccess ||
                cudaMemset(b->d_most.p, 0, sizeof(int) * 2 * (size_t)num_systems) != cudaSuccess ||
                cudaMemset(b->d_ncnt.p, 0, sizeof(int) * u1) != cudaSuccess ||
                cudaMemset(b->d_place.p, 0, sizeof(int) * u1) != cudaSuccess ||
                cudaMemset(b->d_unit_at.p, 0, sizeof(int) * u1) != cudaSuccess))
        rc = set_error(RBX_ERR_CUDA, "initialisation of the force-field arrays failed");
    if (!rc && cudaMallocHost((void**)&b->h_out, sizeof(double) * 3 * (size_t)num_systems) != cudaSuccess)
        rc = set_error(RBX_ERR_CUDA, "pinned allocation failed");
    if (rc) { delete b; return rc; }
    FFDev& D = b->ff;
    D.S = num_systems;
    D.n_int = nint;
    D.n_units = nunit;
    D.n_cells = cells;
    D.sys = b->d_sys.p;
    D.iatom = b->d_iatom.p;
    D.param = b->d_param.p;
    D.unit = b->d_unit.p;
    D.ugrp = b->d_ugrp.p;
    D.usys = b->d_usys.p;
    D.ucen = b->d_ucen.p;
    D.uref = b->d_uref.p;
    D.place = b->d_place.p;
    D.unit_at = b->d_unit_at.p;
    D.cell_count = b->d_cell_count.p;
    D.cell_start = b->d_cell_start.p;
    D.cell_cursor = b->d_cell_cursor.p;
    D.scen = b->d_scen.p;
    D.sgrp = b->d_sgrp.p;
    D.sunit = b->d_sunit.p;
    for (int a = 0; a < kMaxUnit; a++) {
        D.spos[a] = a < slots ? b->d_spos.p + a * u1 : nullptr;
        D.spar[a] = a < slots && !nt ? b->d_spar.p + a * u1 : nullptr;
    }
    D.slots = slots;
    D.e_unit = b->d_e_unit.p;
    D.e_chunks = b->e_chunks.view();
    D.energy = b->d_energy.p;
    D.fcap = 0.0f;
    D.sys_status = b->d_sys_status.p;
    D.force_all = 0;
    D.moved = b->d_moved.p;
    D.build = b->d_build.p;
    D.rebuilds = b->d_rebuilds.p;
    D.nbr = nullptr;  // allocated with the state (size_lists)
    D.ncnt = b->d_ncnt.p;
    D.half_skin2 = (float)(0.25 * kSkin * kSkin);
    D.types = b->d_types.p;
    D.atype = b->d_atype.p;
    D.ntypes = nt;
    D.sys_types = b->d_sys_types.p;
    D.prep_units = 0;
    D.prep_cells = 0;
    D.skey = b->d_skey.p;
    // the owned OpenMM-layout buffers (forces of non-interacting atoms stay zero)
    rbx_buffers rb;
    if ((rc = rbx_context_buffers(b->integ, &rb))) { delete b; return rc; }
    *out = b;
    return RBX_OK;
}

int rbx_batch_destroy(rbx_batch* b) {
    delete b;
    return RBX_OK;
}

int rbx_batch_set_state(rbx_batch* b, void* stream, const double* positions, const double* velocities) {
    int rc = check(b);
    if (rc) return rc;
    b->u_valid = b->f_valid = false;
    b->drop_graph();
    if (!positions || !velocities) return set_error(RBX_ERR_INVALID_ARGUMENT, "null positions or velocities");
    BATCH_TRY(cudaSetDevice(b->device));
    BATCH_TRY(cudaStreamSynchronize((cudaStream_t)stream));  // no force pass in flight on the old lists
    b->d_body0.release();  // no state, until all of the new one is in place
    if ((rc = setup_lists(b, stream, positions))) return rc;
    // positions and velocities into the device buffers, bodies built there (no host round trip)
    if ((rc = rbx_context_load(b->integ, stream, positions, velocities))) return rc;
    rbx_buffers rb;
    if ((rc = rbx_context_buffers(b->integ, &rb))) return rc;
    if ((rc = rbx_upload_state_device(b->integ, stream, &rb))) return rc;
    // body atoms start where the body state puts them (the step kernels' arithmetic), so that a
    // system's trajectory is a function of its body state alone, in or out of a batch
    if ((rc = rbx_context_sync_bodies(b->integ, stream))) return rc;
    if ((rc = size_lists(b, stream))) return rc;
    if ((rc = sync_host_dof(b->integ))) return rc;
    std::vector<int> body0, free0;
    if ((rc = system_ranges(b->integ, b->offsets, body0, free0, b->dof))) return rc;
    if ((rc = upload_vec(b->d_body0, body0)) || (rc = upload_vec(b->d_free0, free0))) return rc;
    if (!b->ke_chunks.chunk.n) {  // the counts are fixed at creation
        std::vector<int> items(b->S);
        for (int s = 0; s < b->S; s++) items[s] = body0[s + 1] - body0[s] + free0[s + 1] - free0[s];
        if ((rc = b->ke_chunks.set(items, kKEChunk, 2))) return rc;
    }
    b->body0_h = body0;
    b->free0_h = free0;
    BATCH_TRY(cudaMemsetAsync(b->d_sys_status.p, 0, sizeof(unsigned int) * (size_t)b->S, (cudaStream_t)stream));
    return RBX_OK;
}

int rbx_batch_get_state(rbx_batch* b, void* stream, double* positions, double* velocities) {
    int rc = check(b);
    if (rc) return rc;
    return rbx_context_get_state(b->integ, stream, positions, velocities);
}

int rbx_batch_get_system_state(rbx_batch* b, void* stream, int s, double* positions, double* velocities) {
    int rc = check(b);
    if (rc) return rc;
    if (s < 0 || s >= b->S) return set_error(RBX_ERR_INVALID_ARGUMENT, "system %d outside [0, %d)", s, b->S);
    return rbx_context_get_range(b->integ, stream, b->offsets[s], b->offsets[s + 1] - b->offsets[s], positions,
                                 velocities);
}

int rbx_batch_get_body_state(rbx_batch* b, void* body_rows) {
    int rc = check(b);
    if (rc) return rc;
    return rbx_get_body_state_raw(b->integ, body_rows);
}

int rbx_batch_restore(rbx_batch* b, void* stream, const void* body_rows, const double* positions,
                      const double* velocities) {
    int rc = check(b);
    if (rc) return rc;
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no geometry: call rbx_batch_set_state with the systems first");
    b->u_valid = b->f_valid = false;
    if ((rc = rbx_context_load(b->integ, stream, positions, velocities))) return rc;
    if ((rc = rbx_set_body_state_raw(b->integ, body_rows))) return rc;
    if ((rc = rbx_context_sync_bodies(b->integ, stream))) return rc;
    BATCH_TRY(cudaMemsetAsync(b->d_sys_status.p, 0, sizeof(unsigned int) * (size_t)b->S, (cudaStream_t)stream));
    return RBX_OK;
}

int rbx_batch_step(rbx_batch* b, void* stream, int nsteps, double dt) {
    int rc = check(b);
    if (rc) return rc;
    if (nsteps < 1) return set_error(RBX_ERR_INVALID_ARGUMENT, "nsteps must be >= 1");
    if (!(dt == dt) || dt == 0.0) return set_error(RBX_ERR_INVALID_ARGUMENT, "step size must be finite and non-zero");
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    BATCH_TRY(cudaSetDevice(b->device));
    b->last_launches = 0;
    // forces at the starting positions: those the previous step call ended with while nothing has
    // changed the state since (formed, as an evaluation here would form them, from lists built at
    // these positions with the energy variant), else one evaluation. The reference likewise keeps
    // the forces of the last step for the next one (CudaRigidBodyKernels.cpp:421-426).
    if (!b->f_valid && (rc = forces(b, stream, true, true))) return rc;
    b->f_valid = false;
    b->u_valid = false;
    if ((rc = integrate(b, stream, STEP_PART1, dt))) return rc;
    int remaining = nsteps - 1;
    if (b->graph_k > 0 && !b->timing && remaining >= b->graph_k) {
        if (!b->graph || b->graph_dt != dt) {
            if ((rc = capture(b, dt))) return rc;
        }
        while (remaining >= b->graph_k) {
            BATCH_TRY(cudaGraphLaunch(b->graph, (cudaStream_t)stream));
            b->last_launches += b->graph_launches;
            remaining -= b->graph_k;
        }
    }
    for (; remaining > 0; remaining--) {
        if ((rc = forces(b, stream, false, false)) || (rc = fused(b, stream, dt))) return rc;
    }
    // the last evaluation builds every list at the final positions and also forms their potential
    // energy
    if ((rc = forces(b, stream, true, true))) return rc;
    if ((rc = integrate(b, stream, STEP_PART2, dt))) return rc;
    b->u_valid = true;
    b->f_valid = true;
    return RBX_OK;
}

int rbx_batch_relax(rbx_batch* b, void* stream, int nsteps, double dt, double max_force, double damping) {
    int rc = check(b);
    if (rc) return rc;
    if (nsteps < 1 || !(dt > 0.0) || !(max_force > 0.0) || !(damping >= 0.0 && damping < 1.0))
        return set_error(RBX_ERR_INVALID_ARGUMENT,
                         "relaxation needs nsteps >= 1, dt > 0, max_force > 0 and 0 <= damping < 1");
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    BATCH_TRY(cudaSetDevice(b->device));
    b->last_launches = 0;
    rbx_buffers rb;
    rbx_context_buffers(b->integ, &rb);
    const DevSys sys = device_system(b->integ);
    b->ff.fcap = (float)max_force;
    b->u_valid = false;
    b->f_valid = false;
    for (int n = 0; n < nsteps && !rc; n++) {
        rc = forces(b, stream, false, n == 0);
        if (!rc && launch_scale_momenta(b->prec, sys, buffers(b), damping, stream) < 0)
            rc = set_error(RBX_ERR_CUDA, "momentum damping failed");
        if (!rc) rc = rbx_integrate_part1(b->integ, stream, &rb, dt);
        b->last_launches += 2;
    }
    b->ff.fcap = 0.0f;
    if (rc) return rc;
    if (launch_scale_momenta(b->prec, sys, buffers(b), 0.0, stream) < 0) return set_error(RBX_ERR_CUDA, "momentum reset failed");
    return RBX_OK;
}

int rbx_batch_energies(rbx_batch* b, void* stream, double* out) {
    int rc = check(b);
    if (rc) return rc;
    if (!out) return set_error(RBX_ERR_INVALID_ARGUMENT, "null output");
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    BATCH_TRY(cudaSetDevice(b->device));
    b->last_launches = 0;
    // the potential energy of the last step call's final positions when it is still current (formed
    // in that call's last force evaluation); otherwise a force evaluation that forms it
    if (!b->u_valid && (rc = forces(b, stream, true, true))) return rc;
    b->u_valid = true;
    b->f_valid = true;
    const int launched = launch_kinetic_systems(b->prec, device_system(b->integ), buffers(b), b->d_body0.p, b->d_free0.p,
                                                b->ke_chunks.view(), b->S, b->d_ke.p, stream);
    if (launched < 0)
        return set_error(RBX_ERR_CUDA, "kinetic-energy kernel failed: %s", cudaGetErrorString(cudaGetLastError()));
    b->last_launches += launched;
    cudaStream_t st = (cudaStream_t)stream;
    BATCH_TRY(cudaMemcpyAsync(b->h_out, b->d_energy.p, sizeof(double) * b->S, cudaMemcpyDeviceToHost, st));
    BATCH_TRY(cudaMemcpyAsync(b->h_out + b->S, b->d_ke.p, sizeof(double) * 2 * b->S, cudaMemcpyDeviceToHost, st));
    BATCH_TRY(cudaStreamSynchronize(st));
    for (int s = 0; s < b->S; s++) {
        out[3 * s] = b->h_out[s];
        out[3 * s + 1] = b->h_out[b->S + 2 * s];
        out[3 * s + 2] = b->h_out[b->S + 2 * s + 1];
    }
    return RBX_OK;
}

int rbx_batch_forces(rbx_batch* b, void* stream, double* forces_out, double* energies) {
    int rc = check(b);
    if (rc) return rc;
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    BATCH_TRY(cudaSetDevice(b->device));
    b->last_launches = 0;
    if ((rc = forces(b, stream, true, true))) return rc;
    b->u_valid = true;
    b->f_valid = true;
    cudaStream_t st = (cudaStream_t)stream;
    const DevBuf d = buffers(b);
    if (forces_out) {
        if (launch_forces_to_user(d.force, d.stride, b->natoms, b->d_user.p, stream) < 0)
            return set_error(RBX_ERR_CUDA, "force conversion failed");
        BATCH_TRY(cudaMemcpyAsync(forces_out, b->d_user.p, sizeof(double) * 3 * (size_t)b->natoms, cudaMemcpyDeviceToHost, st));
    }
    if (energies) BATCH_TRY(cudaMemcpyAsync(energies, b->d_energy.p, sizeof(double) * b->S, cudaMemcpyDeviceToHost, st));
    BATCH_TRY(cudaStreamSynchronize(st));
    return RBX_OK;
}

int rbx_batch_get_num_dof(rbx_batch* b, int* dof) {
    int rc = check(b);
    if (rc) return rc;
    if (b->dof.empty()) return set_error(RBX_ERR_STATE, "degrees of freedom are known after rbx_batch_set_state");
    std::copy(b->dof.begin(), b->dof.end(), dof);
    return RBX_OK;
}

int rbx_batch_list_builds(rbx_batch* b, void* stream, unsigned int* counts) {
    int rc = check(b);
    if (rc) return rc;
    if (!counts) return set_error(RBX_ERR_INVALID_ARGUMENT, "null output");
    BATCH_TRY(cudaSetDevice(b->device));
    BATCH_TRY(cudaMemcpyAsync(counts, b->d_rebuilds.p, sizeof(unsigned int) * (size_t)b->S, cudaMemcpyDeviceToHost,
                              (cudaStream_t)stream));
    BATCH_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    return RBX_OK;
}

int rbx_batch_memory(const rbx_batch* b, size_t* bytes) {
    int rc = check(b);
    if (rc) return rc;
    if (!bytes) return set_error(RBX_ERR_INVALID_ARGUMENT, "null output");
    size_t n = b->d_sys.bytes() + b->d_iatom.bytes() + b->d_param.bytes() + b->d_unit.bytes() + b->d_ugrp.bytes() +
               b->d_usys.bytes() + b->d_ucen.bytes() + b->d_uref.bytes() + b->d_place.bytes() +
               b->d_unit_at.bytes() + b->d_cell_count.bytes() + b->d_cell_start.bytes() + b->d_cell_cursor.bytes() +
               b->d_scen.bytes() + b->d_sgrp.bytes() + b->d_sunit.bytes() + b->d_spos.bytes() + b->d_spar.bytes() +
               b->d_skey.bytes() + b->d_types.bytes() + b->d_sys_types.bytes() + b->d_atype.bytes() + b->d_moved.bytes() +
               b->d_build.bytes() + b->d_nbr.bytes() + b->d_ncnt.bytes() + b->d_rebuilds.bytes() + b->d_most.bytes() +
               b->d_e_unit.bytes() + b->d_energy.bytes() + b->d_body0.bytes() + b->d_free0.bytes() +
               b->d_sys_status.bytes() + b->d_ke.bytes() + b->d_user.bytes() + b->ke_chunks.bytes() +
               b->e_chunks.bytes();
    *bytes = n + (b->integ ? device_bytes(b->integ) : 0);
    return RBX_OK;
}

int rbx_batch_status(rbx_batch* b, void* stream, int* system_status, int* num_failed) {
    int rc = check(b);
    if (rc) return rc;
    if (b->body0_h.empty()) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    BATCH_TRY(cudaSetDevice(b->device));
    std::vector<unsigned int> fs(b->S);
    BATCH_TRY(cudaMemcpyAsync(fs.data(), b->d_sys_status.p, sizeof(unsigned int) * (size_t)b->S, cudaMemcpyDeviceToHost,
                              (cudaStream_t)stream));
    std::vector<uint8_t> bb, fb;
    unsigned int count = 0;
    if ((rc = failure_flags(b->integ, stream, bb, fb, &count))) return rc;  // synchronises the stream
    std::vector<int> failed(b->S, 0);
    for (int s = 0; s < b->S; s++) {
        bool bad = fs[s] != 0;
        if (count) {
            for (int L = b->body0_h[s]; L < b->body0_h[s + 1] && !bad; L++) bad = bb[L] != 0;
            for (int j = b->free0_h[s]; j < b->free0_h[s + 1] && !bad; j++) bad = fb[j] != 0;
        }
        failed[s] = bad ? RBX_ERR_NUMERIC : RBX_OK;
    }
    int n = 0, first = -1;
    for (int s = 0; s < b->S; s++)
        if (failed[s]) {
            if (first < 0) first = s;
            n++;
        }
    if (system_status) std::copy(failed.begin(), failed.end(), system_status);
    if (num_failed) *num_failed = n;
    if (!n) return RBX_OK;
    return set_error(RBX_ERR_NUMERIC, "%d of %d systems failed (first: system %d): a non-finite state after a step, "
                     "or a force beyond the fixed-point range", n, b->S, first);
}

int rbx_batch_autotune(rbx_batch* b, void* stream, double dt, int trial_steps, int* chosen) {
    int rc = check(b);
    if (rc) return rc;
    if (!b->d_body0.p) return set_error(RBX_ERR_STATE, "no state: call rbx_batch_set_state first");
    if (trial_steps < 1) return set_error(RBX_ERR_INVALID_ARGUMENT, "trial_steps must be >= 1");
    if (!(dt == dt) || dt == 0.0) return set_error(RBX_ERR_INVALID_ARGUMENT, "step size must be finite and non-zero");
    BATCH_TRY(cudaSetDevice(b->device));
    cudaStream_t st = (cudaStream_t)stream;
    // the exact state, restored after the trials (they only change how the work is scheduled)
    int nb = 0;
    if ((rc = rbx_get_num_bodies(b->integ, &nb))) return rc;
    std::vector<double> body((size_t)nb * 14 + 1), x((size_t)3 * b->natoms), v((size_t)3 * b->natoms);
    if ((rc = rbx_batch_get_body_state(b, body.data())) || (rc = rbx_batch_get_state(b, stream, x.data(), v.data())))
        return rc;
    const bool timing = b->timing;
    b->timing = false;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    BATCH_TRY(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return set_error(RBX_ERR_CUDA, "cudaEventCreate failed");
    }
    // milliseconds per step of `n` steps after one untimed call of the same length
    auto per_step = [&](int n, float& ms) -> int {
        int r = rbx_batch_step(b, stream, n, dt);
        if (!r && cudaEventRecord(e0, st) != cudaSuccess) r = set_error(RBX_ERR_CUDA, "event record failed");
        if (!r) r = rbx_batch_step(b, stream, n, dt);
        if (!r && (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                   cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
            r = set_error(RBX_ERR_CUDA, "event timing failed");
        ms /= (float)n;
        return r;
    };
    const int k0 = b->graph_k;
    int best_k = k0;
    float best = 0.0f, ms = 0.0f;
    b->graph_k = 0;
    b->drop_graph();
    // 1. tile shape of the step kernel (single/mixed; 128 threads only for bodies of at most 32
    // atoms): the integrator launches alone, event-timed over 2 x trial_steps steps after one
    // untimed run, since they are a small share of a step
    int best_nt = 0;
    if (!rc && (rc = rbx_get_tile_threads(b->integ, &best_nt)) == RBX_OK) {
        const int nts[2] = {kThreadsF, kThreadsFNarrow};
        double best_i = 0.0;
        bool any = false;
        for (int nt : nts) {
            if (rbx_set_tile_threads(b->integ, nt) != RBX_OK) continue;  // shape not supported here
            b->timing = true;
            if ((rc = rbx_batch_step(b, stream, trial_steps, dt)) || (rc = rbx_batch_set_timing(b, 1)) ||
                (rc = rbx_batch_step(b, stream, 2 * trial_steps, dt)))
                break;
            double mf = 0.0, mi = 0.0;
            if ((rc = rbx_batch_kernel_times(b, &mf, &mi, nullptr))) break;
            if (!any || mi < best_i) {
                best_i = mi;
                best_nt = nt;
                any = true;
            }
        }
        b->timing = false;
        const int rc1 = rbx_set_tile_threads(b->integ, best_nt);
        if (!rc) rc = rc1;
    }
    // 2. one step, direct launches
    if (!rc) rc = per_step(trial_steps, best);
    // 3. steps per captured graph, where launch overhead matters (steps under 1 ms)
    if (!rc && best < 1.0f) {
        const int ks[3] = {0, 10, 50};
        float best_g = 0.0f;
        for (int i = 0; i < 3 && !rc; i++) {
            b->graph_k = ks[i];
            b->drop_graph();
            if ((rc = per_step(ks[i] ? 2 * ks[i] + 1 : trial_steps, ms))) break;
            if (i == 0 || ms < best_g) {
                best_g = ms;
                best_k = ks[i];
            }
        }
    } else if (!rc) {
        best_k = k0 > 0 ? k0 : 50;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->graph_k = best_k;
    b->drop_graph();
    b->timing = timing;
    b->ev_marks.clear();
    b->ev_kind.clear();
    b->ev_used = 0;
    const int rc2 = rbx_batch_restore(b, stream, body.data(), x.data(), v.data());
    if (rc) return rc;
    if (rc2) return rc2;
    if (chosen) {
        chosen[0] = b->list_threads;
        chosen[1] = best_k;
    }
    return RBX_OK;
}

int rbx_batch_set_tile_threads(rbx_batch* b, int threads) {
    int rc = check(b);
    if (rc) return rc;
    int cur = 0;
    if ((rc = rbx_get_tile_threads(b->integ, &cur))) return rc;
    if (cur == threads) return RBX_OK;
    b->drop_graph();
    return rbx_set_tile_threads(b->integ, threads);
}

int rbx_batch_get_tile_threads(rbx_batch* b, int* out) {
    int rc = check(b);
    if (rc) return rc;
    return rbx_get_tile_threads(b->integ, out);
}

int rbx_batch_set_tuning(rbx_batch* b, int cell_threads, int graph_steps) {
    int rc = check(b);
    if (rc) return rc;
    if (cell_threads != 64 && cell_threads != 128 && cell_threads != 256)
        return set_error(RBX_ERR_INVALID_ARGUMENT, "cell kernel block size must be 64, 128 or 256");
    if ((rc = rbx_batch_set_graph_steps(b, graph_steps))) return rc;
    b->list_threads = cell_threads;
    return RBX_OK;
}

int rbx_batch_set_graph_steps(rbx_batch* b, int k) {
    int rc = check(b);
    if (rc) return rc;
    if (k < 0) return set_error(RBX_ERR_INVALID_ARGUMENT, "graph run length must be >= 0");
    if (k != b->graph_k) b->drop_graph();
    b->graph_k = k;
    return RBX_OK;
}

int rbx_batch_set_timing(rbx_batch* b, int on) {
    int rc = check(b);
    if (rc) return rc;
    b->timing = on != 0;
    b->ev_marks.clear();
    b->ev_kind.clear();
    b->ev_used = 0;
    return RBX_OK;
}

int rbx_batch_kernel_times(rbx_batch* b, double* ms_forces, double* ms_integrator, int* groups) {
    int rc = check(b);
    if (rc) return rc;
    double t[2] = {0.0, 0.0};
    for (size_t i = 0; i < b->ev_marks.size(); i++) {
        float ms = 0.0f;
        BATCH_TRY(cudaEventSynchronize(b->ev_pool[b->ev_marks[i].second]));
        BATCH_TRY(cudaEventElapsedTime(&ms, b->ev_pool[b->ev_marks[i].first], b->ev_pool[b->ev_marks[i].second]));
        t[b->ev_kind[i]] += ms;
    }
    if (ms_forces) *ms_forces = t[0];
    if (ms_integrator) *ms_integrator = t[1];
    if (groups) *groups = (int)b->ev_marks.size();
    b->ev_marks.clear();
    b->ev_kind.clear();
    b->ev_used = 0;
    return RBX_OK;
}

int rbx_batch_last_launch_count(const rbx_batch* b) { return b ? b->last_launches : 0; }

}  // extern "C"
