// ============================================================================
//  k_squirmer.cuh -- the per-step squirmer update on the device, one CTA:
//
//   stage FORCE: sum the boundary-link partials of the step into Fh, Th
//                (fixed order, deterministic) -- the tail of LBM::step
//                (lbm.cpp:219-223).
//   stage BODY : LBM::applyWallPotential, Squirmer::integrate and
//                LBM::enforceMinimumGap (lbm.cpp:231-253,
//                squirmer.cpp:52-77), FP64.
//   stage REMAP: LBM::updateParticleFlags(false) (lbm.cpp:271-320) with the
//                reference's order-dependent semantics, then a rebuild of the
//                boundary-link list (fluid nodes next to the sphere, in
//                ascending node order) and of the near-particle flag bits.
//                A step that changes at most SQ_FEW nodes takes a short way
//                through the same steps (remap_few); the walk over the whole
//                box runs when the candidate list is rebuilt or more change.
//   stage LOOP : time-loop bookkeeping of src/main.cpp:60-64: schedule the
//                mass correction of correction steps (applied by the next
//                stream kernel on load), record the trajectory row, and set
//                the region whose densities the next step must store.
//
//  Remap ordering. The reference walks the sphere's bounding box in z, y, x
//  order and updates flags, f and rho in place, so an uncovered node sees
//  the new state of nodes visited before it and the old state of the rest.
//  Here the changed nodes are found in parallel and compacted in box order
//  (their order key is the box index of their first visit); each changed
//  node's neighbour data (old flag, old rho, change order) is gathered in
//  parallel into shared memory; one thread then replays the changes in box
//  order, resolving neighbours that changed earlier from shared memory; the
//  writes go out in parallel. Batches of BATCH changed nodes keep the shared
//  memory bounded; a batch sees the global writes of the batches before it.
// ============================================================================
#pragma once
#include <cub/block/block_scan.cuh>

#include "k_logical.cuh"
#include "k_stream.cuh"

namespace lbmgpu {

constexpr int SQ_THREADS = 512;
constexpr int SQ_BATCH = 256;
constexpr int SQ_SORT_CAP = 2048;   // changes ordered in shared memory (3 ints each)
constexpr int SQ_GROUP = 4;         // remap candidates tested per thread with their loads in flight together
constexpr int SQ_PRE = 8;           // candidates per thread fetched ahead: 4096 of them, the shell up to R = 9
constexpr int SQ_FEW = 32;          // changed nodes that remap_few orders: one warp
constexpr int SQ_FEW_LINKS = 4096;  // boundary links that remap_few edits in shared memory (R up to about 15)
constexpr int STAGE_BODY = 1, STAGE_REMAP = 2, STAGE_LOOP = 4, STAGE_FORCE = 8;
// The launch follows a zone kernel that had itself waited for the update before
// and published order_tag: this update may read what that one wrote (its state,
// the candidate list, the node types) before its own pdl_wait.
constexpr int STAGE_PRE = 16;

struct SqArgs {
    void* f;
    uint8_t* flag;
    double* rho; double* ux; double* uy; double* uz;
    int* links;
    int* linkslot;            // node -> row of its boundary-link entry
    int link_cap;
    const double* link_part;
    const double* block_part;     // bulk kernel partials (mass in column 3)
    int nblocks;
    const double* block_part_b;   // zone kernel partials
    int nblocks_b;
    const double* block_part_w;   // wall-row partials of an ensemble member (else unused)
    int nblocks_w;
    int* ordermap;            // N entries, -1 when idle
    int* chg_node;            // changed-node list (capacity chg_cap)
    int* chg_key;
    int* cand;                // candidate nodes of the remap / link scans (chg_cap)
    uint8_t* mark;            // chg_cap bytes: one verdict per candidate
    int chg_cap;
    int* shell;               // cached remap candidates (chg_cap entries)
    ShellCache* shell_hdr;
    double* traj;             // TRAJ_RING x TRAJ_COLS
    SqState* sq;
    int parity;               // parity of the state being remapped
    int stages;
    int corr_step;            // this step is a mass-correction step (time-loop mode)
    int zslot_a, zslot_b;     // zone slots to (re)write from the new position, -1: none
    const int* order;         // STAGE_PRE: the word that the step's zone kernel publishes, and its value
    int order_tag;
};

struct ChgSh {
    double r[3];
    double p[3];
    double mass;
    double rr, ub[3];
    double nbrho[18];
    int nbord[18];
    int node, kind;           // kind: 1 covered, 2 uncovered
    uint8_t nbfl[18];
};

// softWallForce (squirmer.cpp:73-77)
__device__ __forceinline__ double soft_wall_force(double h, double eps, double FS, double hc) {
    if (h >= hc) return 0.0;
    const double s = 1.0 - fmax(h, 0.0) / hc;
    return eps * FS * s * s;
}

// Deterministic block sum of one column of a strided array: each thread its
// rows in order, a shuffle tree per warp, the warps in order.
__device__ __forceinline__ void block_sum_rows(const double* base, int rows, int stride, int col, double* out_sh) {
    __shared__ double red[SQ_THREADS / 32];
    double acc = 0.0;
    constexpr int U = 8;   // rows per thread with their loads in flight together
#pragma unroll 1
    for (int k0 = threadIdx.x; k0 < rows; k0 += U * SQ_THREADS) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * SQ_THREADS;
            v[u] = k < rows ? base[(size_t)k * stride + col] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k0 + u * SQ_THREADS < rows) acc += v[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < SQ_THREADS / 32; ++w) t += red[w];
        *out_sh = t;
    }
    __syncthreads();
}

// The link rows' sums (six columns of `cap` rows each), up to the warps: red[w]
// gets warp w's. In the first level of the tree the half-warps exchange three
// columns each, so that every later level moves three columns instead of six
// (the shuffles are what this stage waits for).
__device__ __forceinline__ void link_warp_sums(const double* part, int rows, size_t cap, double (*red)[6]) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double acc[6] = {0, 0, 0, 0, 0, 0}, half[3] = {0, 0, 0};
    if (wid * 32 < rows) {   // a warp without rows adds 0
#pragma unroll 2
        for (int k = threadIdx.x; k < rows; k += SQ_THREADS)
#pragma unroll
            for (int c = 0; c < 6; ++c) acc[c] += part[c * cap + k];
        const bool hi = lane >= 16;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            half[c] = (hi ? acc[3 + c] : acc[c]) + __shfl_xor_sync(ALL, hi ? acc[c] : acc[3 + c], 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) half[c] += __shfl_down_sync(ALL, half[c], o, 16);
    }
    if ((lane & 15) == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) red[wid][(lane >> 4) * 3 + c] = half[c];
}
__device__ __forceinline__ double link_total(const double (*red)[6], int c) {   // the warps in order
    double v[SQ_THREADS / 32], t = 0.0;
#pragma unroll
    for (int w = 0; w < SQ_THREADS / 32; ++w) v[w] = red[w][c];
#pragma unroll
    for (int w = 0; w < SQ_THREADS / 32; ++w) t += v[w];
    return t;
}

// Coordinates along one axis of a box, visited in ascending wrapped order.
struct AxisRange {
    int start, width, n, wrap;
    __device__ void init(int lo_unwrapped, int w, int nd) {
        if (w >= nd) { start = 0; width = nd; wrap = 0; n = nd; return; }
        start = ((lo_unwrapped % nd) + nd) % nd;
        width = w; n = nd;
        wrap = start + w > nd ? start + w - nd : 0;
    }
    __device__ int at(int b) const { return b < wrap ? b : start + (b - wrap); }
};

static_assert(3 * SQ_SORT_CAP * sizeof(int) <= SQ_BATCH * sizeof(ChgSh), "the change sort fits the batch stage");

// What one update keeps in shared memory besides the batch stage.
struct SqShared {
    SqState s;
    double red[SQ_THREADS / 32][6], sum;
    double mass_delta;            // stored mass that covered and uncovered nodes take or bring (correction steps)
    long long dfluid;
    int total, box[6], rebuild, ncand, few, nins, nrem;
    int wbox[3];                  // the box's corner wrapped into the lattice
    float off[3];                 // the centre from the node below the candidate list's
    typename cub::BlockScan<int, SQ_THREADS>::TempStorage scan;
};

// ---------------------------------------------------------------------------
//  remap_few: the remap of a step that changes at most SQ_FEW nodes and a link
//  list of at most SQ_FEW_LINKS entries, which is nearly every step (a sphere
//  moving U cells a step changes about 2 pi R^2 U nodes: 0.3 to 3 in the
//  channels here). Everything stays in shared memory, one warp replays the
//  changes, and the list is edited (entries gained and lost near the changed
//  nodes) instead of being rebuilt by two walks over the sphere's box.
//  The whole update is bound by latency, on one SM: its dependent loads, its
//  FP64 chains (8 cycles an addition, 130 a division), its barriers and its
//  instruction fetches. Hence reads gathered into one round, ordered sums over
//  values already in registers, divisions done once for all components, and
//  the velocity set from immediates. Launched back to back the update takes
//  7.1 us (64x34x32, R = 4; 14.9 with rebuilt lists and serial parts) to 9.1 us
//  (256x128x128, R = 8; 21.7); a step with changes adds about 4-6 us (before:
//  35-45 us). 64x34x32 FP64 channel: 37.7 -> 20.3 us a step.
// ---------------------------------------------------------------------------
struct FewSh {
    double pop[SQ_FEW][Q];        // covered: the node's stored numbers
    double nbrho[SQ_FEW][Q];      // uncovered: the neighbours' densities
    double part[SQ_FEW][6];       // what the change adds to Fc, Tc
    double ub[SQ_FEW][3], rr[SQ_FEW], mass[SQ_FEW];
    unsigned fnode[SQ_FEW];       // changed nodes as found
    int fkind[SQ_FEW];
    unsigned node[SQ_FEW];        // in the order of their first visit in the box
    int x[SQ_FEW], y[SQ_FEW], z[SQ_FEW], kind[SQ_FEW];   // kind: 1 covered, 2 uncovered
    int8_t nbord[SQ_FEW][Q];      // the change that neighbour j is, or -1
    uint8_t flag[SQ_FEW][Q];      // flag byte of neighbour j (0: the node) before the changes
    uint8_t near[SQ_FEW][Q];      // neighbour j (0: the node) has a PARTICLE neighbour after them
    unsigned ins[SQ_FEW * Q], rem[SQ_FEW * Q];           // nodes that enter / leave the link list
    int list[SQ_FEW_LINKS];       // the link list (fetched ahead)
};
// The candidates fetched ahead, each written and read by the same thread: the
// node, and its offset from the node below the list's reference centre, 10 bits
// an axis (R <= 200), with its type.
struct CandSh {
    unsigned n[SQ_PRE * SQ_THREADS], word[SQ_PRE * SQ_THREADS];
};
constexpr size_t FEW_BYTES = (sizeof(FewSh) + 15) / 16 * 16;
static_assert(FEW_BYTES + sizeof(CandSh) <= SQ_BATCH * sizeof(ChgSh),
              "the few-changes stage and the candidates fit the batch stage");

// index distance a - b on an axis of n nodes, as -1, 0, 1 for neighbours (with
// wrap) and something else otherwise
__device__ __forceinline__ int axis_delta(int a, int b, int n) {
    const int d = a - b;
    return d == n - 1 ? -1 : (d == 1 - n ? 1 : d);
}
__device__ __forceinline__ bool near_or_same(const Lattice& L, const FewSh& w, int e, int x, int y, int z) {
    const int dx = abs(axis_delta(x, w.x[e], L.nx)), dy = abs(axis_delta(y, w.y[e], L.ny)),
              dz = abs(axis_delta(z, w.z[e], L.nz));
    return dx <= 1 && dy <= 1 && dz <= 1 && dx + dy + dz < 3;
}
__device__ __forceinline__ int wrap1(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }
__device__ __forceinline__ unsigned node_at(const Lattice& L, int x, int y, int z) {
    return (unsigned)x + (unsigned)L.nx * ((unsigned)y + (unsigned)L.ny * (unsigned)z);
}
// equilibrium() (lattice.hpp:42-47) of direction i
__device__ __forceinline__ double equilibrium_rt(int i, double rr, const double* ub) {
    const double cu = cx_rt(i) * ub[0] + cy_rt(i) * ub[1] + cz_rt(i) * ub[2];
    const double usq = ub[0] * ub[0] + ub[1] * ub[1] + ub[2] * ub[2];
    return w_rt(i) * rr * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq);
}

// Called by all threads; w.f* hold the nfew changes in any order.
template <class S>
__device__ __forceinline__ void remap_few(const Lattice& L, const SqArgs& a, SqShared& sh, FewSh& w, int nfew,
                                          bool corr_step) {
    SqState& s = sh.s;
    const int tid = threadIdx.x;
    const int nold = s.n_links;
    if (tid < 32) {   // order of the first visit in the box (z, y, x): rank on the visit index
        const unsigned n = tid < nfew ? w.fnode[tid] : 0u, q = n / (unsigned)L.nx, z = q / (unsigned)L.ny;
        const int x = (int)(n - q * (unsigned)L.nx), y = (int)(q - z * (unsigned)L.ny);
        const int kx = x - sh.wbox[0], ky = y - sh.wbox[1], kz = (int)z - sh.wbox[2];
        const int key = ((kz < 0 ? kz + L.nz : kz) * sh.box[4] + (ky < 0 ? ky + L.ny : ky)) * sh.box[3] +
                        (kx < 0 ? kx + L.nx : kx);
        int rank = 0;
#pragma unroll 1
        for (int j = 0; j < nfew; ++j) rank += __shfl_sync(0xffffffffu, key, j) < key;
        if (tid < nfew) {
            w.node[rank] = n;
            w.x[rank] = x; w.y[rank] = y; w.z[rank] = (int)z;
            w.kind[rank] = w.fkind[tid];
        }
    }
    for (int k = tid; k < nfew * Q; k += SQ_THREADS) w.near[k / Q][k % Q] = 0;
    __syncthreads();
    // Everything that is read, in one round: the flags of the changed nodes
    // and their neighbours, a covered node's populations, an uncovered one's
    // neighbouring densities (tasks below nfew Q), and for each of those nodes
    // whether one of its 18 neighbours is PARTICLE once the changes are made
    // (a changed node's type follows from its kind).
#pragma unroll 1
    for (int q = tid; q < nfew * Q * Q; q += SQ_THREADS) {
        const bool near = q >= nfew * Q;
        const int ej = near ? (q - nfew * Q) / 18 : q, i = near ? (q - nfew * Q) % 18 + 1 : 0;
        const int e = ej / Q, j = ej - e * Q;
        int x = wrap1(w.x[e] + cx_rt(j), L.nx), y = wrap1(w.y[e] + cy_rt(j), L.ny), z = wrap1(w.z[e] + cz_rt(j), L.nz);
        if (near) { x = wrap1(x + cx_rt(i), L.nx); y = wrap1(y + cy_rt(i), L.ny); z = wrap1(z + cz_rt(i), L.nz); }
        const unsigned m = node_at(L, x, y, z);
        const uint8_t fm = a.flag[m];
        double v = 0.0;
        if (!near)
            v = w.kind[e] == 1 ? Pop<S>::raw(a.f, logical_slot(L, a.parity, j, w.node[e], w.x[e], w.y[e], w.z[e])) : a.rho[m];
        int o = -1;
#pragma unroll 1
        for (int k = 0; k < nfew; ++k)
            if (w.node[k] == m) o = k;
        if (near) {
            if (o >= 0 ? w.kind[o] == 1 : (fm & TYPE_MASK) == T_PARTICLE) w.near[e][j] = 1;
        } else {
            w.flag[e][j] = fm;
            w.nbord[e][j] = (int8_t)o;
            (w.kind[e] == 1 ? w.pop : w.nbrho)[e][j] = v;
        }
    }
    __syncthreads();
    if (tid < 32) {   // lane e replays change e; an uncovered node waits for the refills it reads
        const int e = tid;
        const bool mine = e < nfew;
        const int kind = mine ? w.kind[e] : 0;
        double r[3] = {0, 0, 0}, p[3] = {0, 0, 0}, nb[Q];
        unsigned dep = 0, fluid = 0;
        if (mine) offset_from_squirmer(L, &s, w.x[e], w.y[e], w.z[e], r);
        if (kind == 1) {   // covered: momentum of the node's populations (lbm.cpp:294-298)
            double m = 0;
#pragma unroll
            for (int i = 0; i < Q; ++i) nb[i] = w.pop[e][i];
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const double fv = S::shifted ? WD(i) + nb[i] : nb[i];
                if (CX(i) > 0) p[0] += fv; else if (CX(i) < 0) p[0] -= fv;
                if (CY(i) > 0) p[1] += fv; else if (CY(i) < 0) p[1] -= fv;
                if (CZ(i) > 0) p[2] += fv; else if (CZ(i) < 0) p[2] -= fv;
                m += nb[i];
            }
            w.mass[e] = m;
        } else if (kind == 2) {
#pragma unroll
            for (int j = 1; j < Q; ++j) {
                const int o = w.nbord[e][j];
                bool fl = (w.flag[e][j] & TYPE_MASK) == T_FLUID;
                nb[j] = w.nbrho[e][j];
                if (o >= 0 && o < e) {   // changed earlier
                    fl = w.kind[o] == 2;
                    if (fl) dep |= 1u << o;
                }
                if (fl) fluid |= 1u << j;
            }
        }
        bool done = kind != 2;
#pragma unroll 1
        for (unsigned all = __ballot_sync(0xffffffffu, done); all != 0xffffffffu;) {
            if (!done && (dep & ~all) == 0) {   // uncovered: refill (lbm.cpp:302-317)
                double rs = 0;
                if (dep)
                    for (int j = 1; j < Q; ++j) {   // a refilled neighbour's density
                        const int o = w.nbord[e][j];
                        if (o >= 0 && o < e && w.kind[o] == 2) w.nbrho[e][j] = w.rr[o];
                    }
#pragma unroll
                for (int j = 1; j < Q; ++j) {
                    const double v = dep ? w.nbrho[e][j] : nb[j];
                    if (fluid >> j & 1u) rs += v;
                }
                const double rr = fluid ? rs / __popc(fluid) : 1.0;
                double ub[3];
                surface_velocity(&s, r, ub, false);
                w.rr[e] = rr;
#pragma unroll
                for (int d = 0; d < 3; ++d) { w.ub[e][d] = ub[d]; p[d] = rr * ub[d]; }
                done = true;
            }
            __syncwarp();
            all = __ballot_sync(0xffffffffu, done);
        }
        if (mine) {   // a covered node's momentum is gained, a refilled one's given
            const double sg = kind == 1 ? 1.0 : -1.0;
            w.part[e][0] = sg * p[0]; w.part[e][1] = sg * p[1]; w.part[e][2] = sg * p[2];
            w.part[e][3] = sg * (r[1] * p[2] - r[2] * p[1]);
            w.part[e][4] = sg * (r[2] * p[0] - r[0] * p[2]);
            w.part[e][5] = sg * (r[0] * p[1] - r[1] * p[0]);
        }
        __syncwarp();   // part and mass are read by other lanes; a vote does not order memory
        const unsigned unc = __ballot_sync(0xffffffffu, kind == 2);
        if (tid < 6) {   // Fc, Tc: the changes in order
            double* acc = tid < 3 ? &s.Fc[tid] : &s.Tc[tid - 3];
            double v = *acc;
#pragma unroll 1
            for (int k = 0; k < nfew; ++k) v += w.part[k][tid];
            *acc = v;
        }
        if (tid == 0) {
            sh.dfluid += 2 * __popc(unc) - nfew;
            if (corr_step) {
                double md = sh.mass_delta;
                for (int k = 0; k < nfew; ++k) {
                    if (w.kind[k] == 1) md -= w.mass[k];
                    else
                        for (int i = 0; i < Q; ++i) md += Pop<S>::stored_raw(equilibrium_rt(i, w.rr[k], w.ub[k]), i);
                }
                sh.mass_delta = md;
            }
        }
    } else {
        // Meanwhile the nodes' new types, and the nodes that enter or leave the
        // link list: only the changed nodes and their neighbours can, each
        // handled once, by the first change it is near.
#pragma unroll 1
        for (int q = tid - 32; q < nfew * Q; q += SQ_THREADS - 32) {
            const int e = q / Q, j = q - e * Q;
            const int x = wrap1(w.x[e] + cx_rt(j), L.nx), y = wrap1(w.y[e] + cy_rt(j), L.ny),
                      z = wrap1(w.z[e] + cz_rt(j), L.nz);
            bool first = true;
#pragma unroll 1
            for (int k = 0; k < e; ++k) first = first && !near_or_same(L, w, k, x, y, z);
            if (!first) continue;
            const unsigned m = node_at(L, x, y, z);
            const int o = w.nbord[e][j];   // the change that m is
            const uint8_t fm = w.flag[e][j];
            uint8_t nf = fm & (uint8_t)~NEAR_PARTICLE;
            if (o >= 0) {
                const bool nw = (L.walls_y && (y == 1 || y == L.ny - 2)) || (L.walls_z && (z == 1 || z == L.nz - 2));
                nf = w.kind[o] == 1 ? T_PARTICLE : (uint8_t)(T_FLUID | (nw ? NEAR_WALL : 0));
            }
            const bool was = (fm & NEAR_PARTICLE) != 0, is = (nf & TYPE_MASK) == T_FLUID && w.near[e][j];
            if (is) nf |= NEAR_PARTICLE;
            if (nf != fm) a.flag[m] = nf;
            if (is && !was) w.ins[atomicAdd(&sh.nins, 1)] = m;
            if (was && !is) w.rem[atomicAdd(&sh.nrem, 1)] = m;
        }
    }
    __syncthreads();
    // the refilled populations, rho and u of uncovered nodes
#pragma unroll 1
    for (int q = tid; q < nfew * Q; q += SQ_THREADS) {
        const int e = q / Q, j = q - e * Q;
        if (w.kind[e] != 2) continue;
        const unsigned n = w.node[e];
        Pop<S>::put(a.f, logical_slot(L, a.parity, j, n, w.x[e], w.y[e], w.z[e]), j, equilibrium_rt(j, w.rr[e], w.ub[e]));
        if (j == 0) { a.rho[n] = w.rr[e]; a.ux[n] = w.ub[e][0]; a.uy[n] = w.ub[e][1]; a.uz[n] = w.ub[e][2]; }
    }
    const int nins = sh.nins, nrem = sh.nrem;
    if (nins + nrem > 0) {   // uniform: every entry to its new place in the ascending list
#pragma unroll 1
        for (int k = SQ_THREADS - 1 - tid; k < nold + nins; k += SQ_THREADS) {
            const bool fresh = k >= nold;
            const unsigned n = fresh ? w.ins[k - nold] : (unsigned)w.list[k];
            int pos = k;
            if (fresh) {   // old entries below n
                int lo = 0, hi = nold;
#pragma unroll 1
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if ((unsigned)w.list[mid] < n) lo = mid + 1; else hi = mid;
                }
                pos = lo;
            }
            bool gone = false;
#pragma unroll 1
            for (int j = 0; j < nrem; ++j) { pos -= w.rem[j] < n; gone = gone || (!fresh && w.rem[j] == n); }
#pragma unroll 1
            for (int j = 0; j < nins; ++j) pos += w.ins[j] < n;
            if (!gone && pos < a.link_cap && (fresh || pos != k)) {
                a.links[pos] = (int)n;
                a.linkslot[n] = pos;
            }
        }
        if (tid == 0) {
            const int nnew = nold + nins - nrem;
            s.n_links = min(nnew, a.link_cap);
            if (nnew > a.link_cap) s.status |= ST_LINK_OVERFLOW;
        }
    }
}

// The remap by the candidate list in full: rebuilds the list where needed,
// orders any number of changes, and rebuilds the link list by walks over the
// sphere's box. Off the usual path (remap_few) except for spheres of R > 15, so
// it is kept out of line; what its walks use of its arguments is held locally,
// since through the references every store might have changed it. A step of a
// fast sphere (U = 0.005): R = 20 333 -> 262 us, R = 40 1,923 -> 1,491, with the
// candidates of long link lists tested here only. (All arguments held locally:
// 254 and 1,468, but a stack frame that costs every update 0.5 us.)
template <class S>
__device__ __noinline__ void remap_walk(const Lattice& lattice, const SqArgs& args, SqShared& sh, int shell_ok,
                                        bool corr_step) {
    Lattice L;
    L.nx = lattice.nx; L.ny = lattice.ny; L.nz = lattice.nz; L.N = lattice.N; L.nxy = lattice.nxy;
    L.walls_y = lattice.walls_y; L.walls_z = lattice.walls_z;
    const SqArgs& a = args;
    int* const a_shell = args.shell;
    int* const a_cand = args.cand;
    const int a_chg_cap = args.chg_cap;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ChgSh* ch = reinterpret_cast<ChgSh*>(smem_raw);
    typedef cub::BlockScan<int, SQ_THREADS> Scan;
    SqState& s = sh.s;
    int &sh_total = sh.total, &sh_rebuild = sh.rebuild, &sh_ncand = sh.ncand;
    double& sh_mass_delta = sh.mass_delta;
    long long& sh_dfluid = sh.dfluid;
    auto& scan_tmp = sh.scan;
    const int tid = threadIdx.x;
    const int bx0 = sh.box[0], by0 = sh.box[1], bz0 = sh.box[2];
    const int bw = sh.box[3], bh = sh.box[4], bd = sh.box[5];
    const int V = bw * bh * bd;
    const double R2 = s.R * s.R;
    // Wrapped centre for the cheap distance filters (X[0] is kept unwrapped).
    const double cxw = s.X[0] - L.nx * floor(s.X[0] / L.nx);
    const double cyw = L.walls_y ? s.X[1] : s.X[1] - L.ny * floor(s.X[1] / L.ny);
    const double czw = L.walls_z ? s.X[2] : s.X[2] - L.nz * floor(s.X[2] / L.nz);
    auto approx_r2 = [&](int x, int y, int z) -> double {
        double dx = x - cxw, dy = y - cyw, dz = z - czw;
        if (dx > 0.5 * L.nx) dx -= L.nx; else if (dx < -0.5 * L.nx) dx += L.nx;
        if (!L.walls_y) { if (dy > 0.5 * L.ny) dy -= L.ny; else if (dy < -0.5 * L.ny) dy += L.ny; }
        if (!L.walls_z) { if (dz > 0.5 * L.nz) dz -= L.nz; else if (dz < -0.5 * L.nz) dz += L.nz; }
        return dx * dx + dy * dy + dz * dz;
    };
    // Only nodes within one cell of the sphere's surface can change: the
    // centre moved less than a cell since the last remap (checked in stage
    // BODY), so nodes deeper than that were and stay PARTICLE and nodes
    // farther out were and stay FLUID. The candidates are the nodes within
    // R +- 1.05 of the centre (0.05 covers the cheap distance against the
    // reference's exact offset, which makes the decision). The shell list
    // widens that by SHELL_SLACK around a reference centre, so it holds
    // every candidate while the centre stays within SHELL_SLACK of it
    // (triangle inequality), and the box walk that builds it runs only
    // when the centre leaves that ball.

    // (1) candidates: the cached shell, rebuilt in box order (z, y, x of
    // the first visit) when the centre has left the slack around the
    // reference centre of the list. A cached list that yields more than
    // SQ_SORT_CAP changes is rebuilt at once (second pass).
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            if (!(!sh_rebuild && sh_total > SQ_SORT_CAP)) break;   // uniform
            __syncthreads();
            if (tid == 0) sh_rebuild = 1;
            __syncthreads();
        }
        const int chunk = (V + SQ_THREADS - 1) / SQ_THREADS;
        const int k0 = min(V, tid * chunk), k1 = min(V, k0 + chunk);
        auto box_walk = [&](auto&& visit) {
            if (k0 >= k1) return;
            int bx = k0 % bw, by = (k0 / bw) % bh, bz = k0 / (bw * bh);
            int x = (((bx0 + bx) % L.nx) + L.nx) % L.nx;
            int y = (((by0 + by) % L.ny) + L.ny) % L.ny;
            int z = (((bz0 + bz) % L.nz) + L.nz) % L.nz;
            for (int k = k0; k < k1; ++k) {
                // a box wider than the lattice revisits nodes; the first visit counts
                if (bx < L.nx && by < L.ny && bz < L.nz) visit(k, x, y, z);
                if (++bx == bw) {
                    bx = 0; x = (((bx0) % L.nx) + L.nx) % L.nx;
                    if (++by == bh) { by = 0; y = (((by0) % L.ny) + L.ny) % L.ny; ++bz; if (++z == L.nz) z = 0; }
                    else if (++y == L.ny) y = 0;
                } else if (++x == L.nx) x = 0;
            }
        };
        if (sh_rebuild) {   // uniform
            const double Sin = fmax(s.R - 1.05 - SHELL_SLACK, 0.0), Sout = s.R + 1.05 + SHELL_SLACK;
            const double Sin2 = Sin * Sin, Sout2 = Sout * Sout;
            int cnt = 0;
            box_walk([&](int, int x, int y, int z) {
                const double r2 = approx_r2(x, y, z);
                cnt += (r2 >= Sin2 && r2 < Sout2);
            });
            int off = 0;
            Scan(scan_tmp).ExclusiveSum(cnt, off, sh_total);
            __syncthreads();
            box_walk([&](int, int x, int y, int z) {
                const double r2 = approx_r2(x, y, z);
                if (r2 >= Sin2 && r2 < Sout2) {
                    if (off < a_chg_cap) a_shell[off] = x + L.nx * (y + L.ny * z);
                    ++off;
                }
            });
            if (tid == 0) {
                sh_ncand = min(sh_total, a_chg_cap);
                ShellCache hc;
                for (int d = 0; d < 3; ++d) hc.X[d] = s.X[d];
                hc.n = sh_ncand;
                hc.valid = shell_ok == 2 ? 2 : 1;
                *a.shell_hdr = hc;
            }
            __syncthreads();
        }
        const int ncand = sh_ncand;
        // (2) exact test of each candidate (flag load + the reference's
        // offset), SQ_GROUP candidates per thread at a time: their node
        // indices and flags are all loaded before the first test
        for (int c0 = tid; c0 < ncand; c0 += SQ_GROUP * SQ_THREADS) {
            unsigned nn[SQ_GROUP];
            uint8_t ty[SQ_GROUP];
#pragma unroll
            for (int g = 0; g < SQ_GROUP; ++g) {
                const int c = c0 + g * SQ_THREADS;
                nn[g] = c < ncand ? (unsigned)a_shell[c] : 0u;
            }
#pragma unroll
            for (int g = 0; g < SQ_GROUP; ++g)
                ty[g] = c0 + g * SQ_THREADS < ncand ? (uint8_t)(a.flag[nn[g]] & TYPE_MASK) : (uint8_t)T_WALL;
#pragma unroll
            for (int g = 0; g < SQ_GROUP; ++g) {
                const int c = c0 + g * SQ_THREADS;
                if (c >= ncand) break;
                const unsigned n = nn[g];
                uint8_t mk = 0;
                if (ty[g] != T_WALL) {
                    const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                              z = (int)(n / L.nxy);
                    double r[3];
                    offset_from_squirmer(L, &s, x, y, z, r);
                    const bool inside = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] < R2;
                    if (inside != (ty[g] == T_PARTICLE)) mk = inside ? 1 : 2;
                }
                a.mark[c] = mk;
            }
        }
        __syncthreads();
        // (3) changed nodes in list order
        {
            const int ch2 = (ncand + SQ_THREADS - 1) / SQ_THREADS;
            const int c0 = min(ncand, tid * ch2), c1 = min(ncand, c0 + ch2);
            int cnt = 0;
            for (int c = c0; c < c1; ++c) cnt += a.mark[c] != 0;
            int off = 0;
            Scan(scan_tmp).ExclusiveSum(cnt, off, sh_total);
            __syncthreads();
            for (int c = c0; c < c1; ++c) {
                const uint8_t mk = a.mark[c];
                if (!mk) continue;
                a.chg_node[off] = a_shell[c];
                a.chg_key[off] = mk;
                ++off;
            }
        }
        __syncthreads();
    }
    // A list cached under an earlier box is in that box's order: put the
    // changes in the order of their first visit in this box (rank sort on
    // the visit index; distinct nodes have distinct indices).
    if (!sh_rebuild && sh_total > 1) {   // uniform
        const int nchg = sh_total;
        int* keys = reinterpret_cast<int*>(smem_raw);
        int* nodes = keys + SQ_SORT_CAP;
        int* kinds = nodes + SQ_SORT_CAP;
        for (int e = tid; e < nchg; e += SQ_THREADS) {
            const unsigned n = (unsigned)a.chg_node[e];
            const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                      z = (int)(n / L.nxy);
            const int kx = ((x - bx0) % L.nx + L.nx) % L.nx;
            const int ky = ((y - by0) % L.ny + L.ny) % L.ny;
            const int kz = ((z - bz0) % L.nz + L.nz) % L.nz;
            keys[e] = (kz * bh + ky) * bw + kx;
            nodes[e] = (int)n;
            kinds[e] = a.chg_key[e];
        }
        __syncthreads();
        for (int e = tid; e < nchg; e += SQ_THREADS) {
            const int ke = keys[e];
            int rank = 0;
            for (int j = 0; j < nchg; ++j) rank += keys[j] < ke;
            a.chg_node[rank] = nodes[e];
            a.chg_key[rank] = kinds[e];
        }
        __syncthreads();
    }
    const int total = sh_total;
    for (int k = tid; k < total; k += SQ_THREADS) a.ordermap[a.chg_node[k]] = k;
    __syncthreads();

    // (4) batches: gather, ordered replay, scatter
    for (int b0 = 0; b0 < total; b0 += SQ_BATCH) {
        const int nb = min(SQ_BATCH, total - b0);
        for (int e = tid; e < nb; e += SQ_THREADS) {
            ChgSh& c = ch[e];
            const unsigned n = (unsigned)a.chg_node[b0 + e];
            c.node = (int)n;
            c.kind = a.chg_key[b0 + e];
            const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                      z = (int)(n / L.nxy);
            offset_from_squirmer(L, &s, x, y, z, c.r);
            if (c.kind == 1) {
                // covered: momentum of the node's populations (lbm.cpp:294-298)
                double p0 = 0, p1 = 0, p2 = 0, m = 0;
                for (int i = 0; i < Q; ++i) {
                    const size_t k = logical_slot(L, a.parity, i, n, x, y, z);
                    const double fv = Pop<S>::get(a.f, k, i);
                    p0 += fv * cx_rt(i); p1 += fv * cy_rt(i); p2 += fv * cz_rt(i);
                    m += Pop<S>::raw(a.f, k);
                }
                c.p[0] = p0; c.p[1] = p1; c.p[2] = p2; c.mass = m;
            }
        }
        __syncthreads();
        for (int q = tid; q < nb * 18; q += SQ_THREADS) {
            const int e = q / 18, j = q % 18 + 1;
            ChgSh& c = ch[e];
            if (c.kind != 2) continue;
            const unsigned n = (unsigned)c.node;
            const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                      z = (int)(n / L.nxy);
            // lbm.cpp:305: neighbour with wrap in every axis
            const int xn = (x + cx_rt(j) + L.nx) % L.nx, yn = (y + cy_rt(j) + L.ny) % L.ny,
                      zn = (z + cz_rt(j) + L.nz) % L.nz;
            const unsigned m = (unsigned)xn + (unsigned)L.nx * ((unsigned)yn + (unsigned)L.ny * (unsigned)zn);
            c.nbfl[j - 1] = a.flag[m] & TYPE_MASK;
            c.nbrho[j - 1] = a.rho[m];
            c.nbord[j - 1] = a.ordermap[m];
        }
        __syncthreads();
        if (tid == 0) {
            for (int e = 0; e < nb; ++e) {
                ChgSh& c = ch[e];
                if (c.kind == 1) {
                    const double t0 = c.r[1] * c.p[2] - c.r[2] * c.p[1];
                    const double t1 = c.r[2] * c.p[0] - c.r[0] * c.p[2];
                    const double t2 = c.r[0] * c.p[1] - c.r[1] * c.p[0];
                    s.Fc[0] += c.p[0]; s.Tc[0] += t0;
                    s.Fc[1] += c.p[1]; s.Tc[1] += t1;
                    s.Fc[2] += c.p[2]; s.Tc[2] += t2;
                    if (corr_step) sh_mass_delta -= c.mass;
                    sh_dfluid -= 1;
                    continue;
                }
                // uncovered: refill (lbm.cpp:302-317)
                double rs = 0; int cntf = 0;
                const int k_me = b0 + e;
                for (int j = 0; j < 18; ++j) {
                    const int o = c.nbord[j];
                    uint8_t ty = c.nbfl[j];
                    double rv = c.nbrho[j];
                    if (o >= b0 && o < k_me) {  // changed earlier in this batch
                        const ChgSh& cc = ch[o - b0];
                        ty = cc.kind == 1 ? T_PARTICLE : T_FLUID;
                        if (cc.kind == 2) rv = cc.rr;
                    }
                    if (ty == T_FLUID) { rs += rv; ++cntf; }
                }
                const double rr = cntf ? rs / cntf : 1.0;
                double ub[3];
                surface_velocity(&s, c.r, ub, false);
                c.rr = rr; c.ub[0] = ub[0]; c.ub[1] = ub[1]; c.ub[2] = ub[2];
                const double p0 = rr * ub[0], p1 = rr * ub[1], p2 = rr * ub[2];
                const double t0 = c.r[1] * p2 - c.r[2] * p1;
                const double t1 = c.r[2] * p0 - c.r[0] * p2;
                const double t2 = c.r[0] * p1 - c.r[1] * p0;
                s.Fc[0] -= p0; s.Tc[0] -= t0;
                s.Fc[1] -= p1; s.Tc[1] -= t1;
                s.Fc[2] -= p2; s.Tc[2] -= t2;
                sh_dfluid += 1;
                if (corr_step) {
                    const double usq = ub[0] * ub[0] + ub[1] * ub[1] + ub[2] * ub[2];
                    for (int i = 0; i < Q; ++i) {
                        const double cu = cx_rt(i) * ub[0] + cy_rt(i) * ub[1] + cz_rt(i) * ub[2];
                        const double feq = w_rt(i) * rr * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq);
                        sh_mass_delta += Pop<S>::stored_raw(feq, i);
                    }
                }
            }
        }
        __syncthreads();
        // scatter: flags, refilled populations, rho/u of uncovered nodes
        for (int q = tid; q < nb * Q; q += SQ_THREADS) {
            const int e = q / Q, i = q % Q;
            const ChgSh& c = ch[e];
            const unsigned n = (unsigned)c.node;
            const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                      z = (int)(n / L.nxy);
            if (i == 0) {
                uint8_t nf = T_PARTICLE;
                if (c.kind == 2) {
                    const bool nw = (L.walls_y && (y == 1 || y == L.ny - 2)) || (L.walls_z && (z == 1 || z == L.nz - 2));
                    nf = T_FLUID | (nw ? NEAR_WALL : 0);
                    a.rho[n] = c.rr; a.ux[n] = c.ub[0]; a.uy[n] = c.ub[1]; a.uz[n] = c.ub[2];
                }
                a.flag[n] = nf;
            }
            if (c.kind == 2) {
                // equilibrium() (lattice.hpp:42-47) at (rr, U + W x r)
                const double cu = cx_rt(i) * c.ub[0] + cy_rt(i) * c.ub[1] + cz_rt(i) * c.ub[2];
                const double usq = c.ub[0] * c.ub[0] + c.ub[1] * c.ub[1] + c.ub[2] * c.ub[2];
                const double feq = w_rt(i) * c.rr * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq);
                Pop<S>::put(a.f, logical_slot(L, a.parity, i, n, x, y, z), i, feq);
            }
        }
        __syncthreads();
    }
    for (int k = tid; k < total; k += SQ_THREADS) a.ordermap[a.chg_node[k]] = -1;

    // (5) boundary-link list: FLUID nodes with a PARTICLE neighbour, in
    // ascending node order over the sphere's box.
    if (total > 0 || s.n_links < 0) {
        const int old = max(0, s.n_links);
        for (int k = tid; k < old; k += SQ_THREADS) {
            const int n = a.links[k];
            a.flag[n] &= (uint8_t)~NEAR_PARTICLE;
        }
        __syncthreads();
        AxisRange ax, ay, az;
        ax.init(bx0, bw, L.nx); ay.init(by0, bh, L.ny); az.init(bz0, bd, L.nz);
        const int V2 = ax.width * ay.width * az.width;
        // after the remap FLUID means r >= R; PARTICLE neighbours lie within sqrt(2)
        const double Lin = fmax(s.R - 0.05, 0.0), Lout = s.R + 1.5;
        const double Lin2 = Lin * Lin, Lout2 = Lout * Lout;
        const int chk = (V2 + SQ_THREADS - 1) / SQ_THREADS;
        const int q0 = min(V2, tid * chk), q1 = min(V2, q0 + chk);
        auto region_walk = [&](auto&& visit) {
            for (int k = q0; k < q1; ++k) {
                const int x = ax.at(k % ax.width), y = ay.at((k / ax.width) % ay.width),
                          z = az.at(k / (ax.width * ay.width));
                visit(x, y, z);
            }
        };
        {
            int cnt = 0;
            region_walk([&](int x, int y, int z) {
                const double r2 = approx_r2(x, y, z);
                cnt += (r2 >= Lin2 && r2 < Lout2);
            });
            int off = 0;
            Scan(scan_tmp).ExclusiveSum(cnt, off, sh_total);
            __syncthreads();
            region_walk([&](int x, int y, int z) {
                const double r2 = approx_r2(x, y, z);
                if (r2 >= Lin2 && r2 < Lout2) {
                    if (off < a_chg_cap) a_cand[off] = x + L.nx * (y + L.ny * z);
                    ++off;
                }
            });
        }
        __syncthreads();
        const int nc2 = min(sh_total, a_chg_cap);
        for (int c = tid; c < nc2; c += SQ_THREADS) {
            const unsigned n = (unsigned)a_cand[c];
            uint8_t mk = 0;
            if ((a.flag[n] & TYPE_MASK) == T_FLUID) {
                const int x = (int)(n % (unsigned)L.nx), y = (int)((n / (unsigned)L.nx) % (unsigned)L.ny),
                          z = (int)(n / L.nxy);
                const Nbr nbh(L, x, y, z);
                bool near = false;
#pragma unroll
                for (int j = 1; j < Q; ++j) near |= (a.flag[nbh.of(n, j)] & TYPE_MASK) == T_PARTICLE;
                mk = near;
            }
            a.mark[c] = mk;
        }
        __syncthreads();
        {
            const int ch2 = (nc2 + SQ_THREADS - 1) / SQ_THREADS;
            const int c0 = min(nc2, tid * ch2), c1 = min(nc2, c0 + ch2);
            int cnt = 0;
            for (int c = c0; c < c1; ++c) cnt += a.mark[c];
            int off = 0;
            Scan(scan_tmp).ExclusiveSum(cnt, off, sh_total);
            __syncthreads();
            for (int c = c0; c < c1; ++c) {
                if (!a.mark[c]) continue;
                const int n = a_cand[c];
                if (off < a.link_cap) {
                    a.links[off] = n;
                    a.linkslot[n] = off;
                    a.flag[n] |= NEAR_PARTICLE;
                }
                ++off;
            }
        }
        __syncthreads();
        if (tid == 0) {
            s.n_links = min(sh_total, a.link_cap);
            if (sh_total > a.link_cap) s.status |= ST_LINK_OVERFLOW;
            a.shell_hdr->valid = 2;
        }
    }
    __syncthreads();
}

// The state a run ends a step with, word by word. The wall force belongs to
// k_finalize, and status bits are only ever added (the bulk's watchdog may set
// one meanwhile).
__device__ __forceinline__ void store_sq_state(SqState* dst, const SqState& s) {
    constexpr int NS = (int)(sizeof(SqState) / 4);
    constexpr int W0 = (int)(offsetof(SqState, wall_force) / 4), W1 = W0 + (int)(sizeof(SqState::wall_force) / 4);
    constexpr int ST = (int)(offsetof(SqState, status) / 4);
    const int t = threadIdx.x;
    if (t < NS && !(t >= W0 && t < W1) && t != ST)
        reinterpret_cast<uint32_t*>(dst)[t] = reinterpret_cast<const uint32_t*>(&s)[t];
    if (t == ST && s.status) atomicOr(&dst->status, s.status);
}

// The rigid body (stage BODY) and what the remap's test needs of the new
// centre. Warp 0 holds the components of X and U in its lanes 0-2, warp 1
// those of W and e: each step of the two chains runs once for all components,
// and side by side. What does not depend on the force is fetched and formed
// before the wait (BodyPre). The values are the reference's, operation for
// operation.
struct BodyPre {
    double X, v, c, M, y;         // component d: X, U, Fc, M, 1/M (warp 0); e, W, Tc, I, 1/I (warp 1)
    double e1, e2;                // warp 1: e[d + 1], e[d + 2]
    double lo, hi, Xs;            // warp 0: the hard gap's bounds, the node below the list's centre
    double R, hc, base;           // base: the list's centre
    int planar;
    bool yfar;
};
__device__ __forceinline__ BodyPre body_pre(const Lattice& L, const SqState& s, const double* shell_X, int warp, int d) {
    BodyPre b;
    const int nd = d == 0 ? L.nx : (d == 1 ? L.ny : L.nz), d1 = d == 2 ? 0 : d + 1, d2 = d == 0 ? 2 : d - 1;
    b.planar = s.planar;
    b.R = s.R; b.hc = s.hc;
    b.X = warp == 0 ? s.X[d] : s.e[d];
    b.v = warp == 0 ? s.U[d] : s.W[d];
    b.c = warp == 0 ? s.Fc[d] : s.Tc[d];
    b.M = warp == 0 ? s.M : s.I;
    b.y = 1.0 / b.M;
    b.yfar = divisor_far(b.M);
    b.e1 = s.e[d1]; b.e2 = s.e[d2];
    b.lo = 0.5 + s.R + s.hmin; b.hi = (nd - 1.5) - s.R - s.hmin;
    b.base = d == 0 ? shell_X[0] : (d == 1 ? shell_X[1] : shell_X[2]);
    b.Xs = floor(b.base);
    return b;
}
__device__ __forceinline__ void body_rotation(SqShared& sh, const BodyPre& b, double T, int lane, int d) {   // warp 1
    SqState& s = sh.s;
    constexpr unsigned ALL = 0xffffffffu;
    const int d1 = d == 2 ? 0 : d + 1, d2 = d == 0 ? 2 : d - 1;
    // Squirmer::integrate (squirmer.cpp:52-68)
    double w = b.v + div_by(T + b.c, b.M, b.y, numerator_far(T + b.c) || b.yfar), e = b.X;
    if (b.planar && d != 2) w = 0.0;
    e += __shfl_sync(ALL, w, d1) * b.e2 - __shfl_sync(ALL, w, d2) * b.e1;
    if (b.planar && d == 2) e = 0.0;
    const double f0 = __shfl_sync(ALL, e, 0), f1 = __shfl_sync(ALL, e, 1), f2 = __shfl_sync(ALL, e, 2);
    e /= sqrt(f0 * f0 + f1 * f1 + f2 * f2);
    if (lane < 3) {
        s.W[d] = w; s.e[d] = e; s.Tc[d] = 0.0;
        if (!(isfinite(w) && isfinite(e) && isfinite(T))) atomicOr(&s.status, ST_NAN);
    }
}
__device__ __forceinline__ void body_motion(const Lattice& L, SqShared& sh, const BodyPre& b, double F, bool body,
                                            int shell_ok, int lane, int d) {   // warp 0
    SqState& s = sh.s;
    constexpr unsigned ALL = 0xffffffffu;
    const bool walled = d == 1 ? L.walls_y != 0 : (d == 2 && L.walls_z != 0);
    double X = b.X;
    if (body) {
        // LBM::applyWallPotential (lbm.cpp:231-241): the lower and the upper wall
        double Fw = 0.0;
        if (walled) {
            const int nd = d == 1 ? L.ny : L.nz;
            const double hl = X - b.R - 0.5, hu = (nd - 1.5) - X - b.R;
            if (hl < b.hc) Fw += soft_wall_force(hl, s.eps, s.FS, b.hc);
            if (hu < b.hc) Fw -= soft_wall_force(hu, s.eps, s.FS, b.hc);
        }
        // Squirmer::integrate (squirmer.cpp:52-68)
        double v = b.v + div_by(F + b.c + Fw, b.M, b.y, numerator_far(F + b.c + Fw) || b.yfar);
        if (b.planar && d == 2) v = 0.0;
        X += v;
        int hits = 0;
        if (walled) {   // LBM::enforceMinimumGap (lbm.cpp:245-253)
            if (X < b.lo) { X = b.lo; if (v < 0) v = 0; ++hits; }
            if (X > b.hi) { X = b.hi; if (v > 0) v = 0; ++hits; }
        }
        if (lane < 3) {
            s.X[d] = X; s.U[d] = v; s.Fw[d] = Fw; s.Fc[d] = 0.0;
            // The densities the refill reads were stored for the box of the
            // previous position widened by 2; that covers this step's box
            // widened by 1 only if the centre moved less than one cell.
            if (!(isfinite(X) && isfinite(v) && isfinite(F))) atomicOr(&s.status, ST_NAN);
            else if (fabs(X - b.X) >= 1.0) atomicOr(&s.status, ST_REMAP_RANGE);
            if (hits) atomicAdd(reinterpret_cast<unsigned long long*>(&s.contacts), (unsigned long long)hits);
            if (d == 0) s.t += 1;
        }
    }
    const double q = X - b.base, q2 = q * q;
    const double r2 = __shfl_sync(ALL, q2, 0) + __shfl_sync(ALL, q2, 1) + __shfl_sync(ALL, q2, 2);
    if (lane == 0) sh.rebuild = !(shell_ok && r2 < SHELL_SLACK * SHELL_SLACK);
    if (lane < 3) sh.off[d] = (float)(X - b.Xs);
}
// The sphere's bounding box (lbm.cpp:272-276) and the zones of the coming steps
// around it (see ZoneBox), beside the remap's test: lane d of one warp.
__device__ __forceinline__ void box_and_zones(const Lattice& L, const SqArgs& a, SqShared& sh, int d) {
    SqState& s = sh.s;
    const int nd = d == 0 ? L.nx : (d == 1 ? L.ny : L.nz);
    const bool walled = d == 1 ? L.walls_y != 0 : (d == 2 && L.walls_z != 0);
    int b0 = (int)floor(s.X[d] - s.R) - 2, b1 = (int)ceil(s.X[d] + s.R) + 2;
    if (d == 1 && walled) { b0 = max(0, b0); b1 = min(nd - 1, b1); }
    const int wb = b0 >= 0 && b0 < nd ? b0 : ((b0 % nd) + nd) % nd;
    sh.box[d] = b0;
    sh.box[3 + d] = b1 - b0 + 1;
    sh.wbox[d] = wb;
    const int wd = zone_width(s.R, nd, walled);
    int lo;
    if (walled) zone_axis(b0, nd, wd, true, lo);
    else lo = wd >= nd ? 0 : wrap1(wb - ZONE_MARGIN, nd);   // zone_axis of the wrapped corner
    if (a.zslot_a >= 0) { s.zone[a.zslot_a].w[d] = wd; s.zone[a.zslot_a].lo[d] = lo; }
    if (a.zslot_b >= 0) { s.zone[a.zslot_b].w[d] = wd; s.zone[a.zslot_b].lo[d] = lo; }
}

// One update. wait() returns once everything the update reads but its own
// earlier writes is complete (false: that never came, and the update leaves).
// early: the state, the candidate list and the node types, which only updates
// write, may be read before it.
template <class S, class Wait>
__device__ __forceinline__ bool squirmer_update(const Lattice& L, const SqArgs& a, bool early, Wait&& wait) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SqShared sh;
    SqState& s = sh.s;
    const int tid = threadIdx.x;
    if (!early && !wait()) return false;
    {   // the state, one word per thread
        constexpr int NS = (int)(sizeof(SqState) / 4);
        static_assert(sizeof(SqState) % 4 == 0 && NS <= SQ_THREADS, "one word per thread");
        if (tid < NS) reinterpret_cast<uint32_t*>(&s)[tid] = __ldcg(reinterpret_cast<const uint32_t*>(a.sq) + tid);
    }
    // the first candidates of the remap (see stage REMAP) and the link list,
    // kept in shared memory until the new centre is known
    const bool remap = (a.stages & STAGE_REMAP) != 0;
    int ncand = 0, shell_ok = 0;
    double shell_X[3] = {0, 0, 0};
    CandSh& cs = *reinterpret_cast<CandSh*>(smem_raw + FEW_BYTES);
    FewSh& fw = *reinterpret_cast<FewSh*>(smem_raw);
    int cb[3] = {0, 0, 0};   // the node below the list's reference centre, wrapped
    auto cand_word = [&](unsigned n) {   // offset from cb and type
        const unsigned q = n / (unsigned)L.nx, z = q / (unsigned)L.ny;
        int dx = (int)(n - q * (unsigned)L.nx) - cb[0], dy = (int)(q - z * (unsigned)L.ny) - cb[1], dz = (int)z - cb[2];
        if (2 * dx > L.nx) dx -= L.nx; else if (2 * dx < -L.nx) dx += L.nx;
        if (!L.walls_y) { if (2 * dy > L.ny) dy -= L.ny; else if (2 * dy < -L.ny) dy += L.ny; }
        if (!L.walls_z) { if (2 * dz > L.nz) dz -= L.nz; else if (2 * dz < -L.nz) dz += L.nz; }
        return (unsigned)(dx + 512) << 22 | (unsigned)(dy + 512) << 12 | (unsigned)(dz + 512) << 2 |
               (unsigned)(__ldcg(a.flag + n) & TYPE_MASK);
    };
    if (remap) {
        shell_ok = __ldcg(&a.shell_hdr->valid);
        ncand = shell_ok ? __ldcg(&a.shell_hdr->n) : 0;
        const int nd[3] = {L.nx, L.walls_y ? 0 : L.ny, L.walls_z ? 0 : L.nz};   // 0: not periodic
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            shell_X[d] = __ldcg(&a.shell_hdr->X[d]);
            const double c0 = floor(shell_X[d]);
            cb[d] = (int)(nd[d] && !(c0 >= 0.0 && c0 < nd[d]) ? c0 - nd[d] * floor(c0 / nd[d]) : c0);
        }
        const int nl = shell_ok == 2 ? min(__ldcg(&a.sq->n_links), SQ_FEW_LINKS) : 0;
#pragma unroll 2
        for (int k = tid; k < nl; k += SQ_THREADS) fw.list[k] = __ldcg(a.links + k);
#pragma unroll 2
        for (int c = tid; c < min(ncand, SQ_PRE * SQ_THREADS); c += SQ_THREADS) {
            const unsigned n = (unsigned)__ldcg(a.shell + c);
            cs.n[c] = n;
            cs.word[c] = cand_word(n);
        }
    }
    if (tid == 0) {
        sh.mass_delta = 0.0;
        sh.dfluid = 0;
        sh.few = sh.nins = sh.nrem = 0;
        sh.ncand = ncand;
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, axis = lane < 3 ? lane : 0;
    BodyPre bp;
    if (warp < 2) bp = body_pre(L, s, shell_X, warp, axis);
    if (early && !wait()) return false;
    // invalid already; the host reports it. Every warp reads the status before
    // the next barrier, behind which the body may set bits: one verdict for all.
    if (s.status & (ST_NAN | ST_REMAP_RANGE | ST_LINK_OVERFLOW)) return true;

    const bool loop = (a.stages & STAGE_LOOP) != 0;
    const bool corr_step = loop && a.corr_step;

    // ---------------- stages FORCE, BODY ----------------
    const bool force = (a.stages & STAGE_FORCE) != 0, body = (a.stages & STAGE_BODY) != 0;
    if (force) link_warp_sums(a.link_part, s.n_links, (size_t)a.link_cap, sh.red);
    __syncthreads();
    if (warp == 0) {
        const double F = force ? link_total(sh.red, axis) : s.Fh[axis];
        if (force && lane < 3) s.Fh[lane] = F;
        body_motion(L, sh, bp, F, body, shell_ok, lane, axis);
    } else if (warp == 1) {
        const double T = force ? link_total(sh.red, 3 + axis) : s.Th[axis];
        if (force && lane < 3) s.Th[lane] = T;
        if (body) body_rotation(sh, bp, T, lane, axis);
    }
    __syncthreads();
    if (s.status & (ST_NAN | ST_REMAP_RANGE)) {
        store_sq_state(a.sq, s);
        return true;
    }

    // ---------------- stage REMAP ----------------
    // Candidates within the cached shell: each is first tested in FP32 (the
    // squared distance is off by less than 1e-6 R^2 there); one within 1e-5 R^2
    // + 1e-3 of the surface by the reference's FP64 offset, as is every one in
    // a lattice hardly wider than the sphere, where the offset may be about
    // half a lattice. If few nodes change, remap_few does the rest.
    if (remap) {
        // A link list too long for remap_few would send every step with a change
        // to the walk, which tests the candidates itself: at once then.
        bool walk = sh.rebuild != 0 || s.n_links > SQ_FEW_LINKS;   // uniform
        if (!walk) {
            const double R2 = s.R * s.R;
            const float R2f = (float)R2, span = 2.0f * (float)s.R + 10.0f, ox = sh.off[0], oy = sh.off[1], oz = sh.off[2];
            const bool tight = L.nx < span || (!L.walls_y && L.ny < span) || (!L.walls_z && L.nz < span);
            const float band = tight ? 3.0e38f : 1e-5f * R2f + 1e-3f;
#pragma unroll 2
            for (int c = tid; c < ncand; c += SQ_THREADS) {
                const unsigned wd = c < SQ_PRE * SQ_THREADS ? cs.word[c] : cand_word((unsigned)a.shell[c]);
                const unsigned ty = wd & 3u;
                if (ty == T_WALL) continue;
                const float ex = (float)((int)(wd >> 22) - 512) - ox, ey = (float)((int)(wd >> 12 & 1023u) - 512) - oy,
                            ez = (float)((int)(wd >> 2 & 1023u) - 512) - oz;
                const float gap = ex * ex + ey * ey + ez * ez - R2f;
                bool inside = gap < 0.f;
                if (inside == (ty == T_PARTICLE) && fabsf(gap) >= band) continue;
                const unsigned n = c < SQ_PRE * SQ_THREADS ? cs.n[c] : (unsigned)a.shell[c];
                const unsigned q = n / (unsigned)L.nx;
                const int x = (int)(n - q * (unsigned)L.nx), y = (int)(q % (unsigned)L.ny), z = (int)(q / (unsigned)L.ny);
                double r[3];
                offset_from_squirmer(L, &s, x, y, z, r);
                inside = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] < R2;
                if (inside != (ty == T_PARTICLE)) {
                    const int k = atomicAdd(&sh.few, 1);
                    if (k < SQ_FEW) {
                        fw.fnode[k] = n;
                        fw.fkind[k] = inside ? 1 : 2;
                    }
                }
            }
        }
        if (tid >= SQ_THREADS - 3) box_and_zones(L, a, sh, SQ_THREADS - 1 - tid);
        __syncthreads();
        const int nfew = sh.few;
        walk = walk || (nfew > 0 && (nfew > SQ_FEW || shell_ok != 2 || s.n_links < 0));
        if (walk) remap_walk<S>(L, a, sh, shell_ok, corr_step);   // uniform
        else if (nfew > 0) remap_few<S>(L, a, sh, fw, nfew, corr_step);
        if (tid == 0) s.n_fluid += sh.dfluid;
    }

    // ---------------- stage LOOP ----------------
    double mstep = 0.0;
    if (corr_step) {
        __syncthreads();
        block_sum_rows(a.block_part, a.nblocks, BLOCK_PART, 3, &sh.sum);
        mstep = sh.sum;
        __syncthreads();
        block_sum_rows(a.block_part_b, a.nblocks_b, BLOCK_PART, 3, &sh.sum);
        mstep += sh.sum;
        if (a.nblocks_w > 0) {
            __syncthreads();
            block_sum_rows(a.block_part_w, a.nblocks_w, BLOCK_PART, 3, &sh.sum);
            mstep += sh.sum;
        }
    }
    if (tid == 0) {
        s.corr_pending = 0;
        if (loop) {
            if (corr_step && s.n_fluid > 0) {
                // LBM::correctMass (lbm.cpp:324-339): d = 1 - m / n_fluid, with m
                // the populations summed after this step and its remap.
                const double m = mstep + sh.mass_delta;
                s.corr_d = S::shifted ? -(m / (double)s.n_fluid) : 1.0 - m / (double)s.n_fluid;
                s.corr_pending = 1;
            }
            const bool row = s.traj_every > 0 && ((unsigned long long)s.t <= 0xffffffffull
                                                      ? (unsigned)s.t % (unsigned)s.traj_every == 0
                                                      : s.t % s.traj_every == 0);
            if (row) {
                double* out = a.traj + (size_t)(s.traj_count % TRAJ_RING) * TRAJ_COLS;
                out[0] = (double)s.t;
                for (int d = 0; d < 3; ++d) {
                    out[1 + d] = s.X[d]; out[4 + d] = s.e[d]; out[7 + d] = s.U[d]; out[10 + d] = s.W[d];
                }
                out[13] = s.Fw[1]; out[14] = s.Fw[2];
                s.traj_count += 1;
            }
        }
    }
    __syncthreads();
    store_sq_state(a.sq, s);
    return true;
}

template <class S>
__global__ void __launch_bounds__(SQ_THREADS, 1) k_squirmer(const __grid_constant__ Lattice L,
                                                         const __grid_constant__ SqArgs a) {
    const bool early = (a.stages & STAGE_PRE) != 0;
    if (early) order_acquire(a.order, a.order_tag);   // each thread for its own reads
    squirmer_update<S>(L, a, early, [] {
        pdl_wait();
        pdl_launch_dependents();
        return true;
    });
}

// Ensemble: one CTA per member, each with its own lattice and arguments; the
// per-step settings are the same for all members.
template <class S>
__global__ void __launch_bounds__(SQ_THREADS, 1) k_squirmer_batch(const Lattice* lat, const SqArgs* args, SqStep st) {
    __shared__ __align__(16) Lattice L;
    __shared__ __align__(16) SqArgs A;
    {   // the member's records, one word per thread, with this step's settings
        constexpr int NL = (int)(sizeof(Lattice) / 4), NA = (int)(sizeof(SqArgs) / 4);
        static_assert(NL <= SQ_THREADS && NA <= SQ_THREADS, "one word per thread");
        const int t = threadIdx.x;
        if (t < NL) reinterpret_cast<uint32_t*>(&L)[t] = reinterpret_cast<const uint32_t*>(lat + blockIdx.x)[t];
        if (t < NA) {
            uint32_t w = reinterpret_cast<const uint32_t*>(args + blockIdx.x)[t];
            if (t == (int)(offsetof(SqArgs, parity) / 4)) w = (uint32_t)st.parity;
            if (t == (int)(offsetof(SqArgs, stages) / 4)) w = (uint32_t)st.stages;
            if (t == (int)(offsetof(SqArgs, corr_step) / 4)) w = (uint32_t)st.corr_step;
            if (t == (int)(offsetof(SqArgs, zslot_a) / 4)) w = (uint32_t)st.zslot_a;
            if (t == (int)(offsetof(SqArgs, zslot_b) / 4)) w = (uint32_t)st.zslot_b;
            reinterpret_cast<uint32_t*>(&A)[t] = w;
        }
    }
    __syncthreads();
    squirmer_update<S>(L, A, false, [] { return true; });
}

}  // namespace lbmgpu
