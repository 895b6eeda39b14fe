// ============================================================================
//  k_cluster.cuh -- many time steps of a small lattice without a squirmer in one
//  launch, with the populations in the shared memory of one thread-block cluster.
//
//  A step of such a lattice by separate kernels is two launches and a chain of
//  global round trips for a few thousand nodes: 3.4 us for the 4x34x34 FP64 duct,
//  whose 0.7 MB of populations would cross HBM in 0.1 us. Here a cluster of up to
//  16 CTAs holds them (each CTA the whole x-rows [rank * rows, + rows) of the
//  lattice, wall layers included, A[i][node] as in global memory), a node's
//  neighbours are read and written through distributed shared memory, and a
//  step ends at the cluster's hardware barrier. The populations are read from
//  global memory once and written back once per launch.
//  The AA pattern, the arithmetic and the values stored are those of k_bulk
//  (halfway bounce-back at a wall layer returns the post-collision value
//  itself), so the results are its bits. The last step of a call, which stores
//  the fields and sums the wall force, runs by the separate kernels.
//  Bound: instruction issue and the FP64 pipe of the few SMs, then the barrier
//  and one remote latency a step. Against the separate kernels (us a step, FP64 /
//  FP32 / FP16): 4x34x34 2.2 / 1.9 / 1.4 against 3.4 / 3.1 / 3.7; 8x32x32, the
//  largest (512 nodes per CTA), 2.9 / 2.4 / 1.7 against 3.5 / 3.2 / 3.6; with two
//  nodes per thread (16x32x32) it was 5.6 against 3.9, hence the limit of one.
// ============================================================================
#pragma once
#include "k_stream.cuh"

namespace lbmgpu {

constexpr int CLUSTER_CTAS = 16;       // CTAs of a cluster, at most (8 where 16 cannot be resident)
constexpr int CLUSTER_THREADS = 512;
constexpr int CLUSTER_NODES = CLUSTER_THREADS;   // nodes per CTA, at most: one per thread

struct ClusterWork {
    int rows;              // x-rows per CTA
    int stride;            // elements per direction in a CTA's shared memory
    int nsteps, parity;    // parity of the state before the first step
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// everything every thread of the cluster wrote to shared memory before is visible after
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t shared_addr, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(shared_addr), "r"(rank));
    return a;
}
// a stored number of a storage form at a cluster shared address, as S::ld / S::st convert it
template <class S>
__device__ __forceinline__ std::conditional_t<S::shifted, float, double> ld_cluster(uint32_t a) {
    if constexpr (sizeof(typename S::T) == 8) {
        double v;
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
        return v;
    } else if constexpr (sizeof(typename S::T) == 4) {
        float v;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
        return v;
    } else {
        unsigned short v;
        asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
        return __half2float(__ushort_as_half(v));
    }
}
template <class S, class V>
__device__ __forceinline__ void st_cluster(uint32_t a, V v) {
    if constexpr (sizeof(typename S::T) == 8) asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"((double)v) : "memory");
    else if constexpr (sizeof(typename S::T) == 4) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"((float)v) : "memory");
    else asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"(__half_as_ushort(__float2half_rn((float)v))) : "memory");
}

// One step of one fluid node. own: address of A[0][node]; slot(i): address of
// A[i][n + c_i]; wr: the wall layers next to its row (wall_row).
template <class S, int PAR, bool FORCE, class Slot>
__device__ __forceinline__ void cluster_node(const Lattice& L, uint32_t own, uint32_t dir_bytes, uint8_t wr, Slot&& slot) {
    using V = std::conditional_t<S::shifted, float, double>;
    V f[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i)
        f[i] = ld_cluster<S>(PAR == 0 || i == 0 ? own + (uint32_t)i * dir_bytes : slot(OPP(i)));
    typename S::A post[Q];
    if constexpr (!S::shifted) {
        double r = 0, mx = 0, my = 0, mz = 0;   // update_node's moments
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            r += f[i];
            if (CX(i) > 0) mx += f[i]; else if (CX(i) < 0) mx -= f[i];
            if (CY(i) > 0) my += f[i]; else if (CY(i) < 0) my -= f[i];
            if (CZ(i) > 0) mz += f[i]; else if (CZ(i) < 0) mz -= f[i];
        }
        const double Fx = L.F[0], Fy = L.F[1], Fz = L.F[2];
        double u, v, wz;
        div3(mx + 0.5 * Fx, my + 0.5 * Fy, mz + 0.5 * Fz, r, u, v, wz);
        const double usq = u * u + v * v + wz * wz, uF = u * Fx + v * Fy + wz * Fz;
        collide_pairs_fp64<FORCE>(L, f, r, u, v, wz, usq, uF, post);
    } else {
        using A = typename S::A;
        A dr, rho, u, v, wz, k15, uF, srho;
        shifted_moments<S>(L, f, dr, rho, u, v, wz);
        shifted_terms<S>(L, rho, u, v, wz, k15, uF, srho);
        post[0] = rest_post<S, FORCE>(L, (A)f[0], dr, srho, k15, uF);
#pragma unroll
        for (int i = 1; i < Q; i += 2)
            pair_post<S, FORCE>(L, i, (A)f[i], (A)f[i + 1], u, v, wz, dr, srho, k15, uF, post[i], post[i + 1]);
    }
    st_cluster<S>(own, post[0]);
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        const uint32_t local = own + (uint32_t)OPP(i) * dir_bytes, remote = slot(i);
        const bool solid = wall_dir(i, wr);
        st_cluster<S>((PAR == 0) == solid ? remote : local, post[i]);
    }
}

template <class S, bool FORCE>
__global__ void __launch_bounds__(CLUSTER_THREADS, 1) k_cluster_steps(const __grid_constant__ Lattice L, void* fv,
                                                                      const ClusterWork w) {
    using T = typename S::T;
    extern __shared__ __align__(16) unsigned char cluster_raw[];
    T* const sh = reinterpret_cast<T*>(cluster_raw);
    // address of the first node of the row at (cy, cz) from row r, for each row of this CTA
    uint32_t* const rowtab = reinterpret_cast<uint32_t*>(cluster_raw + (size_t)Q * w.stride * sizeof(T));   // [rows][9]
    T* const f = static_cast<T*>(fv);
    const int rank = (int)cluster_rank(), r0 = rank * w.rows, nrows = min(w.rows, L.ny * L.nz - r0);   // may be <= 0
    const int nodes = max(0, nrows) * L.nx;
    const size_t n0 = (size_t)r0 * L.nx;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sh), dir_bytes = (uint32_t)(w.stride * sizeof(T));
    for (int i = 0; i < Q; ++i)
        for (int l = threadIdx.x; l < nodes; l += CLUSTER_THREADS) sh[i * w.stride + l] = f[(size_t)i * L.N + n0 + l];
    for (int k = threadIdx.x; k < nrows * 9; k += CLUSTER_THREADS) {
        const int r = r0 + k / 9, c = k % 9;
        const int y = r % L.ny, z = r / L.ny;
        int yn = y + c % 3 - 1, zn = z + c / 3 - 1;
        yn += yn < 0 ? L.ny : (yn >= L.ny ? -L.ny : 0);
        zn += zn < 0 ? L.nz : (zn >= L.nz ? -L.nz : 0);
        const int rn = yn + L.ny * zn, to = rn / w.rows;
        rowtab[k] = cluster_addr(base + (uint32_t)((rn - to * w.rows) * L.nx * (int)sizeof(T)), to);
    }
    cluster_sync();
    // this thread's node, the same in every step
    const int l = threadIdx.x, row = l / L.nx, x = l - row * L.nx, z = (r0 + row) / L.ny, y = r0 + row - z * L.ny;
    const bool fluid = l < nodes && !((L.walls_y && (y == 0 || y == L.ny - 1)) || (L.walls_z && (z == 0 || z == L.nz - 1)));
    const uint8_t wr = wall_row(L, y, z);
    const uint32_t xb[3] = {(uint32_t)((x == 0 ? L.nx - 1 : x - 1) * (int)sizeof(T)), (uint32_t)(x * (int)sizeof(T)),
                            (uint32_t)((x == L.nx - 1 ? 0 : x + 1) * (int)sizeof(T))};
    uint32_t rows9[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) rows9[c] = fluid ? rowtab[row * 9 + c] : 0u;
    auto slot = [&](int i) { return rows9[(CZ(i) + 1) * 3 + CY(i) + 1] + xb[CX(i) + 1] + (uint32_t)i * dir_bytes; };
    const uint32_t own = rows9[4] + xb[1];   // the node's own slots, through the cluster window too
    int k = w.nsteps;
    if (w.parity & 1) {   // a first odd step
        if (fluid) cluster_node<S, 1, FORCE>(L, own, dir_bytes, wr, slot);
        cluster_sync();
        --k;
    }
    for (; k > 0; k -= 2) {
        if (fluid) cluster_node<S, 0, FORCE>(L, own, dir_bytes, wr, slot);
        cluster_sync();
        if (k == 1) break;
        if (fluid) cluster_node<S, 1, FORCE>(L, own, dir_bytes, wr, slot);
        cluster_sync();
    }
    for (int i = 0; i < Q; ++i)
        for (int l = threadIdx.x; l < nodes; l += CLUSTER_THREADS) f[(size_t)i * L.N + n0 + l] = sh[i * w.stride + l];
}

template <class S>
constexpr size_t cluster_smem(int rows, int stride) {
    return (size_t)Q * stride * sizeof(typename S::T) + (size_t)rows * 9 * sizeof(uint32_t);
}

}  // namespace lbmgpu
