// What the two staged collide-and-stream kernels share: the mbarrier and bulk-copy primitives, the
// stage layout, the collision and stores of one cell, and the collision constants of a launch.
#pragma once

#include <algorithm>
#include <cstring>
#include <mutex>
#include <unordered_map>

#include "lattice_common.cuh"

namespace bib {

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// One potentially blocking test of a barrier phase: a thread whose phase is not complete is
// suspended until it completes or about kSuspendNs pass (the suspend-time hint), so that waiting
// warps do not spin through issue slots the working warps need.
constexpr uint32_t kSuspendNs = 20000;
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait for one phase of a stage barrier: gives up after limit_ns (2 s by default; a
// copy of a tile takes microseconds) or 2^26 polls, so that a lost completion can never hang
// the GPU.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, uint64_t limit_ns = kDefaultWaitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0 && global_ns() - t0 > limit_ns) break;
    }
    return false;
}
// Shared -> global bulk copy, completed by the thread's bulk group; dst, src and bytes are multiples of 16.
__device__ __forceinline__ void bulk_copy_s2g(void* dst, const void* src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;" ::"l"(dst),
                 "r"(smem_addr(src)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// A consumer warp hands a stage that it has read into registers back to the producer, which refills it by bulk
// copies.  The copies belong to another proxy than the reads: without the fence of every reading thread the arrival
// orders nothing between the two, and reads that wait in the shared-memory pipe (behind the global loads of
// other warps' face cells) find the next tile's values.  Linear tiles of a 313 x 79 x 89 FP32 lattice: about one warp
// in 3 x 10^8 (one step in 5,000) read a population of the tile after next.
__device__ __forceinline__ void release_stage(uint64_t* empty, int lane) {
    proxy_fence();
    __syncwarp();
    if (lane == 0) mbar_arrive(empty);
}
// Global -> shared bulk copy; dst, src and bytes are multiples of 16.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Values of a staged population row as the compute type, in storage units (FP16 keeps the
// scaled f-bar; the scale is folded into the collision).
template <class T>
struct Staged;
template <>
struct Staged<__half> {
    static __device__ __forceinline__ float one(const __half* p) { return __half2float(*p); }
    static __device__ __forceinline__ void put(__half* p, float a) { *p = __float2half_rn(a); }
};
template <>
struct Staged<float> {
    static __device__ __forceinline__ float one(const float* p) { return *p; }
    static __device__ __forceinline__ void put(float* p, float a) { *p = a; }
};
template <>
struct Staged<double> {
    static __device__ __forceinline__ double one(const double* p) { return *p; }
    static __device__ __forceinline__ void put(double* p, double a) { *p = a; }
};

// The 19 post-collision values of one cell to their arrays (stride apart); FP16 converts two
// values per instruction (same rounding; measured on row tiles with one cell per thread, 400-cell channel:
// 0.1763 -> 0.1748 ms).
template <class T, class C>
__device__ __forceinline__ void store_cell(T* o, int64_t stride, const C* f) {
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        Staged<T>::put(o, f[i]);
        o += stride;
    }
}
template <>
__device__ __forceinline__ void store_cell<__half, float>(__half* o, int64_t stride, const float* f) {
#pragma unroll
    for (int i = 0; i + 1 < Q; i += 2) {
        const __half2 h = __floats2half2_rn(f[i], f[i + 1]);
        o[0] = __low2half(h);
        o[stride] = __high2half(h);
        o += 2 * stride;
    }
    *o = __float2half_rn(f[Q - 1]);
}

// Tile pitch in cells: the shared-memory row of one population holds up to TILE cells, so
// every staged address is a per-thread base plus a compile-time offset.
template <class T>
struct TileOf {
    static constexpr int value = sizeof(T) == 8 ? 256 : 512;
};

// Coupling of a staged launch: lattice only; dense (the velocity field with the previous force,
// which is read and reset to the body force); sparse (the velocity field with the body force,
// the previous force left to the sparse reset); reset (no velocity field, the previous force reset
// without being read).
constexpr int kCplNone = 0, kCplDense = 1, kCplSparse = 2, kCplReset = 3;
__host__ __device__ constexpr bool writes_u(int cpl) { return cpl == kCplDense || cpl == kCplSparse; }
__host__ __device__ constexpr bool resets(int cpl) { return cpl == kCplDense || cpl == kCplReset; }

// Stage layout (compile-time): 19 population rows, the collision force (BGK + Guo) and,
// for the dense coupled step, the previous force (three values per cell), each TILE cells long.
template <class T, int CPL, int COLL>
struct StageLayout {
    using FT = typename Store<T>::F;
    static constexpr int TILE = TileOf<T>::value;
    static constexpr int CELLS = sizeof(T) == 2 ? 2 : 1;  // per consumer thread and tile
    static constexpr int CONSUMERS = TILE / 32 / CELLS;   // consumer warps
    static constexpr int THREADS = 32 * (CONSUMERS + 1);
    static constexpr bool NEED_FCOL = COLL == BIB_COLLISION_BGK_GUO_VOF;
    static constexpr unsigned POP = TILE * sizeof(T);
    static constexpr unsigned FRC = TILE * sizeof(FT);
    static constexpr unsigned OFF_FCOL = Q * POP;
    static constexpr unsigned OFF_FPREV = OFF_FCOL + (NEED_FCOL ? 3 * FRC : 0);
    static constexpr unsigned BYTES = ((OFF_FPREV + (CPL == kCplDense ? 3 * FRC : 0)) + 127) / 128 * 128;
    // dense coupling: one tile of the body force in front of the stages, the source of the reset
    static constexpr unsigned RESET = resets(CPL) ? 3 * FRC : 0;
};

constexpr int kMaxStages = 8;

template <class FT>
__device__ __forceinline__ void fill_reset(FT* reset, const double* body, int n, int t, int nthreads) {
    for (int k = t; k < n; k += nthreads) reset[k] = (FT)body[k % 3];
    proxy_fence();
}

// Collision and stores of one cell k of row y whose gathered populations are in f: a
// BounceBack / NoDynamics node is not collided (zero velocity), every other node collides with
// the force F; the coupled step writes its velocity (j/rho + Fp/2, or the wall's on
// finite-difference wall rows).
template <class T, int CPL, int COLL>
__device__ __forceinline__ void finish_cell(const LatticeDesc& d, const CollideParams<typename Store<T>::C>& cp,
                                            T* __restrict__ fout, typename Store<T>::U* __restrict__ u_out, const uint8_t* __restrict__ phase,
                                            const uint8_t* __restrict__ celltype, int64_t k, int y, bool fd,
                                            typename Store<T>::C* f, const typename Store<T>::C* F,
                                            const typename Store<T>::C* Fp) {
    using C = typename Store<T>::C;
    using UT = typename Store<T>::U;
    constexpr bool UVEL = writes_u(CPL);
    const int ctype = d.has_types ? celltype[k] : BIB_CELL_FLUID;
    if (ctype != BIB_CELL_FLUID) {  // BounceBack / NoDynamics node: no collision, zero velocity
        if (UVEL) store_u<UT>(u_out, k, (UT)0.0f, (UT)0.0f, (UT)0.0f);
        if (ctype == BIB_CELL_BOUNCE_BACK) bounce_back_cell(f);
        store_cell<T, C>(fout + k, d.stride, f);
        return;
    }
    RelaxRates<C> r = cp.r[0];
    if (COLL == BIB_COLLISION_BGK_GUO_VOF && d.use_phase && phase[k]) r = cp.r[1];
    const CellMoments<C> m = moments_compact<C, sizeof(T) == 2>(f, cp.invS);
    if (UVEL) {
        // the velocity is stored before the relaxation, so that the previous force is dead while
        // the relaxation runs
        C u[3];
        if (fd) {
            const int side = y == 0 ? 0 : 1;
#pragma unroll
            for (int q = 0; q < 3; ++q) u[q] = cp.wall_u[side][q];
        } else {
            velocity_compact<C>(m, Fp, u);
        }
        store_u_from<UT, C>(u_out, k, u[0], u[1], u[2]);
    }
    relax_compact<C, COLL>(f, F, r, m);
    store_cell<T, C>(fout + k, d.stride, f);
}

// Resident CTAs per SM the kernels are built for: FP16 needs two (32 consumer warps; 16 of packed pairs) to hide
// the latency of its arithmetic; FP32 and FP64 run one CTA with a deeper pipeline.
template <class T>
constexpr int staged_ctas_per_sm() {
    return sizeof(T) == 2 ? 2 : 1;
}

inline int optin_smem() {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return optin;
}

template <class C>
CollideParams<C> collide_params(const LatticeDesc& d, int storage) {
    CollideParams<C> cp{};
    const double S = storage == BIB_STORAGE_F16 ? (double)d.scale : 1.0;
    const C omm = (C)(1.0 / (d.trt_magic / (1.0 / d.omega - 0.5) + 0.5));
    if (d.collision == BIB_COLLISION_BGK_GUO_VOF) {
        cp.r[0] = relax_rates<C, BIB_COLLISION_BGK_GUO_VOF>((C)d.omega_c0, C(0), (C)S);
        cp.r[1] = relax_rates<C, BIB_COLLISION_BGK_GUO_VOF>((C)d.omega_c1, C(0), (C)S);
    } else if (d.collision == BIB_COLLISION_TRT) {
        cp.r[0] = cp.r[1] = relax_rates<C, BIB_COLLISION_TRT>((C)d.omega, omm, (C)S);
    } else {
        cp.r[0] = cp.r[1] = relax_rates<C, BIB_COLLISION_BGK>((C)d.omega, C(0), (C)S);
    }
    cp.invS = (C)(storage == BIB_STORAGE_F16 ? (double)d.inv_scale : 1.0);
    for (int q = 0; q < 3; ++q) {
        cp.body[q] = (C)d.body[q];
        cp.wall_u[0][q] = (C)d.wall_u[0][q];
        cp.wall_u[1][q] = (C)d.wall_u[1][q];
    }
    for (int face = 0; face < 4; ++face)
        for (int i = 0; i < Q; ++i) {
            const double cu = cx(i) * d.wall_u[face][0] + cy(i) * d.wall_u[face][1] + cz(i) * d.wall_u[face][2];
            cp.mw[face][i] = (C)((C)(6.0 * weight<double>(i) * cu) * (C)S);
        }
    return cp;
}

}  // namespace

}  // namespace bib
