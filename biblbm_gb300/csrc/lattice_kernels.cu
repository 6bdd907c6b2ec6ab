// Lattice kernels: fused pull collide-and-stream (+ velocity field), finite-difference
// velocity walls, state import / export and equilibrium initialisation.
//
// Data layout in HBM: one array per population (structure of arrays), x fastest,
// cell k = x + nx*(y + ny*z), population i at f[i*stride + k].  The buffers hold
// post-collision populations f*(x); the post-streaming state (the reference's state
// between steps) is gathered: f_i(x) = f*_i(x - c_i), periodic by index wrap, halfway
// bounce-back f_i(x) = f*_opp(i)(x) + 6 t_i (c_i . u_wall) where x - c_i lies behind a
// wall, and the nodes of finite-difference velocity walls read a separate wall buffer.
#include <algorithm>

#include "lattice_common.cuh"

namespace bib {

namespace {

// Post-streaming populations of one cell.
template <class T>
__device__ __forceinline__ void gather(const LatticeDesc& d, const T* __restrict__ f, const T* __restrict__ wall, int x,
                                       int y, int z, int64_t k, typename Store<T>::C* out) {
    using C = typename Store<T>::C;
    if (fd_wall_node(d, y)) {
        const int64_t wk = wall_index(d, y == 0 ? 0 : 1, x, z), ws = wall_stride(d);
#pragma unroll
        for (int i = 0; i < Q; ++i) out[i] = Store<T>::load(wall + i * ws + wk, d.inv_scale);
        return;
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        int face;
        const int64_t s = source_cell(d, i, x, y, z, face);
        if (s >= 0) out[i] = Store<T>::load(f + i * d.stride + s, d.inv_scale);
        else out[i] = Store<T>::load(f + opposite(i) * d.stride + k, d.inv_scale) + moving_wall_term<C>(d, i, face);
    }
}

// Inverse of gather for a single population: where the value f_i(x) of a post-streaming
// state has to be stored so that the next gather returns it.
template <class T>
__device__ __forceinline__ void scatter_canonical(const LatticeDesc& d, T* __restrict__ f, T* __restrict__ wall, int i, int x,
                                                  int y, int z, int64_t k, typename Store<T>::C v) {
    using C = typename Store<T>::C;
    if (fd_wall_node(d, y)) {
        Store<T>::store(wall + i * wall_stride(d) + wall_index(d, y == 0 ? 0 : 1, x, z), v, d.scale);
        return;
    }
    int face;
    const int64_t s = source_cell(d, i, x, y, z, face);
    if (s >= 0) Store<T>::store(f + i * d.stride + s, v, d.scale);
    else Store<T>::store(f + opposite(i) * d.stride + k, v - moving_wall_term<C>(d, i, face), d.scale);
}

template <class T, bool COUPLED>
__global__ void __launch_bounds__(256) k_collide_stream(LatticeDesc d, const T* __restrict__ fin, T* __restrict__ fout,
                                                         const T* __restrict__ wall,
                                                         const typename Store<T>::F* __restrict__ Fcol,
                                                         typename Store<T>::F* __restrict__ Fprev,
                                                         typename Store<T>::U* __restrict__ u_out,
                                                         const uint8_t* __restrict__ phase,
                                                         const uint8_t* __restrict__ celltype, int coll) {
    using C = typename Store<T>::C;
    using FT = typename Store<T>::F;
    using UT = typename Store<T>::U;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = blockIdx.z;
    if (x >= d.nx) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    C f[Q];
    gather<T>(d, fin, wall, x, y, z, k, f);
    const int ctype = d.has_types ? celltype[k] : BIB_CELL_FLUID;
    if (ctype != BIB_CELL_FLUID) {  // BounceBack / NoDynamics node: no collision, zero velocity
        if (COUPLED) {
            if (u_out) store_u<UT>(u_out, k, (UT)0.0f, (UT)0.0f, (UT)0.0f);
            if (Fprev)
                for (int c = 0; c < 3; ++c) Fprev[3 * k + c] = (FT)d.body[c];
        }
        if (ctype == BIB_CELL_BOUNCE_BACK) bounce_back_cell(f);
#pragma unroll
        for (int i = 0; i < Q; ++i) Store<T>::store(fout + i * d.stride + k, f[i], d.scale);
        return;
    }
    if (COUPLED) {
        // computeVelocity of the current state (externalForceDynamics.hh:59-74; the wall
        // nodes give their imposed velocity, boundaryDynamics.hh:316-322), with the force of
        // the previous collision; that force buffer is then reset to the body force so the
        // next step can spread into it (setExternalVector).  Without Fprev (sparse force
        // reset) the velocity takes the body force and the interpolation adds the rest.
        if (u_out) {
            C u[3];
            if (fd_wall_node(d, y)) {
                const int side = y == 0 ? 0 : 1;
                u[0] = (C)d.wall_u[side][0];
                u[1] = (C)d.wall_u[side][1];
                u[2] = (C)d.wall_u[side][2];
            } else {
                C Fp[3] = {(C)d.body[0], (C)d.body[1], (C)d.body[2]};
                if (Fprev) {
                    for (int c = 0; c < 3; ++c) Fp[c] = (C)Fprev[3 * k + c];
                }
                velocity_with_force(f, Fp, u);
            }
            store_u<UT>(u_out, k, (UT)u[0], (UT)u[1], (UT)u[2]);
        }
        if (Fprev) {
            for (int c = 0; c < 3; ++c) Fprev[3 * k + c] = (FT)d.body[c];
        }
    }
    C Fc[3] = {(C)__ldg(Fcol + 3 * k), (C)__ldg(Fcol + 3 * k + 1), (C)__ldg(Fcol + 3 * k + 2)};
    if (coll == BIB_COLLISION_BGK_GUO_VOF) {
        C omega = (C)d.omega_c0;
        if (d.use_phase && phase[k]) omega = (C)d.omega_c1;
        collide_unscaled<C, BIB_COLLISION_BGK_GUO_VOF>(f, Fc, omega, C(0));
    } else if (coll == BIB_COLLISION_BGK) {
        collide_unscaled<C, BIB_COLLISION_BGK>(f, Fc, (C)d.omega, C(0));
    } else {
        const C om = (C)d.omega;
        const C omm = C(1) / ((C)d.trt_magic / (C(1) / om - C(0.5)) + C(0.5));
        collide_unscaled<C, BIB_COLLISION_TRT>(f, Fc, om, omm);
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) Store<T>::store(fout + i * d.stride + k, f[i], d.scale);
}

// ---------------------------------------------------------------------------------------
// Row-vectorised pull collide-and-stream (nx even).  A warp covers 64 consecutive cells of
// one x-row, two per thread: every population is read as an aligned pair (half2 / float2 /
// double2) from its source row, and the +-1 shift along x of the populations with
// c_x != 0 is done with one warp shuffle (the lanes at the warp's ends fetch the missing
// neighbour with a scalar load, wrapping periodically at the row ends).  The nine source
// rows (y - c_y, z - c_z) are resolved once per thread.
template <class T, bool COUPLED>
__global__ void __launch_bounds__(256) k_collide_stream_rows(LatticeDesc d, const T* __restrict__ fin, T* __restrict__ fout,
                                                              const T* __restrict__ wall,
                                                              const typename Store<T>::F* __restrict__ Fcol,
                                                              typename Store<T>::F* __restrict__ Fprev,
                                                              typename Store<T>::U* __restrict__ u_out,
                                                              const uint8_t* __restrict__ phase,
                                                              const uint8_t* __restrict__ celltype, int coll) {
    using C = typename Store<T>::C;
    using FT = typename Store<T>::F;
    using UT = typename Store<T>::U;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // grid.x runs over blocks of rows (ny * nz can exceed the 65535 limit of grid.y)
    const int tx = blockIdx.y * blockDim.x + threadIdx.x;
    const int row = blockIdx.x * blockDim.y + threadIdx.y;
    if (row >= d.ny * d.nz) return;  // uniform per warp: a warp never spans two rows
    const int y = row % d.ny, z = row / d.ny;
    const int x0 = 2 * tx;
    const bool active = x0 < d.nx;
    const int64_t k0 = (int64_t)row * d.nx + x0;
    const bool wallrow = fd_wall_node(d, y);
    // ---- phase 1: issue every load of the cell pair before any shuffle or arithmetic, so
    // that all of them are in flight together (the shuffles would otherwise serialise them)
    C pa[Q], pb[Q], edge[Q];
    FT fpa[3], fpb[3], fca[3], fcb[3];
    int sface[3][3];
    if (wallrow) {
        const int64_t ws = wall_stride(d), wk = wall_index(d, y == 0 ? 0 : 1, active ? x0 : 0, z);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            pa[i] = pb[i] = edge[i] = C(0);
            if (active) Pair<T>::load(wall + i * ws + wk, d.inv_scale, pa[i], pb[i]);
        }
    } else {
        int64_t srow[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                int ys = y - (a - 1), zs = z - (b - 1), face = -1;
                if (d.py) ys = (int)wrap_index(ys, d.ny);
                else if (ys < 0 || ys >= d.ny) face = ys < 0 ? 0 : 1;
                if (d.pz) zs = (int)wrap_index(zs, d.nz);
                else if (face < 0 && (zs < 0 || zs >= d.nz)) face = zs < 0 ? 2 : 3;
                sface[a][b] = face;
                srow[a][b] = face >= 0 ? -1 : ((int64_t)ys + (int64_t)d.ny * zs) * d.nx;
            }
        const int xl = x0 == 0 ? d.nx - 1 : x0 - 1;            // left neighbour of the pair
        const int xr = x0 + 2 >= d.nx ? x0 + 2 - d.nx : x0 + 2; // right neighbour of the pair
        const bool need_l = active && lane == 0;
        const bool need_r = active && (lane == 31 || x0 + 2 >= d.nx);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int a = cy(i) + 1, b = cz(i) + 1;
            pa[i] = pb[i] = edge[i] = C(0);
            if (srow[a][b] < 0) {
                // halfway bounce-back: the own node's opposite population, no shift in x
                if (active) Pair<T>::load(fin + opposite(i) * d.stride + k0, d.inv_scale, pa[i], pb[i]);
                continue;
            }
            const T* src = fin + i * d.stride + srow[a][b];
            if (active) Pair<T>::load(src + x0, d.inv_scale, pa[i], pb[i]);
            if (cx(i) == 1 && need_l) edge[i] = Store<T>::load(src + xl, d.inv_scale);
            if (cx(i) == -1 && need_r) edge[i] = Store<T>::load(src + xr, d.inv_scale);
        }
    }
    if (active) {
        load_force2<FT>(Fcol, k0, fca, fcb);
        if (COUPLED && !wallrow && u_out) {
            if (Fprev) {
                load_force2<FT>(Fprev, k0, fpa, fpb);
            } else {  // sparse force reset: the velocity field takes the body force only
                for (int c = 0; c < 3; ++c) fpa[c] = fpb[c] = (FT)d.body[c];
            }
        }
    }
    // ---- phase 2: assemble the gathered populations (x shifts through the warp)
    C f0[Q], f1[Q];
    if (wallrow) {
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            f0[i] = pa[i];
            f1[i] = pb[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int a = cy(i) + 1, b = cz(i) + 1;
            if (sface[a][b] >= 0) {
                const C mw = moving_wall_term<C>(d, i, sface[a][b]);
                f0[i] = pa[i] + mw;
                f1[i] = pb[i] + mw;
            } else if (cx(i) == 0) {
                f0[i] = pa[i];
                f1[i] = pb[i];
            } else if (cx(i) == 1) {  // src[x0 - 1], src[x0]
                const C left = __shfl_up_sync(FULL, pb[i], 1);
                f0[i] = lane == 0 ? edge[i] : left;
                f1[i] = pa[i];
            } else {  // src[x0 + 1], src[x0 + 2]
                const C right = __shfl_down_sync(FULL, pa[i], 1);
                f0[i] = pb[i];
                f1[i] = (lane == 31 || x0 + 2 >= d.nx) ? edge[i] : right;
            }
        }
    }
    if (!active) return;
    int ct0 = BIB_CELL_FLUID, ct1 = BIB_CELL_FLUID;
    if (d.has_types) {
        ct0 = celltype[k0];
        ct1 = celltype[k0 + 1];
    }
    if (COUPLED) {
        if (u_out) {
            C u0[3], u1[3];
            if (wallrow) {
                const int side = y == 0 ? 0 : 1;
                for (int c = 0; c < 3; ++c) u0[c] = u1[c] = (C)d.wall_u[side][c];
            } else {
                C Fa[3] = {(C)fpa[0], (C)fpa[1], (C)fpa[2]}, Fb[3] = {(C)fpb[0], (C)fpb[1], (C)fpb[2]};
                velocity_with_force(f0, Fa, u0);
                velocity_with_force(f1, Fb, u1);
            }
            if (ct0 != BIB_CELL_FLUID) u0[0] = u0[1] = u0[2] = C(0);
            if (ct1 != BIB_CELL_FLUID) u1[0] = u1[1] = u1[2] = C(0);
            store_u<UT>(u_out, k0, (UT)u0[0], (UT)u0[1], (UT)u0[2]);
            store_u<UT>(u_out, k0 + 1, (UT)u1[0], (UT)u1[1], (UT)u1[2]);
        }
        if (Fprev)
            store_force2<FT>(Fprev, k0, d.body);
    }
    C Fa[3] = {(C)fca[0], (C)fca[1], (C)fca[2]}, Fb[3] = {(C)fcb[0], (C)fcb[1], (C)fcb[2]};
    C om0 = (C)d.omega, om1 = (C)d.omega, omm = C(0);
    if (coll == BIB_COLLISION_BGK_GUO_VOF) {
        om0 = om1 = (C)d.omega_c0;
        if (d.use_phase) {
            if (phase[k0]) om0 = (C)d.omega_c1;
            if (phase[k0 + 1]) om1 = (C)d.omega_c1;
        }
    } else if (coll == BIB_COLLISION_TRT) {
        omm = C(1) / ((C)d.trt_magic / (C(1) / om0 - C(0.5)) + C(0.5));
    }
    auto collide_one = [&](C* f, const C* Fx, C om) {
        if (coll == BIB_COLLISION_BGK_GUO_VOF) collide_unscaled<C, BIB_COLLISION_BGK_GUO_VOF>(f, Fx, om, C(0));
        else if (coll == BIB_COLLISION_BGK) collide_unscaled<C, BIB_COLLISION_BGK>(f, Fx, om, C(0));
        else collide_unscaled<C, BIB_COLLISION_TRT>(f, Fx, om, omm);
    };
    // BounceBack nodes swap their incoming populations, NoDynamics nodes keep them
    if (ct0 == BIB_CELL_FLUID) collide_one(f0, Fa, om0);
    else if (ct0 == BIB_CELL_BOUNCE_BACK) bounce_back_cell(f0);
    if (ct1 == BIB_CELL_FLUID) collide_one(f1, Fb, om1);
    else if (ct1 == BIB_CELL_BOUNCE_BACK) bounce_back_cell(f1);
#pragma unroll
    for (int i = 0; i < Q; ++i) Pair<T>::store(fout + i * d.stride + k0, f0[i], f1[i], d.scale);
}

// PlaneFdBoundaryFunctional3D::processCell on the y walls after collide-and-stream,
// src/boundaryCondition/finiteDifferenceBoundaryProcessor3D.hh:68-115: density from the
// known populations (VelocityDirichletBoundaryDynamics::computeRhoBar,
// boundaryDynamics.hh:631-663), one-sided normal velocity derivative
// (finiteDifference3D.h:67-82; tangential derivatives vanish for a uniform wall
// velocity), regularised reconstruction of all 19 populations into the wall buffer.
template <class T>
__device__ __forceinline__ void fd_wall_cell(const LatticeDesc& d, const T* __restrict__ f, T* __restrict__ wall,
                                             const typename Store<T>::F* __restrict__ F, int x, int z, int side);

// GuoRigidWallBoundaryFunctional::process with depth 2 (fsi/GuoBoundaryCondition.hh:133-187),
// one thread per wall node after collide-and-stream: the post-streaming states of the two fluid
// nodes along the node's lattice vector give density, momentum and non-equilibrium parts; the
// node's new state, the equilibrium of the extrapolated wall momentum (0 for a NoDynamics node)
// plus the extrapolated non-equilibrium part, is scattered into the post-collision slots it
// gathers from.  Each slot f*_i(x) is read by the node x + c_i alone, and no wall node's fluid
// nodes are wall nodes (checked on the host), so the threads never touch each other's data.
template <class T>
__global__ void __launch_bounds__(128) k_guo_walls(LatticeDesc d, T* __restrict__ f, const T* __restrict__ wall,
                                                    const GuoNode* __restrict__ nodes, int n) {
    using C = typename Store<T>::C;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const GuoNode w = nodes[g];
    C fc[2][Q], rb[2], j[2][3], fneq[2][Q];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int xs = (int)wrap_index(w.x + (m + 1) * cx(w.dir), d.nx);
        const int ys = (int)wrap_index(w.y + (m + 1) * cy(w.dir), d.ny);
        const int zs = (int)wrap_index(w.z + (m + 1) * cz(w.dir), d.nz);
        gather<T>(d, f, wall, xs, ys, zs, xs + (int64_t)d.nx * (ys + (int64_t)d.ny * zs), fc[m]);
        rho_bar_j<C>(fc[m], rb[m], j[m]);
        const C jsq = j[m][0] * j[m][0] + j[m][1] * j[m][1] + j[m][2] * j[m][2];
        const C invRho = C(1) / (rb[m] + C(1));
#pragma unroll
        for (int i = 0; i < Q; ++i) fneq[m][i] = fc[m][i] - bgk_equilibrium<C>(i, rb[m], invRho, j[m], jsq);
    }
    const C rbw = rb[0], dl = (C)w.delta;
    C wj[3], jw[3], fw[Q];
    for (int c = 0; c < 3; ++c) wj[c] = (rbw + C(1)) * (C)w.u[c];
    if (dl < C(0.75)) {
        for (int c = 0; c < 3; ++c)
            jw[c] = wj[c] + (dl - C(1)) * j[0][c] + (C(1) - dl) / (C(1) + dl) * (C(2) * wj[c] + (dl - C(1)) * j[1][c]);
#pragma unroll
        for (int i = 0; i < Q; ++i) fw[i] = dl * fneq[0][i] + (C(1) - dl) * fneq[1][i];
    } else {
        for (int c = 0; c < 3; ++c) jw[c] = C(1) / dl * (wj[c] + (dl - C(1)) * j[0][c]);
#pragma unroll
        for (int i = 0; i < Q; ++i) fw[i] = fneq[0][i];
    }
    const C jsq = jw[0] * jw[0] + jw[1] * jw[1] + jw[2] * jw[2];
    const C invRho = C(1) / (rbw + C(1));
    const int64_t k = w.x + (int64_t)d.nx * (w.y + (int64_t)d.ny * w.z);
#pragma unroll
    for (int i = 0; i < Q; ++i)
        scatter_canonical<T>(d, f, const_cast<T*>(wall), i, w.x, w.y, w.z, k,
                             (w.nodyn ? C(0) : bgk_equilibrium<C>(i, rbw, invRho, jw, jsq)) + fw[i]);
}

// grid: blocks of wall nodes, two sides
constexpr int kWallBlock = 64;
template <class T>
__global__ void __launch_bounds__(kWallBlock) k_fd_walls(LatticeDesc d, const T* __restrict__ f, T* __restrict__ wall,
                                                         const typename Store<T>::F* __restrict__ F) {
    const uint32_t t = blockIdx.x * kWallBlock + threadIdx.x, nx = (uint32_t)d.nx;
    if (t >= nx * (uint32_t)d.nz) return;
    fd_wall_cell<T>(d, f, wall, F, (int)(t % nx), (int)(t / nx), blockIdx.y);
}

// Batched: grid.z = lattices; each lattice's view of the state after the swap.
template <class T>
__global__ void __launch_bounds__(kWallBlock) k_fd_walls_batch(const CollideView* __restrict__ views) {
    const CollideView& V = views[blockIdx.z];
    const uint32_t t = blockIdx.x * kWallBlock + threadIdx.x, nx = (uint32_t)V.d.nx;
    if (!V.d.fd_walls || t >= nx * (uint32_t)V.d.nz) return;
    fd_wall_cell<T>(V.d, static_cast<const T*>(V.fin), static_cast<T*>(const_cast<void*>(V.wall)),
                    static_cast<const typename Store<T>::F*>(V.Fprev), (int)(t % nx), (int)(t / nx), blockIdx.y);
}

// With a uniform wall velocity the stress has three entries (xy, yy, yz), and a wall row and its
// neighbour gather from rows inside the domain (three rows at least, periodic x and z).  One thread per
// wall node; bound by latency, in FP64 by the FP64 pipe: with all six entries, multiplications by zero
// lattice components and the general gather 18.1 us (64 x 64 nodes on two sides, FP64; 8.6 us FP32 128 x 64),
// now 11.4 and 5.0; 64 lattices in one launch 68 -> 25 us, whose rows of 32 to 96 nodes left lanes idle.
template <class T, int SIDE>
__device__ __forceinline__ void fd_wall_node_rebuild(const LatticeDesc& d, const T* __restrict__ f, T* __restrict__ wall,
                                                     const typename Store<T>::F* __restrict__ F, int x, int z) {
    using C = typename Store<T>::C;
    constexpr int O = SIDE == 0 ? -1 : 1;  // outward normal
    const int y = SIDE == 0 ? 0 : d.ny - 1, y1 = y - O;
    const int64_t plane = (int64_t)d.nx * d.ny;
    // source offsets along x and z of c = -1, 0, 1
    const int xo[3] = {x + 1 == d.nx ? 0 : x + 1, x, x == 0 ? d.nx - 1 : x - 1};
    const int64_t zo[3] = {(z + 1 == d.nz ? 0 : z + 1) * plane, z * plane, (z == 0 ? d.nz - 1 : z - 1) * plane};
    C fc[Q], f1[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const T* p = f + i * d.stride + xo[cx(i) + 1] + zo[cz(i) + 1];
        f1[i] = Store<T>::load(p + (int64_t)d.nx * (y1 - cy(i)), d.inv_scale);
        fc[i] = cy(i) == -O ? C(0) : Store<T>::load(p + (int64_t)d.nx * (y - cy(i)), d.inv_scale);  // unknown ones are not used
    }
    const int64_t k = x + (int64_t)d.nx * y + z * plane, k1 = x + (int64_t)d.nx * y1 + z * plane;
    const C Fy = (C)F[3 * k + 1];
    C F1[3] = {(C)F[3 * k1], (C)F[3 * k1 + 1], (C)F[3 * k1 + 2]};
    const C uw[3] = {(C)d.wall_u[SIDE][0], (C)d.wall_u[SIDE][1], (C)d.wall_u[SIDE][2]};
    C rhoOnWall = 0, rhoNormal = 0;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if (cy(i) == 0) rhoOnWall += fc[i];
        if (cy(i) == O) rhoNormal += fc[i];
    }
    const C velNormal = C(O) * (uw[1] - C(0.5) * Fy);
    const C rhoBarW = (C(2) * rhoNormal + rhoOnWall - velNormal) / (C(1) + velNormal);
    const C rho = rhoBarW + C(1);
    C u1[3];
    velocity_with_force(f1, F1, u1);
    // one-sided normal derivative of the velocity times -rho / (3 omega), fromPiToFneq
    // (src/latticeBoltzmann/offEquilibriumTemplates.h:91-115) times 4.5 and the multiplicities
    const C sToPi = -rho / C(3) / (C)d.omega;
    const C pxy = C(9) * C(-O) * (u1[0] - uw[0]) * sToPi, pyy = C(9) * C(-O) * (u1[1] - uw[1]) * sToPi,
            pyz = C(9) * C(-O) * (u1[2] - uw[2]) * sToPi;
    const C j[3] = {rho * uw[0], rho * uw[1], rho * uw[2]};
    const C rhoBar = rho - C(1), invRho = C(1) / rho;
    // bgk_equilibrium (d3q19.cuh) with the terms of a pair gathered
    const C base = rhoBar - C(1.5) * invRho * (j[0] * j[0] + j[1] * j[1] + j[2] * j[2]);
    const C h = C(4.5) * invRho, third = pyy * (C(1) / C(3));
    const int64_t wk = wall_index(d, SIDE, x, z), ws = wall_stride(d);
    Store<T>::store(wall + wk, weight<C>(0) * (base - third), d.scale);
#pragma unroll
    for (int i = 1; i < 10; ++i) {
        const C cj = cdot<C>(i + 9, j[0], j[1], j[2]);
        C even = fmac(h * cj, cj, base) - third;
        if (cy(i) != 0) {
            even += pyy;
            if (cx(i) != 0) even += C(cx(i) * cy(i)) * pxy;
            if (cz(i) != 0) even += C(cy(i) * cz(i)) * pyz;
        }
        Store<T>::store(wall + i * ws + wk, weight<C>(i) * fmac(C(-3), cj, even), d.scale);
        Store<T>::store(wall + (i + 9) * ws + wk, weight<C>(i) * fmac(C(3), cj, even), d.scale);
    }
}
template <class T>
__device__ __forceinline__ void fd_wall_cell(const LatticeDesc& d, const T* __restrict__ f, T* __restrict__ wall,
                                             const typename Store<T>::F* __restrict__ F, int x, int z, int side) {
    if (side == 0) fd_wall_node_rebuild<T, 0>(d, f, wall, F, x, z);
    else fd_wall_node_rebuild<T, 1>(d, f, wall, F, x, z);
}

// computeVelocity of one cell of the current state with the current external force F (wall nodes give
// the wall velocity, BounceBack / NoDynamics nodes zero).
template <class T>
__device__ __forceinline__ void cell_velocity(const LatticeDesc& d, const T* __restrict__ f, const T* __restrict__ wall,
                                              const typename Store<T>::F* __restrict__ F,
                                              const uint8_t* __restrict__ celltype, int x, int y, int z, int64_t k,
                                              typename Store<T>::C* uc) {
    using C = typename Store<T>::C;
    if (d.has_types && celltype[k] != BIB_CELL_FLUID) {
        uc[0] = uc[1] = uc[2] = C(0);
    } else if (fd_wall_node(d, y)) {
        const int side = y == 0 ? 0 : 1;
        for (int a = 0; a < 3; ++a) uc[a] = (C)d.wall_u[side][a];
    } else {
        C fc[Q];
        gather<T>(d, f, wall, x, y, z, k, fc);
        C Fc[3] = {(C)F[3 * k], (C)F[3 * k + 1], (C)F[3 * k + 2]};
        velocity_with_force(fc, Fc, uc);
    }
}

// The velocity of every cell; OT = double for the host export, the field's storage type otherwise.
template <class T, class OT>
__global__ void k_velocity(LatticeDesc d, const T* __restrict__ f, const T* __restrict__ wall,
                           const typename Store<T>::F* __restrict__ F, OT* __restrict__ u, int64_t cstride,
                           int64_t kstride, const uint8_t* __restrict__ celltype) {
    using C = typename Store<T>::C;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = blockIdx.z;
    if (x >= d.nx) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    C uc[3];
    cell_velocity<T>(d, f, wall, F, celltype, x, y, z, k, uc);
    for (int a = 0; a < 3; ++a) u[a * cstride + k * kstride] = (OT)uc[a];
    if (kstride == 4) u[k * 4 + 3] = OT(0.0f);
}

// The velocity field at the support nodes of the vertices only, one thread per (vertex, node), the
// nodes of a vertex in x order: what the interpolation reads.  Nodes shared by several vertices are
// written several times with the same value.
template <class T, int S>
__global__ void __launch_bounds__(128) k_velocity_support(LatticeDesc d, IbDesc ib, int64_t nthreads,
                                                           const double* __restrict__ pos, const T* __restrict__ f,
                                                           const T* __restrict__ wall,
                                                           const typename Store<T>::F* __restrict__ F,
                                                           typename Store<T>::U* __restrict__ u,
                                                           const uint8_t* __restrict__ celltype) {
    using C = typename Store<T>::C;
    using UT = typename Store<T>::U;
    constexpr double h = S == 4 ? 2.0 : 1.5;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nthreads) return;
    const int64_t v = t / (S * S * S);
    const int m = (int)(t - v * (S * S * S));
    const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
    if (!inside_envelope(d, ib.dirac, p)) return;
    const int off = (int)ib.offset;
    const int x = remap_global(d.px, d.nx, (int64_t)ceil(p[0] - ib.offset - h) + m % S, off);
    const int y = remap_global(d.py, d.ny, (int64_t)ceil(p[1] - ib.offset - h) + (m / S) % S, off);
    const int z = remap_global(d.pz, d.nz, (int64_t)ceil(p[2] - ib.offset - h) + m / (S * S), off);
    if (x < 0 || y < 0 || z < 0) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    C uc[3];
    cell_velocity<T>(d, f, wall, F, celltype, x, y, z, k, uc);
    store_u<UT>(u, k, (UT)uc[0], (UT)uc[1], (UT)uc[2]);
}

// iniCellAtEquilibrium, src/core/cell.hh:124-132, in the storage's compute type (FP64 for FP64
// storage; FP32 otherwise: the FP64 pipe of this part would make the 19 equilibria per cell
// slower than reading the host velocity field over the CPU-GPU link).
template <class T>
__global__ void k_init_eq(LatticeDesc d, T* __restrict__ f, T* __restrict__ wall, const double* __restrict__ rho,
                          const double* __restrict__ u) {
    using C = typename Store<T>::C;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = blockIdx.z;
    if (x >= d.nx) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    const double r = rho ? rho[k] : 1.0;
    const C j[3] = {(C)(u[k] * r), (C)(u[d.n + k] * r), (C)(u[2 * d.n + k] * r)};
    const C jSqr = j[0] * j[0] + j[1] * j[1] + j[2] * j[2];
    const double rb = r - 1.0;
    const C rhoBar = (C)rb, invRho = (C)(1.0 / (rb + 1.0));
#pragma unroll
    for (int i = 0; i < Q; ++i) scatter_canonical<T>(d, f, wall, i, x, y, z, k, bgk_equilibrium<C>(i, rhoBar, invRho, j, jSqr));
}

// Import / export of the planes z0 .. z0 + gridDim.z - 1 from / to a buffer holding, per
// population, `pitch` cells that start with the first cell of plane z0.
template <class T>
__global__ void k_import(LatticeDesc d, T* __restrict__ f, T* __restrict__ wall, const double* __restrict__ src, int z0,
                         int64_t pitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = z0 + (int)blockIdx.z;
    if (x >= d.nx) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    const int64_t j = k - (int64_t)z0 * d.nx * d.ny;
#pragma unroll
    for (int i = 0; i < Q; ++i) scatter_canonical<T>(d, f, wall, i, x, y, z, k, src[i * pitch + j]);
}

template <class T>
__global__ void k_export(LatticeDesc d, const T* __restrict__ f, const T* __restrict__ wall, double* __restrict__ dst,
                         int z0, int64_t pitch) {
    using C = typename Store<T>::C;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y, z = z0 + (int)blockIdx.z;
    if (x >= d.nx) return;
    const int64_t k = x + (int64_t)d.nx * (y + (int64_t)d.ny * z);
    const int64_t j = k - (int64_t)z0 * d.nx * d.ny;
    C fc[Q];
    gather<T>(d, f, wall, x, y, z, k, fc);
    for (int i = 0; i < Q; ++i) dst[i * pitch + j] = (double)fc[i];
}

// Import / export of the x-planes x0 .. x0 + nxc - 1 of the cell-major wire order of Palabos
// (BlockLattice3D static content, blockLattice3D.hh:644-689: x slowest, z fastest; PER = 23
// doubles per cell: 19 f-bar, the force, the phase) and of CoProcessor3D (coProcessor3D.h:84-91:
// the same order, PER = 19 populations only).  `src` / `dst` hold cell (x0, 0, 0) first.
//
// Bound by the CPU-GPU link where the buffer is page-locked host memory.  A CTA moves the 8 x 32
// cells (x, z) of one y through shared memory: on the wire side a warp takes the 32 cells of one
// x, one contiguous run of 32 * PER doubles, 256 bytes per request; on the lattice side
// neighbouring lanes hold neighbouring x, so a population's sectors are written whole.  One thread
// per record straight from the buffer needed 32 sectors of the link per request: 128 x 96 x 80 cells
// of FP64 took 3.95 ms in and 6.15 ms out, 38 and 24 GB/s; send, one step and receive of that lattice
// went from 9.71 to 1.78 ms.
constexpr int kWireX = 8, kWireZ = 32;
// doubles of one x in shared memory: 2 more than its cells (a multiple of 16), so that the 8 x by 2 z
// lanes of a half warp read 16 different banks (19 and 23 are odd)
template <int PER>
__host__ __device__ constexpr int wire_pitch() {
    return kWireZ * PER + 2;
}
struct WireTile {
    int x0, y, z0, nxt, nzt;  // first cell, cells along x and z
};
__device__ __forceinline__ WireTile wire_tile(const LatticeDesc& d, int x0, int nxc) {
    WireTile t;
    t.x0 = x0 + (int)blockIdx.x * kWireX;
    t.y = blockIdx.y;
    t.z0 = (int)blockIdx.z * kWireZ;
    t.nxt = min(kWireX, x0 + nxc - t.x0);
    t.nzt = min(kWireZ, d.nz - t.z0);
    return t;
}

template <class T, int PER>
__global__ void __launch_bounds__(kWireX * kWireZ) k_import_aos(LatticeDesc d, T* __restrict__ f, T* __restrict__ wall,
                                                                typename Store<T>::F* __restrict__ F,
                                                                uint8_t* __restrict__ phase,
                                                                const double* __restrict__ src, int x0, int nxc) {
    __shared__ double sm[kWireX * wire_pitch<PER>()];
    const WireTile t = wire_tile(d, x0, nxc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < t.nxt) {
        const double* s = src + (int64_t)PER * (t.z0 + (int64_t)d.nz * (t.y + (int64_t)d.ny * (t.x0 - x0 + warp)));
        double* o = sm + warp * wire_pitch<PER>();
        const int n = PER * t.nzt;
        double v[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) v[k] = lane + 32 * k < n ? __ldg(s + lane + 32 * k) : 0.0;
#pragma unroll
        for (int k = 0; k < PER; ++k) o[lane + 32 * k] = v[k];
    }
    __syncthreads();
    const int xi = threadIdx.x & (kWireX - 1), zi = threadIdx.x / kWireX;
    if (xi >= t.nxt || zi >= t.nzt) return;
    const int x = t.x0 + xi, z = t.z0 + zi;
    const int64_t k = x + (int64_t)d.nx * (t.y + (int64_t)d.ny * z);
    const double* c = sm + xi * wire_pitch<PER>() + zi * PER;
#pragma unroll
    for (int i = 0; i < Q; ++i) scatter_canonical<T>(d, f, wall, i, x, t.y, z, k, c[i]);
    if (PER == Q + 4) {
        for (int a = 0; a < 3; ++a) F[3 * k + a] = (typename Store<T>::F)c[Q + a];
        if (phase) phase[k] = c[Q + 3] >= 0.5 ? 1 : 0;
    }
}

template <class T, int PER>
__global__ void __launch_bounds__(kWireX * kWireZ) k_export_aos(LatticeDesc d, const T* __restrict__ f,
                                                                const T* __restrict__ wall,
                                                                const typename Store<T>::F* __restrict__ F,
                                                                const uint8_t* __restrict__ phase,
                                                                double* __restrict__ dst, int x0, int nxc) {
    using C = typename Store<T>::C;
    __shared__ double sm[kWireX * wire_pitch<PER>()];
    const WireTile t = wire_tile(d, x0, nxc);
    const int xi = threadIdx.x & (kWireX - 1), zi = threadIdx.x / kWireX;
    if (xi < t.nxt && zi < t.nzt) {
        const int x = t.x0 + xi, z = t.z0 + zi;
        const int64_t k = x + (int64_t)d.nx * (t.y + (int64_t)d.ny * z);
        double* c = sm + xi * wire_pitch<PER>() + zi * PER;
        C fc[Q];
        gather<T>(d, f, wall, x, t.y, z, k, fc);
#pragma unroll
        for (int i = 0; i < Q; ++i) c[i] = (double)fc[i];
        if (PER == Q + 4) {
            for (int a = 0; a < 3; ++a) c[Q + a] = (double)F[3 * k + a];
            c[Q + 3] = phase && phase[k] ? 1.0 : 0.0;
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= t.nxt) return;
    double* o = dst + (int64_t)PER * (t.z0 + (int64_t)d.nz * (t.y + (int64_t)d.ny * (t.x0 - x0 + warp)));
    const double* s = sm + warp * wire_pitch<PER>();
    const int n = PER * t.nzt;
#pragma unroll
    for (int k = 0; k < PER; ++k)
        if (lane + 32 * k < n) o[lane + 32 * k] = s[lane + 32 * k];
}

template <class FT>
__global__ void k_force_import(LatticeDesc d, FT* __restrict__ F, const double* __restrict__ src) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    for (int a = 0; a < 3; ++a) F[3 * k + a] = (FT)src[a * d.n + k];
}

template <class FT>
__global__ void k_force_export(LatticeDesc d, const FT* __restrict__ F, double* __restrict__ dst) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    for (int a = 0; a < 3; ++a) dst[a * d.n + k] = (double)F[3 * k + a];
}

// One component of the cells k0 .. k0 + n - 1 out of (IN: into) the force field, for files that hold one array per
// component.
template <class FT, bool IN>
__global__ void k_force_component(FT* __restrict__ F, FT* __restrict__ part, int a, int64_t k0, int64_t n) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (IN) F[3 * (k0 + k) + a] = part[k];
    else part[k] = F[3 * (k0 + k) + a];
}

template <class FT>
__global__ void k_force_fill(LatticeDesc d, FT* __restrict__ F) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= d.stride) return;
    for (int a = 0; a < 3; ++a) F[3 * k + a] = (FT)d.body[a];
}

__global__ void k_phase_import(LatticeDesc d, uint8_t* __restrict__ ph, const double* __restrict__ src) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    ph[k] = src[k] >= 0.5 ? 1 : 0;
}

template <class T>
__global__ void k_nan_scan(LatticeDesc d, const T* __restrict__ f, int* flag) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    bool bad = false;
    for (int i = 0; i < Q; ++i) {
        const float v = (float)Store<T>::load(f + i * d.stride + k, d.inv_scale);
        bad |= !isfinite(v);
    }
    if (bad) atomicOr(flag, 1);
}

inline int row_block(const LatticeDesc& d) { return d.nx >= 256 ? 256 : (d.nx >= 128 ? 128 : (d.nx >= 64 ? 64 : 32)); }
inline dim3 row_grid(const LatticeDesc& d, int bx) { return dim3((d.nx + bx - 1) / bx, d.ny, d.nz); }
inline unsigned lin_grid(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

template <class T>
void collide_stream_t(const Lattice& L, Coupling mode, cudaStream_t s) {
    using FT = typename Store<T>::F;
    if (L.collide_kernel != BIB_KERNEL_ROWS && (launch_collide_stream_staged(L, mode, s) || launch_collide_stream_linear(L, mode, s)))
        return;
    const bool coupled = mode != Coupling::kNone;
    // the previous force: read for the velocity and reset (dense), or reset alone, without a velocity field
    FT* Fprev = mode == Coupling::kDense || mode == Coupling::kReset ? (FT*)L.F[L.fe] : nullptr;
    auto* u = mode == Coupling::kReset ? nullptr : (typename Store<T>::U*)L.u;
    if (L.d.nx % 2 == 0) {
        const int pairs = L.d.nx / 2;
        const int bx = std::min(256, (pairs + 31) / 32 * 32);
        const int by = std::max(1, 256 / bx);
        const int rows = L.d.ny * L.d.nz;
        dim3 grid((rows + by - 1) / by, (pairs + bx - 1) / bx);
        dim3 block(bx, by);
        const T* fin = (const T*)L.f[L.cur];
        T* fout = (T*)L.f[1 - L.cur];
        if (coupled)
            k_collide_stream_rows<T, true><<<grid, block, 0, s>>>(L.d, fin, fout, (const T*)L.wall, (const FT*)L.F[1 - L.fe],
                                                                  Fprev, u, L.phase, L.celltype, L.d.collision);
        else
            k_collide_stream_rows<T, false><<<grid, block, 0, s>>>(L.d, fin, fout, (const T*)L.wall, (const FT*)L.F[L.fe],
                                                                   nullptr, nullptr, L.phase, L.celltype, L.d.collision);
        return;
    }
    const int bx = row_block(L.d);
    const T* fin = (const T*)L.f[L.cur];
    T* fout = (T*)L.f[1 - L.cur];
    const T* wall = (const T*)L.wall;
    if (coupled) {
        k_collide_stream<T, true><<<row_grid(L.d, bx), bx, 0, s>>>(L.d, fin, fout, wall, (const FT*)L.F[1 - L.fe],
                                                                    Fprev, u, L.phase, L.celltype, L.d.collision);
    } else {
        k_collide_stream<T, false><<<row_grid(L.d, bx), bx, 0, s>>>(L.d, fin, fout, wall, (const FT*)L.F[L.fe], nullptr,
                                                                     nullptr, L.phase, L.celltype, L.d.collision);
    }
}

template <class T>
void fd_walls_batch_t(const BatchLaunch& B, cudaStream_t s) {
    k_fd_walls_batch<T><<<dim3(lin_grid((int64_t)B.nx_max * B.nz_max, kWallBlock), 2, B.n), kWallBlock, 0, s>>>(B.wviews);
}

template <class T>
void fd_walls_t(const Lattice& L, int buf, int fbuf, cudaStream_t s) {
    using FT = typename Store<T>::F;
    k_fd_walls<T><<<dim3(lin_grid((int64_t)L.d.nx * L.d.nz, kWallBlock), 2), kWallBlock, 0, s>>>(
        L.d, (const T*)L.f[buf], (T*)L.wall, (const FT*)L.F[fbuf]);
}

#define BIB_DISPATCH(storage, FN, ...)                          \
    do {                                                       \
        if ((storage) == BIB_STORAGE_F64) FN<double>(__VA_ARGS__); \
        else if ((storage) == BIB_STORAGE_F32) FN<float>(__VA_ARGS__); \
        else FN<__half>(__VA_ARGS__);                          \
    } while (0)

// The velocity field that an interpolation is about to read: at its support nodes where they are at
// most half as many as the cells (short scattered runs against whole rows), on lattices of 2^16 cells
// or more.  Measured, one step with a phase field, support nodes against all cells: 96^3 FP32 113 / 148 us
// at 0.02 nodes per cell, 126 / 150 at 0.31; 64^3 71 / 76 at 0.07, 80.6 / 81.6 at 0.53, 88 / 84 at 1.06; 96^3
// FP64 441 / 523 at 0.02; 32^3 FP32 54.3 / 53.3 at 0.13, 70 / 65 at 4.2.
template <class T>
void velocity_support_t(const Lattice& L, cudaStream_t s) {
    using FT = typename Store<T>::F;
    using UT = typename Store<T>::U;
    const int sup = L.ib.dirac == BIB_DIRAC_PESKIN ? 4 : 3;
    const int64_t nodes = (int64_t)L.nvert * sup * sup * sup;
    auto kern = sup == 4 ? k_velocity_support<T, 4> : k_velocity_support<T, 3>;
    kern<<<lin_grid(nodes, 128), 128, 0, s>>>(L.d, L.ib, nodes, L.pos[L.pcur], (const T*)L.f[L.cur], (const T*)L.wall,
                                              (const FT*)L.F[L.fe], (UT*)L.u, L.celltype);
}
template <class T>
void velocity_field_t(const Lattice& L, cudaStream_t s) {
    using FT = typename Store<T>::F;
    using UT = typename Store<T>::U;
    if (few_support_nodes(L) && L.d.n >= 65536) {
        velocity_support_t<T>(L, s);
        return;
    }
    const int bx = row_block(L.d);
    k_velocity<T, UT><<<row_grid(L.d, bx), bx, 0, s>>>(L.d, (const T*)L.f[L.cur], (const T*)L.wall, (const FT*)L.F[L.fe],
                                                        (UT*)L.u, 1, 4, L.celltype);
}

template <class T>
void velocity_export_t(const Lattice& L, double* u, cudaStream_t s) {
    using FT = typename Store<T>::F;
    const int bx = row_block(L.d);
    k_velocity<T, double><<<row_grid(L.d, bx), bx, 0, s>>>(L.d, (const T*)L.f[L.cur], (const T*)L.wall,
                                                            (const FT*)L.F[L.fe], u, L.d.n, 1, L.celltype);
}

template <class T>
void init_eq_t(const Lattice& L, const double* rho, const double* u, cudaStream_t s) {
    const int bx = row_block(L.d);
    k_init_eq<T><<<row_grid(L.d, bx), bx, 0, s>>>(L.d, (T*)L.f[L.cur], (T*)L.wall, rho, u);
}

template <class T>
void import_t(const Lattice& L, const double* src, int z0, int nzc, int64_t pitch, cudaStream_t s) {
    const int bx = row_block(L.d);
    dim3 g((L.d.nx + bx - 1) / bx, L.d.ny, nzc);
    k_import<T><<<g, bx, 0, s>>>(L.d, (T*)L.f[L.cur], (T*)L.wall, src, z0, pitch);
}

template <class T>
void export_t(const Lattice& L, double* dst, int z0, int nzc, int64_t pitch, cudaStream_t s) {
    const int bx = row_block(L.d);
    dim3 g((L.d.nx + bx - 1) / bx, L.d.ny, nzc);
    k_export<T><<<g, bx, 0, s>>>(L.d, (const T*)L.f[L.cur], (const T*)L.wall, dst, z0, pitch);
}

inline dim3 wire_grid(const LatticeDesc& d, int nxc) {
    return dim3((nxc + kWireX - 1) / kWireX, d.ny, (d.nz + kWireZ - 1) / kWireZ);
}

template <class T>
void import_aos_t(const Lattice& L, const double* src, int per, int x0, int nxc, cudaStream_t s) {
    using FT = typename Store<T>::F;
    auto kern = per == Q ? k_import_aos<T, Q> : k_import_aos<T, Q + 4>;
    kern<<<wire_grid(L.d, nxc), kWireX * kWireZ, 0, s>>>(L.d, (T*)L.f[L.cur], (T*)L.wall, (FT*)L.F[L.fe], L.phase, src, x0, nxc);
}

template <class T>
void export_aos_t(const Lattice& L, double* dst, int per, int x0, int nxc, cudaStream_t s) {
    using FT = typename Store<T>::F;
    auto kern = per == Q ? k_export_aos<T, Q> : k_export_aos<T, Q + 4>;
    kern<<<wire_grid(L.d, nxc), kWireX * kWireZ, 0, s>>>(L.d, (const T*)L.f[L.cur], (const T*)L.wall, (const FT*)L.F[L.fe],
                                                         L.phase, dst, x0, nxc);
}

template <class T>
void nan_scan_t(const Lattice& L, int* flag, cudaStream_t s) {
    k_nan_scan<T><<<lin_grid(L.d.n, 256), 256, 0, s>>>(L.d, (const T*)L.f[L.cur], flag);
}

}  // namespace

void launch_collide_stream(const Lattice& L, Coupling mode, cudaStream_t s) {
    BIB_DISPATCH(L.storage, collide_stream_t, L, mode, s);
}

void launch_fd_walls_batch(const BatchLaunch& B, cudaStream_t s) {
    if (!B.any_fd || B.n == 0) return;
    BIB_DISPATCH(B.storage, fd_walls_batch_t, B, s);
}

template <class T>
void guo_walls_t(const Lattice& L, int buf, cudaStream_t s) {
    k_guo_walls<T><<<(L.nguo + 127) / 128, 128, 0, s>>>(L.d, (T*)L.f[buf], (const T*)L.wall, L.guo, L.nguo);
}

// The wall processors after a collide-and-stream: finite-difference velocity walls, then the
// second-order rigid walls (the latter integrated at processor level 1, after the former)
void launch_fd_walls(const Lattice& L, int buf, int fbuf, cudaStream_t s) {
    if (L.d.fd_walls) BIB_DISPATCH(L.storage, fd_walls_t, L, buf, fbuf, s);
    if (L.nguo > 0) BIB_DISPATCH(L.storage, guo_walls_t, L, buf, s);
}

namespace {
__global__ void __launch_bounds__(256) k_copy_f64(double* __restrict__ dst, const double* __restrict__ src, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = src[i];
}
}  // namespace

void launch_copy_f64(double* dst, const double* src, size_t n, cudaStream_t s) {
    if (n == 0) return;
    const unsigned g = (unsigned)std::min<size_t>((n + 255) / 256, 1024);
    k_copy_f64<<<g, 256, 0, s>>>(dst, src, n);
}

void launch_velocity_field(const Lattice& L, cudaStream_t s) { BIB_DISPATCH(L.storage, velocity_field_t, L, s); }
void launch_velocity_support(const Lattice& L, cudaStream_t s) { BIB_DISPATCH(L.storage, velocity_support_t, L, s); }

void launch_velocity_export(const Lattice& L, double* u, cudaStream_t s) {
    BIB_DISPATCH(L.storage, velocity_export_t, L, u, s);
}

void launch_init_equilibrium(const Lattice& L, const double* rho, const double* u, cudaStream_t s) {
    BIB_DISPATCH(L.storage, init_eq_t, L, rho, u, s);
}

void launch_import_planes(const Lattice& L, const double* src, int z0, int nzc, int64_t pitch, cudaStream_t s) {
    BIB_DISPATCH(L.storage, import_t, L, src, z0, nzc, pitch, s);
}

void launch_export_planes(const Lattice& L, double* dst, int z0, int nzc, int64_t pitch, cudaStream_t s) {
    BIB_DISPATCH(L.storage, export_t, L, dst, z0, nzc, pitch, s);
}

void launch_import_aos(const Lattice& L, const double* src, int per, int x0, int nxc, cudaStream_t s) {
    if (nxc > 0) BIB_DISPATCH(L.storage, import_aos_t, L, src, per, x0, nxc, s);
}

void launch_export_aos(const Lattice& L, double* dst, int per, int x0, int nxc, cudaStream_t s) {
    if (nxc > 0) BIB_DISPATCH(L.storage, export_aos_t, L, dst, per, x0, nxc, s);
}

void launch_force_component(const Lattice& L, int buf, void* part, int a, int64_t k0, int64_t n, bool in, cudaStream_t s) {
    auto run = [&](auto zero) {
        using FT = decltype(zero);
        auto kern = in ? k_force_component<FT, true> : k_force_component<FT, false>;
        kern<<<lin_grid(n, 256), 256, 0, s>>>((FT*)L.F[buf], (FT*)part, a, k0, n);
    };
    if (L.storage == BIB_STORAGE_F64) run(double{});
    else run(float{});
}

void launch_force_import(const Lattice& L, int buf, const double* src, cudaStream_t s) {
    const unsigned g = lin_grid(L.d.n, 256);
    if (L.storage == BIB_STORAGE_F64) k_force_import<double><<<g, 256, 0, s>>>(L.d, (double*)L.F[buf], src);
    else k_force_import<float><<<g, 256, 0, s>>>(L.d, (float*)L.F[buf], src);
}

void launch_force_export(const Lattice& L, int buf, double* dst, cudaStream_t s) {
    const unsigned g = lin_grid(L.d.n, 256);
    if (L.storage == BIB_STORAGE_F64) k_force_export<double><<<g, 256, 0, s>>>(L.d, (const double*)L.F[buf], dst);
    else k_force_export<float><<<g, 256, 0, s>>>(L.d, (const float*)L.F[buf], dst);
}

void launch_force_fill(const Lattice& L, int buf, cudaStream_t s) {
    const size_t fsz = L.storage == BIB_STORAGE_F64 ? sizeof(double) : sizeof(float);
    if (L.d.body[0] == 0.0 && L.d.body[1] == 0.0 && L.d.body[2] == 0.0) {
        cudaMemsetAsync(L.F[buf], 0, 3 * L.d.stride * fsz, s);
        return;
    }
    const unsigned g = lin_grid(L.d.stride, 256);
    if (L.storage == BIB_STORAGE_F64) k_force_fill<double><<<g, 256, 0, s>>>(L.d, (double*)L.F[buf]);
    else k_force_fill<float><<<g, 256, 0, s>>>(L.d, (float*)L.F[buf]);
}

void launch_phase_import(const Lattice& L, const double* src, cudaStream_t s) {
    k_phase_import<<<lin_grid(L.d.n, 256), 256, 0, s>>>(L.d, L.phase, src);
}

void launch_nan_scan(const Lattice& L, int* flag, cudaStream_t s) { BIB_DISPATCH(L.storage, nan_scan_t, L, flag, s); }

}  // namespace bib
