// Immersed-boundary kernels: delta interpolation of the lattice velocity to the
// membrane vertices and their motion, membrane forces (by patches, elements or vertices),
// delta spreading of the vertex forces into the lattice force field, and the area / volume /
// centre-of-mass update.
//
// Vertices of all particles of a lattice are concatenated: positions (FP64, two
// buffers swapped every step), velocities and forces (FP64).
#include <algorithm>
#include <cfloat>

#include <cub/device/device_radix_sort.cuh>

#include "lattice_common.cuh"

namespace bib {

namespace {

// Reduced-precision arithmetic: the FP32 element and weight evaluations use the hardware's
// approximate square root, reciprocal and division (a few ulp); FP64 keeps the IEEE
// operations of the reference's expressions.
__device__ __forceinline__ float fast_sqrt(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double fast_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float fast_rcp(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double fast_rcp(double x) { return 1.0 / x; }
__device__ __forceinline__ float fast_div(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double fast_div(double a, double b) { return a / b; }

// ---------------------------------------------------------------- delta kernels
// RomaDirac<T,3>::eval and PeskinDirac<T,3>::eval(x), src/fsi/Dirac.h:27-31, 78-83
template <class W>
__device__ __forceinline__ W dirac_eval(int dirac, W x) {
    const W dx = fabs(x);
    if (dirac == BIB_DIRAC_PESKIN)
        return W(0.125) * (dx <= W(1) ? (W(3) - W(2) * dx + fast_sqrt(W(1) + W(4) * dx * (W(1) - dx)))
                                      : (W(5) - W(2) * dx - fast_sqrt(W(-7) + W(4) * dx * (W(3) - dx))));
    return (W(1) / W(6)) * (dx > W(0.5) ? (W(5) - W(3) * dx - fast_sqrt(W(-3) * (W(1) - dx) * (W(1) - dx) + W(1)))
                                        : W(2) * (W(1) + fast_sqrt(W(1) - W(3) * dx * dx)));
}

// First support node of one axis as the spreading records it for the sparse force reset: on a
// periodic axis reduced to one period (remap_global of lo + m is unchanged), so that it fits 32
// bits; on a walled axis a vertex inside the envelope is within h + 1 of the domain.
__device__ __forceinline__ int record_lo(int periodic, int N, int64_t lo, int off) {
    return periodic ? pmod(lo + off, N) - off : (int)lo;
}

// Delta weight of support node lo + m on one axis, phi(lo + m - x) with lo = ceil(x - h).
// FP32 weights take the FP64 offset lo - x and add m in FP32.
template <class W>
__device__ __forceinline__ W axis_weight(int dirac, int64_t lo, double x, int m) {
    if (sizeof(W) == sizeof(double)) return dirac_eval<W>(dirac, (W)((double)(lo + m) - x));
    return dirac_eval<W>(dirac, (W)((double)lo - x) + (W)m);
}
template <class W, int S>
__device__ __forceinline__ int64_t axis_weights(double x, W* w) {
    constexpr int dirac = S == 4 ? BIB_DIRAC_PESKIN : BIB_DIRAC_ROMA;
    const int64_t lo = (int64_t)ceil(x - half_support(dirac));
#pragma unroll
    for (int m = 0; m < S; ++m) w[m] = axis_weight<W>(dirac, lo, x, m);
    return lo;
}

// One cell of the velocity field ((ux, uy, uz, 0) per cell), one or two vector loads.
template <class C>
struct U3 {
    C x, y, z;
};
__device__ __forceinline__ U3<float> load_u(const float* u, int64_t k) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(u) + k);
    return U3<float>{v.x, v.y, v.z};
}
__device__ __forceinline__ U3<double> load_u(const double* u, int64_t k) {
    const double2* q = reinterpret_cast<const double2*>(u) + 2 * k;
    const double2 a = __ldg(q), b = __ldg(q + 1);
    return U3<double>{a.x, a.y, b.x};
}
__device__ __forceinline__ U3<float> load_u(const __half* u, int64_t k) {  // FP16 population storage
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(u) + k);
    const float2 ab = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    return U3<float>{ab.x, ab.y, __low2float(*reinterpret_cast<const __half2*>(&v.y))};
}
// Compute type of an interpolation from the velocity field's storage type.
template <class UT>
struct InterpC {
    using type = float;
};
template <>
struct InterpC<double> {
    using type = double;
};

// ---------------------------------------------------------------- pipe boundary
// PipeBoundary::distance_to_boundary (fsi/Boundary.h:158-161) minus the kernel's half support:
// the weight of the supplied kernel against the 2-point TopHat near the wall (>= 1: the
// supplied kernel alone, <= 0: the TopHat alone, _interpolation.hh:181-230, _forces.hh:192-237)
__device__ __forceinline__ double pipe_weight(const IbDesc& ib, const double* p, double h) {
    const double dy = p[1] - ib.pipe_y0, dz = p[2] - ib.pipe_z0;
    return ib.pipe_r - sqrt(dy * dy + dz * dz) - h;
}

// TopHatDirac<T,3> (Dirac.h:47-64): support 2, weight 1 - |x| per axis; the 2 x 2 x 2 nodes
// in GeneralInterpolator / GeneralSpreading order.  mode 0 gathers u into acc, mode 1 adds
// w * fv into the force field.
template <class C, class UT>
__device__ __forceinline__ void tophat_interp(const LatticeDesc& d, const IbDesc& ib, const double* p, const UT* u, C* acc) {
    const int off = (int)ib.offset;
    int64_t lo[3];
    C w[3][2];
    for (int a = 0; a < 3; ++a) {
        const double x = p[a] - ib.offset;
        lo[a] = (int64_t)ceil(x - 1.0);
        w[a][0] = (C)(1. - fabs((double)lo[a] - x));
        w[a][1] = (C)(1. - fabs((double)(lo[a] + 1) - x));
    }
    for (int a = 0; a < 2; ++a) {
        const int gx = remap_global(d.px, d.nx, lo[0] + a, off);
        if (gx < 0) continue;
        for (int b = 0; b < 2; ++b) {
            const int gy = remap_global(d.py, d.ny, lo[1] + b, off);
            if (gy < 0) continue;
            const C wxy = w[0][a] * w[1][b];
            for (int c = 0; c < 2; ++c) {
                const int gz = remap_global(d.pz, d.nz, lo[2] + c, off);
                if (gz < 0) continue;
                const C wt = wxy * w[2][c];
                const U3<C> uc = load_u(u, gx + (int64_t)d.nx * (gy + (int64_t)d.ny * gz));
                acc[0] += wt * uc.x;
                acc[1] += wt * uc.y;
                acc[2] += wt * uc.z;
            }
        }
    }
}
template <class FT>
__device__ __forceinline__ void tophat_spread(const LatticeDesc& d, const IbDesc& ib, const double* p, const FT* fv, FT* F) {
    const int off = (int)ib.offset;
    int64_t lo[3];
    FT w[3][2];
    for (int a = 0; a < 3; ++a) {
        const double x = p[a] - ib.offset;
        lo[a] = (int64_t)ceil(x - 1.0);
        w[a][0] = (FT)(1. - fabs((double)lo[a] - x));
        w[a][1] = (FT)(1. - fabs((double)(lo[a] + 1) - x));
    }
    for (int a = 0; a < 2; ++a) {
        const int gx = remap_global(d.px, d.nx, lo[0] + a, off);
        if (gx < 0) continue;
        for (int b = 0; b < 2; ++b) {
            const int gy = remap_global(d.py, d.ny, lo[1] + b, off);
            if (gy < 0) continue;
            const FT wxy = w[0][a] * w[1][b];
            for (int c = 0; c < 2; ++c) {
                const int gz = remap_global(d.pz, d.nz, lo[2] + c, off);
                if (gz < 0) continue;
                const FT wt = wxy * w[2][c];
                FT* q = F + 3 * (gx + (int64_t)d.nx * (gy + (int64_t)d.ny * gz));
                atomicAdd(q, wt * fv[0]);
                atomicAdd(q + 1, wt * fv[1]);
                atomicAdd(q + 2, wt * fv[2]);
            }
        }
    }
}

// DeformableParticle3D::move_vertices(boundary) (DeformableParticle3D.hh:26-51) with
// PipeBoundary::trace_ray / get_normal (Boundary.h:164-187, 245-249): a step that crosses the
// wall is reflected about the normal at the crossing.
__device__ __forceinline__ void pipe_move(const IbDesc& ib, const double* old, const double* v, double* x) {
    const double y1 = old[1] - ib.pipe_y0, y2 = x[1] - ib.pipe_y0, z1 = old[2] - ib.pipe_z0, z2 = x[2] - ib.pipe_z0;
    const double a = (y2 - y1) * (y2 - y1) + (z2 - z1) * (z2 - z1);
    const double b = y1 * (y2 - y1) + z1 * (z2 - z1);
    const double c = y1 * y1 + z1 * z1 - ib.pipe_r * ib.pipe_r;
    const double disc = b * b - c * a;
    if (disc < 0. || fabs(a) < 10 * DBL_EPSILON) return;
    const double bOverA = -b / a, sqrtDisc = sqrt(disc) / a;
    double t = bOverA - sqrtDisc;
    if (!(t >= 0. && t <= 1.)) {
        t = bOverA + sqrtDisc;
        if (!(t >= 0. && t <= 1.)) return;
    }
    for (int k = 0; k < 3; ++k) x[k] = old[k] + t * v[k];
    const double ny_ = x[1] - ib.pipe_y0, nz_ = x[2] - ib.pipe_z0;
    const double nn = sqrt(0.0 * 0.0 + ny_ * ny_ + nz_ * nz_);
    const double n[3] = {0.0 / nn, ny_ / nn, nz_ / nn};
    const double s2 = 2. * (v[0] * n[0] + v[1] * n[1] + v[2] * n[2]);
    for (int k = 0; k < 3; ++k) x[k] += (v[k] - s2 * n[k]) * (1. - t);
}

// Velocity and move of a vertex in a pipe from the interpolated velocity u3: near the wall blended with
// (or switched to) the TopHat kernel, and a step that crosses the wall reflected.
template <class UT, int S, class C>
__device__ __noinline__ void move_near_pipe(const IbView& V, int v, const C* u3) {
    const double p[3] = {V.pos[3 * v], V.pos[3 * v + 1], V.pos[3 * v + 2]};
    double out[3] = {(double)u3[0], (double)u3[1], (double)u3[2]};
    if (inside_envelope(V.d, V.ib.dirac, p)) {
        const double w = pipe_weight(V.ib, p, S == 4 ? 2.0 : 1.5);
        if (w < 1) {
            C t[3] = {C(0), C(0), C(0)};
            tophat_interp<C, UT>(V.d, V.ib, p, static_cast<const UT*>(V.u), t);
            for (int k = 0; k < 3; ++k) out[k] = w <= 0 ? (double)t[k] : (1. - w) * (double)t[k] + w * out[k];
        }
    }
    double xn[3] = {p[0] + out[0], p[1] + out[1], p[2] + out[2]};
    pipe_move(V.ib, p, out, xn);
    for (int k = 0; k < 3; ++k) {
        V.vel[3 * v + k] = out[k];
        V.pos_next[3 * v + k] = xn[k];
    }
}

// ---------------------------------------------------------------- interpolation
// Interpolation of the velocity field (written by the collide-and-stream kernel or the
// velocity kernel) to every vertex, followed by the explicit Euler move
// X_{n+1} = X_n + U_n (DeformableParticle3D::move_vertices, DeformableParticle3D.hh:26-51).
// Classes and index arithmetic follow interpolate_impl with the Bulk / General
// interpolators, ImmersedBoundaryDynamics_interpolation.hh:13-153.
// BATCH: the vertex numbering runs over the lattices of a batch and each vertex looks its lattice's view
// up through vinst; otherwise v1 is the lattice.
// FOLD (sparse force reset): the velocity field holds j/rho + body/2, and the vertex velocity
// adds the share of the previous step's force, sum of w (Fold - body) / 2 over the support
// nodes off the finite-difference wall rows (whose velocity is the wall's); the sum of the two
// is the interpolation of j/rho + Fold/2, the reference's computeVelocity field.
//
// Many vertices: one thread per vertex.
template <class UT, int S, bool FOLD = false>
__device__ __forceinline__ void interpolate_move_vertex(const IbView& V, int v) {
    using C = typename InterpC<UT>::type;  // also the force field's type
    static_assert(S == 3 || S == 4, "Roma (3) or Peskin (4) support");
    const LatticeDesc& d = V.d;
    const IbDesc& ib = V.ib;
    const double* __restrict__ pos = V.pos;
    double* __restrict__ pos_next = V.pos_next;
    const UT* __restrict__ u = static_cast<const UT*>(V.u);
    double* __restrict__ vel = V.vel;
    const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
    double out[3] = {0.0, 0.0, 0.0};
    if (inside_envelope(d, ib.dirac, p)) {
        const int off = (int)ib.offset;
        constexpr int s = S;
        int64_t lo[3];
        C w[3][4];
        for (int a = 0; a < 3; ++a) lo[a] = axis_weights<C, S>(p[a] - ib.offset, w[a]);
        int gx[4], gy[4], gz[4];
#pragma unroll
        for (int m = 0; m < s; ++m) {
            gx[m] = remap_global(d.px, d.nx, lo[0] + m, off);
            gy[m] = remap_global(d.py, d.ny, lo[1] + m, off);
            gz[m] = remap_global(d.pz, d.nz, lo[2] + m, off);
        }
        int64_t yo[4], zo[4];  // row offsets of the support nodes
#pragma unroll
        for (int m = 0; m < s; ++m) {
            yo[m] = (int64_t)gy[m] * d.nx;
            zo[m] = (int64_t)gz[m] * d.ny * d.nx;
        }
        C acc[3] = {C(0), C(0), C(0)};
        C facc[3] = {C(0), C(0), C(0)};
        const C* __restrict__ Fo = static_cast<const C*>(V.Fold);
        const C body[3] = {(C)d.body[0], (C)d.body[1], (C)d.body[2]};
#pragma unroll
        for (int a = 0; a < s; ++a) {
            if (gx[a] < 0) continue;
#pragma unroll
            for (int b = 0; b < s; ++b) {
                if (gy[b] < 0) continue;
                const C wxy = w[0][a] * w[1][b];
                const int64_t col = gx[a] + yo[b];
                const bool fd_row = FOLD && fd_wall_node(d, gy[b]);
#pragma unroll
                for (int c = 0; c < s; ++c) {
                    if (gz[c] < 0) continue;
                    const C wt = wxy * w[2][c];
                    const U3<C> uc = load_u(u, col + zo[c]);
                    acc[0] += wt * uc.x;
                    acc[1] += wt * uc.y;
                    acc[2] += wt * uc.z;
                    if (FOLD && !fd_row) {
                        const int64_t k = col + zo[c];
                        facc[0] += wt * (__ldg(Fo + 3 * k) - body[0]);
                        facc[1] += wt * (__ldg(Fo + 3 * k + 1) - body[1]);
                        facc[2] += wt * (__ldg(Fo + 3 * k + 2) - body[2]);
                    }
                }
            }
        }
        out[0] = (double)(FOLD ? acc[0] + C(0.5) * facc[0] : acc[0]);
        out[1] = (double)(FOLD ? acc[1] + C(0.5) * facc[1] : acc[1]);
        out[2] = (double)(FOLD ? acc[2] + C(0.5) * facc[2] : acc[2]);
    }
    if (ib.has_pipe) {
        const C u3[3] = {(C)out[0], (C)out[1], (C)out[2]};
        move_near_pipe<UT, S>(V, v, u3);
        return;
    }
    vel[3 * v] = out[0];
    vel[3 * v + 1] = out[1];
    vel[3 * v + 2] = out[2];
    pos_next[3 * v] = p[0] + out[0];
    pos_next[3 * v + 1] = p[1] + out[1];
    pos_next[3 * v + 2] = p[2] + out[2];
}

// 9 CTAs of 128 threads per SM (at most 56 registers): measured 2 % faster than 8 on the
// 400-cell channel (the kernel waits on its gathers; more warps hide more of that)
template <class UT, int S, bool BATCH, bool FOLD = false>
__global__ void __launch_bounds__(128, 9) k_interpolate_vertices(IbView v1, const IbView* __restrict__ views,
                                                           const int* __restrict__ vinst, int nvert) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nvert) return;
    const IbView& V = BATCH ? views[vinst[g]] : v1;
    interpolate_move_vertex<UT, S, FOLD>(V, BATCH ? g - V.vbase : (V.order ? V.order[g] : g));
}

// Few vertices: a CTA takes 32; three warps prepare one axis each (nodes and weights, the FP64 part), then warp r
// gathers row r of every support (one vertex per lane) and 96 threads add the rows up in order and move
// one coordinate each.  Bound by the latency of the gathers and by the FP64 pipe (about 9 operations per
// coordinate); with tens of thousands of vertices the CTAs' barriers cost more than the threads of the
// kernel above wait.  Measured, interpolation and update of a step in 256 x 64 x 64, 32 vertices per CTA against
// one thread per vertex: FP32 Roma 18.7 / 24.4 us at 2,568 vertices, 23.0 / 25.1 at 20,544, 27.2 / 26.2 at 41,088,
// 57 / 35 at 164,352; FP64 Peskin 28.7 / 55.5, 63 / 66, 100 / 88, 319 / 221; the line is between those.
constexpr int kGatherMax = 24576;
constexpr int kGatherVerts = 32;
template <class C, int S>
struct GatherTile {
    int vert[kGatherVerts];         // vertex, -1: none
    int inst[kGatherVerts];         // batch: the lattice
    int node[3][S][kGatherVerts];   // support nodes, -1: none
    C w[3][S][kGatherVerts];
    C part[S * S][3][kGatherVerts];  // of each row
};

template <class UT, int S, bool BATCH, bool FOLD = false>
__global__ void __launch_bounds__(32 * S * S) k_interpolate_move(IbView v1, const IbView* __restrict__ views,
                                                                const int* __restrict__ vinst, int nvert) {
    using C = typename InterpC<UT>::type;  // also the force field's type
    static_assert(S == 3 || S == 4, "Roma (3) or Peskin (4) support");
    constexpr int dirac = S == 4 ? BIB_DIRAC_PESKIN : BIB_DIRAC_ROMA;
    __shared__ GatherTile<C, S> sm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 3) {
        const int g = blockIdx.x * kGatherVerts + lane, a = warp;
        int v = -1, inst = 0;
        if (g < nvert) {
            if (BATCH) inst = vinst[g];
            const IbView& V = BATCH ? views[inst] : v1;
            v = BATCH ? g - V.vbase : (V.order ? V.order[g] : g);
            const LatticeDesc& d = V.d;
            const int off = (int)V.ib.offset, per = a == 0 ? d.px : (a == 1 ? d.py : d.pz);
            const int N = a == 0 ? d.nx : (a == 1 ? d.ny : d.nz);
            const double p = V.pos[3 * v + a];
            const bool in = inside_axis(per, N, dirac, p);
            const double x = p - V.ib.offset;
            const int64_t lo = (int64_t)ceil(x - half_support(dirac));
#pragma unroll
            for (int m = 0; m < S; ++m) {
                sm.node[a][m][lane] = in ? remap_global(per, N, lo + m, off) : -1;
                sm.w[a][m][lane] = axis_weight<C>(dirac, lo, x, m);
            }
        }
        if (a == 0) {
            sm.vert[lane] = v;
            sm.inst[lane] = inst;
        }
    }
    __syncthreads();
    const int v = sm.vert[lane];
    if (v >= 0) {
        const IbView& V = BATCH ? views[sm.inst[lane]] : v1;
        const LatticeDesc& d = V.d;
        const UT* __restrict__ u = static_cast<const UT*>(V.u);
        const int b = warp / S, c = warp % S;
        const int gy = sm.node[1][b][lane], gz = sm.node[2][c][lane];
        C acc[3] = {C(0), C(0), C(0)};
        if (gy >= 0 && gz >= 0) {
            const int64_t row = (int64_t)d.nx * (gy + (int64_t)d.ny * gz);
            const bool fold = FOLD && !fd_wall_node(d, gy);
#pragma unroll
            for (int m = 0; m < S; ++m) {
                const int gx = sm.node[0][m][lane];
                if (gx < 0) continue;
                const C w = sm.w[0][m][lane];
                const U3<C> uc = load_u(u, row + gx);
                acc[0] += w * uc.x;
                acc[1] += w * uc.y;
                acc[2] += w * uc.z;
                if (fold) {
                    const C* __restrict__ Fo = static_cast<const C*>(V.Fold) + 3 * (row + gx);
#pragma unroll
                    for (int q = 0; q < 3; ++q) acc[q] += C(0.5) * (w * (__ldg(Fo + q) - (C)d.body[q]));
                }
            }
            const C wyz = sm.w[1][b][lane] * sm.w[2][c][lane];
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[q] *= wyz;
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) sm.part[warp][q][lane] = acc[q];
    }
    __syncthreads();
    // one coordinate per thread, neighbouring threads the coordinates of a vertex
    const int t = threadIdx.x / 3, q = threadIdx.x - 3 * t;
    if (threadIdx.x >= 3 * kGatherVerts || sm.vert[t] < 0) return;
    const IbView& V = BATCH ? views[sm.inst[t]] : v1;
    const int64_t e = 3LL * sm.vert[t] + q;
    C sum = sm.part[0][q][t];
#pragma unroll
    for (int r = 1; r < S * S; ++r) sum += sm.part[r][q][t];
    if (V.ib.has_pipe) {  // the near-wall blend and the reflection need the whole vector
        if (q == 0) {
            C u3[3] = {sum, sm.part[0][1][t], sm.part[0][2][t]};
#pragma unroll
            for (int r = 1; r < S * S; ++r) {
                u3[1] += sm.part[r][1][t];
                u3[2] += sm.part[r][2][t];
            }
            move_near_pipe<UT, S>(V, sm.vert[t], u3);
        }
        return;
    }
    V.vel[e] = (double)sum;
    V.pos_next[e] = V.pos[e] + (double)sum;
}

// Sparse force reset: F := body force at the support nodes the last spreading into F recorded
// (one thread per vertex and (y, z) row of its support).  Along x the stores cover the aligned
// float4 words around the row's s nodes: a cell of such a word outside the support holds the body
// force already or lies in the support of another vertex, which is reset in the same launch.
template <int S>
__global__ void __launch_bounds__(128) k_force_clear(LatticeDesc d, IbDesc ib, int nvert, const int4* __restrict__ lo,
                                                      float* __restrict__ F) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)nvert * S * S) return;
    const int v = (int)(t / (S * S)), r = (int)(t - (int64_t)v * S * S);
    const int4 l = lo[v];
    if (!l.w) return;
    const int off = (int)ib.offset;
    const int gy = remap_global(d.py, d.ny, (int64_t)l.y + r / S, off);
    const int gz = remap_global(d.pz, d.nz, (int64_t)l.z + r % S, off);
    if (gy < 0 || gz < 0) return;
    const int64_t row = (int64_t)d.nx * (gy + (int64_t)d.ny * gz);
    const float b[3] = {(float)d.body[0], (float)d.body[1], (float)d.body[2]};
    const int gx0 = remap_global(d.px, d.nx, (int64_t)l.x, off);
    const int gxl = remap_global(d.px, d.nx, (int64_t)l.x + S - 1, off);
    if (gx0 >= 0 && gxl == gx0 + S - 1) {
        // the row's values are contiguous: the float4 words around them, component (index mod 3)
        const int64_t k0 = (3 * (row + gx0)) & ~(int64_t)3, k1 = (3 * (row + gxl) + 2) & ~(int64_t)3;
        int c = (int)(k0 % 3);
        for (int64_t k = k0; k <= k1; k += 4) {
            const int c1 = c == 2 ? 0 : c + 1, c2 = c1 == 2 ? 0 : c1 + 1;
            reinterpret_cast<float4*>(F)[k >> 2] = make_float4(b[c], b[c1], b[c2], b[c]);
            c = c1;  // 4 values on is one component on
        }
        return;
    }
#pragma unroll
    for (int m = 0; m < S; ++m) {
        const int gx = remap_global(d.px, d.nx, (int64_t)l.x + m, off);
        if (gx < 0) continue;
        for (int q = 0; q < 3; ++q) F[3 * (row + gx) + q] = b[q];
    }
}

// ---------------------------------------------------------------- spreading
// The whole share of vertex v by one thread, node by node: with a positive field offset, where the periodic
// remap leaves nodes out.
template <class FT, int S>
__device__ __noinline__ void spread_vertex_nodes(const IbView& V, int v) {
    const LatticeDesc& d = V.d;
    const IbDesc& ib = V.ib;
    const double* p = V.pos + 3LL * v;
    const double* force = V.force + 3LL * v;
    FT* F = static_cast<FT*>(V.F);
    const double wp = ib.has_pipe ? pipe_weight(ib, p, S == 4 ? 2.0 : 1.5) : 1.0;
    if (wp <= 0) return;
    const double share = wp < 1 ? (double)(FT)wp : 1.0;
    const FT fv[3] = {(FT)(force[0] * share), (FT)(force[1] * share), (FT)(force[2] * share)};
    const int off = (int)ib.offset;
    int64_t lo[3];
    FT w[3][4];
    for (int a = 0; a < 3; ++a) lo[a] = axis_weights<FT, S>(p[a] - ib.offset, w[a]);
    for (int a = 0; a < S; ++a) {
        const int gx = remap_global(d.px, d.nx, lo[0] + a, off);
        for (int b = 0; b < S; ++b) {
            const int gy = remap_global(d.py, d.ny, lo[1] + b, off);
            for (int c = 0; c < S; ++c) {
                const int gz = remap_global(d.pz, d.nz, lo[2] + c, off);
                if (gx < 0 || gy < 0 || gz < 0) continue;
                const FT wt = w[0][a] * w[1][b] * w[2][c];
                FT* q = F + 3 * (gx + (int64_t)d.nx * (gy + (int64_t)d.ny * gz));
                for (int k = 0; k < 3; ++k) atomicAdd(q + k, wt * fv[k]);
            }
        }
    }
}

// Near the wall of a pipe (weight wp < 1): the TopHat takes the share 1 - wp of a vertex's force, its 24 values
// by one thread; the kernel's share goes by rows like that of any other vertex.  Measured, the step of 300 cells of
// 642 vertices in a 256 x 104 x 104 pipe, FP32: Roma 215 us, Peskin 240; node by node for every vertex of a
// lattice with a pipe boundary 309 and 463.
template <class FT, int S>
__device__ __noinline__ void spread_near_wall(const IbView& V, int v) {
    const double* p = V.pos + 3LL * v;
    const double* force = V.force + 3LL * v;
    const double wp = pipe_weight(V.ib, p, S == 4 ? 2.0 : 1.5);
    if (!(wp < 1)) return;
    const double st = wp <= 0 ? 1.0 : 1. - wp;
    const FT ft[3] = {(FT)(force[0] * st), (FT)(force[1] * st), (FT)(force[2] * st)};
    tophat_spread<FT>(V.d, V.ib, p, ft, static_cast<FT*>(V.F));
}

// Spreading by rows.  A row of a vertex's support, S cells of three components, is one contiguous run
// of 3 S values of the force field.  Three warps of a CTA prepare 32 vertices in shared memory, one axis each
// (the products of x-weight and force, the y and z weights, the rows); then all threads take the
// (vertex, row, word) items in order, neighbouring lanes the neighbouring words of a row.  FP32 fields
// are added to in aligned float4 words (S = 3: three words cover a run at any offset, S = 4: four; values
// outside the run add zero), FP64 fields value by value.
// Bound by the count of its L2 reductions.  With one array per component a vertex had 27 runs of 3 values;
// with the components of a cell together it has 9 of 9 values, 1.25 lines each: 256,800 vertices (Roma) of
// the 400-cell channel 79.5 -> 37.4 us, 128,400 (Peskin) of a 240 x 96 x 90 channel 80 -> 35 us (40.9 and 38 with
// all axes of a vertex prepared by one thread).  64 vertices per CTA were slower (40.6 against 36.8 us alone).
constexpr int kSpreadVerts = 32, kSpreadThreads = 128;
template <class FT, int S>
struct SpreadVertex {
    static constexpr int WORDS = sizeof(FT) == 4 ? (S == 3 ? 3 : 4) : 3 * S;  // per row
    static constexpr int ITEMS = S * S * WORDS;
    FT p[3 * S];  // x-weight times force
    FT wy[S], wz[S];
    int yo[S], zo[S];  // rows and planes, -1: behind a wall
    int gx;            // first cell along x (its run wraps if gx + S > nx), -1: nothing to add
    int inst;          // batch: the lattice
};

template <class FT, int S>
struct SpreadTile {
    SpreadVertex<FT, S> sv[kSpreadVerts];
    int lo_rec[3][kSpreadVerts];  // first support node per axis for the sparse reset
    unsigned inside[3];           // vertices inside the envelope, per axis
};

// The spreading of 32 vertices by a CTA of kSpreadThreads threads: lane l of the first three warps gives
// vertex l of the tile, v (-1: none) of lattice `inst`, and its force; view(inst) is the lattice.
template <class FT, int S, class View>
__device__ __forceinline__ void spread_tile(SpreadTile<FT, S>& T, const View& view, int v, int inst, const FT* f) {
    using SV = SpreadVertex<FT, S>;
    const int a = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (a < 3) {  // warp a prepares axis a of the 32 vertices
        constexpr int dirac = S == 4 ? BIB_DIRAC_PESKIN : BIB_DIRAC_ROMA;
        bool in = false;
        if (v >= 0) {
            const IbView& V = view(inst);
            SV& s = T.sv[lane];
            const LatticeDesc& d = V.d;
            const int off = (int)V.ib.offset, per = a == 0 ? d.px : (a == 1 ? d.py : d.pz);
            const int N = a == 0 ? d.nx : (a == 1 ? d.ny : d.nz);
            const double p = V.pos[3 * v + a];
            in = inside_axis(per, N, dirac, p);
            const double x = p - V.ib.offset;
            const int64_t lo = (int64_t)ceil(x - half_support(dirac));
            T.lo_rec[a][lane] = in ? record_lo(per, N, lo, off) : 0;
            if (a == 0) {
                s.inst = inst;
                s.gx = in ? remap_global(per, N, lo, off) : -1;
                FT g[3] = {f[0], f[1], f[2]};
                if (V.ib.has_pipe) {  // near the wall the rows take the share wp of the force, or nothing
                    const double wp = pipe_weight(V.ib, V.pos + 3LL * v, half_support(dirac));
                    if (wp < 1)
                        for (int q = 0; q < 3; ++q) g[q] = (FT)(V.force[3LL * v + q] * (double)(FT)wp);
                    if (wp <= 0) s.gx = -1;
                }
#pragma unroll
                for (int m = 0; m < S; ++m) {
                    const FT w = axis_weight<FT>(dirac, lo, x, m);
#pragma unroll
                    for (int q = 0; q < 3; ++q) s.p[3 * m + q] = w * g[q];
                }
            } else {
                int* node = a == 1 ? s.yo : s.zo;
                FT* w = a == 1 ? s.wy : s.wz;
#pragma unroll
                for (int m = 0; m < S; ++m) {
                    node[m] = in ? remap_global(per, N, lo + m, off) : -1;
                    w[m] = axis_weight<FT>(dirac, lo, x, m);
                }
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) T.inside[a] = m;
    }
    __syncthreads();
    if (a == 0) {
        const bool in = ((T.inside[0] & T.inside[1] & T.inside[2]) >> lane) & 1u;
        const IbView& V = view(inst);
        const bool nodewise = in && (int)V.ib.offset > 0;
        if (!in || nodewise) T.sv[lane].gx = -1;
        if (v >= 0 && V.spread_lo)
            V.spread_lo[v] = in ? make_int4(T.lo_rec[0][lane], T.lo_rec[1][lane], T.lo_rec[2][lane], 1) : make_int4(0, 0, 0, 0);
        if (nodewise) spread_vertex_nodes<FT, S>(V, v);
        if (in && V.ib.has_pipe) spread_near_wall<FT, S>(V, v);
    }
    __syncthreads();
    for (int it = threadIdx.x; it < kSpreadVerts * SV::ITEMS; it += kSpreadThreads) {
        const int t = it / SV::ITEMS, r = it - t * SV::ITEMS, row = r / SV::WORDS, j = r - row * SV::WORDS;
        const SV& s = T.sv[t];
        if (s.gx < 0) continue;
        const int y = s.yo[row / S], z = s.zo[row % S];
        if (y < 0 || z < 0) continue;
        const IbView& V = view(s.inst);
        const int nx = V.d.nx;
        const FT wyz = s.wy[row / S] * s.wz[row % S];
        const int64_t cell0 = (int64_t)nx * (y + (int64_t)V.d.ny * z);
        FT* F = static_cast<FT*>(V.F);
        if (s.gx + S <= nx) {
            const int64_t e0 = 3 * (cell0 + s.gx);
            if constexpr (sizeof(FT) == 4) {
                const int o = (int)(e0 & 3);
                float w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int e = 4 * j + k - o;
                    w[k] = e >= 0 && e < 3 * S ? s.p[e] * wyz : 0.0f;
                }
                if (4 * j - o < 3 * S) atomicAdd(reinterpret_cast<float4*>(F + (e0 - o)) + j, make_float4(w[0], w[1], w[2], w[3]));
            } else {
                atomicAdd(F + e0 + j, s.p[j] * wyz);
            }
        } else {  // the run wraps periodically along x: value by value
            const int e0 = sizeof(FT) == 4 ? 4 * j : j, e1 = min(sizeof(FT) == 4 ? e0 + 4 : e0 + 1, 3 * S);
            for (int e = e0; e < e1; ++e) {
                const int x = (s.gx + e / 3) % nx;
                atomicAdd(F + 3 * (cell0 + x) + e % 3, s.p[e] * wyz);
            }
        }
    }
}

template <class FT, int S, bool BATCH>
__global__ void __launch_bounds__(kSpreadThreads) k_spread_rows(IbView v1, const IbView* __restrict__ views,
                                                                const int* __restrict__ vinst, int nvert) {
    __shared__ SpreadTile<FT, S> T;
    const int g = blockIdx.x * kSpreadVerts + (threadIdx.x & 31);
    auto view = [&](int inst) -> const IbView& { return BATCH ? views[inst] : v1; };
    int v = -1, inst = 0;
    FT f[3] = {FT(0), FT(0), FT(0)};
    if (threadIdx.x < 96 && g < nvert) {
        if (BATCH) inst = vinst[g];
        const IbView& V = view(inst);
        v = BATCH ? g - V.vbase : g;
        if (threadIdx.x < 32)
            for (int q = 0; q < 3; ++q) f[q] = (FT)V.force[3 * v + q];
    }
    spread_tile<FT, S>(T, view, v, inst, f);
}

// Deterministic spreading.  Every (vertex, stencil node) pair becomes an entry keyed by its
// target cell; a stable radix sort groups the entries of a cell in vertex order, and one
// thread per cell sums its contributions in that order onto the body force already in F.
// The result does not depend on scheduling (the atomic path does, in its last bits).
// Entries that spread nowhere carry the key n (one past the last cell), so the sort needs
// only ceil(log2(n + 1)) key bits.
__host__ __device__ inline int key_bits(int64_t n) {
    int b = 1;
    while (((int64_t)1 << b) <= n) ++b;
    return b;
}

// The two kernels of a lattice's own spreading: its buffers hold a record of every vertex (the weights of
// the three axes and the force in the field's type), so that an entry's share is three products of L2
// reads.  Bound by the sort and by the reduction's scattered reads.  With the weights evaluated again by
// every entry from the FP64 position, the reduction was bound by the FP64 pipe: 166,920 vertices (4.5 M
// entries, FP32 field) 1468 us, now 89 us; the keys, written by one thread per vertex, 69 us, now
// 23 us.
template <class FT, int S>
struct SpreadRecord {
    FT w[3][S];
    FT f[3];
};

template <class FT, int S>
__global__ void __launch_bounds__(kSpreadThreads) k_spread_entries(LatticeDesc d, IbDesc ib, int nvert,
                                                                   const double* __restrict__ pos,
                                                                   const double* __restrict__ force,
                                                                   FT* __restrict__ rec, uint32_t* __restrict__ keys,
                                                                   uint32_t* __restrict__ ids, int4* __restrict__ lo_out) {
    constexpr int S3 = S * S * S, RW = sizeof(SpreadRecord<FT, S>) / sizeof(FT);
    __shared__ SpreadRecord<FT, S> sr[kSpreadVerts];
    __shared__ int node[kSpreadVerts][3][S];  // support nodes per axis, -1: none
    const int g0 = blockIdx.x * kSpreadVerts, cnt = min(kSpreadVerts, nvert - g0);
    if ((int)threadIdx.x < cnt) {
        const int t = threadIdx.x, v = g0 + t;
        const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
        const bool inside = inside_envelope(d, ib.dirac, p);
        const int off = (int)ib.offset, N[3] = {d.nx, d.ny, d.nz}, per[3] = {d.px, d.py, d.pz};
        int lo_rec[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double x = p[a] - ib.offset;
            const int64_t lo = (int64_t)ceil(x - half_support(ib.dirac));
#pragma unroll
            for (int m = 0; m < S; ++m) {
                sr[t].w[a][m] = axis_weight<FT>(S == 4 ? BIB_DIRAC_PESKIN : BIB_DIRAC_ROMA, lo, x, m);
                node[t][a][m] = inside ? remap_global(per[a], N[a], lo + m, off) : -1;
            }
            lo_rec[a] = inside ? record_lo(per[a], N[a], lo, off) : 0;
            sr[t].f[a] = (FT)force[3 * v + a];
        }
        if (lo_out) lo_out[v] = make_int4(lo_rec[0], lo_rec[1], lo_rec[2], inside ? 1 : 0);
    }
    __syncthreads();
    const FT* flat = reinterpret_cast<const FT*>(sr);
    for (int i = threadIdx.x; i < cnt * RW; i += kSpreadThreads) rec[(int64_t)g0 * RW + i] = flat[i];
    for (int i = threadIdx.x; i < cnt * S3; i += kSpreadThreads) {
        const int t = i / S3, m = i - t * S3;
        const int gx = node[t][0][m / (S * S)], gy = node[t][1][(m / S) % S], gz = node[t][2][m % S];
        const int64_t e = (int64_t)g0 * S3 + i;
        keys[e] = gx >= 0 && gy >= 0 && gz >= 0 ? (uint32_t)(gx + (int64_t)d.nx * (gy + (int64_t)d.ny * gz)) : (uint32_t)d.n;
        ids[e] = (uint32_t)e;
    }
}

template <class FT, int S>
__global__ void __launch_bounds__(128) k_spread_sum(int64_t n, int64_t nentries, const uint32_t* __restrict__ keys,
                                                     const uint32_t* __restrict__ ids,
                                                     const SpreadRecord<FT, S>* __restrict__ rec, FT* __restrict__ F) {
    constexpr int S3 = S * S * S;
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= nentries) return;
    const uint32_t key = keys[p];
    if (key == (uint32_t)n || (p > 0 && keys[p - 1] == key)) return;  // not the head of a cell's run
    FT* out = F + 3 * (int64_t)key;
    FT acc[3] = {out[0], out[1], out[2]};
    for (int64_t q = p; q < nentries && keys[q] == key; ++q) {
        const uint32_t e = ids[q], v = e / S3, m = e % S3;
        const SpreadRecord<FT, S>& r = rec[v];
        const FT wt = (r.w[0][m / (S * S)] * r.w[1][(m / S) % S]) * r.w[2][m % S];
        acc[0] += wt * r.f[0];
        acc[1] += wt * r.f[1];
        acc[2] += wt * r.f[2];
    }
    out[0] = acc[0];
    out[1] = acc[1];
    out[2] = acc[2];
}

// The same entries and sums without records, for the spreading that allocates nothing.
__global__ void __launch_bounds__(128) k_spread_keys(LatticeDesc d, IbDesc ib, int nvert, const double* __restrict__ pos,
                                                      uint32_t* __restrict__ keys, uint32_t* __restrict__ ids) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvert) return;
    const int s = support(ib.dirac), s3 = s * s * s;
    const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
    const bool inside = inside_envelope(d, ib.dirac, p);
    const int off = (int)ib.offset;
    const double h = half_support(ib.dirac);
    int64_t lo[3];
    for (int a = 0; a < 3; ++a) lo[a] = (int64_t)ceil(p[a] - ib.offset - h);
    for (int m = 0; m < s3; ++m) {
        const int a = m / (s * s), b = (m / s) % s, c = m % s;
        const int gx = remap_global(d.px, d.nx, lo[0] + a, off);
        const int gy = remap_global(d.py, d.ny, lo[1] + b, off);
        const int gz = remap_global(d.pz, d.nz, lo[2] + c, off);
        const bool ok = inside && gx >= 0 && gy >= 0 && gz >= 0;
        keys[(int64_t)v * s3 + m] = ok ? (uint32_t)(gx + (int64_t)d.nx * (gy + (int64_t)d.ny * gz)) : (uint32_t)d.n;
        ids[(int64_t)v * s3 + m] = (uint32_t)((int64_t)v * s3 + m);
    }
}

template <class FT>
__global__ void __launch_bounds__(128) k_spread_reduce(LatticeDesc d, IbDesc ib, int64_t nentries,
                                                        const uint32_t* __restrict__ keys, const uint32_t* __restrict__ ids,
                                                        const double* __restrict__ pos, const double* __restrict__ force,
                                                        FT* __restrict__ F) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= nentries) return;
    const uint32_t key = keys[p];
    if (key == (uint32_t)d.n || (p > 0 && keys[p - 1] == key)) return;  // not the head of a cell's run
    const int s = support(ib.dirac), s3 = s * s * s;
    const double h = half_support(ib.dirac);
    FT acc[3] = {F[key], F[d.stride + key], F[2 * d.stride + key]};
    for (int64_t q = p; q < nentries && keys[q] == key; ++q) {
        const uint32_t e = ids[q];
        const int v = (int)(e / s3), m = (int)(e % s3);
        const int a = m / (s * s), b = (m / s) % s, c = m % s;
        const double pr[3] = {pos[3 * v] - ib.offset, pos[3 * v + 1] - ib.offset, pos[3 * v + 2] - ib.offset};
        FT w[3];
        const int sel[3] = {a, b, c};
        for (int ax = 0; ax < 3; ++ax) {
            const int64_t lo = (int64_t)ceil(pr[ax] - h);
            w[ax] = axis_weight<FT>(ib.dirac, lo, pr[ax], sel[ax]);
        }
        const FT wt = (w[0] * w[1]) * w[2];
        acc[0] += wt * (FT)force[3 * v];
        acc[1] += wt * (FT)force[3 * v + 1];
        acc[2] += wt * (FT)force[3 * v + 2];
    }
    F[key] = acc[0];
    F[d.stride + key] = acc[1];
    F[2 * d.stride + key] = acc[2];
}

// ---------------------------------------------------------------- interaction forces
// MorsePotential::eval / SpringPotential::operator() (fsi/Potentials.h:29-71), FP64
__device__ __forceinline__ double potential_eval(const PotentialDev& p, double d) {
    if (p.kind == BIB_POTENTIAL_MORSE) {
        if (d < 0) d = 0.0;
        const double x = exp(p.beta * (p.r0 - d));
        return 2 * p.beta * p.strength * x * (x - 1);
    }
    if (p.kind == BIB_POTENTIAL_SPRING) return (p.r0 - d) * p.strength;
    return 0.0;
}

// Sum of the wall-interaction decorators on a vertex at p (WallInteraction::apply_force,
// ForceDecorator.hh:25-32, with ParallelPlatesBoundary, Boundary.h:305-365): for the nearer
// plate at distance dist <= r0, force -= phi(dist) * outward normal.
__device__ __forceinline__ void wall_force(const Interactions& I, const double* p, double* f) {
    f[0] = f[1] = f[2] = 0.0;
    for (int w = 0; w < I.nwall; ++w) {
        const int a = I.wall_axis[w];
        if (a == 3) {  // PipeBoundary: distance_to_boundary and get_normal, Boundary.h:158-161, 245-249
            const double dy = p[1] - I.wall_lo[w], dz = p[2] - I.wall_hi[w];
            const double rr = sqrt(dy * dy + dz * dz);
            const double dist = I.wall_r[w] - rr;
            if (dist <= I.wall[w].r0) {
                // the normal (0, dy, dz) / |.| of get_normal: on the axis (rr = 0) every component,
                // the x one included, is 0/0, as in the reference
                const double phi = potential_eval(I.wall[w], dist);
                f[0] -= phi * (0.0 / rr);
                f[1] -= phi * (dy / rr);
                f[2] -= phi * (dz / rr);
            }
            continue;
        }
        const double r = p[a], lo = I.wall_lo[w], hi = I.wall_hi[w];
        const bool lower = r < 0.5 * (lo + hi);
        const double dist = lower ? r - lo : hi - r;
        if (dist <= I.wall[w].r0) {
            const double phi = potential_eval(I.wall[w], dist);
            f[a] -= lower ? -phi : phi;
        }
    }
}

// ---------------------------------------------------------------- membrane mechanics
template <class M>
struct V3 {
    M x, y, z;
};
template <class M>
__device__ __forceinline__ V3<M> mk3(M a, M b, M c) { return V3<M>{a, b, c}; }
template <class M>
__device__ __forceinline__ V3<M> operator+(V3<M> a, V3<M> b) { return mk3(a.x + b.x, a.y + b.y, a.z + b.z); }
template <class M>
__device__ __forceinline__ V3<M> operator-(V3<M> a, V3<M> b) { return mk3(a.x - b.x, a.y - b.y, a.z - b.z); }
template <class M>
__device__ __forceinline__ V3<M> operator*(M s, V3<M> a) { return mk3(s * a.x, s * a.y, s * a.z); }
template <class M>
__device__ __forceinline__ M dot3(V3<M> a, V3<M> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <class M>
__device__ __forceinline__ M norm3(V3<M> a) { return fast_sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
// a / s by one reciprocal (approximate in FP32)
template <class M>
__device__ __forceinline__ V3<M> div3(V3<M> a, M s) {
    return fast_rcp(s) * a;
}
template <class M>
__device__ __forceinline__ V3<M> cross3(V3<M> a, V3<M> b) {
    return mk3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// Element force consumers: AtomicSink accumulates every corner force into shared memory
// (order of summation left to the hardware); GatherSink keeps the contributions to one
// vertex, in the order the elements are visited (deterministic).
template <class M>
struct AtomicSink {
    M* sf;
    __device__ __forceinline__ void operator()(int v, V3<M> f) const {
        atomicAdd(sf + 3 * v, f.x);
        atomicAdd(sf + 3 * v + 1, f.y);
        atomicAdd(sf + 3 * v + 2, f.z);
    }
};
template <class M>
struct GatherSink {
    int target;
    V3<M> acc;
    __device__ __forceinline__ void operator()(int v, V3<M> f) {
        if (v == target) acc = acc + f;
    }
};

// Vertex positions as the element kernels see them.  GlobalPos reads the FP64 positions
// (relative to c, exact FP64 subtraction, then rounding to M); SharedPos reads a copy of
// the particle's relative positions staged in shared memory.
template <class M>
struct GlobalPos {
    const double* pos;  // particle's first vertex
    double c[3];
    __device__ __forceinline__ V3<M> operator()(int v) const {
        return mk3<M>((M)(pos[3 * v] - c[0]), (M)(pos[3 * v + 1] - c[1]), (M)(pos[3 * v + 2] - c[2]));
    }
};
template <class M>
struct SharedPos {
    const M* sp;
    __device__ __forceinline__ V3<M> operator()(int v) const { return mk3<M>(sp[3 * v], sp[3 * v + 1], sp[3 * v + 2]); }
};

// Per-particle constants of the element kernels, evaluated once per thread in the
// element precision M (the FP64 expressions are the reference's, so M = double gives the
// same values as evaluating them per element).
template <class M>
struct MemCoef {
    M G, C;            // capsule shear modulus and area-dilation ratio
    M kb;              // bending modulus
    M k_area_local;
    M df_area_global;  // k_area_global (A0 - A) / A0
    M df_vol6;         // k_volume (V_desired - V) / V_desired / 6
};
template <class M>
__device__ __forceinline__ MemCoef<M> mem_coef(const ParticleDev& P, double area, double volume) {
    MemCoef<M> k;
    k.G = (M)P.prm[BIB_P_G];
    k.C = (M)P.prm[BIB_P_C];
    k.kb = (M)P.prm[BIB_P_K_BEND];
    k.k_area_local = (M)P.prm[BIB_P_K_AREA_LOCAL];
    k.df_area_global = (M)(P.prm[BIB_P_K_AREA_GLOBAL] * (P.A0 - area) / P.A0);
    k.df_vol6 = (M)(P.prm[BIB_P_K_VOLUME] * (P.prm[BIB_P_VOL_DESIRED] - volume) / P.prm[BIB_P_VOL_DESIRED]) / M(6);
    return k;
}
// Rest state of one triangle at hand (the patch kernel), in place of the particle's tables.
struct TriRest {
    float4 rest;
    float area;
};
template <class M>
struct Rest4 {
    M x, y, z, w;
};
template <class M>
__device__ __forceinline__ Rest4<M> rest_of(const ParticleDev& P, int t) {
    if constexpr (sizeof(M) == sizeof(double)) {
        const double2 a = reinterpret_cast<const double2*>(P.tri_rest)[2 * t], b = reinterpret_cast<const double2*>(P.tri_rest)[2 * t + 1];
        return {a.x, a.y, b.x, b.y};
    } else {
        const float4 r = reinterpret_cast<const float4*>(P.tri_rest_f)[t];
        return {r.x, r.y, r.z, r.w};
    }
}
template <class M>
__device__ __forceinline__ Rest4<M> rest_of(const TriRest& R, int) {
    return {R.rest.x, R.rest.y, R.rest.z, R.rest.w};
}
template <class M>
__device__ __forceinline__ M tri_area_of(const TriRest& R, int) {
    return R.area;
}
template <class M>
__device__ __forceinline__ M tri_area_of(const ParticleDev& P, int t) {
    return sizeof(M) == sizeof(double) ? (M)P.tri_area[t] : (M)P.tri_area_f[t];
}
template <class M>
__device__ __forceinline__ M pair_c(const ParticleDev& P, int p, int k) {
    return sizeof(M) == sizeof(double) ? (M)P.pair_cs[2 * p + k] : (M)P.pair_cs_f[2 * p + k];
}

// DeformableCapsuleParticle::compute_forces for one triangle, src/fsi/DeformableCapsule.hh:68-148
// (with the reference's c = l' sin(phi) / (l' sin(phi0)), line 96).  The rest-state lengths
// and angle come from the FP64 rest mesh (M = double) or its FP32 copies.
template <class M, class PD, class PS, class Sink>
__device__ void capsule_triangle(const PD& P, int t, int4 ti, const PS& ps, int skalak, const MemCoef<M>& k,
                                 Sink& sk) {
    const int i0 = ti.x, i1 = ti.y, i2 = ti.z;
    const V3<M> p0 = ps(i0), p1 = ps(i1), p2 = ps(i2);
    const V3<M> e0 = p1 - p0, e1 = p2 - p0;
    const Rest4<M> r0 = rest_of<M>(P, t);
    const M l0 = r0.x, l0p = r0.y, cos_phi_0 = r0.z, sin_phi_0 = r0.w;
    // The forces with the corner-independent scalars gathered: every gradient of
    // D11, D22, D12 (hence of I1, I2) is a combination of the corner gradients of
    // l, l' and cos(phi) (gl, glp, gc below), so f_i = pref (Cl gl_i + Cp glp_i + Cq gc_i);
    // reciprocals are taken once (FP64: a chain of divisions per gradient bound a warp at 36.9 us).
    const M l = norm3(e0), lp = norm3(e1);
    const M e0e1 = dot3(e0, e1), cr = norm3(cross3(e0, e1));
    const M rl = fast_rcp(l), rlp = fast_rcp(lp), rl0 = fast_rcp(l0), rl0p = fast_rcp(l0p), rs0 = fast_rcp(sin_phi_0);
    const M rllp = rl * rlp;
    const M sin_phi = cr * rllp, cos_phi = e0e1 * rllp;
    const M a = l * rl0;
    const M b = (lp * cos_phi * rl0p - l * cos_phi_0 * rl0) * rs0;
    const M c = sin_phi * rs0;
    const M D11 = (a * a - M(1)) * M(0.5);
    const M D22 = (b * b + c * c - M(1)) * M(0.5);
    const M D12 = a * b * M(0.5);
    const M I1 = M(2) * (D11 + D22);
    const M I2 = I1 + M(4) * (D11 * D22 - D12 * D12);
    M w1, w2;
    if (skalak) {
        w1 = I1 + M(1);
        w2 = k.C * I2 - M(1);
    } else {
        const M q = M(1) + I2;
        w1 = M(1);
        w2 = -fast_rcp(q * q);
    }
    const M A11 = l * rl0 * rl0, s2 = rs0 * rs0;
    const M k22p = s2 * (lp * rl0p * rl0p - l * cos_phi * cos_phi_0 * rl0 * rl0p);
    const M k22l = s2 * (l * cos_phi_0 * cos_phi_0 * rl0 * rl0 - lp * cos_phi * cos_phi_0 * rl0p * rl0);
    const M k22c = -s2 * l * lp * cos_phi_0 * rl0 * rl0p;
    const M k12 = M(0.5) * rl0p * rs0;
    const M k12l = k12 * (lp * cos_phi * rl0p - M(2) * l * cos_phi_0 * rl0);
    const M k12p = k12 * l * cos_phi * rl0p, k12c = k12 * l * lp * rl0p;
    const M al = M(2) + M(4) * D22, be = M(2) + M(4) * D11, ga = M(8) * D12;
    const M Cl = M(2) * w1 * (A11 + k22l) + w2 * (al * A11 + be * k22l - ga * k12l);
    const M Cp = M(2) * w1 * k22p + w2 * (be * k22p - ga * k12p);
    const M Cq = M(2) * w1 * k22c + w2 * (be * k22c - ga * k12c);
    const M t3 = e0e1 * rl * rl * rllp, t4 = e0e1 * rllp * rlp * rlp;
    const M pref = -k.G * M(0.5) * tri_area_of<M>(P, t);
    const V3<M> gl1 = rl * e0, glp2 = rlp * e1;
    const V3<M> gc0 = (t3 - rllp) * e0 + (t4 - rllp) * e1, gc1 = rllp * e1 - t3 * e0, gc2 = rllp * e0 - t4 * e1;
    sk(i0, pref * (M(-1) * (Cl * gl1 + Cp * glp2) + Cq * gc0));
    sk(i1, pref * (Cl * gl1 + Cq * gc1));
    sk(i2, pref * (Cp * glp2 + Cq * gc2));
}

// RBCParticle link term (WLC + POW), src/fsi/RBCParticle.hh:148-169 with
// RBCParameters::in_plane_ks_kp (RBCParticle.hh:27-44), m = 2, x0 = 1/2.2.
template <class M, class PS, class Sink>
__device__ void rbc_link(const ParticleDev& P, int l, const PS& ps, Sink& sk) {
    const double x0 = 1. / 2.2;
    const double ks_c1 = 0.25 * (6. * x0 + (3 * x0 * x0 - 2 * x0 * x0 * x0) / ((1 - x0) * (1 - x0)));
    const double ks_c2 = x0 / (2. * (1 - x0) * (1 - x0) * (1 - x0)) + 0.25 * (1. - 1. / ((1 - x0) * (1 - x0)));
    const double l0 = P.link_len[l];
    const double kp_c1 = -1. / (l0 * l0), kp_c2 = 3. / (l0 * l0);
    const double G_lhs = 4. * l0 * P.prm[BIB_P_SHEAR_MODULUS] / sqrt(3.0);
    const double den = ks_c1 * kp_c2 - ks_c2 * kp_c1;
    const M ks = (M)(-kp_c1 * G_lhs / den), kp = (M)(ks_c1 * G_lhs / den);
    const int a = P.links[2 * l], b = P.links[2 * l + 1];
    const V3<M> dv = ps(a) - ps(b);
    const M L = norm3(dv);
    const M x = L / (M)(l0 * 2.2);
    const M df = M(-0.25) * ks * (M(6) * x + (M(3) * x * x - M(2) * x * x * x) / ((M(1) - x) * (M(1) - x))) + kp / (L * L);
    const V3<M> fv = (df / L) * dv;
    sk(a, fv);
    sk(b, M(-1) * fv);
}

// RBCParticle triangle terms: global + local area and volume penalties,
// src/fsi/RBCParticle.hh:175-213 with tri::triangle_area_and_gradient and
// tri::grad_signed_volume (TriangleUtils.h:58-120).  The volume gradient is
// translation invariant on a closed surface, so it is taken relative to the centre.
template <class M, class PD, class PS, class Sink>
__device__ void rbc_triangle(const PD& P, int t, int4 ti, const PS& ps, const MemCoef<M>& k, Sink& sk) {
    const int i0 = ti.x, i1 = ti.y, i2 = ti.z;
    const V3<M> v0 = ps(i0), v1 = ps(i1), v2 = ps(i2);
    const M v01v11 = v0.y - v1.y, v02v22 = v0.z - v2.z, v02v12 = v0.z - v1.z;
    const M v01v21 = v0.y - v2.y, v00v20 = v0.x - v2.x, v00v10 = v0.x - v1.x;
    const M a = v01v11 * v02v22 - v02v12 * v01v21;
    const M b = v02v12 * v00v20 - v00v10 * v02v22;
    const M c = v00v10 * v01v21 - v01v11 * v00v20;
    const M la = M(0.5) * fast_sqrt(a * a + b * b + c * c);
    const M denom = fast_div(M(1), M(4) * la);
    const V3<M> g0 = mk3<M>((b * (v2.z - v1.z) + c * (v1.y - v2.y)) * denom, (a * (v1.z - v2.z) + c * (v2.x - v1.x)) * denom,
                            (a * (v2.y - v1.y) + b * (v1.x - v2.x)) * denom);
    const V3<M> g1 = mk3<M>((b * v02v22 + c * (v2.y - v0.y)) * denom, (a * (v2.z - v0.z) + c * v00v20) * denom,
                            (a * v01v21 + b * (v2.x - v0.x)) * denom);
    const V3<M> g2 = mk3<M>((b * (v1.z - v0.z) + c * v01v11) * denom, (a * v02v12 + c * (v1.x - v0.x)) * denom,
                            (a * (v1.y - v0.y) + b * v00v10) * denom);
    // the global penalty differences are evaluated once per particle, in FP64
    const M a0t = tri_area_of<M>(P, t);
    M df_area = k.df_area_global;
    df_area += fast_div(k.k_area_local * (a0t - la), a0t);
    sk(i0, df_area * g0);
    sk(i1, df_area * g1);
    sk(i2, df_area * g2);
    sk(i0, k.df_vol6 * cross3(v1, v2));
    sk(i1, k.df_vol6 * cross3(v2, v0));
    sk(i2, k.df_vol6 * cross3(v0, v1));
}

// Dihedral bending of one adjacent-triangle pair, src/fsi/RBCParticle.hh:217-246 with
// tri::grad_angle_between_pair (TriangleUtils.h:139-164).
template <class M, class PS, class Sink>
__device__ void rbc_pair(const ParticleDev& P, int p, const PS& ps, const MemCoef<M>& k, Sink& sk) {
    const int4 qq = __ldg(reinterpret_cast<const int4*>(P.pairs) + p);
    const int q[4] = {qq.x, qq.y, qq.z, qq.w};
    const V3<M> v0 = ps(q[0]), v1 = ps(q[1]), v2 = ps(q[2]), v3 = ps(q[3]);
    const V3<M> e0 = v1 - v0, e1 = v2 - v0, e2 = v3 - v0;
    const M e1n = norm3(e1);
    const V3<M> e1u = div3(e1, e1n);
    const V3<M> n1 = cross3(e0, e1), n2 = cross3(e1, e2);
    const M n1n = norm3(n1), n2n = norm3(n2);
    const V3<M> n1u = div3(n1, n1n), n2u = div3(n2, n2n);
    const M cos_t = dot3(n1u, n2u);
    const M sin_t = (dot3(n1 - n2, v1 - v3) > M(0) ? M(1) : M(-1)) * norm3(cross3(n1u, n2u));
    M c0, c1;
    if constexpr (sizeof(M) == sizeof(float)) {
        const float2 cs = __ldg(reinterpret_cast<const float2*>(P.pair_cs_f) + p);
        c0 = cs.x, c1 = cs.y;
    } else {
        c0 = pair_c<M>(P, p, 0), c1 = pair_c<M>(P, p, 1);
    }
    const M pref = k.kb * (-c0 * sin_t + c1 * cos_t);
    sk(q[0], pref * (fast_div(dot3(e1u, e1 - e2), n2n) * n2u + fast_div(dot3(e1u, e1 - e0), n1n) * n1u));
    sk(q[1], pref * (fast_div(-e1n, n1n) * n1u));
    sk(q[2], pref * (fast_div(dot3(e1u, e2), n2n) * n2u + fast_div(dot3(e1u, e0), n1n) * n1u));
    sk(q[3], pref * (fast_div(-e1n, n2n) * n2u));
}

// Forces on the three corners of one triangle, summed in registers and handed on once.
template <class M>
struct CornerSink {
    int id[3];
    V3<M> f[3];
    __device__ __forceinline__ void operator()(int v, V3<M> g) {
        if (v == id[0]) f[0] = f[0] + g;
        else if (v == id[1]) f[1] = f[1] + g;
        else f[2] = f[2] + g;
    }
};

// One CTA per particle: vertex forces at X_n (ParticleBase3D::reset_forces +
// compute_forces), accumulated in shared memory.
template <class M>
__device__ __forceinline__ void membrane_block(const ParticleDev& P, const IbView& V, unsigned char* smem_raw) {
    M* sf = reinterpret_cast<M*>(smem_raw);
    const double* __restrict__ pos = V.pos;
    double* __restrict__ force = V.force;
    const double* st = V.stats + STATS * P.lpid;
    const double area = st[0], volume = st[1];
    // gridDim.y CTAs share the elements of one particle: each sums its share in shared memory
    // and adds it to the force array (seeded by k_force_seed) with atomics
    const int split = gridDim.y;
    const int e0 = blockIdx.y * blockDim.x + threadIdx.x, es = split * blockDim.x;
    // the force decorators come first (ImmersedBoundaryDynamics_forces.hh:293-296)
    if (split == 1 && V.inter.nwall > 0) {
        for (int i = threadIdx.x; i < P.nv; i += blockDim.x) {
            double fw[3];
            wall_force(V.inter, pos + 3LL * (P.v0 + i), fw);
            sf[3 * i] = (M)fw[0];
            sf[3 * i + 1] = (M)fw[1];
            sf[3 * i + 2] = (M)fw[2];
        }
    } else {
        for (int i = threadIdx.x; i < 3 * P.nv; i += blockDim.x) sf[i] = M(0);
    }
    // FP64 element arithmetic uses absolute positions as the reference does; reduced
    // precision stages the positions relative to the centre of mass in shared memory
    // (exact FP64 subtraction, then rounding) so the element loops read them from there.
    const bool rel = sizeof(M) < sizeof(double);
    M* sp = sf + 3 * P.nv;
    if (rel) {
        const double* pp = pos + 3LL * P.v0;
        const double c[3] = {st[2], st[3], st[4]};
        for (int i = threadIdx.x; i < P.nv; i += blockDim.x) {
            sp[3 * i] = (M)(pp[3 * i] - c[0]);
            sp[3 * i + 1] = (M)(pp[3 * i + 1] - c[1]);
            sp[3 * i + 2] = (M)(pp[3 * i + 2] - c[2]);
        }
    }
    // the per-particle constants (FP64 divisions) once per CTA
    __shared__ MemCoef<M> kc;
    if (threadIdx.x == 0) kc = mem_coef<M>(P, area, volume);
    __syncthreads();
    AtomicSink<M> sk{sf};
    const int skalak = P.model != BIB_MODEL_CAPSULE_NEOHOOKEAN;
    const bool capsule = P.model == BIB_MODEL_CAPSULE_NEOHOOKEAN || P.model == BIB_MODEL_CAPSULE_SKALAK ||
                         P.model == BIB_MODEL_SKALAK_BENDING;
    const bool rbc_terms = P.model == BIB_MODEL_RBC_WLCPOW || P.model == BIB_MODEL_SKALAK_BENDING;
    const MemCoef<M> k = kc;
    auto run = [&](const auto& ps) {
        // triangle terms (capsule law and RBC area / volume penalties) of one triangle are
        // summed per corner before they reach the shared accumulators
        if (capsule || rbc_terms)
            for (int t = e0; t < P.nt; t += es) {
                const V3<M> z = mk3<M>(0, 0, 0);
                const int4 ti = __ldg(reinterpret_cast<const int4*>(P.tri4) + t);
                CornerSink<M> cs{{ti.x, ti.y, ti.z}, {z, z, z}};
                if (capsule) capsule_triangle<M>(P, t, ti, ps, skalak, k, cs);
                if (rbc_terms) rbc_triangle<M>(P, t, ti, ps, k, cs);
                for (int c = 0; c < 3; ++c) sk(cs.id[c], cs.f[c]);
            }
        if (P.model == BIB_MODEL_RBC_WLCPOW)
            for (int l = e0; l < P.nl; l += es) rbc_link<M>(P, l, ps, sk);
        if (rbc_terms)
            for (int p = e0; p < P.np; p += es) rbc_pair<M>(P, p, ps, k, sk);
    };
    if (rel) run(SharedPos<M>{sp});
    else run(GlobalPos<M>{pos + 3LL * P.v0, {0.0, 0.0, 0.0}});
    __syncthreads();
    if (split == 1) {
        for (int i = threadIdx.x; i < 3 * P.nv; i += blockDim.x) force[3LL * P.v0 + i] = (double)sf[i];
    } else {
        for (int i = threadIdx.x; i < 3 * P.nv; i += blockDim.x)
            if (sf[i] != M(0)) atomicAdd(force + 3LL * P.v0 + i, (double)sf[i]);
    }
}

// The vertex forces before a split membrane launch adds into them: the wall-interaction
// decorators, or zero.
__global__ void __launch_bounds__(128) k_force_seed(IbView V) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V.nvert) return;
    double fw[3] = {0.0, 0.0, 0.0};
    if (V.inter.nwall > 0) wall_force(V.inter, V.pos + 3LL * v, fw);
    V.force[3LL * v] = fw[0];
    V.force[3LL * v + 1] = fw[1];
    V.force[3LL * v + 2] = fw[2];
}

template <class M, bool BATCH>
__global__ void __launch_bounds__(512) k_membrane(const ParticleDev* __restrict__ parts, IbView v1,
                                                   const IbView* __restrict__ views) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const ParticleDev& P = parts[blockIdx.x];
    membrane_block<M>(P, BATCH ? views[P.inst] : v1, smem_raw);
}

// Bending across one edge of a triangle, its share on the triangle's own corners: v1 is the corner
// opposite the edge v0 v2, v3 the neighbour's vertex across it, n1 = (v1 - v0) x (v2 - v0) with its length
// n1n.  The forces are along n1 (rbc_pair: the terms of n1u), as factors of its unit vector on v0, v1, v2.
template <class M>
__device__ __forceinline__ void bend_side(V3<M> v0, V3<M> v1, V3<M> v2, V3<M> v3, V3<M> n1, M n1n, V3<M> n1u, M kb, M c0, M c1,
                                          M* s) {
    const V3<M> e0 = v1 - v0, e1 = v2 - v0, e2 = v3 - v0;
    const M e1n = norm3(e1);
    const V3<M> e1u = div3(e1, e1n);
    const V3<M> n2 = cross3(e1, e2);
    const V3<M> n2u = div3(n2, norm3(n2));
    const M cos_t = dot3(n1u, n2u);
    const M sin_t = (dot3(n1 - n2, v1 - v3) > M(0) ? M(1) : M(-1)) * norm3(cross3(n1u, n2u));
    const M pref = fast_div(kb * (-c0 * sin_t + c1 * cos_t), n1n);
    s[0] = pref * dot3(e1u, e1 - e0);
    s[1] = pref * -e1n;
    s[2] = pref * dot3(e1u, e0);
}

// Membrane forces by patches (reduced precision), one CTA per patch of 32 owned vertices.  The CTA stages
// the positions that the patch's triangles and their neighbours need, evaluates every triangle at an owned
// vertex once (capsule law, area and volume penalties, and the triangle's own share of the bending across
// its three edges) into shared memory, and adds up the corners of each owned vertex in triangle order:
// no atomics, the same bits on every run.  SPREAD: the forces go straight on into the force field.
// Bound by instruction issue, and by the FP64 pipe for the staging and the delta offsets.  A triangle on a
// patch boundary is evaluated by each of its patches (1.5 evaluations per triangle).  One CTA per particle
// with a shared-memory float atomic for each corner of each triangle and adjacent-triangle pair: 400 cells
// of 642 vertices 45.8 us plus 37.4 us of spreading, in one launch here 81.8; 200 cells with the 4-point kernel
// 41.2 + 34.8, here 55.7; one of 2562 vertices 20.8 + 2.3 (seeding) + 6.4, here 10.8.  One thread per vertex evaluating
// all its elements (the deterministic mode): 260 cells 199 us, here 34.5.  At 59 % of the issue slots with 7 CTAs
// per SM; 5 take 95 us for the 400 cells, 8 (64 registers, spills) the same.
template <int S, bool BATCH, bool SPREAD>
__global__ void __launch_bounds__(kSpreadThreads, 7) k_membrane_patch(const PatchJob* __restrict__ jobs,
                                                                      const ParticleDev* __restrict__ parts, IbView v1,
                                                                      const IbView* __restrict__ views) {
    static_assert(kPatchOwn == kSpreadVerts, "a patch is a tile of the spreading");
    extern __shared__ __align__(16) float dyn[];
    __shared__ SpreadTile<float, S> T;
    __shared__ double wall[3][kPatchOwn];
    __shared__ MemCoef<float> kc;
    __shared__ float own_f[3][kPatchOwn];
    __shared__ uint16_t inc_off[kPatchOwn + 1];
    const PatchJob& J = jobs[blockIdx.x];
    const ParticleDev& P = parts[J.part];
    const IbView& V = BATCH ? views[J.inst] : v1;
    const double* st = V.stats + STATS * J.lpid;
    const double* pos = V.pos + 3LL * J.v0;
    const int* verts = J.verts;
    const int own = J.own, all = J.all, ntris = J.ntris;
    float* sp = dyn;
    float* tf = dyn + 3 * all;
    uint16_t* inc = reinterpret_cast<uint16_t*>(tf + 9 * ntris);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the thread's first triangle is loaded along with the positions
    uint4 raw[4];
    auto load_tri = [&](int i) {
        const uint4* q = reinterpret_cast<const uint4*>(J.tris + i);
#pragma unroll
        for (int w = 0; w < 4; ++w) raw[w] = __ldg(q + w);
    };
    if ((int)threadIdx.x < ntris) load_tri(threadIdx.x);
    for (int i = threadIdx.x; i < J.nincs; i += kSpreadThreads) inc[i] = J.inc[i];
    if (threadIdx.x <= kPatchOwn) inc_off[threadIdx.x] = J.inc_off[threadIdx.x];
    // positions relative to the centre of mass: exact FP64 subtraction, then rounding
    for (int i = threadIdx.x; i < all; i += kSpreadThreads) {
        const double* p = pos + 3LL * verts[i];
        sp[3 * i] = (float)(p[0] - st[2]);
        sp[3 * i + 1] = (float)(p[1] - st[3]);
        sp[3 * i + 2] = (float)(p[2] - st[4]);
    }
    if (threadIdx.x == 0) {
        kc.G = P.pf[0];
        kc.C = P.pf[1];
        kc.kb = P.pf[2];
        kc.k_area_local = P.pf[3];
        kc.df_area_global = (float)(P.ka_a0 * (P.A0 - st[0]));
        kc.df_vol6 = (float)(P.kv_vd * (P.prm[BIB_P_VOL_DESIRED] - st[1])) / 6.0f;
    }
    // the force decorators come first (ImmersedBoundaryDynamics_forces.hh:293-296)
    if (warp == 3 && V.inter.nwall > 0 && lane < own) {
        double fw[3];
        wall_force(V.inter, pos + 3LL * verts[lane], fw);
        for (int q = 0; q < 3; ++q) wall[q][lane] = fw[q];
    }
    const int skalak = P.model != BIB_MODEL_CAPSULE_NEOHOOKEAN;
    const bool rbc_terms = P.model == BIB_MODEL_SKALAK_BENDING;
    const int v = warp < 3 && lane < own ? J.v0 + verts[lane] : -1;
    __syncthreads();
    const MemCoef<float> k = kc;
    const SharedPos<float> ps{sp};
    for (int i = threadIdx.x; i < ntris; i += kSpreadThreads) {
        if (i >= kSpreadThreads) load_tri(i);
        const int c[3] = {(int)(raw[0].x & 0xffffu), (int)(raw[0].x >> 16), (int)(raw[0].y & 0xffffu)};
        const int nb[3] = {(int)(raw[0].y >> 16), (int)(raw[0].z & 0xffffu), (int)(raw[0].z >> 16)};
        const TriRest R{make_float4(__uint_as_float(raw[1].x), __uint_as_float(raw[1].y), __uint_as_float(raw[1].z),
                                    __uint_as_float(raw[1].w)),
                        __uint_as_float(raw[3].z)};
        const float bend[6] = {__uint_as_float(raw[2].x), __uint_as_float(raw[2].y), __uint_as_float(raw[2].z),
                               __uint_as_float(raw[2].w), __uint_as_float(raw[3].x), __uint_as_float(raw[3].y)};
        const V3<float> z = mk3<float>(0, 0, 0);
        CornerSink<float> cs{{c[0], c[1], c[2]}, {z, z, z}};
        const int4 ti = make_int4(c[0], c[1], c[2], 0);
        capsule_triangle<float>(R, 0, ti, ps, skalak, k, cs);
        if (rbc_terms) {
            rbc_triangle<float>(R, 0, ti, ps, k, cs);
            const V3<float> p[3] = {ps(c[0]), ps(c[1]), ps(c[2])};
            const V3<float> n = cross3(p[1] - p[0], p[2] - p[0]);
            const float nn = norm3(n);
            const V3<float> nu = div3(n, nn);
            float along[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                if (nb[e] == kNoNb) continue;
                const bool flip = (raw[0].w >> e) & 1u;  // the pair runs against the triangle: n1 turns over
                const V3<float> a = p[(e + 2) % 3], b = p[(e + 1) % 3];
                const V3<float> v0 = flip ? b : a, v2 = flip ? a : b;
                const float sign = flip ? -1.0f : 1.0f;
                float s[3];
                bend_side<float>(v0, p[e], v2, ps(nb[e]), sign * n, nn, sign * nu, k.kb, bend[2 * e], bend[2 * e + 1], s);
                along[e] += sign * s[1];
                along[(e + 2) % 3] += sign * (flip ? s[2] : s[0]);
                along[(e + 1) % 3] += sign * (flip ? s[0] : s[2]);
            }
            for (int e = 0; e < 3; ++e) cs.f[e] = cs.f[e] + along[e] * nu;
        }
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            tf[9 * i + 3 * e] = cs.f[e].x;
            tf[9 * i + 3 * e + 1] = cs.f[e].y;
            tf[9 * i + 3 * e + 2] = cs.f[e].z;
        }
    }
    __syncthreads();
    if (v >= 0) {  // one component of an owned vertex per thread
        // summed with the rounding errors beside the sum: an FP64 sum of the corners rounded once, without its
        // FP64 additions (1.5 us of the 400 cells' step against 3)
        float sum = 0.0f, err = 0.0f;
        for (int e = inc_off[lane]; e < inc_off[lane + 1]; ++e) {
            const float a = tf[3 * inc[e] + warp], s = sum + a, t = s - sum;
            err += (sum - (s - t)) + (a - t);
            sum = s;
        }
        sum += err;
        double f = (double)sum;
        if (V.inter.nwall > 0) {  // the wall interactions are FP64 and stay so in the vertex force
            f += wall[warp][lane];
            sum = (float)f;
        }
        V.force[3LL * v + warp] = f;
        own_f[warp][lane] = sum;
    }
    if (!SPREAD) return;
    __syncthreads();
    const float f[3] = {own_f[0][lane], own_f[1][lane], own_f[2][lane]};
    spread_tile<float, S>(T, [&](int) -> const IbView& { return V; }, v, 0, f);
}

// Deterministic membrane forces: one thread per vertex sums the contributions of its
// incident links, triangles and adjacent-triangle pairs, visited in the order of the
// reference's element loops (RBCParticle.hh:148-246: links, then triangles with the area
// term before the volume term, then pairs).  Each incident element is evaluated once per
// corner, so the element arithmetic is repeated 2-4 times; no atomics, bit-reproducible.
// The Skalak + bending composite sums the capsule part and the RBC part separately, as
// the reference does when both particle classes act on the same vertices.
constexpr int INC_LINK = 0, INC_TRI = 1, INC_PAIR = 2;

template <class M>
__global__ void __launch_bounds__(128) k_membrane_gather(int nvert, const int* __restrict__ vert_particle,
                                                          const ParticleDev* __restrict__ parts,
                                                          const double* __restrict__ pos, double* __restrict__ force,
                                                          const double* __restrict__ stats, Interactions inter) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nvert) return;
    const int pid = vert_particle[g];
    const ParticleDev& P = parts[pid];
    const int lv = g - P.v0;
    const double* st = stats + STATS * pid;
    const double area = st[0], volume = st[1];
    const bool rel = sizeof(M) < sizeof(double);
    const GlobalPos<M> ps{pos + 3LL * P.v0, {rel ? st[2] : 0.0, rel ? st[3] : 0.0, rel ? st[4] : 0.0}};
    const bool capsule = P.model == BIB_MODEL_CAPSULE_NEOHOOKEAN || P.model == BIB_MODEL_CAPSULE_SKALAK ||
                         P.model == BIB_MODEL_SKALAK_BENDING;
    const bool rbc_terms = P.model == BIB_MODEL_RBC_WLCPOW || P.model == BIB_MODEL_SKALAK_BENDING;
    const int skalak = P.model != BIB_MODEL_CAPSULE_NEOHOOKEAN;
    const MemCoef<M> k = mem_coef<M>(P, area, volume);
    GatherSink<M> cap{lv, mk3<M>(0, 0, 0)}, rbc{lv, mk3<M>(0, 0, 0)};
    for (int e = P.inc_off[lv]; e < P.inc_off[lv + 1]; ++e) {
        const int code = P.inc[e];
        const int type = code >> 29, id = code & ((1 << 29) - 1);
        if (type == INC_LINK) {
            if (P.model == BIB_MODEL_RBC_WLCPOW) rbc_link<M>(P, id, ps, rbc);
        } else if (type == INC_TRI) {
            const int4 ti = __ldg(reinterpret_cast<const int4*>(P.tri4) + id);
            if (capsule) capsule_triangle<M>(P, id, ti, ps, skalak, k, cap);
            if (rbc_terms) rbc_triangle<M>(P, id, ti, ps, k, rbc);
        } else if (type == INC_PAIR && rbc_terms) {
            rbc_pair<M>(P, id, ps, k, rbc);
        }
    }
    V3<M> f = P.model == BIB_MODEL_SKALAK_BENDING ? cap.acc + rbc.acc : (capsule ? cap.acc : rbc.acc);
    double fw[3] = {0.0, 0.0, 0.0};
    if (inter.nwall > 0) wall_force(inter, pos + 3LL * g, fw);
    force[3LL * g] = fw[0] + (double)f.x;
    force[3LL * g + 1] = fw[1] + (double)f.y;
    force[3LL * g + 2] = fw[2] + (double)f.z;
}

// One CTA per particle: area, signed volume and area-weighted centroid of X_{n+1}
// (DeformableParticle3D::update, DeformableParticle3D.hh:54-82), then the periodic
// centre-of-mass remap (ParticleBase3D::map_center_of_mass_to_periodic_grid,
// ParticleBase.hh:111-136).  M = double follows the reference with absolute positions.
// M = float (reduced-precision lattices) evaluates each triangle in FP32 on positions
// relative to the previous centre of mass (exact FP64 subtraction, then rounding) and
// accumulates in FP64; the signed volume of the closed surface does not depend on the
// origin.
// Sums of five per-thread values over the block into out[0..4] (shared): the partials go
// to red (5 x blockDim.x doubles), then one warp per quantity adds them up.
__device__ __forceinline__ void block_sum5(const double v[5], double* red, double* out) {
    const int n = blockDim.x, t = threadIdx.x;
#pragma unroll
    for (int k = 0; k < 5; ++k) red[k * n + t] = v[k];
    __syncthreads();
    const int lane = t & 31, nw = n >> 5;
    for (int q = t >> 5; q < 5; q += nw) {
        double s = 0.0;
        for (int i = lane; i < n; i += 32) s += red[q * n + i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) out[q] = s;
    }
    __syncthreads();
}

// Per-triangle area, signed volume and area-weighted centroid of X_{n+1}, summed over the
// triangles e0, e0 + es, ... by this CTA into sum[0..4] (shared; valid for every thread).
// M = float with STAGE: the relative positions of the whole particle are staged in sp first (one CTA for
// many triangles); without, each triangle takes its own.
template <class M, bool STAGE>
__device__ __forceinline__ void update_sums(const ParticleDev& P, const IbView& V, float* sp, double* red, double* sum,
                                            int e0, int es) {
    const double* pv = V.pos_next + 3LL * P.v0;
    const double* st = V.stats + STATS * P.lpid;
    const bool rel = sizeof(M) < sizeof(double);
    const double c0 = rel ? st[2] : 0.0, c1 = rel ? st[3] : 0.0, c2 = rel ? st[4] : 0.0;
    if (STAGE && rel) {  // one FP64 subtraction and rounding per vertex coordinate
        for (int i = threadIdx.x; i < P.nv; i += blockDim.x) {
            sp[3 * i] = (float)(pv[3 * i] - c0);
            sp[3 * i + 1] = (float)(pv[3 * i + 1] - c1);
            sp[3 * i + 2] = (float)(pv[3 * i + 2] - c2);
        }
        __syncthreads();
    }
    auto vert = [&](int i) {
        return STAGE && rel ? mk3<M>((M)sp[3 * i], (M)sp[3 * i + 1], (M)sp[3 * i + 2])
                   : mk3<M>((M)(pv[3 * i] - c0), (M)(pv[3 * i + 1] - c1), (M)(pv[3 * i + 2] - c2));
    };
    // per-thread partial sums in M (a few triangles each), block sums in FP64
    M ta = 0, tv = 0, tcx = 0, tcy = 0, tcz = 0;
    for (int t = e0; t < P.nt; t += es) {
        const int4 ti = __ldg(reinterpret_cast<const int4*>(P.tri4) + t);
        const V3<M> A = vert(ti.x), B = vert(ti.y), Cv = vert(ti.z);
        const M dA = norm3(cross3(B - A, Cv - A)) * M(0.5);
        ta += dA;
        // multiplications by 1/6 and 1/3 instead of the reference's divisions (FP64 division
        // is a long instruction sequence on this part); differences are within one ulp per term
        tv += dot3(A, cross3(B, Cv)) * (M(1) / M(6));
        const V3<M> cen = (M(1) / M(3)) * (A + B + Cv);
        tcx += cen.x * dA;
        tcy += cen.y * dA;
        tcz += cen.z * dA;
    }
    const double part[5] = {(double)ta, (double)tv, (double)tcx, (double)tcy, (double)tcz};
    block_sum5(part, red, sum);
}

// A, V and the centre from the sums (relative to the previous centre for M = float), the
// periodic centre-of-mass remap, and the shift of the vertices by whole periods.
template <class M>
__device__ __forceinline__ void update_finish(const ParticleDev& P, const IbView& V, const double* sum, double* delta) {
    const LatticeDesc& d = V.d;
    double* pos_next = V.pos_next;
    double* st = V.stats + STATS * P.lpid;
    if (threadIdx.x == 0) {
        const bool rel = sizeof(M) < sizeof(double);
        const double c0 = rel ? st[2] : 0.0, c1 = rel ? st[3] : 0.0, c2 = rel ? st[4] : 0.0;
        const double sa = sum[0], sv = sum[1];
        const double com[3] = {c0 + sum[2] / sa, c1 + sum[3] / sa, c2 + sum[4] / sa};
        const int N[3] = {d.nx, d.ny, d.nz};
        const int per[3] = {d.px, d.py, d.pz};
        double np_[3];
        for (int a = 0; a < 3; ++a) {
            np_[a] = com[a];
            if (per[a]) np_[a] = com[a] - (double)N[a] * floor((com[a] - (-0.5)) * d.inv_n[a]);
            delta[a] = np_[a] - com[a];
        }
        st[0] = sa;
        st[1] = sv;
        st[2] = np_[0];
        st[3] = np_[1];
        st[4] = np_[2];
    }
    __syncthreads();
    if (delta[0] != 0.0 || delta[1] != 0.0 || delta[2] != 0.0) {
        for (int i = threadIdx.x; i < P.nv; i += blockDim.x) {
            const int64_t g = 3LL * (P.v0 + i);
            pos_next[g] += delta[0];
            pos_next[g + 1] += delta[1];
            pos_next[g + 2] += delta[2];
        }
    }
}

template <class M>
__device__ __forceinline__ void update_block(const ParticleDev& P, const IbView& V, float* sp, double* red,
                                             double* delta) {
    __shared__ double sum[5];
    update_sums<M, true>(P, V, sp, red, sum, threadIdx.x, blockDim.x);
    update_finish<M>(P, V, sum, delta);
}

// Few particles: gridDim.y CTAs per particle write partial sums; the one that finishes last adds them in
// slice order and finishes the update (it waits for nothing: the others have left their sums and their
// ticket).  `ticket` counts the CTAs done, zero between launches.  A triangle takes its vertices from global
// memory: staging the particle in every CTA was bound by the FP64 pipe.  One membrane of 2562 vertices in
// FP32, partial sums and finish in two launches, 11.9 + 5.7 us, now 11.4.
constexpr int kMaxUpdateSplit = 64, kUpdateFew = 128;

template <class M>
__global__ void __launch_bounds__(kUpdateFew) k_update_few(const ParticleDev* __restrict__ parts, IbView v1, double* partial,
                                                           unsigned* ticket) {
    __shared__ double red[5 * kUpdateFew];
    __shared__ double sum[5], delta[3];
    __shared__ bool last;
    const ParticleDev& P = parts[blockIdx.x];
    const int split = gridDim.y;
    update_sums<M, false>(P, v1, nullptr, red, sum, blockIdx.y * kUpdateFew + threadIdx.x, split * kUpdateFew);
    double* mine = partial + (blockIdx.x * (size_t)split) * 5;
    if (threadIdx.x < 5) mine[blockIdx.y * 5 + threadIdx.x] = sum[threadIdx.x];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket + blockIdx.x, 1u) == (unsigned)split - 1u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 5) {
        double a = 0.0;
        for (int y = 0; y < split; ++y) a += __ldcg(mine + y * 5 + threadIdx.x);
        sum[threadIdx.x] = a;
    }
    if (threadIdx.x == 0) ticket[blockIdx.x] = 0;
    __syncthreads();
    update_finish<M>(P, v1, sum, delta);
}

template <class M, bool BATCH>
__global__ void __launch_bounds__(256) k_particle_update(const ParticleDev* __restrict__ parts, IbView v1,
                                                          const IbView* __restrict__ views) {
    __shared__ double red[5 * 256];
    __shared__ double delta[3];
    extern __shared__ __align__(16) float sp[];  // M = float: relative vertex positions
    const ParticleDev& P = parts[blockIdx.x];
    update_block<M>(P, BATCH ? views[P.inst] : v1, sp, red, delta);
}

// ---------------------------------------------------------------- voxelization
// RayTracer::tri_ray_intersect (fsi/RayTracer.hh:80-108) for the ray from (px, py, 0) along
// +z, in the reference's operation order and without fused multiply-adds, so the
// intersection heights (and therefore the phase field) are the reference's to the bit.
__device__ __forceinline__ double dot_nofma(const double* a, const double* b) {
    double r = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) r = __dadd_rn(r, __dmul_rn(a[d], b[d]));
    return r;
}
__device__ __forceinline__ void cross_nofma(const double* a, const double* b, double* c) {
    c[0] = __dsub_rn(__dmul_rn(a[1], b[2]), __dmul_rn(a[2], b[1]));
    c[1] = __dsub_rn(__dmul_rn(a[2], b[0]), __dmul_rn(a[0], b[2]));
    c[2] = __dsub_rn(__dmul_rn(a[0], b[1]), __dmul_rn(a[1], b[0]));
}
__device__ __forceinline__ bool tri_ray_z(const double* v0, const double* v1, const double* v2, double px, double py,
                                          double& dist) {
    const double e1[3] = {__dsub_rn(v1[0], v0[0]), __dsub_rn(v1[1], v0[1]), __dsub_rn(v1[2], v0[2])};
    const double e2[3] = {__dsub_rn(v2[0], v0[0]), __dsub_rn(v2[1], v0[1]), __dsub_rn(v2[2], v0[2])};
    const double dir[3] = {0.0, 0.0, 1.0};
    double q[3];
    cross_nofma(dir, e2, q);
    const double a = dot_nofma(e1, q);
    if (fabs(a) < DBL_EPSILON) return false;
    const double f = __drcp_rn(a);
    const double sv[3] = {__dsub_rn(px, v0[0]), __dsub_rn(py, v0[1]), __dsub_rn(0.0, v0[2])};
    const double u = __dmul_rn(f, dot_nofma(sv, q));
    if (u < 0.0) return false;
    double r[3];
    cross_nofma(sv, e1, r);
    const double v = __dmul_rn(f, dot_nofma(dir, r));
    if (v < 0.0 || __dadd_rn(u, v) > 1.0) return false;
    dist = __dmul_rn(f, dot_nofma(e2, r));
    return true;
}

// One thread per triangle, one warp per CTA (grid: particles x blocks of 32 triangles): z-rays through the integer (x, y) points of
// the triangle's xy box (RayTracer::find_intersections_z, RayTracer.hh:18-40); each hit goes
// to its (periodically wrapped) column, height wrapped into [-1/2, nz - 1/2) (ZBuffer::put,
// Arithmetic1D::remap_pos).  Columns are numbered x fastest.
// Bound by the FP64 pipe (about 80 operations per ray, 2 lanes per cycle and SM): warps spread over all
// SMs.  One 128-thread CTA per particle kept one capsule of 1280 triangles on one SM for 97 us; with 40
// one-warp CTAs the whole step of that capsule (80^3 cells, phase field) went from 250 to 127 us.
__global__ void __launch_bounds__(32) k_voxel_rays(LatticeDesc d, const ParticleDev* __restrict__ parts,
                                                     const double* __restrict__ pos, int* __restrict__ count,
                                                     double* __restrict__ zbuf, int cap, int* __restrict__ overflow) {
    const ParticleDev& P = parts[blockIdx.x];
    const double* pv = pos + 3LL * P.v0;
    const int64_t ncol = (int64_t)d.nx * d.ny;
    for (int t = blockIdx.y * blockDim.x + threadIdx.x; t < P.nt; t += gridDim.y * blockDim.x) {
        const double* v0 = pv + 3 * P.tri[3 * t];
        const double* v1 = pv + 3 * P.tri[3 * t + 1];
        const double* v2 = pv + 3 * P.tri[3 * t + 2];
        double x0 = fmin(v0[0], fmin(v1[0], v2[0])), x1 = fmax(v0[0], fmax(v1[0], v2[0]));
        double y0 = fmin(v0[1], fmin(v1[1], v2[1])), y1 = fmax(v0[1], fmax(v1[1], v2[1]));
        // a triangle wider than the lattice (or not finite) only arises from a diverged
        // membrane: flag it instead of casting rays through a runaway box
        if (!(x1 - x0 < (double)d.nx && y1 - y0 < (double)d.ny)) {
            atomicExch(overflow, 1);
            continue;
        }
        if (!d.px) x0 = fmax(x0, -1.0), x1 = fmin(x1, (double)d.nx);  // rays outside a walled axis are dropped
        if (!d.py) y0 = fmax(y0, -1.0), y1 = fmin(y1, (double)d.ny);
        const int64_t i0 = (int64_t)ceil(x0), i1 = (int64_t)floor(x1);
        const int64_t j0 = (int64_t)ceil(y0), j1 = (int64_t)floor(y1);
        for (int64_t i = i0; i <= i1; ++i)
            for (int64_t j = j0; j <= j1; ++j) {
                double z;
                if (!tri_ray_z(v0, v1, v2, (double)i, (double)j, z)) continue;
                int64_t cx = i, cy = j;
                if (d.px) cx = pmod(cx, d.nx);
                else if (cx < 0 || cx >= d.nx) continue;
                if (d.py) cy = pmod(cy, d.ny);
                else if (cy < 0 || cy >= d.ny) continue;
                if (d.pz) z = __dsub_rn(z, __dmul_rn((double)d.nz, floor(__dmul_rn(__dsub_rn(z, -0.5), d.inv_n[2]))));
                const int64_t c = cx + (int64_t)d.nx * cy;
                const int slot = atomicAdd(count + c, 1);
                if (slot < cap) zbuf[slot * ncol + c] = z;
                else atomicExch(overflow, 1);
            }
    }
}

// One thread per column: sort its heights and fill the column from below by parity
// (apply_voxelization, ImmersedBoundaryDynamics_voxelization.hh:121-161); resets the count.
// Heights of column c sit at zbuf[slot * ncol + c], so a warp reads slot e of 32 columns at once.
__global__ void __launch_bounds__(128) k_voxel_fill(LatticeDesc d, int* __restrict__ count, double* __restrict__ zbuf,
                                                     int cap, uint8_t* __restrict__ phase) {
    const int64_t ncol = (int64_t)d.nx * d.ny;
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= ncol) return;
    const int m = min(count[c], cap);
    count[c] = 0;
    double* zl = zbuf + c;
    for (int e = 1; e < m; ++e) {  // insertion sort, ascending, in place
        const double z = zl[e * ncol];
        int p = e;
        while (p > 0 && zl[(p - 1) * ncol] > z) {
            zl[p * ncol] = zl[(p - 1) * ncol];
            --p;
        }
        zl[p * ncol] = z;
    }
    const int64_t plane = ncol;
    uint8_t inside = 0;
    double z_last = -10000.0;
    for (int e = 0; e <= m; ++e) {
        const double ze = e < m ? zl[e * ncol] : 0.0;
        int64_t lo, hi;
        if (e < m) {
            lo = max((int64_t)ceil(z_last), (int64_t)0);
            hi = min((int64_t)floor(ze), (int64_t)d.nz - 1);
        } else {
            if (!(ceil(z_last) < (double)(d.nz - 1))) break;
            lo = max((int64_t)ceil(z_last), (int64_t)0);
            hi = d.nz - 1;
        }
        for (int64_t z = lo; z <= hi; ++z) phase[c + plane * z] = inside;
        if (e < m) {
            z_last = ze;
            inside ^= 1;
        }
    }
}

// ---------------------------------------------------------------- particle-particle interactions
// Pair search on a hashed cell list: cells of at least the largest cutoff, each vertex keyed
// by the hash of its cell, vertices sorted by key (stable: vertex order within a bucket).
struct PairCells {
    int nc[3];
    double cs[3];
    unsigned mask;
};

__device__ __forceinline__ int pair_cell(const LatticeDesc& d, const PairCells& g, int a, double x) {
    const int N = a == 0 ? d.nx : (a == 1 ? d.ny : d.nz);
    const int per = a == 0 ? d.px : (a == 1 ? d.py : d.pz);
    if (per) x -= (double)N * floor(x * d.inv_n[a]);
    int c = (int)floor(x / g.cs[a]);
    return c < 0 ? 0 : (c >= g.nc[a] ? g.nc[a] - 1 : c);
}
__device__ __forceinline__ unsigned cell_hash(const PairCells& g, int cx, int cy, int cz) {
    return ((unsigned)cx * 73856093u ^ (unsigned)cy * 19349663u ^ (unsigned)cz * 83492791u) & g.mask;
}

// Cell and bucket of every vertex (the cell kept for the search); the buckets of the previous step's
// sort go back to empty.
__global__ void __launch_bounds__(128) k_pp_keys(LatticeDesc d, PairCells g, int nvert, const double* __restrict__ pos,
                                                  const uint32_t* __restrict__ prev_keys, int* __restrict__ start,
                                                  int* __restrict__ end, uint32_t* __restrict__ keys,
                                                  uint32_t* __restrict__ ids, int4* __restrict__ cell) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvert) return;
    start[prev_keys[v]] = 0;
    end[prev_keys[v]] = 0;
    const double* p = pos + 3LL * v;
    const int c[3] = {pair_cell(d, g, 0, p[0]), pair_cell(d, g, 1, p[1]), pair_cell(d, g, 2, p[2])};
    keys[v] = cell_hash(g, c[0], c[1], c[2]);
    ids[v] = (uint32_t)v;
    cell[v] = make_int4(c[0], c[1], c[2], 0);
}

// Bucket bounds, and the sorted vertices' positions in FP32 with their particles for the pre-test of the
// pairs (a position more than 4 periods out becomes NaN, which the pre-test lets through).
__global__ void __launch_bounds__(128) k_pp_bounds(LatticeDesc d, int nvert, const uint32_t* __restrict__ keys,
                                                    const uint32_t* __restrict__ ids, const double* __restrict__ pos,
                                                    const int* __restrict__ owner, int* __restrict__ start,
                                                    int* __restrict__ end, float4* __restrict__ posf) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nvert) return;
    const uint32_t k = keys[s];
    if (s == 0 || keys[s - 1] != k) start[k] = s;
    if (s == nvert - 1 || keys[s + 1] != k) end[k] = s + 1;
    const int v = (int)ids[s];
    const double x = pos[3LL * v], y = pos[3LL * v + 1], z = pos[3LL * v + 2];
    const bool far = !(fabs(x) <= 4.0 * d.nx && fabs(y) <= 4.0 * d.ny && fabs(z) <= 4.0 * d.nz);
    posf[s] = make_float4(far ? nanf("") : (float)x, (float)y, (float)z, __int_as_float(owner[v]));
}

// Arithmetic1D::min_mod_diff (Periodicity.h:27-35, 96-99) on periodic axes
__device__ __forceinline__ double min_image(const LatticeDesc& d, int a, double dx) {
    const int per = a == 0 ? d.px : (a == 1 ? d.py : d.pz);
    if (!per) return dx;
    const double N = (double)(a == 0 ? d.nx : (a == 1 ? d.ny : d.nz));
    return dx - floor(dx * d.inv_n[a] + 0.5) * N;
}

__device__ __forceinline__ float min_image_f(int per, float N, float dx) {
    return per ? dx - floorf(dx / N + 0.5f) * N : dx;
}

// One warp per vertex, one lane per neighbour cell: the sum over partners j of other particles within
// the cutoff of (-phi(d) / d) (x_j - x_i) (CollisionHandler::handle_collision, CollisionForces.h:187-199),
// added to the vertex's force.  Every pair is evaluated from both ends and the lanes are added up in one
// order, so no atomics.  Pairs pass an FP32 distance test first, with `reach` = the cutoff plus 2^-18 of
// the longest axis (more than the FP32 positions and differences can be off within 4 periods); the FP64
// test alone decides the rest.
// Bound by the latency of the bucket lookups: all 27 of a vertex are in flight at once, over FP32
// positions in bucket order.  One thread per vertex that walked its 27 cells and formed every distance
// in FP64 took 156 us for 40 cells of 642 vertices in a 192 x 50 x 50 pipe, whose step went from 274 to
// 145 us.
__global__ void __launch_bounds__(128) k_pp_forces(LatticeDesc d, Interactions I, PairCells g, int nvert, float reach,
                                                    const double* __restrict__ pos, const uint32_t* __restrict__ ids,
                                                    const int4* __restrict__ cell, const float4* __restrict__ posf,
                                                    const int* __restrict__ start, const int* __restrict__ end,
                                                    double* __restrict__ force) {
    const unsigned FULL = 0xffffffffu;
    const int slot = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (slot >= nvert) return;  // whole warps
    const int i = (int)ids[slot];
    const float4 pi = posf[slot];
    const int4 c = cell[i];
    const int per[3] = {d.px, d.py, d.pz};
    int n[3] = {c.x + lane % 3 - 1, c.y + (lane / 3) % 3 - 1, c.z + lane / 9 - 1};
    bool ok = lane < 27;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (n[a] < 0 || n[a] >= g.nc[a]) {
            if (!per[a]) ok = false;
            else n[a] = (n[a] + g.nc[a]) % g.nc[a];
        }
    const unsigned h = ok ? cell_hash(g, n[0], n[1], n[2]) : 0u;
    // neighbour cells that share a bucket are visited once, by the first lane that has it
    const unsigned live = __ballot_sync(FULL, ok), same = __match_any_sync(FULL, h) & live;
    const bool mine = ok && (same & ((1u << lane) - 1)) == 0;
    double f[3] = {0.0, 0.0, 0.0};
    bool hit = false;
    const int s1 = mine ? end[h] : 0;
    for (int s = mine ? start[h] : 0; s < s1; ++s) {
        const float4 q = posf[s];
        if (__float_as_int(q.w) == __float_as_int(pi.w)) continue;
        const float ex = min_image_f(d.px, (float)d.nx, q.x - pi.x), ey = min_image_f(d.py, (float)d.ny, q.y - pi.y),
                    ez = min_image_f(d.pz, (float)d.nz, q.z - pi.z);
        if (ex * ex + ey * ey + ez * ez > reach * reach) continue;
        const double xi[3] = {pos[3LL * i], pos[3LL * i + 1], pos[3LL * i + 2]};
        if (!(isfinite(xi[0]) && isfinite(xi[1]) && isfinite(xi[2]))) continue;
        const int j = (int)ids[s];
        const double dr[3] = {min_image(d, 0, pos[3LL * j] - xi[0]), min_image(d, 1, pos[3LL * j + 1] - xi[1]),
                              min_image(d, 2, pos[3LL * j + 2] - xi[2])};
        const double dsq = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
        if (!(dsq <= I.pp_cut * I.pp_cut)) continue;
        const double dist = sqrt(dsq);
        for (int k = 0; k < I.npp; ++k) {
            if (!(dsq <= I.pp[k].r0 * I.pp[k].r0)) continue;
            const double sc = -potential_eval(I.pp[k], dist) / dist;
            f[0] += sc * dr[0];
            f[1] += sc * dr[1];
            f[2] += sc * dr[2];
            hit = true;
        }
    }
    if (!__any_sync(FULL, hit)) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) f[a] += __shfl_down_sync(FULL, f[a], o);
    if (lane == 0)
        for (int a = 0; a < 3; ++a) force[3LL * i + a] += f[a];
}

}  // namespace

size_t membrane_smem_bytes(int max_nv) { return (size_t)3 * max_nv * sizeof(double); }

size_t spread_sort_temp_bytes(int64_t nentries) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs((void*)nullptr, bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (uint32_t*)nullptr, (int)nentries, 0, 32);  // upper bound over the key widths
    return bytes;
}

int spread_key_bits(int64_t n) { return key_bits(n); }

size_t spread_sort_temp_bytes_pingpong(int64_t nentries, int end_bit) {
    size_t bytes = 0;
    cub::DoubleBuffer<uint32_t> k(nullptr, nullptr), v(nullptr, nullptr);
    if (cub::DeviceRadixSort::SortPairs(nullptr, bytes, k, v, (int)nentries, 0, end_bit) != cudaSuccess) return SIZE_MAX;
    return bytes;
}

cudaError_t launch_spread_sorted(const LatticeDesc& d, const IbDesc& ib, bool f64_field, int nvert, const double* pos,
                                 const double* force, void* field, uint32_t* keys0, uint32_t* keys1, uint32_t* ids0,
                                 uint32_t* ids1, void* temp, size_t temp_bytes, cudaStream_t s) {
    const int sup = ib.dirac == BIB_DIRAC_PESKIN ? 4 : 3;
    const int64_t ne = (int64_t)nvert * sup * sup * sup;
    k_spread_keys<<<(nvert + 127) / 128, 128, 0, s>>>(d, ib, nvert, pos, keys0, ids0);
    cub::DoubleBuffer<uint32_t> k(keys0, keys1), v(ids0, ids1);
    size_t tb = temp_bytes;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(temp, tb, k, v, (int)ne, 0, key_bits(d.n), s);
    if (e != cudaSuccess) return e;
    const unsigned ge = (unsigned)((ne + 127) / 128);
    if (f64_field)
        k_spread_reduce<double><<<ge, 128, 0, s>>>(d, ib, ne, k.Current(), v.Current(), pos, force, (double*)field);
    else
        k_spread_reduce<float><<<ge, 128, 0, s>>>(d, ib, ne, k.Current(), v.Current(), pos, force, (float*)field);
    return cudaGetLastError();
}

void configure_membrane_kernel(size_t smem) {
    // the limit is per kernel function: only ever raise it, other lattices may need more
    static size_t configured = 0;
    if (smem <= configured) return;
    configured = smem;
    cudaFuncSetAttribute(k_membrane<double, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_membrane<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_membrane<double, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaFuncSetAttribute(k_membrane<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    // 3 floats per vertex, at most half of the membrane kernel's 3 doubles per vertex
    cudaFuncSetAttribute(k_particle_update<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem / 2));
    cudaFuncSetAttribute(k_particle_update<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem / 2));
}

IbView single_view(const Lattice& L, int fbuf) {
    IbView v{};
    v.d = L.d;
    v.ib = L.ib;
    v.pos = L.pos[L.pcur];
    v.pos_next = L.pos[1 - L.pcur];
    v.u = L.u;
    v.vel = L.vel;
    v.force = L.force;
    v.F = fbuf >= 0 ? L.F[fbuf] : nullptr;
    v.stats = L.stats;
    v.vbase = 0;
    v.nvert = L.nvert;
    v.inter = L.inter;
    v.order = L.visit_order;
    return v;
}

namespace {

template <class UT, int S, bool BATCH, bool FOLD = false>
void interpolate_inst(const IbView& v1, const IbView* views, const int* vinst, int nvert, cudaStream_t s) {
    if (nvert <= kGatherMax)
        k_interpolate_move<UT, S, BATCH, FOLD>
            <<<(nvert + kGatherVerts - 1) / kGatherVerts, 32 * S * S, 0, s>>>(v1, views, vinst, nvert);
    else
        k_interpolate_vertices<UT, S, BATCH, FOLD><<<(nvert + 127) / 128, 128, 0, s>>>(v1, views, vinst, nvert);
}

template <bool BATCH>
void interpolate_any(int storage, int dirac, const IbView& v1, const IbView* views, const int* vinst, int nvert,
                     cudaStream_t s) {
    const bool peskin = dirac == BIB_DIRAC_PESKIN;
    if (storage == BIB_STORAGE_F64) {
        if (peskin) interpolate_inst<double, 4, BATCH>(v1, views, vinst, nvert, s);
        else interpolate_inst<double, 3, BATCH>(v1, views, vinst, nvert, s);
    } else if (storage == BIB_STORAGE_F32) {
        if (peskin) interpolate_inst<float, 4, BATCH>(v1, views, vinst, nvert, s);
        else interpolate_inst<float, 3, BATCH>(v1, views, vinst, nvert, s);
    } else {
        if (peskin) interpolate_inst<__half, 4, BATCH>(v1, views, vinst, nvert, s);
        else interpolate_inst<__half, 3, BATCH>(v1, views, vinst, nvert, s);
    }
}

template <bool BATCH>
void spread_any(int storage, int dirac, const IbView& v1, const IbView* views, const int* vinst, int nvert,
                cudaStream_t s) {
    const unsigned g = (nvert + kSpreadVerts - 1) / kSpreadVerts;
    const bool peskin = dirac == BIB_DIRAC_PESKIN;
    if (storage == BIB_STORAGE_F64) {
        if (peskin) k_spread_rows<double, 4, BATCH><<<g, kSpreadThreads, 0, s>>>(v1, views, vinst, nvert);
        else k_spread_rows<double, 3, BATCH><<<g, kSpreadThreads, 0, s>>>(v1, views, vinst, nvert);
    } else {
        if (peskin) k_spread_rows<float, 4, BATCH><<<g, kSpreadThreads, 0, s>>>(v1, views, vinst, nvert);
        else k_spread_rows<float, 3, BATCH><<<g, kSpreadThreads, 0, s>>>(v1, views, vinst, nvert);
    }
}

template <bool BATCH>
void membrane_any(int storage, const ParticleDev* parts, int np, const IbView& v1, const IbView* views, size_t smem,
                  int block, cudaStream_t s) {
    if (storage == BIB_STORAGE_F64) k_membrane<double, BATCH><<<np, block, smem, s>>>(parts, v1, views);
    else k_membrane<float, BATCH><<<np, block, smem, s>>>(parts, v1, views);
}

template <bool BATCH>
void update_any(int storage, const ParticleDev* parts, int np, const IbView& v1, const IbView* views, int max_nv,
                cudaStream_t s) {
    if (storage == BIB_STORAGE_F64) k_particle_update<double, BATCH><<<np, 256, 0, s>>>(parts, v1, views);
    else k_particle_update<float, BATCH><<<np, 256, 3 * sizeof(float) * max_nv, s>>>(parts, v1, views);
}

}  // namespace

void launch_interpolate_move(const Lattice& L, cudaStream_t s, int fold) {
    if (L.nvert == 0) return;
    if (fold < 0 || L.storage == BIB_STORAGE_F64) {
        interpolate_any<false>(L.storage, L.ib.dirac, single_view(L, -1), nullptr, nullptr, L.nvert, s);
        return;
    }
    IbView v = single_view(L, -1);
    v.Fold = L.F[fold];
    const bool peskin = L.ib.dirac == BIB_DIRAC_PESKIN;
    if (L.storage == BIB_STORAGE_F32) {
        if (peskin) interpolate_inst<float, 4, false, true>(v, nullptr, nullptr, L.nvert, s);
        else interpolate_inst<float, 3, false, true>(v, nullptr, nullptr, L.nvert, s);
    } else {
        if (peskin) interpolate_inst<__half, 4, false, true>(v, nullptr, nullptr, L.nvert, s);
        else interpolate_inst<__half, 3, false, true>(v, nullptr, nullptr, L.nvert, s);
    }
}

void launch_force_clear(const Lattice& L, int fbuf, cudaStream_t s) {
    if (L.nvert == 0 || L.storage == BIB_STORAGE_F64) return;
    const int sup = L.ib.dirac == BIB_DIRAC_PESKIN ? 4 : 3;
    const int64_t threads = (int64_t)L.nvert * sup * sup;
    const unsigned g = (unsigned)((threads + 127) / 128);
    if (sup == 4) k_force_clear<4><<<g, 128, 0, s>>>(L.d, L.ib, L.nvert, L.spread_lo[fbuf], (float*)L.F[fbuf]);
    else k_force_clear<3><<<g, 128, 0, s>>>(L.d, L.ib, L.nvert, L.spread_lo[fbuf], (float*)L.F[fbuf]);
}

// CTAs per particle: enough to give every SM `per_sm` CTAs, but at least one element per thread
int membrane_split(int np, int max_elems, int block, int per_sm = 2) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    if (np <= 0 || np >= sms) return 1;
    const int want = (per_sm * sms + np - 1) / np;
    const int most = std::max(1, (max_elems + block - 1) / block);
    return std::max(1, std::min(want, most));
}

namespace {
template <bool SPREAD, bool BATCH>
void patch_launch(int dirac, const PatchJob* jobs, const ParticleDev* parts, int npatch, size_t smem, const IbView& v,
                  const IbView* views, cudaStream_t s) {
    if (dirac == BIB_DIRAC_PESKIN) k_membrane_patch<4, BATCH, SPREAD><<<npatch, kSpreadThreads, smem, s>>>(jobs, parts, v, views);
    else k_membrane_patch<3, BATCH, SPREAD><<<npatch, kSpreadThreads, smem, s>>>(jobs, parts, v, views);
}
}  // namespace

bool launch_membrane_spread(const Lattice& L, int fbuf, cudaStream_t s, bool record) {
    if (L.npatch == 0 || L.inter.npp > 0 || L.ib.spread_mode == BIB_SPREAD_DETERMINISTIC) return false;
    IbView v = single_view(L, fbuf);
    v.spread_lo = record ? L.spread_lo[fbuf] : nullptr;
    patch_launch<true, false>(L.ib.dirac, L.patch_jobs, L.pdev, L.npatch, L.patch_smem, v, nullptr, s);
    return true;
}

bool launch_membrane_spread_batch(const BatchLaunch& B, cudaStream_t s) {
    if (B.npatch == 0) return false;
    patch_launch<true, true>(B.dirac, B.patch_jobs, B.parts, B.npatch, B.patch_smem, IbView{}, B.views, s);
    return true;
}

void launch_membrane_forces(const Lattice& L, cudaStream_t s) {
    const int np = (int)L.parts.size();
    if (np == 0) return;
    if (L.npatch > 0) {
        patch_launch<false, false>(L.ib.dirac, L.patch_jobs, L.pdev, L.npatch, L.patch_smem, single_view(L, -1), nullptr, s);
        return;
    }
    if (L.ib.spread_mode == BIB_SPREAD_DETERMINISTIC) {
        // one-warp CTAs: few vertices spread over more SMs (FP64 pipe), many take as long either way.  Step with red
        // cells of 642 vertices, FP64, 32 against 128 threads: 1 cell 350 / 366 us, 10 439 / 460, 30 552 / 552, 260
        // 3637 / 3642; FP32 with link springs the same within 1 % from 1 to 260
        const int block = 32;
        const unsigned g = (L.nvert + block - 1) / block;
        if (L.storage == BIB_STORAGE_F64)
            k_membrane_gather<double><<<g, block, 0, s>>>(L.nvert, L.vert_particle, L.pdev, L.pos[L.pcur], L.force, L.stats, L.inter);
        else
            k_membrane_gather<float><<<g, block, 0, s>>>(L.nvert, L.vert_particle, L.pdev, L.pos[L.pcur], L.force, L.stats, L.inter);
        return;
    }
    // Few particles: each particle's elements over several CTAs so the launch fills the GPU.
    // FP64: about four warps per SM (bound by the FP64 pipe, 2 lanes per cycle and SM: a warp to itself is served
    // as fast as it can issue).  One capsule of 1280 triangles: 8 CTAs of 256 threads 53.8 us, 60 of 32 36.9
    // (23.6 with capsule_triangle's shared scalars); the step of 40 red cells of 2562 vertices with link springs 793 us
    // with the CTAs of the FP32 rule, so 734.
    // FP32 (membranes with link springs, the others go by patches): two CTAs of membrane_block threads per SM, since
    // every CTA clears, stages and adds the whole membrane.  Steps with such red cells, one-warp CTAs as in
    // FP64 against these: 1 of 642 vertices 57.7 / 42.0 us, 10 76.0 / 62.5, 100 169 / 165; 1 of 2562 96.7 / 70.8, 10 112 / 83.6,
    // 40 169 / 162.
    const bool f64 = L.storage == BIB_STORAGE_F64;
    const int warps = (L.max_elems + 31) / 32;
    const int split = f64 ? std::min(warps, membrane_split(np, L.max_elems, 32, 4))
                          : membrane_split(np, L.max_elems, L.membrane_block);
    if (split > 1) {
        const IbView v = single_view(L, -1);
        k_force_seed<<<(L.nvert + 127) / 128, 128, 0, s>>>(v);
        const dim3 grid((unsigned)np, (unsigned)split);
        const int block = f64 ? std::min(L.membrane_block, 32 * ((warps + split - 1) / split)) : L.membrane_block;
        if (L.storage == BIB_STORAGE_F64) k_membrane<double, false><<<grid, block, L.membrane_smem, s>>>(L.pdev, v, nullptr);
        else k_membrane<float, false><<<grid, block, L.membrane_smem, s>>>(L.pdev, v, nullptr);
        return;
    }
    membrane_any<false>(L.storage, L.pdev, np, single_view(L, -1), nullptr, L.membrane_smem, L.membrane_block, s);
}

size_t pp_sort_temp_bytes(int nvert, int bits) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs((void*)nullptr, bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (uint32_t*)nullptr, nvert, 0, bits);
    return bytes;
}

void launch_pp_forces(const Lattice& L, cudaStream_t s) {
    if (L.inter.npp == 0 || L.nvert == 0) return;
    if (L.inter.pp_search == BIB_PAIR_SEARCH_GRID) {
        // one CollisionHandler per potential, in order (ImmersedBoundaryDynamics_forces.hh:299-301)
        if (!L.rgrid.start) return;
        const int64_t box[6] = {0, L.d.nx - 1, 0, L.d.ny - 1, 0, L.d.nz - 1};
        const int per[3] = {L.d.px, L.d.py, L.d.pz};
        for (int k = 0; k < L.inter.npp; ++k)
            launch_ref_grid_forces(ref_grid(box, per, L.inter.pp[k].r0, L.nvert), L.rgrid, L.inter.pp[k],
                                   L.pos[L.pcur], L.vert_particle, L.force, false, nullptr, s);
        return;
    }
    if (!L.pgrid.table) return;
    const PairGrid& G = L.pgrid;
    PairCells g;
    for (int a = 0; a < 3; ++a) {
        g.nc[a] = G.nc[a];
        g.cs[a] = G.cs[a];
    }
    g.mask = G.table - 1;
    const unsigned b = (L.nvert + 127) / 128;
    k_pp_keys<<<b, 128, 0, s>>>(L.d, g, L.nvert, L.pos[L.pcur], G.keys[1], G.start, G.end, G.keys[0], G.ids[0], G.cell);
    size_t tb = G.temp_bytes;
    cub::DeviceRadixSort::SortPairs(G.temp, tb, G.keys[0], G.keys[1], G.ids[0], G.ids[1], L.nvert, 0, G.bits, s);
    k_pp_bounds<<<b, 128, 0, s>>>(L.d, L.nvert, G.keys[1], G.ids[1], L.pos[L.pcur], L.vert_particle, G.start, G.end, G.posf);
    const float reach = (float)(L.inter.pp_cut + std::max(L.d.nx, std::max(L.d.ny, L.d.nz)) / 262144.0);
    k_pp_forces<<<(unsigned)((32LL * L.nvert + 127) / 128), 128, 0, s>>>(L.d, L.inter, g, L.nvert, reach, L.pos[L.pcur],
                                                                         G.ids[1], G.cell, G.posf, G.start, G.end, L.force);
}

void launch_particle_update(const Lattice& L, cudaStream_t s) {
    const int np = (int)L.parts.size();
    if (np == 0) return;
    // FP64 sums, and in FP32 large meshes.  FP32 step of one membrane in 96^3, one CTA against split: 1216 triangles
    // 59.1 / 59.2 us, 1932 61.7 / 61.7, 2592 65.5 / 60.5, 3248 66.2 / 60.6, 4200 71.2 / 62.0; 16 of 3248 129 / 111, 64 of them
    // 132 / 136
    const bool big = L.storage == BIB_STORAGE_F64 || L.max_nt >= 2048;
    const int split = big ? std::min(kMaxUpdateSplit, membrane_split(np, L.max_nt, kUpdateFew)) : 1;
    if (split > 1 && L.upd_partial) {
        const IbView v = single_view(L, -1);
        unsigned* ticket = reinterpret_cast<unsigned*>(L.upd_partial + (size_t)np * kMaxUpdateSplit * 5);
        if (L.storage == BIB_STORAGE_F64) k_update_few<double><<<dim3(np, split), kUpdateFew, 0, s>>>(L.pdev, v, L.upd_partial, ticket);
        else k_update_few<float><<<dim3(np, split), kUpdateFew, 0, s>>>(L.pdev, v, L.upd_partial, ticket);
        return;
    }
    update_any<false>(L.storage, L.pdev, np, single_view(L, -1), nullptr, L.max_nv, s);
}

void launch_membrane_batch(const BatchLaunch& B, int block, cudaStream_t s) {
    if (B.nparts == 0) return;
    membrane_any<true>(B.storage, B.parts, B.nparts, IbView{}, B.views, B.membrane_smem, block, s);
}
void launch_spread_batch(const BatchLaunch& B, cudaStream_t s) {
    if (B.nvert == 0) return;
    spread_any<true>(B.storage, B.dirac, IbView{}, B.views, B.vinst, B.nvert, s);
}
void launch_interpolate_batch(const BatchLaunch& B, cudaStream_t s) {
    if (B.nvert == 0) return;
    interpolate_any<true>(B.storage, B.dirac, IbView{}, B.views, B.vinst, B.nvert, s);
}
void launch_update_batch(const BatchLaunch& B, cudaStream_t s) {
    if (B.nparts == 0) return;
    update_any<true>(B.storage, B.parts, B.nparts, IbView{}, B.views, B.max_nv, s);
}

void launch_spread(const Lattice& L, int fbuf, cudaStream_t s, bool record) {
    if (L.nvert == 0) return;
    const double* pos = L.pos[L.pcur];
    int4* lo = record ? L.spread_lo[fbuf] : nullptr;
    if (L.ib.spread_mode == BIB_SPREAD_DETERMINISTIC) {
        const int sup = L.ib.dirac == BIB_DIRAC_PESKIN ? 4 : 3;
        const int64_t ne = (int64_t)L.nvert * sup * sup * sup;
        auto run = [&](auto zero, auto sup_c) {
            using FT = decltype(zero);
            constexpr int S = decltype(sup_c)::value;
            FT* rec = static_cast<FT*>(L.spread_rec);
            k_spread_entries<FT, S><<<(L.nvert + kSpreadVerts - 1) / kSpreadVerts, kSpreadThreads, 0, s>>>(
                L.d, L.ib, L.nvert, pos, L.force, rec, L.sort_keys[0], L.sort_ids[0], lo);
            size_t tb = L.sort_temp_bytes;
            cub::DeviceRadixSort::SortPairs(L.sort_temp, tb, L.sort_keys[0], L.sort_keys[1], L.sort_ids[0], L.sort_ids[1],
                                            (int)ne, 0, key_bits(L.d.n), s);
            k_spread_sum<FT, S><<<(unsigned)((ne + 127) / 128), 128, 0, s>>>(
                L.d.n, ne, L.sort_keys[1], L.sort_ids[1], reinterpret_cast<const SpreadRecord<FT, S>*>(rec), (FT*)L.F[fbuf]);
        };
        using Roma = std::integral_constant<int, 3>;
        using Peskin = std::integral_constant<int, 4>;
        if (L.storage == BIB_STORAGE_F64) sup == 4 ? run(double{}, Peskin{}) : run(double{}, Roma{});
        else sup == 4 ? run(float{}, Peskin{}) : run(float{}, Roma{});
        return;
    }
    IbView v = single_view(L, fbuf);
    v.spread_lo = lo;
    spread_any<false>(L.storage, L.ib.dirac, v, nullptr, nullptr, L.nvert, s);
}

// Phase field of the membranes at pos (the positions of the current step's end): z-rays of
// every triangle, then the per-column parity fill.  count must be zero on entry (it is left
// zero); a column with more than cap crossings, or a triangle wider than the lattice, sets
// *overflow (the column keeps its first cap crossings, the triangle casts no rays).
void launch_voxelize(const Lattice& L, const double* pos, cudaStream_t s) {
    if (!L.phase || L.parts.empty()) return;
    const dim3 rays((unsigned)L.parts.size(), (unsigned)std::min(65535, (L.max_nt + 31) / 32));
    k_voxel_rays<<<rays, 32, 0, s>>>(L.d, L.pdev, pos, L.vox_count, L.vox_z, kVoxelCap, L.vox_err);
    const int64_t ncol = (int64_t)L.d.nx * L.d.ny;
    k_voxel_fill<<<(unsigned)((ncol + 127) / 128), 128, 0, s>>>(L.d, L.vox_count, L.vox_z, kVoxelCap, L.phase);
}

// ---- RBC shape calibration: RBCParticle::relax_nodes (RBCParticle.hh:318-342) ----
// One iteration of shrink_rbc_volume (progs/common/calibrate_rbc_shape.h:25-33) for the single
// particle of L: vol_desired of iteration it (while it <= n_it) into the particle's parameters,
// node masses M_i = sum over the triangles at i (in triangle order) of area/3, vel += force/M -
// damping vel, pos_next = pos + vel.  The forces of pos_next are computed by the membrane
// kernel afterwards, with the new vol_desired.  Operations are rounded one by one (no
// contraction) in the reference's order.  One block; *iter counts the iterations.
__global__ void __launch_bounds__(256) k_rbc_relax(ParticleDev* P, const double* __restrict__ pos,
                                                   double* __restrict__ pos_next, double* __restrict__ vel,
                                                   const double* __restrict__ force, int nv, double damping,
                                                   long long* iter, long long n_it, double vol_start, double vol_final) {
    const long long it = *iter;
    const ParticleDev& p = *P;
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
        double M = 0.0;
        for (int e = p.inc_off[i]; e < p.inc_off[i + 1]; ++e) {
            const int code = p.inc[e];
            if ((code >> 29) != 1) continue;  // triangles only
            const int t = code & ((1 << 29) - 1);
            const int i0 = p.tri[3 * t], i1 = p.tri[3 * t + 1], i2 = p.tri[3 * t + 2];
            const double ax = pos[3 * i0], ay = pos[3 * i0 + 1], az = pos[3 * i0 + 2];
            const double ux = __dsub_rn(pos[3 * i1], ax), uy = __dsub_rn(pos[3 * i1 + 1], ay),
                         uz = __dsub_rn(pos[3 * i1 + 2], az);
            const double wx = __dsub_rn(pos[3 * i2], ax), wy = __dsub_rn(pos[3 * i2 + 1], ay),
                         wz = __dsub_rn(pos[3 * i2 + 2], az);
            const double cx = __dsub_rn(__dmul_rn(uy, wz), __dmul_rn(uz, wy));
            const double cy = __dsub_rn(__dmul_rn(uz, wx), __dmul_rn(ux, wz));
            const double cz = __dsub_rn(__dmul_rn(ux, wy), __dmul_rn(uy, wx));
            const double n2 = __dadd_rn(__dadd_rn(__dmul_rn(cx, cx), __dmul_rn(cy, cy)), __dmul_rn(cz, cz));
            M = __dadd_rn(M, __ddiv_rn(__dmul_rn(0.5, __dsqrt_rn(n2)), 3.0));
        }
        for (int k = 0; k < 3; ++k) {
            const double v = vel[3 * i + k];
            const double nvk = __dadd_rn(v, __dsub_rn(__ddiv_rn(force[3 * i + k], M), __dmul_rn(damping, v)));
            vel[3 * i + k] = nvk;
            pos_next[3 * i + k] = __dadd_rn(pos[3 * i + k], nvk);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (it <= n_it)
            P->prm[BIB_P_VOL_DESIRED] =
                __dadd_rn(vol_start, __dmul_rn(__ddiv_rn((double)it, (double)n_it), __dsub_rn(vol_final, vol_start)));
        *iter = it + 1;
    }
}

void launch_rbc_relax(const Lattice& L, double damping, long long* iter, long long n_it, double vol_start,
                      double vol_final, cudaStream_t s) {
    k_rbc_relax<<<1, 256, 0, s>>>(L.pdev, L.pos[L.pcur], L.pos[1 - L.pcur], L.vel, L.force, L.nvert, damping, iter,
                                   n_it, vol_start, vol_final);
}

}  // namespace bib
