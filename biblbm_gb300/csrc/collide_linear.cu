// Staged collide-and-stream over linear tiles, for rows that the row tiles do not take (x-rows longer
// than a tile, or whose bytes are no multiple of 16: N + 1 nodes), FP16 and FP32 storage.
//
// A tile is TILE consecutive cells, whatever rows they belong to.  Away from the domain's faces the
// source of population i is the cell a constant distance back, k - (c_x + nx (c_y + ny c_z)), so a tile's
// source is one run per population.  A bulk copy starts on 16 bytes: the run is copied from the boundary
// below its start, and since tiles start on one, the remainder is the same for every tile.  The cells at
// a face have other sources: at the ends of a row the populations that cross it come from the row's
// other end, in the first and last rows and planes from the periodic image, the wall rule or the wall
// buffer.  Those few are read from global memory after the stage has been handed back.
//
// Bound by HBM (FP32) and by HBM and issue (FP16) as the row tiles are: 201^3, 100 steps in a row, FP32 5.6 TB/s (4.0
// with one thread per cell straight from global memory), FP16 4.5 TB/s (1.1).
#include <type_traits>

#include "staged_common.cuh"

namespace bib {

namespace {

template <class T>
struct LinearOf {
    static constexpr int TILE = TileOf<T>::value;
    static constexpr int A = 16 / (int)sizeof(T);  // cells of 16 bytes
    static constexpr int PITCH = TILE + A;
};

template <class T, int CPL, int COLL>
struct LinearLayout {
    using FT = typename Store<T>::F;
    static constexpr int TILE = LinearOf<T>::TILE, PITCH = LinearOf<T>::PITCH;
    static constexpr int CONSUMERS = TILE / 32, THREADS = 32 * (CONSUMERS + 1);
    static constexpr bool NEED_FCOL = COLL == BIB_COLLISION_BGK_GUO_VOF;
    static constexpr unsigned POP = PITCH * sizeof(T);
    static constexpr unsigned FRC = 3 * TILE * sizeof(FT);
    static constexpr unsigned OFF_FCOL = Q * POP;
    static constexpr unsigned OFF_FPREV = OFF_FCOL + (NEED_FCOL ? FRC : 0);
    static constexpr unsigned BYTES = (OFF_FPREV + (CPL == kCplDense ? FRC : 0) + 127) / 128 * 128;
    static constexpr unsigned RESET = resets(CPL) ? FRC : 0;
};

struct LinearGeom {
    int nstages;
    uint32_t ntiles;
    int64_t n, stride;
    int32_t off[Q];  // distance back of each population's source
    int32_t rem[Q];  // (-off) modulo the cells of 16 bytes
    uint64_t wait_ns;
    int64_t withhold;
};

// x, y, z of cell k (n < 2^31)
struct Cell3 {
    int x, y, z;
};
__device__ __forceinline__ Cell3 cell_of(const LatticeDesc& d, uint32_t k) {
    Cell3 c;
    const uint32_t row = k / (uint32_t)d.nx;
    c.x = (int)(k - row * (uint32_t)d.nx);
    c.z = (int)(row / (uint32_t)d.ny);
    c.y = (int)(row - (uint32_t)c.z * (uint32_t)d.ny);
    return c;
}

template <class T, int CPL, int COLL>
__device__ __forceinline__ void load_linear(const LinearGeom& g, uint32_t tile, unsigned char* stage, uint64_t* bar,
                                            const T* fin, const typename Store<T>::F* Fcol,
                                            const typename Store<T>::F* Fprev, int lane, int32_t off) {
    using L = LinearLayout<T, CPL, COLL>;
    using FT = typename Store<T>::F;
    constexpr int A = LinearOf<T>::A;
    const int64_t k0 = (int64_t)tile * L::TILE;
    unsigned char* dst = nullptr;
    const void* src = nullptr;
    unsigned bytes = 0;
    if (lane < Q) {
        // [a, b): the run from the 16-byte boundary below its start, inside the population's array
        int64_t a = (k0 - off) & ~(int64_t)(A - 1), b = a + L::PITCH;
        int skip = 0;
        if (a < 0) skip = (int)min((int64_t)L::PITCH, -a), a = 0;
        b = min(b, g.stride);
        if (b > a) {
            bytes = (unsigned)((b - a) * sizeof(T));
            dst = stage + lane * L::POP + skip * sizeof(T);
            src = fin + lane * g.stride + a;
        }
    } else if ((L::NEED_FCOL && lane == Q) || (CPL == kCplDense && lane == Q + 1)) {
        bytes = (unsigned)(3 * min((int64_t)L::TILE, g.stride - k0) * sizeof(FT));
        dst = stage + (lane == Q ? L::OFF_FCOL : L::OFF_FPREV);
        src = (lane == Q ? Fcol : Fprev) + 3 * k0;
    }
    const unsigned total = __reduce_add_sync(0xffffffffu, bytes);
    if (lane == 0) mbar_arrive_expect_tx(bar, total);
    __syncwarp();
    if (bytes) bulk_copy_g2s(dst, src, bytes, bar);
    __syncwarp();
}

// Post-streaming populations, in storage units, of a cell whose gather crosses a y or z face.
template <class T>
__device__ __noinline__ void gather_face_cell(const LatticeDesc& d, const CollideParams<typename Store<T>::C>& cp,
                                              const T* __restrict__ fin, const T* __restrict__ wall, Cell3 c, int64_t k,
                                              typename Store<T>::C* f) {
    using C = typename Store<T>::C;
    if (fd_wall_node(d, c.y)) {
        const int64_t wk = wall_index(d, c.y == 0 ? 0 : 1, c.x, c.z), ws = wall_stride(d);
#pragma unroll
        for (int i = 0; i < Q; ++i) f[i] = Staged<T>::one(wall + i * ws + wk);
        return;
    }
    // the row of each (c_y, c_z), or the wall face behind it; all loads are issued before the first value
    // is used (a load, its conversion and its wall term in turn would wait 19 times)
    int row[3][3], face[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            int ys = c.y - (a - 1), zs = c.z - (b - 1), at = -1;
            if (zs < 0 || zs >= d.nz) {
                if (d.pz) zs = zs < 0 ? zs + d.nz : zs - d.nz;
                else at = zs < 0 ? 2 : 3;
            }
            if (ys < 0 || ys >= d.ny) {
                if (d.py) ys = ys < 0 ? ys + d.ny : ys - d.ny;
                else at = ys < 0 ? 0 : 1;
            }
            face[a][b] = at;
            row[a][b] = at < 0 ? ys + d.ny * zs : c.y + d.ny * c.z;
        }
    T raw[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int a = cy(i) + 1, b = cz(i) + 1;
        int x = c.x;
        if (cx(i) != 0 && face[a][b] < 0) {
            x -= cx(i);
            x = x < 0 ? x + d.nx : (x >= d.nx ? x - d.nx : x);
        }
        raw[i] = __ldg(fin + (face[a][b] < 0 ? i : opposite(i)) * d.stride + ((int64_t)row[a][b] * d.nx + x));
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const int at = face[cy(i) + 1][cz(i) + 1];
        f[i] = (C)raw[i];
        if (at >= 0) f[i] += cp.mw[at][i];
    }
}

template <class T, int CPL, int COLL>
__global__ void __launch_bounds__(LinearLayout<T, CPL, COLL>::THREADS, staged_ctas_per_sm<T>())
    k_collide_stream_linear(LatticeDesc d, LinearGeom g, CollideParams<typename Store<T>::C> cp, const T* __restrict__ fin,
                            T* __restrict__ fout, const T* __restrict__ wall, const typename Store<T>::F* __restrict__ Fcol,
                            typename Store<T>::F* __restrict__ Fprev, typename Store<T>::U* __restrict__ u_out,
                            const uint8_t* __restrict__ phase, const uint8_t* __restrict__ celltype,
                            int* __restrict__ wait_err) {
    using C = typename Store<T>::C;
    using FT = typename Store<T>::F;
    using L = LinearLayout<T, CPL, COLL>;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + kMaxStages;
    FT* reset = reinterpret_cast<FT*>(smem + 256);
    unsigned char* stages = smem + 256 + L::RESET;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t NS = (uint32_t)g.nstages;
    if (blockIdx.x >= g.ntiles) return;
    if (resets(CPL)) fill_reset(reset, d.body, 3 * L::TILE, tid, L::THREADS);
    if (tid == 0) {
        for (uint32_t k = 0; k < NS; ++k) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], L::CONSUMERS);
        }
        mbar_init_fence();
    }
    __syncthreads();
    // the reset of the previous force of a tile: its cells, and at the array's end what the array holds
    auto reset_linear = [&](uint32_t tile) {
        const int64_t k0 = (int64_t)tile * L::TILE;
        bulk_copy_s2g(Fprev + 3 * k0, reset, (unsigned)(3 * min((int64_t)L::TILE, g.stride - k0) * sizeof(FT)));
    };

    if (warp == 0) {
        // ---- producer: lane i moves population i
        int32_t off = 0;
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if (lane == i) off = g.off[i];
        uint32_t it = 0, withheld = 0xffffffffu;
        for (uint32_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x, ++it) {
            const uint32_t s = it % NS, use = it / NS;
            if (use > 0) {
                const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], (use - 1) & 1u, g.wait_ns));
                if (!ok) {
                    if (lane == 0) atomicExch(wait_err, 1);
                    break;
                }
            }
            if ((int64_t)tile == g.withhold) {  // failure testing: this stage's phase is never completed
                withheld = it;
                continue;
            }
            load_linear<T, CPL, COLL>(g, tile, stages + s * L::BYTES, &full[s], fin, Fcol, Fprev, lane, off);
            if (resets(CPL) && use > 0 && lane == 0) reset_linear(tile - NS * gridDim.x);
        }
        // copies still landing (if the consumers gave up) and the last tiles' reset
        if (lane == 0) {
            for (uint32_t k = it > NS ? it - NS : 0; k < it; ++k)
                if (k != withheld && mbar_wait_bounded(&full[k % NS], (k / NS) & 1u) && resets(CPL))
                    reset_linear(blockIdx.x + k * gridDim.x);
            if (resets(CPL)) bulk_wait_all();
        }
        return;
    }

    // ---- consumers: thread `ct` owns cell ct of every tile
    const int ct = tid - 32;
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x, ++it) {
        const uint32_t s = it % NS;
        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], (it / NS) & 1u, g.wait_ns));
        if (!ok) {
            if (lane == 0) atomicExch(wait_err, 1);
            return;
        }
        const unsigned char* st = stages + s * L::BYTES;
        const uint32_t k = tile * (uint32_t)L::TILE + ct;
        const bool active = (int64_t)k < g.n;
        const T* P = reinterpret_cast<const T*>(st) + ct;
        const FT* SFc = reinterpret_cast<const FT*>(st + L::OFF_FCOL) + 3 * ct;
        const FT* SFp = reinterpret_cast<const FT*>(st + L::OFF_FPREV) + 3 * ct;
        C f[Q], F[3] = {C(0), C(0), C(0)}, Fp[3] = {C(0), C(0), C(0)};
#pragma unroll
        for (int i = 0; i < Q; ++i) f[i] = Staged<T>::one(P + i * L::PITCH + g.rem[i]);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if (L::NEED_FCOL) F[q] = (C)SFc[q];
            if (CPL == kCplDense) Fp[q] = (C)SFp[q];
            else if (CPL == kCplSparse) Fp[q] = cp.body[q];
        }
        release_stage(&empty[s], lane);
        if (!active) continue;
        const Cell3 c = cell_of(d, k);
        if (c.y == 0 || c.y == d.ny - 1 || c.z == 0 || c.z == d.nz - 1) {
            C g_f[Q];  // of its own: f stays in registers
            gather_face_cell<T>(d, cp, fin, wall, c, (int64_t)k, g_f);
#pragma unroll
            for (int i = 0; i < Q; ++i) f[i] = g_f[i];
        } else if (c.x == 0 || c.x == d.nx - 1) {
            // the five populations that cross the row's end come from its other end
            T raw[5];
            auto fetch = [&](auto right) {
                constexpr int dir = decltype(right)::value ? -1 : 1;  // c_x of the populations that cross
                int n = 0;
#pragma unroll
                for (int i = 0; i < Q; ++i)
                    if (cx(i) == dir) raw[n++] = __ldg(fin + i * d.stride + ((int64_t)k - g.off[i] + dir * d.nx));
                n = 0;
#pragma unroll
                for (int i = 0; i < Q; ++i)
                    if (cx(i) == dir) f[i] = (C)raw[n++];
            };
            if (c.x == 0) fetch(std::false_type{});
            else fetch(std::true_type{});
        }
        finish_cell<T, CPL, COLL>(d, cp, fout, u_out, phase, celltype, (int64_t)k, c.y, fd_wall_node(d, c.y), f, F, Fp);
    }
}

template <class T, int CPL, int COLL>
size_t linear_smem(int nstages) {
    return 256 + LinearLayout<T, CPL, COLL>::RESET + (size_t)nstages * LinearLayout<T, CPL, COLL>::BYTES;
}

template <class T, int CPL, int COLL>
bool linear_inst(const Lattice& L, cudaStream_t s) {
    using FT = typename Store<T>::F;
    using C = typename Store<T>::C;
    using LY = LinearLayout<T, CPL, COLL>;
    const LatticeDesc& d = L.d;
    LinearGeom g{};
    g.n = d.n;
    g.stride = d.stride;
    g.ntiles = (uint32_t)((d.n + LY::TILE - 1) / LY::TILE);
    const int A = LinearOf<T>::A;
    for (int i = 0; i < Q; ++i) {
        g.off[i] = (int32_t)(cx(i) + (int64_t)d.nx * (cy(i) + (int64_t)d.ny * cz(i)));
        g.rem[i] = (int32_t)(((-(int64_t)g.off[i]) % A + A) % A);
    }
    g.wait_ns = L.wait_ns;
    g.withhold = L.withhold_tile;
    // pipeline depth: the tuning value, else as many stages as fit the resident CTAs of an SM.  The reset coupling takes
    // them too, beside the membranes' kernels (three against four, steps of one 642-vertex capsule: FP16 65^3 30.3 / 30.7
    // us, 129^3 77.0 / 79.8, FP32 101^3 64.1 / 63.3, 129^3 94.4 / 95.1; the same within 2 us at 33^3 to 129^3)
    const size_t limit = std::min<size_t>((size_t)optin_smem(), 228 * 1024 / staged_ctas_per_sm<T>()) - 1024;
    g.nstages = L.stages >= 2 ? L.stages : 2;
    for (int ns = 2; L.stages < 2 && ns <= kMaxStages; ++ns)
        if (linear_smem<T, CPL, COLL>(ns) <= limit) g.nstages = ns;
    const size_t smem = linear_smem<T, CPL, COLL>(g.nstages);
    if (smem + 1024 > (size_t)optin_smem()) return false;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto kern = k_collide_stream_linear<T, CPL, COLL>;
    // per device: the shared memory allowed (only ever raised) and, for each size, the resident CTAs per SM
    static std::mutex mu;
    static std::unordered_map<int, size_t> allowed;
    static std::unordered_map<int64_t, int> resident;
    int nb = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        size_t& lim = allowed[dev];
        if (smem > lim) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
            lim = smem;
        }
        int& r = resident[((int64_t)dev << 32) | (int64_t)smem];
        if (r == 0 && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kern, LY::THREADS, smem) != cudaSuccess || r < 1)) {
            r = 0;
            return false;
        }
        nb = r;
    }
    const unsigned grid = (unsigned)std::min<int64_t>(g.ntiles, (int64_t)nb * sms);
    const FT* Fcol = (const FT*)(CPL != kCplNone ? L.F[1 - L.fe] : L.F[L.fe]);
    FT* Fprev = resets(CPL) ? (FT*)L.F[L.fe] : nullptr;
    kern<<<grid, LY::THREADS, smem, s>>>(d, g, collide_params<C>(d, L.storage), (const T*)L.f[L.cur], (T*)L.f[1 - L.cur],
                                         (const T*)L.wall, Fcol, Fprev,
                                         writes_u(CPL) ? (typename Store<T>::U*)L.u : nullptr, L.phase, L.celltype,
                                         L.wait_err);
    return true;
}

template <class T, int CPL>
bool linear_coll(const Lattice& L, cudaStream_t s) {
    switch (L.d.collision) {
        case BIB_COLLISION_BGK_GUO_VOF: return linear_inst<T, CPL, BIB_COLLISION_BGK_GUO_VOF>(L, s);
        case BIB_COLLISION_BGK: return linear_inst<T, CPL, BIB_COLLISION_BGK>(L, s);
        default: return linear_inst<T, CPL, BIB_COLLISION_TRT>(L, s);
    }
}

template <class T>
bool linear_t(const Lattice& L, Coupling mode, cudaStream_t s) {
    switch (mode) {
        case Coupling::kDense: return linear_coll<T, kCplDense>(L, s);
        case Coupling::kSparse: return linear_coll<T, kCplSparse>(L, s);
        case Coupling::kReset: return linear_coll<T, kCplReset>(L, s);
        default: return linear_coll<T, kCplNone>(L, s);
    }
}

}  // namespace

// Where the linear tiles take over from the direct kernels (one thread per cell for odd rows, two cells per
// thread for even ones).  Measured, lattice-only steps in a row, linear against direct:
//   FP16, from 2^15 cells: 33^3 10.3 / 10.3 us, 41^3 10.3 / 11.3, 81^3 22 / 41, 129^3 47 / 181, 201^3 138 / 555,
//     1024 x 64 x 64 89 / 266: the direct kernels' 2-byte accesses are half empty;
//   FP32 odd rows, from 2^19: 61^3 16.3 / 12.4, 81^3 20.4 / 32.8, 129^3 65 / 94, 201^3 221 / 305;
//   FP32 even rows, from 2^19, only where the direct kernel leaves a quarter of its lanes without a cell:
//     102 x 101 x 100 45 / 39, 1024 x 64 x 64 141 / 114 (lanes full); 520 x 64 x 64 70 / 97 (half full).
// FP64 is bound by its arithmetic and stays with the direct kernels.
bool launch_collide_stream_linear(const Lattice& L, Coupling mode, cudaStream_t s) {
    const LatticeDesc& d = L.d;
    if (L.storage == BIB_STORAGE_F64 || !L.wait_err || d.n >= ((int64_t)1 << 31) - 4096) return false;
    if (L.storage == BIB_STORAGE_F16) return d.n >= (1 << 15) && linear_t<__half>(L, mode, s);
    const int pairs = d.nx / 2, bx = std::min(256, (pairs + 31) / 32 * 32);
    const bool full = d.nx % 2 == 0 && 4 * pairs >= 3 * bx * ((pairs + bx - 1) / bx);
    return d.n >= (1 << 19) && !full && linear_t<float>(L, mode, s);
}

}  // namespace bib
