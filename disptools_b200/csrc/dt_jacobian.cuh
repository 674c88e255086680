// Jacobian stencil of one field in any row layout (sm_100a): the map, the
// adjoint's weights, or the log of the map added to a running sum.
//
// The TMA kernels need rows a multiple of 16 bytes long.  Every other layout
// (odd widths, a base off a 16-byte boundary), second order, FP64 arithmetic on
// float fields, and FP64 volumes of less than 7.5 million voxels
// (FP64_ELEMENTWISE_VOXELS) come here.
//
// A block of 32 x 8 threads, one voxel each, marches a 32 x 8 tile through
// bz planes.  Boxes of the tile with two voxels of halo on each x-y side and
// three components arrive element by element with cp.async, JA_D planes
// ahead, in a ring of JA_NS slots; values outside the volume arrive as
// zeros.  Each thread keeps its column's values of the planes ze-2 .. ze+2 in
// registers, so a slot is free once its plane has been the stencil's centre
// plane, and one block barrier a plane guards everything.  The geometry is a
// kernel parameter: a launch needs no device memory, no lock and no wait.
//
// What bounds it: instruction issue and the latency of a plane's chain, so
// resident warps: one voxel a thread keeps FP32 at 64 registers (four blocks,
// 32 warps an SM).  Map of 181 x 217 x 181 in FP32 77 us, FP64 108-113 us; the
// plain-load kernel before it (256 threads, a 64-bit index per load, scheme by
// case analysis, a lock and a wait) 230 and 330.
#pragma once

#include <algorithm>
#include <climits>

#include "dt_kernels.cuh"
#include "dt_tma.cuh"

namespace dtb {

constexpr int JA_NT = 256, JA_D = 3, JA_NS = JA_D + 3;

// Tiles are TX voxels wide and JA_NT / TX high: 32 x 8, and 8 x 32 for volumes
// at most 16 voxels wide, which would leave most of a 32-wide tile idle.
template <int TX>
struct JaTile {
    static constexpr int X = TX, Y = JA_NT / TX;
    static constexpr int PX = X + 4, PY = Y + 4, CELLS = PX * PY, PLANE = 3 * CELLS;
    // Copies: the threads take the columns of half a component's rows at a time.
    static constexpr int RG = PY / 2;
    static_assert(RG * PX <= JA_NT && PY % 2 == 0);
};
constexpr int JA_NARROW = 16;

// Resident blocks per SM: 32 warps at 64 registers (FP32), 16 at 128 (FP64).
template <typename T>
__host__ __device__ constexpr int ja_blocks() {
    return sizeof(T) == 4 ? 4 : 2;
}

enum JacEpilogue { JAC_MAP = 0, JAC_WEIGHTS = 1, JAC_LOG = 2 };

// Epilogue arguments; arrays of scalars have the field's row and plane
// strides unless stated.
template <typename T>
struct JacOut {
    T *J = nullptr;          // JAC_MAP
    const T *gJ = nullptr;   // JAC_WEIGHTS: W[c][a] = gJ cof_ca(I + A) ih_a
    T *W = nullptr;          //   component stride wn, row and plane strides wys, wzs
    long long wn = 0, wys = 0, wzs = 0;
    double *acc = nullptr;   // JAC_LOG: the sum so far (not read by the first)
    double eps = 0.0, scale = 0.0;
    int first = 0, last = 0;  // the last writes exp(scale * sum) instead
};

template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The two central schemes of one axis as one expression of the first and
// second differences, so that a warp with voxels of both kinds evaluates it
// once: weights chosen per voxel, and the second difference dropped (not
// multiplied by zero: it may be infinite) where the scheme is second order.
// Each rounds as its scheme does: FP32 d1 k1 + d2 k2 fused, or d1 (ih / 2);
// FP64 ((d1 w1) - d2 / 12) ih half, with w1 = 2/3 and half = 1, or w1 = 1,
// d2 = 0 and half = 1/2 (exact factors).
template <typename T>
struct CentralWeights {
    T k1[3], k2[3];  // FP32; FP64: k2 = ih
    T w1, half;      // FP64
    __device__ __forceinline__ CentralWeights(const T (&ih)[3], bool c4) {
        w1 = c4 ? FD<T>::two_thirds : T(1);
        half = c4 ? T(1) : T(.5);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            k1[a] = c4 ? FD<T>::two_thirds * ih[a] : ih[a] * T(.5);
            k2[a] = sizeof(T) == 4 ? -FD<T>::one_twelfth * ih[a] : ih[a];
        }
    }
    __device__ __forceinline__ T operator()(T d1, T d2, int a) const {
        if constexpr (sizeof(T) == 4) return __fmaf_rn(d1, k1[a], __fmul_rn(d2, k2[a]));
        else return (d1 * w1 - d2 * FD<T>::one_twelfth) * k2[a] * half;
    }
};

// The stencil matrix of a voxel: `p` its element of the centre plane's box,
// zq its column's values of planes ze-2 .. ze+2.  A warp is one row of the
// tile, so `deep` (all its voxels take fourth-order differences) is uniform
// and has code without a choice per voxel.  Other voxels take fourth-order
// differences where `c4`, and are second order along every axis elsewhere
// (schemes_at), one-sided where they lie on a face.
template <int PX, int CELLS, typename TI, typename T>
__device__ __forceinline__ void stencil_voxel(const TI *p, const T (&zq)[3][5], int x, int y, int z, const Geom &g,
                                              const T (&ih)[3], bool deep, bool c4, T (&a)[3][3]) {
    auto central = [&](const CentralWeights<T> &w, auto second) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TI *q = p + c * CELLS;
            a[c][0] = w((T) q[1] - (T) q[-1], second((T) q[2] - (T) q[-2]), 0);
            a[c][1] = w((T) q[PX] - (T) q[-PX], second((T) q[2 * PX] - (T) q[-2 * PX]), 1);
            a[c][2] = w(zq[c][3] - zq[c][1], second(zq[c][4] - zq[c][0]), 2);
        }
    };
    if (deep) {
        central(CentralWeights<T>(ih, true), [](T d2) { return d2; });
        return;
    }
    central(CentralWeights<T>(ih, c4), [&](T d2) { return c4 ? d2 : T(0); });
    if (x == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TI *q = p + c * CELLS;
            a[c][0] = fd_fwd<T>(q[0], q[1], q[2], ih[0]);
        }
    }
    if (x == g.nx - 1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TI *q = p + c * CELLS;
            a[c][0] = fd_bwd<T>(q[0], q[-1], q[-2], ih[0]);
        }
    }
    if (y == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TI *q = p + c * CELLS;
            a[c][1] = fd_fwd<T>(q[0], q[PX], q[2 * PX], ih[1]);
        }
    }
    if (y == g.ny - 1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const TI *q = p + c * CELLS;
            a[c][1] = fd_bwd<T>(q[0], q[-PX], q[-2 * PX], ih[1]);
        }
    }
    if (z == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c][2] = fd_fwd<T>(zq[c][2], zq[c][3], zq[c][4], ih[2]);
    }
    if (z == g.nz - 1) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c][2] = fd_bwd<T>(zq[c][2], zq[c][1], zq[c][0], ih[2]);
    }
}

template <typename TI, typename T, int EPI, int TX>
__global__ void __launch_bounds__(JA_NT, ja_blocks<T>())
    k_jacobian_async(const TI *__restrict__ field, const Geom g, const JacOut<T> out, int bz) {
    using L = JaTile<TX>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TI *ring = reinterpret_cast<TI *>(smem_raw);
    const int tid = threadIdx.x, tx = tid % L::X, ty = tid / L::X;
    const int tiles_x = (g.nx + L::X - 1) / L::X, tiles_y = (g.ny + L::Y - 1) / L::Y;
    const int txy = (int) blockIdx.x / tiles_x;
    const int x0 = ((int) blockIdx.x - txy * tiles_x) * L::X, y0 = (txy % tiles_y) * L::Y, z0 = (txy / tiles_y) * bz;
    const int z1 = min(z0 + bz, g.nz);
    // Box positions outside the volume stay zero: their x and y are the same
    // in every plane, planes below it are never copied, planes above it are
    // cleared.
    if (z0 < 2 || y0 < 2 || x0 < 2 || y0 + L::Y + 2 > g.ny || x0 + L::X + 2 > g.nx) {
        for (int i = tid; i < JA_NS * L::PLANE; i += JA_NT) ring[i] = TI(0);
        __syncthreads();
    }
    const int rg = tid / L::PX, col = tid - rg * L::PX;
    const int gx = x0 - 2 + col, gy = y0 - 2 + rg;
    const bool col_ok = rg < L::RG && gx >= 0 && gx < g.nx;
    const bool lo = col_ok && gy >= 0 && gy < g.ny, hi = col_ok && gy + L::RG >= 0 && gy + L::RG < g.ny;
    const TI *src = field + ((z0 - 2) * g.zs + gy * g.ys + gx);  // in the next plane to copy
    // Copies plane zp (tile and halo) into its slot; always one group.
    auto load_plane = [&](int zp, int slot) {
        if (zp >= 0 && zp <= z1 + 1) {
            TI *dst = ring + slot * L::PLANE + tid;
            if (zp < g.nz) {
                const TI *up = src + L::RG * g.ys;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    if (lo) cp_async_elem<(int) sizeof(TI)>(dst + c * L::CELLS, src + c * g.cs);
                    if (hi) cp_async_elem<(int) sizeof(TI)>(dst + c * L::CELLS + L::RG * L::PX, up + c * g.cs);
                }
            } else {
                for (int i = tid; i < L::PLANE; i += JA_NT) ring[slot * L::PLANE + i] = TI(0);
            }
        }
        src += g.zs;
        cp_async_commit();
    };
    for (int j = 0; j < JA_D; ++j) load_plane(z0 - 2 + j, j);

    const int x = x0 + tx, y = y0 + ty;
    const bool in_xy = x < g.nx && y < g.ny;
    const T ih[3] = {(T) g.ih[0], (T) g.ih[1], (T) g.ih[2]};
    const bool row_in = y >= 2 && y <= g.ny - 3 && g.order == 4;
    // A warp of a wide tile is one row of it.
    const bool tile_in = TX == 32 && row_in && x0 >= 2 && x0 + L::X - 1 <= g.nx - 3;
    const bool voxel_in = row_in && x >= 2 && x <= g.nx - 3;
    const int own = (ty + 2) * L::PX + tx + 2;
    T zq[3][5];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 5; ++k) zq[c][k] = T(0);
    long long off = (z0 - 4) * g.zs + y * g.ys + x;  // of the thread's voxel in plane ze
    int slot = 0;                                    // of plane q
#pragma unroll(sizeof(T) == 4 ? 5 : 1)
    for (int q = z0 - 2; q <= z1 + 1; ++q, off += g.zs) {
        cp_async_wait_group<JA_D - 1>();
        __syncthreads();
        // The slot of plane q + D held plane q - 3, the last centre plane.
        load_plane(q + JA_D, slot + JA_D < JA_NS ? slot + JA_D : slot + JA_D - JA_NS);
        const TI *pl = ring + slot * L::PLANE + own;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int k = 0; k < 4; ++k) zq[c][k] = zq[c][k + 1];
            zq[c][4] = (T) pl[c * L::CELLS];
        }
        const int ze = q - 2;
        const int se = slot >= 2 ? slot - 2 : slot - 2 + JA_NS;
        slot = slot + 1 < JA_NS ? slot + 1 : 0;
        if (ze < z0 || !in_xy) continue;
        // What the epilogue reads, on its way during the stencil.
        T pre = T(0);
        if constexpr (EPI == JAC_WEIGHTS) pre = __ldg(out.gJ + off);
        if constexpr (EPI == JAC_LOG) pre = out.first ? T(0) : out.acc[off];
        const bool plane_in = ze >= 2 && ze <= g.nz - 3;
        T a[3][3];
        stencil_voxel<L::PX, L::CELLS, TI, T>(ring + se * L::PLANE + own, zq, x, y, ze, g, ih, tile_in && plane_in,
                             voxel_in && plane_in, a);
        if constexpr (EPI == JAC_MAP) {
            out.J[off] = det_i_plus<T>(a);
        } else if constexpr (EPI == JAC_LOG) {
            double j = (double) det_i_plus<T>(a);
            j = j < out.eps ? out.eps : j;
            const double s = pre + log(j);
            out.acc[off] = out.last ? exp(out.scale * s) : s;
        } else {
            const T w = pre;
            T *W = out.W + (ze * out.wzs + y * out.wys + x);
            a[0][0] += T(1);
            a[1][1] += T(1);
            a[2][2] += T(1);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int r0 = c == 0 ? 1 : 0, r1 = c == 2 ? 1 : 2;
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const int c0 = b == 0 ? 1 : 0, c1 = b == 2 ? 1 : 2;
                    const T minor = a[r0][c0] * a[r1][c1] - a[r0][c1] * a[r1][c0];
                    const T cof = ((c + b) & 1) ? -minor : minor;
                    W[(c * 3 + b) * out.wn] = w * cof * ih[b];
                }
            }
        }
    }
    cp_async_wait_all();
}

// Planes per block.  A block of bz planes takes bz + 4 plane-times and about
// two more to start; blocks run in waves of `slots`, of which the last is
// shorter where it leaves the SMs fewer than their `resident` blocks (a block
// alone on an SM runs faster, though not in proportion).
inline int jacobian_depth(const Geom &g, long long cols, int resident, int num_sms) {
    const long long slots = (long long) resident * num_sms;
    int best = 1;
    double best_t = 1e300;
    for (int bz = std::min(g.nz, 64); bz >= 2; --bz) {
        const long long blocks = cols * ((g.nz + bz - 1) / bz), rest = blocks % slots;
        const double last = 0.4 + 0.6 * (double) ((rest + num_sms - 1) / num_sms) / resident;
        const double t = (bz + 6) * (blocks <= slots ? 1.0 : (double) (blocks / slots) + (rest ? last : 0.0));
        if (t < best_t) {
            best_t = t;
            best = bz;
        }
    }
    return best;
}

template <typename TI, typename T, int EPI, int TX>
cudaError_t launch_jacobian_tiles(const TI *field, const Geom &g, const JacOut<T> &out, int num_sms, cudaStream_t s) {
    using L = JaTile<TX>;
    constexpr int smem = JA_NS * L::PLANE * (int) sizeof(TI);
    static std::atomic<unsigned long long> devs{0};
    const cudaError_t attr = opt_in_smem(k_jacobian_async<TI, T, EPI, TX>, smem, devs);
    if (attr != cudaSuccess) return attr;
    const long long cols = (long long) ((g.nx + L::X - 1) / L::X) * ((g.ny + L::Y - 1) / L::Y);
    const int bz = jacobian_depth(g, cols, ja_blocks<T>(), num_sms);
    const long long grid = cols * ((g.nz + bz - 1) / bz);
    if (grid > INT_MAX) return cudaErrorInvalidConfiguration;
    k_jacobian_async<TI, T, EPI, TX><<<(unsigned) grid, JA_NT, smem, s>>>(field, g, out, bz);
    count_launch();
    return cudaGetLastError();
}

template <typename TI, typename T, int EPI>
cudaError_t launch_jacobian_async(const TI *field, const Geom &g, const JacOut<T> &out, int num_sms, cudaStream_t s) {
    if (g.nx <= JA_NARROW) return launch_jacobian_tiles<TI, T, EPI, 8>(field, g, out, num_sms, s);
    return launch_jacobian_tiles<TI, T, EPI, 32>(field, g, out, num_sms, s);
}

template <typename T>
cudaError_t launch_jacobian_any(const T *field, const Geom &g, T *J, int num_sms, cudaStream_t s) {
    JacOut<T> o;
    o.J = J;
    return launch_jacobian_async<T, T, JAC_MAP>(field, g, o, num_sms, s);
}

// Whether the adjoint's weights are faster with a thread per voxel than by
// tiles: where most of a tile lies outside the volume, and for small volumes of
// second order, whose neighbours the cache serves as well.  Adjoint by voxels and
// by tiles, us: FP32, order 4 577 x 577 x 3 53 and 72, 100000 x 3 x 3 54 and 171,
// 925 x 925 x 7 421 and 302; FP64 577 x 577 x 9 220 and 248, 707 x 707 x 12 433
// and 418, 594 x 594 x 17 437 and 428; order 2, FP32 40^3 13 and 15, 70^3 24 and
// 29, 90^3 41 and 41, 110^3 75 and 64, 174 x 174 x 33 57 and 63; FP64 40^3 15 and
// 19, 81^3 41 and 43, 90^3 56 and 49.
template <typename T>
bool voxel_weights_pay(const Geom &g) {
    const bool narrow = g.nx <= JA_NARROW;
    const int tx = narrow ? JaTile<8>::X : JaTile<32>::X, ty = narrow ? JaTile<8>::Y : JaTile<32>::Y;
    const double used = (double) g.nx * g.ny / ((double) ((g.nx + tx - 1) / tx * tx) * ((g.ny + ty - 1) / ty * ty));
    if (used < (sizeof(T) == 8 && narrow ? 0.7 : 0.4)) return true;
    return g.order == 2 && used * g.nx * g.ny * g.nz < (sizeof(T) == 8 ? 5.5e5 : 7e5);
}

template <typename T>
cudaError_t launch_weights_any(const T *field, const Geom &g, const T *gJ, T *W, long long wn, long long wys,
                               long long wzs, int num_sms, cudaStream_t s) {
    JacOut<T> o;
    o.gJ = gJ;
    o.W = W;
    o.wn = wn;
    o.wys = wys;
    o.wzs = wzs;
    if (voxel_weights_pay<T>(g)) return launch_weights_voxel<T>(field, g, gJ, W, wn, wys, wzs, s);
    return launch_jacobian_async<T, T, JAC_WEIGHTS>(field, g, o, num_sms, s);
}

template <typename TI>
cudaError_t launch_log_jacobian(const TI *field, const Geom &g, double *acc, double eps, bool first, bool last,
                                double scale, int num_sms, cudaStream_t s) {
    JacOut<double> o;
    o.acc = acc;
    o.eps = eps;
    o.scale = scale;
    o.first = first;
    o.last = last;
    return launch_jacobian_async<TI, double, JAC_LOG>(field, g, o, num_sms, s);
}

#define DTB_INSTANTIATE_JACOBIAN(T)                                                                            \
    template cudaError_t launch_jacobian_any<T>(const T *, const Geom &, T *, int, cudaStream_t);              \
    template cudaError_t launch_weights_any<T>(const T *, const Geom &, const T *, T *, long long, long long,  \
                                               long long, int, cudaStream_t);

}  // namespace dtb
