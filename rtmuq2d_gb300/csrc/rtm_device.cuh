// rtm_device.cuh -- device helpers shared by the kernels: PTX wrappers (mbarriers, TMA, bounded
// waits), 4-wide vectors, ring geometry, 16-bit storage and the scheme's per-quad arithmetic.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "rtm_internal.h"

namespace rtm {

// 8th-order second-derivative weights (SRC/stencilDFM.h:8-12)
#define RTM_AC0 (-2.97399944f)
#define RTM_AC1 (+1.70507669f)
#define RTM_AC2 (-0.25861812f)
#define RTM_AC3 (+0.04577745f)
#define RTM_AC4 (-0.00523630f)
// 8th-order first-derivative weights (SRC/absorbingBoundaryCondition.h:21-24)
#define RTM_B1 (+0.8f)
#define RTM_B2 (-0.2f)
#define RTM_B3 (+0.025396825f)
#define RTM_B4 (-0.001785714f)

// Scale targets of 16-bit storage: the tile's max |u| is stored as this value.
constexpr float kFp16Target = 16384.0f;
constexpr float kBf16Target = 1.0f;

// ---- PTX helpers -------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1,
                                            uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait on an mbarrier phase: gives up after `limit_ns` nanoseconds.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  uint64_t limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (global_ns() - t0 > limit_ns) return false;
    }
    return true;
}

// ---- 4-wide vector helpers (16 B for float, 2 x 16 B for double) -------------------------
__device__ __forceinline__ void ld4(const float *p, float (&q)[4])
{
    const float4 v = *reinterpret_cast<const float4 *>(p);
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}
__device__ __forceinline__ void ld4(const double *p, double (&q)[4])
{
    const double2 a = reinterpret_cast<const double2 *>(p)[0];
    const double2 b = reinterpret_cast<const double2 *>(p)[1];
    q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
}
__device__ __forceinline__ void ldg4(const float *p, float (&q)[4])
{
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
}
__device__ __forceinline__ void ldg4(const double *p, double (&q)[4])
{
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    q[0] = a.x; q[1] = a.y; q[2] = b.x; q[3] = b.y;
}
// 16-byte asynchronous copy global -> shared (cp.async), its group commit and wait.
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)),
                 "l"(__cvta_generic_to_global(src))
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void st4(float *p, const float (&q)[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(q[0], q[1], q[2], q[3]);
}
__device__ __forceinline__ void st4(double *p, const double (&q)[4])
{
    reinterpret_cast<double2 *>(p)[0] = make_double2(q[0], q[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(q[2], q[3]);
}

// ---- geometry predicates -----------------------------------------------------------------
// Index of cell (x,z) in the boundary ring that encloses the reconstruction region
// [rx0,rx1) x [rz0,rz1) with a 4-cell band, or -1.  Bands: top (x-major, 4 z each),
// bottom, left (4 columns of rz1-rz0), right.
__device__ __forceinline__ int ring_index(const Geom &g, int x, int z)
{
    if (x < g.rx0 - 4 || x >= g.rx1 + 4 || z < g.rz0 - 4 || z >= g.rz1 + 4) return -1;
    if (z < g.rz0) return (x - (g.rx0 - 4)) * 4 + (z - (g.rz0 - 4));
    if (z >= g.rz1) return g.ring_w * 4 + (x - (g.rx0 - 4)) * 4 + (z - g.rz1);
    if (x < g.rx0) return g.ring_w * 8 + (x - (g.rx0 - 4)) * g.ring_h + (z - g.rz0);
    if (x >= g.rx1) return g.ring_w * 8 + 4 * g.ring_h + (x - g.rx1) * g.ring_h + (z - g.rz0);
    return -1;
}

// Whether the quad [zq, zq+4) of column x holds a ring cell (a cheap test before ring_index):
// the top and bottom bands span the ring box's columns, the side bands its rows.
__device__ __forceinline__ bool ring_quad(const Geom &g, int x, int zq)
{
    if (x < g.rx0 - 4 || x >= g.rx1 + 4) return false;
    if (x < g.rx0 || x >= g.rx1) return zq < g.rz1 + 4 && zq + 4 > g.rz0 - 4;
    return (zq < g.rz0 && zq + 4 > g.rz0 - 4) || (zq < g.rz1 + 4 && zq + 4 > g.rz1);
}

__device__ __forceinline__ bool in_region(const Geom &g, int x, int z)
{
    return x >= g.rx0 && x < g.rx1 && z >= g.rz0 && z < g.rz1;
}

__device__ __forceinline__ bool in_interior(const Geom &g, int x, int z)
{
    return x >= g.thl && x < g.thl + g.nx && z >= g.thu && z < g.thu + g.nz;
}

// Stored source-wavefield element: full precision (T) or 16-bit with a tile scale.
template <typename T>
__device__ __forceinline__ void store_put(void *base, int prec, size_t i, T v, float inv_scale)
{
    if (prec == 1)
        reinterpret_cast<__nv_bfloat16 *>(base)[i] = __float2bfloat16_rn((float)v * inv_scale);
    else if (prec == 2)
        reinterpret_cast<__half *>(base)[i] = __float2half_rn((float)v * inv_scale);
    else
        reinterpret_cast<T *>(base)[i] = v;
}

template <typename T>
__device__ __forceinline__ T store_get(const void *base, int prec, size_t i, float scale)
{
    if (prec == 1)
        return (T)(__bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(base)[i]) * scale);
    if (prec == 2) return (T)(__half2float(reinterpret_cast<const __half *>(base)[i]) * scale);
    return reinterpret_cast<const T *>(base)[i];
}

// Laplacian of the 4 cells of a quad, from the 9-column window W (x) and the 12-value z
// line zz (zm | centre | zp).  Operand order as SRC/stencilDFM.c:24-28.
template <typename T>
__device__ __forceinline__ T lap8(const T (&W)[9][4], const T (&zz)[12], int j)
{
    const T c0 = (T)2.0f * (T)RTM_AC0;
    return c0 * W[4][j]
        + (T)RTM_AC1 * (((W[3][j] + W[5][j]) + zz[3 + j]) + zz[5 + j])
        + (T)RTM_AC2 * (((W[2][j] + W[6][j]) + zz[2 + j]) + zz[6 + j])
        + (T)RTM_AC3 * (((W[1][j] + W[7][j]) + zz[1 + j]) + zz[7 + j])
        + (T)RTM_AC4 * (((W[0][j] + W[8][j]) + zz[0 + j]) + zz[8 + j]);
}

template <int WARPS>
__device__ __forceinline__ float block_max(float v, float *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = red[0];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) m = fmaxf(m, red[w]);
    __syncthreads();
    return m;
}

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" :::); }

template <typename T>
__device__ __forceinline__ T add_source(const float *wavelet, int t, T v, T cf)
{
    if (sizeof(T) == sizeof(float)) return v + (T)(wavelet[t] * (float)cf);   // float product, as the reference
    return v + (T)wavelet[t] * cf;
}

template <typename T>
__device__ __forceinline__ void image_quad(double *img, double *slf, const T (&s)[4], const T (&r)[4])
{
    double2 i0 = reinterpret_cast<double2 *>(img)[0], i1 = reinterpret_cast<double2 *>(img)[1];
    double2 s0 = reinterpret_cast<double2 *>(slf)[0], s1 = reinterpret_cast<double2 *>(slf)[1];
    i0.x += (double)s[0] * (double)r[0]; i0.y += (double)s[1] * (double)r[1];
    i1.x += (double)s[2] * (double)r[2]; i1.y += (double)s[3] * (double)r[3];
    s0.x += (double)s[0] * (double)s[0]; s0.y += (double)s[1] * (double)s[1];
    s1.x += (double)s[2] * (double)s[2]; s1.y += (double)s[3] * (double)s[3];
    reinterpret_cast<double2 *>(img)[0] = i0; reinterpret_cast<double2 *>(img)[1] = i1;
    reinterpret_cast<double2 *>(slf)[0] = s0; reinterpret_cast<double2 *>(slf)[1] = s1;
}

// First derivative (times dx) of 4 cells along x from a 9-column window W[k] = f(x-4+k):
// B4 (f+4 - f-4) + B3 (f+3 - f-3) + B2 (f+2 - f-2) + B1 (f+1 - f-1), the operand order of
// absorbingBoundaryCondition.c:177-181 (psi) and :198-203 (dpsi).
template <typename T>
__device__ __forceinline__ T d1x_w(const T (&W)[9][4], int j)
{
    return (T)RTM_B4 * (W[8][j] - W[0][j]) + (T)RTM_B3 * (W[7][j] - W[1][j])
         + (T)RTM_B2 * (W[6][j] - W[2][j]) + (T)RTM_B1 * (W[5][j] - W[3][j]);
}
// The same along z from a 12-value line q (q[4+j] is cell j).
template <typename T>
__device__ __forceinline__ T dpsi_z(const T (&q)[12], int j)
{
    return (T)RTM_B4 * (q[8 + j] - q[j]) + (T)RTM_B3 * (q[7 + j] - q[1 + j])
         + (T)RTM_B2 * (q[6 + j] - q[2 + j]) + (T)RTM_B1 * (q[5 + j] - q[3 + j]);
}
template <typename T>
__device__ __forceinline__ T d2x_w(const T (&W)[9][4], int j)
{
    return (T)RTM_AC4 * (W[8][j] + W[0][j]) + (T)RTM_AC3 * (W[7][j] + W[1][j])
         + (T)RTM_AC2 * (W[6][j] + W[2][j]) + (T)RTM_AC1 * (W[5][j] + W[3][j])
         + (T)RTM_AC0 * W[4][j];
}
template <typename T>
__device__ __forceinline__ T d2z_q(const T (&zz)[12], int j)
{
    return (T)RTM_AC4 * (zz[8 + j] + zz[j]) + (T)RTM_AC3 * (zz[7 + j] + zz[1 + j])
         + (T)RTM_AC2 * (zz[6 + j] + zz[2 + j]) + (T)RTM_AC1 * (zz[5 + j] + zz[3 + j])
         + (T)RTM_AC0 * zz[4 + j];
}

// Loads the 12-value z line (zm | centre | zp) of column row `row` of a halo tile.
template <typename T>
__device__ __forceinline__ void z_line(const T *tile, int row, int zi, const T (&c)[4], T (&zz)[12])
{
    T zm[4], zp[4];
    ld4(tile + row * SZ + zi - 4, zm);
    ld4(tile + row * SZ + zi + 4, zp);
#pragma unroll
    for (int j = 0; j < 4; ++j) { zz[j] = zm[j]; zz[4 + j] = c[j]; zz[8 + j] = zp[j]; }
}

// psi of this step on 4 cells of an x-strip column from the 9-column window of u and the
// previous psi (absorbingBoundaryCondition.c:177-181, 269-273): psi = b psi + a D1x(u) / dx on
// z in [4, dimZ-4); the other cells keep their psi.
template <typename T>
__device__ __forceinline__ void psi_x_new(const T (&W)[9][4], T (&ps)[4], T ab, T bb, T h1, int zq, int dimz)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (zq + j >= 4 && zq + j < dimz - 4) ps[j] = bb * ps[j] + ab * d1x_w<T>(W, j) * h1;
}

// Ring offset of the quad [zq, zq+4) of column x (ring_index of its first cell), or -1 when
// the quad holds no ring cell.  With quad-aligned region bounds a quad is either wholly in the
// ring or not, and its 4 cells are consecutive there (ring_save_quad writes the same offsets).
__device__ __forceinline__ long long ring_quad_offset(const Geom &g, int x, int zq)
{
    if (x < g.rx0 - 4 || x >= g.rx1 + 4 || zq < g.rz0 - 4 || zq >= g.rz1 + 4) return -1;
    if (zq < g.rz0) return (long long)(x - (g.rx0 - 4)) * 4;                              // top band
    if (zq >= g.rz1) return (long long)4 * g.ring_w + (long long)(x - (g.rx0 - 4)) * 4;   // bottom
    if (x < g.rx0) return (long long)8 * g.ring_w + (long long)(x - (g.rx0 - 4)) * g.ring_h + (zq - g.rz0);
    if (x >= g.rx1)
        return (long long)8 * g.ring_w + (long long)4 * g.ring_h + (long long)(x - g.rx1) * g.ring_h +
               (zq - g.rz0);
    return -1;
}

// The 16-bit storage scale of a block: max |v| over the cells it stores, mapped to target.
__host__ __device__ __forceinline__ float store_scale_of(float mx, int prec)
{
    const float target = prec == 2 ? kFp16Target : kBf16Target;
    // A block ahead of the wavefront can hold only denormal-size values: clamping keeps the
    // inverse finite (an infinite inverse would turn 0 into NaN).
    return fmaxf(mx, 1e-30f) / target;
}

// Strip quads of one member: every strip column x in [4, thl-4) or [dimx-thr+4, dimx-4)
// with all its z quads in [4, dimz-4) (nA items), then every column x in [0, dimx) with its
// top quads (z in [4, thu-4)) and bottom quads (z in [dimz-thd+4, dimz-4)) -- items of strip
// columns (already covered) or bottom quads outside [4, dimx-4) are skipped (nB items).
struct CorrShape {
    int nql, nA, ntq, q0, nbq, nB;
};
__host__ __device__ __forceinline__ CorrShape corr_shape(const Geom &g)
{
    CorrShape c;
    c.nql = (g.dimz - 8 + 3) / 4;
    c.nA = (g.thl - 8 + g.thr - 8) * c.nql;
    c.ntq = (g.thu - 8 + 3) / 4;
    c.q0 = (g.dimz - g.thd + 4) & ~3;
    c.nbq = (g.dimz - 4 - c.q0 + 3) / 4;
    c.nB = g.dimx * (c.ntq + c.nbq);
    return c;
}
constexpr int kStripBlock = 256;          // strip items per block (and per 16-bit ring scale)
__host__ __device__ __forceinline__ int round_block(int n)
{
    return (n + kStripBlock - 1) / kStripBlock * kStripBlock;
}

// Item index of quad (x, zq) in the list above (the quad holding a ring cell).
__device__ __forceinline__ int strip_item(const Geom &g, const CorrShape &cs, int x, int zq)
{
    if (x >= 4 && x < g.thl - 4) return (x - 4) * cs.nql + (zq - 4) / 4;
    if (x >= g.dimx - g.thr + 4 && x < g.dimx - 4)
        return (g.thl - 8 + x - (g.dimx - g.thr + 4)) * cs.nql + (zq - 4) / 4;
    const int k = zq < g.thu - 4 ? (zq - 4) / 4 : cs.ntq + (zq - cs.q0) / 4;
    return cs.nA + x * (cs.ntq + cs.nbq) + k;
}

// Cell of ring index r (inverse of ring_index).
__device__ __forceinline__ void ring_cell(const Geom &g, int r, int &x, int &z)
{
    const int w4 = g.ring_w * 4;
    if (r < w4) { x = g.rx0 - 4 + r / 4; z = g.rz0 - 4 + r % 4; return; }
    r -= w4;
    if (r < w4) { x = g.rx0 - 4 + r / 4; z = g.rz1 + r % 4; return; }
    r -= w4;
    const int h4 = 4 * g.ring_h;
    if (r < h4) { x = g.rx0 - 4 + r / g.ring_h; z = g.rz0 + r % g.ring_h; return; }
    r -= h4;
    x = g.rx1 + r / g.ring_h;
    z = g.rz0 + r % g.ring_h;
}

}  // namespace rtm
