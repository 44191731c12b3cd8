// rtm_resident.cu -- k_resident: many time steps of a migration's pass in one launch, its fields
// resident on the chip.
//
// The grid is cut into at most one block per SM.  A CTA keeps its block of every field it needs
// (forward: u; backward: the receiver field and, with ring storage, the source field being
// reconstructed) in shared memory with an 8-cell halo, the previous field and the CPML's xi in
// tensor memory (each thread reads back only what it wrote itself, 128 words a thread), and psi in
// shared memory.  Per step it exchanges the cells around its block with its four neighbours and
// reads nothing else of the fields: the per-step kernels re-read 16 B (forward) to 28 B (backward)
// a cell and pay a launch, a grid drain and a chain of dependent global loads in the CPML tiles.
//
// Exchange: each side of a block has a mailbox in global memory, two parities deep.  A value
// travels with the tag of its step in one 8-byte word, so that a reader polls the data itself and
// no fence or separate flag is needed.  A block overwrites a parity two steps later, which it can
// only reach after its neighbour has published the step in between, that is, after that neighbour
// has read this one.  Every wait is bounded and ends with the status flag.
//
// The arithmetic of a cell is the per-step kernels', in the same operand order (lap8, d1x_w, ...):
// SRC/stencilDFM.c:17-29, SRC/absorbingBoundaryCondition.c:150-361, SRC/forward_modeling.c:98-130,
// SRC/backward_modeling.c:268-297.
#include <algorithm>

#include "rtm_device.cuh"

namespace rtm {

// ---- tensor memory as thread-private storage --------------------------------------------------
// 32x32b accesses: lane l of warp w reaches row 32 (w % 4) + l; the four warps of a row group take
// 128 columns each.  Every access is warp-wide.
__device__ __forceinline__ void tm_alloc(uint32_t *dst)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(dst))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tm_free(uint32_t base)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}
template <typename T> struct TmQuad;
template <> struct TmQuad<float> {
    static constexpr int WORDS = 4;
    uint32_t r[4];
    __device__ __forceinline__ void load(uint32_t a)
    {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
    }
    // the values exist only after the wait: it takes them as operands
    __device__ __forceinline__ void wait(float (&q)[4])
    {
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]));
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = __uint_as_float(r[j]);
    }
    static __device__ __forceinline__ void store(uint32_t a, const float (&q)[4])
    {
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a),
                     "r"(__float_as_uint(q[0])), "r"(__float_as_uint(q[1])), "r"(__float_as_uint(q[2])),
                     "r"(__float_as_uint(q[3])));
    }
};
template <> struct TmQuad<double> {
    static constexpr int WORDS = 8;
    uint32_t r[8];
    __device__ __forceinline__ void load(uint32_t a)
    {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                       "=r"(r[7]) : "r"(a));
    }
    __device__ __forceinline__ void wait(double (&q)[4])
    {
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                       "+r"(r[7]));
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = __hiloint2double((int)r[2 * j + 1], (int)r[2 * j]);
    }
    static __device__ __forceinline__ void store(uint32_t a, const double (&q)[4])
    {
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[2 * j] = (uint32_t)__double2loint(q[j]);
            w[2 * j + 1] = (uint32_t)__double2hiint(q[j]);
        }
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a),
                     "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]));
    }
};
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;"); }

// ---- mailboxes -----------------------------------------------------------------------------
// A quad is 4 sizeof(T) / 4 words of (tag << 32 | 32 bits), two words an access; each word is
// read and written whole.
template <typename T> constexpr int kXWords = 4 * (int)sizeof(T) / 4;

__device__ __forceinline__ void x_st2(unsigned long long *p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void x_ld2(const unsigned long long *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
template <typename T>
__device__ __forceinline__ void x_put(unsigned long long *p, const T (&q)[4], unsigned tag)
{
    constexpr int N = kXWords<T>;
    uint32_t w[N];
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __float_as_uint(q[j]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            w[2 * j] = (uint32_t)__double2loint(q[j]);
            w[2 * j + 1] = (uint32_t)__double2hiint(q[j]);
        }
    }
    const unsigned long long hi = (unsigned long long)tag << 32;
#pragma unroll
    for (int j = 0; j < N; j += 2) x_st2(p + j, hi | w[j], hi | w[j + 1]);
}
template <typename T>
struct XQuad {
    static constexpr int N = kXWords<T>;
    unsigned long long w[N];
    __device__ __forceinline__ void load(const unsigned long long *p)
    {
#pragma unroll
        for (int j = 0; j < N; j += 2) x_ld2(p + j, w[j], w[j + 1]);
    }
    __device__ __forceinline__ bool ready(unsigned tag) const
    {
        bool ok = true;
#pragma unroll
        for (int j = 0; j < N; ++j) ok = ok && (unsigned)(w[j] >> 32) == tag;
        return ok;
    }
    __device__ __forceinline__ void get(T (&q)[4]) const
    {
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = __uint_as_float((uint32_t)w[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = __hiloint2double((int)(uint32_t)w[2 * j + 1], (int)(uint32_t)w[2 * j]);
        }
    }
};
constexpr uint64_t kResWaitNs = 2000000000ull;

// Polls the quad at p until it carries `tag`; gives up after kResWaitNs, or as soon as another
// block has (the status word).
template <typename T>
__device__ __forceinline__ bool x_poll(XQuad<T> &x, const unsigned long long *p, unsigned tag, const unsigned *status)
{
    if (x.ready(tag)) return true;
    const uint64_t s0 = global_ns();
    for (unsigned n = 1;; ++n) {
        x.load(p);
        if (x.ready(tag)) return true;
        if ((n & 63u) == 0) {
            if (global_ns() - s0 > kResWaitNs) return false;
            if (*reinterpret_cast<const volatile unsigned *>(status) != 0) return false;
        }
    }
}

// Makes v opaque to the optimiser at this point of a loop: what is computed from it is computed in
// the step, not kept in registers (and, past 128, in local memory) over all steps.
__device__ __forceinline__ void opaque(int &v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void opaque(unsigned &v) { asm volatile("" : "+r"(v)); }

// What one thread of a block works on: quad q of the columns [xk, xk + len) of the block.
struct ResThread {
    int q, xk, len;
    bool own;                   // false: a spare thread (repeats a column, stores nothing)
};

// i / d for 0 <= i < 65536 and inv = 1.0f / d: (i + 1/2) / d is at least 1 / (2 d) from a whole number,
// far above the rounding of the product.
__device__ __forceinline__ int fast_div(int i, float inv) { return (int)(((float)i + 0.5f) * inv); }

// Halo of a block: what crosses its sides, for the propagated field (f = 0: depths d) and, in a
// reconstruction step, the source field (f = 1: depths e).
struct ResHalo {
    int d[4], e[4];             // depths: left, right (columns), up, down (quads)
    int n0, n;                  // items of f = 0, of both
};
__device__ __forceinline__ int halo_count(const ResShape &h, const int (&d)[4])
{
    return (d[0] + d[1]) * h.HQ + (d[2] + d[3]) * h.W;
}
// Item i of the halo (IN: received, else sent), packed: its quad's place in the tiles (f = 1 follows
// f = 0; bits 0-14), its side (15-16), f (17) and its quad in the side's mailbox (18-).  The items
// are the same at every step: a thread works its own out once.
template <bool IN>
__device__ __forceinline__ unsigned halo_item(const ResShape &h, const ResHalo &w, int i)
{
    if (i >= w.n) return 0u;
    const unsigned f = i >= w.n0;
    const int *d = f ? w.e : w.d;
    if (f) i -= w.n0;
    const int nl = d[0] * h.HQ, nx = (d[0] + d[1]) * h.HQ;
    int side, quad, x, z;
    if (i < nx) {
        side = i < nl ? 0 : 1;
        quad = i < nl ? i : i - nl;
        const int k = quad / h.HQ;
        z = 4 * (quad - k * h.HQ);
        // received: left columns -d .. -1, right columns W .. W+d-1 of the block;
        // sent: left columns 0 .. d-1, right columns W-d .. W-1
        x = side == 0 ? (IN ? k - d[0] : k) : (IN ? h.W + k : h.W - d[1] + k);
    } else {
        i -= nx;
        side = i < d[2] * h.W ? 2 : 3;
        quad = side == 2 ? i : i - d[2] * h.W;
        const int dq = d[side];                                   // depth 1 or 2 quads
        x = dq == 1 ? quad : quad >> 1;
        z = dq == 1 ? 0 : 4 * (quad & 1);
        if (side == 2) z += IN ? -4 * dq : 0;
        else z += IN ? h.H : h.H - 4 * dq;
    }
    const int at = (f ? h.field : 0) + (x + kResPad) * h.SP + kResPad + z;
    return (unsigned)(at >> 2) | (unsigned)side << 15 | f << 17 | (unsigned)quad << 18;
}
// Mailboxes of the block, by parity, field and side: the address of each one's first quad.
struct ResBox {
    unsigned long long *at[16];
};
__device__ __forceinline__ unsigned long long *res_box(const unsigned (&off)[4], const int (&cap)[4], int i, unsigned long long *xch,
                                                       int words)
{
    const int side = i & 3, f = (i >> 2) & 1, par = i >> 3;
    return xch + (size_t)(off[side] + (unsigned)((2 * f + par) * cap[side])) * words;
}
// The item's words at parity par.
template <typename T>
__device__ __forceinline__ unsigned long long *halo_word(const ResBox &b, unsigned item, int par)
{
    return b.at[par * 8 + ((item >> 15) & 7u)] + (item >> 18) * kXWords<T>;
}

// Receives the first n items of the halo (this thread's: in[k] = item tid + k kResThreads); false
// when a wait ran out.  Two items a round: their loads are in flight together.
template <typename T>
__device__ __forceinline__ bool res_recv(const ResBox &b, int tid, const unsigned (&in)[kResItems], int n, unsigned tag,
                                         T *tile, const unsigned *status)
{
    const int par = (int)(tag & 1u);
    bool ok = true;
#pragma unroll
    for (int r = 0; r < kResItems; r += 2) {
        if (r > 0 && r * kResThreads >= n) break;
        const unsigned long long *p[2];
        XQuad<T> x[2];
        bool have[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            have[k] = tid + (r + k) * kResThreads < n;
            if (have[k]) {
                p[k] = halo_word<T>(b, in[r + k], par);
                x[k].load(p[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (have[k]) {
                ok = ok && x_poll<T>(x[k], p[k], tag, status);
                T q[4];
                x[k].get(q);
                st4(tile + 4 * (in[r + k] & 0x7fffu), q);
            }
    }
    return ok;
}

// Publishes the first n items that the neighbours need, R a round: their loads are in flight together.
template <typename T, int R>
__device__ __forceinline__ void res_send(const ResBox &b, int tid, const unsigned (&out)[kResItems], int n, unsigned tag,
                                         const T *tile)
{
    const int par = (int)(tag & 1u);
#pragma unroll
    for (int r = 0; r < kResItems; r += R) {
        if (r > 0 && r * kResThreads >= n) break;
        T q[R][4];
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (tid + (r + k) * kResThreads < n) ld4(tile + 4 * (out[r + k] & 0x7fffu), q[k]);
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (tid + (r + k) * kResThreads < n)
                x_put<T>(halo_word<T>(b, out[r + k], par), q[k], tag);
    }
}

// psi of the step on the block's strip cells and 4 beyond (absorbingBoundaryCondition.c:171-189,
// 219-235, 265-281, 312-328): psi = b psi + a D1(u) / dx, in place.  A thread keeps its quad of a
// column and strides over the columns.
struct ResPsi {
    int lo[4], hi[4];           // updated columns (left, right) or rows (top, bottom)
    int rows[4];                // quads of a column of it (0: no such strip in the block)
    float inv[4];               // 1 / rows
};
__device__ __forceinline__ void res_psi_init(const Geom &g, const ResShape &h, ResPsi &w)
{
    for (int k = 0; k < 4; ++k) {
        int lo, hi, rows;
        if (k < 2) {
            const int nc = k == 0 ? h.nl : h.nr, c0 = k == 0 ? h.cl0 : h.cr0;
            lo = max(c0 - 4, k == 0 ? 4 : g.dimx - g.thr + 4);
            hi = min(c0 + nc + 4, k == 0 ? g.thl - 4 : g.dimx - 4);
            rows = nc ? h.HQ : 0;
        } else {
            const int hh = k == 2 ? h.ht : h.hb, q0 = k == 2 ? h.qt0 : h.qb0;
            const int zlo = k == 2 ? 4 : g.dimz - g.thd + 4, zhi = k == 2 ? g.thu - 4 : g.dimz - 4;
            lo = max(q0 - 4, zlo & ~3);
            hi = min(q0 + hh + 4, (zhi + 3) & ~3);
            rows = hh ? (hi - lo) >> 2 : 0;
        }
        w.lo[k] = lo;
        w.hi[k] = hi;
        w.rows[k] = rows;
        w.inv[k] = 1.0f / (float)max(rows, 1);
    }
}
template <typename T>
__device__ __forceinline__ void res_psi(const ResJob<T> &J, const ResCta &c, const ResShape &h, const ResPsi &w, int tid,
                                        const T *su, T *sm, const float *px, const float *pz)
{
    const T h1 = J.h1;
    const int sp = h.SP, dimz = J.g.dimz;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {             // left, right
        const int rows = w.rows[side];
        if (rows == 0) continue;
        const int k = fast_div(tid, w.inv[side]), q = tid - k * rows, ks = fast_div(kResThreads, w.inv[side]);
        const int ph = h.PH, hi = w.hi[side], zq = c.za + 4 * q;
        if (k >= ks) continue;
        int x = w.lo[side] + k;
        T *pp = sm + (side ? h.offr + (x - h.cr0 + 4) * ph : h.offl + (x - h.cl0 + 4) * ph) + 4 * q;
        const T *up = su + (x - 4 - c.xa + kResPad) * sp + kResPad + 4 * q;
        const float2 *pr = reinterpret_cast<const float2 *>(px) + (x - c.xa + 4);
        // two quads at a time: their loads come before either store
#pragma unroll 1
        for (; x < hi; x += 2 * ks, pp += 2 * ks * ph, up += 2 * ks * sp, pr += 2 * ks) {
            const bool two = x + ks < hi;
            T ps[2][4], d1[2][4];
            float2 ab[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int o = u && two ? ks : 0;
                ab[u] = pr[o];
                ld4(pp + o * ph, ps[u]);
                T W[9][4];
#pragma unroll
                for (int m = 0; m < 9; ++m)
                    if (m != 4) ld4(up + (o + m) * sp, W[m]);
#pragma unroll
                for (int j = 0; j < 4; ++j) d1[u][j] = d1x_w<T>(W, j);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u && !two) break;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (zq + j < dimz - 4) ps[u][j] = (T)ab[u].y * ps[u][j] + (T)ab[u].x * d1[u][j] * h1;
                st4(pp + (u ? ks * ph : 0), ps[u]);
            }
        }
    }
#pragma unroll 1
    for (int side = 2; side < 4; ++side) {             // top, bottom
        const int rows = w.rows[side];
        if (rows == 0) continue;
        const int k = fast_div(tid, w.inv[side]), q = tid - k * rows, ks = fast_div(kResThreads, w.inv[side]);
        if (k >= ks) continue;
        const int zq = w.lo[side] + 4 * q, W = h.W, pt = side == 2 ? h.PT : h.PB;
        const int zlo = side == 2 ? 4 : dimz - J.g.thd + 4, zhi = side == 2 ? J.g.thu - 4 : dimz - 4;
        T *pp = sm + (side == 2 ? h.offt + k * pt + (zq - (h.qt0 - 4)) : h.offb + k * pt + (zq - (h.qb0 - 4)));
        const T *up = su + (k + kResPad) * sp + kResPad + (zq - c.za);
        float aa[4], bz[4];
        ld4(pz + 2 * (zq - c.za + kResPad), aa);
        ld4(pz + 2 * (zq - c.za + kResPad) + 4, bz);
#pragma unroll 1
        for (int x = k; x < W; x += 2 * ks, pp += 2 * ks * pt, up += 2 * ks * sp) {
            const bool two = x + ks < W;
            T ps[2][4], d1[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int o = u && two ? ks : 0;
                T zz[12], zm[4], c4[4], zp[4];
                ld4(pp + o * pt, ps[u]);
                ld4(up + o * sp - 4, zm);
                ld4(up + o * sp, c4);
                ld4(up + o * sp + 4, zp);
#pragma unroll
                for (int m = 0; m < 4; ++m) { zz[m] = zm[m]; zz[4 + m] = c4[m]; zz[8 + m] = zp[m]; }
#pragma unroll
                for (int m = 0; m < 4; ++m) d1[u][m] = dpsi_z<T>(zz, m);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u && !two) break;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int z = zq + m;
                    if (z >= zlo && z < zhi) ps[u][m] = (T)bz[m] * ps[u][m] + (T)aa[m] * d1[u][m] * h1;
                }
                st4(pp + (u ? ks * pt : 0), ps[u]);
            }
        }
    }
}

// Blocks of at most NC = 1 or 2 columns a thread keep a thread's private values in registers, the
// others in tensor memory (ResPriv).
template <typename T, int NC>
struct ResPriv {
    T prv[2][NC][4];            // previous field, of f = 0 and 1
    T xx[NC][4], xz[NC][4];     // xi of the x and z strips
    T cf[NC][4];                // coef
    T v[NC][4];                 // new values
};
template <typename T>
struct ResPriv<T, 0> {
    T cf[1][4];                 // coef of the first column, read at every step: tensor memory has the others'
};
// Tensor-memory address of coef of a thread's column col >= 1, behind the private values.
template <typename T>
__device__ __forceinline__ uint32_t res_coef_at(const ResShape &h, uint32_t tm, int col)
{
    return tm + (uint32_t)((h.CW * h.nslot + col - 1) * TmQuad<T>::WORDS);
}

// The leapfrog of one quad (SRC/stencilDFM.c:17-29): W its 9-column window, zz its z line.
template <typename T>
__device__ __forceinline__ void leap_quad(const T (&W)[9][4], const T (&zm)[4], const T (&zp)[4], const T (&cf)[4],
                                          const T (&prv)[4], T (&v)[4])
{
    T zz[12];
#pragma unroll
    for (int j = 0; j < 4; ++j) { zz[j] = zm[j]; zz[4 + j] = W[4][j]; zz[8 + j] = zp[j]; }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = cf[j] * lap8<T>(W, zz, j) + (T)2.0f * W[4][j] - prv[j];
}

// The leapfrog of a thread's columns.  A 9-column register window along x, the column loop unrolled
// so that the window turns without moves: 3 new 16-byte shared loads a quad and two of tensor memory,
// a column ahead (previous field, coef; from the second-level cache, coef made a column take 420 ns
// instead of 330).  The new values go to tensor memory, over the previous field
// they consume (res_store swaps them into the tile): held in registers until the block has read the
// old tile they would spill, and a spill misses the little first-level cache that the tiles leave.
template <typename T, int NC>
__device__ __forceinline__ void res_leap(const ResJob<T> &J, const ResCta &c, const ResShape &h, const ResThread &th,
                                         int f, const T *su, uint32_t tm, ResPriv<T, NC> &me)
{
    constexpr int NU = NC > 0 ? NC : kResCols;
    constexpr int QW = TmQuad<T>::WORDS;
    const int sp = h.SP, cw = h.CW;
    const T *row = su + (th.xk + kResPad - 4) * sp + kResPad + 4 * th.q;
    T W[9][4];
    if constexpr (NC > 0) {
#pragma unroll
        for (int m = 0; m < 8; ++m) ld4(row + m * sp, W[m]);
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            if (u > 0 && u >= cw) break;
            T zm[4], zp[4];
            ld4(row + 8 * sp, W[8]);
            ld4(row + 4 * sp - 4, zm);
            ld4(row + 4 * sp + 4, zp);
            // f is a constant at every call
            leap_quad<T>(W, zm, zp, me.cf[u], f == 0 ? me.prv[0][u] : me.prv[1][u], me.v[u]);
#pragma unroll
            for (int j = 0; j < 4; ++j) (f == 0 ? me.prv[0] : me.prv[1])[u][j] = W[4][j];
            row += sp;
#pragma unroll
            for (int m = 0; m < 8; ++m)
#pragma unroll
                for (int j = 0; j < 4; ++j) W[m][j] = W[m + 1][j];
        }
    } else {
        const uint32_t cstep = (uint32_t)(h.nslot * QW);
        uint32_t ta = tm + (uint32_t)(f * QW), tac = res_coef_at<T>(h, tm, 1);
        TmQuad<T> tp, tc;
        tp.load(ta);
#pragma unroll
        for (int m = 0; m < 8; ++m) ld4(row + m * sp, W[m]);
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            T zm[4], zp[4], cf[4], prv[4], v[4];
            ld4(row + 8 * sp, W[8]);
            ld4(row + 4 * sp - 4, zm);
            ld4(row + 4 * sp + 4, zp);
            tp.wait(prv);
            if (u > 0) tc.wait(cf);
            else {
#pragma unroll
                for (int j = 0; j < 4; ++j) cf[j] = me.cf[0][j];
            }
            const uint32_t to = ta;
            ta += cstep;
            if (u + 1 < cw) {
                tp.load(ta);
                tc.load(tac);
                tac += QW;
            }
            leap_quad<T>(W, zm, zp, cf, prv, v);
            TmQuad<T>::store(to, v);
            if (u + 1 >= cw) break;
            row += sp;
#pragma unroll
            for (int m = 0; m < 8; ++m)
#pragma unroll
                for (int j = 0; j < 4; ++j) W[m][j] = W[m + 1][j];
        }
    }
}

// What stays the same for a thread of a strip block at every step, with NC > 0: its psi quads (a count
// in the left or right strip and one in the top or bottom one, at a fixed stride of columns) and where
// the psi of its own quads lies.  Worked out at every step, the index arithmetic and its chain of
// shared loads took a third of a small grid's step.  (A block that holds both strips of an axis runs
// with NC = 0.)
// Packed: they live in registers over all steps, and a word spilt costs a way to the second-level
// cache at every one (offsets are below 65536: 224 KB hold 57344 values).
struct ResFix {
    unsigned x, z;              // psi (low half), u (high half) of the first x / z quad; u at the first of its rows
    unsigned xw, zw;            // profile's column or quad (10 bits), stride in columns (10), count (9), x: cells before the frame (3)
    unsigned s;                 // psi of the thread's own first quad in the x (low) and z strip
    unsigned bits;              // zlo 3, zhi 3: cells of the z quad; slo 3, shi 3: ... of its own quads in the z strip;
                                // sl 3: their cells before the frame; xm 2: its columns in the x strip; xfirst 1
    __device__ __forceinline__ int get(int at, int n) const { return (int)((bits >> at) & ((1u << n) - 1u)); }
    __device__ __forceinline__ int zlo() const { return get(0, 3); }
    __device__ __forceinline__ int zhi() const { return get(3, 3); }
    __device__ __forceinline__ int slo() const { return get(6, 3); }
    __device__ __forceinline__ int shi() const { return get(9, 3); }
    __device__ __forceinline__ int sl() const { return get(12, 3); }
    __device__ __forceinline__ bool in_x(int u) const { return get(15 + u, 1); }
    __device__ __forceinline__ bool xfirst() const { return get(17, 1); }
};
__device__ __forceinline__ void res_fix_init(const Geom &g, const ResCta &c, const ResShape &h, const ResPsi &w,
                                             const ResThread &th, int tid, ResFix &f)
{
    auto cells = [](int n) { return (unsigned)min(max(n, 0), 4); };
    f.x = f.z = f.xw = f.zw = f.s = 0u;
    const int zq = c.za + 4 * th.q;
    f.bits = cells(g.dimz - 4 - zq) << 12 | 1u << 17;
    int first = 0;              // threads with quads of the x strip, in whole warps
    if (h.nl || h.nr) {
        const int side = h.nl ? 0 : 1, rows = w.rows[side], ks = kResThreads / rows, k = tid / rows, q = tid - k * rows;
        const int x = w.lo[side] + k;
        if (k < ks && x < w.hi[side]) {
            f.x = (unsigned)((side ? h.offr + (x - h.cr0 + 4) * h.PH : h.offl + (x - h.cl0 + 4) * h.PH) + 4 * q) |
                  (unsigned)((x - 4 - c.xa + kResPad) * h.SP + kResPad + 4 * q) << 16;
            f.xw = (unsigned)(x - c.xa + 4) | (unsigned)ks << 10 | (unsigned)((w.hi[side] - x + ks - 1) / ks) << 20 |
                   cells(g.dimz - 4 - (c.za + 4 * q)) << 29;
        }
        const int x0 = c.xa + th.xk;
        for (int u = 0; u < 2; ++u)
            if (side == 0 ? x0 + u < g.thl - 4 : x0 + u >= g.dimx - g.thr + 4) f.bits |= 1u << (15 + u);
        if (f.bits & (3u << 15)) f.s = (unsigned)((side ? h.offr + (x0 - h.cr0 + 4) * h.PH : h.offl + (x0 - h.cl0 + 4) * h.PH) + 4 * th.q);
        first = min(kResThreads, ((w.hi[side] - w.lo[side]) * rows + 31) & ~31);
    }
    if (h.ht || h.hb) {
        // the threads after those of the x strip come first: a corner's two kinds run side by side
        const int turn = (tid - first) & (kResThreads - 1);
        const int side = h.ht ? 2 : 3, rows = w.rows[side], ks = kResThreads / rows, k = turn / rows, q = turn - k * rows;
        const int zp = w.lo[side] + 4 * q, pt = side == 2 ? h.PT : h.PB, off = side == 2 ? h.offt : h.offb;
        const int q0 = (side == 2 ? h.qt0 : h.qb0) - 4;
        const int zlo = side == 2 ? 4 : g.dimz - g.thd + 4, zhi = side == 2 ? g.thu - 4 : g.dimz - 4;
        if (k < ks && k < h.W) {
            f.z = (unsigned)(off + k * pt + (zp - q0)) | (unsigned)((k + kResPad) * h.SP + kResPad + (zp - c.za)) << 16;
            f.zw = (unsigned)((zp - c.za + kResPad) >> 2) | (unsigned)ks << 10 | (unsigned)((h.W - k + ks - 1) / ks) << 20;
            f.bits |= cells(zlo - zp) | cells(zhi - zp) << 3;
        }
        if (zlo - zq < 4 && zhi - zq > 0) {
            f.s |= (unsigned)(off + th.xk * pt + (zq - q0)) << 16;
            f.bits |= cells(zlo - zq) << 6 | cells(zhi - zq) << 9;
        }
        if (!h.nl && side != 3) f.bits &= ~(1u << 17);
    }
}
template <typename T>
__device__ __forceinline__ void res_psi_fix(const ResFix &f, const ResShape &h, T h1, const T *su, T *sm, const float *px,
                                            const float *pz)
{
    const int sp = h.SP;
    if (f.xw) {
        const int ks = (int)((f.xw >> 10) & 1023u), ph = h.PH, xl = (int)(f.xw >> 29);
        T *pp = sm + (f.x & 0xffffu);
        const T *up = su + (f.x >> 16);
        const float2 *pr = reinterpret_cast<const float2 *>(px) + (f.xw & 1023u);
#pragma unroll 1
        for (int i = (int)((f.xw >> 20) & 511u); i > 0; --i, pp += ks * ph, up += ks * sp, pr += ks) {
            T ps[4], W[9][4];
            const float2 ab = *pr;
            ld4(pp, ps);
#pragma unroll
            for (int m = 0; m < 9; ++m)
                if (m != 4) ld4(up + m * sp, W[m]);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < xl) ps[j] = (T)ab.y * ps[j] + (T)ab.x * d1x_w<T>(W, j) * h1;
            st4(pp, ps);
        }
    }
    if (f.zw) {
        const int ks = (int)((f.zw >> 10) & 1023u), pt = h.ht ? h.PT : h.PB;
        T *pp = sm + (f.z & 0xffffu);
        const T *up = su + (f.z >> 16);
        float aa[4], bz[4];
        ld4(pz + 8 * (f.zw & 1023u), aa);
        ld4(pz + 8 * (f.zw & 1023u) + 4, bz);
#pragma unroll 1
        for (int i = (int)(f.zw >> 20); i > 0; --i, pp += ks * pt, up += ks * sp) {
            T ps[4], zz[12], zm[4], c4[4], zp[4];
            ld4(pp, ps);
            ld4(up - 4, zm);
            ld4(up, c4);
            ld4(up + 4, zp);
#pragma unroll
            for (int m = 0; m < 4; ++m) { zz[m] = zm[m]; zz[4 + m] = c4[m]; zz[8 + m] = zp[m]; }
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m >= f.zlo() && m < f.zhi()) ps[m] = (T)bz[m] * ps[m] + (T)aa[m] * dpsi_z<T>(zz, m) * h1;
            st4(pp, ps);
        }
    }
}

// The CPML corrections of quad u of a thread of a strip block (absorbingBoundaryCondition.c:191-217,
// 237-263, 283-310, 330-357), added to its new values v in the reference's order left, top, right,
// bottom; xx, xz: the quad's xi, updated.  up: its u in the tile; psx, psz: its psi.  D1(psi) and D2(u)
// along x are summed a pair of rows at a time, the outermost first, in the operand order of d1x_w / d2x_w.
template <typename T>
__device__ __forceinline__ void res_strip_quad(const ResFix &f, int u, T h1, T h2, T h3, int sp, int ph, const T *up,
                                               const T *psx, const T *psz, float2 pr, const float *pz, const T (&cf)[4],
                                               T (&xx)[4], T (&xz)[4], T (&v)[4])
{
    T dX[4] = {(T)0, (T)0, (T)0, (T)0}, dZ[4] = {(T)0, (T)0, (T)0, (T)0}, uc[4];
    const bool inX = f.in_x(u), inZ = f.slo() < f.shi();
    ld4(up, uc);
    if (inX) {
        const T ab = (T)pr.x, bb = (T)pr.y;
        const T bk[4] = {(T)RTM_B4, (T)RTM_B3, (T)RTM_B2, (T)RTM_B1};
        const T ak[4] = {(T)RTM_AC4, (T)RTM_AC3, (T)RTM_AC2, (T)RTM_AC1};
        T acc[4], d2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            T mk[4], pk[4], um[4], uq[4];
            ld4(psx - (4 - k) * ph, mk);
            ld4(psx + (4 - k) * ph, pk);
            ld4(up - (4 - k) * sp, um);
            ld4(up + (4 - k) * sp, uq);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const T term = bk[k] * (pk[j] - mk[j]);
                acc[j] = k == 0 ? term : acc[j] + term;
                const T dterm = ak[k] * (uq[j] + um[j]);
                d2[j] = k == 0 ? dterm : d2[j] + dterm;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            d2[j] = d2[j] + (T)RTM_AC0 * uc[j];
            if (j < f.sl()) {
                const T dp = acc[j] * h1;
                const T xn = bb * xx[j] + ab * (d2[j] * h3 + dp);
                xx[j] = xn;
                dX[j] = (cf[j] * h2) * (dp + xn);
            }
        }
    }
    if (inZ) {
        float aa[4], bz[4];
        ld4(pz, aa);
        ld4(pz + 4, bz);
        T q[12], zz[12], a0[4], a1[4], a2[4];
        ld4(psz - 4, a0);
        ld4(psz, a1);
        ld4(psz + 4, a2);
#pragma unroll
        for (int j = 0; j < 4; ++j) { q[j] = a0[j]; q[4 + j] = a1[j]; q[8 + j] = a2[j]; }
        ld4(up - 4, a0);
        ld4(up + 4, a2);
#pragma unroll
        for (int j = 0; j < 4; ++j) { zz[j] = a0[j]; zz[4 + j] = uc[j]; zz[8 + j] = a2[j]; }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j >= f.slo() && j < f.shi()) {
                const T dp = dpsi_z<T>(q, j) * h1;
                const T xn = (T)bz[j] * xz[j] + (T)aa[j] * (d2z_q<T>(zz, j) * h3 + dp);
                xz[j] = xn;
                dZ[j] = (cf[j] * h2) * (dp + xn);
            }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (inX && f.xfirst()) v[j] = v[j] + dX[j];
        if (inZ) v[j] = v[j] + dZ[j];
        if (inX && !f.xfirst()) v[j] = v[j] + dX[j];
        if (j >= f.sl()) v[j] = (T)0;                      // the grid's frame stays zero
    }
}

// A product that stays one: the correction is rounded before it is added, as in the other kernels.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// With the values in tensor memory each strip is a pass of its own, in the same order, two columns at
// a time so that one's loads cover the other's arithmetic, and without branches: lanes outside the
// strip work on the strip's nearest quad and keep their values.
// Left (side 0) and right (1) strips: the columns of the thread that lie in them.
template <typename T>
__device__ __forceinline__ void res_strip_x(const ResJob<T> &J, const ResCta &c, const ResShape &h, const ResThread &th,
                                            int side, const T *su, const T *sm, const float *px, uint32_t tm,
                                            const T (&cf0)[4])
{
    constexpr int QW = TmQuad<T>::WORDS, U = 2;
    const uint32_t cstep = (uint32_t)(h.nslot * QW), ox = (uint32_t)(h.xslot * QW);
    const int sp = h.SP, ph = h.PH, zl = J.g.dimz - 4 - c.za - 4 * th.q;              // cells before the frame
    const T h1 = J.h1, h2 = J.h2, h3 = J.h3;
    const int beg = side == 0 ? 0 : h.cr0 - c.xa, end = side == 0 ? h.nl : h.W;       // columns of the block
    // the warp's columns of the strip (a lane's chunk may start a chunk further on)
    const int lo = __reduce_min_sync(0xffffffffu, max(0, beg - th.xk));
    const int hi = __reduce_max_sync(0xffffffffu, min(h.CW, end - th.xk));
    const T *ub = su + kResPad * sp + kResPad + 4 * th.q;
    const T *pb = sm + (side == 0 ? h.offl : h.offr) + 4 * th.q;
    const float2 *pr = reinterpret_cast<const float2 *>(px) + 4;
    const T bk[4] = {(T)RTM_B4, (T)RTM_B3, (T)RTM_B2, (T)RTM_B1};
    const T ak[4] = {(T)RTM_AC4, (T)RTM_AC3, (T)RTM_AC2, (T)RTM_AC1};
#pragma unroll 1
    for (int col = lo; col < hi; col += U) {
        TmQuad<T> tv[U], tc[U], tx[U];
        T acc[U][4], d2[U][4];
        float2 ab[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int cc = min(col + u, hi - 1);
            tv[u].load(tm + cc * cstep);
            tc[u].load(res_coef_at<T>(h, tm, max(cc, 1)));
            tx[u].load(tm + cc * cstep + ox);
            const int xc = th.xk + cc, xs = min(max(xc, beg), end - 1);
            in[u] = xc == xs && col + u < hi;
            const T *up = ub + xs * sp, *ps = pb + (xs - beg + 4) * ph;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                T mk[4], pk[4], um[4], uq[4];
                ld4(ps - (4 - k) * ph, mk);
                ld4(ps + (4 - k) * ph, pk);
                ld4(up - (4 - k) * sp, um);
                ld4(up + (4 - k) * sp, uq);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const T term = bk[k] * (pk[j] - mk[j]);
                    acc[u][j] = k == 0 ? term : acc[u][j] + term;
                    const T dterm = ak[k] * (uq[j] + um[j]);
                    d2[u][j] = k == 0 ? dterm : d2[u][j] + dterm;
                }
            }
            T uc[4];
            ld4(up, uc);
            ab[u] = pr[xs];
#pragma unroll
            for (int j = 0; j < 4; ++j) d2[u][j] = d2[u][j] + (T)RTM_AC0 * uc[j];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            T v[4], cf[4], xx[4];
            tv[u].wait(v);
            tc[u].wait(cf);
            tx[u].wait(xx);
            if (col + u == 0) {
#pragma unroll
                for (int j = 0; j < 4; ++j) cf[j] = cf0[j];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const T dp = acc[u][j] * h1;
                const T xn = (T)ab[u].y * xx[j] + (T)ab[u].x * (d2[u][j] * h3 + dp);
                const T vn = v[j] + mul_rn(cf[j] * h2, dp + xn);
                const bool ok = in[u] && j < zl;
                xx[j] = ok ? xn : xx[j];
                v[j] = ok ? vn : v[j];
            }
            if (u == 0 || col + u < hi) {
                TmQuad<T>::store(tm + (col + u) * cstep, v);
                TmQuad<T>::store(tm + (col + u) * cstep + ox, xx);
            }
        }
    }
}
// Top (side 2) and bottom (3) strips: all of the thread's columns, if its rows lie in them.
template <typename T>
__device__ __forceinline__ void res_strip_z(const ResJob<T> &J, const ResCta &c, const ResShape &h, const ResThread &th,
                                            int side, const T *su, const T *sm, const float *pz, uint32_t tm,
                                            const T (&cf0)[4])
{
    constexpr int QW = TmQuad<T>::WORDS, U = sizeof(T) == 4 ? 2 : 1;
    const Geom &g = J.g;
    const uint32_t cstep = (uint32_t)(h.nslot * QW), oz = (uint32_t)(h.zslot * QW);
    const int sp = h.SP, cw = h.CW, pt = side == 2 ? h.PT : h.PB;
    const T h1 = J.h1, h2 = J.h2, h3 = J.h3;
    const int zlo = side == 2 ? 4 : g.dimz - g.thd + 4, zhi = side == 2 ? g.thu - 4 : g.dimz - 4;
    const int zq = c.za + 4 * th.q, first = side == 2 ? h.qt0 : h.qb0, count = side == 2 ? h.ht : h.hb;
    const int zs = min(max(zq, first), first + count - 4);                            // the strip's nearest quad
    if (!__any_sync(0xffffffffu, zs == zq)) return;
    const T *ub = su + kResPad * sp + kResPad + (zs - c.za);
    const T *pb = sm + (side == 2 ? h.offt : h.offb) + (zs - first + 4);
    float aa[4], bz[4];
    ld4(pz + 2 * (zs - c.za + kResPad), aa);
    ld4(pz + 2 * (zs - c.za + kResPad) + 4, bz);
    bool up_j[4], frame[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        up_j[j] = zs == zq && zq + j >= zlo && zq + j < zhi;
        frame[j] = zq + j >= g.dimz - 4;
    }
#pragma unroll 1
    for (int col = 0; col < cw; col += U) {
        TmQuad<T> tv[U], tc[U], tz[U];
        T dp[U][4], d2[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int cc = min(col + u, cw - 1), xc = min(th.xk + cc, h.W - 1);       // (the spare column)
            tv[u].load(tm + cc * cstep);
            tc[u].load(res_coef_at<T>(h, tm, max(cc, 1)));
            tz[u].load(tm + cc * cstep + oz);
            const T *up = ub + xc * sp, *ps = pb + xc * pt;
            T q[12], zz[12], a0[4], a1[4], a2[4];
            ld4(ps - 4, a0);
            ld4(ps, a1);
            ld4(ps + 4, a2);
#pragma unroll
            for (int j = 0; j < 4; ++j) { q[j] = a0[j]; q[4 + j] = a1[j]; q[8 + j] = a2[j]; }
            ld4(up - 4, a0);
            ld4(up, a1);
            ld4(up + 4, a2);
#pragma unroll
            for (int j = 0; j < 4; ++j) { zz[j] = a0[j]; zz[4 + j] = a1[j]; zz[8 + j] = a2[j]; }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                dp[u][j] = dpsi_z<T>(q, j);
                d2[u][j] = d2z_q<T>(zz, j);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            T v[4], cf[4], xz[4];
            tv[u].wait(v);
            tc[u].wait(cf);
            tz[u].wait(xz);
            if (col + u == 0) {
#pragma unroll
                for (int j = 0; j < 4; ++j) cf[j] = cf0[j];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const T d1 = dp[u][j] * h1;
                const T xn = (T)bz[j] * xz[j] + (T)aa[j] * (d2[u][j] * h3 + d1);
                const T vn = v[j] + mul_rn(cf[j] * h2, d1 + xn);
                xz[j] = up_j[j] ? xn : xz[j];
                v[j] = frame[j] ? (T)0 : up_j[j] ? vn : v[j];                        // the grid's frame stays zero
            }
            if (u == 0 || col + u < cw) {
                TmQuad<T>::store(tm + (col + u) * cstep, v);
                TmQuad<T>::store(tm + (col + u) * cstep + oz, xz);
            }
        }
    }
}
// ... of all of a thread's columns.
template <typename T, int NC>
__device__ __forceinline__ void res_strips(const ResJob<T> &J, const ResCta &c, const ResShape &h, const ResThread &th,
                                           const ResFix &f, const T *su, const T *sm, const float *px, const float *pz,
                                           uint32_t tm, ResPriv<T, NC> &me)
{
    if constexpr (NC > 0) {
        const T h1 = J.h1, h2 = J.h2, h3 = J.h3;
        const int sp = h.SP, ph = h.PH, pt = h.ht ? h.PT : h.PB;
        const float2 *pr = reinterpret_cast<const float2 *>(px) + th.xk + 4;
        const T *up = su + (th.xk + kResPad) * sp + kResPad + 4 * th.q;
#pragma unroll
        for (int u = 0; u < NC; ++u)
            if (u == 0 || u < th.len)
                res_strip_quad<T>(f, u, h1, h2, h3, sp, ph, up + u * sp, sm + (f.s & 0xffffu) + u * ph, sm + (f.s >> 16) + u * pt, pr[u],
                                  pz + 2 * (4 * th.q + kResPad), me.cf[u], me.xx[u], me.xz[u], me.v[u]);
    } else {
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {                     // left, top; right, bottom
            if (k == 0 ? h.nl : h.nr) {
                res_strip_x<T>(J, c, h, th, k, su, sm, px, tm, me.cf[0]);
                tm_wait_st();
            }
            if (k == 0 ? h.ht : h.hb) {
                res_strip_z<T>(J, c, h, th, 2 + k, su, sm, pz, tm, me.cf[0]);
                tm_wait_st();
            }
        }
    }
}

// The new values into the tile, the current ones to where the previous field is kept.  keep(col):
// the column is this thread's to write.
template <typename T, int NC, typename K>
__device__ __forceinline__ void res_store(const ResShape &h, int f, T *own, uint32_t tm, const ResPriv<T, NC> &me, K keep)
{
    if constexpr (NC > 0) {
#pragma unroll
        for (int u = 0; u < NC; ++u)
            if (keep(u)) st4(own + u * h.SP, me.v[u]);
        return;
    } else {
        constexpr int QW = TmQuad<T>::WORDS, U = 2;
        const uint32_t cstep = (uint32_t)(h.nslot * QW);
        uint32_t ta = tm + (uint32_t)(f * QW);
        const int cw = h.CW, sp = h.SP;
        int col = 0;
#pragma unroll 1
        for (; col + U <= cw; col += U) {
            TmQuad<T> n[U];
            T q[U][4], v[U][4];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                n[u].load(ta + u * cstep);
                ld4(own + u * sp, q[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) n[u].wait(v[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                TmQuad<T>::store(ta + u * cstep, q[u]);
                if (keep(col + u)) st4(own + u * sp, v[u]);
            }
            ta += U * cstep;
            own += U * sp;
        }
        if (col < cw) {
            TmQuad<T> n;
            T q[4], v[4];
            n.load(ta);
            ld4(own, q);
            n.wait(v);
            TmQuad<T>::store(ta, q);
            if (keep(col)) st4(own, v);
        }
    }
}

// Ring quads of a block (the 4-cell ring around the reconstruction region): item i -> cell (x, zq)
// and its offset in a slot (ring_quad_offset); ring_items counts them.
struct RingBox {
    int x0, x1, z0, z1;         // block cells within the ring's bounding box
    int nt, nb;                 // top / bottom band quads (one a column)
    int zl, nl, xl0, xl1, xr0, xr1;   // side bands: rows and columns
    float inv;                  // 1 / nl
};
__device__ __forceinline__ RingBox ring_box(const Geom &g, const ResCta &c)
{
    RingBox b;
    b.x0 = max(c.xa, g.rx0 - 4); b.x1 = min(c.xb, g.rx1 + 4);
    const int nx = max(0, b.x1 - b.x0);
    b.z0 = max(c.za, g.rz0); b.z1 = min(c.zb, g.rz1);
    b.nt = c.za <= g.rz0 - 4 && g.rz0 - 4 < c.zb ? nx : 0;
    b.nb = c.za <= g.rz1 && g.rz1 < c.zb ? nx : 0;
    b.zl = b.z0; b.nl = max(0, b.z1 - b.z0) >> 2;
    b.xl0 = max(c.xa, g.rx0 - 4); b.xl1 = max(b.xl0, min(c.xb, g.rx0));
    b.xr0 = max(c.xa, g.rx1); b.xr1 = max(b.xr0, min(c.xb, g.rx1 + 4));
    b.inv = 1.0f / (float)max(1, b.nl);
    return b;
}
__device__ __forceinline__ int ring_items(const RingBox &b)
{
    return b.nt + b.nb + (b.xl1 - b.xl0 + b.xr1 - b.xr0) * b.nl;
}
__device__ __forceinline__ void ring_item(const Geom &g, const RingBox &b, int i, int &x, int &zq)
{
    if (i < b.nt) { x = b.x0 + i; zq = g.rz0 - 4; return; }
    i -= b.nt;
    if (i < b.nb) { x = b.x0 + i; zq = g.rz1; return; }
    i -= b.nb;
    const int k = fast_div(i, b.inv);
    zq = b.zl + 4 * (i - k * b.nl);
    x = k < b.xl1 - b.xl0 ? b.xl0 + k : b.xr0 + (k - (b.xl1 - b.xl0));
}

// A run of steps of one pass on one block.
// What bounds it: on small grids (NC = 1, 2) a chain of latencies -- the exchange through the second-level
// cache, psi, leapfrog and strips a quad a thread, two to four barriers; on large ones (NC = 0) the issue
// slots and shared-memory latency of 16 warps, at the 128 registers that 512 threads leave.  256 threads
// would leave 255 but half the warps; more than 512 fewer registers than the window alone needs.
// A forward and a backward step together, step kernels -> here: 96 x 64 17.2 -> 4.7 us, 400 x 200
// 17.7 -> 5.5, 901 x 301 (FP16 snapshots) 18.3 -> 8.2, 2000 x 600 (snapshots) 25.0 -> 13.5, 3400 x 700
// 38.9 -> 21.5, 400 x 200 in double 120 -> 39.
template <typename T, int NC>
__global__ void __launch_bounds__(kResThreads, 1)
    k_resident(const ResJob<T> *__restrict__ jobs, const ResCta *__restrict__ ctas, unsigned long long *xch, int pt0,
               int pt1, unsigned tag0, T *rec_out, T *pstore, unsigned *status)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *sm = reinterpret_cast<T *>(smem_raw);
    __shared__ ResJob<T> J;
    __shared__ ResCta c;
    __shared__ uint32_t s_tm;
    constexpr int QW = TmQuad<T>::WORDS;
    int tid = threadIdx.x;
    {
        const int *src = reinterpret_cast<const int *>(ctas + blockIdx.x);
        for (int i = tid; i < (int)(sizeof(ResCta) / 4); i += kResThreads) reinterpret_cast<int *>(&c)[i] = src[i];
        __syncthreads();
        const int *js = reinterpret_cast<const int *>(jobs + c.job);
        for (int i = tid; i < (int)(sizeof(ResJob<T>) / 4); i += kResThreads) reinterpret_cast<int *>(&J)[i] = js[i];
        if constexpr (NC == 0) {
            if (tid < 32) tm_alloc(&s_tm);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        } else {
            if (tid == 0) s_tm = 0;
            __syncthreads();
        }
    }
    const Geom &g = J.g;
    const bool back = J.back != 0, ring = J.storage == 1, two = back && ring;
    const int t0 = pt1 < 0 ? J.t0 : pt0, t1 = pt1 < 0 ? J.t1 : pt1;
    T *rec = J.rec_out ? J.rec_out : rec_out, *store = pstore ? pstore : J.store;
    const size_t P = (size_t)g.pitch;
    __shared__ ResShape h;
    if (tid == 0) h = res_shape(g, c.xa, c.xb, c.za, c.zb, two ? 2 : 1, (int)sizeof(T));
    __syncthreads();
    T *su = sm, *ss = sm + h.field;
    // damping profiles of the block: (a, b) by column xa - 4 .., and by quad za - 8 .. (4 a, 4 b)
    float *px = reinterpret_cast<float *>(sm + h.total), *pz = px + res_px_floats(h);
    T *rstage = reinterpret_cast<T *>(pz + res_pz_floats(h));      // the step's ring quads
    __shared__ ResPsi wpsi;
    if (tid == 0) res_psi_init(g, h, wpsi);
    const bool strip = h.nl || h.nr || h.ht || h.hb;
    ResThread th;
    {
        th.q = tid % h.HQ;
        const int k = tid / h.HQ;
        th.own = k < h.K;
        const int kk = min(k, h.K - 1);
        th.xk = (int)((long long)kk * h.W / h.K);
        th.len = (int)((long long)(kk + 1) * h.W / h.K) - th.xk;
    }
    int zq = c.za + 4 * th.q;
    const uint32_t tm = s_tm + ((uint32_t)((tid >> 5) & 3) << 21) + (uint32_t)(tid >> 7) * kResTmemWords;
    const uint32_t cstep = (uint32_t)(h.nslot * QW);
    // the source field's part in this block: its region, ring included
    const bool hasS = two && c.xa < g.rx1 + 4 && c.xb > g.rx0 - 4 && c.za < g.rz1 + 4 && c.zb > g.rz0 - 4;
    const int ua = g.nt & 1, ub = 1 - ua;             // u buffers holding u_nt, u_{nt-1}
    auto s_cur_of = [&](int t) { return ((max(t, 2) - 2) & 1) ? ua : ub; };

    // ---- fields, psi and xi on the chip: zero at the first step, else what the last run left
    const T none[4] = {(T)0, (T)0, (T)0, (T)0};
    // tiles that load_tile does not fill, and psi
    for (int i = (t0 > 0 ? (hasS || !two ? h.offl : h.field) : 0) + 4 * tid; i < h.total; i += 4 * kResThreads) st4(sm + i, none);
    for (int i = tid; i < h.W + 9; i += kResThreads) {
        const int x = c.xa - 4 + i;
        float a = 0.0f, b = 0.0f;
        if (x < g.thl) { a = J.prof[0][x]; b = J.prof[1][x]; }
        else if (x >= g.dimx - g.thr && x < g.dimx) { a = J.prof[2][x - (g.dimx - g.thr)]; b = J.prof[3][x - (g.dimx - g.thr)]; }
        px[2 * i] = a;
        px[2 * i + 1] = b;
    }
    for (int i = tid; i < h.H + 2 * kResPad; i += kResThreads) {
        const int z = c.za - kResPad + i;
        float a = 0.0f, b = 0.0f;
        if (z >= 0 && z < g.thu) { a = J.prof[4][z]; b = J.prof[5][z]; }
        else if (z >= g.zb0 && z < g.dimz) { a = J.prof[6][z - g.zb0]; b = J.prof[7][z - g.zb0]; }
        pz[8 * (i >> 2) + (i & 3)] = a;
        pz[8 * (i >> 2) + 4 + (i & 3)] = b;
    }
    __syncthreads();
    auto load_tile = [&](const T *f, T *tile) {
        // a warp takes whole rows of the tile: its lanes along z, up to 4 rows in flight
        const int nq = h.SP >> 2, rows = h.W + 2 * kResPad, lane = tid & 31;
        for (int k0 = tid >> 5; k0 < rows; k0 += 4 * (kResThreads / 32))
            for (int q0 = lane; q0 < nq; q0 += 32) {
                const int z = c.za - kResPad + 4 * q0;
                const bool zok = z >= 0 && z < g.pitch && 4 * q0 < h.H + 2 * kResPad;
                T q[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int k = k0 + r * (kResThreads / 32), x = c.xa - kResPad + k;
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[r][j] = (T)0;
                    if (zok && k < rows && x >= 0 && x < g.dimx) ld4(f + (size_t)x * P + z, q[r]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int k = k0 + r * (kResThreads / 32);
                    if (k < rows) st4(tile + k * h.SP + 4 * q0, q[r]);
                }
            }
    };
    if (t0 > 0) load_tile(back ? J.r[t0 & 1] : J.u[t0 & 1], su);
    if (hasS) load_tile(J.u[s_cur_of(t0)], ss);
    if (t0 > 0 && strip) {
        for (int side = 0; side < 2; ++side) {
            const int nc = side == 0 ? h.nl : h.nr;
            if (nc == 0) continue;
            const int c0 = side == 0 ? h.cl0 : h.cr0, base = side == 0 ? 0 : g.dimx - g.thr;
            T *ps = sm + (side == 0 ? h.offl : h.offr);
            for (int i = tid; i < (nc + 8) * h.HQ; i += kResThreads) {
                const int k = i / h.HQ, q = i - k * h.HQ, li = c0 - 4 + k - base;
                if (li < 0 || li >= (side == 0 ? g.thl : g.thr)) continue;
                T v4[4];
                ld4(J.psi[t0 & 1][side] + (size_t)li * P + c.za + 4 * q, v4);
                st4(ps + k * h.PH + 4 * q, v4);
            }
        }
        for (int side = 0; side < 2; ++side) {
            const int hh = side == 0 ? h.ht : h.hb;
            if (hh == 0) continue;
            const int q0 = side == 0 ? h.qt0 : h.qb0, nq = (hh + 8) >> 2, Pp = side == 0 ? h.PT : h.PB;
            const int st = side == 0 ? g.st : g.sb, sh = side == 0 ? 0 : g.zb0;
            T *ps = sm + (side == 0 ? h.offt : h.offb);
            for (int i = tid; i < h.W * nq; i += kResThreads) {
                const int k = i / nq, z = q0 - 4 + 4 * (i - k * nq);
                if (z - sh < 0 || z - sh + 4 > st) continue;
                T v4[4];
                ld4(J.psi[t0 & 1][2 + side] + (size_t)(c.xa + k) * st + (z - sh), v4);
                st4(ps + k * Pp + (z - (q0 - 4)), v4);
            }
        }
    }
    // offset of a quad's xi in its global strip array (x strips: which = 0, z strips: 1), or -1
    auto xi_at = [&](int which, int x, T *&arr) -> long long {
        if (which == 0) {
            if (x < g.thl - 4) { arr = J.xi[0]; return (long long)x * (long long)P + zq; }
            if (x >= g.dimx - g.thr + 4) { arr = J.xi[1]; return (long long)(x - (g.dimx - g.thr)) * (long long)P + zq; }
            return -1;
        }
        if (zq < g.thu - 4) { arr = J.xi[2]; return (long long)x * g.st + zq; }
        if (zq + 4 > g.dimz - g.thd + 4) { arr = J.xi[3]; return (long long)x * g.sb + (zq - g.zb0); }
        return -1;
    };
    ResPriv<T, NC> me;
    auto init_col = [&](int col, int u) {
        const int x = c.xa + min(th.xk + col, h.W - 1);
        T q[4] = {(T)0, (T)0, (T)0, (T)0};
        if (t0 > 0) ld4((back ? J.r[1 - (t0 & 1)] : J.u[1 - (t0 & 1)]) + (size_t)x * P + zq, q);
        T p2[4] = {(T)0, (T)0, (T)0, (T)0};
        if (two) ld4(J.u[1 - s_cur_of(t0)] + (size_t)x * P + zq, p2);
        if constexpr (NC == 0) {
            TmQuad<T>::store(tm + col * cstep, q);
            if (two) TmQuad<T>::store(tm + col * cstep + QW, p2);
            if (col > 0) {
                ldg4(J.coef + (size_t)x * P + zq, q);
                TmQuad<T>::store(res_coef_at<T>(h, tm, col), q);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) { me.prv[0][u][j] = q[j]; me.prv[1][u][j] = p2[j]; }
            ldg4(J.coef + (size_t)x * P + zq, me.cf[u]);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int slot = w == 0 ? h.xslot : h.zslot;
            T y[4] = {(T)0, (T)0, (T)0, (T)0}, *arr = nullptr;
            const long long o = slot >= 0 && t0 > 0 ? xi_at(w, x, arr) : -1;
            if (o >= 0) ld4(arr + o, y);
            if constexpr (NC == 0) {
                if (slot >= 0) TmQuad<T>::store(tm + col * cstep + slot * QW, y);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) (w == 0 ? me.xx : me.xz)[u][j] = y[j];
            }
        }
    };
    if constexpr (NC == 0) {
#pragma unroll 4
        for (int col = 0; col < h.CW; ++col) init_col(col, 0);   // (a column's loads take longer than all the rest)
        tm_wait_st();
    } else {
#pragma unroll
        for (int u = 0; u < NC; ++u) init_col(u, u);
    }

    // ---- receivers and shot: thread k patches column k of the block
    const bool recs = g.nrec > 0 && g.zrec >= c.za && g.zrec < c.zb && (back || rec != nullptr);
    const bool shot = g.xs >= c.xa && g.xs < c.xb && g.zs >= c.za && g.zs < c.zb;
    int my_rec = -1, my_cnt = 0;
    if (recs && tid < h.W) {
        if (back) my_rec = J.rec_last[c.xa + tid];
        else { my_rec = J.rec_first[c.xa + tid]; my_cnt = J.rec_cnt[c.xa + tid]; }
    }
    __shared__ RingBox rb;
    if (tid == 0) rb = ring_box(g, c);
    __syncthreads();
    const int nring = ring ? ring_items(rb) : 0;
    __shared__ ResHalo hin, hout;
    __shared__ ResBox box_in, box_out;
    if (tid < 16) {
        box_in.at[tid] = res_box(c.in_off, c.in_cap, tid, xch, kXWords<T>);
        box_out.at[tid] = res_box(c.out_off, c.out_cap, tid, xch, kXWords<T>);
    }
    if (tid < 4) {
        hin.d[tid] = c.din[tid];
        hout.d[tid] = c.dout[tid];
        hin.e[tid] = hout.e[tid] = c.sx[tid] ? (tid < 2 ? 4 : 1) : 0;
    }
    __syncthreads();
    if (tid == 0) {
        hin.n0 = halo_count(h, hin.d);
        hin.n = hin.n0 + (hasS ? halo_count(h, hin.e) : 0);
        hout.n0 = halo_count(h, hout.d);
        hout.n = hout.n0 + (hasS ? halo_count(h, hout.e) : 0);
    }
    const bool live = __any_sync(0xffffffffu, th.own);   // warps of spare threads only sit the leap out
    unsigned in[kResItems], out[kResItems];               // the thread's halo items
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kResItems; ++k) {
        in[k] = halo_item<true>(h, hin, tid + k * kResThreads);
        out[k] = halo_item<false>(h, hout, tid + k * kResThreads);
    }
    const int nin0 = hin.n0, nin = hin.n, nout0 = hout.n0, nout = hout.n;
    ResFix fix;
    if constexpr (NC > 0) res_fix_init(g, c, h, wpsi, th, tid, fix);
    int img_in = back ? (g.nt - 1 - t0) % g.slices : (g.slices - t0 % g.slices) % g.slices;   // steps to the next image / snapshot
    const bool int_any = c.xa < g.thl + g.nx && c.xb > g.thl && c.za < g.thu + g.nz && c.zb > g.thu;
    __syncthreads();

    bool dead = false;
    for (int t = t0; t < t1; ++t) {
        const unsigned tag = tag0 + (unsigned)(t - t0);     // of the fields this step reads
        // (what the compiler worked out of these ahead of the loop it kept in spilt words: 96 x 64
        // 2.69 -> 2.40 us a step, 400 x 200 2.92 -> 2.76, and NC = 0 the more so)
        opaque(tid);
        opaque(zq);
        opaque(th.q);
        opaque(th.xk);
        opaque(th.len);
#pragma unroll
        for (int k = 0; k < kResItems; ++k) { opaque(in[k]); opaque(out[k]); }
        if constexpr (NC > 0)
            for (unsigned *w : {&fix.x, &fix.z, &fix.xw, &fix.zw, &fix.s, &fix.bits}) opaque(*w);
        const bool recon = hasS && t >= 2;
        // inputs of the step that do not depend on the neighbours
        float seis = 0.0f;
        if (back && my_rec >= 0) seis = J.seis_t[(size_t)(g.nt - 1 - t) * g.nrec + my_rec];
        if (recon && nring > 0) {                           // the ring of u_{nt-t}, for the end of the step
            const T *slot = store + (size_t)(g.nt - t) * J.slot_elems;
            for (int i = tid; i < nring; i += kResThreads) {
                int x, z;
                ring_item(g, rb, i, x, z);
                const T *src = slot + ring_quad_offset(g, x, z);
#pragma unroll
                for (int k = 0; k < (int)sizeof(T) / 4; ++k) cp_async16(rstage + 4 * i + k * (16 / (int)sizeof(T)), src + k * (16 / (int)sizeof(T)));
            }
            cp_async_commit();
        }
        if constexpr (NC == 0) ldg4(J.coef + (size_t)(c.xa + th.xk) * P + zq, me.cf[0]);
        bool ok = true;
        if (t > t0) ok = res_recv<T>(box_in, tid, in, t >= 3 ? nin : nin0, tag, sm, status);
        if constexpr (NC == 0) tm_wait_st();
        if (__syncthreads_or(!ok)) {
            if (tid == 0) atomicOr(status, ST_EXCHANGE_TIMEOUT);
            dead = true;
            break;
        }
        if constexpr (NC > 0) {
            if (strip) res_psi_fix<T>(fix, h, J.h1, su, sm, px, pz);
        } else {
            if (strip) res_psi<T>(J, c, h, wpsi, tid, su, sm, px, pz);
        }
        T *own = su + (th.xk + kResPad) * h.SP + kResPad + 4 * th.q;
        auto half = [&](int f) {                              // leapfrog of field f into its tile
            T *tile = sm + f * h.field;
            if (live) {
                res_leap<T, NC>(J, c, h, th, f, tile, tm, me);
                if constexpr (NC == 0) tm_wait_st();
            }
            if (f == 0 && strip) {
                __syncthreads();                             // psi
                if (live) res_strips<T, NC>(J, c, h, th, fix, su, sm, px, pz, tm, me);
            }
            __syncthreads();
            if (live) {
                // of the source field, the region's cells only
                const bool zin = th.own && (f == 0 || (zq >= g.rz0 && zq < g.rz1));
                const int xlo = f == 0 ? 0 : g.rx0 - c.xa - th.xk, xhi = f == 0 ? th.len : min(th.len, g.rx1 - c.xa - th.xk);
                res_store<T, NC>(h, f, own + f * h.field, tm, me, [&](int col) { return zin && col >= xlo && col < xhi; });
            }
        };
        if constexpr (NC > 0) {
            half(0);
            if (recon) half(1);
        } else {                                             // one copy of the long column loop
#pragma unroll 1
            for (int f = 0; f < (recon ? 2 : 1); ++f) half(f);
        }
        if (recon && nring > 0) {                           // each thread takes what it copied
            cp_async_wait_all();
            for (int i = tid; i < nring; i += kResThreads) {
                int x, z;
                ring_item(g, rb, i, x, z);
                T q[4];
                ld4(rstage + 4 * i, q);
                st4(ss + (x - c.xa + kResPad) * h.SP + kResPad + (z - c.za), q);
            }
        }
        __syncthreads();
        if (recs || shot) {              // the source, then the receivers of a column, by its thread
            if (shot && tid == g.xs - c.xa) {
                const int shot_at = (tid + kResPad) * h.SP + kResPad + (g.zs - c.za);
                const T shot_cf = J.coef[(size_t)g.xs * P + g.zs];
                if (!back && t < g.nwav) su[shot_at] = add_source<T>(J.wav, t, su[shot_at], shot_cf);
                if (recon && g.nt + 1 - t < g.nwav) ss[shot_at] = add_source<T>(J.wav, g.nt + 1 - t, ss[shot_at], shot_cf);
            }
            if (my_rec >= 0) {
                const int rec_at = (tid + kResPad) * h.SP + kResPad + (g.zrec - c.za);
                if (back) su[rec_at] = (T)seis;
                else
                    for (int q = 0; q < my_cnt; ++q) rec[(size_t)(my_rec + q) * g.nt + t] = su[rec_at];
            }
            __syncthreads();
        }
        if (t + 1 < t1) res_send<T, (NC == 0 && sizeof(T) == 4 ? 2 : 1)>(box_out, tid, out, recon ? nout : nout0, tag + 1, sm);
        // ---- storage of the forward field, image of the backward ones
        if (!back && ring && t + 1 < g.nt) {            // slot k holds the ring of u_k
            T *slot = store + (size_t)(t + 1) * J.slot_elems;
            for (int i = tid; i < nring; i += kResThreads) {
                int x, z;
                ring_item(g, rb, i, x, z);
                T q[4];
                ld4(su + (x - c.xa + kResPad) * h.SP + kResPad + (z - c.za), q);
                st4(slot + ring_quad_offset(g, x, z), q);
            }
        }
        const int tau = back ? g.nt - 1 - t : t;
        const bool imaged = img_in == 0;
        img_in = imaged ? g.slices - 1 : img_in - 1;
        if (imaged && int_any && th.own && (back || !ring)) {
            T *slot = store + (size_t)(tau / g.slices) * J.slot_elems;
            const bool zfull = zq >= g.thu && zq + 4 <= g.thu + g.nz;
            const bool zany = zq < g.thu + g.nz && zq + 4 > g.thu;
            for (int col = 0; col < th.len && zany; ++col) {
                const int x = c.xa + th.xk + col;
                if (x < g.thl || x >= g.thl + g.nx) continue;
                const size_t o = (size_t)(x - g.thl) * P + zq;
                T q[4];
                ld4(own + col * h.SP, q);
                if (!back) {
                    if (zfull) {
                        st4(slot + o, q);
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (in_interior(g, x, zq + j)) slot[o + j] = q[j];
                    continue;
                }
                T s[4];
                if (!ring) ld4(slot + o, s);
                else if (recon) ld4(ss + (own - su) + col * h.SP, s);
                else ld4(J.u[t == 0 ? ua : ub] + (size_t)x * P + zq, s);
                if (zfull) image_quad<T>(J.img + o, J.slf + o, s, q);
                else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (in_interior(g, x, zq + j)) {
                            J.img[o + j] += (double)s[j] * (double)q[j];
                            J.slf[o + j] += (double)s[j] * (double)s[j];
                        }
                }
            }
        }
    }

    // ---- the fields back to their buffers (and, between the runs of a pass, psi and xi).  Neighbours load
    // some of these cells at their start.  After two steps or more they have: an exchange lies between.  A
    // run of one step has none: it leaves in u and r what a neighbour may still read as it is (the same
    // values again, or the other buffer's), and its psi goes to the buffer it did not come from.
    if (!dead) {
        if constexpr (NC == 0) tm_wait_st();
        const T *own = su + (th.xk + kResPad) * h.SP + kResPad + 4 * th.q;
        T *fc = back ? J.r[t1 & 1] : J.u[t1 & 1], *fp = back ? J.r[1 - (t1 & 1)] : J.u[1 - (t1 & 1)];
        T *sc = J.u[s_cur_of(t1)], *sp = J.u[1 - s_cur_of(t1)];
        const bool sdone = hasS && t1 > 2;
        auto dump_col = [&](int col, int u) {
            const int x = c.xa + th.xk + col;
            const bool mine = th.own && col < th.len;
            TmQuad<T> tq;
            T q[4];
            auto priv = [&](int slot, const T (&reg)[4]) {
                if constexpr (NC == 0) {
                    tq.load(tm + col * cstep + slot * QW);
                    tq.wait(q);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[j] = reg[j];
                }
            };
            if constexpr (NC == 0) priv(0, me.cf[0]);
            else priv(0, me.prv[0][u]);
            if (mine) {
                st4(fp + (size_t)x * P + zq, q);
                ld4(own + col * h.SP, q);
                st4(fc + (size_t)x * P + zq, q);
            }
            if (two) {
                if constexpr (NC == 0) priv(1, me.cf[0]);
                else priv(1, me.prv[1][u]);
                if (mine && sdone && x >= g.rx0 && x < g.rx1 && zq >= g.rz0 && zq < g.rz1) {
                    st4(sp + (size_t)x * P + zq, q);
                    ld4(ss + (own - su) + col * h.SP, q);
                    st4(sc + (size_t)x * P + zq, q);
                }
            }
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int slot = w == 0 ? h.xslot : h.zslot;
                if (slot < 0) continue;
                if constexpr (NC == 0) priv(slot, me.cf[0]);
                else priv(slot, (w == 0 ? me.xx : me.xz)[u]);
                T *arr = nullptr;
                const long long o = mine && t1 < g.nt ? xi_at(w, x, arr) : -1;
                if (o >= 0) st4(arr + o, q);
            }
        };
        if constexpr (NC == 0) {
#pragma unroll 1
            for (int col = 0; col < h.CW; ++col) dump_col(col, 0);
        } else {
#pragma unroll
            for (int u = 0; u < NC; ++u) dump_col(u, u);
        }
        if (sdone)
            for (int i = tid; i < nring; i += kResThreads) {
                int x, z;
                ring_item(g, rb, i, x, z);
                T q[4];
                ld4(ss + (x - c.xa + kResPad) * h.SP + kResPad + (z - c.za), q);
                st4(sc + (size_t)x * P + z, q);
                if (t1 > 3) {                            // the step before's ring, from its slot
                    ld4(store + (size_t)(g.nt - t1 + 2) * J.slot_elems + ring_quad_offset(g, x, z), q);
                    st4(sp + (size_t)x * P + z, q);
                }
            }
        if (t1 < g.nt && strip) {
            for (int side = 0; side < 2; ++side) {
                const int nc = side == 0 ? h.nl : h.nr;
                const int c0 = side == 0 ? h.cl0 : h.cr0, base = side == 0 ? 0 : g.dimx - g.thr;
                const T *ps = sm + (side == 0 ? h.offl : h.offr);
                for (int i = tid; i < nc * h.HQ; i += kResThreads) {
                    const int k = i / h.HQ, q = i - k * h.HQ;
                    T v4[4];
                    ld4(ps + (k + 4) * h.PH + 4 * q, v4);
                    st4(J.psi[t1 & 1][side] + (size_t)(c0 + k - base) * P + c.za + 4 * q, v4);
                }
            }
            for (int side = 0; side < 2; ++side) {
                const int hh = side == 0 ? h.ht : h.hb;
                if (hh == 0) continue;
                const int q0 = side == 0 ? h.qt0 : h.qb0, nq = hh >> 2, Pp = side == 0 ? h.PT : h.PB;
                const int st = side == 0 ? g.st : g.sb, sh = side == 0 ? 0 : g.zb0;
                const T *ps = sm + (side == 0 ? h.offt : h.offb);
                for (int i = tid; i < h.W * nq; i += kResThreads) {
                    const int k = i / nq, z = q0 + 4 * (i - k * nq);
                    T v4[4];
                    ld4(ps + k * Pp + 4 + (z - q0), v4);
                    st4(J.psi[t1 & 1][2 + side] + (size_t)(c.xa + k) * st + (z - sh), v4);
                }
            }
        }
    }
    cp_async_wait_all();                                    // a block that gave up: the ring quads of its step
    if constexpr (NC == 0) {
        __syncthreads();
        if (tid < 32) tm_free(s_tm);
    }
}

// ---- launch -----------------------------------------------------------------------------------
template <typename T, int NC>
static cudaError_t launch_resident_c(const ResLaunch<T> &L, cudaStream_t s)
{
    static cudaError_t conf = cudaFuncSetAttribute(k_resident<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
    if (conf != cudaSuccess) return conf;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.nctas);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_resident<T, NC>, L.jobs, L.ctas, L.xch, L.t0, L.t1, L.tag0, L.rec_out, L.store, L.status);
}
template <typename T>
cudaError_t launch_resident(const ResLaunch<T> &L, cudaStream_t s)
{
    // registers for a thread's private values while they fit: one quad in double, two in float
    if (L.cw <= 1) return launch_resident_c<T, 1>(L, s);
    if (L.cw <= 2 && sizeof(T) == 4) return launch_resident_c<T, (sizeof(T) == 4 ? 2 : 1)>(L, s);
    return launch_resident_c<T, 0>(L, s);
}
template cudaError_t launch_resident<float>(const ResLaunch<float> &, cudaStream_t);
template cudaError_t launch_resident<double>(const ResLaunch<double> &, cudaStream_t);

// ---- 16-bit storage of a resident pass ---------------------------------------------------------
// A resident pass reads and writes full-precision slots; with BF16 / FP16 storage they are a staging
// area of a few slots that these kernels pack into the store after a run of steps, or unpack before
// one.  Values and scales are those of the per-step kernels: a max-abs scale for each group of a slot's
// cells -- a tile of the step kernels (kRingTile, kSnapTile) or a strip block of the batched ones
// (kRingStrip).

// Tile of tile_coords' order that holds cell (x, z).
__device__ __forceinline__ int tile_at(const Geom &g, int x, int z)
{
    const int xt = x / g.tx;
    int zt = 0;
    if (z >= g.ztop) zt = g.zbot > 0 && z >= g.zbot ? g.tiles_z - 1 : 1 + (z - g.ztop) / TZ;
    const int nzb = g.tiles_z > 1 ? 2 : 1;
    if (zt == 0) return xt * nzb;
    if (zt == g.tiles_z - 1) return xt * nzb + 1;
    const int nzi = g.tiles_z - nzb, nxb = g.nxl + (g.tiles_x - g.xr0);
    int t = g.tiles_x * nzb;
    if (xt < g.nxl || xt >= g.xr0) return t + (xt < g.nxl ? xt : g.nxl + xt - g.xr0) * nzi + zt - 1;
    return t + nxb * nzi + (xt - g.nxl) * nzi + zt - 1;
}

// One group of one slot: blockIdx.x, blockIdx.y.
template <int KIND>
__global__ void __launch_bounds__(256) k_pack16(const __grid_constant__ Pack16 a)
{
    const Geom &g = a.g;
    __shared__ float red[8];
    const float *in = a.stage + (size_t)blockIdx.y * a.slot_elems;
    unsigned char *out = static_cast<unsigned char *>(a.store) + (size_t)blockIdx.y * a.slot_elems * 2;
    int x0 = 0, z0 = 0, zend = 0, n = 1;
    const CorrShape cs = corr_shape(g);
    if (KIND != kRingStrip) {
        int xt, zt;
        tile_coords(g, blockIdx.x, xt, zt);
        x0 = xt * g.tx; z0 = ztile_origin(g, zt); zend = min(min(ztile_end(g, zt), z0 + TZ), g.dimz);
        const int x1 = x0 + g.tx;
        if (KIND == kRingTile) {
            const bool inside = x0 >= g.rx0 && x1 <= g.rx1 && z0 >= g.rz0 && zend <= g.rz1;
            if (inside || x0 >= g.rx1 + 4 || x1 <= g.rx0 - 4 || z0 >= g.rz1 + 4 || zend <= g.rz0 - 4) return;
        } else if (x0 >= g.thl + g.nx || x1 <= g.thl || z0 >= g.thu + g.nz || zend <= g.thu) return;
        n = (g.tx * (TZ / 4) + 255) / 256;
    }
    // offset of the thread's k-th quad in the slot (and its stored cells), or -1
    auto quad = [&](int k, int &x, int &zq) -> long long {
        if (KIND == kRingStrip) {
            int i = blockIdx.x * kStripBlock + threadIdx.x;
            if (i >= cs.nA + cs.nB) return -1;
            if (i < cs.nA) {
                const int c = i / cs.nql;
                x = c < g.thl - 8 ? 4 + c : g.dimx - g.thr + 4 + (c - (g.thl - 8));
                zq = 4 + 4 * (i % cs.nql);
            } else {
                i -= cs.nA;
                const int nq = cs.ntq + cs.nbq, q = i % nq;
                x = i / nq;
                zq = q < cs.ntq ? 4 + 4 * q : cs.q0 + 4 * (q - cs.ntq);
                if ((x >= 4 && x < g.thl - 4) || (x >= g.dimx - g.thr + 4 && x < g.dimx - 4)) return -1;
            }
            return ring_quad_offset(g, x, zq);
        }
        const int i = k * 256 + threadIdx.x;
        x = x0 + i / (TZ / 4);
        zq = z0 + 4 * (i % (TZ / 4));
        if (i >= g.tx * (TZ / 4) || x >= g.dimx || zq >= zend) return -1;
        if (KIND == kRingTile) return ring_quad_offset(g, x, zq);
        if (x < g.thl || x >= g.thl + g.nx) return -1;
        return (long long)(x - g.thl) * g.pitch + zq;
    };
    float mx = 0.0f;
    for (int k = 0; k < n; ++k) {
        int x = 0, zq = 0;
        const long long o = quad(k, x, zq);
        if (o < 0) continue;
        for (int j = 0; j < 4; ++j)
            if (KIND != kSnapTile || in_interior(g, x, zq + j)) mx = fmaxf(mx, fabsf(in[o + j]));
    }
    mx = block_max<8>(mx, red);
    const float scale = store_scale_of(mx, a.prec), inv = 1.0f / scale;
    if (threadIdx.x == 0) a.scales[(size_t)blockIdx.y * a.scales_per_slot + blockIdx.x] = scale;
    for (int k = 0; k < n; ++k) {
        int x = 0, zq = 0;
        const long long o = quad(k, x, zq);
        if (o < 0) continue;
        for (int j = 0; j < 4; ++j)
            if (KIND != kSnapTile || in_interior(g, x, zq + j)) store_put<float>(out, a.prec, (size_t)(o + j), in[o + j], inv);
    }
}

// Quads of one slot (blockIdx.y).
template <int KIND>
__global__ void __launch_bounds__(256) k_unpack16(const __grid_constant__ Pack16 a)
{
    const Geom &g = a.g;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if ((size_t)4 * i >= a.slot_elems) return;
    float *out = a.stage + (size_t)blockIdx.y * a.slot_elems + 4 * (size_t)i;
    const unsigned char *in = static_cast<const unsigned char *>(a.store) + (size_t)blockIdx.y * a.slot_elems * 2;
    int x, z, group;
    if (KIND == kSnapTile) {
        const int pq = g.pitch / 4;
        x = g.thl + i / pq;
        z = 4 * (i % pq);
        if (z + 4 <= g.thu || z >= g.thu + g.nz) return;
        group = tile_at(g, x, z);
    } else {
        ring_cell(g, 4 * i, x, z);
        group = KIND == kRingTile ? tile_at(g, x, z) : strip_item(g, corr_shape(g), x, z & ~3) / kStripBlock;
    }
    const float scale = a.scales[(size_t)blockIdx.y * a.scales_per_slot + group];
    float q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = store_get<float>(in, a.prec, 4 * (size_t)i + j, scale);
    st4(out, q);
}

cudaError_t launch_pack16(int kind, bool pack, const Pack16 &all, int slots, cudaStream_t s)
{
    constexpr int kMost = 65535;                         // blocks of a grid's second dimension
    const int groups = kind == kRingStrip ? strip_blocks_host(all.g) : all.g.tiles;
    for (int k = 0; k < slots; k += kMost) {
        Pack16 a = all;
        a.stage += (size_t)k * a.slot_elems;
        a.store = static_cast<unsigned char *>(a.store) + (size_t)k * a.slot_elems * 2;
        a.scales += (size_t)k * a.scales_per_slot;
        const dim3 grid(pack ? groups : (int)((a.slot_elems / 4 + 255) / 256), std::min(slots - k, kMost));
        if (pack) {
            if (kind == kRingTile) k_pack16<kRingTile><<<grid, 256, 0, s>>>(a);
            else if (kind == kSnapTile) k_pack16<kSnapTile><<<grid, 256, 0, s>>>(a);
            else k_pack16<kRingStrip><<<grid, 256, 0, s>>>(a);
        } else {
            if (kind == kRingTile) k_unpack16<kRingTile><<<grid, 256, 0, s>>>(a);
            else if (kind == kSnapTile) k_unpack16<kSnapTile><<<grid, 256, 0, s>>>(a);
            else k_unpack16<kRingStrip><<<grid, 256, 0, s>>>(a);
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace rtm
