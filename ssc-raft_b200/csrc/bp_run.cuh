// bp_run.cuh -- the backprojector whose threads' pixels are runs along the image
// axis on which the detector coordinate moves slowest: 16, 8 or 4 slices per thread
// on slice-interleaved rows, or one on plain rows (included by backproject.cu).
//
// What bounds it, and why runs.  A gather of one 4-byte sample per
// (voxel, angle) is limited by the 128 B/clk shared-memory pipe to 32 updates
// per SM and clock; the kernel that reads one 16-byte element (four slices) per
// (pixel, angle) ran at 87-90 % of that.  But at every angle one image axis has
// |dt/dx| <= 1/sqrt(2) bins per pixel, so four neighbouring pixels along it fall
// into two (|dt/dx| <= 1/3), three or at most four bins: the thread loads those
// bins once and adds the right one to each pixel.  That is 2.64 instead of 4
// shared-memory bytes per update averaged over [0, pi); neighbouring pixels of
// a run start in one of only two bins (slope classes below), so the choice is
// one compare and one select per two slices.  16 x 2048^2 x 900, nearest: 87 % of
// the pipe's wavefronts (80 % shared memory, most of the rest the spills of the
// sixteen-slice form), 2.47 instructions per clock.  Position and rounding
// are computed two pixels per instruction.  The bin of every pixel is still
// computed by itself with the single-pixel kernel's expressions, and the order
// of the additions over angles is the same: the images are bit for bit those of
// bp_kernel.
// The lanes of a warp lie along the other axis (one pixel apart, so a load's
// eight-lane phases read eight neighbouring 16-byte elements without bank
// conflicts): when the run axis changes, which for angles in order happens
// twice over [0, pi), the accumulators change hands through shared memory.
#pragma once
#include "ring.hpp"

namespace raft {

__device__ __forceinline__ u64 add2_rz(u64 a, u64 b)
{
    u64 r;
    asm("add.rz.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Orientation of the runs: 0 along x, 1 along y; +2: pixels in descending order,
// so that the bins of a run never descend.
// Slope classes: the bin of pixel p of a run, relative to pixel 0's, is low or
// low + 1 with low = floor(p * slope), slope <= 1/sqrt(2):
//   RUN_A  slope <= 1/3           low = 0 0 0
//   RUN_B  1/3 .. 1/2             low = 0 0 1
//   RUN_C  1/2 .. 2/3             low = 0 1 1
//   RUN_D  >= 2/3                 low = 0 1 2
//   RUN_G  within eps of a class boundary (the computed positions carry
//          rounding errors), or where bins may be negative (truncation towards
//          zero): every pixel reads its own bin
enum { RUN_A = 0, RUN_B = 1, RUN_C = 2, RUN_D = 3, RUN_G = 4 };

__device__ __forceinline__ int run_mode(float slope_x, float slope_y, float eps, bool general)
{
    const bool along_y = fabsf(slope_x) > fabsf(slope_y);
    const float s = along_y ? slope_y : slope_x, m = fabsf(s);
    int cls = RUN_G;
    if (3.f * m <= 1.f - eps) cls = RUN_A;
    else if (3.f * m >= 1.f + eps && 2.f * m <= 1.f - eps) cls = RUN_B;
    else if (2.f * m >= 1.f + eps && 3.f * m <= 2.f - eps) cls = RUN_C;
    else if (3.f * m >= 2.f + eps) cls = RUN_D;
    if (general) cls = RUN_G;
    return (along_y ? 1 : 0) | (s < 0.f ? 2 : 0) | (cls << 2);
}

// What a stage holds per angle.  Nearest sample: position along x c + y s, c and
// s twice (both lanes of the two-lane instructions); linear interpolation:
// b x + c y + a.  base: bin (as the integer run_positions makes) of window element 0.
struct __align__(16) RunParam {
    float c0, c1, s0, s1;
    float a;
    int base, mode, pad;
};

// One bin of four slices: the samples; for linear interpolation 2 mid and dif
// (2 mid + 2 f dif is twice the sample: scaling by two changes no rounding, and
// the sum is halved at the end), or mid and dif of bf16 pairs.
template <int STORE> struct RunBin {
    u64 m01, m23, d01, d23;
};
template <> struct RunBin<STORE_F32> {
    u64 m01, m23;
};

// A pixel's sums: of G groups of four slices, or of one slice (G = 0).
template <int G> struct RunAcc {
    static constexpr int slices = 4 * G;
    u64 v[G][2];
    __device__ __forceinline__ float get(int q) const
    {
        float lo, hi;
        unpack2(v[q >> 2][(q >> 1) & 1], lo, hi);
        return (q & 1) ? hi : lo;
    }
    __device__ __forceinline__ void set(int q, float x)
    {
        float lo, hi;
        unpack2(v[q >> 2][(q >> 1) & 1], lo, hi);
        v[q >> 2][(q >> 1) & 1] = (q & 1) ? pack2(lo, x) : pack2(x, hi);
    }
};
template <> struct RunAcc<0> {
    static constexpr int slices = 1;
    float v;
    __device__ __forceinline__ float get(int) const { return v; }
    __device__ __forceinline__ void set(int, float x) { v = x; }
};

// the window elements from q on as bins b[0..NB-1] of group g
template <int STORE, int NB, int G>
__device__ __forceinline__ void load_bins(const unsigned char *w, int g, RunBin<STORE> (&b)[NB][G])
{
    if constexpr (STORE == STORE_F32) {
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(w);
#pragma unroll
        for (int j = 0; j < NB; j++) {
            const ulonglong2 v = q[j];
            b[j][g].m01 = v.x;
            b[j][g].m23 = v.y;
        }
    } else if constexpr (STORE == STORE_PAIR_F32) {
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(w);
        const u64 neg = pack2(-1.f, -1.f);
        ulonglong2 lo = q[0];
#pragma unroll
        for (int j = 0; j < NB; j++) {
            const ulonglong2 hi = q[j + 1];
            b[j][g].m01 = add2(lo.x, hi.x);
            b[j][g].m23 = add2(lo.y, hi.y);
            b[j][g].d01 = fma2(lo.x, neg, hi.x);
            b[j][g].d23 = fma2(lo.y, neg, hi.y);
            lo = hi;
        }
    } else {
        const uint4 *q = reinterpret_cast<const uint4 *>(w);
#pragma unroll
        for (int j = 0; j < NB; j++) {
            const uint4 u = q[j];
            b[j][g].m01 = pack2(__uint_as_float(u.x << 16), __uint_as_float(u.y << 16));
            b[j][g].m23 = pack2(__uint_as_float(u.z << 16), __uint_as_float(u.w << 16));
            b[j][g].d01 = pack2(__uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y & 0xffff0000u));
            b[j][g].d23 = pack2(__uint_as_float(u.z & 0xffff0000u), __uint_as_float(u.w & 0xffff0000u));
        }
    }
}

// acc[g] += the sample of bin a[g] (weight f twice in ff)
template <int STORE, int G>
__device__ __forceinline__ void take(u64 (&acc)[G][2], const RunBin<STORE> (&a)[G], u64 ff)
{
#pragma unroll
    for (int g = 0; g < G; g++) {
        if constexpr (STORE == STORE_F32) {
            acc[g][0] = add2(acc[g][0], a[g].m01);
            acc[g][1] = add2(acc[g][1], a[g].m23);
        } else {
            acc[g][0] = add2(acc[g][0], fma2(ff, a[g].d01, a[g].m01));
            acc[g][1] = add2(acc[g][1], fma2(ff, a[g].d23, a[g].m23));
        }
    }
}

// Bins t[] (as integers with a common offset) and, for linear interpolation,
// weights ff[] (in both lanes) of the four pixels of a run at one angle; rc: their
// coordinates along the run axis, fc: the other coordinate twice; Y: runs along y;
// GEN: bins may be negative.
template <int GEOM, int STORE, bool UNIT, bool Y, bool GEN>
__device__ __forceinline__ void run_positions(const ulonglong2 cs, float a, u64 rc0, u64 rc1, u64 fc, u64 ntmin,
                                              u64 rdt2, int (&t)[4], u64 (&ff)[4])
{
    if constexpr (GEOM == GEOM_FBP_LIN) {
        const float MAGIC = 12582912.0f;   // 1.5 * 2^23: adding it rounds to an integer
        const u64 magic = pack2(MAGIC, MAGIC), nmagic = pack2(-MAGIC, -MAGIC), neg = pack2(-1.f, -1.f);
        const u64 aa = pack2(a, a);
        const u64 row = Y ? 0ull : fma2(fc, cs.y, aa);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const u64 rc = i ? rc1 : rc0;
            u64 v;
            if (Y) v = fma2(fc, cs.x, fma2(rc, cs.y, aa));
            else v = fma2(rc, cs.x, row);
            const u64 m = add2(v, magic);
            u64 g = fma2(add2(m, nmagic), neg, v);   // v - round(v)
            if (STORE == STORE_PAIR_F32) g = add2(g, g);
            float m0, m1, f0, f1;
            unpack2(m, m0, m1);
            unpack2(g, f0, f1);
            ff[2 * i] = pack2(f0, f0);
            ff[2 * i + 1] = pack2(f1, f1);
            t[2 * i] = __float_as_int(m0);
            t[2 * i + 1] = __float_as_int(m1);
        }
    } else {
        const u64 ys = Y ? 0ull : mul2(fc, cs.y);
        const u64 big = pack2(8388608.f, 8388608.f);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const u64 rc = i ? rc1 : rc0;
            u64 u;
            if (Y) u = fma2(fc, cs.x, mul2(rc, cs.y));
            else u = fma2(rc, cs.x, ys);
            u = add2(u, ntmin);
            if (!UNIT) u = mul2(u, rdt2);
            float u0, u1;
            // u >= 0: adding 2^23 rounded towards zero truncates u, as the conversion does
            if (!GEN) u = add2_rz(u, big);
            unpack2(u, u0, u1);
            t[2 * i] = GEN ? (int)u0 : __float_as_int(u0);
            t[2 * i + 1] = GEN ? (int)u1 : __float_as_int(u1);
            ff[2 * i] = ff[2 * i + 1] = 0ull;
        }
    }
}

// acc[g] += the sample of bin a[g] where t == ka, of bin b[g] elsewhere.  A select,
// not a multiply by 0 or 1, so that a neighbouring bin's infinity or NaN stays
// there; predicated two-lane adds measured slower (each brings two predicated moves).
template <int STORE, int G>
__device__ __forceinline__ void take_either(u64 (&acc)[G][2], const RunBin<STORE> (&a)[G], const RunBin<STORE> (&b)[G],
                                            u64 ff, int t, int ka)
{
    u64 xa[G], xb[G], ya[G], yb[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
        if constexpr (STORE == STORE_F32) {
            xa[g] = a[g].m01, xb[g] = b[g].m01, ya[g] = a[g].m23, yb[g] = b[g].m23;
        } else {
            xa[g] = fma2(ff, a[g].d01, a[g].m01), xb[g] = fma2(ff, b[g].d01, b[g].m01);
            ya[g] = fma2(ff, a[g].d23, a[g].m23), yb[g] = fma2(ff, b[g].d23, b[g].m23);
        }
    }
#pragma unroll
    for (int g = 0; g + 1 < G; g += 2) {
        u64 v0, v1, v2, v3;
        asm("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %12, %13;\n\tselp.b64 %0, %4, %5, p;\n\t"
            "selp.b64 %1, %6, %7, p;\n\tselp.b64 %2, %8, %9, p;\n\tselp.b64 %3, %10, %11, p;\n\t}"
            : "=l"(v0), "=l"(v1), "=l"(v2), "=l"(v3)
            : "l"(xa[g]), "l"(xb[g]), "l"(ya[g]), "l"(yb[g]), "l"(xa[g + 1]), "l"(xb[g + 1]), "l"(ya[g + 1]),
              "l"(yb[g + 1]), "r"(t), "r"(ka));
        acc[g][0] = add2(acc[g][0], v0);
        acc[g][1] = add2(acc[g][1], v1);
        acc[g + 1][0] = add2(acc[g + 1][0], v2);
        acc[g + 1][1] = add2(acc[g + 1][1], v3);
    }
    if constexpr (G % 2 == 1) {
        u64 v0, v1;
        asm("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %6, %7;\n\tselp.b64 %0, %2, %3, p;\n\t"
            "selp.b64 %1, %4, %5, p;\n\t}"
            : "=l"(v0), "=l"(v1)
            : "l"(xa[G - 1]), "l"(xb[G - 1]), "l"(ya[G - 1]), "l"(yb[G - 1]), "r"(t), "r"(ka));
        acc[G - 1][0] = add2(acc[G - 1][0], v0);
        acc[G - 1][1] = add2(acc[G - 1][1], v1);
    }
}

// Adds the angles al .. end - 1 (all of one mode) to the runs.  Each mode has a
// loop of its own so that the accumulators keep their registers.
template <int GEOM, int STORE, bool UNIT, int CLS, bool Y, int G>
__device__ __forceinline__ void run_angles(RunAcc<G> (&acc)[4], const RunParam *prm, const unsigned char *win,
                                           int wbytes, int al, int end, const u64 (&rc)[2], u64 fc, u64 ntmin,
                                           u64 rdt2, int W)
{
    const unsigned char *w = win + al * (G * wbytes);
    const unsigned kmax = W - 5;   // the window planning keeps every bin below it
    const RunParam *ap = prm + al, *ae = prm + end;
    ulonglong2 cs_next = *reinterpret_cast<const ulonglong2 *>(ap);
    float2 ab_next = *reinterpret_cast<const float2 *>(&ap->a);
#pragma unroll 1
    for (; ap != ae; w += G * wbytes) {
        const ulonglong2 cs = cs_next;
        const float2 ab = ab_next;
        const int base = __float_as_int(ab.y);
        ap++;   // the next angle's parameters (past the last one: unused) are read ahead
        cs_next = *reinterpret_cast<const ulonglong2 *>(ap);
        ab_next = *reinterpret_cast<const float2 *>(&ap->a);
        int t[4];
        u64 ff[4];
        run_positions<GEOM, STORE, UNIT, Y, CLS == RUN_G>(cs, ab.x, rc[0], rc[1], fc, ntmin, rdt2, t, ff);
        const unsigned char *q0 = w + min((unsigned)(t[0] - base), kmax) * 16;
        const unsigned char *q3 = w + min((unsigned)(t[3] - base), kmax) * 16;
        // two groups at a time: the bins of more would not fit the registers
        constexpr int GG = G >= 2 ? 2 : 1;
#pragma unroll
        for (int h = 0; h < G / GG; h++) {
            if (h) asm volatile("" ::: "memory");   // keeps the next groups' loads after these
            const int wh = h * GG * wbytes;
            auto bins = [&](const unsigned char *q, auto &b) {   // element q and the following ones
#pragma unroll
                for (int g = 0; g < GG; g++) load_bins<STORE>(q + wh + g * wbytes, g, b);
            };
            auto at = [&](int p) -> u64(&)[GG][2] { return *reinterpret_cast<u64(*)[GG][2]>(&acc[p].v[h * GG]); };
            if constexpr (CLS == RUN_G) {
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    RunBin<STORE> b[1][GG];
                    bins(w + min((unsigned)(t[p] - base), kmax) * 16, b);
                    take<STORE, GG>(at(p), b[0], ff[p]);
                }
            } else if constexpr (CLS == RUN_A) {   // pixels 1 and 2 are in pixel 0's or pixel 3's bin
                RunBin<STORE> b[1][GG], e[1][GG];
                bins(q0, b);
                bins(q3, e);
                take<STORE, GG>(at(0), b[0], ff[0]);
                take_either<STORE, GG>(at(1), b[0], e[0], ff[1], t[1], t[0]);
                take_either<STORE, GG>(at(2), b[0], e[0], ff[2], t[2], t[0]);
                take<STORE, GG>(at(3), e[0], ff[3]);
            } else {
                constexpr int NB = CLS == RUN_B ? 2 : 3, l2 = NB - 2;
                RunBin<STORE> b[NB][GG];
                bins(q0, b);
                take<STORE, GG>(at(0), b[0], ff[0]);
                take_either<STORE, GG>(at(1), b[0], b[1], ff[1], t[1], t[0]);
                take_either<STORE, GG>(at(2), b[l2], b[l2 + 1], ff[2], t[2], t[0] + l2);
                if constexpr (CLS == RUN_C) {
                    take_either<STORE, GG>(at(3), b[1], b[2], ff[3], t[3], t[0] + 1);
                } else {
                    RunBin<STORE> e[1][GG];
                    bins(q3, e);
                    take<STORE, GG>(at(3), e[0], ff[3]);
                }
            }
        }
    }
}

// The same for one slice on plain rows (four-byte elements, one load per bin).
template <int STORE> struct RunBin1 {
    float m, d;
};
template <int STORE> __device__ __forceinline__ RunBin1<STORE> load_bin1(const unsigned char *q)
{
    RunBin1<STORE> b;
    if constexpr (STORE == STORE_F32) {
        b.m = *reinterpret_cast<const float *>(q);
        b.d = 0.f;
    } else {
        const uint32_t u = *reinterpret_cast<const uint32_t *>(q);
        b.m = __uint_as_float(u << 16);
        b.d = __uint_as_float(u & 0xffff0000u);
    }
    return b;
}
template <int STORE> __device__ __forceinline__ float value1(const RunBin1<STORE> &b, u64 ff)
{
    if constexpr (STORE == STORE_F32) return b.m;
    float f, g;
    unpack2(ff, f, g);
    return __fmaf_rn(f, b.d, b.m);
}
template <int GEOM, int STORE, bool UNIT, int CLS, bool Y>
__device__ __forceinline__ void run_angles(RunAcc<0> (&acc)[4], const RunParam *prm, const unsigned char *win,
                                           int wbytes, int al, int end, const u64 (&rc)[2], u64 fc, u64 ntmin,
                                           u64 rdt2, int W)
{
    const unsigned char *w = win + al * wbytes;
    const unsigned kmax = W - 5;
    const RunParam *ap = prm + al, *ae = prm + end;
#pragma unroll 2
    for (; ap != ae; ap++, w += wbytes) {
        const ulonglong2 cs = *reinterpret_cast<const ulonglong2 *>(ap);
        const float2 ab = *reinterpret_cast<const float2 *>(&ap->a);
        const int base = __float_as_int(ab.y);
        int t[4];
        u64 ff[4];
        run_positions<GEOM, STORE, UNIT, Y, CLS == RUN_G>(cs, ab.x, rc[0], rc[1], fc, ntmin, rdt2, t, ff);
        if constexpr (CLS == RUN_G) {
#pragma unroll
            for (int p = 0; p < 4; p++)
                acc[p].v += value1<STORE>(
                    load_bin1<STORE>(w + min((unsigned)(t[p] - base), kmax) * 4), ff[p]);
        } else {
            const unsigned char *q0 = w + min((unsigned)(t[0] - base), kmax) * 4;
            const RunBin1<STORE> b0 = load_bin1<STORE>(q0);
            const RunBin1<STORE> e = load_bin1<STORE>(w + min((unsigned)(t[3] - base), kmax) * 4);
            acc[0].v += value1<STORE>(b0, ff[0]);
            acc[3].v += value1<STORE>(e, ff[3]);
            if constexpr (CLS == RUN_A) {
                acc[1].v += t[1] == t[0] ? value1<STORE>(b0, ff[1]) : value1<STORE>(e, ff[1]);
                acc[2].v += t[2] == t[0] ? value1<STORE>(b0, ff[2]) : value1<STORE>(e, ff[2]);
            } else {   // pixel 2 by a load of its own: no more loads than the bins between
                const RunBin1<STORE> b1 = load_bin1<STORE>(q0 + 4);
                const RunBin1<STORE> c = CLS == RUN_B ? (t[2] == t[0] ? b0 : b1)
                                                      : load_bin1<STORE>(w + min((unsigned)(t[2] - base), kmax) * 4);
                acc[1].v += t[1] == t[0] ? value1<STORE>(b0, ff[1]) : value1<STORE>(b1, ff[1]);
                acc[2].v += value1<STORE>(c, ff[2]);
            }
        }
    }
}

// CTAs per SM the register allocation must allow
constexpr int run_min_blocks(int store, int groups)
{
    return groups >= 2 ? 2 : (groups == 0 && store == STORE_F32 ? 4 : 3);
}

// tid.x and ctaid.x/y read anew: what rarely run code derives from them is not
// hoisted into (and spilled around) the angle loop
__device__ __forceinline__ int fresh_tid()
{
    int v;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(v));
    return v;
}
__device__ __forceinline__ int fresh_ctaid_x()
{
    int v;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(v));
    return v;
}
__device__ __forceinline__ int fresh_ctaid_y()
{
    int v;
    asm volatile("mov.u32 %0, %%ctaid.y;" : "=r"(v));
    return v;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Tile of 32 x 32 pixels, 256 threads with a run of four pixels each, of G groups
// of four slices (rows interleaved by slice) or of one slice (G = 0, plain rows).
// (Two runs per thread on 64 x 32 pixels: 28.5 ms where two groups take 26.2.)
// A stage (AB angles) is copied while the one before it is summed; the third
// buffer keeps the copying warp from waiting for the slowest one (copying two
// stages ahead, which leaves no such slack: 30.3 ms).
constexpr int kRunStages = 3, kRunTile = 32;
constexpr int kRunScratch = (kRunTile * (kRunTile + 1) * 4 + 127) / 128 * 128;                  // one slice of the tile
constexpr int kRunFixed = 128 + kRunStages * 32 * (int)sizeof(RunParam) + kRunScratch;          // before the windows

template <int GEOM, int STORE, bool UNIT, int G>
__global__ void __launch_bounds__(BP_THREADS, run_min_blocks(STORE, G)) bp_run_kernel(const BpArgs p, const int AB)
{
    constexpr int P = 4, NS = kRunStages, GW = G ? G : 1, ES = G ? 16 : 4;   // windows per angle, element bytes
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + NS, *turned = empty + NS;
    volatile int *armed = reinterpret_cast<volatile int *>(turned + 1);   // last stage copied into each buffer
    using Stages = Ring<NS>;
    RunParam *prm = reinterpret_cast<RunParam *>(smem + 128);
    float *scratch = reinterpret_cast<float *>(smem + kRunFixed - kRunScratch);
    unsigned char *win = smem + kRunFixed;
    const int wbytes = p.W * ES, stage_bytes = AB * GW * wbytes;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int A = p.nangles, nst = (A + AB - 1) / AB;
    const size_t gstride = (size_t)A * p.Wg * ES;
    const unsigned char *rows = p.filt + (size_t)blockIdx.z * GW * gstride;

    if (tid == 0) {
        for (int i = 0; i < NS; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], BP_THREADS / 32);
            armed[i] = -1;
        }
        mbar_init(turned, BP_THREADS / 32);
        fence_mbar_init();
    }
    __syncthreads();

    // Waits are bounded; after one that ran out (reported through the error
    // flag) the rest do not wait, so that every warp reaches the end, and the
    // warp copies nothing more: the copy it waited for may still be on its way.
    bool ok = true;
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (!mbar_wait_bounded(bar, parity, ok ? kWaitLimit : 1)) ok = false;
    };

    // One warp: the window base and mode of every angle of stage s, then one
    // bulk copy per angle and group.  The warps take turns.
    auto issue = [&](int s) {
        const int b = Stages::buffer(s), a0 = s * AB, na = min(AB, A - a0), lane = fresh_tid() & 31;
        const int x0 = fresh_ctaid_x() * kRunTile, y0 = fresh_ctaid_y() * kRunTile;
        if (Stages::reused(s)) wait(&empty[b], Stages::parity(Stages::before(s)));
        if (!__all_sync(0xffffffffu, ok)) return;
        int base = 0;
        if (lane < na) {
            AngleParam ap;
            int tmin_i = 0;
            angle_param<GEOM, kRunTile, kRunTile>(p, a0 + lane, x0, y0, ap, base, tmin_i);
            RunParam rp;
            if constexpr (GEOM == GEOM_FBP_LIN) {
                // positions are floats relative to the 64-pixel-wide tile's window, as
                // in the other kernels, whatever the tile: bins then shift by whole elements
                int b64;
                angle_param<GEOM, 64, kRunTile>(p, a0 + lane, x0 & ~63, y0, ap, b64, tmin_i);
                rp.c0 = rp.c1 = ap.b;
                rp.s0 = rp.s1 = ap.c;
                rp.a = ap.a;
                rp.mode = run_mode(ap.b, ap.c, p.eps, false);
                rp.base = 0x4B400000 + base - b64;
            } else {
                rp.c0 = rp.c1 = ap.a;
                rp.s0 = rp.s1 = GEOM == GEOM_FBP_REF ? -ap.b : ap.b;
                rp.a = 0.f;
                rp.mode = run_mode(rp.c0, rp.s0, p.eps, tmin_i <= 1);
                rp.base = ap.d + ((rp.mode >> 2) == RUN_G ? 0 : 0x4B000000);
            }
            rp.pad = 0;
            prm[b * 32 + lane] = rp;
        }
        __syncwarp();
        if (lane == 0) {
            armed[b] = s;
            mbar_arrive_expect_tx(&full[b], (uint32_t)(na * GW * wbytes));   // releases prm
        }
        __syncwarp();
        if (lane < na) {
            fence_proxy_async_smem();
#pragma unroll
            for (int g = 0; g < GW; g++)
                bulk_g2s(win + (size_t)b * stage_bytes + (size_t)(lane * GW + g) * wbytes,
                         rows + g * gstride + ((size_t)(a0 + lane) * p.Wg + base) * ES, (uint32_t)wbytes, &full[b]);
        }
    };
    if (warp < NS - 2 && warp < nst) issue(warp);

    using Acc = RunAcc<G>;
    Acc acc[P];
#pragma unroll
    for (int i = 0; i < P; i++)
#pragma unroll
        for (int q = 0; q < Acc::slices; q++) acc[i].set(q, 0.f);
    int cur = -1;                 // orientation of the accumulators
    uint32_t nturn = 0;
    u64 rc[P / 2];                // coordinates of the run's pixels, two per register pair
    u64 fc = 0;                   // coordinate on the other axis, twice

    auto xcoord = [&](int x) {
        const int x0 = fresh_ctaid_x() * kRunTile;
        if constexpr (GEOM == GEOM_FBP_REF) return __fmaf_rn((float)(x0 + x + p.offo), p.dx, p.xmin);
        else if constexpr (GEOM == GEOM_EM_REF) return __fmaf_rn((float)(x0 + x), p.dxy, p.xymin);
        else return (float)(x + (x0 & 63));
    };
    auto ycoord = [&](int y) {
        const int y0 = fresh_ctaid_y() * kRunTile;
        if constexpr (GEOM == GEOM_FBP_REF) return __fmaf_rn((float)(y0 + y + p.offo), p.dy, p.ymin);
        else if constexpr (GEOM == GEOM_EM_REF) return __fmaf_rn((float)(y0 + y), p.dxy, p.xymin);
        else return (float)y;
    };
    auto place = [&](int o, int &px, int &py) {     // first pixel of this thread in orientation o
        const int tid = fresh_tid(), lane = tid & 31, warp = tid >> 5;
        if (!(o & 1)) px = warp * P, py = lane;
        else px = lane, py = warp * P;
    };
    auto sync_turn = [&]() {      // all warps, bounded
        __syncwarp();
        if ((fresh_tid() & 31) == 0) mbar_arrive(turned);
        wait(turned, nturn & 1);
        nturn++;
    };
    auto turn = [&](int o) {      // bring the accumulators into orientation o (whole CTA)
        int px, py;
        if (cur >= 0 && ((cur ^ o) & 1)) {
#pragma unroll
            for (int q = 0; q < Acc::slices; q++) {
                place(cur, px, py);
#pragma unroll
                for (int i = 0; i < P; i++) {
                    const int d = (cur & 2) ? P - 1 - i : i;
                    scratch[((cur & 1) ? py + d : py) * (kRunTile + 1) + ((cur & 1) ? px : px + d)] = acc[i].get(q);
                }
                sync_turn();
                place(o, px, py);
#pragma unroll
                for (int i = 0; i < P; i++) {
                    const int d = (o & 2) ? P - 1 - i : i;
                    acc[i].set(q, scratch[((o & 1) ? py + d : py) * (kRunTile + 1) + ((o & 1) ? px : px + d)]);
                }
                sync_turn();
            }
        } else if (cur >= 0 && cur != o) {
#pragma unroll
            for (int i = 0; i < P / 2; i++) {
                const Acc v = acc[i];
                acc[i] = acc[P - 1 - i];
                acc[P - 1 - i] = v;
            }
        }
        cur = o;
        place(o, px, py);
        const float other = (o & 1) ? xcoord(px) : ycoord(py);
        fc = pack2(other, other);
#pragma unroll
        for (int i = 0; i < P; i += 2) {
            const int d0 = (o & 2) ? P - 1 - i : i, d1 = (o & 2) ? P - 2 - i : i + 1;
            rc[i / 2] = (o & 1) ? pack2(ycoord(py + d0), ycoord(py + d1)) : pack2(xcoord(px + d0), xcoord(px + d1));
        }
    };

    const u64 ntmin = pack2(-p.tmin, -p.tmin);
    const float rdt = __fdividef(1.0f, p.dt);   // t / dt is t times this reciprocal
    const u64 rdt2 = pack2(rdt, rdt);

#pragma unroll 1
    for (int s = 0; s < nst; s++) {
        const int b = Stages::buffer(s);
        if (s + NS - 2 < nst && warp == s % (BP_THREADS / 32)) issue(s + NS - 2);
        wait(&full[b], Stages::parity(s));
        const int na = min(AB, A - s * AB), lane = fresh_tid() & 31;
        const unsigned char *w = win + (size_t)b * stage_bytes;
        const RunParam *pb = prm + b * 32;
        const int modes = lane < na ? pb[lane].mode : -1;
#pragma unroll 1
        for (int al = 0; al < na;) {
            const int mode = __shfl_sync(0xffffffffu, modes, al);
            const unsigned other = __ballot_sync(0xffffffffu, modes != mode) & (0xffffffffu << al);
            const int end = other ? __ffs(other) - 1 : 32;   // a mode of -1 ends the stage's angles
            if ((mode & 3) != cur) turn(mode & 3);
            switch (((mode >> 2) << 1) | (mode & 1)) {
#define RAFT_RUN(C, Y)                                                                                           \
    case 2 * C + Y:                                                                                              \
        run_angles<GEOM, STORE, UNIT, C, Y != 0>(acc, pb, w, wbytes, al, end, rc, fc, ntmin, rdt2, p.W); \
        break;
                RAFT_RUN(RUN_A, 0) RAFT_RUN(RUN_A, 1) RAFT_RUN(RUN_B, 0) RAFT_RUN(RUN_B, 1) RAFT_RUN(RUN_C, 0)
                RAFT_RUN(RUN_C, 1) RAFT_RUN(RUN_D, 0) RAFT_RUN(RUN_D, 1) RAFT_RUN(RUN_G, 0)
#undef RAFT_RUN
            default:
                run_angles<GEOM, STORE, UNIT, RUN_G, true>(acc, pb, w, wbytes, al, end, rc, fc, ntmin, rdt2, p.W);
                break;
            }
            al = end;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[b]);
    }
    if (!ok) {
        if (p.err) atomicExch(p.err, 1);
        // shared memory is given back only after the copies into it have landed
        for (int i = 0; i < NS; i++)
            if (const int s = armed[i]; s >= 0) mbar_wait_bounded(&full[i], Stages::parity(s), kWaitLimit);
        return;
    }

    const int slice0 = blockIdx.z * Acc::slices, nsl = min(Acc::slices, p.nslices - slice0);
    const int x0 = fresh_ctaid_x() * kRunTile, y0 = fresh_ctaid_y() * kRunTile;
    int px, py;
    place(cur, px, py);
    const float half = STORE == STORE_PAIR_F32 ? 0.5f : 1.0f;
#pragma unroll
    for (int q = 0; q < Acc::slices; q++) {
        if (q >= nsl) break;
        float *out = p.img + (size_t)(slice0 + q) * p.No * p.No;
        const float *den = p.den ? p.den + (size_t)(slice0 + q) * p.No * p.No : nullptr;
#pragma unroll
        for (int i = 0; i < P; i++) {
            const int d = (cur & 2) ? P - 1 - i : i;
            const int X = x0 + ((cur & 1) ? px : px + d), Y = y0 + ((cur & 1) ? py + d : py);
            if (X < p.No && Y < p.No) {
                const size_t o = (size_t)Y * p.No + X;
                const float v = acc[i].get(q) * half;
                if (p.update) out[o] = out[o] * v / den[o];
                else out[o] = v;
            }
        }
    }
}

}  // namespace raft
