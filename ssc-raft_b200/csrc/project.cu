// project.cu -- the ray-driven parallel-beam projectors.
//
// Reference kernels restated (cnpem/ssc-raft):
//   * Radon_RT_version_sscRadon, cuda/src/geometries/parallel/forward_methods/radon_rt.cu:131-174
//       dx = 2ax/(nx-1), dy = 2ay/(ny-1), t = -ax + i*dx, for r < ny:
//       s = -ay + r*dy, (x, y) = (t c - s s_, t s_ + s c),
//       sum img[(int)((y+1)/dy)][(int)((x+1)/dx)], out = sum*dy
//   * kernel_radon, em_RT_kernel.cu:145-185 (EM forward; one step dt = 2/(nrays-1)
//     for rays, samples and pixels), with the EM epilogues fused:
//       tEM  kernel_flatTimesExp (em_RT_kernel.cu:20-32): q = flat * exp(-p)
//       eEM  kernel_radonWithDivision (em_RT_kernel.cu:188-246):
//            q = max(0, y * SIGN(p) / sqrt(1e-8 + p^2))
//     and the angle step folded in, written straight into the window rows
//     the EM backprojector stages.  Optional FP64 reductions (data residual,
//     Poisson log-likelihood) are accumulated per slice in the same pass.
//
// The sample positions and indices are computed with the reference's FP32
// expressions (this file is compiled with fast math, as the reference is),
// so the nearest-pixel choice is the reference's.  The multiply-adds are
// written out (t = i*d - a, x = t*c - s*sin, y = t*sin + s*c as single-rounding
// fmaf with the product s*sin / s*c rounded first -- the contraction the
// reference build produces) so that no template instance can contract them
// differently.
#include "raft.hpp"
#include "ptx.hpp"
#include "profile.hpp"

#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace raft {

constexpr int PJ_WARPS = 8;   // 256 threads per block

// Thread -> (ray, angle, sample phase) shapes.  A warp covers RW neighbouring
// rays at AW = 32 / (RW PH) neighbouring angles, each ray's samples split over
// PH lanes (lane ph sums samples m = ph, ph + PH, ... in order; the PH partial
// sums are then combined by a fixed butterfly of warp shuffles, so the
// summation order depends on PH alone, not on the slice count, the layout or
// the ray/angle shape); a block covers BR rays x BA angles.  The lanes of a
// warp load their samples together.  With one angle and one phase per warp
// (RW = 32) the 32 pixels lie on a line across the ray direction, one pixel
// apart: along an image row near 0 degrees, but on ~23 different rows near 45
// degrees.  A few rays x a few consecutive samples cover a compact
// parallelogram instead (about 12 cache lines per warp load of 32-byte pixels
// against 15-17 for the line, averaged over angles).  Measured (B200, 512 x
// 1024^2 x 900): interleaved 8-slice images four rays x four phases x two
// angles, Radon 5096 GUPS against 4655 for one angle x 32 rays, tEM 176.7
// against 182.1 ms per iteration; planar single-slice projection (instruction
// issue bound) is best sequential (ragged batch 1863 GUPS) and costs 3.7 % at
// PH = 4 (eight rays x four phases, 1795 GUPS), kept so that every slice count
// sums in the same order.
template <int RW, int PH, int BRS> struct PjShape {
    static_assert(32 % (RW * PH) == 0, "a warp holds whole (ray, phase) groups");
    static constexpr int AW = 32 / (RW * PH);     // angles per warp
    static constexpr int BR = BRS;                // rays per block
    static constexpr int BA = 256 / (BR * PH);    // angles per block
    static constexpr int WR = BR / RW;            // warps along the rays
    static_assert(BR % RW == 0 && BA % AW == 0 && WR * (BA / AW) == 8, "eight warps per block");
};

// S slices per thread share every sample's position and pixel index (the
// geometry is the same for all slices).  Warps whose angle is steeper than
// 45 degrees read a transposed copy of the images (imgT[x][y]) so that the
// 32 rays of the warp touch consecutive addresses; the index arithmetic and
// therefore the chosen pixels are unchanged.  IL = 1 (S = 8) reads the
// slice-interleaved copies instead (il[g][y][x][8], ilT[g][x][y][8]): one
// sample's eight slice values are one 32-byte load (one sector).
// 256-bit read-only load of eight consecutive floats (32-byte aligned)
__device__ __forceinline__ void ldg_v8(const float *p, float (&w)[8])
{
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
                 : "l"(p));
}

// Rows of the interleaved copies start on 128-byte lines.  Rows of 32-byte pixels that
// do not cost every warp load more lines: 8 x 901^2 x 360 621 us with rows nx pixels
// apart, 485 now.
__host__ __device__ __forceinline__ int il_pitch(int n) { return (n + 3) & ~3; }

template <int EM, int EPI, int S, int IL, int RW, int PH, int BRS>
__device__ __forceinline__ void project_block(const ProjLaunch &p, const int bx, const int by, const int bz)
{
    static_assert(!IL || S == 8, "interleaved images hold groups of 8 slices");
    using Sh = PjShape<RW, PH, BRS>;
    const int w = threadIdx.y, lane = threadIdx.x;
    const int ph = lane / (RW * Sh::AW);                                      // sample phase
    const int i = bx * Sh::BR + (w % Sh::WR) * RW + lane % RW;                // ray
    const int j = by * Sh::BA + (w / Sh::WR) * Sh::AW + (lane / RW) % Sh::AW;  // angle
    const int k0 = bz * S;                        // first slice
    const int nsl = min(S, p.nslices - k0);
    const bool valid = (i < p.nrays) && (j < p.nangles);
    const int nx = p.nx, ny = p.ny;
    const size_t plane = (size_t)nx * ny;
    float value[S], linesum[S];
    float step = 0.f;
#pragma unroll
    for (int q = 0; q < S; q++) value[q] = linesum[q] = 0.f;
    if (valid) {
        const float ang = p.angles[j];
        const float ctheta = __cosf(ang);
        const float stheta = __sinf(ang);
        const bool steep = (IL ? p.ilT : p.imgT) && fabsf(stheta) > fabsf(ctheta);
        // address = Y*nx + X (row-major) or X*ny + Y (transposed), rows of interleaved
        // copies il_pitch apart
        const int px = IL ? il_pitch(nx) : nx, py = IL ? il_pitch(ny) : ny;
        const float *img = IL ? (steep ? p.ilT + (size_t)bz * nx * py * 8 : p.il + (size_t)bz * ny * px * 8)
                              : (steep ? p.imgT : p.img) + (size_t)k0 * plane;
        const int sy = steep ? 1 : px, sx = steep ? py : 1;
        // This lane's samples (m = ph, ph + PH, ...) are processed four at a
        // time: the four positions and pixel loads are issued together
        // (independent, so their latency overlaps), then added in sample order.
        auto sample_loop = [&](const float t, const float d0, const float ay0, const float ddx,
                               const float ddy, const int nsamp, const int limx, const int limy) {
            int m = ph;
            if constexpr (IL) {
                // two samples' positions and two slices' sums per instruction (the
                // lanes round as the scalar instructions do); the sample number is
                // counted in float, exactly.  24 x 1024^2 x 900: 4400 -> 4104 us (with rows on
                // 128-byte lines and four blocks per SM).
                const u64 d2 = pack2(d0, d0), na2 = pack2(-ay0, -ay0), t2 = pack2(t, t), c2 = pack2(ctheta, ctheta);
                const u64 s2 = pack2(stheta, stheta), ns2 = pack2(-stheta, -stheta), one2 = pack2(1.f, 1.f);
                const float rx = __fdividef(1.0f, ddx), ry = __fdividef(1.0f, ddy);   // a / ddx is a times this
                const u64 rx2 = pack2(rx, rx), ry2 = pack2(ry, ry), step2 = pack2(2.f * PH, 2.f * PH);
                u64 sum[4];
#pragma unroll
                for (int q = 0; q < 4; q++) sum[q] = 0ull;
                u64 m2 = pack2((float)ph, (float)(ph + PH));   // the next two sample numbers
                constexpr int U = 4;   // samples in flight (6, 8 and 12 measured slower)
                auto sample2 = [&](u64 mm, float (&w0)[8], float (&w1)[8]) {
                    const u64 s = fma2(mm, d2, na2);
                    const u64 x = mul2(add2(fma2(t2, c2, mul2(s, ns2)), one2), rx2);
                    const u64 y = mul2(add2(fma2(t2, s2, mul2(s, c2)), one2), ry2);
                    float x0, x1, y0, y1;
                    unpack2(x, x0, x1);
                    unpack2(y, y0, y1);
                    // one 32-byte load: the pixel's eight slice values, or eight zeros
                    // (p.il_zero) for a sample outside the image
                    const int X0 = (int)x0, Y0 = (int)y0, X1 = (int)x1, Y1 = (int)y1;
                    const bool in0 = ((unsigned)X0 < (unsigned)limx) & ((unsigned)Y0 < (unsigned)limy);
                    const bool in1 = ((unsigned)X1 < (unsigned)limx) & ((unsigned)Y1 < (unsigned)limy);
                    const unsigned p0 = (unsigned)Y0 * (unsigned)sy + (unsigned)X0 * (unsigned)sx;
                    const unsigned p1 = (unsigned)Y1 * (unsigned)sy + (unsigned)X1 * (unsigned)sx;
                    ldg_v8(in0 ? img + (size_t)p0 * 8 : p.il_zero, w0);
                    ldg_v8(in1 ? img + (size_t)p1 * 8 : p.il_zero, w1);
                };
                for (; m + (U - 1) * PH < nsamp; m += U * PH) {
                    float w[U][8];
#pragma unroll
                    for (int u = 0; u < U; u += 2) {
                        sample2(m2, w[u], w[u + 1]);
                        m2 = add2(m2, step2);
                    }
#pragma unroll
                    for (int u = 0; u < U; u++)
#pragma unroll
                        for (int q = 0; q < 4; q++) sum[q] = add2(sum[q], pack2(w[u][2 * q], w[u][2 * q + 1]));
                }
                for (; m + PH < nsamp; m += 2 * PH) {
                    float w[2][8];
                    sample2(m2, w[0], w[1]);
                    m2 = add2(m2, step2);
#pragma unroll
                    for (int u = 0; u < 2; u++)
#pragma unroll
                        for (int q = 0; q < 4; q++) sum[q] = add2(sum[q], pack2(w[u][2 * q], w[u][2 * q + 1]));
                }
#pragma unroll
                for (int q = 0; q < 4; q++) unpack2(sum[q], linesum[2 * q], linesum[2 * q + 1]);
            } else {
                for (; m + 3 * PH < nsamp; m += 4 * PH) {
                    float v[4][S];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float s = __fmaf_rn((float)(m + u * PH), d0, -ay0);
                        const float x = __fmaf_rn(t, ctheta, -__fmul_rn(s, stheta));
                        const float y = __fmaf_rn(t, stheta, __fmul_rn(s, ctheta));
                        const int X = (int)((x + 1) / ddx);
                        const int Y = (int)((y + 1) / ddy);
                        // 32-bit pixel index (the launch checks nx * ny < 2^32), predicated loads
                        const bool in = ((unsigned)X < (unsigned)limx) & ((unsigned)Y < (unsigned)limy);
                        const unsigned pix = (unsigned)Y * (unsigned)sy + (unsigned)X * (unsigned)sx;
#pragma unroll
                        for (int q = 0; q < S; q++) {
                            float val = 0.f;
                            if (in && q < nsl) val = __ldg(img + q * plane + pix);
                            v[u][q] = val;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++)
#pragma unroll
                        for (int q = 0; q < S; q++) linesum[q] += v[u][q];
                }
            }
            for (; m < nsamp; m += PH) {
                const float s = __fmaf_rn((float)m, d0, -ay0);
                const float x = __fmaf_rn(t, ctheta, -__fmul_rn(s, stheta));
                const float y = __fmaf_rn(t, stheta, __fmul_rn(s, ctheta));
                const int X = (int)((x + 1) / ddx);
                const int Y = (int)((y + 1) / ddy);
                if (((unsigned)X < (unsigned)limx) & ((unsigned)Y < (unsigned)limy)) {
                    const unsigned pix = (unsigned)Y * (unsigned)sy + (unsigned)X * (unsigned)sx;
                    if constexpr (IL) {
                        float w[8];
                        ldg_v8(img + (size_t)pix * 8, w);
#pragma unroll
                        for (int q = 0; q < S; q++) linesum[q] += w[q];
                    } else {
#pragma unroll
                        for (int q = 0; q < S; q++)
                            if (q < nsl) linesum[q] += __ldg(img + q * plane + pix);
                    }
                }
            }
        };
        if constexpr (EM) {
            // kernel_radon: dt = 2.0*a/(nrays-1) in double, a = 1; one step for
            // rays, samples and pixels; the image is N x N with N = nx
            const float a = p.ax;
            const float dt = (float)(2.0 * a / (p.nrays - 1));
            const float t = __fmaf_rn((float)i, dt, -a);
            sample_loop(t, dt, a, dt, dt, p.nrays, nx, nx);
            step = dt;
        } else {
            const float dx = 2.0f * p.ax / (float)(unsigned)(nx - 1);
            const float dy = 2.0f * p.ay / (float)(unsigned)(ny - 1);
            const float t = __fmaf_rn((float)i, dx, -p.ax);
            sample_loop(t, dy, p.ay, dx, dy, ny, nx, ny);
            step = dy;
        }
    }
    // combine the PH partial sums of each ray (every lane of the warp takes
    // part; the lanes of one ray share its validity, invalid rays sum zeros):
    // ((p0 + p1) + (p2 + p3)) for PH = 4, the same in every lane of the ray
#pragma unroll
    for (int o = RW * Sh::AW; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < S; q++) linesum[q] += __shfl_xor_sync(0xffffffffu, linesum[q], o);
#pragma unroll
    for (int q = 0; q < S; q++) value[q] = linesum[q] * step;

    // FP64 metric terms of this lane's slices q = ph + PH u (slot u = q / PH)
    constexpr int U = (S + PH - 1) / PH;
    double r2[U], y2[U], nll[U];
#pragma unroll
    for (int u = 0; u < U; u++) r2[u] = y2[u] = nll[u] = 0.0;
#pragma unroll
    for (int q = 0; q < S; q++) {
        const int k = k0 + q;
        if (!valid || q >= nsl || q % PH != ph) continue;   // phase lane ph writes slices q = ph mod PH
        const size_t vox = ((size_t)k * p.nangles + j) * p.nrays + i;
        float out = value[q];
        if constexpr (EPI == 1) {
            // tEM: model = flat * exp(-p); data = counts (kernel_flatTimesExp, em_RT_kernel.cu:20-32)
            const float fl = p.flat[(size_t)k * p.nrays + i];
            out = fl * __expf(-value[q]);
            if (p.metrics) {
                const double y = p.data[vox];
                const double m = fl * exp(-(double)value[q]);
                r2[q / PH] = (m - y) * (m - y);
                y2[q / PH] = y * y;
                nll[q / PH] = m + y * (double)value[q];
            }
        } else if constexpr (EPI == 2) {
            // eEM ratio, APPROXINVX(value, 1e-4) = SIGN/sqrtf(SQR(e)+SQR(x)) (configs.hpp:30-32)
            const float TOLZERO = 0.0001f;
            const float y = p.data[vox];
            const int sgn = (value[q] > 0) ? 1 : ((value[q] < 0) ? -1 : 0);
            out = y * (sgn / sqrtf(TOLZERO * TOLZERO + value[q] * value[q]));
            if (out < 0) out = 0.0f;
            if (p.metrics) {
                const double yd = y, m = value[q];
                r2[q / PH] = (m - yd) * (m - yd);
                y2[q / PH] = yd * yd;
                nll[q / PH] = (m > 0) ? m - yd * log(m) : 0.0;
            }
        }
        if (p.windowed) {
            const float w = p.wt ? p.wt[j] : 1.f;
            const size_t e = (size_t)(i - p.wlo);
            // 2: rows interleaved by slice in groups of four, the layout the
            // four-slice backprojector stages (the four phase lanes of a ray
            // write the four floats of one 16-byte element)
            const size_t o = p.windowed == 2 ? ((((size_t)(k >> 2) * p.nangles + j) * p.Wg + e) << 2) + (k & 3)
                                             : ((size_t)k * p.nangles + j) * p.Wg + e;
            p.out[o] = out * w;
        } else {
            p.out[vox] = out;
        }
    }
    if constexpr (EPI != 0) {
        if (p.metrics) {
            // FP64 per-slice sums: over the warp's lanes of one sample phase
            // (the lanes holding slice q), then across the block's warps
            __shared__ double red[3][S][PJ_WARPS];
            constexpr int G = RW * Sh::AW;   // lanes of one phase
#pragma unroll
            for (int u = 0; u < U; u++) {
                double a0 = r2[u], a1 = y2[u], a2 = nll[u];
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
                    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
                    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
                }
                const int q = ph + PH * u;
                if (threadIdx.x % G == 0 && q < S) {
                    red[0][q][threadIdx.y] = a0;
                    red[1][q][threadIdx.y] = a1;
                    red[2][q][threadIdx.y] = a2;
                }
            }
            __syncthreads();
            if (threadIdx.y == 0 && threadIdx.x < 3 * S) {
                const int q = threadIdx.x / 3, c = threadIdx.x - 3 * q;
                if (q < nsl) {
                    double sum = 0.0;
                    for (int w = 0; w < PJ_WARPS; w++) sum += red[c][q][w];
                    atomicAdd(&p.metrics[(size_t)(k0 + q) * 3 + c], sum);
                }
            }
        }
    }
}

template <int EM, int EPI, int S, int IL, int RW, int PH, int BRS>
// Four blocks per SM on interleaved images (24 x 1024^2 x 900: 4104 us; three blocks:
// 4169, and launches of few blocks, 800^2 x 45, up to a quarter slower for their second
// wave; 53 registers, the compiler's choice for EM: 16 x 1024^2 x 900 tEM 15.18 ->
// 15.69 ms); the compiler's choice on planar ones (a bound of one block costs 7 - 17 %).
__global__ void __launch_bounds__(32 * PJ_WARPS, IL ? 4 : 0)
project_kernel(const ProjLaunch p)
{
    project_block<EM, EPI, S, IL, RW, PH, BRS>(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Launch shapes (rays per warp RW, sample phases PH, rays per block BR): by
// default four rays x four phases x two angles per warp on interleaved images
// and eight rays x four phases on planar ones, 32 rays per block (blocks of
// 16, 8 or 4 rays at more angles measured 8-10 % slower on the interleaved
// images, the same on planar ones); RAFT_PJ_SEQUENTIAL=1 sums every ray in one
// lane in sample order (the reference's order; 32 rays at one angle, or four
// rays at eight angles per warp).  Read at every launch.
struct PjChoice {
    int rw, ph, br;
};
static bool pj_sequential()
{
    const char *e = getenv("RAFT_PJ_SEQUENTIAL");
    return e && atoi(e) == 1;
}
static PjChoice pj_il() { return pj_sequential() ? PjChoice{32, 1, 32} : PjChoice{4, 4, 32}; }
static PjChoice pj_pl() { return pj_sequential() ? PjChoice{4, 1, 32} : PjChoice{8, 4, 32}; }
template <class F>
static void pj_dispatch(PjChoice c, F &&f)
{
    using std::integral_constant;
    if (c.rw == 32) f(integral_constant<int, 32>{}, integral_constant<int, 1>{}, integral_constant<int, 32>{});
    else if (c.ph == 1) f(integral_constant<int, 4>{}, integral_constant<int, 1>{}, integral_constant<int, 32>{});
    else if (c.rw == 4) f(integral_constant<int, 4>{}, integral_constant<int, 4>{}, integral_constant<int, 32>{});
    else f(integral_constant<int, 8>{}, integral_constant<int, 4>{}, integral_constant<int, 32>{});
}

int project_blocks_per_slice(int nrays, int nangles)
{
    int n = 0;
    pj_dispatch(pj_pl(), [&](auto rw, auto ph, auto br) {
        using Sh = PjShape<decltype(rw)::value, decltype(ph)::value, decltype(br)::value>;
        n = ((nrays + Sh::BR - 1) / Sh::BR) * ((nangles + Sh::BA - 1) / Sh::BA);
    });
    return n;
}

// Ragged projector: one launch over many single-slice requests of different
// sizes; block b belongs to the request r with blk_start[r] <= b < blk_start[r+1].
template <int EM, int EPI, int RW, int PH, int BRS>
__global__ void __launch_bounds__(32 * PJ_WARPS)
project_ragged_kernel(const ProjLaunch *__restrict__ reqs, const int *__restrict__ blk_start, int nreq)
{
    __shared__ int s_r;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        int lo = 0, hi = nreq - 1;
        while (lo < hi) {                       // last r with blk_start[r] <= blockIdx.x
            const int mid = (lo + hi + 1) / 2;
            if (blk_start[mid] <= (int)blockIdx.x) lo = mid;
            else hi = mid - 1;
        }
        s_r = lo;
    }
    __syncthreads();
    const int r = s_r;
    const ProjLaunch &p = reqs[r];
    const int local = blockIdx.x - blk_start[r];
    const int nbx = (p.nrays + PjShape<RW, PH, BRS>::BR - 1) / PjShape<RW, PH, BRS>::BR;
    project_block<EM, EPI, 1, 0, RW, PH, BRS>(p, local % nbx, local / nbx, 0);
}

template <int RW, int PH, int BRS>
static void launch_ragged_shape(const ProjLaunch *d_reqs, const int *d_blk_start, int nreq, int total_blocks,
                                int em, int epilogue, cudaStream_t st)
{
    dim3 block(32, PJ_WARPS);
    if (!em)
        project_ragged_kernel<0, 0, RW, PH, BRS><<<total_blocks, block, 0, st>>>(d_reqs, d_blk_start, nreq);
    else if (epilogue == 1)
        project_ragged_kernel<1, 1, RW, PH, BRS><<<total_blocks, block, 0, st>>>(d_reqs, d_blk_start, nreq);
    else if (epilogue == 2)
        project_ragged_kernel<1, 2, RW, PH, BRS><<<total_blocks, block, 0, st>>>(d_reqs, d_blk_start, nreq);
    else
        project_ragged_kernel<1, 0, RW, PH, BRS><<<total_blocks, block, 0, st>>>(d_reqs, d_blk_start, nreq);
}

void launch_project_ragged(const ProjLaunch *d_reqs, const int *d_blk_start, int nreq, int total_blocks, int em,
                           int epilogue, cudaStream_t st)
{
    if (nreq <= 0 || total_blocks <= 0) return;
    ProfScope ps(PROF_PROJECT, st);
    pj_dispatch(pj_pl(), [&](auto rw, auto ph, auto br) {
        launch_ragged_shape<decltype(rw)::value, decltype(ph)::value, decltype(br)::value>(
            d_reqs, d_blk_start, nreq, total_blocks, em, epilogue, st);
    });
    RAFT_CUDA(cudaGetLastError());
}

// Tiled transpose of each slice: out[k][x][y] = in[k][y][x].
__global__ void transpose_kernel(const float *__restrict__ in, float *__restrict__ out, int nx, int ny)
{
    __shared__ float tile[32][33];
    const size_t plane = (size_t)nx * ny;
    const float *src = in + blockIdx.z * plane;
    float *dst = out + blockIdx.z * plane;
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int y = by + r, x = bx + threadIdx.x;
        if (x < nx && y < ny) tile[r][threadIdx.x] = src[(size_t)y * nx + x];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int x = bx + r, y = by + threadIdx.x;
        if (x < nx && y < ny) dst[(size_t)x * ny + y] = tile[threadIdx.x][r];
    }
}

void launch_transpose(const float *in, float *out, int nx, int ny, int nslices, cudaStream_t st)
{
    if (nslices <= 0) return;
    count_launch();
    dim3 grid((nx + 31) / 32, (ny + 31) / 32, nslices);
    transpose_kernel<<<grid, dim3(32, 8), 0, st>>>(in, out, nx, ny);
    RAFT_CUDA(cudaGetLastError());
}

// Slice-interleaved copies of groups of 8 planes, row-major and transposed:
// il[g][y][x][s] = ilT[g][x][y][s] = in[8g + s][y][x] (rows il_pitch apart; zero where 8g + s is
// past the last plane), plus the eight zeros that samples outside the image
// read.  One 32 x TY pixel tile of all 8 planes per block: TY = 32, or 8 where
// that would leave SMs without a block (301^2: 100 blocks, 10.9 us).
template <int TY>
__global__ void __launch_bounds__(256)
interleave_kernel(const float *__restrict__ in, float *__restrict__ il, float *__restrict__ ilT,
                  float *__restrict__ zero8, int nx, int ny, int nslices)
{
    __shared__ float tile[8][TY][33];
    const size_t plane = (size_t)nx * ny;
    const int g = blockIdx.z, tx = threadIdx.x;
    if ((blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.y) == 0 && tx < 8) zero8[tx] = 0.f;
    const int bx = blockIdx.x * 32, by = blockIdx.y * TY;
#pragma unroll
    for (int s = 0; s < 8; s++) {
        const int k = g * 8 + s;
        for (int r = threadIdx.y; r < TY; r += 8) {
            const int y = by + r, x = bx + tx;
            tile[s][r][tx] = (k < nslices && x < nx && y < ny) ? in[(size_t)k * plane + (size_t)y * nx + x] : 0.f;
        }
    }
    __syncthreads();
    const int px = il_pitch(nx), py = il_pitch(ny);
    float *o = il + (size_t)g * ny * px * 8;
    float *oT = ilT + (size_t)g * nx * py * 8;
    auto put = [&](float *p, int r, int c) {
        float4 *d = reinterpret_cast<float4 *>(p);
        d[0] = make_float4(tile[0][r][c], tile[1][r][c], tile[2][r][c], tile[3][r][c]);
        d[1] = make_float4(tile[4][r][c], tile[5][r][c], tile[6][r][c], tile[7][r][c]);
    };
    for (int r = threadIdx.y; r < TY; r += 8) {
        const int y = by + r, x = bx + tx;
        if (x < nx && y < ny) put(o + ((size_t)y * px + x) * 8, r, tx);
    }
    // transposed: TY consecutive y per x
    for (int e = threadIdx.y * 32 + tx; e < 32 * TY; e += 256) {
        const int c = e / TY, r = e % TY, x = bx + c, y = by + r;
        if (x < nx && y < ny) put(oT + ((size_t)x * py + y) * 8, r, c);
    }
}

// Whether the projector reads interleaved copies.  Eight slices and more do.  Fewer share
// a group of eight, whose projection costs the same (us, interleaved | planar): 5 to 7
// slices against two planar groups of four, 1024^2 x 360 604 | 1608; three slices
// against two of two, 304^2 x 96 27 | 35, 1003^2 x 257 446 | 641; four slices against
// one of four, 901^2 x 128 205 | 225, x 360 485 | 594, and at widths that are multiples
// of 32, which make planar rows slower, 512^2 x 64 43 | 55.  The copies (16 planes
// written, 2 us more than the planar transposition at 300^2, 11 at 800^2, 23 at 1024^2,
// 55 at 2048^2) have to be earned by enough angles.  The 16 planes are not taken for
// few planes of a size where they would claim a good part of the memory.
static bool use_interleaved(int nx, int ny, int nslices, int nangles)
{
    if (nslices >= 8) return true;
    if (nslices < 3 || (size_t)nx * ny > ((size_t)1 << 26)) return false;
    if (nslices >= 5) return nangles >= 16;
    if (nslices == 3) return nangles >= 48;
    return nangles >= ((nx | ny) % 32 ? 128 : 16);
}

static size_t il_bytes(int nx, int ny, int nslices)
{
    const size_t pixels = (size_t)ny * il_pitch(nx) + (size_t)nx * il_pitch(ny);
    return ((nslices + 7) / 8 * pixels + 1) * 8 * sizeof(float);
}

// of up to nslices planes: a last, smaller chunk may be the one that takes the copies
size_t proj_scratch_bytes(int nx, int ny, int nslices, int nangles)
{
    const size_t plane = (size_t)nx * ny * sizeof(float);
    if (nslices <= 0) return 16;
    size_t bytes = 0;
    for (int n = nslices < 8 ? 1 : nslices; n <= nslices; n++)
        bytes = std::max(bytes, use_interleaved(nx, ny, n, nangles)
                                    ? il_bytes(nx, ny, n)
                                    : n * plane);
    return bytes;
}

void stage_proj_images(ProjLaunch &pl, void *scratch, cudaStream_t st)
{
    if (pl.nslices <= 0) return;
    if (use_interleaved(pl.nx, pl.ny, pl.nslices, pl.nangles)) {
        // the projector indexes a pixel of the interleaved copies in 32 bits
        RAFT_CHECK(std::max((size_t)pl.ny * il_pitch(pl.nx), (size_t)pl.nx * il_pitch(pl.ny)) <= 0xffffffffull,
                   "projector: image plane above 2^32 pixels");
        const int G = (pl.nslices + 7) / 8;
        float *il = (float *)scratch;
        float *ilT = il + (size_t)G * 8 * pl.ny * il_pitch(pl.nx);
        float *zero8 = ilT + (size_t)G * 8 * pl.nx * il_pitch(pl.ny);
        count_launch();
        const unsigned bx = (pl.nx + 31) / 32, by = (pl.ny + 31) / 32;
        if ((long long)bx * by * G < 2 * 148)
            interleave_kernel<8><<<dim3(bx, (pl.ny + 7) / 8, G), dim3(32, 8), 0, st>>>(pl.img, il, ilT, zero8, pl.nx, pl.ny,
                                                                                    pl.nslices);
        else
            interleave_kernel<32><<<dim3(bx, by, G), dim3(32, 8), 0, st>>>(pl.img, il, ilT, zero8, pl.nx, pl.ny,
                                                                        pl.nslices);
        RAFT_CUDA(cudaGetLastError());
        pl.il = il;
        pl.ilT = ilT;
        pl.il_zero = zero8;
        pl.imgT = nullptr;
    } else {
        float *t = (float *)scratch;
        launch_transpose(pl.img, t, pl.nx, pl.ny, pl.nslices, st);
        pl.imgT = t;
        pl.il = pl.ilT = pl.il_zero = nullptr;
    }
}

template <int EM, int EPI, int S, int IL, int RW, int PH, int BRS>
static void launch_project_shape(const ProjLaunch &pl, cudaStream_t st)
{
    using Sh = PjShape<RW, PH, BRS>;
    dim3 grid((pl.nrays + Sh::BR - 1) / Sh::BR, (pl.nangles + Sh::BA - 1) / Sh::BA, (pl.nslices + S - 1) / S);
    project_kernel<EM, EPI, S, IL, RW, PH, BRS><<<grid, dim3(32, PJ_WARPS), 0, st>>>(pl);
}

template <int EM, int EPI>
static void launch_project_s(const ProjLaunch &pl, int S, cudaStream_t st)
{
    ProfScope ps(PROF_PROJECT, st);
    if (S == 8) {
        pj_dispatch(pj_il(), [&](auto rw, auto ph, auto br) {
            launch_project_shape<EM, EPI, 8, 1, decltype(rw)::value, decltype(ph)::value, decltype(br)::value>(pl, st);
        });
    } else {
        pj_dispatch(pj_pl(), [&](auto rw, auto ph, auto br) {
            constexpr int RW = decltype(rw)::value, PH = decltype(ph)::value, BR = decltype(br)::value;
            if (S == 4) launch_project_shape<EM, EPI, 4, 0, RW, PH, BR>(pl, st);
            else if (S == 2) launch_project_shape<EM, EPI, 2, 0, RW, PH, BR>(pl, st);
            else launch_project_shape<EM, EPI, 1, 0, RW, PH, BR>(pl, st);
        });
    }
    RAFT_CUDA(cudaGetLastError());
}

void launch_project(const ProjLaunch &pl, cudaStream_t st)
{
    if (pl.nslices <= 0 || pl.nangles <= 0 || pl.nrays <= 0) return;
    // the projector indexes a pixel of a plane in 32 bits
    RAFT_CHECK((size_t)pl.nx * pl.ny <= 0xffffffffull, "projector: image plane above 2^32 pixels");
    RAFT_CHECK((pl.il == nullptr) == (pl.ilT == nullptr) && (pl.il == nullptr) == (pl.il_zero == nullptr),
               "projector: interleaved copies come with their transposed copy and zero pixel");
    const int S = pl.il ? 8 : (pl.nslices >= 4 ? 4 : (pl.nslices >= 2 ? 2 : 1));
    if (!pl.em) {
        launch_project_s<0, 0>(pl, S, st);
    } else {
        switch (pl.epilogue) {
        case 1: launch_project_s<1, 1>(pl, S, st); break;
        case 2: launch_project_s<1, 2>(pl, S, st); break;
        default: launch_project_s<1, 0>(pl, S, st); break;
        }
    }
}

// Plain sinogram -> weighted window rows interleaved by slice in groups of four
// (the bins and slices it does not write stay as they are: zero).
// sino == nullptr writes the weight itself (back-projection of ones).
__global__ void to_window4_kernel(const float *__restrict__ sino, float *__restrict__ rows,
                                  const float *__restrict__ wt, int nslices, int nangles, int nrays, int wlo, int Wg)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrays) return;
    const long long nrow = (long long)((nslices + 3) / 4) * nangles;
    for (long long r = blockIdx.y; r < nrow; r += gridDim.y) {
        const int g = (int)(r / nangles), a = (int)(r - (long long)g * nangles);
        const float w = wt[a];
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = 4 * g + q;
            v[q] = k < nslices ? (sino ? sino[((size_t)k * nangles + a) * nrays + i] : 1.f) * w : 0.f;
        }
        reinterpret_cast<float4 *>(rows)[r * Wg + (i - wlo)] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

void launch_to_window4(const float *sino, float *rows, const float *wt, int nslices, int nangles, int nrays, int wlo,
                       int Wg, cudaStream_t st)
{
    if (nslices <= 0 || nangles <= 0) return;
    const long long nrow = (long long)((nslices + 3) / 4) * nangles;
    dim3 grid((nrays + 255) / 256, (unsigned)(nrow < 65535 ? nrow : 65535));
    count_launch();
    to_window4_kernel<<<grid, 256, 0, st>>>(sino, rows, wt, nslices, nangles, nrays, wlo, Wg);
    RAFT_CUDA(cudaGetLastError());
}

// Plain sinogram -> weighted window rows (the rest of each row stays zero).
// sino == nullptr writes the weight itself (back-projection of ones).
__global__ void to_window_kernel(const float *__restrict__ sino, float *__restrict__ rows,
                                 const float *__restrict__ wt, int nrows, int nangles, int nrays, int wlo,
                                 int Wg)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrays) return;
    for (int r = blockIdx.y; r < nrows; r += gridDim.y) {
        const float w = wt ? wt[r % nangles] : 1.f;
        const float v = sino ? sino[(size_t)r * nrays + i] : 1.f;
        rows[(size_t)r * Wg + (i - wlo)] = v * w;
    }
}

void launch_to_window(const float *sino, float *rows, const float *wt, int nrows, int nangles, int nrays,
                      int wlo, int Wg, cudaStream_t st)
{
    if (nrows <= 0) return;
    dim3 grid((nrays + 255) / 256, nrows < 65535 ? nrows : 65535);
    count_launch();
    to_window_kernel<<<grid, 256, 0, st>>>(sino, rows, wt, nrows, nangles, nrays, wlo, Wg);
    RAFT_CUDA(cudaGetLastError());
}

}  // namespace raft
