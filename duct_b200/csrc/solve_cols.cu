// solve_cols.cu -- the flip-symmetric FP64 GEMM pass (the operator algebra is
// described at fold_operators in setup.cu) on the resident-operator core of
// cols.cuh.
//
// A unit is 4 complex lines of a field: a P^-1 pass (par 1) folds them as
// they are read and writes the even modes, then the odd ones, over the
// eigenvalue divide where asked; a P pass (par 2) reads the two mode blocks
// and unfolds P +- M as it writes.  Fragments, K order and epilogue arithmetic
// are those of pass_s_tile (solve_fp64.cu): equal bit for bit.
//
// What bounds it: the FP64 tensor pipe, 4 n (he^2 + ho^2) flops a plane.
// 255 planes of my = 193 take 133 us a pass (137 with the divide), 0.75 of the
// DMMA rate with the padding to 96 rows counted; the form before, whose CTAs
// staged 8 lines and streamed the operator, 151 to 166.  Graph replays of whole
// solves, before / after, us: 255 planes of my = 193 650 / 567, 256 of my =
// 129 238 / 220 (before: producer and consumer warps, resident operator), of
// my = 145 500 / 442, of my = 35 55 / 41, 84 of my = 65 39 / 37.
#include <math.h>

#include "cols.cuh"
#include "internal.h"

namespace duct {

struct ColsParams {
    PassParams p;
    long long unit0[kMaxFields + 1];   // first unit of each field
};

// Two warps a scheduler where a third's accumulators would cost the registers
// that keep a unit's next lines in flight (96 rows: 567 us with 8 warps, 590 with
// 12 that spill) or has nothing to hide (32 rows: 60 / 66); three at 64 rows
// (220 / 225).
template <int MT> constexpr int kPassWarps = MT == 4 ? 12 : 8;

template <int MT, bool DIV>
__global__ void __launch_bounds__(32 * kPassWarps<MT>, 1) k_pass_cols(const __grid_constant__ ColsParams q, int *err)
{
    constexpr int W = kPassWarps<MT>, GM = 2;
    extern __shared__ __align__(128) double smem[];
    double *Op = smem, *Es = smem + ColShape<MT>::op;   // Es: [2 H]
    __shared__ __align__(8) uint64_t bar;
    const PassParams &p = q.p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    if (tid == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;\n" ::"r"(col_smem(&bar)));
    const long long all = q.unit0[p.nf], a0 = all * blockIdx.x / gridDim.x, a1 = all * (blockIdx.x + 1) / gridDim.x;
    const double *have = nullptr;
    unsigned loads = 0;
#pragma unroll 1
    for (int fi = 0; fi < p.nf; ++fi) {
        if (q.unit0[fi + 1] <= a0 || q.unit0[fi] >= a1) continue;
        const PassField &F = p.f[fi];
        const int u0 = (int)(a0 > q.unit0[fi] ? a0 - q.unit0[fi] : 0);
        const int u1 = (int)((a1 < q.unit0[fi + 1] ? a1 : q.unit0[fi + 1]) - q.unit0[fi]);
        const int n = F.n, he = F.he, ho = F.ho, nlines = F.nlines, lines = F.nmodes * F.nlines;
        const long long sk = F.sk, sl = F.sl, plane = F.plane_stride / 2;
        const bool fold = F.par == 1;
        // the field's operator and eigenvalues, once every warp is done with the last one's
        __syncthreads();
        const bool fresh = F.A != have;
        if (fresh && tid == 0) col_load(Op, F.A, (unsigned)(ColShape<MT>::op * sizeof(double)), &bar);
        have = F.A;
        if (DIV)
            for (int i = tid; i < n; i += 32 * W) Es[i] = F.E[i];
        ColIn in;
        in.first[0] = 0, in.step[0] = 1, in.count[0] = he;
        in.first[1] = fold ? n - 1 : he, in.step[1] = fold ? -1 : 1, in.count[1] = ho;
        in.fold = fold, in.es = sk;
        const double2 *src = reinterpret_cast<const double2 *>(F.src) + F.off * (sk + sl);
        auto line_of = [&](int l) -> const double2 * {
            if (l >= lines) return nullptr;
            const int pl = l / nlines;
            return src + pl * plane + (l - pl * nlines) * sl;
        };
        ColLane cl;
        if (u0 + warp < u1) cl.start(in, line_of((u0 + warp) * 4 + (g >> 1)), lane);
        const bool landed = !fresh || col_landed(&bar, loads);
        loads += fresh ? 1 : 0;
        if (__syncthreads_or(!landed)) {
            if (tid == 0) atomicExch(err, 1);
            if (fresh) col_landed(&bar, loads - 1);   // no copy may land in a CTA that is gone
            return;
        }
        double2 *dst = reinterpret_cast<double2 *>(F.dst) + F.off * (sk + sl);
#pragma unroll 1
        for (int u = u0 + warp; u < u1; u += W) {
            double acc[2][MT][4];
            // this thread's line: columns (2t, 2t+1) are its (re, im)
            const int lt = u * 4 + t;
            const bool lok = lt < lines;
            const int pl = lok ? lt / nlines : 0, l = lok ? lt - pl * nlines : 0;
            const double lam = p.lam[F.plane0 + pl];
            const double el = DIV ? F.El[l] - lam : 0.0;
            col_multiply<MT, 512 * MT, 256 * MT>(acc, Op, cl, in, lane, [](int, const double (&)[4], const double (&)[4]) {});
            // the next unit's first K step while this one is written
            if (u + W < u1) cl.start(in, line_of((u + W) * 4 + (g >> 1)), lane);
            double2 *out = dst + pl * plane + l * sl;
            const bool im0 = p.zero_im_mode0 && F.mode0 && pl == 0;
            const bool singular = F.sing_io >= 0 && fabs(lam) <= 1.0e-10 && l == F.sing_l;
#pragma unroll
            for (int m1 = 0; m1 < MT; m1 += GM) {
                double2 w[2][2 * GM];      // [even / odd or plain / mirrored][row]
                auto row = [&](int i) { return (m1 + (i >> 1)) * 16 + g + 8 * (i & 1); };
#pragma unroll
                for (int i = 0; i < 2 * GM; ++i) {
                    const double2 P = make_double2(acc[0][m1 + (i >> 1)][2 * (i & 1)], acc[0][m1 + (i >> 1)][2 * (i & 1) + 1]);
                    const double2 M = make_double2(acc[1][m1 + (i >> 1)][2 * (i & 1)], acc[1][m1 + (i >> 1)][2 * (i & 1) + 1]);
                    if (fold) {
                        w[0][i] = P;
                        w[1][i] = M;
                    } else {
                        // the middle point (he > ho) has no odd part
                        const bool pair = row(i) < ho;
                        w[0][i] = pair ? make_double2(P.x + M.x, P.y + M.y) : P;
                        w[1][i] = make_double2(P.x - M.x, P.y - M.y);
                    }
                }
                if (DIV) {
                    double den[2][2 * GM], rec[2][2 * GM];
                    bool good = true;
#pragma unroll
                    for (int pm = 0; pm < 2; ++pm)
#pragma unroll
                        for (int i = 0; i < 2 * GM; ++i) {
                            den[pm][i] = row(i) < (pm ? ho : he) ? Es[pm ? he + row(i) : row(i)] + el : 1.0;
                            rec[pm][i] = col_recip(den[pm][i], good);
                        }
                    if (!__all_sync(0xffffffffu, good)) {
#pragma unroll
                        for (int pm = 0; pm < 2; ++pm)
#pragma unroll
                            for (int i = 0; i < 2 * GM; ++i) rec[pm][i] = col_reciprocal(den[pm][i]);
                    }
#pragma unroll
                    for (int pm = 0; pm < 2; ++pm)
#pragma unroll
                        for (int i = 0; i < 2 * GM; ++i) {
                            const bool pin = singular && (pm ? he + row(i) : row(i)) == F.sing_io;
                            const double r = rec[pm][i];
                            w[pm][i] = pin ? make_double2(0.0, 0.0) : make_double2(w[pm][i].x * r, w[pm][i].y * r);
                        }
                }
#pragma unroll
                for (int pm = 0; pm < 2; ++pm)
#pragma unroll
                    for (int i = 0; i < 2 * GM; ++i) {
                        const int r = row(i), o = pm == 0 ? r : (fold ? he + r : n - 1 - r);
                        if (im0) w[pm][i].y = 0.0;
                        if (lok && r < (pm ? ho : he)) out[o * sk] = w[pm][i];
                    }
            }
        }
    }
}

// The wait of the kernel above on a barrier that nothing completes.
__global__ void k_wait_selftest(unsigned limit, int *err)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;\n" ::"r"(col_smem(&bar)));
    __syncthreads();
    const bool ok = col_landed(&bar, 0, limit);
    if (!__all_sync(0xffffffffu, ok) && threadIdx.x == 0) atomicExch(err, 3);
}

cudaError_t wait_selftest(ductgpu_ctx ctx, unsigned polls)
{
    LaunchScope ls(ctx, DUCTGPU_K_OTHER);
    k_wait_selftest<<<1, 32, 0, ctx->stream>>>(polls, ctx->dev_err);
    return cudaGetLastError();
}

// The reciprocals of the passes: y[0] with the fallback, y[1] whether x is in the
// range that needs none, y[2] the division.
__global__ void k_recip_selftest(const double *x, double *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool ok = true;
    col_recip(x[i], ok);
    y[i] = col_reciprocal(x[i]);
    y[n + i] = ok ? 1.0 : 0.0;
    y[2 * (long long)n + i] = 1.0 / x[i];
}

cudaError_t recip_selftest(ductgpu_ctx ctx, const double *x, double *y, int n)
{
    LaunchScope ls(ctx, DUCTGPU_K_OTHER);
    k_recip_selftest<<<(n + 255) / 256, 256, 0, ctx->stream>>>(x, y, n);
    return cudaGetLastError();
}

template <int MT, bool DIV> static cudaError_t launch_cols(ductgpu_ctx ctx, const PassParams &pp)
{
    ColsParams q;
    q.p = pp;
    long long units = 0;
    for (int i = 0; i < pp.nf; ++i) {
        q.unit0[i] = units;
        units += ((long long)pp.f[i].nmodes * pp.f[i].nlines + 3) / 4;
    }
    q.unit0[pp.nf] = units;
    constexpr int W = kPassWarps<MT>;
    const size_t smem = (ColShape<MT>::op + (DIV ? 32 * MT : 0)) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_pass_cols<MT, DIV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = units < ctx->num_sms ? (int)units : ctx->num_sms;
    LaunchScope ls(ctx, DUCTGPU_K_PASS_FP64);
    k_pass_cols<MT, DIV><<<grid, 32 * W, smem, ctx->stream>>>(q, ctx->dev_err);
    return cudaGetLastError();
}

cudaError_t fp64_pass_cols(ductgpu_ctx ctx, const PassParams &pp, int hpad)
{
    if (pp.divide)
        return hpad == 32 ? launch_cols<2, true>(ctx, pp) : hpad == 64 ? launch_cols<4, true>(ctx, pp) : launch_cols<6, true>(ctx, pp);
    return hpad == 32 ? launch_cols<2, false>(ctx, pp) : hpad == 64 ? launch_cols<4, false>(ctx, pp) : launch_cols<6, false>(ctx, pp);
}

}  // namespace duct
