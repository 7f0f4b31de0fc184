// mode_lines.cu -- products along the lines of a field whose operator splits by
// the parity of the mode index, on the resident-operator core of cols.cuh
// (k_mode_lines).  With nn = 2 ho + 1, N = nn - 1:
//   forward DCT-I  c_{2r} = sum_{j<ho} E(r,j) (x_j + x_{N-j}) + E(r,ho) x_ho,  r <= ho
//                  c_{2r+1} = sum_{j<ho} O(r,j) (x_j - x_{N-j}),               r < ho
//   inverse DCT-I  x_j, x_{N-j} = P_j +- M_j with P_j = sum_{r<ho} E'(j,r) c_{2r} +
//                  E'(j,ho) c_N, M_j = sum_{r<ho} O'(j,r) c_{2r+1}, and x_ho = P_ho
//   mode operator  d_{2r} = sum_{q<=ho} A(2r,2q) c_{2q}, d_{2r+1} the same of the odd
//                  modes (Chebyshev to Legendre and back)
// so the forward transform folds its loads, the inverse unfolds its stores,
// and modes are read and written two apart.  A warp's unit is 4 whole lines,
// read before they are written: a field may be transformed in place.
//
// What bounds it: memory (one read and one write) up to about 97 points, the
// FP64 tensor pipe above, 2 (ho^2) real products a column; beside the half-length
// FFT, which is bound by its instructions, it pays up to 109 points.  FFT forms / this, us, 85 modes,
// along y: 65 10.8 / 7.5, 97 16.8 / 12.2, 109 (no half-length plan) 35.2 / 17.8,
// 129 21.0 / 24.7 (z 24.7 / 22.6), 145 29.1 / 31.3, 163 (no plan) 69 / 42, 193 41.6 /
// 52.5; 24 modes: 97 9.5 / 7.0, 129 10.6 / 10.7; 5 modes: 97 8.6 / 6.6, 129 7.5 / 8.6.
#include <math.h>

#include <vector>

#include "cols.cuh"
#include "internal.h"

namespace duct {

enum { kForward, kInverse, kModes };

// ---------------------------------------------------------------------------
struct ModeLines {
    const double2 *src;
    double2 *dst;
    const double *op;
    long long ms;              // complex strides: mode, line, element
    long long ls, es;
    int lpm, lines, units, nn, ho;
};

template <int MT, int KIND>
__global__ void __launch_bounds__(32 * ColShape<MT>::W, 1) k_mode_lines(const __grid_constant__ ModeLines q, int *err)
{
    constexpr int HR = 16 * MT, W = ColShape<MT>::W;
    extern __shared__ __align__(128) double Op[];   // E, O, then E(r, ho), E(ho, j), unused, E(ho, ho)
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nn = q.nn, ho = q.ho, N = nn - 1;
    const long long es = q.es;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tfence.mbarrier_init.release.cluster;\n" ::"r"(col_smem(&bar)));
        col_load(Op, q.op, (unsigned)(dl_chunk(HR) * sizeof(double)), &bar);
    }
    __syncthreads();
    const int u0 = (int)((long long)q.units * blockIdx.x / gridDim.x), u1 = (int)((long long)q.units * (blockIdx.x + 1) / gridDim.x);
    ColIn in;
    constexpr bool MODES = KIND != kForward;      // the input is a line of modes
    in.first[0] = 0, in.step[0] = MODES ? 2 : 1;
    in.first[1] = MODES ? 1 : N, in.step[1] = MODES ? 2 : -1;
    in.count[0] = in.count[1] = ho;
    in.fold = !MODES, in.es = es;
    auto line_of = [&](int l) -> const double2 * {
        if (l >= q.lines) return nullptr;
        const int mode = l / q.lpm;
        return q.src + mode * q.ms + (l - mode * q.lpm) * q.ls;
    };
    auto out_of = [&](int l) { return l < q.lines ? q.dst + (line_of(l) - q.src) : nullptr; };
    ColLane cl;
    if (u0 + warp < u1) cl.start(in, line_of((u0 + warp) * 4 + (g >> 1)), lane);
    if (__syncthreads_or(!col_landed(&bar, 0))) {
        if (tid == 0) atomicExch(err, 1);
        col_landed(&bar, 0);               // no copy may land in a CTA that is gone
        return;
    }
    const double *vecD = Op + 2 * (size_t)HR * HR, *row = vecD + HR, *dmid = row + 2 * HR;
#pragma unroll 1
    for (int u = u0 + warp; u < u1; u += W) {
        double2 *out_m = out_of(u * 4 + (g >> 1)), *out = out_of(u * 4 + t);
        const double xmid = cl.point(in, MODES ? N : ho);
        double acc[2][MT][4];
        double dot[4] = {0.0, 0.0, 0.0, 0.0};   // the last even row's dot product for column g
        col_multiply<MT, 256 * MT, 256 * MT * MT>(acc, Op, cl, in, lane,
                                                  [&](int ks, const double (&bu)[4], const double (&)[4]) {
#pragma unroll
                                                      for (int v = 0; v < 4; ++v)
                                                          dot[v] = fma(row[ks * 16 + t + 4 * v], bu[v], dot[v]);
                                                  });
        // the next unit's first K step while this one is written
        if (u + W < u1) cl.start(in, line_of((u + W) * 4 + (g >> 1)), lane);
        const double xr = __shfl_sync(0xffffffffu, xmid, 8 * t), xi = __shfl_sync(0xffffffffu, xmid, 8 * t + 4);
        double part = (dot[0] + dot[1]) + (dot[2] + dot[3]);
        part += __shfl_xor_sync(0xffffffffu, part, 1);
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        part = fma(dmid[0], xmid, part);
        const double part_i = __shfl_down_sync(0xffffffffu, part, 4);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = mt * 16 + g + 8 * h;
                if (!out || r >= ho) continue;
                const double d = vecD[r];
                const double2 P = make_double2(fma(d, xr, acc[0][mt][2 * h]), fma(d, xi, acc[0][mt][2 * h + 1]));
                const double2 M = make_double2(acc[1][mt][2 * h], acc[1][mt][2 * h + 1]);
                if (KIND == kInverse) {
                    out[r * es] = make_double2(P.x + M.x, P.y + M.y);
                    out[(N - r) * es] = make_double2(P.x - M.x, P.y - M.y);
                } else {
                    out[2 * r * es] = P;
                    out[(2 * r + 1) * es] = M;
                }
            }
        if (t == 0 && !(g & 1) && out_m) out_m[(KIND == kInverse ? ho : N) * es] = make_double2(part, part_i);
    }
}

// DCT-I matrices of N + 1 points: c_k = w_k (x_0 + (-1)^k x_N + 2 sum x_j
// cos(pi j k / N)), w_k = 1/N, 1/(2N) at the ends; x_j = sum_k c_k cos(pi j k / N).
struct DctMatrix {
    int N;
    long double cosine(long j, long k) const
    {
        return cosl(3.141592653589793238462643383279502884L * (long double)(j * k % (2L * N)) / (long double)N);
    }
    double forward(int k, int j) const
    {
        return (double)(((k == 0 || k == N) ? 0.5L : 1.0L) / N * ((j == 0 || j == N) ? 1.0L : 2.0L) * cosine(j, k));
    }
    double inverse(int j, int k) const { return (double)cosine(j, k); }
};

// The transforms' operators for line length nn, built on first use: [forward
// chunk][inverse chunk], entries from the definition in long double.  First use
// may be inside a stream capture, which records none of this (a length has one
// form, captured or not), and there is a slot for every length that comes here:
// 2^a 3^b + 1 from 17 to 193 points, less 145 and 193.
static int dct_ops(ductgpu_ctx ctx, int nn, const double **ops)
{
    const int N = nn - 1, ho = N / 2, MT = (ho + 15) / 16, HR = 16 * MT;
    const size_t blk = (size_t)HR * HR, chunk = dl_chunk(HR);
    int slot = -1;
    for (int i = 0; i < ductgpu_ctx_s::kDctSlots; ++i)
        if (ctx->dct_nn[i] == nn) { *ops = ctx->dct_ops[i]; return DUCTGPU_OK; }
    for (int i = 0; i < ductgpu_ctx_s::kDctSlots && slot < 0; ++i)
        if (!ctx->dct_nn[i]) slot = i;
    if (slot < 0) return set_error(ctx, DUCTGPU_ESTATE, "transyz: more than %d line lengths", ductgpu_ctx_s::kDctSlots);
    const DctMatrix m{N};
    std::vector<double> packed(2 * chunk, 0.0);
    for (int d = 0; d < 2; ++d) {
        double *dst = packed.data() + d * chunk;
        for (size_t idx = 0; idx < blk; ++idx) {
            int r, c;
            pack_slot((int)idx, MT, r, c);
            if (r >= ho || c >= ho) continue;
            dst[idx] = d ? m.inverse(r, 2 * c) : m.forward(2 * r, c);
            dst[blk + idx] = d ? m.inverse(r, 2 * c + 1) : m.forward(2 * r + 1, c);
        }
        for (int r = 0; r < ho; ++r) {
            dst[2 * blk + r] = d ? m.inverse(r, N) : m.forward(2 * r, ho);
            dst[2 * blk + HR + r] = d ? m.inverse(ho, 2 * r) : m.forward(N, r);
        }
        dst[2 * blk + 3 * HR] = d ? m.inverse(ho, N) : m.forward(N, ho);
    }
    double *dev = nullptr;
    const size_t bytes = packed.size() * sizeof(double);
    cudaStream_t st = nullptr;                              // no part of any capture
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&dev, bytes);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dev, packed.data(), bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) cudaFree(dev);
    if (st) cudaStreamDestroy(st);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return check_cuda(ctx, e, "transform operators");
    ctx->dct_ops[slot] = dev;
    ctx->dct_nn[slot] = nn;
    *ops = dev;
    return DUCTGPU_OK;
}

template <int MT> static cudaError_t launch_lines(ductgpu_ctx ctx, const ModeLines &q, int kind)
{
    const size_t smem = dl_chunk(16 * MT) * sizeof(double);
    auto kernel = kind == kForward ? k_mode_lines<MT, kForward> : kind == kInverse ? k_mode_lines<MT, kInverse> : k_mode_lines<MT, kModes>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = q.units < ctx->num_sms ? q.units : ctx->num_sms;
    LaunchScope ls(ctx, kind == kModes ? DUCTGPU_K_PASS_FP64 : DUCTGPU_K_TRANSFORM);
    kernel<<<grid, 32 * ColShape<MT>::W, smem, ctx->stream>>>(q, ctx->dev_err);
    return cudaGetLastError();
}

static int mode_lines(ductgpu_ctx ctx, const double *src, double *dst, const double *op, int my, int mz, int nmodes, bool y, int kind)
{
    ModeLines q;
    q.src = reinterpret_cast<const double2 *>(src);
    q.dst = reinterpret_cast<double2 *>(dst);
    q.op = op;
    q.nn = y ? my : mz;
    q.ho = q.nn / 2;
    q.lpm = y ? mz : my;
    q.ms = (long long)my * mz;
    q.ls = y ? my : 1;
    q.es = y ? 1 : my;
    q.lines = q.lpm * nmodes;
    q.units = (q.lines + 3) / 4;
    if (q.units == 0) return DUCTGPU_OK;
    cudaError_t e;
    switch ((q.ho + 15) / 16) {
    case 1: e = launch_lines<1>(ctx, q, kind); break;
    case 2: e = launch_lines<2>(ctx, q, kind); break;
    case 3: e = launch_lines<3>(ctx, q, kind); break;
    case 4: e = launch_lines<4>(ctx, q, kind); break;
    case 5: e = launch_lines<5>(ctx, q, kind); break;
    default: e = launch_lines<6>(ctx, q, kind); break;
    }
    return check_cuda(ctx, e, "k_mode_lines");
}

// transyz along one direction; -1 where the FFT forms are to be used: line
// kernel 0 and lengths without this form
int dct_lines(ductgpu_ctx ctx, double *f, int my, int mz, int nmodes, char dir, int iopt)
{
    const int nn = (dir == 'y') ? my : mz;
    const long long lines = (long long)((dir == 'y') ? mz : my) * nmodes;
    const int MT = (nn / 2 + 15) / 16;
    if (!ctx->dlines || !(nn & 1) || nn < 17 || MT > 6 || lines > (1LL << 30)) return -1;
    // where a half-length FFT plan exists: up to three row tiles, and four along z
    // (the figures above; 129 points along z, FFT / this, us: 1 mode 7.2 / 8.3, 5 8.3 /
    // 8.3, 32 12.4 / 10.3, 64 20.9 / 16.5, 128 32.9 / 28.7; along y only 64 modes and
    // their like gain, 21.3 / 20.8).  The forms round differently, so the number of
    // lines has no say: a mode's transform must not depend on the batch it is in.
    if (lines_supported(nn) && MT > (dir == 'z' ? 4 : 3)) return -1;
    const double *ops = nullptr;
    int rc = dct_ops(ctx, nn, &ops);
    if (rc) return rc;
    const bool inverse = iopt >= 0;
    return mode_lines(ctx, f, f, ops + (inverse ? dl_chunk(16 * MT) : 0), my, mz, nmodes, dir == 'y',
                      inverse ? kInverse : kForward);
}

// One chunk of a mode operator A (nn x nn, column-major, modes of equal parity
// coupled only).
__global__ void k_pack_modes(const double *A, double *dst, int nn, int MT)
{
    const int HR = 16 * MT, ho = nn / 2, blk = HR * HR;
    auto at = [&](int r, int c) { return A[r + (long long)nn * c]; };
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < blk; i += gridDim.x * blockDim.x) {
        int r, c;
        pack_slot(i, MT, r, c);
        const bool in = r < ho && c < ho;
        dst[i] = in ? at(2 * r, 2 * c) : 0.0;
        dst[blk + i] = in ? at(2 * r + 1, 2 * c + 1) : 0.0;
        if (i < HR) {
            dst[2 * blk + i] = i < ho ? at(2 * i, nn - 1) : 0.0;
            dst[2 * blk + HR + i] = i < ho ? at(nn - 1, 2 * i) : 0.0;
            dst[2 * blk + 2 * HR + i] = 0.0;
            dst[2 * blk + 3 * HR + i] = i == 0 ? at(nn - 1, nn - 1) : 0.0;
        }
    }
}

size_t mode_operator_size(int nn) { return dl_chunk((nn / 2 + 15) / 16 * 16); }
int pack_mode_operator(ductgpu_ctx ctx, const double *A, double *dst, int nn)
{
    k_pack_modes<<<32, 256, 0, ctx->stream>>>(A, dst, nn, (nn / 2 + 15) / 16);
    ctx->launches += 1;
    return check_cuda(ctx, cudaGetLastError(), "k_pack_modes");
}
int mode_operator(ductgpu_ctx ctx, const double *src, double *dst, const double *op, int m, int nmodes, bool y)
{
    return mode_lines(ctx, src, dst, op, m, m, nmodes, y, kModes);
}

}  // namespace duct
