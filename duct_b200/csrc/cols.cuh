// cols.cuh -- products of a resident half-size operator pair with streamed
// lines on the FP64 tensor cores: the core of the flip-symmetric GEMM pass
// (solve_cols.cu), the derivative lines and the transforms (dlines.cu).
//
// One CTA per SM keeps the two blocks of an operator (2 HR x HR doubles, HR =
// 16 MT, DMMA A-fragment order) in shared memory.  Its warps share nothing
// else and never wait for each other: a warp takes a unit of 4 complex lines
// (8 real columns, one n-tile) at a time and keeps all 2 MT row tiles of P =
// A0 u and M = A1 v in its accumulators, so whatever joins the two halves of a
// line is done in its registers.  The lines come straight from global memory
// in B-fragment order, a K step ahead (each element is used by one lane, once;
// 4 lanes read 64 consecutive bytes along either direction).
//
// What shapes it: DMMA and the FP64 vector instructions share a pipe.  Where
// two warps of a scheduler multiply, a third gets one vector instruction in
// per two MMAs (257 cycles each, measured; 13 with one warp multiplying, 2.5
// with none), so an epilogue has as few of them as it can.  One warp
// multiplying alone leaves a quarter of the pipe to its stalls (measured, with
// its lines staged or not, the warps taking turns); three or four together
// hide each other's.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace duct {

// Three or four warps a scheduler, as their accumulators (16 MT registers a
// thread) allow; a kernel may take fewer.
template <int MT> struct ColShape {
    static constexpr int HR = 16 * MT, W = MT > 4 ? 12 : 16;
    static constexpr size_t op = 2 * (size_t)HR * HR;            // doubles of the operator pair
};

// Operators of lines of nn = 2 ho + 1 points (the derivative matrices' folded
// halves; the transforms' by parity of the mode), HR = 16 MT >= ho: two blocks
// A0 and A1 (HR x HR each, rows and columns >= ho zero, DMMA A-fragment order),
// then, HR doubles each, the vectors over the middle point or the last even
// mode: D(r, ho) (r < ho), A0(ho, c) and A1(ho, c) (c < ho), and D(ho, ho).
__host__ __device__ constexpr size_t dl_chunk(int HR) { return 2 * (size_t)HR * HR + 4 * (size_t)HR; }

constexpr unsigned kColSpin = 1u << 22;

__device__ __forceinline__ unsigned col_smem(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// D += A(16x16) B(16x8), m16n8k16 f64 fragments (PTX ISA):
// a[v] = A[g + 8(v&1)][t + 4(v>>1)], b[v] = B[t + 4v][g],
// d = {D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1]}.
__device__ __forceinline__ void col_mma(double (&d)[4], const double (&a)[8], const double (&b)[4])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
          "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// Thread 0: bytes of an operator from global to shared memory, completing on bar.
__device__ __forceinline__ void col_load(void *dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile("fence.proxy.async.shared::cta;\n\t"
                 "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t"
                 "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%2], [%3], %1, [%0];\n" ::"r"(
                     col_smem(bar)),
                 "r"(bytes), "r"(col_smem(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ bool col_try(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok) : "r"(col_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// bounded wait for the operator of load number `phase`
__device__ __forceinline__ bool col_landed(uint64_t *bar, unsigned phase, unsigned limit = kColSpin)
{
    bool ok = false;
    for (unsigned it = 0; !ok && it < limit; ++it) ok = col_try(bar, phase & 1);
    return ok;
}

// The two inputs of a product: element k of input h (h = 0, 1) is point
// first[h] + step[h] k of the line, k < count[h], zero beyond; fold: u = x0 +
// x1, v = x0 - x1, else u = x0, v = x1.  es: complex stride of the points.
struct ColIn {
    int first[2], step[2], count[2];
    bool fold;
    long long es;
};

// A lane's column (line g / 2 of the unit, its real or imaginary part) and the
// K step in flight.
struct ColLane {
    const double *col;
    bool ok;
    double raw[2][4];

    // line: the column's line, null beyond the field
    __device__ __forceinline__ void start(const ColIn &in, const double2 *line, int lane)
    {
        ok = line != nullptr;
        col = reinterpret_cast<const double *>(line) + ((lane >> 2) & 1);
        fetch(in, lane, 0);
    }
    __device__ __forceinline__ void fetch(const ColIn &in, int lane, int ks)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int k = ks * 16 + (lane & 3) + 4 * v;
                raw[h][v] = ok && k < in.count[h] ? col[2 * (in.first[h] + in.step[h] * k) * in.es] : 0.0;
            }
    }
    __device__ __forceinline__ double point(const ColIn &in, int i) const { return ok ? col[2 * i * in.es] : 0.0; }
};

// The products of one unit: acc[0] = A0 u, acc[1] = A1 v.  use(ks, u, v) sees
// every B fragment (rows ks 16 + t + 4 v, column g).  KSTEP, BLOCK: doubles
// from one K step's tiles to the next, and from A0's to A1's.
template <int MT, int KSTEP, int BLOCK, class Use>
__device__ __forceinline__ void col_multiply(double (&acc)[2][MT][4], const double *Op, ColLane &cl, const ColIn &in, int lane,
                                             Use use)
{
#pragma unroll
    for (int pm = 0; pm < 2; ++pm)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[pm][mt][v] = 0.0;
#pragma unroll 1
    for (int ks = 0; ks < MT; ++ks) {
        double b[2][4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            b[0][v] = in.fold ? cl.raw[0][v] + cl.raw[1][v] : cl.raw[0][v];
            b[1][v] = in.fold ? cl.raw[0][v] - cl.raw[1][v] : cl.raw[1][v];
        }
        if (ks + 1 < MT) cl.fetch(in, lane, ks + 1);
        use(ks, b[0], b[1]);
        const double2 *A = reinterpret_cast<const double2 *>(Op + (size_t)ks * KSTEP) + lane;
#pragma unroll
        for (int pm = 0; pm < 2; ++pm)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                double a[8];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const double2 v = A[pm * (BLOCK / 2) + mt * 128 + 32 * h];
                    a[2 * h] = v.x;
                    a[2 * h + 1] = v.y;
                }
                col_mma(acc[pm][mt], a, b[pm]);
            }
    }
}

// 1 / x by one step of Householder's method of order 2 for 1 / r - x (A. S.
// Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970; the
// third-order hyperpower iteration): r (1 + e + e^2), e = 1 - x r, with the
// hardware's 20-bit estimate as r.  The remainder e^3 leaves 2^-60 before the one
// rounding of the last step: 0.51 ulp (test_gpu_reciprocal.py), against 0.5 of a
// division.  No branch, so a thread's reciprocals overlap, and three FP64
// operations: each costs its share of the tensor pipe.  ok comes back false
// unless 2^-1000 <= |x| < 2^1001 (zero, infinity and NaN are outside), where the
// caller divides.  Every flip-symmetric pass takes its reciprocals here, so that
// they agree bit for bit.
__device__ __forceinline__ double col_recip(double x, bool &ok)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;\n" : "=d"(r) : "d"(x));
    ok = ok && ((__double2hiint(x) >> 20) & 0x7ff) - 23u < 2001u;
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
static __device__ __noinline__ double col_divide(double x) { return 1.0 / x; }
// one reciprocal, whatever x
__device__ __forceinline__ double col_reciprocal(double x)
{
    bool ok = true;
    const double r = col_recip(x, ok);
    return ok ? r : col_divide(x);
}

}  // namespace duct
