// solve_plane.cu -- the whole flip-symmetric solve of a plane with up to 63
// interior points a side on chip (k_plane): the four GEMM passes (solve_cols.cu;
// the operator algebra is described at fold_operators in setup.cu) without the
// three round trips of the field through memory and the launches between them.
//
// With both directions folded a real plane is four independent quadrants
// (y parity x z parity) from the first pass to the last.  A cluster of four
// CTAs takes a complex plane: a CTA keeps the modes of one y parity of one
// component (re or im), D[z][y'] with both z parities' blocks of rows, in
// shared memory (2 H x (H + 4) doubles) for all four passes:
//   load: the lines z are dealt to the CTAs of the cluster, read once, folded
//     along y, and each part stored into its CTA's D through distributed
//     shared memory;
//   pass 1 (y, P^-1): a warp owns 8 first-half columns z and their mirror
//     images, in place; the two accumulators are folded along z on the way
//     back to shared memory;
//   pass 2 (z, P^-1, divide) and pass 3 (z, P): a warp owns 16 columns y' of
//     one z parity, in place, without any barrier between warps;
//   pass 4 (y, P): the z unfold is two additions on the B fragments;
//   store: the lines are dealt out again, the parts of a point gathered and
//     unfolded along y, and the points and the zero walls written.
// The K order, the fragments and the places of the fold and unfold additions
// are those of the four-pass form: the results are equal bit for bit.
//
// What bounds it: small batches its own latency (load, four dependent
// products, store), large ones the FP64 tensor pipe (DMMA, mma.sync m16n8k16
// f64; tcgen05 has no f64 kind), 16 n (he^2 + ho^2) flops a complex plane;
// memory is touched once.  DMMA and the FP64 vector instructions share a
// pipe: where two warps of a scheduler multiply a third gets one vector
// instruction in per two MMAs (257 cycles each; 13 with one warp multiplying,
// 2.5 with none).  So the five CTAs that share an SM have one warp a scheduler,
// and one CTA's divide, fold, load and store run under the others' products.
// The operators stream through a ring of K-step slabs (bulk copies of the
// packed fragments; a slab is refilled by whichever warp is the last to leave
// it, so no warp ever waits for the others to free one).
//
// Graph replays, four passes and their wall kernel before / this: my = 65, 4
// planes 20.5 / 12.4 us, 84 with 21 of them Neumann (and its fill) 39 / 30.8,
// 256 65.6 / 52.7, 1280 223 / 179; my = 33, 17 planes 18.6 / 12.4.  The same kernel
// with larger half blocks measured slower than the passes: 64 rows (my = 129,
// 256 planes) 283 us against 238, 96 rows (my = 193, 255 planes) 649 against 567 --
// fewer CTAs an SM, whose divide and fold phases then stall each other --
// and 32 x 64 rows (my = 65, mz = 129) 110 against 121 alone but 443 against 395
// in a batch of four shapes, beside the others' passes.
#include <math.h>

#include "cols.cuh"
#include "internal.h"

namespace duct {

namespace {

// rows of a half block, CTAs of a cluster, operator slabs in the ring, CTAs an SM
constexpr int H = 32, CL = 4, SLOTS = 2, kPlaneCtas = 5;
constexpr int W = H / 8, THREADS = 32 * W, LD = H + 4;
constexpr int SLAB = 2 * H * 16;                 // one K step: the y block of a parity (half of it), or both z blocks
constexpr int CELLS = 2 * H / CL * H / THREADS;  // points of a CTA's share of the lines a thread
constexpr size_t kDataSize = (size_t)2 * H * LD, kRingSize = (size_t)SLOTS * SLAB;
constexpr size_t kPlaneSmem = (kDataSize + kRingSize + 3 * H) * sizeof(double) + SLOTS * (8 + 2 * 4) + 16;
static_assert(CELLS * THREADS * CL == 2 * H * H);

__device__ __forceinline__ void pl_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;\n" ::: "memory");
}

// the address in the shared memory of the cluster's CTA `rank` of what `p` is in this one's
__device__ __forceinline__ unsigned pl_map(const void *p, unsigned rank)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(col_smem(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ double pl_get(unsigned a)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void pl_put(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(a), "d"(v) : "memory");
}

// acc += A b: MT row tiles of operator fragments against NT column tiles
template <int MT, int NT>
__device__ __forceinline__ void pl_multiply(double (&acc)[MT][NT][4], const double *A, const double (&b)[NT][4], int lane)
{
    // fragments one row tile ahead, in two register sets
    const unsigned at = col_smem(A) + lane * 16;
    double a[2][8];
    auto fragment = [&](double (&f)[8], int mt) {
#pragma unroll
        for (int h = 0; h < 4; ++h)
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(f[2 * h]), "=d"(f[2 * h + 1]) : "r"(at + mt * 2048 + h * 512));
    };
    fragment(a[0], 0);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            col_mma(acc[mt][nt], a[mt & 1], b[nt]);
            if (nt == 0 && mt + 1 < MT) fragment(a[(mt + 1) & 1], mt + 1);
        }
    }
}

template <int MT, int NT> __device__ __forceinline__ void pl_clear(double (&acc)[MT][NT][4])
{
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[i][nt][v] = 0.0;
}

}  // namespace

__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(THREADS, kPlaneCtas)
    k_plane(const __grid_constant__ PlaneParams p, int *err)
{
    constexpr int MT = H / 16, STEPS = 4 * MT;  // K steps of 16 of a pass, of the four
    extern __shared__ __align__(128) double smem[];
    double *Dt = smem;                     // [2 H][LD]: rows z' (even block, odd block), columns y'
    double *ring = Dt + kDataSize;
    double *Ez = ring + kRingSize;           // [2 H] by row z', [H] by column y', less lambda
    double *Ey = Ez + 2 * H;
    uint64_t *full = reinterpret_cast<uint64_t *>(Ey + H);
    int *left = reinterpret_cast<int *>(full + SLOTS);     // warps that have left a slab, all uses
    volatile int *last = left + SLOTS;                     // the last use a slab was filled for
    volatile int *abort = last + SLOTS;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int rank = blockIdx.x & (CL - 1), c = rank & 1, comp = rank >> 1;   // place in the cluster: y parity, component
    const int item = blockIdx.x / CL;
    int fi = 0;
    while (fi + 1 < p.nf && item >= p.start[fi + 1]) ++fi;
    const PlaneField &F = p.f[fi];
    const int plane = item - p.start[fi];
    const int my = F.my, mz = F.mz, ny = my - 2, nz = mz - 2;
    const int ey = (ny + 1) / 2, oy = ny / 2, ez = (nz + 1) / 2, oz = nz / 2;   // even / odd extents
    const int hc = c ? oy : ey;            // this CTA's modes along y
    const long long stride = 2LL * my * mz;
    const double lam = p.lam[F.plane0 + plane];

    // K step s of the solve: P^-1 along y (block c), P^-1 along z (both
    // blocks), P along z, P along y (block c)
    auto issue = [&](int s) {
        const double *src;
        unsigned bytes = 2 * MT * 2048;
        if (s < MT) src = F.Qy + (size_t)(2 * s + c) * MT * 256, bytes = MT * 2048;
        else if (s < 2 * MT) src = F.Qz + (size_t)(s - MT) * 2 * MT * 256;
        else if (s < 3 * MT) src = F.Pz + (size_t)(s - 2 * MT) * 2 * MT * 256;
        else src = F.Py + (size_t)(2 * (s - 3 * MT) + c) * MT * 256, bytes = MT * 2048;
        const unsigned bar = col_smem(full + s % SLOTS);
        last[s % SLOTS] = s / SLOTS;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                         col_smem(ring + (size_t)(s % SLOTS) * SLAB)),
                     "l"(src), "r"(bytes), "r"(bar)
                     : "memory");
    };
    if (tid == 0) {
        for (int s = 0; s < SLOTS; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(col_smem(full + s)));
            left[s] = 0;
        }
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;\n" ::: "memory");
        for (int s = 0; s < SLOTS && s < STEPS; ++s) issue(s);
    }
    for (int i = tid; i < 2 * H; i += THREADS)
        Ez[i] = i < H ? (i < ez ? F.Ez[i] : 0.0) : (i - H < oz ? F.Ez[ez + i - H] : 0.0);
    for (int i = tid; i < H; i += THREADS) Ey[i] = (i < hc ? F.Ey[c ? ey + i : i] : 0.0) - lam;

    // Load: row R = (z half, r) of D holds line z = r or its mirror image
    // nz - 1 - r; this CTA reads the rows R = rank, rank + CL, ...  Of a point
    // k and its partner ny - 1 - k the sums go to the CTAs of even, the
    // differences to those of odd y parity; zero outside the half blocks.
    // All of a thread's loads are in flight at once.
    auto cell = [&](int e, int &R, int &k, int &z) {
        const int idx = tid + e * THREADS;
        R = (idx / H) * CL + rank;
        k = idx % H;
        const int r = R < H ? R : R - H;
        z = r < (R < H ? ez : oz) ? (R < H ? r : nz - 1 - r) : -1;
    };
    unsigned peer[CL];
#pragma unroll
    for (int i = 0; i < CL; ++i) peer[i] = pl_map(Dt, i);
    {
        const double *in = F.rhs + (long long)plane * stride + 2 * (my + 1);   // point (1, 1)
        double2 x[CELLS], y[CELLS];
#pragma unroll
        for (int e = 0; e < CELLS; ++e) {
            int R, k, z;
            cell(e, R, k, z);
            const double2 *line = reinterpret_cast<const double2 *>(in + 2LL * my * z);
            x[e] = y[e] = make_double2(0.0, 0.0);
            if (z >= 0 && k < ey) x[e] = line[k];
            if (z >= 0 && k < oy) y[e] = line[ny - 1 - k];
        }
        pl_cluster_sync();                 // every CTA of the cluster runs: its memory may be written
#pragma unroll
        for (int e = 0; e < CELLS; ++e) {
            int R, k, z;
            cell(e, R, k, z);
            const unsigned off = (unsigned)(R * LD + k) * 8;
            const bool pair = k < oy;
            pl_put(peer[0] + off, x[e].x + y[e].x);
            pl_put(peer[1] + off, pair ? x[e].x - y[e].x : 0.0);
            pl_put(peer[2] + off, x[e].y + y[e].y);
            pl_put(peer[3] + off, pair ? x[e].y - y[e].y : 0.0);
        }
    }
    pl_cluster_sync();                     // D is complete (and the barriers and eigenvalues are set)
    const int r0 = warp * 8 + g;      // this lane's first column z of passes 1 and 4

    bool ok = true;
    // the slab of K step s, once it has landed
    auto enter = [&](int s) -> const double * {
        uint64_t *bar = full + s % SLOTS;
        const unsigned parity = (s / SLOTS) & 1;
        for (unsigned it = 0; ok && !col_try(bar, parity); ++it)
            if (it >= kColSpin || ((it & 255) == 255 && *abort)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        return ring + (size_t)(s % SLOTS) * SLAB;
    };
    auto leave = [&](int s) {
        __syncwarp();
        if (lane == 0) {
            if (!ok) {
                *abort = 1;
                atomicExch(err, 1);
            } else if (s + SLOTS < STEPS) {
                __threadfence_block();
                if (atomicAdd(left + s % SLOTS, 1) == W * (s / SLOTS + 1) - 1) {
                    __threadfence_block();
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    issue(s + SLOTS);
                }
            }
        }
    };

    // ---- pass 1: y, P^-1 -------------------------------------------------
    {
        double acc[MT][2][4];
        pl_clear(acc);
#pragma unroll 1
        for (int ks = 0; ks < MT; ++ks) {
            double b[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int v = 0; v < 4; ++v) b[i][v] = Dt[(i * H + r0) * LD + ks * 16 + t + 4 * v];
            const double *A = enter(ks);
            if (ok) pl_multiply(acc, A, b, lane);
            leave(ks);
        }
        __syncwarp();                      // the columns are read: replaced in place
        // z fold: sums to row r, differences to row H + r (zero from oz on)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int r = warp * 8 + 2 * t + (v & 1), y = mt * 16 + g + 8 * (v >> 1);
                Dt[r * LD + y] = acc[mt][0][v] + acc[mt][1][v];
                Dt[(H + r) * LD + y] = r < oz ? acc[mt][0][v] - acc[mt][1][v] : 0.0;
            }
    }
    __syncthreads();

    // ---- passes 2 and 3: z, P^-1 with the divide, then P -------------------
    {
        const int zp = warp & 1, n0 = (warp >> 1) * 16;     // z parity, first of 16 columns y'
        double *Dz = Dt + zp * H * LD + n0;
        const int hz = zp ? oz : ez;
        const bool singular = F.sing_y >= 0 && fabs(lam) <= 1.0e-10;
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
            double acc[MT][2][4];
            pl_clear(acc);
#pragma unroll 1
            for (int ks = 0; ks < MT; ++ks) {
                double b[2][4];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int v = 0; v < 4; ++v) b[nt][v] = Dz[(ks * 16 + t + 4 * v) * LD + nt * 8 + g];
                const double *A = enter((1 + q) * MT + ks) + zp * MT * 256;
                if (ok) pl_multiply(acc, A, b, lane);
                leave((1 + q) * MT + ks);
            }
            // pass 2 over E_z + (E_y - lambda); the pinned pair of a singular plane is zero
            auto denominator = [&](int o, int l, bool &live) {
                live = o < hz && l < hc &&
                       !(singular && (zp ? ez + o : o) == F.sing_z && (c ? ey + l : l) == F.sing_y);
                return live ? Ez[zp * H + o] + Ey[l] : 1.0;
            };
            bool rest = false;             // divisors left to the division below
            if (q == 0) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            bool live, good = true;
                            const double den = denominator(mt * 16 + g + 8 * (v >> 1), n0 + nt * 8 + 2 * t + (v & 1), live);
                            const double rec = col_recip(den, good);
                            rest = rest || !good;
                            acc[mt][nt][v] = live ? (good ? acc[mt][nt][v] * rec : acc[mt][nt][v]) : 0.0;
                        }
            }
            __syncwarp();                  // the columns are read: replaced in place
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        *reinterpret_cast<double2 *>(Dz + (mt * 16 + g + 8 * h) * LD + nt * 8 + 2 * t) =
                            make_double2(acc[mt][nt][2 * h], acc[mt][nt][2 * h + 1]);
            __syncwarp();
            if (__any_sync(0xffffffffu, rest)) {
                for (int i = lane; i < H * 16; i += 32) {
                    const int o = i / 16, l = i % 16;
                    bool live, good = true;
                    const double den = denominator(o, n0 + l, live);
                    col_recip(den, good);
                    if (!good) Dz[o * LD + l] = Dz[o * LD + l] * (1.0 / den);
                }
                __syncwarp();
            }
        }
    }
    __syncthreads();

    // ---- pass 4: y, P, on columns z = r (even + odd) and mirrored (even - odd)
    {
        double acc[MT][2][4];
        pl_clear(acc);
#pragma unroll 1
        for (int ks = 0; ks < MT; ++ks) {
            double b[2][4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int k = ks * 16 + t + 4 * v;
                const double e = Dt[r0 * LD + k], o = Dt[(H + r0) * LD + k];
                b[0][v] = e + o;
                b[1][v] = e - o;
            }
            const double *A = enter(3 * MT + ks);
            if (ok) pl_multiply(acc, A, b, lane);
            leave(3 * MT + ks);
        }
        __syncwarp();
        // this CTA's part of column r to row r, of the mirrored column to row H + r
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int r = warp * 8 + 2 * t + (v & 1), y = mt * 16 + g + 8 * (v >> 1);
                Dt[r * LD + y] = acc[mt][0][v];
                Dt[(H + r) * LD + y] = acc[mt][1][v];
            }
    }
    pl_cluster_sync();

    // ---- store: the parts of this CTA's rows, unfolded along y ---------------
    const bool zero = F.mode0 && plane == 0;               // mode 0 is real
    if (ok) {
        double *out = F.sol + (long long)plane * stride + 2 * (my + 1);
        double v[CELLS][CL];
#pragma unroll
        for (int e = 0; e < CELLS; ++e) {
            int R, k, z;
            cell(e, R, k, z);
#pragma unroll
            for (int i = 0; i < CL; ++i) v[e][i] = pl_get(peer[i] + (unsigned)(R * LD + k) * 8);
        }
#pragma unroll
        for (int e = 0; e < CELLS; ++e) {
            int R, k, z;
            cell(e, R, k, z);
            if (z < 0 || k >= ey) continue;
            double2 *line = reinterpret_cast<double2 *>(out + 2LL * my * z);
            const bool pair = k < oy;      // else the middle point, which has no odd part
            const double ore = pair ? v[e][1] : 0.0, oim = pair ? v[e][3] : 0.0;
            line[k] = make_double2(v[e][0] + ore, zero ? 0.0 : v[e][2] + oim);
            if (pair) line[ny - 1 - k] = make_double2(v[e][0] - ore, zero ? 0.0 : v[e][2] - oim);
        }
    }
    // helm3d zeroes the Dirichlet walls of rhs in place and the solution
    // keeps them (src/helm3d.f90:48-60, src/solvediag.f90:131-135): the y walls
    // by one component's CTAs, the z walls by the other's
    if (F.walls) {
        double2 *rhs = reinterpret_cast<double2 *>(F.rhs + (long long)plane * stride);
        double2 *sol = reinterpret_cast<double2 *>(F.sol + (long long)plane * stride);
        for (int q = tid; q < (comp ? my : mz); q += THREADS) {
            const long long off = comp ? q + (c ? (long long)my * (mz - 1) : 0) : (c ? my - 1 : 0) + (long long)my * q;
            if (F.walls == 1) rhs[off] = make_double2(0.0, 0.0);
            sol[off] = make_double2(0.0, 0.0);
        }
    }
    pl_cluster_sync();                     // the others have read this CTA's part
    // after a failed wait: no copy may land in a CTA that is gone
    if (!ok)
        for (int s = 0; s < SLOTS; ++s)
            for (unsigned it = 0; it < kColSpin && !col_try(full + s, last[s] & 1); ++it) {}
}

bool plane_arrays_apart(const PlaneParams &p)
{
    // the clusters of a plane read and write it in their own time: a
    // solution array may be its own right-hand side (read in full before the
    // cluster's first store) but must not meet anything else of the call
    auto bytes = [&](int i) { return (size_t)p.f[i].nmodes * 2 * p.f[i].my * p.f[i].mz * sizeof(double); };
    auto meet = [&](const double *a, size_t na, const double *b, size_t nb) {
        return (uintptr_t)a < (uintptr_t)b + nb && (uintptr_t)b < (uintptr_t)a + na;
    };
    for (int i = 0; i < p.nf; ++i)
        for (int j = 0; j < p.nf; ++j) {
            if (!(i == j && p.f[i].sol == p.f[j].rhs) && meet(p.f[i].sol, bytes(i), p.f[j].rhs, bytes(j))) return false;
            if (i != j && meet(p.f[i].sol, bytes(i), p.f[j].sol, bytes(j))) return false;
            if (i != j && p.f[i].walls == 1 && meet(p.f[i].rhs, bytes(i), p.f[j].rhs, bytes(j))) return false;
        }
    return true;
}

// On chip a plane costs the same whatever its size, in the passes its lines
// count as they are: a call of more planes than the GPU has SMs goes to the
// passes when its sides have fewer than 55 interior points.  256 planes, graph
// replays of the solve on chip / in passes, us: my = 57 51.8 / 51.3, 49 51.7 /
// 49.3, 35 50.7 / 41.0.  Up to one plane an SM the four launches that go matter more than
// the products, wherever the solve is one of a chain: direct calls of 112 and 144
// planes of my = 33 25.6 / 31.8 and 27.7 / 31.8, of 17 23.9 / 31.8 and 27.5 / 31.8; a
// time step with 144-plane predictor solves (mgalx = 144, graph) at my = 17 367 / 388,
// 25 383 / 392, 33 389 / 407, 49 497 / 516.  (Replays of nothing but such a
// solve hide the launches behind each other: my = 33, 112 planes 22.5 / 20.5.)
bool plane_wanted(ductgpu_ctx ctx, const PlaneParams &p)
{
    int planes = 0, n = p.f[0].my - 2;
    for (int i = 0; i < p.nf; ++i) {
        planes += p.f[i].nmodes;
        for (int side : {p.f[i].my - 2, p.f[i].mz - 2}) {
            if (side > 2 * H - 1) return false;
            n = side < n ? side : n;
        }
    }
    return n >= 55 || planes <= ctx->num_sms;
}

int plane_solve(ductgpu_ctx ctx, PlaneParams &p)
{
    int planes = 0;
    for (int i = 0; i < p.nf; ++i) {
        p.start[i] = planes;
        planes += p.f[i].nmodes;
    }
    p.start[p.nf] = planes;
    DUCT_CUDA(ctx, cudaFuncSetAttribute(k_plane, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlaneSmem));
    {
        LaunchScope ls(ctx, DUCTGPU_K_PASS_FP64);
        k_plane<<<CL * planes, THREADS, kPlaneSmem, ctx->stream>>>(p, ctx->dev_err);
    }
    return check_cuda(ctx, cudaGetLastError(), "k_plane");
}

}  // namespace duct
