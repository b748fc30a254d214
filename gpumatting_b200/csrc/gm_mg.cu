// gm_mg.cu -- CG preconditioned with an aggregation multigrid V-cycle on the
// symmetric Levin store (GM_SOLVER_MG).
//
// The reference's unfinished direction for faster solves is a hierarchy of
// piecewise-constant aggregation operators (gridoperators.h:18-138: restriction
// matrices with unit entries, pixel -> label) over superpixels (SLIC.cpp:32;
// the call sits commented out at main.cu:201-218).  Here the aggregates are
// fixed 2x2 blocks, so every level keeps a banded stencil that streams like
// the fine one:
//
//   level 0      the store's iteration operator (12 upper planes w + the
//                diagonal d; FP16 / BF16 / FP32 planes);
//   level l+1    Galerkin P^T A_l P with P the 2x2 aggregation: 4 FP32 upper
//                coupling planes (E, SW, S, SE) + diagonal Gamma + sum of the
//                couplings leaving the aggregate;
//   coarsest     the first level with <= kCoarseMax cells, inverted once per
//                solve (FP64 Gauss-Jordan in shared memory).
//
// V-cycle on level l with right-hand side b: x1 = omega b / D,
// b_{l+1} = P^T (b - A x1), recurse, y = x1 + scale P x_{l+1},
// x = y + omega (b - A y) / D.  Each level above the dense one costs two streaming
// kernels ("down": smoothing + residual + restriction; "up": prolongation +
// smoothing), both the persistent TMA-ring stencil kernel mg_fine_kernel; x1
// is recomputed from b in "up" instead of stored.  From the first level of at
// most kDenseMax cells down, the cycle is one dense matrix, formed once per
// solve (mg_dense_build_kernel) and applied as a matrix-vector product
// (mg_dense_kernel).
//
// Outer loop: PCG with FP64 solution (plus an FP32 increment folded in after
// each replacement), FP32 vectors and FP64 scalars, on the FP16 planes where
// outer_low_for allows it and else on the true FP32 operator; the
// preconditioner reads the low-precision planes.  The true residual b - A x in FP64 arithmetic
// replaces the recurrence every `replace_every` iterations and decides
// convergence (the same reliable-update rule as the fused CG).
// All scalars stay on the device: every reduction adds per-CTA partials in a
// fixed order (so results are deterministic), p.q and r.z in the kernel that
// needs them, and the whole solve is ONE CUDA graph launch with two device-side conditional WHILE loops,
// over the residual replacements and, inside, over the iterations between
// them -- no host round trip per iteration.  Kernels are
// chained with programmatic dependent launch.  gm_levin_solve_mg_many runs
// many such solves on concurrent streams.
#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "gm_graph_cache.h"
#include "gm_internal.cuh"

namespace gm {
namespace mg {

constexpr int kCoarseMax = 128;   // cells of the directly solved level
// Smoother damping and coarse-correction scale.  A sweep on the GPU over
// omega in {0.7 .. 1.0} x scale in {1.5 .. 2.4} put (0.8, 1.5) among the
// fastest at 640x480, 1920x1080 and 4096^2 (eps 1e-7); omega = 1.0 stalls.
constexpr float kDefaultOmega = 0.8f;
constexpr float kDefaultScale = 1.5f;
constexpr int kMaxLevels = 24;
constexpr int kThreads = 256;     // 32 x 8
constexpr int kTX = 64;           // tile columns (2 per thread)
constexpr int kTY = 8;            // tile rows of apply / up / replacement tiles
constexpr int kHalo = 2;
constexpr int kPW = kTX + 16;     // plane tile width: tile + 8 columns each side (16-byte aligned loads)
constexpr int kVW = kTX + 2 * kHalo;
constexpr int kMaxParts = 4096;

// Stencils.  Fine: 12 upper planes, plane k couples (x, y) with
// (x + du, y + dv), du = ((k + 3) % 5) - 2, dv = (k + 3) / 5 (k = 0..11 is the
// store's k = 1..12).  Coarse: 4 upper planes E (1,0), SW (-1,1), S (0,1),
// SE (1,1).
struct FineSten {
    static constexpr int NP = 12;
    __host__ __device__ static constexpr int du(int k) { return ((k + 3) % 5) - 2; }
    __host__ __device__ static constexpr int dv(int k) { return (k + 3) / 5; }
};
struct CoarseSten {
    static constexpr int NP = 4;
    __host__ __device__ static constexpr int du(int k) { return k == 0 ? 1 : (k == 1 ? -1 : (k == 2 ? 0 : 1)); }
    __host__ __device__ static constexpr int dv(int k) { return k == 0 ? 0 : 1; }
};

// Device-resident solver state (scalars of the outer PCG).
//
// The sums r.z, p.q and r.r of an iteration are left as per-CTA partials by
// the kernel that forms them and added up by every CTA of the kernel that
// needs them, in index order (so all agree bit for bit), while its first
// loads are in flight; a last-CTA sum costs 2.5-4 us at the end of each of the
// three kernels instead.  A field is never written by a kernel whose other
// CTAs may still read it: the matrix product of iteration k reads rz[(k - 1) & 1]
// and writes rz[k & 1], the update reads iter and writes iter_next, the
// restriction takes iter_next over into iter.
struct State {
    double rz[2], rr, bn2, rr_true;
    int iter, iter_next, done, status, need_replace, replacements;
    int fold_at;     // iteration whose update folds the FP32 increment into x
    int restart_at;  // iteration whose search direction is z alone (beta = 0)
    unsigned ticket[2];
};
enum { T_RR = 0, T_TRUE = 1 };
// Partial sums: p.q of the matrix product, r.r of the update, the true r.r and
// b.b of the replacement, r.z of the level-0 prolongation.
enum { S_PQ = 0, S_RR = 1, S_TRUE = 2, S_RZ = 4 };

// One level's operator and vectors (l >= 1: FP32 planes of its own; level 0
// points into the store and the fine work vectors).
struct Lev {
    int W, H, P;          // cells, rows, pitch (elements)
    void* c;              // planes [NP][H][P] (level 0: the store's w, type T)
    size_t ps;            // plane stride (elements)
    float* D;             // diagonal [H][P]
    float* Di;            // 1 / D (0 where D = 0): the smoothers multiply
    float* gam;           // summed scribble weight (l >= 1)
    float* b;             // right-hand side of the V-cycle on this level
    float* x;             // V-cycle result on this level
    double* M;            // levels lt .. L: the V-cycle from this level down as a dense matrix [n][n]
};

struct Args {
    Lev lev[kMaxLevels];
    int L;                // index of the coarsest level
    int lt;               // the level whose V-cycle is applied as a dense matrix (1 <= lt <= L)
    int W, H, P;          // fine grid (== lev[0])
    const float* w32;     // true operator: FP32 planes, gamma and d32 = gamma + row sum
    size_t ps32;
    const float* gamma;
    const float* d32;
    const float* bvec;    // right-hand side [H][bpitch]
    int bpitch;
    const float* alpha_in;
    float* alpha_out;     // [H][W]
    double* x;            // FP64 solution [H][P]; the solution is x + xinc
    float* xinc;          // FP32 increment since the last replacement [H][P]
    float *r, *q, *p0, *p1;  // fine vectors [H][P]; z is lev[0].x
    double* parts;        // [5][kMaxParts], S_*
    int planes_first;     // plane_policy of the level-0 planes
    int n_pq, n_rr, n_rz; // partials per sum: the CTAs of the kernel that leaves them
    State* st;
    double rtol;
    int max_iters, replace_every;
    int outer_low;  // the level-0 SpMV streams the FP16 iteration planes, not w32
    int rows0;      // tile rows of the level-0 kernels on 2-byte planes
    float omega, scale;
    // conditional-node handles (0 = host-driven loop): the loop over iterations
    // up to the next residual replacement, and the loop over replacements
    unsigned long long cond, cond_outer;
};

// ---------------------------------------------------------------------------
// Tile loaders
// ---------------------------------------------------------------------------

template <class T> __device__ __forceinline__ float tof(T v) { return Cvt<T>::to_f(v); }

// Programmatic dependent launch: every kernel of the solve is launched with
// programmatic stream serialisation, waits for its predecessor's completion
// (and memory), and lets its successor start launching only then.  So when a
// kernel starts, all kernels before its predecessor are complete: ahead of the
// wait it may read what those wrote, and only that.  Their writes are in L2 by
// then (the predecessor's wait is for that too); what changes from iteration to
// iteration is read from there (__ldcg, TMA), because no wait of the reading
// kernel's own has dropped older lines from L1 yet.  What the set-up wrote is
// constant in the iterations, and plain loads do.  This hides the launch gap
// between the many short kernels of a V-cycle.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter()
{
    pdl_wait();
    pdl_trigger();
}

// Starts copying a plane tile: NP planes x ROWS rows (y0 - 2 .. y0 + ROWS - 3) x
// kPW columns starting at x0 - 8 (16-byte aligned: x0 is a multiple of 64 and P
// of 8).  Elements outside the W x H level read as zero (a partial copy fills
// with zeros).  All of a tile's copies are in flight together.
template <class T, int NP, int ROWS>
__device__ __forceinline__ void load_planes(T* sm, const T* g, size_t ps, int P, int W, int H, int x0, int y0)
{
    constexpr int EPV = 16 / sizeof(T);
    constexpr int VPR = kPW / EPV;
    constexpr int TOTAL = NP * ROWS * VPR;
#pragma unroll
    for (int j = 0; j < (TOTAL + kThreads - 1) / kThreads; ++j) {
        const int i = threadIdx.x + j * kThreads;
        const int v = i % VPR, r = (i / VPR) % ROWS, k = i / (VPR * ROWS);
        const int gx = x0 - 8 + v * EPV, gy = y0 - kHalo + r;
        const bool in = gy >= 0 && gy < H && gx >= 0 && gx < W;
        const int bytes = in ? min(EPV, W - gx) * (int)sizeof(T) : 0;
        if (i < TOTAL)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sm + (size_t)(i / VPR) * kPW + v * EPV)),
                         "l"(g + (in ? (size_t)k * ps + (size_t)gy * P + gx : 0)), "r"(bytes)
                         : "memory");
    }
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Deterministic grid reductions: each CTA publishes its partial sums, and
// either the last CTA to arrive adds them in index order (the sums that end a
// recurrence) or every CTA of the consuming kernel does (p.q, r.z: no ticket,
// and the sum is formed after a wait that the consumer makes anyway).
// ---------------------------------------------------------------------------
template <int NV>
__device__ __forceinline__ bool last_cta_total(double (&v)[NV], double* parts, unsigned* ticket)
{
    __shared__ double red[32 * NV + NV];
    __shared__ int s_last;
    block_sum<NV>(v, red);
    const unsigned G = gridDim.x;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) parts[(size_t)k * kMaxParts + blockIdx.x] = v[k];
        __threadfence();
        const unsigned t = atomicAdd(ticket, 1u);
        s_last = (t == G - 1);
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (wid < NV) {
        const double t = warp_sum_range(parts + (size_t)wid * kMaxParts, 0, (int)G);
        if (lane == 0) red[32 * NV + wid] = t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = red[32 * NV + k];
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// This CTA's share of sum `which`, for the consuming kernel.
__device__ __forceinline__ void publish(double v, const Args& a, int which)
{
    __shared__ double red[32];
    double t[1] = {v};
    block_sum<1>(t, red);
    if (threadIdx.x == 0) a.parts[(size_t)which * kMaxParts + blockIdx.x] = t[0];
}

// The iteration now complete (k of them) ends the recurrence: converged by its
// own residual, at the replacement period or at the limit.
__device__ __forceinline__ bool replacement_due(const Args& a, const State* st, int k, double rr)
{
    return (a.rtol > 0.0 && rr <= a.rtol * a.rtol * st->bn2) || (a.replace_every > 0 && k % a.replace_every == 0) ||
           k >= a.max_iters || !isfinite(rr);
}

// Whether the kernels of an iteration have nothing to do: the solve is over, or
// the residual replacement at the end of the unrolled loop body is due first.
__device__ __forceinline__ bool paused(const State* st) { return st->done || st->need_replace; }

__device__ __forceinline__ void set_loop(unsigned long long h, bool go)
{
    if (h) cudaGraphSetConditional((cudaGraphConditionalHandle)h, go ? 1u : 0u);
}

// The smoother steps written with 1 / D only.  With S = sum_j w_ij v_j, so
// that (A v)_i = D_i v_i - S_i, and x1 = omega b / D:
//   rho = b - A x1 = (1 - omega) b + S(x1)            (D > 0; rho = b + S if D = 0)
//   x = y + omega (b - A y) / D = (1 - omega) y + omega (b + S(y)) / D
__device__ __forceinline__ float rho_of(float b, float di, float om, float S)
{
    return (di > 0.f ? (1.f - om) * b : b) + S;
}
__device__ __forceinline__ float smooth_of(float y, float b, float di, float om, float S)
{
    return di > 0.f ? fmaf(om * di, b + S, (1.f - om) * y) : y;
}

// ---------------------------------------------------------------------------
// Outer PCG kernels (level 0)
// ---------------------------------------------------------------------------

// x += alpha p_new, r -= alpha q, r . r, with alpha = r.z / p.q from the matrix
// product's partials.  The last update of a loop pass (LAST) sums r . r itself
// and decides whether the loop goes on; after the others the restriction does.
// Four pixels per step (16-byte vectors; the pitch is a multiple of 8); lanes
// past W are written as zero and left out of the sum.
template <bool LAST>
__global__ void __launch_bounds__(kThreads) mg_update_kernel(Args a)
{
    // What kernels before the predecessor left (they are complete: the
    // predecessor started after them) is read ahead of the wait for it.
    State* st = a.st;
    const int W = a.W, H = a.H, P = a.P;
    __shared__ int s_it, s_fold;
    if (threadIdx.x == 0) {  // (one thread: every warp's request for the one line would queue up in L2)
        s_it = __ldcg(&st->iter);
        s_fold = __ldcg(&st->fold_at);
    }
    const int qpr = (W + 3) / 4;
    const size_t nq = (size_t)qpr * H, step = (size_t)gridDim.x * kThreads;
    struct Quad {
        size_t o;
        int x;
        float4 p, q, r, xi;
    };
    auto load_old = [&](Quad& d, size_t qi) {
        d.x = (int)(qi % qpr) * 4;
        d.o = (qi / qpr) * P + d.x;
        d.r = __ldcg(reinterpret_cast<const float4*>(a.r + d.o));
        d.xi = __ldcg(reinterpret_cast<const float4*>(a.xinc + d.o));
    };
    const float* pn = nullptr;
    auto load_new = [&](Quad& d) {
        d.p = *reinterpret_cast<const float4*>(pn + d.o);
        d.q = *reinterpret_cast<const float4*>(a.q + d.o);
    };
    size_t qi = (size_t)blockIdx.x * kThreads + threadIdx.x;
    Quad c, n;
    if (qi < nq) load_old(c, qi);
    __syncthreads();
    const int it = s_it;
    const bool fold = s_fold == it;  // a replacement ran: move the increment into x
    pn = (it & 1) ? a.p0 : a.p1;
    pdl_enter();
    if (qi < nq) load_new(c);
    const double rz = st->rz[it & 1];
    const double pq = warp_sum_range(a.parts + (size_t)S_PQ * kMaxParts, 0, a.n_pq);
    const bool stop = paused(st);  // (done is set below only when every thread returns)
    const bool bad = !(pq > 0.0) || !isfinite(pq) || !isfinite(rz);
    if (stop || bad) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (!stop) {
                st->status = GM_ERR_BREAKDOWN;
                st->done = 1;
            }
            if (LAST) set_loop(a.cond, false);
        }
        return;
    }
    const float alf = (float)(rz / pq);
    double acc = 0.0;
    for (; qi < nq; qi += step) {
        if (qi + step < nq) {
            load_old(n, qi + step);
            load_new(n);
        }
        const bool v1 = c.x + 1 < W, v2 = c.x + 2 < W, v3 = c.x + 3 < W;
        if (fold) {
            double2 x01 = *reinterpret_cast<const double2*>(a.x + c.o);
            double2 x23 = *reinterpret_cast<const double2*>(a.x + c.o + 2);
            x01.x += (double)c.xi.x;
            x01.y = v1 ? x01.y + (double)c.xi.y : 0.0;
            x23.x = v2 ? x23.x + (double)c.xi.z : 0.0;
            x23.y = v3 ? x23.y + (double)c.xi.w : 0.0;
            *reinterpret_cast<double2*>(a.x + c.o) = x01;
            *reinterpret_cast<double2*>(a.x + c.o + 2) = x23;
            c.xi = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        c.xi.x = fmaf(alf, c.p.x, c.xi.x);
        c.xi.y = v1 ? fmaf(alf, c.p.y, c.xi.y) : 0.f;
        c.xi.z = v2 ? fmaf(alf, c.p.z, c.xi.z) : 0.f;
        c.xi.w = v3 ? fmaf(alf, c.p.w, c.xi.w) : 0.f;
        c.r.x = fmaf(-alf, c.q.x, c.r.x);
        c.r.y = v1 ? fmaf(-alf, c.q.y, c.r.y) : 0.f;
        c.r.z = v2 ? fmaf(-alf, c.q.z, c.r.z) : 0.f;
        c.r.w = v3 ? fmaf(-alf, c.q.w, c.r.w) : 0.f;
        *reinterpret_cast<float4*>(a.xinc + c.o) = c.xi;
        *reinterpret_cast<float4*>(a.r + c.o) = c.r;
        acc += (double)c.r.x * c.r.x + (double)c.r.y * c.r.y + ((double)c.r.z * c.r.z + (double)c.r.w * c.r.w);
        c = n;
    }
    if (LAST) {
        double v[1] = {acc};
        if (last_cta_total<1>(v, a.parts + (size_t)S_RR * kMaxParts, &st->ticket[T_RR]) && threadIdx.x == 0) {
            const bool replace = replacement_due(a, st, it + 1, v[0]);
            st->iter = it + 1;
            st->rr = v[0];
            if (replace) st->need_replace = 1;
            set_loop(a.cond, !replace);
        }
    } else {
        publish(acc, a, S_RR);
        if (blockIdx.x == 0 && threadIdx.x == 0) st->iter_next = it + 1;
    }
}

// True residual r = b - A x with the FP32 planes in FP64 arithmetic (runs
// only when a replacement is due).  Four CTAs per SM hide one tile's loads
// behind the others' arithmetic, at the price of 32 spilled bytes a thread: 62 us
// at 1080p, 452 at 4096^2 (with 3 CTAs, or with gamma and b loaded where they
// are used, 73 and 560; 92 B per pixel take 29 and 235).  Also forms ||b||^2 on
// the first call.
__global__ void __launch_bounds__(kThreads, 4) mg_replace_kernel(Args a)
{
    pdl_enter();
    State* st = a.st;
    if (st->done || !st->need_replace) {
        if (st->done && blockIdx.x == 0 && threadIdx.x == 0) {
            set_loop(a.cond, false);
            set_loop(a.cond_outer, false);
        }
        return;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    float* pt = reinterpret_cast<float*>(smem);
    double* xt = reinterpret_cast<double*>(smem + sizeof(float) * FineSten::NP * (kTY + kHalo) * kPW);
    const int W = a.W, H = a.H, P = a.P;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int tiles_x = (W + kTX - 1) / kTX, tiles = tiles_x * ((H + kTY - 1) / kTY);
    double rr = 0.0, bb = 0.0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int x0 = (t % tiles_x) * kTX, y0 = (t / tiles_x) * kTY;
        __syncthreads();
        load_planes<float, FineSten::NP, kTY + kHalo>(pt, a.w32, a.ps32, P, W, H, x0, y0);
        constexpr int XT = (kTY + 2 * kHalo) * kVW, XI = (XT + kThreads - 1) / kThreads;
        double xv[XI];
#pragma unroll
        for (int j = 0; j < XI; ++j) {
            const int i = threadIdx.x + j * kThreads;
            const int gx = x0 - kHalo + i % kVW, gy = y0 - kHalo + i / kVW;
            const size_t o = (size_t)gy * P + gx;
            xv[j] = (i < XT && gx >= 0 && gx < W && gy >= 0 && gy < H) ? a.x[o] + (double)a.xinc[o] : 0.0;
        }
        // the pixels' own values, in flight with the rest
        float gv[2], bw[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int gx = x0 + tx + 32 * h, gy = y0 + ty;
            const bool in = gx < W && gy < H;
            gv[h] = in ? a.gamma[(size_t)gy * P + gx] : 0.f;
            bw[h] = in ? a.bvec[(size_t)gy * a.bpitch + gx] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < XI; ++j) {
            const int i = threadIdx.x + j * kThreads;
            if (i < XT) xt[i] = xv[j];
        }
        copies_done();
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int lx = tx + 32 * h, gx = x0 + lx, gy = y0 + ty;
            if (gx < W && gy < H) {
                const size_t o = (size_t)gy * P + gx;
                const int vc = (ty + kHalo) * kVW + lx + kHalo;
                const double xc = xt[vc];
                double y = (double)gv[h] * xc;
#pragma unroll
                for (int k = 0; k < FineSten::NP; ++k) {
                    const int du = FineSten::du(k), dv = FineSten::dv(k);
                    const double wu = pt[((size_t)k * (kTY + kHalo) + ty + kHalo) * kPW + lx + 8];
                    const double wl = pt[((size_t)k * (kTY + kHalo) + ty + kHalo - dv) * kPW + lx + 8 - du];
                    y += wu * (xc - xt[vc + dv * kVW + du]) + wl * (xc - xt[vc - dv * kVW - du]);
                }
                const double bv = bw[h];
                const double r = bv - y;
                a.r[o] = (float)r;
                rr += r * r;
                bb += bv * bv;
            }
        }
    }
    double v[2] = {rr, bb};
    if (last_cta_total<2>(v, a.parts + (size_t)S_TRUE * kMaxParts, &st->ticket[T_TRUE]) && threadIdx.x == 0) {
        if (st->replacements == 0) st->bn2 = v[1];
        st->replacements += 1;
        st->fold_at = st->iter;
        st->need_replace = 0;
        // A true residual well above the recurrence's (more than twice its
        // norm) means the FP32 recurrences drifted: from a zero guess the
        // first cycle can carry the whole solution in the FP32 increment.
        // The old direction is then conjugate to a residual that no longer
        // exists, and beta = true r.z / recurrence r.z would let it swamp
        // the new one (the iteration stalls), so the next direction restarts
        // from z.  Forward solves never open such a gap.
        st->restart_at = v[0] > 4.0 * st->rr ? st->iter : -1;
        st->rr_true = v[0];
        st->rr = v[0];
        const double bn2 = st->bn2;
        if (!(bn2 > 0.0)) {
            st->done = 1;          // b = 0: the solution is 0
            st->status = GM_OK;
        } else if (!isfinite(v[0])) {
            st->done = 1;
            st->status = GM_ERR_BREAKDOWN;
        } else if (a.rtol > 0.0 && v[0] <= a.rtol * a.rtol * bn2) {
            st->done = 1;
            st->status = GM_OK;
        } else if (st->iter >= a.max_iters) {
            st->done = 1;
            st->status = a.rtol > 0.0 ? GM_ERR_NOT_CONVERGED : GM_OK;
        }
        set_loop(a.cond, !st->done);
        set_loop(a.cond_outer, !st->done);
    }
}

// ---------------------------------------------------------------------------
// V-cycle kernels
// ---------------------------------------------------------------------------

// The V-cycle from level lt down is a linear map of at most kDenseMax cells, so
// it is formed once per solve as a dense FP64 matrix and applied as one
// matrix-vector product, spread over the GPU.  On level l, with S the
// couplings, R = (1 - omega) I + omega D^-1 S and T = R P, the smoothing
// steps and the coarse correction compose to
//     M_l = omega D^-1 + R omega D^-1 + scale T M_{l+1} T^T,
// from M_L, the coarsest inverse.  A row of T has four entries: a cell couples
// to its own aggregate and to the three on its side of it.
// Run level by level in one CTA these levels took 15-24 us of every
// iteration (17 block barriers, and 75 KB staged by one SM); the product takes
// 3-5, and forming the matrix 20-40 us per solve.  Per iteration: 46.0 -> 37.6
// us at 317 x 211, 58.2 -> 47.2 at 640 x 480, 117.4 -> 106.5 at 1080p.
struct TRow {
    double w[4];  // own aggregate, x side, y side, diagonal
    int I[4];
};

__device__ __forceinline__ TRow t_row(const Lev& F, const Lev& C, int i, double om)
{
    const int x = i % F.W, y = i / F.W;
    const float* c = static_cast<const float*>(F.c);
    const size_t o = (size_t)y * F.P + x;
    const int sx = (x & 1) ? 1 : -1, sy = (y & 1) ? 1 : -1;
    const int X = x >> 1, Y = y >> 1;
    double own = 0.0, wx = 0.0, wy = 0.0, wd = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            const int du = dir ? -CoarseSten::du(k) : CoarseSten::du(k), dv = dir ? -CoarseSten::dv(k) : CoarseSten::dv(k);
            const int xj = x + du, yj = y + dv;
            if (xj < 0 || xj >= F.W || yj < 0 || yj >= F.H) continue;
            const double w = c[(size_t)k * F.ps + (dir ? (size_t)yj * F.P + xj : o)];
            const bool ox = du == sx, oy = dv == sy;  // leaves the aggregate in x, in y
            if (ox && oy) wd += w;
            else if (ox) wx += w;
            else if (oy) wy += w;
            else own += w;
        }
    const double di = F.Di[o];
    TRow t;
    t.w[0] = di > 0.0 ? (1.0 - om) + om * di * own : 1.0;
    t.w[1] = om * di * wx;
    t.w[2] = om * di * wy;
    t.w[3] = om * di * wd;
    // a side outside the grid has no coupling; its index only has to be readable
    const int Xs = min(max(X + sx, 0), C.W - 1), Ys = min(max(Y + sy, 0), C.H - 1);
    t.I[0] = Y * C.W + X;
    t.I[1] = Y * C.W + Xs;
    t.I[2] = Ys * C.W + X;
    t.I[3] = Ys * C.W + Xs;
    return t;
}

// Cells of the largest dense level.  Us per iteration with 700 / 1300 / 2100:
// 42.1 / 37.6 / 39.2 at 317 x 211 (420 or 1080 cells), 50.7 / 47.2 / 52.6 at
// 640 x 480 (300 or 1200), 103.8 / 106.5 / 111.1 at 1080p (510, 510, 2040): one
// level less costs a row of 2 K doubles per warp, more than its two launches.
// One limit for all sizes, taken for the small ones, where it gains most; the
// figures are from before the levels above ran in pairs.
constexpr int kDenseMax = 1300;

// M_l from M_{l+1}.  A CTA forms the rows of 8 cells next to each other: their T
// rows reach 6 x 2 aggregates, whose rows of M_{l+1} it stages in shared
// memory; thread j applies T to those from the right (12 numbers), then to
// them from the left, for column j of the 8 rows.  (16 gathers per entry from
// L2 instead: 54 against 35 us cold for the two levels of 317 x 211.)
constexpr int kDenseRun = 8;
constexpr int kDenseParts = 4;  // CTAs per run: 256 columns each at a time
static int dense_build_smem(int nc) { return 2 * (kDenseRun / 2 + 2) * nc * (int)sizeof(double); }

__global__ void __launch_bounds__(kThreads) mg_dense_build_kernel(Args a, int l)
{
    pdl_enter();
    constexpr int NX = kDenseRun / 2 + 2;
    extern __shared__ __align__(16) unsigned char smem[];
    double* Ms = reinterpret_cast<double*>(smem);  // [2][NX][nc]
    __shared__ TRow rows[kDenseRun];
    const Lev& F = a.lev[l];
    const Lev& C = a.lev[l + 1];
    const int n = F.W * F.H, nc = C.W * C.H, runs = (F.W + kDenseRun - 1) / kDenseRun;
    const double om = (double)a.omega, sc = (double)a.scale;
    const float* c = static_cast<const float*>(F.c);
    for (int item = blockIdx.x; item < runs * F.H * kDenseParts; item += gridDim.x) {
        const int run = item / kDenseParts, part = item % kDenseParts;
        const int x0 = (run % runs) * kDenseRun, y = run / runs, X0 = x0 >> 1, Y = y >> 1;
        const int Ys = min(max(Y + ((y & 1) ? 1 : -1), 0), C.H - 1);
        const int cells = min(kDenseRun, F.W - x0);
        __syncthreads();
        for (int e = 0; e < 2 * NX; ++e) {
            const int X = min(max(X0 - 1 + e % NX, 0), C.W - 1);
            const double* src = C.M + (size_t)((e < NX ? Y : Ys) * C.W + X) * nc;
            for (int j = threadIdx.x; j < nc; j += kThreads) Ms[e * nc + j] = src[j];
        }
        if ((int)threadIdx.x < cells) rows[threadIdx.x] = t_row(F, C, y * F.W + x0 + threadIdx.x, om);
        __syncthreads();
        for (int j = part * kThreads + threadIdx.x; j < n; j += kDenseParts * kThreads) {
            const TRow tj = t_row(F, C, j, om);
            double u[2 * NX];
#pragma unroll
            for (int e = 0; e < 2 * NX; ++e) {
                const double* row = Ms + e * nc;
                u[e] = tj.w[0] * row[tj.I[0]] + tj.w[1] * row[tj.I[1]] + tj.w[2] * row[tj.I[2]] + tj.w[3] * row[tj.I[3]];
            }
            const int xj = j % F.W, yj = j / F.W, dv = yj - y;
            const size_t oj = (size_t)yj * F.P + xj;
            const double dj = F.Di[oj];
#pragma unroll
            for (int q = 0; q < kDenseRun; ++q) {
                if (q >= cells) break;
                const int own = 1 + q / 2, side = (q & 1) ? 2 + q / 2 : q / 2;  // x0 is even
                double v = sc * (rows[q].w[0] * u[own] + rows[q].w[1] * u[side] + rows[q].w[2] * u[NX + own] +
                                 rows[q].w[3] * u[NX + side]);
                const int xi = x0 + q, du = xj - xi;
                if (du == 0 && dv == 0) v += om * (2.0 - om) * dj;
                else if (du >= -1 && du <= 1 && dv >= -1 && dv <= 1) {
                    // the coupling is stored at the upper end of the pair: planes E, SW, S, SE
                    const bool up = dv > 0 || (dv == 0 && du > 0);
                    const int k = dv == 0 ? 0 : 2 + (up ? du : -du);
                    const size_t oi = (size_t)y * F.P + xi;
                    v += om * om * (double)c[(size_t)k * F.ps + (up ? oi : oj)] * (double)F.Di[oi] * dj;
                }
                F.M[(size_t)(y * F.W + xi) * n + j] = v;
            }
        }
    }
}

// x_lt = M_lt b_lt, one warp per row.  The rows are constant during a solve
// and were written before this kernel's predecessor started, so they are
// loaded into registers ahead of the wait for b_lt.
constexpr int kDenseLoads = (kDenseMax + 31) / 32;
__global__ void __launch_bounds__(kThreads) mg_dense_kernel(Args a)
{
    __shared__ float b[kDenseMax];
    const Lev& G = a.lev[a.lt];
    const int n = G.W * G.H, lane = threadIdx.x & 31, step = gridDim.x * (kThreads / 32);
    int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    double m[kDenseLoads];
    auto load_row = [&]() {
        const double* row = G.M + (size_t)min(i, n - 1) * n;
#pragma unroll
        for (int q = 0; q < kDenseLoads; ++q) m[q] = lane + 32 * q < n ? __ldg(row + lane + 32 * q) : 0.0;
    };
    load_row();
    constexpr int NB = (kDenseMax + kThreads - 1) / kThreads;
    const float* src[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        const int j = min((int)threadIdx.x + k * kThreads, n - 1);
        src[k] = G.b + (size_t)(j / G.W) * G.P + j % G.W;
    }
    pdl_enter();
    float bv[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) bv[k] = __ldcg(src[k]);
    const bool stop = paused(a.st);
#pragma unroll
    for (int k = 0; k < NB; ++k)
        if ((int)threadIdx.x + k * kThreads < n) b[threadIdx.x + k * kThreads] = bv[k];
    if (stop) return;
    __syncthreads();
    for (;;) {
        double s[2] = {0.0, 0.0};
#pragma unroll
        for (int q = 0; q < kDenseLoads; ++q)
            if (lane + 32 * q < n) s[q & 1] = fma(m[q], (double)b[lane + 32 * q], s[q & 1]);
        double t = s[0] + s[1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0 && i < n) G.x[(size_t)(i / G.W) * G.P + i % G.W] = (float)t;
        i += step;
        if (i >= n) break;
        load_row();
    }
}

// ---------------------------------------------------------------------------
// The kernels of level 0 and of the large coarse levels: persistent CTAs
// streaming 128-column tiles through a TMA ring of two stages (one where every
// tile has a CTA of its own; the pattern of the standalone SpMV).  One elected
// thread issues, per tile, a 3-D box {144, TH + 2, 12} of the affinity planes
// (8 columns each side so the box starts on a 16-byte boundary, 2 rows above
// for the mirrored couplings) and 2-D boxes {144, TH + 4} of the vectors the
// stencil input is made of; TMA's zero fill stands in for everything outside
// the image.  After a stage lands, the CTA forms the stencil input in a
// shared tile, then each thread takes two rows of a column pair with a 5 x 6
// window of it in registers.
//   FM_SPMV  input z + beta p_old, beta from the prolongation's r . z;
//            q = A p_new with the FP32 planes and d32 (FP16 planes and d when
//            Args::outer_low); writes p_new and q, sums p_new . q.
//   FM_DOWN  input x1 = omega b / d; rho = b - A x1, summed over 2 x 2 blocks
//            into the level-1 right-hand side.  On level 0 with `pending`: the
//            update before it left r . r as partials, so this kernel counts
//            the iteration and stops when a replacement is due.
//   FM_UP    input y = x1 + scale x_1[aggregate]; z = y + omega (b - A y) / d,
//            sums r . z.
// ---------------------------------------------------------------------------
enum { FM_SPMV = 0, FM_DOWN = 1, FM_UP = 2 };
constexpr int kFTW = 128;             // output columns per tile
constexpr int kFBW = kFTW + 16;       // box width
constexpr int kXBW = kFTW / 2 + 8;    // coarse box width (FM_UP)

// SPMV: m[0] w32 planes, m[1] z, m[2] p0, m[3] p1, m[4] d32 (tile rows only)
// DOWN: m[0] iteration planes, m[1] r, m[2] d
// UP:   m[0] iteration planes, m[1] r, m[2] d, m[3] level-1 x
struct TMaps {
    CUtensorMap m[5];
};

// Tile rows of the TMA kernels: 8 with 4-byte planes (two CTAs per SM fit); with
// the 2-byte planes of level 0, 16 (one CTA per SM, a smaller share of halo rows) or
// 8, chosen per solve by level0_rows.
constexpr int kRows = 8, kTallRows = 16;
__host__ __device__ constexpr int b128(int x) { return (x + 127) & ~127; }

template <int MODE, int ES, int NP, int ROWS>
struct FineLayout {
    static constexpr int TH = ROWS;
    static constexpr int THR = 32 * TH;  // threads: 64 column pairs x TH / 2 row pairs
    static constexpr int PB = NP * (TH + 2) * kFBW * ES;
    static constexpr int VB = (TH + 4) * kFBW * 4;
    static constexpr int XB = MODE == FM_UP ? (TH / 2 + 2) * kXBW * 4 : 0;
    static constexpr int DB = MODE == FM_SPMV ? TH * kFTW * 4 : 0;
    static constexpr int v0_off = b128(PB);
    static constexpr int v1_off = v0_off + b128(VB);
    static constexpr int x_off = v1_off + b128(VB);
    static constexpr int d_off = x_off + b128(XB);
    static constexpr int stage = d_off + b128(DB);
    // nst stages, the stencil input, the barriers; + room to align the base to 128 bytes
    static constexpr int total(int nst) { return nst * stage + b128(VB) + 64 + 128; }
    static constexpr uint32_t bytes = (uint32_t)(PB + 2 * VB + XB + DB);
};

// Element type of the planes a level-0 kernel streams: the iteration planes.
// The SpMV of a BF16 store reads the FP32 planes instead (a BF16 outer
// operator costs more iterations than its bytes save); so does an FP16
// store's when the tolerance is tight (Args::outer_low = 0), through the
// float instantiation.
template <int MODE, class T>
struct FinePlanes {
    using PT = typename std::conditional<MODE == FM_SPMV && !std::is_same<T, __half>::value, float, T>::type;
    static constexpr int ES = (int)sizeof(PT);
};

template <class T> __device__ __forceinline__ float2 ld2(const T* p);
template <> __device__ __forceinline__ float2 ld2<float>(const float* p) { return *reinterpret_cast<const float2*>(p); }
template <> __device__ __forceinline__ float2 ld2<__half>(const __half* p)
{
    return __half22float2(*reinterpret_cast<const __half2*>(p));
}
template <> __device__ __forceinline__ float2 ld2<__nv_bfloat16>(const __nv_bfloat16* p)
{
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}

// Adds expected TMA bytes to the current phase without arriving.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Waits for a TMA stage with a wall-clock limit (2 s); on expiry the solve
// ends with GM_ERR_TIMEOUT.
__device__ __forceinline__ bool stage_wait(uint64_t* bar, uint32_t parity, State* st)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    unsigned spins = 0;
    while (!mbar_try_wait_hint(bar, parity, 100000u)) {
        if ((++spins & 15u) == 0 && globaltimer_ns() - t0 > 2000000000ull) {
            atomicCAS(&st->status, (int)GM_OK, (int)GM_ERR_TIMEOUT);
            st->done = 1;
            return false;
        }
    }
    return true;
}

template <int MODE, class S, class T, int ROWS>
__global__ void __launch_bounds__(32 * ROWS, 1)
    mg_fine_kernel(const __grid_constant__ TMaps tm, Args a, int l, int nst, int pending)
{
    constexpr int ES = FinePlanes<MODE, T>::ES;
    using PT = typename FinePlanes<MODE, T>::PT;
    using LY = FineLayout<MODE, ES, S::NP, ROWS>;
    constexpr int TH = LY::TH, NT = LY::THR, RPT = TH / (NT / 64);
    static_assert(RPT == 2, "each thread covers one row pair");
    constexpr int PW = (TH + 2) * kFBW;  // elements per plane in the box
    // TMA destinations must be 128-byte aligned; the dynamic region follows
    // the reduction's static shared memory, so align its base by hand.
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    float* vt = reinterpret_cast<float*>(smem + nst * LY::stage);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + nst * LY::stage + b128(LY::VB));
    const Lev& F = a.lev[l];
    const int W = F.W, H = F.H, P = F.P, tid = threadIdx.x, G = gridDim.x;
    const int ntx = (W + kFTW - 1) / kFTW, ntiles = ntx * ((H + TH - 1) / TH);
    const int t0 = blockIdx.x;
    State* st = a.st;
    // (of FM_SPMV's predecessors only those long complete write iter; one thread
    // reads it, as every warp's request for the one line would queue up in L2)
    int it = MODE == FM_SPMV && tid == 0 ? __ldcg(&st->iter) : 0;
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue_planes = [&](int t, int s) {
        const int u0 = (t % ntx) * kFTW, v0 = (t / ntx) * TH;
        if (S::NP == 12)
            tma_load_3d_hint(smem + s * LY::stage, &tm.m[0], u0 - 8, v0 - 2, 0, &full[s], plane_policy(a.planes_first));
        else
            tma_load_3d(smem + s * LY::stage, &tm.m[0], u0 - 8, v0 - 2, 0, &full[s]);
    };
    // The planes are constant during a solve (written by the store's assembly
    // or the set-up kernels, which completed before this kernel's predecessor
    // began), so the first stages' plane boxes are requested before the
    // wait for the predecessor; the stage's arrival comes with the vectors.
    const int npre = (t0 < ntiles ? 1 : 0) + (nst > 1 && t0 + G < ntiles ? 1 : 0);
    if (tid == 0)
        for (int k = 0; k < npre; ++k) {
            mbar_expect_tx(&full[k], (uint32_t)LY::PB);
            issue_planes(t0 + k * G, k);
        }
    pdl_enter();
    const float om = a.omega, sc = a.scale;
    const CUtensorMap* mv1 = MODE == FM_SPMV && (it & 1) ? &tm.m[3] : &tm.m[2];  // (for thread 0)
    const Lev& C = a.lev[l + 1];
    auto issue_vectors = [&](int t, int s) {
        const int u0 = (t % ntx) * kFTW, v0 = (t / ntx) * TH;
        unsigned char* sp = smem + s * LY::stage;
        tma_load_2d(sp + LY::v0_off, &tm.m[1], u0 - 8, v0 - 2, &full[s]);
        tma_load_2d(sp + LY::v1_off, mv1, u0 - 8, v0 - 2, &full[s]);
        if (MODE == FM_UP) tma_load_2d(sp + LY::x_off, &tm.m[3], u0 / 2 - 4, v0 / 2 - 1, &full[s]);
        if (MODE == FM_SPMV) tma_load_2d(sp + LY::d_off, &tm.m[4], u0, v0, &full[s]);
    };
    auto issue = [&](int t, int s) {
        mbar_arrive_expect_tx(&full[s], LY::bytes);
        issue_planes(t, s);
        issue_vectors(t, s);
    };
    auto drain = [&]() {  // let the requested stages land
        for (int k = 0; k < npre; ++k) stage_wait(&full[k], 0u, st);
    };
    // The vectors are requested before it is known whether there is anything
    // to do, and the sums of the kernels before are added up while they are on
    // their way.
    if (tid == 0)
        for (int k = 0; k < npre; ++k) {
            mbar_arrive_expect_tx(&full[k], LY::bytes - (uint32_t)LY::PB);
            issue_vectors(t0 + k * G, k);
        }
    float beta = 0.f;
    const bool summing = MODE == FM_SPMV || (MODE == FM_DOWN && pending);
    __shared__ double s_sum;
    __shared__ int s_stop, s_it;
    if (tid == 0) s_it = it;
    if (summing && tid >= 32 && tid < 64) {
        const double t = MODE == FM_SPMV ? warp_sum_range(a.parts + (size_t)S_RZ * kMaxParts, 0, a.n_rz)
                                         : warp_sum_range(a.parts + (size_t)S_RR * kMaxParts, 0, a.n_rr);
        if (tid == 32) s_sum = t;
    }
    // One thread looks: the lead CTA of this kernel may set need_replace or done
    // while others start, and a CTA has to take one path.
    if (tid == 64) s_stop = paused(st);
    __syncthreads();
    if (s_stop) {
        drain();
        return;
    }
    it = s_it;
    const bool first = it == 0;
    float* pnew = (it & 1) ? a.p0 : a.p1;
    if (summing) {
        const double sum = s_sum;
        const bool lead = blockIdx.x == 0 && tid == 0;
        if (MODE == FM_SPMV) {
            if (!isfinite(sum)) {
                if (lead) {
                    st->status = GM_ERR_BREAKDOWN;
                    st->done = 1;
                }
                drain();
                return;
            }
            if (!first && st->restart_at != it) beta = (float)(sum / st->rz[(it & 1) ^ 1]);
            if (lead) st->rz[it & 1] = sum;
        } else {
            const int k = st->iter_next;
            const bool replace = replacement_due(a, st, k, sum);
            if (lead) {
                st->iter = k;
                st->rr = sum;
                if (replace) st->need_replace = 1;
            }
            if (replace) {
                drain();
                return;
            }
        }
    }
    const int cp = tid & 63, rg = tid >> 6;
    const int lu = 8 + 2 * cp;
    const int r0 = rg * RPT;
    double acc = 0.0;
    int s = 0;
    uint32_t phase = 0u;
    bool ok = true;
    for (int t = t0; t < ntiles; t += G) {
        if (!stage_wait(&full[s], (phase >> s) & 1u, st)) { ok = false; break; }
        phase ^= 1u << s;
        const unsigned char* sp = smem + s * LY::stage;
        const PT* wb = reinterpret_cast<const PT*>(sp);
        const float* v0b = reinterpret_cast<const float*>(sp + LY::v0_off);
        const float* v1b = reinterpret_cast<const float*>(sp + LY::v1_off);
        const int u0 = (t % ntx) * kFTW, v0 = (t / ntx) * TH;
        // stencil input tile
        for (int i = tid; i < (TH + 4) * kFBW; i += NT) {
            float v;
            if (MODE == FM_SPMV) {
                v = first ? v0b[i] : fmaf(beta, v1b[i], v0b[i]);
            } else {
                v = om * v0b[i] * v1b[i];  // x1 = omega b / d (v1 holds 1 / d)
                if (MODE == FM_UP) {
                    // 1/d is zero outside the image (zero fill) and on pixels
                    // with no coupling and no scribble: y = 0 there
                    const int row = i / kFBW, col = i - row * kFBW;
                    const float* xb = reinterpret_cast<const float*>(sp + LY::x_off);
                    v = v1b[i] > 0.f ? fmaf(sc, xb[(row >> 1) * kXBW + (col >> 1)], v) : 0.f;
                }
            }
            vt[i] = v;
        }
        __syncthreads();
        float xw[5][6];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float* xr = vt + (r0 + j) * kFBW + lu - 2;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float2 q = *reinterpret_cast<const float2*>(xr + 2 * c);
                xw[j + 1][2 * c] = q.x;
                xw[j + 1][2 * c + 1] = q.y;
            }
        }
        float cs = 0.f;  // FM_DOWN: 2 x 2 block sum
#pragma unroll
        for (int rr = 0; rr < RPT; ++rr) {
            const int r = r0 + rr;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < 6; ++c) xw[j][c] = xw[j + 1][c];
            {
                const float* xr = vt + (r + 4) * kFBW + lu - 2;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float2 q = *reinterpret_cast<const float2*>(xr + 2 * c);
                    xw[4][2 * c] = q.x;
                    xw[4][2 * c + 1] = q.y;
                }
            }
            const float xi0 = xw[2][2], xi1 = xw[2][3];
            // S = sum_j w_ij x_j, two chains per pixel
            float a0[2] = {0.f, 0.f}, a1[2] = {0.f, 0.f};
#pragma unroll
            for (int k = 0; k < S::NP; ++k) {
                const int dv = S::dv(k), du = S::du(k);
                const PT* pk = wb + k * PW;
                const float2 wo = ld2<PT>(pk + (r + 2) * kFBW + lu);
                const PT* pm = pk + (r + 2 - dv) * kFBW + lu - du;
                const float wm0 = tof(pm[0]), wm1 = tof(pm[1]);
                a0[k & 1] = fmaf(wo.x, xw[2 + dv][2 + du], a0[k & 1]);
                a1[k & 1] = fmaf(wo.y, xw[2 + dv][3 + du], a1[k & 1]);
                a0[k & 1] = fmaf(wm0, xw[2 - dv][2 - du], a0[k & 1]);
                a1[k & 1] = fmaf(wm1, xw[2 - dv][3 - du], a1[k & 1]);
            }
            const float S0 = a0[0] + a0[1], S1 = a1[0] + a1[1];
            const int u = u0 + 2 * cp, v = v0 + r;
            if (MODE == FM_SPMV) {
                const float2 dg = *reinterpret_cast<const float2*>(sp + LY::d_off + (size_t)(r * kFTW + 2 * cp) * 4);
                const float q0 = fmaf(dg.x, xi0, -S0), q1 = fmaf(dg.y, xi1, -S1);
                if (v < H) {
                    const size_t o = (size_t)v * P + u;
                    if (u + 1 < W) {
                        *reinterpret_cast<float2*>(pnew + o) = make_float2(xi0, xi1);
                        *reinterpret_cast<float2*>(a.q + o) = make_float2(q0, q1);
                        acc += (double)xi0 * q0 + (double)xi1 * q1;
                    } else if (u < W) {
                        pnew[o] = xi0;
                        a.q[o] = q0;
                        acc += (double)xi0 * q0;
                    }
                }
            } else {
                const float2 bb = *reinterpret_cast<const float2*>(v0b + (r + 2) * kFBW + lu);
                const float2 dd = *reinterpret_cast<const float2*>(v1b + (r + 2) * kFBW + lu);  // 1 / d
                if (MODE == FM_DOWN) {
                    // rho = b - A x1; zero outside the image (zero fill)
                    cs += rho_of(bb.x, dd.x, om, S0) + rho_of(bb.y, dd.y, om, S1);
                    if (rr & 1) {
                        const int X = (u0 >> 1) + cp, Y = v >> 1;
                        if (X < C.W && Y < C.H) C.b[(size_t)Y * C.P + X] = cs;
                        cs = 0.f;
                    }
                } else {
                    const float z0 = smooth_of(xi0, bb.x, dd.x, om, S0);
                    const float z1 = smooth_of(xi1, bb.y, dd.y, om, S1);
                    if (v < H) {
                        float* zr = F.x + (size_t)v * P + u;
                        if (u + 1 < W) {
                            *reinterpret_cast<float2*>(zr) = make_float2(z0, z1);
                            acc += (double)bb.x * z0 + (double)bb.y * z1;
                        } else if (u < W) {
                            *zr = z0;
                            acc += (double)bb.x * z0;
                        }
                    }
                }
            }
        }
        __syncthreads();  // every thread is done with stage s and the input tile
        if (tid == 0 && t + nst * G < ntiles) issue(t + nst * G, s);
        s ^= nst - 1;
    }
    if (!ok) return;
    static_assert(NT <= 1024, "");
    if (MODE == FM_SPMV) publish(acc, a, S_PQ);
    else if (MODE == FM_UP && l == 0) publish(acc, a, S_RZ);
}

// ---------------------------------------------------------------------------
// Two coarse levels in one kernel.  A restriction or prolongation of a small
// level is a chain of latencies (launch, loads, two barriers, stores: 2-2.5 us
// for a few thousand cells), so two of them run as one: a CTA takes 32 x 8
// cells of the middle level l + 1 (64 x 16 of level l) and repeats what its
// neighbours compute one cell beyond its edge.  The operators and whatever
// older kernels left are staged ahead of the wait.  Every value is formed by
// the operations of the single-level kernels in their order, so results are
// the same bits.  A pair of restrictions takes 2.0-2.2 us instead of 3.9-4.3, a
// pair of prolongations 1.7-2.5 instead of 4.7-5.2; per iteration 24.7 -> 20.6
// us at 317 x 211, 37.4 -> 32.2 at 640 x 480, 88.3 -> 80.9 at 1080p.
// ---------------------------------------------------------------------------
constexpr int kPW1 = 32, kPH1 = 8;  // middle-level cells of a tile
constexpr int kPairThreads = 512;

// Starts copying RW x RH cells of a level from (x0, y0), zero outside it, to
// shared memory (4-byte asynchronous copies, all in flight together).
template <int RW, int RH>
__device__ __forceinline__ void stage(float* dst, const float* g, int P, int W, int H, int x0, int y0)
{
#pragma unroll
    for (int j = 0; j < (RW * RH + kPairThreads - 1) / kPairThreads; ++j) {
        const int i = threadIdx.x + j * kPairThreads, x = x0 + i % RW, y = y0 + i / RW;
        const bool in = x >= 0 && x < W && y >= 0 && y < H;
        if (i < RW * RH)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst + i)),
                         "l"(g + (in ? (size_t)y * P + x : 0)), "r"(in ? 4 : 0)
                         : "memory");
    }
}

// S = sum_j w_ij v_j at index i of rows of RW cells; the planes are RC cells apart.
template <int RW, int RC>
__device__ __forceinline__ float pair_sum(const float* c, const float* v, int i)
{
    float s[2] = {0.f, 0.f};
#pragma unroll
    for (int k = 0; k < CoarseSten::NP; ++k) {
        const int o = CoarseSten::dv(k) * RW + CoarseSten::du(k);
        s[k & 1] = fmaf(c[k * RC + i], v[i + o], s[k & 1]);
        s[k & 1] = fmaf(c[k * RC + i - o], v[i - o], s[k & 1]);
    }
    return s[0] + s[1];
}

// b_{l+1} and b_{l+2} from b_l.
__global__ void __launch_bounds__(kPairThreads) mg_pair_down_kernel(Args a, int l)
{
    constexpr int MW = kPW1 + 2, MH = kPH1 + 2;        // middle cells with their halo
    constexpr int FW = 2 * MW + 2, FH = 2 * MH + 2;    // level-l cells those need
    constexpr int NF = (FW * FH + kPairThreads - 1) / kPairThreads, NM = (MW * MH + kPairThreads - 1) / kPairThreads;
    __shared__ float cf[4 * (FH - 1) * FW], x1[FH * FW], rb[FH * FW];
    __shared__ float cm[4 * (MH - 1) * MW], xm[MH * MW], rm[MH * MW], rho[kPH1 * kPW1];
    const Lev& F = a.lev[l];
    const Lev& G = a.lev[l + 1];
    const Lev& C = a.lev[l + 2];
    const float om = a.omega;
    const int tx = (G.W + kPW1 - 1) / kPW1, tiles = tx * ((G.H + kPH1 - 1) / kPH1), tid = threadIdx.x;
    bool waited = false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int mx0 = (t % tx) * kPW1, my0 = (t / tx) * kPH1;
        const int fx0 = 2 * mx0 - 3, fy0 = 2 * my0 - 3;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            stage<FW, FH - 1>(cf + k * (FH - 1) * FW, static_cast<const float*>(F.c) + k * F.ps, F.P, F.W, F.H, fx0, fy0);
            stage<MW, MH - 1>(cm + k * (MH - 1) * MW, static_cast<const float*>(G.c) + k * G.ps, G.P, G.W, G.H, mx0 - 1,
                              my0 - 1);
        }
        float df[NF], dm[NM];
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int i = tid + j * kPairThreads, x = fx0 + i % FW, y = fy0 + i / FW;
            df[j] = i < FW * FH && x >= 0 && x < F.W && y >= 0 && y < F.H ? F.Di[(size_t)y * F.P + x] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < NM; ++j) {
            const int i = tid + j * kPairThreads, x = mx0 - 1 + i % MW, y = my0 - 1 + i / MW;
            dm[j] = i < MW * MH && x >= 0 && x < G.W && y >= 0 && y < G.H ? G.Di[(size_t)y * G.P + x] : 0.f;
        }
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        float bf[NF];
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int i = tid + j * kPairThreads, x = fx0 + i % FW, y = fy0 + i / FW;
            bf[j] = i < FW * FH && x >= 0 && x < F.W && y >= 0 && y < F.H ? __ldcg(F.b + (size_t)y * F.P + x) : 0.f;
        }
        if (paused(a.st)) {
            copies_done();
            return;
        }
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int i = tid + j * kPairThreads;
            if (i < FW * FH) {
                x1[i] = om * bf[j] * df[j];
                rb[i] = rho_of(bf[j], df[j], om, 0.f);
            }
        }
        copies_done();
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NM; ++j) {
            const int i = tid + j * kPairThreads, mx = i % MW, my = i / MW;
            if (i < MW * MH) {
                float sum = 0.f;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int f = (1 + 2 * my + q) * FW + 1 + 2 * mx;
                    sum += (rb[f] + pair_sum<FW, (FH - 1) * FW>(cf, x1, f)) +
                           (rb[f + 1] + pair_sum<FW, (FH - 1) * FW>(cf, x1, f + 1));
                }
                xm[i] = om * sum * dm[j];
                rm[i] = rho_of(sum, dm[j], om, 0.f);
                const int x = mx0 - 1 + mx, y = my0 - 1 + my;
                if (mx >= 1 && mx <= kPW1 && my >= 1 && my <= kPH1 && x < G.W && y < G.H) G.b[(size_t)y * G.P + x] = sum;
            }
        }
        __syncthreads();
        if (tid < kPW1 * kPH1) {
            const int i = (1 + (tid >> 5)) * MW + 1 + (tid & 31);
            rho[tid] = rm[i] + pair_sum<MW, (MH - 1) * MW>(cm, xm, i);
        }
        __syncthreads();
        if (tid < kPW1 * kPH1 / 4) {
            const int X = tid & 15, Y = tid >> 4, f = 2 * Y * kPW1 + 2 * X;
            float sum = 0.f;
            sum += rho[f] + rho[f + 1];
            sum += rho[f + kPW1] + rho[f + kPW1 + 1];
            const int x = (mx0 >> 1) + X, y = (my0 >> 1) + Y;
            if (x < C.W && y < C.H) C.b[(size_t)y * C.P + x] = sum;
        }
        __syncthreads();
    }
}

// x_l from x_{l+2}, b_{l+1} and b_l (x_{l+1} stays in the CTA).
__global__ void __launch_bounds__(kPairThreads) mg_pair_up_kernel(Args a, int l)
{
    constexpr int YW = kPW1 + 4, YH = kPH1 + 4;          // middle cells of y
    constexpr int MW = kPW1 + 2, MH = kPH1 + 2;          // middle cells of x
    constexpr int FW = 2 * kPW1 + 2, FH = 2 * kPH1 + 2;  // level-l cells of y
    constexpr int NY = (YW * YH + kPairThreads - 1) / kPairThreads, NM = (MW * MH + kPairThreads - 1) / kPairThreads,
                  NF = (FW * FH + kPairThreads - 1) / kPairThreads;
    __shared__ float cm[4 * (YH - 1) * YW], bm[YW * YH], dm[YW * YH], ym[YW * YH], xm[MW * MH];
    __shared__ float cf[4 * (FH - 1) * FW], bf[FW * FH], df[FW * FH], yf[FW * FH];
    const Lev& F = a.lev[l];
    const Lev& G = a.lev[l + 1];
    const Lev& C = a.lev[l + 2];
    const float om = a.omega, sc = a.scale;
    const int tx = (G.W + kPW1 - 1) / kPW1, tiles = tx * ((G.H + kPH1 - 1) / kPH1), tid = threadIdx.x;
    bool waited = false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int mx0 = (t % tx) * kPW1, my0 = (t / tx) * kPH1;
        const int fx0 = 2 * mx0, fy0 = 2 * my0;
        float gb[NY], fb[NF];
#pragma unroll
        for (int j = 0; j < NY; ++j) {
            const int i = tid + j * kPairThreads, x = mx0 - 2 + i % YW, y = my0 - 2 + i / YW;
            gb[j] = i < YW * YH && x >= 0 && x < G.W && y >= 0 && y < G.H ? __ldcg(G.b + (size_t)y * G.P + x) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int i = tid + j * kPairThreads, x = fx0 - 1 + i % FW, y = fy0 - 1 + i / FW;
            fb[j] = i < FW * FH && x >= 0 && x < F.W && y >= 0 && y < F.H ? __ldcg(F.b + (size_t)y * F.P + x) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            stage<YW, YH - 1>(cm + k * (YH - 1) * YW, static_cast<const float*>(G.c) + k * G.ps, G.P, G.W, G.H, mx0 - 2,
                              my0 - 2);
            stage<FW, FH - 1>(cf + k * (FH - 1) * FW, static_cast<const float*>(F.c) + k * F.ps, F.P, F.W, F.H, fx0 - 1,
                              fy0 - 1);
        }
        stage<YW, YH>(dm, G.Di, G.P, G.W, G.H, mx0 - 2, my0 - 2);
        stage<FW, FH>(df, F.Di, F.P, F.W, F.H, fx0 - 1, fy0 - 1);
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        float xc[NY];
#pragma unroll
        for (int j = 0; j < NY; ++j) {
            const int i = tid + j * kPairThreads, x = mx0 - 2 + i % YW, y = my0 - 2 + i / YW;
            xc[j] = i < YW * YH && x >= 0 && x < G.W && y >= 0 && y < G.H ? __ldcg(C.x + (size_t)(y >> 1) * C.P + (x >> 1))
                                                                          : 0.f;
        }
        copies_done();
        if (paused(a.st)) return;
#pragma unroll
        for (int j = 0; j < NY; ++j) {  // (each thread reads what it staged itself)
            const int i = tid + j * kPairThreads;
            if (i < YW * YH) {
                ym[i] = dm[i] > 0.f ? fmaf(sc, xc[j], om * gb[j] * dm[i]) : 0.f;
                bm[i] = gb[j];
            }
        }
#pragma unroll
        for (int j = 0; j < NF; ++j)
            if (tid + j * kPairThreads < FW * FH) bf[tid + j * kPairThreads] = fb[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NM; ++j) {
            const int i = tid + j * kPairThreads, f = (1 + i / MW) * YW + 1 + i % MW;
            if (i < MW * MH) xm[i] = smooth_of(ym[f], bm[f], dm[f], om, pair_sum<YW, (YH - 1) * YW>(cm, ym, f));
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int i = tid + j * kPairThreads, x = i % FW, y = i / FW;
            if (i < FW * FH)
                yf[i] = df[i] > 0.f ? fmaf(sc, xm[((y + 1) >> 1) * MW + ((x + 1) >> 1)], om * bf[i] * df[i]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4 * kPW1 * kPH1 / kPairThreads; ++j) {
            const int i = tid + j * kPairThreads, lx = i % (2 * kPW1), ly = i / (2 * kPW1), f = (1 + ly) * FW + 1 + lx;
            const int x = fx0 + lx, y = fy0 + ly;
            if (x < F.W && y < F.H)
                F.x[(size_t)y * F.P + x] = smooth_of(yf[f], bf[f], df[f], om, pair_sum<FW, (FH - 1) * FW>(cf, yf, f));
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Set-up kernels
// ---------------------------------------------------------------------------

// Galerkin coarsening, one thread per coarse cell: the couplings of the cell's
// (up to 4) fine cells in both directions are summed per neighbouring
// aggregate (FP64), in a fixed order.  weight(k, dir, bq, aq) is the coupling
// of plane k of fine cell (2 X + aq, 2 Y + bq) towards its upper (dir 0) or
// lower (dir 1) neighbour, 0 where there is none.
template <class S, class F>
__device__ __forceinline__ void coarsen(const Lev& C, int X, int Y, double gam, F weight)
{
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    double ext = 0.0;
#pragma unroll
    for (int bq = 0; bq < 2; ++bq)
#pragma unroll
        for (int aq = 0; aq < 2; ++aq)
#pragma unroll
            for (int k = 0; k < S::NP; ++k)
#pragma unroll
                for (int dir = 0; dir < 2; ++dir) {
                    const int du = dir ? -S::du(k) : S::du(k), dv = dir ? -S::dv(k) : S::dv(k);
                    const int ox = (aq + du) >> 1, oy = (bq + dv) >> 1;  // aggregate of the neighbour, from (X, Y)
                    if (ox == 0 && oy == 0) continue;
                    const double wv = weight(k, dir, bq, aq);
                    ext += wv;
#pragma unroll
                    for (int o = 0; o < 4; ++o)
                        if (ox == CoarseSten::du(o) && oy == CoarseSten::dv(o)) c[o] += wv;
                }
    const size_t oc = (size_t)Y * C.P + X;
    float* cp = static_cast<float*>(C.c);
#pragma unroll
    for (int o = 0; o < 4; ++o) cp[(size_t)o * C.ps + oc] = (float)c[o];
    C.gam[oc] = (float)gam;
    C.D[oc] = (float)(gam + ext);
    C.Di[oc] = gam + ext > 0.0 ? (float)(1.0 / (gam + ext)) : 0.f;
}

// Summed scribble weight of a coarse cell's fine cells.
__device__ __forceinline__ double gamma_sum(const Lev& F, const float* g, int gp, int X, int Y)
{
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int x = 2 * X + (q & 1), y = 2 * Y + (q >> 1);
        if (x < F.W && y < F.H) t += g[(size_t)y * gp + x];
    }
    return t;
}

// Level 0 into level 1: tiles of 32 x 8 coarse cells, whose 64 x 16 pixels of
// the 12 planes (with the halo of the mirrored couplings) go through shared
// memory, so that the planes are read once and coalesced (1080p, FP16: 143 us
// cold with each thread loading its own 96 couplings, 28 now, 9 us at the copy
// rate).
constexpr int kBuildTY = 16;
template <class T>
__global__ void __launch_bounds__(kThreads) mg_build0_kernel(Args a)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem[];
    T* pt = reinterpret_cast<T*>(smem);
    const Lev& F = a.lev[0];
    const Lev& C = a.lev[1];
    const int cx = threadIdx.x & 31, cy = threadIdx.x >> 5;
    const int tiles_x = (F.W + kTX - 1) / kTX, tiles = tiles_x * ((F.H + kBuildTY - 1) / kBuildTY);
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int x0 = (t % tiles_x) * kTX, y0 = (t / tiles_x) * kBuildTY;
        __syncthreads();
        load_planes<T, FineSten::NP, kBuildTY + kHalo>(pt, static_cast<const T*>(F.c), F.ps, F.P, F.W, F.H, x0, y0);
        const int X = (x0 >> 1) + cx, Y = (y0 >> 1) + cy;
        const double gam = gamma_sum(F, a.gamma, a.P, X, Y);
        copies_done();
        __syncthreads();
        if (X < C.W && Y < C.H)
            coarsen<FineSten>(C, X, Y, gam, [&](int k, int dir, int bq, int aq) {
                const int lx = 2 * cx + aq + 8 - (dir ? FineSten::du(k) : 0);
                const int ly = 2 * cy + bq + kHalo - (dir ? FineSten::dv(k) : 0);
                return (double)tof(pt[((size_t)k * (kBuildTY + kHalo) + ly) * kPW + lx]);
            });
    }
}

// Level l >= 1 into l + 1, one cell.
__device__ __forceinline__ void coarsen_cell(const Args& a, int l, int i)
{
    const Lev& F = a.lev[l];
    const Lev& C = a.lev[l + 1];
    const float* w = static_cast<const float*>(F.c);
    const int X = i % C.W, Y = i / C.W;
    coarsen<CoarseSten>(C, X, Y, gamma_sum(F, F.gam, F.P, X, Y), [&](int k, int dir, int bq, int aq) {
        const int du = CoarseSten::du(k), dv = CoarseSten::dv(k);
        const int x = 2 * X + aq, y = 2 * Y + bq;
        const int xn = dir ? x - du : x + du, yn = dir ? y - dv : y + dv;
        const bool in = x < F.W && y < F.H && xn >= 0 && xn < F.W && yn >= 0 && yn < F.H;
        return in ? (double)w[(size_t)k * F.ps + (dir ? (size_t)yn * F.P + xn : (size_t)y * F.P + x)] : 0.0;
    });
}

__global__ void __launch_bounds__(128) mg_build_kernel(Args a, int l)
{
    pdl_enter();
    const Lev& C = a.lev[l + 1];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C.W * C.H; i += gridDim.x * blockDim.x) coarsen_cell(a, l, i);
}

// The levels after lb in one CTA (each depends on the one before), then the
// dense FP64 inverse of the coarsest operator by Gauss-Jordan elimination (SPD:
// no pivoting).  The matrix stays in registers: thread (row, sub) holds the
// columns sub, sub + 8, ...; a step publishes the pivot's row and column and its
// reciprocal in shared memory (two copies in turn, so one barrier a step).
// Bound by the chain of one step (FP64 reciprocal, barrier, update: 0.45-0.6 us);
// with the matrix in shared memory, two barriers and an index division per
// entry it was 1.2 us for n = 40 and 2.8 for n = 70.
// NC: columns per thread, 8 NC >= n; 8 n threads, rounded up to a warp.
constexpr int kOneCtaCells = 1024;  // a level this small is built by one CTA
template <int NC>
__global__ void __launch_bounds__(64 * NC) mg_coarse_kernel(Args a, int lb)
{
    pdl_enter();
    for (int l = lb; l < a.L; ++l) {
        for (int i = threadIdx.x; i < a.lev[l + 1].W * a.lev[l + 1].H; i += blockDim.x) coarsen_cell(a, l, i);
        __syncthreads();
    }
    __shared__ double s_row[2][kCoarseMax], s_col[2][kCoarseMax];
    __shared__ double s_inv[2], s_dmax;
    const Lev& C = a.lev[a.L];
    const int n = C.W * C.H, row = threadIdx.x >> 3, sub = threadIdx.x & 7;
    const float* cp = static_cast<const float*>(C.c);
    double v[NC];
    const int xr = row % C.W, yr = row / C.W;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        const int col = sub + 8 * j, xc = col % C.W, yc = col / C.W, du = xc - xr, dv = yc - yr;
        v[j] = 0.0;
        if (row < n && col < n && du >= -1 && du <= 1 && dv >= -1 && dv <= 1) {
            const size_t orow = (size_t)yr * C.P + xr, ocol = (size_t)yc * C.P + xc;
            const bool up = dv > 0 || (dv == 0 && du > 0);
            const int k = dv == 0 ? 0 : 2 + (up ? du : -du);
            v[j] = row == col ? (double)C.D[orow] : -(double)cp[(size_t)k * C.ps + (up ? orow : ocol)];
        }
    }
    // Zero rows (aggregates with no coupling and no scribble weight, as in
    // images less than 3 pixels wide or tall, where no 3x3 window exists) are
    // left out: for a positive semidefinite matrix a zero pivot means a zero
    // row and column, and the inverse on the remaining rows is exact.
    if (threadIdx.x < 32) {
        double m = 0.0;
        for (int i = threadIdx.x; i < n; i += 32) m = fmax(m, (double)C.D[(size_t)(i / C.W) * C.P + i % C.W]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) s_dmax = m;
    }
    __syncthreads();
    const double tiny = 1e-300 + 1e-14 * s_dmax;
    bool bad = false;
#pragma unroll
    for (int jb = 0; jb < NC; ++jb) {
        for (int m = 0; m < 8; ++m) {
            const int k = 8 * jb + m;
            if (k >= n || bad) break;
            double* pr = s_row[m & 1];
            double* pc = s_col[m & 1];
            if (row == k) {
#pragma unroll
                for (int j = 0; j < NC; ++j) pr[sub + 8 * j] = v[j];
                if (sub == m) {
                    const double piv = v[jb];
                    const bool fine = isfinite(piv) && piv >= 0.0;
                    s_inv[m & 1] = !fine ? -1.0 : (piv <= tiny ? 0.0 : 1.0 / piv);
                }
            }
            if (sub == m) pc[row] = v[jb];
            __syncthreads();
            const double inv = s_inv[m & 1];  // 0: a zero row, -1: not positive semidefinite
            if (inv < 0.0) {
                bad = true;
                break;
            }
            if (row == k) {
#pragma unroll
                for (int j = 0; j < NC; ++j) v[j] *= inv;
                if (sub == m) v[jb] = inv;
            } else {
                const double f = pc[row] * inv;
#pragma unroll
                for (int j = 0; j < NC; ++j) v[j] = fma(-f, pr[sub + 8 * j], v[j]);
                if (sub == m) v[jb] = -f;
            }
        }
    }
    if (bad) {
        if (threadIdx.x == 0) {
            a.st->status = GM_ERR_BREAKDOWN;
            a.st->done = 1;
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < NC; ++j)
        if (row < n && sub + 8 * j < n) C.M[(size_t)row * n + sub + 8 * j] = v[j];
}

// 1 / d of the level-0 iteration diagonal (0 where d = 0), FP64 solution from
// the FP32 guess (none: only the hierarchy is set up), initial state.
__global__ void mg_init_kernel(Args a)
{
    pdl_enter();
    const int W = a.W, H = a.H, P = a.P;
    const size_t n = (size_t)W * H;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t o = (i / W) * P + i % W;
        const float d = a.lev[0].D[o];
        a.lev[0].Di[o] = d > 0.f ? 1.f / d : 0.f;
        if (a.alpha_in) {
            a.x[o] = (double)a.alpha_in[i];
            a.xinc[o] = 0.f;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        State* st = a.st;
        st->rz[0] = st->rz[1] = st->rr = st->bn2 = st->rr_true = 0.0;
        st->iter = 0;
        st->iter_next = 0;
        st->done = 0;
        st->status = GM_OK;
        st->need_replace = a.alpha_in ? 1 : 0;
        st->replacements = 0;
        st->fold_at = -1;
        st->restart_at = -1;
        for (int k = 0; k < 2; ++k) st->ticket[k] = 0u;
    }
}

// Solution out (FP32), zero when b = 0.
__global__ void mg_final_kernel(Args a)
{
    pdl_enter();
    const int W = a.W, H = a.H, P = a.P;
    const bool zero = !(a.st->bn2 > 0.0) && a.st->replacements > 0;
    const size_t n = (size_t)W * H;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int y = (int)(i / W), x = (int)(i % W);
        const size_t o = (size_t)y * P + x;
        a.alpha_out[(size_t)y * W + x] = zero ? 0.f : (float)(a.x[o] + (double)a.xinc[o]);
    }
}

}  // namespace mg
}  // namespace gm

// ===========================================================================
// Host driver
// ===========================================================================
namespace gm {
namespace mg {

// Cells of the middle level up to which two levels run as one kernel.  With
// pairs everywhere below it: 1501 x 703 (levels 1 + 2, 66 K cells in the middle)
// 53.5 -> 52.0 us per iteration; the next larger middle level of that kind has
// 330 K cells, where the repeated halo (1.5x the work of level l) is no longer
// hidden by latency.
constexpr int kPairMax = 140000;

struct Plan {
    int L, lt;
    int W[kMaxLevels], H[kMaxLevels];
};

static int make_plan(int W, int H, Plan& pl)
{
    pl.W[0] = W;
    pl.H[0] = H;
    int l = 0;
    for (;;) {
        const int w = (pl.W[l] + 1) / 2, h = (pl.H[l] + 1) / 2;
        if (++l >= kMaxLevels) { gm_set_error_msg("multigrid: too many levels"); return GM_ERR_UNSUPPORTED; }
        pl.W[l] = w;
        pl.H[l] = h;
        if ((long long)w * h <= kCoarseMax) break;
    }
    pl.L = l;
    // the dense level: the first one small enough
    pl.lt = pl.L;
    while (pl.lt > 1 && (long long)pl.W[pl.lt - 1] * pl.H[pl.lt - 1] <= kDenseMax) --pl.lt;
    return GM_OK;
}

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// Workspace carve: fine vectors r, q, p0, p1, z (FP32) and x (FP64) with the
// store's pitch; per coarse level 4 coupling planes, D, Gamma, b, x (FP32,
// pitch a multiple of 32); the matrices of the dense levels (FP64, 13.5 MB at
// most for the largest); reduction partials; state.
static size_t carve(const Plan& pl, int P0, char* base, Args* a)
{
    size_t off = 0;
    auto take = [&](size_t bytes) -> char* { char* p = base ? base + off : nullptr; off += al256(bytes); return p; };
    const size_t n0 = (size_t)pl.H[0] * P0;
    float* r = (float*)take(n0 * 4);
    float* q = (float*)take(n0 * 4);
    float* p0 = (float*)take(n0 * 4);
    float* p1 = (float*)take(n0 * 4);
    float* z = (float*)take(n0 * 4);
    float* di0 = (float*)take(n0 * 4);
    float* xinc = (float*)take(n0 * 4);
    double* x = (double*)take(n0 * 8);
    if (a) {
        a->r = r; a->q = q; a->p0 = p0; a->p1 = p1; a->x = x; a->xinc = xinc;
        a->lev[0].b = r;
        a->lev[0].x = z;
        a->lev[0].Di = di0;
    }
    for (int l = 1; l <= pl.L; ++l) {
        const int P = (pl.W[l] + 31) & ~31;
        const size_t n = (size_t)pl.H[l] * P;
        char* c = take(4 * n * 4);
        float* D = (float*)take(n * 4);
        float* Di = (float*)take(n * 4);
        float* gam = (float*)take(n * 4);
        float* b = (float*)take(n * 4);
        float* xl = (float*)take(n * 4);
        const size_t cells = (size_t)pl.W[l] * pl.H[l];
        double* M = l >= pl.lt ? (double*)take(cells * cells * 8) : nullptr;
        if (a) {
            Lev& v = a->lev[l];
            v.W = pl.W[l]; v.H = pl.H[l]; v.P = P;
            v.c = c; v.ps = n; v.D = D; v.Di = Di; v.gam = gam; v.b = b; v.x = xl; v.M = M;
        }
    }
    double* parts = (double*)take((size_t)5 * kMaxParts * 8);
    State* st = (State*)take(sizeof(State));
    if (a) { a->parts = parts; a->st = st; }
    return off;
}

// Per-device solver slots: each has a grow-only workspace, capture streams,
// an execution stream (for batches), pinned state for the read-back, timing
// events and a cache of instantiated graphs (gm_graph_cache.h).  Single solves use slot 0;
// gm_levin_solve_mg_many spreads its images over the slots.
//
// A graph serves any buffers of its shape and parameters: the kernels that use
// a store's planes or the caller's vectors (the set-up, the replacement, the
// level-0 passes and the final write, about 35 of 120 nodes) are given new ones
// before a launch (10-25 us; a capture and instantiation takes 1-2 ms).
enum { B_INIT = 0, B_BUILD0 = 1, B_REPLACE = 2, B_FINAL = 3, B_FINE = 4 };  // B_FINE + FM_*
struct BoundNode {
    cudaGraphNode_t node;
    void* fn;
    unsigned grid, threads, smem;
    int kind, nst, pending;
    unsigned long long cond, cond_outer;
};
struct Graph {
    Args key;             // the solve it is bound to
    Args shape;           // the same without the fields a binding sets
    Args launch;          // as captured (with the partial-sum counts)
    int tcode;
    cudaGraph_t graph;    // owns the nodes
    cudaGraphExec_t exec;
    std::vector<BoundNode> nodes;
    int rebinds;
    unsigned long long used;
};

struct Dev {
    void* ws = nullptr;
    size_t ws_bytes = 0;
    cudaStream_t cap = nullptr, cap2 = nullptr, cap3 = nullptr, run = nullptr;
    State* host_state = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr;
    std::vector<Graph> graphs;
    unsigned long long clock = 0;
    int sms = 0;
    int cond_ok = -1;  // conditional nodes usable (-1 unknown)
    State* pin = nullptr;  // slot 0 only: pinned result states of a batch
    int pin_n = 0;
};

constexpr int kSlots = 8;        // concurrent solves of gm_levin_solve_mg_many

// GM_MG_GRAPH=0 selects the host-driven loop (the same kernels launched
// one by one, the done flag read every 4 iterations), e.g. for profilers
// that do not look inside conditional graph nodes.
static bool graph_enabled()
{
    const char* e = getenv("GM_MG_GRAPH");
    return !(e && e[0] == '0');
}

static std::mutex g_mu;
static Dev g_dev[64][kSlots];

static void free_graph(Graph& g)
{
    cudaGraphExecDestroy(g.exec);
    cudaGraphDestroy(g.graph);
}

static void drop_graphs(Dev& d)
{
    for (Graph& g : d.graphs) free_graph(g);
    d.graphs.clear();
}

static int dev_setup(Dev& d, size_t bytes)
{
    if (!d.cap) {
        GM_CUDA_TRY(cudaStreamCreateWithFlags(&d.cap, cudaStreamNonBlocking));
        GM_CUDA_TRY(cudaStreamCreateWithFlags(&d.cap2, cudaStreamNonBlocking));
        GM_CUDA_TRY(cudaStreamCreateWithFlags(&d.cap3, cudaStreamNonBlocking));
        GM_CUDA_TRY(cudaStreamCreateWithFlags(&d.run, cudaStreamNonBlocking));
        GM_CUDA_TRY(cudaMallocHost((void**)&d.host_state, sizeof(State)));
        GM_CUDA_TRY(cudaEventCreate(&d.e0));
        GM_CUDA_TRY(cudaEventCreate(&d.e1));
        GM_CUDA_TRY(cudaEventCreate(&d.e2));
    }
    if (d.ws_bytes < bytes) {
        drop_graphs(d);
        if (d.ws) cudaFree(d.ws);
        d.ws = nullptr;
        d.ws_bytes = 0;
        if (cudaMalloc(&d.ws, bytes) != cudaSuccess) {
            cudaGetLastError();
            gm_set_error_msg("multigrid workspace allocation (%zu bytes) failed", bytes);
            return GM_ERR_NOMEM;
        }
        d.ws_bytes = bytes;
    }
    return GM_OK;
}

static int occupancy(const void* fn, int smem, int threads)
{
    struct E { const void* fn; int dev, smem, occ; };
    static std::vector<E> cache;  // guarded by g_mu
    int dev = 0;
    cudaGetDevice(&dev);
    for (const E& e : cache)
        if (e.fn == fn && e.dev == dev && e.smem == smem) return e.occ;
    if (smem > 48 * 1024) {
        // the largest size the kernel may ask for (opt-in maximum less its
        // static shared memory), so graphs captured with other sizes stay valid
        int optin = 0;
        cudaFuncAttributes fa;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, fn) == cudaSuccess)
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 std::max(smem, optin - (int)fa.sharedSizeBytes));
        cudaGetLastError();
    }
    int o = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fn, threads, smem) != cudaSuccess) o = 1;
    if (o < 1) o = 1;
    cache.push_back({fn, dev, smem, o});
    return o;
}

static int tiles_of(int W, int H, int ty) { return ((W + kTX - 1) / kTX) * ((H + ty - 1) / ty); }

// Enqueues kernels on one stream.  The template argument is the element type
// of the fine iteration planes.  A dry pass only computes the launch shapes
// (it sets the kernels' shared-memory limits before any stream capture).
// Tensor maps of the TMA-pipelined kernels: the level-0 SpMV, and the
// restriction / prolongation of every level above the dense one.
struct FineMaps {
    TMaps spmv, down[kMaxLevels], up[kMaxLevels];
};

// Whether the outer SpMV streams the FP16 iteration planes (tcode 1) rather
// than the FP32 ones.  It saves 24 of ~180 B per pixel-iteration, and the
// FP16 outer operator costs 1 % more iterations at rtol 1e-6 (1080p: 87
// against 86).  Between replacements each cycle can refine less, so below
// 1e-7 the extra iterations outweigh it (1e-10: 408 against 331), and the
// FP32 planes stay.  rtol <= 0 (a fixed iteration count) takes the FP16 ones.
constexpr double kOuterLowMinRtol = 1e-7;
static int outer_low_for(int tcode, double rtol)
{
    return tcode == 1 && !(rtol > 0.0 && rtol < kOuterLowMinRtol) ? 1 : 0;
}

// Tile rows of the level-0 kernels on 2-byte planes.  Short tiles spread a small
// image over more SMs and leave room for a second CTA (the next kernel's, or
// another solve's) on each; their halo rows (10 of 8 plane rows, 12 of 8 vector
// rows) cost more L2 and DRAM reads on a large one.  Us per iteration with 16 and 8
// rows: 20.7 / 19.5 at 317 x 211, 32.6 / 30.7 at 640 x 480, 45 / 45 at 960 x 720 (eight
// such solves at once 284 / 273 us), 51.8 / 52.6 at 1501 x 703, 500 / 547 at 4096^2.
static int level0_rows(int W, int H, int sms)
{
    const long long tiles = (long long)((W + kFTW - 1) / kFTW) * ((H + kRows - 1) / kRows);
    return tiles <= 5LL * sms ? kRows : kTallRows;
}

// Tensor maps of the level-0 kernels (es: bytes per element of the
// iteration planes).
static int make_maps(const Args& a, int es, CUtensorMapDataType dt, FineMaps& fm)
{
    const uint64_t W = (uint64_t)a.W, H = (uint64_t)a.H, P = (uint64_t)a.P;
    auto planes = [&](CUtensorMap* m, const void* base, CUtensorMapDataType t, uint64_t e, uint64_t ps, int th) {
        const uint64_t d3[3] = {W, H, 12};
        const uint64_t s3[2] = {P * e, ps * e};
        const uint32_t b3[3] = {(uint32_t)kFBW, (uint32_t)(th + 2), 12u};
        return gm_make_tmap(m, t, 3, const_cast<void*>(base), d3, s3, b3);
    };
    auto vec = [&](CUtensorMap* m, const float* base, uint64_t w, uint64_t h, uint64_t pitch, int bw, int bh) {
        const uint64_t d2[2] = {w, h};
        const uint64_t s2[1] = {pitch * 4};
        const uint32_t b2[2] = {(uint32_t)bw, (uint32_t)bh};
        return gm_make_tmap(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), d2, s2, b2);
    };
    const int t32 = kRows, tlo = es == 2 ? a.rows0 : kRows;
    const Lev& L0 = a.lev[0];
    // the SpMV streams the FP16 iteration planes and their diagonal d when
    // outer_low is set, else the FP32 planes and d32
    const bool lo16 = es == 2 && dt == CU_TENSOR_MAP_DATA_TYPE_FLOAT16 && a.outer_low;
    const int ts = lo16 ? tlo : t32;
    if (lo16) GM_TRY(planes(&fm.spmv.m[0], L0.c, dt, 2, L0.ps, ts));
    else GM_TRY(planes(&fm.spmv.m[0], a.w32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.ps32, ts));
    GM_TRY(vec(&fm.spmv.m[1], L0.x, W, H, P, kFBW, ts + 4));
    GM_TRY(vec(&fm.spmv.m[2], a.p0, W, H, P, kFBW, ts + 4));
    GM_TRY(vec(&fm.spmv.m[3], a.p1, W, H, P, kFBW, ts + 4));
    GM_TRY(vec(&fm.spmv.m[4], lo16 ? L0.D : a.d32, W, H, P, kFTW, ts));
    for (int l = 0; l < a.lt; ++l) {
        // level 0: the store's planes (12, iteration precision); below: 4 FP32 planes
        const Lev& F = a.lev[l];
        const Lev& Cl = a.lev[l + 1];
        const int np = l == 0 ? 12 : 4;
        const uint64_t e = l == 0 ? (uint64_t)es : 4;
        const int th = l == 0 ? tlo : t32;
        const uint64_t Wl = (uint64_t)F.W, Hl = (uint64_t)F.H, Pl = (uint64_t)F.P;
        const uint64_t d3[3] = {Wl, Hl, (uint64_t)np};
        const uint64_t s3[2] = {Pl * e, (uint64_t)F.ps * e};
        const uint32_t b3[3] = {(uint32_t)kFBW, (uint32_t)(th + 2), (uint32_t)np};
        GM_TRY(gm_make_tmap(&fm.down[l].m[0], l == 0 ? dt : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, F.c, d3, s3, b3));
        GM_TRY(vec(&fm.down[l].m[1], F.b, Wl, Hl, Pl, kFBW, th + 4));
        GM_TRY(vec(&fm.down[l].m[2], F.Di, Wl, Hl, Pl, kFBW, th + 4));
        fm.up[l] = fm.down[l];
        GM_TRY(vec(&fm.up[l].m[3], Cl.x, (uint64_t)Cl.W, (uint64_t)Cl.H, (uint64_t)Cl.P, kXBW, th / 2 + 2));
    }
    return GM_OK;
}

template <class T>
struct Enq {
    const Args& a;
    int sms;
    cudaStream_t s;
    bool dry;
    const FineMaps* fm;
    std::vector<BoundNode>* rec = nullptr;  // capture only: the nodes a binding sets

    // Notes the kernel node captured last.
    template <class K> void note(K fn, int tiles, int smem, int threads, int kind, int nst = 0, int pending = 0) const
    {
        if (!rec || dry) return;
        cudaStreamCaptureStatus cs;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        BoundNode b = {};
        if (cudaStreamGetCaptureInfo(s, &cs, nullptr, nullptr, &deps, &nd) == cudaSuccess && nd == 1) b.node = deps[0];
        b.fn = (void*)fn;
        b.grid = (unsigned)ctas(fn, tiles, smem, threads);
        b.threads = (unsigned)threads;
        b.smem = (unsigned)smem;
        b.kind = kind;
        b.nst = nst;
        b.pending = pending;
        b.cond = a.cond;
        b.cond_outer = a.cond_outer;
        rec->push_back(b);
    }

    template <class K> int ctas(K fn, int tiles, int smem, int threads) const
    {
        const int g = std::min(tiles, sms * occupancy((const void*)fn, smem, threads));
        return std::max(1, std::min(g, kMaxParts));
    }

    template <class K, class... X> void go(K fn, int tiles, int smem, int threads, X... args) const
    {
        const int g = ctas(fn, tiles, smem, threads);
        if (dry) return;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)g);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = (size_t)smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, fn, args...);
    }

    int pointwise_tiles() const
    {
        return (int)std::min<size_t>((size_t)sms * 4, ((size_t)(a.W + 3) / 4 * a.H + kThreads - 1) / kThreads);
    }

    // The TMA-pipelined kernels: level 0 with the store's 12 planes in the
    // iteration precision, the levels below with their 4 FP32 planes.
    template <int MODE> void fine(int l, int pending = 0) const
    {
        const TMaps& m = MODE == FM_SPMV ? fm->spmv : (MODE == FM_DOWN ? fm->down[l] : fm->up[l]);
        with_fine<MODE>(l, [&](auto fn, int tiles, int smem, int threads, int nst) {
            go(fn, tiles, smem, threads, m, a, l, nst, pending);
            if (l == 0) note(fn, tiles, smem, threads, B_FINE + MODE, nst, pending);
        });
    }

    // The kernel and launch shape of one level's pass.  One ring stage where
    // every tile gets a CTA of its own: nothing is left to prefetch, and with
    // half the shared memory a second CTA (the next kernel's, or another
    // solve's) fits beside it.
    template <int MODE, class F> auto with_fine(int l, F f) const
    {
        const Lev& G = a.lev[l];
        auto shape = [&](auto fn, auto layout) {
            using LY = decltype(layout);
            const int tiles = ((G.W + kFTW - 1) / kFTW) * ((G.H + LY::TH - 1) / LY::TH);
            const int nst = tiles <= sms * occupancy((const void*)fn, LY::total(1), LY::THR) ? 1 : 2;
            return f(fn, tiles, LY::total(nst), LY::THR, nst);
        };
        constexpr int ES = FinePlanes<MODE, T>::ES;
        if (l > 0) return shape(mg_fine_kernel<MODE, CoarseSten, float, kRows>, FineLayout<MODE, 4, 4, kRows>());
        if (MODE == FM_SPMV && !a.outer_low)
            return shape(mg_fine_kernel<MODE, FineSten, float, kRows>, FineLayout<MODE, 4, 12, kRows>());
        if constexpr (ES == 2)
            if (a.rows0 == kTallRows)
                return shape(mg_fine_kernel<MODE, FineSten, T, kTallRows>, FineLayout<MODE, ES, 12, kTallRows>());
        return shape(mg_fine_kernel<MODE, FineSten, T, kRows>, FineLayout<MODE, ES, 12, kRows>());
    }

    // Partials per sum: the CTAs of the kernels that leave them.
    void count_parts(Args& out) const
    {
        auto n = [&](auto fn, int tiles, int smem, int threads, int) { return ctas(fn, tiles, smem, threads); };
        out.n_pq = with_fine<FM_SPMV>(0, n);
        out.n_rz = with_fine<FM_UP>(0, n);
        out.n_rr = ctas(mg_update_kernel<false>, pointwise_tiles(), 0, kThreads);
    }

    // Whether levels l and l + 1 run as one kernel: pairs from the dense level
    // up, while the middle level is small.
    bool paired(int l) const
    {
        return l >= 1 && l + 1 < a.lt && (a.lt - l) % 2 == 0 && (long long)a.lev[l + 1].W * a.lev[l + 1].H <= kPairMax;
    }
    int pair_tiles(int l) const
    {
        return ((a.lev[l + 1].W + kPW1 - 1) / kPW1) * ((a.lev[l + 1].H + kPH1 - 1) / kPH1);
    }

    void vcycle(int pending) const
    {
        for (int l = 0; l < a.lt;) {
            if (paired(l)) {
                go(mg_pair_down_kernel, pair_tiles(l), 0, kPairThreads, a, l);
                l += 2;
            } else {
                fine<FM_DOWN>(l, l == 0 ? pending : 0);
                ++l;
            }
        }
        const int n = a.lev[a.lt].W * a.lev[a.lt].H;
        go(mg_dense_kernel, (n + kThreads / 32 - 1) / (kThreads / 32), 0, kThreads, a);
        for (int l = a.lt - 1; l >= 0; --l) {
            if (paired(l - 1)) {
                --l;
                go(mg_pair_up_kernel, pair_tiles(l), 0, kPairThreads, a, l);
            } else {
                fine<FM_UP>(l);
            }
        }
    }

    void replace() const
    {
        constexpr int sm = (int)(sizeof(float) * FineSten::NP * (kTY + kHalo) * kPW +
                                 sizeof(double) * (kTY + 2 * kHalo) * kVW);
        go(mg_replace_kernel, tiles_of(a.W, a.H, kTY), sm, kThreads, a);
        note(mg_replace_kernel, tiles_of(a.W, a.H, kTY), sm, kThreads, B_REPLACE);
    }

    void setup() const
    {
        go(mg_init_kernel, pointwise_tiles(), 0, kThreads, a);
        note(mg_init_kernel, pointwise_tiles(), 0, kThreads, B_INIT);
        constexpr int sm0 = (int)sizeof(T) * FineSten::NP * (kBuildTY + kHalo) * kPW;
        go(mg_build0_kernel<T>, tiles_of(a.W, a.H, kBuildTY), sm0, kThreads, a);
        note(mg_build0_kernel<T>, tiles_of(a.W, a.H, kBuildTY), sm0, kThreads, B_BUILD0);
        int l = 1;
        for (; l < a.L && (long long)a.lev[l + 1].W * a.lev[l + 1].H > kOneCtaCells; ++l)
            go(mg_build_kernel, (a.lev[l + 1].W * a.lev[l + 1].H + 127) / 128, 0, 128, a, l);
        const int nc = a.lev[a.L].W * a.lev[a.L].H, threads = (8 * nc + 31) / 32 * 32;
        static_assert(kCoarseMax == 128, "columns per thread");
        if (nc <= 40) go(mg_coarse_kernel<5>, 1, 0, threads, a, l);
        else if (nc <= 64) go(mg_coarse_kernel<8>, 1, 0, threads, a, l);
        else if (nc <= 96) go(mg_coarse_kernel<12>, 1, 0, threads, a, l);
        else go(mg_coarse_kernel<16>, 1, 0, threads, a, l);
        for (l = a.L - 1; l >= a.lt; --l)
            go(mg_dense_build_kernel, (a.lev[l].W + kDenseRun - 1) / kDenseRun * a.lev[l].H * kDenseParts,
               dense_build_smem(a.lev[l + 1].W * a.lev[l + 1].H), kThreads, a, l);
    }

    // One loop pass of preconditioner, matrix product and update; an iteration
    // does nothing when a replacement is due before it.
    void iterations(int count) const
    {
        for (int k = 0; k < count; ++k) {
            vcycle(k > 0);
            fine<FM_SPMV>(0);
            if (k + 1 < count) go(mg_update_kernel<false>, pointwise_tiles(), 0, kThreads, a);
            else go(mg_update_kernel<true>, pointwise_tiles(), 0, kThreads, a);
        }
    }

    void finish() const
    {
        go(mg_final_kernel, pointwise_tiles(), 0, kThreads, a);
        note(mg_final_kernel, pointwise_tiles(), 0, kThreads, B_FINAL);
    }
};

// Iterations per pass of the inner loop.  Going round a WHILE node costs 3-6 us
// more than the next kernel of a chain, and an iteration that is skipped
// because the replacement comes first about 12, so a pass is as long as
// divides the distance between replacements well.  With the replacement check
// out of the iteration and ten iterations a pass: 37.6 -> 34.8 us per iteration
// at 317 x 211, 47.2 -> 44.6 at 640 x 480, 106.5 -> 99.6 at 1080p.
static int unroll_for(const Args& a)
{
    const int period = std::max(1, std::min(a.max_iters, a.replace_every > 0 ? a.replace_every : a.max_iters));
    int best = 1, best_cost = INT_MAX;
    for (int u = 1; u <= 10; ++u) {
        const int passes = (int)std::min<long long>(1000, ((long long)std::min(period, 1000) + u - 1) / u);
        const int cost = 5 * passes + 12 * (passes * u - std::min(period, 1000));
        if (cost < best_cost) { best_cost = cost; best = u; }
    }
    return best;
}

// Adds a WHILE node to the capture on stream s (condition 1 at its start),
// with the handle *h or, where that is 0, a new one; returns its body.
static cudaError_t add_while(cudaStream_t s, cudaGraphConditionalHandle* h, cudaGraph_t* body)
{
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, &ndeps);
    if (e != cudaSuccess) return e;
    if (*h == 0) e = cudaGraphConditionalHandleCreate(h, g, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = *h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    e = cudaGraphAddNode(&node, g, deps, ndeps, &cp);
    if (e != cudaSuccess) return e;
    *body = cp.conditional.phGraph_out[0];
    return cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies);
}

// Captures the whole solve into one graph:
//   set-up; WHILE { replacement; WHILE { unrolled iterations } }; finish.
// The replacement kernel keeps or ends both loops, the update kernel ends the
// inner one when a replacement is due.
template <class T>
static int build_graph(Dev& d, Args a, const FineMaps& fm, Graph& out)
{
    cudaGraph_t g = nullptr, outer = nullptr, inner = nullptr;
    a.cond = a.cond_outer = 0;
    {
        const Enq<T> dry{a, d.sms, d.cap, true, &fm};  // sets the kernels' shared-memory limits too
        dry.setup();
        dry.replace();
        dry.iterations(2);
        dry.count_parts(a);
        dry.finish();
    }
    out.launch = a;
    GM_CUDA_TRY(cudaStreamBeginCapture(d.cap, cudaStreamCaptureModeThreadLocal));
    Enq<T>{a, d.sms, d.cap, false, &fm, &out.nodes}.setup();
    cudaGraphConditionalHandle ho = 0, hi = 0;
    cudaError_t e = add_while(d.cap, &ho, &outer);
    if (e == cudaSuccess) {
        // (the body's capture ends on every path: an unfinished one would
        // leave the stream unusable)
        e = cudaStreamBeginCaptureToGraph(d.cap2, outer, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            Args ab = a;
            ab.cond_outer = (unsigned long long)ho;
            cudaStreamCaptureStatus cs;
            cudaGraph_t og = nullptr;
            // the inner handle is needed by the replacement kernel, which
            // comes before the inner node
            e = cudaStreamGetCaptureInfo(d.cap2, &cs, nullptr, &og, nullptr, nullptr);
            if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&hi, og, 1, cudaGraphCondAssignDefault);
            ab.cond = (unsigned long long)hi;
            if (e == cudaSuccess) Enq<T>{ab, d.sms, d.cap2, false, &fm, &out.nodes}.replace();
            if (e == cudaSuccess) e = add_while(d.cap2, &hi, &inner);
            if (e == cudaSuccess) {
                e = cudaStreamBeginCaptureToGraph(d.cap3, inner, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
                if (e == cudaSuccess) {
                    const Enq<T> q{ab, d.sms, d.cap3, false, &fm, &out.nodes};
                    q.iterations(unroll_for(a));
                    cudaGraph_t x = nullptr;
                    e = cudaStreamEndCapture(d.cap3, &x);
                }
            }
            cudaGraph_t x = nullptr;
            const cudaError_t e1 = cudaStreamEndCapture(d.cap2, &x);
            if (e == cudaSuccess) e = e1;
        }
    }
    if (e == cudaSuccess) Enq<T>{a, d.sms, d.cap, false, &fm, &out.nodes}.finish();
    cudaError_t e2 = cudaStreamEndCapture(d.cap, &g);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&out.exec, g, 0);
    out.graph = g;
    if (e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        gm_set_error_msg("multigrid graph capture: %s", cudaGetErrorString(e));
        return GM_ERR_CUDA;
    }
    return GM_OK;
}

// The fields of a solve that a binding sets: copied from src, or cleared.
static void bind_fields(Args& a, const Args* src)
{
    a.lev[0].c = src ? src->lev[0].c : nullptr;
    a.lev[0].ps = src ? src->lev[0].ps : 0;
    a.lev[0].D = src ? src->lev[0].D : nullptr;
    a.w32 = src ? src->w32 : nullptr;
    a.ps32 = src ? src->ps32 : 0;
    a.gamma = src ? src->gamma : nullptr;
    a.d32 = src ? src->d32 : nullptr;
    a.bvec = src ? src->bvec : nullptr;
    a.bpitch = src ? src->bpitch : 0;
    a.alpha_in = src ? src->alpha_in : nullptr;
    a.alpha_out = src ? src->alpha_out : nullptr;
}

// Gives the graph the buffers of solve a.  (Launches that are already enqueued
// keep theirs.)  After a failure the graph is of no use: its nodes may have
// two solves' buffers.
static int rebind(Graph& g, const Args& a, const FineMaps& fm)
{
    Args b = g.launch;
    bind_fields(b, &a);
    for (const BoundNode& n : g.nodes) {
        b.cond = n.cond;
        b.cond_outer = n.cond_outer;
        TMaps m;
        int l = 0, nst = n.nst, pending = n.pending;
        void* fine[] = {&m, &b, &l, &nst, &pending};
        void* plain[] = {&b};
        cudaKernelNodeParams kp = {};
        kp.func = n.fn;
        kp.gridDim = dim3(n.grid);
        kp.blockDim = dim3(n.threads);
        kp.sharedMemBytes = n.smem;
        kp.kernelParams = plain;
        if (n.kind >= B_FINE) {
            const int mode = n.kind - B_FINE;
            m = mode == FM_SPMV ? fm.spmv : (mode == FM_DOWN ? fm.down[0] : fm.up[0]);
            kp.kernelParams = fine;
        }
        if (!n.node || cudaGraphExecKernelNodeSetParams(g.exec, n.node, &kp) != cudaSuccess) {
            cudaGetLastError();
            return GM_ERR_CUDA;
        }
    }
    memcpy(&g.key, &a, sizeof(Args));
    return GM_OK;
}

// A solve, as the cache of graphs asks about it.
template <class T>
struct GraphOps {
    Dev& d;
    const Args& a;
    const FineMaps& fm;
    int tcode;
    Args shape;

    GraphOps(Dev& dev, const Args& args, const FineMaps& maps, int tc) : d(dev), a(args), fm(maps), tcode(tc)
    {
        memcpy(&shape, &a, sizeof(Args));
        bind_fields(shape, nullptr);
    }
    bool same_shape(const Graph& g) const { return g.tcode == tcode && memcmp(&g.shape, &shape, sizeof(Args)) == 0; }
    bool bound(const Graph& g) const { return memcmp(&g.key, &a, sizeof(Args)) == 0; }
    int bind(Graph& g) const { return rebind(g, a, fm); }
    int build(Graph& g) const
    {
        GM_TRY(build_graph<T>(d, a, fm, g));
        memcpy(&g.key, &a, sizeof(Args));
        memcpy(&g.shape, &shape, sizeof(Args));
        g.tcode = tcode;
        return GM_OK;
    }
    void drop(Graph& g) const { free_graph(g); }
};

template <class T>
static int run(Dev& d, const Args& a0, const FineMaps& fm, int tcode, cudaStream_t st, float* ms)
{
    Args a = a0;
    if (d.cond_ok != 0 && graph_enabled()) {
        Graph* hit = nullptr;
        const int rc = cached_graph(d.graphs, d.clock, kSameShape, GraphOps<T>(d, a, fm, tcode), &hit);
        if (rc == GM_OK) {
            d.cond_ok = 1;
        } else if (d.cond_ok == -1) {
            d.cond_ok = 0;  // conditional nodes unavailable: host-driven loop from now on
            if (getenv("GM_MG_DEBUG")) fprintf(stderr, "gm_mg: graph path unavailable (%s)\n", gm_last_error());
        } else {
            return rc;
        }
        if (hit) {
            GM_CUDA_TRY(cudaEventRecord(d.e0, st));
            GM_CUDA_TRY(cudaGraphLaunch(hit->exec, st));
            GM_CUDA_TRY(cudaEventRecord(d.e1, st));
            GM_CUDA_TRY(cudaMemcpyAsync(d.host_state, a.st, sizeof(State), cudaMemcpyDeviceToHost, st));
            GM_CUDA_TRY(cudaStreamSynchronize(st));
            cudaEventElapsedTime(ms, d.e0, d.e1);
            return GM_OK;
        }
    }
    // Host-driven loop: the same kernels, the done flag read every 4 iterations.
    // (every pass takes an iteration or a replacement, and a replacement is
    // followed by an iteration or the end)
    a.cond = a.cond_outer = 0;
    Enq<T>{a, d.sms, st, true, &fm}.count_parts(a);
    Enq<T> q{a, d.sms, st, false, &fm};
    GM_CUDA_TRY(cudaEventRecord(d.e0, st));
    q.setup();
    for (int it = 0; it <= a.max_iters + 4; ++it) {
        q.replace();
        q.iterations(4);
        GM_CUDA_TRY(cudaMemcpyAsync(d.host_state, a.st, sizeof(State), cudaMemcpyDeviceToHost, st));
        GM_CUDA_TRY(cudaStreamSynchronize(st));
        if (d.host_state->done) break;
    }
    q.finish();
    GM_CUDA_TRY(cudaEventRecord(d.e1, st));
    GM_CUDA_TRY(cudaMemcpyAsync(d.host_state, a.st, sizeof(State), cudaMemcpyDeviceToHost, st));
    GM_CUDA_TRY(cudaStreamSynchronize(st));
    GM_CUDA_TRY(cudaGetLastError());
    cudaEventElapsedTime(ms, d.e0, d.e1);
    return GM_OK;
}

// One image of gm_levin_solve_mg_many.
struct Item {
    Plan pl;
    Args a;
    size_t bytes;
    FineMaps fm;
    int slot;
    int same;  // images of this size on the slot
};

// Every image's graph goes to the execution stream of its slot, forked
// from and joined back to st, and each image's final state to pinned memory on
// the same stream.  The images of one slot run one after another (they share
// its workspace); different slots run concurrently.  One host synchronisation
// for the whole batch.
template <class T>
struct ManyOps {
    Dev* slots;
    int K;
    std::vector<Item>& items;
    int tcode;
    cudaStream_t st;
    float* ms;

    int keep(int k) const { return std::max(kSameShape, std::min(items[k].same, (int)kGraphCache)); }
    int ready(int k) const
    {
        Dev& d = slots[items[k].slot];
        return ready_graph(d.graphs, d.clock, keep(k), GraphOps<T>(d, items[k].a, items[k].fm, tcode));
    }
    int begin() const
    {
        Dev& d0 = slots[0];
        const int n = (int)items.size();
        if (d0.pin_n < n) {
            if (d0.pin) cudaFreeHost(d0.pin);
            d0.pin = nullptr;
            d0.pin_n = 0;
            GM_CUDA_TRY(cudaMallocHost((void**)&d0.pin, (size_t)n * sizeof(State)));
            d0.pin_n = n;
        }
        GM_CUDA_TRY(cudaEventRecord(d0.e0, st));
        for (int j = 0; j < K; ++j) GM_CUDA_TRY(cudaStreamWaitEvent(slots[j].run, d0.e0, 0));
        d0.cond_ok = 1;
        return GM_OK;
    }
    int launch(int k) const
    {
        Dev& d = slots[items[k].slot];
        Graph* g = nullptr;
        GM_TRY(cached_graph(d.graphs, d.clock, keep(k), GraphOps<T>(d, items[k].a, items[k].fm, tcode), &g));
        GM_CUDA_TRY(cudaGraphLaunch(g->exec, d.run));
        GM_CUDA_TRY(cudaMemcpyAsync(slots[0].pin + k, items[k].a.st, sizeof(State), cudaMemcpyDeviceToHost, d.run));
        return GM_OK;
    }
    int join() const
    {
        for (int j = 0; j < K; ++j) {
            GM_CUDA_TRY(cudaEventRecord(slots[j].e1, slots[j].run));
            GM_CUDA_TRY(cudaStreamWaitEvent(st, slots[j].e1, 0));
        }
        GM_CUDA_TRY(cudaEventRecord(slots[0].e2, st));
        GM_CUDA_TRY(cudaStreamSynchronize(st));
        cudaEventElapsedTime(ms, slots[0].e0, slots[0].e2);
        return GM_OK;
    }
    void drain() const
    {
        for (int j = 0; j < K; ++j) cudaStreamSynchronize(slots[j].run);
        cudaGetLastError();
    }
};

// Fills the level-0 fields and the carve of an Args for the store.
static int prepare(const gm_levin_store* store, int use_low, Plan& pl, Args& a, size_t* bytes, int* tcode)
{
    const int W = store->W, H = store->H, P = store->pitch;
    if (W <= 0 || H <= 0 || P < W || (P & 7)) { gm_set_error_msg("multigrid: bad store shape"); return GM_ERR_INVALID; }
    GM_TRY(make_plan(W, H, pl));
    memset(&a, 0, sizeof(Args));
    const bool low = use_low && store->precision != GM_PREC_FP32;
    const size_t ps = store->plane_stride ? store->plane_stride : (size_t)H * P;
    const int esz = low ? 2 : 4;
    const void* wp = low ? store->w : (const void*)store->w32;
    if (((uintptr_t)wp & 15) || ((uintptr_t)store->w32 & 15) || ((ps * esz) & 15) || ((ps * 4) & 15)) {
        gm_set_error_msg("multigrid: planes must be 16-byte aligned");
        return GM_ERR_INVALID;
    }
    *tcode = low ? (store->precision == GM_PREC_FP16 ? 1 : 2) : 0;
    a.L = pl.L;
    a.lt = pl.lt;
    a.W = W; a.H = H; a.P = P;
    Lev& f = a.lev[0];
    f.W = W; f.H = H; f.P = P;
    f.c = const_cast<void*>(wp);
    f.ps = ps;
    f.D = low ? store->d : store->d32;
    a.w32 = store->w32;
    a.ps32 = ps;
    a.gamma = store->gamma;
    a.d32 = store->d32;
    *bytes = carve(pl, P, nullptr, nullptr);
    return GM_OK;
}

static CUtensorMapDataType tcode_dtype(int tcode)
{
    return tcode == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                      : (tcode == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32);
}

static int dev_index(int* dev)
{
    GM_CUDA_TRY(cudaGetDevice(dev));
    if (*dev < 0 || *dev >= 64) { gm_set_error_msg("device index out of range"); return GM_ERR_UNSUPPORTED; }
    return GM_OK;
}

}  // namespace mg

// Solve with the multigrid-preconditioned CG (called from the store solvers).
int run_mg_solver(const gm_levin_store* store, const float* b, int bpitch, const float* alpha_in, float* alpha_out,
                  const gm_solve_params* p, gm_solve_info* info, cudaStream_t st)
{
    using namespace mg;
    int sms = 0;
    GM_TRY(gm_check_device(&sms));
    if (p->max_iters < 0) { gm_set_error_msg("max_iters must be >= 0"); return GM_ERR_INVALID; }
    Plan pl;
    Args a;
    size_t bytes = 0;
    int tcode = 0;
    GM_TRY(prepare(store, p->use_low, pl, a, &bytes, &tcode));
    int dev = 0;
    GM_TRY(dev_index(&dev));
    std::lock_guard<std::mutex> g(g_mu);
    Dev& d = g_dev[dev][0];
    d.sms = sms;
    GM_TRY(dev_setup(d, bytes));
    carve(pl, a.P, (char*)d.ws, &a);
    a.bvec = b;
    a.bpitch = bpitch;
    a.alpha_in = alpha_in;
    a.alpha_out = alpha_out;
    a.rtol = p->rtol;
    a.outer_low = outer_low_for(tcode, a.rtol);
    a.rows0 = level0_rows(a.W, a.H, sms);
    a.planes_first = planes_leave_first((long long)a.W * a.H);
    a.max_iters = p->max_iters;
    a.replace_every = p->replace_every;
    a.omega = p->mg_omega > 0.f ? p->mg_omega : kDefaultOmega;
    a.scale = p->mg_scale > 0.f ? p->mg_scale : kDefaultScale;
    FineMaps fm;
    GM_TRY(make_maps(a, tcode ? 2 : 4, tcode_dtype(tcode), fm));
    float ms = 0.f;
    int rc;
    if (tcode == 1) rc = run<__half>(d, a, fm, tcode, st, &ms);
    else if (tcode == 2) rc = run<__nv_bfloat16>(d, a, fm, tcode, st, &ms);
    else rc = run<float>(d, a, fm, tcode, st, &ms);
    if (rc != GM_OK) return rc;
    const State& s = *d.host_state;
    if (info) {
        memset(info, 0, sizeof(*info));
        info->status = s.status;
        info->iters = s.iter;
        info->replacements = s.replacements;
        info->bnorm = std::sqrt(s.bn2);
        info->rel_residual = s.bn2 > 0.0 ? std::sqrt(s.rr_true / s.bn2) : 0.0;
        info->kernel_ms = ms;
        info->grid = pl.L + 1;
        info->where = 0;
        info->solver = GM_SOLVER_MG;
    }
    if (s.status != GM_OK) {
        gm_set_error_msg(s.status == GM_ERR_NOT_CONVERGED ? "multigrid CG: max_iters reached above rtol"
                                                         : "multigrid CG: breakdown (non-positive curvature, "
                                                           "singular coarse operator or non-finite value)");
    }
    return s.status;
}

static void fill_info(gm_solve_info* info, const mg::State& s, float ms, int levels)
{
    memset(info, 0, sizeof(*info));
    info->status = s.status;
    info->iters = s.iter;
    info->replacements = s.replacements;
    info->bnorm = std::sqrt(s.bn2);
    info->rel_residual = s.bn2 > 0.0 ? std::sqrt(s.rr_true / s.bn2) : 0.0;
    info->kernel_ms = ms;
    info->grid = levels;
    info->where = 0;
    info->solver = GM_SOLVER_MG;
}

}  // namespace gm

// Many independent multigrid solves at once (see gpumat.h).
extern "C" int gm_levin_solve_mg_many(const gm_levin_store* const* stores, float* const* alphas, int count,
                                      const gm_solve_params* prm, gm_solve_info* infos, void* stream)
{
    using namespace gm;
    using namespace gm::mg;
    gm_solve_params p;
    if (prm) p = *prm; else gm_default_params(&p);
    if (count < 0 || (count > 0 && (!stores || !alphas))) {
        gm_set_error_msg("gm_levin_solve_mg_many: bad arguments");
        return GM_ERR_INVALID;
    }
    if (count == 0) return GM_OK;
    if (p.max_iters < 0) { gm_set_error_msg("max_iters must be >= 0"); return GM_ERR_INVALID; }
    int sms = 0;
    GM_TRY(gm_check_device(&sms));
    std::vector<Item> items((size_t)count);
    int tcode = -1;
    for (int k = 0; k < count; ++k) {
        if (!stores[k] || !stores[k]->w32 || !alphas[k]) {
            gm_set_error_msg("gm_levin_solve_mg_many: image %d has no store or alpha", k);
            return GM_ERR_INVALID;
        }
        int tc = 0;
        GM_TRY(prepare(stores[k], p.use_low, items[k].pl, items[k].a, &items[k].bytes, &tc));
        if (tcode >= 0 && tc != tcode) {
            gm_set_error_msg("gm_levin_solve_mg_many: all stores must have the same precision");
            return GM_ERR_INVALID;
        }
        tcode = tc;
    }
    int dev = 0;
    GM_TRY(dev_index(&dev));
    std::lock_guard<std::mutex> g(g_mu);
    Dev* slots = g_dev[dev];
    const bool graphs = graph_enabled() && slots[0].cond_ok != 0;
    const int K = graphs ? std::min(kSlots, count) : 1;
    // Deal the images to the slots largest first, each to the least-loaded
    // slot (a fixed per-solve cost plus the pixels); the deal depends only
    // on the shapes, so repeated calls reuse each slot's cached graphs.
    {
        std::vector<int> order(count);
        for (int k = 0; k < count; ++k) order[k] = k;
        auto cost = [&](int k) { return (double)items[k].a.W * items[k].a.H + 2.0e5; };
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost(x) > cost(y); });
        std::vector<double> load(K, 0.0);
        for (int k : order) {
            const int j = (int)(std::min_element(load.begin(), load.end()) - load.begin());
            items[k].slot = j;
            load[j] += cost(k);
        }
        std::map<std::array<int, 3>, int> same;
        for (const Item& x : items) ++same[{x.slot, x.a.W, x.a.H}];
        for (Item& x : items) x.same = same[{x.slot, x.a.W, x.a.H}];
    }
    for (int j = 0; j < K; ++j) {
        size_t need = 0;
        for (int k = 0; k < count; ++k)
            if (items[k].slot == j) need = std::max(need, items[k].bytes);
        slots[j].sms = sms;
        GM_TRY(dev_setup(slots[j], need));
    }
    for (int k = 0; k < count; ++k) {
        Args& a = items[k].a;
        carve(items[k].pl, a.P, (char*)slots[items[k].slot].ws, &a);
        a.bvec = stores[k]->b;
        a.bpitch = stores[k]->pitch;
        a.alpha_in = alphas[k];
        a.alpha_out = alphas[k];
        a.rtol = p.rtol;
        a.outer_low = outer_low_for(tcode, a.rtol);
        a.rows0 = level0_rows(a.W, a.H, sms);
        a.planes_first = planes_leave_first((long long)a.W * a.H);
        a.max_iters = p.max_iters;
        a.replace_every = p.replace_every;
        a.omega = p.mg_omega > 0.f ? p.mg_omega : kDefaultOmega;
        a.scale = p.mg_scale > 0.f ? p.mg_scale : kDefaultScale;
        GM_TRY(make_maps(a, tcode ? 2 : 4, tcode_dtype(tcode), items[k].fm));
    }
    cudaStream_t st = (cudaStream_t)stream;
    int worst = GM_OK;
    if (!graphs) {
        // no conditional graphs here: one solve after another on slot 0
        for (int k = 0; k < count; ++k) {
            float ms = 0.f;
            int rc;
            if (tcode == 1) rc = run<__half>(slots[0], items[k].a, items[k].fm, tcode, st, &ms);
            else if (tcode == 2) rc = run<__nv_bfloat16>(slots[0], items[k].a, items[k].fm, tcode, st, &ms);
            else rc = run<float>(slots[0], items[k].a, items[k].fm, tcode, st, &ms);
            if (rc != GM_OK) return rc;
            if (infos) fill_info(&infos[k], *slots[0].host_state, ms, items[k].pl.L + 1);
            worst = std::max(worst, slots[0].host_state->status);
        }
    } else {
        float ms = 0.f;
        int rc;
        bool launched = false;
        if (tcode == 1) rc = run_images(count, ManyOps<__half>{slots, K, items, tcode, st, &ms}, &launched);
        else if (tcode == 2) rc = run_images(count, ManyOps<__nv_bfloat16>{slots, K, items, tcode, st, &ms}, &launched);
        else rc = run_images(count, ManyOps<float>{slots, K, items, tcode, st, &ms}, &launched);
        if (rc != GM_OK && !launched && slots[0].cond_ok == -1) {
            // the first capture failed: no conditional graphs here, so solve
            // the images one after another with the host-driven loop
            slots[0].cond_ok = 0;
            if (getenv("GM_MG_DEBUG")) fprintf(stderr, "gm_mg: graph path unavailable (%s)\n", gm_last_error());
            for (int k = 0; k < count; ++k) {
                GM_TRY(dev_setup(slots[0], items[k].bytes));
                Args& a = items[k].a;
                carve(items[k].pl, a.P, (char*)slots[0].ws, &a);
                GM_TRY(make_maps(a, tcode ? 2 : 4, tcode_dtype(tcode), items[k].fm));
                float ms1 = 0.f;
                if (tcode == 1) rc = run<__half>(slots[0], a, items[k].fm, tcode, st, &ms1);
                else if (tcode == 2) rc = run<__nv_bfloat16>(slots[0], a, items[k].fm, tcode, st, &ms1);
                else rc = run<float>(slots[0], a, items[k].fm, tcode, st, &ms1);
                if (rc != GM_OK) return rc;
                if (infos) fill_info(&infos[k], *slots[0].host_state, ms1, items[k].pl.L + 1);
                worst = std::max(worst, slots[0].host_state->status);
            }
            if (worst != GM_OK) gm_set_error_msg("multigrid batch: an image ended with status %d", worst);
            return worst;
        }
        if (rc != GM_OK) return rc;
        for (int k = 0; k < count; ++k) {
            if (infos) fill_info(&infos[k], slots[0].pin[k], ms, items[k].pl.L + 1);
            worst = std::max(worst, slots[0].pin[k].status);
        }
    }
    if (worst != GM_OK) gm_set_error_msg("multigrid batch: an image ended with status %d", worst);
    return worst;
}

// ---------------------------------------------------------------------------
// C ABI: level shapes and an inspection entry for tests
// ---------------------------------------------------------------------------
extern "C" int gm_levin_mg_levels(int W, int H, int* nlevels, int* dims, int cap)
{
    using namespace gm::mg;
    if (W <= 0 || H <= 0 || !nlevels) { gm_set_error_msg("gm_levin_mg_levels: bad arguments"); return GM_ERR_INVALID; }
    Plan pl;
    GM_TRY(make_plan(W, H, pl));
    *nlevels = pl.L + 1;
    if (dims)
        for (int l = 0; l <= pl.L && l < cap; ++l) { dims[2 * l] = pl.W[l]; dims[2 * l + 1] = pl.H[l]; }
    return GM_OK;
}

extern "C" int gm_levin_mg_inspect(const gm_levin_store* store, int use_low, const float* r, float* z, int level,
                                   float* c_host, float* d_host, void* stream)
{
    using namespace gm;
    using namespace gm::mg;
    if (!store || !store->w32) { gm_set_error_msg("gm_levin_mg_inspect: bad arguments"); return GM_ERR_INVALID; }
    int sms = 0;
    GM_TRY(gm_check_device(&sms));
    Plan pl;
    Args a;
    size_t bytes = 0;
    int tcode = 0;
    GM_TRY(prepare(store, use_low, pl, a, &bytes, &tcode));
    if (level < 0 || level > pl.L) { gm_set_error_msg("gm_levin_mg_inspect: level out of range"); return GM_ERR_INVALID; }
    int dev = 0;
    GM_TRY(dev_index(&dev));
    std::lock_guard<std::mutex> g(g_mu);
    Dev& d = g_dev[dev][0];
    d.sms = sms;
    GM_TRY(dev_setup(d, bytes));
    carve(pl, a.P, (char*)d.ws, &a);
    a.omega = kDefaultOmega;
    a.scale = kDefaultScale;
    a.max_iters = 1;
    a.rows0 = level0_rows(a.W, a.H, sms);
    a.planes_first = planes_leave_first((long long)a.W * a.H);
    FineMaps fm;
    GM_TRY(make_maps(a, tcode ? 2 : 4, tcode_dtype(tcode), fm));
    cudaStream_t st = (cudaStream_t)stream;
    auto go = [&](auto tag) {
        using T = decltype(tag);
        Enq<T> q{a, sms, st, false, &fm};
        q.setup();
        if (r && z) {
            cudaMemcpy2DAsync(a.r, (size_t)a.P * 4, r, (size_t)a.W * 4, (size_t)a.W * 4, a.H, cudaMemcpyDeviceToDevice,
                              st);
            q.vcycle(0);
            cudaMemcpy2DAsync(z, (size_t)a.W * 4, a.lev[0].x, (size_t)a.P * 4, (size_t)a.W * 4, a.H,
                              cudaMemcpyDeviceToDevice, st);
        }
    };
    if (tcode == 1) go(__half());
    else if (tcode == 2) go(__nv_bfloat16());
    else go(0.0f);
    if (level >= 1 && (c_host || d_host)) {
        const Lev& v = a.lev[level];
        for (int k = 0; k < 4 && c_host; ++k)
            GM_CUDA_TRY(cudaMemcpy2DAsync(c_host + (size_t)k * v.W * v.H, (size_t)v.W * 4,
                                          static_cast<float*>(v.c) + (size_t)k * v.ps, (size_t)v.P * 4,
                                          (size_t)v.W * 4, v.H, cudaMemcpyDeviceToHost, st));
        if (d_host)
            GM_CUDA_TRY(cudaMemcpy2DAsync(d_host, (size_t)v.W * 4, v.D, (size_t)v.P * 4, (size_t)v.W * 4, v.H,
                                          cudaMemcpyDeviceToHost, st));
    }
    GM_CUDA_TRY(cudaMemcpyAsync(d.host_state, a.st, sizeof(State), cudaMemcpyDeviceToHost, st));
    GM_CUDA_TRY(cudaStreamSynchronize(st));
    GM_CUDA_TRY(cudaGetLastError());
    if (d.host_state->status != GM_OK) {
        gm_set_error_msg("multigrid: singular coarse operator");
        return d.host_state->status;
    }
    return GM_OK;
}
