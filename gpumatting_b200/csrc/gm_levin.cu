// gm_levin.cu -- Levin matting Laplacian assembly on the GPU.
//
// No atomics: every entry is written once, by one thread.  Per pixel i and
// each of the 24 neighbours j of the 5x5 stencil, the window terms
//     (1 + (x_i - mu)^T (Sigma + eps/9 I)^-1 (x_j - mu)) / 9
// are summed over the 3x3 windows holding both (Matting.cu:79-189,
// matlab/getLevinLapRaster.m:22-62).  levin_sym_kernel goes by windows (one
// thread per window column, marching down); levin_ref_kernel gathers: a CTA
// stages a TW x TH pixel tile with a 2-pixel halo and the statistics of every
// window that touches it, then each thread sums its pixel's rows in window
// raster order.
//
// Two arithmetic modes:
//   levin_sym_kernel   FP64 throughout, rounded once to the store types
//                      (symmetric store + optional 25-band FP32 copy).
//   levin_ref_kernel   the reference's own float/double mix with IEEE
//                      round-to-nearest intrinsics and no FMA contraction,
//                      bit-identical to hostLevinLaplacian (Matting.cu:39-219).
#include <string.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "gm_internal.cuh"

int gm_note_status(int s);

namespace gm {

constexpr int TW = 32, TH = 8;
constexpr int NWIN = (TW + 2) * (TH + 2);

struct ImgView {
    const unsigned char* data;
    int format;
    size_t pitch;
};

__device__ __forceinline__ void load_rgb_d(const ImgView& im, int u, int v, double& r, double& g, double& b)
{
    if (im.format == GM_IMAGE_RGB8) {
        const unsigned char* p = im.data + (size_t)v * im.pitch + 3 * (size_t)u;
        r = (double)p[0] / 255.0;
        g = (double)p[1] / 255.0;
        b = (double)p[2] / 255.0;
    } else {
        const float4 q = reinterpret_cast<const float4*>(im.data + (size_t)v * im.pitch)[u];
        r = q.x; g = q.y; b = q.z;
    }
}

// ppm.h:325-327: channel / maxval in float (maxval = 255).
__device__ __forceinline__ void load_rgb_f(const ImgView& im, int u, int v, float& r, float& g, float& b)
{
    if (im.format == GM_IMAGE_RGB8) {
        const unsigned char* p = im.data + (size_t)v * im.pitch + 3 * (size_t)u;
        r = __fdiv_rn((float)p[0], 255.0f);
        g = __fdiv_rn((float)p[1], 255.0f);
        b = __fdiv_rn((float)p[2], 255.0f);
    } else {
        const float4 q = reinterpret_cast<const float4*>(im.data + (size_t)v * im.pitch)[u];
        r = q.x; g = q.y; b = q.z;
    }
}

struct ScribView {
    const unsigned char* map;
    size_t map_pitch;
    float gamma_value;
    const float* gamma_map;
    const float* s_map;
    int W;
};

// Matting.cu:205-216: 255 -> (gamma, b = gamma), 0 -> (gamma, b = 0), else
// (0, 0); or per-pixel weights and targets.  Returns whether gamma is added
// to the diagonal (the reference adds nothing on unknown pixels).
__device__ __forceinline__ bool scribble(const ScribView& s, int u, int v, float& gam, float& bv)
{
    if (s.gamma_map) {
        gam = s.gamma_map[(size_t)v * s.W + u];
        bv = s.s_map ? gam * s.s_map[(size_t)v * s.W + u] : 0.f;
        return true;
    }
    if (s.map) {
        const unsigned char c = s.map[(size_t)v * s.map_pitch + u];
        if (c == 255) { gam = s.gamma_value; bv = s.gamma_value; return true; }
        if (c == 0) { gam = s.gamma_value; bv = 0.f; return true; }
    }
    gam = 0.f;
    bv = 0.f;
    return false;
}

template <class T> __device__ __forceinline__ T from_double(double x);
template <> __device__ __forceinline__ float from_double<float>(double x) { return __double2float_rn(x); }
template <> __device__ __forceinline__ __half from_double<__half>(double x) { return __double2half(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_double<__nv_bfloat16>(double x) { return __double2bfloat16(x); }

struct SymOut {
    void* w;          // [12][H][pitch] in T
    float* w32;       // [12][H][pitch]
    float* gamma;     // [H][pitch]
    float* b;         // [H][pitch]
    int pitch;
    size_t plane;     // elements between planes of w / w32
    float* a25;       // optional [25][apitch]
    size_t apitch;
    float* b25;       // optional [N]
    float* d;         // [H][pitch] gamma + row sum of w
    float* d32;       // [H][pitch] gamma + row sum of w32; NULL: 25 bands only (w, w32, gamma, b, d unset)
};

// ---- FP64 assembly: one streaming pass over the image ----
//
// With S = sum of a window's 9 colours, D_i = 9 x_i - S and
// N = 9 sum(x x^T) - S S^T = 81 Sigma, a window's term of the pair (i, j) is
//     (1 + (x_i - mu)^T (Sigma + eps/9 I)^-1 (x_j - mu)) / 9
//         = (1 + e_i . D_j) / 9,     e_i = (N + 9 eps I)^-1 D_i,
// one solve per pixel of the window and one 3-vector product per pair: about
// 340 FP64 operations per pixel of the image (24 neighbours of 9 windows each
// on their own, with an FP64 division each, took 1,500).  Only the 12 upper
// couplings are formed.  Colours of an RGB8 image stay whole numbers
// (x = 0..255, eps scaled by 255^2), so S, N and D are exact.
//
// Thread t of a CTA owns the windows centred on column u0 - 1 + t and marches
// down the rows with the 9 colours of its window in registers.  Sums over the
// vertically neighbouring windows stay in registers; the horizontal ones
// (3 - |du| windows per pair) take 9 values per row through shared memory.
// The thread of column u finishes the couplings with du = -1, 0, 1 of pixel u,
// du = 2 of pixel u - 1 and du = -2 of pixel u + 1 (one window column only).
// The diagonal (the FP64 sum of exactly the stored weights) is formed in the same
// pass instead of in a second one that reads all planes again (84 B/px): the
// thread that finishes a coupling adds it to the sums of both its pixels, which
// lie in its own column or a neighbouring one, in this row or the two below, and
// hands the neighbours' sums over once per row.  The first
// rows of a run repeat the couplings of the two rows above it; runs are as
// long as one wave of CTAs allows.
//
// Measured with the FP16 store: 1080p RGB8 450 -> 114 us, 4096^2 4.3 -> 0.82 ms in a
// row, 0.95-1.05 where another kernel's data has to leave L2 first (88 B written
// per pixel are 28 and 225 us); FP32 store, 4001 x 2999: 2,400 -> 494 (RGB8), 550
// us (float).  Bound by instruction issue at 12 warps per SM (about 60 % of the
// slots, FP64 pipe 37 %).  Forms before: windows in shared memory 156 us
// (12 shared wavefronts per 32 pixels and window); all rounded couplings through a
// shared ring for the diagonal 122.
constexpr int kAT = 128;              // threads = window columns
constexpr int kAW = kAT - 2;          // output columns per CTA
constexpr int kAP = kAT + 4;          // row length in shared memory (two pad columns each side)
// CTAs per SM the registers are cut for.  A float image's 27 colours and 18 row
// sums in 64 bits do not fit 168 registers (1080p: 160 us with 3 CTAs per SM, 135
// with 2).  An RGB8 image's nearly do: 116 bytes a thread are spilled with a 2-byte
// store (152 with the 25 bands), 8 with an FP32 one.  The 12 warps are worth
// that: 122 us with 3 CTAs per SM and 135 with 2 before the diagonal's sums moved
// to registers (4 bytes spilled then), 114 since.
__host__ __device__ constexpr int asm_ctas(bool f32) { return f32 ? 2 : 3; }
constexpr int kMinRows = 2;

// Rows of the coupling rings (the 25-band output, whose lower bands repeat the
// couplings of rows above, and the low-precision weights of float images): couplings to the same row are read in the step that
// forms them, those to the next row one step later, to the second row two
// steps later.
__host__ __device__ constexpr int ring_base(int k) { return k <= 2 ? k - 1 : (k <= 7 ? 2 + 2 * (k - 3) : 12 + 3 * (k - 8)); }
__host__ __device__ constexpr int ring_len(int k) { return k <= 2 ? 1 : (k <= 7 ? 2 : 3); }
constexpr int kRingRows = 27;

// |n| < 2^31, given as n + 2^31, to double with one FP64 addition (the
// conversion instruction runs at a quarter of the FP64 rate).
__device__ __forceinline__ double biased_to_double(unsigned n)
{
    return __hiloint2double(0x43300000, (int)n) - 4503601774854144.0;  // 2^52 + 2^31
}

// What is added to the diagonal of N: e9 + rel sum(x x), with
// e9 = 9 eps.  A window of fewer than three independent colours has a singular
// N, and with eps = 0 (or too little to show beside N's entries in 64 bits) a
// pivot of zero, whose reciprocal makes the window NaN.  As much is added then as
// keeps every pivot positive in rounding, which gives the limit of small eps:
// colours of a window lie in the range of its N, and a flat window couples its
// pixels with 1/9.  RGB8: N is whole, at most 81 127.5^2 < 2^21, and the last pivot
// is at least e9 N_00 with an error of 2^-51 N_00 N_22: e9 = 2^-26 is 16 times that.
// Float: the sums err by up to 2^-49 of 9 sum(x x), 2^-47 is 4 times that; so
// little it changes nothing where eps counts, and it is left out from 1e-10 on.
struct Ridge {
    double e9, rel;
};
static Ridge ridge_for(double eps, bool f32img)
{
    if (!f32img) return {std::max(9.0 * eps * (255.0 * 255.0), std::ldexp(1.0, -26)), 0.0};
    return {std::max(9.0 * eps, 1e-60), eps < 1e-10 ? std::ldexp(9.0, -47) : 0.0};
}

template <class T, bool F32IMG, bool BANDS>
__global__ void __launch_bounds__(kAT, asm_ctas(F32IMG)) levin_sym_kernel(ImgView im, ScribView sc, Ridge ridge, int W,
                                                                       int H, int rows, SymOut o)
{
    constexpr bool kLow = sizeof(T) == 2;
    // Two sets of nine FP64 sums do not fit beside a float image's registers
    // (1080p: 148 us against 130): there the low-precision weights go through a
    // ring in shared memory and are summed from it.
    constexpr bool kLowRing = kLow && F32IMG;
    using Sum = typename std::conditional<F32IMG, double, int>::type;
    using Pix = typename std::conditional<F32IMG, float, int>::type;
    __shared__ double xch[9][kAP];
    __shared__ double sums[kLow && !kLowRing ? 4 : 2][kAP];  // this row's shares of the left and right columns' diagonals
    __shared__ float hi[BANDS ? kRingRows : 1][kAP];
    __shared__ T lo[kLowRing ? kRingRows : 1][kAP];
    const int t = threadIdx.x, c = t + 2, u = blockIdx.x * kAW - 1 + t;
    const int r0 = blockIdx.y * rows, r1 = min(r0 + rows, H), rs0 = max(r0 - 2, 0);
    const bool ok_col = u >= 1 && u <= W - 2;
    if (BANDS || kLowRing)
        for (int i = t; i < kRingRows * kAP; i += kAT) {
            if (BANDS) hi[i / kAP][i % kAP] = 0.f;
            if (kLowRing) lo[i / kAP][i % kAP] = T(0.f);
        }

    // Colours (u - 1, u, u + 1) of row v, zero outside the image and for columns
    // that are no window's centre.  (The zero factors of a window outside the image
    // do not make a float image's infinities and NaN zero: to the sides they are
    // left out here, below the image the couplings they reach are cut.)  With an
    // FP32 store a float image's three colours are loaded under a test each, which
    // the middle one's, hidden from the compiler, keeps apart: as one block of loads
    // they took the kernel from 562 to 715 us at 4001 x 2999 (550 this way).
    constexpr bool kByPixel = F32IMG && !kLow;
    const bool any = (kByPixel || ok_col) && H >= 3;
    int in[3] = {ok_col, ok_col, ok_col};
    if (kByPixel) asm volatile("" : "+r"(in[1]));
    auto fetch = [&](int v, Pix (&p)[9]) {
#pragma unroll
        for (int q = 0; q < 9; ++q) p[q] = 0;
        if (any && v >= 0 && v < H) {
            const unsigned char* row = im.data + (size_t)v * im.pitch;
#pragma unroll
            for (int b = 0; b < 3; ++b)
                if (!kByPixel || in[b]) {
                    if constexpr (F32IMG) {
                        const float4 q = reinterpret_cast<const float4*>(row)[u - 1 + b];
                        p[3 * b] = q.x; p[3 * b + 1] = q.y; p[3 * b + 2] = q.z;
                    } else {
                        const unsigned char* q = row + 3 * (ptrdiff_t)(u - 1 + b);
                        p[3 * b] = q[0]; p[3 * b + 1] = q[1]; p[3 * b + 2] = q[2];
                    }
                }
        }
    };
    // Row sums of the three colours and their six products.
    auto row_sums = [&](const Pix (&p)[9], Sum (&s)[9]) {
        int n = 3;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            s[a] = (Sum)p[a] + (Sum)p[3 + a] + (Sum)p[6 + a];
#pragma unroll
            for (int b = a; b < 3; ++b, ++n)
                s[n] = (Sum)p[a] * (Sum)p[b] + (Sum)p[3 + a] * (Sum)p[3 + b] + (Sum)p[6 + a] * (Sum)p[6 + b];
        }
    };

    Pix pa[9], pb[9], pc[9], pn[9];  // rows v - 1, v, v + 1 of the window, and the one after
    Sum sa[9], sb[9], sn[9];         // row sums of rows v - 1 and v
    fetch(rs0 - 2, pa);
    fetch(rs0 - 1, pb);
    fetch(rs0, pc);
    row_sums(pa, sa);
    row_sums(pb, sb);
    // Sums over the windows so far: rows v -> v + 1 (9 pairs of columns) and
    // within rows v and v + 1 (column pairs 01, 02, 12).
    double dn1[9], in0[3], in1[3];
#pragma unroll
    for (int n = 0; n < 9; ++n) dn1[n] = 0.0;
#pragma unroll
    for (int n = 0; n < 3; ++n) in0[n] = in1[n] = 0.0;
    // Diagonal sums of rows r, r + 1, r + 2 in the columns left of, at and right of
    // this thread's: of the FP32 weights, and of the low-precision ones.
    double d32[3][3] = {}, dlo[3][3] = {};
    const size_t plane = o.plane;
    T* wl = reinterpret_cast<T*>(o.w);
    const bool own_w = o.w != (void*)o.w32;  // an FP32 store may keep w apart from w32
    // Output columns: [first, first + kAW) of the image.
    const int first = blockIdx.x * kAW, last = min(first + kAW, W) - 1;
    const bool out_col = u >= first && u <= last;
    __syncthreads();

#pragma unroll F32IMG ? 1 : 2
    for (int v = rs0 - 1; v <= r1; ++v) {  // window centre row; finishes pixel row r = v - 1
        const int r = v - 1;
        fetch(v + 2, pn);
        const bool out = out_col && r >= r0;
        // the scribble's raw values, looked at only when the row is done
        float sc_g = 0.f, sc_s = 0.f;
        unsigned char sc_m = 128;
        if (out) {
            if (sc.gamma_map) {
                sc_g = sc.gamma_map[(size_t)r * W + u];
                if (sc.s_map) sc_s = sc.s_map[(size_t)r * W + u];
            } else if (sc.map) {
                sc_m = sc.map[(size_t)r * sc.map_pitch + u];
            }
        }
        row_sums(pc, sn);
        // --- window statistics and the factors of N + e9 I = L diag(d) L^T
        // (the error of a solve with them grows with the condition number,
        // that of the cofactors' inverse with its square); two divisions give
        // the three 1 / d.
        const bool ok = ok_col && v >= 1 && v <= H - 2;
        Sum s[9];
#pragma unroll
        for (int n = 0; n < 9; ++n) s[n] = sa[n] + sb[n] + sn[n];
        double N[6];
        if constexpr (F32IMG) {
            N[0] = fma(-s[0], s[0], 9.0 * s[3]); N[1] = fma(-s[0], s[1], 9.0 * s[4]); N[2] = fma(-s[0], s[2], 9.0 * s[5]);
            N[3] = fma(-s[1], s[1], 9.0 * s[6]); N[4] = fma(-s[1], s[2], 9.0 * s[7]); N[5] = fma(-s[2], s[2], 9.0 * s[8]);
        } else {
            const unsigned B = 0x80000000u;
            N[0] = biased_to_double(9 * s[3] - s[0] * s[0] + B); N[1] = biased_to_double(9 * s[4] - s[0] * s[1] + B);
            N[2] = biased_to_double(9 * s[5] - s[0] * s[2] + B); N[3] = biased_to_double(9 * s[6] - s[1] * s[1] + B);
            N[4] = biased_to_double(9 * s[7] - s[1] * s[2] + B); N[5] = biased_to_double(9 * s[8] - s[2] * s[2] + B);
        }
        double e9 = ridge.e9;
        if (F32IMG && ridge.rel > 0.0) e9 = fma(ridge.rel, (double)(s[3] + s[6] + s[8]), e9);
        const double s00 = N[0] + e9, s11 = N[3] + e9, s22 = N[5] + e9;
        const double c22 = fma(s00, s11, -N[1] * N[1]), c12 = fma(s00, N[4], -N[2] * N[1]),
                     c11 = fma(s00, s22, -N[2] * N[2]);
        const double ri = 1.0 / (s00 * c22), rc = ri * s00;  // 1 / c22 = rc
        const double i0 = ok ? ri * c22 : 0.0, i1 = ok ? s00 * rc : 0.0;
        const double l1 = ok ? N[1] * i0 : 0.0, l2 = ok ? N[2] * i0 : 0.0, l3 = ok ? c12 * rc : 0.0;
        const double i2 = ok ? s00 * (1.0 / fma(-c12, l3, c11)) : 0.0;
        const double one = ok ? 1.0 : 0.0;
        auto dev = [&](const Pix (&p)[9], int b, double (&d)[3]) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if constexpr (F32IMG) d[a] = fma(9.0, (double)p[3 * b + a], -s[a]);
                else d[a] = biased_to_double(9u * (unsigned)p[3 * b + a] + (0x80000000u - (unsigned)s[a]));
            }
        };
        auto solve = [&](const double (&d)[3], double (&e)[3]) {
            const double z1 = fma(-l1, d[0], d[1]), z2 = fma(-l3, z1, fma(-l2, d[0], d[2]));
            e[2] = i2 * z2;
            e[1] = fma(i1, z1, -l3 * e[2]);
            e[0] = fma(i0, d[0], -fma(l1, e[1], l2 * e[2]));
        };
        auto pair = [](double acc, const double (&e)[3], const double (&d)[3]) {
            return fma(e[0], d[0], fma(e[1], d[1], fma(e[2], d[2], acc)));
        };
        double da[3][3], db[3][3], dc[3][3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            dev(pa, b, da[b]);
            dev(pb, b, db[b]);
            dev(pc, b, dc[b]);
        }
        // --- pairs whose upper pixel is in row r: their last window
        double p2[9], p1[9], p0[3], e[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            solve(da[a], e);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                p2[3 * a + b] = pair(one, e, dc[b]);
                p1[3 * a + b] = pair(dn1[3 * a + b] + one, e, db[b]);
            }
            if (a == 0) {
                p0[0] = pair(in0[0] + one, e, da[1]);
                p0[1] = pair(in0[1] + one, e, da[2]);
            }
            if (a == 1) p0[2] = pair(in0[2] + one, e, da[2]);
        }
        if (F32IMG && r + 2 >= H) {  // couplings to rows below the image
#pragma unroll
            for (int n = 0; n < 9; ++n) {
                p2[n] = 0.0;
                if (r + 1 >= H) p1[n] = 0.0;
            }
        }
        // shares of the neighbouring columns' couplings: [9] planes, read from
        // t - 1 (0, 1, 4, 5) or t + 1 (2, 3, 6, 7, 8)
        xch[0][c] = p2[8]; xch[1][c] = p2[7]; xch[2][c] = p2[0]; xch[3][c] = p2[1];
        xch[4][c] = p1[8]; xch[5][c] = p1[7]; xch[6][c] = p1[0]; xch[7][c] = p1[1];
        xch[8][c] = p0[0];
        // --- pairs whose upper pixel is in row v or v + 1: sums to go on with
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            solve(db[a], e);
#pragma unroll
            for (int b = 0; b < 3; ++b) dn1[3 * a + b] = pair(one, e, dc[b]);
            if (a == 0) {
                in0[0] = pair(in1[0] + one, e, db[1]);
                in0[1] = pair(in1[1] + one, e, db[2]);
            }
            if (a == 1) in0[2] = pair(in1[2] + one, e, db[2]);
        }
        solve(dc[0], e);
        in1[0] = pair(one, e, dc[1]);
        in1[1] = pair(one, e, dc[2]);
        solve(dc[1], e);
        in1[2] = pair(one, e, dc[2]);
#pragma unroll
        for (int n = 0; n < 9; ++n) {
            pa[n] = pb[n]; pb[n] = pc[n]; pc[n] = pn[n];
            sa[n] = sb[n]; sb[n] = sn[n];
        }
        if (r < rs0) continue;
        __syncthreads();
        // --- finish the couplings of row r
        const int r2 = r & 1, r3 = r % 3;
        const bool row_out = r >= r0 && o.w32 != nullptr;
        const bool st[3] = {row_out && u > first && u <= last + 1, row_out && out_col, row_out && u >= first - 1 && u < last};
        float* w32 = o.w32 + (size_t)r * o.pitch + u;
        T* wlo = wl + (size_t)r * o.pitch + u;
        // x: column of the upper pixel less u; the lower one is du further, dv below
        auto finish = [&](int k, int x, double w9) {
            const int dv = (k + 2) / 5, du = k - 5 * dv;
            const double w = w9 * (1.0 / 9.0);
            const float wf = __double2float_rn(w);
            const int row = ring_base(k) + (dv == 0 ? 0 : (dv == 1 ? r2 : r3));
            if (BANDS) hi[row][c + x] = wf;
            const double wd = (double)wf;
            d32[0][1 + x] += wd;
            d32[dv][1 + x + du] += wd;
            if (st[x + 1]) w32[(size_t)(k - 1) * plane + x] = wf;
            if (kLow) {
                const T wt = from_double<T>(w);
                if (kLowRing) {
                    lo[row][c + x] = wt;
                } else {
                    const double wd2 = (double)Cvt<T>::to_f(wt);
                    dlo[0][1 + x] += wd2;
                    dlo[dv][1 + x + du] += wd2;
                }
                if (st[x + 1]) wlo[(size_t)(k - 1) * plane + x] = wt;
            } else if (own_w && st[x + 1]) {
                wlo[(size_t)(k - 1) * plane + x] = from_double<T>(w);
            }
        };
        finish(10, 0, xch[0][c - 1] + p2[4] + xch[2][c + 1]);
        finish(9, 0, xch[1][c - 1] + p2[3]);
        finish(11, 0, p2[5] + xch[3][c + 1]);
        finish(12, -1, p2[2]);
        finish(8, 1, p2[6]);
        finish(5, 0, xch[4][c - 1] + p1[4] + xch[6][c + 1]);
        finish(4, 0, xch[5][c - 1] + p1[3]);
        finish(6, 0, p1[5] + xch[7][c + 1]);
        finish(7, -1, p1[2]);
        finish(3, 1, p1[6]);
        finish(1, 0, p0[2] + xch[8][c + 1]);
        finish(2, -1, p0[1]);
        sums[0][c] = d32[0][0];
        sums[1][c] = d32[0][2];
        if (kLow && !kLowRing) {
            sums[2][c] = dlo[0][0];
            sums[3][c] = dlo[0][2];
        }
        const double own32 = d32[0][1], own = dlo[0][1];
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            d32[0][n] = d32[1][n]; d32[1][n] = d32[2][n]; d32[2][n] = 0.0;
            dlo[0][n] = dlo[1][n]; dlo[1][n] = dlo[2][n]; dlo[2][n] = 0.0;
        }
        __syncthreads();
        // --- diagonal of row r
        if (out) {
            const size_t gi = (size_t)r * o.pitch + u;
            // Matting.cu:205-216: 255 -> (gamma, b = gamma), 0 -> (gamma, b = 0)
            const bool mark = sc_m == 255 || sc_m == 0;
            const float gam = sc.gamma_map ? sc_g : (mark ? sc.gamma_value : 0.f);
            const float bv = sc.gamma_map ? (sc.s_map ? sc_g * sc_s : 0.f) : (sc_m == 255 ? sc.gamma_value : 0.f);
            const int r2b = r2 ^ 1, r3b = r3 == 2 ? 0 : r3 + 1;  // rows r - 1 (mod 2), r - 2 (mod 3)
            double s1 = 0.0;
            if (kLowRing) {
#pragma unroll
                for (int k = 1; k <= 12; ++k) {
                    const int dv = (k + 2) / 5, du = k - 5 * dv;
                    s1 += (double)Cvt<T>::to_f(lo[ring_base(k) + (dv == 0 ? 0 : (dv == 1 ? r2 : r3))][c]);
                    s1 += (double)Cvt<T>::to_f(lo[ring_base(k) + (dv == 0 ? 0 : (dv == 1 ? r2b : r3b))][c - du]);
                }
            } else if (kLow) {
                s1 = own + (sums[2][c + 1] + sums[3][c - 1]);
            }
            const double s32 = (double)gam + (own32 + (sums[0][c + 1] + sums[1][c - 1]));
            if (o.d32) {
                o.gamma[gi] = gam;
                o.b[gi] = bv;
                o.d[gi] = __double2float_rn(kLow ? (double)gam + s1 : s32);
                o.d32[gi] = __double2float_rn(s32);
            }
            if (BANDS) {
                const size_t i = (size_t)r * W + u;
                double rs = 0.0;
#pragma unroll
                for (int k = -12; k <= 12; ++k) {
                    if (k == 0) continue;
                    const int ka = k < 0 ? -k : k, dv = (ka + 2) / 5, du = ka - 5 * dv;
                    const int row = ring_base(ka) + (dv == 0 ? 0 : (dv == 1 ? (k < 0 ? r2b : r2) : (k < 0 ? r3b : r3)));
                    const float a = -(k < 0 ? hi[row][c - du] : hi[row][c]);
                    o.a25[(size_t)(12 + k) * o.apitch + i] = a;
                    rs -= (double)a;
                }
                o.a25[(size_t)12 * o.apitch + i] = __double2float_rn(rs + (double)gam);
                if (o.b25) o.b25[i] = bv;
            }
        }
    }
}

// ---- reference arithmetic (Matting.cu:79-218), bit-exact ----
struct RefWin {
    float mx, my, mz;
    double d11, d12, d13, d22, d23, d33, cdet;
};

__global__ void __launch_bounds__(TW * TH) levin_ref_kernel(ImgView im, ScribView sc, float lambda, int W, int H,
                                                            float* a, size_t apitch, float* bout)
{
    __shared__ float col[TH + 4][TW + 4][3];
    __shared__ RefWin win[NWIN];
    const int u0 = blockIdx.x * TW, v0 = blockIdx.y * TH;
    const int tid = threadIdx.x;
    for (int t = tid; t < (TH + 4) * (TW + 4); t += blockDim.x) {
        const int x = t % (TW + 4), y = t / (TW + 4);
        const int u = u0 - 2 + x, v = v0 - 2 + y;
        float r = 0, g = 0, b = 0;
        if (u >= 0 && u < W && v >= 0 && v < H) load_rgb_f(im, u, v, r, g, b);
        col[y][x][0] = r; col[y][x][1] = g; col[y][x][2] = b;
    }
    __syncthreads();
    for (int t = tid; t < NWIN; t += blockDim.x) {
        const int wx = t % (TW + 2), wy = t / (TW + 2);
        const int cu = u0 - 1 + wx, cv = v0 - 1 + wy;
        if (cu < 1 || cu > W - 2 || cv < 1 || cv > H - 2) continue;
        float mx = 0.f, my = 0.f, mz = 0.f;
        double c11 = 0, c12 = 0, c13 = 0, c22 = 0, c23 = 0, c33 = 0;
        for (int q = 0; q < 9; ++q) {  // Matting.cu:98-113, raster order
            const float* p = col[wy + q / 3][wx + q % 3];
            mx = __fadd_rn(mx, p[0]); my = __fadd_rn(my, p[1]); mz = __fadd_rn(mz, p[2]);
            c11 = __dadd_rn(c11, (double)__fmul_rn(p[0], p[0]));
            c12 = __dadd_rn(c12, (double)__fmul_rn(p[0], p[1]));
            c13 = __dadd_rn(c13, (double)__fmul_rn(p[0], p[2]));
            c22 = __dadd_rn(c22, (double)__fmul_rn(p[1], p[1]));
            c23 = __dadd_rn(c23, (double)__fmul_rn(p[1], p[2]));
            c33 = __dadd_rn(c33, (double)__fmul_rn(p[2], p[2]));
        }
        mx = __fdiv_rn(mx, 9.0f); my = __fdiv_rn(my, 9.0f); mz = __fdiv_rn(mz, 9.0f);
        const double l9 = (double)__fdiv_rn(lambda, 9.0f);
        c11 = __dadd_rn(__dsub_rn(__ddiv_rn(c11, 9.0), (double)__fmul_rn(mx, mx)), l9);
        c12 = __dsub_rn(__ddiv_rn(c12, 9.0), (double)__fmul_rn(mx, my));
        c13 = __dsub_rn(__ddiv_rn(c13, 9.0), (double)__fmul_rn(mx, mz));
        c22 = __dadd_rn(__dsub_rn(__ddiv_rn(c22, 9.0), (double)__fmul_rn(my, my)), l9);
        c23 = __dsub_rn(__ddiv_rn(c23, 9.0), (double)__fmul_rn(my, mz));
        c33 = __dadd_rn(__dsub_rn(__ddiv_rn(c33, 9.0), (double)__fmul_rn(mz, mz)), l9);
        // Matting.cu:130-137, left to right
        const double t1 = __dmul_rn(__dmul_rn(c11, c22), c33);
        const double t2 = __dmul_rn(__dmul_rn(c12, c23), c13);
        const double t3 = __dmul_rn(__dmul_rn(c13, c12), c23);
        const double t4 = __dmul_rn(__dmul_rn(c13, c22), c13);
        const double t5 = __dmul_rn(__dmul_rn(c12, c12), c33);
        const double t6 = __dmul_rn(__dmul_rn(c11, c23), c23);
        RefWin w;
        w.cdet = __dsub_rn(__dsub_rn(__dsub_rn(__dadd_rn(__dadd_rn(t1, t2), t3), t4), t5), t6);
        w.d11 = __dsub_rn(__dmul_rn(c33, c22), __dmul_rn(c23, c23));
        w.d12 = __dsub_rn(__dmul_rn(c13, c23), __dmul_rn(c33, c12));
        w.d13 = __dsub_rn(__dmul_rn(c23, c12), __dmul_rn(c22, c13));
        w.d22 = __dsub_rn(__dmul_rn(c33, c11), __dmul_rn(c13, c13));
        w.d23 = __dsub_rn(__dmul_rn(c12, c13), __dmul_rn(c23, c11));
        w.d33 = __dsub_rn(__dmul_rn(c22, c11), __dmul_rn(c12, c12));
        w.mx = mx; w.my = my; w.mz = mz;
        win[t] = w;
    }
    __syncthreads();
    const int lx = tid % TW, ly = tid / TW;
    const int u = u0 + lx, v = v0 + ly;
    if (u >= W || v >= H) return;
    float acc[25];
#pragma unroll
    for (int k = 0; k < 25; ++k) acc[k] = 0.f;
    const float* xi = col[ly + 2][lx + 2];
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int cu = u + dx, cv = v + dy;
            if (cu < 1 || cu > W - 2 || cv < 1 || cv > H - 2) continue;
            const RefWin& w = win[(ly + 1 + dy) * (TW + 2) + (lx + 1 + dx)];
            const float rx = __fsub_rn(xi[0], w.mx), ry = __fsub_rn(xi[1], w.my), rz = __fsub_rn(xi[2], w.mz);
            // Matting.cu:151-153
            const float wx = __double2float_rn(__ddiv_rn(
                __dadd_rn(__dadd_rn(__dmul_rn(w.d11, (double)rx), __dmul_rn(w.d12, (double)ry)), __dmul_rn(w.d13, (double)rz)),
                w.cdet));
            const float wy = __double2float_rn(__ddiv_rn(
                __dadd_rn(__dadd_rn(__dmul_rn(w.d12, (double)rx), __dmul_rn(w.d22, (double)ry)), __dmul_rn(w.d23, (double)rz)),
                w.cdet));
            const float wz = __double2float_rn(__ddiv_rn(
                __dadd_rn(__dadd_rn(__dmul_rn(w.d13, (double)rx), __dmul_rn(w.d23, (double)ry)), __dmul_rn(w.d33, (double)rz)),
                w.cdet));
#pragma unroll
            for (int qy = -1; qy <= 1; ++qy) {
#pragma unroll
                for (int qx = -1; qx <= 1; ++qx) {
                    const int ju = dx + qx, jv = dy + qy;
                    const float* xj = col[ly + 2 + jv][lx + 2 + ju];
                    const float sx = __fsub_rn(xj[0], w.mx), sy = __fsub_rn(xj[1], w.my), sz = __fsub_rn(xj[2], w.mz);
                    // Matting.cu:177
                    const float t = __fadd_rn(__fadd_rn(__fadd_rn(1.0f, __fmul_rn(wx, sx)), __fmul_rn(wy, sy)),
                                              __fmul_rn(wz, sz));
                    const float neg = __fdiv_rn(-t, 9.0f);
                    acc[12 + ju + 5 * jv] = __fadd_rn(acc[12 + ju + 5 * jv], neg);
                }
            }
        }
    }
    // Matting.cu:192-216
    double rs = 0.0;
#pragma unroll
    for (int k = 0; k < 25; ++k) rs = __dadd_rn(rs, (double)acc[k]);
    float diag = __double2float_rn(__dsub_rn((double)acc[12], rs));
    float gam, bv;
    if (scribble(sc, u, v, gam, bv)) diag = __fadd_rn(diag, gam);
    acc[12] = diag;
    const size_t i = (size_t)v * W + u;
#pragma unroll
    for (int k = 0; k < 25; ++k) a[(size_t)k * apitch + i] = acc[k];
    if (bout) bout[i] = bv;
}

// d_i = gamma_i + sum of the affinities of row i as stored (upper planes at
// i, lower ones at the neighbour), summed in FP64 and rounded once, for the
// low-precision planes (d) and the FP32 planes (d32).
template <class T>
__global__ void levin_diag_kernel(const T* __restrict__ w, const float* __restrict__ w32,
                                  const float* __restrict__ gamma, float* d, float* d32, int W, int H, int pitch,
                                  size_t plane)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (u >= W) return;
    const size_t i = (size_t)v * pitch + u;
    double s = gamma[i], s32 = gamma[i];
#pragma unroll
    for (int k = 1; k <= 12; ++k) {
        const int dv = (k + 2) / 5, du = k - 5 * dv;
        s += (double)Cvt<T>::to_f(w[(k - 1) * plane + i]);
        s32 += (double)w32[(k - 1) * plane + i];
        const int ul = u - du, vl = v - dv;
        if (ul >= 0 && ul < W && vl >= 0) {
            const size_t j = (size_t)vl * pitch + ul;
            s += (double)Cvt<T>::to_f(w[(k - 1) * plane + j]);
            s32 += (double)w32[(k - 1) * plane + j];
        }
    }
    d[i] = __double2float_rn(s);
    d32[i] = __double2float_rn(s32);
}

template <class T, bool F32IMG, bool BANDS>
static int launch_sym3(const ImgView& im, const ScribView& sc, double eps, int W, int H, const SymOut& o, int sms,
                       cudaStream_t st)
{
    // One wave: every CTA that fits the GPU gets a run of rows of one strip.
    const int strips = (W + kAW - 1) / kAW;
    const int runs = max(1, asm_ctas(F32IMG) * sms / strips);
    const int rows = max(kMinRows, (H + runs - 1) / runs);
    const dim3 grid(strips, (H + rows - 1) / rows);
    levin_sym_kernel<T, F32IMG, BANDS><<<grid, kAT, 0, st>>>(im, sc, ridge_for(eps, F32IMG), W, H, rows, o);
    GM_CUDA_TRY(cudaGetLastError());
    return GM_OK;
}

template <class T>
static int launch_sym(const ImgView& im, const ScribView& sc, double eps, int W, int H, const SymOut& o, int sms,
                      cudaStream_t st)
{
    if (im.format == GM_IMAGE_RGBA32F)
        return o.a25 ? launch_sym3<T, true, true>(im, sc, eps, W, H, o, sms, st)
                     : launch_sym3<T, true, false>(im, sc, eps, W, H, o, sms, st);
    return o.a25 ? launch_sym3<T, false, true>(im, sc, eps, W, H, o, sms, st)
                 : launch_sym3<T, false, false>(im, sc, eps, W, H, o, sms, st);
}

// ---------------------------------------------------------------------------
// Adjoint of the assembly
// ---------------------------------------------------------------------------
// For a loss of alpha with lam = A^-1 dloss/dalpha (A is symmetric), every
// pair (i, j) the store couples has dloss/dw_ij = -(lam_i - lam_j)(alpha_i -
// alpha_j), and each window k adds w_ij += (1 + x_i^T K^-1 x_j) / 9 with
// x = I - mu_k and K = Sigma_k + eps/9 I.  Summing the pair gradients of one
// window collapses to two 3-vectors,
//   ka = K^-1 sum_a x_a alpha_a,   kl = K^-1 sum_a x_a lam_a,
// and pixel a of the window receives
//   dI_a += [(lam_a - mean lam) ka + (alpha_a - mean alpha) kl] / 9
//           - [(x_a . kl) ka + (x_a . ka) kl] / 81.
// The window statistics are recomputed from the image (the forward pass
// stores none).  FP64 throughout, one FP32 rounding per output.

// Scribble target s_i: the value b_i / gamma_i the forward pass encodes
// (0 where the pixel carries no scribble).
__device__ __forceinline__ float scribble_target(const ScribView& s, int u, int v)
{
    if (s.gamma_map) return s.s_map ? s.s_map[(size_t)v * s.W + u] : 0.f;
    if (s.map) return s.map[(size_t)v * s.map_pitch + u] == 255 ? 1.f : 0.f;
    return 0.f;
}

struct AdjOut {
    float* dimage;   // [H][dpitch] floats, `channels` per pixel
    size_t dpitch;
    int channels;    // 3 or 4 (the fourth is written as 0)
    float* dgamma;   // [H][W] or NULL
};

__global__ void __launch_bounds__(TW * TH) levin_adjoint_kernel(ImgView im, ScribView sc, double eps, int W, int H,
                                                                const float* __restrict__ lam,
                                                                const float* __restrict__ alpha, AdjOut o)
{
    __shared__ double col[TH + 4][TW + 4][3];
    __shared__ double sl[TH + 4][TW + 4];
    __shared__ double sa[TH + 4][TW + 4];
    __shared__ double wmu[NWIN][3];
    __shared__ double wka[NWIN][3];
    __shared__ double wkl[NWIN][3];
    __shared__ double wbar[NWIN][2];  // mean lam, mean alpha
    const int u0 = blockIdx.x * TW, v0 = blockIdx.y * TH;
    const int tid = threadIdx.x;
    for (int t = tid; t < (TH + 4) * (TW + 4); t += blockDim.x) {
        const int x = t % (TW + 4), y = t / (TW + 4);
        const int u = u0 - 2 + x, v = v0 - 2 + y;
        double r = 0, g = 0, b = 0, l = 0, a = 0;
        if (u >= 0 && u < W && v >= 0 && v < H) {
            load_rgb_d(im, u, v, r, g, b);
            l = lam[(size_t)v * W + u];
            a = alpha[(size_t)v * W + u];
        }
        col[y][x][0] = r; col[y][x][1] = g; col[y][x][2] = b;
        sl[y][x] = l;
        sa[y][x] = a;
    }
    __syncthreads();
    for (int t = tid; t < NWIN; t += blockDim.x) {
        const int wx = t % (TW + 2), wy = t / (TW + 2);
        const int cu = u0 - 1 + wx, cv = v0 - 1 + wy;
        if (cu < 1 || cu > W - 2 || cv < 1 || cv > H - 2) continue;
        double m[3] = {0, 0, 0}, c[6] = {0, 0, 0, 0, 0, 0}, lb = 0, ab = 0;
        for (int q = 0; q < 9; ++q) {
            const double* p = col[wy + q / 3][wx + q % 3];
            m[0] += p[0]; m[1] += p[1]; m[2] += p[2];
            c[0] += p[0] * p[0]; c[1] += p[0] * p[1]; c[2] += p[0] * p[2];
            c[3] += p[1] * p[1]; c[4] += p[1] * p[2]; c[5] += p[2] * p[2];
            lb += sl[wy + q / 3][wx + q % 3];
            ab += sa[wy + q / 3][wx + q % 3];
        }
        for (int a = 0; a < 3; ++a) m[a] /= 9.0;
        const double e9 = eps / 9.0;
        const double s00 = c[0] / 9.0 - m[0] * m[0] + e9, s01 = c[1] / 9.0 - m[0] * m[1],
                     s02 = c[2] / 9.0 - m[0] * m[2], s11 = c[3] / 9.0 - m[1] * m[1] + e9,
                     s12 = c[4] / 9.0 - m[1] * m[2], s22 = c[5] / 9.0 - m[2] * m[2] + e9;
        const double a00 = s11 * s22 - s12 * s12, a01 = s02 * s12 - s01 * s22, a02 = s01 * s12 - s02 * s11;
        const double a11 = s00 * s22 - s02 * s02, a12 = s02 * s01 - s00 * s12, a22 = s00 * s11 - s01 * s01;
        const double id = 1.0 / (s00 * a00 + s01 * a01 + s02 * a02);
        double va[3] = {0, 0, 0}, vl[3] = {0, 0, 0};
        for (int q = 0; q < 9; ++q) {
            const double* p = col[wy + q / 3][wx + q % 3];
            const double l = sl[wy + q / 3][wx + q % 3], a = sa[wy + q / 3][wx + q % 3];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const double x = p[e] - m[e];
                va[e] += x * a;
                vl[e] += x * l;
            }
        }
        wmu[t][0] = m[0]; wmu[t][1] = m[1]; wmu[t][2] = m[2];
        wka[t][0] = (a00 * va[0] + a01 * va[1] + a02 * va[2]) * id;
        wka[t][1] = (a01 * va[0] + a11 * va[1] + a12 * va[2]) * id;
        wka[t][2] = (a02 * va[0] + a12 * va[1] + a22 * va[2]) * id;
        wkl[t][0] = (a00 * vl[0] + a01 * vl[1] + a02 * vl[2]) * id;
        wkl[t][1] = (a01 * vl[0] + a11 * vl[1] + a12 * vl[2]) * id;
        wkl[t][2] = (a02 * vl[0] + a12 * vl[1] + a22 * vl[2]) * id;
        wbar[t][0] = lb / 9.0;
        wbar[t][1] = ab / 9.0;
    }
    __syncthreads();
    const int lx = tid % TW, ly = tid / TW;
    const int u = u0 + lx, v = v0 + ly;
    if (u >= W || v >= H) return;
    const double* xi = col[ly + 2][lx + 2];
    const double li = sl[ly + 2][lx + 2], ai = sa[ly + 2][lx + 2];
    double g[3] = {0, 0, 0};
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int cu = u + dx, cv = v + dy;
            if (cu < 1 || cu > W - 2 || cv < 1 || cv > H - 2) continue;
            const int t = (ly + 1 + dy) * (TW + 2) + (lx + 1 + dx);
            const double x0 = xi[0] - wmu[t][0], x1 = xi[1] - wmu[t][1], x2 = xi[2] - wmu[t][2];
            const double* ka = wka[t];
            const double* kl = wkl[t];
            const double xkl = x0 * kl[0] + x1 * kl[1] + x2 * kl[2];
            const double xka = x0 * ka[0] + x1 * ka[1] + x2 * ka[2];
            const double dl = (li - wbar[t][0]) / 9.0 - xkl / 81.0;
            const double da = (ai - wbar[t][1]) / 9.0 - xka / 81.0;
#pragma unroll
            for (int e = 0; e < 3; ++e) g[e] += dl * ka[e] + da * kl[e];
        }
    }
    float* out = o.dimage + (size_t)v * o.dpitch + (size_t)o.channels * u;
    out[0] = __double2float_rn(g[0]);
    out[1] = __double2float_rn(g[1]);
    out[2] = __double2float_rn(g[2]);
    if (o.channels == 4) out[3] = 0.f;
    if (o.dgamma) {
        const double s = scribble_target(sc, u, v);
        o.dgamma[(size_t)v * W + u] = __double2float_rn(li * (s - ai));
    }
}

// ---------------------------------------------------------------------------
// Restriction to the unknown pixels (hard constraints)
// ---------------------------------------------------------------------------
// Pixels with a scribble (or a positive gamma_map weight) are known: their
// value is fixed at the target s.  The store becomes the system on the
// unknown pixels with the known ones eliminated: for an unknown pixel i and a
// known neighbour j, w_ij (x_i - s_j) moves to the diagonal (gamma_i += w_ij)
// and the right-hand side (b_i += w_ij s_j); known rows become x_i = s_i;
// every coupling that touches a known pixel is removed.  Pass 1 gathers the
// new gamma and b per pixel (reads planes only), pass 2 zeroes the removed
// couplings, then the diagonal planes are recomputed.

__device__ __forceinline__ bool known_at(const ScribView& s, int u, int v, float& target)
{
    float gam, bv;
    const bool has = scribble(s, u, v, gam, bv);
    target = scribble_target(s, u, v);
    return has && gam > 0.f;
}

__global__ void levin_restrict_gather_kernel(ScribView sc, const float* __restrict__ w32, float* gamma, float* b,
                                             int W, int H, int pitch, size_t plane)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (u >= W) return;
    const size_t i = (size_t)v * pitch + u;
    float si;
    if (known_at(sc, u, v, si)) {
        gamma[i] = 1.f;
        b[i] = si;
        return;
    }
    double g = gamma[i], bb = b[i];
#pragma unroll
    for (int k = 1; k <= 12; ++k) {
        const int dv = (k + 2) / 5, du = k - 5 * dv;
        const int uf = u + du, vf = v + dv;  // upper partner: coupling stored at i
        float sj;
        if (uf >= 0 && uf < W && vf < H && known_at(sc, uf, vf, sj)) {
            const double w = w32[(size_t)(k - 1) * plane + i];
            g += w;
            bb += w * (double)sj;
        }
        const int ul = u - du, vl = v - dv;  // lower partner: coupling stored at the partner
        if (ul >= 0 && ul < W && vl >= 0 && known_at(sc, ul, vl, sj)) {
            const double w = w32[(size_t)(k - 1) * plane + (size_t)vl * pitch + ul];
            g += w;
            bb += w * (double)sj;
        }
    }
    gamma[i] = __double2float_rn(g);
    b[i] = __double2float_rn(bb);
}

template <class T>
__global__ void levin_restrict_cut_kernel(ScribView sc, T* w, float* w32, int W, int H, int pitch, size_t plane)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (u >= W) return;
    const size_t i = (size_t)v * pitch + u;
    float t;
    const bool ki = known_at(sc, u, v, t);
#pragma unroll
    for (int k = 1; k <= 12; ++k) {
        const int dv = (k + 2) / 5, du = k - 5 * dv;
        const int uf = u + du, vf = v + dv;
        const bool kj = uf >= 0 && uf < W && vf < H && known_at(sc, uf, vf, t);
        if (ki || kj) {
            w[(size_t)(k - 1) * plane + i] = from_double<T>(0.0);
            w32[(size_t)(k - 1) * plane + i] = 0.f;
        }
    }
}

}  // namespace gm

using namespace gm;

static int make_views(const gm_image* im, const gm_scribbles* sc, int W, ImgView& iv, ScribView& sv)
{
    if (!im || !im->data) { gm_set_error_msg("image is NULL"); return GM_ERR_INVALID; }
    if (im->format != GM_IMAGE_RGB8 && im->format != GM_IMAGE_RGBA32F) { gm_set_error_msg("unknown image format"); return GM_ERR_INVALID; }
    iv.data = (const unsigned char*)im->data;
    iv.format = im->format;
    iv.pitch = im->pitch_bytes;
    if (im->format == GM_IMAGE_RGBA32F && (((uintptr_t)im->data & 15) || (im->pitch_bytes & 15))) {
        gm_set_error_msg("RGBA32F image must be 16-byte aligned with a 16-byte multiple pitch");
        return GM_ERR_INVALID;
    }
    memset(&sv, 0, sizeof(sv));
    sv.W = W;
    if (sc) {
        sv.map = sc->map;
        sv.map_pitch = sc->map_pitch ? sc->map_pitch : (size_t)W;
        sv.gamma_value = sc->gamma_value;
        sv.gamma_map = sc->gamma_map;
        sv.s_map = sc->s_map;
    }
    return GM_OK;
}

extern "C" int gm_levin_store_alloc(gm_levin_store* st, int W, int H, int precision)
{
    if (!st || W <= 0 || H <= 0) { gm_set_error_msg("bad store size"); return GM_ERR_INVALID; }
    if (precision < GM_PREC_FP32 || precision > GM_PREC_BF16) { gm_set_error_msg("bad precision"); return GM_ERR_INVALID; }
    memset(st, 0, sizeof(*st));
    st->W = W;
    st->H = H;
    st->pitch = (W + 7) & ~7;
    st->precision = precision;
    const size_t plane = (size_t)H * st->pitch;
    const size_t esz = precision == GM_PREC_FP32 ? 4 : 2;
    const size_t lo_bytes = precision == GM_PREC_FP32 ? 0 : ((12 * plane * esz + 255) & ~(size_t)255);
    const size_t b32 = (12 * plane * 4 + 255) & ~(size_t)255;
    const size_t b1 = (plane * 4 + 255) & ~(size_t)255;
    unsigned char* m = nullptr;
    if (cudaMalloc((void**)&m, lo_bytes + b32 + 4 * b1) != cudaSuccess) {
        cudaGetLastError();
        gm_set_error_msg("store allocation failed");
        return GM_ERR_NOMEM;
    }
    st->w32 = (float*)m;
    st->w = precision == GM_PREC_FP32 ? (void*)m : (void*)(m + b32);
    st->gamma = (float*)(m + b32 + lo_bytes);
    st->b = (float*)(m + b32 + lo_bytes + b1);
    st->d = (float*)(m + b32 + lo_bytes + 2 * b1);
    st->d32 = (float*)(m + b32 + lo_bytes + 3 * b1);
    st->owns = 1;
    return GM_OK;
}

extern "C" int gm_levin_store_free(gm_levin_store* st)
{
    if (!st) return GM_ERR_INVALID;
    // cudaFree waits for every use of the block by itself, on any device and
    // while other threads capture; a pool's free would need a wait of the
    // device, which a capture anywhere on it refuses and is broken by.
    if (st->owns && st->w32) cudaFree(st->w32);
    memset(st, 0, sizeof(*st));
    return GM_OK;
}

extern "C" int gm_levin_assemble(gm_levin_store* st, const gm_image* im, const gm_scribbles* sc, double eps,
                                 BandedMatrix* bands25, float* b25, void* stream)
{
    if (!st || !st->w || !st->w32 || !st->gamma || !st->b || !st->d || !st->d32) {
        gm_set_error_msg("store not allocated");
        return GM_ERR_INVALID;
    }
    if (!(eps >= 0.0)) { gm_set_error_msg("eps must be >= 0"); return GM_ERR_INVALID; }
    int sms = 0;
    GM_TRY(gm_check_device(&sms));
    ImgView iv;
    ScribView sv;
    GM_TRY(make_views(im, sc, st->W, iv, sv));
    SymOut o;
    memset(&o, 0, sizeof(o));
    o.w = st->w;
    o.w32 = st->w32;
    o.gamma = st->gamma;
    o.b = st->b;
    o.d = st->d;
    o.d32 = st->d32;
    o.pitch = st->pitch;
    o.plane = st->plane_stride ? st->plane_stride : (size_t)st->H * st->pitch;
    if (bands25) {
        if (!bands25->a || bands25->nbands != 25 || bands25->rows != st->W * st->H ||
            bands25->apitch < (size_t)bands25->rows) {
            gm_set_error_msg("bands25 must be a device BandedMatrix of 25 bands and W*H rows");
            return GM_ERR_INVALID;
        }
        o.a25 = bands25->a;
        o.apitch = bands25->apitch;
        o.b25 = b25;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (st->precision == GM_PREC_FP16) return launch_sym<__half>(iv, sv, eps, st->W, st->H, o, sms, s);
    if (st->precision == GM_PREC_BF16) return launch_sym<__nv_bfloat16>(iv, sv, eps, st->W, st->H, o, sms, s);
    return launch_sym<float>(iv, sv, eps, st->W, st->H, o, sms, s);
}

extern "C" int gm_levin_assemble_bands25(float* a, size_t apitch, float* b, const gm_image* im,
                                         const gm_scribbles* sc, double eps, int W, int H, int arithmetic,
                                         void* stream)
{
    if (!a || W <= 0 || H <= 0 || apitch < (size_t)W * H) { gm_set_error_msg("bad 25-band output"); return GM_ERR_INVALID; }
    int sms = 0;
    GM_TRY(gm_check_device(&sms));
    ImgView iv;
    ScribView sv;
    GM_TRY(make_views(im, sc, W, iv, sv));
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid((W + TW - 1) / TW, (H + TH - 1) / TH);
    if (arithmetic == GM_ASSEMBLY_REFERENCE) {
        levin_ref_kernel<<<grid, TW * TH, 0, s>>>(iv, sv, (float)eps, W, H, a, apitch, b);
    } else {
        if (!(eps >= 0.0)) { gm_set_error_msg("eps must be >= 0"); return GM_ERR_INVALID; }
        SymOut o;
        memset(&o, 0, sizeof(o));
        o.a25 = a;
        o.apitch = apitch;
        o.b25 = b;
        return launch_sym<float>(iv, sv, eps, W, H, o, sms, s);
    }
    GM_CUDA_TRY(cudaGetLastError());
    return GM_OK;
}

// Image and scribble-weight gradients from lam and alpha (both [H][W] floats
// on the device).  Used by gm_levin_adjoint after its lam solve.
int gm_levin_adjoint_grads(const gm_image* im, const gm_scribbles* sc, double eps, int W, int H,
                           const float* lam, const float* alpha, float* dimage, size_t dimage_pitch,
                           int dimage_channels, float* dgamma, cudaStream_t stream)
{
    if (W <= 0 || H <= 0 || !lam || !alpha || !dimage) { gm_set_error_msg("adjoint: bad arguments"); return GM_ERR_INVALID; }
    if (dimage_channels != 3 && dimage_channels != 4) { gm_set_error_msg("adjoint: dimage_channels must be 3 or 4"); return GM_ERR_INVALID; }
    if (dimage_pitch < (size_t)dimage_channels * W) { gm_set_error_msg("adjoint: dimage_pitch below channels * W"); return GM_ERR_INVALID; }
    if (!(eps >= 0.0)) { gm_set_error_msg("eps must be >= 0"); return GM_ERR_INVALID; }
    ImgView iv;
    ScribView sv;
    GM_TRY(make_views(im, sc, W, iv, sv));
    AdjOut o;
    o.dimage = dimage;
    o.dpitch = dimage_pitch;
    o.channels = dimage_channels;
    o.dgamma = dgamma;
    dim3 grid((W + TW - 1) / TW, (H + TH - 1) / TH);
    levin_adjoint_kernel<<<grid, TW * TH, 0, stream>>>(iv, sv, eps, W, H, lam, alpha, o);
    GM_CUDA_TRY(cudaGetLastError());
    return GM_OK;
}

extern "C" int gm_levin_restrict(gm_levin_store* st, const gm_scribbles* sc, void* stream)
{
    if (!st || !st->w || !st->w32 || !st->gamma || !st->b || !st->d || !st->d32 || !sc) {
        gm_set_error_msg("gm_levin_restrict: bad arguments");
        return GM_ERR_INVALID;
    }
    if (!sc->map && !sc->gamma_map) { gm_set_error_msg("gm_levin_restrict: no known pixels given"); return GM_ERR_INVALID; }
    GM_TRY(gm_check_device(nullptr));
    ScribView sv;
    memset(&sv, 0, sizeof(sv));
    sv.W = st->W;
    sv.map = sc->map;
    sv.map_pitch = sc->map_pitch ? sc->map_pitch : (size_t)st->W;
    sv.gamma_value = 1.f;  // only "known or not" matters here
    sv.gamma_map = sc->gamma_map;
    sv.s_map = sc->s_map;
    const int W = st->W, H = st->H, P = st->pitch;
    const size_t plane = st->plane_stride ? st->plane_stride : (size_t)H * P;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 g((W + 127) / 128, H);
    levin_restrict_gather_kernel<<<g, 128, 0, s>>>(sv, st->w32, st->gamma, st->b, W, H, P, plane);
    if (st->precision == GM_PREC_FP16)
        levin_restrict_cut_kernel<__half><<<g, 128, 0, s>>>(sv, (__half*)st->w, st->w32, W, H, P, plane);
    else if (st->precision == GM_PREC_BF16)
        levin_restrict_cut_kernel<__nv_bfloat16><<<g, 128, 0, s>>>(sv, (__nv_bfloat16*)st->w, st->w32, W, H, P, plane);
    else
        levin_restrict_cut_kernel<float><<<g, 128, 0, s>>>(sv, (float*)st->w, st->w32, W, H, P, plane);
    if (st->precision == GM_PREC_FP16)
        levin_diag_kernel<__half><<<g, 128, 0, s>>>((const __half*)st->w, st->w32, st->gamma, st->d, st->d32, W, H, P, plane);
    else if (st->precision == GM_PREC_BF16)
        levin_diag_kernel<__nv_bfloat16><<<g, 128, 0, s>>>((const __nv_bfloat16*)st->w, st->w32, st->gamma, st->d,
                                                           st->d32, W, H, P, plane);
    else
        levin_diag_kernel<float><<<g, 128, 0, s>>>((const float*)st->w, st->w32, st->gamma, st->d, st->d32, W, H, P, plane);
    GM_CUDA_TRY(cudaGetLastError());
    return GM_OK;
}
