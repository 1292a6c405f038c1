// Adjoint force path: exact forces and torques of the pair energy
// E = en_min + (en_max - en_min) * net(g(cloud)) instead of the reference's
// ten finite-difference evaluations (ForceEvaluator.py:86-112).
//
// One CTA works on tiles of 128 pairs with 256 threads; thread t handles pair
// p = t % 128 and the half h = t / 128 of the harmonics (and the same TMEM
// lane p in the tensor-core epilogues). Per tile:
//   1  stage the rotated body points of the pairs in shared memory;
//   2  descriptor forward (FP32): g = [sum_a f_n(a) | sum_m N_lm^2 A_{n,lm}^2];
//   3  net forward and backward on the tensor cores: every product is three
//      bf16 x bf16 -> fp32 MMAs (hi*hi + hi*lo + lo*hi of the bf16 splits of
//      activations and weights), accumulators in TMEM; gives dE/dg;
//   4  descriptor backward (FP32): the per-point quantities are recomputed
//      instead of stored (only the per-pair sums A stay in registers across the
//      net): dE/dA = 2 dE/dg_ang A, then per point
//      dE/dr_a = sum_n dE/df_n f_n'(d) rhat + sum_lm dE/dY_lm grad Y_lm;
//   5  F_pair = -sum_{a in i} dE/dp_a, T_i = -sum_{a in i} p_a x dE/dp_a,
//      T_j = -sum_{a in j} (p_a - t) x dE/dp_a (dE/dp_a = dE/dr_a minus the mean,
//      the centroid moving with every point), times (en_max - en_min), clipped
//      to [-100, 100] and scattered like the reference (ForceEvaluator.py:119-142).
// Nets: 1 to 3 hidden layers of width <= 64, D <= 64.
#include "descriptor.cuh"
#include "descriptor_direct.cuh"
#include "tcgen05.cuh"

namespace amlp {

__device__ unsigned int g_amlp_device_error = 0;
// Test hook (amlp_test_first_wait_limit): polls allowed to the first MMA-completion
// wait of every CTA of k_forces_adjoint and k_mlp_grad; -1 keeps the normal limit. 0
// makes that wait give up at once, which exercises the abort path without any fault
// (in k_mlp_pair 0 makes the teams give up before their first product).
__device__ int g_amlp_first_wait_limit = -1;

namespace {

constexpr int kAP = 128;          // pairs per tile of the fused kernel (MMA M)
constexpr int kAThreads = 2 * kAP;
// Pairs per tile of the wide path's descriptor kernels: two CTAs of 64 pairs on an
// SM, so that one's loads, staging and scatter run under the other's point loops
// (backward 1,376 -> 1,222 us at 60,001 cylinders against one CTA of 128).
constexpr int kDP = 64;
constexpr int kDThreads = 2 * kDP;
constexpr int kMaxHidden = 3;      // hidden layers of the fused kernel
constexpr int kMaxHiddenWide = 4;  // hidden layers of the wide path: layer_first + 3 (TheEnergyNet(150, 3, D))
constexpr int kWpad = 64;          // hidden widths padded to 64 in TMEM regions
constexpr uint32_t kErrMbarTimeout = 1u;
// Shared-memory row strides of per-pair arrays, odd so that the 32 pairs of a
// warp (thread = pair) hit 32 different banks.
constexpr int kGS = 49;           // descriptor partials / dE/dg rows (48 used)
constexpr int kPartStride = 13;   // gradient partial sums (12 used)

struct AdjNet {
    int nh;                              // hidden layers
    int act;
    int kin[kMaxHiddenWide + 1];         // padded input width of hidden layer k (multiple of 16)
    int nout[kMaxHiddenWide + 1];        // padded output width of hidden layer k (multiple of 16)
    int dims[kMaxHiddenWide + 2];        // true dims: D, h1, .., h_nh, 1
    long long woff[kMaxHiddenWide + 1];  // offset of W_k in the packed global weights (k = 0..nh)
    int wsm_off[kMaxHiddenWide];         // byte offset of W_k (hi) in the weight area; lo follows (the wide
                                         // path: in the pre-split global copy of the weights)
    int wsm_total;                       // bytes of the weight area
    int bias_off[kMaxHiddenWide + 1];    // float offsets of b_k in the fp32 parameter area; last = w_last
    int par_total;
    // the wide path's net kernels only (set by wide_net): row strides of the g and dE/dg rows, widest
    // hidden layer, TMEM columns of the product region, act'(z) as bits (ReLU),
    // shared-memory carve-up and whether the next tile's g rows are prefetched
    int g_ld, gp, wmax, zbw, relu_bits;
    int wbuf_off, par_off, eps_off, gbuf_off, prefetch_g, smem;
    // k_mlp_pair: 0 not taken, 1 both operand tiles in shared memory, 2 the first in TMEM
    int pair, pair_d, pair_tile, pair_wbuf, pair_par, pair_eps, pair_smem;
};

// Activation and its derivative from one exponential, for the tensor-core
// epilogues (the net there is accurate to about 1e-5 relative, so the fast
// exponential's few-ulp error does not show): tanh(z) = 1 - 2 / (1 + e^(2z)),
// tanh' = 1 - tanh^2; silu(z) = z s, silu' = s (1 + z (1 - s)), s = 1 / (1 + e^-z).
// The exponential and the reciprocal flush subnormals: where one occurs it is added
// to 1 or is a saturated derivative's factor, and every float gives the value that
// the general forms give, at less than half of their instructions.
template <int ACT>
__device__ __forceinline__ void act_pair(float z, float &f, float &df) {
    constexpr float kLog2e = 1.4426950408889634f;
    if (ACT == AMLP_ACT_RELU) {
        f = fmaxf(z, 0.0f);
        df = z > 0.0f ? 1.0f : 0.0f;
    } else if (ACT == AMLP_ACT_TANH) {
        const float t = fmaf(-2.0f, rcp_ftz(1.0f + exp2_ftz(z * (2.0f * kLog2e))), 1.0f);
        f = t;
        df = fmaf(-t, t, 1.0f);
    } else {
        const float sg = rcp_ftz(1.0f + exp2_ftz(-z * kLog2e));
        f = z * sg;
        df = sg * fmaf(z, 1.0f - sg, 1.0f);
    }
}

// Eight of them, one branch on the activation.
__device__ __forceinline__ void act8(int act, const float *z, float *f, float *df) {
    if (act == AMLP_ACT_RELU) {
#pragma unroll
        for (int k = 0; k < 8; ++k) act_pair<AMLP_ACT_RELU>(z[k], f[k], df[k]);
    } else if (act == AMLP_ACT_TANH) {
#pragma unroll
        for (int k = 0; k < 8; ++k) act_pair<AMLP_ACT_TANH>(z[k], f[k], df[k]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) act_pair<AMLP_ACT_SILU>(z[k], f[k], df[k]);
    }
}

// ---------------------------------------------------------------- harmonic halves
// The 24 harmonics of l = 1..4 split over the two threads of a pair by order m,
// twelve each: half 0 holds m = 0 and 1, half 1 holds m = 2, 3 and 4. Half 0 needs
// the polynomials in z and x, y themselves, half 1 the powers
// C_m + i S_m = (x + i y)^m and few polynomials, so neither runs recurrences that
// only the other uses, and both take about the same time. Split by index (l = 1, 2
// and part of 3 | the rest), half 1 ran every recurrence up to l = m = 4 while
// half 0's warps waited at the barrier.
//
// The radial functions are f_n = h (1 + T_n(x)) with h = fc / 2. The backward
// holds, per harmonic, the coefficients of q_k(x) = sum_n G_nk (1 + T_n(x)) in
// the basis 1, T_1, .., T_8, and forms neither f_n nor f_n' per point. Its
// harmonics carry the scale that makes their derivatives come out of the same
// few polynomials, with c3 = 5 z^2 - 1, c4 = z (7 z^2 - 3), c7 = 7 z^2 - 1:
//   m = 0: z, z^2/2 - 1/6, 5/3 z^3 - z, 7/4 z^4 - 3/2 z^2 + 3/20  (d/dz: 1, z, c3, c4)
//   m = 1: {x, y} times 1, z, c3, c4      (d/dz of the last three: 1, 10 z, 21 z^2 - 3)
//   m = 2: {C_2, S_2} times 1, z, c7      (d/dz: 0, 1, 14 z)
//   m = 3: {C_3, S_3} times 1, z;  m = 4: {C_4, S_4}
// The sums over harmonics run on pairs of them (fma.rn.f32x2): two multiply-adds
// per instruction at the same rate, which keeps the unrolled loops half as long.
//
// The FP32 pipe bounds both loops, with two warps per scheduler to fill it: a
// multiply-add of the 9 x 24 sums (108 per point and half forward, 204 backward)
// comes with about as many others. 131,072 cubes, fused kernel: 4.20 ms (5.02 with
// halves by index); 60,001 cylinders: descriptor forward 617 us (751), backward
// 1,160 us (1,594).
constexpr int kHalfK = 12;  // harmonics per half
constexpr int kHalfP = kHalfK / 2;
// Points per iteration of the forward's loop: four overlap one point's chain
// (load, square root, cosine, recurrences) with another's sums (60,001 cylinders: 617
// us against 669 with one); the fused kernel, whose code is longer, is faster with one
// (131,072 cubes: 4.20 ms against 4.23). The backward takes two (1,160 us against 1,203).
constexpr int kWideUnroll = 4, kFusedUnroll = 1, kBackwardUnroll = 2;

__host__ __device__ constexpr int half_l(int H, int kk) {
    constexpr int t[2][kHalfK] = {{1, 2, 3, 4, 1, 2, 3, 4, 1, 2, 3, 4}, {2, 3, 4, 2, 3, 4, 3, 4, 3, 4, 4, 4}};
    return t[H][kk];
}
__host__ __device__ constexpr int half_m(int H, int kk) {
    return H == 0 ? (kk < 4 ? 0 : 1) : (kk < 6 ? 2 : (kk < 10 ? 3 : 4));
}
__host__ __device__ constexpr bool half_sin(int H, int kk) {
    return H == 0 ? kk >= 8 : kk == 11 || kk == 8 || kk == 9 || (kk >= 3 && kk < 6);
}
// N_lm^2 = 2 (l - m)! / (l + m)! (1 for m = 0): the weight of a squared sum of Q_l^m {C_m, S_m},
// so that g[n][l] = sum_m N_lm^2 (sum_a f_n Q_l^m {C_m, S_m})^2.
__host__ __device__ constexpr float half_weight(int H, int kk) {
    const int l = half_l(H, kk), m = half_m(H, kk);
    if (m == 0) return 1.0f;
    double num = 2.0, den = 1.0;
    for (int v = 2; v <= l - m; ++v) num *= v;
    for (int v = 2; v <= l + m; ++v) den *= v;
    return (float)(num / den);
}
// Q_l^m {C_m, S_m} over the backward's harmonic.
__host__ __device__ constexpr float half_scale(int H, int kk) {
    constexpr float t[2][kHalfK] = {{1.0f, 3.0f, 1.5f, 2.5f, 1.0f, 3.0f, 1.5f, 2.5f, 1.0f, 3.0f, 1.5f, 2.5f},
                                    {3.0f, 15.0f, 7.5f, 3.0f, 15.0f, 7.5f, 15.0f, 105.0f, 15.0f, 105.0f, 105.0f, 105.0f}};
    return t[H][kk];
}

// Element kk of an array of pairs (kk a constant after unrolling).
__device__ __forceinline__ float &pick(float2 *v, int kk) { return kk & 1 ? v[kk >> 1].y : v[kk >> 1].x; }

// T_1 .. T_N of x, t[n] = T_n (t[0] unused).
template <int N>
__device__ __forceinline__ void chebyshev(float x, float *t) {
    const float x2 = x + x;
    t[1] = x;
    t[2] = fmaf(x2, x, -1.0f);
#pragma unroll
    for (int n = 3; n <= N; ++n) t[n] = fmaf(x2, t[n - 1], -t[n - 2]);
}

// The half's harmonics Q_l^m(z) {C_m, S_m} of the unit vector (x, y, z),
// Q_l^m = d^m P_l / dz^m by the recurrence in l (what a half does not use is
// never computed).
template <int H>
__device__ __forceinline__ void half_harmonics(float x, float y, float z, float (&Y)[kHalfK]) {
    constexpr int LM = 4;
    float C[LM + 1], S[LM + 1], Q[LM + 1][LM + 1];
    C[0] = 1.0f;
    S[0] = 0.0f;
#pragma unroll
    for (int m = 1; m <= LM; ++m) {
        C[m] = fmaf(x, C[m - 1], -y * S[m - 1]);
        S[m] = fmaf(x, S[m - 1], y * C[m - 1]);
    }
#pragma unroll
    for (int m = 0; m <= LM; ++m) {
#pragma unroll
        for (int l = m; l <= LM; ++l) {
            if (l == m) Q[l][m] = (float)dfact_odd(m);
            else if (l == m + 1) Q[l][m] = (float)(2 * m + 1) * z * Q[l - 1][m];
            else
                Q[l][m] = ((float)(2 * l - 1) * z * Q[l - 1][m] - (float)(l + m - 1) * Q[l - 2][m]) *
                          (1.0f / (float)(l - m));
        }
    }
#pragma unroll
    for (int kk = 0; kk < kHalfK; ++kk) {
        const int l = half_l(H, kk), m = half_m(H, kk);
        Y[kk] = m == 0 ? Q[l][0] : Q[l][m] * (half_sin(H, kk) ? S[m] : C[m]);
    }
}

// s plus the weighted squares of row n's sums over the half's harmonics k0 .. k1 - 1 of degree l.
template <int H>
__device__ __forceinline__ float add_squares(float2 *An, int l, int k0, int k1, float s) {
#pragma unroll
    for (int kk = 0; kk < kHalfK; ++kk)
        if (kk >= k0 && kk < k1 && half_l(H, kk) == l) s = fmaf(half_weight(H, kk) * pick(An, kk), pick(An, kk), s);
    return s;
}

// Forward of one half: A[n][k] = sum_a f_n(a) Y_k(a), kept in the caller's
// registers for the backward, and its share of the descriptor row gp[0..47]: half
// 0 the radial sums n = 0..5 and, per (n, l), its weighted squares; half 1 the
// radial sums n = 6..10 and the padding column. half_forward_finish adds half 1's
// squares. r holds the pair's 2 npts centred points (x, y, z each).
template <class Cfg, int H, int UNROLL>
__device__ __forceinline__ void half_forward(const float *r, int npts, float inv_rc, float *gp,
                                              float2 (&A)[Cfg::NA][kHalfP]) {
    static_assert(Cfg::LMAX == 4 && Cfg::K == 2 * kHalfK && Cfg::NA == 9 && Cfg::NR == 11, "hypers (10, 8, 4)");
    constexpr int NR = Cfg::NR, NA = Cfg::NA, NS = 6;  // radial sums split at n = NS
    constexpr int NT = H == 0 ? NA - 1 : NR - 1;       // Chebyshev polynomials this half needs
#pragma unroll
    for (int n = 0; n < NA; ++n)
#pragma unroll
        for (int k2 = 0; k2 < kHalfP; ++k2) A[n][k2] = make_float2(0.f, 0.f);
    float R[NR];
#pragma unroll
    for (int n = 0; n < NR; ++n) R[n] = 0.f;
#pragma unroll UNROLL
    for (int a = 2 * npts; a > 0; --a, r += 3) {
        const float rx = r[0], ry = r[1], rz = r[2];
        const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
        const float inv_d = rsqrt_ftz(d2);
        const float u = d2 * inv_d * inv_rc, um1 = u - 1.0f;
        // the hardware cosine (an absolute error of a few 1e-7 for the arguments here, far
        // below the tensor-core net's 1e-5)
        const float h = fmaf(0.25f, __cosf(3.14159265358979f * u), 0.25f);  // fc / 2
        float f[NT + 1], Y[kHalfK];
        chebyshev<NT>(fmaf(2.0f * um1, um1, -1.0f), f);
        half_harmonics<H>(rx * inv_d, ry * inv_d, rz * inv_d, Y);
#pragma unroll
        for (int n = 0; n <= NT; ++n) f[n] = n == 0 ? 2.0f * h : fmaf(h, f[n], h);
#pragma unroll
        for (int n = H == 0 ? 0 : NS; n < (H == 0 ? NS : NR); ++n) R[n] += f[n];
#pragma unroll
        for (int n = 0; n < NA; ++n)
#pragma unroll
            for (int k2 = 0; k2 < kHalfP; ++k2)
                A[n][k2] = fma2(make_float2(f[n], f[n]), make_float2(Y[2 * k2], Y[2 * k2 + 1]), A[n][k2]);
    }
#pragma unroll
    for (int n = H == 0 ? 0 : NS; n < (H == 0 ? NS : NR); ++n) gp[n] = R[n];
    if (H == 1) {
        gp[Cfg::D] = 0.f;
        return;
    }
#pragma unroll
    for (int n = 0; n < NA; ++n)
#pragma unroll
        for (int l = 1; l <= Cfg::LMAX; ++l) gp[NR + n * Cfg::LMAX + l - 1] = add_squares<H>(A[n], l, 0, kHalfK, 0.f);
}

// Half 1's weighted squares onto half 0's in the row gp (after a barrier). The
// squares of one (n, l) add up in the order of the index split, l = 1, 2 and the
// first four of l = 3 before the rest: the descriptor stays the same to the bit,
// and with it the branch a ReLU net takes and the slope of a saturated unit.
template <class Cfg>
__device__ __forceinline__ void half_forward_finish(float *gp, float2 (&A)[Cfg::NA][kHalfP]) {
#pragma unroll
    for (int n = 0; n < Cfg::NA; ++n) {
        float *g = gp + Cfg::NR + n * Cfg::LMAX;
        g[1] = add_squares<1>(A[n], 2, 0, kHalfK, g[1]);
        g[2] = add_squares<1>(A[n], 3, 0, 3, g[2]) + add_squares<1>(A[n], 3, 3, kHalfK, 0.f);
        g[3] = add_squares<1>(A[n], 4, 0, kHalfK, g[3]);
    }
}

// Backward of one half: given dE/dg (dg) and the forward sums A of this half
// (overwritten), the partial sums over the centred points r_a of dE/dr_a
// needed for the pair force and torques: sum_{a in i} G_a, sum_a G_a,
// sum_{a in i} r_a x G_a, sum_{a in j} r_a x G_a -> out[12] (the caller adds
// the centroid terms). Per point, with G_nk = dE/dA_nk,
//   phi = h sum_k q_k Y_k + h p  (p: the radial descriptor's polynomial, half 0),
//   dphi/dd = h' (sum_k q_k Y_k + p) + h x' (sum_n s_n T_n'(x)),  s_n = sum_k G_nk Y_k (+ dE/dg_n),
// the last sum by Clenshaw's recurrence on T_n' = n U_(n-1). The angular
// gradient is h sum_k q_k grad Y_k, assembled from the sums U, V (over the
// half's cos and sin harmonics of one order m, times their polynomial in z)
// and W, X (the same with its derivative):
//   gx = sum_m m (U C_(m-1) + V S_(m-1)), gy = sum_m m (V C_(m-1) - U S_(m-1)),
//   gz = sum_m W C_m + X S_m, sum_k q_k Y_k = sum_m U C_m + V S_m (m >= 1) and
//   x gx + y gy = sum_m m (U C_m + V S_m).
template <class Cfg, int H>
__device__ __forceinline__ void half_backward(const float *r, int npts, float inv_rc, const float *dg, float *out,
                                               float2 (&A)[Cfg::NA][kHalfP]) {
    constexpr int NR = Cfg::NR, NA = Cfg::NA;
    constexpr int NT = H == 0 ? NR - 1 : NA - 1;
#pragma unroll
    for (int kk = 0; kk < kHalfK; ++kk) {
        const float w2 = 2.0f * half_weight(H, kk) * half_scale(H, kk);
        float s = 0.f;
#pragma unroll
        for (int n = 0; n < NA; ++n) {
            float &a = pick(A[n], kk);
            a *= w2 * dg[NR + n * Cfg::LMAX + half_l(H, kk) - 1];
            s += a;
        }
        pick(A[0], kk) += s;  // coefficient of 1: sum_n G_nk, and T_0 = 1 once more for n = 0
    }
    float gr[NR];  // the same of the radial descriptor
    if (H == 0) {
        float s = 0.f;
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            gr[n] = dg[n];
            s += gr[n];
        }
        gr[0] += s;
    }
    float Si[3], Xi[3];
#pragma unroll 1  // the same code for both bodies: one set of sums, no branch per point
    for (int body = 0; body < 2; ++body) {
        float G[3] = {0, 0, 0}, X[3] = {0, 0, 0};
#pragma unroll kBackwardUnroll
        for (int a = npts; a > 0; --a, r += 3) {
            const float rx = r[0], ry = r[1], rz = r[2];
            const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
            const float inv_d = rsqrt_ftz(d2);
            const float x = rx * inv_d, y = ry * inv_d, z = rz * inv_d, z2 = z * z;
            const float u = d2 * inv_d * inv_rc, um1 = u - 1.0f;
            float sn, cs;
            __sincosf(3.14159265358979f * u, &sn, &cs);
            const float h = fmaf(0.25f, cs, 0.25f);                        // fc / 2
            const float hd = (-0.25f * 3.14159265358979f * inv_rc) * sn;    // dh/dd
            const float hdx = (4.0f * inv_rc) * um1 * h;                    // h dx/dd
            const float cx = fmaf(2.0f * um1, um1, -1.0f), cx2 = cx + cx;
            float t[NT + 1], Y[kHalfK], q[kHalfK], s[NA];
            chebyshev<NT>(cx, t);
            // the harmonics, and the polynomials and powers that the gradient needs too
            float c3 = 0.f, c4 = 0.f, c7 = 0.f;
            if (H == 0) {
                c3 = fmaf(5.0f, z2, -1.0f), c4 = z * fmaf(7.0f, z2, -3.0f);
                Y[0] = z;
                Y[1] = fmaf(0.5f, z2, -1.0f / 6.0f);
                Y[2] = z * fmaf(5.0f / 3.0f, z2, -1.0f);
                Y[3] = fmaf(z2, fmaf(1.75f, z2, -1.5f), 0.15f);
                Y[4] = x, Y[5] = x * z, Y[6] = x * c3, Y[7] = x * c4;
                Y[8] = y, Y[9] = y * z, Y[10] = y * c3, Y[11] = y * c4;
            } else {
                c7 = fmaf(7.0f, z2, -1.0f);
                const float C2 = fmaf(x, x, -y * y), S2 = (x + x) * y;
                const float C3 = fmaf(x, C2, -y * S2), S3 = fmaf(x, S2, y * C2);
                Y[0] = C2, Y[1] = C2 * z, Y[2] = C2 * c7;
                Y[3] = S2, Y[4] = S2 * z, Y[5] = S2 * c7;
                Y[6] = C3, Y[7] = C3 * z, Y[8] = S3, Y[9] = S3 * z;
                Y[10] = fmaf(C2, C2, -S2 * S2), Y[11] = (C2 + C2) * S2;
            }
#pragma unroll
            for (int k2 = 0; k2 < kHalfP; ++k2) {
                float2 v = A[0][k2];
#pragma unroll
                for (int n = 1; n < NA; ++n) v = fma2(A[n][k2], make_float2(t[n], t[n]), v);
                q[2 * k2] = v.x;
                q[2 * k2 + 1] = v.y;
            }
#pragma unroll
            for (int n = 1; n < NA; ++n) {
                float2 v = make_float2(H == 0 ? gr[n] : 0.f, 0.f);
#pragma unroll
                for (int k2 = 0; k2 < kHalfP; ++k2) v = fma2(A[n][k2], make_float2(Y[2 * k2], Y[2 * k2 + 1]), v);
                s[n] = v.x + v.y;
            }
            // sum_n s_n n U_(n-1)(cx), n descending
            float b1 = 0.f, b2 = 0.f;
            if (H == 0) {
                b2 = (float)(NR - 1) * gr[NR - 1];
                b1 = fmaf(cx2, b2, (float)(NR - 2) * gr[NR - 2]);
            }
#pragma unroll
            for (int n = NA - 1; n >= 1; --n) {
                const float b0 = fmaf(cx2, b1, fmaf((float)n, s[n], -b2));
                b2 = b1;
                b1 = b0;
            }
            float gx, gy, gz, e, phi;  // sum_k q_k grad Y_k, x gx + y gy, sum_k q_k Y_k (+ the radial polynomial)
            if (H == 0) {
                const float z10 = 10.0f * z, c21 = fmaf(21.0f, z2, -3.0f);
                gx = fmaf(q[7], c4, fmaf(q[6], c3, fmaf(q[5], z, q[4])));
                gy = fmaf(q[11], c4, fmaf(q[10], c3, fmaf(q[9], z, q[8])));
                const float W0 = fmaf(q[3], c4, fmaf(q[2], c3, fmaf(q[1], z, q[0])));
                const float W1 = fmaf(q[7], c21, fmaf(q[6], z10, q[5])), X1 = fmaf(q[11], c21, fmaf(q[10], z10, q[9]));
                gz = fmaf(x, W1, fmaf(y, X1, W0));
                e = fmaf(x, gx, y * gy);
                float p = gr[0];
#pragma unroll
                for (int n = 1; n < NR; ++n) p = fmaf(gr[n], t[n], p);
                phi = fmaf(q[0], Y[0], fmaf(q[1], Y[1], fmaf(q[2], Y[2], fmaf(q[3], Y[3], e)))) + p;
            } else {
                const float z14 = 14.0f * z, C2 = Y[0], S2 = Y[3], C3 = Y[6], S3 = Y[8];
                const float U2 = fmaf(q[2], c7, fmaf(q[1], z, q[0])), V2 = fmaf(q[5], c7, fmaf(q[4], z, q[3]));
                const float U3 = fmaf(q[7], z, q[6]), V3 = fmaf(q[9], z, q[8]);
                const float W2 = fmaf(q[2], z14, q[1]), X2 = fmaf(q[5], z14, q[4]);
                const float x2 = x + x, y2 = y + y, C23 = 3.0f * C2, S23 = 3.0f * S2, C34 = 4.0f * C3, S34 = 4.0f * S3;
                gx = fmaf(U2, x2, fmaf(V2, y2, fmaf(U3, C23, fmaf(V3, S23, fmaf(q[10], C34, q[11] * S34)))));
                gy = fmaf(V2, x2, fmaf(-U2, y2, fmaf(V3, C23, fmaf(-U3, S23, fmaf(q[11], C34, -q[10] * S34)))));
                gz = fmaf(W2, C2, fmaf(X2, S2, fmaf(q[7], C3, q[9] * S3)));
                const float w2 = fmaf(U2, C2, V2 * S2), w3 = fmaf(U3, C3, V3 * S3), w4 = fmaf(q[10], Y[10], q[11] * Y[11]);
                e = fmaf(4.0f, w4, fmaf(3.0f, w3, w2 + w2));
                phi = w2 + w3 + w4;
            }
            // dE/dr = phi' rhat + (h g - rhat (rhat . h g)) / d
            const float hi = h * inv_d;
            const float dot = fmaf(z, gz, e);
            const float c1 = fmaf(-dot, hi, fmaf(hd, phi, hdx * b1));
            const float Gx = fmaf(x, c1, gx * hi);
            const float Gy = fmaf(y, c1, gy * hi);
            const float Gz = fmaf(z, c1, gz * hi);
            G[0] += Gx;
            G[1] += Gy;
            G[2] += Gz;
            X[0] += ry * Gz - rz * Gy;
            X[1] += rz * Gx - rx * Gz;
            X[2] += rx * Gy - ry * Gx;
        }
        if (body == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) Si[k] = G[k], Xi[k] = X[k];
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                out[k] = Si[k];
                out[3 + k] = Si[k] + G[k];
                out[6 + k] = Xi[k];
                out[9 + k] = X[k];
            }
        }
    }
}

struct AdjShared {
    float *R;          // rotated body points, NP x rs (may alias the MLP operand area)
    char *ops;         // MLP operand area (bf16 hi/lo tiles)
    char *wts;         // weights (bf16 hi/lo), resident
    float *par;        // biases + last-layer weights (fp32)
    float *g;          // descriptor rows, then dE/dg, NP x kGS
    float *t;          // translations, NP x 3
    float *cen;        // centroids, NP x 3
    float *part;       // per-half gradient partial sums, 2 x NP x kPartStride
    float *eps;        // per-half energy partials, 2 x NP
    float *fd;         // per-pair F, T_i, T_j, NP x 9
    int *ij;           // pair indices, NP x 2
    float *pts;        // body points
    float4 *q;         // orientations of the tile's pairs, NP x 2 (i, j)
    float *psum;       // sum of the body points (body frame), 3
};

// Per-pair areas of a tile of NP pairs (the fused kernel's and the wide path's
// descriptor kernels'), taken from `base`.
template <int NP>
constexpr size_t pair_area_bytes() {
    return (size_t)NP * 4 * (8 + 3 + 3 + 2 + 2 + 2 * kPartStride + 9);
}
template <int NP>
__device__ __forceinline__ void take_pair_areas(AdjShared &S, char *base) {
    float *f = reinterpret_cast<float *>(base);
    S.q = reinterpret_cast<float4 *>(f);
    S.t = f + 8 * NP;
    S.cen = f + 11 * NP;
    S.eps = f + 14 * NP;
    S.ij = reinterpret_cast<int *>(f + 16 * NP);
    S.part = f + 18 * NP;
    S.fd = S.part + 2 * NP * kPartStride;
}

// Sum of the body-frame points into S.psum (one warp; call before a barrier).
__device__ __forceinline__ void body_point_sum(const AdjShared &S, int npts) {
    if (threadIdx.x < 32) {
        float v[3] = {0.f, 0.f, 0.f};
        for (int a = threadIdx.x; a < npts; a += 32)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] += S.pts[3 * a + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (threadIdx.x == 0)
#pragma unroll
            for (int k = 0; k < 3; ++k) S.psum[k] = v[k];
    }
}

// Activation tile of layer k in the operand area (hi at its base, lo after it).
// Only two are live at a time (the one an MMA reads and the one its epilogue
// writes), so the layers alternate between two buffers.
__device__ __forceinline__ char *op_tile(char *ops, int k) { return ops + (k & 1) * (2 * kAP * kWpad * 2); }

// A (128 x K) times B, three split terms, into TMEM columns at d_tmem.
// STEP_DESC: build the four descriptors of K-step 0 once and move only their
// start address (bits 0-13, in 16-byte units, below 2^14 for any shared-memory
// address) from step to step; otherwise build them per MMA. Measured: stepping
// is 0.4 % faster in the fused kernel (K <= 64) and 0.7 % slower in k_mlp_grad.
template <bool STEP_DESC>
__device__ __forceinline__ void mma3(uint32_t d_tmem, const char *a_hi, int K, const char *b_hi, size_t b_lo_off,
                                     int N, bool b_mn, int b_kstride /* bytes per K-step of 16 */, uint32_t b_lbo,
                                     uint32_t b_sbo) {
    const uint32_t idesc = tc::idesc_bf16(N, b_mn ? 1 : 0);
    const uint32_t a0 = tc::smem_u32(a_hi), a1 = a0 + (uint32_t)(kAP * K * 2);
    const uint32_t b0 = tc::smem_u32(b_hi), b1 = b0 + (uint32_t)b_lo_off;
    const uint32_t a_sbo = (uint32_t)K * 16;
    if constexpr (STEP_DESC) {
        const uint64_t da = tc::smem_desc(a0, 128, a_sbo), da1 = tc::smem_desc(a1, 128, a_sbo);
        const uint64_t db = tc::smem_desc(b0, b_lbo, b_sbo), db1 = tc::smem_desc(b1, b_lbo, b_sbo);
        for (int ks = 0; ks < K / 16; ++ks) {
            const uint64_t oa = (uint64_t)(ks * 16), ob = (uint64_t)((ks * b_kstride) >> 4);
            tc::mma_bf16(d_tmem, da + oa, db + ob, idesc, ks > 0 ? 1u : 0u);
            tc::mma_bf16(d_tmem, da + oa, db1 + ob, idesc, 1u);
            tc::mma_bf16(d_tmem, da1 + oa, db + ob, idesc, 1u);
        }
    } else {
        for (int ks = 0; ks < K / 16; ++ks) {
            const uint32_t ao = ks * 256, bo = ks * b_kstride;
            tc::mma_bf16(d_tmem, tc::smem_desc(a0 + ao, 128, a_sbo), tc::smem_desc(b0 + bo, b_lbo, b_sbo), idesc,
                         ks > 0 ? 1u : 0u);
            tc::mma_bf16(d_tmem, tc::smem_desc(a0 + ao, 128, a_sbo), tc::smem_desc(b1 + bo, b_lbo, b_sbo), idesc,
                         1u);
            tc::mma_bf16(d_tmem, tc::smem_desc(a1 + ao, 128, a_sbo), tc::smem_desc(b0 + bo, b_lbo, b_sbo), idesc,
                         1u);
        }
    }
}

// bf16 hi and lo of 8 values, rounded two at a time (one packed conversion per
// pair, round to nearest even): hi + lo == v to about 2^-16 relative.
__device__ __forceinline__ void split8(const float *v, uint4 &hi, uint4 &lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        const float2 hf = __bfloat1622float2(h2);
        const float2 r = fma2(hf, make_float2(-1.f, -1.f), make_float2(v[2 * k], v[2 * k + 1]));  // v - hi
        const __nv_bfloat162 l2 = __floats2bfloat162_rn(r.x, r.y);
        h[k] = *reinterpret_cast<const uint32_t *>(&h2);
        l[k] = *reinterpret_cast<const uint32_t *>(&l2);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Write 8 consecutive values of row p, columns c0..c0+7 into a K-major bf16
// hi/lo tile of width K.
__device__ __forceinline__ void store_split8(char *tile_hi, int K, int p, int c0, const float *v) {
    uint4 hi, lo;
    split8(v, hi, lo);
    const uint32_t off = tc::kmajor_offset(p, c0, K);
    *reinterpret_cast<uint4 *>(tile_hi + off) = hi;
    *reinterpret_cast<uint4 *>(tile_hi + kAP * K * 2 + off) = lo;
}

// The weights of a layer (N x K, row-major) as a zero-padded Np x Kp K-major bf16
// hi/lo operand: hi at `hi`, lo after it. Eight weights per thread and step
// (independent loads, 16-byte stores), `first` of `stride` threads.
// One weight per step, with a division and 2-byte stores each, took every block of
// the fused kernel 6 us: 83.6 us a pass over 1,000 cubes, 77.5 us so.
__device__ __forceinline__ void split_layer(const float *W, int N, int K, int Np, int Kp, char *hi, int first,
                                            int stride) {
    char *lo = hi + (size_t)Np * Kp * 2;
    const int per_row = Kp / 8;
    for (int c = first; c < Np * per_row; c += stride) {
        const int n = c / per_row, k0 = 8 * (c - n * per_row);
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = n < N && k0 + u < K ? W[(size_t)n * K + k0 + u] : 0.f;
        uint4 h, l;
        split8(v, h, l);
        const uint32_t off = tc::kmajor_offset(n, k0, Kp);
        *reinterpret_cast<uint4 *>(hi + off) = h;
        *reinterpret_cast<uint4 *>(lo + off) = l;
    }
}

// Centroid of pair q's cloud into S.cen from its orientations and translation
// (S.q, S.t): c = (R_i s + R_j s + npts t) / (2 npts), s the sum of the
// body-frame points. Called by the thread that wrote pair q's S.q and S.t.
__device__ __forceinline__ void store_centroid(const AdjShared &S, int q, int npts) {
    const float3 ps = make_float3(S.psum[0], S.psum[1], S.psum[2]);
    const float3 a = rotate_ref(S.q[2 * q], ps), b = rotate_ref(S.q[2 * q + 1], ps);
    const float inv = 1.0f / (float)(2 * npts), n = (float)npts;
    S.cen[3 * q] = fmaf(n, S.t[3 * q], a.x + b.x) * inv;
    S.cen[3 * q + 1] = fmaf(n, S.t[3 * q + 1], a.y + b.y) * inv;
    S.cen[3 * q + 2] = fmaf(n, S.t[3 * q + 2], a.z + b.z) * inv;
}

// Centred cloud points of the tile's pairs into S.R: row q holds body i's
// points R_i b_a - c, then body j's R_j b_a + t - c (c = S.cen). Thread
// (q, body) = (tid % NP, tid / NP) rotates all points of one body of one pair
// (body points broadcast from shared memory, rows of odd stride rs: no bank
// conflicts, no index divisions) with the matrix of q v q* for q = (w, u),
// (w^2 - |u|^2) I + 2 u u^T + 2 w [u]x, built once: 9 FMAs per point.
template <int NP>
__device__ __forceinline__ void rotate_tile(const AdjShared &S, int npts, int rs) {
    const int q = threadIdx.x & (NP - 1), body = threadIdx.x / NP;
    const float4 qq = S.q[2 * q + body];
    const float w = qq.x, x = qq.y, y = qq.z, z = qq.w;
    const float a0 = w * w - (x * x + y * y + z * z);
    const float m00 = fmaf(2.f * x, x, a0), m01 = 2.f * (x * y - w * z), m02 = 2.f * (x * z + w * y);
    const float m10 = 2.f * (x * y + w * z), m11 = fmaf(2.f * y, y, a0), m12 = 2.f * (y * z - w * x);
    const float m20 = 2.f * (x * z - w * y), m21 = 2.f * (y * z + w * x), m22 = fmaf(2.f * z, z, a0);
    const float ox = body ? S.t[3 * q] - S.cen[3 * q] : -S.cen[3 * q];
    const float oy = body ? S.t[3 * q + 1] - S.cen[3 * q + 1] : -S.cen[3 * q + 1];
    const float oz = body ? S.t[3 * q + 2] - S.cen[3 * q + 2] : -S.cen[3 * q + 2];
    float *dst = S.R + q * rs + body * 3 * npts;
    for (int a = 0; a < npts; ++a) {
        const float px = S.pts[3 * a], py = S.pts[3 * a + 1], pz = S.pts[3 * a + 2];
        dst[3 * a] = fmaf(m00, px, fmaf(m01, py, fmaf(m02, pz, ox)));
        dst[3 * a + 1] = fmaf(m10, px, fmaf(m11, py, fmaf(m12, pz, oy)));
        dst[3 * a + 2] = fmaf(m20, px, fmaf(m21, py, fmaf(m22, pz, oz)));
    }
}

// Torque sums about the body origins from those about the centroid:
// sum_{a in i} (r_a + c) x G_a = Xi + c x Si and
// sum_{a in j} (r_a + c - t) x G_a = Xj + (c - t) x (Sa - Si).
__device__ __forceinline__ void add_centroid_terms(const AdjShared &S, int q, const float *Si, const float *Sa,
                                                   float *Xi, float *Xj) {
    const float c[3] = {S.cen[3 * q], S.cen[3 * q + 1], S.cen[3 * q + 2]};
    const float e[3] = {c[0] - S.t[3 * q], c[1] - S.t[3 * q + 1], c[2] - S.t[3 * q + 2]};
    const float Sj[3] = {Sa[0] - Si[0], Sa[1] - Si[1], Sa[2] - Si[2]};
    Xi[0] += c[1] * Si[2] - c[2] * Si[1];
    Xi[1] += c[2] * Si[0] - c[0] * Si[2];
    Xi[2] += c[0] * Si[1] - c[1] * Si[0];
    Xj[0] += e[1] * Sj[2] - e[2] * Sj[1];
    Xj[1] += e[2] * Sj[0] - e[0] * Sj[2];
    Xj[2] += e[0] * Sj[1] - e[1] * Sj[0];
}

// Pair indices, orientations, translations and centroids of the tile's pairs
// p0 .. p0 + NP - 1 (past the last pair: that pair again), then their rotated,
// centred points into S.R.
template <int NP, bool MULTI>
__device__ __forceinline__ void load_pairs(const AdjShared &S, const float *pos, const float *quat, float L,
                                           const int *pairs, long long P, long long p0, int npts, int rs,
                                           const int *rep, const amlp_replica *rp) {
    const int tid = threadIdx.x;
    if (tid < NP) {
        long long pr = min(p0 + tid, P - 1);
        int i = pairs[2 * pr], j = pairs[2 * pr + 1];
        S.q[2 * tid] = load_quat(quat, i);
        S.q[2 * tid + 1] = load_quat(quat, j);
        float dd;
        float3 tt = min_image(pos, i, j, MULTI ? rp[rep[i]].box : L, &dd);
        S.t[3 * tid] = tt.x;
        S.t[3 * tid + 1] = tt.y;
        S.t[3 * tid + 2] = tt.z;
        S.ij[2 * tid] = i;
        S.ij[2 * tid + 1] = j;
        store_centroid(S, tid, npts);
    }
    __syncthreads();
    rotate_tile<NP>(S, npts, rs);
}

// Per-pair force/torque from the two halves' partial sums, scaled, clipped
// (unless clip == 0), then scattered with runs of equal i summed in the warp
// (the first NP threads, thread = pair). y_of(q) is the net output of the tile's pair q.
template <int NP, bool MULTI, class Y>
__device__ __forceinline__ void adj_finish_tile(const AdjShared &S, int npts, int valid, float en_min, float en_range,
                                                const Y &y_of, float *F, float *T, double *pe, const int *rep,
                                                double &pe_acc, int clip) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int nd = 2 * npts;
    if (tid < NP) {
        const int p = tid;
        const float *a0 = S.part + p * kPartStride, *a1 = a0 + NP * kPartStride;
        float Si[3], Sa[3], Xi[3], Xj[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Si[k] = a0[k] + a1[k];
            Sa[k] = a0[3 + k] + a1[3 + k];
            Xi[k] = a0[6 + k] + a1[6 + k];
            Xj[k] = a0[9 + k] + a1[9 + k];
        }
        add_centroid_terms(S, p, Si, Sa, Xi, Xj);
        const float3 ps = make_float3(S.psum[0], S.psum[1], S.psum[2]);
        const float3 pi3 = rotate_ref(S.q[2 * p], ps), qj3 = rotate_ref(S.q[2 * p + 1], ps);
        const float Pi[3] = {pi3.x, pi3.y, pi3.z}, Qj[3] = {qj3.x, qj3.y, qj3.z};
        const float inv_nd = 1.0f / (float)nd;
        float Gm[3] = {Sa[0] * inv_nd, Sa[1] * inv_nd, Sa[2] * inv_nd};
        float Fp[3], Ti[3], Tj[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) Fp[k] = -(Si[k] - (float)npts * Gm[k]);
        Ti[0] = -(Xi[0] - (Pi[1] * Gm[2] - Pi[2] * Gm[1]));
        Ti[1] = -(Xi[1] - (Pi[2] * Gm[0] - Pi[0] * Gm[2]));
        Ti[2] = -(Xi[2] - (Pi[0] * Gm[1] - Pi[1] * Gm[0]));
        Tj[0] = -(Xj[0] - (Qj[1] * Gm[2] - Qj[2] * Gm[1]));
        Tj[1] = -(Xj[1] - (Qj[2] * Gm[0] - Qj[0] * Gm[2]));
        Tj[2] = -(Xj[2] - (Qj[0] * Gm[1] - Qj[1] * Gm[0]));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float f = Fp[k] * en_range, ti = Ti[k] * en_range, tj = Tj[k] * en_range;
            S.fd[9 * p + k] = clip ? clip100(f) : f;
            S.fd[9 * p + 3 + k] = clip ? clip100(ti) : ti;
            S.fd[9 * p + 6 + k] = clip ? clip100(tj) : tj;
        }
        if (!MULTI && p < valid) pe_acc += (double)en_min + (double)en_range * (double)y_of(p);
    }
    __syncthreads();
    if (tid < NP) {
        const int q = tid;
        const bool ok = q < valid;
        const int i = S.ij[2 * q], j = S.ij[2 * q + 1];
        float v[6];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            v[k] = ok ? S.fd[9 * q + k] : 0.f;
            v[3 + k] = ok ? S.fd[9 * q + 3 + k] : 0.f;
        }
        if (ok) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicAdd(F + 3 * j + k, -v[k]);
                atomicAdd(T + 3 * j + k, S.fd[9 * q + 6 + k]);
            }
        }
        const bool runs = warp_keys_sorted(i, ok);  // every lane takes part (warp vote)
        int key = ok && runs ? i : -1 - q;  // unsorted pairs: no merging
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int ko = __shfl_up_sync(0xffffffffu, key, o);
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                float yv = __shfl_up_sync(0xffffffffu, v[k], o);
                if (lane >= o && ko == key) v[k] += yv;
            }
        }
        int kn = __shfl_down_sync(0xffffffffu, key, 1);
        if (ok && (lane == 31 || kn != key)) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicAdd(F + 3 * i + k, v[k]);
                atomicAdd(T + 3 * i + k, v[3 + k]);
            }
        }
        if (MULTI && pe) {
            double e = ok ? (double)en_min + (double)en_range * (double)y_of(q) : 0.0;
            const int sys = ok ? rep[i] : 0;
            const bool sys_runs = warp_keys_sorted(sys, ok);
            int rk = ok && sys_runs ? sys : -1 - lane;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int ro = __shfl_up_sync(0xffffffffu, rk, o);
                double yv = __shfl_up_sync(0xffffffffu, e, o);
                if (lane >= o && ro == rk) e += yv;
            }
            int rn = __shfl_down_sync(0xffffffffu, rk, 1);
            if (ok && (lane == 31 || rn != rk)) atomicAdd(pe + sys, e);
        }
    }
    __syncthreads();
}

// MULTI: the pairs come from many systems in one launch; body i's system is
// rep[i], its box rp[rep[i]].box, and the pair energies are summed per system
// into pe[rep[i]].
template <class Cfg, bool MULTI>
__global__ void __launch_bounds__(kAThreads, 1) k_forces_adjoint(const float *pos, const float *quat, float L,
                                                                const int *pairs, const long long *d_np, long long cap,
                                                                const float *pts, int npts, float inv_rc, float en_min,
                                                                float en_range, AdjNet net, const float *w, float *F,
                                                                float *T, double *pe, const int *rep,
                                                                const amlp_replica *rp, int keep_r) {
    constexpr int DP = kGS;  // row stride of the fp32 descriptor staging
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ double pe_s[kAThreads / 32];
    __shared__ float psum_s[3];

    const int tid = threadIdx.x, p = tid & (kAP - 1), h = tid / kAP, warp = tid >> 5, lane = tid & 31;
    const int rs = 6 * npts + 1 - ((6 * npts) & 1);
    const int Kg = net.kin[0];
    const int first_limit = g_amlp_first_wait_limit;

    // ---- shared memory carve-up (offsets are multiples of 128 bytes)
    AdjShared S;
    size_t off = 0;
    // Two layouts. keep_r: the rotated points R have their own area and the
    // descriptor rows live in the first operand tile (free whenever the rows are
    // live), so R survives the net and is rotated once per tile.
    // Otherwise (when that does not fit) R shares its area with the operand
    // tiles and is rotated again after the net.
    const size_t r_bytes = (size_t)kAP * rs * 4, ops_bytes = (size_t)2 * 2 * kAP * kWpad * 2;
    if (keep_r) {
        S.R = reinterpret_cast<float *>(smem_raw);
        off = align_up(r_bytes, 128);
        S.ops = smem_raw + off;
        off += align_up(ops_bytes, 128);
    } else {
        S.ops = smem_raw;
        S.R = reinterpret_cast<float *>(smem_raw);
        off = align_up(r_bytes > ops_bytes ? r_bytes : ops_bytes, 128);
    }
    S.wts = smem_raw + off;
    off += align_up(net.wsm_total, 128);
    S.par = reinterpret_cast<float *>(smem_raw + off);
    off += align_up((size_t)net.par_total * 4, 128);
    if (keep_r) {
        S.g = reinterpret_cast<float *>(op_tile(S.ops, 0));
    } else {
        S.g = reinterpret_cast<float *>(smem_raw + off);
        off += (size_t)kAP * DP * 4;
    }
    take_pair_areas<kAP>(S, smem_raw + off);
    off += pair_area_bytes<kAP>();
    S.pts = reinterpret_cast<float *>(smem_raw + off);
    S.psum = psum_s;

    // ---- one-time set-up: weights (bf16 hi/lo, K-major), biases, TMEM, mbarrier
    for (int k = tid; k < 3 * npts; k += kAThreads) S.pts[k] = pts[k];
    __syncthreads();
    body_point_sum(S, npts);
    for (int L2 = 0; L2 < net.nh; ++L2) {
        const int K = net.dims[L2], N = net.dims[L2 + 1], Kp = net.kin[L2], Np = net.nout[L2];
        const float *W = w + net.woff[L2];
        split_layer(W, N, K, Np, Kp, S.wts + net.wsm_off[L2], tid, kAThreads);
        const float *b = W + (size_t)N * K;
        for (int n = tid; n < Np; n += kAThreads) S.par[net.bias_off[L2] + n] = n < N ? b[n] : 0.f;
    }
    {
        const int K = net.dims[net.nh];
        const float *Wl = w + net.woff[net.nh];
        for (int k = tid; k < kWpad; k += kAThreads) S.par[net.bias_off[net.nh] + k] = k < K ? Wl[k] : 0.f;
        if (tid == 0) S.par[net.bias_off[net.nh] + kWpad] = Wl[K];  // last bias
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    if (tid == 0) tc::mbar_init(&mbar, 1);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t bar = tc::smem_u32(&mbar);
    uint32_t phase = 0;
    // A bounded wait that gives up sets gave_up in its thread; the barrier that
    // ends each net stage ORs it over the block into `aborted`, so that every
    // thread agrees on it: no further MMA is issued or waited for, the tile loop
    // ends, and the MMA still in flight is drained before TMEM is released.
    bool gave_up = false, aborted = false;
    int waits = 0, commits = 0;
    // TMEM column regions: Z_k (hidden layer k) at 64k, backward product at 192, dE/dg at 192 too,
    // act'(Z_k) of the hidden layers before the last at 256 + 64k
    auto zcol = [&](int k) { return (uint32_t)(k * kWpad); };
    const uint32_t bcol = (uint32_t)(3 * kWpad);
    auto dfcol = [&](int k) { return (uint32_t)(4 * kWpad + k * kWpad); };
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

    auto wait_mma = [&]() {
        if (aborted) return;  // nothing was issued
        const int limit = (waits++ == 0 && first_limit >= 0) ? first_limit : tc::kWaitLimit;
        if (!tc::mbar_wait(bar, phase, limit)) gave_up = true;
        phase ^= 1u;
        tc::fence_after();
    };
    const long long P = min(*d_np, cap);
    const long long ntiles = (P + kAP - 1) / kAP;
    double pe_acc = 0.0;

    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long p0 = tile * kAP;
        const int valid = (int)min((long long)kAP, P - p0);
        // ---- 1. pair indices, orientations, translations, then the rotated body points
        load_pairs<kAP, MULTI>(S, pos, quat, L, pairs, P, p0, npts, rs, rep, rp);
        __syncthreads();
        // ---- 2. descriptor forward
        const float *Rp = S.R + p * rs;  // the pair's centred points
        float2 A[Cfg::NA][kHalfP];  // this half's sum_a f_n Y_k, kept in registers for the backward
        if (h == 0) half_forward<Cfg, 0, kFusedUnroll>(Rp, npts, inv_rc, S.g + p * DP, A);
        else half_forward<Cfg, 1, kFusedUnroll>(Rp, npts, inv_rc, S.g + p * DP, A);
        __syncthreads();
        if (h == 1) half_forward_finish<Cfg>(S.g + p * DP, A);
        __syncthreads();
        // ---- 3. net forward + backward on the tensor cores
        {
            char *tG = op_tile(S.ops, 0);
            // this thread's half of its row of g (kin[0] = 48 columns, set by the
            // launcher, 24 per half), read completely before the tile is written:
            // with keep_r, the rows occupy the operand tile
            float v[24];
#pragma unroll
            for (int k = 0; k < 24; ++k) {
                int d = h * 24 + k;
                v[k] = S.g[p * DP + d];
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 3; ++c) store_split8(tG, Kg, p, h * 24 + 8 * c, v + 8 * c);
        }
        tc::fence_async_smem();
        __syncthreads();
        // forward layers
        for (int L2 = 0; L2 < net.nh; ++L2) {
            const int Kp = net.kin[L2], Np = net.nout[L2];
            if (tid == 0 && !aborted) {
                tc::fence_after();
                const char *wb = S.wts + net.wsm_off[L2];
                mma3<true>(tmem + zcol(L2), op_tile(S.ops, L2), Kp, wb, (size_t)Np * Kp * 2, Np, false, 256, 128,
                     (uint32_t)Kp * 16);
                tc::commit(bar);
                ++commits;
            }
            wait_mma();
            // epilogue: a = act(z + b) into the next operand tile; the last hidden
            // layer also forms e and delta = w_last * act'(z)
            const bool last = L2 == net.nh - 1;
            const float *bias = S.par + net.bias_off[L2];
            const float *wl = S.par + net.bias_off[net.nh];
            char *dst = op_tile(S.ops, L2 + 1);
            float esum = 0.f;
            // this thread's Np / 2 columns from cb: nch chunks of 8, two per TMEM wait
            const int cb = h * (Np / 2), nch = Np / 16;
            for (int g = 0; g < nch; g += 2) {
                float z[2 * 8];
                tc::tmem_ld8_many<2>(tmem + lane_base + zcol(L2) + cb + 8 * g, min(2, nch - g), z);
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    if (g + ch < nch) {
                        const int c0 = cb + 8 * (g + ch);
                        float v[8], dv[8], bb[8], ww[8];
                        // bias_off is a multiple of 16 floats and c0 of 8: 16-byte loads
                        *reinterpret_cast<float4 *>(bb) = *reinterpret_cast<const float4 *>(bias + c0);
                        *reinterpret_cast<float4 *>(bb + 4) = *reinterpret_cast<const float4 *>(bias + c0 + 4);
                        if (last) {
                            *reinterpret_cast<float4 *>(ww) = *reinterpret_cast<const float4 *>(wl + c0);
                            *reinterpret_cast<float4 *>(ww + 4) = *reinterpret_cast<const float4 *>(wl + c0 + 4);
                        }
#pragma unroll
                        for (int k = 0; k < 8; ++k) bb[k] += z[8 * ch + k];
                        act8(net.act, bb, v, dv);
                        if (last) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                esum = fmaf(ww[k], v[k], esum);
                                v[k] = ww[k] * dv[k];
                            }
                        }
                        store_split8(dst, Np, p, c0, v);
                        if (!last) tc::tmem_st8(tmem + lane_base + dfcol(L2) + c0, dv);  // for the backward
                    }
                }
            }
            if (last) S.eps[h * kAP + p] = esum;
            else tc::tmem_wait_st();
            tc::fence_before();
            tc::fence_async_smem();
            aborted = __syncthreads_or(gave_up) != 0;
        }
        // backward layers: delta_{k-1} = (delta_k W_k) * act'(z_{k-1}); dE/dg = delta_1 W_1
        for (int L2 = net.nh - 1; L2 >= 0; --L2) {
            const int Kp = net.kin[L2], Np = net.nout[L2];
            if (tid == 0 && !aborted) {
                tc::fence_after();
                const char *wb = S.wts + net.wsm_off[L2];
                // B = W_k read as MN-major (the transpose): N' = Kp, K' = Np
                mma3<true>(tmem + bcol, op_tile(S.ops, L2 + 1), Np, wb, (size_t)Np * Kp * 2, Kp, true,
                     2 * Kp * 16, (uint32_t)Kp * 16, 128);
                tc::commit(bar);
                ++commits;
            }
            wait_mma();
            const int cb = h * (Kp / 2), nch = Kp / 16;
            if (L2 > 0) {
                char *dst = op_tile(S.ops, L2);
                for (int ch = 0; ch < nch; ++ch) {  // a chunk of dz and of act'(z) per TMEM wait
                    const int c0 = cb + 8 * ch;
                    uint32_t r[16];
                    float x[16];
                    tc::tmem_ld8_issue(tmem + lane_base + bcol + c0, r);
                    tc::tmem_ld8_issue(tmem + lane_base + dfcol(L2 - 1) + c0, r + 8);
                    tc::tmem_wait_ld<16>(r, x);
                    float v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = x[k] * x[8 + k];
                    store_split8(dst, Kp, p, c0, v);
                }
                tc::fence_async_smem();
            } else {
                for (int g = 0; g < nch; g += 2) {
                    float dg[2 * 8];
                    tc::tmem_ld8_many<2>(tmem + lane_base + bcol + cb + 8 * g, min(2, nch - g), dg);
#pragma unroll
                    for (int ch = 0; ch < 2; ++ch)
                        if (g + ch < nch)
#pragma unroll
                            for (int k = 0; k < 8; ++k) S.g[p * DP + cb + 8 * (g + ch) + k] = dg[8 * ch + k];
                }
            }
            tc::fence_before();
            aborted = __syncthreads_or(gave_up) != 0;
        }
        if (aborted) break;  // the net's outputs are not to be trusted: no forces from this tile
        // ---- 4. recompute the rotated points (their area held the MLP tiles)
        if (!keep_r) {
            rotate_tile<kAP>(S, npts, rs);
            __syncthreads();
        }
        // ---- descriptor backward
        float *part = S.part + (h * kAP + p) * kPartStride;
        if (h == 0) half_backward<Cfg, 0>(Rp, npts, inv_rc, S.g + p * DP, part, A);
        else half_backward<Cfg, 1>(Rp, npts, inv_rc, S.g + p * DP, part, A);
        __syncthreads();
        // ---- 5. per-pair forces and torques, scatter
        const float b_last = S.par[net.bias_off[net.nh] + kWpad];
        adj_finish_tile<kAP, MULTI>(
            S, npts, valid, en_min, en_range,
            [&](int q) { return S.eps[q] + S.eps[kAP + q] + b_last; }, F, T, pe, rep, pe_acc, 1);
    }
    if (aborted && tid == 0) {
        atomicOr(&g_amlp_device_error, kErrMbarTimeout);
        // the last MMA issued may still be in flight (thread 0 flipped `phase` after waiting for it):
        // let it finish, with the normal limit, before TMEM is released
        if (commits > 0) tc::mbar_wait(bar, phase ^ 1u, tc::kWaitLimit);
    }
    // ---- pair-energy sum, TMEM release
    if (!MULTI && pe) {
        double v = pe_acc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) pe_s[warp] = v;
    }
    tc::fence_before();
    __syncthreads();
    if (!MULTI && pe && tid == 0) {
        double s = 0.0;
        for (int k = 0; k < kAThreads / 32; ++k) s += pe_s[k];
        if (s != 0.0) atomicAdd(pe, s);
    }
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

// ============================================================================
// Wide nets (hidden widths up to 128): three kernels instead of one, since the
// descriptor state and the resident weights of a 128-wide net do not share one
// CTA's shared memory. g, dE/dg and the net output go through a caller
// workspace:
//   k_adj_desc<..., false>  descriptor forward per pair -> g (P x 48 fp32);
//   k_mlp_pair, k_mlp_grad  net forward + backward on the tensor cores per row,
//                           weights staged layer by layer -> y and dE/dg;
//   k_adj_desc<..., true>   recomputes the per-pair sums, descriptor backward,
//                           forces, torques, scatter.
// ============================================================================
constexpr int kWideMax = 160;  // hidden widths up to 150 (the reference's nets), padded to 160
constexpr int kGP = 48;  // padded descriptor width in the workspace rows
// Row stride of the descriptor rows in the workspace and in k_mlp_grad's shared
// copy: 52 floats, 13 units of 16 bytes, odd, so that the 16-byte reads of 32
// consecutive rows by a warp fall in distinct bank groups.
constexpr int kGRow = 52;
// The same for the hypers (10, 10, 10), D = 121: padded to 128, rows of 132 floats (33 x 16 bytes)
constexpr int kGP2 = 128;
constexpr int kGRow2 = 132;
constexpr size_t kWeightSplitBytes = (size_t)kMaxHiddenWide * kWideMax * kWideMax * 4;  // bf16 hi/lo, every layer
constexpr size_t kAdjAFloats = 2 * 9 * kHalfK;  // harmonic sums per pair kept between the passes

__host__ __device__ inline size_t adj_a_bytes(long long cap) {
    return (size_t)((cap + kDP - 1) / kDP) * kDP * kAdjAFloats * 4;
}

// dE/dg rows of the tile's pairs into S.g (row stride kGS), weighted by wt
// when given; rows past `valid` are zero. One row per warp, lanes over columns.
__device__ __forceinline__ void load_dg_rows(const AdjShared &S, const float *dg_rows, const float *wt, long long p0,
                                             int valid) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = warp; q < kDP; q += kDThreads / 32) {
        const float w = q < valid ? (wt ? wt[p0 + q] : 1.0f) : 0.f;
        for (int d = lane; d < kGP; d += 32) S.g[q * kGS + d] = q < valid ? w * dg_rows[(p0 + q) * kGP + d] : 0.f;
    }
}

// Descriptor pass of the wide path: BWD = false writes g rows (row stride
// g_ld >= D, zero padded); BWD = true reads dE/dg rows (stride kGP) and the net
// outputs and produces forces, torques and energies. wt (BWD, may be null)
// weights pair p's dE/dg by wt[p] (a vector-Jacobian product); clip = 0 turns
// the +-100 clip of the per-pair forces and torques off.
template <class Cfg, bool MULTI, bool BWD>
__global__ void __launch_bounds__(kDThreads, 2) k_adj_desc(const float *pos, const float *quat, float L,
                                                          const int *pairs, const long long *d_np, long long cap,
                                                          const float *pts, int npts, float inv_rc, float en_min,
                                                          float en_range, float *g_rows, int g_ld,
                                                          const float *dg_rows, const float *y_rows, const float *wt,
                                                          int clip, float *F, float *T, double *pe, const int *rep,
                                                          const amlp_replica *rp, float *a_rows) {
    constexpr int KC = kHalfK;
    static_assert(2 * Cfg::NA * KC == kAdjAFloats, "harmonic sums per pair in the workspace");
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ double pe_s[kDThreads / 32];
    __shared__ float psum_s[3];
    const int tid = threadIdx.x, p = tid & (kDP - 1), h = tid / kDP, warp = tid >> 5, lane = tid & 31;
    const int rs = 6 * npts + 1 - ((6 * npts) & 1);
    AdjShared S;
    S.psum = psum_s;
    size_t off = 0;
    S.R = reinterpret_cast<float *>(smem_raw);
    off = align_up((size_t)kDP * rs * 4, 128);
    S.g = reinterpret_cast<float *>(smem_raw + off);
    off += (size_t)kDP * kGS * 4;
    take_pair_areas<kDP>(S, smem_raw + off);
    off += pair_area_bytes<kDP>();
    S.pts = reinterpret_cast<float *>(smem_raw + off);
    for (int k = tid; k < 3 * npts; k += kDThreads) S.pts[k] = pts[k];
    __syncthreads();
    body_point_sum(S, npts);
    __syncthreads();
    const long long P = min(*d_np, cap);
    const long long ntiles = (P + kDP - 1) / kDP;
    double pe_acc = 0.0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long p0 = tile * kDP;
        const int valid = (int)min((long long)kDP, P - p0);
        // this thread's harmonic sums: computed by the forward pass (and stored
        // for the backward pass when a_rows is given), read back by the backward
        // pass; layout [tile][half][n][kk][pair] so that a warp's accesses coalesce
        float2 A[Cfg::NA][kHalfP];
        float *a_tile = a_rows ? a_rows + ((size_t)tile * 2 + h) * (Cfg::NA * KC) * kDP + p : nullptr;
        if (BWD && a_rows && tid == 0 && tile + gridDim.x < ntiles) {
            // the next tile's harmonic sums and dE/dg rows into L2 while this tile runs
            const long long nt = tile + gridDim.x;
            const char *an = reinterpret_cast<const char *>(a_rows + (size_t)nt * 2 * (Cfg::NA * KC) * kDP);
            constexpr uint32_t kABytes = 2u * Cfg::NA * KC * kDP * 4u, kPiece = 16384u;
            for (uint32_t o = 0; o < kABytes; o += kPiece) tc::bulk_prefetch_l2(an + o, min(kPiece, kABytes - o));
            const uint32_t gb = (uint32_t)(min((long long)kDP, P - nt * kDP) * kGP * 4);
            tc::bulk_prefetch_l2(dg_rows + nt * kDP * kGP, gb);
        }
        if (BWD && a_rows) {
            // the backward's inputs first, so that their loads overlap the rotation pass
#pragma unroll
            for (int n = 0; n < Cfg::NA; ++n)
#pragma unroll
                for (int kk = 0; kk < KC; ++kk) pick(A[n], kk) = a_tile[(n * KC + kk) * kDP];
            load_dg_rows(S, dg_rows, wt, p0, valid);
        }
        load_pairs<kDP, MULTI>(S, pos, quat, L, pairs, P, p0, npts, rs, rep, rp);
        __syncthreads();
        const float *Rp = S.R + p * rs;  // the pair's centred points
        if (!BWD || !a_rows) {
            if (h == 0) half_forward<Cfg, 0, kWideUnroll>(Rp, npts, inv_rc, S.g + p * kGS, A);
            else half_forward<Cfg, 1, kWideUnroll>(Rp, npts, inv_rc, S.g + p * kGS, A);
            __syncthreads();
            if (h == 1) half_forward_finish<Cfg>(S.g + p * kGS, A);
            if (!BWD && a_tile) {
#pragma unroll
                for (int n = 0; n < Cfg::NA; ++n)
#pragma unroll
                    for (int kk = 0; kk < KC; ++kk) a_tile[(n * KC + kk) * kDP] = pick(A[n], kk);
            }
        }
        __syncthreads();
        if (!BWD) {
            for (int q = warp; q < valid; q += kDThreads / 32)  // one row per warp: coalesced
                for (int d = lane; d < g_ld; d += 32)
                    g_rows[(p0 + q) * g_ld + d] = d < Cfg::D ? S.g[q * kGS + d] : 0.f;
            __syncthreads();
            continue;
        }
        if (!a_rows) {  // the descriptor rows held S.g until now
            load_dg_rows(S, dg_rows, wt, p0, valid);
        }
        __syncthreads();
        float *part = S.part + (h * kDP + p) * kPartStride;
        if (h == 0) half_backward<Cfg, 0>(Rp, npts, inv_rc, S.g + p * kGS, part, A);
        else half_backward<Cfg, 1>(Rp, npts, inv_rc, S.g + p * kGS, part, A);
        __syncthreads();
        adj_finish_tile<kDP, MULTI>(
            S, npts, valid, en_min, en_range, [&](int q) { return y_rows[p0 + q]; }, F, T, pe, rep, pe_acc, clip);
    }
    if (BWD && !MULTI && pe) {
        double v = pe_acc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) pe_s[warp] = v;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int k = 0; k < kDThreads / 32; ++k) s += pe_s[k];
            if (s != 0.0) atomicAdd(pe, s);
        }
    }
}

// The hidden layers' weights split into bf16 hi/lo once per launch, in the
// K-major layout of the shared-memory operand (per layer: hi, then lo), so that
// the net kernels load a layer with one bulk copy.
__global__ void k_split_weights(AdjNet net, const float *w, char *dst) {
    for (int L2 = 0; L2 < net.nh; ++L2) {
        const int K = net.dims[L2], N = net.dims[L2 + 1], Kp = net.kin[L2], Np = net.nout[L2];
        split_layer(w + net.woff[L2], N, K, Np, Kp, dst + net.wsm_off[L2], blockIdx.x * blockDim.x + threadIdx.x,
                    gridDim.x * blockDim.x);
    }
}

// y and dE/dg of the tiles tl, tl + step, ... to zero: what a wait that gave up leaves
// behind is not to be trusted, and with dE/dg zero the pairs exert no force.
__device__ void drop_rows(long long tl, long long step, long long P, int gp, int first, int stride, float *y_rows,
                          float *dg_rows) {
    for (; tl * kAP < P; tl += step) {
        const long long r0 = tl * kAP;
        const int valid = (int)min((long long)kAP, P - r0);
        for (int k = first; k < valid; k += stride) y_rows[r0 + k] = 0.f;
        for (int k = first; k < valid * gp; k += stride) dg_rows[r0 * gp + k] = 0.f;
    }
}

// Net forward and backward over rows of g on the tensor cores (bf16x3 splits,
// fp32 TMEM accumulators), hidden layers up to 160 wide and up to four of them
// (the reference's TheEnergyNet(150, 3, D): layer_first and three hidden
// layers). 16 warps: warp w reads TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31 (its
// rows) and, of every layer's columns, the 8-column chunks c with
// c % 4 == w / 4, so that four warps share each epilogue's rows.
// Shared memory holds one operand tile: each epilogue overwrites the tile its
// MMA read, complete by then. One layer's weights at a time sit beside it,
// brought in by a bulk copy from the pre-split copy (k_split_weights) that
// thread 0 starts as soon as the previous layer's MMAs are done, so that it
// overlaps the epilogue; the layer order fwd 0..nh-1, bwd nh-1..0 reuses the
// last forward layer and, across tiles, layer 0. One TMEM region (net.zbw
// columns) takes every product in turn. The forward epilogues keep act'(z) of
// each hidden layer but the last for the backward: for ReLU (derivative 0 or
// 1) as bits in registers, otherwise in TMEM after the product region.
// Outputs per row: y = net(g) and dE/dg (net.gp floats).
constexpr int kMQ = 4;                  // column groups of the k_mlp_grad epilogues
constexpr int kMThreads = kMQ * kAP;    // 512
static_assert(kWideMax <= 8 * kMQ * 8, "a thread's 8-column chunks of a layer fit one 64-bit mask");
__global__ void __launch_bounds__(kMThreads, 1) k_mlp_grad(const float *g_rows, const long long *d_np, long long cap,
                                                          AdjNet net, const float *w, const char *wsplit,
                                                          float *y_rows, float *dg_rows) {
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ uint64_t mbar, wbar, gbar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, p = tid & (kAP - 1), h = tid >> 7, warp = tid >> 5;
    char *tile = smem_raw;  // the operand tile: bf16 hi, then lo
    char *wbuf = smem_raw + net.wbuf_off;
    float *par = reinterpret_cast<float *>(smem_raw + net.par_off);
    float *eps = reinterpret_cast<float *>(smem_raw + net.eps_off);
    float *gbuf = reinterpret_cast<float *>(smem_raw + net.gbuf_off);
    for (int L2 = 0; L2 < net.nh; ++L2) {
        const int N = net.dims[L2 + 1], Np = net.nout[L2];
        const float *b = w + net.woff[L2] + (size_t)N * net.dims[L2];
        for (int n = tid; n < Np; n += kMThreads) par[net.bias_off[L2] + n] = n < N ? b[n] : 0.f;
    }
    {
        const int K = net.dims[net.nh];
        const float *Wl = w + net.woff[net.nh];
        for (int k = tid; k < kWideMax; k += kMThreads) par[net.bias_off[net.nh] + k] = k < K ? Wl[k] : 0.f;
        if (tid == 0) par[net.bias_off[net.nh] + kWideMax] = Wl[K];
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    if (tid == 0) {
        tc::mbar_init(&mbar, 1);
        tc::mbar_init(&wbar, 1);
        tc::mbar_init(&gbar, 1);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_slot, bar = tc::smem_u32(&mbar);
    uint32_t phase = 0;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    auto dfcol = [&](int k) { return (uint32_t)(net.zbw + k * net.wmax); };  // act'(z_k), smooth activations
    const bool relu = net.relu_bits != 0;
    // A bounded wait that gives up sets gave_up in its thread; the barriers that
    // end the stages OR it over the block into `aborted`: no further MMA or copy
    // is issued, the tile loop ends and what is in flight is drained at the end.
    bool gave_up = false, aborted = false;
    int commits = 0;
    int limit = g_amlp_first_wait_limit >= 0 ? g_amlp_first_wait_limit : tc::kWaitLimit;
    auto wait_mma = [&]() {
        if (aborted) return;  // nothing was issued
        if (!tc::mbar_wait(bar, phase, limit)) gave_up = true;
        limit = tc::kWaitLimit;
        phase ^= 1u;
        tc::fence_after();
    };
    // weights: `in_buf` (tracked identically by every thread) is the layer whose
    // weights are in wbuf or on their way; thread 0 starts the copies and waits
    // for them before its MMAs.
    int in_buf = -1;
    bool w_pending = false;
    uint32_t wphase = 0;
    const uint32_t wb_u32 = tc::smem_u32(wbuf), wbar_u32 = tc::smem_u32(&wbar);
    auto request = [&](int L2) {
        if (L2 == in_buf) return;
        in_buf = L2;
        if (tid == 0 && !aborted && !gave_up) {
            const uint32_t bytes = (uint32_t)(4 * net.nout[L2] * net.kin[L2]);
            tc::mbar_arrive_expect_tx(wbar_u32, bytes);
            tc::bulk_g2s(wb_u32, wsplit + net.wsm_off[L2], bytes, wbar_u32);
            w_pending = true;
        }
    };
    auto ensure = [&]() {  // thread 0 only
        if (!w_pending) return;
        if (!tc::mbar_wait(wbar_u32, wphase)) gave_up = true;
        wphase ^= 1u;
        w_pending = false;
    };
    request(0);
    const long long P = min(*d_np, cap);
    const long long ntiles = (P + kAP - 1) / kAP;
    const int Kg = net.kin[0];
    // descriptor rows of tile tl into gbuf (thread 0; rows r0 .. r0 + valid are contiguous)
    bool g_pending = false;
    uint32_t gphase = 0;
    const uint32_t gbuf_u32 = tc::smem_u32(gbuf), gbar_u32 = tc::smem_u32(&gbar);
    auto request_g = [&](long long tl) {
        if (!net.prefetch_g || tid != 0 || aborted || gave_up || tl >= ntiles) return;
        const long long r0 = tl * kAP;
        const uint32_t bytes = (uint32_t)(min((long long)kAP, P - r0) * net.g_ld * 4);
        tc::mbar_arrive_expect_tx(gbar_u32, bytes);
        tc::bulk_g2s(gbuf_u32, g_rows + r0 * net.g_ld, bytes, gbar_u32);
        g_pending = true;
    };
    request_g(blockIdx.x);
    for (long long tl = blockIdx.x; tl < ntiles; tl += gridDim.x) {
        if (aborted) break;
        const long long r0 = tl * kAP;
        const int valid = (int)min((long long)kAP, P - r0);
        if (net.prefetch_g) {  // every thread reads gbuf
            if (!tc::mbar_wait(gbar_u32, gphase)) gave_up = true;
            gphase ^= 1u;
            if (tid == 0) g_pending = false;
        }
        for (int c0 = 8 * h; c0 < Kg; c0 += 8 * kMQ) {
            float v[8];
            const float *src = net.prefetch_g ? gbuf + p * net.g_ld + c0 : g_rows + (r0 + p) * net.g_ld + c0;
            const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 lo4 = p < valid ? reinterpret_cast<const float4 *>(src)[0] : zero4;
            const float4 hi4 = p < valid ? reinterpret_cast<const float4 *>(src)[1] : zero4;
            v[0] = lo4.x, v[1] = lo4.y, v[2] = lo4.z, v[3] = lo4.w;
            v[4] = hi4.x, v[5] = hi4.y, v[6] = hi4.z, v[7] = hi4.w;
            store_split8(tile, Kg, p, c0, v);
        }
        uint64_t m0 = 0, m1 = 0, m2 = 0;  // ReLU: act'(z) bits of hidden layers 0, 1, 2 (this thread's chunks)
        for (int L2 = 0; L2 < net.nh; ++L2) {
            const int Kp = net.kin[L2], Np = net.nout[L2];
            request(L2);
            if (L2 == 0) {  // later layers start right after the previous epilogue's barrier
                tc::fence_async_smem();
                aborted = __syncthreads_or(gave_up) != 0;
                request_g(tl + gridDim.x);  // gbuf has been read: prefetch the next tile
            }
            if (tid == 0) ensure();
            if (tid == 0 && !aborted && !gave_up) {
                tc::fence_after();
                mma3<false>(tmem, tile, Kp, wbuf, (size_t)Np * Kp * 2, Np, false, 256, 128, (uint32_t)Kp * 16);
                tc::commit(bar);
                ++commits;
            }
            wait_mma();
            if (L2 + 1 < net.nh) request(L2 + 1);  // overlaps this layer's epilogue
            const bool last = L2 == net.nh - 1;
            const float *bias = par + net.bias_off[L2];
            const float *wl = par + net.bias_off[net.nh];
            float esum = 0.f;
            uint64_t bits = 0;
            for (int j = 0, c0 = 8 * h; c0 < Np; ++j, c0 += 8 * kMQ) {
                float z[8], v[8], dv[8], bb[8], ww[8];
                tc::tmem_ld8(tmem + lane_base + c0, z);
                *reinterpret_cast<float4 *>(bb) = *reinterpret_cast<const float4 *>(bias + c0);
                *reinterpret_cast<float4 *>(bb + 4) = *reinterpret_cast<const float4 *>(bias + c0 + 4);
                if (last) {
                    *reinterpret_cast<float4 *>(ww) = *reinterpret_cast<const float4 *>(wl + c0);
                    *reinterpret_cast<float4 *>(ww + 4) = *reinterpret_cast<const float4 *>(wl + c0 + 4);
                }
                uint32_t b8 = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) bb[k] += z[k];
                act8(net.act, bb, v, dv);
                if (last) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        esum = fmaf(ww[k], v[k], esum);
                        v[k] = ww[k] * dv[k];
                    }
                } else if (relu) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) b8 |= (dv[k] != 0.f ? 1u : 0u) << k;
                }
                if (!last) bits |= (uint64_t)b8 << (8 * j);
                store_split8(tile, Np, p, c0, v);  // the MMA that read the tile is complete
                if (!last && !relu) tc::tmem_st8(tmem + lane_base + dfcol(L2) + c0, dv);  // for the backward
            }
            if (last) {
                eps[h * kAP + p] = esum;
            } else if (relu) {
                if (L2 == 0) m0 = bits;
                else if (L2 == 1) m1 = bits;
                else m2 = bits;
            } else {
                tc::tmem_wait_st();
            }
            tc::fence_before();
            tc::fence_async_smem();
            aborted = __syncthreads_or(gave_up) != 0;
        }
        if (tid < kAP && p < valid)
        {
            float ysum = par[net.bias_off[net.nh] + kWideMax];
#pragma unroll
            for (int g = 0; g < kMQ; ++g) ysum += eps[g * kAP + p];
            y_rows[r0 + p] = ysum;
        }
        // backward: delta_{k-1} = (delta_k W_k) * act'(z_{k-1}); dE/dg = delta_0 W_0
        for (int L2 = net.nh - 1; L2 >= 0; --L2) {  // each layer starts right after the previous barrier
            const int Kp = net.kin[L2], Np = net.nout[L2];
            request(L2);
            if (tid == 0) ensure();
            if (tid == 0 && !aborted && !gave_up) {
                tc::fence_after();
                // B = W_k read as MN-major (the transpose): N' = Kp, K' = Np
                mma3<false>(tmem, tile, Np, wbuf, (size_t)Np * Kp * 2, Kp, true, 2 * Kp * 16, (uint32_t)Kp * 16, 128);
                tc::commit(bar);
                ++commits;
            }
            wait_mma();
            request(L2 > 0 ? L2 - 1 : 0);  // the next layer needed (layer 0 again for the next tile)
            if (L2 > 0) {
                const uint64_t bits = L2 == 1 ? m0 : (L2 == 2 ? m1 : m2);
                for (int j = 0, c0 = 8 * h; c0 < Kp; ++j, c0 += 8 * kMQ) {
                    float dz[8], df[8], v[8];
                    tc::tmem_ld8(tmem + lane_base + c0, dz);
                    if (relu) {
                        const uint32_t b8 = (uint32_t)(bits >> (8 * j));
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = (b8 >> k) & 1u ? dz[k] : 0.f;
                    } else {
                        tc::tmem_ld8(tmem + lane_base + dfcol(L2 - 1) + c0, df);
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = dz[k] * df[k];
                    }
                    store_split8(tile, Kp, p, c0, v);
                }
            } else {
                for (int c0 = 8 * h; c0 < Kp; c0 += 8 * kMQ) {
                    float dg[8];
                    tc::tmem_ld8(tmem + lane_base + c0, dg);
                    if (p < valid) {
                        float4 *dst = reinterpret_cast<float4 *>(dg_rows + (r0 + p) * net.gp + c0);
                        dst[0] = make_float4(dg[0], dg[1], dg[2], dg[3]);
                        dst[1] = make_float4(dg[4], dg[5], dg[6], dg[7]);
                    }
                }
            }
            tc::fence_before();
            tc::fence_async_smem();
            aborted = __syncthreads_or(gave_up) != 0;
        }
    }
    aborted = __syncthreads_or(gave_up) != 0;
    if (tid == 0) {
        bool drained = true;
        // the last MMA issued (commit number `commits`, parity (commits - 1) & 1) may still be in flight
        if (commits > 0) drained &= tc::mbar_wait(bar, (uint32_t)((commits - 1) & 1));
        if (w_pending) drained &= tc::mbar_wait(wbar_u32, wphase);  // no copy may still write shared memory
        if (g_pending) drained &= tc::mbar_wait(gbar_u32, gphase);
        if (aborted || !drained) atomicOr(&g_amlp_device_error, kErrMbarTimeout);
    }
    __syncthreads();
    if (aborted) drop_rows(blockIdx.x, gridDim.x, P, net.gp, tid, kMThreads, y_rows, dg_rows);
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

// The same net pass with two tiles in flight per CTA. k_mlp_grad runs a tile's products
// and epilogues one after the other: of its 51 k cycles a tile (four 160-wide layers)
// the tensor cores worked 20 k. Here two teams of twelve warps each have a tile of their
// own (operand tile, product region, mbarrier), so that one team's epilogue runs under
// the other's product, and one copy of the running layer's weights serves both.
//  - The last warp issues the products, team 0's then team 1's of each layer, when a team
//    signals that its operand tile is written (ready) and the weights are there (wfull).
//    All its lanes compute the descriptors, so that they stay in uniform registers:
//    issued by a thread of the team under a divergent branch, between its scheduler's
//    epilogues, the 30 MMAs of a 160-wide layer took 3.9 k cycles to issue and 2.4 k to run.
//  - The warp before it copies the next layer's weights when both products are complete (wfree).
//  - A team without a tile (last round) is left out of the round.
//  - A role whose wait gives up sets `quit` and leaves; the others follow (pair_wait, or at
//    worst their own limit), the products in flight are drained, and the block's rows are
//    zeroed (drop_rows).
// Two 160-wide operand tiles and a layer's weights do not fit shared memory: with TMEM_A
// the first team's operand tile is in TMEM (bf16 pairs, hi and lo), which ReLU leaves
// room for (its derivatives are bits in registers). Smooth activations take this kernel
// when both tiles fit shared memory and both teams' act'(z) fit TMEM; up to two 128-wide
// hidden layers do. A product is the same sequence of MMAs as in k_mlp_grad. A team's
// chain of product and epilogue bounds the kernel (the activation is known at compile
// time, and three column groups per row shorten it: 3 % faster than two; a fourth would
// pass 1,024 threads), with the weights' copies, 2.7 k cycles for a 160-wide layer.
// Measured against k_mlp_grad: 5,465 tiles of four 150-wide ReLU layers 960 -> 581 us
// (tensor pipe busy 336 us), 5,715 tiles of two 128-wide silu layers 490 -> 335 us.
constexpr int kPG = 3;               // column groups of a team's epilogues
constexpr int kPTeam = kPG * kAP;
constexpr int kPThreads = 2 * kPTeam + 64;
static_assert(kWideMax <= 8 * 8 * kPG, "a thread's chunks of a layer fit two words of bits");

__device__ __forceinline__ bool pair_sync_or(int team, bool v) {
    uint32_t o;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(o)
        : "r"((uint32_t)v), "r"(1 + team), "n"(kPTeam)
        : "memory");
    return o != 0;
}

// Bounded wait that ends early (false) when another role of the block has given up, as
// that sets `quit`. It is looked at every 64 polls, to keep the polling itself short.
__device__ __forceinline__ bool pair_wait(uint32_t bar, uint32_t phase, const volatile int *quit) {
    for (int i = 0; i < tc::kWaitLimit; i += 64) {
        if (tc::mbar_wait(bar, phase, 64)) return true;
        if (*quit) return false;
    }
    return false;
}

// mma3's sequence with the descriptors' steps added to their address fields (a shared-memory
// address is below 2^18, so a field holds it) and, with a_tmem, A's hi and lo in TMEM.
// Every lane of the issuing warp runs it, so that its arithmetic is uniform; `leader`
// issues.
__device__ __forceinline__ void issue3(bool leader, uint32_t d_tmem, bool a_tmem, uint32_t a_hi, uint32_t a_lo, int K,
                                       uint32_t b_hi, uint32_t b_lo, int N, bool b_mn, uint32_t b_kstride,
                                       uint32_t b_lbo, uint32_t b_sbo) {
    const uint32_t idesc = tc::idesc_bf16(N, b_mn ? 1 : 0);
    uint64_t b0 = tc::smem_desc(b_hi, b_lbo, b_sbo), b1 = tc::smem_desc(b_lo, b_lbo, b_sbo);
    const uint64_t bstep = b_kstride >> 4;
    if (a_tmem) {
#pragma unroll 2
        for (int ks = 0; ks < K / 16; ++ks) {
            if (leader) {
                tc::mma_bf16_ts(d_tmem, a_hi, b0, idesc, ks > 0 ? 1u : 0u);
                tc::mma_bf16_ts(d_tmem, a_hi, b1, idesc, 1u);
                tc::mma_bf16_ts(d_tmem, a_lo, b0, idesc, 1u);
            }
            a_hi += 8, a_lo += 8, b0 += bstep, b1 += bstep;
        }
    } else {
        uint64_t a0 = tc::smem_desc(a_hi, 128, (uint32_t)K * 16), a1 = tc::smem_desc(a_lo, 128, (uint32_t)K * 16);
#pragma unroll 2
        for (int ks = 0; ks < K / 16; ++ks) {
            if (leader) {
                tc::mma_bf16(d_tmem, a0, b0, idesc, ks > 0 ? 1u : 0u);
                tc::mma_bf16(d_tmem, a0, b1, idesc, 1u);
                tc::mma_bf16(d_tmem, a1, b0, idesc, 1u);
            }
            a0 += 16, a1 += 16, b0 += bstep, b1 += bstep;
        }
    }
}

// z[0..8) += b[0..8), two sums an instruction.
__device__ __forceinline__ void bias8(const float *b, float *z) {
    const float4 b0 = reinterpret_cast<const float4 *>(b)[0], b1 = reinterpret_cast<const float4 *>(b)[1];
    const float2 bb[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                          make_float2(b1.z, b1.w)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 r = add2(make_float2(z[2 * k], z[2 * k + 1]), bb[k]);
        z[2 * k] = r.x, z[2 * k + 1] = r.y;
    }
}

template <int ACT, bool TMEM_A>
__global__ void __launch_bounds__(kPThreads, 1) k_mlp_pair(const float *g_rows, const long long *d_np, long long cap,
                                                          AdjNet net, const float *w, const char *wsplit,
                                                          float *y_rows, float *dg_rows) {
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ uint64_t mbar[2], ready_s[2], wfull_s, wfree_s, done_s;
    __shared__ uint32_t tmem_slot;
    __shared__ int quit;  // a wait of some role has given up
    const int tid = threadIdx.x, warp = tid >> 5, team = tid / kPTeam, tt = tid - team * kPTeam;
    const int p = tt & (kAP - 1), h = tt / kAP;
    char *wbuf = smem_raw + net.pair_wbuf;
    float *par = reinterpret_cast<float *>(smem_raw + net.pair_par);
    float *eps = reinterpret_cast<float *>(smem_raw + net.pair_eps) + (team & 1) * kPG * kAP;
    char *tile = smem_raw + (TMEM_A ? 0 : (team & 1) * net.pair_tile);
    const bool a_tmem = TMEM_A && team == 0;
    for (int L2 = 0; L2 < net.nh; ++L2) {
        const int N = net.dims[L2 + 1], Np = net.nout[L2];
        const float *b = w + net.woff[L2] + (size_t)N * net.dims[L2];
        for (int n = tid; n < Np; n += kPThreads) par[net.bias_off[L2] + n] = n < N ? b[n] : 0.f;
    }
    {
        const int K = net.dims[net.nh];
        const float *Wl = w + net.woff[net.nh];
        for (int k = tid; k < kWideMax; k += kPThreads) par[net.bias_off[net.nh] + k] = k < K ? Wl[k] : 0.f;
        if (tid == 0) par[net.bias_off[net.nh] + kWideMax] = Wl[K];
    }
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    if (tid == 0) {
        tc::mbar_init(&mbar[0], 1);
        tc::mbar_init(&mbar[1], 1);
        tc::mbar_init(&ready_s[0], 1);
        tc::mbar_init(&ready_s[1], 1);
        tc::mbar_init(&wfull_s, 1);
        tc::mbar_init(&wfree_s, 1);
        tc::mbar_init(&done_s, 1);
        quit = 0;
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t wfull = tc::smem_u32(&wfull_s), wfree = tc::smem_u32(&wfree_s);
    const int nh = net.nh, np = 2 * nh;  // products of a tile: layers 0 .. nh - 1 forward, nh - 1 .. 0 backward
    auto layer_of = [&](int s) { return s < nh ? s : np - 1 - s; };
    // the weights change before product s (the same layer's serve the last forward and
    // the first backward one, and layer 0's the next round's first)
    auto loads_before = [&](int s, bool first_round) { return s == 0 ? first_round : s != nh; };
    const long long P = min(*d_np, cap);
    const long long ntiles = (P + kAP - 1) / kAP;
    const long long step = 2LL * gridDim.x;
    const long long rounds = blockIdx.x < ntiles ? (ntiles - blockIdx.x + step - 1) / step : 0;
    bool gave_up = team < 2 && g_amlp_first_wait_limit == 0, aborted = false;
    const uint32_t a_hi = tmem_slot + (uint32_t)(2 * net.pair_d), a_lo = a_hi + (uint32_t)(net.pair_d / 2);  // TMEM_A
    if (warp == 2 * kPTeam / 32) {  // weights
        if (tid == 2 * kPTeam) {
            uint32_t fphase = 0, loads = 0;
            for (long long r = 0; r < rounds && !gave_up; ++r)
                for (int s = 0; s < np && !gave_up; ++s) {
                    if (!loads_before(s, r == 0)) continue;
                    if (loads > 0) {
                        if (!pair_wait(wfree, fphase, &quit)) gave_up = true;
                        fphase ^= 1u;
                    }
                    if (gave_up) break;
                    const int L2 = layer_of(s);
                    const uint32_t bytes = (uint32_t)(4 * net.nout[L2] * net.kin[L2]);
                    tc::mbar_arrive_expect_tx(wfull, bytes);
                    tc::bulk_g2s(tc::smem_u32(wbuf), wsplit + net.wsm_off[L2], bytes, wfull);
                    ++loads;
                }
            // no copy may still write shared memory when the block ends
            if (loads > 0 && !tc::mbar_wait(wfull, (loads - 1) & 1u)) gave_up = true;
            if (gave_up) quit = 1;
        }
        __syncwarp();
    } else if (team == 2) {  // products
        const bool leader = tc::elect_one();
        const uint32_t wb = tc::smem_u32(wbuf), t0 = tc::smem_u32(smem_raw);
        const uint32_t tm0 = __shfl_sync(~0u, tmem_slot, 0);
        uint32_t wphase = 0, rphase = 0;  // both teams' tiles change phase together
        for (long long r = 0; r < rounds && !gave_up; ++r)
            for (int s = 0; s < np && !gave_up; ++s) {
                const int L2 = layer_of(s), Kp = net.kin[L2], Np = net.nout[L2];
                const bool fwd = s < nh;
                if (loads_before(s, r == 0)) {
                    if (!tc::mbar_wait(wfull, wphase)) gave_up = true;
                    wphase ^= 1u;
                }
                // forward: B = W_k (N' = Np, K' = Kp); backward: W_k read as MN-major (N' = Kp, K' = Np)
                const int N = fwd ? Np : Kp, K = fwd ? Kp : Np;
                const uint32_t b_lo = wb + (uint32_t)(Np * Kp * 2), ks = fwd ? 256 : 2 * Kp * 16;
                const uint32_t lbo = fwd ? 128u : (uint32_t)Kp * 16, sbo = fwd ? (uint32_t)Kp * 16 : 128u;
#pragma unroll
                for (int tm = 0; tm < 2; ++tm) {
                    if (blockIdx.x + (2 * r + tm) * gridDim.x >= ntiles) continue;
                    if (!pair_wait(tc::smem_u32(&ready_s[tm]), rphase, &quit)) gave_up = true;
                    gave_up = __any_sync(~0u, gave_up);
                    if (gave_up) break;
                    tc::fence_after();
                    const uint32_t d = tm0 + (uint32_t)(tm * net.pair_d);
                    if (TMEM_A && tm == 0) {
                        const uint32_t a0 = tm0 + (uint32_t)(2 * net.pair_d);
                        issue3(leader, d, true, a0, a0 + (uint32_t)(net.pair_d / 2), K, wb, b_lo, N, !fwd, ks, lbo, sbo);
                    } else {
                        const uint32_t a0 = t0 + (TMEM_A ? 0 : tm * net.pair_tile);
                        issue3(leader, d, false, a0, a0 + (uint32_t)(kAP * K * 2), K, wb, b_lo, N, !fwd, ks, lbo, sbo);
                    }
                    if (leader) tc::commit(tc::smem_u32(&mbar[tm]));
                    __syncwarp();
                }
                rphase ^= 1u;
                if (leader && s + 1 < np && loads_before(s + 1, false)) tc::commit(wfree);
                __syncwarp();
            }
        // products may still be in flight
        if (leader) tc::commit(tc::smem_u32(&done_s));
        __syncwarp();
        if (!tc::mbar_wait(tc::smem_u32(&done_s), 0)) gave_up = true;
        if (gave_up) quit = 1;
    } else {
        const uint32_t bar = tc::smem_u32(&mbar[team]);
        const uint32_t dcol = tmem_slot + (uint32_t)(team * net.pair_d);  // this team's product region
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t ready = tc::smem_u32(&ready_s[team]);
        constexpr bool relu = ACT == AMLP_ACT_RELU;
        auto dfcol = [&](int k) {  // act'(z_k), smooth activations
            return tmem_slot + (uint32_t)(2 * net.pair_d + (team * (nh - 1) + k) * net.wmax);
        };
        uint32_t phase = 0;
        const uint32_t row8 = (p & 7) * 16, rows = p >> 3;
        auto store_a = [&](int K, int c0, const float *v) {
            uint4 hi, lo;
            split8(v, hi, lo);
            if (a_tmem) {
                tc::tmem_st4(a_hi + lane_base + c0 / 2, hi);
                tc::tmem_st4(a_lo + lane_base + c0 / 2, lo);
            } else {
                char *dst = tile + row8 + rows * (K * 16) + c0 * 16;  // tc::kmajor_offset(p, c0, K)
                *reinterpret_cast<uint4 *>(dst) = hi;
                *reinterpret_cast<uint4 *>(dst + kAP * K * 2) = lo;
            }
        };
        // the end of a stage that wrote the operand tile or read TMEM
        auto stage_end = [&]() {
            if (a_tmem || !relu) tc::tmem_wait_st();
            tc::fence_before();
            tc::fence_async_smem();
            aborted = pair_sync_or(team, gave_up);
        };
        for (long long r = 0; r < rounds && !aborted; ++r) {
            const long long tl = blockIdx.x + (2 * r + team) * gridDim.x;
            if (tl >= ntiles) break;  // no tile in the last round
            const long long r0 = tl * kAP;
            const int valid = (int)min((long long)kAP, P - r0), Kg = net.kin[0];
            if (tt == 0 && tl + step < ntiles) {  // the next tile's descriptor rows into L2
                const long long n0 = (tl + step) * kAP;
                tc::bulk_prefetch_l2(g_rows + n0 * net.g_ld, (uint32_t)(min((long long)kAP, P - n0) * net.g_ld * 4));
            }
            const float4 *src = reinterpret_cast<const float4 *>(g_rows + (r0 + p) * net.g_ld);
            for (int c0 = 8 * h; c0 < Kg; c0 += 16 * kPG) {  // two chunks' loads in flight
                const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
                const bool two = c0 + 8 * kPG < Kg;
                float4 q[4] = {zero4, zero4, zero4, zero4};
                if (p < valid) {
                    q[0] = src[c0 / 4], q[1] = src[c0 / 4 + 1];
                    if (two) q[2] = src[c0 / 4 + 2 * kPG], q[3] = src[c0 / 4 + 2 * kPG + 1];
                }
                const float v[16] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w,
                                     q[2].x, q[2].y, q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w};
                store_a(Kg, c0, v);
                if (two) store_a(Kg, c0 + 8 * kPG, v + 8);
            }
            stage_end();
            uint32_t m[6];  // ReLU: act'(z) bits of hidden layers 0, 1, 2 (this thread's chunks)
            for (int s = 0; s < np && !aborted; ++s) {
                const int L2 = layer_of(s), Kp = net.kin[L2], Np = net.nout[L2];
                const bool fwd = s < nh;
                if (tt == 0) tc::mbar_arrive(ready);
                if (!tc::mbar_wait(bar, phase)) gave_up = true;
                phase ^= 1u;
                __syncwarp();
                tc::fence_after();
                // columns in chunks of 8: c0 = 8 h, 8 h + 8 kPG, ...
                const bool last = L2 == nh - 1;
                if (fwd) {
                    const float *bias = par + net.bias_off[L2], *wl = par + net.bias_off[nh];
                    uint32_t w0 = 0, w1 = 0;
                    float esum = 0.f;
                    for (int j = 0, c0 = 8 * h; c0 < Np; ++j, c0 += 8 * kPG) {
                        float z[8], v[8];
                        tc::tmem_ld8(dcol + lane_base + c0, z);
                        bias8(bias + c0, z);
                        if (last) {
                            float ww[8];
                            *reinterpret_cast<float4 *>(ww) = *reinterpret_cast<const float4 *>(wl + c0);
                            *reinterpret_cast<float4 *>(ww + 4) = *reinterpret_cast<const float4 *>(wl + c0 + 4);
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                float fz, dfz;
                                act_pair<ACT>(z[k], fz, dfz);
                                esum = fmaf(ww[k], fz, esum);
                                v[k] = ww[k] * dfz;
                            }
                        } else if (relu) {
                            uint32_t b8 = 0;
#pragma unroll
                            for (int k = 7; k >= 0; --k) {
                                v[k] = fmaxf(z[k], 0.f);
                                b8 = __funnelshift_l(__float_as_uint(0.f - z[k]), b8, 1);  // its sign: z > 0
                            }
                            b8 <<= 8 * (j & 3);
                            if (j < 4) w0 |= b8;
                            else w1 |= b8;
                        } else {
                            float dv[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) act_pair<ACT>(z[k], v[k], dv[k]);
                            tc::tmem_st8(dfcol(L2) + lane_base + c0, dv);  // for the backward
                        }
                        store_a(Np, c0, v);  // the MMA that read the tile is complete
                    }
                    if (last) eps[h * kAP + p] = esum;
                    else if (relu) {
                        if (L2 == 0) m[0] = w0, m[1] = w1;
                        else if (L2 == 1) m[2] = w0, m[3] = w1;
                        else m[4] = w0, m[5] = w1;
                    }
                } else if (L2 > 0) {
                    uint32_t w0 = 0, w1 = 0;
                    if (relu) {
                        w0 = L2 == 1 ? m[0] : (L2 == 2 ? m[2] : m[4]);
                        w1 = L2 == 1 ? m[1] : (L2 == 2 ? m[3] : m[5]);
                    }
                    for (int j = 0, c0 = 8 * h; c0 < Kp; ++j, c0 += 8 * kPG) {
                        float z[8];
                        if (relu) {
                            tc::tmem_ld8(dcol + lane_base + c0, z);
                            const uint32_t b8 = (j < 4 ? w0 : w1) >> (8 * (j & 3));
#pragma unroll
                            for (int k = 0; k < 8; ++k) z[k] = (b8 >> k) & 1u ? z[k] : 0.f;
                        } else {
                            uint32_t r2[16];
                            float x[16];
                            tc::tmem_ld8_issue(dcol + lane_base + c0, r2);
                            tc::tmem_ld8_issue(dfcol(L2 - 1) + lane_base + c0, r2 + 8);
                            tc::tmem_wait_ld<16>(r2, x);
#pragma unroll
                            for (int k = 0; k < 8; ++k) z[k] = x[k] * x[8 + k];
                        }
                        store_a(Kp, c0, z);
                    }
                } else {
                    float4 *dst = reinterpret_cast<float4 *>(dg_rows + (r0 + p) * net.gp);
                    for (int c0 = 8 * h; c0 < Kp; c0 += 8 * kPG) {
                        float z[8];
                        tc::tmem_ld8(dcol + lane_base + c0, z);
                        if (p < valid) {
                            dst[c0 / 4] = make_float4(z[0], z[1], z[2], z[3]);
                            dst[c0 / 4 + 1] = make_float4(z[4], z[5], z[6], z[7]);
                        }
                    }
                }
                stage_end();
                if (fwd && last && tt < kAP && p < valid) {
                    float ysum = par[net.bias_off[nh] + kWideMax];
#pragma unroll
                    for (int q = 0; q < kPG; ++q) ysum += eps[q * kAP + p];
                    y_rows[r0 + p] = ysum;
                }
            }
        }
        if (tt == 0 && (aborted || gave_up)) quit = 1;
        __syncwarp();
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tmem_slot, 512);
    }
    if (quit) {
        if (tid == 0) atomicOr(&g_amlp_device_error, kErrMbarTimeout);
        drop_rows(blockIdx.x, gridDim.x, P, net.gp, tid, kPThreads, y_rows, dg_rows);
    }
}

}  // namespace

amlp_status check_nep(const amlp_nep *n);
int hyper_kind(const amlp_nep *n);
int nep_D(const amlp_nep *n);
amlp_status check_mlp(const amlp_mlp *m, int D);

}  // namespace amlp

using namespace amlp;

static amlp_status launch_adjoint(const float *d_pos, const float *d_quat, float box, const int *d_pairs,
                                  const long long *d_npairs, long long cap, const amlp_nep *nep, const amlp_mlp *mlp,
                                  float *d_F, float *d_T, double *d_pe, const int *d_rep, const amlp_replica *d_rp,
                                  void *stream) {
    amlp_status st = check_nep(nep);
    if (st) return st;
    const int D = nep_D(nep);
    if ((st = check_mlp(mlp, D))) return st;
    if (!d_pos || !d_quat || !d_npairs || !d_F || !d_T || cap < 0 || (cap > 0 && !d_pairs)) return AMLP_ERR_INVALID_ARG;
    if (cap == 0) return AMLP_OK;
    if (hyper_kind(nep) != 1 || D > 48) return AMLP_ERR_UNSUPPORTED;
    const int nh = mlp->n_layers - 1;
    if (nh < 1 || nh > kMaxHidden) return AMLP_ERR_UNSUPPORTED;
    AdjNet net{};
    net.nh = nh;
    net.act = mlp->act;
    long long off = 0;
    int wsm = 0, par = 0;
    for (int k = 0; k <= mlp->n_layers; ++k) net.dims[k] = mlp->dims[k];
    for (int k = 0; k <= nh; ++k) {
        net.woff[k] = off;
        off += (long long)mlp->dims[k + 1] * mlp->dims[k] + mlp->dims[k + 1];
    }
    for (int k = 0; k < nh; ++k) {
        if (mlp->dims[k + 1] > kWpad) return AMLP_ERR_UNSUPPORTED;
        net.kin[k] = k == 0 ? 48 : net.nout[k - 1];
        net.nout[k] = (mlp->dims[k + 1] + 15) / 16 * 16;
        net.wsm_off[k] = wsm;
        wsm += 2 * net.nout[k] * net.kin[k] * 2;
        net.bias_off[k] = par;
        par += net.nout[k];
    }
    net.bias_off[nh] = par;
    par += kWpad + 4;
    net.wsm_total = wsm;
    net.par_total = par;
    const int npts = nep->npts;
    const int rs = 6 * npts + 1 - ((6 * npts) & 1);
    const size_t r_bytes = align_up((size_t)kAP * rs * 4, 128), ops_bytes = (size_t)2 * 2 * kAP * kWpad * 2;
    static_assert((size_t)kAP * kGS * 4 <= (size_t)2 * kAP * kWpad * 2, "descriptor rows fit an operand tile");
    const size_t tail = align_up(wsm, 128) + align_up((size_t)par * 4, 128) + pair_area_bytes<kAP>() +
                        (size_t)3 * npts * 4 + 16 + 128;
    // R kept apart from the operand tiles (one rotation pass per tile) when it fits
    const size_t row_bytes = (size_t)kAP * kGS * 4;
    const size_t smem_keep = r_bytes + ops_bytes + tail;
    const size_t smem_shared = std::max(r_bytes, ops_bytes) + row_bytes + tail;
    const int keep_r = smem_keep <= 220 * 1024 ? 1 : 0;
    const size_t smem = keep_r ? smem_keep : smem_shared;
    // the shapes and nets taken: those that leave room for a second copy of the rows
    if (smem + (keep_r ? 0 : row_bytes) > 220 * 1024) return AMLP_ERR_UNSUPPORTED;
    using Cfg = NepCfg<10, 8, 4, 12>;
    cudaStream_t s = as_stream(stream);
    const float inv_rc = 1.0f / nep->nep_cutoff, rng = nep->en_max - nep->en_min;
    if (d_rep) {
        AMLP_CHECK_CUDA(cudaFuncSetAttribute(k_forces_adjoint<Cfg, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem));
        k_forces_adjoint<Cfg, true><<<kNumSM, kAThreads, smem, s>>>(d_pos, d_quat, box, d_pairs, d_npairs, cap,
                                                                    nep->d_pts, npts, inv_rc, nep->en_min, rng, net,
                                                                    mlp->d_w, d_F, d_T, d_pe, d_rep, d_rp, keep_r);
    } else {
        AMLP_CHECK_CUDA(cudaFuncSetAttribute(k_forces_adjoint<Cfg, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem));
        k_forces_adjoint<Cfg, false><<<kNumSM, kAThreads, smem, s>>>(d_pos, d_quat, box, d_pairs, d_npairs, cap,
                                                                     nep->d_pts, npts, inv_rc, nep->en_min, rng, net,
                                                                     mlp->d_w, d_F, d_T, d_pe, nullptr, nullptr,
                                                                     keep_r);
    }
    return check_launch();
}

extern "C" amlp_status amlp_forces_adjoint(const float *d_pos, const float *d_quat, float box, const int *d_pairs,
                                           const long long *d_npairs, long long cap, const amlp_nep *nep,
                                           const amlp_mlp *mlp, float *d_F, float *d_T, double *d_pe,
                                           void *stream) {
    return launch_adjoint(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep, mlp, d_F, d_T, d_pe, nullptr, nullptr,
                          stream);
}

extern "C" amlp_status amlp_multi_forces_adjoint(const float *d_pos, const float *d_quat, const int *d_rep,
                                                 const amlp_replica *d_rp, const int *d_pairs,
                                                 const long long *d_npairs, long long cap, const amlp_nep *nep,
                                                 const amlp_mlp *mlp, float *d_F, float *d_T, double *d_pe,
                                                 void *stream) {
    if (!d_rep || !d_rp) return AMLP_ERR_INVALID_ARG;
    return launch_adjoint(d_pos, d_quat, 0.f, d_pairs, d_npairs, cap, nep, mlp, d_F, d_T, d_pe, d_rep, d_rp, stream);
}


constexpr size_t kMlpSmemMax = 226 * 1024;  // dynamic shared memory of k_mlp_grad and k_mlp_pair

// The net of the wide path and its kernels' geometry: Kg = padded descriptor
// width (the first layer's K), g_ld = row stride of the g rows.
static amlp_status wide_net(const amlp_mlp *mlp, int Kg, int g_ld, AdjNet *net) {
    const int nh = mlp->n_layers - 1;
    if (nh < 1 || nh > kMaxHiddenWide) return AMLP_ERR_UNSUPPORTED;
    *net = AdjNet{};
    net->nh = nh;
    net->act = mlp->act;
    long long off = 0;
    int par = 0, wbytes = 0;
    for (int k = 0; k <= mlp->n_layers; ++k) net->dims[k] = mlp->dims[k];
    for (int k = 0; k <= nh; ++k) {
        net->woff[k] = off;
        off += (long long)mlp->dims[k + 1] * mlp->dims[k] + mlp->dims[k + 1];
    }
    for (int k = 0; k < nh; ++k) {
        if (mlp->dims[k + 1] > kWideMax) return AMLP_ERR_UNSUPPORTED;
        net->kin[k] = k == 0 ? Kg : net->nout[k - 1];
        net->nout[k] = (mlp->dims[k + 1] + 15) / 16 * 16;
        net->bias_off[k] = par;
        par += net->nout[k];
        net->wsm_off[k] = net->wsm_total;  // pre-split weights of layer k: hi then lo
        net->wsm_total += 4 * net->nout[k] * net->kin[k];
        wbytes = std::max(wbytes, 4 * net->nout[k] * net->kin[k]);
        net->wmax = std::max(net->wmax, net->nout[k]);
    }
    net->bias_off[nh] = par;
    par += kWideMax + 4;
    net->par_total = par;
    net->g_ld = g_ld;
    net->gp = Kg;
    net->zbw = std::max(Kg, net->wmax);
    net->relu_bits = mlp->act == AMLP_ACT_RELU ? 1 : 0;
    // smooth activations keep act'(z) of nh - 1 layers in TMEM beside the product region
    if (!net->relu_bits && net->zbw + (nh - 1) * net->wmax > 512) return AMLP_ERR_UNSUPPORTED;
    size_t o = align_up((size_t)2 * kAP * net->zbw * 2, 128);  // operand tile, bf16 hi + lo
    net->wbuf_off = (int)o;
    o += align_up((size_t)wbytes, 128);
    net->par_off = (int)o;
    o += align_up((size_t)par * 4, 128);
    net->eps_off = (int)o;
    o += align_up((size_t)kMQ * kAP * 4, 128);
    net->gbuf_off = (int)o;
    const size_t with_g = o + (size_t)kAP * g_ld * 4;
    net->prefetch_g = with_g <= kMlpSmemMax ? 1 : 0;
    net->smem = (int)(net->prefetch_g ? with_g : o);
    if ((size_t)net->smem > kMlpSmemMax) return AMLP_ERR_UNSUPPORTED;
    // two tiles in flight (k_mlp_pair) where both operand tiles fit beside a layer's weights
    // (faster at every width measured: 128 x 2 silu 490 -> 335 us, 150 x 4 ReLU with the first
    // tile in TMEM 960 -> 581 us); the other nets take k_mlp_grad. TMEM regions start at
    // multiples of 32 columns.
    const size_t tile = align_up((size_t)2 * kAP * net->zbw * 2, 128);
    const size_t rest = align_up((size_t)wbytes, 128) + align_up((size_t)par * 4, 128) + (size_t)2 * kPG * kAP * 4;
    const int df = net->relu_bits ? 0 : 2 * (nh - 1) * net->wmax;
    net->pair_d = (int)align_up((size_t)net->zbw, 32);
    net->pair = 0;
    if (2 * tile + rest <= kMlpSmemMax && 2 * net->pair_d + df <= 512) net->pair = 1;
    else if (net->relu_bits && tile + rest <= kMlpSmemMax && 3 * net->pair_d <= 512) net->pair = 2;
    net->pair_tile = (int)tile;
    net->pair_wbuf = (int)(net->pair == 1 ? 2 * tile : tile);
    net->pair_par = net->pair_wbuf + (int)align_up((size_t)wbytes, 128);
    net->pair_eps = net->pair_par + (int)align_up((size_t)par * 4, 128);
    net->pair_smem = net->pair_eps + 2 * kPG * kAP * 4;
    return AMLP_OK;
}

// The net pass over the g rows: the weights split once, then k_mlp_pair or k_mlp_grad.
static amlp_status launch_net(const AdjNet &net, const float *g_rows, const long long *d_npairs, long long cap,
                              const float *d_w, char *wsplit, float *y_rows, float *dg_rows, cudaStream_t s) {
    k_split_weights<<<kNumSM, 128, 0, s>>>(net, d_w, wsplit);
    auto kern = k_mlp_grad;
    if (net.pair == 2) kern = k_mlp_pair<AMLP_ACT_RELU, true>;
    else if (net.pair && net.relu_bits) kern = k_mlp_pair<AMLP_ACT_RELU, false>;
    else if (net.pair) kern = net.act == AMLP_ACT_TANH ? k_mlp_pair<AMLP_ACT_TANH, false> : k_mlp_pair<AMLP_ACT_SILU, false>;
    const int smem = net.pair ? net.pair_smem : net.smem;
    AMLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<kNumSM, net.pair ? kPThreads : kMThreads, smem, s>>>(g_rows, d_npairs, cap, net, d_w, wsplit, y_rows,
                                                               dg_rows);
    return AMLP_OK;
}

extern "C" amlp_status amlp_adjoint_workspace_bytes(long long cap, size_t *bytes) {
    if (cap < 0 || !bytes) return AMLP_ERR_INVALID_ARG;
    *bytes = align_up((size_t)cap * kGRow * 4) + align_up((size_t)cap * kGP * 4) + align_up((size_t)cap * 4) +
             align_up(kWeightSplitBytes) + align_up(adj_a_bytes(cap)) + 256;
    return AMLP_OK;
}

// Body points the harmonic descriptor passes take (at 48, 98 KB of shared memory per block).
constexpr int kHarmonicMaxPts = 48;
static size_t wide_desc_smem(int npts) {
    const int rs = 6 * npts + 1 - ((6 * npts) & 1);
    return align_up((size_t)kDP * rs * 4, 128) + (size_t)kDP * kGS * 4 + pair_area_bytes<kDP>() +
           (size_t)3 * npts * 4;
}

static amlp_status check_pair_args(const float *d_pos, const float *d_quat, const int *d_pairs,
                                   const long long *d_npairs, long long cap, const amlp_nep *nep) {
    amlp_status st = check_nep(nep);
    if (st) return st;
    if (!d_pos || !d_quat || !d_npairs || cap < 0 || (cap > 0 && !d_pairs)) return AMLP_ERR_INVALID_ARG;
    if (hyper_kind(nep) == 2) return 2 * nep->npts <= direct::kMaxNd ? AMLP_OK : AMLP_ERR_UNSUPPORTED;
    if (hyper_kind(nep) != 1 || nep_D(nep) > kGP) return AMLP_ERR_UNSUPPORTED;
    return AMLP_OK;
}

// The wide path and amlp_pair_descriptors take the direct-form descriptor
// passes for the hypers (10, 10, 10) and, for (10, 8, 4), for clouds of at most
// 12 points (th_v1, cube_v2), where the O(Nd^2) sum costs less than the
// harmonic form; the multi-system path keeps the harmonic form.
constexpr int kDirectMaxNd47 = 12;
static bool use_direct(const amlp_nep *nep) {
    return hyper_kind(nep) == 2 || (hyper_kind(nep) == 1 && 2 * nep->npts <= kDirectMaxNd47);
}

// Launch of a direct-form descriptor kernel: one thread per pair, grid-stride
// over at most 16 blocks per SM, one float4 of shared memory per point and thread.
template <class K, class... Args>
static amlp_status launch_direct(K kernel, long long cap, int npts, cudaStream_t s, Args... args) {
    const size_t smem = direct::smem_bytes(2 * npts);
    if (smem > 48 * 1024)
        AMLP_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long blocks = min((cap + direct::kThreads - 1) / direct::kThreads, (long long)kNumSM * 16);
    kernel<<<(unsigned)blocks, direct::kThreads, smem, s>>>(args...);
    return AMLP_OK;
}

// Stage events of the wide path (amlp_stage_timing): one set for the library,
// recorded by the last call on its stream.
static bool g_stage_timing = false;
static bool g_stage_recorded = false;
static cudaEvent_t g_stage_ev[4];

static void stage_mark(int k, cudaStream_t s) {
    if (!g_stage_timing) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;  // not in graphs
    cudaEventRecord(g_stage_ev[k], s);
    if (k == 3) g_stage_recorded = true;
}

static amlp_status launch_adjoint_wide(const float *d_pos, const float *d_quat, float box, const int *d_pairs,
                                       const long long *d_npairs, long long cap, const amlp_nep *nep,
                                       const amlp_mlp *mlp, const float *d_wt, int clip, float *d_F, float *d_T,
                                       double *d_pe, const int *d_rep, const amlp_replica *d_rp, void *d_ws,
                                       size_t ws_bytes, void *stream) {
    amlp_status st = check_pair_args(d_pos, d_quat, d_pairs, d_npairs, cap, nep);
    if (st) return st;
    if ((st = check_mlp(mlp, nep_D(nep)))) return st;
    if (!d_F || !d_T) return AMLP_ERR_INVALID_ARG;
    if (cap == 0) return AMLP_OK;
    size_t need;
    amlp_adjoint_workspace_bytes(cap, &need);
    if (!d_ws || ws_bytes < need) return AMLP_ERR_WORKSPACE;
    cudaStream_t s = as_stream(stream);
    const float inv_rc = 1.0f / nep->nep_cutoff, rng = nep->en_max - nep->en_min;
    AdjNet net;
    if (hyper_kind(nep) == 2 || (use_direct(nep) && !d_rep)) {  // the direct-form passes around the same net kernel
        if (d_rep) return AMLP_ERR_UNSUPPORTED;
        const bool k2 = hyper_kind(nep) == 2;
        const int gp = k2 ? kGP2 : kGP, grow = k2 ? kGRow2 : kGRow;
        if ((st = wide_net(mlp, gp, grow, &net))) return st;
        Carver c(d_ws, ws_bytes);
        float *g_rows = c.take<float>((size_t)cap * grow);
        float *dg_rows = c.take<float>((size_t)cap * gp);
        float *y_rows = c.take<float>((size_t)cap);
        char *wsplit = c.take<char>(kWeightSplitBytes);
        if (!c.ok()) return AMLP_ERR_WORKSPACE;
        const int npts = nep->npts;
        auto fwd = k2 ? direct::k_desc_direct_fwd<11, 11, 10> : direct::k_desc_direct_fwd<11, 9, 4>;
        auto bwd = k2 ? direct::k_desc_direct_bwd<11, 11, 10> : direct::k_desc_direct_bwd<11, 9, 4>;
        stage_mark(0, s);
        if ((st = launch_direct(fwd, cap, npts, s, d_pos, d_quat, box, d_pairs, d_npairs, cap,
                                (const float *)nep->d_pts, npts, inv_rc, g_rows, grow)))
            return st;
        stage_mark(1, s);
        if ((st = launch_net(net, g_rows, d_npairs, cap, mlp->d_w, wsplit, y_rows, dg_rows, s))) return st;
        stage_mark(2, s);
        if ((st = launch_direct(bwd, cap, npts, s, d_pos, d_quat, box, d_pairs, d_npairs, cap,
                                (const float *)nep->d_pts, npts, inv_rc, nep->en_min, rng, (const float *)dg_rows, gp,
                                (const float *)y_rows, d_wt, clip, d_F, d_T, d_pe)))
            return st;
        stage_mark(3, s);
        return check_launch();
    }
    if ((st = wide_net(mlp, kGP, kGRow, &net))) return st;
    Carver c(d_ws, ws_bytes);
    float *g_rows = c.take<float>((size_t)cap * kGRow);
    float *dg_rows = c.take<float>((size_t)cap * kGP);
    float *y_rows = c.take<float>((size_t)cap);
    char *wsplit = c.take<char>(kWeightSplitBytes);
    float *a_rows = c.take<float>(adj_a_bytes(cap) / 4);
    const int npts = nep->npts;
    const size_t smem_desc = wide_desc_smem(npts);
    if (npts > kHarmonicMaxPts) return AMLP_ERR_UNSUPPORTED;
    using Cfg = NepCfg<10, 8, 4, 12>;
    const bool multi = d_rep != nullptr;
    auto fwd = multi ? k_adj_desc<Cfg, true, false> : k_adj_desc<Cfg, false, false>;
    auto bwd = multi ? k_adj_desc<Cfg, true, true> : k_adj_desc<Cfg, false, true>;
    AMLP_CHECK_CUDA(cudaFuncSetAttribute(fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_desc));
    AMLP_CHECK_CUDA(cudaFuncSetAttribute(bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_desc));
    stage_mark(0, s);
    fwd<<<2 * kNumSM, kDThreads, smem_desc, s>>>(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep->d_pts, npts, inv_rc,
                                             nep->en_min, rng, g_rows, kGRow, nullptr, nullptr, nullptr, clip, d_F,
                                             d_T, d_pe, d_rep, d_rp, a_rows);
    stage_mark(1, s);
    if ((st = launch_net(net, g_rows, d_npairs, cap, mlp->d_w, wsplit, y_rows, dg_rows, s))) return st;
    stage_mark(2, s);
    bwd<<<2 * kNumSM, kDThreads, smem_desc, s>>>(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep->d_pts, npts, inv_rc,
                                             nep->en_min, rng, nullptr, kGP, dg_rows, y_rows, d_wt, clip, d_F, d_T,
                                             d_pe, d_rep, d_rp, a_rows);
    stage_mark(3, s);
    return check_launch();
}

extern "C" amlp_status amlp_forces_adjoint_wide(const float *d_pos, const float *d_quat, float box,
                                                const int *d_pairs, const long long *d_npairs, long long cap,
                                                const amlp_nep *nep, const amlp_mlp *mlp, float *d_F, float *d_T,
                                                double *d_pe, void *d_ws, size_t ws_bytes, void *stream) {
    return launch_adjoint_wide(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep, mlp, nullptr, 1, d_F, d_T, d_pe,
                               nullptr, nullptr, d_ws, ws_bytes, stream);
}

extern "C" amlp_status amlp_multi_forces_adjoint_wide(const float *d_pos, const float *d_quat, const int *d_rep,
                                                      const amlp_replica *d_rp, const int *d_pairs,
                                                      const long long *d_npairs, long long cap, const amlp_nep *nep,
                                                      const amlp_mlp *mlp, float *d_F, float *d_T, double *d_pe,
                                                      void *d_ws, size_t ws_bytes, void *stream) {
    if (!d_rep || !d_rp) return AMLP_ERR_INVALID_ARG;
    return launch_adjoint_wide(d_pos, d_quat, 0.f, d_pairs, d_npairs, cap, nep, mlp, nullptr, 1, d_F, d_T, d_pe,
                               d_rep, d_rp, d_ws, ws_bytes, stream);
}

extern "C" amlp_status amlp_pair_energy_vjp(const float *d_pos, const float *d_quat, float box, const int *d_pairs,
                                            const long long *d_npairs, long long cap, const amlp_nep *nep,
                                            const amlp_mlp *mlp, const float *d_wt, int clip, float *d_F,
                                            float *d_T, double *d_pe, void *d_ws, size_t ws_bytes, void *stream) {
    return launch_adjoint_wide(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep, mlp, d_wt, clip ? 1 : 0, d_F, d_T,
                               d_pe, nullptr, nullptr, d_ws, ws_bytes, stream);
}

extern "C" amlp_status amlp_pair_descriptors(const float *d_pos, const float *d_quat, float box, const int *d_pairs,
                                             const long long *d_npairs, long long cap, const amlp_nep *nep,
                                             float *d_g, int ld_g, void *stream) {
    amlp_status st = check_pair_args(d_pos, d_quat, d_pairs, d_npairs, cap, nep);
    if (st) return st;
    if (!d_g || ld_g < nep_D(nep)) return AMLP_ERR_INVALID_ARG;
    if (cap == 0) return AMLP_OK;
    if (use_direct(nep)) {
        auto fwd = hyper_kind(nep) == 2 ? direct::k_desc_direct_fwd<11, 11, 10> : direct::k_desc_direct_fwd<11, 9, 4>;
        if ((st = launch_direct(fwd, cap, nep->npts, as_stream(stream), d_pos, d_quat, box, d_pairs, d_npairs, cap,
                                (const float *)nep->d_pts, nep->npts, 1.0f / nep->nep_cutoff, d_g, ld_g)))
            return st;
        return check_launch();
    }
    const size_t smem = wide_desc_smem(nep->npts);
    if (nep->npts > kHarmonicMaxPts) return AMLP_ERR_UNSUPPORTED;
    using Cfg = NepCfg<10, 8, 4, 12>;
    auto fwd = k_adj_desc<Cfg, false, false>;
    AMLP_CHECK_CUDA(cudaFuncSetAttribute(fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fwd<<<2 * kNumSM, kDThreads, smem, as_stream(stream)>>>(d_pos, d_quat, box, d_pairs, d_npairs, cap, nep->d_pts,
                                                        nep->npts, 1.0f / nep->nep_cutoff, nep->en_min,
                                                        nep->en_max - nep->en_min, d_g, ld_g, nullptr, nullptr,
                                                        nullptr, 1, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                        nullptr);
    return check_launch();
}

extern "C" amlp_status amlp_stage_timing(int enable) {
    if (enable && !g_stage_ev[0]) {
        for (auto &e : g_stage_ev) AMLP_CHECK_CUDA(cudaEventCreate(&e));
    }
    g_stage_timing = enable != 0;
    return AMLP_OK;
}

extern "C" amlp_status amlp_stage_times(float *h_ms3) {
    if (!h_ms3) return AMLP_ERR_INVALID_ARG;
    if (!g_stage_recorded) return AMLP_ERR_INVALID_ARG;  // no call recorded its stages yet
    AMLP_CHECK_CUDA(cudaEventSynchronize(g_stage_ev[3]));
    for (int k = 0; k < 3; ++k) AMLP_CHECK_CUDA(cudaEventElapsedTime(h_ms3 + k, g_stage_ev[k], g_stage_ev[k + 1]));
    return AMLP_OK;
}

extern "C" amlp_status amlp_test_first_wait_limit(int polls) {
    if (polls < -1) return AMLP_ERR_INVALID_ARG;
    AMLP_CHECK_CUDA(cudaMemcpyToSymbol(g_amlp_first_wait_limit, &polls, sizeof(int)));
    return AMLP_OK;
}

// The sticky flags as a status, for the handles' synchronisation points (reads
// the flags without clearing them).
amlp_status amlp::device_wait_status() {
    unsigned int f = 0;
    AMLP_CHECK_CUDA(cudaMemcpyFromSymbol(&f, g_amlp_device_error, sizeof(unsigned int)));
    return f ? AMLP_ERR_DEVICE_WAIT : AMLP_OK;
}

extern "C" amlp_status amlp_device_error(unsigned int *flags, int clear) {
    if (!flags) return AMLP_ERR_INVALID_ARG;
    AMLP_CHECK_CUDA(cudaMemcpyFromSymbol(flags, g_amlp_device_error, sizeof(unsigned int)));
    if (clear) {
        unsigned int z = 0;
        AMLP_CHECK_CUDA(cudaMemcpyToSymbol(g_amlp_device_error, &z, sizeof(unsigned int)));
    }
    return AMLP_OK;
}
