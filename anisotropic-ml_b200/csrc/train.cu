// Weight gradient of the pair-energy net for a training step, the loss of the
// reference's training loop (05/FFNN.py:95-106, torch.nn.MSELoss over a batch)
// on energies normalised as 05/FFNN.py:59-63 does (the caller passes
// y = clamp((min(E, en_max) - en_min) / (en_max - en_min), 0, 1)):
//   L = (1/B) sum_r (net(g_r) - y_r)^2.
// The same kernel also backpropagates a given per-row upstream gradient dy_r
// (a vector-Jacobian product, sum_r dy_r d net(g_r) / d theta).
// Backpropagation into every weight and bias, FP32.
//
// A CTA keeps all activations of a tile of R rows in shared memory, feature-major
// (a feature's R values contiguous), and runs the three products of every layer on
// them as register tiles:
//   forward   z[r][n]  = b[n] + sum_k W[n][k] a[r][k]  (ascending k, one rounding per
//             multiply-add), thread = 4 rows x NC columns;
//   gradient  dW[n][k] = sum_r delta[r][n] a[r][k], thread = NJ x NI weights over all
//             rows, a warp's lanes 4 n x 8 consecutive k: one reduction per weight and
//             tile into the caller's gradient buffer, 32 bytes of a row at a time;
//   deltas    delta_prev[r][k] = act' sum_n W[n][k] delta[r][n], thread as forward,
//             written over the activations they belong to (ReLU's and tanh's
//             derivatives follow from the activation; SiLU keeps z beside it).
// The weights are read through L1 (a warp shares each of them), so that the shared
// memory holds rows alone: the more rows per tile, the fewer reductions. R is
// chosen so that the tiles fill whole rounds of the SMs, at most 64.
// Bound by latency with four warps per scheduler: the weights' loads (77 % of them hit
// L1), the barriers between layers and the rows' loads keep the multiply-add pipe at 37 %.
// The forward and the deltas take about three quarters of the time. 16,384 rows of the
// 47-150-150-150-150-1 ReLU net: 330 us, 22 TFLOP/s. Before the tiles, 3,254 us: a
// thread walked one output column over 32 rows with a shared-memory load per
// multiply-add, and every 32 rows paid one reduction per weight.
#include <algorithm>

#include "common.cuh"

namespace amlp {
namespace {

constexpr int kTrainThreads = 512;       // threads per block, one block per SM
// Nets whose inputs and layers are at most 16 wide take four blocks of 128 threads: their tiles
// are barriers and latency, which other blocks' tiles fill. 300,000 rows of 1-3-1 (ReLU): 89
// us, with one block of 512 threads 257, 170 before the tiles; 8-16-16-1: 144 against 404. With 47
// inputs the blocks gain less, and at 1,000 rows (47-16-1) they lose, 14.4 us against 12.3.
constexpr int kTrainSmallThreads = 128;
constexpr int kTrainSmallWidth = 16;
constexpr int kTrainMaxRows = 64;
constexpr int kTrainMaxWidth = 256;
constexpr size_t kTrainSmem = 226 * 1024;

struct TrainNet {
    int n_layers, act;
    int dims[AMLP_MAX_LAYERS + 1];
    long long woff[AMLP_MAX_LAYERS];
    int feat[AMLP_MAX_LAYERS + 1];  // first feature of layer k's activations (then deltas)
    int zfeat[AMLP_MAX_LAYERS + 1]; // SiLU: first feature of layer k's pre-activations
    int rg, ld;                     // row groups of 4 per tile, floats per feature
};

// Features are ld floats apart: ld / 4 is odd, so that 8 lanes' 16-byte reads of
// consecutive features fall in distinct bank groups.
__host__ __device__ constexpr int train_ld(int rg) { return 4 * (rg | 1); }

// acc[i][c] (rows 2 i, 2 i + 1) += sum over k = 0 .. K - 1, ascending, of x[k][rows]
// times the weight of column c: x points at the thread's four rows of feature 0
// (features ld apart). ROWS: column c's weights are consecutive floats at w + c col
// (the forward's, one row of W per column), otherwise the
// columns are consecutive and k's weights are the floats at w + k step (the
// deltas', one row of W per k). The next four k's weights load while four k's
// multiply-adds issue, VEC floats to a load (the rows' alignment; without ROWS, 4 columns):
// at compile time, as the loads' registers decide the loop's (at the 128 registers of the
// block's 512 threads it spills 164 bytes). 50,021 rows of 47-128-128-128-1: 608 us with
// 16-byte loads, 686 with 8 bytes (4 for the deltas) chosen inside the loop; 16,384 rows of
// 47-150 x 4-1, whose rows allow 8 bytes: 323 us against 347.
template <int NC, bool ROWS, int VEC>
__device__ __forceinline__ void train_product(float2 (&acc)[2][NC], const float *x, int ld, int K, const float *w,
                                              int col, int step) {
    const float *p[ROWS ? NC : 1];
    p[0] = w;
    if (ROWS) {
#pragma unroll
        for (int c = 1; c < NC; ++c) p[c] = w + c * col;
    }
    auto mul = [&](const float4 &xv, const float (&wv)[NC]) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            acc[0][c] = fma2(make_float2(xv.x, xv.y), make_float2(wv[c], wv[c]), acc[0][c]);
            acc[1][c] = fma2(make_float2(xv.z, xv.w), make_float2(wv[c], wv[c]), acc[1][c]);
        }
    };
    auto load1 = [&](float (&wv)[NC]) {  // the next k's weights
#pragma unroll
        for (int c = 0; c < NC; ++c) wv[c] = ROWS ? __ldg(p[c]) : __ldg(p[0] + c);
        if (ROWS) {
#pragma unroll
            for (int c = 0; c < NC; ++c) ++p[c];
        } else {
            p[0] += step;
        }
    };
    auto load4 = [&](float (&wv)[4][NC]) {
        if constexpr (ROWS && VEC == 4) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(p[c]));
                wv[0][c] = a.x, wv[1][c] = a.y, wv[2][c] = a.z, wv[3][c] = a.w;
                p[c] += 4;
            }
        } else if constexpr (!ROWS && VEC == 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(p[0]));
                wv[u][0] = a.x, wv[u][1] = a.y, wv[u][2] = a.z, wv[u][3] = a.w;
                p[0] += step;
            }
        } else if constexpr (ROWS && VEC == 2) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float2 a = __ldg(reinterpret_cast<const float2 *>(p[c]));
                const float2 b = __ldg(reinterpret_cast<const float2 *>(p[c]) + 1);
                wv[0][c] = a.x, wv[1][c] = a.y, wv[2][c] = b.x, wv[3][c] = b.y;
                p[c] += 4;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) load1(wv[u]);
        }
    };
    int k = 0;
    if (K >= 4) {
        float cur[4][NC];
        load4(cur);
#pragma unroll 1
        for (k = 4; k + 4 <= K; k += 4, x += 4 * ld) {
            float nxt[4][NC];
            load4(nxt);
#pragma unroll
            for (int u = 0; u < 4; ++u) mul(*reinterpret_cast<const float4 *>(x + u * ld), cur[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int c = 0; c < NC; ++c) cur[u][c] = nxt[u][c];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) mul(*reinterpret_cast<const float4 *>(x + u * ld), cur[u]);
        x += 4 * ld;
    }
#pragma unroll 1
    for (; k < K; ++k, x += ld) {
        float wv[NC];
        load1(wv);
        mul(*reinterpret_cast<const float4 *>(x), wv);
    }
}

// Floats per load that the rows of W (K each) are aligned to: 4, 2 or 1.
__device__ __forceinline__ int train_vec(const float *W, int K) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(W) | (uintptr_t)K * sizeof(float);
    return (a & 15) == 0 ? 4 : ((a & 7) == 0 ? 2 : 1);
}

// Consecutive columns per thread of a layer of n, ncg column groups: 1 to 5, or two
// groups of 4.
__device__ __forceinline__ int train_columns(int n, int ncg) {
    const int nc = (n + ncg - 1) / ncg;
    return nc > 5 ? 8 : nc;
}

// First of a thread's NC consecutive columns from c0, moved back so that all lie
// below n (the columns below c0 then belong to another thread).
__device__ __forceinline__ int train_first(int c0, int nc, int n) { return max(0, min(c0, n - nc)); }

struct TrainTile {
    float *sm;
    int tid, rg, cg, ncg;  // row group (4 rows), column group and their number
    int nr;                // rows of the batch in the tile
    bool on;               // threads past the last whole column group idle in the products
};

// The thread's four rows v, zero past the tile's last one. Those rows' forward runs on zero
// inputs, and a net that overflows there would turn their zero deltas into NaN.
__device__ __forceinline__ float4 train_rows(const TrainTile &t, float4 v) {
    const int left = t.nr - 4 * t.rg;
    if (left < 4) {
        v.w = 0.f;
        if (left < 3) v.z = 0.f;
        if (left < 2) v.y = 0.f;
        if (left < 1) v.x = 0.f;
    }
    return v;
}

// Layer L forward for NC columns per thread from n0.
template <int NC>
__device__ __forceinline__ void train_forward(const TrainNet &net, const TrainTile &t, const float *wts, int L,
                                              int n0) {
    const int K = net.dims[L], N = net.dims[L + 1], ld = net.ld;
    const float *W = wts + net.woff[L], *b = W + (size_t)N * K;
    const bool last = L == net.n_layers - 1;
    const int f = train_first(n0, NC, N);
    float2 acc[2][NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const float bv = __ldg(b + f + c);
        acc[0][c] = acc[1][c] = make_float2(bv, bv);
    }
    const float *x = t.sm + net.feat[L] * ld + 4 * t.rg, *Wf = W + (size_t)f * K;
    const int vec = train_vec(W, K);
    if (vec == 4) train_product<NC, true, 4>(acc, x, ld, K, Wf, K, 0);
    else if (vec == 2) train_product<NC, true, 2>(acc, x, ld, K, Wf, K, 0);
    else train_product<NC, true, 1>(acc, x, ld, K, Wf, K, 0);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const int n = f + c;
        if (n < n0) continue;
        const float z[4] = {acc[0][c].x, acc[0][c].y, acc[1][c].x, acc[1][c].y};
        float a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = last ? z[i] : act_f(net.act, z[i]);
        *reinterpret_cast<float4 *>(t.sm + (net.feat[L + 1] + n) * ld + 4 * t.rg) =
            train_rows(t, make_float4(a[0], a[1], a[2], a[3]));
        if (!last && net.act == AMLP_ACT_SILU)
            *reinterpret_cast<float4 *>(t.sm + (net.zfeat[L + 1] + n) * ld + 4 * t.rg) =
                train_rows(t, make_float4(z[0], z[1], z[2], z[3]));
    }
}

// The deltas of layer L's inputs without act', for NC columns per thread from
// train_first(k0, NC, K), into out.
template <int NC>
__device__ __forceinline__ void train_deltas(const TrainNet &net, const TrainTile &t, const float *wts, int L, int k0,
                                             float4 *out) {
    const int K = net.dims[L], N = net.dims[L + 1], ld = net.ld;
    const float *W = wts + net.woff[L];
    float2 acc[2][NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[0][c] = acc[1][c] = make_float2(0.f, 0.f);
    const float *x = t.sm + net.feat[L + 1] * ld + 4 * t.rg, *Wk = W + train_first(k0, NC, K);
    if constexpr (NC == 4) {
        if (train_vec(W, K) == 4 && (k0 & 3) == 0) {
            train_product<NC, false, 4>(acc, x, ld, N, Wk, 0, K);
        } else {
            train_product<NC, false, 1>(acc, x, ld, N, Wk, 0, K);
        }
    } else {
        train_product<NC, false, 1>(acc, x, ld, N, Wk, 0, K);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = make_float4(acc[0][c].x, acc[0][c].y, acc[1][c].x, acc[1][c].y);
}

// act' times the delta d of the thread's rows of feature k, over the activations.
__device__ __forceinline__ void train_store_delta(const TrainNet &net, const TrainTile &t, int L, int k, float4 dv) {
    float4 *dst = reinterpret_cast<float4 *>(t.sm + (net.feat[L] + k) * net.ld + 4 * t.rg);
    const float4 av = *dst;
    const float a[4] = {av.x, av.y, av.z, av.w};
    float d[4] = {dv.x, dv.y, dv.z, dv.w};
    if (net.act == AMLP_ACT_SILU) {
        const float4 zv = *reinterpret_cast<const float4 *>(t.sm + (net.zfeat[L] + k) * net.ld + 4 * t.rg);
        const float z[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] *= act_df(AMLP_ACT_SILU, z[i]);
    } else if (net.act == AMLP_ACT_TANH) {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] *= 1.0f - a[i] * a[i];
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] *= a[i] > 0.0f ? 1.0f : 0.0f;
    }
    *dst = train_rows(t, make_float4(d[0], d[1], d[2], d[3]));
}

// dL/dW of layer L from its deltas and inputs, in tiles of 4 NJ x 8 NI weights per warp:
// lane (n, k) of 4 x 8 takes rows n + 4 j and columns k + 8 i. A warp's 16-byte reads of
// four rows of the activations then touch 8 features (one wavefront) and those of the
// deltas 4; with all lanes along k, the same 40 multiply-adds took 21 wavefronts instead
// of 9 and the shared memory bounded them (47-128-128-128-1, 50,021 rows: 608 -> 589 us;
// the reductions, in 32-byte pieces now, cost the 150-wide net 1 %).
template <int NT, int NI, int NJ>
__device__ __forceinline__ void train_weights(const TrainNet &net, const TrainTile &t, float *grad, int L) {
    constexpr int nw = NT / 32;
    const int K = net.dims[L], N = net.dims[L + 1], ld = net.ld, R = 4 * net.rg;
    const int lane = t.tid & 31, nkb = (K + 8 * NI - 1) / (8 * NI), nnb = (N + 4 * NJ - 1) / (4 * NJ);
    float *gW = grad + net.woff[L];
#pragma unroll 1
    for (int tl = t.tid >> 5; tl < nkb * nnb; tl += nw) {
        const int nb = tl / nkb, k0 = (tl - nb * nkb) * 8 * NI + (lane & 7), n0 = nb * 4 * NJ + (lane >> 3);
        const float *a[NI], *d[NJ];
        float2 acc[NJ][NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) a[i] = t.sm + (net.feat[L] + min(k0 + 8 * i, K - 1)) * ld;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            d[j] = t.sm + (net.feat[L + 1] + min(n0 + 4 * j, N - 1)) * ld;
#pragma unroll
            for (int i = 0; i < NI; ++i) acc[j][i] = make_float2(0.f, 0.f);
        }
#pragma unroll 1
        for (int r = 0; r < R; r += 4) {
            float4 av[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) av[i] = *reinterpret_cast<const float4 *>(a[i] + r);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float4 dv = *reinterpret_cast<const float4 *>(d[j] + r);
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    acc[j][i] = fma2(make_float2(dv.x, dv.y), make_float2(av[i].x, av[i].y), acc[j][i]);
                    acc[j][i] = fma2(make_float2(dv.z, dv.w), make_float2(av[i].z, av[i].w), acc[j][i]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int n = n0 + 4 * j;
            if (n >= N) break;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int k = k0 + 8 * i;
                if (k < K) atomicAdd(gW + (size_t)n * K + k, acc[j][i].x + acc[j][i].y);
            }
        }
    }
}

// Multiply-adds per lane and row of a layer's tiles: whole rounds of the warps.
template <int NT>
__device__ __forceinline__ int train_tile_cost(int N, int K, int NI, int NJ) {
    const int tiles = ((K + 8 * NI - 1) / (8 * NI)) * ((N + 4 * NJ - 1) / (4 * NJ));
    constexpr int nw = NT / 32;
    return (tiles + nw - 1) / nw * NI * NJ;
}

// dL/db of layer L.
template <int NT>
__device__ __forceinline__ void train_bias(const TrainNet &net, const TrainTile &t, float *grad, int L) {
    const int K = net.dims[L], N = net.dims[L + 1], ld = net.ld, R = 4 * net.rg;
    float *gb = grad + net.woff[L] + (size_t)N * K;
    for (int n = t.tid; n < N; n += NT) {
        const float *d = t.sm + (net.feat[L + 1] + n) * ld;
        float s = 0.f;
        for (int r = 0; r < R; r += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(d + r);
            s += (v.x + v.y) + (v.z + v.w);
        }
        atomicAdd(gb + n, s);
    }
}

template <int NT>
__global__ void __launch_bounds__(NT, kTrainThreads / NT) k_mlp_loss_grad(const float *g, const float *y,
                                                                         const float *dy, long long rows, TrainNet net,
                                                                         const float *w, float *grad, double *loss) {
    extern __shared__ __align__(16) float sm[];
    const int ld = net.ld, R = 4 * net.rg;
    TrainTile t;
    t.sm = sm;
    t.tid = threadIdx.x;
    t.ncg = NT / net.rg;
    t.cg = t.tid / net.rg;
    t.rg = t.tid - t.cg * net.rg;
    t.on = t.cg < t.ncg;
    const float inv_b = 1.0f / (float)rows;
    for (long long r0 = (long long)blockIdx.x * R; r0 < rows; r0 += (long long)gridDim.x * R) {
        const int nr = t.nr = (int)min((long long)R, rows - r0);
        const int D = net.dims[0];
        // the tile's descriptor rows, a warp per row (coalesced); rows past the end are zero
        for (int r = t.tid >> 5; r < R; r += NT / 32)
            for (int d = t.tid & 31; d < D; d += 32) sm[d * ld + r] = r < nr ? g[(r0 + r) * D + d] : 0.f;
        __syncthreads();
        for (int L = 0; L < net.n_layers; ++L) {
            if (t.on) {
                // nc consecutive columns per thread
                const int N = net.dims[L + 1], nc = train_columns(N, t.ncg), n0 = t.cg * nc;
                if (n0 < N) {
                    if (nc == 8) {
                        train_forward<4>(net, t, w, L, n0);
                        if (n0 + 4 < N) train_forward<4>(net, t, w, L, n0 + 4);
                    } else if (nc == 5) train_forward<5>(net, t, w, L, n0);
                    else if (nc == 4) train_forward<4>(net, t, w, L, n0);
                    else if (nc == 3) train_forward<3>(net, t, w, L, n0);
                    else if (nc == 2) train_forward<2>(net, t, w, L, n0);
                    else train_forward<1>(net, t, w, L, n0);
                }
            }
            __syncthreads();
        }
        // output delta: dy, or dL/dz_last = 2 (net - y) / B and the loss
        if (t.tid < kTrainMaxRows) {
            float *out = sm + net.feat[net.n_layers] * ld + t.tid;
            float d = 0.f;
            double l = 0.0;
            if (t.tid < nr && dy) {
                d = dy[r0 + t.tid];
            } else if (t.tid < nr) {
                float e = *out - y[r0 + t.tid];
                d = 2.0f * e * inv_b;
                l = (double)e * (double)e / (double)rows;
            }
            if (t.tid < R) *out = d;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if ((t.tid & 31) == 0 && loss && l != 0.0) atomicAdd(loss, l);
        }
        __syncthreads();
        for (int L = net.n_layers - 1; L >= 0; --L) {
            const int K = net.dims[L], N = net.dims[L + 1];
            // the tile with which the layer's tiles cost the warps least
            const int c55 = train_tile_cost<NT>(N, K, 5, 5), c54 = train_tile_cost<NT>(N, K, 5, 4);
            const int c44 = train_tile_cost<NT>(N, K, 4, 4), c34 = train_tile_cost<NT>(N, K, 3, 4);
            const int least = min(min(c55, c54), min(c44, c34));
            if (c55 == least) train_weights<NT, 5, 5>(net, t, grad, L);
            else if (c54 == least) train_weights<NT, 5, 4>(net, t, grad, L);
            else if (c44 == least) train_weights<NT, 4, 4>(net, t, grad, L);
            else train_weights<NT, 3, 4>(net, t, grad, L);
            train_bias<NT>(net, t, grad, L);
            if (L == 0) break;
            const int nc = train_columns(K, t.ncg), k0 = t.cg * nc;
            const bool mine = t.on && k0 < K;
            float4 d[8];
            if (mine) {
                if (nc == 8) {
                    train_deltas<4>(net, t, w, L, k0, d);
                    if (k0 + 4 < K) train_deltas<4>(net, t, w, L, k0 + 4, d + 4);
                } else if (nc == 5) train_deltas<5>(net, t, w, L, k0, d);
                else if (nc == 4) train_deltas<4>(net, t, w, L, k0, d);
                else if (nc == 3) train_deltas<3>(net, t, w, L, k0, d);
                else if (nc == 2) train_deltas<2>(net, t, w, L, k0, d);
                else train_deltas<1>(net, t, w, L, k0, d);
            }
            __syncthreads();  // every thread has read layer L's activations (its weight gradient)
            if (mine) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    // d[c] is the delta of column train_first(s0, ..) + c of its group
                    const int s0 = nc == 8 && c >= 4 ? k0 + 4 : k0;
                    const int k = nc == 8 ? train_first(s0, 4, K) + (c & 3) : train_first(s0, nc, K) + c;
                    if (c < nc && s0 < K && k >= s0) train_store_delta(net, t, L, k, d[c]);
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

}  // namespace

amlp_status check_mlp(const amlp_mlp *m, int D);

}  // namespace amlp

using namespace amlp;

static amlp_status launch_grad(const float *d_g, const float *d_y, const float *d_dy, long long rows,
                               const amlp_mlp *mlp, float *d_grad, double *d_loss, void *stream) {
    if (!mlp || rows < 0) return AMLP_ERR_INVALID_ARG;
    amlp_status st = check_mlp(mlp, mlp->dims[0]);
    if (st) return st;
    if (rows == 0) return AMLP_OK;
    if (!d_g || !(d_y || d_dy) || !d_grad) return AMLP_ERR_INVALID_ARG;
    TrainNet net{};
    net.n_layers = mlp->n_layers;
    net.act = mlp->act;
    long long off = 0;
    int feat = 0;
    for (int k = 0; k <= mlp->n_layers; ++k) {
        net.dims[k] = mlp->dims[k];
        if (mlp->dims[k] > kTrainMaxWidth) return AMLP_ERR_UNSUPPORTED;
        net.feat[k] = feat;
        feat += mlp->dims[k];
    }
    if (feat > 880) return AMLP_ERR_UNSUPPORTED;  // the nets taken: layer widths, D and 1 included, adding up to 880
    if (mlp->act == AMLP_ACT_SILU)
        for (int k = 1; k < mlp->n_layers; ++k) {
            net.zfeat[k] = feat;
            feat += mlp->dims[k];
        }
    for (int k = 0; k < mlp->n_layers; ++k) {
        net.woff[k] = off;
        off += (long long)mlp->dims[k + 1] * mlp->dims[k] + mlp->dims[k + 1];
    }
    int wide = 0;
    for (int k = 0; k < mlp->n_layers; ++k) wide = std::max(wide, mlp->dims[k]);
    const bool small = wide <= kTrainSmallWidth;
    const int blocks = small ? kNumSM * (kTrainThreads / kTrainSmallThreads) : kNumSM;  // running at once
    const size_t room = small ? kTrainSmem / (kTrainThreads / kTrainSmallThreads) : kTrainSmem;
    // Rows per tile: as many as the shared memory holds, at most 64, then the fewest
    // (a multiple of 4) with which the tiles make as few rounds of the blocks
    int rg = kTrainMaxRows / 4;
    while (rg > 1 && (size_t)feat * train_ld(rg) * sizeof(float) > room) --rg;
    const long long rounds = (rows + (long long)blocks * 4 * rg - 1) / ((long long)blocks * 4 * rg);
    const long long per = (rows + blocks * rounds - 1) / (blocks * rounds);
    rg = (int)std::min<long long>(rg, std::max<long long>(1, (per + 3) / 4));
    net.rg = rg;
    net.ld = train_ld(rg);
    const size_t smem = (size_t)feat * net.ld * sizeof(float);
    if (smem > room) return AMLP_ERR_UNSUPPORTED;
    const auto kern = small ? k_mlp_loss_grad<kTrainSmallThreads> : k_mlp_loss_grad<kTrainThreads>;
    AMLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long tiles = (rows + 4 * rg - 1) / (4 * rg);
    const int grid = (int)std::min<long long>(tiles, blocks);
    kern<<<grid, small ? kTrainSmallThreads : kTrainThreads, smem, as_stream(stream)>>>(
        d_g, d_y, d_dy, rows, net, mlp->d_w, d_grad, d_dy ? nullptr : d_loss);
    return check_launch();
}

extern "C" amlp_status amlp_mlp_loss_grad(const float *d_g, const float *d_y, long long rows, const amlp_mlp *mlp,
                                          float *d_grad, double *d_loss, void *stream) {
    if (!d_y && rows > 0) return AMLP_ERR_INVALID_ARG;
    return launch_grad(d_g, d_y, nullptr, rows, mlp, d_grad, d_loss, stream);
}

extern "C" amlp_status amlp_mlp_backward(const float *d_g, const float *d_dy, long long rows, const amlp_mlp *mlp,
                                         float *d_grad, void *stream) {
    if (!d_dy && rows > 0) return AMLP_ERR_INVALID_ARG;
    return launch_grad(d_g, nullptr, d_dy, rows, mlp, d_grad, nullptr, stream);
}
