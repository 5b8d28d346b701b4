// gate.cu — learned smoothness gate of the face flux.
//
// A small MLP (8 -> 32 -> 32 -> 1, GELU, sigmoid; BF16 weights and
// activations, FP32 accumulation on the tensor cores through
// mma.sync.m16n8k16) decides per face whether the linear WCNS weights
// suffice.  On such faces the flux is the component-wise linear
// reconstruction of the conserved variables and fluxes (no characteristic
// projection, no nonlinear weights); everywhere else the plain scheme of
// numerics.cuh runs unchanged.  No reference counterpart: the reference
// always evaluates the nonlinear weights (src/nnd_center_RK.F90:310-353).
//
// The same file holds the training side: per-face (features, target)
// samples emitted by the plain solver, a fused forward+backward kernel that
// accumulates the gradients of a minibatch, and Adam.
#include <algorithm>

#include "gate_items.cuh"

namespace fdm {

static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

// The gate's per-direction arguments of the two kernels below, which take
// the warps' chunks of 32 x faces and then those of the y faces in one
// launch (half the launches of a stage, one partial wave instead of two).
struct GateDir {
    double4 *F;
    int32_t *hard;
    float *jump1;
};
// Stage 1, persistent: each warp takes 32 faces at a time.  Bound by issue
// slots and the XU pipe (64 tanh, 8 logarithms and 14 conversions from FP64
// per face): the weights stay in registers, the FP32 arithmetic runs on
// packed pairs and two values are rounded to BF16 at once.  1.03 M leaves
// 103 us in a step of 0.472 ms; 155 in 0.528 with one value per instruction,
// single roundings and the weights read from shared memory each time.
__global__ void __launch_bounds__(128, 4) k_gate_linear(Tables T, const double4 *__restrict__ cur,
                                                        const float *__restrict__ P, float logit_thr,
                                                        float jump_thr, const DevScalars *__restrict__ sc, double g,
                                                        double ig1, GateDir X, GateDir Y, uint32_t *count) {
    __shared__ GateWeights W;
    __shared__ XTile tiles[4];
    load_weights_smem(W, P);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t wx = (T.NI + T.nux + 31) / 32, wy = (T.NI + T.nuy + 31) / 32;
    XTile &Tt = tiles[wid];
    for (int k = GF; k < XLD; ++k) Tt.X[lane][k] = __float2bfloat16_rn(0.f);
    const GateFrag frag(W);
    const int64_t nwarps = (int64_t)gridDim.x * 4;
    for (int64_t w = blockIdx.x * 4 + wid; w < wx + wy; w += nwarps) {
        if (w < wx)
            gate_linear_chunk<0>(T, cur, X.F, frag, Tt, logit_thr, jump_thr, sc->lambda_x, ig1, g, X.hard, count, X.jump1,
                                 w);
        else
            gate_linear_chunk<1>(T, cur, Y.F, frag, Tt, logit_thr, jump_thr, sc->lambda_y, ig1, g, Y.hard, count + 1,
                                 Y.jump1, w - wx);
    }
}

// Stages 2 and 3: the guard on the faces that were linear at stage 1.
__global__ void __launch_bounds__(256) k_guard_linear(Tables T, const double4 *__restrict__ cur,
                                                      const DevScalars *__restrict__ sc, double g, double ig1,
                                                      GateDir X, GateDir Y, uint32_t *count) {
    const int64_t wx = (T.NI + T.nux + 31) / 32, wy = (T.NI + T.nuy + 31) / 32;
    const int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w < wx) guard_linear_chunk<0>(T, cur, X.F, X.jump1, sc->lambda_x, ig1, g, X.hard, count, w);
    else if (w < wx + wy)
        guard_linear_chunk<1>(T, cur, Y.F, Y.jump1, sc->lambda_y, ig1, g, Y.hard, count + 1, w - wx);
}

// full WCNS flux of the faces on the hard list
__global__ void __launch_bounds__(128, 4) k_faces_list(Tables T, const double4 *__restrict__ cur, double4 *Fx,
                                                       double4 *Fy, const int32_t *__restrict__ hx,
                                                       const int32_t *__restrict__ hy,
                                                       const uint32_t *__restrict__ count,
                                                       const DevScalars *__restrict__ sc, double g, FluxDen den) {
    // the x list, then the y list, whole warps to each
    const int64_t nx = count[0], ny = count[1], px = (nx + 31) / 32 * 32, stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < px + ny; i += stride) {
        if (i < px) {
            if (i < nx) face_item<0>(T, cur, Fx, sc->lambda_x, g, den, hx[i]);
        } else {
            face_item<1>(T, cur, Fy, sc->lambda_y, g, den, hy[i - px]);
        }
    }
}

// --------------------------------------------------- training samples
// (features, target) of every stride-th face of the current state; target
// = exp(-dev/tau) with dev the largest nonlinear-weight deviation.
template <int DIR>
__global__ void k_face_samples(Tables T, const double4 *__restrict__ cur, double gama, int64_t stride, int64_t phase,
                               double tau, float *feat, float *target, int64_t out0, int64_t cap) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nf = T.NI + (DIR == 0 ? T.nux : T.nuy);
    const int64_t f = j * stride + phase;
    if (f >= nf) return;
    const int64_t o = out0 + j;
    if (o >= cap) return;
    int32_t a, b, c, d;
    face_slots<DIR>(T, f, a, b, c, d);
    const Prim p0 = load_prim(cur, a), p1 = load_prim(cur, b), p2 = load_prim(cur, c), p3 = load_prim(cur, d);
    float fv[GF];
    face_features<DIR>(p0, p1, p2, p3, gama, fv);
    for (int k = 0; k < GF; ++k) feat[o * GF + k] = fv[k];
    target[o] = (float)exp(-face_weight_deviation<DIR>(p0, p1, p2, p3, gama) / tau);
}

// ----------------------------------------------------------- training
// Fused forward + backward of the weighted cross entropy
// -(y log g + neg_w (1-y) log(1-g)), g = sigmoid(z), for a minibatch; gradients
// of the mean loss accumulate into grad (FP32 atomics), the loss sum into
// loss.  Samples idx0 + k*step (mod n), k < B.
//
// A warp takes 32 samples at a time and keeps everything in registers: the
// accumulators of one product are the fragments of the next (as in
// mlp_logits_regs), and the products over the samples take theirs transposed
// (movmatrix).  The warps' gradients are summed in shared memory, so each
// block adds once to the result.  Bound by the latency of that chain (two
// groups of samples per warp at 65536) and by the call's three launches: one
// step 16 us at 65536 samples and 29 at 262144; 66 and 84 through tiles in
// shared memory, with an atomic per warp and gradient and two memsets before.
// Blocks of eight warps at 255 registers; of four or twelve 4 to 6 us more.
constexpr int TRAIN_TB = 256, TRAIN_ACC = 44;
// 8 x 8 transpose of a fragment block
__device__ __forceinline__ uint32_t transposed(uint32_t a) {
    uint32_t d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ F2 bf16_pair(uint32_t p) {
    return F2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}
// forward GELU of a layer's accumulators: fragments h of the next layer and
// the derivatives dg
__device__ __forceinline__ void gelu_layer(const float c[4][4], uint32_t h[2][4], F2 dg[4][2]) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i) h[nt >> 1][2 * (nt & 1) + i] = gelu_bf16(c[nt][2 * i], c[nt][2 * i + 1], &dg[nt][i]);
}
// adds the two row halves of a fragment's columns (nt, pair) to sum
__device__ __forceinline__ void add_columns(const uint32_t h[2][4], F2 s0, F2 s1, F2 sum[4]) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
        sum[nt] = sum[nt] + (bf16_pair(h[nt >> 1][2 * (nt & 1)]) * s0 + bf16_pair(h[nt >> 1][2 * (nt & 1) + 1]) * s1);
}
// column nt*8 + 2t + i summed over the warp's rows: lane (g, t) gets the one
// with nt = g/2, i = g%2
__device__ __forceinline__ float lane_column(const F2 sum[4]) {
    const int g = (threadIdx.x & 31) >> 2;
    float out = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float v[2];
        sum[c >> 1].get(v[0], v[1]);
        float x = v[c & 1];
        x += __shfl_xor_sync(0xffffffffu, x, 4);
        x += __shfl_xor_sync(0xffffffffu, x, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 16);
        if (g == c) out = x;
    }
    return out;
}
// where accumulator e = acc*32 + lane of a warp belongs: an index into grad,
// -1 the loss, -2 nothing
__device__ __forceinline__ int train_index(int e) {
    const int acc = e >> 5, lane = e & 31, g = lane >> 2, t = lane & 3;
    if (acc < 32) {
        const int mt = acc >> 4, nt = (acc >> 2) & 3, i = acc & 3;
        return P_W2 + (mt * 16 + g + 8 * (i >> 1)) * GH + nt * 8 + 2 * t + (i & 1);
    }
    if (acc < 40) {
        const int mt = (acc - 32) >> 2, i = acc & 3;
        return P_W1 + (mt * 16 + g + 8 * (i >> 1)) * GF + 2 * t + (i & 1);
    }
    const int col = (g >> 1) * 8 + 2 * t + (g & 1);
    if (acc == 40) return P_B1 + col;
    if (acc == 41) return P_B2 + col;
    if (acc == 42) return P_W3 + col;
    return lane == 0 ? P_B3 : lane == 1 ? -1 : -2;
}
__global__ void __launch_bounds__(TRAIN_TB) k_mlp_grad(const float *__restrict__ X, const float *__restrict__ Y,
                                                       int64_t n, int64_t idx0, int64_t step, int64_t B,
                                                       const float *__restrict__ P, float neg_w, float *grad,
                                                       float *loss) {
    constexpr int NW = TRAIN_TB / 32;
    __shared__ GateWeights W;
    __shared__ uint4 xs[NW][32];
    __shared__ float red[NW / 2][TRAIN_ACC * 32];
    load_weights_smem(W, P);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const GateFrag fr(W);
    uint32_t w2t[4][2][2];   // B[k = out][n = in] = W2[out][in]
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int kc = 0; kc < 2; ++kc)
#pragma unroll
            for (int i = 0; i < 2; ++i) w2t[nt][kc][i] = transposed(fr.w2[2 * kc + i][nt >> 1][nt & 1]);
    F2 w3c[4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) w3c[nt] = bf16_pair(*reinterpret_cast<const uint32_t *>(W.w3 + nt * 8 + 2 * t));
    float acc[TRAIN_ACC];    // dW2 [mt over out][nt over in][i], dW1 [mt over out][i]
#pragma unroll
    for (int a = 0; a < TRAIN_ACC; ++a) acc[a] = 0.f;
    F2 gb1[4], gb2[4], gw3[4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) gb1[nt] = gb2[nt] = gw3[nt] = F2(0.f);
    float gb3 = 0.f, ls = 0.f;
    const float invB = 1.0f / (float)B;
    const bool wide = ((uintptr_t)X & 15u) == 0;   // rows of 32 bytes: as two vectors where the base allows
    const int64_t ngroups = (B + 31) / 32;
    for (int64_t grp = blockIdx.x * (int64_t)NW + wid; grp < ngroups; grp += (int64_t)gridDim.x * NW) {
        const int64_t k = grp * 32 + lane;
        const bool valid = k < B;
        const int64_t s = (idx0 + k * step) % n;
        float y = 0.f, x[GF];
#pragma unroll
        for (int q = 0; q < GF; ++q) x[q] = 0.f;
        if (valid) {
            y = Y[s];
            if (wide) {
                const float4 u = *reinterpret_cast<const float4 *>(X + s * GF);
                const float4 v = *reinterpret_cast<const float4 *>(X + s * GF + 4);
                x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
                x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
            } else {
#pragma unroll
                for (int q = 0; q < GF; ++q) x[q] = X[s * GF + q];
            }
        }
        __syncwarp();
        xs[wid][lane] = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]),
                                   pack_bf16(x[6], x[7]));
        __syncwarp();
        const uint32_t *xw = reinterpret_cast<const uint32_t *>(xs[wid]);
        uint32_t xa[4];      // rows g, g+8, g+16, g+24, features 2t and 2t+1
#pragma unroll
        for (int q = 0; q < 4; ++q) xa[q] = xw[(g + 8 * q) * 4 + t];
        uint32_t h1[2][2][4], h2[2][2][4];
        F2 d1[2][4][2], d2[2][4][2];
        float z[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const uint32_t a[4] = {xa[2 * mt], xa[2 * mt + 1], 0u, 0u};
            float c4[4][4];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float c[4] = {fr.b1[nt][0], fr.b1[nt][1], fr.b1[nt][0], fr.b1[nt][1]};
                mma16816(c4[nt], a, fr.w1[nt], c);
            }
            gelu_layer(c4, h1[mt], d1[mt]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float c[4] = {fr.b2[nt][0], fr.b2[nt][1], fr.b2[nt][0], fr.b2[nt][1]};
                float d[4];
                mma16816(d, h1[mt][0], fr.w2[nt][0], c);
                mma16816(c4[nt], h1[mt][1], fr.w2[nt][1], d);
            }
            gelu_layer(c4, h2[mt], d2[mt]);
            const float c[4] = {fr.b3, 0.f, fr.b3, 0.f};
            float d[4], e[4];
            mma16816(d, h2[mt][0], fr.w3[0], c);
            mma16816(e, h2[mt][1], fr.w3[1], d);
            z[mt][0] = e[0];
            z[mt][1] = e[2];
        }
        const float zl = row_logit(z, lane);
        const float gs = 1.0f / (1.0f + expf(-zl));
        if (valid) {
            const float e = 1e-7f;
            ls += -(y * logf(gs + e) + neg_w * (1.0f - y) * logf(1.0f - gs + e));
        }
        // d/dz of -(y log g + a (1-y) log(1-g)) = g (y + a (1-y)) - y
        const float dz = valid ? (gs * (y + neg_w * (1.0f - y)) - y) * invB : 0.f;
        gb3 += dz;
        uint32_t a2[2][2][4], a1[2][2][4];   // dA2, dA1 as fragments
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const F2 z0(__shfl_sync(0xffffffffu, dz, mt * 16 + g)), z1(__shfl_sync(0xffffffffu, dz, mt * 16 + g + 8));
            // dw3[j] = sum_s h2[s][j] dz[s]
            add_columns(h2[mt], z0, z1, gw3);
            // dh2 = dz w3, da2 = dh2 gelu'(a2); db2[j] = sum_s da2[s][j]
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float lo, hi;
                    ((i ? z1 : z0) * w3c[nt] * d2[mt][nt][i]).get(lo, hi);
                    a2[mt][nt >> 1][2 * (nt & 1) + i] = pack_bf16(lo, hi);
                }
            add_columns(a2[mt], F2(1.f), F2(1.f), gb2);
            // dh1 = dA2 W2; da1 = dh1 gelu'(a1)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float c[4] = {0.f, 0.f, 0.f, 0.f};
                float d[4], e[4];
                mma16816(d, a2[mt][0], w2t[nt][0], c);
                mma16816(e, a2[mt][1], w2t[nt][1], d);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float lo, hi;
                    (F2(e[2 * i], e[2 * i + 1]) * d1[mt][nt][i]).get(lo, hi);
                    a1[mt][nt >> 1][2 * (nt & 1) + i] = pack_bf16(lo, hi);
                }
            }
            add_columns(a1[mt], F2(1.f), F2(1.f), gb1);
        }
        // dW2[o][i] += sum_s dA2[s][o] H1[s][i], dW1[o][f] += sum_s dA1[s][o] X[s][f]:
        // A[m = o][k = s] and B[k = s][n = i] are the transposed blocks
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {     // samples 16 ks .. 16 ks + 15
            uint32_t bh[4][2];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                bh[nt][0] = transposed(h1[ks][nt >> 1][2 * (nt & 1)]);
                bh[nt][1] = transposed(h1[ks][nt >> 1][2 * (nt & 1) + 1]);
            }
            const uint32_t bx[2] = {transposed(xa[2 * ks]), transposed(xa[2 * ks + 1])};
#pragma unroll
            for (int mo = 0; mo < 2; ++mo) { // outputs 16 mo .. 16 mo + 15: rows o, o+8 by samples s, s+8
                const uint32_t at2[4] = {transposed(a2[ks][mo][0]), transposed(a2[ks][mo][2]),
                                         transposed(a2[ks][mo][1]), transposed(a2[ks][mo][3])};
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    float *c = acc + mo * 16 + nt * 4, d[4];
                    mma16816(d, at2, bh[nt], c);
                    c[0] = d[0]; c[1] = d[1]; c[2] = d[2]; c[3] = d[3];
                }
                const uint32_t at1[4] = {transposed(a1[ks][mo][0]), transposed(a1[ks][mo][2]),
                                         transposed(a1[ks][mo][1]), transposed(a1[ks][mo][3])};
                float *c = acc + 32 + mo * 4, d[4];
                mma16816(d, at1, bx, c);
                c[0] = d[0]; c[1] = d[1]; c[2] = d[2]; c[3] = d[3];
            }
        }
    }
    acc[40] = lane_column(gb1);
    acc[41] = lane_column(gb2);
    acc[42] = lane_column(gw3);
    for (int o = 16; o; o >>= 1) {
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
        ls += __shfl_xor_sync(0xffffffffu, ls, o);
    }
    acc[43] = lane == 0 ? gb3 : ls;
    dep_begin();   // the results are cleared; what is read above was final before the kernel that clears them
    // the upper half of the warps to the lower half, those to all threads
    if (wid >= NW / 2)
#pragma unroll
        for (int a = 0; a < TRAIN_ACC; ++a) red[wid - NW / 2][a * 32 + lane] = acc[a];
    __syncthreads();
    if (wid < NW / 2)
#pragma unroll
        for (int a = 0; a < TRAIN_ACC; ++a) red[wid][a * 32 + lane] += acc[a];
    __syncthreads();
    for (int e = threadIdx.x; e < TRAIN_ACC * 32; e += TRAIN_TB) {
        float v = red[0][e];
#pragma unroll
        for (int w = 1; w < NW / 2; ++w) v += red[w][e];
        const int at = train_index(e);
        if (at >= 0) atomicAdd(grad + at, v);
        else if (at == -1) atomicAdd(loss, v);
    }
}

__global__ void k_train_clear(float *grad, float *loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P_N) grad[i] = 0.f;
    else if (i == P_N) *loss = 0.f;
}

// Adam (FP32 master weights)
__global__ void k_adam(float *P, const float *grad, float *m, float *v, int64_t n, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    dep_begin();
    if (i >= n) return;
    const float gi = grad[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// gate probabilities of given feature rows (evaluation / tests)
__global__ void __launch_bounds__(128) k_mlp_eval(const float *__restrict__ X, int64_t n, const float *__restrict__ P,
                                                  float *prob) {
    __shared__ GateWeights W;
    __shared__ XTile tiles[4];
    load_weights_smem(W, P);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t r = (blockIdx.x * 4 + wid) * 32 + lane;
    XTile &Tt = tiles[wid];
    for (int q = 0; q < XLD; ++q) Tt.X[lane][q] = __float2bfloat16_rn(r < n && q < GF ? X[r * GF + q] : 0.f);
    __syncwarp();
    float z[2][2];
    mlp_logits_regs(GateFrag(W), Tt.X, z);
    const float zl = row_logit(z, lane);
    if (r < n) prob[r] = 1.0f / (1.0f + expf(-zl));
}

// ------------------------------------------------------ gated face flux
static int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

void launch_gated_faces(fdm_handle *h, const double4 *cur, int krk) {
    const Tables T = h->tables();
    const DevScalars *sc = h->scal.as<DevScalars>();
    const int64_t nfx = h->NI + h->nux, nfy = h->NI + h->nuy;
    const GateLists GL = gate_lists(h->gate_flag.p, nfx, nfy);
    uint32_t *cnt = GL.cnt;
    int32_t *hx = GL.hx, *hy = GL.hy;
    float *jx = GL.jx, *jy = GL.jy;
    const float *P = h->gate_params.as<float>();
    const int sms = sm_count();
    const int lx = (int)std::min<int64_t>(nblk(nfx, 256), 2 * sms), ly = (int)std::min<int64_t>(nblk(nfy, 256), 2 * sms);
    const GateDir X{h->Fx.as<double4>(), hx, jx}, Y{h->Fy.as<double4>(), hy, jy};
    const int64_t warps = (nfx + 31) / 32 + (nfy + 31) / 32;
    if (krk == 1 || !h->gate_stage1_valid) {
        cudaMemsetAsync(cnt, 0, 2 * sizeof(uint32_t), h->s);
        k_gate_linear<<<(int)std::min<int64_t>(nblk(warps, 4), 4 * sms), 128, 0, h->s>>>(
            T, cur, P, h->gate_logit_thr, h->gate_jump_thr, sc, h->G.gama, 1.0 / (h->G.gama - 1.0), X, Y, cnt);
        cudaMemcpyAsync(cnt + 2, cnt, 2 * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->s);
        h->gate_stage1_valid = true;
    } else {
        cudaMemcpyAsync(cnt, cnt + 2, 2 * sizeof(uint32_t), cudaMemcpyDeviceToDevice, h->s);
        k_guard_linear<<<nblk(warps, 8), 256, 0, h->s>>>(T, cur, sc, h->G.gama, 1.0 / (h->G.gama - 1.0), X, Y, cnt);
    }
    if (h->p.flux_variant == 1) {
        launch_faces_list_fast(h, cur, hx, hy, cnt, lx, ly);
        return;
    }
    k_faces_list<<<(int)std::min<int64_t>(nblk(nfx + nfy, 128), 4 * sms), 128, 0, h->s>>>(
        T, cur, h->Fx.as<double4>(), h->Fy.as<double4>(), hx, hy, cnt, sc, h->G.gama, flux_den(h->G.gama));
}

size_t gate_list_bytes(const fdm_handle *h) {
    return (size_t)(GATE_LIST_HEAD + 2 * (2 * h->NI + h->nux + h->nuy)) * sizeof(int32_t);
}

}  // namespace fdm

using namespace fdm;

extern "C" int fdm_gate_param_count(void) { return P_N; }

// faces that took the linear path in the last gated stage, and all faces
extern "C" int fdm_gate_stats(fdm_handle *h, int64_t *gated, int64_t *total) {
    if (!h) return FDM_ERR_ARG;
    if (!h->loaded) return FDM_ERR_STATE;
    const int64_t n = 2 * h->NI + h->nux + h->nuy;
    if (total) *total = n;
    if (!gated) return FDM_OK;
    if (!h->gate_on) { *gated = 0; return FDM_OK; }
    uint32_t c[2] = {0, 0};
    cudaMemcpyAsync(c, h->gate_flag.p, sizeof c, cudaMemcpyDeviceToHost, h->s);
    const cudaError_t e = cudaStreamSynchronize(h->s);
    if (e != cudaSuccess) return cuda_fail(h, e, "fdm_gate_stats");
    *gated = n - (int64_t)c[0] - (int64_t)c[1];
    return FDM_OK;
}

extern "C" int fdm_gate_set(fdm_handle *h, const float *params, float threshold, int32_t enable) {
    if (!h) return FDM_ERR_ARG;
    if (enable) {
        if (!params || !(threshold > 0.f && threshold < 1.f)) return FDM_ERR_ARG;
        FDM_CK(h, h->gate_params.ensure(P_N * sizeof(float)));
        FDM_CK(h, cudaMemcpy(h->gate_params.p, params, P_N * sizeof(float), cudaMemcpyHostToDevice));
        h->gate_logit_thr = logf(threshold / (1.f - threshold));
        h->gate_jump_thr = -1.f;
    }
    h->gate_on = enable != 0;
    h->gate_stage1_valid = false;
    h->graph_version = -1;
    return FDM_OK;
}

// The plain jump rule in place of the network: a face is linear at stage 1
// when its largest normalised jump (the unsquashed gate features) is at most
// jump_threshold; a negative value restores the network.  The gate must have
// been enabled by fdm_gate_set.
extern "C" int fdm_gate_set_jump_rule(fdm_handle *h, float jump_threshold) {
    if (!h) return FDM_ERR_ARG;
    if (!h->gate_on || !h->gate_params.p) { h->err = "the gate is off: fdm_gate_set first"; return FDM_ERR_STATE; }
    h->gate_jump_thr = jump_threshold >= 0.f ? jump_threshold : -1.f;
    h->gate_stage1_valid = false;
    h->graph_version = -1;
    return FDM_OK;
}

extern "C" int fdm_gate_samples(fdm_handle *h, int64_t stride, int64_t phase, double tau, float *feat_dev,
                                float *target_dev, int64_t offset, int64_t cap, int64_t *n_written) {
    if (!h || stride <= 0 || phase < 0 || phase >= stride || !(tau > 0) || !feat_dev || !target_dev) return FDM_ERR_ARG;
    if (!h->loaded) return FDM_ERR_STATE;
    const Tables T = h->tables();
    const int64_t nfx = h->NI + h->nux, nfy = h->NI + h->nuy;
    const int64_t jx = (nfx - phase + stride - 1) / stride, jy = (nfy - phase + stride - 1) / stride;
    const double4 *cur = h->B[0].as<double4>();
    launch_requests(h, cur);
    if (jx > 0)
        k_face_samples<0><<<nblk(jx, 128), 128, 0, h->s>>>(T, cur, h->G.gama, stride, phase, tau, feat_dev,
                                                            target_dev, offset, cap);
    if (jy > 0)
        k_face_samples<1><<<nblk(jy, 128), 128, 0, h->s>>>(T, cur, h->G.gama, stride, phase, tau, feat_dev,
                                                            target_dev, offset + jx, cap);
    FDM_CK(h, cudaStreamSynchronize(h->s));
    int64_t w = jx + jy;
    if (offset + w > cap) w = cap > offset ? cap - offset : 0;
    if (n_written) *n_written = w;
    return FDM_OK;
}

// One Adam step on a minibatch of B samples (idx0 + k*step mod n).
extern "C" int fdm_gate_train_step(const float *X, const float *Y, int64_t n, int64_t idx0, int64_t step, int64_t B,
                                   float neg_weight, float *params, float *grad, float *adam_m, float *adam_v,
                                   int64_t t, float lr, float *loss, void *stream) {
    if (!X || !Y || n <= 0 || B <= 0 || !params || !grad || !adam_m || !adam_v || !loss || t <= 0 ||
        !(neg_weight > 0.f))
        return FDM_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // waits for all of the caller's work before it, so the weights and samples
    // are final for the next kernel however early that one starts
    k_train_clear<<<(P_N + 256) / 256, 256, 0, s>>>(grad, loss);
    const int64_t ngroups = (B + 31) / 32;
    const int64_t blocks = std::min<int64_t>((ngroups + TRAIN_TB / 32 - 1) / (TRAIN_TB / 32), sm_count());
    launch_after(s, (unsigned)blocks, TRAIN_TB, k_mlp_grad, X, Y, n, idx0, step, B, params, neg_weight, grad, loss);
    if (lr > 0.f) {
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
        launch_after(s, (P_N + 255) / 256, 256, k_adam, params, grad, adam_m, adam_v, P_N, lr, b1, b2, 1e-8f, c1, c2);
    }
    return cudaGetLastError() == cudaSuccess ? FDM_OK : FDM_ERR_CUDA;
}

extern "C" int fdm_gate_eval(const float *X, int64_t n, const float *params, float *prob, void *stream) {
    if (!X || n <= 0 || !params || !prob) return FDM_ERR_ARG;
    k_mlp_eval<<<(int)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(X, n, params, prob);
    return cudaGetLastError() == cudaSuccess ? FDM_OK : FDM_ERR_CUDA;
}
