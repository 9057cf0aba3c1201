// Depthwise causal convolution over channel-last activations (Mamba-2 / gated delta net short convolutions):
//   z[b, t, c] = bias[c] + sum_j w[c, j] * x[b, t - (K-1) + j, c],   y = silu(z) or z,   K <= 8
// with x[b, t < 0, c] taken from init[b, c, K-1+t] (or 0).  One thread owns 8 channels (one 16-byte vector) and a
// run of CHUNK time steps and slides a register window over it, so every x element is read once (+ K-1 halo rows per
// chunk) and consecutive threads touch consecutive channels (fully coalesced rows).
// Backward recomputes z (nothing but x is saved), forms dz = dy * act'(z), and produces dx (needs dz of the next K-1
// steps: a forward halo), the gradient of the initial state, and per-thread partial sums of dw / dbias that are
// added atomically into fp32 accumulators.
// Role of causal_conv1d_fn / causal_conv1d_update in the reference
// (lm_engine/modeling_utils/depthwise_causal_convolution.py:110-206).
namespace lme {

static constexpr int CONV_MAX_K = 8;
static constexpr int CONV_CHUNK = 32;

__device__ __forceinline__ void conv_load_row(const __nv_bfloat16* x, const __nv_bfloat16* init, long long b, int t,
                                              int S, int C, int K, int c, float (&out)[8]) {
    if (t >= 0) {
        if (t < S) load8(x + (b * S + t) * C + c, out);
        else {
#pragma unroll
            for (int i = 0; i < 8; ++i) out[i] = 0.f;
        }
    } else if (init != nullptr) {
        // init [B, C, K-1]: element (c + i, K-1+t)
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __bfloat162float(init[(b * C + c + i) * (K - 1) + (K - 1 + t)]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = 0.f;
    }
}

// up to KM taps (four-tap filters have their own kernels below)
template <int KM>
__global__ void __launch_bounds__(128)
causal_conv1d_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                         const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ init,
                         __nv_bfloat16* __restrict__ y, int B, int S, int C, int K, int silu) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= C) return;
    const int t0 = blockIdx.y * CONV_CHUNK;
    const long long b = blockIdx.z;
    float wv[KM][8], bv[8], win[KM][8];
#pragma unroll
    for (int j = 0; j < KM; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[j][i] = j < K ? __bfloat162float(w[(c + i) * K + j]) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) bv[i] = bias != nullptr ? __bfloat162float(bias[c + i]) : 0.f;
    // window slots 0 .. K-2 hold x[t - (K-1)] .. x[t - 1]
#pragma unroll
    for (int j = 0; j < KM - 1; ++j)
        if (j < K - 1) conv_load_row(x, init, b, t0 - (K - 1) + j, S, C, K, c, win[j]);
    const int t1 = min(t0 + CONV_CHUNK, S);
    for (int t = t0; t < t1; ++t) {
        float cur[8], z[8];
        load8(x + (b * S + t) * C + c, cur);
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = bv[i];
#pragma unroll
        for (int j = 0; j < KM - 1; ++j)
            if (j < K - 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) z[i] += wv[j][i] * win[j][i];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float wk = 0.f;
#pragma unroll
            for (int j = 0; j < KM; ++j) wk = (j == K - 1) ? wv[j][i] : wk;
            z[i] += wk * cur[i];
            if (silu) z[i] = silu_f(z[i]);
        }
        store8(y + (b * S + t) * C + c, z);
#pragma unroll
        for (int j = 0; j < KM - 2; ++j)
            if (j < K - 2) {
#pragma unroll
                for (int i = 0; i < 8; ++i) win[j][i] = win[j + 1][i];
            }
#pragma unroll
        for (int j = 0; j < KM - 1; ++j)
            if (j == K - 2) {
#pragma unroll
                for (int i = 0; i < 8; ++i) win[j][i] = cur[i];
            }
    }
}

// dz at time t for the thread's 8 channels (0 outside [0, S))
template <int KM>
__device__ __forceinline__ void conv_dz(const __nv_bfloat16* x, const __nv_bfloat16* init, const __nv_bfloat16* dy,
                                        const float (&wv)[KM][8], const float (&bv)[8], long long b, int t,
                                        int S, int C, int K, int c, int silu, float (&dz)[8]) {
    if (t < 0 || t >= S) {
#pragma unroll
        for (int i = 0; i < 8; ++i) dz[i] = 0.f;
        return;
    }
    float z[8], g[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = bv[i];
    for (int j = 0; j < K; ++j) {
        float xr[8];
        conv_load_row(x, init, b, t - (K - 1) + j, S, C, K, c, xr);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float wj = 0.f;
#pragma unroll
            for (int jj = 0; jj < KM; ++jj) wj = (jj == j) ? wv[jj][i] : wj;
            z[i] += wj * xr[i];
        }
    }
    load8(dy + (b * S + t) * C + c, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (silu) {
            const float sg = 1.f / (1.f + __expf(-z[i]));
            dz[i] = g[i] * sg * (1.f + z[i] * (1.f - sg));
        } else {
            dz[i] = g[i];
        }
    }
}

template <int KM>
__global__ void __launch_bounds__(128)
causal_conv1d_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                         const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ init,
                         const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx,
                         float* __restrict__ dw, float* __restrict__ dbias, float* __restrict__ dinit, int B, int S,
                         int C, int K, int silu) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c >= C) return;
    const int t0 = blockIdx.y * CONV_CHUNK;
    const long long b = blockIdx.z;
    float wv[KM][8], bv[8];
#pragma unroll
    for (int j = 0; j < KM; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[j][i] = j < K ? __bfloat162float(w[(c + i) * K + j]) : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) bv[i] = bias != nullptr ? __bfloat162float(bias[c + i]) : 0.f;
    float dwacc[KM][8], dbacc[8];
#pragma unroll
    for (int j = 0; j < KM; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) dwacc[j][i] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) dbacc[i] = 0.f;
    // dzw slot j holds dz[t + j]; dx[t] = sum_j w[K-1-j] * dz[t + j]
    float dzw[KM][8];
#pragma unroll
    for (int j = 0; j < KM; ++j)
        if (j < K) conv_dz<KM>(x, init, dy, wv, bv, b, t0 + j, S, C, K, c, silu, dzw[j]);
    const int t1 = min(t0 + CONV_CHUNK, S);
    for (int t = t0; t < t1; ++t) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = 0.f;
#pragma unroll
        for (int j = 0; j < KM; ++j)
            if (j < K) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float wr = 0.f;
#pragma unroll
                    for (int jj = 0; jj < KM; ++jj) wr = (jj == K - 1 - j) ? wv[jj][i] : wr;
                    o[i] += wr * dzw[j][i];
                }
            }
        store8(dx + (b * S + t) * C + c, o);
        // weight / bias gradients of output step t (dz[t] = slot 0) against its K inputs
        for (int j = 0; j < K; ++j) {
            float xr[8];
            conv_load_row(x, init, b, t - (K - 1) + j, S, C, K, c, xr);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
                for (int jj = 0; jj < KM; ++jj)
                    if (jj == j) dwacc[jj][i] += dzw[0][i] * xr[i];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) dbacc[i] += dzw[0][i];
        // slide: slot j <- slot j + 1, new last slot = dz[t + K]
#pragma unroll
        for (int j = 0; j < KM - 1; ++j)
            if (j < K - 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) dzw[j][i] = dzw[j + 1][i];
            }
        float nxt[8];
        conv_dz<KM>(x, init, dy, wv, bv, b, t + K, S, C, K, c, silu, nxt);
#pragma unroll
        for (int j = 0; j < KM; ++j)
            if (j == K - 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) dzw[j][i] = nxt[i];
            }
    }
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v = 0.f;
#pragma unroll
            for (int jj = 0; jj < KM; ++jj) v = (jj == j) ? dwacc[jj][i] : v;
            atomicAdd(&dw[(c + i) * K + j], v);
        }
    if (dbias != nullptr)
#pragma unroll
        for (int i = 0; i < 8; ++i) atomicAdd(&dbias[c + i], dbacc[i]);
    // gradient of the initial state: x at time s = i - (K-1) (i = 0 .. K-2) feeds output t = s + (K-1) - j, t >= 0
    if (dinit != nullptr && blockIdx.y == 0) {
        for (int i = 0; i < K - 1; ++i) {
            float acc[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] = 0.f;
            for (int j = 0; j <= i; ++j) {
                float dz[8];
                conv_dz<KM>(x, init, dy, wv, bv, b, i - j, S, C, K, c, silu, dz);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    float wj = 0.f;
#pragma unroll
                    for (int jj = 0; jj < KM; ++jj) wj = (jj == j) ? wv[jj][q] : wj;
                    acc[q] += wj * dz[q];
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) dinit[(b * C + c + q) * (K - 1) + i] = acc[q];
        }
    }
}

// ---- four taps (every configuration of the repository): sliding windows in registers
// The work per element is a few multiplies, but IEEE divisions in the activation and re-read rows made it more than its
// HBM traffic (x in, y out; x and dy in, dx out).  A thread owns a run of CONV4_STEPS time steps of four channels and
// requests rows ahead of the arithmetic.  The backward pass reads every x and dy row once: step t's pre-activation,
// its weight gradient and the window of dz that dx[t - 3] needs all come from the same four rows of x in registers.  A
// block sums the weight gradients of its eight time runs before it adds them to memory.  x may be a slice of a wider
// row (element strides x_b, x_t), so that a projection's output is read in place.
// Measured (4096 steps x 4352 channels, silu): forward 41 -> 22 us and no copy of x before it (71 MB: issue slots 70 %
// busy), backward 150 -> 85 us (107 MB: 16 warps per SM wait for rows).
static constexpr int CONV4_STEPS = 16;
static constexpr int CONV4_AHEAD = 4;   // forward

struct Conv4 {
    const __nv_bfloat16 *x, *w, *bias, *init;
    long long x_b, x_t;
    int S, C, silu;
};

__device__ __forceinline__ void conv_unpack(const uint2& r, float (&f)[4]) {
    const float2 lo = unpack_bf16x2(r.x), hi = unpack_bf16x2(r.y);
    f[0] = lo.x; f[1] = lo.y; f[2] = hi.x; f[3] = hi.y;
}
__device__ __forceinline__ uint2 conv_pack(const float (&f)[4]) {
    return make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
}
// four channels of row t of x, of the initial state for t < 0, zeros outside
__device__ __forceinline__ uint2 conv4_row(const Conv4& p, long long b, int t, int c) {
    uint2 r = make_uint2(0, 0);
    if (t >= 0) {
        if (t < p.S) r = *reinterpret_cast<const uint2*>(p.x + b * p.x_b + t * p.x_t + c);
    } else if (p.init != nullptr) {
        float f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = __bfloat162float(p.init[(b * p.C + c + i) * 3 + 3 + t]);
        r = conv_pack(f);
    }
    return r;
}
__device__ __forceinline__ void conv4_filter(const Conv4& p, int c, float (&w)[4][4], float (&bv)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint2 r = *reinterpret_cast<const uint2*>(p.w + (c + i) * 4);
        const float2 lo = unpack_bf16x2(r.x), hi = unpack_bf16x2(r.y);
        w[0][i] = lo.x; w[1][i] = lo.y; w[2][i] = hi.x; w[3][i] = hi.y;
        bv[i] = p.bias != nullptr ? __bfloat162float(p.bias[c + i]) : 0.f;
    }
}

// Channel groups in grid.x and time runs in grid.y: blocks that run together read whole rows (22.3 us at 4096 steps x 4352
// channels, 23.3 with the two exchanged).  More runs than grid.y holds, a million steps, exchange them all the same.
__global__ void __launch_bounds__(128, 8)
causal_conv4_fwd_kernel(const Conv4 p, __nv_bfloat16* __restrict__ y, const bool exchanged) {
    constexpr int V = 4;
    const int run = exchanged ? blockIdx.x : blockIdx.y;
    const int c = ((exchanged ? blockIdx.y : blockIdx.x) * 128 + threadIdx.x) * V;
    if (c >= p.C) return;
    const long long b = blockIdx.z;
    const int t0 = run * CONV4_STEPS, t1 = min(t0 + CONV4_STEPS, p.S);
    float w[4][V], bv[V], x0[V], x1[V], x2[V];
    conv4_filter(p, c, w, bv);
    conv_unpack(conv4_row(p, b, t0 - 3, c), x0);
    conv_unpack(conv4_row(p, b, t0 - 2, c), x1);
    conv_unpack(conv4_row(p, b, t0 - 1, c), x2);
    uint2 ahead[CONV4_AHEAD];
#pragma unroll
    for (int u = 0; u < CONV4_AHEAD; ++u) ahead[u] = conv4_row(p, b, t0 + u, c);
    for (int t = t0; t < t1; t += CONV4_AHEAD) {
        uint2 now[CONV4_AHEAD];
#pragma unroll
        for (int u = 0; u < CONV4_AHEAD; ++u) {
            now[u] = ahead[u];
            if (t + CONV4_AHEAD < t1) ahead[u] = conv4_row(p, b, t + CONV4_AHEAD + u, c);
        }
#pragma unroll
        for (int u = 0; u < CONV4_AHEAD; ++u) {
            if (t + u >= t1) break;
            float x3[V], z[V];
            conv_unpack(now[u], x3);
#pragma unroll
            for (int i = 0; i < V; ++i) {
                z[i] = bv[i] + w[0][i] * x0[i] + w[1][i] * x1[i] + w[2][i] * x2[i] + w[3][i] * x3[i];
                if (p.silu) z[i] *= sigmoid_fast(z[i]);
                x0[i] = x1[i];
                x1[i] = x2[i];
                x2[i] = x3[i];
            }
            *reinterpret_cast<uint2*>(y + (b * p.S + t + u) * p.C + c) = conv_pack(z);
        }
    }
}

// block (32, 8): 32 groups of 4 channels x 8 consecutive time runs
__global__ void __launch_bounds__(256, 2)
causal_conv4_bwd_kernel(const Conv4 p, const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx,
                        float* __restrict__ dw, float* __restrict__ dbias, float* __restrict__ dinit) {
    constexpr int V = 4, AHEAD = 2;     // 128 registers, two blocks per SM; four rows ahead spill (118 us instead of 85)
    __shared__ float part[8][5 * V][33];
    const int c = (blockIdx.x * 32 + threadIdx.x) * V;
    const long long b = blockIdx.z;
    const int t0 = (blockIdx.y * 8 + threadIdx.y) * CONV4_STEPS, t1 = min(t0 + CONV4_STEPS, p.S);
    float dwa[4][V] = {}, dba[V] = {};
    if (c < p.C && t0 < p.S) {
        float w[4][V], bv[V], x0[V], x1[V], x2[V];
        float d0[V] = {}, d1[V] = {}, d2[V] = {};      // dz of the three steps before the current one
        conv4_filter(p, c, w, bv);
        conv_unpack(conv4_row(p, b, t0 - 3, c), x0);
        conv_unpack(conv4_row(p, b, t0 - 2, c), x1);
        conv_unpack(conv4_row(p, b, t0 - 1, c), x2);
        const __nv_bfloat16* dyp = dy + b * p.S * p.C + c;
        uint2 ax[AHEAD], ad[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            ax[u] = conv4_row(p, b, t0 + u, c);
            ad[u] = make_uint2(0, 0);
            if (t0 + u < p.S) ad[u] = *reinterpret_cast<const uint2*>(dyp + static_cast<long long>(t0 + u) * p.C);
        }
        for (int t = t0; t < t1 + 3; t += AHEAD) {
            uint2 nx[AHEAD], nd[AHEAD];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                nx[u] = ax[u];
                nd[u] = ad[u];
                const int ta = t + AHEAD + u;
                if (ta < t1 + 3) {
                    ax[u] = conv4_row(p, b, ta, c);
                    ad[u] = make_uint2(0, 0);
                    if (ta < p.S) ad[u] = *reinterpret_cast<const uint2*>(dyp + static_cast<long long>(ta) * p.C);
                }
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
                const int tt = t + u;
                if (tt >= t1 + 3) break;
                float x3[V], gd[V], o[V];
                conv_unpack(nx[u], x3);
                conv_unpack(nd[u], gd);
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    float dz = gd[i];       // zero beyond the sequence
                    if (p.silu) {
                        const float z = bv[i] + w[0][i] * x0[i] + w[1][i] * x1[i] + w[2][i] * x2[i] + w[3][i] * x3[i];
                        const float sg = sigmoid_fast(z);
                        dz *= sg * (1.f + z * (1.f - sg));
                        if (tt >= p.S) dz = 0.f;
                    }
                    if (tt < t1) {
                        dwa[0][i] += dz * x0[i];
                        dwa[1][i] += dz * x1[i];
                        dwa[2][i] += dz * x2[i];
                        dwa[3][i] += dz * x3[i];
                        dba[i] += dz;
                    }
                    o[i] = w[3][i] * d0[i] + w[2][i] * d1[i] + w[1][i] * d2[i] + w[0][i] * dz;
                    d0[i] = d1[i];
                    d1[i] = d2[i];
                    d2[i] = dz;
                    x0[i] = x1[i];
                    x1[i] = x2[i];
                    x2[i] = x3[i];
                }
                if (tt - 3 >= t0)
                    *reinterpret_cast<uint2*>(dx + (b * p.S + tt - 3) * p.C + c) = conv_pack(o);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) part[threadIdx.y][i * 5 + j][threadIdx.x] = dwa[j][i];
        part[threadIdx.y][i * 5 + 4][threadIdx.x] = dba[i];
    }
    __syncthreads();
    if (c < p.C)
        for (int v = threadIdx.y; v < 5 * V; v += 8) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) s += part[k][v][threadIdx.x];
            const int i = v / 5, j = v % 5;
            if (j < 4) atomicAdd(&dw[(c + i) * 4 + j], s);
            else if (dbias != nullptr) atomicAdd(&dbias[c + i], s);
        }
    // gradient of the initial state: x at time i - 3 (i = 0 .. 2) feeds outputs 0 .. i
    if (dinit != nullptr && t0 == 0 && c < p.C) {
        float w[4][V], bv[V], dz[3][V], row[6][V];
        conv4_filter(p, c, w, bv);
#pragma unroll
        for (int r = 0; r < 6; ++r) conv_unpack(conv4_row(p, b, r - 3, c), row[r]);
#pragma unroll
        for (int t = 0; t < 3; ++t)
#pragma unroll
            for (int i = 0; i < V; ++i) {
                dz[t][i] = 0.f;
                if (t >= p.S) continue;
                dz[t][i] = __bfloat162float(dy[(b * p.S + t) * p.C + c + i]);
                if (p.silu) {
                    const float z = bv[i] + w[0][i] * row[t][i] + w[1][i] * row[t + 1][i] + w[2][i] * row[t + 2][i] +
                                    w[3][i] * row[t + 3][i];
                    const float sg = sigmoid_fast(z);
                    dz[t][i] *= sg * (1.f + z * (1.f - sg));
                }
            }
#pragma unroll
        for (int i = 0; i < V; ++i) {
            float* o = dinit + (b * p.C + c + i) * 3;
            o[0] = w[0][i] * dz[0][i];
            o[1] = w[1][i] * dz[0][i] + w[0][i] * dz[1][i];
            o[2] = w[2][i] * dz[0][i] + w[1][i] * dz[1][i] + w[0][i] * dz[2][i];
        }
    }
}

}  // namespace lme

using namespace lme;

// x: element strides x_b (batch) and x_t (time), multiples of 8; y, dy, dx: contiguous [B, S, C]
extern "C" int lme_causal_conv1d_fwd(const void* x, long long x_b, long long x_t, const void* w, const void* bias,
                                     const void* init, void* y, int B, int S, int C, int K, int silu, void* stream) {
    if (B <= 0 || S <= 0 || C <= 0) return LME_OK;
    if (C % 8 || K < 1 || K > CONV_MAX_K || x_b % 8 || x_t % 8) return LME_ERR_SHAPE;
    if (K != 4 && (x_t != C || (B > 1 && x_b != static_cast<long long>(S) * C))) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) return LME_ERR_ALIGN;
    dim3 grid((C / 8 + 127) / 128, (S + CONV_CHUNK - 1) / CONV_CHUNK, B);
    auto X = static_cast<const __nv_bfloat16*>(x);
    auto W = static_cast<const __nv_bfloat16*>(w);
    auto BI = static_cast<const __nv_bfloat16*>(bias);
    auto IN = static_cast<const __nv_bfloat16*>(init);
    auto Y = static_cast<__nv_bfloat16*>(y);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (K == 4) {
        if (reinterpret_cast<uintptr_t>(w) & 7) return LME_ERR_ALIGN;
        const Conv4 p{X, W, BI, IN, x_b, x_t, S, C, silu};
        const int runs = (S + CONV4_STEPS - 1) / CONV4_STEPS, groups = (C / 4 + 127) / 128;
        const bool exchanged = runs > 65535;
        causal_conv4_fwd_kernel<<<exchanged ? dim3(runs, groups, B) : dim3(groups, runs, B), 128, 0, st>>>(p, Y, exchanged);
    } else if (K < 4) causal_conv1d_fwd_kernel<4><<<grid, 128, 0, st>>>(X, W, BI, IN, Y, B, S, C, K, silu);
    else causal_conv1d_fwd_kernel<CONV_MAX_K><<<grid, 128, 0, st>>>(X, W, BI, IN, Y, B, S, C, K, silu);
    return cudaGetLastError() == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}

// dw [C, K], dbias [C] (may be null), dinit [B, C, K-1] (may be null) are fp32; dw / dbias must be zeroed by the caller
// (they are accumulated atomically), dinit is written.
extern "C" int lme_causal_conv1d_bwd(const void* x, long long x_b, long long x_t, const void* w, const void* bias,
                                     const void* init, const void* dy, void* dx, float* dw, float* dbias, float* dinit,
                                     int B, int S, int C, int K, int silu, void* stream) {
    if (B <= 0 || S <= 0 || C <= 0) return LME_OK;
    if (C % 8 || K < 1 || K > CONV_MAX_K || x_b % 8 || x_t % 8) return LME_ERR_SHAPE;
    if (K != 4 && (x_t != C || (B > 1 && x_b != static_cast<long long>(S) * C))) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 15)
        return LME_ERR_ALIGN;
    dim3 grid((C / 8 + 127) / 128, (S + CONV_CHUNK - 1) / CONV_CHUNK, B);
    auto X = static_cast<const __nv_bfloat16*>(x);
    auto W = static_cast<const __nv_bfloat16*>(w);
    auto BI = static_cast<const __nv_bfloat16*>(bias);
    auto IN = static_cast<const __nv_bfloat16*>(init);
    auto DY = static_cast<const __nv_bfloat16*>(dy);
    auto DX = static_cast<__nv_bfloat16*>(dx);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (K == 4) {
        if (reinterpret_cast<uintptr_t>(w) & 7) return LME_ERR_ALIGN;
        const Conv4 p{X, W, BI, IN, x_b, x_t, S, C, silu};
        const int runs = 8 * CONV4_STEPS;
        causal_conv4_bwd_kernel<<<dim3((C / 4 + 31) / 32, (S + runs - 1) / runs, B), dim3(32, 8), 0, st>>>(
            p, DY, DX, dw, dbias, dinit);
    } else if (K < 4)
        causal_conv1d_bwd_kernel<4><<<grid, 128, 0, st>>>(X, W, BI, IN, DY, DX, dw, dbias, dinit, B, S, C, K, silu);
    else
        causal_conv1d_bwd_kernel<CONV_MAX_K><<<grid, 128, 0, st>>>(X, W, BI, IN, DY, DX, dw, dbias, dinit, B, S, C,
                                                                          K, silu);
    return cudaGetLastError() == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}
