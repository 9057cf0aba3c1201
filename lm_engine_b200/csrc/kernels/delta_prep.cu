// Everything of the chunk-parallel gated delta rule that is local to a 64-step block, forward and backward, in one
// kernel each way (the chain over the blocks is delta_rule.cu).  With q^ = scale q / |q|, k^ = k / |k| (rows), G the
// cumulative log-decay inside the block and D[t, i] = e^{G_t - G_i}:
//     A = strict_tril(beta_t D k^ k^T),  X = (I + A)^{-1},  W_v = X (beta v),  W_k = X (beta e^G k^)
//     QK = tril(D q^ k^T),  Q_e = e^G q^,  K_e = e^{G_L - G} k^,  a = e^{G_L}
// and the reverse pass takes the gradients of those operands back to q, k, v, g and beta.
//
// The work is a few MFLOP per block on 200 KB of operands: bound by launches and passes when it is a sequence of
// tensor operations, by HBM when it is one.  fp32 accuracy is kept on the tensor cores: q, k, v and the chain's U / dU
// ARE bf16, so products of two of them (K K^T, Q K^T, dU V^T) are exact bf16 products accumulated in fp32 with the row
// scales applied afterwards, and a product of an fp32 coefficient matrix with one of them splits the coefficients into
// three bf16 terms (24 bits of mantissa).  Contractions along a row read their fragments straight from global memory
// in 16-byte pieces (the contraction index is numbered so that a piece is a fragment).
// Measured (batch 2, 2048 steps, 4 heads, K = 256, V = 512: 256 blocks): 57 us forward, 153 us backward (217 us with eight
// warps per block instead of sixteen); the tensor operations took about 800 us and 1100 us in 180 launches.  The backward
// waits for memory a third of the time (one CTA per SM, 1.7 waves); its tensor pipe is at 15 %.
// Included by lme_cuda.cu after delta_rule.cu.

namespace lme {
namespace dp {

using m2::mma16816;

constexpr int L = 64;
constexpr int LD = 68;        // floats per row of a 64 x 64 matrix in shared memory (16-byte rows, banks spread)
constexpr int THREADS = 256;  // of the forward kernel; warp w: rows 16 (w & 3) .. + 16, column group w >> 2

struct Rows {                 // one head's rows of a [B, S, N, X] tensor with unit inner stride
    const __nv_bfloat16* p;
    long long b, s, n;        // element strides
};

struct FwdArgs {
    Rows q, k, v;
    const float *g, *beta;                                // [B, S, N] contiguous
    __nv_bfloat16 *wk, *qe, *ke, *ket, *qk;               // [B N nc] x [L, K], [L, K], [L, K], [K, L], [L, L]
    float *wv, *x, *a;                                    // [L, V], [L, L], scalar
    int S, N, nc, V, l2norm;
    float scale;
};

struct BwdArgs {
    Rows q, k, v;
    const float *g, *beta, *x;
    const __nv_bfloat16 *du, *h, *dh;                     // [L, V], [K, V], [K, V]
    const float *duh, *dqe, *dqk, *dke;                   // dU h^T = -dW_k [L, K], [L, K], [L, L], [L, K]
    __nv_bfloat16 *dq, *dk, *dv;                          // [B, S, N, X] contiguous
    float *dg, *dbeta;                                    // [B, S, N]
    int S, N, nc, V, l2norm;
    float scale;
};

__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }

// the block's row vectors
struct Vectors {
    float G[L], E[L], beta[L];
    float rq[L], rk[L];       // scale / (|q| + eps), 1 / (|k| + eps)
    float nq[L], nk[L];       // |q|, |k|
};

template <int K>
__device__ __forceinline__ void load_vectors(Vectors& s, const __nv_bfloat16* q, long long qs, const __nv_bfloat16* k,
                                             long long ks, const float* g, const float* beta, int N, int valid,
                                             int l2norm, float scale) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < L; r += blockDim.x >> 5) {
        float sq = 0.f, sk = 0.f;
        if (r < valid && lane * 8 < K) {
            const uint4 a = *reinterpret_cast<const uint4*>(q + r * qs + lane * 8);
            const uint4 b = *reinterpret_cast<const uint4*>(k + r * ks + lane * 8);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float2 f = unpack_bf16x2(word(a, i));
                sq += f.x * f.x + f.y * f.y;
                f = unpack_bf16x2(word(b, i));
                sk += f.x * f.x + f.y * f.y;
            }
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        if (lane == 0) {
            s.nq[r] = sqrtf(sq);
            s.nk[r] = sqrtf(sk);
            s.rq[r] = l2norm ? scale / (s.nq[r] + 1e-6f) : scale;
            s.rk[r] = l2norm ? 1.f / (s.nk[r] + 1e-6f) : 1.f;
        }
    }
    if (warp == 0) {
        const int r = 2 * lane;
        const float g0 = r < valid ? g[static_cast<long long>(r) * N] : 0.f;
        const float g1 = r + 1 < valid ? g[static_cast<long long>(r + 1) * N] : 0.f;
        float sum = g0 + g1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        const float before = sum - (g0 + g1);
        s.G[r] = before + g0;
        s.G[r + 1] = sum;
        s.E[r] = expf(before + g0);
        s.E[r + 1] = expf(sum);
        s.beta[r] = r < valid ? beta[static_cast<long long>(r) * N] : 0.f;
        s.beta[r + 1] = r + 1 < valid ? beta[static_cast<long long>(r + 1) * N] : 0.f;
    }
}

// 16 bytes of row r (zeros beyond `valid`)
__device__ __forceinline__ uint4 piece(const __nv_bfloat16* p, long long stride, int r, int valid) {
    return r < valid ? __ldg(reinterpret_cast<const uint4*>(p + r * stride)) : make_uint4(0, 0, 0, 0);
}

// acc[nt] += A[m0 .. m0+16) B[n0 + 8 nt ..)^T over `len` (a multiple of 32) columns, both row-major bf16 in global memory
template <int NT>
__device__ __forceinline__ void rows_by_rows(float (&acc)[NT][4], const __nv_bfloat16* A, long long as, int avalid, int m0,
                                             const __nv_bfloat16* B, long long bs, int bvalid, int n0, int len) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 2
    for (int j = 0; j < len; j += 32) {
        const uint4 lo = piece(A + j + 8 * t, as, m0 + g, avalid), hi = piece(A + j + 8 * t, as, m0 + g + 8, avalid);
        const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const uint4 b = piece(B + j + 8 * t, bs, n0 + nt * 8 + g, bvalid);
            mma16816(acc[nt], a0, b.x, b.y);
            mma16816(acc[nt], a1, b.z, b.w);
        }
    }
}

// fragment (value pairs) of product tile nt: rows m0 + g and m0 + g + 8, columns n0 + 8 nt + 2t, + 1
template <int NT, typename F>
__device__ __forceinline__ void each_pair(const float (&acc)[NT][4], int m0, int n0, F f) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half)
            f(m0 + g + 8 * half, n0 + nt * 8 + 2 * t, acc[nt][2 * half], acc[nt][2 * half + 1]);
}

// acc (16 rows x 64 columns) += sum over rows c of k-steps [ks0, ks1) of coef(r, c) B[c][64 columns], coef in fp32 as
// three bf16 terms.  Tile i of acc, product column n: column 8 n + i of the slab.
template <typename F>
__device__ __forceinline__ void coef_by_rows(float (&acc)[8][4], F coef, int m0, int ks0, int ks1,
                                             const __nv_bfloat16* B, long long bs, int bvalid) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    for (int ks = ks0; ks < ks1; ++ks) {
        const int c = ks * 16 + 2 * t;
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = m0 + g + 8 * (e & 1), cc = c + 8 * (e >> 1);
            split3(coef(r, cc), coef(r, cc + 1), a[0][e], a[1][e], a[2][e]);
        }
        const uint4 w0 = piece(B + 8 * g, bs, c, bvalid), w1 = piece(B + 8 * g, bs, c + 1, bvalid);
        const uint4 w2 = piece(B + 8 * g, bs, c + 8, bvalid), w3 = piece(B + 8 * g, bs, c + 9, bvalid);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
            const uint32_t b0 = __byte_perm(word(w0, i >> 1), word(w1, i >> 1), sel);
            const uint32_t b1 = __byte_perm(word(w2, i >> 1), word(w3, i >> 1), sel);
            mma16816(acc[i], a[0], b0, b1);
            mma16816(acc[i], a[1], b0, b1);
            mma16816(acc[i], a[2], b0, b1);
        }
    }
}

// the same with fp32 rows B (contiguous, `bs` floats apart): six of the nine products of the two splits reach 2^-24
template <typename F>
__device__ __forceinline__ void coef_by_rows_f32(float (&acc)[8][4], F coef, int m0, int ks0, int ks1, const float* B,
                                                 int bs) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    for (int ks = ks0; ks < ks1; ++ks) {
        const int c = ks * 16 + 2 * t;
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = m0 + g + 8 * (e & 1), cc = c + 8 * (e >> 1);
            split3(coef(r, cc), coef(r, cc + 1), a[0][e], a[1][e], a[2][e]);
        }
        const float* p = B + static_cast<long long>(c) * bs + 8 * g;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 r0 = __ldg(reinterpret_cast<const float4*>(p + 4 * h));
            const float4 r1 = __ldg(reinterpret_cast<const float4*>(p + bs + 4 * h));
            const float4 r2 = __ldg(reinterpret_cast<const float4*>(p + 8 * bs + 4 * h));
            const float4 r3 = __ldg(reinterpret_cast<const float4*>(p + 9 * bs + 4 * h));
            const float x0[4] = {r0.x, r0.y, r0.z, r0.w}, x1[4] = {r1.x, r1.y, r1.z, r1.w};
            const float x2[4] = {r2.x, r2.y, r2.z, r2.w}, x3[4] = {r3.x, r3.y, r3.z, r3.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t b0[3], b1[3];
                split3(x0[i], x1[i], b0[0], b0[1], b0[2]);
                split3(x2[i], x3[i], b1[0], b1[1], b1[2]);
#pragma unroll
                for (int u = 0; u < 3; ++u)
#pragma unroll
                    for (int w = 0; w < 3 - u; ++w) mma16816(acc[4 * h + i], a[u], b0[w], b1[w]);
            }
        }
    }
}

// a lane's 16 consecutive columns (16 t ..) of the slab in row `half` of its pair: f(value index j, value)
__device__ __forceinline__ void lane_columns(const float (&acc)[8][4], int half, float (&out)[16]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        out[i] = acc[i][2 * half];
        out[8 + i] = acc[i][2 * half + 1];
    }
}
__device__ __forceinline__ void clear(float (&acc)[8][4]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
}
__device__ __forceinline__ void store16(__nv_bfloat16* p, const float (&v)[16]) {
    uint4 o[2];
    uint32_t* w = reinterpret_cast<uint32_t*>(o);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
    reinterpret_cast<uint4*>(p)[0] = o[0];
    reinterpret_cast<uint4*>(p)[1] = o[1];
}
__device__ __forceinline__ void load16(const __nv_bfloat16* p, float (&v)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(p) + h);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = unpack_bf16x2(word(u, i));
            v[8 * h + 2 * i] = f.x;
            v[8 * h + 2 * i + 1] = f.y;
        }
    }
}
__device__ __forceinline__ void load16(const float* p, float (&v)[16]) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p) + h);
        v[4 * h] = f.x; v[4 * h + 1] = f.y; v[4 * h + 2] = f.z; v[4 * h + 3] = f.w;
    }
}

struct FwdSmem {
    float at[L][LD];      // at[i][t] = A[t][i]
    float x[L][LD];       // X
    Vectors s;
};

template <int K>
__global__ void __launch_bounds__(THREADS, 2) delta_prep_fwd_kernel(const FwdArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FwdSmem& sm = *reinterpret_cast<FwdSmem*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m0 = (warp & 3) * 16, nh = warp >> 2;
    const long long blk = blockIdx.x;
    const int c = blk % p.nc;
    const long long bn = blk / p.nc, b = bn / p.N, n = bn % p.N;
    const int s0 = c * L, valid = min(L, p.S - s0);
    const __nv_bfloat16* q = p.q.p + b * p.q.b + s0 * p.q.s + n * p.q.n;
    const __nv_bfloat16* k = p.k.p + b * p.k.b + s0 * p.k.s + n * p.k.n;
    const __nv_bfloat16* v = p.v.p + b * p.v.b + s0 * p.v.s + n * p.v.n;
    const long long go = (b * p.S + s0) * p.N + n;
    load_vectors<K>(sm.s, q, p.q.s, k, p.k.s, p.g + go, p.beta + go, p.N, valid, p.l2norm, p.scale);
    __syncthreads();
    const Vectors& s = sm.s;

    // A^T to shared memory, QK to global memory
    {
        float kk[4][4] = {}, qk[4][4] = {};
        const int n0 = nh * 32;
        if (n0 < m0 + 16) {
            rows_by_rows(kk, k, p.k.s, valid, m0, k, p.k.s, valid, n0, K);
            rows_by_rows(qk, q, p.q.s, valid, m0, k, p.k.s, valid, n0, K);
        }
        each_pair(kk, m0, n0, [&](int r, int i, float x0, float x1) {
            const float f = s.beta[r] * s.rk[r];
            sm.at[i][r] = i < r ? f * expf(s.G[r] - s.G[i]) * s.rk[i] * x0 : 0.f;
            sm.at[i + 1][r] = i + 1 < r ? f * expf(s.G[r] - s.G[i + 1]) * s.rk[i + 1] * x1 : 0.f;
        });
        each_pair(qk, m0, n0, [&](int r, int i, float x0, float x1) {
            x0 = i <= r ? s.rq[r] * expf(s.G[r] - s.G[i]) * s.rk[i] * x0 : 0.f;
            x1 = i + 1 <= r ? s.rq[r] * expf(s.G[r] - s.G[i + 1]) * s.rk[i + 1] * x1 : 0.f;
            *reinterpret_cast<uint32_t*>(p.qk + (blk * L + r) * L + i) = pack_bf16x2(x0, x1);
        });
    }
    __syncthreads();
    if (threadIdx.x < L) {
        // column j of X by forward substitution, sixteen rows at a time
        const int j = threadIdx.x;
        for (int r0 = 0; r0 < L; r0 += 16) {
            float acc[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) acc[r] = r0 + r == j ? 1.f : 0.f;
            for (int i = 0; i < r0; ++i) {
                const float xi = sm.x[i][j];
#pragma unroll
                for (int r = 0; r < 16; r += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(&sm.at[i][r0 + r]);
                    acc[r] -= a.x * xi; acc[r + 1] -= a.y * xi; acc[r + 2] -= a.z * xi; acc[r + 3] -= a.w * xi;
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                sm.x[r0 + i][j] = acc[i];
#pragma unroll
                for (int r = i + 1; r < 16; ++r) acc[r] -= sm.at[r0 + i][r0 + r] * acc[i];
            }
        }
    } else {
        // meanwhile: Q_e, K_e and K_e^T (eight rows x eight columns per step, transposed in registers)
        const float gl = s.G[L - 1];
        for (int u = threadIdx.x - L; u < (L / 8) * (K / 8); u += THREADS - L) {
            const int r0 = (u % (L / 8)) * 8, d = (u / (L / 8)) * 8;
            float kt[8][8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint4 a = piece(q + d, p.q.s, r0 + r, valid), w = piece(k + d, p.k.s, r0 + r, valid);
                const float fq = s.E[r0 + r] * s.rq[r0 + r], fk = expf(gl - s.G[r0 + r]) * s.rk[r0 + r];
                uint4 oq, ok;
                uint32_t* pq = reinterpret_cast<uint32_t*>(&oq);
                uint32_t* pk = reinterpret_cast<uint32_t*>(&ok);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float2 f = unpack_bf16x2(word(a, i));
                    pq[i] = pack_bf16x2(f.x * fq, f.y * fq);
                    f = unpack_bf16x2(word(w, i));
                    kt[2 * i][r] = f.x * fk;
                    kt[2 * i + 1][r] = f.y * fk;
                    pk[i] = pack_bf16x2(kt[2 * i][r], kt[2 * i + 1][r]);
                }
                *reinterpret_cast<uint4*>(p.qe + (blk * L + r0 + r) * K + d) = oq;
                *reinterpret_cast<uint4*>(p.ke + (blk * L + r0 + r) * K + d) = ok;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint4 o;
                uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
                for (int r = 0; r < 4; ++r) po[r] = pack_bf16x2(kt[i][2 * r], kt[i][2 * r + 1]);
                *reinterpret_cast<uint4*>(p.ket + (blk * K + d + i) * L + r0) = o;
            }
        }
        if (threadIdx.x == L) p.a[blk] = expf(gl);
    }
    __syncthreads();
    for (int u = threadIdx.x; u < L * L / 4; u += THREADS)
        *reinterpret_cast<float4*>(p.x + blk * L * L + 4 * u) =
            *reinterpret_cast<const float4*>(&sm.x[u / (L / 4)][4 * (u % (L / 4))]);
    const int ks1 = m0 / 16 + 1;     // X is lower triangular
    for (int slab = nh; slab < p.V / 64; slab += 2) {
        float acc[8][4];
        clear(acc);
        coef_by_rows(acc, [&](int r, int i) { return sm.x[r][i] * s.beta[i]; }, m0, 0, ks1, v + slab * 64, p.v.s, valid);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float o[16];
            lane_columns(acc, half, o);
            float* dst = p.wv + (blk * L + m0 + g + 8 * half) * p.V + slab * 64 + 16 * t;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                reinterpret_cast<float4*>(dst)[i] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        }
    }
    for (int slab = nh; slab < K / 64; slab += 2) {
        float acc[8][4];
        clear(acc);
        coef_by_rows(acc, [&](int r, int i) { return sm.x[r][i] * (s.beta[i] * s.E[i] * s.rk[i]); }, m0, 0, ks1,
                     k + slab * 64, p.k.s, valid);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float o[16];
            lane_columns(acc, half, o);
            store16(p.wk + (blk * L + m0 + g + 8 * half) * K + slab * 64 + 16 * t, o);
        }
    }
}

// HG: groups of columns, four warps each (the 64 rows of a block): a slab of 64 columns of q / k per warp, so that a
// block of K = 256 runs on sixteen warps and its chains of dependent products overlap
template <int HG>
struct BwdSmem {
    float x[L][LD];
    float n1[L][LD];      // dU V^T, then the combined N, then the coefficients F1 of dK K^T
    float n2[L][LD];      // dW_k K^T, then X^T N, then the decay gradients D-weighted (row minus column sums go to dG)
    float kk[L][LD];      // K K^T, then the coefficients F2 of dQ K^T
    float qk[L][LD];      // Q K^T
    Vectors s;
    float el[L];          // e^{G_L - G}
    float dG[L], dbeta[L];
    float dot[4][HG][L];  // row dots by column group: dq.q, dqe.q, dk.k, dke.k
    float red[32];
    float da;
};

template <int K>
__global__ void __launch_bounds__(2 * K, 1) delta_prep_bwd_kernel(const BwdArgs p) {
    constexpr int HG = K / 64, THREADS = 128 * HG;   // hides the forward kernel's thread count
    constexpr int NT = 8 / HG;                       // 8-column tiles of a 64 x 64 product per warp
    constexpr int TR = 64 * 16 / THREADS;            // rows of the register tile of the 64 x 64 fp32 products
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BwdSmem<HG>& sm = *reinterpret_cast<BwdSmem<HG>*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int m0 = (warp & 3) * 16, nh = warp >> 2;
    const long long blk = blockIdx.x;
    const int c = blk % p.nc, V = p.V;
    const long long bn = blk / p.nc, b = bn / p.N, n = bn % p.N;
    const int s0 = c * L, valid = min(L, p.S - s0);
    const __nv_bfloat16* q = p.q.p + b * p.q.b + s0 * p.q.s + n * p.q.n;
    const __nv_bfloat16* k = p.k.p + b * p.k.b + s0 * p.k.s + n * p.k.n;
    const __nv_bfloat16* v = p.v.p + b * p.v.b + s0 * p.v.s + n * p.v.n;
    const long long go = (b * p.S + s0) * p.N + n;
    const __nv_bfloat16* du = p.du + blk * L * V;
    const float* duh = p.duh + blk * L * K;
    load_vectors<K>(sm.s, q, p.q.s, k, p.k.s, p.g + go, p.beta + go, p.N, valid, p.l2norm, p.scale);
    for (int u = tid; u < L * L / 4; u += THREADS)
        *reinterpret_cast<float4*>(&sm.x[u / (L / 4)][4 * (u % (L / 4))]) =
            *reinterpret_cast<const float4*>(p.x + blk * L * L + 4 * u);
    {   // da = sum of dh * h over the state entering the block
        const uint4* ph = reinterpret_cast<const uint4*>(p.h + blk * K * V);
        const uint4* pd = reinterpret_cast<const uint4*>(p.dh + blk * K * V);
        float sum = 0.f;
#pragma unroll 4
        for (int u = tid; u < K * V / 8; u += THREADS) {
            const uint4 x = __ldg(ph + u), y = __ldg(pd + u);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 e = unpack_bf16x2(word(x, i)), f = unpack_bf16x2(word(y, i));
                sum += e.x * f.x + e.y * f.y;
            }
        }
        sum = block_sum(sum, sm.red);
        if (tid == 0) sm.da = sum;
    }
    __syncthreads();
    const Vectors& s = sm.s;
    if (tid < L) sm.el[tid] = expf(s.G[L - 1] - s.G[tid]);

    {
        const int n0 = nh * 8 * NT;
        float acc[NT][4] = {};
        rows_by_rows(acc, du, V, L, m0, v, p.v.s, valid, n0, V);
        each_pair(acc, m0, n0, [&](int r, int i, float x0, float x1) { sm.n1[r][i] = x0; sm.n1[r][i + 1] = x1; });
        // dW_k K^T with dW_k = -dU h^T in fp32 (three bf16 terms)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        for (int j = 0; j < K; j += 32) {
            uint32_t a[2][3][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const float* pa = duh + (m0 + g + 8 * half) * K + j + 8 * t;
                const float4 f0 = __ldg(reinterpret_cast<const float4*>(pa)), f1 = __ldg(reinterpret_cast<const float4*>(pa) + 1);
                split3(-f0.x, -f0.y, a[0][0][half], a[0][1][half], a[0][2][half]);
                split3(-f0.z, -f0.w, a[0][0][2 + half], a[0][1][2 + half], a[0][2][2 + half]);
                split3(-f1.x, -f1.y, a[1][0][half], a[1][1][half], a[1][2][half]);
                split3(-f1.z, -f1.w, a[1][0][2 + half], a[1][1][2 + half], a[1][2][2 + half]);
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 w = piece(k + j + 8 * t, p.k.s, n0 + nt * 8 + g, valid);
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    mma16816(acc[nt], a[0][u], w.x, w.y);
                    mma16816(acc[nt], a[1][u], w.z, w.w);
                }
            }
        }
        each_pair(acc, m0, n0, [&](int r, int i, float x0, float x1) { sm.n2[r][i] = x0; sm.n2[r][i + 1] = x1; });
        float kk[NT][4] = {}, qk[NT][4] = {};
        if (n0 < m0 + 16) {
            rows_by_rows(kk, k, p.k.s, valid, m0, k, p.k.s, valid, n0, K);
            rows_by_rows(qk, q, p.q.s, valid, m0, k, p.k.s, valid, n0, K);
        }
        each_pair(kk, m0, n0, [&](int r, int i, float x0, float x1) { sm.kk[r][i] = x0; sm.kk[r][i + 1] = x1; });
        each_pair(qk, m0, n0, [&](int r, int i, float x0, float x1) { sm.qk[r][i] = x0; sm.qk[r][i + 1] = x1; });
    }
    __syncthreads();
    if (tid < L) {
        float d1 = 0.f, d2 = 0.f;
        for (int r = tid; r < L; ++r) {
            d1 += sm.x[r][tid] * sm.n1[r][tid];
            d2 += sm.x[r][tid] * sm.n2[r][tid];
        }
        const float e = s.E[tid] * s.rk[tid] * d2;
        sm.dbeta[tid] = d1 + e;
        sm.dG[tid] = s.beta[tid] * e;
    }
    __syncthreads();
    const int ty = tid >> 4, tx = tid & 15;
    for (int u = tid; u < L * L; u += THREADS) {
        const int r = u / L, i = u % L;
        sm.n1[r][i] = s.beta[i] * (sm.n1[r][i] + s.E[i] * s.rk[i] * sm.n2[r][i]);
    }
    __syncthreads();
    {   // Y = X^T N: rows TR ty + i, columns 4 tx + j
        float y[TR][4] = {};
        for (int r = TR * ty; r < L; ++r) {     // X[r][i] = 0 for r < i
            const float4 nb = *reinterpret_cast<const float4*>(&sm.n1[r][4 * tx]);
            const float ns[4] = {nb.x, nb.y, nb.z, nb.w};
#pragma unroll
            for (int i = 0; i < TR; ++i) {
                const float xi = sm.x[r][TR * ty + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) y[i][j] += xi * ns[j];
            }
        }
#pragma unroll
        for (int i = 0; i < TR; ++i)
            *reinterpret_cast<float4*>(&sm.n2[TR * ty + i][4 * tx]) = make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
    }
    __syncthreads();
    {   // dA = -strict_tril(Y X^T); rows TR ty + i, columns tx + 16 j
        float da[TR][4] = {};
        for (int m = 0; m < L; m += 4) {
            float4 yv[TR], xv[4];
#pragma unroll
            for (int i = 0; i < TR; ++i) yv[i] = *reinterpret_cast<const float4*>(&sm.n2[TR * ty + i][m]);
#pragma unroll
            for (int i = 0; i < 4; ++i) xv[i] = *reinterpret_cast<const float4*>(&sm.x[tx + 16 * i][m]);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    da[i][j] -= yv[i].x * xv[j].x + yv[i].y * xv[j].y + yv[i].z * xv[j].z + yv[i].w * xv[j].w;
        }
        __syncthreads();      // Y and N are read no more
#pragma unroll
        for (int i = 0; i < TR; ++i) {
            const int r = TR * ty + i;
            float db = 0.f, rows = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = tx + 16 * j;
                float f1 = 0.f, f2 = 0.f, z = 0.f;
                if (col <= r) {
                    const float D = expf(s.G[r] - s.G[col]);
                    if (col < r) {
                        const float a1 = D * sm.kk[r][col] * s.rk[r] * s.rk[col];
                        db += da[i][j] * a1;
                        z = da[i][j] * s.beta[r] * a1;
                        f1 = da[i][j] * s.beta[r] * D;
                    }
                    f2 = __ldg(p.dqk + blk * L * L + r * L + col) * D;
                    z += f2 * sm.qk[r][col] * s.rq[r] * s.rk[col];
                }
                rows += z;
                sm.n1[r][col] = f1;
                sm.n2[r][col] = z;
                sm.kk[r][col] = f2;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                db += __shfl_xor_sync(0xffffffffu, db, o);
                rows += __shfl_xor_sync(0xffffffffu, rows, o);
            }
            if (tx == 0) {
                sm.dbeta[r] += db;
                sm.dG[r] += rows;
            }
        }
    }
    __syncthreads();
    if (tid < L) {
        float cols = 0.f;
        for (int r = tid; r < L; ++r) cols += sm.n2[r][tid];
        sm.dG[tid] -= cols;
    }
    const int mi = m0 / 16;
    const long long tok = (b * p.S + s0) * p.N + n;      // first token's row of a [B, S, N, *] tensor
    // dv_i = beta_i sum_t X[t, i] dU_t
    for (int slab = nh; slab < V / 64; slab += HG) {
        float acc[8][4];
        clear(acc);
        coef_by_rows(acc, [&](int r, int i) { return sm.x[i][r] * s.beta[r]; }, m0, mi, 4, du + slab * 64, V, L);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = m0 + g + 8 * half;
            float o[16];
            lane_columns(acc, half, o);
            if (r < valid) store16(p.dv + (tok + static_cast<long long>(r) * p.N) * V + slab * 64 + 16 * t, o);
        }
    }
    // dq and dk: the gradient of the normalised row, then the projection of the normalisation
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
        const __nv_bfloat16* raw = which == 0 ? q : k;
        const long long rs = which == 0 ? p.q.s : p.k.s;
        const float* direct = (which == 0 ? p.dqe : p.dke) + blk * L * K;
        float acc[8][4];
        float dot[2] = {}, ddot[2] = {};
        const int col = nh * 64;
        clear(acc);
        if (which == 0) {
            coef_by_rows(acc, [&](int r, int i) { return sm.kk[r][i] * s.rk[i]; }, m0, 0, mi + 1, k + col, p.k.s, valid);
        } else {
            coef_by_rows(acc, [&](int r, int i) { return (sm.n1[r][i] + sm.n1[i][r]) * s.rk[i]; }, m0, 0, 4, k + col,
                         p.k.s, valid);
            coef_by_rows(acc, [&](int r, int i) { return sm.kk[i][r] * s.rq[i]; }, m0, mi, 4, q + col, p.q.s, valid);
            coef_by_rows_f32(acc, [&](int r, int i) { return -sm.x[i][r] * (s.beta[r] * s.E[r]); }, m0, mi, 4, duh + col, K);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = m0 + g + 8 * half;
            const float f = which == 0 ? s.E[r] : sm.el[r];
            float d[16], w[16] = {};
            load16(direct + r * K + col + 16 * t, d);
            if (r < valid) load16(raw + r * rs + col + 16 * t, w);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float& a = acc[i & 7][2 * half + (i >> 3)];
                a += f * d[i];
                dot[half] += a * w[i];
                ddot[half] += d[i] * w[i];
            }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            dot[half] += __shfl_xor_sync(0xffffffffu, dot[half], 1);
            dot[half] += __shfl_xor_sync(0xffffffffu, dot[half], 2);
            ddot[half] += __shfl_xor_sync(0xffffffffu, ddot[half], 1);
            ddot[half] += __shfl_xor_sync(0xffffffffu, ddot[half], 2);
            if (t == 0) {
                sm.dot[2 * which][nh][m0 + g + 8 * half] = dot[half];
                sm.dot[2 * which + 1][nh][m0 + g + 8 * half] = ddot[half];
            }
        }
        __syncthreads();
        __nv_bfloat16* out = which == 0 ? p.dq : p.dk;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = m0 + g + 8 * half;
            if (r >= valid) continue;
            const float rr = which == 0 ? s.rq[r] : s.rk[r], norm = which == 0 ? s.nq[r] : s.nk[r];
            const float inv = 1.f / (norm + 1e-6f);
            float total = 0.f;
#pragma unroll
            for (int i = 0; i < HG; ++i) total += sm.dot[2 * which][i][r];
            const float proj = p.l2norm && norm > 0.f ? total * rr * inv / norm : 0.f;
            float o[16], w[16];
            lane_columns(acc, half, o);
            load16(raw + r * rs + col + 16 * t, w);
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = rr * o[i] - proj * w[i];
            store16(out + (tok + static_cast<long long>(r) * p.N) * K + col + 16 * t, o);
        }
    }
    __syncthreads();
    // dG: dqe . qe to its step, dke . ke from its step to the end of the block, da e^{G_L}; dg is the suffix sum
    if (tid < L) {
        float dqq = 0.f, dkk = 0.f;
#pragma unroll
        for (int i = 0; i < HG; ++i) {
            dqq += sm.dot[1][i][tid];
            dkk += sm.dot[3][i][tid];
        }
        const float e = sm.el[tid] * s.rk[tid] * dkk;
        sm.dG[tid] += s.E[tid] * s.rq[tid] * dqq - e;
        sm.n2[0][tid] = e;
    }
    __syncthreads();
    if (tid < 32) {
        float x0 = sm.dG[2 * lane], x1 = sm.dG[2 * lane + 1];
        const float all = warp_sum(sm.n2[0][2 * lane] + sm.n2[0][2 * lane + 1]);
        if (lane == 31) x1 += all + sm.da * s.E[L - 1];
        float sum = x0 + x1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float dn = __shfl_down_sync(0xffffffffu, sum, o);
            if (lane + o < 32) sum += dn;
        }
        const int r = 2 * lane;
        if (r < valid) p.dg[tok + static_cast<long long>(r) * p.N] = sum;
        if (r + 1 < valid) p.dg[tok + static_cast<long long>(r + 1) * p.N] = sum - x0;
    }
    if (tid < valid) p.dbeta[tok + static_cast<long long>(tid) * p.N] = sm.dbeta[tid];
}

static int check(const Rows& q, const Rows& k, const Rows& v, int B, int S, int N, int K, int V) {
    if (B <= 0 || S <= 0 || N <= 0 || (K != 128 && K != 256) || V <= 0 || V % 64) return LME_ERR_SHAPE;
    if ((q.b | q.s | q.n | k.b | k.s | k.n | v.b | v.s | v.n) % 8) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(q.p) | reinterpret_cast<uintptr_t>(k.p) | reinterpret_cast<uintptr_t>(v.p)) & 15)
        return LME_ERR_ALIGN;
    if (static_cast<long long>(B) * N * ((S + L - 1) / L) > 0x7fffffffll) return LME_ERR_SHAPE;
    return LME_OK;
}

template <auto Kern, typename Args>
static int launch(const Args& a, int threads, int smem, long long blocks, void* stream) {
    if (!opt_in<Kern>(cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) return LME_ERR_LAUNCH;
    Kern<<<static_cast<unsigned>(blocks), threads, smem, static_cast<cudaStream_t>(stream)>>>(a);
    return cudaGetLastError() == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}

}  // namespace dp
}  // namespace lme

// strides: nine element strides, (batch, token, head) of q, k and v
extern "C" int lme_delta_prep_fwd(const void* q, const void* k, const void* v, const long long* strides, const float* g,
                                  const float* beta, void* wk, void* qe, void* ke, void* ket, void* qk, float* wv,
                                  float* x, float* a, int B, int S, int N, int K, int V, int l2norm, float scale,
                                  void* stream) {
    using namespace lme::dp;
    using bf = __nv_bfloat16;
    const Rows rq{static_cast<const bf*>(q), strides[0], strides[1], strides[2]};
    const Rows rk{static_cast<const bf*>(k), strides[3], strides[4], strides[5]};
    const Rows rv{static_cast<const bf*>(v), strides[6], strides[7], strides[8]};
    if (int rc = check(rq, rk, rv, B, S, N, K, V)) return rc;
    const int nc = (S + L - 1) / L;
    const FwdArgs p{rq, rk, rv, g, beta, static_cast<bf*>(wk), static_cast<bf*>(qe), static_cast<bf*>(ke),
                    static_cast<bf*>(ket), static_cast<bf*>(qk), wv, x, a, S, N, nc, V, l2norm, scale};
    const long long blocks = static_cast<long long>(B) * N * nc;
    return K == 256 ? launch<delta_prep_fwd_kernel<256>>(p, THREADS, static_cast<int>(sizeof(FwdSmem)), blocks, stream)
                    : launch<delta_prep_fwd_kernel<128>>(p, THREADS, static_cast<int>(sizeof(FwdSmem)), blocks, stream);
}

extern "C" int lme_delta_prep_bwd(const void* q, const void* k, const void* v, const long long* strides, const float* g,
                                  const float* beta, const float* x, const void* du, const void* h, const void* dh,
                                  const float* duh, const float* dqe, const float* dqk, const float* dke, void* dq,
                                  void* dk, void* dv, float* dg, float* dbeta, int B, int S, int N, int K, int V,
                                  int l2norm, float scale, void* stream) {
    using namespace lme::dp;
    using bf = __nv_bfloat16;
    const Rows rq{static_cast<const bf*>(q), strides[0], strides[1], strides[2]};
    const Rows rk{static_cast<const bf*>(k), strides[3], strides[4], strides[5]};
    const Rows rv{static_cast<const bf*>(v), strides[6], strides[7], strides[8]};
    if (int rc = check(rq, rk, rv, B, S, N, K, V)) return rc;
    const int nc = (S + L - 1) / L;
    const BwdArgs p{rq, rk, rv, g, beta, x, static_cast<const bf*>(du), static_cast<const bf*>(h),
                    static_cast<const bf*>(dh), duh, dqe, dqk, dke, static_cast<bf*>(dq), static_cast<bf*>(dk),
                    static_cast<bf*>(dv), dg, dbeta, S, N, nc, V, l2norm, scale};
    const long long blocks = static_cast<long long>(B) * N * nc;
    return K == 256 ? launch<delta_prep_bwd_kernel<256>>(p, 512, static_cast<int>(sizeof(BwdSmem<4>)), blocks, stream)
                    : launch<delta_prep_bwd_kernel<128>>(p, 256, static_cast<int>(sizeof(BwdSmem<2>)), blocks, stream);
}
