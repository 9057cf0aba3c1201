// Mamba-2 SSD, intra-chunk part: y[l] = sum_{s <= l} exp(cum[l] - cum[s]) (C_l . B_s) xdt[s] per head and chunk.
//
//   ssd_decay_matrix : M[b,c,n,l,s] = CB[b,c,g(n),l,s] * exp(cum[b,c,n,l] - cum[b,c,n,s]) for s <= l, else 0   (bf16)
//                      -- one pass that replaces the difference / mask / exp / repeat / multiply chain over
//                      [chunks, heads, L, L] fp32 tensors; y = M @ xdt then runs on the tensor cores as a batched GEMM
//   ssd_dcb          : dCB[b,c,g,l,s] = sum_{n in g} dM[b,c,n,l,s] * exp(cum[n,l] - cum[n,s]) for s <= l
//                      -- one warp per (b, c, g, l) row loops over the heads of the group: no atomics
// The gradient with respect to cum needs no L x L pass: sum_s dM[l,s] M[l,s] = dy[l] . y[l] and
// sum_l dM[l,s] M[l,s] = xdt[s] . dxdt[s] (both are products of the same three factors), evaluated by the caller.
// Role of the chunk-scan kernels of mamba_ssm used by the reference
// (lm_engine/modeling_utils/sequence_mixer_blocks/mamba2/op.py:385-457).
namespace lme {

// Bound by its instructions (84 % of the issue slots; the write of m alone would take 20 us).  A block owns 32 rows of one
// head, so the index arithmetic is a few 32-bit operations per 16-byte vector (64-bit divisions per vector cost more than
// the exponentials).  1024 heads of 256 x 256 (134 MB): 89 -> 57 us.
constexpr int DECAY_ROWS = 32;

__global__ void __launch_bounds__(256)
ssd_decay_matrix_kernel(const __nv_bfloat16* __restrict__ cb, const float* __restrict__ cum,
                        __nv_bfloat16* __restrict__ m, int N, int G, int L) {
    const int vec_per_row = L / 8;
    const long long head = blockIdx.x;                   // (b*nc + c) * N + n
    const long long bc = head / N;
    const int g = static_cast<int>(head - bc * N) / (N / G);
    const int l0 = blockIdx.y * DECAY_ROWS, rows = min(DECAY_ROWS, L - l0);
    const float* cu = cum + head * L;
    const __nv_bfloat16* src = cb + (bc * G + g) * L * L;
    __nv_bfloat16* dst = m + head * L * L;
#pragma unroll 4
    for (int u = threadIdx.x; u < rows * vec_per_row; u += blockDim.x) {
        const int r = u / vec_per_row, s0 = (u - r * vec_per_row) * 8, l = l0 + r;
        float out[8];
        if (s0 > l) {
#pragma unroll
            for (int j = 0; j < 8; ++j) out[j] = 0.f;
        } else {
            float c8[8];
            load8(src + l * L + s0, c8);
            const float cl = __ldg(cu + l);
            const float4 a = __ldg(reinterpret_cast<const float4*>(cu + s0));
            const float4 b = __ldg(reinterpret_cast<const float4*>(cu + s0 + 4));
            const float cs[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) out[j] = (s0 + j <= l) ? c8[j] * __expf(cl - cs[j]) : 0.f;
        }
        store8(dst + l * L + s0, out);
    }
}

// one warp per (bc, g, l); block = 8 warps
template <int MAXV>
__global__ void __launch_bounds__(256)
ssd_dcb_kernel(const __nv_bfloat16* __restrict__ dm, const float* __restrict__ cum, __nv_bfloat16* __restrict__ dcb,
               long long rows_total, int N, int G, int L) {
    const int lane = threadIdx.x & 31;
    const long long row = blockIdx.x * 8ll + (threadIdx.x >> 5);   // (bc * G + g) * L + l
    if (row >= rows_total) return;
    const int l = static_cast<int>(row % L);
    const long long bcg = row / L;
    const int g = static_cast<int>(bcg % G);
    const long long bc = bcg / G;
    const int rep = N / G;
    const int nvec = L / 8;
    float acc[MAXV][8];
#pragma unroll
    for (int k = 0; k < MAXV; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[k][j] = 0.f;
    for (int r = 0; r < rep; ++r) {
        const long long head = bc * N + g * rep + r;
        const float* cu = cum + head * L;
        const float cl = cu[l];
        const __nv_bfloat16* drow = dm + (head * L + l) * L;
#pragma unroll
        for (int k = 0; k < MAXV; ++k) {
            const int v = lane + 32 * k;
            const int s0 = v * 8;
            if (v < nvec && s0 <= l) {
                float d8[8];
                load8(drow + s0, d8);
                const float4 a = *reinterpret_cast<const float4*>(cu + s0);
                const float4 b = *reinterpret_cast<const float4*>(cu + s0 + 4);
                const float cs[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (s0 + j <= l) acc[k][j] += d8[j] * __expf(cl - cs[j]);
            }
        }
    }
    __nv_bfloat16* orow = dcb + row * L;
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
        const int v = lane + 32 * k;
        if (v < nvec) store8(orow + v * 8, acc[k]);
    }
}

// ------------------------------------------------------------------------------------------------ decays
// Per-(token, head) scalars of the chunked scan.  dt [BC, L, N] -> cum (inclusive sums of dt A inside the chunk), laid
// out for its readers: ct = cum, dtt = dt and tail = exp(cum_last - cum) as [BC, N, L], ecum = exp(cum) as [BC, L, N],
// decay = exp(cum_last) [BC, N].  A CTA holds eight heads of a chunk in shared memory and a warp scans a head 32 steps
// at a time (the library's scan along an outer dimension takes 64 us for the same 1 MB; with 32 heads per CTA only 32
// CTAs existed for 16 chunks x 64 heads and the reverse took 41 us).
constexpr int DECAY_HEADS = 8;                       // one per warp
constexpr int DECAY_LD = DECAY_HEADS + 1;           // at most 1024 rows of it: 36 KB

__global__ void __launch_bounds__(256)
ssd_decay_fwd_kernel(const float* __restrict__ dt, const float* __restrict__ A, float* __restrict__ ct,
                     float* __restrict__ dtt, float* __restrict__ tail, float* __restrict__ ecum,
                     float* __restrict__ decay, int N, int L) {
    extern __shared__ float tile[];                  // [L][DECAY_LD]
    const long long bc = blockIdx.x;
    const int n0 = blockIdx.y * DECAY_HEADS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hh = threadIdx.x % DECAY_HEADS, l0t = threadIdx.x / DECAY_HEADS;      // the thread's column of the tile
    const bool has = n0 + hh < N;
    for (int l = l0t; l < L; l += 32) tile[l * DECAY_LD + hh] = has ? dt[(bc * L + l) * N + n0 + hh] : 0.f;
    __syncthreads();
    if (n0 + warp < N) {
        const float a = A[n0 + warp];
        float carry = 0.f;
        const long long row = (bc * N + n0 + warp) * L;
        for (int l0 = 0; l0 < L; l0 += 32) {
            float x = tile[(l0 + lane) * DECAY_LD + warp];
            dtt[row + l0 + lane] = x;
            x *= a;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += up;
            }
            x += carry;
            carry = __shfl_sync(0xffffffffu, x, 31);
            tile[(l0 + lane) * DECAY_LD + warp] = x;
            ct[row + l0 + lane] = x;
        }
        for (int l = lane; l < L; l += 32) tail[row + l] = expf(carry - tile[l * DECAY_LD + warp]);
        if (lane == 0) decay[bc * N + n0 + warp] = expf(carry);
    }
    __syncthreads();
    if (!has) return;
    for (int l = l0t; l < L; l += 32) ecum[(bc * L + l) * N + n0 + hh] = expf(tile[l * DECAY_LD + hh]);
}

// The reverse: with sy = dy . y_intra and decum ([BC, L, N]), sh = xh . dxh, sw = sum_p x dxw and ddt0, the direct gradient
// of dt ([BC, N, L]), dcum = sy - sh + ecum decum - tail dt sw, plus at the last step what tail and the chunk's decay
// send there; ddt = ddt0 + A * (suffix sums of dcum); per (chunk, head) sums of dt * suffix (dA) and of dDp (dD).
__global__ void __launch_bounds__(256)
ssd_decay_bwd_kernel(const float* __restrict__ dtt, const float* __restrict__ A, const float* __restrict__ tail,
                     const float* __restrict__ ecum, const float* __restrict__ decay, const float* __restrict__ sy,
                     const float* __restrict__ decum, const float* __restrict__ ddt0, const float* __restrict__ sw,
                     const float* __restrict__ sh, const float* __restrict__ ddecay_parts, int parts,
                     const float* __restrict__ dDp, float* __restrict__ ddt, float* __restrict__ dA_part,
                     float* __restrict__ dD_part, int N, int L) {
    extern __shared__ float tile[];                  // [L][DECAY_LD]
    __shared__ float red[32][DECAY_LD];
    const long long bc = blockIdx.x;
    const int n0 = blockIdx.y * DECAY_HEADS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hh = threadIdx.x % DECAY_HEADS, l0t = threadIdx.x / DECAY_HEADS;
    const bool has = n0 + hh < N;
    float dD = 0.f;
    for (int l = l0t; l < L; l += 32) {
        float v = 0.f;
        if (has) {
            const long long o = (bc * L + l) * N + n0 + hh;
            v = sy[o] + ecum[o] * decum[o];
            dD += dDp[o];
        }
        tile[l * DECAY_LD + hh] = v;
    }
    red[l0t][hh] = dD;
    __syncthreads();
    if (n0 + warp < N) {
        const long long bn = bc * N + n0 + warp, row = bn * L;
        float dd = 0.f, to_last = 0.f, dA = 0.f;
        for (int i = lane; i < parts; i += 32) dd += ddecay_parts[bn * parts + i];
        for (int l = lane; l < L; l += 32) {
            const float tw = tail[row + l] * dtt[row + l] * sw[row + l];
            to_last += tw;
            tile[l * DECAY_LD + warp] -= tw + sh[row + l];
        }
        float carry = warp_sum(to_last) + decay[bn] * warp_sum(dd);
        const float a = A[n0 + warp];
        __syncwarp();
        for (int l0 = L - 32; l0 >= 0; l0 -= 32) {
            float x = tile[(l0 + lane) * DECAY_LD + warp];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float dn = __shfl_down_sync(0xffffffffu, x, o);
                if (lane + o < 32) x += dn;
            }
            x += carry;
            carry = __shfl_sync(0xffffffffu, x, 0);
            dA += dtt[row + l0 + lane] * x;
            tile[(l0 + lane) * DECAY_LD + warp] = ddt0[row + l0 + lane] + a * x;
        }
        dA = warp_sum(dA);
        dD = warp_sum(red[lane][warp]);
        if (lane == 0) {
            dA_part[bn] = dA;
            dD_part[bn] = dD;
        }
    }
    __syncthreads();
    if (!has) return;
    for (int l = l0t; l < L; l += 32) ddt[(bc * L + l) * N + n0 + hh] = tile[l * DECAY_LD + hh];
}

// ------------------------------------------------------------------------------------------------ scan glue
// The element-wise passes around the products of the chunked scan, one kernel per direction instead of a chain of
// PyTorch ops over [tokens, heads, P] fp32 tensors (BC = batch x chunks, rows l of a chunk, heads n, P values; x may be a
// slice of wider rows, xs elements from token to token):
//   prep     xh [BC,N,L,P]  = x[BC,L,N,P] * dt[BC,N,L]                         (operand of the intra-chunk product)
//            xwT[BC,N,P,L]  = x * dt * tail[BC,N,L], transposed                 (operand of the chunk-state product)
//   prep^T   dx = dt (dxh + tail dxwT^T) + D dy;  row sums [BC,N,L]: ddt0 = sum_p x (dxh + tail dxwT^T),
//            sw = sum_p x dxwT^T, sh = sum_p xh dxh   (sy - sh is the intra-chunk gradient of cum: the two cancel over
//            a chunk, so both take the rounded xh that the products multiplied)
//   combine  y[BC,L,N,P] = yin[BC,N,L,P] + off[BC,G,L,rep*P] * ecum[BC,L,N] + D[n] * x
//   combine^T dyin = dy, doff = dy * ecum, sy = sum_p dy yin, decum = sum_p dy off, dDp = sum_p dy x   (sums [BC,L,N])
// prep: one block handles 32 rows of one (BC, n); a warp owns a row at a time (coalesced along P); the transposed
// operand goes through a padded shared-memory tile so that both its reads and writes are coalesced.
// combine: P / 8 lanes per row of P values, 16-byte accesses on the bf16 streams.  Row scalars are laid out for their
// readers ([BC,N,L] where a block owns a head, [BC,L,N] where it owns a token): 4-byte accesses 256 bytes apart took as
// long as the rest of the pass.  4096 tokens x 64 heads of 64: prep 24 / 49 us, combine 34 / 43 us (backward of prep 65, combine 63 / 74 before,
// with 2-byte accesses and a separate pass for D dy).
constexpr int GLUE_ROWS = 32;

template <int P>
__global__ void __launch_bounds__(256)
ssd_prep_kernel(const __nv_bfloat16* __restrict__ x, long long xs, const float* __restrict__ dt,
                const float* __restrict__ tail, __nv_bfloat16* __restrict__ xh, __nv_bfloat16* __restrict__ xwT, int N,
                int L) {
    __shared__ float tile[GLUE_ROWS][P + 1];
    const int l0 = blockIdx.x * GLUE_ROWS, n = blockIdx.y;
    const long long bc = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int r = warp; r < GLUE_ROWS; r += 8) {
        const int l = l0 + r;
        const long long tok = bc * L + l;
        const float d = dt[(bc * N + n) * L + l], tl = tail[(bc * N + n) * L + l];
        const __nv_bfloat16* xr = x + tok * xs + n * P;
        __nv_bfloat16* hr = xh + ((bc * N + n) * L + l) * P;
#pragma unroll
        for (int p = 2 * lane; p < P; p += 64) {
            float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(xr + p));
            v.x *= d;
            v.y *= d;
            *reinterpret_cast<uint32_t*>(hr + p) = pack_bf16x2(v.x, v.y);
            tile[r][p] = v.x * tl;
            tile[r][p + 1] = v.y * tl;
        }
    }
    __syncthreads();
    __nv_bfloat16* wt = xwT + (bc * N + n) * static_cast<long long>(P) * L + l0;
    // a half warp per row p: 16 lanes x 2 of the 32 steps
    for (int p = threadIdx.x >> 4; p < P; p += 16) {
        const int i = 2 * (threadIdx.x & 15);
        *reinterpret_cast<uint32_t*>(wt + static_cast<long long>(p) * L + i) = pack_bf16x2(tile[i][p], tile[i + 1][p]);
    }
}

template <int P>
__global__ void __launch_bounds__(256)
ssd_prep_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long xs, const float* __restrict__ dt,
                    const float* __restrict__ tail, const float* __restrict__ dxh,
                    const __nv_bfloat16* __restrict__ dxwT, const __nv_bfloat16* __restrict__ dy,
                    const float* __restrict__ D, __nv_bfloat16* __restrict__ dx, float* __restrict__ ddt0,
                    float* __restrict__ sw, float* __restrict__ sh, int N, int L) {
    __shared__ float tile[GLUE_ROWS][P + 1];
    const int l0 = blockIdx.x * GLUE_ROWS, n = blockIdx.y;
    const long long bc = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const __nv_bfloat16* wt = dxwT + (bc * N + n) * static_cast<long long>(P) * L + l0;
    for (int p = threadIdx.x >> 4; p < P; p += 16) {
        const int i = 2 * (threadIdx.x & 15);
        const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(wt + static_cast<long long>(p) * L + i));
        tile[i][p] = v.x;
        tile[i + 1][p] = v.y;
    }
    __syncthreads();
    constexpr int LANES = P / 4;           // lanes per row: 32 / LANES rows of the block at a time in a warp
    const float dn = D[n];
    const int p = 4 * (lane % LANES);
#pragma unroll
    for (int r = warp * (32 / LANES) + lane / LANES; r < GLUE_ROWS; r += 8 * (32 / LANES)) {
        const int l = l0 + r;
        const long long tok = bc * L + l, row = tok * N + n, hrow = (bc * N + n) * L + l;
        const float d = dt[hrow], tl = tail[hrow];
        const uint2 xr = *reinterpret_cast<const uint2*>(x + tok * xs + n * P + p);
        const float4 gv = *reinterpret_cast<const float4*>(dxh + hrow * P + p);
        const uint2 yr = *reinterpret_cast<const uint2*>(dy + row * P + p);
        const float2 x0 = unpack_bf16x2(xr.x), x1 = unpack_bf16x2(xr.y), y0 = unpack_bf16x2(yr.x), y1 = unpack_bf16x2(yr.y);
        const float w0 = tile[r][p], w1 = tile[r][p + 1], w2 = tile[r][p + 2], w3 = tile[r][p + 3];
        const float g0 = gv.x + tl * w0, g1 = gv.y + tl * w1, g2 = gv.z + tl * w2, g3 = gv.w + tl * w3;
        *reinterpret_cast<uint2*>(dx + row * P + p) = make_uint2(pack_bf16x2(d * g0 + dn * y0.x, d * g1 + dn * y0.y),
                                                                 pack_bf16x2(d * g2 + dn * y1.x, d * g3 + dn * y1.y));
        // xh as the products saw it
        const float2 h0 = unpack_bf16x2(pack_bf16x2(x0.x * d, x0.y * d)), h1 = unpack_bf16x2(pack_bf16x2(x1.x * d, x1.y * d));
        float s_dt = x0.x * g0 + x0.y * g1 + x1.x * g2 + x1.y * g3;
        float s_w = x0.x * w0 + x0.y * w1 + x1.x * w2 + x1.y * w3;
        float s_h = h0.x * gv.x + h0.y * gv.y + h1.x * gv.z + h1.y * gv.w;
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            s_dt += __shfl_xor_sync(0xffffffffu, s_dt, o);
            s_w += __shfl_xor_sync(0xffffffffu, s_w, o);
            s_h += __shfl_xor_sync(0xffffffffu, s_h, o);
        }
        if (p == 0) {
            ddt0[hrow] = s_dt;
            sw[hrow] = s_w;
            sh[hrow] = s_h;
        }
    }
}

__device__ __forceinline__ void load8f(const float* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// P / 8 lanes per (bc, l, n) row; blockIdx.y = bc * L + l, threads over n and p
template <int P>
__global__ void __launch_bounds__(256)
ssd_combine_kernel(const float* __restrict__ yin, const float* __restrict__ off, const float* __restrict__ ecum,
                   const float* __restrict__ D, const __nv_bfloat16* __restrict__ x, long long xs,
                   __nv_bfloat16* __restrict__ y, int N, int L, int G) {
    const long long tok = blockIdx.x;
    const long long bc = tok / L;
    const int l = static_cast<int>(tok - bc * L), rep = N / G;
    for (int u = threadIdx.x; u < N * (P / 8); u += blockDim.x) {
        const int n = u / (P / 8), p = u % (P / 8) * 8, g = n / rep;
        const float e = ecum[tok * N + n], dn = D[n];
        float a[8], o[8], xv[8];
        load8f(yin + ((bc * N + n) * L + l) * P + p, a);
        load8f(off + ((bc * G + g) * L + l) * static_cast<long long>(rep) * P + (n - g * rep) * P + p, o);
        load8(x + tok * xs + n * P + p, xv);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += o[j] * e + dn * xv[j];
        store8(y + (tok * N + n) * P + p, a);
    }
}

template <int P>
__global__ void __launch_bounds__(256)
ssd_combine_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const float* __restrict__ yin,
                       const float* __restrict__ off, const float* __restrict__ ecum,
                       const __nv_bfloat16* __restrict__ x, long long xs, __nv_bfloat16* __restrict__ dyin,
                       __nv_bfloat16* __restrict__ doff, float* __restrict__ sy, float* __restrict__ decum,
                       float* __restrict__ dDp, int N, int L, int G) {
    constexpr int LANES = P / 8;
    const long long tok = blockIdx.x;
    const long long bc = tok / L;
    const int l = static_cast<int>(tok - bc * L), rep = N / G;
    const int total = N * LANES;
    for (int u0 = 0; u0 < total; u0 += blockDim.x) {       // whole warps stay together for the row sums
        const int u = u0 + threadIdx.x;
        const bool in = u < total;
        const int n = in ? u / LANES : 0, p = u % LANES * 8, g = n / rep;
        const long long row = tok * N + n;
        float s_y = 0.f, s_e = 0.f, s_d = 0.f;
        if (in) {
            const float e = ecum[row];
            const long long o_in = ((bc * N + n) * L + l) * P + p;
            const long long o_off = ((bc * G + g) * L + l) * static_cast<long long>(rep) * P + (n - g * rep) * P + p;
            const uint4 raw = *reinterpret_cast<const uint4*>(dy + row * P + p);
            float gy[8], a[8], o[8], xv[8], w[8];
            unpack8(raw, gy);
            load8f(yin + o_in, a);
            load8f(off + o_off, o);
            load8(x + tok * xs + n * P + p, xv);
            *reinterpret_cast<uint4*>(dyin + o_in) = raw;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                w[j] = gy[j] * e;
                s_y += gy[j] * a[j];
                s_e += gy[j] * o[j];
                s_d += gy[j] * xv[j];
            }
            store8(doff + o_off, w);
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            s_y += __shfl_xor_sync(0xffffffffu, s_y, o);
            s_e += __shfl_xor_sync(0xffffffffu, s_e, o);
            s_d += __shfl_xor_sync(0xffffffffu, s_d, o);
        }
        if (in && u % LANES == 0) {
            sy[row] = s_y;
            decum[row] = s_e;
            dDp[row] = s_d;
        }
    }
}

}  // namespace lme

using namespace lme;

// cb [BC, G, L, L] bf16, cum [BC, N, L] fp32 (inclusive cumulative sums of dt * A inside the chunk) -> m [BC, N, L, L]
extern "C" int lme_ssd_decay_matrix(const void* cb, const float* cum, void* m, long long BC, int N, int G, int L,
                                    void* stream) {
    if (BC <= 0) return LME_OK;
    if (L % 8 || N % G || L > 1024) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(cb) | reinterpret_cast<uintptr_t>(cum) | reinterpret_cast<uintptr_t>(m)) & 15)
        return LME_ERR_ALIGN;
    const long long heads = BC * N;
    if (heads > 0x7fffffffll) return LME_ERR_SHAPE;
    const dim3 grid(static_cast<unsigned>(heads), (L + DECAY_ROWS - 1) / DECAY_ROWS);
    ssd_decay_matrix_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(cb), cum, static_cast<__nv_bfloat16*>(m), N, G, L);
    return LME_LAUNCH_OK();
}

// dm [BC, N, L, L] bf16, cum [BC, N, L] fp32 -> dcb [BC, G, L, L] bf16
extern "C" int lme_ssd_dcb(const void* dm, const float* cum, void* dcb, long long BC, int N, int G, int L,
                           void* stream) {
    if (BC <= 0) return LME_OK;
    if (L % 8 || N % G || L > 1024) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(dm) | reinterpret_cast<uintptr_t>(cum) | reinterpret_cast<uintptr_t>(dcb)) & 15)
        return LME_ERR_ALIGN;
    const long long rows = BC * G * L;
    const unsigned int grid = static_cast<unsigned int>((rows + 7) / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto DM = static_cast<const __nv_bfloat16*>(dm);
    auto DC = static_cast<__nv_bfloat16*>(dcb);
    if (L <= 256) ssd_dcb_kernel<1><<<grid, 256, 0, st>>>(DM, cum, DC, rows, N, G, L);
    else if (L <= 512) ssd_dcb_kernel<2><<<grid, 256, 0, st>>>(DM, cum, DC, rows, N, G, L);
    else ssd_dcb_kernel<4><<<grid, 256, 0, st>>>(DM, cum, DC, rows, N, G, L);
    return LME_LAUNCH_OK();
}

// Decays and scan glue (see the kernels): BC = batch x chunks, L % 32 == 0, L <= 1024, P in {32, 64, 128}, N % G == 0;
// x rows xs elements apart (a multiple of 8).
extern "C" int lme_ssd_decay_fwd(const float* dt, const float* A, float* ct, float* dtt, float* tail, float* ecum,
                                 float* decay, long long BC, int N, int L, void* stream) {
    if (BC <= 0) return LME_OK;
    if (L % 32 || L > 1024 || BC > 0x7fffffffll) return LME_ERR_SHAPE;
    const int smem = L * DECAY_LD * 4;
    ssd_decay_fwd_kernel<<<dim3(static_cast<unsigned>(BC), (N + DECAY_HEADS - 1) / DECAY_HEADS), 256, smem,
                           static_cast<cudaStream_t>(stream)>>>(dt, A, ct, dtt, tail, ecum, decay, N, L);
    return LME_LAUNCH_OK();
}
extern "C" int lme_ssd_decay_bwd(const float* dtt, const float* A, const float* tail, const float* ecum,
                                 const float* decay, const float* sy, const float* decum, const float* ddt0,
                                 const float* sw, const float* sh, const float* ddecay_parts, int parts,
                                 const float* dDp, float* ddt, float* dA_part, float* dD_part, long long BC, int N, int L,
                                 void* stream) {
    if (BC <= 0) return LME_OK;
    if (L % 32 || L > 1024 || BC > 0x7fffffffll) return LME_ERR_SHAPE;
    const int smem = L * DECAY_LD * 4;
    ssd_decay_bwd_kernel<<<dim3(static_cast<unsigned>(BC), (N + DECAY_HEADS - 1) / DECAY_HEADS), 256, smem,
                           static_cast<cudaStream_t>(stream)>>>(dtt, A, tail, ecum, decay, sy, decum, ddt0, sw,
                                                                sh, ddecay_parts, parts, dDp, ddt, dA_part, dD_part, N,
                                                                L);
    return LME_LAUNCH_OK();
}

static int ssd_glue_check(const void* x, long long xs, long long BC, int N, int L, int G, int P) {
    if (L % GLUE_ROWS || L > 1024 || BC > 65535 || N <= 0 || N > 65535 || G <= 0 || N % G || xs % 8 || BC * L > 0x7fffffffll)
        return LME_ERR_SHAPE;
    if (P != 32 && P != 64 && P != 128) return LME_ERR_SHAPE;
    return (reinterpret_cast<uintptr_t>(x) & 15) ? LME_ERR_ALIGN : LME_OK;
}
#define LME_SSD_P(CALL)                                                                                              \
    do {                                                                                                             \
        if (P == 32) { CALL(32); } else if (P == 64) { CALL(64); } else { CALL(128); }                               \
    } while (0)

extern "C" int lme_ssd_prep_fwd(const void* x, long long xs, const float* dt, const float* tail, void* xh, void* xwT,
                                long long BC, int N, int L, int P, void* stream) {
    if (BC <= 0) return LME_OK;
    if (int rc = ssd_glue_check(x, xs, BC, N, L, 1, P)) return rc;
    const dim3 grid(L / GLUE_ROWS, N, static_cast<unsigned>(BC));
#define LME_CALL(PP)                                                                                                 \
    ssd_prep_kernel<PP><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(                                        \
        static_cast<const __nv_bfloat16*>(x), xs, dt, tail, static_cast<__nv_bfloat16*>(xh),                         \
        static_cast<__nv_bfloat16*>(xwT), N, L)
    LME_SSD_P(LME_CALL);
#undef LME_CALL
    return LME_LAUNCH_OK();
}
extern "C" int lme_ssd_prep_bwd(const void* x, long long xs, const float* dt, const float* tail, const float* dxh,
                                const void* dxwT, const void* dy, const float* D, void* dx, float* ddt0, float* sw,
                                float* sh, long long BC, int N, int L, int P, void* stream) {
    if (BC <= 0) return LME_OK;
    if (int rc = ssd_glue_check(x, xs, BC, N, L, 1, P)) return rc;
    const dim3 grid(L / GLUE_ROWS, N, static_cast<unsigned>(BC));
#define LME_CALL(PP)                                                                                                 \
    ssd_prep_bwd_kernel<PP><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(                                    \
        static_cast<const __nv_bfloat16*>(x), xs, dt, tail, dxh, static_cast<const __nv_bfloat16*>(dxwT),            \
        static_cast<const __nv_bfloat16*>(dy), D, static_cast<__nv_bfloat16*>(dx), ddt0, sw, sh, N, L)
    LME_SSD_P(LME_CALL);
#undef LME_CALL
    return LME_LAUNCH_OK();
}
extern "C" int lme_ssd_combine_fwd(const float* yin, const float* off, const float* ecum, const float* D, const void* x,
                                   long long xs, void* y, long long BC, int N, int L, int G, int P, void* stream) {
    if (BC <= 0) return LME_OK;
    if (int rc = ssd_glue_check(x, xs, BC, N, L, G, P)) return rc;
    const unsigned grid = static_cast<unsigned>(BC * L);
#define LME_CALL(PP)                                                                                                 \
    ssd_combine_kernel<PP><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(                                     \
        yin, off, ecum, D, static_cast<const __nv_bfloat16*>(x), xs, static_cast<__nv_bfloat16*>(y), N, L, G)
    LME_SSD_P(LME_CALL);
#undef LME_CALL
    return LME_LAUNCH_OK();
}
extern "C" int lme_ssd_combine_bwd(const void* dy, const float* yin, const float* off, const float* ecum, const void* x,
                                   long long xs, void* dyin, void* doff, float* sy, float* decum, float* dDp,
                                   long long BC, int N, int L, int G, int P, void* stream) {
    if (BC <= 0) return LME_OK;
    if (int rc = ssd_glue_check(x, xs, BC, N, L, G, P)) return rc;
    const unsigned grid = static_cast<unsigned>(BC * L);
#define LME_CALL(PP)                                                                                                 \
    ssd_combine_bwd_kernel<PP><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(                                 \
        static_cast<const __nv_bfloat16*>(dy), yin, off, ecum, static_cast<const __nv_bfloat16*>(x), xs,             \
        static_cast<__nv_bfloat16*>(dyin), static_cast<__nv_bfloat16*>(doff), sy, decum, dDp, N, L, G)
    LME_SSD_P(LME_CALL);
#undef LME_CALL
    return LME_LAUNCH_OK();
}
#undef LME_SSD_P

// ----------------------------------------------------------------------------------------------------------------
// Chunk-boundary recurrence of the SSD scan:  h_0 = h_init,  h_{c+1} = decay[c] * h_c + S_c  per (batch, head), where
// S_c [P * Sd] is the summary of chunk c and decay[c] = exp(sum of dt A over the chunk).  The forward kernel walks the
// chunks once and writes the state at every chunk start (bf16: the operand of the carried-state product; optionally
// fp32 for the backward pass) and the final state; the backward kernel walks them in reverse:
//   dS_c = g,   d decay[c] = <g, h_c>,   g <- decay[c] * g + dh_c        (g starts as d h_final, ends as d h_init)
// 16 chunks x 64 heads x 8192 elements: backward 118 -> 16 us.  A thread owns four state elements for the whole walk: nothing is shared between threads, so the loads of the next
// chunks are in flight while the recurrence advances (a CTA per (batch, head) with a block sum per chunk for d decay
// waited for memory twice per chunk on 64 of 148 SMs).  d decay comes as one partial sum per warp (E / 128 of them per
// row), added up by whoever reads it.
namespace lme {

// E = P * Sd (multiple of 4).  states / h0_f32 / dh0 / dstates: [B, NC, N, E];  decay: [B, NC, N].
__global__ void __launch_bounds__(256)
ssd_boundary_fwd_kernel(const float* __restrict__ states, const float* __restrict__ decay,
                        const float* __restrict__ h_init, __nv_bfloat16* __restrict__ h0_bf16,
                        float* __restrict__ h0_f32, float* __restrict__ h_final, int NC, int N, int E) {
    const int slices = (E / 4 + 255) / 256, bn = blockIdx.x / slices, slice = blockIdx.x - bn * slices;
    const int b = bn / N, n = bn - b * N;
    const int e = (slice * 256 + threadIdx.x) * 4;
    if (e >= E) return;
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
    if (h_init != nullptr) h = *reinterpret_cast<const float4*>(h_init + (static_cast<long long>(b) * N + n) * E + e);
#pragma unroll 4
    for (int c = 0; c < NC; ++c) {
        const long long row = (static_cast<long long>(b) * NC + c) * N + n;
        const long long off = row * E + e;
        const float d = __ldg(decay + row);
        const float4 s = __ldg(reinterpret_cast<const float4*>(states + off));
        uint2 o;
        o.x = pack_bf16x2(h.x, h.y);
        o.y = pack_bf16x2(h.z, h.w);
        *reinterpret_cast<uint2*>(h0_bf16 + off) = o;
        if (h0_f32 != nullptr) *reinterpret_cast<float4*>(h0_f32 + off) = h;
        h.x = h.x * d + s.x; h.y = h.y * d + s.y; h.z = h.z * d + s.z; h.w = h.w * d + s.w;
    }
    *reinterpret_cast<float4*>(h_final + (static_cast<long long>(b) * N + n) * E + e) = h;
}

// dstates in fp32 or bf16 (the operand of the products that read it); ddecay_parts [B, NC, N, parts]
template <typename T>
__global__ void __launch_bounds__(256)
ssd_boundary_bwd_kernel(const float* __restrict__ dh0, const float* __restrict__ dh_final,
                        const float* __restrict__ h0_f32, const float* __restrict__ decay, T* __restrict__ dstates,
                        float* __restrict__ ddecay_parts, int parts, float* __restrict__ dh_init, int NC, int N, int E) {
    const int slices = (E / 4 + 255) / 256, bn = blockIdx.x / slices, slice = blockIdx.x - bn * slices;
    const int b = bn / N, n = bn - b * N;
    const int e = (slice * 256 + threadIdx.x) * 4;
    const int part = (slice * 256 + threadIdx.x) >> 5;
    const bool in = e < E;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in && dh_final != nullptr) g = *reinterpret_cast<const float4*>(dh_final + (static_cast<long long>(b) * N + n) * E + e);
#pragma unroll 4
    for (int c = NC - 1; c >= 0; --c) {
        const long long row = (static_cast<long long>(b) * NC + c) * N + n;
        const long long off = row * E + e;
        const float d = __ldg(decay + row);
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f), a = h;
        if (in) {
            h = __ldg(reinterpret_cast<const float4*>(h0_f32 + off));
            if (dh0 != nullptr) a = __ldg(reinterpret_cast<const float4*>(dh0 + off));
            if constexpr (sizeof(T) == 2) {
                uint2 o;
                o.x = pack_bf16x2(g.x, g.y);
                o.y = pack_bf16x2(g.z, g.w);
                *reinterpret_cast<uint2*>(dstates + off) = o;
            } else {
                *reinterpret_cast<float4*>(dstates + off) = g;
            }
        }
        const float dot = warp_sum(g.x * h.x + g.y * h.y + g.z * h.z + g.w * h.w);
        if ((threadIdx.x & 31) == 0 && part < parts) ddecay_parts[row * parts + part] = dot;
        g.x = g.x * d + a.x; g.y = g.y * d + a.y; g.z = g.z * d + a.z; g.w = g.w * d + a.w;
    }
    if (in && dh_init != nullptr) *reinterpret_cast<float4*>(dh_init + (static_cast<long long>(b) * N + n) * E + e) = g;
}

}  // namespace lme

extern "C" int lme_ssd_boundary_fwd(const float* states, const float* decay, const float* h_init, void* h0_bf16,
                                    float* h0_f32, float* h_final, int B, int NC, int N, int E, void* stream) {
    if (B <= 0 || NC <= 0 || N <= 0 || E <= 0 || (E % 4)) return LME_ERR_SHAPE;
    const long long blocks = static_cast<long long>(B) * N * ((E / 4 + 255) / 256);
    if (blocks > 0x7fffffffll) return LME_ERR_SHAPE;
    lme::ssd_boundary_fwd_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        states, decay, h_init, static_cast<__nv_bfloat16*>(h0_bf16), h0_f32, h_final, NC, N, E);
    return cudaGetLastError() == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}

// ddecay_parts: [B, NC, N, (E + 127) / 128]
extern "C" int lme_ssd_boundary_bwd(const float* dh0, const float* dh_final, const float* h0_f32, const float* decay,
                                    void* dstates, int dstates_bf16, float* ddecay_parts, float* dh_init, int B, int NC,
                                    int N, int E, void* stream) {
    if (B <= 0 || NC <= 0 || N <= 0 || E <= 0 || (E % 4)) return LME_ERR_SHAPE;
    const long long blocks = static_cast<long long>(B) * N * ((E / 4 + 255) / 256);
    if (blocks > 0x7fffffffll) return LME_ERR_SHAPE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned grid = static_cast<unsigned>(blocks);
    const int parts = (E + 127) / 128;
    if (dstates_bf16)
        lme::ssd_boundary_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(
            dh0, dh_final, h0_f32, decay, static_cast<__nv_bfloat16*>(dstates), ddecay_parts, parts, dh_init, NC, N, E);
    else
        lme::ssd_boundary_bwd_kernel<float><<<grid, 256, 0, st>>>(
            dh0, dh_final, h0_f32, decay, static_cast<float*>(dstates), ddecay_parts, parts, dh_init, NC, N, E);
    return cudaGetLastError() == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}
