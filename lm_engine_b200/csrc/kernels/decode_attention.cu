// Attention of ONE new query token per sequence over its key / value cache (generation): grouped query heads, head
// dim 64 or 128, optional sliding window and padding mask.
//
// Bound by reading K and V once.  A CTA of four warps owns a slice of the keys of one (batch, K / V head) and serves
// up to eight query heads of its group from the registers the keys pass through; the slices of one (batch, head)
// form a cluster and merge their softmax partials through distributed shared memory, so there is one launch and no
// workspace.  A warp takes 16 keys per step:
//   scores  mma.sync m16n8k16 with the queries as the 16-row operand (rows 8..15 zero): a lane's 16-byte pieces of a
//           key ARE its B fragment when the contraction index is numbered accordingly (queries use the same order),
//           so keys go from global memory to the tensor core without shared memory, shuffles or conversions;
//   values  the weights stay fp32-exact: p = hi + mid + lo in bf16 (3 x 8 bits of mantissa), hi in rows 0..7, mid in
//           rows 8..15 of one operand, lo in a second product, all accumulated in fp32; the score fragment's layout is
//           the weight operand's, and two keys' 16-byte pieces give the value fragments with one byte permute per
//           register.
// tcgen05 has nothing to add: one row per head is used, and the bound is HBM.
// Measured (24 sequences x 3001 keys, 8 K / V heads of 128, 295 MB): 76 us = 3.9 TB/s (84 us without the loads one block
// ahead); the PyTorch statement that served this case before expands K and V to one fp32 copy per query head and took
// 2640 us.  What is left is latency: 12 warps per SM at 168 registers, a quarter of the issue slots used.
// Included by lme_cuda.cu after m2rnn.cu (mma helper).

namespace lme {
namespace da {

using m2::mma16816;

constexpr int WARPS = 4;
constexpr int MAX_SPLITS = 16;

struct Args {
    const __nv_bfloat16 *q, *k, *v;
    __nv_bfloat16* out;                     // [B, Hkv * G, D] contiguous
    const unsigned char* mask;              // [B, Sk] bytes, 0 = hidden, or null
    long long q_b, q_h, k_b, k_s, k_h, v_b, v_s, v_h, mask_b;   // element strides
    int first, Sk;                          // keys [first, Sk) are attended
    int Hkv, G, head_blocks;                // head_blocks = ceil(G / 8): groups of eight query heads
    float scale;
};

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }
// 0xffff in the halves of a bf16 pair that are infinite or not a number
__device__ __forceinline__ uint32_t not_finite(uint32_t w) {
    return ((w & 0x7f80u) == 0x7f80u ? 0xffffu : 0u) | ((w & 0x7f800000u) == 0x7f800000u ? 0xffff0000u : 0u);
}
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t cta) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int D>
struct Partials {          // of the warps
    float acc[WARPS][8][D];
    float m[WARPS][8], l[WARPS][8];
};

// One warp's share of the keys [k0, k1); returns whether any of its sums is not finite.
// An infinite value times the zero or negative lower terms of its weight is not the infinity that it should be, so a
// warp with such a sum goes over its keys a second time, out of line, where values that are not finite meet the
// leading term alone (!FINITE).
template <int D, bool FINITE>
__device__ __forceinline__ bool attend_keys(const Args& p, Partials<D>& s, int kvh, int hb, long long b, int heads, int k0,
                                            int k1) {
    constexpr int KC = D / 32;    // 16-byte pieces of a key per lane
    constexpr int VC = D / 64;    // 16-byte pieces of a value row per lane
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;

    // query fragments; rows >= heads are zero
    uint32_t qa[D / 16][2];
    {
        const __nv_bfloat16* qp = p.q + b * p.q_b + (static_cast<long long>(kvh) * p.G + hb * 8 + g) * p.q_h + 8 * t;
#pragma unroll
        for (int j = 0; j < KC; ++j) {
            uint4 w = make_uint4(0, 0, 0, 0);
            if (g < heads) w = *reinterpret_cast<const uint4*>(qp + 32 * j);
            qa[2 * j][0] = w.x;
            qa[2 * j][1] = w.y;
            qa[2 * j + 1][0] = w.z;
            qa[2 * j + 1][1] = w.w;
        }
    }
    const __nv_bfloat16* kb = p.k + b * p.k_b + static_cast<long long>(kvh) * p.k_h + 8 * t;
    const __nv_bfloat16* vb = p.v + b * p.v_b + static_cast<long long>(kvh) * p.v_h + 8 * g;
    const unsigned char* mb = p.mask != nullptr ? p.mask + b * p.mask_b : nullptr;

    float acc[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    float m = -INFINITY, l = 0.f;     // row g; l is this lane's share

    // Loads run one block of 16 keys ahead in the registers that the current block frees: the next keys are requested
    // right after the scores, the next values (with their mask) right after the products with the weights.
    uint4 kw[2][KC], vw[4][VC];
    unsigned ok = 0;            // bit e: the lane's e-th key of the block is attended
    auto load_keys = [&](int base) {
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
            const int key = min(base + tile * 8 + g, k1 - 1);
#pragma unroll
            for (int j = 0; j < KC; ++j) kw[tile][j] = ld_stream(kb + key * p.k_s + 32 * j);
        }
    };
    auto load_values = [&](int base) {
        ok = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int key = base + (e >> 1) * 8 + 2 * t + (e & 1);
            bool in = key < k1;
            if (in && mb != nullptr) in = mb[key] != 0;
            ok |= in ? 1u << e : 0u;
#pragma unroll
            for (int j = 0; j < VC; ++j)
                vw[e][j] = in ? ld_stream(vb + key * p.v_s + 64 * j) : make_uint4(0, 0, 0, 0);
        }
    };
    constexpr int STEP = WARPS * 16;
    if (k0 + warp * 16 < k1) {
        load_keys(k0 + warp * 16);
        load_values(k0 + warp * 16);
    }
    for (int base = k0 + warp * 16; base < k1; base += STEP) {
        float sc[2][4];
#pragma unroll
        for (int tile = 0; tile < 2; ++tile) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sc[tile][i] = 0.f;
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                const uint32_t a[4] = {qa[ks][0], 0u, qa[ks][1], 0u};
                mma16816(sc[tile], a, word(kw[tile][ks >> 1], 2 * (ks & 1)), word(kw[tile][ks >> 1], 2 * (ks & 1) + 1));
            }
        }
        if (base + STEP < k1) load_keys(base + STEP);
        float x[4], mx = m;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[e] = (ok >> e & 1) ? sc[e >> 1][e & 1] * p.scale : -INFINITY;
            mx = fmaxf(mx, x[e]);
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if (__any_sync(0xffffffffu, mx > m)) {
            const float c = m == -INFINITY ? 0.f : __expf(m - mx);
            l *= c;
#pragma unroll
            for (int i = 0; i < D / 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] *= c;
            m = mx;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            x[e] = x[e] == -INFINITY ? 0.f : __expf(x[e] - m);
            l += x[e];
        }
        uint32_t hi[2], mid[2], lo[2];
        split3(x[0], x[1], hi[0], mid[0], lo[0]);
        split3(x[2], x[3], hi[1], mid[1], lo[1]);
        const uint32_t a0[4] = {hi[0], mid[0], hi[1], mid[1]}, a1[4] = {lo[0], 0u, lo[1], 0u};
#pragma unroll
        for (int j = 0; j < VC; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
                uint32_t b0 = __byte_perm(word(vw[0][j], i >> 1), word(vw[1][j], i >> 1), sel);
                uint32_t b1 = __byte_perm(word(vw[2][j], i >> 1), word(vw[3][j], i >> 1), sel);
                if (!FINITE) {
                    const uint32_t ah[4] = {hi[0], hi[0], hi[1], hi[1]}, n0 = not_finite(b0), n1 = not_finite(b1);
                    mma16816(acc[j * 8 + i], ah, b0 & n0, b1 & n1);
                    b0 &= ~n0;
                    b1 &= ~n1;
                }
                mma16816(acc[j * 8 + i], a0, b0, b1);
                mma16816(acc[j * 8 + i], a1, b0, b1);
            }
        if (base + STEP < k1) load_values(base + STEP);
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    // accumulator i of piece j: columns 2t, 2t + 1 of the product are dims 64 j + 8 (2t) + i and 64 j + 8 (2t + 1) + i
    float zero = 0.f;
#pragma unroll
    for (int j = 0; j < VC; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float* a = acc[j * 8 + i];
            const float c0 = a[0] + a[2], c1 = a[1] + a[3];
            s.acc[warp][g][64 * j + 16 * t + i] = c0;
            s.acc[warp][g][64 * j + 16 * t + 8 + i] = c1;
            zero += (c0 + c1) * 0.f;
        }
    if (t == 0) {
        s.m[warp][g] = m;
        s.l[warp][g] = l;
    }
    return __any_sync(0xffffffffu, zero != 0.f);
}
template <int D>
__device__ __noinline__ void attend_keys_not_finite(const Args& p, Partials<D>& s, int kvh, int hb, long long b, int heads,
                                                    int k0, int k1) {
    attend_keys<D, false>(p, s, kvh, hb, b, heads, k0, k1);
}

template <int D>
__global__ void __launch_bounds__(WARPS * 32, 3) decode_attention_kernel(const __grid_constant__ Args p) {
    __shared__ Partials<D> part;
    __shared__ float c_acc[8][D];
    __shared__ float c_m[8], c_l[8];
    const int splits = gridDim.x, split = blockIdx.x;
    const int kvh = blockIdx.y / p.head_blocks, hb = blockIdx.y % p.head_blocks;
    const long long b = blockIdx.z;
    const int heads = min(8, p.G - hb * 8);
    const int n = p.Sk - p.first;
    const int per = ((n + splits - 1) / splits + 15) & ~15;
    const int k0 = p.first + min(n, split * per), k1 = p.first + min(n, (split + 1) * per);
    if (attend_keys<D, true>(p, part, kvh, hb, b, heads, k0, k1))
        attend_keys_not_finite<D>(p, part, kvh, hb, b, heads, k0, k1);
    __syncthreads();
    for (int u = threadIdx.x; u < heads * D; u += WARPS * 32) {
        const int r = u / D, d = u % D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) M = fmaxf(M, part.m[w][r]);
        float a = 0.f, ls = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = part.m[w][r] == -INFINITY ? 0.f : __expf(part.m[w][r] - M);
            a += f * part.acc[w][r][d];
            ls += f * part.l[w][r];
        }
        c_acc[r][d] = a;
        if (d == 0) {
            c_m[r] = M;
            c_l[r] = ls;
        }
    }
    cluster_sync();
    for (int u = split * (WARPS * 32) + threadIdx.x; u < heads * D; u += splits * (WARPS * 32)) {
        const int r = u / D, d = u % D;
        float M = -INFINITY;
        for (int c = 0; c < splits; ++c) M = fmaxf(M, ld_cluster(&c_m[r], c));
        float a = 0.f, ls = 0.f;
        for (int c = 0; c < splits; ++c) {
            const float mc = ld_cluster(&c_m[r], c);
            const float f = mc == -INFINITY ? 0.f : __expf(mc - M);
            a += f * ld_cluster(&c_acc[r][d], c);
            ls += f * ld_cluster(&c_l[r], c);
        }
        // a row that attends to nothing, or whose scores are not finite, is zero (as in the PyTorch statement)
        const float o = ls > 0.f && ls < INFINITY ? a / ls : 0.f;
        p.out[(b * p.Hkv * p.G + static_cast<long long>(kvh) * p.G + hb * 8 + r) * D + d] = __float2bfloat16_rn(o);
    }
    cluster_sync();   // the others may still read this CTA's partials
}

template <int D>
static int launch_decode_attention(const Args& a, int B, int splits, cudaStream_t st) {
    auto kern = decode_attention_kernel<D>;
    if (!opt_in<decode_attention_kernel<D>>(cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) return LME_ERR_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, a.Hkv * a.head_blocks, B);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess ? LME_OK : LME_ERR_LAUNCH;
}

}  // namespace da
}  // namespace lme

extern "C" int lme_decode_attention(const void* q, long long q_b, long long q_h, const void* k, long long k_b,
                                    long long k_s, long long k_h, const void* v, long long v_b, long long v_s,
                                    long long v_h, const void* mask, long long mask_b, void* out, int B, int Sk,
                                    int Hkv, int G, int D, int window, float scale, void* stream) {
    if (B <= 0 || Hkv <= 0 || G <= 0) return LME_OK;
    if (Sk <= 0 || window <= 0 || (D != 64 && D != 128)) return LME_ERR_SHAPE;
    if ((q_b | q_h | k_b | k_s | k_h | v_b | v_s | v_h) % 8) return LME_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)
        return LME_ERR_ALIGN;
    lme::da::Args a = {};
    a.q = static_cast<const __nv_bfloat16*>(q);
    a.k = static_cast<const __nv_bfloat16*>(k);
    a.v = static_cast<const __nv_bfloat16*>(v);
    a.out = static_cast<__nv_bfloat16*>(out);
    a.mask = static_cast<const unsigned char*>(mask);
    a.q_b = q_b; a.q_h = q_h;
    a.k_b = k_b; a.k_s = k_s; a.k_h = k_h;
    a.v_b = v_b; a.v_s = v_s; a.v_h = v_h;
    a.mask_b = mask_b;
    a.first = Sk > window ? Sk - window : 0;
    a.Sk = Sk;
    a.Hkv = Hkv;
    a.G = G;
    a.head_blocks = (G + 7) / 8;
    a.scale = scale;
    if (B > 65535 || static_cast<long long>(Hkv) * a.head_blocks > 65535) return LME_ERR_SHAPE;
    // The keys are split until there is a CTA for every slot of the chip (three fit an SM), and no further once a slice is
    // down to the 64 keys that the four warps take in one step: a slice costs a prologue and a merge of about 4 us.  Slices
    // therefore keep more than 32 keys (48 with the rounding to blocks of 16); the last ones get what is left, or nothing.
    const long long rows = static_cast<long long>(B) * Hkv * a.head_blocks;
    int splits = 1;
    while (splits < lme::da::MAX_SPLITS && rows * splits < 3 * 148 && (Sk - a.first) > splits * 64) splits *= 2;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return D == 64 ? lme::da::launch_decode_attention<64>(a, B, splits, st)
                   : lme::da::launch_decode_attention<128>(a, B, splits, st);
}
