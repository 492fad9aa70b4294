// grad_input of the QuantizedLinear backward pass: grad_in[M,K] = grad_out[M,N] . W[N,K],
// W = GradT( scale * (code - zero_point) ) evaluated in fp32 and cast to the gradient dtype.
//
// Replaces the eager unpack loop + fp32 dequantize + matmul of
// QuantizedLinearFunction.backward (bitween/modules.py:108-141) without materialising W.
// Each thread owns one packed word column (32/bits consecutive k) for a block of up to 8
// tokens and walks down the rows, so packed words are read coalesced across the warp and
// each is expanded once per token block.  That CUDA-core kernel serves fp32 gradients and
// layouts the tensor-core kernel below cannot take.
//
// fp16 / bf16 gradients (what LoRA fine-tuning and mixed-precision retraining produce) run on the
// tcgen05 kernel at the end of this file where TMA can stride over their layout, else on an
// mma.sync kernel: a CTA owns 128 tokens x 64 k of grad_in and walks over N in steps of 64 rows;
// each step the CTA expands the [64 rows x 64 k] block of W ONCE (exactly GradT(scale * (code -
// zp)), fp32 arithmetic, one rounding) into shared memory, transposed and padded so that the
// mma.sync B fragments are conflict-free 32-bit loads, while the eight warps multiply the
// previous block: mma.sync.m16n8k16 with grad_out as the row-major A operand, fp32 accumulators.
#include <cooperative_groups.h>
#include <cuda.h>

#include "bw_common.cuh"
#include "qmm_dequant.cuh"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace cgx = cooperative_groups;

namespace bw {
namespace {

constexpr int TOK = 8;

template <int BITS, typename GT>
__global__ void __launch_bounds__(128)
grad_input_kernel(const GT *__restrict__ go, int64_t M, int64_t N, int64_t K,
                  const int32_t *__restrict__ q, const __half *__restrict__ scale,
                  const __half *__restrict__ zp, GT *__restrict__ gi, int g, int words_per_row,
                  int64_t G) {
    constexpr int VPI = 32 / BITS;
    constexpr int32_t MASK = (1 << BITS) - 1;
    const int wi = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m0 = (int64_t)blockIdx.y * TOK;
    if (wi >= words_per_row) return;
    float acc[TOK][VPI];
#pragma unroll
    for (int j = 0; j < TOK; ++j)
#pragma unroll
        for (int i = 0; i < VPI; ++i) acc[j][i] = 0.0f;
    const bool one_group = (g % VPI) == 0;
    for (int64_t n = 0; n < N; ++n) {
        const int32_t word = q[n * words_per_row + wi];
        float wv[VPI];
        if (one_group) {
            const int64_t gidx = n * G + ((int64_t)wi * VPI) / g;
            const float s = __half2float(scale[gidx]), z = __half2float(zp[gidx]);
#pragma unroll
            for (int i = 0; i < VPI; ++i)
                wv[i] = to_f32<GT>(from_f32<GT>(__fmul_rn(s, __fsub_rn((float)((word >> (i * BITS)) & MASK), z))));
        } else {
#pragma unroll
            for (int i = 0; i < VPI; ++i) {
                const int64_t gidx = n * G + ((int64_t)wi * VPI + i) / g;
                const float s = __half2float(scale[gidx]), z = __half2float(zp[gidx]);
                wv[i] = to_f32<GT>(from_f32<GT>(__fmul_rn(s, __fsub_rn((float)((word >> (i * BITS)) & MASK), z))));
            }
        }
#pragma unroll
        for (int j = 0; j < TOK; ++j) {
            if (m0 + j < M) {
                const float gv = to_f32<GT>(go[(m0 + j) * N + n]);
#pragma unroll
                for (int i = 0; i < VPI; ++i) acc[j][i] = fmaf(gv, wv[i], acc[j][i]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < TOK; ++j) {
        if (m0 + j < M) {
#pragma unroll
            for (int i = 0; i < VPI; ++i) gi[(m0 + j) * K + (int64_t)wi * VPI + i] = from_f32<GT>(acc[j][i]);
        }
    }
}

// ---- tensor-core kernel --------------------------------------------------------------------
constexpr int GI_BM = 128, GI_BK = 64, GI_BN = 64;   // tokens x k per CTA, weight rows per step
constexpr int GI_PITCH = GI_BN + 8;                  // elements between k columns of the expanded block: conflict-free
                                                     // 32-bit fragment loads (36 words: 8 columns land on banks 0,4,...,28)

template <typename GT> __device__ __forceinline__ void mma_grad(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma_grad<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma_grad<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Each step the CTA expands the [64 rows x 64 k] block of W once into shared memory (transposed,
// [k][row]) while the eight warps multiply the previous block; the packed words, their scales and
// zero points and the grad_out fragments of the NEXT step are already in registers by then, so
// the global-memory latency hides behind the 32 MMAs of a step.
template <int BITS, typename GT>
__global__ void __launch_bounds__(256)
grad_input_tc_kernel(const GT *__restrict__ go, int64_t M, int64_t N, int64_t K, const int32_t *__restrict__ q,
                     const __half *__restrict__ scale, const __half *__restrict__ zp, GT *__restrict__ gi, int g,
                     int words_per_row, int64_t G) {
    constexpr int VPI = 32 / BITS;
    constexpr int32_t MASK = (1 << BITS) - 1;
    constexpr int WPB = GI_BK / VPI;                       // packed words per row of the block: 16 / 8 / 4
    constexpr int WPT = GI_BN * WPB / 256;                 // words per thread and step: 4 / 2 / 1
    __shared__ __align__(16) GT wt[2][GI_BK * GI_PITCH];   // [buffer][k][row] expanded weights
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t = lane & 3;
    const int64_t k0 = (int64_t)blockIdx.x * GI_BK, m0 = (int64_t)blockIdx.y * GI_BM + warp * 16;
    const bool one_group = (g % VPI) == 0;                 // a packed word lies in one quantization group
    float acc[GI_BK / 8][4];
#pragma unroll
    for (int j = 0; j < GI_BK / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.0f;

    // registers holding the next step's global data
    int32_t words[WPT];
    float sv[WPT], zv[WPT];
    uint32_t a_next[GI_BN / 16][4];
    auto fetch = [&](int64_t n0) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int w = tid + u * 256, er = w % GI_BN, ew = w / GI_BN;   // rows vary fastest: conflict-free stores below
            const int64_t n = n0 + er, kw = k0 + (int64_t)ew * VPI;
            words[u] = 0; sv[u] = 0.0f; zv[u] = 0.0f;
            if (n < N && kw < K) {
                words[u] = __ldg(q + n * words_per_row + kw / VPI);
                const int64_t gidx = n * G + kw / g;
                sv[u] = __half2float(__ldg(scale + gidx));
                zv[u] = __half2float(__ldg(zp + gidx));
            }
        }
#pragma unroll
        for (int sub = 0; sub < GI_BN / 16; ++sub)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int64_t m = m0 + gq + (e & 1) * 8, n = n0 + sub * 16 + 2 * t + (e >> 1) * 8;
                a_next[sub][e] = (m < M && n < N) ? __ldg(reinterpret_cast<const unsigned int *>(go + m * N + n)) : 0u;
            }
    };
    auto expand = [&](int64_t n0, int buf) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int w = tid + u * 256, er = w % GI_BN, ew = w / GI_BN;
            const int64_t n = n0 + er, kw = k0 + (int64_t)ew * VPI;
            GT *dst = wt[buf] + (size_t)(ew * VPI) * GI_PITCH + er;
            const bool live = n < N && kw < K;
#pragma unroll
            for (int i = 0; i < VPI; ++i) {
                float s1 = sv[u], z1 = zv[u];
                if (!one_group && live) {
                    const int64_t gidx = n * G + (kw + i) / g;
                    s1 = __half2float(__ldg(scale + gidx));
                    z1 = __half2float(__ldg(zp + gidx));
                }
                const float wv = live ? __fmul_rn(s1, __fsub_rn((float)((words[u] >> (i * BITS)) & MASK), z1)) : 0.0f;
                dst[(size_t)i * GI_PITCH] = from_f32<GT>(wv);
            }
        }
    };
    const int64_t steps = (N + GI_BN - 1) / GI_BN;
    fetch(0);
    expand(0, 0);
    uint32_t a_cur[GI_BN / 16][4];
#pragma unroll
    for (int sub = 0; sub < GI_BN / 16; ++sub)
#pragma unroll
        for (int e = 0; e < 4; ++e) a_cur[sub][e] = a_next[sub][e];
    __syncthreads();
    for (int64_t st = 0; st < steps; ++st) {
        const int buf = (int)(st & 1);
        if (st + 1 < steps) fetch((st + 1) * GI_BN);              // in flight during the MMAs below
        const GT *wb = wt[buf];
#pragma unroll
        for (int sub = 0; sub < GI_BN / 16; ++sub)
#pragma unroll
            for (int j = 0; j < GI_BK / 8; ++j) {
                const GT *col = wb + (size_t)(j * 8 + gq) * GI_PITCH + sub * 16 + 2 * t;
                mma_grad<GT>(acc[j], a_cur[sub], *reinterpret_cast<const uint32_t *>(col), *reinterpret_cast<const uint32_t *>(col + 8));
            }
        if (st + 1 < steps) {
            expand((st + 1) * GI_BN, buf ^ 1);
#pragma unroll
            for (int sub = 0; sub < GI_BN / 16; ++sub)
#pragma unroll
                for (int e = 0; e < 4; ++e) a_cur[sub][e] = a_next[sub][e];
        }
        __syncthreads();
    }
    // C fragment: rows m0+gq / +8, columns k0 + 8j + 2t, +1
#pragma unroll
    for (int j = 0; j < GI_BK / 8; ++j) {
        const int64_t k = k0 + j * 8 + 2 * t;
        if (k >= K) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t m = m0 + gq + h * 8;
            if (m >= M) continue;
            GT pair[2] = {from_f32<GT>(acc[j][2 * h]), from_f32<GT>(acc[j][2 * h + 1])};
            *reinterpret_cast<uint32_t *>(gi + m * K + k) = *reinterpret_cast<const uint32_t *>(pair);
        }
    }
}

template <int BITS, typename GT>
int launch_tc(const void *go, int64_t M, int64_t N, int64_t K, const int32_t *q, const __half *scale,
              const __half *zp, void *gi, int g, cudaStream_t st) {
    const int64_t kblocks = (K + GI_BK - 1) / GI_BK, mblocks = (M + GI_BM - 1) / GI_BM;
    if (kblocks > 0x7fffffff || mblocks > 65535) return BW_ERR_SHAPE;
    dim3 grid((unsigned)kblocks, (unsigned)mblocks, 1);
    grad_input_tc_kernel<BITS, GT><<<grid, 256, 0, st>>>((const GT *)go, M, N, K, q, scale, zp, (GT *)gi, g,
                                                         (int)(K / (32 / BITS)), K / g);
    return check_launch("grad_input_tc_kernel");
}

// 16-bit gradients whose rows allow 32-bit accesses at even columns run on the tensor cores.
inline bool grad_tc_ok(const void *go, const void *gi, int dt, int64_t N, int64_t K) {
    return (dt == BW_F16 || dt == BW_BF16) && N % 2 == 0 && K % 2 == 0 && aligned_to(go, 4) && aligned_to(gi, 4);
}

// ---- tcgen05 kernel ------------------------------------------------------------------------
// 16-bit gradients whose layout TMA can stride over.  The product is formed transposed, as in the
// forward GEMM: the MMA's M dimension holds 128 k columns (one TMEM lane each), its N dimension up
// to 256 tokens, and the reduction walks over the weight rows n in stages of 64:
//     D^T[k, m] += W^T[k, n] . go[m, n].
// The expanded weights keep the order in which packed words hold them -- 64 consecutive k of one
// row n are 128 contiguous bytes -- which is the MN-major form of the A operand, so nothing is
// transposed: each dequantization thread expands 64 codes of one row and writes eight 16-byte
// chunks into the 128-byte-swizzled shared-memory tile.  (The forward keeps A in tensor memory;
// here a TMEM lane would need one code from each of 64 different words.)  Tensor memory holds only
// accumulators, two of them, so the output stage of a tile runs beside the MMAs of the next one.
//
// Warps: 0 TMA producer of grad_out tiles, 1 MMA issuer, 2 TMA producer of the packed words with
// their scales and zero points, 3 allocates tensor memory, 4-7 output stage, 8-23 four groups of
// dequantization threads (group g expands stages g, g+4, ...).  Persistent: one CTA per SM walks the
// tile list; when there are fewer tiles than SMs, the CTAs of a cluster split the rows n and add
// their partial tiles through distributed shared memory.
//
// Bound: per stage a CTA moves ~104 KB through shared memory (32 KB of grad_out in and read again,
// 16 KB of weights written and read, packed words) against 512 cycles of MMAs, so shared-memory
// bandwidth, not the tensor pipe, sets the pace of 256-token tiles.  Measured: forward and backward of a
// Llama-3-8B block's seven linears at 2048 tokens (W4 g128, 1.8 TFLOP, half of it here) 11.6 ms with the
// mma.sync kernel above (which re-expands the weights for every 128 tokens and multiplies at 80 TFLOP/s),
// 1.76 ms with this one.
constexpr int GU_BK = 128;          // k columns per tile (MMA M)
constexpr int GU_BN = 64;           // weight rows per stage (reduction)
constexpr int GU_AS = 4;            // stages of expanded weights == dequantization groups
constexpr int GU_GROUPS = 4;
constexpr int GU_WS = 4;            // slots of packed words
constexpr int GU_THREADS = 24 * 32;
constexpr int GU_A_BYTES = GU_BK * GU_BN * 2;
constexpr int GU_C_BYTES = GU_BN * 16;             // scales (or zero points) of a stage: 64 rows x 8 groups
constexpr int GU_O_BYTES = 32 * GU_BK * 2;         // output staging: 32 tokens x 128 k
// (reduced sums, one accumulator per split) and the ring depths below rely on these
static_assert(GU_AS >= GU_GROUPS && GU_WS == GU_GROUPS, "a group always uses one word slot; parity waits never lag two phases");

__device__ int g_grad_status = 0;

using namespace umma;
__device__ __forceinline__ bool gu_wait(uint64_t *bar, unsigned parity, volatile int *abort_flag, int code) {
    return umma::mbar_wait(bar, parity, abort_flag, code, &g_grad_status);
}

// Named barrier 1 over the output stage's 128 threads; true if `ok` holds on all of them.
__device__ __forceinline__ bool gu_all_128(bool ok) {
    unsigned r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, 128, p;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r) : "r"((unsigned)ok) : "memory");
    return r != 0;
}

struct GuParams {
    const __half *scale, *zp;
    void *gi;
    int64_t M, N, K;
    int g_shift, G;
    int bn;                 // tokens per tile
    int x_stages;           // ring of grad_out tiles
    int steps;              // ceil(N / 64)
    int splits, per_split;  // cluster size along z, steps per CTA of it
    int k_tiles, tiles;
    int const_tma;          // 1: scales / zero points arrive with the packed words
};

// 64 codes of one row -> 64 16-bit weights GradT(scale * (code - zp)), as eight 16-byte chunks.
// The expression is evaluated in fp32 and rounded once (modules.py:131-139); 2^23 + code is built by
// inserting the code into the significand, so the difference to 2^23 is the exact code.
template <int BITS, typename GT>
__device__ __forceinline__ uint32_t gu_pair(uint32_t word, int i, float s, float z) {
    constexpr uint32_t MASK = (1u << BITS) - 1u;
    const float c0 = __uint_as_float(lop3_and_or(word >> (i * BITS), MASK, 0x4B000000u)) - 8388608.0f;
    const float c1 = __uint_as_float(lop3_and_or(word >> ((i + 1) * BITS), MASK, 0x4B000000u)) - 8388608.0f;
    const float w0 = __fmul_rn(s, __fsub_rn(c0, z)), w1 = __fmul_rn(s, __fsub_rn(c1, z));
    if constexpr (sizeof(GT) == 2 && __is_same(GT, __half)) return h2_as_u32(__floats2half2_rn(w0, w1));
    else {
        const __nv_bfloat162 b = __floats2bfloat162_rn(w0, w1);
        return *reinterpret_cast<const uint32_t *>(&b);
    }
}
// The fp16 form on packed pairs: the same bits when the zero point is an integer of at most 1024
// (1024 + code - (1024 + zp) is exact and one rounding follows, in the product).
template <int BITS>
__device__ __forceinline__ void gu_word_h2(const Dequant<BITS> &dq, uint32_t w, uint32_t (&r)[16 / BITS]) {
    uint32_t p[16 / BITS];
    dq.run(w, p);
    constexpr int H = 16 / BITS;           // p[j] = (c_j, c_{j+H})
#pragma unroll
    for (int j = 0; j < H; j += 2) {
        r[j / 2] = pair_lo(p[j], p[j + 1]);
        r[H / 2 + j / 2] = pair_hi(p[j], p[j + 1]);
    }
}

// A thread's 64 codes (one row, `w`) -> eight 16-byte chunks of its 128-byte row of the A tile, swizzled.
// FAST: packed fp16 arithmetic; ONE: all 64 codes lie in one quantization group.
template <int BITS, typename GT, bool FAST, bool ONE>
__device__ __forceinline__ void gu_expand(const uint32_t (&w)[2 * BITS], const uint32_t (&sz)[4], int g_shift, unsigned char *dst, int swz) {
    constexpr int VPI = 32 / BITS, PPW = 16 / BITS;        // codes, pairs per word
    Dequant<BITS> dq;
    float s = 0.0f, z = 0.0f;
    auto set = [&](uint32_t c) {
        if constexpr (FAST) {
            GroupConst gc;
            gc.s2 = __byte_perm(c, 0, 0x1010);
            gc.z1024 = h2_as_u32(__hadd2(u32_as_h2(__byte_perm(c, 0, 0x3232)), __float2half2_rn(1024.0f)));
            dq.set(gc);
        } else {
            s = __half2float(__ushort_as_half((unsigned short)(c & 0xffffu)));
            z = __half2float(__ushort_as_half((unsigned short)(c >> 16)));
        }
    };
    if constexpr (ONE) set(sz[0]);
    int cur = -1;
    uint32_t q[PPW < 4 ? 4 : PPW];                          // at least one chunk
#pragma unroll
    for (int j = 0; j < 2 * BITS; ++j) {
        if constexpr (!ONE) {
            const int gl = (j * VPI) >> g_shift;
            if (gl != cur) { set(gl == 0 ? sz[0] : gl == 1 ? sz[1] : gl == 2 ? sz[2] : sz[3]); cur = gl; }
        }
        const int q0 = PPW < 4 ? (j & 1) * PPW : 0;
        if constexpr (FAST) {
            uint32_t t[PPW];
            gu_word_h2<BITS>(dq, w[j], t);
#pragma unroll
            for (int e = 0; e < PPW; ++e) q[q0 + e] = t[e];
        } else {
#pragma unroll
            for (int e = 0; e < PPW; ++e) q[q0 + e] = gu_pair<BITS, GT>(w[j], 2 * e, s, z);
        }
        if (PPW >= 4 || (j & 1)) {
            const int c0 = PPW >= 4 ? j * (PPW / 4) : j / 2;
#pragma unroll
            for (int c = 0; c < (PPW < 4 ? 1 : PPW / 4); ++c)
                *reinterpret_cast<uint4 *>(dst + (((c0 + c) ^ swz) << 4)) = make_uint4(q[4 * c], q[4 * c + 1], q[4 * c + 2], q[4 * c + 3]);
        }
    }
}

template <int BITS, typename GT>
__global__ void __launch_bounds__(GU_THREADS, 1)
grad_input_umma_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map,
                       const __grid_constant__ CUtensorMap s_map, const __grid_constant__ CUtensorMap z_map,
                       const __grid_constant__ CUtensorMap out_map, const GuParams p) {
    constexpr int VPI = 32 / BITS;
    constexpr int ROW_BYTES = GU_BK * BITS / 8;                  // packed bytes of a row in a tile: 32 / 64 / 128
    constexpr int W_BYTES = GU_BN * ROW_BYTES;
    constexpr int SLOT = W_BYTES + 2 * GU_C_BYTES;
    constexpr int SWZ_SHIFT = BITS == 8 ? 0 : (BITS == 4 ? 1 : 2), SWZ_MASK = ROW_BYTES / 16 - 1;
    constexpr int VECS = 64 / VPI / 4;                           // 16-byte vectors of packed words per thread: 1 / 2 / 4
    constexpr int WPT = 64 / VPI;                                // words per thread
    extern __shared__ unsigned char gu_smem[];
    unsigned char *smem = gu_smem + ((1024u - (smem_addr(gu_smem) & 1023u)) & 1023u);
    const int bn = p.bn, NSX = p.x_stages;
    unsigned char *a_tiles = smem;                                           // [GU_AS][2 halves][64 n][128 B]
    unsigned char *x_tiles = a_tiles + GU_AS * GU_A_BYTES;                   // [NSX][bn][128 B]
    unsigned char *w_slots = x_tiles + (size_t)NSX * bn * 128;               // [GU_WS][words | scales | zero points]
    unsigned char *o_stage = w_slots + GU_WS * SLOT;
    uint64_t *bars = reinterpret_cast<uint64_t *>(o_stage + GU_O_BYTES);
    uint64_t *a_full = bars, *a_empty = bars + GU_AS, *w_full = a_empty + GU_AS, *w_empty = w_full + GU_WS;
    uint64_t *x_full = w_empty + GU_WS, *acc_full = x_full + GU_AS, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    // (Broadcast, so that the compiler knows the roles' branches, loops and addresses to be warp-uniform: the
    // operands of tcgen05 and mbarrier instructions then stay in uniform registers: 908 -> 740 us for the
    // seven linears of a Llama-3-8B block at 2048 tokens.)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int st0 = blockIdx.z * p.per_split;
    const int nk = max(min(st0 + p.per_split, p.steps) - st0, 0);            // stages of this CTA per tile
    const int first_tile = (int)blockIdx.x, tile_step = (int)gridDim.x;
    const uint32_t acc_cols = bn < 32 ? 32u : (uint32_t)bn;
    const uint32_t tmem_cols = 2 * acc_cols;                                 // a power of two, 64 .. 512

    if (tid == 0) {
        for (int s = 0; s < GU_AS; ++s) { mbar_init(&a_full[s], 4); mbar_init(&a_empty[s], 1); mbar_init(&x_full[s], 1); }
        for (int s = 0; s < GU_WS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 4); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async_smem();
    }
    if (warp == 3) tmem_alloc(tmem_slot, tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 0) {
        // ---- TMA producer of grad_out tiles [bn tokens x 64 n] ----
        if (lane == 0) {
            int sx = 0, gx = 0;
            bool alive = true;
            for (int t = first_tile; t < p.tiles && alive; t += tile_step) {
                const int m0 = (t / p.k_tiles) * bn;
                for (int i = 0; i < nk; ++i, ++gx) {
                    const int jf = gx - NSX;      // its MMAs also free the slot (NSX <= GU_AS)
                    if (jf >= 0 && !gu_wait(&a_empty[jf % GU_AS], (unsigned)(jf / GU_AS) & 1u, abort_flag, 1)) { alive = false; break; }
                    mbar_expect_tx(&x_full[sx], (unsigned)bn * 128u);
                    tma_load_2d(x_tiles + (size_t)sx * bn * 128, &x_map, (st0 + i) * GU_BN, m0, &x_full[sx]);
                    if (++sx == NSX) sx = 0;
                }
            }
        }
    } else if (warp == 2) {
        // ---- TMA producer of packed words, scales, zero points of [64 n x 128 k] ----
        if (lane == 0) {
            int gw = 0;
            bool alive = true;
            for (int t = first_tile; t < p.tiles && alive; t += tile_step) {
                const int kt = t % p.k_tiles;
                const int grp0 = ((kt * GU_BK) >> p.g_shift) & ~7;           // boxes start on 16-byte boundaries
                for (int i = 0; i < nk; ++i, ++gw) {
                    const int sw = gw % GU_WS;
                    if (!gu_wait(&w_empty[sw], ((unsigned)(gw / GU_WS) & 1u) ^ 1u, abort_flag, 2)) { alive = false; break; }
                    unsigned char *slot = w_slots + (size_t)sw * SLOT;
                    mbar_expect_tx(&w_full[sw], (unsigned)(W_BYTES + (p.const_tma ? 2 * GU_C_BYTES : 0)));
                    tma_load_2d(slot, &w_map, kt * (GU_BK / VPI), (st0 + i) * GU_BN, &w_full[sw]);
                    if (p.const_tma) {
                        tma_load_2d(slot + W_BYTES, &s_map, grp0, (st0 + i) * GU_BN, &w_full[sw]);
                        tma_load_2d(slot + W_BYTES + GU_C_BYTES, &z_map, grp0, (st0 + i) * GU_BN, &w_full[sw]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer (the whole warp runs the loop, one elected lane issues) ----
        const uint32_t idesc = umma_idesc_f16(bn, !__is_same(GT, __half), true);
        bool ok = true;
        int sx = 0, gi = 0, it = 0;
        unsigned phx = 0;
        for (int t = first_tile; t < p.tiles && ok; t += tile_step, ++it) {
            const uint32_t acc = tmem_base + (uint32_t)(it & 1) * acc_cols;
            // the output stage has read this accumulator's previous tile (passes at once the first time round)
            ok = __all_sync(0xffffffffu, gu_wait(&acc_empty[it & 1], ((unsigned)(it >> 1) & 1u) ^ 1u, abort_flag, 3));
            if (!ok) break;
            tc_fence_after();
            for (int i = 0; i < nk; ++i, ++gi) {
                const int sa = gi % GU_AS;
                const bool got = gu_wait(&x_full[sx], phx, abort_flag, 4) &&
                                 gu_wait(&a_full[sa], (unsigned)(gi / GU_AS) & 1u, abort_flag, 5);
                ok = __all_sync(0xffffffffu, got);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_addr = smem_addr(a_tiles + (size_t)sa * GU_A_BYTES);
                const uint32_t b_addr = smem_addr(x_tiles + (size_t)sx * bn * 128);
#pragma unroll
                for (int k4 = 0; k4 < GU_BN / 16; ++k4)
                    umma_f16_ss(acc, umma_smem_desc_mn(a_addr + k4 * 2048, GU_BN * 128), umma_smem_desc(b_addr + k4 * 32), idesc,
                                (i | k4) != 0 ? 1u : 0u);
                umma_commit(&a_empty[sa]);
                if (++sx == NSX) { sx = 0; phx ^= 1u; }
            }
            if (ok) umma_commit(&acc_full[it & 1]);
        }
    } else if (warp >= 8) {
        // ---- dequantization: this thread expands 64 codes of one row of its group's stages ----
        const int grp = (warp - 8) >> 2, tg = tid & 127;
        const int row = tg & 63, half = tg >> 6;
        const int gps = max(1, 64 >> p.g_shift);                             // quantization groups per thread and stage
        const int swz = (row >> SWZ_SHIFT) & SWZ_MASK;
        bool ok = true;
        int gbase = 0;
        for (int t = first_tile; t < p.tiles && ok; t += tile_step, gbase += nk) {
            const int kt = t % p.k_tiles;
            const int grp_first = (kt * GU_BK + half * 64) >> p.g_shift;     // first group of this thread's 64 codes
            for (int i = (grp - gbase) & (GU_GROUPS - 1); i < nk; i += GU_GROUPS) {
                const int gi = gbase + i, sa = gi % GU_AS, sw = gi % GU_WS;
                const unsigned ph = (unsigned)(gi / GU_WS) & 1u;
                uint32_t sz[4];                              // scale | zero point << 16 of the thread's groups
                if (!p.const_tma) {
                    const int64_t n = (int64_t)(st0 + i) * GU_BN + row;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool live = j < gps && n < p.N && grp_first + j < p.G;
                        sz[j] = 0;
                        if (live) sz[j] = (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(p.scale) + n * p.G + grp_first + j) |
                                          (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(p.zp) + n * p.G + grp_first + j) << 16;
                    }
                }
                ok = __all_sync(0xffffffffu, gu_wait(&w_full[sw], ph, abort_flag, 6));
                if (!ok) break;
                const unsigned char *slot = w_slots + (size_t)sw * SLOT;
                uint32_t w[WPT];
#pragma unroll
                for (int v = 0; v < VECS; ++v) {
                    const uint4 tq = *reinterpret_cast<const uint4 *>(slot + (size_t)row * ROW_BYTES + (((half * VECS + v) ^ swz) << 4));
                    w[4 * v] = tq.x; w[4 * v + 1] = tq.y; w[4 * v + 2] = tq.z; w[4 * v + 3] = tq.w;
                }
                if (p.const_tma) {
                    const unsigned short *cs = reinterpret_cast<const unsigned short *>(slot + W_BYTES) + row * 8;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (j < gps) {
                            const int o = (grp_first + j) & 7;
                            sz[j] = (uint32_t)cs[o] | (uint32_t)cs[o + GU_C_BYTES / 2] << 16;
                        } else {
                            sz[j] = 0;
                        }
                    }
                }
                fence_proxy_async_smem();                    // reads of the slot before its refill by TMA
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_empty[sw]);
                ok = __all_sync(0xffffffffu, gu_wait(&a_empty[sa], ((unsigned)(gi / GU_AS) & 1u) ^ 1u, abort_flag, 7));
                if (!ok) break;
                unsigned char *dst = a_tiles + (size_t)sa * GU_A_BYTES + (size_t)half * (GU_BN * 128) + (size_t)row * 128;
                bool fast = __is_same(GT, __half);
                if (fast) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float zf = __half2float(__ushort_as_half((unsigned short)(sz[j] >> 16)));
                        fast = fast && (j >= gps || (zf == rintf(zf) && fabsf(zf) <= 1024.0f));
                    }
                }
                if (!fast) gu_expand<BITS, GT, false, false>(w, sz, p.g_shift, dst, row & 7);
                else if (gps == 1) gu_expand<BITS, GT, true, true>(w, sz, p.g_shift, dst, row & 7);
                else gu_expand<BITS, GT, true, false>(w, sz, p.g_shift, dst, row & 7);
                fence_proxy_async_smem();                    // generic-proxy writes before the MMAs read them
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[sa]);
            }
        }
    } else if (warp >= 4) {
        // ---- output stage: 32 tokens at a time, fp32 -> GradT, staged and stored by TMA ----
        const int quad = warp & 3, row = quad * 32 + lane;
        const bool issuer = tid == 4 * 32;
        const int nblk = bn < 32 ? 1 : bn / 32;
        int it = 0;
        for (int t = first_tile; t < p.tiles; t += tile_step, ++it) {
            // the four warps agree on whether the wait succeeded: they meet at named barriers below
            const bool done = __all_sync(0xffffffffu, gu_wait(&acc_full[it & 1], (unsigned)(it >> 1) & 1u, abort_flag, 8));
            if (!gu_all_128(done)) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(it & 1) * acc_cols;
            const int k0 = (t % p.k_tiles) * GU_BK, m0 = (t / p.k_tiles) * bn;
            for (int cb = 0; cb < nblk; ++cb) {
                uint32_t r[32];
                tmem_ld_32x32b_x32(acc + (uint32_t)(cb * 32), r);
                if (cb == nblk - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[it & 1]);
                }
                if (p.splits > 1) {
                    // park the partial tile in the idle rings as red[token][k]; the cluster adds it below
                    float *red = reinterpret_cast<float *>(a_tiles);
#pragma unroll
                    for (int j = 0; j < 32; ++j) red[(cb * 32 + j) * GU_BK + row] = nk > 0 ? __uint_as_float(r[j]) : 0.0f;
                    continue;
                }
                if (m0 + cb * 32 >= p.M) continue;                           // nothing of this block is inside the output
                if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                asm volatile("bar.sync 1, 128;" ::: "memory");
                GT *dst = reinterpret_cast<GT *>(o_stage) + row;
#pragma unroll
                for (int j = 0; j < 32; ++j) dst[j * GU_BK] = from_f32<GT>(__uint_as_float(r[j]));
                fence_proxy_async_smem();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (issuer) {
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                                 ::"l"(&out_map), "r"(smem_addr(o_stage)), "r"(k0), "r"(m0 + cb * 32) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the staging tile outlives the stores
    }
    if (p.splits > 1) {
        // every thread of every CTA of the cluster reaches these barriers (also after an abort)
        __syncwarp();
        cgx::cluster_group cluster = cgx::this_cluster();
        float *red = reinterpret_cast<float *>(a_tiles);
        cluster.sync();
        if (*abort_flag == 0) {
            const int rank = (int)cluster.block_rank(), nranks = (int)cluster.num_blocks();
            const int k0 = (first_tile % p.k_tiles) * GU_BK, m0 = (first_tile / p.k_tiles) * bn;
            const int per_rank = (bn + nranks - 1) / nranks, c0 = rank * per_rank, c1 = min(bn, c0 + per_rank);
            for (int e = tid; e < (c1 - c0) * (GU_BK / 2); e += GU_THREADS) {
                const int c = c0 + e / (GU_BK / 2), kk = (e % (GU_BK / 2)) * 2;
                float2 v = make_float2(0.0f, 0.0f);
                for (int q = 0; q < nranks; ++q) {
                    const float2 a = *reinterpret_cast<const float2 *>(cluster.map_shared_rank(red, q) + c * GU_BK + kk);
                    v.x += a.x; v.y += a.y;
                }
                if (m0 + c < p.M && k0 + kk < p.K) {                         // K is even
                    const GT pair[2] = {from_f32<GT>(v.x), from_f32<GT>(v.y)};
                    *reinterpret_cast<uint32_t *>(reinterpret_cast<GT *>(p.gi) + (int64_t)(m0 + c) * p.K + k0 + kk) =
                        *reinterpret_cast<const uint32_t *>(pair);
                }
            }
        }
        cluster.sync();                                     // shared memory stays until every peer has read it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 3) tmem_dealloc(tmem_base, tmem_cols);
}

// Products that the mma.sync kernel does faster: one or two steps of weight rows and at most about two of its blocks an
// SM.  The tcgen05 kernel's fixed part (rings, tensor memory, 24 warps; 4.5 us, 7 us with a tile of 256 tokens) is then
// the whole call; at 8 bits a step there costs twice as much.  us there / here, W4 g128: N 64, K 1024: 4.1 / 5.2 at 64
// tokens, 5.0 / 7.5 at 1024; N 96, K 1024: 6.0 / 5.3 at 64, 7.2 / 7.7 at 1024; N 128: 6.7 / 5.4 and 8.3 / 7.6; N 64,
// K 4096: 11.7 / 7.8 at 1024 tokens.  W8 g32: N 64, K 4096: 6.0 / 7.6 at 256 tokens, 9.0 / 7.6 at 512.
bool grad_small(int64_t M, int64_t N, int64_t K, int bits) {
    if (M > (1 << 20) || K > (1 << 20)) return false;
    const int64_t blocks = (M + GI_BM - 1) / GI_BM * ((K + GI_BK - 1) / GI_BK);
    const int64_t room = (M > 128 ? 16384 : 8192) / (bits == 8 ? 2 : 1);
    return N <= (M > 128 && bits < 8 ? 120 : 64) && blocks <= 256 && N * blocks <= room;
}

// What the tcgen05 kernel can take: 16-bit gradients in rows that TMA can stride over (whole 16-byte units,
// 16-byte aligned), power-of-two groups of at least 16 codes that hold whole words, whole 16-byte vectors
// of packed words per row, at least one full tile of columns.  The rest runs on the kernels above.
bool grad_umma_ok(const void *go, const void *gi, int dt, int64_t M, int64_t N, int64_t K, const int32_t *q, int bits, int g) {
    if (dt != BW_F16 && dt != BW_BF16) return false;
    const int vpi = 32 / bits;
    if (M < 1 || N < 8 || K < GU_BK) return false;
    if ((g & (g - 1)) || g < 16 || g < vpi) return false;
    if (N % 8 || K % (4 * vpi) || K % 8) return false;
    if (M > 0x7ffffeff || K > 0x7ffffeff || N > 0x7ffffeff) return false;
    if (!aligned_to(go, 16) || !aligned_to(gi, 16) || !aligned_to(q, 16)) return false;
    return encode_tiled_fn() != nullptr;
}

// BW_ERR_UNSUPPORTED: nothing was launched.
template <int BITS, typename GT>
int launch_umma(const void *go, int64_t M, int64_t N, int64_t K, const int32_t *q, const __half *scale, const __half *zp,
                void *gi, int g, cudaStream_t st) {
    constexpr int VPI = 32 / BITS;
    constexpr int SLOT = GU_BN * (GU_BK * BITS / 8) + 2 * GU_C_BYTES;
    GuParams p = {};
    p.scale = scale; p.zp = zp; p.gi = gi; p.M = M; p.N = N; p.K = K;
    while ((1 << p.g_shift) < g) ++p.g_shift;
    p.G = (int)(K / g);
    p.bn = M > 128 ? 256 : (M > 64 ? 128 : (M > 32 ? 64 : (M > 16 ? 32 : 16)));
    p.steps = (int)((N + GU_BN - 1) / GU_BN);
    p.k_tiles = (int)((K + GU_BK - 1) / GU_BK);
    const int64_t tiles = (int64_t)p.k_tiles * ((M + p.bn - 1) / p.bn);
    if (tiles > 1 << 30) return BW_ERR_UNSUPPORTED;
    p.tiles = (int)tiles;
    const size_t fixed = 1024 + 512 + (size_t)GU_AS * GU_A_BYTES + (size_t)GU_WS * SLOT + GU_O_BYTES;
    const size_t x_stage = (size_t)p.bn * 128;
    p.x_stages = (int)((227 * 1024 - fixed) / x_stage);
    if (p.x_stages > GU_AS) p.x_stages = GU_AS;
    const size_t smem = fixed + (size_t)p.x_stages * x_stage;
    int dev = 0, sms = 0;
    BW_CUDA_TRY(cudaGetDevice(&dev));
    BW_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // fewer tiles than SMs: split the rows over a cluster, at least four stages a CTA
    int splits = 1;
    if (tiles < sms) {
        splits = (int)(sms / tiles);
        if (splits > 8) splits = 8;
        if (splits > p.steps / 4) splits = p.steps / 4;
        if (splits < 1) splits = 1;
    }
    p.splits = splits;
    p.per_split = (p.steps + splits - 1) / splits;
    p.const_tma = p.G % 8 == 0 && aligned_to(scale, 16) && aligned_to(zp, 16);

    CUtensorMap xm, wm, sm, zm, om;
    const CUtensorMapSwizzle wswz = BITS == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : (BITS == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    bool ok = encode_2d(&xm, CU_TENSOR_MAP_DATA_TYPE_UINT16, go, N, M, N * 2, GU_BN, p.bn, CU_TENSOR_MAP_SWIZZLE_128B) &&
              encode_2d(&wm, CU_TENSOR_MAP_DATA_TYPE_INT32, q, K / VPI, N, K / VPI * 4, GU_BK / VPI, GU_BN, wswz) &&
              encode_2d(&om, CU_TENSOR_MAP_DATA_TYPE_UINT16, gi, K, M, K * 2, GU_BK, 32, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (ok && p.const_tma)
        ok = encode_2d(&sm, CU_TENSOR_MAP_DATA_TYPE_UINT16, scale, p.G, N, (int64_t)p.G * 2, 8, GU_BN, CU_TENSOR_MAP_SWIZZLE_NONE) &&
             encode_2d(&zm, CU_TENSOR_MAP_DATA_TYPE_UINT16, zp, p.G, N, (int64_t)p.G * 2, 8, GU_BN, CU_TENSOR_MAP_SWIZZLE_NONE);
    else { sm = wm; zm = wm; }
    if (!ok) return BW_ERR_UNSUPPORTED;

    auto kern = grad_input_umma_kernel<BITS, GT>;
    BW_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles < sms ? tiles : sms), 1, (unsigned)splits);
    cfg.blockDim = dim3(GU_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (splits > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = (unsigned)splits;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    BW_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, xm, wm, sm, zm, om, p));
    note_launch("grad_input_umma_kernel");
    return BW_OK;
}

template <int BITS, typename GT>
int launch(const void *go, int64_t M, int64_t N, int64_t K, const int32_t *q, const __half *scale,
           const __half *zp, void *gi, int g, cudaStream_t st) {
    const int wpr = (int)(K / (32 / BITS));
    const int64_t mblocks = (M + TOK - 1) / TOK;
    if (mblocks > 65535) return BW_ERR_SHAPE;
    dim3 grid((unsigned)((wpr + 127) / 128), (unsigned)mblocks, 1);
    grad_input_kernel<BITS, GT><<<grid, 128, 0, st>>>((const GT *)go, M, N, K, q, scale, zp, (GT *)gi, g,
                                                      wpr, K / g);
    return check_launch("grad_input_kernel");
}

template <int BITS>
int launch_dt(const void *go, int dt, int64_t M, int64_t N, int64_t K, const int32_t *q,
              const __half *scale, const __half *zp, void *gi, int g, cudaStream_t st) {
    if (grad_umma_ok(go, gi, dt, M, N, K, q, BITS, g) && !grad_small(M, N, K, BITS)) {
        const int rc = dt == BW_F16 ? launch_umma<BITS, __half>(go, M, N, K, q, scale, zp, gi, g, st)
                                    : launch_umma<BITS, __nv_bfloat16>(go, M, N, K, q, scale, zp, gi, g, st);
        if (rc != BW_ERR_UNSUPPORTED) return rc;
    }
    if (grad_tc_ok(go, gi, dt, N, K)) {
        if (dt == BW_F16) return launch_tc<BITS, __half>(go, M, N, K, q, scale, zp, gi, g, st);
        return launch_tc<BITS, __nv_bfloat16>(go, M, N, K, q, scale, zp, gi, g, st);
    }
    switch (dt) {
        case BW_F32: return launch<BITS, float>(go, M, N, K, q, scale, zp, gi, g, st);
        case BW_F16: return launch<BITS, __half>(go, M, N, K, q, scale, zp, gi, g, st);
        case BW_BF16: return launch<BITS, __nv_bfloat16>(go, M, N, K, q, scale, zp, gi, g, st);
        default: return BW_ERR_DTYPE;
    }
}

}  // namespace

int grad_device_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_grad_status, sizeof(int)) != cudaSuccess) return -1;
    if (v) (void)cudaMemcpyToSymbol(g_grad_status, &zero, sizeof(int));
    return v;
}

int qmatmul_grad_input(const void *go, int dtype, int64_t M, int64_t N, int64_t K, const int32_t *q,
                       const __half *scale, const __half *zp, void *gi, int bits, int g, cudaStream_t st) {
    if (K > (int64_t)1 << 31) return BW_ERR_SHAPE;
    switch (bits) {
        case 2: return launch_dt<2>(go, dtype, M, N, K, q, scale, zp, gi, g, st);
        case 4: return launch_dt<4>(go, dtype, M, N, K, q, scale, zp, gi, g, st);
        case 8: return launch_dt<8>(go, dtype, M, N, K, q, scale, zp, gi, g, st);
        default: return BW_ERR_BITS;
    }
}

}  // namespace bw
