// Quantized matmul of at most 8 tokens: out[M,N] = x[M,K] . W[N,K]^T (+bias), W = fp16(scale * (code - zero_point))
// bit-identical to the reference's dequantized weights (bitween/modules.py:55-58), fp32 accumulation, fp16 output
// rounding and a separate fp16 bias add as in bitween/modules.py:97,101.  One launch, no scratch.
//
// What bounds it: the bytes of a layer take 1.3 us (4096 x 4096, W4) to 4.5 us (14336 x 4096) when they are only read,
// in launches that follow each other through programmatic dependent launch; beyond that the dequantization, which needs
// three half-rate instructions for two weights (3.4 us for 14336 x 4096), and the chain from the preceding kernel's end
// to the first sum.  The ring kernel (qmatmul_decode.cu) has one 220 KB CTA an SM, so that the next launch's CTAs only
// enter when those of the launch before have left: 5.7 us a launch in which no weights stream.  Hence here
//   * CTAs of 8 warps, two an SM, or of 16 warps (below): the CTAs of the next launch enter one by one, and their first
//     words and constants are requested before griddepcontrol.wait;
//   * row tiles of 16 rows (one MMA's) for whole CTAs, K cut into one contiguous range a warp: warps meet once, at
//     the end, when the shares of all of the CTA's tiles are added in the order of the k ranges (a barrier a tile
//     cost 0.4 us on 14336 x 4096);
//   * packed words go from memory to registers, eight 16-byte loads a lane in flight, a block of four chunks (64 bytes
//     of each row) ahead across tiles;
//   * a warp prepares the activations of its own k range once, in the order of the MMAs' B fragments, and reuses them
//     for all of the CTA's tiles.
// us in a CUDA graph of layers that are not in L2, ring kernel / this one, W4 g128, 1 token: 4096 x 4096 6.88 / 4.56,
// 1024 x 4096 4.54 / 3.02, 14336 x 4096 13.0 / 10.0, 4096 x 14336 13.4 / 10.8.  Tried and slower on
// 14336 x 4096: words through a shared-memory ring with cp.async 16.5, 3 CTAs an SM at 80 registers 11.0, one tile a CTA
// (the preparation again for every tile) 15.4, a shared memory carve-out that leaves 28 KB of L1 for the loads in flight
// 15.9 against 11.7.
#include <atomic>

#include "bw_common.cuh"
#include "qmm_dequant.cuh"

namespace bw {
namespace {

struct RowsParams {
    const void *x;
    const uint4 *q;
    const __half *scale, *zp, *bias;
    void *out;
    int64_t N, K;
    int M;
    int out_dtype;
    int g_shift, G;
    int vpr;              // 16-byte vectors per row of packed words
    int chunks, cpw;      // k-chunks of a row, of a warp
    int tiles;            // row tiles of 16
    int tmax;             // row tiles of a CTA
    int x_magic;          // 2^20 / units of a token in a warp's k range, rounded up
    int ne;               // groups of a warp's table
    int const_vec;        // groups can be read two at a time
    int tab_off, red_off; // shared memory: activations | constants [WK][ne][16] | sums [tmax][WK][M][RS]
};

__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// 16 bytes of two rows, read once (predicated in place instead of branched around: 1 % of a pass)
__device__ __forceinline__ void ld_stream(uint4 &v, uint4 &w, const uint4 *p, const uint4 *q, bool live) {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %10, 0;\n"
                 " @p ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%8];\n"
                 " @p ld.global.nc.L1::no_allocate.v4.u32 {%4,%5,%6,%7}, [%9];\n}"
                 : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w), "+r"(w.x), "+r"(w.y), "+r"(w.z), "+r"(w.w)
                 : "l"(p), "l"(q), "r"((int)live));
}
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int BITS> struct Geo {
    static constexpr int VPI = 32 / BITS, KL = 4 * VPI, KC = 4 * KL;
    static constexpr int NP = KL / 8;                     // 16-byte pieces of fp16 activations per lane and chunk
    static constexpr int UNIT = VPI > 8 ? VPI : 8;        // k values prepared at a time
    static constexpr int UPC = KC / UNIT, UPL = KL / UNIT;
};
__device__ __forceinline__ uint32_t bf2h(uint32_t u) { return h2_as_u32(__floats2half2_rn(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u))); }
template <int V> struct Int { static constexpr int value = V; };
template <int UNIT, typename XT> struct Raw { uint4 v[UNIT * sizeof(XT) / 16]; };
// fp16 pairs (0,1) (2,3) ... of the unit
template <int UNIT, typename XT> __device__ __forceinline__ void to_h2(const Raw<UNIT, XT> &r, uint32_t (&h)[UNIT / 2]) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(r.v);
#pragma unroll
    for (int i = 0; i < UNIT / 2; ++i) {
        if constexpr (sizeof(XT) == 4) h[i] = h2_as_u32(__floats2half2_rn(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1])));
        else if constexpr (__is_same(XT, __half)) h[i] = w[i];
        else h[i] = bf2h(w[i]);
    }
}

template <int BITS, int WK, int OCC, typename XT>
__global__ void __launch_bounds__(WK * 32, OCC)
qmm_rows_kernel(const __grid_constant__ RowsParams p, const __grid_constant__ Epilogue ep) {
    using G_ = Geo<BITS>;
    constexpr int R = 16, RS = 20, THREADS = WK * 32, PS = G_::NP + 1, D = 4, NPF = 4;
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, wk = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int g = lane >> 2, t = lane & 3;
    const int stride = gridDim.x;
    const int c0 = min(wk * p.cpw, p.chunks), c1 = min(c0 + p.cpw, p.chunks);
    const int my_tiles = c0 < c1 ? (p.tiles - (int)blockIdx.x + stride - 1) / stride : 0;

    // ---- packed words: blocks of D chunks, requested one block ahead ----
    const int lane_c1 = min(c1, (p.vpr - t + 3) / 4);    // chunks of which this lane's vector lies inside the row
    int ptile = 0, pc = c0, plim = my_tiles > 0 ? lane_c1 : c0;
    const uint4 *pa, *pb;
    auto set_rows = [&]() {
        const int64_t n0 = ((int64_t)blockIdx.x + (int64_t)ptile * stride) * R + g;
        pa = p.q + min(n0, p.N - 1) * p.vpr + c0 * 4 + t;
        pb = p.q + min(n0 + 8, p.N - 1) * p.vpr + c0 * 4 + t;
    };
    set_rows();
    uint4 wa[D] = {}, wb[D] = {};
    auto request = [&](int d) {
        ld_stream(wa[d], wb[d], pa + d * 4, pb + d * 4, pc + d < plim);
    };
    auto advance = [&]() {
        pc += D; pa += D * 4; pb += D * 4;
        if (pc >= c1) {
            pc = c0;
            if (++ptile < my_tiles) set_rows();
            else plim = c0;
        }
    };
#pragma unroll
    for (int d = 0; d < D; ++d) request(d);
    advance();

    // ---- constants of a tile's rows and this warp's groups: {scale, scale}, {1024 + zp, 1024 + zp} by [group][row]; a lane takes pairs of groups of a row ----
    const int crow = lane & 15, cpart = lane >> 4;
    uint2 *const tab = reinterpret_cast<uint2 *>(smem + p.tab_off) + (size_t)wk * p.ne * R;
    const int e0 = (int)(((int64_t)c0 * G_::KC) >> p.g_shift) & ~1;
    const int ng = c0 < c1 ? (int)((((int64_t)c1 * G_::KC - 1) >> p.g_shift) + 1) - e0 : 0;
    uint32_t sv[NPF], zv[NPF];
    auto pair_at = [&](const unsigned short *src, int e) {
        if (p.const_vec) return e < p.G ? __ldg(reinterpret_cast<const uint32_t *>(src + e)) : 0u;
        return (e < p.G ? (uint32_t)__ldg(src + e) : 0u) | (e + 1 < p.G ? (uint32_t)__ldg(src + e + 1) << 16 : 0u);
    };
    auto const_row = [&](const __half *base, int ti) {
        const int64_t n = min(((int64_t)blockIdx.x + (int64_t)ti * stride) * R + crow, p.N - 1);
        return reinterpret_cast<const unsigned short *>(base) + n * p.G;
    };
    auto put = [&](int e, uint32_t s, uint32_t z) {
        const __half2 k1024 = __float2half2_rn(1024.0f);
        uint2 *d = tab + e * R + crow;
        d[0] = make_uint2(__byte_perm(s, s, 0x1010), h2_as_u32(__hadd2(u32_as_h2(__byte_perm(z, z, 0x1010)), k1024)));
        d[R] = make_uint2(__byte_perm(s, s, 0x3232), h2_as_u32(__hadd2(u32_as_h2(__byte_perm(z, z, 0x3232)), k1024)));
    };
    auto fetch_consts = [&](int ti) {
        if (ti < my_tiles) {
            const unsigned short *sp = const_row(p.scale, ti), *zq = const_row(p.zp, ti);
#pragma unroll
            for (int i = 0; i < NPF; ++i)
                if (i * 4 < ng) { sv[i] = pair_at(sp, e0 + i * 4 + cpart * 2); zv[i] = pair_at(zq, e0 + i * 4 + cpart * 2); }
        }
    };
    auto store_consts = [&](int ti) {
#pragma unroll
        for (int i = 0; i < NPF; ++i)
            if (i * 4 < ng) put(i * 4 + cpart * 2, sv[i], zv[i]);
        if (ng > NPF * 4) {
            const unsigned short *sp = const_row(p.scale, ti), *zq = const_row(p.zp, ti);
            for (int e = NPF * 4 + cpart * 2; e < ng; e += 4) put(e, pair_at(sp, e0 + e), pair_at(zq, e0 + e));
        }
    };
    fetch_consts(0);

    pdl_wait();

    // ---- this warp's activations, cast to fp16, as B fragments: [chunk][token][t][piece], the pieces of a lane in a row ----
    uint4 *xs = reinterpret_cast<uint4 *>(smem) + (size_t)c0 * p.M * 4 * PS;
    // (units of all tokens at the warp's pitch, so that token and unit come from one multiplication; a few or many in flight)
    auto prepare = [&](auto batch) {
        constexpr int B = decltype(batch)::value;
        const int per = (c1 - c0) * G_::UPC, pitch = p.cpw * G_::UPC, units = pitch * p.M;
        for (int i0 = lane; i0 < units; i0 += B * 32) {
            Raw<G_::UNIT, XT> raw[B];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const int i = i0 + j * 32, m = (int)((unsigned)i * (unsigned)p.x_magic >> 20), u = i - m * pitch;
                const int k = c0 * G_::KC + u * G_::UNIT;
                const bool live = i < units && u < per && k < p.K;
                const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const XT *>(p.x) + m * p.K + k);
#pragma unroll
                for (int e = 0; e < (int)(sizeof(raw[j].v) / 16); ++e) raw[j].v[e] = live ? __ldcg(src + e) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const int i = i0 + j * 32, m = (int)((unsigned)i * (unsigned)p.x_magic >> 20), u = i - m * pitch;
                if (i < units && u < per) {
                    uint32_t r[G_::UNIT / 2];
                    to_h2<G_::UNIT, XT>(raw[j], r);
                    const int c = u / G_::UPC, tt = u % G_::UPC / G_::UPL, sub = u % G_::UPL;
                    uint4 *dst = xs + ((c * p.M + m) * 4 + tt) * PS + (BITS == 2 ? 2 * sub : sub);
                    if constexpr (BITS == 4) {
                        *dst = make_uint4(pair_lo(r[0], r[2]), pair_hi(r[0], r[2]), pair_lo(r[1], r[3]), pair_hi(r[1], r[3]));
                    } else if constexpr (BITS == 8) {
                        *dst = make_uint4(pair_lo(r[0], r[1]), pair_hi(r[0], r[1]), pair_lo(r[2], r[3]), pair_hi(r[2], r[3]));
                    } else {
                        dst[0] = make_uint4(pair_lo(r[0], r[4]), pair_hi(r[0], r[4]), pair_lo(r[1], r[5]), pair_hi(r[1], r[5]));
                        dst[1] = make_uint4(pair_lo(r[2], r[6]), pair_hi(r[2], r[6]), pair_lo(r[3], r[7]), pair_hi(r[3], r[7]));
                    }
                }
            }
        }
    };
    constexpr int FLY = 128 / (G_::UNIT * (int)sizeof(XT));          // 32 registers
    if (p.cpw * G_::UPC * p.M <= 64) prepare(Int<2>{});
    else prepare(Int<FLY>{});

    const int xstep = p.M * 4 * PS;
    const uint4 *const x0 = xs + (min(g, p.M - 1) * 4 + t) * PS;     // this lane's token (columns past the last token are not stored)
    const uint4 *xl;                                                 // the same at the current chunk
    float acc[2][4];                                                 // two chains of MMAs
    auto compute = [&](const uint4 &va, const uint4 &vb, const uint2 *tb, int k) {
        Dequant<BITS> dqa, dqb;
        auto set = [&](int kk) {
            const uint2 *cs = tb + (kk >> p.g_shift) * R;
            const uint2 ca = cs[0], cb = cs[8];
            dqa.set(GroupConst{ca.x, ca.y});
            dqb.set(GroupConst{cb.x, cb.y});
        };
        set(k);
        uint4 xq8;
        (void)xq8;
#pragma unroll
        for (int wi = 0; wi < 4; ++wi) {
            const uint32_t wwa = (&va.x)[wi], wwb = (&vb.x)[wi];
            if constexpr (BITS == 4) {
                const uint4 xf = xl[wi];
                uint32_t qa[4], qb[4];
                dqa.run(wwa, qa);
                dqb.run(wwb, qb);
                mma(acc[0], qa[0], qb[0], qa[1], qb[1], xf.x, xf.y);
                mma(acc[1], qa[2], qb[2], qa[3], qb[3], xf.z, xf.w);
            } else if constexpr (BITS == 8) {
                if ((wi & 1) == 0) xq8 = xl[wi >> 1];
                uint32_t qa[2], qb[2];
                dqa.run(wwa, qa);
                dqb.run(wwb, qb);
                mma(acc[wi & 1], qa[0], qb[0], qa[1], qb[1], wi & 1 ? xq8.z : xq8.x, wi & 1 ? xq8.w : xq8.y);
            } else {
                if (wi == 2 && (1 << p.g_shift) < G_::KL) set(k + G_::KL / 2);   // groups of 32: two in a lane's 64 codes
                const uint4 xa = xl[2 * wi], xb = xl[2 * wi + 1];
                uint32_t qa[8], qb[8];
                dqa.run(wwa, qa);
                dqb.run(wwb, qb);
                mma(acc[0], qa[0], qb[0], qa[1], qb[1], xa.x, xa.y);
                mma(acc[1], qa[2], qb[2], qa[3], qb[3], xa.z, xa.w);
                mma(acc[0], qa[4], qb[4], qa[5], qb[5], xb.x, xb.y);
                mma(acc[1], qa[6], qb[6], qa[7], qb[7], xb.z, xb.w);
            }
        }
    };

    float *red = reinterpret_cast<float *>(smem + p.red_off);
    for (int ti = 0; ti < my_tiles; ++ti) {
        __syncwarp();                                    // the previous tile's constants are done with
        store_consts(ti);
        __syncwarp();                                    // (and, the first time round, the activations are in place)
        fetch_consts(ti + 1);
        const uint2 *tb = tab + g - e0 * R;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[0][e] = acc[1][e] = 0.0f;
        xl = x0;
        int k = c0 * G_::KC + t * G_::KL;
        for (int c = c0; c < c1; c += D) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                if (c + d < c1) {
                    compute(wa[d], wb[d], tb, k);
                    k += G_::KC;
                    xl += xstep;
                }
                request(d);
            }
            advance();
        }
        float *rw = red + (size_t)(ti * WK + wk) * p.M * RS + g;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int m = 2 * t + (e & 1);
            if (m < p.M) rw[m * RS + (e >> 1) * 8] = acc[0][e] + acc[1][e];
        }
    }
    __syncthreads();
    // the shares of each tile, added in the order of the k ranges
    const int nt = (p.tiles - (int)blockIdx.x + stride - 1) / stride, nw = (p.chunks + p.cpw - 1) / p.cpw;
    for (int i = threadIdx.x; i < nt * p.M * R; i += THREADS) {
        const int r = i % R, mm = i / R, ti = mm / p.M, m = mm - ti * p.M;
        const float *rr = red + (size_t)(ti * WK * p.M + m) * RS + r;
        float v = 0.0f;
        if (nw == WK) {
#pragma unroll
            for (int q = 0; q < WK; ++q) v += rr[q * p.M * RS];
        } else {
            for (int q = 0; q < nw; ++q) v += rr[q * p.M * RS];
        }
        const int64_t n = ((int64_t)blockIdx.x + (int64_t)ti * stride) * R + r;
        if (n < p.N) store_output(p.out, p.out_dtype, m * p.N + n, v, p.bias != nullptr, p.bias ? p.bias[n] : __half(), ep);
    }
}

int rows_sms(int dev) {
    static std::atomic<int> cached[64];
    int n = cached[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// BW_ERR_UNSUPPORTED, with nothing launched, when the activations and sums of a CTA do not fit its shared memory.
template <int BITS, int WK, int OCC, typename XT>
int launch_rows(RowsParams p, cudaStream_t st) {
    auto kern = qmm_rows_kernel<BITS, WK, OCC, XT>;
    using G_ = Geo<BITS>;
    int dev = 0;
    BW_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return BW_ERR_UNSUPPORTED;
    p.chunks = (int)((p.K + G_::KC - 1) / G_::KC);
    p.cpw = (p.chunks + WK - 1) / WK;
    p.tiles = (int)((p.N + 15) / 16);
    const int64_t pitch = (int64_t)p.cpw * G_::UPC;
    // (unit i belongs to token i * magic >> 20: exact while i * pitch < 2^20, and i < pitch * M)
    if (pitch * pitch * p.M >= 1 << 20) return BW_ERR_UNSUPPORTED;
    p.x_magic = (int)(((1 << 20) + pitch - 1) / pitch);
    p.ne = (int)((((int64_t)p.cpw * G_::KC - 1) >> p.g_shift) + 6) & ~3;
    const int ctas = p.tiles < OCC * rows_sms(dev) ? p.tiles : OCC * rows_sms(dev);
    p.tmax = (p.tiles + ctas - 1) / ctas;
    const int64_t tab_off = (int64_t)p.chunks * p.M * 4 * (G_::NP + 1) * 16, red_off = tab_off + (int64_t)WK * p.ne * 16 * 8;
    const int64_t smem = red_off + (int64_t)p.tmax * WK * p.M * 20 * 4;
    if (smem > (227 / OCC - 1) * 1024) return BW_ERR_UNSUPPORTED;
    p.tab_off = (int)tab_off; p.red_off = (int)red_off;
    static std::atomic<bool> configured[64];             // per instantiation and device
    if (!configured[dev].load(std::memory_order_relaxed)) {
        BW_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (227 / OCC - 1) * 1024));
        configured[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(WK * 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BW_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p, current_epilogue()));
    return BW_OK;
}

// 8 warps, two CTAs an SM, where a token or four of ordinary length leave little to prepare; otherwise 16 warps, one CTA
// an SM, which share the preparation of a row of activations among twice the warps and have room for longer ones.
// us with 8 / 16 warps, W4 g128: 4096 x 4096, 1 token 4.56 / 5.09, 4 tokens 5.52 / 5.88, 8 tokens 7.5 / 6.3; 14336 x 4096,
// 1 token 10.0 / 12.5, 8 tokens 15.1 / 14.4; 4096 x 11008, 5 tokens: does not fit / 11.8.  In sum over 960 random
// layers of 2 / 4 / 8 bits, groups of 32..128, 1..8 tokens: ring and cluster kernels 7.42 ms, 8 warps for M * K <= 8192 /
// 16384 / 24576: 5.62 / 5.60 / 5.66 ms (5.50 for the better one each time).
template <int BITS, typename XT>
int launch_rows_warps(const RowsParams &p, cudaStream_t st) {
    if (p.M * p.K <= 16384) {
        const int rc = launch_rows<BITS, 8, 2, XT>(p, st);
        if (rc != BW_ERR_UNSUPPORTED) return rc;
    }
    return launch_rows<BITS, 16, 1, XT>(p, st);
}
template <typename XT>
int launch_rows_bits(const RowsParams &p, int bits, cudaStream_t st) {
    switch (bits) {
        case 2: return launch_rows_warps<2, XT>(p, st);
        case 4: return launch_rows_warps<4, XT>(p, st);
        default: return launch_rows_warps<8, XT>(p, st);
    }
}

}  // namespace

// At most 8 tokens (one MMA's columns), power-of-two groups that hold a lane's 16-byte vector of codes (2 bits: half
// of one), rows of whole such vectors, activations in 16-byte units.
bool rows_path_ok(const void *x, int x_dtype, int64_t M, int64_t N, int64_t K, const int32_t *q, int bits, int g) {
    if (bits != 2 && bits != 4 && bits != 8) return false;
    const int kl = 128 / bits;
    if (M < 1 || M > 8 || N < 1 || K < 1 || N > 1 << 30 || K > 1 << 20) return false;
    if ((g & (g - 1)) || g < (bits == 2 ? kl / 2 : kl) || K % kl) return false;
    if (current_epilogue().act == BW_ACT_SILU_MUL) return false;         // (pairs rows in its output stage)
    return aligned_to(q, 16) && aligned_to(x, 16) && (K * dtype_size(x_dtype)) % 16 == 0;
}

// BW_ERR_UNSUPPORTED: nothing was launched (rows of activations too long for shared memory); another kernel takes the call.
int qmatmul_rows(const void *x, int x_dtype, int64_t M, int64_t N, int64_t K, const int32_t *q,
                 const __half *scale, const __half *zp, const __half *bias, void *out, int out_dtype,
                 int bits, int g, cudaStream_t st) {
    RowsParams p = {};
    p.x = x; p.q = reinterpret_cast<const uint4 *>(q); p.scale = scale; p.zp = zp; p.bias = bias; p.out = out;
    p.M = (int)M; p.N = N; p.K = K; p.out_dtype = out_dtype;
    while ((1 << p.g_shift) < g) ++p.g_shift;
    p.G = (int)(K / g);
    p.vpr = (int)(K * bits / 128);
    p.const_vec = p.G % 2 == 0 && aligned_to(scale, 4) && aligned_to(zp, 4);
    switch (x_dtype) {
        case BW_F16: return launch_rows_bits<__half>(p, bits, st);
        case BW_BF16: return launch_rows_bits<__nv_bfloat16>(p, bits, st);
        default: return launch_rows_bits<float>(p, bits, st);
    }
}

}  // namespace bw
