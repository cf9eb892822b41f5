// 4-bit weights x bf16 activations on the 5th-generation tensor cores, weights dequantised into TENSOR MEMORY:
//   out[M, N] = act(alpha * sum_k x[m, k] * w[n, k] + bias[n]) + beta * out
//
// A tile is 128 weight rows x NT tokens (NT a multiple of 16, up to 256).  The weight rows are the M side of
// tcgen05.mma kind::f16 and come from tensor memory, the tokens are the N side and come from shared memory, so a
// few tokens cost a few columns instead of a padded 128-row tile.  Groups of four warps (four groups, or two where two CTAs
// share an SM) turn codes into bf16 in registers (thread = weight row) and store them with tcgen05.st; nothing dequantised
// passes through shared memory, whose port the activation tiles and the MMAs need.  What a weight becomes:
//   NVFP4        e2m1 x UE4M3 has six significant bits: the product is EXACT in bf16, and so is the result up to the
//                fp32 accumulation -- activations need no residual pieces and no quantiser launch in front
//   INT4 k-block (q - 8) * scale with an 11-bit fp16 scale, rounded once to bf16: the scale is split into two bf16
//                parts, q * low part is exact, so one fused multiply-add rounds like the fp32 product would
//   INT4 plugin  q * scale + zero, one fused multiply-add
//
// Split K: the CTAs of a thread-block cluster take K ranges of one tile; each parks its partial sums in its own
// shared memory, and every CTA finishes its share of the tokens from all of them through distributed shared
// memory, summed in rank order (deterministic; no workspace, no counters, no waiting on other clusters).
//
// What bounds it: four 128 x NT x 16 MMAs with A in tensor memory take exactly 2 NT cycles (measured, NT 32..256), the
// dequantisation of their 128 x 64 weights 250 (NVFP4) to 340 (INT4) cycles of an SM's instruction issue, ~350 to 450 with the
// loop around it (470-530 before a unit was two parts and the positions were counted), and the token tiles are re-read once
// per 128 weight rows (434 MB through the L2 at 712 x 16384 x 2048).  Counters of that launch and of 712 x 2048 x 16384: issue
// slots used in 53 and 66 % of the active cycles, tensor pipe 52 and 61 %; the rest is fill, hand-over and epilogue.  B200, in a
// chain of programmatic dependent launches: INT4 712 x 16384 x 2048 47 us (85 us with weights dequantised through shared
// memory), 712 x 2048 x 16384 45 and 397 x 2048 x 16384 29 us with K split (265 without).  Pairs of CTAs sharing the token tile
// (cta_group::2) halve those reads but were slower (147 against 103 us at 712 x 32768 x 2048): the barrier round trips
// between the two SMs sit on the issuing warp's path.
//
// Roles: warp 0 activation tiles (TMA), warp 1 tensor memory + MMA issue, warp 2 weight blocks (256 K values of 128 rows:
// 16 KB of codes + scales), then 16 warps (8 where two CTAs share an SM) of dequantisation and epilogue.  Weight blocks are
// requested and dequantised BEFORE griddepcontrol.wait: under programmatic dependent launch a launch's weights are
// already in tensor memory when its predecessor's activations arrive.  Every wait is bounded.
#include <algorithm>
#include <atomic>

#include "tcgen05.cuh"

namespace tpb {

bool make_tensor_map_2d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t dim0, uint64_t dim1,
                        uint64_t pitch_bytes, uint32_t box0, uint32_t box1, bool swizzle128);

namespace {

constexpr int kRows = 128;                       // weight rows per tile
constexpr int kBlkK = 256;                       // K values of one weight block
constexpr int kPartK = 64;                       // K values of one part of a step: a 128-byte row of bf16
constexpr int kSlabBytes = 2048;                 // scales of 128 rows x 256 K
constexpr int kCodeBytes = kRows * kBlkK / 2;    // 16 KB
constexpr int kWSlot = kCodeBytes + 2 * kSlabBytes;
constexpr int kMaxW = 4, kMaxS = 14;
constexpr int kXWarp = 0, kMmaWarp = 1, kWWarp = 2, kDqWarp0 = 3;
constexpr long long kWaitG = 400000000LL;        // ~0.2 s
constexpr long long kLandCycles = 2000000LL;     // ~1 ms

enum { kFmtNvfp4 = 0, kFmtKblock = 1, kFmtPlugin = 2, kFmtNvfp4T = 3 };   // 3: the w4a8 plugin's transposed operand
// Epilogues.  Direct (K not split, no partner rows) has a kernel of its own, the others share one: a chain of short launches
// fetches its instructions anew unless the launches before ran the same ones.  All five in one kernel cost the 50-token
// launches 0.6 us each, a kernel for each of the five 0.4.
enum { kEpiDirect = 0, kEpiSplit = 1, kEpiResidual = 2, kEpiGated = 3, kEpiQkv = 4 };

struct W4gParams {
    CUtensorMap map_x;                           // bf16 [M, K], box 64 x NT, 128-byte swizzle
    CUtensorMap map_w;                           // codes (unused with a tiled image)
    CUtensorMap map_s;                           // k-block scales
    const uint8_t* image;                        // tiled NVFP4 image or null
    const uint8_t* sf;                           // row-major NVFP4: scale atoms
    const __half* kb_scale;                      // k-block scales that TMA cannot fetch (base not 16-byte aligned), else null
    const __nv_bfloat16* pl_scale;               // plugin: [N, K / 128]
    const __nv_bfloat16* pl_zero;
    const void* bias;
    void* out;
    int bias_dtype, out_dtype, ldo, activation;
    float alpha, beta;
    int M, N, K;
    int nt;                                      // tokens per tile
    int splits;                                  // CTAs (cluster size) per tile, each with a K range
    int k_blocks, k_steps;
    int parts;                                   // consecutive 64-K parts a group of warps dequantises: 1, or 2 for narrow token tiles
    int merge;                                   // such units per operand step (what one barrier hands to the tensor cores)
    int n_w, n_s;                                // ring depths: weight blocks, operand steps
    int tmem_cols, a_col;
    int epilogue;
    int gated_rows;                              // kEpiGated: rows of one half (I), W = [gate; up]
    int img_kblocks;                             // K blocks per 256-row block of the image / atoms per row tile / 4
    int q_dim, ldq;
    __nv_bfloat16* k_rows;
    __nv_bfloat16* v_rows;
    const int* positions;
    const __nv_bfloat16* rope_cos;
    const __nv_bfloat16* rope_sin;
    // The norm in front of this linear, folded: x holds h * (1 + scale), the row's RMS factor and W * shift come here
    const float* in_sumsq;                       // [M, in_parts] partial sums of h^2, or null
    const float* in_shift;                       // fp32 [N] or null
    int in_parts;
    float in_eps, in_inv_k;
    // kEpiResidual: the residual stream and the next norm's input
    const __nv_bfloat16* res;
    const __nv_bfloat16* gate;
    const __nv_bfloat16* scale;
    __nv_bfloat16* h_out;
    float* out_sumsq;                            // [M, N / 128]
    __nv_bfloat16* copy_out;                     // kEpiSplit: the result once more, bf16 [M, N], or null
};

struct W4gControl {
    uint64_t w_full[kMaxW], w_empty[kMaxW];      // raw weight blocks
    uint64_t full[kMaxS], empty[kMaxS];          // operand steps: weights in tensor memory + activations in shared memory
    uint64_t acc_full;
    uint32_t tmem_base;
    int failed;                                  // a wait ran out
};

__device__ __forceinline__ void give_up(W4gControl& ctl, int error) {
    record_error(error);
    ctl.failed = 1;
}

__device__ __forceinline__ uint32_t idesc_bf16(int n) {
    // D = f32, A = B = bf16, both K-major, N >> 3 at [17,23), M = 128
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}

// D[tmem] (+)= A[tmem] * B[smem]^T
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
}

// the four K = 16 products of one 64-K part; `acc` = 0: the first of them starts the sum
__device__ __forceinline__ void mma_part(uint32_t tmem_d, uint32_t a_col, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        mma_bf16_ts(tmem_d, a_col + kk * 8, tc::desc_from_words(b_lo + kk * 2, tc::kDescHiKmajorSw128), idesc, kk > 0 ? 1u : acc);
    }
}

__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// two E4M3 bytes -> fp16 pair (exact)
__device__ __forceinline__ __half2 decode_e4m3x2_h(uint16_t v) {
    uint32_t r;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
    return *reinterpret_cast<__half2*>(&r);
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) { return __byte_perm(a, b, s); }
__device__ __forceinline__ uint32_t bits(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }

// Eight e2m1 codes (code i at bits 4 i) -> bf16 pairs in K order, times the block scale.  The product is formed in fp16,
// where it is exact (six significant bits, 2^-10 .. 2688), and stays exact through fp32 to bf16.  Half the cycles of
// assembling bf16 from byte tables with prmt (729 against 1243 per 64-K step with 16 warps on the SM): the integer pipe
// runs at half rate, the converter and the FMA pipe share this form's work.
__device__ __forceinline__ void dequant_e2m1x8(uint32_t w, __half2 s, uint32_t* out) {
    __half2 h[4];
    decode_e2m1x8(w, h);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(__hmul2(h[i], s));
        out[i] = bits(__floats2bfloat162_rn(f.x, f.y));
    }
}

// Eight unsigned nibbles (zero point 8) -> q - 8 as exact bf16 pairs in K order
__device__ __forceinline__ void nibbles_minus8(uint32_t w, __nv_bfloat162* q) {
    const __nv_bfloat162 k136 = as_bf162(0x43084308u);
    uint32_t h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = bits(__hsub2(as_bf162(((w >> (4 * j)) & 0x000F000Fu) | 0x43004300u), k136));
    q[0] = as_bf162(prmt(h[0], h[1], 0x5410));
    q[1] = as_bf162(prmt(h[2], h[3], 0x5410));
    q[2] = as_bf162(prmt(h[0], h[1], 0x7632));
    q[3] = as_bf162(prmt(h[2], h[3], 0x7632));
}

__device__ __forceinline__ float act_fast(float x, int act) {
    if (act == TPB200_ACT_GELU) {   // 0.5 x (1 + tanh z) == x * sigmoid(2 z), without cancellation for negative x
        const float z2 = 1.5957691216057308f * (x + 0.044715f * x * x * x);
        return __fdividef(x, 1.0f + __expf(-z2));
    }
    if (act == TPB200_ACT_SILU) return __fdividef(x, 1.0f + __expf(-x));
    return x;
}
__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ uint2 pack4(const float (&v)[4]) {
    return make_uint2(bits(__floats2bfloat162_rn(v[0], v[1])), bits(__floats2bfloat162_rn(v[2], v[3])));
}
__device__ __forceinline__ void unpack4(uint2 u, float (&v)[4]) {
    const float2 a = __bfloat1622float2(as_bf162(u.x)), b = __bfloat1622float2(as_bf162(u.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void act4(float (&v)[4], int act) {
    if (act == TPB200_ACT_GELU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = act_fast(v[e], TPB200_ACT_GELU);
    } else if (act == TPB200_ACT_SILU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = act_fast(v[e], TPB200_ACT_SILU);
    }
}

// Sums of up to S CTAs' partial results at one offset, in rank order.  All loads leave before the first sum needs one (a
// loop that added while it loaded paid a distributed-shared-memory round trip per CTA: 1.4 us of a 5 us launch at 8).
template <int S>
__device__ __forceinline__ float4 sum_ranks(uint32_t base, uint32_t off, int splits) {
    float4 x[S];
#pragma unroll
    for (int p = 0; p < S; ++p) x[p] = ld_cluster_f4(map_to_rank(base, p < splits ? p : 0) + off);
    float4 a = x[0];
#pragma unroll
    for (int p = 1; p < S; ++p) {
        if (p < splits) { a.x += x[p].x; a.y += x[p].y; a.z += x[p].z; a.w += x[p].w; }
    }
    return a;
}

// A load for the line's sake: into this SM's L1, the value unused
__device__ __forceinline__ void touch(const void* p) {
    uint32_t v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
}

// What one unit of the epilogue (a token, 4 weight rows or 4 + 4) reads for the norms folded into a launch.
//   in:   RMSNorm(h) (1 + scale) + shift in front of a linear is  rstd * W (h (1 + scale)) + W shift.  The elementwise
//         product is what the launch before wrote as x; rstd needs its sums of squares and W * shift is a constant vector.
//   out:  (kEpiResidual) the launch that ends a residual branch writes h, h (1 + scale) and the sums of squares itself.
// Between them no launch has to see a whole row before it can start, and the row kernel that stood there is gone.
struct NormUnit {
    float rstd;
    float4 shift_a, shift_b;
    uint2 res, gate, scale, h, cos, sin;

    template <bool kPairs>
    __device__ __forceinline__ void load(const W4gParams& P, int m, int n, int n2) {
        if (P.in_sumsq != nullptr) {
            const float4* sp = reinterpret_cast<const float4*>(P.in_sumsq + static_cast<size_t>(m) * P.in_parts);
            float4 a = sp[0];
            for (int i = 1; i < P.in_parts / 4; ++i) {
                const float4 f = sp[i];
                a.x += f.x; a.y += f.y; a.z += f.z; a.w += f.w;
            }
            rstd = rsqrtf(((a.x + a.y) + (a.z + a.w)) * P.in_inv_k + P.in_eps);
            shift_a = shift_b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (P.in_shift != nullptr) {
                shift_a = *reinterpret_cast<const float4*>(P.in_shift + n);
                if (kPairs) shift_b = *reinterpret_cast<const float4*>(P.in_shift + n2);
            }
        }
        if (kPairs && P.epilogue == kEpiQkv && n < P.q_dim + 256) {  // a Q or K head: 128-row tiles, two per head
            const size_t p = static_cast<size_t>(P.positions[m]) * 128 + (n >> 7 & 1) * 64 + (n & 63);
            cos = *reinterpret_cast<const uint2*>(P.rope_cos + p);
            sin = *reinterpret_cast<const uint2*>(P.rope_sin + p);
        }
        if (!kPairs && P.epilogue == kEpiResidual) {
            if (P.res != nullptr) res = *reinterpret_cast<const uint2*>(P.res + static_cast<size_t>(m) * P.N + n);
            if (P.gate != nullptr) gate = *reinterpret_cast<const uint2*>(P.gate + n);
            scale = *reinterpret_cast<const uint2*>(P.scale + n);
        }
    }
    __device__ __forceinline__ void apply(const W4gParams& P, const float4& s, float (&v)[4]) const {
        if (P.in_sumsq == nullptr) return;
        v[0] = fmaf(v[0], rstd, s.x);
        v[1] = fmaf(v[1], rstd, s.y);
        v[2] = fmaf(v[2], rstd, s.z);
        v[3] = fmaf(v[3], rstd, s.w);
    }
    // y (this linear's output) -> h, and in `v` the next norm's input; returns the token's sum of h^2 over the tile's 128
    // rows, which are the 32 lanes of a warp
    __device__ __forceinline__ float residual(const W4gParams& P, float (&v)[4]) {
        float r[4], s[4], ss = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = bf16r(v[e]);
        if (P.gate != nullptr) {
            float g[4];
            unpack4(gate, g);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = bf16r(v[e] * g[e]);
        }
        if (P.res != nullptr) {
            unpack4(res, r);
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = bf16r(r[e] + v[e]);
        }
        h = pack4(v);
        unpack4(scale, s);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            ss = fmaf(v[e], v[e], ss);
            v[e] *= 1.0f + s[e];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        return ss;
    }
};

// What the epilogue will read besides the sums, brought into the SM's L1 by one warp that has nothing else left to do: read
// first behind the last barrier, these lines (some from HBM) were 1.2 us of a 6 us launch.  Vectors that are parameters of
// the launch like the weights come before griddepcontrol.wait, rows of the launches before it behind it.
__device__ __forceinline__ void touch_parameters(const W4gParams& P, int row_a, int row_b, int lane) {
    const int row = (lane < 16 ? row_a : row_b) + (lane & 15) * 4;   // 64 rows from row_a, 64 from row_b
    if (P.in_shift != nullptr && row < P.N && (lane & 7) == 0) touch(P.in_shift + row);
    if (P.epilogue == kEpiResidual && (lane & 15) == 0) {
        touch(P.scale + row);
        if (P.gate != nullptr) touch(P.gate + row);
    }
}
__device__ __forceinline__ void touch_rows(const W4gParams& P, int row_a, int m0, int m1, int lane) {
    for (int m = m0 + lane; m < m1; m += 32) {
        if (P.in_sumsq != nullptr) touch(P.in_sumsq + static_cast<size_t>(m) * P.in_parts);
        if (P.epilogue == kEpiResidual && P.res != nullptr) {
            touch(P.res + static_cast<size_t>(m) * P.N + row_a);
            touch(P.res + static_cast<size_t>(m) * P.N + row_a + 64);
        }
        if (P.epilogue == kEpiQkv && row_a < P.q_dim + 256) {
            const size_t p = static_cast<size_t>(P.positions[m]) * 128 + (row_a >> 7 & 1) * 64;
            touch(P.rope_cos + p);
            touch(P.rope_sin + p);
        }
    }
}

// Tiles that no other CTA adds to go from tensor memory to the result by the warps that hold them, without a barrier.  A
// warp has 32 rows of W (its lanes) for 32 tokens; 16-bit results are turned through 2 KB of its own shared memory so that
// a lane stores 8 neighbouring rows of a token: a 128 x 240 tile is 128 stores of 512 bytes a warp.  (The tile staged as
// fp32, a barrier and a second pass over it: 4.0 us of the tile's 18; 16 stores of 64 bytes straight from the
// registers: 3.2; this: 2.3.)
// kDtype -1: any type, with beta.
template <int kDtype>
__device__ __forceinline__ void store_columns(const W4gParams& P, uint32_t lane_addr, int c_first, int c_step, int t0, int valid,
                                              int row0, float bias, uint8_t* buf, int lane) {
    auto result = [&](int col, float (&v)[16]) {                             // 16 columns at a time: 64 registers a thread in all
        uint32_t raw[16];
        tmem_ld_32x32b_x16(lane_addr + col, raw);
        tc::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = fmaf(__uint_as_float(raw[e]), P.alpha, bias);
        if (P.activation == TPB200_ACT_GELU) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = act_fast(v[e], TPB200_ACT_GELU);
        } else if (P.activation == TPB200_ACT_SILU) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = act_fast(v[e], TPB200_ACT_SILU);
        }
    };
    // 16-byte chunk c (8 tokens) of row n lies at c ^ key(n): the lanes' stores and the transposing loads hit all banks
    auto key = [](int n) { return ((n >> 3) ^ (n >> 1)) & 3; };
    const int tn = 8 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);     // the row whose address this lane gives to ldmatrix
    for (int c0 = c_first; c0 < valid; c0 += c_step) {
        if constexpr (kDtype == TPB200_BF16 || kDtype == TPB200_F16) {
            __syncwarp();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float v[16];
                result(c0 + 16 * half, v);
                uint32_t w[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    if (kDtype == TPB200_BF16) {
                        w[e] = bits(__floats2bfloat162_rn(v[2 * e], v[2 * e + 1]));
                    } else {
                        const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
                        w[e] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    *reinterpret_cast<uint4*>(buf + lane * 64 + (((2 * half + c) ^ key(lane)) << 4)) =
                        make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
                }
            }
            __syncwarp();
            const int n = row0 + 8 * (lane & 3);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t q[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                             : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3])
                             : "r"(smem_u32(buf + tn * 64 + ((c ^ key(tn)) << 4)))
                             : "memory");
                const int t = c0 + 8 * c + (lane >> 2);
                if (t < valid && n < P.N) {                          // N is a multiple of 8
                    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(P.out) + static_cast<size_t>(t0 + t) * P.ldo + n) =
                        make_uint4(q[0], q[1], q[2], q[3]);
                }
            }
        } else {
            for (int half = 0; half < 2; ++half) {
                float v[16];
                result(c0 + 16 * half, v);
                size_t o = static_cast<size_t>(t0 + c0 + 16 * half) * P.ldo + row0 + lane;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    if (row0 + lane < P.N && c0 + 16 * half + e < valid) {
                        if (kDtype == TPB200_F32) {
                            static_cast<float*>(P.out)[o] = v[e];
                        } else {
                            const float y = fmaf(P.beta, load_as_float(P.out, P.out_dtype, o), v[e]);
                            if (P.out_dtype == TPB200_BF16) static_cast<__nv_bfloat16*>(P.out)[o] = __float2bfloat16_rn(y);
                            else if (P.out_dtype == TPB200_F16) static_cast<__half*>(P.out)[o] = __float2half_rn(y);
                            else static_cast<float*>(P.out)[o] = y;
                        }
                    }
                    o += P.ldo;
                }
            }
        }
    }
}

template <int kFmt, bool kDirect>
__device__ __forceinline__ void w4_gemm_tile(const W4gParams& P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sW = smem;                                              // [n_w][16 KB codes | 2 scale slabs]
    uint8_t* sB = sW + P.n_w * kWSlot;                               // [n_b][nt rows of 128 bytes]
    const int part_bytes = P.nt * 128, step_parts = P.parts * P.merge, b_bytes = part_bytes * step_parts;
    __shared__ W4gControl ctl;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp-uniform, and known to be
    const int splits = kDirect ? 1 : P.splits;
    const int tile = blockIdx.x / splits;
    const int rank = blockIdx.x - tile * splits;                     // K range
    const int groups = ((blockDim.x >> 5) - kDqWarp0) >> 2;          // of four dequantisation warps
    const int t0 = blockIdx.y * P.nt;                                // first token
    const int blk0 = rank * P.k_blocks / splits, blk1 = (rank + 1) * P.k_blocks / splits;
    const int nblk = blk1 - blk0;
    const int parts = P.parts, merge = P.merge;                      // a part past the end of K multiplies zeros
    const int steps = (min(blk1 * 4, P.k_steps) - blk0 * 4 + step_parts - 1) / step_parts;
    // weight rows of the tile: rows 0..63 start at row_a, 64..127 at row_b (apart only in the gated form)
    const bool gated = !kDirect && kFmt == kFmtNvfp4 && P.epilogue == kEpiGated;
    const int row_a = gated ? tile * 64 : tile * kRows;
    const int row_b = gated ? P.gated_rows + row_a : row_a + 64;

    if (threadIdx.x == 0) {
        for (int s = 0; s < P.n_w; ++s) {
            mbar_init(&ctl.w_full[s], 1);
            mbar_init(&ctl.w_empty[s], 16 / P.parts);                // 4 or 2 steps x 4 warps
        }
        for (int s = 0; s < P.n_s; ++s) {
            mbar_init(&ctl.full[s], 1 + 4 * merge);                  // the activation tiles and four dequantising warps a unit
            mbar_init(&ctl.empty[s], 1);
        }
        mbar_init(&ctl.acc_full, 1);
        ctl.failed = 0;
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        __syncwarp();
        tc::tmem_alloc(&ctl.tmem_base, P.tmem_cols);
        tc::tmem_relinquish();
    }
    if (warp == kXWarp && lane == 0) tc::prefetch_tensormap(&P.map_x);
    if (warp == kWWarp && lane == 0 && P.image == nullptr) tc::prefetch_tensormap(&P.map_w);
    tc::fence_before_thread_sync();
    __syncthreads();
    tc::fence_after_thread_sync();
    const uint32_t tmem = ctl.tmem_base;
    pdl_launch_dependents();

    if (warp == kXWarp) {
        // ------------------------------------------------------------ activation tiles
        if (lane == 0) {
            pdl_wait_prior_grids();
            int s = 0, ph = 1;
            for (int i = 0; i < steps; ++i) {
                if (i >= P.n_s && !mbar_wait_bounded(&ctl.empty[s], ph, kWaitG)) {
                    give_up(ctl, kErrGemmEmptyBarrierTimeout);
                    break;
                }
                mbar_expect_tx(&ctl.full[s], b_bytes);
                for (int u = 0; u < step_parts; ++u) {
                    tc::tma_load_2d(sB + s * b_bytes + u * part_bytes, &P.map_x, (blk0 * 4 + i * step_parts + u) * kPartK, t0,
                                    &ctl.full[s]);
                }
                if (++s == P.n_s) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == kWWarp) {
        // ------------------------------------------------------------ weight blocks
        const uint64_t policy = l2_policy_evict_first();
        const uint32_t bytes = kFmt == kFmtNvfp4 ? (gated ? kCodeBytes + 2 * kSlabBytes : kCodeBytes + kSlabBytes)
                               : kFmt == kFmtNvfp4T || (kFmt == kFmtKblock && P.kb_scale == nullptr) ? kCodeBytes + kSlabBytes
                                                                                                      : kCodeBytes;
        for (int j = 0; j < nblk; ++j) {
            const int s = j % P.n_w, kb = blk0 + j;
            uint8_t* slot = sW + s * kWSlot;
            if (j >= P.n_w && !__all_sync(0xffffffffu, mbar_wait_bounded(&ctl.w_empty[s], ((j / P.n_w) - 1) & 1, kWaitG))) {
                if (lane == 0) give_up(ctl, kErrGemmEmptyBarrierTimeout);
                break;                                               // the slot may still be read
            }
            if (lane == 0) mbar_expect_tx(&ctl.w_full[s], bytes);
            __syncwarp();
            // the requests of a block leave from different lanes: one lane needs ~0.3 us per request
            if (kFmt == kFmtNvfp4) {
                const int half = lane & 1, row = half ? row_b : row_a;
                if (lane < 2) {
                    if (P.image != nullptr) {
                        const uint8_t* b = P.image + (static_cast<size_t>(row >> 8) * P.img_kblocks + kb) * 36864;
                        bulk_copy_g2s_hint(slot + half * 8192, b + (row & 255) * 128, 8192, &ctl.w_full[s], policy);
                    } else {
                        tc::tma_load_2d(slot + half * 8192, &P.map_w, kb * 128, row, &ctl.w_full[s]);
                    }
                } else if (lane < (gated ? 4 : 3)) {
                    const uint8_t* src = P.image != nullptr
                                             ? P.image + (static_cast<size_t>(row >> 8) * P.img_kblocks + kb) * 36864 + 32768 +
                                                   ((row >> 7) & 1) * kSlabBytes
                                             : P.sf + (static_cast<size_t>(row >> 7) * P.img_kblocks + kb) * kSlabBytes;
                    bulk_copy_g2s_hint(slot + kCodeBytes + half * kSlabBytes, src, kSlabBytes, &ctl.w_full[s], policy);
                }
            } else if (kFmt == kFmtNvfp4T) {                         // [128 code bytes of K][128 rows], [16 scales][128 rows]
                if (lane == 0) tc::tma_load_2d(slot, &P.map_w, row_a, kb * 128, &ctl.w_full[s]);
                if (lane == 1) tc::tma_load_2d(slot + kCodeBytes, &P.map_s, row_a, kb * 16, &ctl.w_full[s]);
            } else if (kFmt == kFmtKblock) {
                if (lane == 0) tc::tma_load_2d(slot, &P.map_w, row_a * 2, kb * 8, &ctl.w_full[s]);
                if (lane == 1 && P.kb_scale == nullptr) tc::tma_load_2d(slot + kCodeBytes, &P.map_s, row_a, kb * 8, &ctl.w_full[s]);
            } else {
                if (lane < 2) tc::tma_load_2d(slot + lane * 8192, &P.map_w, kb * 128, lane ? row_b : row_a, &ctl.w_full[s]);
            }
            __syncwarp();
        }
        if (kFmt == kFmtNvfp4 && !kDirect) {
            touch_parameters(P, row_a, row_b, lane);
            pdl_wait_prior_grids();
            const int valid = min(P.nt, P.M - t0);
            touch_rows(P, row_a, t0 + rank * valid / splits, t0 + (rank + 1) * valid / splits, lane);
        }
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------ MMA issue
        // The whole warp walks the loop and one elected lane issues: with warp-uniform control flow the operands of
        // tcgen05.mma stay in uniform registers.  Under `if (lane == 0)` every MMA and commit took ~70 cycles to issue
        // and this one thread was the kernel's critical path (750 cycles per 64-K step for 128-480 cycles of MMA).
        {
            const uint32_t idesc = idesc_bf16(P.nt);
            const uint32_t b16 = (smem_u32(sB) & 0x3FFFFu) >> 4;      // without the bits that name the CTA in its cluster
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            int s = 0, ph = 0;
            for (int i = 0; i < steps; ++i) {
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&ctl.full[s], ph, kWaitG))) {
                    if (lane == 0) give_up(ctl, kErrGemmTmaBarrierTimeout);
                    break;
                }
                tc::fence_after_thread_sync();
                const uint32_t a_col = tm + P.a_col + s * 32 * step_parts, b_lo = b16 + ((s * b_bytes) >> 4), pb = part_bytes >> 4;
                if (tc::elect_one()) {
                    mma_part(tm, a_col, b_lo, idesc, i > 0 ? 1u : 0u);
                    if (step_parts >= 2) mma_part(tm, a_col + 32, b_lo + pb, idesc, 1u);
                    if (step_parts == 4) {
                        mma_part(tm, a_col + 64, b_lo + 2 * pb, idesc, 1u);
                        mma_part(tm, a_col + 96, b_lo + 3 * pb, idesc, 1u);
                    }
                    tc::commit(&ctl.empty[s]);
                }
                __syncwarp();
                if (++s == P.n_s) { s = 0; ph ^= 1; }
            }
            if (tc::elect_one()) tc::commit(&ctl.acc_full);
        }
    } else {
        // ------------------------------------------------------------ codes -> bf16 -> tensor memory; thread = weight row
        const int grp = (warp - kDqWarp0) >> 2;                      // takes every groups-th K step
        const int r = (warp & 3) * 32 + lane;                        // the lanes of tensor memory this warp can reach
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        const int row = r < 64 ? row_a + r : row_b + r - 64;
        const int sf_off = (r >= 64 && gated ? kSlabBytes : 0) + (row & 31) * 16 + ((row >> 5) & 3) * 4;
        bool ok = true;
        float psc[2] = {0.0f, 0.0f}, pzp[2] = {0.0f, 0.0f};
        // Ring positions and phases of this group's units, kept by counting: the loop is bound by instruction issue (of ~420
        // instructions per part and warp once, 220 were the arithmetic).
        int sw = 0, wph = 0, next_j = 1, sa = 0, sub = grp, sph = 1;   // weight slot and phase; operand slot, unit in it, empty phase
        bool fresh = true;                                           // no operand slot has been used twice yet
        auto settle = [&] {
            while (sub >= merge) {
                sub -= merge;
                if (++sa == P.n_s) { sa = 0; sph ^= 1; fresh = false; }
            }
        };
        settle();
        const uint32_t code_off = kFmt == kFmtKblock ? r * 16 : r * 128 + ((r & 7) << 4);
        const int live = P.k_steps - blk0 * 4;                       // parts before the end of K
        uint8_t* slot = sW;
        for (int i = grp; i < steps * merge; i += groups) {
            const int p0 = i * parts;
            while (next_j <= p0 >> 2) {
                ++next_j;
                slot += kWSlot;
                if (++sw == P.n_w) { sw = 0; wph ^= 1; slot = sW; }
            }
            // asked before the arithmetic, used behind it: by then the slot is mostly free and the answer there
            const bool slot_free = fresh || mbar_test_wait(&ctl.empty[sa], sph);
            // The plugin's scales, two per 256 K and one for all parts of a unit, come straight from global memory: asked for before
            // the codes are waited for.  (Behind the wait, once per part: 20 x 13624 x 3968 25.0 us, here 23.4.)
            if (kFmt == kFmtPlugin && row < P.N && p0 < live) {
                const size_t g = static_cast<size_t>(row) * (P.K / 128) + (blk0 + (p0 >> 2)) * 2 + ((p0 & 3) >> 1);
                psc[0] = __bfloat162float(__ldg(P.pl_scale + g));
                pzp[0] = P.pl_zero != nullptr ? __bfloat162float(__ldg(P.pl_zero + g)) : 0.0f;
            }
            if (!mbar_wait_bounded(&ctl.w_full[sw], wph, kWaitG)) ok = false;
            for (int u = 0; u < parts; ++u) {
                const int kk = (p0 + u) & 3;
                const bool past = p0 + u >= live;                    // of an operand step's last parts only: zeros
                uint32_t out[32];
                uint4 c[2];
                if (kFmt == kFmtNvfp4T) {                            // a row's codes lie 128 bytes apart
                    uint32_t* cw = reinterpret_cast<uint32_t*>(c);
#pragma unroll
                    for (int wd = 0; wd < 8; ++wd) {
                        const uint8_t* p4 = slot + (32 * kk + 4 * wd) * kRows + r;
                        cw[wd] = p4[0] | p4[kRows] << 8 | p4[2 * kRows] << 16 | static_cast<uint32_t>(p4[3 * kRows]) << 24;
                    }
                } else if (kFmt == kFmtKblock) {
                    const uint8_t* p16 = slot + code_off + kk * 4096;
                    c[0] = *reinterpret_cast<const uint4*>(p16);
                    c[1] = *reinterpret_cast<const uint4*>(p16 + 2048);
                } else {                                             // 16-byte chunks 2 kk, 2 kk + 1 of the row, each XOR r & 7
                    const uint32_t o16 = code_off ^ (kk << 5);
                    c[0] = *reinterpret_cast<const uint4*>(slot + o16);
                    c[1] = *reinterpret_cast<const uint4*>(slot + (o16 ^ 16));
                }
                uint32_t sc = 0;
                if (kFmt == kFmtNvfp4) sc = *reinterpret_cast<const uint32_t*>(slot + kCodeBytes + kk * 512 + sf_off);
                if (kFmt == kFmtNvfp4T) {
                    const uint8_t* p4 = slot + kCodeBytes + 4 * kk * kRows + r;
                    sc = p4[0] | p4[kRows] << 8 | p4[2 * kRows] << 16 | static_cast<uint32_t>(p4[3 * kRows]) << 24;
                }
                if (kFmt == kFmtKblock) {
                    if (P.kb_scale == nullptr) {
                        const __half* sp = reinterpret_cast<const __half*>(slot + kCodeBytes) + (2 * kk) * kRows + r;
                        psc[0] = __half2float(sp[0]);
                        psc[1] = __half2float(sp[kRows]);
                    } else if (row < P.N && !past) {
                        const __half* sp = P.kb_scale + static_cast<size_t>((blk0 + (p0 >> 2)) * 8 + 2 * kk) * P.N + row;
                        psc[0] = __half2float(__ldg(sp));
                        psc[1] = __half2float(__ldg(sp + P.N));
                    }
                }
                if (past) {                                          // codes and scales of zero: zeros, whatever the slot holds
                    c[0] = c[1] = make_uint4(0, 0, 0, 0);
                    sc = 0;
                    psc[0] = psc[1] = pzp[0] = 0.0f;
                }
                if (u == parts - 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl.w_empty[sw]);        // every lane's codes are in registers
                }
                const uint32_t w[8] = {c[0].x, c[0].y, c[0].z, c[0].w, c[1].x, c[1].y, c[1].z, c[1].w};
                if (kFmt == kFmtNvfp4 || kFmt == kFmtNvfp4T) {
                    const __half2 s01 = decode_e4m3x2_h(static_cast<uint16_t>(sc)), s23 = decode_e4m3x2_h(static_cast<uint16_t>(sc >> 16));
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const __half2 s2 = b < 2 ? (b ? __high2half2(s01) : __low2half2(s01)) : b == 3 ? __high2half2(s23) : __low2half2(s23);
                        dequant_e2m1x8(w[2 * b], s2, out + 8 * b);
                        dequant_e2m1x8(w[2 * b + 1], s2, out + 8 * b + 4);
                    }
                } else {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const float s = kFmt == kFmtKblock ? psc[b] : psc[0];
                        const __nv_bfloat162 s_hi = __float2bfloat162_rn(s);
                        const __nv_bfloat162 s_lo = __float2bfloat162_rn(s - __low2float(s_hi));
                        const __nv_bfloat162 zp = __float2bfloat162_rn(pzp[0]);
#pragma unroll
                        for (int wd = 0; wd < 4; ++wd) {
                            __nv_bfloat162 q[4];
                            nibbles_minus8(w[4 * b + wd] ^ (kFmt == kFmtPlugin ? 0x88888888u : 0u), q);
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                out[16 * b + 4 * wd + e] = kFmt == kFmtKblock ? bits(__hfma2(q[e], s_hi, __hmul2(q[e], s_lo)))
                                                                             : bits(__hfma2(q[e], s_hi, zp));
                            }
                        }
                    }
                }
                if (u == 0) {                                        // the arithmetic above needs no free slot
                    if (!slot_free && !mbar_wait_bounded(&ctl.empty[sa], sph, kWaitG)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc::fence_after_thread_sync();
                }
                __syncwarp();                                        // lane 0 may be behind: it has arrived on w_empty
                tmem_st_32x32b_x32(lane_addr + P.a_col + (sa * step_parts + sub * parts + u) * 32, out);
            }
            if (!ok) {
                if (lane == 0) give_up(ctl, kErrGemmEmptyBarrierTimeout);
                break;
            }
            tmem_st_wait();
            tc::fence_before_thread_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl.full[sa]);
            sub += groups;
            settle();
        }
        // ------------------------------------------------------------ accumulator -> result, or -> shared memory
        float bias = 0.0f;
        if (kDirect) {
            pdl_wait_prior_grids();                                  // long over by now; orders the stores (and reads of `out`)
            if (P.bias != nullptr && row < P.N) bias = load_as_float(P.bias, P.bias_dtype, row);
        }
        if (ok && !mbar_wait_bounded(&ctl.acc_full, 0, kWaitG)) {
            give_up(ctl, kErrGemmMmaBarrierTimeout);
            ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc::fence_after_thread_sync();
            const int valid = min(P.nt, P.M - t0);
            if constexpr (kDirect) {
                if (*static_cast<volatile int*>(&ctl.failed) == 0) {
                    uint8_t* buf = smem + (warp - kDqWarp0) * 2048;  // the rings: every slot has been consumed
                    const int row0 = row_a + (warp & 3) * 32;
                    if (P.beta != 0.0f) store_columns<-1>(P, lane_addr, grp * 32, groups * 32, t0, valid, row0, bias, buf, lane);
                    else if (P.out_dtype == TPB200_BF16) store_columns<TPB200_BF16>(P, lane_addr, grp * 32, groups * 32, t0, valid, row0, bias, buf, lane);
                    else if (P.out_dtype == TPB200_F16) store_columns<TPB200_F16>(P, lane_addr, grp * 32, groups * 32, t0, valid, row0, bias, buf, lane);
                    else store_columns<TPB200_F32>(P, lane_addr, grp * 32, groups * 32, t0, valid, row0, bias, buf, lane);
                }
            } else {
                float* st = reinterpret_cast<float*>(smem);          // every ring slot has been consumed; [token][128 rows]
                for (int c0 = grp * 16; c0 < valid; c0 += groups * 16) {
                    uint32_t v[16];
                    tmem_ld_32x32b_x16(lane_addr + c0, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        if (c0 + e < valid) st[(c0 + e) * kRows + r] = __uint_as_float(v[e]);
                    }
                }
            }
        }
        tc::fence_before_thread_sync();
    }

    pdl_wait_prior_grids();                                          // a no-op by now; orders reads of `out` (beta) and of the norms' inputs
    const int valid = min(P.nt, P.M - t0);
    const int tb = rank * valid / splits, te = (rank + 1) * valid / splits;
    // A unit of the epilogue is a token x 4 weight rows (4 + 4 where rows come in pairs): neighbouring lanes read and write
    // neighbouring 16 and 8 bytes.
    const bool pairs = kFmt == kFmtNvfp4 && (P.epilogue == kEpiGated || P.epilogue == kEpiQkv);
    const int per_token = pairs ? 16 : 32;
    const int u_first = tb * per_token + threadIdx.x, u_end = te * per_token;

    if (splits > 1) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        __syncwarp();
        tc::fence_after_thread_sync();
        tc::tmem_dealloc(tmem, P.tmem_cols);
    }

    // ---------------------------------------------------------------- this CTA's share of the tokens, all 128 rows
    const bool failed = ctl.failed != 0;                             // then nothing is stored
    {
        const uint32_t base = smem_u32(smem);
        auto sum4 = [&](int t, int c, float (&v)[4]) {
            const uint32_t off = static_cast<uint32_t>((t * kRows + c) * 4);
            float4 a;
            if (splits == 1) a = *reinterpret_cast<const float4*>(smem + off);
            else if (splits == 2) a = sum_ranks<2>(base, off, 2);
            else if (splits <= 4) a = sum_ranks<4>(base, off, splits);
            else a = sum_ranks<8>(base, off, splits);
            v[0] = a.x * P.alpha; v[1] = a.y * P.alpha; v[2] = a.z * P.alpha; v[3] = a.w * P.alpha;
        };
        if constexpr (kDirect) {
            // stored by the warps that read the accumulator
        } else if (!pairs) {
            for (int u = u_first; u < u_end; u += static_cast<int>(blockDim.x)) {
                const int t = u >> 5, c = (u & 31) * 4, n = row_a + c;
                if (n >= P.N) continue;                              // N is a multiple of 8
                float v[4];
                NormUnit nu;
                if (kFmt == kFmtNvfp4) nu.load<false>(P, t0 + t, n, 0);
                sum4(t, c, v);
                if (kFmt == kFmtNvfp4) nu.apply(P, nu.shift_a, v);
                if (P.bias != nullptr) {
                    if (P.bias_dtype == TPB200_F32 && (reinterpret_cast<uintptr_t>(P.bias) & 15) == 0) {
                        const float4 b0 = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(P.bias) + n));
                        v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[e] += load_as_float(P.bias, P.bias_dtype, n + e);
                    }
                }
                act4(v, P.activation);
                if (kFmt == kFmtNvfp4 && P.epilogue == kEpiResidual) {
                    // h = res + y * gate and the next norm's input h * (1 + scale), each rounded to bf16 (N % 128 == 0: all
                    // 32 lanes are here)
                    const float ss = nu.residual(P, v);
                    if (failed) continue;
                    *reinterpret_cast<uint2*>(P.h_out + static_cast<size_t>(t0 + t) * P.N + n) = nu.h;
                    if ((threadIdx.x & 31) == 0) P.out_sumsq[static_cast<size_t>(t0 + t) * (P.N / kRows) + tile] = ss;
                }
                if (failed) continue;                                // asked here: the flag arrives beside the sums
                const size_t o = static_cast<size_t>(t0 + t) * P.ldo + n;
                if (P.beta != 0.0f) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = fmaf(P.beta, load_as_float(P.out, P.out_dtype, o + e), v[e]);
                }
                if (kFmt == kFmtNvfp4 && P.copy_out != nullptr) {
                    *reinterpret_cast<uint2*>(P.copy_out + static_cast<size_t>(t0 + t) * P.N + n) = pack4(v);
                }
                if (P.out_dtype == TPB200_BF16) {
                    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(P.out) + o) = pack4(v);
                } else if (P.out_dtype == TPB200_F32) {
                    *reinterpret_cast<float4*>(static_cast<float*>(P.out) + o) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
                    const __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
                    *reinterpret_cast<uint2*>(static_cast<__half*>(P.out) + o) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
                }
            }
        } else if (P.epilogue == kEpiGated) {
            // gate rows 0..63, up rows 64..127 of the tile; the roundings of the module: both projections, the
            // activation and the product go to bf16
            for (int u = u_first; u < u_end; u += static_cast<int>(blockDim.x)) {
                const int t = u >> 4, c = (u & 15) * 4;
                float g[4], up[4];
                NormUnit nu;
                if (kFmt == kFmtNvfp4) nu.load<true>(P, t0 + t, row_a + c, row_b + c);
                sum4(t, c, g);
                sum4(t, c + 64, up);
                if (kFmt == kFmtNvfp4) {
                    nu.apply(P, nu.shift_a, g);
                    nu.apply(P, nu.shift_b, up);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) g[e] = bf16r(g[e]);
                act4(g, P.activation);
#pragma unroll
                for (int e = 0; e < 4; ++e) g[e] = bf16r(g[e]) * bf16r(up[e]);
                if (failed) continue;
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(P.out) + static_cast<size_t>(t0 + t) * P.ldo + row_a + c) =
                    pack4(g);
            }
        } else {
            // rows 0..63 of the tile are head offsets i, rows 64..127 their rotate-half partners i + 128; the rotation
            // in bf16, each product and the sum rounded, as torch does it.  V heads pass through.
            const int head = tile >> 1, i0 = (tile & 1) * 64, heads = P.q_dim >> 8;
            for (int u = u_first; u < u_end; u += static_cast<int>(blockDim.x)) {
                const int t = u >> 4, c = (u & 15) * 4, m = t0 + t;
                float lo[4], hi[4];
                NormUnit nu;
                if (kFmt == kFmtNvfp4) nu.load<true>(P, m, row_a + c, row_b + c);
                sum4(t, c, lo);
                sum4(t, c + 64, hi);
                if (kFmt == kFmtNvfp4) {
                    nu.apply(P, nu.shift_a, lo);
                    nu.apply(P, nu.shift_b, hi);
                }
                uint32_t olo[2], ohi[2];
                const uint32_t cw[2] = {nu.cos.x, nu.cos.y}, sw[2] = {nu.sin.x, nu.sin.y};
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    __nv_bfloat162 a = __floats2bfloat162_rn(lo[2 * e], lo[2 * e + 1]);
                    __nv_bfloat162 b = __floats2bfloat162_rn(hi[2 * e], hi[2 * e + 1]);
                    if (head <= heads) {
                        const __nv_bfloat162 co = as_bf162(cw[e]), si = as_bf162(sw[e]);
                        const __nv_bfloat162 ra = __hadd2(__hmul2(a, co), __hmul2(__hneg2(b), si));
                        const __nv_bfloat162 rb = __hadd2(__hmul2(b, co), __hmul2(a, si));
                        a = ra;
                        b = rb;
                    }
                    olo[e] = bits(a);
                    ohi[e] = bits(b);
                }
                if (failed) continue;
                __nv_bfloat16* dst = head < heads ? static_cast<__nv_bfloat16*>(P.out) + static_cast<size_t>(m) * P.ldq + head * 256
                                     : (head == heads ? P.k_rows : P.v_rows) + static_cast<size_t>(m) * 256;
                *reinterpret_cast<uint2*>(dst + i0 + c) = make_uint2(olo[0], olo[1]);
                *reinterpret_cast<uint2*>(dst + i0 + c + 128) = make_uint2(ohi[0], ohi[1]);
            }
        }
    }
    if (failed) {
        // The CTA stays until the copies it has requested (microseconds of work) have landed: its shared memory goes to
        // another CTA afterwards.
        const long long start = clock64();
        while (clock64() - start < kLandCycles) __nanosleep(1000);
    }
    if (splits > 1) {                                                // nobody leaves while a peer still reads its sums
        __syncwarp();
        cluster_arrive_relaxed();                                    // its loads have returned; the stores need not land first
        cluster_wait();
    }
}

// at most 93 registers: two CTAs of 352 threads, or one of 608, fit an SM
constexpr int kBoundThreads = 704;
template <bool kDirect>
__global__ void __launch_bounds__(kBoundThreads, 1) w4_nvfp4_gemm_kernel(const __grid_constant__ W4gParams P) {
    w4_gemm_tile<kFmtNvfp4, kDirect>(P);
}
template <bool kDirect>
__global__ void __launch_bounds__(kBoundThreads, 1) w4_nvfp4_gemm_kernel_transposed(const __grid_constant__ W4gParams P) {
    w4_gemm_tile<kFmtNvfp4T, kDirect>(P);
}
template <bool kDirect>
__global__ void __launch_bounds__(kBoundThreads, 1) w4_int4_kblock_gemm_kernel(const __grid_constant__ W4gParams P) {
    w4_gemm_tile<kFmtKblock, kDirect>(P);
}
template <bool kDirect>
__global__ void __launch_bounds__(kBoundThreads, 1) w4_int4_plugin_gemm_kernel(const __grid_constant__ W4gParams P) {
    w4_gemm_tile<kFmtPlugin, kDirect>(P);
}

// ---------------------------------------------------------------- launch plan
// 64-K parts per unit, the share of a weight block that a group of warps dequantises at a time: two where four such units
// (one per group) fit the step ring.  What a unit costs beside its arithmetic (barriers, positions, phases) is ~100
// instructions of a loop that is bound by their issue.
constexpr int unit_parts(int nt, bool half) { return nt <= (half ? 64 : 144) ? 2 : 1; }

// Tokens per tile, K ranges per tile, and whether two CTAs share an SM (8 dequantising warps each) or one has it
// to itself (16 warps).
struct W4gPlan { int nt, splits; bool half; };

// What a launch takes, about in microseconds on a B200; it only has to rank the candidates.  One per weight form, fitted to 665 shapes
// (1 to 1000 tokens, 512 to 32768 rows, K 512 to 16384) with every candidate measured as a plain launch and in a chain of
// programmatic dependent ones.  A shape has one plan for both (a launch flag does not change a result's bits): NVFP4 weighs the
// chains of the modules and the pipeline more, INT4 plain calls; the transposed form is fitted to plain launches alone.  How many K
// ranges NVFP4 weights get is ranked by a cost of its own, good for nothing but that: it decides in which order a result's sums
// are added, and the pipeline hands on fp32 actions that follow every rounding before them, so it is fitted with the condition
// that no linear of the pipeline changes its ranges.  Off the best candidate on average, plain / in a chain: INT4 2.0 / 1.6 %, NVFP4
// 2.3 / 1.8, transposed 0.7.  One model for all forms was 10 / 6, 7 / 4 and 9 % off, 86 % at worst: it had 0.33 us per 64 K for
// two CTAs that share an SM, which take 0.62 with INT4 codes, as long as one after the other (712 x 2048 x 16384: 89 us, 48 as
// planned now).
struct W4gCost {
    // 64 K values: max(a, b + c NT), for a CTA with an SM of its own, two that share one, and the narrow form of a CTA
    // where it has the SM to itself
    float own[3], shared[3], alone[3];
    float unpaired[2];                               // more where a unit is one part only (ring_of), whole and narrow
    float round[2], round_nt[2];                     // per round of CTAs, whole and narrow, and its NT x ...
    float narrow;                                    // a launch of narrow CTAs
    float split[4], split_nt;                        // 1, 2, 4, 8 K ranges: barrier and sums; NT x 512 bytes per CTA move
    float cta;                                       // each of up to 150
    float crowd[2];                                  // a grid of more than half the room leaves the next launch of a chain less to
                                                     // start in: [0] from a share [1] beyond the half on, in proportion before
};
constexpr W4gCost kCostNvfp4Ranges = {{0.246f, 0.0f, 0.0012f}, {1.96f, 0.0f, 0.0f}, {0.303f, 0.0283f, 0.00875f},
    {0.0f, 0.133f}, {6.66f, 1.95f}, {0.0138f, 0.0384f}, 1.9f,
    {0.0f, 0.7f, 1.89f, 1.87f}, 0.0295f, 0.0203f, {1.28f, 0.516f}};
constexpr W4gCost kCostNvfp4 = {{0.0723f, 0.0677f, 0.000111f}, {0.247f, 0.0499f, 0.000327f}, {0.00406f, 0.119f, 0.00163f},
    {0.00399f, 0.00399f}, {3.93f, 2.74f}, {0.014f, 0.0149f}, 0.32f,
    {0.0f, 0.112f, 0.0622f, 0.0429f}, 0.00508f, 0.00958f, {0.638f, 0.214f}};
constexpr W4gCost kCostInt4 = {{0.00801f, 0.13f, 0.000399f}, {0.431f, 0.0927f, 0.000306f}, {0.303f, 0.139f, 0.00361f},
    {0.0027f, 0.0027f}, {2.09f, 0.0589f}, {0.0176f, 0.033f}, -0.11f,
    {0.0f, 0.02f, 0.0365f, 0.0585f}, 0.00405f, 0.0133f, {1.34f, 0.0866f}};
constexpr W4gCost kCostTransposed = {{0.308f, 0.0662f, 0.00107f}, {0.744f, 0.332f, 0.00168f}, {0.347f, 0.0999f, 0.00141f},
    {0.0599f, 0.0599f}, {5.9f, 6.86f}, {0.0382f, 0.0202f}, 0.574f,
    {0.0f, 0.361f, 0.131f, -0.147f}, 0.00485f, 0.0121f, {0.0f, 1.0f}};

// Clusters of 1, 2, 4 and 8 CTAs that run at once with an SM each (GPCs of 16 to 20 SMs hold whole clusters only), as
// cudaOccupancyMaxActiveClusters has it for every one of these kernels.  Two narrow CTAs do share an SM: times step where
// twice as many clusters are exceeded (296 CTAs, 148 pairs, 66 fours).  The occupancy calls cannot be asked for that: they allow
// a kernel that allocates tensor memory one CTA per SM.
constexpr int kFit[4] = {148, 74, 33, 15};

// The cheapest plan, of `ranges` K ranges where that is not 0
W4gPlan cheapest_plan(const W4gCost& C, int tiles, int M, int k_blocks, int sms, int ranges) {
    W4gPlan best{256, 1, false};
    float best_cost = 1e30f;
    for (int nt = 16; nt <= 256; nt += 16) {
        const int tt = (M + nt - 1) / nt;
        if (tt > 65535 || (nt > 16 && (M + nt - 17) / (nt - 16) == tt)) continue;      // a narrower tile does the same
        const long long clusters = static_cast<long long>(tiles) * tt;
        for (int s = 1, l = 0; s <= 8 && s <= k_blocks; s *= 2, ++l) {
            if (ranges != 0 && s != ranges) continue;
            const long long ctas = clusters * s, fit = std::max(1, kFit[l] * sms / 148);
            const int steps = (k_blocks + s - 1) / s * 4;            // parts of 64 K values
            for (int half = 0; half <= (nt <= 128 ? 1 : 0); ++half) {
                auto round = [&](const float (&t)[3]) {
                    const float step = std::max(t[0], t[1] + t[2] * nt) + (unit_parts(nt, half) == 1 ? C.unpaired[half] : 0.0f);
                    return C.round[half] + C.round_nt[half] * nt + steps * step;
                };
                float cost;
                if (half) {                                          // rounds that share SMs; the last one may not need to
                    const long long rounds = clusters / (2 * fit), rest = clusters - rounds * 2 * fit;
                    cost = C.narrow + rounds * round(C.shared) + (rest == 0 ? 0.0f : round(rest <= fit ? C.alone : C.shared));
                } else {
                    cost = (clusters + fit - 1) / fit * round(C.own);
                }
                cost += C.split[l] + (l > 0 ? C.split_nt * nt : 0.0f) + C.cta * std::min(ctas, 150LL);
                const float over = 2.0f * ctas / (sms * (1 + half)) - 1.0f;
                cost += C.crowd[0] * std::min(1.0f, std::max(0.0f, over / C.crowd[1]));
                if (cost < best_cost) {
                    best_cost = cost;
                    best = {nt, s, half != 0};
                }
            }
        }
    }
    return best;
}

W4gPlan plan_w4_gemm(int tiles, int M, int k_blocks, int sms, int fmt) {
    if (fmt != kFmtNvfp4) return cheapest_plan(fmt == kFmtNvfp4T ? kCostTransposed : kCostInt4, tiles, M, k_blocks, sms, 0);
    const int ranges = cheapest_plan(kCostNvfp4Ranges, tiles, M, k_blocks, sms, 0).splits;
    return cheapest_plan(kCostNvfp4, tiles, M, k_blocks, sms, ranges);
}

// The last plans of this thread: a call's host side is a few microseconds, ranking the candidates is one of them.
W4gPlan plan_cached(int tiles, int M, int k_blocks, int sms, int fmt) {
    struct Entry { int tiles, M, k_blocks, sms, fmt; W4gPlan plan; };
    static thread_local Entry cache[32] = {};
    Entry& e = cache[(static_cast<unsigned>(tiles) * 31u + static_cast<unsigned>(M) * 7u + static_cast<unsigned>(k_blocks)) % 32u];
    if (e.tiles != tiles || e.M != M || e.k_blocks != k_blocks || e.sms != sms || e.fmt != fmt) {
        e = {tiles, M, k_blocks, sms, fmt, plan_w4_gemm(tiles, M, k_blocks, sms, fmt)};
    }
    return e.plan;
}

// Ring depths.  Up to 128 tokens: half an SM's shared and tensor memory, so that two CTAs (of this launch or of the
// next one in the stream) share an SM; more tokens: one CTA per SM.
struct W4gRing { int groups, parts, merge, n_w, n_s, tmem_cols, a_col; };

W4gRing ring_of(const W4gPlan& plan, int k_blocks, int k_steps) {
    W4gRing r;
    r.tmem_cols = plan.half ? 256 : 512;
    r.a_col = (plan.nt + 31) / 32 * 32;
    const int blocks_per = (k_blocks + plan.splits - 1) / plan.splits, steps_per = std::min(blocks_per * 4, k_steps);
    const int budget = (plan.half ? 112 : 225) * 1024 - 1024;
    r.parts = unit_parts(plan.nt, plan.half);
    r.groups = plan.half ? 2 : 4;
    // A group takes every `stride`-th weight block.  A parity wait tells a phase from the one before it only, so a group
    // must have waited for EVERY earlier block of a slot it comes to: with more blocks than slots, the number of slots is
    // a multiple of the stride.  (Three slots under a stride of two: a group could take a block's codes out of a slot that
    // was still receiving the block before, and hand the slot back in another group's place.)
    const int stride = std::max(1, r.groups * r.parts / 4);
    const int slots = stride == 2 ? 4 : plan.half && plan.nt > 64 ? 2 : 3;
    static_assert(kMaxW >= 4, "two blocks ahead for each half of the groups");
    r.n_w = std::min(slots, blocks_per);
    auto depth = [&](int merge) {
        const int units = merge * r.parts;
        return std::min(std::min(kMaxS, (r.tmem_cols - r.a_col) / (32 * units)),
                        std::min((steps_per + units - 1) / units, (budget - r.n_w * kWSlot) / (plan.nt * 128 * units)));
    };
    // Two units per operand step where K is long and three such steps fit: handing a step to the tensor cores costs the
    // issuing warp ~250 cycles (barrier, commit, loop) beside 35 per MMA.
    r.merge = steps_per >= 32 && depth(2) >= 3 ? 2 : 1;
    // Operand steps: a group's wait for the MMAs of its previous unit covers every slot's last but one use as long as there
    // is room for a unit of each group (5 units for 256 tokens, the fewest), or no slot is used twice.
    r.n_s = depth(r.merge);
    return r;
}

// Dynamic shared memory: the rings, then the accumulators of the epilogue in their place; K ranges summed inside a cluster
// keep other clusters off the SM if their tensor memory would not fit beside this one's.
int smem_of(const W4gPlan& plan, const W4gRing& r, bool direct) {
    const int rings = r.n_w * kWSlot + r.n_s * plan.nt * 128 * r.parts * r.merge;
    const int smem = std::max(rings, direct ? r.groups * 4 * 2048 : plan.nt * kRows * 4) + 1024;
    return plan.splits > 1 ? std::max(smem, min_smem_of_columns(r.tmem_cols)) : smem;
}

}  // namespace

int device_error_w4_gemm(int clear) { return read_device_error(clear); }

// `transposed` (internal, TPB200_W4_NVFP4_ROWMAJOR only): w = [K / 2, N] code bytes, w_scales = [K / 16, N] UE4M3 bytes, N % 16 == 0
int w4_gemm_launch(const tpb200_w4_gemm_args* a, cudaStream_t stream, bool transposed, const tpb200_w4_norm_args* norm) {
    TPB_REQUIRE(a != nullptr && a->x != nullptr && a->w != nullptr && a->out != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE(a->format >= TPB200_W4_NVFP4_ROWMAJOR && a->format <= TPB200_W4_INT4_PLUGIN, TPB200_ERR_ENUM);
    TPB_REQUIRE((a->flags & ~TPB200_FLAG_PDL) == 0, TPB200_ERR_ENUM);
    TPB_REQUIRE(a->activation >= TPB200_ACT_NONE && a->activation <= TPB200_ACT_SILU, TPB200_ERR_ENUM);
    const int M = a->M, N = a->N, K = a->K;
    const bool nv = a->format == TPB200_W4_NVFP4_ROWMAJOR || a->format == TPB200_W4_NVFP4_TILED;
    const bool qkv = a->qkv_k_rows != nullptr;
    const bool gated = a->gated != 0;
    TPB_REQUIRE(M >= 1 && M <= 65535 * 256 && N >= 8 && N % 8 == 0 && K >= 16, TPB200_ERR_SHAPE);
    TPB_REQUIRE(nv ? K % 16 == 0 : K % 128 == 0, TPB200_ERR_SHAPE);
    TPB_REQUIRE(a->ldx >= K && a->ldx % 8 == 0 && tpb_aligned16(a->x) && tpb_aligned16(a->w) && tpb_aligned16(a->out),
                TPB200_ERR_ALIGN);
    TPB_REQUIRE(a->format != TPB200_W4_NVFP4_ROWMAJOR || tpb_aligned16(a->w_scales), TPB200_ERR_ALIGN);
    TPB_REQUIRE(a->format == TPB200_W4_NVFP4_TILED || a->w_scales != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE(a->w_zeros == nullptr || a->format == TPB200_W4_INT4_PLUGIN, TPB200_ERR_ENUM);
    TPB_REQUIRE(!(qkv && gated) && (nv || (!qkv && !gated)), TPB200_ERR_ENUM);
    if (qkv) {
        TPB_REQUIRE(a->qkv_v_rows && a->qkv_positions && a->qkv_rope_cos && a->qkv_rope_sin, TPB200_ERR_NULL);
        TPB_REQUIRE(a->qkv_q_dim >= 256 && a->qkv_q_dim % 256 == 0 && N == a->qkv_q_dim + 512 && a->ldo >= a->qkv_q_dim &&
                        a->ldo % 8 == 0,
                    TPB200_ERR_SHAPE);
        TPB_REQUIRE(tpb_aligned16(a->qkv_k_rows) && tpb_aligned16(a->qkv_v_rows) && tpb_aligned16(a->qkv_rope_cos) &&
                        tpb_aligned16(a->qkv_rope_sin),
                    TPB200_ERR_ALIGN);
        TPB_REQUIRE(a->out_dtype == TPB200_BF16 && a->bias == nullptr && a->beta == 0.0f && a->activation == TPB200_ACT_NONE,
                    TPB200_ERR_ENUM);
    } else if (gated) {
        TPB_REQUIRE(N % 128 == 0 && a->ldo >= N / 2 && a->ldo % 8 == 0, TPB200_ERR_SHAPE);
        TPB_REQUIRE(a->out_dtype == TPB200_BF16 && a->bias == nullptr && a->beta == 0.0f && a->activation != TPB200_ACT_NONE,
                    TPB200_ERR_ENUM);
    } else {
        TPB_REQUIRE(tpb_valid_dtype(a->out_dtype) && (a->bias == nullptr || tpb_valid_dtype(a->bias_dtype)), TPB200_ERR_ENUM);
        TPB_REQUIRE(a->ldo >= N, TPB200_ERR_SHAPE);
        TPB_REQUIRE(static_cast<long long>(a->ldo) * tpb_dtype_size(a->out_dtype) % 16 == 0, TPB200_ERR_ALIGN);
    }
    const bool norm_in = norm != nullptr && norm->in_sumsq != nullptr, norm_out = norm != nullptr && norm->h_out != nullptr;
    TPB_REQUIRE(norm == nullptr || norm_in || (norm->in_shift == nullptr && norm->copy_out == nullptr), TPB200_ERR_NULL);
    if (norm_in) {
        TPB_REQUIRE(nv, TPB200_ERR_ENUM);
        TPB_REQUIRE(norm->in_parts >= 4 && norm->in_parts % 4 == 0, TPB200_ERR_SHAPE);
        TPB_REQUIRE(tpb_aligned16(norm->in_sumsq) && tpb_aligned16(norm->in_shift), TPB200_ERR_ALIGN);
        TPB_REQUIRE(norm->copy_out == nullptr || (!qkv && !gated && !norm_out), TPB200_ERR_ENUM);
        TPB_REQUIRE(tpb_aligned16(norm->copy_out), TPB200_ERR_ALIGN);
    }
    if (norm_out) {
        TPB_REQUIRE(nv && !qkv && !gated && a->out_dtype == TPB200_BF16 && a->activation == TPB200_ACT_NONE && a->beta == 0.0f,
                    TPB200_ERR_ENUM);
        TPB_REQUIRE(norm->scale != nullptr && norm->out_sumsq != nullptr, TPB200_ERR_NULL);
        TPB_REQUIRE(N % kRows == 0, TPB200_ERR_SHAPE);
        TPB_REQUIRE(tpb_aligned16(norm->h_out) && tpb_aligned16(norm->res_in) && tpb_aligned16(norm->gate) &&
                        tpb_aligned16(norm->scale),
                    TPB200_ERR_ALIGN);
    }
    W4gParams P = {};
    if (norm_in) {
        P.in_sumsq = norm->in_sumsq;
        P.in_shift = norm->in_shift;
        P.in_parts = norm->in_parts;
        P.in_eps = norm->in_eps;
        P.copy_out = static_cast<__nv_bfloat16*>(norm->copy_out);
        P.in_inv_k = 1.0f / static_cast<float>(K);
    }
    if (norm_out) {
        P.res = static_cast<const __nv_bfloat16*>(norm->res_in);
        P.gate = static_cast<const __nv_bfloat16*>(norm->gate);
        P.scale = static_cast<const __nv_bfloat16*>(norm->scale);
        P.h_out = static_cast<__nv_bfloat16*>(norm->h_out);
        P.out_sumsq = norm->out_sumsq;
    }
    TPB_REQUIRE(!transposed || (a->format == TPB200_W4_NVFP4_ROWMAJOR && !qkv && !gated && N % 16 == 0), TPB200_ERR_ENUM);
    const int fmt = transposed ? kFmtNvfp4T : nv ? kFmtNvfp4 : a->format == TPB200_W4_INT4_KBLOCK ? kFmtKblock : kFmtPlugin;
    const int tiles = (N + kRows - 1) / kRows;
    P.k_blocks = (K + kBlkK - 1) / kBlkK;
    P.k_steps = (K + kPartK - 1) / kPartK;
    P.img_kblocks = P.k_blocks;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const W4gPlan plan = plan_cached(tiles, M, P.k_blocks, sms, fmt);
    P.nt = plan.nt;
    P.splits = plan.splits;
    bool ok = make_tensor_map_2d(&P.map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a->x, K, M, static_cast<uint64_t>(a->ldx) * 2, 64,
                                 P.nt, true);
    if (transposed) {
        ok = ok && make_tensor_map_2d(&P.map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, a->w, N, K / 2, N, 128, 128, false) &&
             make_tensor_map_2d(&P.map_s, CU_TENSOR_MAP_DATA_TYPE_UINT8, a->w_scales, N, K / 16, N, 128, 16, false);
    } else if (a->format == TPB200_W4_NVFP4_TILED) {
        P.image = static_cast<const uint8_t*>(a->w);
    } else if (a->format == TPB200_W4_INT4_KBLOCK) {
        ok = ok && make_tensor_map_2d(&P.map_w, CU_TENSOR_MAP_DATA_TYPE_UINT64, a->w, 2ull * N, K / 32, 16ull * N, 256, 8, false);
        if (tpb_aligned16(a->w_scales)) {
            ok = ok && make_tensor_map_2d(&P.map_s, CU_TENSOR_MAP_DATA_TYPE_UINT16, a->w_scales, N, K / 32, 2ull * N, 128, 8, false);
        } else {
            P.kb_scale = static_cast<const __half*>(a->w_scales);
        }
    } else {
        const int pitch = a->format == TPB200_W4_INT4_PLUGIN ? K / 2 : a->w_pitch;
        TPB_REQUIRE(pitch >= K / 2 && pitch % 16 == 0, TPB200_ERR_ALIGN);
        ok = ok && make_tensor_map_2d(&P.map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, a->w, K / 2, N, pitch, 128, 64, true);
    }
    if (!ok) return TPB200_ERR_CUDA;
    P.sf = static_cast<const uint8_t*>(a->w_scales);
    P.pl_scale = static_cast<const __nv_bfloat16*>(a->w_scales);
    P.pl_zero = static_cast<const __nv_bfloat16*>(a->w_zeros);
    P.bias = a->bias;
    P.bias_dtype = a->bias_dtype;
    P.out = a->out;
    P.out_dtype = a->out_dtype;
    P.ldo = a->ldo;
    P.activation = a->activation;
    P.alpha = a->alpha;
    P.beta = a->beta;
    P.M = M;
    P.N = N;
    P.K = K;
    P.epilogue = qkv ? kEpiQkv : gated ? kEpiGated : norm_out ? kEpiResidual : P.splits > 1 || norm_in ? kEpiSplit : kEpiDirect;
    P.gated_rows = N / 2;
    P.q_dim = a->qkv_q_dim;
    P.ldq = a->ldo;
    P.k_rows = static_cast<__nv_bfloat16*>(a->qkv_k_rows);
    P.v_rows = static_cast<__nv_bfloat16*>(a->qkv_v_rows);
    P.positions = a->qkv_positions;
    P.rope_cos = static_cast<const __nv_bfloat16*>(a->qkv_rope_cos);
    P.rope_sin = static_cast<const __nv_bfloat16*>(a->qkv_rope_sin);

    const W4gRing ring = ring_of(plan, P.k_blocks, P.k_steps);
    P.tmem_cols = ring.tmem_cols;
    P.a_col = ring.a_col;
    P.parts = ring.parts;
    P.merge = ring.merge;
    P.n_w = ring.n_w;
    P.n_s = ring.n_s;

    using Kernel = void (*)(const W4gParams);
    static const Kernel kernels[4][2] = {{w4_nvfp4_gemm_kernel<false>, w4_nvfp4_gemm_kernel<true>},
                                         {w4_int4_kblock_gemm_kernel<false>, w4_int4_kblock_gemm_kernel<true>},
                                         {w4_int4_plugin_gemm_kernel<false>, w4_int4_plugin_gemm_kernel<true>},
                                         {w4_nvfp4_gemm_kernel_transposed<false>, w4_nvfp4_gemm_kernel_transposed<true>}};
    const int direct = P.epilogue == kEpiDirect;
    const Kernel kernel = kernels[fmt][direct];
    static std::atomic<uint64_t> configured[4][2] = {};
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured[fmt][direct].load(std::memory_order_relaxed) & bit)) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) {
            return TPB200_ERR_CUDA;
        }
        configured[fmt][direct].fetch_or(bit, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * P.splits, (M + P.nt - 1) / P.nt, 1);
    cfg.blockDim = dim3((kDqWarp0 + 4 * ring.groups) * 32, 1, 1);
    cfg.dynamicSmemBytes = smem_of(plan, ring, direct != 0);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (P.splits > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = P.splits;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (a->flags & TPB200_FLAG_PDL) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kernel, P) == cudaSuccess ? TPB200_OK : TPB200_ERR_CUDA;
}

}  // namespace tpb

extern "C" int tpb200_w4_gemm(const tpb200_w4_gemm_args* a, tpb200_stream_t stream) {
    return tpb::w4_gemm_launch(a, reinterpret_cast<cudaStream_t>(stream), false, nullptr);
}

extern "C" int tpb200_w4_gemm_norm(const tpb200_w4_gemm_args* a, const tpb200_w4_norm_args* norm, tpb200_stream_t stream) {
    TPB_REQUIRE(norm != nullptr, TPB200_ERR_NULL);
    return tpb::w4_gemm_launch(a, reinterpret_cast<cudaStream_t>(stream), false, norm);
}

extern "C" int tpb200_w4_gemm_plan(int M, int N, int K, int sms, tpb200_w4_gemm_plan_info* info) {
    TPB_REQUIRE(info != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE(M >= 1 && M <= 65535 * 256 && N >= 8 && K >= 16 && sms >= 1, TPB200_ERR_SHAPE);
    const int k_blocks = (K + tpb::kBlkK - 1) / tpb::kBlkK, k_steps = (K + tpb::kPartK - 1) / tpb::kPartK;
    const tpb::W4gPlan plan = tpb::plan_w4_gemm((N + tpb::kRows - 1) / tpb::kRows, M, k_blocks, sms, tpb::kFmtNvfp4);
    const tpb::W4gRing r = tpb::ring_of(plan, k_blocks, k_steps);
    *info = {plan.nt, plan.splits, plan.half ? 2 : 1, r.groups, r.parts, r.n_w, r.n_s * r.merge, k_blocks, k_steps};
    return TPB200_OK;
}

extern "C" int tpb200_w4_gemm_describe(int M, int N, int K, int format, int flags, int sms, tpb200_w4_gemm_launch_info* info) {
    TPB_REQUIRE(info != nullptr, TPB200_ERR_NULL);
    TPB_REQUIRE(M >= 1 && M <= 65535 * 256 && N >= 8 && K >= 16 && sms >= 1, TPB200_ERR_SHAPE);
    TPB_REQUIRE(format >= TPB200_W4_NVFP4_ROWMAJOR && format <= TPB200_W4_INT4_PLUGIN && (flags & ~TPB200_FLAG_PDL) == 0, TPB200_ERR_ENUM);
    const int k_blocks = (K + tpb::kBlkK - 1) / tpb::kBlkK, k_steps = (K + tpb::kPartK - 1) / tpb::kPartK;
    const tpb::W4gPlan plan = tpb::plan_w4_gemm((N + tpb::kRows - 1) / tpb::kRows, M, k_blocks, sms,
                                               format >= TPB200_W4_INT4_KBLOCK ? tpb::kFmtKblock : tpb::kFmtNvfp4);
    const tpb::W4gRing r = tpb::ring_of(plan, k_blocks, k_steps);
    *info = {plan.nt, plan.splits, plan.half ? 2 : 1, r.groups, r.parts, r.merge, r.n_w, r.n_s, k_blocks, k_steps, r.tmem_cols,
             tpb::smem_of(plan, r, plan.splits == 1)};
    return TPB200_OK;
}

extern "C" int tpb200_w4a16_gemm(const void* x, const void* weight, const void* scales, const void* zeros,
                                 const void* bias, int bias_dtype, void* out, int out_dtype, int M, int N, int K, int ldo,
                                 int layout, float alpha, float beta, int flags, tpb200_stream_t stream) {
    TPB_REQUIRE((flags & ~TPB200_FLAG_PDL) == 0, TPB200_ERR_ENUM);
    TPB_REQUIRE(layout == TPB200_INT4_KBLOCK || layout == TPB200_INT4_PLUGIN, TPB200_ERR_ENUM);
    TPB_REQUIRE(tpb_valid_dtype(out_dtype) && tpb_valid_dtype(bias_dtype), TPB200_ERR_ENUM);
    tpb200_w4_gemm_args a = {};
    a.x = x;
    a.ldx = K;
    a.format = layout == TPB200_INT4_KBLOCK ? TPB200_W4_INT4_KBLOCK : TPB200_W4_INT4_PLUGIN;
    a.w = weight;
    a.w_scales = scales;
    a.w_zeros = zeros;
    a.alpha = alpha;
    a.beta = beta;
    a.bias = bias;
    a.bias_dtype = bias_dtype;
    a.out = out;
    a.out_dtype = out_dtype;
    a.ldo = ldo == 0 ? N : ldo;
    a.M = M;
    a.N = N;
    a.K = K;
    a.flags = flags;
    return tpb::w4_gemm_launch(&a, reinterpret_cast<cudaStream_t>(stream), false, nullptr);
}
