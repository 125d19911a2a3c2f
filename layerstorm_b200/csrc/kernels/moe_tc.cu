// Tensor-core routed-expert FFN for many tokens (prefill chunks, verify batches, large decode
// batches): a grouped GEMM over expert-sorted token rows with the weight de-quantisation fused
// into the operand pipeline.
//
//   moe_tc_sort     counting sort of (row, slot) pairs by expert + list of [expert, first row, rows]
//                   token tiles of at most BN rows (device-side, no host round trip)
//   moe_tc_gather   xs[pos] = fp16(x[pair / S]) in sorted order (the TMA-loadable "B" operand)
//   moe_tc_ffn      persistent, one CTA per SM walking (token tile, 128 weight rows) work items:
//        warp 0      TMA producer for the token tiles (cp.async.bulk.tensor, 128-byte swizzle)
//        warp 1      tensor-memory owner and tcgen05.mma issuer (kind::f16, fp16 x fp16 -> fp32 in TMEM,
//                    A = weights read from tensor memory, B = tokens read from shared memory)
//        warps 2-17  weight converters: stream the expert's NVFP4 / FP8-block / Q4_K / BF16 rows from HBM
//                    exactly once into registers, expand them to fp16 (group / block scale folded in) and
//                    write them with tcgen05.st into a ring of operand stages in tensor memory
//        warp 22     TMA producer for the raw weight bytes
//        warps 18-21 epilogue (tcgen05.ld -> SwiGLU(+clamp) -> fp16, or -> fp32 / bf16 rows, or NVLink stores)
//     With few rows per expert the kernel is bound by the converters' instructions and by what the roles spend on barriers, with some 60 rows by these and
//     the traffic of tensor memory (operands stored, MMAs), not by DRAM or the tensor cores alone.  Measured (gate/up, down; us) with one converter set, a single
//     thread walking the issue loop and 64 elements per operand stage: 32 rows x top-8 of 288 + 1 shared NVFP4 experts of 4096 x 2048 (173 hit) 773 and 590,
//     2048 rows 1508 and 1221, 777 rows over 256 FP8 experts of 7168 x 2048 2310 and 1717; with two sets and stages of 128 and 256 elements 379 and 276, 910 and
//     643, 1307 and 860; with a token ring as long as the weights', row sets for down and an epilogue that waits for nothing 329 and 219, 843 and 510, 1262 and 778
//     (weights at DRAM's rate: 253 and 126, 422 and 211, 1168 and 584).  With nothing converted the first are 305 and 192, without MMAs 295 and 206.
//     gate and up tiles share one token tile and accumulate into two TMEM regions, so SwiGLU is
//     fused and the [tokens, 2F] intermediate never exists.
// Per-tensor NVFP4 scales are applied in the epilogue in fp32.  Every wait is bounded and reports
// through an error word.
// Reference seams replaced: moe_permute + external grouped GEMM + fused SwiGLU + unpermute
// (src/core/expert_device.h:31-52, E/smxx/permute/moe_permute.cu, G/sm120/gemm/grouped).
#include "tc_common.cuh"
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include "gemv_core.cuh"
#include "moe_fmt.cuh"
#include "ep_comm.cuh"

namespace lsb {
using namespace tc;

int cached_map_2d(CUtensorMap* out, const void* ptr, CUtensorMapDataType dt, int esize, uint64_t rows, uint64_t cols, uint64_t ld,
                  uint32_t br, uint32_t bc);

constexpr int kTBM = 128;   // weight rows per UMMA
constexpr int kTBK = 64;    // fp16 elements per stage row (128 bytes = one swizzle span)

// ------------------------------------------------------------------------------------------ sort
// Single block.  ids[npairs] = expert of pair i (or < 0 / >= E_total: ignored).
__global__ void __launch_bounds__(1024) moe_tc_sort_kernel(const int* __restrict__ ids, int npairs, int E_total, int BN,
                                                           int* __restrict__ sorted_pair, int* __restrict__ tile_expert,
                                                           int* __restrict__ tile_row0, int* __restrict__ tile_n,
                                                           int* __restrict__ counters /* [0]=tiles [1]=sorted pairs */) {
    extern __shared__ int sm[];
    int* cnt = sm;                  // [E_total]
    int* off = sm + E_total;        // [E_total + 1]
    int* tb = off + E_total + 1;    // [E_total + 1]
    pdl_wait();
    pdl_launch_dependents();
    for (int e = threadIdx.x; e < E_total; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
        const int e = ids[i];
        if (e >= 0 && e < E_total) atomicAdd(&cnt[e], 1);
    }
    __syncthreads();
    // first pair and first tile of every expert: a warp takes 32 experts at a time (one thread over 289 of them: 13 us)
    if (threadIdx.x < 32) {
        int o = 0, t = 0;
        for (int e0 = 0; e0 < E_total; e0 += 32) {
            const int e = e0 + threadIdx.x, c = e < E_total ? cnt[e] : 0, nt = (c + BN - 1) / BN;
            int so = c, st = nt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, so, d), b = __shfl_up_sync(0xffffffffu, st, d);
                if ((int)threadIdx.x >= d) { so += a; st += b; }
            }
            if (e < E_total) { off[e] = o + so - c; tb[e] = t + st - nt; }
            o += __shfl_sync(0xffffffffu, so, 31); t += __shfl_sync(0xffffffffu, st, 31);
        }
        if (threadIdx.x == 0) { off[E_total] = o; tb[E_total] = t; counters[0] = t; counters[1] = o; }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E_total; e += blockDim.x) {
        const int c = cnt[e];
        for (int j = 0, t = tb[e]; j < c; j += BN, ++t) { tile_expert[t] = e; tile_row0[t] = off[e] + j; tile_n[t] = min(BN, c - j); }
        cnt[e] = 0;                 // reused as the placement cursor
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
        const int e = ids[i];
        if (e >= 0 && e < E_total) sorted_pair[off[e] + atomicAdd(&cnt[e], 1)] = i;
    }
    pdl_launch_dependents();
}

// xs[pos][:] = fp16(x[sorted_pair[pos] / S][:]), finite numbers beyond fp16 as its largest
__global__ void __launch_bounds__(128) moe_tc_gather_kernel(const bf16* __restrict__ x, const int* __restrict__ sorted_pair,
                                                            const int* __restrict__ counters, __half* __restrict__ xs, int S, int H) {
    pdl_wait();
    pdl_launch_dependents();
    const int pos = blockIdx.x;
    if (pos >= counters[1]) return;
    const bf16* src = x + (size_t)(sorted_pair[pos] / S) * H;
    __half* dst = xs + (size_t)pos * H;
    for (int k = threadIdx.x * 8; k < H; k += blockDim.x * 8) {
        float f[8];
        unpack_bf16x8(__ldg(reinterpret_cast<const uint4*>(src + k)), f);
        __half2 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = half2_finite(f[2 * i], f[2 * i + 1]);
        *reinterpret_cast<uint4*>(dst + k) = *reinterpret_cast<uint4*>(h);
    }
    pdl_launch_dependents();
}

// The same with the rows as they are (bf16).
__global__ void __launch_bounds__(128) moe_tc_gather_bf16_kernel(const bf16* __restrict__ x, const int* __restrict__ sorted_pair,
                                                                 const int* __restrict__ counters, bf16* __restrict__ xs, int S, int H) {
    pdl_wait();
    pdl_launch_dependents();
    const int pos = blockIdx.x;
    if (pos >= counters[1]) return;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(sorted_pair[pos] / S) * H);
    uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)pos * H);
    for (int k = threadIdx.x; k < H / 8; k += blockDim.x) dst[k] = __ldg(src + k);
}

// ------------------------------------------------------------------------------------------ converters
__device__ __forceinline__ __half2 e4m3x2_to_half2(uint16_t v) {
    uint32_t r;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
    return *reinterpret_cast<__half2*>(&r);
}
__device__ __forceinline__ uint32_t h2_bits(const __half2& h) { return *reinterpret_cast<const uint32_t*>(&h); }

// Weight path of the grouped GEMM:  HBM --TMA--> raw ring in shared memory --ld.shared--> registers --convert-->
// tcgen05.st --> operand ring in tensor memory --> tcgen05.mma (A from TMEM).
// A pipeline stage is 64 reduction elements of 128 weight rows per matrix, SBYTES of every row.  What travels is a box of 128 bytes of
// every row (SUB stages) of the [slot][row][byte] view of the arena, written with the 128-byte swizzle: whole DRAM lines, and one barrier
// round trip of the converters for all of them.  One converter thread owns one
// weight row (TMEM lane = row) and 64 / NH consecutive elements of a stage: it reads its 16-byte chunks from the
// swizzled box (conflict free: the 8 lanes of a quarter-warp phase hit 8 different 16-byte bank groups), expands
// them to fp16 pairs with the group / block scale folded in and writes them into its TMEM lane with one tcgen05.st.
// The converted operand never exists in shared memory, which carries only raw bytes (once in, once out) and the
// token tiles; staging fp16 weight tiles there would cost about four times the shared-memory bandwidth.
//   RowConv<FMT, NH>::SBYTES                   raw bytes per row and stage
//   stage_x(it)                                byte offset of stage `it` inside a weight row
//   fetch(raw, tile, r, h, sub)                read this thread's chunks of row r (part h of NH) of stage `sub` of the box at `tile`
//   convert(raw, out, k0, h)                   expand to 32 / NH packed fp16 pairs
constexpr float kFp8Unscale = 1.f / 256.f;
constexpr int kBoxBytes = 128;
__device__ __forceinline__ uint32_t swz_chunk(uint32_t tile, int r, int c) { return tile + (uint32_t)(r * kBoxBytes + ((c ^ (r & 7)) << 4)); }
template <int FMT, int NH> struct RowConv;

template <int NH> struct RowConv<2, NH> {     // NVFP4: 32 bytes per row-stage; 4 group scales in one word
    static constexpr int SBYTES = 32, NV = 2 / NH, AUX = 512;              // AUX: a stage's 128 x 4 scale atom
    struct Raw { uint4 v[NV]; uint32_t sc; };
    static __device__ __forceinline__ int pitch(int K) { return K >> 1; }
    static __device__ __forceinline__ int stage_x(int it) { return it * 32; }
    static __device__ __forceinline__ void fetch(Raw& r, uint32_t tile, int row, int h, int sub) {
#pragma unroll
        for (int i = 0; i < NV; ++i) r.v[i] = ld_shared_16(swz_chunk(tile, row, sub * 2 + h * NV + i));
    }
    static __device__ __forceinline__ void convert(const Raw& r, uint32_t* out, int, int h) {
        // two scales per conversion; the products take them as halves of a register (a conversion of each scale in both halves: 8 more instructions a scheduler
        // has to place in every 64 elements of a warp, 133 cycles instead of 114)
        const __half2 s01 = e4m3x2_to_half2((uint16_t)(NH == 2 && h ? r.sc >> 16 : r.sc));
        const __half2 s23 = NH == 1 ? e4m3x2_to_half2((uint16_t)(r.sc >> 16)) : s01;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t wv[4] = {r.v[i].x, r.v[i].y, r.v[i].z, r.v[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {             // one word = 8 elements; 16-group index = word / 2
                __half2 hh[4];
                fp4x8_to_half2x4(wv[j], hh);
                const int grp = (4 * i + j) >> 1;
                const __half2 s2 = grp == 0 ? __low2half2(s01) : (grp == 1 ? __high2half2(s01) : (grp == 2 ? __low2half2(s23) : __high2half2(s23)));
#pragma unroll
                for (int q = 0; q < 4; ++q) out[(4 * i + j) * 4 + q] = h2_bits(__hmul2(hh[q], s2));
            }
        }
    }
};

template <int NH> struct RowConv<1, NH> {     // FP8 e4m3 with 128 x 128 block scales: 64 bytes per row-stage
    static constexpr int SBYTES = 64, NV = 4 / NH, AUX = 0;
    struct Raw { uint4 v[NV]; float sc; };
    static __device__ __forceinline__ int pitch(int K) { return K; }
    static __device__ __forceinline__ int stage_x(int it) { return it * 64; }
    static __device__ __forceinline__ void fetch(Raw& r, uint32_t tile, int row, int h, int sub) {
#pragma unroll
        for (int i = 0; i < NV; ++i) r.v[i] = ld_shared_16(swz_chunk(tile, row, sub * 4 + h * NV + i));
    }
    static __device__ __forceinline__ void convert(const Raw& r, uint32_t* out, int, int) {
        // block scales of small weights sit near the bottom of the fp16 range: carry them times 2^8 (exact; block scales up to 146 / 256, weights up to 255)
        // and take the factor out again in the fp32 epilogue (kFp8Unscale)
        const __half2 s2 = __float2half2_rn(r.sc * 256.f);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t wv[4] = {r.v[i].x, r.v[i].y, r.v[i].z, r.v[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                out[(4 * i + j) * 2 + 0] = h2_bits(__hmul2(e4m3x2_to_half2((uint16_t)(wv[j] & 0xffffu)), s2));
                out[(4 * i + j) * 2 + 1] = h2_bits(__hmul2(e4m3x2_to_half2((uint16_t)(wv[j] >> 16)), s2));
            }
        }
    }
};

template <int NH> struct RowConv<3, NH> {     // GGUF Q4_K: a stage = 32 quant bytes: low nibbles = sub-block 2s, high nibbles = 2s + 1
    static constexpr int SBYTES = 32, AUX = 0;
    struct Raw { uint4 hdr; uint4 q[2]; };
    static __device__ __forceinline__ int pitch(int K) { return (K >> 8) * 144; }
    static __device__ __forceinline__ int stage_x(int it) { return (it >> 2) * 144 + 16 + (it & 3) * 32; }
    static __device__ __forceinline__ void fetch(Raw& r, uint32_t tile, int row, int, int sub) {
        r.q[0] = ld_shared_16(swz_chunk(tile, row, sub * 2));
        r.q[1] = ld_shared_16(swz_chunk(tile, row, sub * 2 + 1));
    }
    static __device__ __forceinline__ void convert(const Raw& r, uint32_t* out, int k0, int h) {
        const __half2 dd = *reinterpret_cast<const __half2*>(&r.hdr.x);
        const float d = __low2float(dd), dmin = __high2float(dd);
        uint8_t sc12[12];
        const uint32_t hw[3] = {r.hdr.y, r.hdr.z, r.hdr.w};
#pragma unroll
        for (int i = 0; i < 12; ++i) sc12[i] = (uint8_t)(hw[i >> 2] >> (8 * (i & 3)));
        const uint32_t wv[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
        const int j2 = ((k0 & 255) >> 6) * 2;                      // first sub-block of this stage
#pragma unroll
        for (int hi = 0; hi < 2 / NH; ++hi) {                      // which nibble: elements 32 * nib .. 32 * nib + 31
            const int nib = NH == 1 ? hi : h;
            float sc, mn;
            q4k_scale_min(sc12, j2 + nib, sc, mn);
            const __half2 a2 = __float2half2_rn(d * sc), b2 = __float2half2_rn(-dmin * mn);
#pragma unroll
            for (int pr = 0; pr < 16; ++pr) {                      // byte pair (2 pr, 2 pr + 1) -> two consecutive elements
                const uint32_t wq = wv[pr >> 1] >> ((pr & 1) * 16 + nib * 4);
                // two 4-bit values as exact fp16 integers (1024 + v) - 1024
                const uint32_t bits = 0x64006400u | (wq & 0xFu) | (((wq >> 8) & 0xFu) << 16);
                const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&bits), __float2half2_rn(1024.f));
                out[hi * 16 + pr] = h2_bits(__hfma2(v, a2, b2));
            }
        }
    }
};

template <int NH> struct RowConv<0, NH> {     // BF16: 128 bytes per row-stage
    static constexpr int SBYTES = 128, NV = 8 / NH, AUX = 0;
    struct Raw { uint4 v[NV]; };
    static __device__ __forceinline__ int pitch(int K) { return K * 2; }
    static __device__ __forceinline__ int stage_x(int it) { return it * 128; }
    static __device__ __forceinline__ void fetch(Raw& r, uint32_t tile, int row, int h, int) {
#pragma unroll
        for (int i = 0; i < NV; ++i) r.v[i] = ld_shared_16(swz_chunk(tile, row, h * NV + i));
    }
    static __device__ __forceinline__ void convert(const Raw& r, uint32_t* out, int, int) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            float f[8];
            unpack_bf16x8(r.v[i], f);
#pragma unroll
            for (int q = 0; q < 4; ++q) out[4 * i + q] = h2_bits(__floats2half2_rn(f[2 * q], f[2 * q + 1]));
        }
    }
};

// ------------------------------------------------------------------------------------------ main kernel
struct MoeTcParams {
    const uint8_t* arena; const int* slot_of; ExpertFmt ef;
    const int* tile_expert; const int* tile_row0; const int* tile_n; const int* counters;
    const int* sorted_pair;
    __half* act;          // gate/up output, [pairs, F] fp16 (kDirectBf16: bf16) in sorted order
    float* y;             // down output, [npairs, H] fp32 in pair order
    GluAct ga;
    int* miss_flag; int* err;
    // expert-parallel mode (ep.nranks > 0): the gate/up kernel waits for the peers' token rows (phase 1) before its
    // first load, the down kernel stores its rows straight into the token owners' buffers and publishes phase 2
    EpComm ep;
    // dense-linear mode of the down kernel (one "expert" = the whole matrix): row stride and type of the output and the
    // per-tensor scale (0 = read it from the slot tail)
    int ldo, out_bf16; float down_scale;
    int up;               // one-matrix form of the kernel over the up matrices of experts without a gate: relu(up x)^2 into `act`
};

// DIRECT (bf16 weights over bf16 tokens): nothing to convert, the weight boxes in shared memory are the MMA's A operand as TMA wrote them; tensor
// memory holds accumulators only, two sets of them.  kDirect: gate / up with fp16 hidden values; kDirectBf16: both halves, hidden values in bf16.
constexpr int kDirect = 1, kDirectBf16 = 2;
template <int FMT, int BN, bool GATEUP, int DIRECT = 0> struct MoeTcCfg {
    static_assert(!DIRECT || (FMT == 0 && (GATEUP || DIRECT == kDirectBf16)), "direct operands: bf16 weights and tokens");
    static constexpr int A_TILES = GATEUP ? 2 : 1;
    static constexpr int NH = GATEUP || FMT != 0 ? 1 : 2;                 // converter threads per (row, sub-stage) of a matrix; bf16 rows take too many registers for one
    using CV = RowConv<FMT, NH>;
    // Token tiles of 256 rows (bf16 experts): a copy of 128 rows and an MMA of 128 columns where no more are there, else two and 256.  Half the weights per product
    // through L2 and shared memory, which bound tiles of 128 (12.7 TB/s of L2); tensor memory then holds one accumulator set.
    static constexpr int B_BOX = BN > 128 ? 128 : BN;
    static constexpr int B_BYTES = BN * kTBK * 2;                         // token tile of a sub-stage
    // An operand stage is KS sub-stages of 64 reduction elements behind one pair of barriers: the issuing warp's waits and commit cost a few
    // hundred cycles a stage beside the converters' instruction streams, which is more than the MMAs of 64 elements of a small token tile take.
#ifndef LSB_MOE_KS_GU
#define LSB_MOE_KS_GU 2
#endif
#ifndef LSB_MOE_KS_DN
#define LSB_MOE_KS_DN 4
#endif
    static constexpr int KS = GATEUP ? (BN > 128 ? 1 : LSB_MOE_KS_GU) : (BN <= 64 || FMT != 0 ? LSB_MOE_KS_DN : 2);
    static constexpr int ACC_COLS = A_TILES * BN;                         // one accumulator set (gate [+ up])
    // Tensor memory (512 columns): accumulator sets first, then the ring of converted weight stages
    // (32 columns = 64 fp16 per matrix and sub-stage).  Two accumulator sets let the epilogue of one item overlap the
    // main loop of the next; at ACC_COLS = 256 only one fits beside the weight ring.
#ifndef LSB_MOE_NBUF1_COLS
#define LSB_MOE_NBUF1_COLS 128
#endif
    static constexpr int NBUF = ACC_COLS > LSB_MOE_NBUF1_COLS && (!DIRECT || ACC_COLS > 256) ? 1 : 2;
    static constexpr int A_COLS = 32 * A_TILES * KS;
    static constexpr int A_BASE = NBUF * ACC_COLS;
    static constexpr int S_FIT = DIRECT ? 2 : (512 - A_BASE) / A_COLS;
    static constexpr int S = S_FIT > 3 ? 3 : S_FIT;                       // operand stages of the weights, in tensor memory
    static constexpr int TMEM_COLS = 512;
    // A set of converter warps covers one sub-stage (4 lane quarters x gate and up, or x the parts of a row); the sets take the sub-stages in turns, so
    // that a warp has as many sub-stage times for its serial read -> convert -> store chain.  Down over quantised weights: four sets whose threads take
    // a whole row of 64 elements; two sets with half rows spent as much on barriers as on converting.
    static constexpr int PARTS = GATEUP ? 2 : NH;
    static constexpr int SET_WARPS = 4 * PARTS;
    static constexpr int CONV_SETS = 16 / SET_WARPS;
    static constexpr int CONV_WARPS = DIRECT ? 0 : 16;
    static_assert(DIRECT || KS % CONV_SETS == 0, "all sets have part in every operand stage");
    static constexpr int EPI_WARPS = 4;
    static constexpr int RAW_WARP = 2 + CONV_WARPS + EPI_WARPS;           // last warp: TMA producer of the raw weight ring
    static constexpr int THREADS = (RAW_WARP + 1) * 32;
    // raw weight ring (shared memory): per entry a box of SUB stages per matrix (+ the NVFP4 scale atoms of these)
    static constexpr int SUB = kBoxBytes / CV::SBYTES;
    static constexpr int W_TILE = kTBM * kBoxBytes;
    static constexpr int RAW_STAGE = A_TILES * (W_TILE + SUB * CV::AUX);
    static constexpr int BAR_BYTES = 512;
    // The token tiles have a ring of their own (SB operand stages) that reaches as far ahead as the raw weights': a copy of theirs waits in the SM's copy
    // engine behind the weights that have been asked for, some 3000 cycles.  With as many stages as the weights have in tensor memory (3 of 128
    // elements) the tensor core waited for tokens: 2048 rows of 288 NVFP4 experts, gate/up 600 cycles per 64 elements whether weights were converted or not.
    static constexpr int BUDGET = 224 * 1024 - BAR_BYTES - 1024;
    static constexpr int RD_FIT = BUDGET / (RAW_STAGE + SUB * B_BYTES);
    // Where the converter sets are in entries of their own (ADV > 1), a slot is one set's: a set may be 12 sub-stages ahead, and coming to a slot whose round before
    // is the other's and still on its way (copies out of L2 overtake), it would take the round two before for its own, as the parity is the same.
    static constexpr int ADV = CONV_SETS > SUB && !DIRECT ? CONV_SETS / SUB : 1;
    static constexpr int RD = (RD_FIT > 12 ? 12 : (RD_FIT < 3 ? 3 : RD_FIT)) / ADV * ADV;
    static constexpr int SB_FIT = (BUDGET - RD * RAW_STAGE) / (KS * B_BYTES), SB_ALL = (RD * SUB + KS - 1) / KS;
    static constexpr int SB = SB_FIT < SB_ALL ? SB_FIT : SB_ALL;
    // One CTA per SM by construction (the CTA owns all of tensor memory): ask for more than half of the SM's shared memory.
    static constexpr int SMEM_NEED = SB * KS * B_BYTES + RD * RAW_STAGE + BAR_BYTES + 1024;
    static constexpr int SMEM = SMEM_NEED < 120 * 1024 ? 120 * 1024 : SMEM_NEED;
    static_assert(S >= 2 && A_BASE + (DIRECT ? 0 : S * A_COLS) <= 512, "tensor memory budget");
    static_assert(RD >= 3 && SB >= 2 && SMEM <= 227 * 1024, "shared memory budget");
    static_assert((2 * S + 2 * SB + 2 * RD + 4) * 8 + 8 <= BAR_BYTES, "barrier area");
};
constexpr int kMaxSlots = 1 << 16;
// Role-level time breakdown for tuning builds (-DLSB_MOE_PROFILE): block 0 accumulates the cycles each role spends
// waiting on each barrier and working; lsb_moe_tc_prof_read copies the table out.
#ifdef LSB_MOE_PROFILE
__device__ unsigned long long g_moe_prof[32];
#define PROF_DECL() long long _pacc[4] = {0, 0, 0, 0}; const long long _pt0 = clock64()
#define PROF_SCOPE(j, stmt) do { const long long _t = clock64(); stmt; _pacc[j] += clock64() - _t; } while (0)
#define PROF_FLUSH(j, i) do { if (blockIdx.x == 0) g_moe_prof[i] += (unsigned long long)_pacc[j]; } while (0)
#define PROF_TOTAL(i) do { if (blockIdx.x == 0) g_moe_prof[i] += (unsigned long long)(clock64() - _pt0); } while (0)
#else
#define PROF_DECL()
#define PROF_SCOPE(j, stmt) do { stmt; } while (0)
#define PROF_FLUSH(j, i)
#define PROF_TOTAL(i)
#endif               // slot extent of the weight tensor maps

// Work item w -> (token tile t, weight tile j).  Items are grouped by kTileGroup consecutive token tiles (tiles are sorted
// by expert, so a group mostly belongs to one expert); inside a group the token tile runs fastest, so the CTAs that
// are in flight together read the same 128 weight rows and all but the first hit L2.
constexpr int kTileGroup = 8;
__device__ __forceinline__ void work_item(int w, int ntiles, int NT, int& t, int& j) {
    const int per = kTileGroup * NT;
    const int gi = w / per, r = w % per;
    const int t0 = gi * kTileGroup;
    const int gsz = min(kTileGroup, ntiles - t0);
    t = t0 + r % gsz;
    j = r / gsz;
}

// Persistent kernel: one CTA per SM walks the work list (token tile x 128-row weight tile); the rings, their barrier
// phases and the accumulator sets carry over from one work item to the next, so the producers run ahead across
// item boundaries.
// Position in a ring of N entries and the parity of the round.
template <int N> struct RingPos {
    uint32_t i = 0, ph = 0;
    __device__ __forceinline__ void next() { if (++i == N) { i = 0; ph ^= 1u; } }
    __device__ __forceinline__ void skip(uint32_t n) { i += n; if (i >= N) { i -= N; ph ^= 1u; } }       // n <= N
};

template <int FMT, int BN, bool GATEUP, int DIRECT = 0>
__global__ void __launch_bounds__(MoeTcCfg<FMT, BN, GATEUP, DIRECT>::THREADS, 1) moe_tc_ffn_kernel(const __grid_constant__ CUtensorMap map_b,
                                                                                       const __grid_constant__ CUtensorMap map_w0,
                                                                                       const __grid_constant__ CUtensorMap map_w1, MoeTcParams p) {
    using C = MoeTcCfg<FMT, BN, GATEUP, DIRECT>;
    using CV = typename C::CV;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_b = smem;                                   // [SB][KS] token tiles
    uint8_t* smem_r = smem + C::SB * C::KS * C::B_BYTES;      // [RD] raw weight entries
    uint64_t* full_a = reinterpret_cast<uint64_t*>(smem_r + C::RD * C::RAW_STAGE);
    uint64_t* empty_a = full_a + C::S;
    uint64_t* full_b = empty_a + C::S;
    uint64_t* empty_b = full_b + C::SB;
    uint64_t* full_r = empty_b + C::SB;
    uint64_t* empty_r = full_r + C::RD;
    uint64_t* acc_full = empty_r + C::RD;        // [NBUF]
    uint64_t* acc_empty = acc_full + 2;          // [NBUF]
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool up = !GATEUP && p.up;
    const int K = GATEUP || up ? p.ef.H : p.ef.F;          // reduction length
    const int NOUT = GATEUP || up ? p.ef.F : p.ef.H;       // weight rows
    const int NT = NOUT / kTBM;
    const int nkb = K / kTBK, nops = (nkb + C::KS - 1) / C::KS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::S; ++s) { mbar_init(&full_a[s], DIRECT ? 1 : C::CONV_WARPS); mbar_init(&empty_a[s], 1); }
        for (int s = 0; s < C::SB; ++s) { mbar_init(&full_b[s], 1); mbar_init(&empty_b[s], 1); }
        for (int s = 0; s < C::RD; ++s) { mbar_init(&full_r[s], 1); mbar_init(&empty_r[s], DIRECT ? 1 : C::CONV_WARPS / C::ADV); }
        for (int b = 0; b < C::NBUF; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], C::EPI_WARPS); }
        fence_barrier_init();
        fence_proxy_async();
        tma_prefetch_desc(&map_b);
        tma_prefetch_desc(&map_w0);
        if (GATEUP) tma_prefetch_desc(&map_w1);
    }
    if (warp == 1) tmem_alloc(tmem_holder, C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_holder;
    pdl_wait();
    pdl_launch_dependents();
    const bool ep_mode = p.ep.nranks > 0;
    const unsigned ep_epoch = ep_mode ? *p.ep.epoch + 1u : 0u;
    if (ep_mode && GATEUP) {
        ep_wait(p.ep, 1, ep_epoch);                  // peers' rows have landed in this rank's staging buffer
        asm volatile("fence.proxy.async;" ::: "memory");   // ... and are ordered before the TMA (async proxy) reads
    }
    const int ntiles = p.counters[0];
    const int total = ntiles * NT;
    // an expert that is not resident on this GPU (or a slot the weight maps do not cover): every role skips the item
    auto slot_ok = [&](int slot) { return slot >= 0 && slot < kMaxSlots; };

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer: token tiles ----------------
            RingPos<C::SB> r;
            uint32_t g = 0;
            bool ok = true;
            PROF_DECL();
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
                int t, jn;
                work_item(w, ntiles, NT, t, jn);
                const int e = p.tile_expert[t];
                if (!slot_ok(p.slot_of[e])) {
                    if ((GATEUP || up) && p.miss_flag && jn == 0) atomicExch(p.miss_flag, e + 1);
                    continue;
                }
                const int row0 = p.tile_row0[t];
                const int boxes = BN > 128 && p.tile_n[t] > 128 ? 2 : 1;
                for (int o = 0; o < nops; ++o, ++g, r.next()) {
                    PROF_SCOPE(0, ok = mbar_wait(&empty_b[r.i], r.ph ^ 1, p.err, 11));
                    if (!ok) break;
                    const int n = min(C::KS, nkb - o * C::KS);
                    mbar_expect_tx(&full_b[r.i], (uint32_t)(n * boxes * C::B_BOX * kTBK * 2));
                    for (int j = 0; j < n; ++j) {
                        uint8_t* dst = smem_b + (r.i * C::KS + j) * C::B_BYTES;
                        tma_load_2d(dst, &map_b, &full_b[r.i], (o * C::KS + j) * kTBK, row0);
                        if (BN > 128 && boxes > 1) tma_load_2d(dst + C::B_BOX * kTBK * 2, &map_b, &full_b[r.i], (o * C::KS + j) * kTBK, row0 + C::B_BOX);
                    }
                }
            }
            PROF_FLUSH(0, 1);
            if (!ok) {
                // loads in flight still write this CTA's shared memory: let them land (bounded, no error code)
                for (uint32_t i = g > (uint32_t)C::SB ? g - C::SB : 0; i < g; ++i) mbar_wait(&full_b[i % C::SB], (i / C::SB) & 1, nullptr, 0);
            }
        }
    } else if (warp == C::RAW_WARP) {
        if (lane == 0) {
            // ---------------- TMA producer: raw weight bytes (and NVFP4 scale atoms) ----------------
            uint32_t g = 0;
            bool ok = true;
            PROF_DECL();
            for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
                int t, jn;
                work_item(w, ntiles, NT, t, jn);
                const int slot = p.slot_of[p.tile_expert[t]];
                if (!slot_ok(slot)) continue;
                const uint8_t* base = p.arena + (size_t)slot * p.ef.stride;
                const uint8_t* sf0 = base + (GATEUP ? p.ef.off_sg : (up ? p.ef.off_su : p.ef.off_sd));
                const uint8_t* sf1 = base + p.ef.off_su;
                const int gtiles = ((K >> 4) + 3) >> 2;        // NVFP4: 512-byte scale atoms per 128-row tile
                for (int it = 0; it < nkb; it += C::SUB, ++g) {
                    const int s = g % C::RD;
                    PROF_SCOPE(0, ok = mbar_wait(&empty_r[s], ((g / C::RD) & 1) ^ 1, p.err, 16));
                    if (!ok) break;
                    uint8_t* dst = smem_r + s * C::RAW_STAGE;
                    // (a row's last box may reach past the row: zeros, never read; its scale atoms are those of the stages that are left)
                    const uint32_t aux = (uint32_t)(min(C::SUB, nkb - it) * CV::AUX);
                    mbar_expect_tx(&full_r[s], C::A_TILES * (C::W_TILE + aux));
                    const int x = CV::stage_x(it);
                    tma_load_3d(dst, &map_w0, &full_r[s], x, jn * kTBM, slot);
                    if (GATEUP) tma_load_3d(dst + C::W_TILE, &map_w1, &full_r[s], x, jn * kTBM, slot);
                    if (CV::AUX) {
                        const size_t so = ((size_t)jn * gtiles + it) * 512;
                        bulk_load_1d(dst + C::A_TILES * C::W_TILE, sf0 + so, aux, &full_r[s]);
                        if (GATEUP) bulk_load_1d(dst + C::A_TILES * C::W_TILE + C::SUB * CV::AUX, sf1 + so, aux, &full_r[s]);
                    }
                }
            }
            PROF_FLUSH(0, 0);
            if (!ok) {
                for (uint32_t i = g > (uint32_t)C::RD ? g - C::RD : 0; i < g; ++i) mbar_wait(&full_r[i % C::RD], (i / C::RD) & 1, nullptr, 0);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: A (weights) from tensor memory, B (tokens) from shared memory ----------------
        // The whole warp walks the list (loop bounds and ring positions stay warp-uniform, so the operands of the instructions are uniform
        // registers) and one elected lane issues.
        const int utotal = __reduce_max_sync(0xffffffffu, total), untiles = __reduce_max_sync(0xffffffffu, ntiles);
        const uint32_t ut = __reduce_max_sync(0xffffffffu, tmem_d);
        RingPos<C::S> ra;                                      // weights in tensor memory
        RingPos<C::SB> r;                                      // token tiles
        RingPos<C::RD> rr;                                     // (direct: raw entries)
        uint32_t lt = 0;
        bool ok = true;
        PROF_DECL();
        for (int w = blockIdx.x; w < utotal && ok; w += gridDim.x) {
            int t, jn;
            work_item(w, untiles, NT, t, jn);
            if (!__reduce_or_sync(0xffffffffu, slot_ok(p.slot_of[p.tile_expert[t]]) ? 1u : 0u)) continue;
            constexpr uint32_t idesc_all = idesc_f16(kTBM, BN, DIRECT ? 1 : 0), idesc_box = idesc_f16(kTBM, C::B_BOX, DIRECT ? 1 : 0);
            uint32_t idesc = idesc_all;
            if constexpr (BN > 128) idesc = __reduce_or_sync(0xffffffffu, p.tile_n[t] > C::B_BOX ? 1u : 0u) ? idesc_all : idesc_box;
            const uint32_t buf = lt % C::NBUF;
            PROF_SCOPE(0, ok = mbar_wait(&acc_empty[buf], ((lt / C::NBUF) & 1u) ^ 1u, p.err, 15));   // epilogue has drained this accumulator set
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = ut + buf * C::ACC_COLS;
            for (int o = 0; o < nops; ++o, r.next(), ra.next()) {
                PROF_SCOPE(1, ok = mbar_wait(&full_b[r.i], r.ph, p.err, 12));
                if constexpr (DIRECT) {
                    ok = __all_sync(0xffffffffu, ok);
                    const int n = min(C::KS, nkb - o * C::KS);
                    for (int j = 0; j < n && ok; ++j, rr.next()) {
                        PROF_SCOPE(2, ok = mbar_wait(&full_r[rr.i], rr.ph, p.err, 12));
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                        const uint8_t* a = smem_r + rr.i * C::RAW_STAGE;
                        const uint64_t dg = smem_desc_sw128(a), du = smem_desc_sw128(a + C::W_TILE), db = smem_desc_sw128(smem_b + (r.i * C::KS + j) * C::B_BYTES);
                        PROF_SCOPE(3, {
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < kTBK / 16; ++k) {
                                const uint32_t accum = (o > 0 || j > 0 || k > 0) ? 1u : 0u;
                                umma_f16(acc, dg + 2 * k, db + 2 * k, idesc, accum);
                                if (GATEUP) umma_f16(acc + BN, du + 2 * k, db + 2 * k, idesc, accum);
                            }
                            umma_commit(&empty_r[rr.i]);
                        }
                        __syncwarp(); });
                    }
                    if (!ok) break;
                    if (elect_one()) umma_commit(&empty_b[r.i]);
                    __syncwarp();
                    continue;
                }
                if (ok) PROF_SCOPE(2, ok = mbar_wait(&full_a[ra.i], ra.ph, p.err, 12));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a_t = ut + C::A_BASE + ra.i * C::A_COLS;
                const uint64_t db = smem_desc_sw128(smem_b + r.i * C::KS * C::B_BYTES);
                const int n = min(C::KS, nkb - o * C::KS);
                PROF_SCOPE(3, {
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < C::KS; ++j) {
                        if (j > 0 && j >= n) break;
#pragma unroll
                        for (int k = 0; k < kTBK / 16; ++k) {
                            const uint32_t accum = (o > 0 || j > 0 || k > 0) ? 1u : 0u;
                            const uint64_t b = db + (uint64_t)(j * (C::B_BYTES >> 4) + 2 * k);
                            umma_f16_ts(acc, a_t + j * 32 * C::A_TILES + 8 * k, b, idesc, accum);
                            if (GATEUP) umma_f16_ts(acc + BN, a_t + j * 32 * C::A_TILES + 32 + 8 * k, b, idesc, accum);
                        }
                    }
                    umma_commit(&empty_a[ra.i]);
                    umma_commit(&empty_b[r.i]);
                }
                __syncwarp(); });
            }
            if (ok && elect_one()) umma_commit(&acc_full[buf]);
            __syncwarp();
            ++lt;
        }
        if (lane == 0) { PROF_FLUSH(0, 4); PROF_FLUSH(1, 2); PROF_FLUSH(2, 3); PROF_FLUSH(3, 14); PROF_TOTAL(5); }
    } else if (warp < 2 + C::CONV_WARPS) {
        // ---------------- weight converters ----------------
        constexpr int NC = 32 / C::NH;
        const int q = warp & 3;                                // TMEM lane quarter this warp may access
        const int part = ((warp - 2) >> 2) % C::PARTS;         // gate/up: matrix (0 gate, 1 up); down: part of the sub-stage's elements
        const int set = (warp - 2) / C::SET_WARPS;             // this warp converts the sub-stages `it` with it % CONV_SETS == set
        const int row = q * 32 + lane;                         // row of the 128-row weight tile = TMEM lane
        const int h = GATEUP ? 0 : part;
        const int mat = GATEUP ? part : 0;
        const uint32_t t_lane = tmem_d + C::A_BASE + ((uint32_t)(q * 32) << 16) + (GATEUP ? part * 32 : part * NC);
        RingPos<C::S> ra;                                      // operand stages
        RingPos<C::RD> rr;                                     // raw entries
        bool ok = true;
        PROF_DECL();
        for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
            int t, jn;
            work_item(w, ntiles, NT, t, jn);
            const int slot = p.slot_of[p.tile_expert[t]];
            if (!slot_ok(slot)) continue;
            const uint8_t* base = p.arena + (size_t)slot * p.ef.stride;
            const uint8_t* wm = base + (GATEUP ? (part ? p.ef.off_up : p.ef.off_gate) : (up ? p.ef.off_up : p.ef.off_down));
            const uint8_t* sf = base + (GATEUP ? (part ? p.ef.off_su : p.ef.off_sg) : (up ? p.ef.off_su : p.ef.off_sd));
            const int n = jn * kTBM + row;                     // weight row in the expert matrix
            // side data that does not travel through the ring: the FP8 block scale (one float per 128 x 128 block, the
            // same for the whole tile) and the Q4_K super-block header (16 bytes per row and 256 elements), both read
            // one stage ahead of their use
            const float* fsc = reinterpret_cast<const float*>(sf) + (size_t)(n >> 7) * ((K + 127) >> 7);
            const uint8_t* qrow = wm + (size_t)n * CV::pitch(K);
            // this warp's place among the sub-stages that the sets take side by side (an item with an odd number of entries leaves the sets' slots shifted)
            const int own = C::ADV > 1 ? ((set / C::SUB + C::ADV - (int)rr.i % C::ADV) % C::ADV) * C::SUB + set % C::SUB : set;
            float sc_next = 0.f;
            uint4 hdr_next = make_uint4(0, 0, 0, 0);
            if (FMT == 1) sc_next = __ldg(fsc + (C::ADV > 1 && own / C::SUB < nkb / C::SUB ? own / C::SUB : 0));
            if (FMT == 3) hdr_next = __ldg(reinterpret_cast<const uint4*>(qrow));
            const int nent = (nkb + C::SUB - 1) / C::SUB;
            typename CV::Raw raw;
            // Straight-line code for the sub-stages of whole entries and whole operand stages: the instructions around a sub-stage (ring
            // positions, which barrier is due) cost as much as its conversion when they are decided at run time.
            constexpr int BLK = C::SUB > C::KS ? C::SUB : C::KS;
#pragma unroll 1
            for (int b0 = 0; b0 < nkb && ok; b0 += BLK) {
#pragma unroll
                for (int i = 0; i < BLK / C::CONV_SETS; ++i) {
                    const int l0 = i * C::CONV_SETS, l = l0 + own;       // sub-stages of all sets; this warp's
                    if (b0 + l0 >= nkb) break;
                    // (past the end: zeros into columns that no MMA reads, or no entry at all)
                    const bool mine = C::ADV == 1 || b0 + l / C::SUB * C::SUB < nkb;
                    RingPos<C::RD> re = rr;
                    if (C::ADV > 1) re.skip(l / C::SUB);
                    if (C::ADV > 1 || l0 % C::SUB == 0) {
                        if constexpr (FMT == 1) {
                            raw.sc = sc_next;
                            const int e = (b0 + (C::ADV > 1 ? l : l0)) / C::SUB + C::ADV;
                            if (e < nent) sc_next = __ldg(fsc + e);
                        }
                        if constexpr (FMT == 3) {
                            raw.hdr = hdr_next;
                            const int e = (b0 + l0) / C::SUB + 1;
                            if (e < nent) hdr_next = __ldg(reinterpret_cast<const uint4*>(qrow + (size_t)e * 144));
                        }
                        // (the warp polls as a whole: a lane's poll handed round by a shuffle is a longer chain, 556 instead of 512 cycles per 64 elements of 32 rows)
                        if (mine) PROF_SCOPE(0, ok = mbar_wait(&full_r[re.i], re.ph, p.err, 17));
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                    }
                    uint32_t out[NC];
                    if (mine) {
                        const uint32_t entry = smem_u32(smem_r + re.i * C::RAW_STAGE);
                        const int sub = l % C::SUB;
                        CV::fetch(raw, entry + mat * C::W_TILE, row, h, sub);
                        if constexpr (FMT == 2) {
                            // scale atom of the 128-row tile: word (row % 32) * 4 + row / 32
                            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(raw.sc) : "r"(entry + C::A_TILES * C::W_TILE + (mat * C::SUB + sub) * 512 + lane * 16 + q * 4) : "memory");
                        }
                        CV::convert(raw, out, (b0 + l) * kTBK, h);       // consumes every byte read above
                    }
                    if (C::ADV > 1 || (l0 + C::CONV_SETS) % C::SUB == 0 || b0 + l0 + C::CONV_SETS >= nkb) {
                        __syncwarp();
                        if (lane == 0 && mine) mbar_arrive(&empty_r[re.i]);        // the raw entry may be refilled
                        if (C::ADV == 1) rr.next();
                    }
                    if (l0 % C::KS == 0) {
                        PROF_SCOPE(1, ok = mbar_wait(&empty_a[ra.i], ra.ph ^ 1, p.err, 13));
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();                      // the MMAs that read this operand stage have completed
                    }
                    if (mine) {
                        const uint32_t dst = t_lane + ra.i * C::A_COLS + (l % C::KS) * 32 * C::A_TILES;
                        if (NC == 32) tmem_st32(dst, out);
                        else tmem_st16(dst, out);
                    }
                    if ((l0 + C::CONV_SETS) % C::KS == 0 || b0 + l0 + C::CONV_SETS >= nkb) {
                        PROF_SCOPE(3, tmem_wait_st());
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&full_a[ra.i]);
                        ra.next();
                    }
                }
                if (C::ADV > 1) rr.skip((min(BLK, nkb - b0) + C::SUB - 1) / C::SUB);
            }
        }
        if (warp == 2 && lane == 0) { PROF_FLUSH(0, 6); PROF_FLUSH(1, 8); PROF_FLUSH(2, 7); PROF_FLUSH(3, 9); PROF_TOTAL(10); }
    } else {
        // ---------------- epilogue (4 warps: one TMEM lane quarter each) ----------------
        const int q = warp & 3;
        uint32_t lt = 0;
        bool ok = true;
        PROF_DECL();
        for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
            int t, jn;
            work_item(w, ntiles, NT, t, jn);
            const int e = p.tile_expert[t];
            const int slot = p.slot_of[e];
            if (!slot_ok(slot)) continue;
            const int row0 = p.tile_row0[t], ncols = p.tile_n[t];
            const int n = jn * kTBM + q * 32 + lane;
            const uint8_t* base = p.arena + (size_t)slot * p.ef.stride;
            const uint32_t buf = lt % C::NBUF;
            // what 32 columns need, a lane each, fetched while the tile or the 32 in front of them are worked on: the factor on the expert's input, or the output
            // row of the down projection (read between the stores, which it has to stay behind as far as the compiler knows, the pair index made a chain of 64
            // loads that took longer than the tile's MMAs: the down projection of 2048 rows of 288 NVFP4 experts waited for its epilogue a quarter of the time)
            const bool scaled = GATEUP && p.ga.in_scale != nullptr;
            const bool scatter = !GATEUP && !up && !ep_mode;
            float cs = 1.f, cs_next = 1.f;
            int ct = 0, ct_next = 0;
            auto fetch = [&](int c) {
                ct_next = (scaled || scatter) && c < ncols ? p.sorted_pair[row0 + c] : 0;
                cs_next = scaled && c < ncols ? p.ga.in_scale[ct_next] : 1.f;
            };
            fetch(lane);
            int okw = 1;
            if (lane == 0) { if (q == 0) PROF_SCOPE(0, okw = mbar_wait_relaxed(&acc_full[buf], (lt / C::NBUF) & 1u, p.err, 14) ? 1 : 0); else okw = mbar_wait_relaxed(&acc_full[buf], (lt / C::NBUF) & 1u, p.err, 14) ? 1 : 0; }
            ok = __shfl_sync(0xffffffffu, okw, 0) != 0;
            tc_fence_after();
            if (ok) {
                float sg = 1.f, su = 1.f;
                if (FMT == 2 && (GATEUP || p.down_scale == 0.f)) {
                    const float* tail = reinterpret_cast<const float*>(base + p.ef.off_tail);
                    if (GATEUP) { sg = tail[0]; su = tail[1]; } else sg = tail[up ? 1 : 2];
                } else if (FMT == 2) {
                    sg = p.down_scale;
                } else if (FMT == 1) {
                    sg = su = kFp8Unscale;
                }
                const uint32_t lane_addr = tmem_d + buf * C::ACC_COLS + ((uint32_t)(q * 32) << 16);
                const GluAct ga = p.ga;
                // (NOUT is whole tiles, so every lane has a row of the matrix; which columns are stored is a predicate of the store)
                __half* act = p.act + (size_t)row0 * NOUT + n;
                float* yf = p.y + n;
                bf16* yh = reinterpret_cast<bf16*>(p.y) + n;
#pragma unroll 1
                for (int c0 = 0; c0 < ncols; c0 += 16) {
                    if ((c0 & 31) == 0) { ct = ct_next; cs = cs_next; fetch(c0 + 32 + lane); }
                    float gq[16], uq[16];
                    tmem_ld16(lane_addr + (uint32_t)c0, gq);
                    if (GATEUP) tmem_ld16(lane_addr + (uint32_t)(BN + c0), uq);
                    if (GATEUP) {
#pragma unroll
                        for (int j = 0; j < 16; ++j, act += NOUT) {
                            const float c = __shfl_sync(0xffffffffu, cs, (c0 + j) & 31);
                            if (DIRECT == kDirectBf16) st_global_if(reinterpret_cast<bf16*>(act), __float2bfloat16(glu_act(gq[j] * c, uq[j] * c, ga)), c0 + j < ncols);
                            else st_global_if(act, __float2half_rn(half_range(glu_act(gq[j] * sg * c, uq[j] * su * c, ga))), c0 + j < ncols);
                        }
                    } else if (up) {
                        // (fp16 range: far outside what normed inputs reach, kept finite all the same)
#pragma unroll
                        for (int j = 0; j < 16; ++j, act += NOUT) st_global_if(act, __float2half_rn(fminf(relu2_act(gq[j] * sg), 65504.f)), c0 + j < ncols);
                    } else if (ep_mode) {
#pragma unroll 1
                        for (int j = 0; j < 16 && c0 + j < ncols; ++j) {
                            float v = gq[0];
#pragma unroll
                            for (int i = 1; i < 16; ++i) v = i == j ? gq[i] : v;
                            const int2 ra = p.ep.ret[p.ep.rank][row0 + c0 + j];      // (token owner, pair index there)
                            p.ep.y[ra.x][(size_t)ra.y * NOUT + n] = v * sg;           // NVLink store into the owner's buffer
                        }
                    } else if (p.out_bf16) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int r = __shfl_sync(0xffffffffu, ct, (c0 + j) & 31);
                            st_global_if(yh + (size_t)r * p.ldo, __float2bfloat16(gq[j] * sg), c0 + j < ncols);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int r = __shfl_sync(0xffffffffu, ct, (c0 + j) & 31);
                            st_global_if(yf + (size_t)r * p.ldo, gq[j] * sg, c0 + j < ncols);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);       // the MMA issuer may overwrite this accumulator set
            ++lt;
        }
        if (q == 0 && lane == 0) { PROF_FLUSH(0, 11); PROF_TOTAL(13); }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_d, C::TMEM_COLS);
    if (ep_mode && !GATEUP) ep_signal(p.ep, 2, ep_epoch, gridDim.x);
    pdl_launch_dependents();
}

int make_map_bytes_3d(CUtensorMap* map, const void* ptr, uint64_t pitch, uint64_t rows, uint64_t slot_stride, uint64_t nslots,
                      uint32_t box_bytes, uint32_t box_rows);
static int cached_map_w(CUtensorMap* out, const void* ptr, uint64_t pitch, uint64_t rows, uint64_t sstride, uint64_t nslots) {
    struct Key {
        const void* p; uint64_t pitch, rows, ss, ns;
        bool operator<(const Key& o) const { return std::tie(p, pitch, rows, ss, ns) < std::tie(o.p, o.pitch, o.rows, o.ss, o.ns); }
    };
    static std::map<Key, CUtensorMap> cache;
    static std::mutex mu;
    std::lock_guard<std::mutex> g(mu);
    const Key k{ptr, pitch, rows, sstride, nslots};
    auto it = cache.find(k);
    if (it != cache.end()) { *out = it->second; return 0; }
    CUtensorMap m;
    const int rc = make_map_bytes_3d(&m, ptr, pitch, rows, sstride, nslots, (uint32_t)kBoxBytes, (uint32_t)kTBM);
    if (rc) return rc;
    if (cache.size() > 65536) cache.clear();
    cache[k] = m;
    *out = m;
    return 0;
}

static int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

template <int FMT, int BN, bool GATEUP, int DIRECT = 0>
static int launch_moe_tc(const CUtensorMap& mb, const MoeTcParams& p, int nout, int max_tiles, cudaStream_t st) {
    const int Kred = GATEUP || p.up ? p.ef.H : p.ef.F;
    CUtensorMap mw0, mw1;
    {
        // byte views of the weight matrices over every slot of the arena (dense mode: one "slot")
        const uint64_t pitch = (uint64_t)(FMT == 0 ? Kred * 2 : FMT == 1 ? Kred : FMT == 2 ? Kred / 2 : Kred / 256 * 144);
        const bool dense = p.ef.stride == 0;
        const uint64_t sstride = dense ? pitch * (uint64_t)nout : (uint64_t)p.ef.stride;
        const uint64_t nslots = dense ? 1 : (uint64_t)kMaxSlots;
        int rc = cached_map_w(&mw0, p.arena + (GATEUP ? p.ef.off_gate : (p.up ? p.ef.off_up : p.ef.off_down)), pitch, (uint64_t)nout, sstride, nslots);
        if (rc) return rc;
        if (GATEUP) { rc = cached_map_w(&mw1, p.arena + p.ef.off_up, pitch, (uint64_t)nout, sstride, nslots); if (rc) return rc; }
        else mw1 = mw0;
    }
    using C = MoeTcCfg<FMT, BN, GATEUP, DIRECT>;
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(moe_tc_ffn_kernel<FMT, BN, GATEUP, DIRECT>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM); attr = true; }
    const long long work = (long long)(nout / kTBM) * max_tiles;
    const int grid = (int)(work < sm_count() ? (work > 0 ? work : 1) : sm_count());
    launch_pdl((moe_tc_ffn_kernel<FMT, BN, GATEUP, DIRECT>), grid, C::THREADS, C::SMEM, st, mb, mw0, mw1, p);
    return (int)cudaGetLastError();
}

template <int BN, bool GATEUP>
static int dispatch_fmt(int fmt, const CUtensorMap& mb, const MoeTcParams& p, int nout, int max_tiles, cudaStream_t st) {
    switch (fmt) {
        case 0: return launch_moe_tc<0, BN, GATEUP>(mb, p, nout, max_tiles, st);
        case 1: return launch_moe_tc<1, BN, GATEUP>(mb, p, nout, max_tiles, st);
        case 2: return launch_moe_tc<2, BN, GATEUP>(mb, p, nout, max_tiles, st);
        case 3: return launch_moe_tc<3, BN, GATEUP>(mb, p, nout, max_tiles, st);
    }
    return -1;
}

}  // namespace lsb
using namespace lsb;

// Role-level cycle table of tuning builds (see PROF_SCOPE); -1 in a normal build.
LSB_API int lsb_moe_tc_prof_read(void* out32, int reset, void* stream) {
    (void)stream;
#ifdef LSB_MOE_PROFILE
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(out32, g_moe_prof, sizeof(unsigned long long) * 32);
    if (reset) { unsigned long long z[32] = {0}; cudaMemcpyToSymbol(g_moe_prof, z, sizeof(z)); }
    return 0;
#else
    (void)out32; (void)reset;
    return -1;
#endif
}

// Tiles of at most `BN` (32, 64, 128; 256 over bf16 experts) sorted rows.  tile_* arrays hold npairs / BN + E_total + 1 entries,
// counters 2 ints, sorted_pair npairs ints.
LSB_API int lsb_moe_tc_sort(const void* ids, int npairs, int E_total, int BN, void* sorted_pair, void* tile_expert, void* tile_row0,
                            void* tile_n, void* counters, void* stream) {
    if (E_total > 4000 || (BN != 32 && BN != 64 && BN != 128 && BN != 256)) return -1;
    launch_pdl((moe_tc_sort_kernel), 1, 1024, (size_t)(3 * E_total + 2) * 4, (cudaStream_t)stream, (const int*)ids, npairs, E_total, BN,
               (int*)sorted_pair, (int*)tile_expert, (int*)tile_row0, (int*)tile_n, (int*)counters);
    LSB_CHECK_LAUNCH();
}

LSB_API int lsb_moe_tc_gather(const void* x, const void* sorted_pair, const void* counters, void* xs, int npairs, int S, int H, void* stream) {
    if (H % 8) return -1;
    launch_pdl((moe_tc_gather_kernel), npairs, 128, 0, (cudaStream_t)stream, (const bf16*)x, (const int*)sorted_pair, (const int*)counters,
               (__half*)xs, S, H);
    LSB_CHECK_LAUNCH();
}

LSB_API int lsb_moe_tc_gather_bf16(const void* x, const void* sorted_pair, const void* counters, void* xs, int npairs, int S, int H, void* stream) {
    if (H % 8 || (((uintptr_t)x | (uintptr_t)xs) & 15)) return -1;
    launch_pdl((moe_tc_gather_bf16_kernel), npairs, 128, 0, (cudaStream_t)stream, (const bf16*)x, (const int*)sorted_pair, (const int*)counters, (bf16*)xs, S, H);
    LSB_CHECK_LAUNCH();
}

// gateup != 0: act[pos][f] = SwiGLU(xs[pos] . Wgate[f], xs[pos] . Wup[f]) for every sorted position (fp16, [cap_rows, F]).
// gateup == 0: y[pair][h] = act[pos] . Wdown[h]  (fp32, [npairs, H], rows in pair order).
// gateup == 2: act[pos][f] = relu(xs[pos] . Wup[f])^2 (experts without a gate).
// `b` is the fp16 token operand ([cap_rows, K], K = H for gate/up and F for down), 16-byte aligned.
static int moe_tc_ffn(int gateup, const void* b, int cap_rows, const void* arena, const void* slot_of, const void* fmt_struct,
                           const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                           const void* sorted_pair, void* out, int BN, int max_tiles, GluAct ga, void* miss_flag, void* err,
                           const void* ep, void* stream, int direct = 0) {
    const ExpertFmt* ef = (const ExpertFmt*)fmt_struct;
    const int K = gateup ? ef->H : ef->F, nout = gateup ? ef->F : ef->H;
    if (gateup == 2 && ep) return -1;
    if (K % kTBK || nout % kTBM || ((uintptr_t)b & 15)) return -1;
    if (ef->fmt == 1 && (K % 128)) return -1;
    if (ef->fmt == 3 && (K % 256)) return -1;
    CUtensorMap mb;
    int rc = cached_map_2d(&mb, b, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)cap_rows, (uint64_t)K, (uint64_t)K, BN > 128 ? 128u : (uint32_t)BN, kTBK);
    if (rc) return rc;
    MoeTcParams p;
    p.arena = (const uint8_t*)arena; p.slot_of = (const int*)slot_of; p.ef = *ef;
    p.tile_expert = (const int*)tile_expert; p.tile_row0 = (const int*)tile_row0; p.tile_n = (const int*)tile_n;
    p.counters = (const int*)counters; p.sorted_pair = (const int*)sorted_pair;
    p.act = gateup ? (__half*)out : nullptr; p.y = gateup ? nullptr : (float*)out;
    p.ga = ga; p.miss_flag = (int*)miss_flag; p.err = (int*)err;
    if (ep) p.ep = *(const EpComm*)ep; else { memset(&p.ep, 0, sizeof(p.ep)); }
    p.ldo = nout; p.out_bf16 = 0; p.down_scale = 0.f; p.up = gateup == 2;
    cudaStream_t st = (cudaStream_t)stream;
    if (direct == kDirectBf16) {
        if (gateup < 0 || gateup > 1 || ef->fmt != 0 || BN != 32 || ep) return -1;
        return gateup ? launch_moe_tc<0, 32, true, kDirectBf16>(mb, p, nout, max_tiles, st) : launch_moe_tc<0, 32, false, kDirectBf16>(mb, p, nout, max_tiles, st);
    } else if (direct) {
        if (gateup != 1 || ef->fmt != 0 || ep) return -1;
        switch (BN) {
            case 32: return launch_moe_tc<0, 32, true, kDirect>(mb, p, nout, max_tiles, st);
            case 64: return launch_moe_tc<0, 64, true, kDirect>(mb, p, nout, max_tiles, st);
            case 128: return launch_moe_tc<0, 128, true, kDirect>(mb, p, nout, max_tiles, st);
            case 256: return launch_moe_tc<0, 256, true, kDirect>(mb, p, nout, max_tiles, st);
        }
    } else if (gateup == 1) {
        switch (BN) {
            case 32: return dispatch_fmt<32, true>(ef->fmt, mb, p, nout, max_tiles, st);
            case 64: return dispatch_fmt<64, true>(ef->fmt, mb, p, nout, max_tiles, st);
            case 128: return dispatch_fmt<128, true>(ef->fmt, mb, p, nout, max_tiles, st);
        }
    } else {
        switch (BN) {
            case 32: return dispatch_fmt<32, false>(ef->fmt, mb, p, nout, max_tiles, st);
            case 64: return dispatch_fmt<64, false>(ef->fmt, mb, p, nout, max_tiles, st);
            case 128: return dispatch_fmt<128, false>(ef->fmt, mb, p, nout, max_tiles, st);
            case 256: if (ef->fmt == 0 && !ep) return launch_moe_tc<0, 256, false>(mb, p, nout, max_tiles, st);
        }
    }
    return -1;
}

LSB_API int lsb_moe_tc_ffn(int gateup, const void* b, int cap_rows, const void* arena, const void* slot_of, const void* fmt_struct,
                           const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                           const void* sorted_pair, void* out, int BN, int max_tiles, float limit, void* miss_flag, void* err,
                           const void* ep, void* stream) {
    return moe_tc_ffn(gateup, b, cap_rows, arena, slot_of, fmt_struct, tile_expert, tile_row0, tile_n, counters, sorted_pair, out, BN, max_tiles,
                      GluAct{limit, 1.f, 0.f, nullptr}, miss_flag, err, ep, stream);
}

// The gate/up half over bf16 experts and bf16 token rows (lsb_moe_tc_gather_bf16): both go to the tensor core as they are, which is exact where the other
// form rounds weights outside fp16's normal range, and needs no converters.  1500 rows x top-8 of 64 experts of 4096 x 2048: 832 us through the converters,
// 505 us so in tiles of 128 (bound by shared memory: 112 KB of operands read and written per 64 elements, 875 cycles beside 512 of MMA), 424 in tiles of 256.
LSB_API int lsb_moe_tc_gateup_bf16(const void* b, int cap_rows, const void* arena, const void* slot_of, const void* fmt_struct,
                                   const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                                   const void* sorted_pair, void* out, int BN, int max_tiles, float limit, float alpha, float shift, const void* in_scale,
                                   void* miss_flag, void* err, void* stream) {
    return moe_tc_ffn(1, b, cap_rows, arena, slot_of, fmt_struct, tile_expert, tile_row0, tile_n, counters, sorted_pair, out, BN, max_tiles,
                      GluAct{limit, alpha, shift, (const float*)in_scale}, miss_flag, err, nullptr, stream, kDirect);
}

// Both halves over bf16 experts with hidden values in bf16 (`act` [cap_rows, F] bf16: out of gateup = 1, `b` of gateup = 0), in tiles of 32 rows: the roundings
// and the range of the weight-streaming kernels, for steps of few rows.
LSB_API int lsb_moe_tc_ffn_bf16(int gateup, const void* b, int cap_rows, const void* arena, const void* slot_of, const void* fmt_struct,
                                const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                                const void* sorted_pair, void* out, int BN, int max_tiles, float limit, float alpha, float shift, const void* in_scale,
                                void* miss_flag, void* err, void* stream) {
    return moe_tc_ffn(gateup, b, cap_rows, arena, slot_of, fmt_struct, tile_expert, tile_row0, tile_n, counters, sorted_pair, out, BN, max_tiles,
                      GluAct{limit, alpha, shift, (const float*)in_scale}, miss_flag, err, nullptr, stream, kDirectBf16);
}

// The gate/up half with another gated unit (GluAct): in_scale [npairs] in pair order, or null.
LSB_API int lsb_moe_tc_gateup_act(const void* b, int cap_rows, const void* arena, const void* slot_of, const void* fmt_struct,
                                  const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                                  const void* sorted_pair, void* out, int BN, int max_tiles, float limit, float alpha, float shift, const void* in_scale,
                                  void* miss_flag, void* err, void* stream) {
    return moe_tc_ffn(1, b, cap_rows, arena, slot_of, fmt_struct, tile_expert, tile_row0, tile_n, counters, sorted_pair, out, BN, max_tiles,
                      GluAct{limit, alpha, shift, (const float*)in_scale}, miss_flag, err, nullptr, stream);
}

// Dense linear layer with quantised weights on the tensor cores: out[m][n] = alpha * sum_k x16[m][k] * W[n][k].
// x16: fp16 [M, K] contiguous; W in storage format `fmt` (0 bf16, 1 fp8 e4m3 + 128x128 block scales, 2 nvfp4 + group-scale
// atoms) with `scales`; out fp32 or bf16 with row stride ldo.  The caller provides the (constant per M) tile description:
// tile_expert = 0, tile_row0 = t*BN, tile_n, counters = {tiles, M}, ident[m] = m, slot0 = {0}.
LSB_API int lsb_gemm_q_tc(void* out, const void* x16, const void* w, const void* scales, int fmt, int M, int N, int K, int ldo, int out_bf16,
                          float alpha, const void* tile_expert, const void* tile_row0, const void* tile_n, const void* counters,
                          const void* ident, const void* slot0, int BN, int n_tiles, void* err, void* stream) {
    if (K % kTBK || N % kTBM || ((uintptr_t)x16 & 15) || fmt < 0 || fmt > 3) return -1;
    if ((fmt == 1 && (K % 128)) || (fmt == 3 && (K % 256))) return -1;
    CUtensorMap mb;
    int rc = cached_map_2d(&mb, x16, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)BN, kTBK);
    if (rc) return rc;
    MoeTcParams p;
    memset(&p, 0, sizeof(p));
    p.arena = (const uint8_t*)w; p.slot_of = (const int*)slot0;
    p.ef.fmt = fmt; p.ef.H = N; p.ef.F = K; p.ef.stride = 0; p.ef.off_down = 0;
    p.ef.off_sd = scales ? (long long)((const uint8_t*)scales - (const uint8_t*)w) : 0;
    p.tile_expert = (const int*)tile_expert; p.tile_row0 = (const int*)tile_row0; p.tile_n = (const int*)tile_n;
    p.counters = (const int*)counters; p.sorted_pair = (const int*)ident;
    p.y = (float*)out; p.err = (int*)err; p.ldo = ldo; p.out_bf16 = out_bf16;
    p.down_scale = fmt == 2 ? alpha : 0.f;
    if (fmt != 2 && alpha != 1.0f) return -1;
    cudaStream_t st = (cudaStream_t)stream;
    switch (BN) {
        case 32: return dispatch_fmt<32, false>(fmt, mb, p, N, n_tiles, st);
        case 64: return dispatch_fmt<64, false>(fmt, mb, p, N, n_tiles, st);
        case 128: return dispatch_fmt<128, false>(fmt, mb, p, N, n_tiles, st);
    }
    return -1;
}

LSB_API int lsb_trace_set_moe_tc(void* buf) { return lsb_trace_install(buf); }
