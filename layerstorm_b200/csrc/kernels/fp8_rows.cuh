// Few rows over FP8 weights (e4m3, fp32 scales of 128 x 128 blocks): dense matrices and the experts of decode and verification steps.
//
// A warp owns 16 weight rows and every KW-th block of 128 reduction elements.  A thread's 16-byte pieces are already its share of the mma fragments when
// the reduction is taken in another order (thread c of a row's four: elements 16 c .. 16 c + 15 of 64), so weights go from DRAM into a ring in shared memory, from there
// to the registers of the thread that copied them, from e4m3 to bf16 (exact), and into mma.sync (m16n8k16, fp32 sums) for up to eight activation rows at once,
// which are bf16 as they come; a block's sum is multiplied by its scale in fp32.  Products are exact, whatever lies beside them.
// Bound by DRAM and, with several rows, by the warps' chains of conversions and products.  The form with a multiplication per weight and row took 8 scheduler cycles for two
// weights and one row (conversion, two halves to floats, two FMAs), and read the weights again from the fifth row on.  Before, now (us), out of a clean cache: 36864 x 7168
// 1 row 64, 57, 6 rows 203, 61 (DRAM's rate: 41); 7168 x 16384 36, 38 and 118, 55 (18); 256 + 1 experts of 7168 x 2048, top 8 + 1, gate/up and down: 1 row 94 and 59, 61 and 35
// (41 and 20), 6 rows 442 and 266, 307 and 162 (209 and 104).  Against 64 bits 36864 x 7168 is off 8e-8, 2e-7 before.  fp16 operands, a conversion less per weight, take
// 2 to 6 % less (54, 57; 36, 50; experts of 6 rows 300 and 156) but need a power of two per row, and what lies 2^-31 below a row's largest element loses bits.
#pragma once
#include "gemv_core.cuh"
#include "moe_fmt.cuh"

namespace lsb {

constexpr int kF8Cols = 8;             // activation rows of an mma
constexpr int kF8Warps = 16;           // one block per SM
constexpr int kF8Smem = 210 * 1024;    // staged rows and the ring of weight blocks (17 KB more are static)
constexpr int kF8Ring = kF8Warps * 2048;                               // a block of 16 x 128 weights for every warp
constexpr int kF8Rows = kF8Smem - 3 * kF8Ring;                         // staged rows at most

enum { kF8Dense = 0, kF8GateUp = 1, kF8Down = 2 };

struct Fp8RowsArgs {
    const bf16* x; int ldx;                                            // dense: [M, ldx]; experts: token rows / hidden values, contiguous
    int N, K, M, kw, cols;                                             // warps per 16 rows, activation rows per pass
    const uint8_t* w; const float* scales;                             // dense
    void* out; int ldo, out_bf16; float alpha; const float* bias;      // dense; down: out = y [pairs, N] fp32; gate/up: act [pairs, N] bf16
    const uint8_t* arena; const int* slot_of; ExpertFmt ef;
    const int* group_expert; const int* group_n; const int* group_pairs; const int* n_groups;
    int S; GluAct ga; int* miss_flag;
};

// Two weights as bf16, which holds every e4m3 value, NaN among them.
__device__ __forceinline__ uint32_t f8_pair(uint32_t two) {
    uint32_t r;
    asm("{\n .reg .b32 h;\n .reg .b16 l, u;\n .reg .f32 fl, fu;\n cvt.rn.f16x2.e4m3x2 h, %1;\n mov.b32 {l, u}, h;\n cvt.f32.f16 fl, l;\n cvt.f32.f16 fu, u;\n"
        " cvt.rn.bf16x2.f32 %0, fu, fl;\n}" : "=r"(r) : "h"((uint16_t)two));
    return r;
}
__device__ __forceinline__ void rows_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void f8_copy(uint32_t dst, const uint8_t* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 f8_read(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// NS: weight blocks in flight per warp, in a ring in shared memory of which every thread copies and reads its own 16-byte pieces (registers hold three at the
// most: 3 TB/s).
template <int MODE, int NS>
__global__ void __launch_bounds__(kF8Warps * 32, 1) fp8_rows_kernel(const Fp8RowsArgs a) {
    constexpr int NT = kF8Warps * 32;
    extern __shared__ __align__(16) uint8_t f8_smem[];                 // [NS][warps][4][32] 16-byte pieces, then
    bf16* xs = reinterpret_cast<bf16*>(f8_smem + NS * kF8Ring);        // [cols][K + 8]: rows 16 bytes apart in the banks
    __shared__ float red[2][kF8Warps][16][kF8Cols];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int K = a.K, nkb = K >> 7, kw = a.kw, ks = warp % kw, sub = warp / kw, per = MODE == kF8GateUp ? 1 : kF8Warps / kw;
    // A block stages its rows once and takes every step-th unit of `per` tiles of 16 weight rows; what a warp asks for next runs on from one to the next.
    const int units = (a.N / 16 + per - 1) / per, passes = MODE == kF8Dense ? (a.M + a.cols - 1) / a.cols : 1;
    const int step = gridDim.x / passes, u0 = MODE == kF8Dense ? blockIdx.x / passes : blockIdx.x;       // the passes over a unit run side by side
    int ncols;
    const uint8_t* w;
    const float* scales;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(f8_smem) + (uint32_t)(warp * 2048 + lane * 16);
    int pu = u0, pk = ks;                                              // unit and block that are asked for next
    auto ask = [&](int stage) {                                        // rows g and g + 8, both halves of 64: one group, empty behind the end
        const int tile = MODE == kF8GateUp ? pu : pu * per + sub;
        if (pu < units && tile * 16 < a.N) {
            const uint8_t* p = w + (size_t)(tile * 16 + g) * K + c * 16 + pk * 128;
            const uint32_t d = ring + (uint32_t)(stage * kF8Ring);
            f8_copy(d, p); f8_copy(d + 512, p + (size_t)K * 8); f8_copy(d + 1024, p + 64); f8_copy(d + 1536, p + (size_t)K * 8 + 64);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        pk += kw;
        if (pk >= nkb) { pk = ks; pu += step; }
    };
    if constexpr (MODE == kF8Dense) {
        const int pass = blockIdx.x % passes;
        ncols = min(a.cols, a.M - pass * a.cols);
        w = a.w; scales = a.scales;
#pragma unroll
        for (int i = 0; i < NS; ++i) ask(i);                      // weights do not depend on the kernel before
        pdl_wait();
        pdl_launch_dependents();
    } else {
        pdl_wait();
        pdl_launch_dependents();
        const int grp = blockIdx.y;
        if (grp >= a.n_groups[0]) return;
        const int e = a.group_expert[grp], slot = a.slot_of[e];
        if (slot < 0) {
            if (MODE == kF8GateUp && a.miss_flag && tid == 0 && blockIdx.x == 0) atomicExch(a.miss_flag, e + 1);
            return;
        }
        const uint8_t* base = a.arena + (size_t)slot * a.ef.stride;
        w = base + (MODE == kF8Down ? a.ef.off_down : (sub ? a.ef.off_up : a.ef.off_gate));
        scales = reinterpret_cast<const float*>(base + (MODE == kF8Down ? a.ef.off_sd : (sub ? a.ef.off_su : a.ef.off_sg)));
#pragma unroll
        for (int i = 0; i < NS; ++i) ask(i);
        ncols = min(a.group_n[grp], 4);
    }
    auto pair_of = [&](int m) { return MODE == kF8Dense ? (int)(blockIdx.x % passes) * a.cols + m : a.group_pairs[blockIdx.y * 4 + m]; };
    // ---- rows: some warps for each, a row's loads on their way together
    const int wpr = kF8Warps / ncols, xm = warp / wpr;
    if (xm < ncols) {
        const int p = pair_of(xm);
        const uint4* xp = reinterpret_cast<const uint4*>(MODE == kF8Dense ? a.x + (size_t)p * a.ldx : a.x + (size_t)(MODE == kF8GateUp ? p / a.S : p) * K);
#pragma unroll 8
        for (int k = warp % wpr * 32 + lane; k < K / 8; k += wpr * 32) *reinterpret_cast<uint4*>(xs + (size_t)xm * (K + 8) + k * 8) = __ldg(xp + k);
    }
    __syncthreads();
    // ---- products
    float tot[4] = {0.f, 0.f, 0.f, 0.f};
    const bf16* xb = xs + (size_t)min(g, ncols - 1) * (K + 8) + c * 16;
    const bool have = g < ncols;
    int u = u0, kb = ks, par = 0;
    auto finish = [&]() {
        // the warps' shares in order; the next unit's go to the other half of `red`
        float (*r)[16][kF8Cols] = red[par];
        r[warp][g][2 * c] = tot[0]; r[warp][g][2 * c + 1] = tot[1];
        r[warp][g + 8][2 * c] = tot[2]; r[warp][g + 8][2 * c + 1] = tot[3];
        __syncthreads();
        for (int o = tid; o < per * 16 * ncols; o += NT) {
            const int rr = o & 15, m = (o >> 4) % ncols, t = (o >> 4) / ncols, n = (u * per + t) * 16 + rr;
            if (n >= a.N) continue;
            float v = 0.f, up = 0.f;
            for (int i = 0; i < kw; ++i) {
                v += r[t * kw + i][rr][m];
                if (MODE == kF8GateUp) up += r[kw + i][rr][m];
            }
            const int pair = pair_of(m);
            if constexpr (MODE == kF8GateUp) {
                const float f = glu_in_scale(a.ga, pair);
                reinterpret_cast<bf16*>(a.out)[(size_t)pair * a.N + n] = __float2bfloat16(glu_act(v * f, up * f, a.ga));
            } else if constexpr (MODE == kF8Down) {
                reinterpret_cast<float*>(a.out)[(size_t)pair * a.N + n] = v;
            } else {
                float y = v * a.alpha;
                if (a.bias) y += a.bias[n];
                if (a.out_bf16) reinterpret_cast<bf16*>(a.out)[(size_t)pair * a.ldo + n] = __float2bfloat16(y);
                else reinterpret_cast<float*>(a.out)[(size_t)pair * a.ldo + n] = y;
            }
        }
        par ^= 1;
        tot[0] = tot[1] = tot[2] = tot[3] = 0.f;
        kb = ks;
        u += step;
    };
    // (every warp has at least one block of a unit; all finish the same units)
    int stage = 0;
#pragma unroll 1
    while (u < units) {
        const int tile = MODE == kF8GateUp ? u : u * per + sub;
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
        if (tile * 16 < a.N) {
            const float s = __ldg(scales + (size_t)(tile >> 3) * nkb + kb);
            const uint32_t d = ring + (uint32_t)(stage * kF8Ring);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 lo = f8_read(d + 1024 * h), hi = f8_read(d + 1024 * h + 512);
                uint4 b[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
                if (have) {
                    const uint4* xp = reinterpret_cast<const uint4*>(xb + kb * 128 + h * 64);
                    b[0] = xp[0]; b[1] = xp[1];
                }
                __syncwarp();
                const uint32_t wl[4] = {lo.x, lo.y, lo.z, lo.w}, wh[4] = {hi.x, hi.y, hi.z, hi.w};
                const uint32_t bb[8] = {b[0].x, b[0].y, b[0].z, b[0].w, b[1].x, b[1].y, b[1].z, b[1].w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    rows_mma(acc, f8_pair(wl[j]), f8_pair(wh[j]), f8_pair(wl[j] >> 16), f8_pair(wh[j] >> 16), bb[2 * j], bb[2 * j + 1]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) tot[q] = fmaf(s, acc[q], tot[q]);
        }
        ask(stage);
        stage = stage + 1 == NS ? 0 : stage + 1;
        kb += kw;
        if (kb >= nkb) finish();
    }
    pdl_launch_dependents();
}

constexpr int kF8Resident = 148;       // blocks on the GPU at a time

// Warps that share 16 rows: as few as leave each six blocks of 128 elements, more (down to four blocks) where units are too few for two a thread block.  A matrix'
// own choice, whatever the rows, so that a row's sums do not depend on its company.
inline int fp8_rows_kw(int N, int K) {
    const int nkb = K >> 7;
    int kw = 1;
    while (kw < kF8Warps && nkb >= 12 * kw) kw *= 2;
    while (kw < kF8Warps && nkb >= 8 * kw && N / 16 * kw < 2 * kF8Warps * kF8Resident) kw *= 2;
    return kw;
}
inline bool fp8_rows_ok(const void* x, long long ldx, const void* w, int N, int K) {
    return K % 128 == 0 && N % 16 == 0 && ldx % 8 == 0 && (K + 8) * 2 <= kF8Rows && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
}
template <int MODE, int NS> inline int fp8_rows_start(const Fp8RowsArgs& a, dim3 grid, int rows, cudaStream_t st) {
    static const cudaError_t attr = cudaFuncSetAttribute(fp8_rows_kernel<MODE, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kF8Smem);
    (void)attr;
    launch_pdl((fp8_rows_kernel<MODE, NS>), grid, kF8Warps * 32, (size_t)(NS * kF8Ring + rows), st, a);
    return (int)cudaGetLastError();
}
template <int MODE> inline int fp8_rows_launch(Fp8RowsArgs a, int max_groups, cudaStream_t st) {
    const int row = (a.K + 8) * 2, most = MODE == kF8Dense ? kF8Cols : 4, fit = kF8Rows / row;
    if (MODE == kF8Dense ? a.M < 1 : max_groups < 1) return -1;
    if (MODE != kF8Dense && (fit < most || (MODE == kF8GateUp && a.K < 1024))) return -2;      // a group's rows are staged together; every warp has a block
    a.kw = MODE == kF8GateUp ? kF8Warps / 2 : fp8_rows_kw(a.N, a.K);
    a.cols = a.M < most ? a.M : most;
    if (a.cols > fit) a.cols = fit;
    const int passes = MODE == kF8Dense ? (a.M + a.cols - 1) / a.cols : 1;
    if (MODE == kF8Dense) a.cols = (a.M + passes - 1) / passes;        // evenly
    const int per = MODE == kF8GateUp ? 1 : kF8Warps / a.kw, units = (a.N / 16 + per - 1) / per;
    // one wave of blocks for a matrix or the experts of one or two rows; four for more experts, whose number is not known here
    int step = MODE == kF8Dense ? kF8Resident / passes : (max_groups <= 24 ? kF8Resident : 4 * kF8Resident) / max_groups;
    step = step < 1 ? 1 : (step > units ? units : step);
    const dim3 grid(step * passes, MODE == kF8Dense ? 1 : max_groups);
    const int rows = (MODE == kF8Dense ? a.cols : most) * row;
    if (rows + 6 * kF8Ring <= kF8Smem) return fp8_rows_start<MODE, 6>(a, grid, rows, st);
    if (rows + 4 * kF8Ring <= kF8Smem) return fp8_rows_start<MODE, 4>(a, grid, rows, st);
    return fp8_rows_start<MODE, 3>(a, grid, rows, st);
}

}  // namespace lsb
