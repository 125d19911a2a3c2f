// Five to sixteen rows over a bf16 matrix: the scheme of fp8_rows.cuh without conversions.
//
// A warp owns 16 weight rows and every kw-th block of 64 reduction elements; a thread's 16-byte pieces, copied into a ring in shared memory and read by the thread that
// copied them, are its fragments of four mma.sync (m16n8k16, fp32 sums) when the reduction is taken in another order (thread c of a row's four: elements
// 8 c .. 8 c + 7 of 32).  One block per SM, which stages the activation rows once.  Bound by DRAM; the tcgen05 GEMM gives 128 weight rows to a CTA, so that few-row
// products have CTAs of up to two different loads per SM, or a reduction that is split and added up by a launch of its own.
#pragma once
#include "fp8_rows.cuh"

namespace lsb {

struct Bf16RowsArgs {
    const bf16* x; int ldx; const bf16* w; int ldw;
    void* out; int ldo, out_bf16; const float* bias;
    int M, N, K, kw, cols;                                             // warps per 16 rows, activation rows per pass
    int steady;                                                        // the kernel before does not write w
};

// NC: sets of eight activation rows; NS: weight blocks in flight per warp.
template <int NC, int NS>
__global__ void __launch_bounds__(kF8Warps * 32, 1) bf16_rows_kernel(const Bf16RowsArgs a) {
    constexpr int NT = kF8Warps * 32;
    extern __shared__ __align__(16) uint8_t b16_smem[];                // [NS][warps][4][32] 16-byte pieces, then
    bf16* xs = reinterpret_cast<bf16*>(b16_smem + NS * kF8Ring);       // [cols][K + 8]
    __shared__ float red[kF8Warps][16][8 * NC + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int K = a.K, nkb = K >> 6, kw = a.kw, ks = warp % kw, sub = warp / kw, per = kF8Warps / kw;
    const int units = (a.N / 16 + per - 1) / per, passes = (a.M + a.cols - 1) / a.cols;
    const int step = gridDim.x / passes, u0 = blockIdx.x / passes, pass = blockIdx.x % passes, m0 = pass * a.cols, ncols = min(a.cols, a.M - m0);
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(b16_smem) + (uint32_t)(warp * 2048 + lane * 16);
    int pu = u0, pk = ks;                                              // unit and block that are asked for next
    auto ask = [&](int stage) {                                        // rows g and g + 8, both halves of 32: one group, empty behind the end
        const int tile = pu * per + sub;
        if (pu < units && tile * 16 < a.N) {
            const uint8_t* p = reinterpret_cast<const uint8_t*>(a.w + (size_t)(tile * 16 + g) * a.ldw + c * 8 + pk * 64);
            const size_t r8 = (size_t)a.ldw * 16;
            const uint32_t d = ring + (uint32_t)(stage * kF8Ring);
            f8_copy(d, p); f8_copy(d + 512, p + r8); f8_copy(d + 1024, p + 64); f8_copy(d + 1536, p + r8 + 64);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        pk += kw;
        if (pk >= nkb) { pk = ks; pu += step; }
    };
    if (!a.steady) pdl_wait();
#pragma unroll
    for (int i = 0; i < NS; ++i) ask(i);
    if (a.steady) pdl_wait();
    pdl_launch_dependents();
    for (int i = tid; i < ncols * (K / 8); i += NT) {
        const int m = i / (K / 8), k = i - m * (K / 8);
        *reinterpret_cast<uint4*>(xs + (size_t)m * (K + 8) + k * 8) = __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)(m0 + m) * a.ldx) + k);
    }
    __syncthreads();
    float tot[NC][4];
#pragma unroll
    for (int n = 0; n < NC; ++n) tot[n][0] = tot[n][1] = tot[n][2] = tot[n][3] = 0.f;
    int u = u0, kb = ks, stage = 0;
#pragma unroll 1
    while (u < units) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
        if ((u * per + sub) * 16 < a.N) {
            const uint32_t d = ring + (uint32_t)(stage * kF8Ring);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 lo = f8_read(d + 1024 * h), hi = f8_read(d + 1024 * h + 512);
                uint4 b[NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    b[n] = make_uint4(0u, 0u, 0u, 0u);
                    if (n * 8 + g < ncols) b[n] = *reinterpret_cast<const uint4*>(xs + (size_t)(n * 8 + g) * (K + 8) + kb * 64 + h * 32 + c * 8);
                }
                __syncwarp();
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    rows_mma(tot[n], lo.x, hi.x, lo.y, hi.y, b[n].x, b[n].y);
                    rows_mma(tot[n], lo.z, hi.z, lo.w, hi.w, b[n].z, b[n].w);
                }
            }
        }
        ask(stage);
        stage = stage + 1 == NS ? 0 : stage + 1;
        kb += kw;
        if (kb >= nkb) {                                               // (every warp has a block of every unit)
            __syncthreads();                                           // readers of the unit before are done
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                red[warp][g][n * 8 + 2 * c] = tot[n][0]; red[warp][g][n * 8 + 2 * c + 1] = tot[n][1];
                red[warp][g + 8][n * 8 + 2 * c] = tot[n][2]; red[warp][g + 8][n * 8 + 2 * c + 1] = tot[n][3];
                tot[n][0] = tot[n][1] = tot[n][2] = tot[n][3] = 0.f;
            }
            __syncthreads();
            for (int o = tid; o < per * 16 * ncols; o += NT) {
                const int rr = o & 15, m = (o >> 4) % ncols, t = (o >> 4) / ncols, n = (u * per + t) * 16 + rr;
                if (n >= a.N) continue;
                float y = a.bias ? a.bias[n] : 0.f;
                for (int i = 0; i < kw; ++i) y += red[t * kw + i][rr][m];
                if (a.out_bf16) reinterpret_cast<bf16*>(a.out)[(size_t)(m0 + m) * a.ldo + n] = __float2bfloat16(y);
                else reinterpret_cast<float*>(a.out)[(size_t)(m0 + m) * a.ldo + n] = y;
            }
            kb = ks;
            u += step;
        }
    }
    pdl_launch_dependents();
}

// Up to eight rows that are staged in one pass, of matrices up to 256 MB (behind that both forms run at DRAM's rate; out of a clean cache, us, 5 and 8 rows):
//   576 x 4096   before 6.4, 6.7   here 3.8, 4.2       16384 x 1536   12.1, 12.4   9.5, 10.1       4096 x 8192    15.9, 16.1   13.6, 16.5 (two passes)
//   4096 x 4096  10.4, 10.7        7.3, 7.7            24896 x 4096   37.0, 37.2   34.8, 35.5      4096 x 12288   21.4, 21.8   23.9, 25.2 (two passes)
// More rows, which cost an mma and shared memory reads per set of eight, only in matrices below 64 MB, where the two launches of a split reduction count (12 and 16 rows):
//   576 x 4096   before 7.1, 7.5   here 5.4, 4.3       16384 x 1536   13.1, 13.9   11.5, 12.5      16384 x 4096   26.3, 27.0   27.9, 29.9
//   4096 x 4096  11.2, 11.7        9.3, 10.5           2048 x 12288   14.3, 14.9   18.3, 22.2      24896 x 4096   37.7, 38.2   39.4, 44.6
// Against 64 bits 4096 x 8192 is off 5e-7, 2e-6 before.
inline bool bf16_rows_ok(int M, int N, int K, int ldx, int ldw, const void* x, const void* w) {
    if (M < 1 || M > 16 || N < 16 || N % 16 || K < 64 || K % 64 || ldx % 8 || ldw % 8 || (((uintptr_t)x | (uintptr_t)w) & 15)) return false;
    const long long nk = (long long)N * K;
    return M <= 8 ? M * (K + 8) * 2 <= kF8Rows && nk <= (128 << 20) : K <= 4096 && nk < (32 << 20);
}
template <int NC, int NS> inline int bf16_rows_start(const Bf16RowsArgs& a, int grid, int rows, cudaStream_t st) {
    static const cudaError_t attr = cudaFuncSetAttribute(bf16_rows_kernel<NC, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kF8Smem);
    (void)attr;
    launch_pdl((bf16_rows_kernel<NC, NS>), grid, kF8Warps * 32, (size_t)(NS * kF8Ring + rows), st, a);
    return (int)cudaGetLastError();
}
inline int bf16_rows_launch(Bf16RowsArgs a, cudaStream_t st) {
    const int row = (a.K + 8) * 2;
    a.kw = fp8_rows_kw(a.N, a.K * 2);
    a.cols = a.M < kF8Rows / row ? a.M : kF8Rows / row;
    const int passes = (a.M + a.cols - 1) / a.cols;
    a.cols = (a.M + passes - 1) / passes;                              // evenly
    const int per = kF8Warps / a.kw, units = (a.N / 16 + per - 1) / per, rows = a.cols * row;
    int step = kF8Resident / passes;
    step = step < 1 ? 1 : (step > units ? units : step);
    if (a.cols <= 8) {
        if (rows + 6 * kF8Ring <= kF8Smem) return bf16_rows_start<1, 6>(a, step * passes, rows, st);
        if (rows + 4 * kF8Ring <= kF8Smem) return bf16_rows_start<1, 4>(a, step * passes, rows, st);
        return bf16_rows_start<1, 3>(a, step * passes, rows, st);
    }
    if (rows + 4 * kF8Ring <= kF8Smem) return bf16_rows_start<2, 4>(a, step * passes, rows, st);
    return bf16_rows_start<2, 3>(a, step * passes, rows, st);
}

}  // namespace lsb
