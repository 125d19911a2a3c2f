// Tensor-core GEMM for sm_100a: Y[m][n] = sum_k X[m][k] * W[n][k]  (both operands K-major).
//
// The weight matrix is the 128-row UMMA "A" operand and the activations are the "B" operand
// (swap-AB), so any token count from 16 to thousands maps onto full 128-row tcgen05.mma
// instructions: N_umma = the token tile (16..256).  One CTA computes one [128 x BN] output
// tile (optionally one K split of it):
//     warp 0   one thread issues TMA tile loads (cp.async.bulk.tensor, 128-byte swizzle) into a
//              multi-stage shared-memory ring, completion on mbarriers
//     warp 1   allocates tensor memory; one thread issues tcgen05.mma (kind::f16, fp32 accumulate
//              in TMEM) and tcgen05.commit to release stages / publish the accumulator
//     warps 2-5 epilogue: tcgen05.ld the accumulator (one TMEM lane = one output column n), optional bias; bf16 rows of
//              16-byte pitch through shared memory and TMA, others and fp32 by stores coalesced over n
// This replaces the reference's CUDA-core tiled GEMM (src/compute/kernels/sm120/gemm/bf16_gemm.cu:156)
// and the external FP8 GEMM launcher (G/sm120/gemm/fp8/fp8_gemm.h).  Up to 16 rows of suitable matrices run on the few-row
// form of bf16_rows.cuh instead.
#include "tc_common.cuh"
#include "bf16_rows.cuh"
#include "comm.cuh"

#include <map>
#include <mutex>
#include <tuple>

namespace lsb {
using namespace tc;

constexpr int BM = 128;   // weight rows per tile (UMMA M)
constexpr int kSms = 148;
constexpr int BK = 64;    // bf16 elements per stage row = 128 bytes = one swizzle span

struct GemmTcParams {
    void* out; int ldo;            // [M, ldo] fp32 or bf16
    float* partial;                // [splits, M, N] fp32 when splits > 1
    const float* bias;             // [N] or null
    int M, N, K, out_bf16, splits, kb_per_split;
    int* err;
    long long out_bs;              // batched mode: elements between consecutive batches of `out` (blockIdx.z = batch)
    int tma_out;                   // bf16 rows that TMA can store (map_o)
    // fused all-reduce epilogue (row-parallel layers under tensor parallelism): instead of a local store, every tile of
    // the fp32 partial is stored into this rank's slot of every peer's receive buffer over NVLink; the last CTA
    // publishes the epoch.  The consuming kernel sums the slots in rank order.
    PeerComm comm;
};

// A CTA computes MT weight tiles of 128 rows against one token tile.  MT = 2 (512 x 256 outputs of TMEM, one CTA per SM) brings a third less
// through L2 per product than two CTAs of 128 x 256; MT = 1 has half the shared memory of an SM, so that two CTAs share one and the epilogue of
// one runs under the main loop of the other.  Measured (one CTA of 128 x 256 per SM, MT = 1 at half an SM, MT = 2): 2048 x 24896 x 4096 534, 446,
// 422 us; 2048 x 4096 x 12288 205, 182, 165 us; 391 x 16640 x 4096 119, 94, 89 us; MT = 1 with 64-row tiles and smaller: 32 x 24896 x 4096 66 -> 55 us
// (with an epilogue that took longer than the present one).
// DEEP: MT = 1 with twice the stages, for grids that give an SM one CTA at a time anyway.
template <int BN, int MT, bool DEEP = false> struct TcCfg {
    static constexpr int A_BYTES = BM * BK * 2;
    static constexpr int B_BYTES = BN * BK * 2;
    static constexpr int STAGE_BYTES = MT * A_BYTES + B_BYTES;
    static constexpr int STAGES = MT == 2 ? 3 : (BN >= 256 ? 2 : (BN >= 128 ? 3 : 4)) * (DEEP ? 2 : 1);
    static constexpr int TMEM_COLS = MT * (BN < 32 ? 32 : BN);
    static constexpr int THREADS = 64 + 128 * MT;
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

template <int BN, int MT = 1, bool BATCHED = false, bool DEEP = false>
__global__ void __launch_bounds__(TcCfg<BN, MT, DEEP>::THREADS) gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                                        const __grid_constant__ CUtensorMap map_o, GemmTcParams p) {
    using C = TcCfg<BN, MT, DEEP>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::STAGES * C::STAGE_BYTES);
    uint64_t* empty = full + C::STAGES;
    uint64_t* acc_full = empty + C::STAGES;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // token-row tiles are the fastest grid dimension: the blocks that share a weight tile run together, so the weight
    // matrix streams from DRAM once and the (much smaller) activation tiles stay in L2
    const int n0 = blockIdx.y * (BM * MT), m0 = blockIdx.x * BN;
    const int split = BATCHED ? 0 : blockIdx.z, batch = BATCHED ? blockIdx.z : 0;
    const int nkb_total = (p.K + BK - 1) / BK;
    const int kb0 = split * p.kb_per_split;
    const int kb1 = min(nkb_total, kb0 + p.kb_per_split);
    const int nkb = max(0, kb1 - kb0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        fence_barrier_init();
        fence_proxy_async();
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_x);
    }
    if (warp == 1) tmem_alloc(tmem_holder, C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = *tmem_holder;
    pdl_wait();
    pdl_launch_dependents();
    const unsigned next_epoch = p.comm.nranks ? *p.comm.epoch + 1u : 0u;

    if (warp == 0 && lane == 0) {
        // ---------------- TMA producer ----------------
        int issued = 0;
        bool ok = true;
        for (int it = 0; it < nkb && ok; ++it) {
            const int s = it % C::STAGES;
            const uint32_t ph = (it / C::STAGES) & 1;
            ok = mbar_wait(&empty[s], ph ^ 1, p.err, 1);
            if (!ok) break;
            uint8_t* a = smem + s * C::STAGE_BYTES;
            mbar_expect_tx(&full[s], C::STAGE_BYTES);
            if (BATCHED) {
                tma_load_3d(a, &map_w, &full[s], (kb0 + it) * BK, n0, batch);
                tma_load_3d(a + MT * C::A_BYTES, &map_x, &full[s], (kb0 + it) * BK, m0, batch);
            } else {
#pragma unroll
                for (int m = 0; m < MT; ++m) tma_load_2d(a + m * C::A_BYTES, &map_w, &full[s], (kb0 + it) * BK, n0 + m * BM);
                tma_load_2d(a + MT * C::A_BYTES, &map_x, &full[s], (kb0 + it) * BK, m0);
            }
            ++issued;
        }
        if (!ok) {
            // error path: let the loads already in flight land before this CTA's shared memory is released
            for (int it = max(0, issued - C::STAGES); it < issued; ++it) mbar_wait(&full[it % C::STAGES], (it / C::STAGES) & 1, nullptr, 0);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: the whole warp walks the stages, so that the operands of the instructions are warp-uniform; one elected
        // lane issues (a single thread's own loop takes about 90 cycles per instruction, more than the MMAs of a 256-row tile) ----------------
        constexpr uint32_t idesc = idesc_f16(BM, BN, 1);
        const uint32_t d = __reduce_max_sync(0xffffffffu, tmem_d);
        bool ok = true;
        uint32_t s = 0, ph = 0;
        for (int it = 0; it < nkb; ++it) {
            ok = __all_sync(0xffffffffu, mbar_wait(&full[s], ph, p.err, 2));
            if (!ok) break;
            tc_fence_after();
            const uint8_t* a = smem + s * C::STAGE_BYTES;
            const uint64_t da = smem_desc_sw128(a), db = smem_desc_sw128(a + MT * C::A_BYTES);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
#pragma unroll
                    for (int m = 0; m < MT; ++m) umma_f16(d + m * BN, da + m * (C::A_BYTES >> 4) + 2 * k, db + 2 * k, idesc, (it > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == C::STAGES) { s = 0; ph ^= 1u; }
        }
        if (ok && elect_one()) umma_commit(acc_full);
        __syncwarp();
    } else if (warp >= 2) {
        // ---------------- epilogue ----------------
        // Where the results go is settled once per tile, and lanes never part: what a lane must not store is a predicate of the store.  Worked out for
        // every output, the destination took 25 dependent instructions with one or two warps per scheduler - a quarter of the kernel's time at K = 4096 and
        // most of it at K = 256.  bf16 rows leave through shared memory (the stages, which nothing reads any more): 16 x 8 pieces of the accumulator
        // are packed and stored transposed by one instruction for 256 values, and TMA writes 64 columns of up to 64 rows and drops what lies
        // outside the matrix.  Before, now (us): 2048 x 24896 x 4096 fp32 408, 297 (1406 TFLOP/s), bf16 390, 279 (1500); 2048 x 4096 x 12288 156, 133;
        // 2048 x 20480 x 1536 bf16 207, 107; 391 x 16640 x 4096 bf16 80, 57; 64 products of 2048 x 512 x 256 207, 66; 128 of 777 x 512 x 128 176, 47.
        const int q = warp & 3, mt = (warp - 2) >> 2;
        bool ok = __all_sync(0xffffffffu, nkb > 0 ? mbar_wait(acc_full, 0, p.err, 3) : true);      // one answer for the warp: its loads are warp-wide
        if (p.tma_out) ok = bar_all(1 + mt * 2 + (q >> 1), 64, ok);        // and for the pair of warps that store together: their limits end at different times
        tc_fence_after();
        const int rows = min(BN, p.M - m0);
        const uint32_t lane_addr = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(mt * BN);
        const bool has_bias = p.bias && p.splits == 1;
        if (ok && p.tma_out) {
            constexpr int CH = BN < 64 ? BN : 64;                          // rows of a store
            const int nh = n0 + mt * BM + (q >> 1) * 64;                   // first column of this pair of warps
            float b[2][2];                                                 // bias of the rows of the accumulator that this thread's pieces hold
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int n = nh + (q & 1) * 32 + h * 16 + r * 8 + (lane >> 2);
                    b[h][r] = has_bias && n < p.N ? p.bias[n] : 0.f;
                }
            uint8_t* stage = smem + (mt * 2 + (q >> 1)) * (BN * 128);
            if (nh < p.N)
#pragma unroll 1
            for (int c0 = 0; c0 < rows; c0 += CH) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t r[CH / 2];
                    tmem_ld_pieces<CH>(lane_addr + ((uint32_t)(h * 16) << 16) + (uint32_t)c0, r);
#pragma unroll
                    for (int g = 0; g < CH / 16; ++g) {
                        uint32_t v[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            v[i] = pack_bf16x2(__uint_as_float(r[8 * g + 2 * i]) + b[h][i & 1], __uint_as_float(r[8 * g + 2 * i + 1]) + b[h][i & 1]);
                        const int m = c0 + g * 16 + (lane >> 4) * 8 + (lane & 7), c = (q & 1) * 4 + h * 2 + ((lane >> 3) & 1);
                        stmatrix_x4_trans(smem_u32(stage) + (uint32_t)(m * 128 + ((c ^ (m & 7)) << 4)), v);
                    }
                }
                fence_proxy_async();
                bar_sync(1 + mt * 2 + (q >> 1), 64);
                if (!(q & 1)) {
                    if (elect_one()) {
                        if (BATCHED) tma_store_3d(stage + c0 * 128, &map_o, nh, m0 + c0, batch);
                        else tma_store_2d(stage + c0 * 128, &map_o, nh, m0 + c0);
                    }
                    __syncwarp();
                }
            }
            if (!(q & 1)) {
                bulk_commit_wait();                                        // (the group of the thread that stored is the only one that is not empty)
                __syncwarp();
            }
        } else if (ok) {
            const int n = n0 + mt * BM + q * 32 + lane;
            const bool nin = n < p.N;
            const float b = has_bias && nin ? p.bias[n] : 0.f;
            const bool f32 = p.splits > 1 || !p.out_bf16 || p.comm.nranks;
            const size_t step = p.splits > 1 ? (size_t)p.N : (size_t)p.ldo;
            const size_t at = p.splits > 1 ? ((size_t)split * p.M + m0) * p.N + n : (size_t)batch * p.out_bs + (size_t)m0 * p.ldo + n;
            float* of = (p.splits > 1 ? p.partial : reinterpret_cast<float*>(p.out)) + at;
            bf16* oh = reinterpret_cast<bf16*>(p.out) + at;
#pragma unroll 1
            for (int c0 = 0; c0 < rows; c0 += 16) {
                float v[16];
                tmem_ld16(lane_addr + (uint32_t)c0, v);
                if (nkb == 0) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.f;
                }
                if (p.comm.nranks) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (nin && c0 + j < rows) comm_push(p.comm, next_epoch, (size_t)(m0 + c0 + j) * p.ldo + n, v[j]);
                    __syncwarp();
                } else if (f32) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) { st_global_if(of, v[j] + b, nin && c0 + j < rows); of += step; }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) { st_global_if(oh, __float2bfloat16(v[j] + b), nin && c0 + j < rows); oh += step; }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_d, C::TMEM_COLS);
    if (p.comm.nranks) comm_signal(p.comm, next_epoch, gridDim.x * gridDim.y * gridDim.z);
    pdl_launch_dependents();
}

// Sum K-split partials in split order (deterministic), add bias, convert.
__global__ void splitk_reduce_kernel(void* __restrict__ out, int ldo, const float* __restrict__ partial, const float* __restrict__ bias,
                                     int M, int N, int splits, int out_bf16) {
    pdl_wait();
    pdl_launch_dependents();
    const int n = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
    if (n >= N) return;
    float a = 0.f;
    for (int s = 0; s < splits; ++s) a += partial[((size_t)s * M + m) * N + n];
    if (bias) a += bias[n];
    if (out_bf16) reinterpret_cast<bf16*>(out)[(size_t)m * ldo + n] = __float2bfloat16(a);
    else reinterpret_cast<float*>(out)[(size_t)m * ldo + n] = a;
    pdl_launch_dependents();
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess) fn = (EncodeTiledFn)f;
    }
    return fn;
}

// 2-D row-major tensor [rows, cols] of `esize`-byte elements, box [box_rows, box_cols], 128B swizzle.
int make_map_2d(CUtensorMap* map, const void* ptr, CUtensorMapDataType dt, int esize, uint64_t rows, uint64_t cols, uint64_t ld_elems,
                uint32_t box_rows, uint32_t box_cols) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return -2;
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstr[1] = {ld_elems * (uint64_t)esize};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, dt, 2, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -3;
}

// 3-D view [batch][rows][cols] with element strides (batch_stride, ld, 1); box [1][box_rows][box_cols].
int make_map_3d(CUtensorMap* map, const void* ptr, CUtensorMapDataType dt, int esize, uint64_t rows, uint64_t cols, uint64_t ld_elems,
                uint64_t batch, uint64_t batch_stride_elems, uint32_t box_rows, uint32_t box_cols) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return -2;
    cuuint64_t gdim[3] = {cols, rows, batch};
    cuuint64_t gstr[2] = {ld_elems * (uint64_t)esize, batch_stride_elems * (uint64_t)esize};
    cuuint32_t box[3] = {box_cols, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, dt, 3, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -3;
}

// 3-D byte view [slot][row][byte] of quantised weight matrices that sit at the same offset in every slot of an arena
// (strides: slot_stride, pitch, 1 bytes); box [1][box_rows][box_bytes] with the swizzle mode that matches box_bytes
// (32, 64 or 128), so that a thread reading its own row of the box hits every bank once.
int make_map_bytes_3d(CUtensorMap* map, const void* ptr, uint64_t pitch, uint64_t rows, uint64_t slot_stride, uint64_t nslots,
                      uint32_t box_bytes, uint32_t box_rows) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return -2;
    if (((uintptr_t)ptr & 15) || (pitch & 15) || (slot_stride & 15)) return -4;
    cuuint64_t gdim[3] = {pitch, rows, nslots};
    cuuint64_t gstr[2] = {pitch, slot_stride};
    cuuint32_t box[3] = {box_bytes, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapSwizzle sw = box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : -3;
}

struct MapKey {
    const void* p; uint64_t rows, cols, ld; uint32_t br, bc; int dt;
    bool operator<(const MapKey& o) const { return std::tie(p, rows, cols, ld, br, bc, dt) < std::tie(o.p, o.rows, o.cols, o.ld, o.br, o.bc, o.dt); }
};
static std::map<MapKey, CUtensorMap> g_maps;
static std::mutex g_maps_mu;

int cached_map_2d(CUtensorMap* out, const void* ptr, CUtensorMapDataType dt, int esize, uint64_t rows, uint64_t cols, uint64_t ld,
                  uint32_t br, uint32_t bc) {
    std::lock_guard<std::mutex> g(g_maps_mu);
    MapKey k{ptr, rows, cols, ld, br, bc, (int)dt};
    auto it = g_maps.find(k);
    if (it != g_maps.end()) { *out = it->second; return 0; }
    CUtensorMap m;
    int rc = make_map_2d(&m, ptr, dt, esize, rows, cols, ld, br, bc);
    if (rc) return rc;
    if (g_maps.size() > 65536) g_maps.clear();
    g_maps[k] = m;
    *out = m;
    return 0;
}

template <int BN, int MT = 1, bool DEEP = false>
static int launch_tc(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mo, const GemmTcParams& p, cudaStream_t st) {
    using C = TcCfg<BN, MT, DEEP>;
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(gemm_tc_kernel<BN, MT, false, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM); attr = true; }
    dim3 grid((p.M + BN - 1) / BN, (p.N + BM * MT - 1) / (BM * MT), p.splits);
    launch_pdl((gemm_tc_kernel<BN, MT, false, DEEP>), grid, C::THREADS, C::SMEM, st, mw, mx, mo, p);
    return (int)cudaGetLastError();
}


template <int BN>
static int launch_tc_batched(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mo, const GemmTcParams& p, int batch, cudaStream_t st) {
    using C = TcCfg<BN, 1>;
    static bool attr = false;
    if (!attr) { cudaFuncSetAttribute(gemm_tc_kernel<BN, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM); attr = true; }
    dim3 grid((p.M + BN - 1) / BN, (p.N + BM - 1) / BM, batch);
    launch_pdl((gemm_tc_kernel<BN, 1, true>), grid, C::THREADS, C::SMEM, st, mw, mx, mo, p);
    return (int)cudaGetLastError();
}

}  // namespace lsb
using namespace lsb;

// Batched product for b in [0, B): out[b][m][n] = sum_k x[b][m][k] * w[b][n][k] with element strides
// x: (xs_b, ldx, 1), w: (ws_b, ldw, 1), out: (os_b, ldo, 1).  One launch, grid.z = batch.  Strides % 8 == 0.
LSB_API int lsb_gemm_bf16_tc_batched(void* out, const void* x, const void* w, int M, int N, int K, int B, int ldx, long long xs_b, int ldw,
                                     long long ws_b, int ldo, long long os_b, int out_bf16, void* err, void* stream) {
    if (K % 8 || ldx % 8 || ldw % 8 || xs_b % 8 || ws_b % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) || B < 1 || B > 65535) return -1;
    int BN = 16;
    while (BN < 256 && BN < M) BN <<= 1;
    static std::map<std::tuple<const void*, int, int, int, long long, int, int>, CUtensorMap> cache;      // per (ptr, rows, cols, ld, batch stride, B, box rows)
    static std::mutex mu;
    auto get = [&](const void* ptr, int rows, int cols, int ld, long long bs, int box_rows, CUtensorMap* o) -> int {
        std::lock_guard<std::mutex> g(mu);
        const auto key = std::make_tuple(ptr, rows, cols, ld, bs, B, box_rows);
        auto it = cache.find(key);
        if (it != cache.end()) { *o = it->second; return 0; }
        CUtensorMap m;
        const int rc = make_map_3d(&m, ptr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows, cols, ld, B, bs, box_rows, BK);
        if (rc) return rc;
        if (cache.size() > 4096) cache.clear();
        cache[key] = m;
        *o = m;
        return 0;
    };
    CUtensorMap mw, mx;
    int rc = get(w, N, K, ldw, ws_b, BM, &mw);
    if (rc) return rc;
    rc = get(x, M, K, ldx, xs_b, BN, &mx);
    if (rc) return rc;
    GemmTcParams p;
    p.out = out; p.ldo = ldo; p.partial = nullptr; p.bias = nullptr; p.M = M; p.N = N; p.K = K; p.out_bf16 = out_bf16; p.err = (int*)err;
    p.splits = 1; p.kb_per_split = (K + BK - 1) / BK; p.out_bs = os_b; p.comm.nranks = 0;
    p.tma_out = out_bf16 && K > 0 && ldo % 8 == 0 && os_b % 8 == 0 && ldo >= N && os_b > 0 && ((uintptr_t)out & 15) == 0;
    CUtensorMap mo = mx;
    if (p.tma_out && get(out, M, N, ldo, os_b, BN < 64 ? BN : 64, &mo) != 0) p.tma_out = 0;
    cudaStream_t st = (cudaStream_t)stream;
    switch (BN) {
        case 16: return launch_tc_batched<16>(mw, mx, mo, p, B, st);
        case 32: return launch_tc_batched<32>(mw, mx, mo, p, B, st);
        case 64: return launch_tc_batched<64>(mw, mx, mo, p, B, st);
        case 128: return launch_tc_batched<128>(mw, mx, mo, p, B, st);
        default: return launch_tc_batched<256>(mw, mx, mo, p, B, st);
    }
}

LSB_API int lsb_gemm_tc_workspace_floats(int M, int N, int K) {
    // upper bound on split-K partial storage: at most 16 splits
    return 16 * M * N;
}

// x bf16 [M, ldx], w bf16 [N, ldw], out fp32/bf16 [M, ldo]; K % 8 == 0; ldx, ldw % 8 == 0; pointers 16-byte aligned.
// partial: fp32 scratch of partial_cap floats (split-K is limited to what fits) or null to disable split-K.
// err: int error word (0 = ok; 1-3 = a bounded pipeline wait gave up).
// out_bf16: 1 = bf16 output, + 2 = no kernel that may still run writes w, so that few-row products ask for their weights before they wait for the kernel in front
// (weights of a model; 1 to 2 us per product).
LSB_API int lsb_gemm_bf16_tc(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx, int ldw,
                             int ldo, int out_bf16, void* partial, long long partial_cap, void* err, const void* comm, void* stream) {
    const int steady = (out_bf16 >> 1) & 1;
    out_bf16 &= 1;
    if (K % 8 || ldx % 8 || ldw % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return -1;
    if (comm) { partial = nullptr; if (out_bf16 || bias || (long long)M * ldo > ((const PeerComm*)comm)->cap) return -1; }
    cudaStream_t st = (cudaStream_t)stream;
    if (!comm && bf16_rows_ok(M, N, K, ldx, ldw, x, w)) {
        Bf16RowsArgs a{};
        a.x = (const bf16*)x; a.ldx = ldx; a.w = (const bf16*)w; a.ldw = ldw; a.out = out; a.ldo = ldo; a.out_bf16 = out_bf16;
        a.bias = (const float*)bias; a.M = M; a.N = N; a.K = K; a.steady = steady;
        return bf16_rows_launch(a, st);
    }
    int BN = 16;
    while (BN < 256 && BN < M) BN <<= 1;
    CUtensorMap mw, mx;
    int rc = cached_map_2d(&mw, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, N, K, ldw, BM, BK);
    if (rc) return rc;
    rc = cached_map_2d(&mx, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, K, ldx, BN, BK);
    if (rc) return rc;
    GemmTcParams p;
    p.out = out; p.ldo = ldo; p.partial = (float*)partial; p.bias = (const float*)bias; p.M = M; p.N = N; p.K = K;
    p.out_bf16 = out_bf16; p.err = (int*)err; p.out_bs = 0;
    if (comm) p.comm = *(const PeerComm*)comm; else p.comm.nranks = 0;
    const int nkb = (K + BK - 1) / BK;
    const int tiles = ((N + BM - 1) / BM) * ((M + BN - 1) / BN);
    int splits = 1;
    if (partial && tiles < kSms) {
        splits = (kSms + tiles - 1) / tiles;
        if (splits > 16) splits = 16;
        if (splits > nkb / 4) splits = nkb / 4 > 0 ? nkb / 4 : 1;
        while (splits > 1 && (long long)splits * M * N > partial_cap) --splits;
    }
    p.kb_per_split = (nkb + splits - 1) / splits;
    p.splits = (nkb + p.kb_per_split - 1) / p.kb_per_split;
    const int ctas = tiles * p.splits;                     // of one weight tile each
    p.tma_out = out_bf16 && K > 0 && p.splits == 1 && !comm && ldo % 8 == 0 && ldo >= N && ((uintptr_t)out & 15) == 0;
    CUtensorMap mo = mx;
    if (p.tma_out && cached_map_2d(&mo, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, N, ldo, BN < 64 ? BN : 64, BK) != 0) p.tma_out = 0;
    switch (BN) {
        case 16: rc = launch_tc<16>(mw, mx, mo, p, st); break;
        case 32: rc = launch_tc<32>(mw, mx, mo, p, st); break;
        case 64: rc = launch_tc<64>(mw, mx, mo, p, st); break;
        case 128: rc = launch_tc<128>(mw, mx, mo, p, st); break;
        // (one CTA of 128 x 256 per SM before there was a choice, one weight tile, one and deep, two; us).  A grid that one CTA per SM takes in one wave is deep:
        // 160 x 576 x 4096 27.8, 26.4, 25.9, 28.9; 256 x 2048 x 2048 36.6, 35.1, 33.8, 38.1.  So is one of two to three such waves over a long reduction, which
        // takes CTAs of two tiles two waves: 1500 x 7168 x 12288 298, 334, 291, 306; 391 x 24896 x 12288 304, 343, 301, 312, but 391 x 24896 x 4096 146, 139, 143,
        // 130 and 1000 x 24896 x 12288 (780 CTAs) 659, 554, 645, 518.  Two weight tiles per CTA pay from a reduction of 2048 on (K = 1536 and below: the same; a
        // short one leaves the longer epilogue bare) unless half the grid no longer covers the SMs: 300 x 576 x 4096 (150 CTAs) 36.6, 37.1, -, 40.2.
        default:
            if (ctas <= kSms || (K >= 8192 && ctas > 2 * kSms && ctas <= 3 * kSms)) rc = launch_tc<256, 1, true>(mw, mx, mo, p, st);
            else rc = K >= 2048 && !comm && ctas >= 160 ? launch_tc<256, 2>(mw, mx, mo, p, st) : launch_tc<256>(mw, mx, mo, p, st);
            break;
    }
    if (rc) return rc;
    if (p.splits > 1) {
        launch_pdl((splitk_reduce_kernel), dim3((N + 255) / 256, M), 256, 0, st, out, ldo, (const float*)partial, (const float*)bias, M, N, p.splits, out_bf16);
        return (int)cudaGetLastError();
    }
    return 0;
}

LSB_API int lsb_trace_set_gemm_tc(void* buf) { return lsb_trace_install(buf); }
