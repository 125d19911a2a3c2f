#pragma once
// ------------------------------------------------------------------------------------------------ chunk-parallel recurrence
// The gated delta rule in chunks of 64 tokens of one sequence (prefill chunks), for any head sizes: key channels padded to DK (32, 64 or
// 128), value channels in tiles of 64.  With G_t = sum_{s<=t} log d_s inside a chunk:
//   A[t][s] = sum_c k_t k_s exp(G_t - G_s) (s < t),  B[t][s] = sum_c q_t k_s exp(G_t - G_s) (s <= t)    every exponent <= 0
//   W = (I + diag(beta) tril(A,-1))^-1 diag(beta),  U = W (V - Kp S0^T),  O = Qp S0^T + tril(B) U,  S = S0 diag(gC) + U^T Km
//   Kp = K exp(G), Qp = Q exp(G), Km = K exp(G_last - G), gC = exp(G_last)
// delta_chunk_prep: everything that does not depend on the state, one block per (chunk, head); rewrites qn -> Qp, decay -> Kp, kn -> Km in
// place.  delta_chunk_scan: sequential over the chunks, one block per (head, value tile, sequence) - value channels are independent.
// A step may hold several sequences; those with fewer than `min_rows` rows are left to the token recurrence.  fp32 on the CUDA cores.
constexpr int kCh = 64;            // tokens per chunk
constexpr int kLdC = kCh + 4;      // row stride of [*, 64] tiles
constexpr int kSub = 16;           // tokens per sub-chunk of the A / B factorisation
template <int DK> struct ChunkDims {
    static constexpr int kLdK = DK + 4;       // shared-memory row stride (floats) of [*, DK] tiles: 16-byte aligned rows, conflict-free float4 columns
    static constexpr int kTileRows = 2 * kSub + kCh - kSub;   // rescaled rows of a sub-chunk (k and q) and the k rows in front of it; at least kCh
    static constexpr size_t kPrepSmem = (size_t)(3 * kCh * kLdK + 3 * kCh * kLdC + kCh + kTileRows * kLdK) * sizeof(float);
    static constexpr size_t kScanSmem = (size_t)(4 * kCh * kLdK + 4 * kCh * kLdC) * sizeof(float);
    static constexpr int kWsFloats = 2 * kCh * kCh + DK;      // workspace floats per (chunk, head)
};

struct DeltaChunkArgs {
    float* qn; float* kn; float* decay;      // [rows, H, DK]; decay: the factors, or their logarithms with `log_decay`
    float* vo;                               // [rows, H, dv]  v in, o out
    const float* beta;                       // [rows, H]
    float* state;                            // [slots, H, dv, DK]
    const int* seq_row0; const int* seq_nrows; const int* seq_slot;
    int nseq, min_rows, H, dv, log_decay;
    float* W;     // [chunks, H, 64, 64]
    float* B;     // [chunks, H, 64, 64] lower triangle incl. diagonal, zero above
    float* gC;    // [chunks, H, DK]
};

// V consecutive floats of a row whose start is aligned to them.
template <int V> __device__ __forceinline__ void chunk_ld(float (&o)[V], const float* p) {
    if constexpr (V == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else {
        for (int i = 0; i < V; ++i) o[i] = p[i];
    }
}

// Rows ty (k) and ty + 16 (q) of the tile L against rows tx + 16 j of R, j < NJ, over K channels.
template <int K, int NJ>
__device__ __forceinline__ void chunk_pairs(const float* L, const float* R, int ld, int tx, int ty, float* A, float* B) {
    float acc[2][NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[0][j] = acc[1][j] = 0.f;
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        const float4 a0 = *reinterpret_cast<const float4*>(L + ty * ld + k), a1 = *reinterpret_cast<const float4*>(L + (ty + kSub) * ld + k);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const float4 b = *reinterpret_cast<const float4*>(R + (tx + kSub * j) * ld + k);
            acc[0][j] = fmaf(a0.x, b.x, fmaf(a0.y, b.y, fmaf(a0.z, b.z, fmaf(a0.w, b.w, acc[0][j]))));
            acc[1][j] = fmaf(a1.x, b.x, fmaf(a1.y, b.y, fmaf(a1.z, b.z, fmaf(a1.w, b.w, acc[1][j]))));
        }
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) { A[ty * kLdC + tx + kSub * j] = acc[0][j]; B[ty * kLdC + tx + kSub * j] = acc[1][j]; }
}

// One block per (chunk, head), 256 threads; fp32 throughout.  Bound by the issue rate of one block an SM (196 KB of shared memory at 128 key
// channels).  2048 rows of 64 heads of 128 channels: 1075 us
// when every pair was summed across a warp's lanes by itself and a thread walked down each column of W, 407 us now (traffic at DRAM's rate: 75 us).
template <int kD>
__global__ void __launch_bounds__(256) delta_chunk_prep_kernel(DeltaChunkArgs a_) {
    constexpr int kLdK = ChunkDims<kD>::kLdK;
    constexpr int V = kD / 32;                                // channels per lane
    extern __shared__ __align__(16) float csm[];
    float* sK = csm;
    float* sQ = sK + kCh * kLdK;
    float* sG = sQ + kCh * kLdK;
    float* sA = sG + kCh * kLdK;
    float* sB = sA + kCh * kLdC;
    float* sW = sB + kCh * kLdC;
    float* sBeta = sW + kCh * kLdC;
    float* sD = sBeta + kCh;                                  // [64][kLdK] the decay factors, while the pairs inside sub-chunks are formed
    float* sL = sD;                                           // then [16 + 16][kLdK] k and q rows of the current sub-chunk times exp(G - G_ref)
    float* sR = sL + 2 * kSub * kLdK;                         //      [48][kLdK] earlier k rows times exp(G_ref - G)
    const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    pdl_wait();
    pdl_launch_dependents();
    // this block's sequence and its chunk inside it (chunks are numbered over the chunked sequences in order)
    int row0 = 0, cc = 0, c0 = 0;
    for (int s_ = 0, base = 0; s_ < a_.nseq; ++s_) {
        const int n = a_.seq_nrows[s_];
        if (n < a_.min_rows) continue;
        const int nc = (n + kCh - 1) / kCh;
        if (chunk < base + nc) { row0 = a_.seq_row0[s_]; c0 = (chunk - base) * kCh; cc = min(kCh, n - c0); break; }
        base += nc;
    }
    if (cc <= 0) return;
    const int C = a_.H * kD;
    // 1. k, q, decay and log-decay tiles (rows past the chunk: zeros, i.e. no decay and no write)
#pragma unroll 4
    for (int idx = tid; idx < kCh * (kD / 4); idx += 256) {
        const int t = idx / (kD / 4), c4 = idx % (kD / 4);
        float4 k4 = make_float4(0.f, 0.f, 0.f, 0.f), q4 = k4, g4 = k4, d4 = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < cc) {
            const size_t off = (size_t)(row0 + c0 + t) * C + h * kD + c4 * 4;
            k4 = *reinterpret_cast<const float4*>(a_.kn + off);
            q4 = *reinterpret_cast<const float4*>(a_.qn + off);
            const float4 d = *reinterpret_cast<const float4*>(a_.decay + off);
            g4 = a_.log_decay ? d : make_float4(logf(d.x), logf(d.y), logf(d.z), logf(d.w));
            d4 = a_.log_decay ? make_float4(expf(d.x), expf(d.y), expf(d.z), expf(d.w)) : d;
        }
        *reinterpret_cast<float4*>(sK + t * kLdK + c4 * 4) = k4;
        *reinterpret_cast<float4*>(sQ + t * kLdK + c4 * 4) = q4;
        *reinterpret_cast<float4*>(sG + t * kLdK + c4 * 4) = g4;
        *reinterpret_cast<float4*>(sD + t * kLdK + c4 * 4) = d4;
    }
    for (int idx = tid; idx < kCh * kLdC; idx += 256) { sA[idx] = 0.f; sB[idx] = 0.f; sW[idx] = 0.f; }
    if (tid < kCh) sBeta[tid] = tid < cc ? a_.beta[(size_t)(row0 + c0 + tid) * a_.H + h] : 0.f;
    __syncthreads();
    // 2. cumulative log-decay per channel (non-increasing in t)
    if (tid < kD) {
        float acc = 0.f;
#pragma unroll 16
        for (int t = 0; t < kCh; ++t) { acc += sG[t * kLdK + tid]; sG[t * kLdK + tid] = acc; }
    }
    // 3. A and B.  The 64 tokens are four sub-chunks of 16.
    // Pairs inside a sub-chunk: a warp walks back from its row t over the rows s in front of it, its k and q rows times the decays that lie
    // between; the 16 + 16 sums over the lanes come out of one exchange of halves (lane l: sum l).
    for (int t = warp; t < cc; t += 8) {
        const int dt = t % kSub;
        float kf[V], qf[V], v[2 * kSub];
        chunk_ld<V>(kf, sK + t * kLdK + lane * V);
        chunk_ld<V>(qf, sQ + t * kLdK + lane * V);
#pragma unroll
        for (int d = 0; d < kSub; ++d) {
            float a = 0.f, b = 0.f;
            if (d <= dt) {                                    // warp-uniform
                float ks[V];
                chunk_ld<V>(ks, sK + (t - d) * kLdK + lane * V);
                if (d) {
                    float f[V];
                    chunk_ld<V>(f, sD + (t - d + 1) * kLdK + lane * V);
#pragma unroll
                    for (int i = 0; i < V; ++i) { kf[i] *= f[i]; qf[i] *= f[i]; }
                }
#pragma unroll
                for (int i = 0; i < V; ++i) { a = fmaf(kf[i], ks[i], a); b = fmaf(qf[i], ks[i], b); }
            }
            v[d] = a; v[kSub + d] = b;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        const int d = lane % kSub;
        if (d <= dt) (lane < kSub ? sA : sB)[t * kLdC + t - d] = v[0];
    }
    // Pairs (t in sub-chunk I, s before it) factor through the first token of I:
    //     exp(G_t - G_s) = exp(G_t - G_ref) * exp(G_ref - G_s),   G_ref = G[16 I]:   both exponents <= 0 (G is non-increasing),
    // so the block is a plain product of two rescaled tiles (L = rows of I times exp(G - G_ref), R = earlier rows times exp(G_ref - G))
    // with no exponential in the inner loop.
    for (int I = 1; I < kCh / kSub; ++I) {
        const int t0 = I * kSub;
        if (t0 >= cc) break;                                  // block-uniform
        __syncthreads();                                      // readers of the tiles (the decays, the sub-chunk before) and writers of G are done
        const float* gref = sG + t0 * kLdK;
#pragma unroll 2
        for (int idx = tid; idx < (kSub + t0) * (kD / 4); idx += 256) {
            const int tt = idx / (kD / 4), c = idx % (kD / 4) * 4, src = tt < kSub ? t0 + tt : tt - kSub;
            const float4 g = *reinterpret_cast<const float4*>(sG + src * kLdK + c), r = *reinterpret_cast<const float4*>(gref + c);
            const float4 k4 = *reinterpret_cast<const float4*>(sK + src * kLdK + c);
            const float sg = tt < kSub ? 1.f : -1.f;
            const float4 e = make_float4(__expf(fminf(sg * (g.x - r.x), 0.f)), __expf(fminf(sg * (g.y - r.y), 0.f)), __expf(fminf(sg * (g.z - r.z), 0.f)),
                                         __expf(fminf(sg * (g.w - r.w), 0.f)));
            *reinterpret_cast<float4*>((tt < kSub ? sL + tt * kLdK : sR + src * kLdK) + c) = make_float4(k4.x * e.x, k4.y * e.y, k4.z * e.z, k4.w * e.w);
            if (tt < kSub) {
                const float4 q4 = *reinterpret_cast<const float4*>(sQ + src * kLdK + c);
                *reinterpret_cast<float4*>(sL + (kSub + tt) * kLdK + c) = make_float4(q4.x * e.x, q4.y * e.y, q4.z * e.z, q4.w * e.w);
            }
        }
        __syncthreads();
        // (rows past the chunk are zeros and give zeros)
        if (I == 1) chunk_pairs<kD, 1>(sL, sR, kLdK, tx, ty, sA + t0 * kLdC, sB + t0 * kLdC);
        else if (I == 2) chunk_pairs<kD, 2>(sL, sR, kLdK, tx, ty, sA + t0 * kLdC, sB + t0 * kLdC);
        else chunk_pairs<kD, 3>(sL, sR, kLdK, tx, ty, sA + t0 * kLdC, sB + t0 * kLdC);
    }
    __syncthreads();
    // 4. W = (I + N)^-1 diag(beta), N = diag(beta) tril(A, -1), by blocks of 16: the inverses of the diagonal blocks by forward substitution
    // (one warp each, a lane per column, the column in registers), then the blocks d below the diagonal for d = 1, 2, 3:
    // X_IJ = -X_II sum_{J <= K < I} N_IK X_KJ, a thread per element.
    if (warp < kCh / kSub && lane < kSub) {
        float x[kSub];
        const int b0 = warp * kSub;
#pragma unroll
        for (int t = 0; t < kSub; ++t) {
            float acc = 0.f;
#pragma unroll
            for (int s = 0; s < t; ++s) acc = fmaf(sA[(b0 + t) * kLdC + b0 + s], x[s], acc);
            x[t] = (t == lane ? 1.f : 0.f) - sBeta[b0 + t] * acc;
            sW[(b0 + t) * kLdC + b0 + lane] = x[t];
        }
    }
    float* sY = sL;                                           // [blocks of the diagonal][16][16]
    for (int d = 1; d < kCh / kSub; ++d) {
        __syncthreads();
        for (int J = 0; J + d < kCh / kSub; ++J) {
            const float* ar = sA + ((J + d) * kSub + ty) * kLdC;
            float acc0 = 0.f, acc1 = 0.f;
#pragma unroll 8
            for (int s = J * kSub; s < (J + d) * kSub; s += 2) {
                acc0 = fmaf(ar[s], sW[s * kLdC + J * kSub + tx], acc0);
                acc1 = fmaf(ar[s + 1], sW[(s + 1) * kLdC + J * kSub + tx], acc1);
            }
            sY[(J * kSub + ty) * kSub + tx] = sBeta[(J + d) * kSub + ty] * (acc0 + acc1);
        }
        __syncthreads();
        for (int J = 0; J + d < kCh / kSub; ++J) {
            const float* xr = sW + ((J + d) * kSub + ty) * kLdC + (J + d) * kSub;
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < kSub; ++k) acc = fmaf(xr[k], sY[(J * kSub + k) * kSub + tx], acc);
            sW[((J + d) * kSub + ty) * kLdC + J * kSub + tx] = -acc;
        }
    }
    __syncthreads();
    // 5. results: W, tril(B), the rescaled tiles in place, the chunk's total decay
    float* Wg = a_.W + ((size_t)chunk * a_.H + h) * kCh * kCh;
    float* Bg = a_.B + ((size_t)chunk * a_.H + h) * kCh * kCh;
    for (int idx = tid; idx < kCh * kCh; idx += 256) {
        const int t = idx / kCh, s = idx % kCh;
        Wg[idx] = sW[t * kLdC + s] * sBeta[s];
        Bg[idx] = sB[t * kLdC + s];
    }
    const float* gl = sG + (cc - 1) * kLdK;
#pragma unroll 2
    for (int idx = tid; idx < cc * (kD / 4); idx += 256) {
        const int t = idx / (kD / 4), c4 = idx % (kD / 4);
        const float4 k4 = *reinterpret_cast<const float4*>(sK + t * kLdK + c4 * 4);
        const float4 q4 = *reinterpret_cast<const float4*>(sQ + t * kLdK + c4 * 4);
        const float4 g4 = *reinterpret_cast<const float4*>(sG + t * kLdK + c4 * 4);
        const float4 l4 = *reinterpret_cast<const float4*>(gl + c4 * 4);
        const float4 eg = make_float4(expf(g4.x), expf(g4.y), expf(g4.z), expf(g4.w));
        const float4 el = make_float4(expf(fminf(l4.x - g4.x, 0.f)), expf(fminf(l4.y - g4.y, 0.f)), expf(fminf(l4.z - g4.z, 0.f)),
                                      expf(fminf(l4.w - g4.w, 0.f)));
        const size_t off = (size_t)(row0 + c0 + t) * C + h * kD + c4 * 4;
        *reinterpret_cast<float4*>(a_.qn + off) = make_float4(q4.x * eg.x, q4.y * eg.y, q4.z * eg.z, q4.w * eg.w);
        *reinterpret_cast<float4*>(a_.decay + off) = make_float4(k4.x * eg.x, k4.y * eg.y, k4.z * eg.z, k4.w * eg.w);
        *reinterpret_cast<float4*>(a_.kn + off) = make_float4(k4.x * el.x, k4.y * el.y, k4.z * el.z, k4.w * el.w);
    }
    if (tid < kD) a_.gC[((size_t)chunk * a_.H + h) * kD + tid] = expf(gl[tid]);
}

// 16 bytes global -> shared, asynchronous on the device; zeros where !valid (src must be a readable address all the same).
__device__ __forceinline__ void chunk_copy16(float* dst, const float* src, bool valid) {
#ifdef __CUDACC__
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
#else
    for (int i = 0; i < 4; ++i) dst[i] = valid ? src[i] : 0.f;
#endif
}
__device__ __forceinline__ void chunk_copy_commit() {
#ifdef __CUDACC__
    asm volatile("cp.async.commit_group;" ::: "memory");
#endif
}
template <int N> __device__ __forceinline__ void chunk_copy_wait() {
#ifdef __CUDACC__
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
#endif
}

// acc[i][j] += sum over the lane's quarter of k of A[i][k] B[cl + 8 j][k]: rows i of the warp, kq = lane / 8 the quarter (quads kq, kq + 4, ..), cl = lane % 8.
// 16 16-byte shared reads (8 of them one address per quarter-warp) feed 256 FMAs; `A2` shares B's reads.
template <int K, bool TWO = false>
__device__ __forceinline__ void chunk_mm(const float* A, int lda, const float* B, int ldb, float (&acc)[8][8], int kq, int cl, const float* A2 = nullptr,
                                         float (*acc2)[8] = nullptr) {
#pragma unroll 1
    for (int k = kq * 4; k < K; k += 16) {
        float4 b[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(B + (cl + 8 * j) * ldb + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(A + i * lda + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a.x, b[j].x, fmaf(a.y, b[j].y, fmaf(a.z, b[j].z, fmaf(a.w, b[j].w, acc[i][j]))));
            if (TWO) {
                const float4 c = *reinterpret_cast<const float4*>(A2 + i * lda + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc2[i][j] = fmaf(c.x, b[j].x, fmaf(c.y, b[j].y, fmaf(c.z, b[j].z, fmaf(c.w, b[j].w, acc2[i][j]))));
            }
        }
    }
}
// Sums of the four quarters by exchanging halves: acc[0..1] of lane l become rows 4 (l / 16) + 2 (l / 8 % 2) + {0, 1}.
__device__ __forceinline__ void chunk_quarters(float (&acc)[8][8], int lane) {
#pragma unroll
    for (int o = 16, n = 4; n >= 2; o >>= 1, n >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float send = up ? acc[i][j] : acc[i + n][j], keep = up ? acc[i + n][j] : acc[i][j];
                acc[i][j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
}

// `tail(h, value tile, thread, row0, nrows, slot)` runs after the block's last chunk (convolution histories of the caller).
// One block per (head, 64 value channels, sequence), 256 threads, fp32 FMAs.  A warp owns eight rows of every product and its lanes split the reduction in
// four, so that a lane's 8 x 8 sums take as many shared-memory cycles as FMA cycles (4 x 4 sums per thread: twice as many); the tiles of the next products
// arrive by cp.async meanwhile.  2048 rows of 64 heads of 128 + 128 channels: 805 us
// before, 567 us now (273 us of FMA issue on the 128 SMs that 64 heads give work to).
template <int kD, class Tail>
__global__ void __launch_bounds__(256) delta_chunk_scan_kernel(DeltaChunkArgs a_, Tail tail) {
    constexpr int kLdK = ChunkDims<kD>::kLdK;
    constexpr int NK = kD / 16;                               // key columns per lane of the state's update
    extern __shared__ __align__(16) float csm[];
    float* sS = csm;                         // [64 value channels][128 key channels] state slice
    float* sKp = sS + kCh * kLdK;            // [t][k]
    float* sQp = sKp + kCh * kLdK;
    float* sKm = sQp + kCh * kLdK;
    float* sW = sKm + kCh * kLdK;            // [t][s]
    float* sBm = sW + kCh * kLdC;
    float* sX = sBm + kCh * kLdC;            // (V - Kp S^T)^T : [v][t]
    float* sU = sX + kCh * kLdC;             // U^T : [v][t]
    const int h = blockIdx.x, vs = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, kq = lane >> 3, cl = lane & 7;
    pdl_wait();
    pdl_launch_dependents();
    const int seq = blockIdx.z;
    const int row0 = a_.seq_row0[seq], nrows = a_.seq_nrows[seq], slot = a_.seq_slot[seq];
    if (nrows <= 0 || nrows < a_.min_rows) return;
    int chunk0 = 0;                                           // first chunk of this sequence in the workspace
    for (int s_ = 0; s_ < seq; ++s_) {
        const int n = a_.seq_nrows[s_];
        if (n >= a_.min_rows) chunk0 += (n + kCh - 1) / kCh;
    }
    const int C = a_.H * kD, Cv = a_.H * a_.dv, vbase = h * a_.dv + vs * kCh;
    const int nv = min(kCh, a_.dv - vs * kCh);                // value channels of this tile
    float* sp = a_.state + (((size_t)slot * a_.H + h) * a_.dv + vs * kCh) * kD;
    for (int idx = tid; idx < kCh * (kD / 4); idx += 256) {
        const int v = idx / (kD / 4), c4 = idx % (kD / 4);
        *reinterpret_cast<float4*>(sS + v * kLdK + c4 * 4) =
            v < nv ? *reinterpret_cast<const float4*>(sp + (size_t)v * kD + c4 * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int nchunks = (nrows + kCh - 1) / kCh;
    // rows past a chunk's end: zeros
    auto fetch_rows = [&](float* dst, const float* src, int chunk) {
        const int c0 = chunk * kCh, cc = min(kCh, nrows - c0);
#pragma unroll 4
        for (int idx = tid; idx < kCh * (kD / 4); idx += 256) {
            const int t = idx / (kD / 4), c4 = idx % (kD / 4);
            chunk_copy16(dst + t * kLdK + c4 * 4, src + (size_t)(row0 + c0 + min(t, cc - 1)) * C + h * kD + c4 * 4, t < cc);
        }
    };
    auto fetch_square = [&](float* dst, const float* src, int chunk) {
        const float* g = src + ((size_t)(chunk0 + chunk) * a_.H + h) * kCh * kCh;
#pragma unroll 4
        for (int idx = tid; idx < kCh * (kCh / 4); idx += 256) chunk_copy16(dst + idx / (kCh / 4) * kLdC + idx % (kCh / 4) * 4, g + idx * 4, true);
    };
    auto fetch_first = [&](int chunk) {                       // what the products with the state and U take
        fetch_rows(sKp, a_.decay, chunk);
        fetch_rows(sQp, a_.qn, chunk);
        fetch_square(sW, a_.W, chunk);
        chunk_copy_commit();
    };
    fetch_first(0);
    const int r0 = warp * 8, rt = r0 + (lane >> 4) * 4 + (lane >> 3 & 1) * 2;      // the warp's rows; first of the two that chunk_quarters leaves here
    for (int chunk = 0; chunk < nchunks; ++chunk) {
        const int c0 = chunk * kCh, cc = min(kCh, nrows - c0);
        fetch_rows(sKm, a_.kn, chunk);
        fetch_square(sBm, a_.B, chunk);
        chunk_copy_commit();
        float vreg[2][8], gc[NK];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) vreg[i][j] = (rt + i < cc && cl + 8 * j < nv) ? a_.vo[(size_t)(row0 + c0 + rt + i) * Cv + vbase + cl + 8 * j] : 0.f;
#pragma unroll
        for (int j = 0; j < NK; ++j) gc[j] = a_.gC[((size_t)(chunk0 + chunk) * a_.H + h) * kD + (lane & 15) + 16 * j];
        chunk_copy_wait<1>();
        __syncthreads();
        float acc[8][8], out[8][8];
        auto clear = [&](float (&x)[8][8]) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) x[i][j] = 0.f;
        };
        auto put = [&](float* dst) {                          // transposed: [v][t]
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                dst[(cl + 8 * j) * kLdC + rt] = acc[0][j];
                dst[(cl + 8 * j) * kLdC + rt + 1] = acc[1][j];
            }
        };
        // a. X = V - Kp S^T, and the state's part of the outputs, Qp S^T (its quarters stay apart until the other part is there)
        clear(acc);
        clear(out);
        chunk_mm<kD, true>(sKp + r0 * kLdK, kLdK, sS, kLdK, acc, kq, cl, sQp + r0 * kLdK, out);
        chunk_quarters(acc, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) { acc[0][j] = vreg[0][j] - acc[0][j]; acc[1][j] = vreg[1][j] - acc[1][j]; }
        put(sX);
        __syncthreads();
        // b. U = W X
        clear(acc);
        chunk_mm<kCh>(sW + r0 * kLdC, kLdC, sX, kLdC, acc, kq, cl);
        chunk_quarters(acc, lane);
        put(sU);
        chunk_copy_wait<0>();
        __syncthreads();
        if (chunk + 1 < nchunks) fetch_first(chunk + 1);
        // c. O = Qp S^T + tril(B) U
        chunk_mm<kCh>(sBm + r0 * kLdC, kLdC, sU, kLdC, out, kq, cl);
        chunk_quarters(out, lane);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (rt + i < cc) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (cl + 8 * j < nv) a_.vo[(size_t)(row0 + c0 + rt + i) * Cv + vbase + cl + 8 * j] = out[i][j];
            }
        // d. S = S diag(gC) + U^T Km : value rows of the warp, key columns lane % 16 + 16 j; the half-warps take the tokens four apart in turns
        // (their rows of Km lie 16 banks apart).  Every warp has read S in (a).
        float a2[8][NK];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < NK; ++j) a2[i][j] = 0.f;
#pragma unroll 1
        for (int tb = (lane >> 4) * 4; tb < kCh; tb += 8) {
            float4 u[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) u[i] = *reinterpret_cast<const float4*>(sU + (r0 + i) * kLdC + tb);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float km[NK];
#pragma unroll
                for (int j = 0; j < NK; ++j) km[j] = sKm[(tb + q) * kLdK + (lane & 15) + 16 * j];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float ui = q == 0 ? u[i].x : q == 1 ? u[i].y : q == 2 ? u[i].z : u[i].w;
#pragma unroll
                    for (int j = 0; j < NK; ++j) a2[i][j] = fmaf(ui, km[j], a2[i][j]);
                }
            }
        }
        const bool up = lane & 16;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NK; ++j) {
                const float send = up ? a2[i][j] : a2[i + 4][j], keep = up ? a2[i + 4][j] : a2[i][j];
                float* s = sS + (r0 + (up ? 4 : 0) + i) * kLdK + (lane & 15) + 16 * j;
                *s = fmaf(*s, gc[j], keep + __shfl_xor_sync(0xffffffffu, send, 16));
            }
        __syncthreads();
    }
    for (int idx = tid; idx < kCh * (kD / 4); idx += 256) {
        const int v = idx / (kD / 4), c4 = idx % (kD / 4);
        if (v < nv) *reinterpret_cast<float4*>(sp + (size_t)v * kD + c4 * 4) = *reinterpret_cast<const float4*>(sS + v * kLdK + c4 * 4);
    }
    tail(h, vs, tid, row0, nrows, slot);
    pdl_launch_dependents();
}
