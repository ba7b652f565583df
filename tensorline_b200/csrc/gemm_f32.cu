// C[M,N] = A[M,K] * W[N,K]^T (+ bias), true 32-bit: float inputs (weights may be stored as
// bfloat16 and are widened exactly), FFMA accumulation, no tensor-core mode of reduced precision.
//
// Every output element is one chain of fmaf over k = 0..K-1 in ascending order, whatever M is
// and wherever the element falls in a tile; a row's result therefore does not depend on which
// other rows share the launch.  This is the matrix product of the 32-bit engine for float weights, for small matrices and for
// rows that are not 16-byte aligned; large matrices of bfloat16 weights go to gemm_f32_parts.cu.
//
// Three kernels, the same floats: tiles (many rows), few rows, and a plain one for strides and sizes without 16-byte rows.
#include "common.cuh"

__device__ __forceinline__ void f32_copy16(void* dst, const void* src, bool ok) {      // zeros where !ok
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
// the weights of a 16-byte load as floats (a byte permutation and a mask: both leave the FMA pipe alone)
__device__ __forceinline__ void widen(const uint4 v, float (&w)[4]) {
    w[0] = __uint_as_float(v.x); w[1] = __uint_as_float(v.y); w[2] = __uint_as_float(v.z); w[3] = __uint_as_float(v.w);
}
__device__ __forceinline__ void widen(const uint4 v, float (&w)[8]) {
    const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { w[2 * i] = __uint_as_float(__byte_perm(u[i], 0, 0x1044)); w[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
// (d0, d1) += a * (b0, b1), each as fmaf
__device__ __forceinline__ void fma2(float& d0, float& d1, float a, float b0, float b1) {
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "+f"(d0), "+f"(d1) : "f"(a), "f"(b0), "f"(b1));
}
// four weights of a row as floats
__device__ __forceinline__ void widen4(const float* p, float (&w)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
}
__device__ __forceinline__ void widen4(const bf16* p, float (&w)[4]) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    w[0] = __uint_as_float(__byte_perm(v.x, 0, 0x1044)); w[1] = __uint_as_float(v.x & 0xffff0000u);
    w[2] = __uint_as_float(__byte_perm(v.y, 0, 0x1044)); w[3] = __uint_as_float(v.y & 0xffff0000u);
}

// ------------------------------------------------------------------ many rows
// Tiles of (16 TM) x (16 TN) outputs, 256 threads with TM x TN outputs each (rows and columns 16 apart), k in steps of 32 through
// a ring of cp.async stages in the operands' own layout and type.  The chain of an output cannot be cut, so what bounds it is
// the FMA pipe: a k costs a thread TM * TN / 2 pairs of multiply-adds, TM doublings of a value of A for them, TN widenings and
// (TM + TN) / 4 loads from shared memory (four k of a row at a time; the rows lie so that a warp, 8 threads along n and 4 along
// m, hits no bank twice).  Measured with bfloat16 weights, K 3,584: 1,024 x 37,888 outputs 5.8 ms, 48 TFLOP/s of multiply-adds
// (11.6 ms as 64 x 64 tiles of 4 x 4 outputs a thread with loads of single floats, the kernel below); 336 x 3,584 0.30 (0.58) ms.
// Single multiply-adds instead of pairs: 5 % slower; operands k-major with the weights twice in shared memory: half the rate.
constexpr int GF_BK = 32;
template <typename TW, int TM, int TN> struct TileShape {
    static constexpr int BM = 16 * TM, BN = 16 * TN;
    static constexpr int LA = GF_BK + 4, LW = GF_BK + 16 / (int)sizeof(TW);      // elements a row
    static constexpr int A_BYTES = BM * LA * 4, STAGE = A_BYTES + BN * LW * (int)sizeof(TW);
    static constexpr int STAGES = TM * TN >= 64 ? 3 : 4;
};

template <typename TW, int TM, int TN>
__global__ void __launch_bounds__(256)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                     const TW* __restrict__ bias, float* __restrict__ C, int ldc, int M, int N, int K) {
    using Sh = TileShape<TW, TM, TN>;
    constexpr int BM = Sh::BM, BN = Sh::BN, LA = Sh::LA, LW = Sh::LW, WV = 16 / (int)sizeof(TW), S = Sh::STAGES;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int tx = (wid & 1) * 8 + (lane & 7), ty = (wid >> 1) * 4 + (lane >> 3);
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    auto fetch = [&](int step, int stage) {
        unsigned char* st = smem + stage * Sh::STAGE;
        const int k0 = step * GF_BK;
#pragma unroll
        for (int i = tid; i < BM * (GF_BK / 4); i += 256) {
            const int r = i / (GF_BK / 4), c = (i % (GF_BK / 4)) * 4;
            const bool ok = m0 + r < M && k0 + c < K;
            f32_copy16(st + (r * LA + c) * 4, ok ? A + (size_t)(m0 + r) * lda + k0 + c : A, ok);
        }
#pragma unroll
        for (int i = tid; i < BN * (GF_BK / WV); i += 256) {
            const int r = i / (GF_BK / WV), c = (i % (GF_BK / WV)) * WV;
            const bool ok = n0 + r < N && k0 + c < K;
            f32_copy16(st + Sh::A_BYTES + (r * LW + c) * (int)sizeof(TW), ok ? W + (size_t)(n0 + r) * ldw + k0 + c : W, ok);
        }
    };
    const int steps = (K + GF_BK - 1) / GF_BK;
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (s < steps) fetch(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    int stage = 0, ahead = S - 1;
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncthreads();                                 // step s has landed for everybody, and step s - 1 is read by everybody
        if (s + S - 1 < steps) fetch(s + S - 1, ahead);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = reinterpret_cast<const float*>(smem + stage * Sh::STAGE) + ty * LA;
        const TW* ws = reinterpret_cast<const TW*>(smem + stage * Sh::STAGE + Sh::A_BYTES) + tx * LW;
        // behind the end of K the step holds zeros, which a chain takes like any other product, up to a multiple of 16
        const int kn = min(GF_BK, (K - s * GF_BK + 15) & ~15);
#pragma unroll 4
        for (int k = 0; k < kn; k += 4) {
            float w[TN][4];
            float4 a[TM];
#pragma unroll
            for (int j = 0; j < TN; ++j) widen4(ws + 16 * j * LW + k, w[j]);
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + 16 * i * LA + k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float x = e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w;
#pragma unroll
                    for (int j = 0; j < TN; j += 2) fma2(acc[i][j], acc[i][j + 1], x, w[j][e], w[j + 1][e]);
                }
        }
        stage = stage + 1 == S ? 0 : stage + 1;
        ahead = ahead + 1 == S ? 0 : ahead + 1;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + 16 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + 16 * j;
            if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j] + (bias ? to_f<TW>(bias[gn]) : 0.f);
        }
    }
}

// ------------------------------------------------------------------ few rows (decoding)
// A block has 32 outputs n; a lane one of them, a warp MT of the rows.  What the launch moves is the weights, once: their
// rows come in pieces of ROW bytes through a ring of S stages of cp.async.  A lane reads its own weight row 16 bytes at a time
// (rows ROW + 16 bytes apart: no bank is hit twice) and the activations as broadcasts.  An output is one chain, so K
// multiply-adds of latency are the other bound (4 cycles each: 38 us for K = 18,944).  Where the outputs are few, every
// chain gets a lane of its own (MT 1) and long pieces; where they fill the GPU several times, a warp takes several rows, so
// that a weight is read and widened once for all of them, and pieces are short, so that more blocks share an SM.
constexpr int GF_FEW_N = 32, GF_FEW_MAX = 32;

template <typename TW, int MT, int ROW, int S>
__global__ void __launch_bounds__(256)
gemm_f32_few_kernel(const float* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, const TW* __restrict__ bias,
                    float* __restrict__ C, int ldc, int M, int N, int K) {
    constexpr int BK = ROW / sizeof(TW), WV = 16 / sizeof(TW), PAD = ROW + 16;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x;
    const int n0 = blockIdx.x * GF_FEW_N, m0 = blockIdx.y * GF_FEW_MAX, rows = MT * (nt >> 5);
    const int w_bytes = GF_FEW_N * PAD, stage_bytes = w_bytes + rows * BK * 4;
    auto fetch = [&](int step, int stage) {
        unsigned char* st = smem + stage * stage_bytes;
        const int k0 = step * BK;
        for (int i = tid; i < GF_FEW_N * (ROW / 16); i += nt) {
            const int r = i / (ROW / 16), c = i % (ROW / 16), k = k0 + c * WV;
            const bool ok = n0 + r < N && k < K;
            f32_copy16(st + r * PAD + c * 16, ok ? W + (size_t)(n0 + r) * ldw + k : W, ok);
        }
        for (int i = tid; i < rows * (BK / 4); i += nt) {
            const int r = i / (BK / 4), k = k0 + (i % (BK / 4)) * 4;
            const bool ok = m0 + r < M && k < K;
            f32_copy16(st + w_bytes + i * 16, ok ? A + (size_t)(m0 + r) * lda + k : A, ok);
        }
    };
    const int steps = (K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (s < steps) fetch(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0.f;
    int stage = 0, ahead = S - 1;
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncthreads();                                 // step s has landed for everybody, and step s - 1 is read by everybody
        if (s + S - 1 < steps) fetch(s + S - 1, ahead);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const unsigned char* st = smem + stage * stage_bytes;
        const TW* ws = reinterpret_cast<const TW*>(st + lane * PAD);
        const float* as = reinterpret_cast<const float*>(st + w_bytes) + wid * MT * BK;
        // 16 k at a time, the next 16 fetched from shared memory in front of this one's chains; zeros behind the end of K up to
        // a multiple of 16, as in the tiles
        const int kn = min(BK, (K - s * BK + 15) & ~15);
        float w[2][16];
        float4 x[2][MT][4];
        auto load = [&](int b, int k) {
#pragma unroll
            for (int e = 0; e < 16; e += WV) {
                float v[WV];
                widen(*reinterpret_cast<const uint4*>(ws + k + e), v);
#pragma unroll
                for (int c = 0; c < WV; ++c) w[b][e + c] = v[c];
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) x[b][i][e] = *reinterpret_cast<const float4*>(as + i * BK + k + 4 * e);
        };
        auto chain = [&](int b) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[b][i][e].x, w[b][4 * e], acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[b][i][e].y, w[b][4 * e + 1], acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[b][i][e].z, w[b][4 * e + 2], acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(x[b][i][e].w, w[b][4 * e + 3], acc[i]);
            }
        };
        load(0, 0);
        if (kn == BK) {
#pragma unroll
            for (int k = 0; k < BK; k += 16) {
                if (k + 16 < BK) load((k / 16 + 1) & 1, k + 16);
                chain((k / 16) & 1);
            }
        } else {
            for (int k = 0; k < kn; k += 16) { load(0, k); chain(0); }
        }
        stage = stage + 1 == S ? 0 : stage + 1;
        ahead = ahead + 1 == S ? 0 : ahead + 1;
    }
    const int n = n0 + lane;
    if (n < N) {
        const float bv = bias ? to_f<TW>(bias[n]) : 0.f;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const int m = m0 + wid * MT + i;
            if (m < M) C[(size_t)m * ldc + n] = acc[i] + bv;
        }
    }
}

// ------------------------------------------------------------------ any strides
constexpr int GP_M = 64, GP_N = 64, GP_K = 16;

template <typename TW>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                const TW* __restrict__ bias, float* __restrict__ C, int ldc, int M, int N, int K) {
    __shared__ float As[GP_K][GP_M + 4];
    __shared__ float Ws[GP_K][GP_N + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;      // 16 x 16 threads, 4 x 4 outputs each
    const int m0 = blockIdx.y * GP_M, n0 = blockIdx.x * GP_N;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += GP_K) {
        // 64 x 16 elements per tile, 256 threads: 4 each; consecutive threads walk k (contiguous)
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int idx = threadIdx.x + it * 256;
            const int r = idx >> 4, kk = idx & 15;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
            As[kk][r] = (gm < M && gk < K) ? A[(size_t)gm * lda + gk] : 0.f;
            Ws[kk][r] = (gn < N && gk < K) ? to_f<TW>(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GP_K; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j] + (bias ? to_f<TW>(bias[gn]) : 0.f);
        }
    }
}

template <typename TW, int MT, int ROW, int S>
static int launch_few(const float* A, int lda, const TW* W, int ldw, const TW* bias, float* C, int ldc, int M, int N, int K,
                      cudaStream_t stream) {
    constexpr int BK = ROW / (int)sizeof(TW), MOST = S * (GF_FEW_N * (ROW + 16) + 8 * MT * BK * 4);      // at most 8 warps
    static bool raised[TL_MAX_DEVICES] = {};
    const int e = tl_raise_smem(gemm_f32_few_kernel<TW, MT, ROW, S>, raised, MOST);
    if (e) return e;
    const int m = M < GF_FEW_MAX ? M : GF_FEW_MAX, warps = m > MT ? (m + MT - 1) / MT : 2;      // one warp alone would fetch too slowly
    const int smem = S * (GF_FEW_N * (ROW + 16) + warps * MT * BK * 4);
    const dim3 grid((N + GF_FEW_N - 1) / GF_FEW_N, (M + GF_FEW_MAX - 1) / GF_FEW_MAX);
    gemm_f32_few_kernel<TW, MT, ROW, S><<<grid, warps * 32, smem, stream>>>(A, lda, W, ldw, bias, C, ldc, M, N, K);
    return tl_launch_status();
}

template <typename TW, int TM, int TN>
static int launch_tile(const float* A, int lda, const TW* W, int ldw, const TW* bias, float* C, int ldc, int M, int N, int K,
                       cudaStream_t stream) {
    using Sh = TileShape<TW, TM, TN>;
    constexpr int SMEM = Sh::STAGES * Sh::STAGE;
    static bool raised[TL_MAX_DEVICES] = {};
    const int e = tl_raise_smem(gemm_f32_tile_kernel<TW, TM, TN>, raised, SMEM);
    if (e) return e;
    const dim3 grid((M + Sh::BM - 1) / Sh::BM, (N + Sh::BN - 1) / Sh::BN);
    if (grid.y > 65535) return 1;
    gemm_f32_tile_kernel<TW, TM, TN><<<grid, 256, SMEM, stream>>>(A, lda, W, ldw, bias, C, ldc, M, N, K);
    return tl_launch_status();
}

template <typename TW>
static int launch_gemm_f32(const float* A, int lda, const TW* W, int ldw, const TW* bias, float* C, int ldc, int M, int N, int K,
                           cudaStream_t stream) {
    const bool wide = K % (16 / (int)sizeof(TW)) == 0 && K % 4 == 0 && lda % 4 == 0 && ldw % (16 / (int)sizeof(TW)) == 0 &&
                      ((((uintptr_t)A) | ((uintptr_t)W)) & 15) == 0;
    if (!wide) {
        dim3 grid((N + GP_N - 1) / GP_N, (M + GP_M - 1) / GP_M);
        if (grid.y > 65535) return 1;
        gemm_f32_kernel<TW><<<grid, 256, 0, stream>>>(A, lda, W, ldw, bias, C, ldc, M, N, K);
        return tl_launch_status();
    }
#define GO(F) return F(A, lda, W, ldw, bias, C, ldc, M, N, K, stream)
    // Few rows.  Outputs that fill the SMs at most twice over: a chain a lane, long pieces (N 3,584, K 18,944, 4 rows: 112 us; two
    // rows a warp 154, short pieces 159).  More outputs: rows share a warp, short pieces (N 37,888, K 3,584: 1 row 63 us against
    // 89; 4 rows 76 us with two rows a warp, 93 with one, 111 with four; 8 rows 111 us with four, 127 with two).
    const long long sms = tl_num_sms();
    const bool wide_n = (long long)N > 2 * sms * GF_FEW_N;
    if (M <= 32 && !wide_n) {
        if (M <= 8) GO((launch_few<TW, 1, 512, 4>));
        if (M <= 16) GO((launch_few<TW, 2, 256, 4>));
        GO((launch_few<TW, 4, 256, 4>));
    }
    if (M == 1) GO((launch_few<TW, 1, 128, 4>));
    if (M <= 4) GO((launch_few<TW, 2, 128, 4>));
    if (M <= 16) GO((launch_few<TW, 4, 128, 4>));        // 16 rows: 203 us against 272 as tiles; 32 rows: 371 against 272
    // The tile that is done first: rounds of tiles over the SMs times a tile's outputs, over the rate measured for that size (in
    // outputs of 3,584 products a us) where one block has an SM to itself and where several share it.
    auto cost = [&](int bm, int bn, double alone, double shared) {
        const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn), rounds = (tiles + sms - 1) / sms;
        return (double)rounds * bm * bn / (rounds == 1 ? alone : shared);
    };
    const double c[6] = {cost(128, 128, 42.4, 42.9), cost(96, 128, 41.0, 46.0), cost(128, 96, 40.5, 43.0), cost(96, 96, 38.0, 44.0),
                         cost(64, 128, 36.4, 44.0), cost(64, 64, 27.9, 38.0)};
    int best = 0;
    for (int i = 1; i < 6; ++i) if (c[i] < c[best]) best = i;
    if (cost(32, 64, 21.6, 35.7) < c[best]) GO((launch_tile<TW, 2, 4>));
    switch (best) {
        case 0: GO((launch_tile<TW, 8, 8>));
        case 1: GO((launch_tile<TW, 6, 8>));
        case 2: GO((launch_tile<TW, 8, 6>));
        case 3: GO((launch_tile<TW, 6, 6>));
        case 4: GO((launch_tile<TW, 4, 8>));
        default: GO((launch_tile<TW, 4, 4>));
    }
#undef GO
}

TL_EXPORT int tl_gemm_f32(const float* A, int lda, const void* W, int ldw, int w_dtype, const void* bias,
                          float* C, int ldc, int M, int N, int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (w_dtype == TL_F32) return launch_gemm_f32<float>(A, lda, (const float*)W, ldw, (const float*)bias, C, ldc, M, N, K, stream);
    return launch_gemm_f32<bf16>(A, lda, (const bf16*)W, ldw, (const bf16*)bias, C, ldc, M, N, K, stream);
}
