// C[M,N] = A[M,K] * W[N,K]^T (+ bias) of the 32-bit engine for weights stored as bfloat16, on the tensor cores without giving up a
// bit of an operand of 2^-110 or more: a float is the sum of three bfloat16 parts (24 bits, cut off one after the other, so that
// the parts are exact and none overflows), a product of a part and a weight is exact in float, and the sums are float.  Of smaller
// operands what lies below 2^-133, the smallest bfloat16, is lost.  Outputs that come out as no number (an infinite weight times
// a part that is zero is none) are taken again as chains.
//
// What a row's result is does not depend on the rows beside it, nor on how many there are: every output is
//     sum over groups of 4,096 k ( sum over segments of 1,024 k ( sum over chunks of 64 k ( the tensor cores' sum of the chunk's products )))
// in ascending order, each plus sign an addition that rounds.  Only a chunk is added up by the tensor cores, which cut an
// accumulator's last bits off instead of rounding it: the lowest parts first, while the accumulator is small, twelve instructions
// of 16 k.  How the work is dealt out - tiles of 32 to 176 tokens, an item a segment or a group, its sums kept by the
// block or added up by a second kernel - leaves the order as it is.
//
// Two thread blocks on neighbouring SMs (a cluster of two) work on 256 rows of W and BN tokens: tcgen05.mma.cta_group::2 with W on the
// 256-row side, the three parts of the tokens after one another on the other.  Each block brings its own 128 rows of W and half of
// the tokens' parts by TMA.  The accumulator of a chunk is double-buffered in tensor memory: eight warps of each block take one
// into registers and add it to the segment's sum while the next is made; a group's sum waits in tensor memory.
// What bounds it: with few tokens the weights from memory (a chunk of W takes an SM about 700 cycles at HBM's rate; the three
// passes over it from shared memory take 512 + 3 BN), with many the tensor cores (6 BN cycles a chunk: 1,056 measured at BN 176).
// 176 tokens are the widest tile whose copies still have four stages in shared memory (a stage of 181 would be a quarter of it), and a
// group's sums in tensor memory beside two accumulators but for nine columns a warp.
// Measured beside chains of float multiply-adds (gemm_f32.cu), us and error against 64 bits, norm over norm:
//     N 37,888  K 3,584     336 rows 186 (2,101)   64 rows 60 (396)   4 rows 51 (72)    1.2e-7 (1.1e-6)
//     N  3,584  K 18,944    336 rows 111 (1,703)   64 rows 41 (470)   4 rows 35 (109)   1.3e-7 (2.5e-6)
//     N  2,048  K 2,048     336 rows  21 (116)     64 rows 13 (53)    4 rows 13 (14)    1.1e-7 (8.1e-7)
//     N  1,024  K 1,024     336 rows  12 (43)      64 rows 11 (28)    4 rows 11 (8)     1.1e-7 (5.7e-7), so left to the chains (ops.py)
#include "umma_pair.cuh"

namespace {

constexpr int GP_ROWS = 128;                             // rows of W a block (a pair: 256)
constexpr int GP_CHUNK = 64;                             // k a chunk: 64 bfloat16 = 128 bytes = one swizzle row
constexpr int GP_SEG = 16, GP_GROUP = 64;                // chunks a segment, a group
constexpr int GP_THREADS = 320;                          // warp 0: TMA, warp 1: tensor memory + MMA, warps 2..9: sums
constexpr int GP_W_BYTES = GP_ROWS * GP_CHUNK * 2;
constexpr int GP_SLAB = 2048;                            // rows of A at a time, at most: bounds the scratch for their parts
constexpr long long GP_SUMS = 256LL << 20;               // bytes of the items' sums, at most: bounds the rows at a time as well (parts_rows)

template <int BN> struct PartsShape {
    static constexpr int B_BYTES = (BN / 2) * GP_CHUNK * 2;              // a block's half of one part of the tokens
    static constexpr int STAGE = GP_W_BYTES + 3 * B_BYTES;
    static constexpr int STAGES = (200 * 1024) / STAGE < 8 ? (200 * 1024) / STAGE : 8;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 512;
    static constexpr int CW = BN / 2;                                    // columns a warp sums
    static constexpr int BUFS = BN <= 32 ? 8 : BN <= 64 ? 6 : BN <= 96 ? 4 : BN <= 128 ? 3 : 2;      // accumulators in turn
    static constexpr int KEPT = 512 - BUFS * BN >= BN ? CW : (512 - BUFS * BN) / 2;      // columns of a group's sums in tensor memory
    static_assert(BN % 32 == 0 || BN % 16 == 0, "rows of a half lie in groups of 8");
};

struct PartsArgs {
    float* out; int ldo;                                 // [M, ldo], or
    float* partial;                                      // [items' sums along K][M, N], bias left out
    const bf16* bias;
    int M, N, K;
    int m_tiles, t_tiles, k_parts, part_chunks;          // tiles of W rows, of tokens; items along K and their chunks
    int* status;
    const float* A; int lda; const bf16* W;              // the operands themselves, for gp_chains
};

// Sums of parts that are no number: an infinite weight times a part that is zero is none, the float itself times it may be an infinity.
// Outputs `at`, `at` + ld .. (rows m .. m + rows - 1 of A, row n of W) that are none are taken again as gemm_f32.cu takes them, in one
// chain of multiply-adds.
__device__ __forceinline__ void gp_chains(const PartsArgs& G, const bf16* bias, int m, int rows, int n, float* at, size_t ld) {
    for (int x0 = 0; x0 < rows; x0 += 8) {
        bool odd = false;
        for (int x = x0; x < min(rows, x0 + 8); ++x) odd = odd || at[x * ld] != at[x * ld];
        if (!odd) continue;
        float sum[8] = {};
        for (int k = 0; k < G.K; k += 4) {
            const uint2 w = *reinterpret_cast<const uint2*>(G.W + (size_t)n * G.K + k);
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float4 a = *reinterpret_cast<const float4*>(G.A + (size_t)(m + min(x0 + x, rows - 1)) * G.lda + k);
                sum[x] = fmaf(a.x, __uint_as_float(w.x << 16), sum[x]);
                sum[x] = fmaf(a.y, __uint_as_float(w.x & 0xffff0000u), sum[x]);
                sum[x] = fmaf(a.z, __uint_as_float(w.y << 16), sum[x]);
                sum[x] = fmaf(a.w, __uint_as_float(w.y & 0xffff0000u), sum[x]);
            }
        }
#pragma unroll
        for (int x = 0; x < 8; ++x)
            if (x0 + x < rows && at[(x0 + x) * ld] != at[(x0 + x) * ld]) at[(x0 + x) * ld] = bias ? sum[x] + to_f<bf16>(bias[n]) : sum[x];
    }
}

// the largest of N sums and `w`, no number if one of them is none: an instruction for two
template <int N> __device__ __forceinline__ float gp_worst(const float (&x)[N], float w) {
#pragma unroll
    for (int i = 0; i < N; i += 2) asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(w) : "f"(x[i]), "f"(x[i + 1 < N ? i + 1 : i]));
    return w;
}
__device__ __forceinline__ void gp_ld8(uint32_t at, float* r) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]) : "r"(at));
}
__device__ __forceinline__ void gp_ld16(uint32_t at, float* r) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
                   "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]) : "r"(at));
}
__device__ __forceinline__ void gp_st8(uint32_t at, const float* r) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(r);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(at), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]) : "memory");
}
// N (a multiple of 8) columns at `at`
template <int N> __device__ __forceinline__ void gp_ld(uint32_t at, float (&r)[N]) {
#pragma unroll
    for (int c = 0; c + 16 <= N; c += 16) gp_ld16(at + c, r + c);
    if (N % 16) gp_ld8(at + N - 8, r + N - 8);
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_f32_parts_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const PartsArgs G) {
    using Sh = PartsShape<BN>;
    constexpr int S = Sh::STAGES, CW = Sh::CW, KEPT = Sh::KEPT, NB = Sh::BUFS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + S * Sh::STAGE);      // leader's: both blocks' bytes of a stage
    uint64_t* empty_bar = full_bar + S;                  // in each block: the MMAs that read the stage are done
    uint64_t* acc_full = empty_bar + S;                  // [NB] in each block: a chunk's accumulator is complete
    uint64_t* acc_empty = acc_full + NB;                 // [NB] leader's: the summing warps of both blocks have read it
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + NB);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = pair_rank();                     // 0: the leader, which issues the MMAs
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int chunks = (G.K + GP_CHUNK - 1) / GP_CHUNK, items = G.m_tiles * G.t_tiles * G.k_parts;
    struct Item { int m, t, k, c0, c1; };
    auto item_at = [&](int i) {                          // tokens' tiles next to one another: they share the tile of W in L2
        Item it;
        it.t = i % G.t_tiles; i /= G.t_tiles;
        it.m = i % G.m_tiles; it.k = i / G.m_tiles;
        it.c0 = it.k * G.part_chunks; it.c1 = min(chunks, it.c0 + G.part_chunks);
        return it;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        for (int b = 0; b < NB; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 16); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        pair_tmem_alloc(tmem_slot);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_cluster_sync();                                   // both blocks' barriers exist before anyone signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA (both blocks)
        const uint32_t one = pair_elect(), lead = rank == 0 ? one : 0u;
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        auto load_w = [&](const Item& t, int c, int s) {
            pair_expect(full_bar + s, 2 * Sh::STAGE, lead);
            pair_load(smem_addr(tiles + s * Sh::STAGE), &map_w, pair_peer(smem_addr(full_bar + s), 0), c * GP_CHUNK,
                      t.m * 2 * GP_ROWS + (int)rank * GP_ROWS, one);
        };
        auto load_x = [&](const Item& t, int c, int s) {
            const uint32_t bar = pair_peer(smem_addr(full_bar + s), 0), st = smem_addr(tiles + s * Sh::STAGE) + GP_W_BYTES;
#pragma unroll
            for (int p = 0; p < 3; ++p) pair_load(st + p * Sh::B_BYTES, &map_x, bar, c * GP_CHUNK, p * G.M + t.t * BN + (int)rank * (BN / 2), one);
        };
        // W is nobody's output: its first tiles are asked for before the wait for the kernel that writes the tokens' parts
        const Item first = item_at(pair);
        const int ahead = min(S, first.c1 - first.c0);
        for (int i = 0; i < ahead; ++i) load_w(first, first.c0 + i, i);
        grid_dependency_wait();
        grid_dependency_trigger();
        for (int i = 0; i < ahead; ++i) load_x(first, first.c0 + i, i);
        int it = 0;
        bool ok = true;
        for (int i = pair; i < items && ok; i += pairs) {
            const Item t = item_at(i);
            for (int c = t.c0; c < t.c1; ++c, ++it) {
                if (it < ahead) continue;
                const int s = it % S;
                if (it >= S && !mbar_wait(empty_bar + s, ((it / S) - 1) & 1, abort_flag, G.status, 41)) { ok = false; break; }
                load_w(t, c, s);
                load_x(t, c, s);
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------------------------------------------------------- MMA issuer (leader block)
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * GP_ROWS) >> 4) << 24);
        const uint32_t one = pair_elect();
        int it = 0;
        bool ok = true;
        grid_dependency_wait();                          // the bounded waits below start counting once the copies can land
        for (int i = pair; i < items && ok; i += pairs) {
            const Item t = item_at(i);
            for (int c = t.c0; c < t.c1; ++c, ++it) {
                const int s = it % S, buf = it % NB;
                if (it >= NB && !mbar_wait(acc_empty + buf, ((it / NB) - 1) & 1, abort_flag, G.status, 42)) { ok = false; break; }
                if (!mbar_wait(full_bar + s, (it / S) & 1, abort_flag, G.status, 43)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
                const uint32_t wa = smem_addr(tiles + s * Sh::STAGE), xa = wa + GP_W_BYTES;
#pragma unroll
                for (int p = 2; p >= 0; --p)             // the lowest parts first
#pragma unroll
                    for (int k = 0; k < GP_CHUNK / 16; ++k)
                        pair_mma(acc, desc_kmajor(wa + k * 32), desc_kmajor(xa + p * Sh::B_BYTES + k * 32), idesc, (p < 2 || k > 0) ? 1u : 0u, one);
                pair_commit(empty_bar + s, one);
                pair_commit(acc_full + buf, one);
            }
        }
    } else if (warp >= 2) {
        // ---------------------------------------------------------------- sums: 32 lanes (rows of W) and half of the columns (tokens) a warp
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t group_at = lanes + NB * BN + (uint32_t)(half * KEPT);
        const uint32_t leader_empty = pair_peer(smem_addr(acc_empty), 0);
        int it = 0;
        bool ok = true;
        float worst = 0.f;                               // no number if an output is none
        grid_dependency_wait();
        for (int i = pair; i < items && ok; i += pairs) {
            const Item t = item_at(i);
            float seg[CW], over[CW - KEPT + 1];          // `over`: a group's sums that tensor memory has no room for
#pragma unroll
            for (int c = 0; c < CW; ++c) seg[c] = 0.f;
            const bool grouped = G.part_chunks > GP_SEG;
            for (int c = t.c0; c < t.c1; ++c, ++it) {
                const int buf = it % NB;
                if (!mbar_wait(acc_full + buf, (it / NB) & 1, abort_flag, G.status, 44)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = lanes + (uint32_t)(buf * BN + half * CW);
#pragma unroll
                for (int x0 = 0; x0 + 32 <= CW; x0 += 32) {
                    float r[32];
                    gp_ld(at + x0, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int x = 0; x < 32; ++x) seg[x0 + x] += r[x];
                }
                if constexpr (CW % 32 > 0) {
                    float r[CW % 32];
                    gp_ld(at + CW / 32 * 32, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int x = 0; x < CW % 32; ++x) seg[CW / 32 * 32 + x] += r[x];
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) pair_arrive(leader_empty + (uint32_t)(buf * 8));
                if (grouped && ((c + 1) % GP_SEG == 0 || c + 1 == t.c1)) {       // a segment ends: into the group's sum
                    if (c / GP_SEG != t.c0 / GP_SEG) {   // not the first of its group
#pragma unroll
                        for (int x = 0; x < KEPT; x += 8) {
                            float g[8];
                            gp_ld8(group_at + x, g);
                            tmem_ld_wait();
#pragma unroll
                            for (int y = 0; y < 8; ++y) seg[x + y] += g[y];
                        }
#pragma unroll
                        for (int x = KEPT; x < CW; ++x) seg[x] += over[x - KEPT];
                    }
                    if (c + 1 != t.c1) {
#pragma unroll
                        for (int x = 0; x < KEPT; x += 8) {
                            gp_st8(group_at + x, seg + x);
#pragma unroll
                            for (int y = 0; y < 8; ++y) seg[x + y] = 0.f;
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int x = KEPT; x < CW; ++x) { over[x - KEPT] = seg[x]; seg[x] = 0.f; }
                    }
                }
            }
            if (!ok) break;
            const int n = t.m * 2 * GP_ROWS + (int)rank * GP_ROWS + quarter * 32 + lane, t0 = t.t * BN + half * CW;
            if (n < G.N) {
                float* dst = G.partial ? G.partial + ((size_t)t.k * G.M + t0) * G.N + n : G.out + (size_t)t0 * G.ldo + n;
                const size_t ld = G.partial ? G.N : G.ldo;
                const float b = !G.partial && G.bias ? to_f<bf16>(G.bias[n]) : 0.f;
                const bool add = !G.partial && G.bias;
#pragma unroll
                for (int x = 0; x < CW; ++x, dst += ld)
                    if (t0 + x < G.M) *dst = add ? seg[x] + b : seg[x];
                worst = gp_worst(seg, worst);
            }
        }
        if (worst != worst && ok && !G.partial)         // behind the loop, and inline: a call took 0.8 us of every launch for its stack
            for (int i = pair; i < items; i += pairs) {
                const Item t = item_at(i);
                const int n = t.m * 2 * GP_ROWS + (int)rank * GP_ROWS + quarter * 32 + lane, t0 = t.t * BN + half * CW;
                if (n < G.N && t0 < G.M) gp_chains(G, G.bias, t0, min(CW, G.M - t0), n, G.out + (size_t)t0 * G.ldo + n, G.ldo);
            }
    }
    // ---------------------------------------------------------------- teardown
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {                                   // give copies in flight time to land before the shared memory is handed on
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) { }
    }
    pair_cluster_sync();
    if (warp == 1) pair_tmem_free(tmem_base);
}

// ------------------------------------------------------------------ the parts of A
// x = p0 + p1 + p2, each the leading 8 bits of what is left (cut, not rounded: nothing overflows, and the three are exact);
// infinities and not-a-numbers are their first part alone.
__device__ __forceinline__ void gp_cut(float x, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    const uint32_t u = __float_as_uint(x);
    p0 = u & 0xffff0000u; p1 = 0u; p2 = 0u;
    if ((u & 0x7f800000u) == 0x7f800000u) {
        if (u & 0x007fffffu) p0 = 0x7fc00000u;
        return;
    }
    const float r = x - __uint_as_float(p0);
    p1 = __float_as_uint(r) & 0xffff0000u;
    p2 = __float_as_uint(r - __uint_as_float(p1));
}
// P[3][M][K] from A[M, K], K % 8 == 0: eight k a thread.  Moves 10 bytes an element, once for the whole product.
__global__ void __launch_bounds__(256) gemm_f32_cut_kernel(const float* __restrict__ A, int lda, bf16* __restrict__ P, int M, int K) {
    grid_dependency_wait();
    grid_dependency_trigger();
    const int k8 = K / 8;
    const long long total = (long long)M * k8;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const int m = (int)(i / k8), k = (int)(i - (long long)m * k8) * 8;
        const float4 a = *reinterpret_cast<const float4*>(A + (size_t)m * lda + k), b = *reinterpret_cast<const float4*>(A + (size_t)m * lda + k + 4);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t o[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t l[3], h[3];
            gp_cut(v[2 * e], l[0], l[1], l[2]);
            gp_cut(v[2 * e + 1], h[0], h[1], h[2]);
#pragma unroll
            for (int p = 0; p < 3; ++p) o[p][e] = __byte_perm(l[p], h[p], 0x7632);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint4*>(P + ((size_t)p * M + m) * K + k) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
    }
}

// ------------------------------------------------------------------ items' sums
// out = the sums of `parts` items along K; `seg`: items are segments, and four of them a group
template <int V>
__global__ void __launch_bounds__(256) gemm_f32_sum_kernel(const PartsArgs G, const bf16* __restrict__ bias, float* out, int ldo, int parts, int seg) {
    const float* __restrict__ partial = G.partial;
    const int M = G.M, N = G.N;
    grid_dependency_wait();
    grid_dependency_trigger();
    const int nv = N / V;
    const size_t stride = (size_t)M * N;
    float worst = 0.f;                                   // no number if a sum is none
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)M * nv; i += (long long)gridDim.x * 256) {
        const int m = (int)(i / nv), n = (int)(i - (long long)m * nv) * V;
        const float* src = partial + (size_t)m * N + n;
        float total[V], group[V];
#pragma unroll
        for (int x = 0; x < V; ++x) total[x] = group[x] = 0.f;
        const int run = seg ? GP_GROUP / GP_SEG : 1;
        for (int p = 0; p < parts; p += run) {
            float v[4][V];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (r >= run || p + r >= parts) break;
                if constexpr (V == 4) *reinterpret_cast<float4*>(v[r]) = *reinterpret_cast<const float4*>(src + (size_t)(p + r) * stride);
                else v[r][0] = src[(size_t)(p + r) * stride];
            }
#pragma unroll
            for (int x = 0; x < V; ++x) group[x] = v[0][x];
#pragma unroll
            for (int r = 1; r < 4; ++r) {
                if (r >= run || p + r >= parts) break;
#pragma unroll
                for (int x = 0; x < V; ++x) group[x] += v[r][x];
            }
#pragma unroll
            for (int x = 0; x < V; ++x) total[x] += group[x];
        }
        float* dst = out + (size_t)m * ldo + n;
#pragma unroll
        for (int x = 0; x < V; ++x) if (bias) total[x] += to_f<bf16>(bias[n + x]);
        if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(total[0], total[1], total[2], total[3]);
        else dst[0] = total[0];
        worst = gp_worst(total, worst);
    }
    if (worst != worst)
        for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)M * nv; i += (long long)gridDim.x * 256) {
            const int m = (int)(i / nv), n = (int)(i - (long long)m * nv) * V;
            for (int x = 0; x < V; ++x) gp_chains(G, bias, m, 1, n + x, out + (size_t)m * ldo + n + x, 0);
        }
}

// ------------------------------------------------------------------ the plan
constexpr int GP_WIDTHS[5] = {32, 64, 96, 128, 176};
struct PartsPlan { int bn, part_chunks, k_parts; double cycles; };

// The tile width and the length of an item along K that are done first, in cycles: rounds of items over the pairs of SMs, a chunk the
// longest of the tensor cores' time (6 BN), shared memory's (512 + 3 BN) and HBM's (700, where the whole GPU reads), and the
// writing and reading of the items' sums.
PartsPlan parts_plan(int M, int N, int K) {
    const int chunks = (K + GP_CHUNK - 1) / GP_CHUNK, pairs = tl_num_sms() / 2 > 0 ? tl_num_sms() / 2 : 1, m_tiles = (N + 255) / 256;
    PartsPlan best{0, 0, 0, 1e300};
    for (int bn : GP_WIDTHS)
        for (int len : {GP_SEG, GP_GROUP}) {
            const long long t_tiles = (M + bn - 1) / bn, k_parts = (chunks + len - 1) / len, items = t_tiles * m_tiles * k_parts;
            if (len == GP_SEG && k_parts > 1 && 4 * k_parts * M * N > GP_SUMS) continue;
            const long long rounds = (items + pairs - 1) / pairs, most = chunks < len ? chunks : len;
            const double hbm = 700.0 * (items < pairs ? (double)items / pairs : 1.0) / t_tiles, mma = 6.0 * bn, smem = 512.0 + 3.0 * bn;
            double c = mma > smem ? mma : smem;
            if (hbm > c) c = hbm;
            double cycles = rounds * (most * c + 800.0);
            if (k_parts > 1) cycles += 5000.0 + 8.0 * k_parts * M * (double)N / 2000.0;
            if (cycles < best.cycles) best = PartsPlan{bn, len, (int)k_parts, cycles};
        }
    return best;
}
// Rows of A at a time: the sums of items of a group fit in GP_SUMS (152,064 outputs of K 5,120: 176 rows; a product of 2,048 rows would need
// 2.5 GB), whole tiles of the widest kind, or of the narrowest.  A row's floats do not depend on them.
int parts_rows(int N, int K) {
    const long long groups = (K + GP_CHUNK * GP_GROUP - 1) / (GP_CHUNK * GP_GROUP);
    if (groups == 1) return GP_SLAB;
    const long long rows = GP_SUMS / (4 * groups * N);
    const int widest = GP_WIDTHS[4], narrowest = GP_WIDTHS[0];
    return rows >= GP_SLAB ? GP_SLAB : rows >= widest ? (int)(rows / widest) * widest : rows >= narrowest ? (int)(rows / narrowest) * narrowest : narrowest;
}
bool parts_takes(const void* A, int lda, const void* W, int N, int K) {
    // Whether a product comes here depends on the weights' size and the rows' alignment alone, never on M: a row's floats do not change
    // with the step it is in.  Smaller matrices (N 2,048, K 512: 4 rows 13 us against 8 as chains, 336 rows 15 against 37) are two or
    // three launches instead of one for single tokens and are left to the chains (so are longer rows up to where the caller draws its line).
    return K % 8 == 0 && K >= 1024 && (long long)N * K >= (1 << 20) && lda % 4 == 0 && ((((uintptr_t)A) | ((uintptr_t)W)) & 15) == 0;
}
size_t parts_bytes(int K, int m) { return ((size_t)3 * m * K * sizeof(bf16) + 255) & ~(size_t)255; }

template <int BN>
int parts_launch(const CUtensorMap& mw, const bf16* P, const PartsArgs& G, cudaStream_t stream) {
    using Sh = PartsShape<BN>;
    static bool raised[TL_MAX_DEVICES] = {};
    int e = tl_raise_smem(gemm_f32_parts_kernel<BN>, raised, Sh::SMEM);
    if (e) return e;
    CUtensorMap mx;
    if ((e = pair_map(&mx, P, 3LL * G.M, G.K, BN / 2))) return e;
    const long long items = (long long)G.m_tiles * G.t_tiles * G.k_parts;
    int pairs = tl_num_sms() / 2;
    if (items < pairs) pairs = (int)items;
    return launch_after_wait(gemm_f32_parts_kernel<BN>, dim3(2 * pairs), dim3(GP_THREADS), Sh::SMEM, stream, mw, mx, G);
}

}  // namespace

// The scratch that tl_gemm_f32_parts wants for a product in units of 256 bytes, 0 if it does not take it (a question of W and of
// alignment, not of M).
TL_EXPORT int tl_gemm_f32_parts_scratch(const float* A, int lda, const void* W, int M, int N, int K) {
    if (M <= 0 || N <= 0 || !parts_takes(A, lda, W, N, K)) return 0;
    size_t most = 0;
    const int rows = parts_rows(N, K);
    for (int m : {M < rows ? M : rows, M % rows}) {      // whole slabs and the last one
        if (m == 0) continue;
        const PartsPlan p = parts_plan(m, N, K);
        const size_t b = parts_bytes(K, m) + (p.k_parts > 1 ? (size_t)p.k_parts * m * N * sizeof(float) : 0);
        if (b > most) most = b;
    }
    return (int)((most + 255) / 256);
}

// How many kernels the function below launches.
TL_EXPORT int tl_gemm_f32_parts_launches(int M, int N, int K) {
    int n = 0;
    const int rows = parts_rows(N, K);
    for (int m0 = 0; m0 < M; m0 += rows) n += parts_plan(M - m0 < rows ? M - m0 : rows, N, K).k_parts > 1 ? 3 : 2;
    return n;
}

// C = A W^T (+ bias), W and bias bfloat16.  `scratch`: as much as the function above says, 256-byte aligned; `status`: device int.
TL_EXPORT int tl_gemm_f32_parts(const float* A, int lda, const void* W, const void* bias, float* C, int ldc, int M, int N, int K,
                                void* scratch, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (!parts_takes(A, lda, W, N, K) || scratch == nullptr || status == nullptr) return 1;
    int e = load_encode();
    if (e) return e;
    CUtensorMap mw;
    if ((e = pair_map(&mw, W, N, K, GP_ROWS))) return e;
    const long long cap = (long long)tl_num_sms() * 8;
    const int rows = parts_rows(N, K);
    for (int m0 = 0; m0 < M; m0 += rows) {
        const int m = M - m0 < rows ? M - m0 : rows;
        const PartsPlan plan = parts_plan(m, N, K);
        bf16* P = (bf16*)scratch;
        float* partial = plan.k_parts > 1 ? (float*)((unsigned char*)scratch + parts_bytes(K, m)) : nullptr;
        float* out = C + (size_t)m0 * ldc;
        const long long cut = ((long long)m * (K / 8) + 255) / 256;
        if ((e = launch_after_wait(gemm_f32_cut_kernel, dim3((unsigned)(cut < cap ? cut : cap)), dim3(256), 0, stream, A + (size_t)m0 * lda, lda, P, m, K))) return e;
        const PartsArgs G{out, ldc, partial, (const bf16*)bias, m, N, K, (N + 255) / 256, (m + plan.bn - 1) / plan.bn, plan.k_parts, plan.part_chunks, status, A + (size_t)m0 * lda, lda, (const bf16*)W};
        switch (plan.bn) {
            case 32: e = parts_launch<32>(mw, P, G, stream); break;
            case 64: e = parts_launch<64>(mw, P, G, stream); break;
            case 96: e = parts_launch<96>(mw, P, G, stream); break;
            case 128: e = parts_launch<128>(mw, P, G, stream); break;
            default: e = parts_launch<176>(mw, P, G, stream);
        }
        if (e) return e;
        if (!partial) continue;
        const int seg = plan.part_chunks == GP_SEG;
        const bool vec = N % 4 == 0 && ldc % 4 == 0 && ((uintptr_t)out & 15) == 0;
        const long long blocks = ((long long)m * N / (vec ? 4 : 1) + 255) / 256;
        const dim3 grid((unsigned)(blocks < cap ? blocks : cap));
        e = vec ? launch_after_wait(gemm_f32_sum_kernel<4>, grid, dim3(256), 0, stream, G, (const bf16*)bias, out, ldc, plan.k_parts, seg)
                : launch_after_wait(gemm_f32_sum_kernel<1>, grid, dim3(256), 0, stream, G, (const bf16*)bias, out, ldc, plan.k_parts, seg);
        if (e) return e;
    }
    return 0;
}
