// The experts' products of a step of many tokens, without padding and without the host: rows sorted by expert (moe_sort, moe_gather
// with the runs one behind the other), every expert's run times its own matrix, the runs' bounds read on the device.
//
//     up:    a[p, f] = act(x[p] . gate row f of e) * (x[p] . up row f of e)      (or relu(.)^2 of one product), [P, F]
//     down:  y[p, n] = a[p] . row n of e,                                        [P, N]
//
// Two thread blocks on neighbouring SMs (a cluster of two) work on one tile: 256 rows of an expert's matrix on the MMA's M side
// (tcgen05.mma.cta_group::2, 128 rows a block) and up to 256 rows of its run on the N side.  A run is cut into equal tiles, and the MMA's
// N is the tile's own width rounded up to 32, so that short runs (a step of 40 tokens gives an expert five rows) cost their weights'
// way from memory and little else, and long ones lose less than 32 rows; rows behind a run's end belong to the next expert and are
// not stored.  Blocks are persistent and take tiles pair, pair + pairs, ... of a list of which shared memory holds every expert's first
// entry.  The accumulator is double-buffered in tensor memory: eight warps turn one into bfloat16 rows while the next is made.
// For gated products a block's 128 rows are four groups of 16 gate rows and the 16 up rows of the same features (one copy of a box
// over five dimensions): a warp holds both and hands them over by shuffles, so the epilogue leaves shared memory to the products.
// What bounds it: with long runs shared memory and the tensor cores alike (a chunk of 64 k: 512 cycles each at width 256), with
// short ones the weights from HBM.  Measured with 32 experts, 4 a token, of 2,048 x 1,024, us beside the library's batched product over
// runs padded to the longest (and a kernel for the activation, and the read-back that the padding needs): 2,048 tokens up 78 (88 + 13),
// down 47 (44); 512 tokens 68 (72), 39 (41); 40 tokens 66 (68), 39 (39).  A step of 2,048 tokens, all in all: 221 (276); with the exchange of gate and
// up values through shared memory, by four warps, the up product alone took 121.
#include "umma_pair.cuh"

namespace {

constexpr int MP_ROWS = 128, MP_CHUNK = 64, MP_WIDE = 256, MP_STAGES = 6, MP_THREADS = 320;
constexpr int MP_W_BYTES = MP_ROWS * MP_CHUNK * 2, MP_STAGE = MP_W_BYTES + (MP_WIDE / 2) * MP_CHUNK * 2;
constexpr int MP_BOX = 16, MP_TALL = 64;                 // rows of a box of tokens; of a tall one
constexpr int MP_GROUP = 16;                             // gate rows beside their up rows
constexpr int MP_MAX_E = 1024;
constexpr int MP_SMEM = MP_STAGES * MP_STAGE + 2 * (MP_MAX_E + 1) * 4 + 1024 + 256;

struct MoeProductArgs {
    void* out; int ldo;                                  // [P, ldo] bfloat16 (KIND 8: float)
    const int* offsets; int E;                           // [E + 1]: expert e's run of rows
    int R, K;                                            // rows of an expert's matrix in memory, and their length
    int cols;                                            // columns of out: R, gated R / 2
    int m_tiles;                                         // pairs of blocks' tiles an expert
    float limit, alpha;
    int* status;
};

// one tile of the list: expert, tile of its matrix, the first row and the rows of its run, the MMA's width
struct MoeTile { int e, m, row, rows, width; };
// The i-th tile, by a whole warp; `e` is where the search starts (tiles are asked for in ascending order).  Tiles of an expert are (m, t), t fastest: they
// share the matrix's rows in L2.  False behind the last.
__device__ __forceinline__ bool moe_tile(int i, int& e, const int* offsets, const int* first, int E, MoeTile& t) {
    const int lane = threadIdx.x & 31;
    while (true) {                                       // the experts whose tiles all lie before i
        const int past = __popc(__ballot_sync(0xffffffffu, e + lane < E && first[e + lane + 1] <= i));
        e += past;
        if (past < 32) break;
    }
    if (e >= E) return false;
    const int row0 = offsets[e], run = offsets[e + 1] - row0, tiles = (run + MP_WIDE - 1) / MP_WIDE;
    const int j = i - first[e], m = j / tiles, tt = j - m * tiles;
    t.e = e; t.m = m;
    t.width = ((run + tiles - 1) / tiles + 31) & ~31;
    t.row = row0 + tt * t.width;
    t.rows = min(t.width, run - tt * t.width);
    return true;
}

__device__ __forceinline__ void moe_load5(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int group, int e, uint32_t one) {
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "setp.ne.b32 q, %6, 0;\n\t"
                 "@q cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %7, %7, %4, %5}], [%2];\n\t}"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(group), "r"(e), "r"(one), "r"(0) : "memory");
}

// KIND 0: as it is, 1..3: gates (tl_gate_mul), 4: relu(.)^2, each of values rounded to bfloat16 first, as a stored product would have been.
// Eight more: of the accumulators themselves, and 8 as floats, the gates by exact divisions (tl_act_pair: what streamed experts compute).  A
// parameter of the kernel: with
// the choice inside the loop over a thread's elements their chains did not overlap.
__device__ __forceinline__ float moe_rounded(float v, bool raw) { return raw ? v : __bfloat162float(__float2bfloat16_rn(v)); }
template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MP_THREADS, 1)
moe_product_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_tall,
                   const MoeProductArgs G) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + MP_STAGES * MP_STAGE);      // leader's
    uint64_t* empty_bar = full_bar + MP_STAGES;
    uint64_t* acc_full = empty_bar + MP_STAGES;          // [2] in each block
    uint64_t* acc_empty = acc_full + 2;                  // [2] leader's
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* offsets = reinterpret_cast<int*>(tmem_slot + 2);                                // [E + 1]
    int* first = offsets + G.E + 1;                                                      // [E + 1]: where an expert's tiles start in the list

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = pair_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, chunks = (G.K + MP_CHUNK - 1) / MP_CHUNK;
    constexpr bool raw = KIND >= 8, gated = KIND % 8 >= 1 && KIND % 8 <= 3;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MP_STAGES; ++s) { mbar_init(full_bar + s, 1); mbar_init(empty_bar + s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 16); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) pair_tmem_alloc(tmem_slot);
    grid_dependency_wait();
    grid_dependency_trigger();
    if (warp == 0) {                                     // the list
        int before = 0;
        for (int e0 = 0; e0 < G.E; e0 += 32) {
            const int e = e0 + lane, lo = e <= G.E ? G.offsets[e] : 0, hi = e < G.E ? G.offsets[e + 1] : lo;
            int sum = (hi - lo + MP_WIDE - 1) / MP_WIDE * G.m_tiles;
            const int here = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int x = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += x; }
            if (e < G.E) { offsets[e] = lo; offsets[e + 1] = hi; first[e] = before + sum - here; first[e + 1] = before + sum; }
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_cluster_sync();                                 // both blocks' barriers exist before anyone signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    MoeTile t;
    int e = 0;
    if (warp == 0) {
        // ---------------------------------------------------------------- TMA (both blocks)
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_tall) : "memory");
        const uint32_t one = pair_elect(), lead = rank == 0 ? one : 0u;
        int it = 0;
        bool ok = true;
        for (int i = pair; ok && moe_tile(i, e, offsets, first, G.E, t); i += pairs) {
            const int half = t.width / 2, x0 = t.row + (int)rank * half, block = t.m * 2 + (int)rank;
            const uint32_t bytes = 2 * (MP_W_BYTES + half * MP_CHUNK * 2);
            for (int c = 0; c < chunks; ++c, ++it) {
                const int s = it % MP_STAGES;
                if (it >= MP_STAGES && !mbar_wait(empty_bar + s, ((it / MP_STAGES) - 1) & 1, abort_flag, G.status, 45)) { ok = false; break; }
                pair_expect(full_bar + s, bytes, lead);
                const uint32_t bar = pair_peer(smem_addr(full_bar + s), 0), st = smem_addr(tiles + s * MP_STAGE);
                if (gated) moe_load5(st, &map_w, bar, c * MP_CHUNK, block * (MP_ROWS / 2 / MP_GROUP), t.e, one);
                else pair_load(st, &map_w, bar, c * MP_CHUNK, t.e * G.R + block * MP_ROWS, one);
                int r = 0;
                for (; r + MP_TALL <= half; r += MP_TALL) pair_load(st + MP_W_BYTES + r * MP_CHUNK * 2, &map_tall, bar, c * MP_CHUNK, x0 + r, one);
                for (; r < half; r += MP_BOX) pair_load(st + MP_W_BYTES + r * MP_CHUNK * 2, &map_x, bar, c * MP_CHUNK, x0 + r, one);
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ---------------------------------------------------------------- MMA issuer (leader block)
        const uint32_t one = pair_elect();
        int it = 0, ti = 0;
        bool ok = true;
        for (int i = pair; ok && moe_tile(i, e, offsets, first, G.E, t); i += pairs, ++ti) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(t.width >> 3) << 17) | ((uint32_t)((2 * MP_ROWS) >> 4) << 24);
            const int buf = ti & 1;
            if (ti >= 2 && !mbar_wait(acc_empty + buf, ((ti >> 1) - 1) & 1, abort_flag, G.status, 46)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_base + (uint32_t)(buf * MP_WIDE);
            for (int c = 0; c < chunks; ++c, ++it) {
                const int s = it % MP_STAGES;
                if (!mbar_wait(full_bar + s, (it / MP_STAGES) & 1, abort_flag, G.status, 47)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t wa = smem_addr(tiles + s * MP_STAGE), xa = wa + MP_W_BYTES;
#pragma unroll
                for (int k = 0; k < MP_CHUNK / 16; ++k)
                    pair_mma(acc, desc_kmajor(wa + k * 32), desc_kmajor(xa + k * 32), idesc, (c > 0 || k > 0) ? 1u : 0u, one);
                pair_commit(empty_bar + s, one);
            }
            if (ok) pair_commit(acc_full + buf, one);
        }
    } else if (warp >= 2) {
        // ---------------------------------------------------------------- epilogue: 32 of the block's 128 rows a warp, 16 rows of the run at a time;
        // two halves of four warps take turns of 16 rows
        const int quarter = warp & 3, turn = (warp - 2) >> 2;
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t leader_empty = pair_peer(smem_addr(acc_empty), 0);
        int ti = 0;
        for (int i = pair; moe_tile(i, e, offsets, first, G.E, t); i += pairs, ++ti) {
            const int buf = ti & 1, block = t.m * 2 + (int)rank;
            if (!mbar_wait(acc_full + buf, (ti >> 1) & 1, abort_flag, G.status, 48)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int col = gated ? block * (MP_ROWS / 2) + quarter * MP_GROUP + (lane & 15) : block * MP_ROWS + quarter * 32 + lane;
            for (int c0 = 16 * turn; c0 < t.rows; c0 += 32) {
                float r[16];
                {
                    uint32_t* u = reinterpret_cast<uint32_t*>(r);
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
                                   "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                                 : "r"(lanes + (uint32_t)(buf * MP_WIDE + c0)));
                }
                tmem_ld_wait();
                if (gated) {
                    // a feature's gate value is in lane f, its up value in lane 16 + f: the lower lanes finish the first eight rows, the
                    // upper ones the others, and each hands over what the other needs, rounded to bfloat16 like a stored product
                    const bool up = lane >= 16;
                    const int left = t.rows - c0 - (up ? 8 : 0);
                    float y[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float give = up ? r[j] : r[8 + j], keep = up ? r[8 + j] : r[j];
                        const float a = moe_rounded(keep, raw), b = moe_rounded(__shfl_xor_sync(0xffffffffu, give, 16), raw);
                        y[j] = raw ? tl_act_pair(up ? b : a, up ? a : b, KIND == 11 ? TL_ACT_SWISH_CLAMPED : KIND == 10 ? TL_ACT_GELU_TANH : TL_ACT_SILU, G.limit, G.alpha)
                                   : tl_gate_mul(up ? b : a, up ? a : b, KIND % 8, G.limit, G.alpha);
                    }
                    if (col < G.cols) {
                        bf16* dst = (bf16*)G.out + (size_t)(t.row + c0 + (up ? 8 : 0)) * G.ldo + col;
#pragma unroll
                        for (int j = 0; j < 8; ++j, dst += G.ldo) if (j < left) *dst = __float2bfloat16_rn(y[j]);
                    }
                } else if (col < G.cols) {
                    const int left = t.rows - c0;
                    const size_t at = (size_t)(t.row + c0) * G.ldo + col;
                    if (KIND == 8) {
                        float* dst = (float*)G.out + at;
#pragma unroll
                        for (int j = 0; j < 16; ++j, dst += G.ldo) if (j < left) *dst = r[j];
                    } else {
                        bf16* dst = (bf16*)G.out + at;
#pragma unroll
                        for (int j = 0; j < 16; ++j, dst += G.ldo) {
                            const float v = KIND == 12 ? fmaxf(r[j], 0.f) * fmaxf(r[j], 0.f) : KIND == 4 ? tl_relu_squared_rounded(r[j]) : r[j];
                            if (j < left) *dst = __float2bfloat16_rn(v);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) pair_arrive(leader_empty + (uint32_t)(buf * 8));
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

// w [E, 2 F, K] as (k, row of a group, gate or up, group, expert): a box is four groups of 16 gate and 16 up rows, 64 k wide
int gated_map(CUtensorMap* map, const void* base, int E, int F, int K) {
    const cuuint64_t row = (cuuint64_t)K * 2;
    cuuint64_t dims[5] = {(cuuint64_t)K, MP_GROUP, 2, (cuuint64_t)F / MP_GROUP, (cuuint64_t)E};
    cuuint64_t strides[4] = {row, row * F, row * MP_GROUP, row * 2 * F};
    cuuint32_t box[5] = {MP_CHUNK, MP_GROUP, 2, MP_ROWS / 2 / MP_GROUP, 1}, elem[5] = {1, 1, 1, 1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, elem,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 101;
}

template <int KIND>
int launch_product(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mt, const MoeProductArgs& G, int P, cudaStream_t stream) {
    static bool raised[TL_MAX_DEVICES] = {};
    const int e = tl_raise_smem(moe_product_kernel<KIND>, raised, MP_SMEM);
    if (e) return e;
    // no more pairs than there can be tiles: every expert's last tile may be short
    const long long most = (long long)G.m_tiles * (P / MP_WIDE + (P < G.E ? P : G.E));
    int pairs = tl_num_sms() / 2;
    if (most < pairs) pairs = (int)most;
    return launch_after_wait(moe_product_kernel<KIND>, dim3(2 * pairs), dim3(MP_THREADS), MP_SMEM, stream, mw, mx, mt, G);
}

}  // namespace

// Whether tl_moe_product takes products of rows of K values into `cols` columns.
TL_EXPORT int tl_moe_product_takes(int E, int K, int cols, int gated) {
    return E >= 1 && E <= MP_MAX_E && K >= 8 && K % 8 == 0 && cols >= 1 && (!gated || cols % MP_GROUP == 0);
}

// out[p, :] = rows p = offsets[e] .. offsets[e + 1] - 1 of x [P, K] times w[e] [R, K]^T, e = 0 .. E - 1, through `kind` (see the
// kernel).  x, w and out (kind 8: float) bfloat16, x and w 16-byte aligned; out [P, cols], rows ldo elements apart.
TL_EXPORT int tl_moe_product(const void* x, const void* w, const int* offsets, void* out, int ldo, int P, int E, int R, int K, int kind,
                             float limit, float alpha, int* status, cudaStream_t stream) {
    if (P <= 0) return 0;
    const bool gated = kind % 8 >= 1 && kind % 8 <= 3;
    const int cols = gated ? R / 2 : R;
    if (kind < 0 || kind > 12 || kind % 8 > 4 || (gated && R % 2) || !tl_moe_product_takes(E, K, cols, gated) || (long long)E * R > 2147483647LL ||
        ((((uintptr_t)x) | ((uintptr_t)w)) & 15) || status == nullptr) return 1;
    int e = load_encode();
    if (e) return e;
    CUtensorMap mw, mx, mt;
    if ((e = gated ? gated_map(&mw, w, E, cols, K) : pair_map(&mw, w, (long long)E * R, K, MP_ROWS))) return e;
    if ((e = pair_map(&mx, x, P, K, MP_BOX))) return e;
    if ((e = pair_map(&mt, x, P, K, MP_TALL))) return e;
    const MoeProductArgs G{out, ldo, offsets, E, R, K, cols, gated ? (cols + 127) / 128 : (cols + 255) / 256, limit, alpha, status};
    switch (kind) {
        case 0: return launch_product<0>(mw, mx, mt, G, P, stream);
        case 1: return launch_product<1>(mw, mx, mt, G, P, stream);
        case 2: return launch_product<2>(mw, mx, mt, G, P, stream);
        case 3: return launch_product<3>(mw, mx, mt, G, P, stream);
        case 4: return launch_product<4>(mw, mx, mt, G, P, stream);
        case 8: return launch_product<8>(mw, mx, mt, G, P, stream);
        case 9: return launch_product<9>(mw, mx, mt, G, P, stream);
        case 10: return launch_product<10>(mw, mx, mt, G, P, stream);
        case 11: return launch_product<11>(mw, mx, mt, G, P, stream);
        default: return launch_product<12>(mw, mx, mt, G, P, stream);
    }
}
