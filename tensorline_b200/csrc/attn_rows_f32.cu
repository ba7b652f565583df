// Exact-order paged attention of the 32-bit engine, the same floats as attn_tokenwise.cu gives: per (token, query head) tiles of
// 32 keys aligned to absolute position 0 in ascending order, every dot product one chain of fmaf over the head's dimensions, the
// softmax's sums over the 32 keys of a tile in the order of a warp's shuffles, every output element one chain of fmaf over the
// keys.  What the token-wise kernel spends its time on is fetching every key anew for every token and head, one row a lane; here
// the rows (token, head) that read the same keys share them through shared memory, and a step of few tokens has its dot products
// taken by as many blocks as there are tiles.
//
//   attn_rows       a block has up to 64 (or 32) rows: neighbouring tokens of one request times the query heads of one KV head.
//                   Four warps; a warp owns 16 (or 8) rows from the dot products over the softmax to the values, so between tiles only the
//                   tiles themselves are waited for: K of the next tile arrives while the values are summed, V of it while
//                   the dot products are taken; where a tile's keys lie is looked up a tile ahead.  Operands come from shared memory
//                   a step ahead of the multiply-adds.  A tile costs 2 x 64 x 32 x d multiply-adds; what bounds it is the latency of a
//                   warp's instructions (one in 3.6 cycles) as long as few warps share an SM, then their issue.
//   attn_dots, attn_chain   steps of few tokens: the chains over the keys are all that is left in order.  attn_dots: a thread
//                   a key, all tiles at once, scores to memory; attn_chain: a warp a head and 32 output columns, the softmax of
//                   128 keys at a time and then their chain.
// Measured with 28 query heads of 128 on 4 KV heads: 333 tokens on 700 cached 254 us (the token-wise kernel 5,076; blocks of 64 rows
// without the look-ahead 350), 2,048 tokens 1.29 ms (33.4; 1.31); single tokens at position 1,800: 4 of them 56 us (1,842; attn_rows 478), 64 of them 265 us (3,577; 611).
// Masks, sinks, gates, caps and slopes: as described in attn_tokenwise.cu.  The roundings are spelt out here
// and there: which kernel a row is given to does not show in its floats.
#include "common.cuh"

struct RowsArgs {
    const float* q; int q_stride; float* out;
    const float* k_pages; const float* v_pages;
    const int* table; int max_pages; int page_size;
    const int* pos; const int* req_slot;
    int T, nq, nkv, d, window; float scale;
    const float* sink; int keep_first; const float* gate;
    int chunk; const float* slopes; float cap;
    float* scores; int keys;               // attn_dots / attn_chain: [T, nq, keys]
    int tq;                                // attn_rows: tokens a block
    TlLimits L;
};

__device__ __forceinline__ void rows_copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
#define ROWS_COMMIT() asm volatile("cp.async.commit_group;" ::: "memory")
#define ROWS_WAIT(n) asm volatile("cp.async.wait_group %0;" ::"n"(n) : "memory")

__device__ __forceinline__ void rows_fma2(float& d0, float& d1, float a, float b0, float b1) {       // (d0, d1) += a (b0, b1)
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 z, {%0, %1};\n\t"
        "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "+f"(d0), "+f"(d1) : "f"(a), "f"(b0), "f"(b1));
}

__device__ __forceinline__ int rows_low(const RowsArgs& A, int p) {
    return A.chunk > 0 ? (p / A.chunk) * A.chunk : (A.window > 0 && p - A.window + 1 > 0) ? p - A.window + 1 : 0;
}
__device__ __forceinline__ size_t rows_offset(const RowsArgs& A, const int* tab, int j, int kh) {
    const int page = tl_checked(tab[tl_checked(j / A.page_size, A.max_pages, A.L, TL_K_TOKENWISE)], A.L.total_pages, A.L, TL_K_TOKENWISE);
    return (((size_t)page * A.nkv + kh) * A.page_size + (j % A.page_size)) * A.d;
}
__device__ __forceinline__ const float* rows_at(const RowsArgs& A, const float* pages, const int* tab, int j, int kh) {
    return pages + rows_offset(A, tab, j, kh);
}
// The position of a token whose scores lie in `scores`: one beyond the table is recorded by the checking build, and cut in every build, so
// that nothing outside the scratch is touched.
__device__ __forceinline__ int rows_position(const RowsArgs& A, int t) {
    const int p = A.pos[t];
    return p < 0 ? p : min(tl_checked(p, A.keys, A.L, TL_K_TOKENWISE), A.keys - 1);
}
__device__ __forceinline__ float rows_score(const RowsArgs& A, float dot, float slope, int p, int j) {
    float s = __fmul_rn(dot, A.scale);                   // spelt out: the same roundings in every kernel
    if (A.cap > 0.f) s = __fmul_rn(A.cap, tanhf(s / A.cap));
    if (A.slopes) s = fmaf(-slope, (float)(p - j), s);
    return s;
}
constexpr int ROWS_MAX = 64;

// NC: groups of 64 output columns (d <= 64 NC); ROWS: rows a block, RW: a warp
template <int NC, int ROWS, int RW>
__global__ void __launch_bounds__(ROWS / RW * 32, NC == 1 && RW == 16 ? 4 : 0) attn_rows_kernel(const RowsArgs A) {
    constexpr int NT = ROWS / RW * 32, TK = NT / 32, ROWS_PS = ROWS + 4;                      // threads, and those that fetch a key
    // Operands a step ahead of the multiply-adds: not in blocks of 64 rows of short heads, where four blocks an SM hide the latency (40 heads of 64 on
    // 1, 4,096 tokens 4.73 ms; ahead 4.98, and ahead with the registers that leave three blocks 5.39)
    constexpr bool AHEAD = NC > 1 || RW == 8;
    constexpr int LC = RW == 16 || NC == 1 ? 16 : 32, VR = RW * LC / 32, VC = 16 * NC / LC;      // values: lanes over columns, rows and column groups a lane
    extern __shared__ __align__(16) float sm[];
    const int d = A.d, g = A.nq / A.nkv, ld = d + 4;
    float* Qs = sm;                                      // [64][ld], rows beyond the block's last are zeros
    float* Ks = Qs + ROWS * ld;                      // [32][ld]
    float* Vs = Ks + 32 * ld;                            // [32][ld]
    float* Ps = Vs + 32 * ld;                            // [32 keys][ROWS_PS rows]: dot products, then weights
    float* al = Ps + 32 * ROWS_PS;                       // [64]
    const int kh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    // the block's run: the blockIdx.z-th maximal range of tokens of one request among its tq tokens (tq <= 32)
    const int tb = blockIdx.x * A.tq, te = min(A.T, tb + A.tq);
    unsigned starts;
    {
        const int t = tb + lane;
        starts = __ballot_sync(0xffffffffu, t < te && (lane == 0 || A.req_slot[t] != A.req_slot[t - 1]));
    }
    if ((int)blockIdx.z >= __popc(starts)) return;
    for (unsigned i = 0; i < blockIdx.z; ++i) starts &= starts - 1;
    const int first = __ffs(starts) - 1;
    starts &= starts - 1;
    const int n = (starts ? __ffs(starts) - 1 : te - tb) - first, t0 = tb + first, rows = n * g;
    const int* tab = A.table + (size_t)tl_checked(A.req_slot[t0], A.L.table_rows, A.L, TL_K_TOKENWISE) * A.max_pages;
    for (int i = tid; i < ROWS * d; i += NT) {
        const int r = i / d, e = i - r * d;
        Qs[r * ld + e] = r < rows ? A.q[(size_t)(t0 + r / g) * A.q_stride + (size_t)(kh * g + r % g) * d + e] : 0.f;
    }
    // the softmax's row of this lane: the G lanes RW apart share a row, every G-th key each
    constexpr int G = 32 / RW;
    const int row = wid * RW + lane % RW, kb = lane / RW;
    const bool live = row < rows;
    const int p = live ? A.pos[t0 + row / g] : -1, head = kh * g + row % g;
    const int lo = live ? rows_low(A, p) : 0, kept = min(A.keep_first, lo);
    const float slope = A.slopes && live ? A.slopes[head] : 0.f;
    float m = -INFINITY, l = 0.f;
    int last = -1, low = 0x7fffffff, keep = 0;           // of all the run's tokens
    for (int i = 0; i < n; ++i) {
        const int pi = A.pos[t0 + i], li = rows_low(A, pi);
        last = max(last, pi); low = min(low, li); keep = max(keep, min(A.keep_first, li));
    }
    auto next = [&](int j0) { return (j0 >= keep && j0 + 32 <= low) ? (low / 32) * 32 : j0; };
    // TK threads a key; keys that no row sees are not read.  Where a tile's keys lie is looked up a tile ahead, once for K and V.
    constexpr size_t NOWHERE = ~(size_t)0;
    auto where = [&](int j0) {
        const int j = j0 + tid / TK;
        return j <= last && (j >= low || j < keep) ? rows_offset(A, tab, j, kh) : NOWHERE;
    };
    auto fetch = [&](float* dst, const float* pages, size_t at) {
        if (at != NOWHERE)
            for (int e = tid % TK * 4; e < d; e += TK * 4) rows_copy16(dst + tid / TK * ld + e, pages + at + e);
        ROWS_COMMIT();
    };
    float acc[VR][4 * VC];
#pragma unroll
    for (int r = 0; r < VR; ++r)
#pragma unroll
        for (int c = 0; c < 4 * VC; ++c) acc[r][c] = 0.f;
    const int kl = lane & 7, rl = lane >> 3;             // dot products: keys kl + 8 j, rows RW wid + 4 i + rl
    const int dg = lane % LC * 4, rg = wid * RW + lane / LC * VR;      // values: columns dg + 4 LC c, rows rg ..
    int j0 = next(0);
    {
        const size_t at = where(j0);
        fetch(Ks, A.k_pages, at);
        fetch(Vs, A.v_pages, at);
    }
    while (j0 <= last) {
        const int j1 = next(j0 + 32);
        const size_t at = where(j1);
        ROWS_WAIT(1);
        __syncthreads();
        {
            float s[RW / 4][4];
#pragma unroll
            for (int i = 0; i < RW / 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
            const float* qp = Qs + (wid * RW + rl) * ld;
            const float* kp = Ks + kl * ld;
            // the next four dimensions are on their way from shared memory while these are multiplied
            float4 q4[2][RW / 4], k4[2][4];
            auto load = [&](int b, int e) {
#pragma unroll
                for (int i = 0; i < RW / 4; ++i) q4[b][i] = *reinterpret_cast<const float4*>(qp + 4 * i * ld + e);
#pragma unroll
                for (int j = 0; j < 4; ++j) k4[b][j] = *reinterpret_cast<const float4*>(kp + 8 * j * ld + e);
            };
            auto dots = [&](int b) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int i = 0; i < RW / 4; ++i) {
                        const float x = c == 0 ? q4[b][i].x : c == 1 ? q4[b][i].y : c == 2 ? q4[b][i].z : q4[b][i].w;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            s[i][j] = fmaf(x, c == 0 ? k4[b][j].x : c == 1 ? k4[b][j].y : c == 2 ? k4[b][j].z : k4[b][j].w, s[i][j]);
                    }
            };
            if constexpr (AHEAD) {
                load(0, 0);
                int e = 0;
                for (; e + 8 < d; e += 8) {
                    load(1, e + 4);
                    dots(0);
                    load(0, e + 8);
                    dots(1);
                }
                if (e + 4 < d) { load(1, e + 4); dots(0); dots(1); } else dots(0);
            } else {
#pragma unroll 2
                for (int e = 0; e < d; e += 4) { load(0, e); dots(0); }
            }
#pragma unroll
            for (int i = 0; i < RW / 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) Ps[(kl + 8 * j) * ROWS_PS + wid * RW + 4 * i + rl] = s[i][j];
        }
        __syncthreads();                                 // K is read; a warp's scores are its own
        fetch(Ks, A.k_pages, at);
        bool full;
        {
            float s[RW];
            float top = -INFINITY;
            int any = 0;
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const int j = j0 + kb + G * i;
                s[i] = -INFINITY;
                if ((j >= lo || j < kept) && j <= p) {
                    s[i] = rows_score(A, Ps[(kb + G * i) * ROWS_PS + row], slope, p, j);
                    any = 1;
                }
                top = fmaxf(top, s[i]);
            }
#pragma unroll
            for (int o = 16; o >= RW; o >>= 1) {
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                any |= __shfl_xor_sync(0xffffffffu, any, o);
            }
            const float m_new = fmaxf(m, top);
            const float alpha = any ? expf(m - m_new) : 1.0f;        // a row without keys in this tile stays as it is
            bool nonzero = true;
            float sum[RW];
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const int j = j0 + kb + G * i;
                const float pj = ((j >= lo || j < kept) && j <= p) ? expf(s[i] - m_new) : 0.f;
                Ps[(kb + G * i) * ROWS_PS + row] = pj;
                nonzero = nonzero && pj != 0.f;
                sum[i] = pj;
            }
#pragma unroll
            for (int o = RW / 2; o > 0; o >>= 1)         // the order of a warp's sum: keys 16 apart, then 8, 4, 2, 1
#pragma unroll
                for (int i = 0; i < o; ++i) sum[i] += sum[i + o];
#pragma unroll
            for (int o = 16; o >= RW; o >>= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
            if (any) { l = fmaf(l, alpha, sum[0]); m = m_new; }
            if (kb == 0) al[row] = alpha;
            full = __all_sync(0xffffffffu, nonzero || !live);        // no weight of the warp's rows is zero
        }
        ROWS_WAIT(1);
        __syncthreads();                                 // V has landed
        {
            float av[VR];
#pragma unroll
            for (int r = 0; r < VR; r += 4) *reinterpret_cast<float4*>(av + r) = *reinterpret_cast<const float4*>(al + rg + r);
#pragma unroll
            for (int r = 0; r < VR; ++r)
#pragma unroll
                for (int c = 0; c < 4 * VC; ++c) acc[r][c] *= av[r];
            const int keys = min(32, last - j0 + 1);
            auto load = [&](int k, float (&pv)[VR], float4 (&v)[VC]) {
#pragma unroll
                for (int r = 0; r < VR; r += 4) *reinterpret_cast<float4*>(pv + r) = *reinterpret_cast<const float4*>(Ps + k * ROWS_PS + rg + r);
#pragma unroll
                for (int c = 0; c < VC; ++c) {
                    const int e = dg + 4 * LC * c;
                    v[c] = e < d ? *reinterpret_cast<const float4*>(Vs + k * ld + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            };
            auto key = [&](const float (&pv)[VR], const float4 (&v)[VC], bool all) {
#pragma unroll
                for (int c = 0; c < VC; ++c)
#pragma unroll
                    for (int r = 0; r < VR; ++r) {
                        if (all || pv[r] != 0.f) {       // a weight of zero (no key, or one far below the maximum) adds nothing,
                            rows_fma2(acc[r][4 * c], acc[r][4 * c + 1], pv[r], v[c].x, v[c].y);      // whatever its value holds
                            rows_fma2(acc[r][4 * c + 2], acc[r][4 * c + 3], pv[r], v[c].z, v[c].w);
                        }
                    }
            };
            float pv[2][VR];
            float4 v[2][VC];
            if (!AHEAD && full && keys == 32) {
#pragma unroll 2
                for (int k = 0; k < 32; ++k) { load(k, pv[0], v[0]); key(pv[0], v[0], true); }
            } else if (full && keys == 32) {
                load(0, pv[0], v[0]);
#pragma unroll
                for (int k = 0; k < 32; k += 2) {
                    load(k + 1, pv[1], v[1]);
                    key(pv[0], v[0], true);
                    if (k + 2 < 32) load(k + 2, pv[0], v[0]);
                    key(pv[1], v[1], true);
                }
            } else {
                for (int k = 0; k < keys; ++k) { load(k, pv[0], v[0]); key(pv[0], v[0], false); }
            }
        }
        __syncthreads();                                 // V and the weights are read
        fetch(Vs, A.v_pages, at);
        j0 = j1;
    }
    ROWS_WAIT(0);
    {
        float alpha = 1.0f;
        if (A.sink && live) {
            const float2 r = tl_attn_sink(m, l, A.sink[head]);
            l = r.x; alpha = r.y;
        }
        float inv = 1.0f / l;
        if (A.gate && live) inv *= 1.0f / (1.0f + expf(-A.gate[(size_t)(t0 + row / g) * A.nq + head]));
        if (kb == 0) { al[row] = alpha; Ps[row] = inv; }
    }
    __syncwarp();                                        // rows rg .. of this lane are its own warp's
#pragma unroll
    for (int r = 0; r < VR; ++r) {
        if (rg + r >= rows) continue;
        const float alpha = al[rg + r], inv = Ps[rg + r];
        float* o = A.out + ((size_t)(t0 + (rg + r) / g) * A.nq + kh * g + (rg + r) % g) * d;
#pragma unroll
        for (int c = 0; c < VC; ++c) {
            const int e = dg + 4 * LC * c;
            if (e >= d) continue;
            float4 v = make_float4(acc[r][4 * c], acc[r][4 * c + 1], acc[r][4 * c + 2], acc[r][4 * c + 3]);
            if (A.sink) { v.x *= alpha; v.y *= alpha; v.z *= alpha; v.w *= alpha; }
            v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
            *reinterpret_cast<float4*>(o + e) = v;
        }
    }
}

// ------------------------------------------------------------------ few tokens
constexpr int DOTS_KEYS = 128, DOTS_HEADS = 8, DOTS_BLOCKS = 32;

// scores[t, h, j] for every key j that token t's heads see: grid (x, KV heads, T), a thread a key.  A block a group of 128 keys; LOOP: no more
// blocks than fill the GPU (DOTS_BLOCKS an SM), each several groups, for tables much longer than the contexts may be (table of 131,072
// positions, 4 tokens at position 10: 16.6 us against 22.7, at 300 23.7 against 28.8, at 1,800 60.0 against 61.1; where the blocks fit
// anyway the loop's code costs: 16 tokens at 1,800, table of 2,048, 95 against 82).
template <bool LOOP>
__global__ void __launch_bounds__(DOTS_KEYS) attn_dots_kernel(const RowsArgs A) {
    extern __shared__ __align__(16) float qs[];          // [heads of the group][d]
    const int t = blockIdx.z, kh = blockIdx.y, g = A.nq / A.nkv, d = A.d;
    const int p = rows_position(A, t), lo = rows_low(A, p), kept = min(A.keep_first, lo);
    int c0 = blockIdx.x * DOTS_KEYS;
    if (c0 > p || (!LOOP && c0 >= kept && c0 + DOTS_KEYS <= lo)) return;
    for (int i = threadIdx.x; i < g * d; i += DOTS_KEYS) qs[i] = A.q[(size_t)t * A.q_stride + (size_t)kh * g * d + i];
    __syncthreads();
    const int* tab = A.table + (size_t)tl_checked(A.req_slot[t], A.L.table_rows, A.L, TL_K_TOKENWISE) * A.max_pages;
    do {
        const int j = c0 + threadIdx.x;
        c0 += gridDim.x * DOTS_KEYS;
        if (!((j >= lo || j < kept) && j <= p)) continue;
        const float* kr = rows_at(A, A.k_pages, tab, j, kh);
        for (int h0 = 0; h0 < g; h0 += DOTS_HEADS) {
            float dot[DOTS_HEADS];
#pragma unroll
            for (int h = 0; h < DOTS_HEADS; ++h) dot[h] = 0.f;
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kr + e);
#pragma unroll
                for (int h = 0; h < DOTS_HEADS; ++h) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + min(h0 + h, g - 1) * d + e);
                    dot[h] = fmaf(q4.x, k4.x, dot[h]);
                    dot[h] = fmaf(q4.y, k4.y, dot[h]);
                    dot[h] = fmaf(q4.z, k4.z, dot[h]);
                    dot[h] = fmaf(q4.w, k4.w, dot[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < DOTS_HEADS; ++h) {
                if (h0 + h >= g) break;
                const int head = kh * g + h0 + h;
                A.scores[((size_t)t * A.nq + head) * A.keys + j] = rows_score(A, dot[h], A.slopes ? A.slopes[head] : 0.f, p, j);
            }
        }
    } while (LOOP && c0 <= p);
}

// grid (slices of 32 columns, KV heads * groups of up to 8 of their query heads, T), a warp a head
constexpr int CHAIN_KEYS = 128, CHAIN_STAGES = 4;
constexpr int CHAIN_SMEM = (CHAIN_STAGES * CHAIN_KEYS * 32 + DOTS_HEADS * CHAIN_KEYS) * (int)sizeof(float);

__global__ void __launch_bounds__(32 * DOTS_HEADS) attn_chain_kernel(const RowsArgs A) {
    extern __shared__ __align__(16) float sm[];
    float (*vs)[CHAIN_KEYS][32] = reinterpret_cast<float (*)[CHAIN_KEYS][32]>(sm);
    float (*ws)[CHAIN_KEYS] = reinterpret_cast<float (*)[CHAIN_KEYS]>(sm + CHAIN_STAGES * CHAIN_KEYS * 32);
    const int t = blockIdx.z, g = A.nq / A.nkv, d = A.d, groups = (g + DOTS_HEADS - 1) / DOTS_HEADS;
    const int kh = blockIdx.y / groups, h0 = (blockIdx.y % groups) * DOTS_HEADS;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    const int p = rows_position(A, t), lo = rows_low(A, p), kept = min(A.keep_first, lo);
    const int e0 = blockIdx.x * 32, e = e0 + lane;
    const bool live = h0 + wid < g;
    const int head = kh * g + min(h0 + wid, g - 1);
    const int* tab = A.table + (size_t)tl_checked(A.req_slot[t], A.L.table_rows, A.L, TL_K_TOKENWISE) * A.max_pages;
    const float* sr = A.scores + ((size_t)t * A.nq + head) * A.keys;
    // groups of 128 keys; those wholly between the kept first keys and the window are left out
    auto next = [&](int c) { return (c >= kept && c + CHAIN_KEYS <= lo) ? (lo / CHAIN_KEYS) * CHAIN_KEYS : c; };
    auto valid = [&](int j) { return (j >= lo || j < kept) && j <= p; };
    auto fetch = [&](int c, int stage) {
        if (c <= p) {
            for (int i = tid; i < CHAIN_KEYS * 8; i += nt) {
                const int j = c + (i >> 3), x = (i & 7) * 4;
                if (valid(j) && e0 + x < d) rows_copy16(&vs[stage][i >> 3][x], rows_at(A, A.v_pages, tab, j, kh) + e0 + x);
            }
        }
        ROWS_COMMIT();
    };
    auto load = [&](int c, float (&s)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = c + 32 * i + lane;
            s[i] = valid(j) ? sr[j] : -INFINITY;
        }
    };
    float m = -INFINITY, l = 0.f, acc = 0.f;
    int c = next(0), ahead = c;
    for (int i = 0; i < CHAIN_STAGES - 1; ++i) { fetch(ahead, i); ahead = next(ahead + CHAIN_KEYS); }
    float s[4];
    load(c, s);
    for (int step = 0; c <= p; ++step) {
        const int after = next(c + CHAIN_KEYS);
        fetch(ahead, (step + CHAIN_STAGES - 1) % CHAIN_STAGES);
        ahead = next(ahead + CHAIN_KEYS);
        float top[4], w[4], sum[4], alpha[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) top[i] = warp_max(s[i]);
        unsigned any = 0;                                // tiles with a key; the others leave everything as it is
        bool full = true;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool here = __any_sync(0xffffffffu, valid(c + 32 * i + lane));
            if (here) any |= 1u << i;
            const float m_new = here ? fmaxf(m, top[i]) : m;
            alpha[i] = here ? expf(m - m_new) : 1.0f;
            w[i] = valid(c + 32 * i + lane) ? expf(s[i] - m_new) : 0.f;
            m = m_new;
            full = full && w[i] != 0.f;
        }
        full = __all_sync(0xffffffffu, full);
#pragma unroll
        for (int i = 0; i < 4; ++i) { sum[i] = warp_sum(w[i]); ws[wid][32 * i + lane] = w[i]; }
#pragma unroll
        for (int i = 0; i < 4; ++i) if ((any >> i) & 1u) l = fmaf(l, alpha[i], sum[i]);
        if (after <= p) load(after, s);
        ROWS_WAIT(CHAIN_STAGES - 1);
        __syncthreads();                                 // the step's values have landed
        const float (*vt)[32] = vs[step % CHAIN_STAGES];
        if (full) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc *= alpha[i];
#pragma unroll
                for (int k = 32 * i; k < 32 * i + 32; k += 4) {
                    const float4 w4 = *reinterpret_cast<const float4*>(&ws[wid][k]);
                    acc = fmaf(w4.x, vt[k][lane], acc);
                    acc = fmaf(w4.y, vt[k + 1][lane], acc);
                    acc = fmaf(w4.z, vt[k + 2][lane], acc);
                    acc = fmaf(w4.w, vt[k + 3][lane], acc);
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc *= alpha[i];
                for (int k = 32 * i; k < 32 * i + 32; ++k) {
                    const float wk = ws[wid][k];
                    if (wk != 0.f) acc = fmaf(wk, vt[k][lane], acc);
                }
            }
        }
        __syncthreads();                                 // the stage and the weights are read
        c = after;
    }
    ROWS_WAIT(0);
    if (A.sink) {
        const float2 r = tl_attn_sink(m, l, A.sink[head]);
        l = r.x;
        acc *= r.y;
    }
    float inv = 1.0f / l;
    if (A.gate) inv *= 1.0f / (1.0f + expf(-A.gate[(size_t)t * A.nq + head]));
    if (live && e < d) A.out[((size_t)t * A.nq + head) * d + e] = acc * inv;
}

template <int NC, int ROWS, int RW>
static int launch_rows(RowsArgs A, cudaStream_t stream) {
    constexpr auto bytes = [](int d) { return ((ROWS + 64) * (d + 4) + 32 * (ROWS + 4) + ROWS) * (int)sizeof(float); };
    static bool raised[TL_MAX_DEVICES] = {};
    const int e = tl_raise_smem(attn_rows_kernel<NC, ROWS, RW>, raised, bytes(64 * NC));
    if (e) return e;
    const int g = A.nq / A.nkv;
    A.tq = ROWS / g < 32 ? ROWS / g : 32;
    const dim3 grid((A.T + A.tq - 1) / A.tq, A.nkv, A.tq < A.T ? A.tq : A.T);
    attn_rows_kernel<NC, ROWS, RW><<<grid, ROWS / RW * 32, bytes(A.d), stream>>>(A);
    return tl_launch_status();
}

// `scores` (float [T, nq, keys], keys >= every position of the step + 1, or null): scratch of the two kernels of few tokens.
// Returns 1 for shapes that these kernels do not take; the caller gives those to the token-wise kernel beforehand.
TL_EXPORT int tl_attn_rows(const float* q, int q_stride, float* out, const float* k_pages, const float* v_pages, const int* table,
                           int max_pages, int page_size, const int* pos, const int* req_slot, int T, int nq, int nkv, int d, int window,
                           float scale, const float* sink, int keep_first, const float* gate, int chunk, const float* slopes, float cap,
                           float* scores, int keys, int table_rows, int total_pages, int* fault, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (nq % nkv || (chunk > 0 && window > 0) || chunk < 0 || d < 4 || d % 4 || d > 256 ||
        ((((uintptr_t)k_pages) | ((uintptr_t)v_pages) | ((uintptr_t)out)) & 15)) return 1;
    const int g = nq / nkv;
    static bool rc[TL_MAX_DEVICES] = {};
    int e = tl_raise_smem(attn_chain_kernel, rc, CHAIN_SMEM);
    if (e) return e;
    RowsArgs A{q, q_stride, out, k_pages, v_pages, table, max_pages, page_size, pos, req_slot, T, nq, nkv, d, window, scale,
               sink, window > 0 ? keep_first : 0, gate, chunk, slopes, cap, scores, keys, 0, TlLimits{table_rows, total_pages, fault}};
    if (scores) {
        const int groups = (g + DOTS_HEADS - 1) / DOTS_HEADS;
        const size_t smem = (size_t)g * d * sizeof(float);
        if (smem > 48 * 1024 || nkv > 65535 || T > 65535 || nkv * groups > 65535) return 1;
        const long long most = (long long)DOTS_BLOCKS * tl_num_sms() / ((long long)nkv * T), tiles = (keys + DOTS_KEYS - 1) / DOTS_KEYS;
        if (tiles > most && most > 0) attn_dots_kernel<true><<<dim3((unsigned)most, nkv, T), DOTS_KEYS, smem, stream>>>(A);
        else attn_dots_kernel<false><<<dim3((unsigned)tiles, nkv, T), DOTS_KEYS, smem, stream>>>(A);
        if ((e = tl_launch_status())) return e;
        attn_chain_kernel<<<dim3((d + 31) / 32, nkv * groups, T), 32 * (g < DOTS_HEADS ? g : DOTS_HEADS), CHAIN_SMEM, stream>>>(A);
        return tl_launch_status();
    }
    if (g > ROWS_MAX || nkv > 65535) return 1;
    // Blocks of 64 rows, 16 a warp, where they are three an SM or more (2,048 tokens, 28 heads: 1,294 us against 1,430); else of 32
    // rows, 8 a warp: more of them, and a warp is done with a tile sooner (333 tokens on 700 cached: 254 us against 336; 100 on 300:
    // 158 against 293; 700 tokens, 40 heads, three an SM: 300 both).
    // A block has at most 32 tokens: with one query head a KV head 64 rows would be half empty (32 heads of 64, 2,048 tokens: 1,548 us in such blocks, 834 in
    // those of 32; of 128 2,445 and 1,455).
    const int tokens = ROWS_MAX / g < 32 ? ROWS_MAX / g : 32;
    const bool wide = g > ROWS_MAX / 2 || (g > 1 && (long long)((T + tokens - 1) / tokens) * nkv >= 3LL * tl_num_sms());
#define ROWS_GO(NC) (wide ? launch_rows<NC, ROWS_MAX, 16>(A, stream) : launch_rows<NC, ROWS_MAX / 2, 8>(A, stream))
    return d <= 64 ? ROWS_GO(1) : d <= 128 ? ROWS_GO(2) : ROWS_GO(4);
#undef ROWS_GO
}
