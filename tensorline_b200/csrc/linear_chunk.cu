// The recurrences of recurrent.cu with one decay a head (fixed, or gated with a normaliser) for steps of many tokens: chunks of a
// request's tokens side by side, their sums as matrix products.
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T,  o_t = S_t^T q_t  (gated: divided by max(|n_t . q_t|, exp(-m_t)) + den_eps)
//
// With F_t the sum of the log decays of a chunk up to t and i_s the log input gate (0 for a fixed decay), a token's weight in the
// state after t is exp(F_t - F_s + i_s - m_t), and of the chunk's start state S exp(F_t + m_start - m_t): nothing but the
// running maximum m (0 for a fixed decay) passes from token to token.
//   rotate   retention: q and k rotated and scaled, once for all that read them
//   local    every chunk: its end state from zero, K^T (w V) [d, dv], against a maximum of its own
//   carry    per state element, chunk after chunk: the chunk's start state takes the place of its end state; the slot's new state
//   outputs  every chunk: P = (Q K^T) * weights, then [P | w Q] [V ; S] in one product
// F and the maxima are sums and maxima in double (64 tokens a chunk and head: a warp's work), every weight the float exponential
// of one difference of doubles; the products have a float's accuracy.  The state in the slots has the layout of the scan
// kernel, so the two may take turns on one request.  A position's sums depend on where its step began, to rounding.
//
// What the scan kernel is bound by is the chain over the tokens at one block a head and 16 columns (128 blocks, 0.36 us a token);
// here everything but the carry is products of bfloat16 parts on the tensor cores.
// Measured, 2,048 tokens, 8 heads of 128 x 256: gated 728 us token by token; now gates 4.6, local 30, carry 24, outputs 64 us
// (81 as float multiply-adds).  Fixed decay, 1,650 tokens in 3 requests: local 23, carry 18, outputs 44 us (70 as multiply-adds).
// 64 tokens a chunk: P costs as much as the two products with the state at 128 tokens, and the start states, which pass through
// L2 once each way, weigh half as much again at 32.
#include "umma.cuh"
#include "parts_mma.cuh"

constexpr int LC_C = 64;                 // tokens a chunk
constexpr int LC_WIDE = 128;             // tokens a chunk where a head's 33 to 128 rows fill the 5th-generation tensor cores' tiles
constexpr int LC_COLS = 16;              // columns a slice of the state's layout (the scan kernel's)

struct LinearChunkArgs {
    const float* q; const float* k; int qk_stride;           // element (t, h, e) at t * stride + h * d + e
    const float* v; int v_stride;
    const float* gates; float cap; const float* decay;       // gated: [T, 2H] pre-activations; else decay [H]
    float q_scale, k_scale;
    float* state; long long slot_stride;
    const int* q_start; const int* slots;
    const int4* chunks;                  // (request, number of the chunk, the request's chunks, first chunk of the request in the list)
    const int* firsts;                   // the requests' first chunks
    float* ends;                         // [chunks][H][d dv (+ d)]: end states from zero, then start states
    double* marks;                       // [chunks][H][3]: the chunk's F, its maximum, the running maximum in front of it
    double* weights;                     // gated: [chunks][H][3][64], F, u and top of lc_weights
    int* marked; int tiles;              // [chunks][H][tiles]: operands that the scan kernel has to take (common.cuh)
    float* out;
    int H, d, dv, nz; float den_eps;
    int* status;
};

__device__ __forceinline__ float lc_log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// A warp, gated: for the n tokens of a chunk of C that starts at row t0, F[t] (the log decays' sum up to t), u[t] = i_t - F[t] and the
// running maximum top[t] of u.
template <int C>
__device__ __forceinline__ void lc_weights(const LinearChunkArgs& A, int t0, int n, int h, int lane, double* F, double* u, double* top) {
    constexpr int N = C / 32;                            // tokens a lane
    double f[N], w[N], best = -INFINITY, sum = 0.0;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        const int t = N * lane + e;
        f[e] = 0.0; w[e] = -INFINITY;
        if (t < n) {
            const float* g = A.gates + (size_t)(t0 + t) * 2 * A.H;
            w[e] = A.cap * tanhf(g[h] / A.cap);
            f[e] = lc_log_sigmoid(A.cap * tanhf(g[A.H + h] / A.cap));
        }
        sum += f[e];
    }
    const double mine = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += x;
    }
    double at = sum - mine;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        at += f[e];
        f[e] = at;
        w[e] -= at;
        best = fmax(best, w[e]);
    }
    double before = best;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before = fmax(before, x);
    }
    before = __shfl_up_sync(0xffffffffu, before, 1);
    if (lane == 0) before = -INFINITY;
#pragma unroll
    for (int e = 0; e < N; ++e) {
        before = fmax(before, w[e]);
        F[N * lane + e] = f[e]; u[N * lane + e] = w[e]; top[N * lane + e] = before;
    }
}

// A warp a (chunk, head): the gated kinds' weights, once for all blocks that need them (worked out in each of them, warp 0 held the
// others up: end states 36 us, 33.5 without and 4.6 here, and the outputs need them without a wait).
template <int C>
__global__ void __launch_bounds__(32) lc_gates_kernel(const LinearChunkArgs A) {
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, lane = threadIdx.x, t0 = A.q_start[ck.x] + ck.y * C, n = min(C, A.q_start[ck.x + 1] - t0);
    const size_t at = (size_t)blockIdx.x * A.H + h;
    double* w = A.weights + at * 3 * C;
    lc_weights<C>(A, t0, n, h, lane, w, w + C, w + 2 * C);
    __syncwarp();
    if (lane == 0) {
        const double end = w[n - 1];
        A.marks[at * 3] = end;
        A.marks[at * 3 + 1] = (double)(float)(end + w[2 * C + n - 1]);
    }
}

// ------------------------------------------------------------------ rotation
// rows [T][2 H d]: q rotated and scaled, k rotated and scaled; a block a token.  VEC: four floats at a time, the first ones on their way
// before the angles are known (8 heads of 128, 1,650 tokens: 7.5 us, a float at a time 11); rotations that don't cut a head into
// whole 16-byte pieces stay with the latter.
template <bool VEC>
__global__ void __launch_bounds__(256) lc_rotate_kernel(const float* __restrict__ proj, int stride, int q_off, int k_off, const float* __restrict__ inv_freq,
                                                        int rot, int interleaved, const int* __restrict__ pos, float q_scale, float k_scale,
                                                        float* __restrict__ rows, int H, int d) {
    extern __shared__ __align__(16) float cs[];          // cos [rot / 2], sin [rot / 2]
    const int t = blockIdx.x, half = rot >> 1, tid = threadIdx.x, rest = d - rot;
    const float* row = proj + (size_t)t * stride;
    float* to = rows + (size_t)t * 2 * H * d;
    auto angles = [&]() {
        for (int i = tid; i < half; i += 256) sincosf(__fmul_rn((float)pos[t], inv_freq[i]), &cs[half + i], &cs[i]);
        __syncthreads();
    };
    if constexpr (VEC) {
        const int per = interleaved ? rot / 4 : half / 4, units = 2 * H * per;      // a unit: four pairs, interleaved two
        auto place = [&](int i, bool& isk, int& e) {     // the unit's first element, its place among the angles
            isk = i >= H * per;
            const int j = isk ? i - H * per : i, h = j / per, p = (j - h * per) * 4;
            e = h * d + p;
            return p;
        };
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
        auto fetch = [&](int i) {
            bool isk; int e;
            if (i >= units) return;
            place(i, isk, e);
            const float* from = row + (isk ? k_off : q_off) + e;
            x = *reinterpret_cast<const float4*>(from);
            if (!interleaved) y = *reinterpret_cast<const float4*>(from + half);
        };
        fetch(tid);
        angles();
        for (int i = tid; i < units; i += 256) {
            bool isk; int e;
            const int p = place(i, isk, e);
            const float4 a = x, b = y;
            fetch(i + 256);
            const float sc = isk ? k_scale : q_scale;
            float* out = to + (isk ? H * d : 0) + e;
            auto first = [&](float u, float v, float c, float s) { return (__fmul_rn(u, c) - __fmul_rn(v, s)) * sc; };
            auto second = [&](float u, float v, float c, float s) { return (__fmul_rn(v, c) + __fmul_rn(u, s)) * sc; };
            if (interleaved) {
                const float c0 = cs[p / 2], c1 = cs[p / 2 + 1], s0 = cs[half + p / 2], s1 = cs[half + p / 2 + 1];
                *reinterpret_cast<float4*>(out) = make_float4(first(a.x, a.y, c0, s0), second(a.x, a.y, c0, s0), first(a.z, a.w, c1, s1), second(a.z, a.w, c1, s1));
            } else {
                const float4 c = *reinterpret_cast<const float4*>(cs + p), s = *reinterpret_cast<const float4*>(cs + half + p);
                *reinterpret_cast<float4*>(out) = make_float4(first(a.x, b.x, c.x, s.x), first(a.y, b.y, c.y, s.y), first(a.z, b.z, c.z, s.z), first(a.w, b.w, c.w, s.w));
                *reinterpret_cast<float4*>(out + half) = make_float4(second(a.x, b.x, c.x, s.x), second(a.y, b.y, c.y, s.y), second(a.z, b.z, c.z, s.z), second(a.w, b.w, c.w, s.w));
            }
        }
        for (int i = tid; i < 2 * H * rest / 4; i += 256) {
            const bool isk = i >= H * rest / 4;
            const int j = (isk ? i - H * rest / 4 : i) * 4, e = (j / rest) * d + rot + j % rest;
            const float sc = isk ? k_scale : q_scale;
            float4 v = *reinterpret_cast<const float4*>(row + (isk ? k_off : q_off) + e);
            v.x *= sc; v.y *= sc; v.z *= sc; v.w *= sc;
            *reinterpret_cast<float4*>(to + (isk ? H * d : 0) + e) = v;
        }
    } else {
        angles();
        const int pairs = H * half;
        for (int i = tid; i < 2 * pairs; i += 256) {
            const bool isk = i >= pairs;
            const int j = isk ? i - pairs : i, h = j / half, p = j - h * half;
            const int e1 = h * d + (interleaved ? 2 * p : p), e2 = h * d + (interleaved ? 2 * p + 1 : p + half);
            const float* x = row + (isk ? k_off : q_off);
            float* y = to + (isk ? H * d : 0);
            const float sc = isk ? k_scale : q_scale, x1 = x[e1], x2 = x[e2], c = cs[p], s = cs[half + p];
            y[e1] = (__fmul_rn(x1, c) - __fmul_rn(x2, s)) * sc;
            y[e2] = (__fmul_rn(x2, c) + __fmul_rn(x1, s)) * sc;
        }
        for (int i = tid; i < 2 * H * rest; i += 256) {
            const bool isk = i >= H * rest;
            const int j = isk ? i - H * rest : i, e = (j / rest) * d + rot + j % rest;
            to[(isk ? H * d : 0) + e] = row[(isk ? k_off : q_off) + e] * (isk ? k_scale : q_scale);
        }
    }
}

// ------------------------------------------------------------------ end states from zero
// grid (chunks, H, tiles of RB rows and CB columns); 256 threads: two warps along the rows, four along the columns.  The block's K (weighted)
// and V are cut into parts once; a chunk's 64 tokens are four steps of the tensor cores, so the five small products go first and
// the leading one on top of them in the same accumulator: as exact as one of its own, and half the registers, which leaves
// two blocks an SM.  8 heads of 128 x 256, 2,048 tokens, gated: 30 us, as float multiply-adds (tiles of 8 x 8 a thread, bound by the
// floats they take from shared memory) 33.5; fixed decay, 1,650 tokens: 23.3 against 25.9.
template <int RB, int CB> struct LocalShape {
    static constexpr int RK = RB * 2 + 16, RV = CB * 2 + 16;        // bytes of a row of a part of K, of V
    static constexpr int K = 3 * LC_C * RK, BYTES = K + 3 * LC_C * RV;
};

template <int RB, int CB, bool GATED>
__global__ void __launch_bounds__(256, 2) lc_local_kernel(const LinearChunkArgs A) {
    using Sh = LocalShape<RB, CB>;
    constexpr int RK = Sh::RK, RV = Sh::RV, MT = RB / 32, NJ = CB / 32, KPER = LC_C * RB / 4 / 256, VPER = LC_C * CB / 4 / 256;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float w[LC_C];
    const uint32_t kb = (uint32_t)__cvta_generic_to_shared(smem), vb = kb + Sh::K;
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, col_tiles = (A.dv + CB - 1) / CB, row0 = (blockIdx.z / col_tiles) * RB, col0 = (blockIdx.z % col_tiles) * CB;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = A.q_start[ck.x] + ck.y * LC_C, n = min(LC_C, A.q_start[ck.x + 1] - t0);
    float4 x[KPER], y[VPER];
#pragma unroll
    for (int i = 0; i < KPER; ++i) {
        const int t = (tid + 256 * i) / (RB / 4), e = ((tid + 256 * i) % (RB / 4)) * 4;
        x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n && row0 + e < A.d) x[i] = *reinterpret_cast<const float4*>(A.k + (size_t)(t0 + t) * A.qk_stride + h * A.d + row0 + e);
    }
#pragma unroll
    for (int i = 0; i < VPER; ++i) {
        const int t = (tid + 256 * i) / (CB / 4), c = ((tid + 256 * i) % (CB / 4)) * 4;
        y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n && col0 + c < A.dv) y[i] = *reinterpret_cast<const float4*>(A.v + (size_t)(t0 + t) * A.v_stride + h * A.dv + col0 + c);
    }
    const size_t ch = (size_t)blockIdx.x * A.H + h;
    if (GATED) {
        const double* g = A.weights + ch * 3 * LC_C;
        if (tid < LC_C) w[tid] = tid < n ? (float)exp(A.marks[ch * 3] + g[LC_C + tid] - A.marks[ch * 3 + 1]) * A.k_scale : 0.f;
    } else if (tid < LC_C) {
        const double la = log((double)A.decay[h]);
        w[tid] = tid < n ? (float)exp((n - 1 - tid) * la) * A.k_scale : 0.f;
        if (tid == 0 && blockIdx.z == 0) { A.marks[ch * 3] = n * la; A.marks[ch * 3 + 1] = 0.0; }
    }
    bool odd = tid < LC_C && w[tid] != w[tid];           // a gate that is no number
#pragma unroll
    for (int i = 0; i < KPER; ++i) odd = odd || tl_chunk_odd(x[i].x) || tl_chunk_odd(x[i].y) || tl_chunk_odd(x[i].z) || tl_chunk_odd(x[i].w);
#pragma unroll
    for (int i = 0; i < VPER; ++i) odd = odd || tl_chunk_odd(y[i].x) || tl_chunk_odd(y[i].y) || tl_chunk_odd(y[i].z) || tl_chunk_odd(y[i].w);
    auto put4 = [&](unsigned char* to, int part, const float4 z) {      // four values' parts, `part` bytes from one part to the next
        uint2 p[3];
        parts_cut(z.x, z.y, p[0].x, p[1].x, p[2].x);
        parts_cut(z.z, z.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(to + e * part) = p[e];
    };
#pragma unroll
    for (int i = 0; i < VPER; ++i)
        put4(smem + Sh::K + (tid + 256 * i) / (CB / 4) * RV + ((tid + 256 * i) % (CB / 4)) * 8, LC_C * RV, y[i]);
    odd = __syncthreads_or(odd);
    if (tid == 0) A.marked[ch * A.tiles + blockIdx.z] = odd;
#pragma unroll
    for (int i = 0; i < KPER; ++i) {
        const int t = (tid + 256 * i) / (RB / 4);
        const float wt = w[t];
        put4(smem + t * RK + ((tid + 256 * i) % (RB / 4)) * 8, LC_C * RK, make_float4(x[i].x * wt, x[i].y * wt, x[i].z * wt, x[i].w * wt));
    }
    __syncthreads();
    const int wm = wid >> 2, wn = wid & 3, steps = (n + 15) / 16;       // RB / 2 rows and CB / 4 columns a warp
    // K transposed: tokens (lane & 7) and 8 further from lane 16 on, rows 8 further in every other group; V as in the outputs
    const uint32_t k_at = kb + ((lane & 7) + (lane >> 4) * 8) * RK + ((lane >> 3) & 1) * 16 + wm * RB;
    const uint32_t v_at = vb + ((lane & 7) + ((lane >> 3) & 1) * 8) * RV + (lane >> 4) * 16 + wn * (CB / 2);
    float acc[MT][NJ][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    for (int s = 0; s < steps; ++s) {                    // the small products
        uint32_t b[NJ / 2][3][4];
#pragma unroll
        for (int j = 0; j < NJ / 2; ++j)
#pragma unroll
            for (int p = 0; p < 3; ++p) parts_load4_trans(b[j][p], v_at + (p * LC_C + 16 * s) * RV + j * 32);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            uint32_t a[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) parts_load4_trans(a[p], k_at + (p * LC_C + 16 * s) * RK + i * 32);
#pragma unroll
            for (int p = 0; p < 5; ++p) {                // (lo, hi), (hi, lo), (mid, mid), (mid, hi), (hi, mid)
                const int pa = p == 0 ? 2 : p == 2 || p == 3 ? 1 : 0, pb = p == 1 ? 2 : p == 2 || p == 4 ? 1 : 0;
#pragma unroll
                for (int j = 0; j < NJ; ++j) parts_mma(acc[i][j], a[pa], b[j / 2][pb][(j & 1) * 2], b[j / 2][pb][(j & 1) * 2 + 1]);
            }
        }
    }
    for (int s = 0; s < steps; ++s) {                    // the leading one
        uint32_t b[NJ / 2][4];
#pragma unroll
        for (int j = 0; j < NJ / 2; ++j) parts_load4_trans(b[j], v_at + 16 * s * RV + j * 32);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            uint32_t a[4];
            parts_load4_trans(a, k_at + 16 * s * RK + i * 32);
#pragma unroll
            for (int j = 0; j < NJ; ++j) parts_mma_add(acc[i][j], a, b[j / 2][(j & 1) * 2], b[j / 2][(j & 1) * 2 + 1]);
        }
    }
    const size_t per = (size_t)A.d * A.dv + (GATED ? A.d : 0);
    float* to = A.ends + ch * per;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = row0 + wm * (RB / 2) + 16 * i + 8 * e + (lane >> 2);
            if (row >= A.d) continue;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int col = col0 + wn * (CB / 4) + 8 * j + (lane & 3) * 2;
                if (col < A.dv) *reinterpret_cast<float2*>(to + (size_t)row * A.dv + col) = make_float2(acc[i][j][2 * e], acc[i][j][2 * e + 1]);
            }
        }
    if (GATED && col0 == 0 && tid < RB && row0 + tid < A.d) {        // the normaliser: the same with v = 1
        float s[8] = {};                                 // eight chains of eight tokens
#pragma unroll
        for (int t = 0; t < LC_C; ++t) {
            const unsigned char* k = smem + t * RK + tid * 2;
            auto part = [&](int p) { return __bfloat162float(*reinterpret_cast<const bf16*>(k + p * LC_C * RK)); };
            s[t & 7] += part(0) + (part(1) + part(2));
        }
        to[(size_t)A.d * A.dv + row0 + tid] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
    }
}

// ------------------------------------------------------------------ carry
// grid (groups of 4 state elements / 256, H, requests)
constexpr int LC_CARRY = 64;             // chunks whose factors a block holds at a time

template <int R, int IS, bool GATED>
__global__ void __launch_bounds__(256) lc_carry_kernel(const LinearChunkArgs A) {
    constexpr int NT = (IS * (LC_COLS + (GATED ? 1 : 0)) + 31) / 32 * 32, PB = R * NT + (GATED ? 4 : 0);
    __shared__ double mk[LC_CARRY][2];
    __shared__ double ms[LC_CARRY + 1];
    __shared__ float keep[LC_CARRY], gain[LC_CARRY];
    const int first = A.firsts[blockIdx.z], h = blockIdx.y, tid = threadIdx.x;
    const int4 ck = A.chunks[first];
    const size_t per = (size_t)A.d * A.dv + (GATED ? A.d : 0);
    const size_t i4 = ((size_t)blockIdx.x * 256 + tid) * 4;
    float* slot = A.state + (size_t)A.slots[ck.x] * A.slot_stride + (size_t)h * A.nz * PB;
    const bool mine = i4 < per, norm = GATED && i4 >= (size_t)A.d * A.dv;
    const int row = norm ? (int)(i4 - (size_t)A.d * A.dv) : (int)(i4 / A.dv), col = norm ? 0 : (int)(i4 % A.dv);
    // element c of the four: four columns of a row, or four rows of the normaliser (which every slice of the slot holds)
    auto at = [&](int c, int z) {
        const int r = norm ? row + c : row, j = norm ? LC_COLS : (col + c) % LC_COLS, zz = norm ? z : (col + c) / LC_COLS;
        return (size_t)zz * PB + (size_t)(r % R) * NT + j * IS + r / R;
    };
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mine) S = make_float4(slot[at(0, 0)], slot[at(1, 0)], slot[at(2, 0)], slot[at(3, 0)]);
    double m = GATED ? (double)slot[R * NT] : 0.0;
    if (tl_chunk_marked(A.marked, A.tiles, first, ck.z, h, A.H)) return;      // the scan kernel's, outputs as well
    float* e = A.ends + ((size_t)first * A.H + h) * per + i4;
    const size_t step = (size_t)A.H * per;
    for (int c0 = 0; c0 < ck.z; c0 += LC_CARRY) {
        const int nc = min(LC_CARRY, ck.z - c0);
        __syncthreads();
        for (int c = tid; c < nc; c += 256) {
            const double* g = A.marks + ((size_t)(first + c0 + c) * A.H + h) * 3;
            mk[c][0] = g[0]; mk[c][1] = g[1];
        }
        __syncthreads();
        if (tid == 0) {
            double x = m;
            for (int c = 0; c < nc; ++c) {
                ms[c] = x;
                if (GATED) x = (double)(float)fmax(mk[c][0] + x, mk[c][1]);      // a maximum that a float holds: the slot keeps it
            }
            ms[nc] = x;
        }
        __syncthreads();
        for (int c = tid; c < nc; c += 256) {
            keep[c] = (float)exp(mk[c][0] + ms[c] - ms[c + 1]);
            gain[c] = (float)exp(mk[c][1] - ms[c + 1]);
            if (blockIdx.x == 0) A.marks[((size_t)(first + c0 + c) * A.H + h) * 3 + 2] = ms[c];
        }
        __syncthreads();
        m = ms[nc];
        if (mine) {
            float4 next[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) if (x < nc) next[x] = *reinterpret_cast<const float4*>(e + (size_t)x * step);
            for (int c = 0; c < nc; c += 4) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    if (c + x < nc) {
                        const float4 E = next[x];
                        if (c + x + 4 < nc) next[x] = *reinterpret_cast<const float4*>(e + (size_t)(c + x + 4) * step);
                        *reinterpret_cast<float4*>(e + (size_t)(c + x) * step) = S;
                        const float a = keep[c + x], b = gain[c + x];
                        S.x = fmaf(a, S.x, b * E.x); S.y = fmaf(a, S.y, b * E.y); S.z = fmaf(a, S.z, b * E.z); S.w = fmaf(a, S.w, b * E.w);
                    }
                }
            }
        }
        e += (size_t)nc * step;
    }
    if (mine) {
        for (int z = 0; z < (norm ? A.nz : 1); ++z) { slot[at(0, z)] = S.x; slot[at(1, z)] = S.y; slot[at(2, z)] = S.z; slot[at(3, z)] = S.w; }
    }
}
// The running maximum into every slice of the slot, by the outputs' block of the request's last chunk: all blocks of the carry have read
// the old one by then (a kernel of its own took 3 to 4 us).
template <int DP>
__device__ __forceinline__ void lc_maximum(const LinearChunkArgs& A, const int4 ck, int h) {
    constexpr int R = DP == 32 ? 4 : 8, IS = DP / R, NT = (IS * (LC_COLS + 1) + 31) / 32 * 32, PB = R * NT + 4;
    if (blockIdx.z || ck.y != ck.z - 1 || tl_chunk_marked(A.marked, A.tiles, ck.w, ck.z, h, A.H)) return;
    const double* g = A.marks + ((size_t)blockIdx.x * A.H + h) * 3;
    const float m = (float)fmax(g[0] + g[2], g[1]);
    float* slot = A.state + (size_t)A.slots[ck.x] * A.slot_stride + (size_t)h * A.nz * PB;
    for (int z = threadIdx.x; z < A.nz; z += blockDim.x) slot[(size_t)z * PB + R * NT] = m;
}

// ------------------------------------------------------------------ outputs
// grid (chunks, H, slices of CB columns); DP: rows a head, padded.  256 threads; a block cuts its Q and K (32 tokens at a time) into
// parts once, P where it is made, and the rows of [S ; V] as they come, 16 at a time, the next ones on their way in registers: little
// enough shared memory for two blocks an SM, one of which computes while the other waits for its rows (gated, 8 heads
// of 128 x 256, 2,048 tokens: 64 us; with all of K and 32 rows at a time, one block an SM, 83; multiply-adds 81).  Heads of 256
// need 178 KB, one block an SM (4 heads of 256 x 256, 1,024 tokens: 34 us; as multiply-adds 43, and in single chains of 320 their outputs were
// 4.9e-7 off the recurrence in 64 bits where the token-by-token kernel is 1.8e-7 off; now 1.4e-7).  Q S is taken first and weighted by token, P V added to it.
template <int DP, int CB> struct OutShape {
    static constexpr int RQ = DP * 2 + 16, RB = CB * 2 + 16, RP = LC_C * 2 + 16;       // bytes of a row of a part of Q and K, of [S ; V], of P
    static constexpr int Q = 3 * LC_C * RQ, STAGE = 3 * 16 * RB, KB = Q / 2 > 2 * STAGE ? Q / 2 : 2 * STAGE, P = 3 * LC_C * RP;
    static constexpr int BYTES = Q + KB + P;             // K's parts lie where the stages of [S ; V] come later
};

template <int DP, int CB, bool GATED>
__global__ void __launch_bounds__(256, DP <= 128 ? 2 : 1) lc_out_kernel(const LinearChunkArgs A) {
    using Sh = OutShape<DP, CB>;
    constexpr int RQ = Sh::RQ, RB = Sh::RB, RP = Sh::RP, NJ = CB / 32, PER = 16 * CB / 4 / 256;      // n8 tiles a warp, 16-byte loads of a thread a step
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem), kb = base + Sh::Q, pb = kb + Sh::KB;
    constexpr int LPT = DP / 4 < 32 ? DP / 4 : 32;       // lanes of a warp that share a token's q
    __shared__ double u[LC_C], top[LC_C], nq[DP / 4 / LPT][LC_C], rowsum[2][LC_C];
    __shared__ float coef[LC_C], den[LC_C];
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, col0 = blockIdx.z * CB, d = A.d;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
    const int t0 = A.q_start[ck.x] + ck.y * LC_C, n = min(LC_C, A.q_start[ck.x + 1] - t0);
    if (GATED) lc_maximum<DP>(A, ck, h);
    const size_t per = (size_t)d * A.dv + (GATED ? d : 0);
    const float* start = A.ends + ((size_t)blockIdx.x * A.H + h) * per;
    const double m0 = GATED ? A.marks[((size_t)blockIdx.x * A.H + h) * 3 + 2] : 0.0;
    const int s_steps = (d + 15) / 16, steps = s_steps + (n + 15) / 16;
    float4 ahead[PER];
    auto fetch = [&](int step) {                         // 16 rows of S, then of V; zeros where there are none
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = (tid + 256 * i) / (CB / 4), c = col0 + ((tid + 256 * i) % (CB / 4)) * 4;
            ahead[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c >= A.dv) continue;
            if (step < s_steps) {
                if (step * 16 + r < d) ahead[i] = *reinterpret_cast<const float4*>(start + (size_t)(step * 16 + r) * A.dv + c);
            } else if ((step - s_steps) * 16 + r < n)
                ahead[i] = *reinterpret_cast<const float4*>(A.v + (size_t)(t0 + (step - s_steps) * 16 + r) * A.v_stride + h * A.dv + c);
        }
    };
    auto put4 = [&](unsigned char* to, int part, const float4 x) {      // four values' parts, `part` bytes from one part to the next
        uint2 p[3];
        parts_cut(x.x, x.y, p[0].x, p[1].x, p[2].x);
        parts_cut(x.z, x.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(to + e * part) = p[e];
    };
    auto put = [&](int step) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int r = (tid + 256 * i) / (CB / 4), c = ((tid + 256 * i) % (CB / 4)) * 4;
            put4(smem + Sh::Q + (step & 1) * Sh::STAGE + r * RB + c * 2, 16 * RB, ahead[i]);
        }
    };
#pragma unroll
    for (int i = tid; i < LC_C * DP / 4; i += 256) {
        const int t = i / (DP / 4), e = (i % (DP / 4)) * 4;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        double r = 0.0;                                  // n . q of the chunk's start state
        if (t < n && e < d) {
            q = *reinterpret_cast<const float4*>(A.q + (size_t)(t0 + t) * A.qk_stride + h * d + e);
            q.x *= A.q_scale; q.y *= A.q_scale; q.z *= A.q_scale; q.w *= A.q_scale;
            if (GATED) {
                const float4 x = *reinterpret_cast<const float4*>(start + (size_t)d * A.dv + e);
                r = (double)q.x * x.x + (double)q.y * x.y + (double)q.z * x.z + (double)q.w * x.w;
            }
        }
        put4(smem + t * RQ + e * 2, LC_C * RQ, q);
        if (GATED) {
#pragma unroll
            for (int o = 1; o < LPT; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
            if ((lane & (LPT - 1)) == 0) nq[e / 4 / LPT][t] = r;
        }
    }
    constexpr int KPER = 32 * DP / 4 / 256;              // 16-byte loads of a thread for 32 tokens of K
    float4 keys[KPER];
    auto fetch_keys = [&](int half) {
#pragma unroll
        for (int i = 0; i < KPER; ++i) {
            const int t = 32 * half + (tid + 256 * i) / (DP / 4), e = ((tid + 256 * i) % (DP / 4)) * 4;
            keys[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < n && e < d) {
                keys[i] = *reinterpret_cast<const float4*>(A.k + (size_t)(t0 + t) * A.qk_stride + h * d + e);
                keys[i].x *= A.k_scale; keys[i].y *= A.k_scale; keys[i].z *= A.k_scale; keys[i].w *= A.k_scale;
            }
        }
    };
    auto put_keys = [&]() {
#pragma unroll
        for (int i = 0; i < KPER; ++i)
            put4(smem + Sh::Q + (tid + 256 * i) / (DP / 4) * RQ + ((tid + 256 * i) % (DP / 4)) * 8, 32 * RQ, keys[i]);
    };
    fetch_keys(0);
    if (tid < LC_C) {                                    // top: the running maximum less F; u: what is added to it for a weight
        const int t = tid;
        if (GATED) {
            const double* w = A.weights + ((size_t)blockIdx.x * A.H + h) * 3 * LC_C;
            const double f = w[t], mm = fmax(m0, w[2 * LC_C + t]);
            u[t] = w[LC_C + t];
            coef[t] = (float)exp(m0 - mm);
            den[t] = expf((float)(-(f + mm)));
            top[t] = -mm;
        } else {
            const double f = (t + 1) * log((double)A.decay[h]);
            u[t] = -f;
            top[t] = f;
            coef[t] = (float)exp(f);
        }
    }
    put_keys();
    fetch_keys(1);
    __syncthreads();
    const uint32_t a_at = (lane & 15), a_hi = (lane >> 4) * 16;                          // rows of a first operand's tile, its second eight k
    const uint32_t b_at = (lane & 7) + (lane >> 4) * 8, b_hi = ((lane >> 3) & 1) * 16;   // rows (tokens) of two tiles of K
    const uint32_t v_at = (lane & 7) + ((lane >> 3) & 1) * 8, v_hi = (lane >> 4) * 16;   // rows of [S ; V], transposed
    double sum[2] = {0.0, 0.0};
    for (int half = 0; half < 2; ++half) {               // P: 16 tokens of the first operand a pair of warps, 16 of the second's 32 a warp
        const int mi = wid >> 1, s0 = 32 * half + 16 * (wid & 1);
        float big[2][4] = {}, rest[2][4] = {};
        if (s0 <= 16 * mi + 15) {
#pragma unroll 2
            for (int k = 0; k < DP / 16; ++k) {
                uint32_t a[3][4], b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    parts_load4(a[p], base + (p * LC_C + 16 * mi + a_at) * RQ + a_hi + k * 32);
                    parts_load4(b[p], kb + (p * 32 + 16 * (wid & 1) + b_at) * RQ + b_hi + k * 32);
                }
                parts_mma6_round(big[0], rest[0], a, b, 0);
                parts_mma6_round(big[1], rest[1], a, b, 2);
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int s = s0 + 8 * j + q2;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int t = 16 * mi + g + 8 * x;
                float v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    v[e] = s + e <= t && t < n ? (big[j][2 * x + e] + rest[j][2 * x + e]) * expf((float)(top[t] + u[s + e])) : 0.f;
                    sum[x] += v[e];
                }
                uint32_t p[3];
                parts_cut(v[0], v[1], p[0], p[1], p[2]);
#pragma unroll
                for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(smem + Sh::Q + Sh::KB + (e * LC_C + t) * RP + s * 2) = p[e];
            }
        }
        if (half == 0) {
            __syncthreads();                             // the first half of K is read
            put_keys();
            __syncthreads();
        }
    }
    fetch(0);
    if (GATED) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            sum[x] += __shfl_xor_sync(0xffffffffu, sum[x], 1);
            sum[x] += __shfl_xor_sync(0xffffffffu, sum[x], 2);
            if (q2 == 0) rowsum[wid & 1][16 * (wid >> 1) + g + 8 * x] = sum[x];
        }
    }
    __syncthreads();                                     // K is read, P is written
    if (GATED && tid < LC_C) {
        double r = nq[0][tid];
        if (DP / 4 > LPT) r += nq[DP / 4 / LPT - 1][tid];
        den[tid] = fmaxf(fabsf((float)(rowsum[0][tid] + rowsum[1][tid] + coef[tid] * r)), den[tid]) + A.den_eps;
    }
    const int wm = wid >> 2, wn = wid & 3;               // 32 tokens and CB / 4 columns a warp
    float big[2][NJ][4], rest[2][NJ][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) big[i][j][x] = rest[i][j][x] = 0.f;
    put(0);
    for (int step = 0; step < steps; ++step) {
        __syncthreads();                                 // the step's rows are there, the step's before last are read
        if (step + 1 < steps) fetch(step + 1);
        const bool values = step >= s_steps;
        if (step == s_steps) {                           // all of Q S is there: each token's weight
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const float c = coef[32 * wm + 16 * i + g + (x >> 1) * 8];
                        big[i][j][x] *= c; rest[i][j][x] *= c;
                    }
        }
        const int r0 = values ? (step - s_steps) * 16 : step * 16;
        if (!values || r0 <= 32 * wm + 31) {             // values of later tokens meet zeros only
            const uint32_t st = kb + (step & 1) * Sh::STAGE;
            uint32_t a[2][3][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const uint32_t row = p * LC_C + 32 * wm + 16 * i + a_at;
                    parts_load4(a[i][p], (values ? pb + row * RP : base + row * RQ) + a_hi + r0 * 2);
                }
#pragma unroll
            for (int j = 0; j < NJ; j += 2) {
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) parts_load4_trans(b[p], st + (p * 16 + v_at) * RB + v_hi + (wn * (CB / 4) + 8 * j) * 2);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    parts_mma6_round(big[i][j], rest[i][j], a[i], b, 0);
                    parts_mma6_round(big[i][j + 1], rest[i][j + 1], a[i], b, 2);
                }
            }
        }
        if (step + 1 < steps) put(step + 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int t = 32 * wm + 16 * i + g + 8 * x;
            if (t >= n) continue;
            float* to = A.out + (size_t)(t0 + t) * A.H * A.dv + (size_t)h * A.dv;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int col = col0 + wn * (CB / 4) + 8 * j + q2;
                float2 o = make_float2(big[i][j][2 * x] + rest[i][j][2 * x], big[i][j][2 * x + 1] + rest[i][j][2 * x + 1]);
                if (GATED) { o.x /= den[t]; o.y /= den[t]; }
                if (col < A.dv) *reinterpret_cast<float2*>(to + col) = o;
            }
        }
}

// ------------------------------------------------------------------ wide chunks on the 5th-generation tensor cores
// Heads of 33 to 128 rows: chunks of 128 tokens, so that tokens (outputs) and rows (end states) fill the MMA's 128.  Everything is a sum
// over k (rows, tokens) of twelve tcgen05 products of bfloat16 parts for every 32 k: the five small products of the six have one
// accumulator in tensor memory for a whole sum, the leading products of 16 k one each, and sixteen worker warps add these up with additions
// that round (the tensor cores cut; see parts_mma.cuh), so that no sum is further from 64 bits than in chunks of 64.  A worker owns a
// lane of tensor memory (a token or a row) and a quarter of the columns.  One more warp issues.  Operands are cut into parts on their
// way to shared memory, in the 128-byte swizzle: rows of 64 values, K-major for Q, K and P, MN-major for what is summed over its rows
// (V, S, and K for the end states).  192 KB, one block an SM.
//   outputs     Q K^T, its sum back into the fourth accumulator; Q S, 32 rows of S a stage through a ring of four in K's place; P takes
//               Q's place, then P V likewise.  A stage's leading products are read while the next one's small ones run.
// Loops stay rolled: a block runs once through its code, and what is not in the instruction cache comes at one instruction in
// about 13 cycles (the weights unrolled over a worker's 64 keys took 18,000 cycles).
//   end states  K^T V, 32 tokens a stage; the small products of all tokens first, then the leading ones, three accumulators in turn.
// Measured beside the mma.sync kernels (chunks of 64), 8 heads of 128 x 256, 2,048 tokens: end states 23 us (28), start states 16 (18),
// outputs 48 (65); all of a gated memory 85 (124), a fixed decay's 70 (101).  Against 64 bits, gated / fixed decay: outputs (the median of tokens and
// heads) 1.16e-7 / 1.10e-7 (chunks of 64 1.16 / 1.11), states 0.85e-7 / 1.00e-7 (0.85 / 1.76); with the leading products in the small ones'
// accumulators 1.25 / 1.34 and 0.89 / 1.09.  With the code of a stage's sums in the outputs' loop four times instead of once they took 59 us.  A block runs
// its phases one after the other, about 35 us whatever else there is, so short steps stay with the chunks of 64 (ops.py).
constexpr int LW_WORK = 512, LW_THREADS = LW_WORK + 32, LW_MMA = LW_WORK / 32, LW_REGION = 3 * LC_WIDE * LC_WIDE * 2;
constexpr int LW_SMEM = 2 * LW_REGION + 1024;

__device__ __forceinline__ uint32_t lw_elect() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one;
}
// by a whole warp, the instruction itself by one lane: its operands are uniform registers then (umma_pair.cuh)
__device__ __forceinline__ void lw_mma(uint32_t acc, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t one) {
    asm volatile("{\n\t.reg .pred p, q;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "setp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(acc), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(one) : "memory");
}
__device__ __forceinline__ void lw_commit(uint64_t* bar, uint32_t one) {
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "setp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
                 ::"r"(smem_addr(bar)), "r"(one) : "memory");
}
// The five small products of parts of 32 k, into `acc` (`more`: to what it holds).  a(p, k), b(p, k): descriptors of part p, k in steps of 16.
template <typename FA, typename FB>
__device__ __forceinline__ void lw_small(uint32_t acc, bool more, uint32_t idesc, uint32_t one, FA a, FB b) {
    constexpr int pa[5] = {2, 0, 1, 1, 0}, pb[5] = {0, 2, 1, 0, 1};
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) lw_mma(acc, a(pa[i], k), b(pb[i], k), idesc, (i || k || more) ? 1u : 0u, one);
}
// the leading products of 16 k each
template <typename FA, typename FB>
__device__ __forceinline__ void lw_lead(uint32_t first, uint32_t second, uint32_t idesc, uint32_t one, FA a, FB b) {
    lw_mma(first, a(0, 0), b(0, 0), idesc, 0u, one);
    lw_mma(second, a(0, 1), b(0, 1), idesc, 0u, one);
}
// eight values' parts into the 16 bytes at `at` of three tiles, `part` bytes apart
__device__ __forceinline__ void lw_put8(unsigned char* at, int part, const float (&x)[8]) {
    uint4 p[3];
    uint32_t* w[3] = {reinterpret_cast<uint32_t*>(&p[0]), reinterpret_cast<uint32_t*>(&p[1]), reinterpret_cast<uint32_t*>(&p[2])};
#pragma unroll
    for (int e = 0; e < 4; ++e) parts_cut(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e]);
#pragma unroll
    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint4*>(at + e * part) = p[e];
}
// eight floats of a row, zeros where !ok or behind `left` values (a multiple of 4)
__device__ __forceinline__ void lw_get8(float (&x)[8], const float* from, bool ok, int left) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(x) = ok && left > 0 ? *reinterpret_cast<const float4*>(from) : z;
    *reinterpret_cast<float4*>(x + 4) = ok && left > 4 ? *reinterpret_cast<const float4*>(from + 4) : z;
}
__device__ __forceinline__ void lw_ld16(uint32_t at, float (&r)[16]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
                   "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]) : "r"(at));
}
__device__ __forceinline__ void lw_ld8(uint32_t at, float (&r)[8]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]) : "r"(at));
}
__device__ __forceinline__ void lw_st16(uint32_t at, const float (&r)[16]) {
    const uint32_t* u = reinterpret_cast<const uint32_t*>(r);
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n\t"
                 "tcgen05.wait::st.sync.aligned;"
                 ::"r"(at), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]),
                   "r"(u[8]), "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]) : "memory");
}
// N columns of two leading products added to `sum`, one after the other
template <int N> __device__ __forceinline__ void lw_add(float (&sum)[N], uint32_t first, uint32_t second) {
#pragma unroll
    for (int c = 0; c < N; c += 8) {
        uint32_t a[8], b[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
                     "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
                     "tcgen05.wait::ld.sync.aligned;"
                     : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
                       "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7])
                     : "r"(first + c), "r"(second + c));
#pragma unroll
        for (int x = 0; x < 8; ++x) sum[c + x] = (sum[c + x] + __uint_as_float(a[x])) + __uint_as_float(b[x]);
    }
}
template <int N> __device__ __forceinline__ void lw_put(const float (&sum)[N], uint32_t at) {
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        float r[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) r[x] = sum[c + x];
        lw_st16(at + c, r);
    }
}
// one of them
template <int N> __device__ __forceinline__ void lw_add_one(float (&sum)[N], uint32_t at) {
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        float r[16];
        lw_ld16(at + c, r);
#pragma unroll
        for (int x = 0; x < 16; ++x) sum[c + x] += r[x];
    }
}
// and the small products' accumulator at the end of a sum: sum = weight (sum + small)
template <int N> __device__ __forceinline__ void lw_end_sum(float (&sum)[N], uint32_t small, float weight) {
#pragma unroll
    for (int c = 0; c < N; c += 8) {
        float r[8];
        lw_ld8(small + c, r);
#pragma unroll
        for (int x = 0; x < 8; ++x) sum[c + x] = fmaf(weight, sum[c + x], weight * r[x]);
    }
}
__device__ __forceinline__ void lw_sync() { asm volatile("bar.sync 1, %0;" ::"n"(LW_WORK) : "memory"); }      // the workers
// A tile of floats out of registers (a lane a row, a quarter of the columns) through shared memory into rows `ld` floats apart, in whole
// rows; by the worker warps.  Lane by lane, 16 bytes of 32 rows at a time, the outputs took 15,000 cycles.  `by`: what a row is divided by, `over` one over it.
template <int CB>
__device__ __forceinline__ void lw_store(float* tile, const float (&sum)[CB / 4], float* to, size_t ld, int rows, int cols, const float* by, const float* over) {
    constexpr int LD = CB + 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row = (warp & 3) * 32 + lane;
#pragma unroll
    for (int c = 0; c < CB / 4; c += 4)
        *reinterpret_cast<float4*>(tile + row * LD + (warp >> 2) * (CB / 4) + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
    lw_sync();
    constexpr int STEP = LW_WORK / (CB / 4);             // rows from one piece of a thread to its next
    const int c = tid % (CB / 4) * 4;
    if (c >= cols) return;
    int r = tid / (CB / 4);
    const float* at = tile + r * LD + c;
    to += (size_t)r * ld + c;
#pragma unroll 4
    for (; r < rows; r += STEP, at += STEP * LD, to += STEP * ld) {
        float4 x = *reinterpret_cast<const float4*>(at);
        if (by) {
            const float b = by[r], o = over[r];
            // A quotient by the reciprocal, corrected once with its remainder (Markstein 1990); where a quotient or its remainder leaves a float's
            // range (infinities, numerators below 2^-80) the division itself.
            auto fits = [&](float z) { const float q = fabsf(z * o); return q > 1e-30f && q < 1e38f && fabsf(z) > 1e-24f; };
            if (b > 1e-30f && b < 1e30f && fits(x.x) && fits(x.y) && fits(x.z) && fits(x.w)) {
                auto quotient = [&](float z) { const float q = z * o; return fmaf(fmaf(-q, b, z), o, q); };
                x.x = quotient(x.x); x.y = quotient(x.y); x.z = quotient(x.z); x.w = quotient(x.w);
            } else { x.x /= b; x.y /= b; x.z /= b; x.w /= b; }
        }
        *reinterpret_cast<float4*>(to) = x;
    }
}
// Sums of floats, or of products of two, with what their additions and roundings lose, which is itself a float sum (about 2^-46 of the
// largest partial sum) and on the float pipe (in double the weights and sums of a chunk took 16,000 cycles).
struct LwSum {
    float s = 0.f, lost = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x, b = t - s;
        lost += (s - (t - b)) + (x - b);
        s = t;
    }
    __device__ __forceinline__ void add_product(float x, float y) {
        const float p = x * y;
        lost += fmaf(x, y, -p);
        add(p);
    }
    __device__ __forceinline__ double value() const { return (double)s + (lost == lost ? (double)lost : 0.0); }      // (an infinity has lost nothing)
};
struct LwBars { uint64_t full[4], done[4], free[4]; uint32_t tmem; int gave_up; };
__device__ __forceinline__ void lw_start(LwBars& B, int warp) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) { mbar_init(B.full + i, LW_MMA); mbar_init(B.done + i, 1); mbar_init(B.free + i, LW_MMA); }
        B.gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == LW_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&B.tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
__device__ __forceinline__ void lw_end(LwBars& B, int warp, uint32_t tmem) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == LW_MMA) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}
// a barrier of the workers alone (the MMA warp may be waiting for them): does `x` hold for any?
__device__ __forceinline__ bool lw_workers_or(bool x) {
    int any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.s32 %0, 1, 0, q;\n}" : "=r"(any) : "r"((int)x), "n"(LW_WORK) : "memory");
    return any != 0;
}
// a worker warp has read its part of the accumulators
__device__ __forceinline__ void lw_taken(uint64_t* bar, int lane) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
// a worker warp's part of a stage is in shared memory
__device__ __forceinline__ void lw_filled(uint64_t* bar, int lane) {
    fence_async_proxy();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// grid (chunks, H, slices of CB columns)
template <int DP, int CB, bool GATED>
__global__ void __launch_bounds__(LW_THREADS, 1) lw_local_kernel(const LinearChunkArgs A) {
    constexpr int C = LC_WIDE, PK = C * DP * 2, PV = C * CB * 2, HC = CB / 4;        // bytes of a part of K, of V; columns a worker
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ks = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* vs = ks + LW_REGION;
    __shared__ LwBars B;
    __shared__ float w[C];
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, col0 = blockIdx.z * CB, d = A.d;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int t0 = A.q_start[ck.x] + ck.y * C, n = min(C, A.q_start[ck.x + 1] - t0), stages = (n + 31) / 32;
    const size_t ch = (size_t)blockIdx.x * A.H + h;
    lw_start(B, warp);
    if (GATED) {
        const double* g = A.weights + ch * 3 * C;
        if (tid < C) w[tid] = tid < n ? (float)exp(A.marks[ch * 3] + g[C + tid] - A.marks[ch * 3 + 1]) * A.k_scale : 0.f;
    } else if (tid < C) {
        const double la = log((double)A.decay[h]);
        w[tid] = tid < n ? (float)exp((n - 1 - tid) * la) * A.k_scale : 0.f;
        if (tid == 0 && blockIdx.z == 0) { A.marks[ch * 3] = n * la; A.marks[ch * 3 + 1] = 0.0; }
    }
    bool odd = tid < C && w[tid] != w[tid];              // a gate that is no number
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = B.tmem;
    volatile int* gave_up = &B.gave_up;
    if (warp == LW_MMA) {
        // A: K^T, B: V, both MN-major; heads of up to 64 rows: the upper half of the tile is whatever lies behind, and nobody reads it
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(CB >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t one = lw_elect(), ka = smem_addr(ks), va = smem_addr(vs);
        auto k_at = [&](int i, int p, int k) { return desc_mnmajor(ka + p * PK + (i * 2 + k) * 16 * 128, C * 128); };
        auto v_at = [&](int i, int p, int k) { return desc_mnmajor(va + p * PV + (i * 2 + k) * 16 * 128, C * 128); };
        bool ok = true;
        for (int i = 0; ok && i < stages; ++i) {
            ok = mbar_wait(B.full + i, 0, gave_up, A.status, 61);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            lw_small(tmem, i > 0, idesc, one, [&](int p, int k) { return k_at(i, p, k); }, [&](int p, int k) { return v_at(i, p, k); });
        }
        lw_commit(B.done + 3, one);
        int slot = 0, lap = 0;
        for (int g = 0; ok && g < 2 * stages; ++g) {
            if (lap && !mbar_wait(B.free + slot, (lap - 1) & 1, gave_up, A.status, 66)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            lw_mma(tmem + 128 + slot * 128, k_at(g >> 1, 0, g & 1), v_at(g >> 1, 0, g & 1), idesc, 0u, one);
            lw_commit(B.done + slot, one);
            if (++slot == 3) { slot = 0; ++lap; }
        }
    } else {
        constexpr int KN = 32 * DP / 8, VN = 32 * CB / 8, KPER = (KN + LW_WORK - 1) / LW_WORK, VPER = (VN + LW_WORK - 1) / LW_WORK;      // pieces of eight a stage, a thread
        float keys[2][KPER][8], values[2][VPER][8];      // two stages on their way
        auto fetch = [&](float (&x)[KPER][8], float (&y)[VPER][8], int i) {
#pragma unroll
            for (int j = 0; j < KPER; ++j) {
                if (KN % LW_WORK && tid >= KN) continue;
                const int t = 32 * i + (tid + LW_WORK * j) / (DP / 8), e = (tid + LW_WORK * j) % (DP / 8) * 8;
                lw_get8(x[j], A.k + (size_t)(t0 + t) * A.qk_stride + h * d + e, t < n, d - e);
            }
#pragma unroll
            for (int j = 0; j < VPER; ++j) {
                if (VN % LW_WORK && tid >= VN) continue;
                const int t = 32 * i + (tid + LW_WORK * j) / (CB / 8), c = (tid + LW_WORK * j) % (CB / 8) * 8;
                lw_get8(y[j], A.v + (size_t)(t0 + t) * A.v_stride + h * A.dv + col0 + c, t < n, A.dv - col0 - c);
            }
        };
        auto fill = [&](float (&x)[KPER][8], float (&y)[VPER][8], int i) {
#pragma unroll
            for (int j = 0; j < KPER; ++j) {
                if (KN % LW_WORK && tid >= KN) continue;
                const int t = 32 * i + (tid + LW_WORK * j) / (DP / 8), c = (tid + LW_WORK * j) % (DP / 8);
                const float wt = w[t];
#pragma unroll
                for (int e = 0; e < 8; ++e) { odd = odd || tl_chunk_odd(x[j][e]); x[j][e] *= wt; }
                lw_put8(ks + swz(C, t, c), PK, x[j]);
            }
#pragma unroll
            for (int j = 0; j < VPER; ++j) {
                if (VN % LW_WORK && tid >= VN) continue;
                const int t = 32 * i + (tid + LW_WORK * j) / (CB / 8), c = (tid + LW_WORK * j) % (CB / 8);
#pragma unroll
                for (int e = 0; e < 8; ++e) odd = odd || tl_chunk_odd(y[j][e]);
                lw_put8(vs + swz(C, t, c), PV, y[j]);
            }
            lw_filled(B.full + i, lane);
            if (i + 2 < stages) fetch(x, y, i + 2);
        };
        fetch(keys[0], values[0], 0);
        fetch(keys[1], values[1], 1);
#pragma unroll 1
        for (int i = 0; i < stages; i += 2) {
            fill(keys[0], values[0], i);
            if (i + 1 < stages) fill(keys[1], values[1], i + 1);
        }
    }
    if (warp < LW_MMA) {
        odd = lw_workers_or(odd);                        // (also: all of K is there for the normaliser)
        if (tid == 0) A.marked[ch * A.tiles + blockIdx.z] = odd;
        const size_t per = (size_t)d * A.dv + (GATED ? d : 0);
        float* to = A.ends + ch * per;
        if (GATED && col0 == 0 && tid < DP && tid < d) { // the normaliser: the same with v = 1, sixteen chains of eight tokens
            float s[16] = {};
            for (int t = 0; t < 32 * stages; t += 16)
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const unsigned char* k = ks + swz(C, t + r, tid >> 3) + (tid & 7) * 2;
                    auto part = [&](int p) { return __bfloat162float(*reinterpret_cast<const bf16*>(k + p * PK)); };
                    s[r] += part(0) + (part(1) + part(2));
                }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int r = 0; r < o; ++r) s[r] += s[r + o];
            to[(size_t)d * A.dv + tid] = s[0];
        }
        const int quarter = warp & 3, share = warp >> 2;
        float sum[HC];
#pragma unroll
        for (int c = 0; c < HC; ++c) sum[c] = 0.f;
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + share * HC;
        mbar_wait(B.done + 3, 0, gave_up, A.status, 62);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        lw_add_one(sum, at);
        int slot = 0, lap = 0;
#pragma unroll 1
        for (int g = 0; g < 2 * stages; ++g) {
            if (!GATED && g == 4) {                      // like terms: the first 64 tokens' sum waits in tensor memory for the others' (gated, the later
                lw_put(sum, at);                         // terms are the large ones)
#pragma unroll
                for (int c = 0; c < HC; ++c) sum[c] = 0.f;
            }
            mbar_wait(B.done + slot, lap & 1, gave_up, A.status, 62);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            lw_add_one(sum, at + 128 + slot * 128);
            lw_taken(B.free + slot, lane);
            if (++slot == 3) { slot = 0; ++lap; }
        }
        if (!GATED && stages > 2) lw_add_one(sum, at);
        lw_store<CB>(reinterpret_cast<float*>(vs), sum, to + col0, A.dv, d, A.dv - col0, nullptr, nullptr);      // (V is read)
    }
    lw_end(B, warp, tmem);
}

// grid (chunks, H, slices of NT tiles of CB columns)
template <int DP, int CB, int NT, bool GATED>
__global__ void __launch_bounds__(LW_THREADS, 1) lw_out_kernel(const LinearChunkArgs A) {
    constexpr int C = LC_WIDE, PQ = C * DP * 2, PP = C * C * 2, PS = 32 * CB * 2, HC = CB / 4, GROUPS = DP / 32;      // bytes of a part of Q and K, of P, of a stage
    extern __shared__ unsigned char smem_raw[];
    unsigned char* qs = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);            // Q, then P
    unsigned char* ks = qs + LW_REGION;                                                                               // K, then the ring
    __shared__ LwBars B;
    __shared__ double rowsum[4][C], nq[C];
    __shared__ float2 u[C];                              // a double as two floats
    __shared__ float coef[C], den[C], over[C];
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, col0 = blockIdx.z * NT * CB, d = A.d;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int t0 = A.q_start[ck.x] + ck.y * C, n = min(C, A.q_start[ck.x + 1] - t0), nv = (n + 31) / 32, stages = NT * (GROUPS + nv);      // stages: Q S of every tile, P V of every tile
    if (GATED) lc_maximum<DP>(A, ck, h);
    const size_t ch = (size_t)blockIdx.x * A.H + h, per = (size_t)d * A.dv + (GATED ? d : 0);
    const float* start = A.ends + ch * per;
    const double m0 = GATED ? A.marks[ch * 3 + 2] : 0.0;
    lw_start(B, warp);
    if (warp < LW_MMA) {
        constexpr int PER = C * DP / 8 / LW_WORK, PR = DP / 8, N = 2;        // pieces of eight a thread, of a row; on their way together
        float norm[8], x[2][N][8];
        if (GATED) lw_get8(norm, start + (size_t)d * A.dv + tid % PR * 8, true, d - tid % PR * 8);
        auto get = [&](float (&to)[N][8], int j0) {      // Q's pieces, then K's
            const float* from = (j0 < PER ? A.q : A.k) + h * d + tid % PR * 8;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int t = (tid + LW_WORK * (j0 + j - (j0 < PER ? 0 : PER))) / PR;
                lw_get8(to[j], from + (size_t)(t0 + t) * A.qk_stride, t < n && j0 < 2 * PER, d - tid % PR * 8);
            }
        };
        auto put = [&](float (&v)[N][8], int j0) {
            const bool isq = j0 < PER;
            const float scale = isq ? A.q_scale : A.k_scale;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int t = (tid + LW_WORK * (j0 + j - (isq ? 0 : PER))) / PR;
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j][e] *= scale;
                lw_put8((isq ? qs : ks) + swz(C, t, tid % PR), PQ, v[j]);
                if (GATED && isq) {
                    LwSum r;                             // n . q of the chunk's start state
#pragma unroll
                    for (int e = 0; e < 8; ++e) r.add_product(v[j][e], norm[e]);
#pragma unroll
                    for (int o = 1; o < PR; o <<= 1) {
                        const float lost = __shfl_xor_sync(0xffffffffu, r.lost, o);
                        r.add(__shfl_xor_sync(0xffffffffu, r.s, o));
                        r.lost += lost;
                    }
                    if (lane % PR == 0) nq[t] = r.value();
                }
            }
        };
        get(x[0], 0);
#pragma unroll 1
        for (int j0 = 0; j0 < 2 * PER; j0 += 2 * N) {
            get(x[1], j0 + N);
            put(x[0], j0);
            get(x[0], j0 + 2 * N);
            put(x[1], j0 + N);
        }
        fence_async_proxy();
    }
    auto pair = [](double x) { const float hi = (float)x; return make_float2(hi, (float)(x - (double)hi)); };
    float2 top = make_float2(0.f, 0.f);                  // a token's running maximum less F; u: what is added to it for a weight
    if (warp < LW_MMA) {
        const int t = tid & (C - 1);                     // the worker's token: all that share it need top
        double uv;
        if (GATED) {
            const double* w = A.weights + ch * 3 * C;
            const double f = w[t], mm = fmax(m0, w[2 * C + t]);
            uv = w[C + t];
            if (tid < C) { coef[t] = (float)exp(m0 - mm); den[t] = expf((float)(-(f + mm))); }
            top = pair(-mm);
        } else {
            const double f = (t + 1) * log((double)A.decay[h]);
            uv = -f;
            if (tid < C) coef[t] = (float)exp(f);
            top = pair(f);
        }
        if (warp < 4) u[t] = pair(uv);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = B.tmem;
    volatile int* gave_up = &B.gave_up;
    if (warp == LW_MMA) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);
        const uint32_t one = lw_elect(), qa = smem_addr(qs), ka = smem_addr(ks);
        auto kmajor = [&](uint32_t tile, int k) { return tile + (k >> 2) * C * 128 + (k & 3) * 32; };       // k in steps of 16
        int turn = 0;
        auto products = [&](bool more, uint32_t kind, auto a, auto b) {  // of 32 k; a new sum starts once the one before has been read
            auto freed = [&]() { return !turn || mbar_wait(B.free, (turn - 1) & 1, gave_up, A.status, 67); };
            if (!more && !freed()) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            lw_small(tmem + 128, more, kind, one, a, b);
            if (more && !freed()) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            lw_lead(tmem + 256, tmem + 384, kind, one, a, b);
            lw_commit(B.done, one);
            ++turn;
            return true;
        };
        bool ok = true;
#pragma unroll 1
        for (int i = 0; ok && i < GROUPS; ++i)
            ok = products(i > 0, idesc | ((uint32_t)(C >> 3) << 17), [&](int p, int k) { return desc_kmajor(kmajor(qa + p * PQ, 2 * i + k)); },
                          [&](int p, int k) { return desc_kmajor(kmajor(ka + p * PQ, 2 * i + k)); });
        int group = 0;
#pragma unroll 1
        for (int i = 0; ok && i < stages; ++i) {
            const bool values = i >= NT * GROUPS;
            if (!mbar_wait(B.full + (i & 3), (i >> 2) & 1, gave_up, A.status, 63)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = ka + (i & 3) * 3 * PS, at = kmajor(qa, 2 * group), part = values ? PP : PQ;
            ok = products(group > 0, idesc | (1u << 16) | ((uint32_t)(CB >> 3) << 17), [&](int p, int k) { return desc_kmajor(at + p * part + k * 32); },
                          [&](int p, int k) { return desc_mnmajor(st + p * PS + k * 16 * 128, 32 * 128); });
            group = group + 1 == (values ? nv : GROUPS) ? 0 : group + 1;
        }
    } else {
        constexpr int SN = 32 * CB / 8, SPER = (SN + LW_WORK - 1) / LW_WORK;     // pieces of eight a stage, a thread
        static_assert(SPER == 1, "a piece a thread");
        const int quarter = warp & 3, share = warp >> 2, t = quarter * 32 + lane;
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16);
        const int r = tid / (CB / 8), col = tid % (CB / 8) * 8;
        float ahead[8];
        // 32 rows of S, then of V, tile after tile; zeros where there are none.  A cursor over the stages: the next one's first row and tile.
        const float* from_s = start + (size_t)r * A.dv + col0 + col;
        const float* from_v = A.v + (size_t)(t0 + r) * A.v_stride + h * A.dv + col0 + col;
        int next_row = r, next_col = col0 + col;
        bool values = false;
        auto fetch = [&]() {
            const int z = next_col - col0 - col, rows = values ? n : d;
            const float* from = values ? from_v + (size_t)(next_row - r) * A.v_stride + z : from_s + (size_t)(next_row - r) * A.dv + z;
            if (SN % LW_WORK == 0 || tid < SN) lw_get8(ahead, from, next_row < rows, A.dv - next_col);
            next_row += 32;
            if (next_row - r >= (values ? 32 * nv : DP)) {
                next_row = r;
                next_col += CB;
                if (next_col - col0 >= NT * CB) { next_col = col0 + col; values = true; }
            }
        };
        fetch();
        const bool sees = share <= quarter;              // keys behind all of the warp's tokens weigh nothing
        {                                                // Q K^T, into the fourth accumulator; all of it is there before the ring takes K's place
            float qk[32] = {};
#pragma unroll 1
            for (int i = 0; i < GROUPS; ++i) {
                mbar_wait(B.done, i & 1, gave_up, A.status, 64);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (sees) {
                    lw_add(qk, acc + 256 + 32 * share, acc + 384 + 32 * share);
                    if (i + 1 == GROUPS) lw_end_sum(qk, acc + 128 + 32 * share, 1.0f);
                }
                lw_taken(B.free, lane);
            }
            if (sees) lw_put(qk, acc + 32 * share);
        }
        float sum[NT][HC];
#pragma unroll
        for (int z = 0; z < NT; ++z)
#pragma unroll
            for (int c = 0; c < HC; ++c) sum[z][c] = 0.f;
        int taken = 0, tile = 0, group = 0;
        const float weight = coef[t];                    // the token's, of the chunk's start state
        auto take = [&](int below) {                     // the accumulators of the stages below (GROUPS is even: a stage's parity is its own)
            static_assert(GROUPS % 2 == 0, "parity of the stages");
#pragma unroll 1
            for (; taken < below; ++taken) {
                mbar_wait(B.done, taken & 1, gave_up, A.status, 65);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = acc + share * HC;
                const bool states = taken < NT * GROUPS, last = ++group == (states ? GROUPS : nv);
#pragma unroll
                for (int z = 0; z < NT; ++z) {
                    if (tile != z) continue;
                    lw_add(sum[z], at + 256, at + 384);
                    if (last) lw_end_sum(sum[z], at + 128, states ? weight : 1.0f);
                }
                lw_taken(B.free, lane);
                if (last) { group = 0; tile = tile + 1 == NT ? 0 : tile + 1; }
            }
        };
        auto weigh = [&]() {                             // all of Q S is there: P takes Q's place
            LwSum total;
            const int last = t < n ? t : -1;
#pragma unroll 1
            for (int s = 32 * share; s < 32 * share + 32; s += 8) {
                float P[8] = {};
                if (sees) {
                    lw_ld8(acc + s, P);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {        // no branch in here: the chains overlap.  A key behind the token is left out, not weighed with
                                                         // zero: its product may be an infinity
                        const float2 v = u[s + e];
                        const float y = top.x + v.x, b = y - top.x;      // the sum of two doubles, rounded once
                        const float x = y + (((top.x - (y - b)) + (v.x - b)) + (top.y + v.y));
                        P[e] = s + e <= last ? P[e] * expf(x) : 0.f;
                    }
                    if (GATED) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) total.add(P[e]);
                    }
                }
                lw_put8(qs + swz(C, t, s / 8), PP, P);
            }
            if (GATED) {
                rowsum[share][t] = total.value();
                lw_sync();
                if (share == 0) {
                    den[t] = fmaxf(fabsf((float)((rowsum[0][t] + rowsum[1][t]) + (rowsum[2][t] + rowsum[3][t]) + coef[t] * nq[t])), den[t]) + A.den_eps;
                    over[t] = 1.0f / den[t];
                }
            }
        };
        // Each part of this loop stands in it once (see above): a stage's accumulators are taken while the next stage's products run.
#pragma unroll 1
        for (int i = 0; i <= stages; ++i) {
            take(i == NT * GROUPS || i == stages ? i : i - 1);
            if (i == stages) break;
            if (i == NT * GROUPS) weigh();
            if (!(SN % LW_WORK) || tid < SN) lw_put8(ks + (i & 3) * 3 * PS + swz(32, r, tid % (CB / 8)), PS, ahead);
            lw_filled(B.full + (i & 3), lane);
            if (i + 1 < stages) fetch();
        }
        // (the ring is read: its last sums have been taken; the barrier in there stands between den and its readers)
#pragma unroll
        for (int z = 0; z < NT; ++z) {
            if (z) lw_sync();
            lw_store<CB>(reinterpret_cast<float*>(ks), sum[z], A.out + (size_t)t0 * A.H * A.dv + (size_t)h * A.dv + col0 + z * CB, (size_t)A.H * A.dv, n,
                         A.dv - col0 - z * CB, GATED ? den : nullptr, over);
        }
    }
    lw_end(B, warp, tmem);
}

template <int DP, int CB, bool GATED>
static int lw_launch(const LinearChunkArgs& A, int n_chunks, int requests, cudaStream_t stream) {
    static bool r1[TL_MAX_DEVICES] = {}, r2[TL_MAX_DEVICES] = {};
    static bool r3[TL_MAX_DEVICES] = {};
    int e = tl_raise_smem(lw_local_kernel<DP, CB, GATED>, r1, LW_SMEM);
    if (!e) e = tl_raise_smem(lw_out_kernel<DP, CB, 1, GATED>, r2, LW_SMEM);
    if (!e) e = tl_raise_smem(lw_out_kernel<DP, CB, 2, GATED>, r3, LW_SMEM);
    if (e) return e;
    const int tiles = (A.dv + CB - 1) / CB;
    if (GATED) {
        lc_gates_kernel<LC_WIDE><<<dim3(n_chunks, A.H), 32, 0, stream>>>(A);
        if ((e = tl_launch_status())) return e;
    }
    lw_local_kernel<DP, CB, GATED><<<dim3(n_chunks, A.H, tiles), LW_THREADS, LW_SMEM, stream>>>(A);
    if ((e = tl_launch_status())) return e;
    const size_t per = (size_t)A.d * A.dv + (GATED ? A.d : 0);
    lc_carry_kernel<8, DP / 8, GATED><<<dim3((unsigned)((per / 4 + 255) / 256), A.H, requests), 256, 0, stream>>>(A);
    if ((e = tl_launch_status())) return e;
    // Two tiles a block share its Q K^T and weights; where single tiles fit the GPU at once, they are done sooner.
    if ((long long)n_chunks * A.H * tiles > tl_num_sms() && tiles > 1)
        lw_out_kernel<DP, CB, 2, GATED><<<dim3(n_chunks, A.H, (tiles + 1) / 2), LW_THREADS, LW_SMEM, stream>>>(A);
    else
        lw_out_kernel<DP, CB, 1, GATED><<<dim3(n_chunks, A.H, tiles), LW_THREADS, LW_SMEM, stream>>>(A);
    return tl_launch_status();
}

template <int DP>
static int lw_pick(const LinearChunkArgs& A, int n_chunks, int requests, cudaStream_t stream) {
    if (A.gates) return A.dv <= 64 ? lw_launch<DP, 64, true>(A, n_chunks, requests, stream) : lw_launch<DP, 128, true>(A, n_chunks, requests, stream);
    return A.dv <= 64 ? lw_launch<DP, 64, false>(A, n_chunks, requests, stream) : lw_launch<DP, 128, false>(A, n_chunks, requests, stream);
}

template <int DP, int CB, bool GATED>
static int lc_launch(const LinearChunkArgs& A, int n_chunks, int requests, cudaStream_t stream) {
    constexpr int RB = DP < 128 ? DP : 128, R = DP == 32 ? 4 : 8, IS = DP / R;
    constexpr int local_smem = LocalShape<RB, CB>::BYTES, out_smem = OutShape<DP, CB>::BYTES;
    static bool r1[TL_MAX_DEVICES] = {}, r2[TL_MAX_DEVICES] = {};
    int e = tl_raise_smem(lc_local_kernel<RB, CB, GATED>, r1, local_smem);
    if (!e) e = tl_raise_smem(lc_out_kernel<DP, CB, GATED>, r2, out_smem);
    if (e) return e;
    const int col_tiles = (A.dv + CB - 1) / CB, row_tiles = (A.d + RB - 1) / RB;
    if (GATED) {
        lc_gates_kernel<LC_C><<<dim3(n_chunks, A.H), 32, 0, stream>>>(A);
        if ((e = tl_launch_status())) return e;
    }
    lc_local_kernel<RB, CB, GATED><<<dim3(n_chunks, A.H, row_tiles * col_tiles), 256, local_smem, stream>>>(A);
    if ((e = tl_launch_status())) return e;
    const size_t per = (size_t)A.d * A.dv + (GATED ? A.d : 0);
    lc_carry_kernel<R, IS, GATED><<<dim3((unsigned)((per / 4 + 255) / 256), A.H, requests), 256, 0, stream>>>(A);
    if ((e = tl_launch_status())) return e;
    lc_out_kernel<DP, CB, GATED><<<dim3(n_chunks, A.H, col_tiles), 256, out_smem, stream>>>(A);
    return tl_launch_status();
}

template <int DP>
static int lc_pick(const LinearChunkArgs& A, int n_chunks, int requests, cudaStream_t stream) {
    if (A.gates) return A.dv <= 64 ? lc_launch<DP, 64, true>(A, n_chunks, requests, stream) : lc_launch<DP, 128, true>(A, n_chunks, requests, stream);
    return A.dv <= 64 ? lc_launch<DP, 64, false>(A, n_chunks, requests, stream) : lc_launch<DP, 128, false>(A, n_chunks, requests, stream);
}

// Blocks of the end states a (chunk, head).
static int lc_tiles(int d, int dv) {
    const int cb = dv <= 64 ? 64 : 128, rb = d <= 32 ? 32 : d <= 64 ? 64 : 128;
    return ((d + rb - 1) / rb) * ((dv + cb - 1) / cb);
}
// Tokens a chunk; the wide ones where heads have the rows for them (else 0).
TL_EXPORT int tl_linear_chunk(int d, int wide) { return !wide ? LC_C : d > 32 && d <= 128 ? LC_WIDE : 0; }
TL_EXPORT int tl_linear_chunk_tiles(int d, int dv) { return lc_tiles(d, dv); }

// `rows` (float [T, 2 H d], with a rotation): where q and k go.  ends: float [n_chunks, H, d dv (+ d with gates)], marks: double
// [n_chunks, H, 3], with gates then [n_chunks, H, 3 chunk].  chunk: what a chunk of `chunks` holds, one of tl_linear_chunk's.  marked: int [n_chunks, H, tl_linear_chunk_tiles(d, dv)], for the scan kernel.  d, dv, the offsets and the stride are multiples of 4 and the pointers 16-byte aligned.
TL_EXPORT int tl_linear_chunks(const float* proj, int T, int stride, int q_off, int k_off, int v_off, const float* gates, float cap,
                               const float* decay, const float* inv_freq, int rot, int interleaved, const int* pos, float q_scale,
                               float k_scale, float* rows, float* state, long long slot_stride, const int* q_start, const int* slots,
                               const int* chunks, int n_chunks, const int* firsts, int requests, float* ends, double* marks, int* marked, float* out,
                               int H, int d, int dv, float den_eps, int chunk, int* status, cudaStream_t stream) {
    if (n_chunks <= 0 || H <= 0) return 0;
    if (status == nullptr || (chunk != LC_C && chunk != tl_linear_chunk(d, 1))) return 1;
    if (H > 65535 || requests > 65535 || d < 4 || d > 256 || ((d | dv | stride | q_off | k_off | v_off) & 3) || (rot & 1) || rot > d ||
        (rot && !rows) || (gates != nullptr) == (decay != nullptr) ||
        ((((uintptr_t)proj) | ((uintptr_t)rows) | ((uintptr_t)ends) | ((uintptr_t)out)) & 15)) return 1;
    LinearChunkArgs A{proj + q_off, proj + k_off, stride, proj + v_off, stride, gates, cap, decay, q_scale, k_scale, state, slot_stride,
                      q_start, slots, (const int4*)chunks, firsts, ends, marks, marks + (size_t)n_chunks * H * 3, marked, lc_tiles(d, dv), out, H, d, dv, (dv + LC_COLS - 1) / LC_COLS, den_eps, status};
    if (rot) {
        if (rot % (interleaved ? 4 : 8) == 0)
            lc_rotate_kernel<true><<<T, 256, rot * sizeof(float), stream>>>(proj, stride, q_off, k_off, inv_freq, rot, interleaved, pos, q_scale, k_scale, rows, H, d);
        else
            lc_rotate_kernel<false><<<T, 256, rot * sizeof(float), stream>>>(proj, stride, q_off, k_off, inv_freq, rot, interleaved, pos, q_scale, k_scale, rows, H, d);
        const int e = tl_launch_status();
        if (e) return e;
        A.q = rows; A.k = rows + (size_t)H * d; A.qk_stride = 2 * H * d;
        A.q_scale = A.k_scale = 1.0f;
    }
    if (d <= 32) return lc_pick<32>(A, n_chunks, requests, stream);
    if (chunk == LC_WIDE) return d <= 64 ? lw_pick<64>(A, n_chunks, requests, stream) : lw_pick<128>(A, n_chunks, requests, stream);
    if (d <= 64) return lc_pick<64>(A, n_chunks, requests, stream);
    if (d <= 128) return lc_pick<128>(A, n_chunks, requests, stream);
    return lc_pick<256>(A, n_chunks, requests, stream);
}
