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
#include "common.cuh"
#include "parts_mma.cuh"

constexpr int LC_C = 64;                 // tokens a chunk
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
};

__device__ __forceinline__ float lc_log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// A warp, gated: for the n tokens of a chunk that starts at row t0, F[t] (the log decays' sum up to t), u[t] = i_t - F[t] and the running
// maximum top[t] of u.
__device__ __forceinline__ void lc_weights(const LinearChunkArgs& A, int t0, int n, int h, int lane, double* F, double* u, double* top) {
    double f[2], in[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        f[e] = 0.0; in[e] = -INFINITY;
        if (t < n) {
            const float* g = A.gates + (size_t)(t0 + t) * 2 * A.H;
            in[e] = A.cap * tanhf(g[h] / A.cap);
            f[e] = lc_log_sigmoid(A.cap * tanhf(g[A.H + h] / A.cap));
        }
    }
    double sum = f[0] + f[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += x;
    }
    const double F1 = sum, F0 = sum - f[1], u0 = in[0] - F0, u1 = in[1] - F1;
    double best = fmax(u0, u1);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, best, o);
        if (lane >= o) best = fmax(best, x);
    }
    double before = __shfl_up_sync(0xffffffffu, best, 1);
    if (lane == 0) before = -INFINITY;
    F[2 * lane] = F0; F[2 * lane + 1] = F1;
    u[2 * lane] = u0; u[2 * lane + 1] = u1;
    top[2 * lane] = fmax(before, u0); top[2 * lane + 1] = best;
}

// A warp a (chunk, head): the gated kinds' weights, once for all blocks that need them (worked out in each of them, warp 0 held the
// others up: end states 36 us, 33.5 without and 4.6 here, and the outputs need them without a wait).
__global__ void __launch_bounds__(32) lc_gates_kernel(const LinearChunkArgs A) {
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, lane = threadIdx.x, t0 = A.q_start[ck.x] + ck.y * LC_C, n = min(LC_C, A.q_start[ck.x + 1] - t0);
    const size_t at = (size_t)blockIdx.x * A.H + h;
    double* w = A.weights + at * 3 * LC_C;
    lc_weights(A, t0, n, h, lane, w, w + LC_C, w + 2 * LC_C);
    __syncwarp();
    if (lane == 0) {
        const double end = w[n - 1];
        A.marks[at * 3] = end;
        A.marks[at * 3 + 1] = (double)(float)(end + w[2 * LC_C + n - 1]);
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
        lc_gates_kernel<<<dim3(n_chunks, A.H), 32, 0, stream>>>(A);
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
TL_EXPORT int tl_linear_chunk() { return LC_C; }
TL_EXPORT int tl_linear_chunk_tiles(int d, int dv) { return lc_tiles(d, dv); }

// `rows` (float [T, 2 H d], with a rotation): where q and k go.  ends: float [n_chunks, H, d dv (+ d with gates)], marks: double
// [n_chunks, H, 3], with gates then [n_chunks, H, 192].  marked: int [n_chunks, H, tl_linear_chunk_tiles(d, dv)], for the scan kernel.  d, dv, the offsets and the stride are multiples of 4 and the pointers 16-byte aligned.
TL_EXPORT int tl_linear_chunks(const float* proj, int T, int stride, int q_off, int k_off, int v_off, const float* gates, float cap,
                               const float* decay, const float* inv_freq, int rot, int interleaved, const int* pos, float q_scale,
                               float k_scale, float* rows, float* state, long long slot_stride, const int* q_start, const int* slots,
                               const int* chunks, int n_chunks, const int* firsts, int requests, float* ends, double* marks, int* marked, float* out,
                               int H, int d, int dv, float den_eps, cudaStream_t stream) {
    if (n_chunks <= 0 || H <= 0) return 0;
    if (H > 65535 || requests > 65535 || d < 4 || d > 256 || ((d | dv | stride | q_off | k_off | v_off) & 3) || (rot & 1) || rot > d ||
        (rot && !rows) || (gates != nullptr) == (decay != nullptr) ||
        ((((uintptr_t)proj) | ((uintptr_t)rows) | ((uintptr_t)ends) | ((uintptr_t)out)) & 15)) return 1;
    LinearChunkArgs A{proj + q_off, proj + k_off, stride, proj + v_off, stride, gates, cap, decay, q_scale, k_scale, state, slot_stride,
                      q_start, slots, (const int4*)chunks, firsts, ends, marks, marks + (size_t)n_chunks * H * 3, marked, lc_tiles(d, dv), out, H, d, dv, (dv + LC_COLS - 1) / LC_COLS, den_eps};
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
    if (d <= 64) return lc_pick<64>(A, n_chunks, requests, stream);
    if (d <= 128) return lc_pick<128>(A, n_chunks, requests, stream);
    return lc_pick<256>(A, n_chunks, requests, stream);
}
