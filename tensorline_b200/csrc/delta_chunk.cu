// The gated delta rule of delta.cu for steps of many tokens: chunks of 32 tokens, inside a chunk matrix products, from chunk to chunk
// the state.
//
//   S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
//
// With F_t the sum of the log decays of a chunk up to t and S0 its start state, the corrections of a chunk solve a triangular system
//   u_t + sum_{s<t} A_ts u_s = beta_t (v_t - e^F_t S0^T k_t),      A_ts = beta_t e^(F_t - F_s) k_t . k_s
// so U = U0 - W S0 with U0 = (I + A)^-1 (beta V) and W = (I + A)^-1 (beta e^F K), and
//   o_t = e^F_t S0^T q_t + sum_{s<=t} e^(F_t - F_s) (q_t . k_s) u_s,      S = e^F_end S0 + sum_t e^(F_end - F_t) k_t u_t^T.
//   prepare   every chunk of every head at once: A, the weights P of the outputs, U0 and W (a thread a column of the system)
//   walk      a block a request, head and 16 columns of the state: chunk after chunk U, the outputs and the state
//
// Everything is held in float, and the walk's products are float products on the tensor cores: each factor is cut into three
// bfloat16 parts (24 bits of it), six of the nine products of parts are taken (the other three lie below a float's last
// bit), the leading one in an accumulator of its own, so that the others' roundings count 2^-8.  F is a sum of doubles, every weight
// the float exponential of one difference of them.  The state in the slots has the layout of the scan kernel.  A position's
// sums depend on where its step began, to rounding.
//
// The token-by-token kernel is bound by its chain: two column sums with shuffles a token, 0.31 us.  As float multiply-adds the walk
// is bound by shared memory: a warp gets 32 floats of it a cycle and needs one for two multiply-adds with 16 columns a
// block (measured 286 us for 2,048 tokens, 8 heads of 128 x 256; token by token 642).  On mma.sync a warp holds 32 rows of the transposed state [16 columns x 128 rows] as
// accumulators, which are the next product's first operand as they lie; W, K, Q and P come as bfloat16 parts, cut once
// by prepare, in rows padded for ldmatrix, so that a chunk's operands are linear copies.  With four warps that do everything and copy by
// 16-byte cp.async the walk took 132 us; four more warps for the outputs 130, bulk copies 123, W a chunk and a half ahead 113 (the chain
// alone, without outputs, 93).  Prepare 33.
#include "umma.cuh"
#include "parts_mma.cuh"

constexpr int DC_C = 32;                 // tokens a chunk
constexpr int DC_COLS = 16;              // columns a block of the walk and a slice of the state's layout
constexpr int DC_UB = DC_C * 20 * 4;     // bytes of a slice of U0: 32 rows of 16 floats, 20 apart
constexpr int DC_PROW = DC_C * 2 + 16, DC_PB = 3 * DC_C * DC_PROW;      // a row of a part of P, the three parts
constexpr int DC_MB = 2 * DC_C * 4;      // e^F_t, then e^(F_end - F_t)
__host__ __device__ constexpr int dc_row(int dp) { return dp * 2 + 16; }              // bytes of a row of a part of W, K, Q
__host__ __device__ constexpr int dc_parts(int dp) { return 3 * DC_C * dc_row(dp); }  // bytes of the three parts

struct DeltaChunkArgs {
    const float* qkv; int stride; int q_off, k_off, v_off;      // as conv_prep left them
    const float* gates; int gate_stride; const float* A_log; const float* dt_bias;
    float* state; long long slot_stride;
    const int* q_start; const int* slots;
    const int4* chunks;                  // (request, number of the chunk, the request's chunks, first chunk of the request in the list)
    const int* firsts;                   // the requests' first chunks
    unsigned char* W;                    // [chunks][H] parts of W
    unsigned char* P;                    // [chunks][H] parts of P, row t
    unsigned char* M;                    // [chunks][H] marks
    unsigned char* U;                    // [chunks][H][nz] slices of U0
    unsigned char* K;                    // [chunks][nqk] parts of K, then of Q
    int* marked;                         // [chunks][H]: operands that the scan kernel has to take (common.cuh)
    float* out;
    int H, nqk, d, dv, nz;
    int* status;
};

__device__ __forceinline__ float dc_softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// ------------------------------------------------------------------ prepare
// grid (chunks, H); shared memory K, Q [32][DP + 4], V [32][dv].  384 threads: the columns of a head of 128 x 256 at once.  The dot
// products of a chunk's keys and queries are taken on parts as well: as single chains of multiply-adds over 128 rows they were what
// the outputs lost most by (130 tokens: 2.1e-7 off the recurrence in 64 bits, now 1.1e-7; the token-by-token kernel 1.5e-7).
constexpr int DC_PREP = 384;
template <int DP>
__global__ void __launch_bounds__(DC_PREP) dc_prepare_kernel(const DeltaChunkArgs A) {
    constexpr int LD = DP + 4, ROW = dc_row(DP);
    extern __shared__ __align__(16) float sm[];
    float* Ks = sm;
    float* Qs = sm + DC_C * LD;
    float* Vs = Qs + DC_C * LD;
    __shared__ __align__(16) float As[DC_C][DC_C];       // A, row t: read as broadcasts
    __shared__ __align__(16) float Ps[DC_C][DC_C + 4];
    __shared__ double F[DC_C];
    __shared__ float beta[DC_C], grow[DC_C];
    const int4 ck = A.chunks[blockIdx.x];
    const int h = blockIdx.y, rep = A.H / A.nqk, hq = h / rep, d = A.d, dv = A.dv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t0 = A.q_start[ck.x] + ck.y * DC_C, n = min(DC_C, A.q_start[ck.x + 1] - t0);
    const size_t at = (size_t)blockIdx.x * A.H + h;
    auto copy16 = [&](float* dst, const float* src, bool ok) {       // zeros where !ok
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(ok ? src : A.qkv), "r"(ok ? 16 : 0)
                     : "memory");
    };
    for (int i = tid; i < DC_C * DP / 4; i += DC_PREP) {
        const int t = i / (DP / 4), e = (i % (DP / 4)) * 4;
        const float* row = A.qkv + (size_t)(t0 + t) * A.stride + hq * d + e;
        copy16(Qs + t * LD + e, row + A.q_off, t < n && e < d);
        copy16(Ks + t * LD + e, row + A.k_off, t < n && e < d);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = tid; i < DC_C * dv / 4; i += DC_PREP) {
        const int t = i / (dv / 4), e = (i - t * (dv / 4)) * 4;
        copy16(Vs + t * dv + e, A.qkv + (size_t)(t0 + t) * A.stride + A.v_off + h * dv + e, t < n);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (wid == 0) {
        double x = 0.0;
        float b = 0.f;
        if (lane < n) {
            const float* g = A.gates + (size_t)(t0 + lane) * A.gate_stride;
            b = 1.0f / (1.0f + expf(-g[h]));
            x = -expf(A.A_log[h]) * dc_softplus(g[A.H + h] + A.dt_bias[h]);
            if (x < -1e4) x = -1e4;                      // a decay of zero all the same; the differences behind it stay exact, -inf gives none
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const double end = __shfl_sync(0xffffffffu, x, 31);          // tokens behind the chunk's last add nothing
        F[lane] = x; beta[lane] = b; grow[lane] = expf((float)x);
        float* mk = reinterpret_cast<float*>(A.M + at * DC_MB);
        mk[lane] = expf((float)x);
        mk[DC_C + lane] = expf((float)(end - x));
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (h == hq * rep) {                                 // the parts of K and Q, once for the heads that share them
        unsigned char* to = A.K + ((size_t)blockIdx.x * A.nqk + hq) * 2 * dc_parts(DP);
        for (int i = tid; i < 2 * DC_C * DP / 4; i += DC_PREP) {
            const bool isq = i >= DC_C * DP / 4;
            const int j = isq ? i - DC_C * DP / 4 : i, t = j / (DP / 4), e = (j % (DP / 4)) * 4;
            const float4 x = *reinterpret_cast<const float4*>((isq ? Qs : Ks) + t * LD + e);
            uint2 p[3];
            parts_cut(x.x, x.y, p[0].x, p[1].x, p[2].x);
            parts_cut(x.z, x.w, p[0].y, p[1].y, p[2].y);
#pragma unroll
            for (int c = 0; c < 3; ++c) *reinterpret_cast<uint2*>(to + (isq ? dc_parts(DP) : 0) + (c * DC_C + t) * ROW + e * 2) = p[c];
        }
    }
    if (wid < 8) {                                       // k_t . k_s (even warps) and q_t . k_s: a warp 16 tokens t and 16 tokens s
        const int g = lane >> 2, q2 = (lane & 3) * 2, t0w = ((wid >> 1) & 1) * 16, s0w = (wid >> 2) * 16;
        const bool qk = wid & 1;
        float big[2][4] = {}, rest[2][4] = {};
        if (s0w <= t0w) {
            const float* at = (qk ? Qs : Ks) + (t0w + g) * LD + q2;
            const float* bt = Ks + (s0w + g) * LD + q2;
            auto cut = [&](const float* x, uint32_t (&p)[3][4], int i) {
                const float2 v = *reinterpret_cast<const float2*>(x);
                parts_cut(v.x, v.y, p[0][i], p[1][i], p[2][i]);
            };
#pragma unroll 2
            for (int e = 0; e < DP; e += 16) {
                uint32_t a[3][4], b[3][4];
                cut(at + e, a, 0); cut(at + 8 * LD + e, a, 1); cut(at + e + 8, a, 2); cut(at + 8 * LD + e + 8, a, 3);
                cut(bt + e, b, 0); cut(bt + e + 8, b, 1); cut(bt + 8 * LD + e, b, 2); cut(bt + 8 * LD + e + 8, b, 3);
                parts_mma6_round(big[0], rest[0], a, b, 0);
                parts_mma6_round(big[1], rest[1], a, b, 2);
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int t = t0w + g + (x >> 1) * 8, s = s0w + 8 * j + q2 + (x & 1);
                const float dot = big[j][x] + rest[j][x], w = s <= t && t < n ? expf((float)(F[t] - F[s])) : 0.f;
                if (qk) Ps[t][s] = w * dot;
                else As[t][s] = s < t ? beta[t] * (w * dot) : 0.f;
            }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int i = tid; i < DC_C * DC_C / 2; i += DC_PREP) {
        const int t = i / (DC_C / 2), x = (i % (DC_C / 2)) * 2;
        const float2 v = *reinterpret_cast<const float2*>(&Ps[t][x]);
        uint32_t p[3];
        parts_cut(v.x, v.y, p[0], p[1], p[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) *reinterpret_cast<uint32_t*>(A.P + at * DC_PB + (c * DC_C + t) * DC_PROW + x * 2) = p[c];
    }
    const int wide = (dv + 15) & ~15;                    // columns behind the last are zeros, like rows behind d
    bool odd = false;                                    // a decay or a beta that is no number shows in W's columns
    for (int c = tid; c < wide + DP; c += DC_PREP) {
        float u[DC_C];
        const bool isw = c >= wide;
        const int e = c - wide;
#pragma unroll
        for (int t = 0; t < DC_C; ++t) {
            if (isw) u[t] = beta[t] * (grow[t] * Ks[t * LD + e]);
            else u[t] = c < dv ? beta[t] * Vs[t * dv + c] : 0.f;
            odd = odd || tl_chunk_odd(isw ? u[t] + Ks[t * LD + e] : c < dv ? Vs[t * dv + c] : 0.f);
        }
#pragma unroll
        for (int t = 1; t < DC_C; ++t) {
            float s0 = 0.f, s1 = 0.f;                    // two chains a row
#pragma unroll
            for (int s = 0; s < t; s += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&As[t][s]);
                s0 = fmaf(a.x, u[s], s0);
                if (s + 1 < t) s1 = fmaf(a.y, u[s + 1], s1);
                if (s + 2 < t) s0 = fmaf(a.z, u[s + 2], s0);
                if (s + 3 < t) s1 = fmaf(a.w, u[s + 3], s1);
            }
            u[t] -= s0 + s1;
        }
        if (isw) {
            __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(A.W + at * dc_parts(DP)) + e;
#pragma unroll
            for (int t = 0; t < DC_C; ++t) {
                float x = u[t];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const __nv_bfloat16 b = __float2bfloat16_rn(x);
                    to[(p * DC_C + t) * (ROW / 2)] = b;
                    x -= __bfloat162float(b);
                }
            }
        } else {
            float* to = reinterpret_cast<float*>(A.U + (at * A.nz + c / DC_COLS) * DC_UB) + c % DC_COLS;
#pragma unroll
            for (int t = 0; t < DC_C; ++t) to[t * 20] = u[t];
        }
    }
    odd = __syncthreads_or(odd);
    if (tid == 0) A.marked[at] = odd;
}

// ------------------------------------------------------------------ walk
template <int DP> struct WalkShape {
    static constexpr int PARTS = dc_parts(DP), KT = DP / 4 / 16;
    static constexpr int W = 0, K = PARTS, Q = 2 * PARTS, P = 3 * PARTS, U = P + DC_PB, M = U + DC_UB, E = M + DC_MB,
                         BUF = E + DC_C * 4;             // bytes of a buffer; E: the outputs' own copy of e^F_t
    static constexpr int LP = 40;                        // stride of a column of the partial sums, in tokens: float pairs of 16 lanes meet no bank twice
    static constexpr int SUMS = 4 * DC_COLS * LP * 4;    // bytes: [warp][column][LP]
    static constexpr int SF = 4 * KT * 3 * 512, UF = 2 * 3 * 512;      // bytes of the state's and of u's parts, as fragments
    static constexpr int BYTES = 2 * BUF + 2 * SUMS + 2 * (SF + UF) + 64;      // behind them six barriers and a flag
};
// c[j] and s[j] += the parts of A times those of B's four tiles of 8, each sum in the order of parts_mma6; a product of parts at a time for all
// four, so that neighbouring instructions do not wait for one another
__device__ __forceinline__ void dc_mma6x4(float (&c)[4][4], float (&s)[4][4], const uint32_t (&a)[3][4], const uint32_t (&b)[2][3][4]) {
    constexpr int pa[6] = {0, 2, 0, 1, 1, 0}, pb[6] = {0, 0, 2, 1, 0, 1};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) parts_mma(i ? s[j] : c[j], a[pa[i]], b[j >> 1][pb[i]][(j & 1) * 2], b[j >> 1][pb[i]][(j & 1) * 2 + 1]);
}
// named barriers of the walk: the four warps of the chain, the four of the outputs, and what they hand over (for either buffer)
enum { DC_BAR_CHAIN = 1, DC_BAR_OUT = 2, DC_BAR_S = 3, DC_BAR_U = 5, DC_BAR_FREE = 7 };
__device__ __forceinline__ void dc_sync(int bar, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory"); }
__device__ __forceinline__ void dc_arrive(int bar) { asm volatile("bar.arrive %0, 256;" ::"r"(bar) : "memory"); }

// grid (requests, H, slices of 16 columns), eight warps.  Four carry the chain from chunk to chunk, DP / 4 rows of the state each: W S, u, the
// new state.  Four follow a chunk behind with what nothing waits for: Q S, P u and the outputs, from the parts of the state and of u
// that the others leave in shared memory (two buffers).  The chain is what bounds the kernel (its latency: one warp a scheduler).
template <int DP>
__global__ void __launch_bounds__(256, 1) dc_walk_kernel(const DeltaChunkArgs A) {
    using Sh = WalkShape<DP>;
    constexpr int ROW = dc_row(DP), RW = DP / 4, NT = RW / 8, KT = Sh::KT, LP = Sh::LP;
    constexpr int R = 8, IS = DP / R, LAYOUT = IS * DC_COLS, PB = R * LAYOUT;      // the slot's layout
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    float* sums_w = reinterpret_cast<float*>(smem + 2 * Sh::BUF);
    float* sums_q = sums_w + Sh::SUMS / 4;
    unsigned char* frags = smem + 2 * Sh::BUF + 2 * Sh::SUMS;        // per buffer: the state's parts [warp][k][part][lane], u's [k][part][lane]
    const int first = A.firsts[blockIdx.x], h = blockIdx.y, hq = h / (A.H / A.nqk), z = blockIdx.z, dv = A.dv;
    const int4 ck = A.chunks[first];
    const int tid = threadIdx.x & 127, lane = tid & 31, wid = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
    const bool chain = threadIdx.x < 128;
    const int row0 = A.q_start[ck.x], T = A.q_start[ck.x + 1] - row0;
    if (tl_chunk_marked(A.marked, 1, first, ck.z, h, A.H)) return;       // the scan kernel's
    uint64_t* landed = reinterpret_cast<uint64_t*>(smem + Sh::BYTES - 64);       // [2] W, [2] the chain's other operands, [2] the outputs'
    volatile int* gave_up = reinterpret_cast<volatile int*>(smem + Sh::BYTES - 16);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 6; ++i) mbar_init(landed + i, 1);
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Operands are linear copies, which one thread of those that use them asks for.  W is what a chunk starts with, and is read
    // first: the next but one is asked for as soon as it is (a chunk and a half ahead).
    enum { OF_W = 0, OF_CHAIN = 2, OF_OUT = 4 };
    auto fetch = [&](int which, int c) {
        if (tid || c >= ck.z) return;
        const uint32_t to = base + (c & 1) * Sh::BUF;
        uint64_t* bar = landed + which + (c & 1);
        auto copy = [&](int at, const unsigned char* from, int bytes) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(to + at), "l"(from), "r"(bytes), "r"(smem_addr(bar)) : "memory");
        };
        const size_t at = (size_t)(first + c) * A.H + h;
        const unsigned char* k = A.K + ((size_t)(first + c) * A.nqk + hq) * 2 * Sh::PARTS;      // K, then Q
        mbar_expect_tx(bar, which == OF_W ? Sh::PARTS : which == OF_CHAIN ? Sh::PARTS + DC_UB + DC_MB : Sh::PARTS + DC_PB + DC_C * 4);
        if (which == OF_W) copy(Sh::W, A.W + at * Sh::PARTS, Sh::PARTS);
        if (which == OF_CHAIN) {
            copy(Sh::U, A.U + (at * A.nz + z) * DC_UB, DC_UB);
            copy(Sh::M, A.M + at * DC_MB, DC_MB);
            copy(Sh::K, k, Sh::PARTS);
        }
        if (which == OF_OUT) {
            copy(Sh::Q, k + Sh::PARTS, Sh::PARTS);
            copy(Sh::P, A.P + at * DC_PB, DC_PB);
            copy(Sh::E, A.M + at * DC_MB, DC_C * 4);
        }
    };
    // a wait that runs out is recorded; the walk goes on with what there is (its result is not valid), so that no other warp waits for this one
    auto wait = [&](int which, int c) { mbar_wait(landed + which + (c & 1), (c >> 1) & 1, gave_up, A.status, 51 + which / 2); };
    // this lane's addresses in fragments of two tiles: rows (tokens) of W, Q, P, and of K as it is transposed
    const uint32_t x_at = ((lane & 7) + (lane >> 4) * 8) * ROW + ((lane >> 3) & 1) * 16 + wid * RW * 2;
    const uint32_t k_at = ((lane & 7) + ((lane >> 3) & 1) * 8) * ROW + (lane >> 4) * 16 + wid * RW * 2;
    const uint32_t p_at = (wid * 8 + (lane & 7)) * DC_PROW + (lane >> 3) * 16;
    // (X S)^T over this warp's rows of the state, X the rows at `from`: [16 columns][32 tokens], to the partial sums
    auto times_state = [&](uint32_t from, const uint32_t (&sa)[KT][3][4], float* sums) {
        float big[4][4], rest[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) big[j][x] = rest[j][x] = 0.f;
#pragma unroll
        for (int k = 0; k < KT; ++k) {
            uint32_t b[2][3][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int p = 0; p < 3; ++p) parts_load4(b[j][p], from + (p * DC_C + j * 16) * ROW + x_at + k * 32);
            dc_mma6x4(big, rest, sa[k], b);
        }
        float* to = sums + (wid * DC_COLS + g) * LP + q2;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            *reinterpret_cast<float2*>(to + 8 * j) = make_float2(big[j][0] + rest[j][0], big[j][1] + rest[j][1]);
            *reinterpret_cast<float2*>(to + 8 * LP + 8 * j) = make_float2(big[j][2] + rest[j][2], big[j][3] + rest[j][3]);
        }
    };
    if (chain) {
        fetch(OF_W, 0);
        fetch(OF_CHAIN, 0);
        fetch(OF_W, 1);
        float* slot = A.state + (size_t)A.slots[ck.x] * A.slot_stride + ((size_t)h * A.nz + z) * PB;
        auto place = [&](int row, int c) { return (row % R) * LAYOUT + c * IS + row / R; };
        // S transposed: element (column g or g + 8, row wid RW + 8 i + q2 or + 1)
        float S[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int row = wid * RW + 8 * i + q2;
            S[i][0] = slot[place(row, g)]; S[i][1] = slot[place(row + 1, g)];
            S[i][2] = slot[place(row, g + 8)]; S[i][3] = slot[place(row + 1, g + 8)];
        }
        for (int c = 0; c < ck.z; ++c) {
            const int n = min(DC_C, T - c * DC_C), half = c & 1;
            dc_sync(DC_BAR_CHAIN, 128);                  // the chunk before is read
            fetch(OF_CHAIN, c + 1);
            wait(OF_W, c);
            const uint32_t at = base + half * Sh::BUF;
            const float* u0 = reinterpret_cast<const float*>(smem + half * Sh::BUF + Sh::U);
            const float* mk = reinterpret_cast<const float*>(smem + half * Sh::BUF + Sh::M);
            uint4* sf = reinterpret_cast<uint4*>(frags + half * (Sh::SF + Sh::UF)) + wid * KT * 3 * 32 + lane;
            uint4* uf = reinterpret_cast<uint4*>(frags + half * (Sh::SF + Sh::UF) + Sh::SF) + lane;
            uint32_t sa[KT][3][4];                       // S transposed as a first operand: [columns][rows]
#pragma unroll
            for (int k = 0; k < KT; ++k)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float (&v)[4] = S[2 * k + (x >> 1)];
                    parts_cut(v[(x & 1) * 2], v[(x & 1) * 2 + 1], sa[k][0][x], sa[k][1][x], sa[k][2][x]);
                }
            if (c >= 2) dc_sync(DC_BAR_FREE + half, 256);          // the outputs of chunk c - 2 have read this buffer
#pragma unroll
            for (int k = 0; k < KT; ++k)
#pragma unroll
                for (int p = 0; p < 3; ++p) sf[(k * 3 + p) * 32] = make_uint4(sa[k][p][0], sa[k][p][1], sa[k][p][2], sa[k][p][3]);
            dc_arrive(DC_BAR_S + half);
            times_state(at + Sh::W, sa, sums_w);
            dc_sync(DC_BAR_CHAIN, 128);
            fetch(OF_W, c + 2);
            wait(OF_CHAIN, c);
            // u transposed as a first operand [columns][tokens]: weighted for the end state, and as it is for the outputs
            uint32_t wa[2][3][4];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t ua[3][4];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int col = g + (x & 1) * 8, t = 16 * k + (x >> 1) * 8 + q2;
                    float2 s = make_float2(0.f, 0.f);
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const float2 v = *reinterpret_cast<const float2*>(sums_w + (w * DC_COLS + col) * LP + t);
                        s.x += v.x; s.y += v.y;
                    }
                    const float a = u0[t * 20 + col] - s.x, b = u0[(t + 1) * 20 + col] - s.y;
                    if (wid == k) parts_cut(a, b, ua[0][x], ua[1][x], ua[2][x]);
                    parts_cut(a * mk[DC_C + t], b * mk[DC_C + t + 1], wa[k][0][x], wa[k][1][x], wa[k][2][x]);
                }
                if (wid == k)                            // every warp holds all of u: two of them hand it over, half each
#pragma unroll
                    for (int p = 0; p < 3; ++p) uf[(k * 3 + p) * 32] = make_uint4(ua[p][0], ua[p][1], ua[p][2], ua[p][3]);
            }
            dc_arrive(DC_BAR_U + half);
            // the new state
            const float end = mk[n - 1];
            float big[NT][4] = {}, rest[NT][4] = {};
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if constexpr (NT == 4) {
                    uint32_t b[2][3][4];
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int p = 0; p < 3; ++p) parts_load4_trans(b[j][p], at + Sh::K + (p * DC_C + 16 * k) * ROW + k_at + j * 32);
                    dc_mma6x4(big, rest, wa[k], b);
                } else {
                    uint32_t b[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) parts_load4_trans(b[p], at + Sh::K + (p * DC_C + 16 * k) * ROW + k_at);
                    parts_mma6(big[0], rest[0], wa[k], b, 0);
                    parts_mma6(big[1], rest[1], wa[k], b, 2);
                }
            }
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int x = 0; x < 4; ++x) S[i][x] = fmaf(end, S[i][x], big[i][x] + rest[i][x]);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int row = wid * RW + 8 * i + q2;
            slot[place(row, g)] = S[i][0]; slot[place(row + 1, g)] = S[i][1];
            slot[place(row, g + 8)] = S[i][2]; slot[place(row + 1, g + 8)] = S[i][3];
        }
    } else {
        fetch(OF_OUT, 0);
    }
    for (int c = 0; !chain && c < ck.z; ++c) {
        const int n = min(DC_C, T - c * DC_C), half = c & 1;
        dc_sync(DC_BAR_OUT, 128);                        // the chunk before is read
        fetch(OF_OUT, c + 1);
        wait(OF_OUT, c);
        const uint32_t at = base + half * Sh::BUF;
        const float* grown = reinterpret_cast<const float*>(smem + half * Sh::BUF + Sh::E);
        const uint4* sf = reinterpret_cast<const uint4*>(frags + half * (Sh::SF + Sh::UF)) + wid * KT * 3 * 32 + lane;
        const uint4* uf = reinterpret_cast<const uint4*>(frags + half * (Sh::SF + Sh::UF) + Sh::SF) + lane;
        dc_sync(DC_BAR_S + half, 256);
        {
            uint32_t sa[KT][3][4];
#pragma unroll
            for (int k = 0; k < KT; ++k)
#pragma unroll
                for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(sa[k][p]) = sf[(k * 3 + p) * 32];
            times_state(at + Sh::Q, sa, sums_q);
        }
        dc_sync(DC_BAR_OUT, 128);
        dc_sync(DC_BAR_U + half, 256);
        // outputs of tokens 8 wid ..
        float big[4] = {}, rest[4] = {};
        uint32_t b[3][4], ua[2][3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) parts_load4(b[p], at + Sh::P + p * DC_C * DC_PROW + p_at);
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(ua[k][p]) = uf[(k * 3 + p) * 32];
        if (c + 2 < ck.z) dc_arrive(DC_BAR_FREE + half);
        parts_mma6(big, rest, ua[0], b, 0);
        parts_mma6(big, rest, ua[1], b, 2);
        const int t = 8 * wid + q2;
        const float2 e = *reinterpret_cast<const float2*>(grown + t);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            float2 s = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float2 v = *reinterpret_cast<const float2*>(sums_q + (w * DC_COLS + g + 8 * x) * LP + t);
                s.x += v.x; s.y += v.y;
            }
            const int col = z * DC_COLS + g + 8 * x;
            if (col < dv) {
                float* to = A.out + (size_t)(row0 + c * DC_C + t) * A.H * dv + (size_t)h * dv + col;
                if (t < n) to[0] = fmaf(e.x, s.x, big[2 * x] + rest[2 * x]);
                if (t + 1 < n) to[(size_t)A.H * dv] = fmaf(e.y, s.y, big[2 * x + 1] + rest[2 * x + 1]);
            }
        }
    }
    if (*gave_up) {                                      // give copies in flight time to land before the shared memory is handed on
        const long long start = clock64();
        while (clock64() - start < 2000000LL) { }
    }
}

constexpr int DC_DV_MAX = 1024;          // V of a chunk lies in shared memory beside K and Q

template <int DP>
static int dc_launch(DeltaChunkArgs A, unsigned char* scratch, int* marked, int n_chunks, int requests, cudaStream_t stream) {
    using Sh = WalkShape<DP>;
    constexpr int row_bytes = 2 * DC_C * (DP + 4) * 4;
    static bool prepare[TL_MAX_DEVICES] = {}, walk[TL_MAX_DEVICES] = {};
    int e = tl_raise_smem(dc_prepare_kernel<DP>, prepare, row_bytes + DC_C * DC_DV_MAX * 4);
    if (!e) e = tl_raise_smem(dc_walk_kernel<DP>, walk, Sh::BYTES);
    if (e) return e;
    if (A.status == nullptr) return 1;                   // the walk's waits are bounded: it has to be able to say that one ran out
    const size_t ch = (size_t)n_chunks * A.H;
    A.W = scratch;
    A.P = A.W + ch * Sh::PARTS;
    A.M = A.P + ch * DC_PB;
    A.U = A.M + ch * DC_MB;
    A.K = A.U + ch * A.nz * DC_UB;
    A.marked = marked;
    dc_prepare_kernel<DP><<<dim3(n_chunks, A.H), DC_PREP, row_bytes + DC_C * A.dv * 4, stream>>>(A);
    if ((e = tl_launch_status())) return e;
    dc_walk_kernel<DP><<<dim3(requests, A.H, A.nz), 256, Sh::BYTES, stream>>>(A);
    return tl_launch_status();
}

TL_EXPORT int tl_delta_chunk() { return DC_C; }
// Bytes of scratch a chunk; 0: these sizes run token by token (heads of up to 32, whose state has another layout, and wide ones,
// whose operands fill shared memory once).
TL_EXPORT int tl_delta_chunk_bytes(int H, int nqk, int d, int dv) {
    if (d <= 32 || d > 128 || (d & 3) || (dv & 3) || dv > DC_DV_MAX) return 0;
    const int parts = d <= 64 ? dc_parts(64) : dc_parts(128);
    return H * (parts + DC_PB + DC_MB + (dv + DC_COLS - 1) / DC_COLS * DC_UB) + nqk * 2 * parts;
}

// scratch: `tl_delta_chunk_bytes` bytes a chunk; marked: int [n_chunks, H], for the scan kernel (tiles: 1); status: device int.  The offsets and the stride are multiples of 4, the pointers 16-byte aligned.
TL_EXPORT int tl_delta_chunks(const float* qkv, int stride, int q_off, int k_off, int v_off, const float* gates, int gate_stride,
                              const float* A_log, const float* dt_bias, float* state, long long slot_stride, const int* q_start,
                              const int* slots, const int* chunks, int n_chunks, const int* firsts, int requests, void* scratch, int* marked, float* out,
                              int H, int nqk, int d, int dv, cudaStream_t stream, int* status = nullptr) {
    if (n_chunks <= 0 || H <= 0) return 0;
    if (H > 65535 || nqk < 1 || H % nqk || !tl_delta_chunk_bytes(H, nqk, d, dv) || ((stride | q_off | k_off | v_off) & 3) ||
        ((((uintptr_t)qkv) | ((uintptr_t)scratch) | ((uintptr_t)out)) & 15)) return 1;
    const DeltaChunkArgs A{qkv, stride, q_off, k_off, v_off, gates, gate_stride, A_log, dt_bias, state, slot_stride, q_start, slots,
                           (const int4*)chunks, firsts, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, out, H, nqk, d, dv, (dv + DC_COLS - 1) / DC_COLS, status};
    if (d <= 64) return dc_launch<64>(A, (unsigned char*)scratch, marked, n_chunks, requests, stream);
    return dc_launch<128>(A, (unsigned char*)scratch, marked, n_chunks, requests, stream);
}
