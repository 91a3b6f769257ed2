// prima.cpp_b200/csrc/delta.cu — the gated delta rule with a decay per head and key channel for the usual head sizes (declaration and semantics:
// layers.h, GatedLinParams; any other size runs through the kernels of gated.cu).  Keys, queries, decays, step sizes, values and the state are fp32
// in either compute type.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "launch.h"
#include "layers.h"
#include "mixers.cuh"

namespace pb {
namespace {

// ---- head sizes N = 32, 64, 128, 256 ----
//   S <- diag(g_t) S,  u = beta_t (v_t - S^T k_t),  S <- S + k_t u^T,  y_t = S^T q_t
// CTA = one head x 16 value columns of one entry.  LN = N / 8 lanes share a pair of columns: a lane keeps S[n][2 columns] for 8 n (four
// consecutive ones in either half of the key size), so the 16-byte loads of a token's q, k, g rows from shared memory serve two columns.  Tokens
// arrive in chunks of 16 through two cp.async stages.  The chain from token to token is decay, product with the key, its sum over the lanes (the
// two columns' shuffles side by side) and the rank-one write; the read-out with the query leaves it aside: a full chunk keeps its 32 partial sums
// (16 tokens x 2 columns) in registers and sums them together (30 shuffles at most instead of 32 log2(LN)).
constexpr int DS_CHUNK = 16, DS_COLS = 16, DS_STAGES = 2, DS_NREG = 8;
template <int N> constexpr int ds_stage_floats() { return DS_CHUNK * (3 * N + DS_COLS + 1); }

template <int N>
__global__ void __launch_bounds__(DS_COLS / 2 * (N / DS_NREG)) k_delta_scan(GatedLinIO io, const int32_t * __restrict__ slot, const int32_t * __restrict__ off,
                                                                           GatedLinParams p, float * __restrict__ state, int64_t slot_stride, float * __restrict__ y) {
    pdl_enter();
    extern __shared__ __align__(16) float sm[];   // [stages][ q [16][N] | k [16][N] | g [16][N] | v [16][16] | beta [16] ]
    constexpr int LN = N / DS_NREG, NT = DS_COLS / 2 * LN, STAGE = ds_stage_floats<N>();
    const int P = p.vdim, inner = p.heads * P, ptiles = (P + DS_COLS - 1) / DS_COLS;
    const int h = blockIdx.x / ptiles, pt = blockIdx.x - h * ptiles, e = blockIdx.y;
    const int hk = h / (p.heads / p.qk_heads);
    const int tid = threadIdx.x, lane = tid & 31, ng = tid % LN, cp = tid / LN;   // this thread: n = n_of(0..7), columns 2 cp, 2 cp + 1 of the tile
    auto n_of = [&](int j) { return (j >> 2) * (N / 2) + 4 * ng + (j & 3); };
    const int col = pt * DS_COLS + 2 * cp;
    const bool ok0 = col < P, ok1 = col + 1 < P;
    float * gst = state + (int64_t) slot[e] * slot_stride + (int64_t) h * N * P;
    const int t0 = off[e], n = off[e + 1] - t0;
    auto stage_in = [&](int c0, float * st) {
        const int nc = min(DS_CHUNK, n - c0);
        constexpr int Q = N / 4;                     // 16-byte pieces of a row
#pragma unroll 4
        for (int i = tid; i < 3 * DS_CHUNK * Q; i += NT) {
            const int which = i / (DS_CHUNK * Q), rem = i % (DS_CHUNK * Q), tt = rem / Q, q = rem % Q;
            const int64_t tok = t0 + c0 + min(tt, nc - 1);
            const float * src = which == 0 ? io.q + tok * io.ldq + hk * N : which == 1 ? io.k + tok * io.ldk + hk * N : io.decay + tok * io.ldd + h * N;
            cp_async16(st + which * DS_CHUNK * N + tt * N + 4 * q, src + 4 * q, tt < nc);
        }
        for (int i = tid; i < DS_CHUNK * (DS_COLS / 4); i += NT) {
            const int tt = i / (DS_COLS / 4), q = i % (DS_COLS / 4), c = pt * DS_COLS + 4 * q;
            const bool ok = tt < nc && c < P;        // P is a multiple of 4
            cp_async16(st + 3 * DS_CHUNK * N + tt * DS_COLS + 4 * q, ok ? io.v + (int64_t) (t0 + c0 + tt) * io.ldv + h * P + c : io.v, ok);
        }
        if (tid < DS_CHUNK) {
            const bool ok = tid < nc;
            cp_async4(st + DS_CHUNK * (3 * N + DS_COLS) + tid, ok ? io.beta + (int64_t) (t0 + c0 + tid) * io.ldb + h : io.beta, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (n > 0) stage_in(0, sm);
    float S0[DS_NREG], S1[DS_NREG];
#pragma unroll
    for (int j = 0; j < DS_NREG; j++) {
        const float * g = gst + (int64_t) n_of(j) * P + col;
        S0[j] = ok0 ? g[0] : 0.f;
        S1[j] = ok1 ? g[1] : 0.f;
    }
    for (int c0 = 0, it = 0; c0 < n; c0 += DS_CHUNK, it++) {
        const int nc = min(DS_CHUNK, n - c0);
        float * st = sm + (it & 1) * STAGE;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                             // the stage is complete, and everybody is done with the other one
        if (c0 + DS_CHUNK < n) stage_in(c0 + DS_CHUNK, sm + ((it + 1) & 1) * STAGE);
        const float * Qs = st, * Ks = st + DS_CHUNK * N, * Gs = st + 2 * DS_CHUNK * N, * Vs = st + 3 * DS_CHUNK * N, * Bs = Vs + DS_CHUNK * DS_COLS;
        auto token = [&](int tt, float & y0, float & y1) {
            float kk[DS_NREG], x0 = 0.f, x1 = 0.f;
#pragma unroll
            for (int j = 0; j < DS_NREG; j += 4) {
                const int o = tt * N + n_of(j);
                const float4 k = *reinterpret_cast<const float4 *>(Ks + o), g = *reinterpret_cast<const float4 *>(Gs + o);
                const float gg[4] = {g.x, g.y, g.z, g.w};
                kk[j] = k.x; kk[j + 1] = k.y; kk[j + 2] = k.z; kk[j + 3] = k.w;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    S0[j + i] *= gg[i];
                    S1[j + i] *= gg[i];
                    x0 = fmaf(S0[j + i], kk[j + i], x0);
                    x1 = fmaf(S1[j + i], kk[j + i], x1);
                }
            }
#pragma unroll
            for (int o = 1; o < LN; o <<= 1) {
                x0 += __shfl_xor_sync(0xffffffffu, x0, o);
                x1 += __shfl_xor_sync(0xffffffffu, x1, o);
            }
            const float2 v = *reinterpret_cast<const float2 *>(Vs + tt * DS_COLS + 2 * cp);
            const float b = Bs[tt], u0 = b * (v.x - x0), u1 = b * (v.y - x1);
            y0 = y1 = 0.f;
#pragma unroll
            for (int j = 0; j < DS_NREG; j += 4) {
                const float4 q = *reinterpret_cast<const float4 *>(Qs + tt * N + n_of(j));
                const float qq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    S0[j + i] = fmaf(kk[j + i], u0, S0[j + i]);
                    S1[j + i] = fmaf(kk[j + i], u1, S1[j + i]);
                    y0 = fmaf(S0[j + i], qq[i], y0);
                    y1 = fmaf(S1[j + i], qq[i], y1);
                }
            }
        };
        if (nc == DS_CHUNK) {
            constexpr int M = 2 * DS_CHUNK, KEEP = M / LN;   // partial sums, and how many whole ones a lane ends up with
            float acc[M];                                    // value token * 2 + column
#pragma unroll
            for (int tt = 0; tt < DS_CHUNK; tt++) token(tt, acc[2 * tt], acc[2 * tt + 1]);
            joint_sum<M, LN / 2>(acc, lane);
#pragma unroll
            for (int i = 0; i < KEEP; i++) {
                const int idx = ng * KEEP + i, tt = idx >> 1, c = idx & 1;
                if (c == 0 ? ok0 : ok1) y[(int64_t) (t0 + c0 + tt) * inner + h * P + col + c] = acc[i];
            }
        } else {
            for (int tt = 0; tt < nc; tt++) {
                float y0, y1;
                token(tt, y0, y1);
#pragma unroll
                for (int o = 1; o < LN; o <<= 1) {
                    y0 += __shfl_xor_sync(0xffffffffu, y0, o);
                    y1 += __shfl_xor_sync(0xffffffffu, y1, o);
                }
                if (ng == 0 && ok0) y[(int64_t) (t0 + c0 + tt) * inner + h * P + col] = y0;
                if (ng == 0 && ok1) y[(int64_t) (t0 + c0 + tt) * inner + h * P + col + 1] = y1;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < DS_NREG; j++) {
        float * g = gst + (int64_t) n_of(j) * P + col;
        if (ok0) g[0] = S0[j];
        if (ok1) g[1] = S1[j];
    }
}

// ---- the same in blocks of four tokens, for entries of at least so many ----
// Within a block everything refers to the state S in front of it.  With G_t the product of the decays up to token t of the block and w_st = k_s times the decays
// behind token s up to t (products only, no quotient: a decay may be zero),
//   x_t = S^T (G_t k_t),   u_t = beta_t (v_t - x_t - sum_{s<t} (k_t . w_st) u_s),   y_t = S^T (G_t q_t) + sum_{s<=t} (q_t . w_st) u_s,   S <- diag(G_4) S + sum_s w_s4 u_s^T
// so a block costs one sum over the lanes and one pass over the state instead of four.  What does not depend on the columns (G_t k_t, G_t q_t, w_s4, G_4 and the 16
// scalars) is prepared a chunk of 16 tokens ahead by a warp a block, the loads another chunk ahead by four more warps; the others hold the state as above.
// Bound: some 260 instructions a block of the one warp to a scheduler that walks it, a chain of 1150 clocks; preparation alone takes 30 us of a prompt, loads 19.
// 512 tokens, 16 heads of 128 x 128: 101 us token by token (360 clocks each), 78 in blocks.  With a column to eight lanes, or four columns to a whole warp, instead of
// two to half a warp, 150 and 106; products one by one instead of in pairs 84.
constexpr int DB_BLOCK = 4, DB_BLOCKS = DS_CHUNK / DB_BLOCK, DB_LOADERS = 128, DB_PRODUCERS = 32 * DB_BLOCKS + DB_LOADERS;
template <int N> struct DbRaw { float q[DS_CHUNK][N], k[DS_CHUNK][N], g[DS_CHUNK][N]; };
template <int N> struct DbReady { float q[DS_CHUNK][N], k[DS_CHUNK][N], w[DS_CHUNK][N], g[DB_BLOCKS][N], dots[DB_BLOCKS][16]; };
struct DbVals { float v[DS_CHUNK][DS_COLS], beta[DS_CHUNK]; };
template <int N> struct __align__(16) DbSmem { DbRaw<N> raw[2]; DbReady<N> ready[2]; DbVals vals[3]; };

// E = N / 32 neighbouring floats of a lane
template <int E> __device__ __forceinline__ void db_load(const float * p, float (&x)[E]) {
    if constexpr (E == 1) x[0] = p[0];
    else if constexpr (E == 2) { const float2 a = *reinterpret_cast<const float2 *>(p); x[0] = a.x; x[1] = a.y; }
    else {
#pragma unroll
        for (int i = 0; i < E; i += 4) { const float4 a = *reinterpret_cast<const float4 *>(p + i); x[i] = a.x; x[i + 1] = a.y; x[i + 2] = a.z; x[i + 3] = a.w; }
    }
}
template <int E> __device__ __forceinline__ void db_store(float * p, const float (&x)[E]) {
    if constexpr (E == 1) p[0] = x[0];
    else if constexpr (E == 2) *reinterpret_cast<float2 *>(p) = make_float2(x[0], x[1]);
    else {
#pragma unroll
        for (int i = 0; i < E; i += 4) *reinterpret_cast<float4 *>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    }
}
// two floats in a register pair: one instruction for two products
using F2 = uint64_t;
__device__ __forceinline__ F2 f2_pair(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float2 f2_split(F2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
// block b of a chunk: scalars k_t . w_st of (2,1) (3,1) (3,2) (4,1) (4,2) (4,3) in [0, 6), q_t . w_st of (1,1) (2,1) (2,2) ... (4,4) in [6, 16).  Tokens from nc on
// leave the state alone.
template <int N>
__device__ __forceinline__ void db_prepare(const DbRaw<N> & in, DbReady<N> & out, int b, int nc, int lane) {
    constexpr int E = N / 32;
    float w[DB_BLOCK][E], g_all[E], acc[16];
#pragma unroll
    for (int i = 0; i < 16; i++) acc[i] = 0.f;
#pragma unroll
    for (int t = 0; t < DB_BLOCK; t++) {
        const int row = DB_BLOCK * b + t;
        float q[E], g[E], x[E];
        db_load<E>(&in.q[row][E * lane], q);
        db_load<E>(&in.k[row][E * lane], w[t]);
        db_load<E>(&in.g[row][E * lane], g);
#pragma unroll
        for (int i = 0; i < E; i++) {
            if (row >= nc) g[i] = 1.f;
            g_all[i] = t == 0 ? g[i] : g_all[i] * g[i];
            x[i] = w[t][i] * g_all[i];
        }
        db_store<E>(&out.k[row][E * lane], x);
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = q[i] * g_all[i];
        db_store<E>(&out.q[row][E * lane], x);
#pragma unroll
        for (int s = 0; s <= t; s++)
#pragma unroll
            for (int i = 0; i < E; i++) {
                if (s < t) {
                    w[s][i] *= g[i];
                    acc[t * (t - 1) / 2 + s] = fmaf(w[t][i], w[s][i], acc[t * (t - 1) / 2 + s]);
                }
                acc[6 + t * (t + 1) / 2 + s] = fmaf(q[i], w[s][i], acc[6 + t * (t + 1) / 2 + s]);
            }
    }
#pragma unroll
    for (int s = 0; s < DB_BLOCK; s++) db_store<E>(&out.w[DB_BLOCK * b + s][E * lane], w[s]);
    db_store<E>(&out.g[b][E * lane], g_all);
    joint_sum<16, 16>(acc, lane);
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    if ((lane & 1) == 0) out.dots[b][lane >> 1] = acc[0];
}

template <int N>
__global__ void __launch_bounds__(DS_COLS / 2 * (N / DS_NREG) + DB_PRODUCERS) k_delta_blocks(GatedLinIO io, const int32_t * __restrict__ slot, const int32_t * __restrict__ off,
                                                                                            GatedLinParams p, float * __restrict__ state, int64_t slot_stride,
                                                                                            float * __restrict__ y) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t db_raw[];
    DbSmem<N> & sm = *reinterpret_cast<DbSmem<N> *>(db_raw);
    constexpr int LN = N / DS_NREG, NT = DS_COLS / 2 * LN;
    const int P = p.vdim, inner = p.heads * P, ptiles = (P + DS_COLS - 1) / DS_COLS;
    const int h = blockIdx.x / ptiles, pt = blockIdx.x - h * ptiles, e = blockIdx.y, hk = h / (p.heads / p.qk_heads);
    const int tid = threadIdx.x, lane = tid & 31;
    const int t0 = off[e], n = off[e + 1] - t0, chunks = (n + DS_CHUNK - 1) / DS_CHUNK;
    if (tid >= NT) {
        if (tid < NT + 32 * DB_BLOCKS) {             // ---- a warp prepares a block of every chunk ----
            const int b = (tid - NT) >> 5;
            for (int c = 0; c <= chunks; c++) {
                if (c < chunks) {
                    asm volatile("bar.sync 1, %0;" ::"n"(DB_PRODUCERS) : "memory");
                    db_prepare<N>(sm.raw[c & 1], sm.ready[c & 1], b, n - c * DS_CHUNK, lane);
                }
                __syncthreads();
            }
            return;
        }
        // ---- loads: chunk c + 2 is asked for while c + 1 is prepared and c met by the state ----
        const int pid = tid - NT - 32 * DB_BLOCKS;
        auto fetch = [&](int c) {
            if (c < chunks) {
                const int c0 = c * DS_CHUNK, nc = min(DS_CHUNK, n - c0);
                DbRaw<N> & raw = sm.raw[c & 1];
                DbVals & vals = sm.vals[c % 3];
                constexpr int Q = N / 4;             // 16-byte pieces of a row
#pragma unroll 8
                for (int i = pid; i < DS_CHUNK * Q; i += DB_LOADERS) {
                    const int tt = i / Q, d = i % Q * 4;
                    const int64_t tok = t0 + c0 + min(tt, nc - 1);
                    cp_async16(&raw.q[tt][d], io.q + tok * io.ldq + hk * N + d, tt < nc);
                    cp_async16(&raw.k[tt][d], io.k + tok * io.ldk + hk * N + d, tt < nc);
                    cp_async16(&raw.g[tt][d], io.decay + tok * io.ldd + h * N + d, tt < nc);
                }
                if (pid < DS_CHUNK * (DS_COLS / 4)) {
                    const int tt = pid / (DS_COLS / 4), d = pid % (DS_COLS / 4) * 4, col = pt * DS_COLS + d;
                    const bool ok = tt < nc && col < P;   // P is a multiple of 4
                    cp_async16(&vals.v[tt][d], ok ? io.v + (int64_t) (t0 + c0 + tt) * io.ldv + h * P + col : io.v, ok);
                }
                if (pid < DS_CHUNK) cp_async4(&vals.beta[pid], pid < nc ? io.beta + (int64_t) (t0 + c0 + pid) * io.ldb + h : io.beta, pid < nc);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(0);
        for (int c = 0; c <= chunks; c++) {
            fetch(c + 1);
            if (c < chunks) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                asm volatile("bar.arrive 1, %0;" ::"n"(DB_PRODUCERS) : "memory");
            }
            __syncthreads();
        }
        return;
    }
    // ---- state ----
    const int ng = tid % LN, cp = tid / LN;          // this thread: n = n_of(0..7), columns 2 cp, 2 cp + 1 of the tile
    auto n_of = [&](int j) { return (j >> 2) * (N / 2) + 4 * ng + (j & 3); };
    const int col = pt * DS_COLS + 2 * cp;
    const bool ok0 = col < P, ok1 = col + 1 < P;
    float * gst = state + (int64_t) slot[e] * slot_stride + (int64_t) h * N * P;
    F2 S0[DS_NREG / 2], S1[DS_NREG / 2];             // neighbouring n of the first, the second column
#pragma unroll
    for (int j = 0; j < DS_NREG; j += 2) {
        const float * g = gst + (int64_t) n_of(j) * P + col;
        S0[j / 2] = f2_pair(ok0 ? g[0] : 0.f, ok0 ? g[P] : 0.f);
        S1[j / 2] = f2_pair(ok1 ? g[1] : 0.f, ok1 ? g[P + 1] : 0.f);
    }
    auto sum = [](F2 v) { const float2 x = f2_split(v); return x.x + x.y; };
    __syncthreads();
    for (int c = 0; c < chunks; c++) {
        const DbReady<N> & in = sm.ready[c & 1];
        const DbVals & vals = sm.vals[c % 3];
        constexpr int M = 2 * DS_CHUNK, KEEP = M / LN;   // partial results, and how many whole ones a lane ends up with
        float acc[M];                                    // value token * 2 + column
#pragma unroll
        for (int b = 0; b < DB_BLOCKS; b++) {
            float x[2 * DB_BLOCK];
#pragma unroll
            for (int t = 0; t < DB_BLOCK; t++) {
                const int row = DB_BLOCK * b + t;
                F2 x0 = 0, x1 = 0, y0 = 0, y1 = 0;   // two zeros each
#pragma unroll
                for (int j = 0; j < DS_NREG; j += 4) {
                    const ulonglong2 k4 = *reinterpret_cast<const ulonglong2 *>(&in.k[row][n_of(j)]), q4 = *reinterpret_cast<const ulonglong2 *>(&in.q[row][n_of(j)]);
                    x0 = f2_fma(S0[j / 2 + 1], k4.y, f2_fma(S0[j / 2], k4.x, x0));
                    x1 = f2_fma(S1[j / 2 + 1], k4.y, f2_fma(S1[j / 2], k4.x, x1));
                    y0 = f2_fma(S0[j / 2 + 1], q4.y, f2_fma(S0[j / 2], q4.x, y0));
                    y1 = f2_fma(S1[j / 2 + 1], q4.y, f2_fma(S1[j / 2], q4.x, y1));
                }
                x[2 * t] = sum(x0); x[2 * t + 1] = sum(x1);
                acc[2 * row] = sum(y0); acc[2 * row + 1] = sum(y1);
            }
            // the block's eight sums over the lanes together, then to all lanes
            joint_sum<2 * DB_BLOCK, LN / 2>(x, lane);
            constexpr int SPREAD = LN > 8 ? LN / 8 : 1, HELD = LN < 8 ? 8 / LN : 1;
#pragma unroll
            for (int o = SPREAD / 2; o > 0; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
            float u[2 * DB_BLOCK];
#pragma unroll
            for (int i = 0; i < 2 * DB_BLOCK; i++) u[i] = __shfl_sync(0xffffffffu, x[i % HELD], i / HELD * SPREAD, LN);
            float d[16];
#pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4 *>(d + i) = *reinterpret_cast<const float4 *>(&in.dots[b][i]);
#pragma unroll
            for (int t = 0; t < DB_BLOCK; t++) {
                const int row = DB_BLOCK * b + t;
                const float2 v = *reinterpret_cast<const float2 *>(&vals.v[row][2 * cp]);
                const float beta = vals.beta[row];
                float r0 = v.x - u[2 * t], r1 = v.y - u[2 * t + 1];
#pragma unroll
                for (int s = 0; s < t; s++) {
                    r0 = fmaf(-d[t * (t - 1) / 2 + s], u[2 * s], r0);
                    r1 = fmaf(-d[t * (t - 1) / 2 + s], u[2 * s + 1], r1);
                }
                u[2 * t] = beta * r0; u[2 * t + 1] = beta * r1;
                if (ng == 0) {
#pragma unroll
                    for (int s = 0; s <= t; s++) {
                        acc[2 * row] = fmaf(d[6 + t * (t + 1) / 2 + s], u[2 * s], acc[2 * row]);
                        acc[2 * row + 1] = fmaf(d[6 + t * (t + 1) / 2 + s], u[2 * s + 1], acc[2 * row + 1]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < DS_NREG; j += 4) {
                const ulonglong2 g4 = *reinterpret_cast<const ulonglong2 *>(&in.g[b][n_of(j)]);
                S0[j / 2] = f2_mul(S0[j / 2], g4.x); S0[j / 2 + 1] = f2_mul(S0[j / 2 + 1], g4.y);
                S1[j / 2] = f2_mul(S1[j / 2], g4.x); S1[j / 2 + 1] = f2_mul(S1[j / 2 + 1], g4.y);
            }
#pragma unroll
            for (int s = 0; s < DB_BLOCK; s++) {
                const F2 u0 = f2_pair(u[2 * s], u[2 * s]), u1 = f2_pair(u[2 * s + 1], u[2 * s + 1]);
#pragma unroll
                for (int j = 0; j < DS_NREG; j += 4) {
                    const ulonglong2 w4 = *reinterpret_cast<const ulonglong2 *>(&in.w[DB_BLOCK * b + s][n_of(j)]);
                    S0[j / 2] = f2_fma(w4.x, u0, S0[j / 2]); S0[j / 2 + 1] = f2_fma(w4.y, u0, S0[j / 2 + 1]);
                    S1[j / 2] = f2_fma(w4.x, u1, S1[j / 2]); S1[j / 2 + 1] = f2_fma(w4.y, u1, S1[j / 2 + 1]);
                }
            }
        }
        joint_sum<M, LN / 2>(acc, lane);
        const int nc = min(DS_CHUNK, n - c * DS_CHUNK);
#pragma unroll
        for (int i = 0; i < KEEP; i++) {
            const int idx = ng * KEEP + i, tt = idx >> 1, cc = idx & 1;
            if (tt < nc && (cc == 0 ? ok0 : ok1)) y[(int64_t) (t0 + c * DS_CHUNK + tt) * inner + h * P + col + cc] = acc[i];
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < DS_NREG; j += 2) {
        float * g = gst + (int64_t) n_of(j) * P + col;
        const float2 a = f2_split(S0[j / 2]), b = f2_split(S1[j / 2]);
        if (ok0) { g[0] = a.x; g[P] = a.y; }
        if (ok1) { g[1] = b.x; g[P + 1] = b.y; }
    }
}

// ---- one token per entry ----
// CTA = one head x 32 value columns of one entry, a lane to a column, a warp to N / 8 key entries: the state comes and goes in whole lines, all of a thread's loads at
// once, and the two sums over the keys meet in shared memory.  Bound: the state's way from memory and back.  16 heads of 128 x 128, us: one entry 4.0 with the scan
// above, 2.4 here; eight (17 MB) 18.7, 5.2.
constexpr int DT_WARPS = 8;
template <int N>
__global__ void __launch_bounds__(DT_WARPS * 32) k_delta_token(GatedLinIO io, const int32_t * __restrict__ slot, const int32_t * __restrict__ off, GatedLinParams p,
                                                               float * state, int64_t slot_stride, float * y) {
    constexpr int ROWS = N / DT_WARPS;
    __shared__ float ks[N], gs[N], qs[N], part[2][DT_WARPS][32];
    pdl_enter();
    const int P = p.vdim, ptiles = (P + 31) / 32, h = blockIdx.x / ptiles, pt = blockIdx.x - h * ptiles, e = blockIdx.y, hk = h / (p.heads / p.qk_heads);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = pt * 32 + lane;
    const bool ok = col < P;
    const int64_t t = off[e];
    float * S0 = state + (int64_t) slot[e] * slot_stride + ((int64_t) h * N + warp * ROWS) * P + col;
    float S[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; i++) S[i] = ok ? S0[(int64_t) i * P] : 0.f;
    for (int i = tid; i < N; i += DT_WARPS * 32) {
        ks[i] = io.k[t * io.ldk + hk * N + i];
        gs[i] = io.decay[t * io.ldd + h * N + i];
        qs[i] = io.q[t * io.ldq + hk * N + i];
    }
    const float v = ok ? io.v[t * io.ldv + h * P + col] : 0.f, beta = io.beta[t * io.ldb + h];
    __syncthreads();
    float x = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        S[i] *= gs[warp * ROWS + i];
        x = fmaf(S[i], ks[warp * ROWS + i], x);
    }
    part[0][warp][lane] = x;
    __syncthreads();
    x = 0.f;
#pragma unroll
    for (int w = 0; w < DT_WARPS; w++) x += part[0][w][lane];
    const float u = beta * (v - x);
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        S[i] = fmaf(ks[warp * ROWS + i], u, S[i]);
        o = fmaf(S[i], qs[warp * ROWS + i], o);
        if (ok) S0[(int64_t) i * P] = S[i];
    }
    part[1][warp][lane] = o;
    __syncthreads();
    if (warp == 0 && ok) {
        o = 0.f;
#pragma unroll
        for (int w = 0; w < DT_WARPS; w++) o += part[1][w][lane];
        y[t * ((int64_t) p.heads * P) + h * P + col] = o;
    }
}

template <int N>
int delta_scan_launch(const GatedLinIO & io, const BatchView & b, const GatedLinParams & p, float * state, int64_t slot_stride, float * y, cudaStream_t st) {
    if (b.max_n == 1)
        return ck_launch([&] {
            launch_dep(k_delta_token<N>, dim3((unsigned) (p.heads * ((p.vdim + 31) / 32)), (unsigned) b.n_entries), dim3(DT_WARPS * 32), 0, st, io, b.slot, b.off, p, state, slot_stride, y);
        });
    const dim3 grid((unsigned) (p.heads * ((p.vdim + DS_COLS - 1) / DS_COLS)), (unsigned) b.n_entries);
    // Blocks of four where every CTA has an SM of its own: 384 threads and 106 KB a CTA leave room for one or two, and with more CTAs than SMs it is throughput that
    // counts (eight prompts of 9 to 128 tokens: 26 us token by token, 52 in blocks).  Entries of fewer tokens are not a block.  The two forms round differently: a prompt's
    // last bits depend on how many others share its batch.
    if (b.max_n >= DB_BLOCK && (int64_t) grid.x * grid.y <= sm_count()) {
        const int rc = raise_smem(k_delta_blocks<N>, sizeof(DbSmem<N>));
        if (rc) return rc;
        return ck_launch([&] { launch_dep(k_delta_blocks<N>, dim3(grid), dim3(DS_COLS / 2 * (N / DS_NREG) + DB_PRODUCERS), sizeof(DbSmem<N>), st, io, b.slot, b.off, p, state, slot_stride, y); });
    }
    const size_t smem = (size_t) DS_STAGES * ds_stage_floats<N>() * sizeof(float);
    const int rc = raise_smem(k_delta_scan<N>, smem);
    if (rc) return rc;
    return ck_launch([&] { launch_dep(k_delta_scan<N>, dim3(grid), dim3(DS_COLS / 2 * (N / DS_NREG)), smem, st, io, b.slot, b.off, p, state, slot_stride, y); });
}

}  // namespace

// 1: the kernel above takes this recurrence (a head size it is built for, rows that 16-byte copies can read)
int delta_scan_ok(const GatedLinIO & io, const GatedLinParams & p) {
    auto al = [](const float * q, int64_t ld) { return ((uintptr_t) q & 15) == 0 && ld % 4 == 0; };
    return p.delta && p.decay_per_channel && (p.dim == 32 || p.dim == 64 || p.dim == 128 || p.dim == 256) && p.vdim % 4 == 0 && al(io.q, io.ldq) &&
           al(io.k, io.ldk) && al(io.v, io.ldv) && al(io.decay, io.ldd);
}
int launch_delta_scan(const GatedLinIO & io, const BatchView & b, const GatedLinParams & p, float * state, int64_t slot_stride, float * y, cudaStream_t st) {
    if (p.dim == 32) return delta_scan_launch<32>(io, b, p, state, slot_stride, y, st);
    if (p.dim == 64) return delta_scan_launch<64>(io, b, p, state, slot_stride, y, st);
    if (p.dim == 128) return delta_scan_launch<128>(io, b, p, state, slot_stride, y, st);
    if (p.dim == 256) return delta_scan_launch<256>(io, b, p, state, slot_stride, y, st);
    return (int) cudaErrorInvalidValue;
}

}  // namespace pb
