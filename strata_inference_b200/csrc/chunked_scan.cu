// The recurrences of recurrent.cu over prompts, 64 tokens at a time, in 32-bit.
//
// Token by token (recurrent_scan_kernel) a sequence is a chain of dependent steps of about 600 cycles:
// 2 048 tokens of 8 heads of 128 x 256 take 0.65 to 1.0 ms with a tenth of the chip's arithmetic.  Within
// a chunk of C tokens the chain unrolls: with D(t, s) = a_{s+1} .. a_t and A_t = a_1 .. a_t,
//
//     o_t = A_t S^T q_t + sum_{s <= t} D(t, s) (q_t . k_s) u_s         S: the matrix before the chunk
//     S'  = A_C S + sum_s D(C, s) k_s u_s^T
//     u_t = b_t v_t                                                    memory, retention, gated
//     u_t = b_t (v_t - A_t S^T k_t - sum_{s < t} D(t, s) (k_t . k_s) u_s)    delta rule
//
// The delta rule's system is unit lower triangular, (I + L) U = b V - b A K S: with T = (I + L)^-1,
// U = U0 - W S, U0 = T (b V), W = T (b A K).  What does not contain S is made for all chunks at once, and so
// are the outputs once every chunk's S is known; between them lies the walk from chunk to chunk:
//
//   delta rule    chunk_prepare   T, W, U0, Kd = D(C, .) K
//                 chunk_walk      U = U0 - W S,  S' = A_C S + Kd^T U, a block per 16 columns; keeps U and every S
//   the others    chunk_update    B = Kd^T (b V)
//                 chunk_pass      S' = A_C S + B, element by element; keeps every S
//   all           chunk_out       P[t, s] = D(t, s) (q_t . k_s);  O = P U + A Q S
//
// Measured (8 heads of 128 x 256, token by token -> in chunks): one sequence of 2 048 tokens, delta rule 702 -> 255 us,
// gated 639 -> 163; of 300 tokens 111 -> 93 and 101 -> 60; of 160 tokens 63 -> 87 and 58 -> 56; eight of 300 341 ->
// 325 and 309 -> 214 (more in kernels/native.py, beside the rule). All of it is bound by shared memory's bandwidth: a
// thread's tile of 8 x 4 loads a word for 2.7 FMAs.  Against 64 bits the outputs are 1.3e-7 to 1.7e-7 off (token by
// token 0.9e-7), the matrices 7e-8 (6e-8).  That is further than before, so the engine's parts take these kernels
// only where an engine's owner asks for them (parts/base.py Runtime.chunked_scans).
//
// The decays enter as products of the given factors, never as differences of logarithms or quotients:
// a factor of 0 is an ordinary value.  All sums are 32-bit FMAs; pairs of them issue as one
// instruction (fma.rn.f32x2, the same rounding).
//
// Plain counterparts: tests/plain_karupel.py delta_mixer(), mlstm_mixer().
#include "common.cuh"

namespace {

constexpr int C = 64;            // tokens of a chunk
constexpr int NT = 256;          // threads of a block of chunk_prepare and chunk_walk
constexpr int MS = C + 4;        // row stride of a C x C matrix in shared memory
constexpr int CB = 16;           // columns of a block of the walk

struct ChunkArgs {
    const void* q;               // row r, key head g at q + r * q_stride + g * kd
    const void* k;
    const void* v;               // row r, head h at v + r * v_stride + h * vd
    const float* keep;           // [rows, H] a_t, or null: head_decay
    const float* take;           // [rows, H] b_t, or null: 1
    const float* head_decay;     // [H]
    float* state;                // [slots, state_stride]: [heads][cols][kd]
    float* out;                  // [rows, H * cols]
    float* kd_;                  // [rows, H, KP]  Kd (delta rule)
    float* w;                    // [rows, H, KP]  W (delta rule)
    float* u;                    // [rows, H, cp]  U0, then U (delta rule); zeros from column cols on
    float* sc;                   // [chunks, H, KP, cp]  B, then S before the chunk
    float* ac;                   // [chunks, H]  A_C
    const int* seq_slot;
    const int* seq_start;
    const int* seq_end;
    const int* seq_row0;
    long long q_stride, k_stride, v_stride, state_stride;
    int H, G, kd, vd, cols, cp;  // cols: vd, or vd + 1 with a last column whose v is 1; cp: cols in whole tiles of CB
    float q_scale;
};

// The number of a sequence's first chunk among all chunks: every sequence has as many numbers as it
// may need and shares none (sum of ceil(n / C) <= rows / C + sequences).
__device__ __forceinline__ size_t first_chunk(const ChunkArgs& p, int b) { return (size_t)(p.seq_row0[b] / C) + b; }

__device__ __forceinline__ uint64_t pair_of(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(uint64_t& d, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ ulonglong2 pairs4(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// acc[i][.] += sum_{s <= t} M[t][s] X[s][4 cq + 64 j ..] for the rows t = rq + 16 i, M[C][MS].  What a row
// may not see is not multiplied by zero but left out: an infinity in a later token stays in that
// token.  Whole 16 x 16 blocks below the diagonal go four rows at a time, then the diagonal's blocks.
template <int NQ>
__device__ __forceinline__ void lower_product(const float* M, const float* X, int xs, int rq, int cq,
                                              uint64_t (&acc)[4][2 * NQ]) {
#pragma unroll
    for (int sb = 0; sb < 3; ++sb) {
        uint64_t part[4][2 * NQ];        // (16 terms, then their sums: less rounding than one long sum)
#pragma unroll
        for (int i = sb + 1; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2 * NQ; ++j) part[i][j] = 0ull;
#pragma unroll 1
        for (int s = 16 * sb; s < 16 * sb + 16; s += 4) {
            float4 m[4];
#pragma unroll
            for (int i = sb + 1; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(M + (rq + 16 * i) * MS + s);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ulonglong2 x[NQ];
#pragma unroll
                for (int j = 0; j < NQ; ++j) x[j] = pairs4(X + (s + e) * xs + 4 * cq + 64 * j);
#pragma unroll
                for (int i = sb + 1; i < 4; ++i) {
                    const uint64_t a = pair_of(e == 0 ? m[i].x : e == 1 ? m[i].y : e == 2 ? m[i].z : m[i].w);
#pragma unroll
                    for (int j = 0; j < NQ; ++j) {
                        fma2(part[i][2 * j], a, x[j].x);
                        fma2(part[i][2 * j + 1], a, x[j].y);
                    }
                }
            }
        }
#pragma unroll
        for (int i = sb + 1; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2 * NQ; ++j) add2(acc[i][j], part[i][j]);
    }
#pragma unroll 2
    for (int s = 0; s <= rq; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t a = pair_of(M[(rq + 16 * i) * MS + 16 * i + s]);
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const ulonglong2 x = pairs4(X + (16 * i + s) * xs + 4 * cq + 64 * j);
                fma2(acc[i][2 * j], a, x.x);
                fma2(acc[i][2 * j + 1], a, x.y);
            }
        }
}

template <int NQ> __device__ __forceinline__ void clear(uint64_t (&acc)[4][NQ]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NQ; ++j) acc[i][j] = 0ull;
}

// a_t, b_t, A_t and D(C, s) of the chunk's tokens in av, bv, Av, Dv [C], and (D not null) D(t, s) for s <= t in
// D[C][MS]; all by products.  Tokens behind the sequence's end count as q = k = v = 0, a = 1, b = 0: they
// change nothing.  Ends without a barrier.
__device__ __forceinline__ void chunk_factors(const ChunkArgs& p, size_t row0, int count, int h, float* av, float* bv,
                                              float* Av, float* Dv, float* D) {
    const int tid = threadIdx.x;
    if (tid < C) {
        const bool in = tid < count;
        av[tid] = !in ? 1.f : p.keep ? p.keep[(row0 + tid) * p.H + h] : p.head_decay[h];
        bv[tid] = !in ? 0.f : p.take ? p.take[(row0 + tid) * p.H + h] : 1.f;
    }
    __syncthreads();
    if (tid < C) {
        float d = 1.f;
        if (D) D[tid * MS + tid] = 1.f;
#pragma unroll 4
        for (int t = tid + 1; t < C; ++t) {
            d *= av[t];
            if (D) D[t * MS + tid] = d;
        }
        Dv[tid] = d;
    } else if (tid == C) {
        float d = 1.f;
#pragma unroll 4
        for (int t = 0; t < C; ++t) {
            d *= av[t];
            Av[t] = d;
        }
    }
}

// Rows of q or k of the chunk, times `scale`, into dst[C][KS].
template <typename T, int KP>
__device__ __forceinline__ void load_rows(const T* src, long long stride, size_t row0, int count, int kd, float scale,
                                          float* dst, int threads) {
    constexpr int KS = KP + 4;
#pragma unroll 8
    for (int i = threadIdx.x; i < C * KP; i += threads) {
        const int t = i / KP, d = i % KP;
        dst[t * KS + d] = t < count && d < kd ? to_f32(src[(row0 + t) * stride + d]) * scale : 0.f;
    }
}

// The delta rule's part that does not contain S, one block per (chunk, head, sequence).
template <int KP>
__global__ void __launch_bounds__(NT, 2) chunk_prepare_kernel(ChunkArgs p) {
    constexpr int KS = KP + 4;
    constexpr int NQ = KP / 64;
    extern __shared__ __align__(16) float sm[];
    float* Ks = sm;                      // [C][KS] K, then A K
    float* Ts = Ks + C * KS;             // [C][MS] D, then L, then T b
    float* Vs = Ts + C * MS;             // [C][MS]
    float* av = Vs + C * MS;             // a_t
    float* bv = av + C;                  // b_t
    float* Av = bv + C;                  // A_t
    float* Dv = Av + C;                  // D(C, s)
    float* tmp = Dv + C;                 // [32][33]
    pdl_trigger();
    const int tid = threadIdx.x;
    const int h = blockIdx.y, b = blockIdx.z;
    const int t0 = blockIdx.x * C;
    const int n = p.seq_end[b] - p.seq_start[b];
    if (t0 >= n) return;
    const int count = min(C, n - t0);
    const size_t row0 = (size_t)p.seq_row0[b] + t0;
    const int g = h / (p.H / p.G);
    pdl_wait();
    load_rows<float, KP>((const float*)p.k + (size_t)g * p.kd, p.k_stride, row0, count, p.kd, 1.f, Ks, NT);
    chunk_factors(p, row0, count, h, av, bv, Av, Dv, Ts);
    __syncthreads();
    if (tid == 0) p.ac[(first_chunk(p, b) + blockIdx.x) * p.H + h] = Av[C - 1];

    // L: 4 x 4 of its elements a thread, the 16 x 16 blocks on and below the diagonal
    const int rq = tid / 16, cq = tid % 16;
    {
        uint64_t kk[4][4];
        clear(kk);
#pragma unroll 2
        for (int d = 0; d < KP; d += 4) {
            ulonglong2 kc[4], kr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                kc[i] = pairs4(Ks + (cq + 16 * i) * KS + d);
                kr[i] = pairs4(Ks + (rq + 16 * i) * KS + d);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    fma2(kk[i][j], kr[i].x, kc[j].x);
                    fma2(kk[i][j], kr[i].y, kc[j].y);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = rq + 16 * i;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int s = cq + 16 * j;
                const float2 c = unpair(kk[i][j]);
                const bool seen = j <= i && s < t;
                Ts[t * MS + s] = seen ? bv[t] * Ts[t * MS + s] * (c.x + c.y) : 0.f;
            }
        }
    }
    __syncthreads();

    // Kd, and A K in K's place
#pragma unroll 4
    for (int i = tid; i < C * KP; i += NT) {
        const int t = i / KP, d = i % KP;
        const float kv = Ks[t * KS + d];
        if (t < count) p.kd_[((row0 + t) * p.H + h) * KP + d] = Dv[t] * kv;
        Ks[t * KS + d] = Av[t] * kv;
    }
    // T = (I + L)^-1: the 16 x 16 blocks on the diagonal by a thread per column, then
    // [A 0; B C]^-1 = [A^-1 0; -C^-1 B A^-1 C^-1] for blocks of 16 and of 32
    if (tid < C) {
        const int o = tid & ~15, j = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float v = i == j ? 1.f : 0.f;
#pragma unroll
            for (int s = 0; s < i; ++s) v -= Ts[(o + i) * MS + o + s] * x[s];
            x[i] = v;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; ++i) Ts[(o + i) * MS + o + j] = x[i];
    }
    __syncthreads();
#pragma unroll
    for (int size = 16; size <= 32; size *= 2) {
        const int blocks = 32 / size, each = size * size;
        for (int e = tid; e < blocks * each; e += NT) {          // B A^-1
            const int o = (e / each) * 2 * size, i = (e % each) / size, j = e % size;
            float v = 0.f;
            for (int s = 0; s < size; ++s) v += Ts[(o + size + i) * MS + o + s] * Ts[(o + s) * MS + o + j];
            tmp[((e / each) * size + i) * 33 + j] = v;
        }
        __syncthreads();
        for (int e = tid; e < blocks * each; e += NT) {          // -C^-1 (B A^-1)
            const int o = (e / each) * 2 * size, i = (e % each) / size, j = e % size;
            float v = 0.f;
            for (int s = 0; s <= i; ++s)
                v -= Ts[(o + size + i) * MS + o + size + s] * tmp[((e / each) * size + s) * 33 + j];
            Ts[(o + size + i) * MS + o + j] = v;
        }
        __syncthreads();
    }
    for (int e = tid; e < C * C; e += NT) Ts[(e / C) * MS + e % C] *= bv[e % C];
    __syncthreads();
    {
        uint64_t acc[4][2 * NQ];
        clear(acc);
        lower_product<NQ>(Ts, Ks, KS, rq, cq, acc);                  // W = (T b) (A K)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const int t = rq + 16 * i, d = 4 * cq + 64 * j;
                if (t < count)
                    *reinterpret_cast<ulonglong2*>(p.w + ((row0 + t) * p.H + h) * KP + d) =
                        make_ulonglong2(acc[i][2 * j], acc[i][2 * j + 1]);
            }
    }
    // U0 = (T b) V, 64 columns at a time
    const float* vp = (const float*)p.v + (size_t)h * p.vd;
    for (int c0 = 0; c0 < p.cp; c0 += 64) {
        __syncthreads();
#pragma unroll 8
        for (int i = tid; i < C * 64; i += NT) {
            const int t = i / 64, col = c0 + i % 64;
            Vs[t * MS + i % 64] = t < count && col < p.vd ? vp[(row0 + t) * p.v_stride + col] : 0.f;
        }
        __syncthreads();
        uint64_t acc[4][2];
        clear(acc);
        lower_product<1>(Ts, Vs, MS, rq, cq, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = rq + 16 * i;
            if (t < count && c0 + 4 * cq < p.cp)
                *reinterpret_cast<ulonglong2*>(p.u + ((row0 + t) * p.H + h) * p.cp + c0 + 4 * cq) =
                    make_ulonglong2(acc[i][0], acc[i][1]);
        }
    }
}

// B = Kd^T (b V), one block per (chunk, 64 columns of a head, sequence): 8 keys x 4 columns a thread.
template <typename T, int KP>
__global__ void __launch_bounds__(KP * 2) chunk_update_kernel(ChunkArgs p) {
    constexpr int KS = KP + 4, THREADS = KP * 2;
    extern __shared__ __align__(16) float sm[];
    float* Ks = sm;                      // [C][KS] Kd
    float* Vs = Ks + C * KS;             // [C][MS] b V
    float* av = Vs + C * MS;
    float* bv = av + C;
    float* Av = bv + C;
    float* Dv = Av + C;
    pdl_trigger();
    const int tid = threadIdx.x;
    const int tiles = (p.cp + 63) / 64, h = blockIdx.y / tiles, c0 = (blockIdx.y % tiles) * 64, b = blockIdx.z;
    const int t0 = blockIdx.x * C, n = p.seq_end[b] - p.seq_start[b];
    if (t0 >= n) return;
    const int count = min(C, n - t0);
    const size_t row0 = (size_t)p.seq_row0[b] + t0, chunk = first_chunk(p, b) + blockIdx.x;
    const int g = h / (p.H / p.G);
    pdl_wait();
    load_rows<T, KP>((const T*)p.k + (size_t)g * p.kd, p.k_stride, row0, count, p.kd, 1.f, Ks, THREADS);
    const T* vp = (const T*)p.v + (size_t)h * p.vd;
#pragma unroll 8
    for (int i = tid; i < C * 64; i += THREADS) {
        const int t = i / 64, col = c0 + i % 64;
        Vs[t * MS + i % 64] = t >= count ? 0.f : col < p.vd ? to_f32(vp[(row0 + t) * p.v_stride + col]) : col < p.cols ? 1.f : 0.f;
    }
    chunk_factors(p, row0, count, h, av, bv, Av, Dv, nullptr);
    __syncthreads();
    if (tid == 0 && c0 == 0) p.ac[chunk * p.H + h] = Av[C - 1];
    for (int i = tid; i < C * 64; i += THREADS) Vs[(i / 64) * MS + i % 64] *= Dv[i / 64] * bv[i / 64];
    __syncthreads();
    const int kq = tid / 16, cq = tid % 16;        // keys 8 kq .. + 7, columns 4 cq .. + 3
    uint64_t acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll 4
    for (int t = 0; t < C; ++t) {
        const float4 k0 = *reinterpret_cast<const float4*>(Ks + t * KS + 8 * kq);
        const float4 k1 = *reinterpret_cast<const float4*>(Ks + t * KS + 8 * kq + 4);
        const ulonglong2 v = pairs4(Vs + t * MS + 4 * cq);
        const float k[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t x = pair_of(k[i]);
            fma2(acc[i][0], x, v.x);
            fma2(acc[i][1], x, v.y);
        }
    }
    if (c0 + 4 * cq >= p.cp) return;
    float* to = p.sc + ((chunk * p.H + h) * KP + 8 * kq) * p.cp + c0 + 4 * cq;
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<ulonglong2*>(to + (size_t)i * p.cp) = make_ulonglong2(acc[i][0], acc[i][1]);
}

// S' = A_C S + B from chunk to chunk; every chunk's B is replaced by the S before it.  A thread takes four
// neighbouring columns of a key.
template <int KP>
__global__ void __launch_bounds__(128) chunk_pass_kernel(ChunkArgs p) {
    pdl_trigger();
    const int h = blockIdx.y, b = blockIdx.z;
    const int e = blockIdx.x * 128 + threadIdx.x, quads = p.cp / 4;
    const int slot = p.seq_slot[b], n = p.seq_end[b] - p.seq_start[b], chunks = (n + C - 1) / C;
    const size_t first = first_chunk(p, b);
    pdl_wait();
    if (e >= KP * quads) return;
    const int k = e / quads, col = 4 * (e % quads);
    float* mine = slot >= 0 && k < p.kd
        ? p.state + (size_t)slot * p.state_stride + ((size_t)h * p.cols + col) * p.kd + k : nullptr;
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = mine && col + j < p.cols ? mine[(size_t)j * p.kd] : 0.f;
    float* at = p.sc + ((first * p.H + h) * KP + k) * p.cp + col;
    const size_t step = (size_t)p.H * KP * p.cp;
    const float* keep = p.ac + first * p.H + h;
    constexpr int AHEAD = 4;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 add[AHEAD];
        float a[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) {
                add[i] = *reinterpret_cast<const float4*>(at + (c0 + i) * step);
                a[i] = keep[(size_t)(c0 + i) * p.H];
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) {
                *reinterpret_cast<float4*>(at + (c0 + i) * step) = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = a[i] * s[0] + add[i].x;
                s[1] = a[i] * s[1] + add[i].y;
                s[2] = a[i] * s[2] + add[i].z;
                s[3] = a[i] * s[3] + add[i].w;
            }
    }
    if (!mine) return;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (col + j < p.cols) mine[(size_t)j * p.kd] = s[j];
}

// O = P U + A Q S, one block per (chunk, head, sequence) and run of `span` columns: 8 rows x 4 columns a
// thread, 64 columns at a time.  DELTA: U from p.u, else b V.
constexpr int OT = 128;
template <bool DELTA, typename T, int KP>
__global__ void __launch_bounds__(OT, 2) chunk_out_kernel(ChunkArgs p, int span) {
    constexpr int KS = KP + 4;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                      // [C][KS] Q, then A Q
    float* Ks = Qs + C * KS;             // [C][KS] K, then S [KP][64]
    float* Ps = Ks + C * KS;             // [C][MS] D, then P
    float* Us = Ps + C * MS;             // [C][64]
    float* av = Us + C * 64;
    float* bv = av + C;
    float* Av = bv + C;
    float* Dv = Av + C;
    pdl_trigger();
    const int tid = threadIdx.x;
    const int runs = (p.cp + span - 1) / span, h = blockIdx.y / runs, first = (blockIdx.y % runs) * span, b = blockIdx.z;
    const int t0 = blockIdx.x * C, n = p.seq_end[b] - p.seq_start[b];
    if (t0 >= n) return;
    const int count = min(C, n - t0);
    const size_t row0 = (size_t)p.seq_row0[b] + t0, chunk = first_chunk(p, b) + blockIdx.x;
    const int g = h / (p.H / p.G);
    pdl_wait();
    load_rows<T, KP>((const T*)p.q + (size_t)g * p.kd, p.q_stride, row0, count, p.kd, p.q_scale, Qs, OT);
    load_rows<T, KP>((const T*)p.k + (size_t)g * p.kd, p.k_stride, row0, count, p.kd, 1.f, Ks, OT);
    chunk_factors(p, row0, count, h, av, bv, Av, Dv, Ps);
    __syncthreads();
    const int rq = tid / 16, cq = tid % 16;        // rows rq + 8 i
    {
        uint64_t qk[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) qk[i][j] = 0ull;
#pragma unroll 1
        for (int d = 0; d < KP; d += 4) {
            ulonglong2 kc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kc[j] = pairs4(Ks + (cq + 16 * j) * KS + d);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const ulonglong2 q = pairs4(Qs + (rq + 8 * i) * KS + d);
#pragma unroll
                for (int j = 0; j <= i / 2; ++j) {
                    fma2(qk[i][j], q.x, kc[j].x);
                    fma2(qk[i][j], q.y, kc[j].y);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = rq + 8 * i;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int s = cq + 16 * j;
                const float2 x = unpair(qk[i][j]);
                const bool seen = j <= i / 2 && s <= t;
                Ps[t * MS + s] = seen ? Ps[t * MS + s] * (x.x + x.y) : 0.f;
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < C * KP; i += OT) Qs[(i / KP) * KS + i % KP] *= Av[i / KP];
    const T* vp = (const T*)p.v + (size_t)h * p.vd;
    for (int c0 = first; c0 < min(first + span, p.cp); c0 += 64) {
        __syncthreads();
        const float* sc = p.sc + ((chunk * p.H + h) * KP) * p.cp + c0;
#pragma unroll 8
        for (int i = tid; i < KP * 16; i += OT) {
            const int k = i / 16, d = 4 * (i % 16);
            *reinterpret_cast<float4*>(Ks + k * 64 + d) =
                c0 + d < p.cp ? *reinterpret_cast<const float4*>(sc + (size_t)k * p.cp + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (DELTA) {
#pragma unroll 8
            for (int i = tid; i < C * 16; i += OT) {
                const int t = i / 16, d = 4 * (i % 16);
                *reinterpret_cast<float4*>(Us + t * 64 + d) =
                    t < count && c0 + d < p.cp ? *reinterpret_cast<const float4*>(p.u + ((row0 + t) * p.H + h) * p.cp + c0 + d)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else {
#pragma unroll 8
            for (int i = tid; i < C * 64; i += OT) {
                const int t = i / 64, col = c0 + i % 64;
                const float v = t >= count ? 0.f : col < p.vd ? to_f32(vp[(row0 + t) * p.v_stride + col]) : col < p.cols ? 1.f : 0.f;
                Us[i] = bv[t] * v;
            }
        }
        __syncthreads();
        uint64_t acc[8][2], sum[8][2];       // (runs of 32, then their sums: half the rounding of one long sum)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = sum[i][0] = sum[i][1] = 0ull;
        // P U: rows 8 i + rq see whole groups of 8 tokens below their own, and of that the tokens up to rq
#pragma unroll
        for (int sb = 0; sb < 7; ++sb) {
#pragma unroll
            for (int s4 = 0; s4 < 8; s4 += 4) {
                ulonglong2 u[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) u[e] = pairs4(Us + (8 * sb + s4 + e) * 64 + 4 * cq);
#pragma unroll
                for (int i = sb + 1; i < 8; ++i) {
                    const float4 m = *reinterpret_cast<const float4*>(Ps + (rq + 8 * i) * MS + 8 * sb + s4);
                    const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint64_t x = pair_of(mv[e]);
                        fma2(acc[i][0], x, u[e].x);
                        fma2(acc[i][1], x, u[e].y);
                    }
                }
            }
            if (sb == 3) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    add2(sum[i][0], acc[i][0]);
                    add2(sum[i][1], acc[i][1]);
                    acc[i][0] = acc[i][1] = 0ull;
                }
            }
        }
#pragma unroll 1
        for (int s = 0; s <= rq; ++s)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t x = pair_of(Ps[(rq + 8 * i) * MS + 8 * i + s]);
                const ulonglong2 u = pairs4(Us + (8 * i + s) * 64 + 4 * cq);
                fma2(acc[i][0], x, u.x);
                fma2(acc[i][1], x, u.y);
            }
        // A Q S
#pragma unroll 1
        for (int k0 = 0; k0 < KP; k0 += 32) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                add2(sum[i][0], acc[i][0]);
                add2(sum[i][1], acc[i][1]);
                acc[i][0] = acc[i][1] = 0ull;
            }
#pragma unroll 2
            for (int k = k0; k < k0 + 32; k += 4) {
                ulonglong2 x[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = pairs4(Ks + (k + e) * 64 + 4 * cq);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 q = *reinterpret_cast<const float4*>(Qs + (rq + 8 * i) * KS + k);
                    const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint64_t y = pair_of(qv[e]);
                        fma2(acc[i][0], y, x[e].x);
                        fma2(acc[i][1], y, x[e].y);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            add2(sum[i][0], acc[i][0]);
            add2(sum[i][1], acc[i][1]);
            const int t = rq + 8 * i;
            const float2 x = unpair(sum[i][0]), y = unpair(sum[i][1]);
            const float o[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (t < count && c0 + 4 * cq + e < p.cols)
                    p.out[((row0 + t) * p.H + h) * p.cols + c0 + 4 * cq + e] = o[e];
        }
    }
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = in ? 16 : 0;               // 0: the 16 bytes are set to zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// The delta rule's walk, one block per (16 columns, head, sequence).  Per chunk: U = U0 - W S (64 x 16, the
// eight warps take 16 of the keys each, a thread 8 rows x 4 columns; their parts are added through shared
// memory), then S' = A_C S + Kd^T U (KP x 16, four runs of 16 tokens, 8 keys x 4 columns a thread, added
// likewise).  W and U0 of the next chunk are copied while Kd^T U runs, Kd of this one while W S does.
template <int KP>
__global__ void __launch_bounds__(NT, 1) chunk_walk_kernel(ChunkArgs p) {
    constexpr int KS = KP + 4;
    constexpr int KW = KP / 8;                   // keys of a warp's part of W S
    constexpr int KG = KP / 64;                  // groups of 64 keys: warps side by side in Kd^T U
    constexpr int TS = 8 / KG;                   // runs of tokens
    constexpr int TR = C / TS;                   // tokens of a run
    extern __shared__ __align__(16) float sm[];
    float* W = sm;                               // [C][KS]
    float* Kd = W + C * KS;                      // [C][KP]
    float* U0 = Kd + C * KP;                     // [C][CB]
    float* U = U0 + C * CB;                      // [C][CB]
    float* S = U + C * CB;                       // [KP][CB]
    float* parts = S + KP * CB;                  // [8][C][CB] of W S, then [TS][KP][CB] of Kd^T U
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = blockIdx.x * CB, h = blockIdx.y, b = blockIdx.z;
    const int slot = p.seq_slot[b];
    const size_t row0 = p.seq_row0[b], first = first_chunk(p, b);
    const int n = p.seq_end[b] - p.seq_start[b];
    const int chunks = (n + C - 1) / C;
    const int cq = 4 * (lane & 3), rl = lane >> 2;
    pdl_wait();

    auto copy_w = [&](int c) {                   // W and U0
        const int t0 = c * C, count = min(C, n - t0);
#pragma unroll
        for (int i = 0; i < C * KP / 4 / NT; ++i) {
            const int e = tid + NT * i, t = e / (KP / 4), d = 4 * (e % (KP / 4));
            copy16(W + t * KS + d, p.w + ((row0 + t0 + min(t, count - 1)) * p.H + h) * KP + d, t < count);
        }
        const int t = tid / (CB / 4), d = 4 * (tid % (CB / 4));
        copy16(U0 + t * CB + d, p.u + ((row0 + t0 + min(t, count - 1)) * p.H + h) * p.cp + col0 + d, t < count);
    };
    auto copy_kd = [&](int c) {
        const int t0 = c * C, count = min(C, n - t0);
#pragma unroll
        for (int i = 0; i < C * KP / 4 / NT; ++i) {
            const int e = tid + NT * i, t = e / (KP / 4), d = 4 * (e % (KP / 4));
            copy16(Kd + t * KP + d, p.kd_ + ((row0 + t0 + min(t, count - 1)) * p.H + h) * KP + d, t < count);
        }
    };

    // (a thread answers for the quads tid, tid + NT of the matrix: key (quad / 4), columns 4 (quad % 4))
    constexpr int QUADS = KP * CB / 4 / NT;
    float* mine = slot >= 0 ? p.state + (size_t)slot * p.state_stride + ((size_t)h * p.cols + col0) * p.kd : nullptr;
#pragma unroll
    for (int i = 0; i < QUADS; ++i) {
        const int k = (tid + NT * i) / 4, c = 4 * (tid % 4);
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            v[j] = mine && col0 + c + j < p.cols && k < p.kd ? mine[(size_t)(c + j) * p.kd + k] : 0.f;
        *reinterpret_cast<float4*>(S + k * CB + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
    if (chunks > 0) {
        copy_w(0);
        copies_commit();
    }
    for (int c = 0; c < chunks; ++c) {
        const int t0 = c * C, count = min(C, n - t0);
        const float keep = p.ac[(first + c) * p.H + h];
        copies_wait();
        __syncthreads();                                      // W, U0 and S are there; Kd and the parts are free
        copy_kd(c);
        copies_commit();
        // every chunk's S, for the outputs
        float* sc = p.sc + (((first + c) * p.H + h) * KP) * p.cp + col0;
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int k = (tid + NT * i) / 4, q = 4 * (tid % 4);
            *reinterpret_cast<float4*>(sc + (size_t)k * p.cp + q) = *reinterpret_cast<const float4*>(S + k * CB + q);
        }
        {
            uint64_t acc[8][2];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll
            for (int k = warp * KW; k < warp * KW + KW; k += 4) {
                ulonglong2 s[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) s[e] = pairs4(S + (k + e) * CB + cq);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 w = *reinterpret_cast<const float4*>(W + (rl + 8 * i) * KS + k);
                    const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint64_t x = pair_of(wv[e]);
                        fma2(acc[i][0], x, s[e].x);
                        fma2(acc[i][1], x, s[e].y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<ulonglong2*>(parts + (warp * C + rl + 8 * i) * CB + cq) = make_ulonglong2(acc[i][0], acc[i][1]);
        }
        __syncthreads();                                      // the parts are there; W is free
        {
            const int t = tid / 4, q = 4 * (tid % 4);
            float4 u = *reinterpret_cast<const float4*>(U0 + t * CB + q), s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const float4 x = *reinterpret_cast<const float4*>(parts + (w * C + t) * CB + q);
                s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
            }
            u = make_float4(u.x - s.x, u.y - s.y, u.z - s.z, u.w - s.w);
            *reinterpret_cast<float4*>(U + t * CB + q) = u;
            if (t < count) *reinterpret_cast<float4*>(p.u + ((row0 + t0 + t) * p.H + h) * p.cp + col0 + q) = u;
        }
        copies_wait();
        __syncthreads();                                      // Kd and U are there; U0 and the parts are free
        if (c + 1 < chunks) {
            copy_w(c + 1);
            copies_commit();
        }
        {
            const int kg = warp % KG, run = warp / KG, k = 64 * kg + 8 * rl;
            uint64_t acc[8][2];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll 4
            for (int t = run * TR; t < run * TR + TR; ++t) {
                const float4 k0 = *reinterpret_cast<const float4*>(Kd + t * KP + k);
                const float4 k1 = *reinterpret_cast<const float4*>(Kd + t * KP + k + 4);
                const ulonglong2 u = pairs4(U + t * CB + cq);
                const float kv[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint64_t x = pair_of(kv[i]);
                    fma2(acc[i][0], x, u.x);
                    fma2(acc[i][1], x, u.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<ulonglong2*>(parts + (run * KP + k + i) * CB + cq) = make_ulonglong2(acc[i][0], acc[i][1]);
        }
        __syncthreads();                                      // the parts are there
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int k = (tid + NT * i) / 4, q = 4 * (tid % 4);
            float4 s = *reinterpret_cast<const float4*>(S + k * CB + q), add = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int r = 0; r < TS; ++r) {
                const float4 x = *reinterpret_cast<const float4*>(parts + (r * KP + k) * CB + q);
                add.x += x.x; add.y += x.y; add.z += x.z; add.w += x.w;
            }
            *reinterpret_cast<float4*>(S + k * CB + q) =
                make_float4(keep * s.x + add.x, keep * s.y + add.y, keep * s.z + add.z, keep * s.w + add.w);
        }
    }
    if (!mine) return;
#pragma unroll
    for (int i = 0; i < QUADS; ++i) {                         // (a thread's own quads)
        const int k = (tid + NT * i) / 4, c = 4 * (tid % 4);
        const float4 s = *reinterpret_cast<const float4*>(S + k * CB + c);
        const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col0 + c + j < p.cols && k < p.kd) mine[(size_t)(c + j) * p.kd + k] = v[j];
    }
}

// The matrix memory's factors: a warp per (sequence, head) walks the tokens 32 at a time.  With F the
// running sum of the log forget gates and M_t = max_{s <= t} (i_s + F_t - F_s), both from the group's
// first token on, m_t = max(F_t + m, M_t); pairs (F, M) compose, so a group is one warp scan.
struct GateArgs {
    const void* gate_i;          // row r, head h at gate_i + r * stride + h (before bias and cap)
    const void* gate_f;
    const float* bias_i;
    const float* bias_f;
    float* state;                // the slot's running maxima lie `m_offset` floats into its state
    float* keep;                 // [rows, H]
    float* take;
    float* m_out;                // [rows, H]
    const int* seq_slot;
    const int* seq_start;
    const int* seq_end;
    const int* seq_row0;
    long long stride, state_stride, m_offset;
    int H;
    float cap;
};

template <typename T> __global__ void __launch_bounds__(32) memory_gates_kernel(GateArgs p) {
    pdl_trigger();
    const int lane = threadIdx.x, h = blockIdx.x, b = blockIdx.y;
    const int slot = p.seq_slot[b], n = p.seq_end[b] - p.seq_start[b];
    const size_t row0 = p.seq_row0[b];
    float* cell = slot >= 0 ? p.state + (size_t)slot * p.state_stride + p.m_offset + h : nullptr;
    const float bias_i = p.bias_i[h], bias_f = p.bias_f[h];
    pdl_wait();
    float m = cell ? *cell : 0.f;
    const T* gi = (const T*)p.gate_i + h;
    const T* gf = (const T*)p.gate_f + h;
    // (the gates' inputs of AHEAD groups are asked for while the AHEAD before them are worked on)
    constexpr int AHEAD = 4;
    T ri[AHEAD], rf[AHEAD];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int t = t0 + 32 * i + lane;
            ri[i] = rf[i] = from_f32<T>(0.f);
            if (t < n) {
                ri[i] = gi[(row0 + t) * p.stride];
                rf[i] = gf[(row0 + t) * p.stride];
            }
        }
    };
    fetch(0);
    for (int t00 = 0; t00 < n; t00 += 32 * AHEAD) {
        float gate[AHEAD], forget[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int t = t00 + 32 * k + lane;
            const float z = p.cap * tanhf((to_f32(rf[k]) + bias_f) / p.cap);
            gate[k] = t < n ? p.cap * tanhf((to_f32(ri[k]) + bias_i) / p.cap) : -INFINITY;
            forget[k] = t < n ? -(fmaxf(-z, 0.f) + log1pf(expf(-fabsf(z)))) : 0.f;      // log sigmoid
        }
        fetch(t00 + 32 * AHEAD);
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int t = t00 + 32 * k + lane;
            const float i = gate[k], f = forget[k];
            float F = f, M = i;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float F1 = __shfl_up_sync(0xffffffffu, F, o), M1 = __shfl_up_sync(0xffffffffu, M, o);
                if (lane >= o) {
                    M = fmaxf(M1 + F, M);
                    F += F1;
                }
            }
            const float now = fmaxf(F + m, M);
            float before = __shfl_up_sync(0xffffffffu, now, 1);
            if (lane == 0) before = m;
            if (t < n) {
                const size_t at = (row0 + t) * p.H + h;
                p.keep[at] = expf(f + before - now);
                p.take[at] = expf(i - now);
                p.m_out[at] = now;
            }
            m = __shfl_sync(0xffffffffu, now, 31);
        }
    }
    if (cell && lane == 0) *cell = m;
}

template <typename K> int allow(K kernel, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    SIB_REQUIRE(e == cudaSuccess, "chunked_scan: %s", cudaGetErrorString(e));
    return 0;
}

template <bool DELTA, typename T, int KP>
int launch_chunks(const ChunkArgs& p, int n_seqs, int longest, cudaStream_t s) {
    constexpr int KS = KP + 4;
    const int chunks = (longest + C - 1) / C;
    if constexpr (DELTA) {
        const size_t prepare = ((size_t)C * KS + 2 * C * MS + 4 * C + 32 * 33) * sizeof(float);
        const size_t walk = ((size_t)C * KS + C * KP + 2 * C * CB + KP * CB + 8 * C * CB) * sizeof(float);
        static_assert(8 * C * CB >= (8 / (KP / 64)) * KP * CB, "both kinds of parts fit");
        if (allow(chunk_prepare_kernel<KP>, prepare) || allow(chunk_walk_kernel<KP>, walk)) return -1;
        sib_launch_chained(chunk_prepare_kernel<KP>, dim3(chunks, p.H, n_seqs), dim3(NT), prepare, s, p);
        int rc = sib_check_launch("chunk_prepare");
        if (rc) return rc;
        sib_launch_chained(chunk_walk_kernel<KP>, dim3(p.cp / CB, p.H, n_seqs), dim3(NT), walk, s, p);
        rc = sib_check_launch("chunk_walk");
        if (rc) return rc;
    } else {
        const size_t update = ((size_t)C * KS + C * MS + 4 * C) * sizeof(float);
        if (allow(chunk_update_kernel<T, KP>, update)) return -1;
        sib_launch_chained(chunk_update_kernel<T, KP>, dim3(chunks, p.H * ((p.cp + 63) / 64), n_seqs), dim3(2 * KP), update, s, p);
        int rc = sib_check_launch("chunk_update");
        if (rc) return rc;
        sib_launch_chained(chunk_pass_kernel<KP>, dim3((KP * (p.cp / 4) + 127) / 128, p.H, n_seqs), dim3(128), 0, s, p);
        rc = sib_check_launch("chunk_pass");
        if (rc) return rc;
    }
    const size_t out = ((size_t)2 * C * KS + C * MS + C * 64 + 4 * C) * sizeof(float);
    if (allow(chunk_out_kernel<DELTA, T, KP>, out)) return -1;
    // (P is made once per run of columns: all of them where the chunks alone fill the device)
    const long long blocks = (long long)chunks * p.H * n_seqs;
    const int span = blocks >= 296 ? p.cp : blocks >= 148 ? max(64, (p.cp / 2 + 63) / 64 * 64) : 64;
    sib_launch_chained(chunk_out_kernel<DELTA, T, KP>, dim3(chunks, p.H * ((p.cp + span - 1) / span), n_seqs), dim3(OT), out,
                       s, p, span);
    return sib_check_launch("chunk_out");
}

template <bool DELTA, typename T>
int launch_chunks(ChunkArgs p, float* scratch, long long rows, int n_seqs, int longest, cudaStream_t s) {
    const int KP = p.kd <= 64 ? 64 : 128;
    p.cp = (p.cols + CB - 1) / CB * CB;
    const long long units = rows * p.H, chunks = rows / C + n_seqs;
    SIB_REQUIRE((long long)p.H * ((p.cp + 63) / 64) < 65536, "chunked_scan: %d heads of %d columns", p.H, p.cols);
    p.kd_ = scratch;
    p.w = p.kd_ + (DELTA ? units * KP : 0);
    p.u = p.w + (DELTA ? units * KP : 0);
    p.sc = p.u + (DELTA ? units * p.cp : 0);
    p.ac = p.sc + chunks * p.H * KP * p.cp;
    return KP == 64 ? launch_chunks<DELTA, T, 64>(p, n_seqs, longest, s)
                    : launch_chunks<DELTA, T, 128>(p, n_seqs, longest, s);
}

int check_chunks(const char* what, int rows, int n_seqs, int longest, int H, int G, int kd, int vd, const float* scratch) {
    SIB_REQUIRE(rows > 0 && n_seqs > 0 && n_seqs < 65536 && H > 0 && H < 65536 && G > 0 && H % G == 0 && longest > 0,
                "%s: rows=%d sequences=%d (of up to %d rows) heads=%d key heads=%d", what, rows, n_seqs, longest, H, G);
    SIB_REQUIRE(kd > 0 && kd <= 128 && vd > 0, "%s: key width %d (at most 128) and value width %d", what, kd, vd);
    SIB_REQUIRE(scratch != nullptr && ((uintptr_t)scratch % 16) == 0, "%s: 16-byte aligned scratch memory is needed", what);
    return 0;
}

}  // namespace

// 32-bit floats of scratch memory a chunked scan of this shape takes (0: not a shape it takes).
// `cols`: columns of a head's matrix; `delta`: the delta rule; `memory`: the matrix memory.
SIB_EXPORT long long sib_chunked_scan_floats(long long rows, int n_seqs, int H, int kd, int cols, int delta, int memory) {
    if (kd <= 0 || kd > 128 || rows <= 0 || n_seqs <= 0 || H <= 0 || cols <= 0) return 0;
    const int KP = kd <= 64 ? 64 : 128, cp = (cols + CB - 1) / CB * CB;
    if ((long long)H * ((cp + 63) / 64) >= 65536) return 0;
    return rows * H * ((delta ? 2 * KP + cp : 0) + (memory ? 2 : 0)) + (rows / C + n_seqs) * H * ((long long)KP * cp + 1);
}

SIB_EXPORT int sib_delta_scan_chunked(const float* qn, const float* kn, const float* vc, const float* decay,
                                      const float* beta, float* state, long long state_stride, float* out,
                                      float* scratch, const int* seq_slot, const int* seq_start,
                                      const int* seq_end, const int* seq_row0, int rows, int n_seqs,
                                      int longest, int H, int G, int kd, int vd, void* stream) {
    if (rows == 0) return 0;
    if (check_chunks("delta_scan", rows, n_seqs, longest, H, G, kd, vd, scratch)) return -1;
    ChunkArgs p{qn, kn, vc, decay, beta, nullptr, state, out, nullptr, nullptr, nullptr, nullptr, nullptr,
                seq_slot, seq_start, seq_end, seq_row0, (long long)G * kd, (long long)G * kd,
                (long long)H * vd, state_stride, H, G, kd, vd, vd, 0, 1.0f};
    return launch_chunks<true, float>(p, scratch, rows, n_seqs, longest, (cudaStream_t)stream);
}

SIB_EXPORT int sib_memory_scan_chunked(const void* proj, long long stride, int dtype, long long gate_i_col,
                                       long long gate_f_col, const float* bias_i, const float* bias_f,
                                       float cap, float* state, long long state_stride, float* out,
                                       float* m_out, float* scratch, const int* seq_slot,
                                       const int* seq_start, const int* seq_end, const int* seq_row0,
                                       int rows, int n_seqs, int longest, int H, int kd, int vd,
                                       void* stream) {
    if (rows == 0) return 0;
    if (check_chunks("memory_scan", rows, n_seqs, longest, H, H, kd, vd, scratch)) return -1;
    SIB_REQUIRE(cap > 0.f && bias_i && bias_f && m_out, "memory_scan: the gates need a cap, biases and a place for the maxima");
    const size_t esz = dtype == SIB_F32 ? 4 : 2;
    const char* base = (const char*)proj;
    // keep and take lie behind the chunks' own scratch memory
    float* keep = scratch + sib_chunked_scan_floats(rows, n_seqs, H, kd, vd + 1, 0, 0);
    float* take = keep + (size_t)rows * H;
    GateArgs gates{base + (size_t)gate_i_col * esz, base + (size_t)gate_f_col * esz, bias_i, bias_f, state,
                   keep, take, m_out, seq_slot, seq_start, seq_end, seq_row0, stride, state_stride,
                   (long long)H * (vd + 1) * kd, H, cap};
    ChunkArgs p{base, base + (size_t)H * kd * esz, base + (size_t)2 * H * kd * esz, keep, take, nullptr,
                state, out, nullptr, nullptr, nullptr, nullptr, nullptr, seq_slot, seq_start, seq_end,
                seq_row0, stride, stride, stride, state_stride, H, H, kd, vd, vd + 1, 0, 1.0f / sqrtf((float)kd)};
    cudaStream_t s = (cudaStream_t)stream;
    SIB_DISPATCH_DTYPE(dtype, {
        sib_launch_chained(memory_gates_kernel<T>, dim3(H, n_seqs), dim3(32), 0, s, gates);
        const int rc = sib_check_launch("memory_gates");
        return rc ? rc : (launch_chunks<false, T>(p, scratch, rows, n_seqs, longest, s));
    });
    return 0;
}

// Retention (head_decay, take null) and the gated recurrence (keep and take) over 32-bit rows.
SIB_EXPORT int sib_gated_scan_chunked(const float* q, const float* k, const float* v, long long q_stride,
                                      long long k_stride, long long v_stride, const float* keep,
                                      const float* take, const float* head_decay, float* state,
                                      long long state_stride, float* out, float* scratch,
                                      const int* seq_slot, const int* seq_start, const int* seq_end,
                                      const int* seq_row0, int rows, int n_seqs, int longest, int H,
                                      int G, int kd, int vd, void* stream) {
    if (rows == 0) return 0;
    if (check_chunks("gated_scan", rows, n_seqs, longest, H, G, kd, vd, scratch)) return -1;
    SIB_REQUIRE((keep != nullptr && take != nullptr) || head_decay != nullptr, "gated_scan: the rows' or the heads' factors are needed");
    ChunkArgs p{q, k, v, keep, take, head_decay, state, out, nullptr, nullptr, nullptr, nullptr, nullptr,
                seq_slot, seq_start, seq_end, seq_row0, q_stride, k_stride, v_stride, state_stride, H, G,
                kd, vd, vd, 0, 1.0f};
    return launch_chunks<false, float>(p, scratch, rows, n_seqs, longest, (cudaStream_t)stream);
}
