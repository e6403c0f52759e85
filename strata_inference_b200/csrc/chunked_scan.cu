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
// U = U0 - W S, U0 = T (b V), W = T (b A K).  Everything that does not contain S is made for all chunks at
// once (chunk_prepare_kernel): with P[t, s] = D(t, s) (q_t . k_s),
//
//     O0 = P U0,   Q' = A Q - P W,   Kd = D(C, .) K
//
// so that the walk from chunk to chunk (chunk_walk_kernel) is left with two products of 16 columns a block:
// [Q' ; W] S, which gives the outputs and U, and Kd^T U, the matrix's update.
//
// Measured (one sequence, 8 heads of 128 x 256, token by token -> in chunks): 2 048 tokens, delta rule
// 634 -> 285 us, memory 763 -> 253, gated 574 -> 237; 512 tokens, delta rule 170 -> 112; 128 tokens 56 -> 76,
// hence the least number of rows in kernels/native.py.  Both kernels are bound by shared memory's
// bandwidth (a thread's tile of 2 x 4 or 4 x 8 loads a word for 1.3 to 2.7 FMAs).  Against 64 bits the
// outputs are 1.6e-7 off (token by token 0.9e-7), the matrices 4.9e-8 (5.4e-8).
//
// The decays enter as products of the given factors, never as differences of logarithms or quotients:
// a factor of 0 is an ordinary value.  All sums are 32-bit FMAs; pairs of them issue as one
// instruction (fma.rn.f32x2, the same rounding).
//
// Plain counterparts: tests/plain_karupel.py delta_mixer(), mlstm_mixer().
#include "common.cuh"

namespace {

constexpr int C = 64;            // tokens of a chunk
constexpr int NT = 256;          // threads of a block, in both kernels
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
    float* qd;                   // [rows, H, KP]  Q'
    float* kd_;                  // [rows, H, KP]  Kd
    float* w;                    // [rows, H, KP]  W (delta rule)
    float* u0;                   // [rows, H, cp]  U0, zeros from column cols on
    float* ac;                   // [rows, H]  A_C at each chunk's first row
    const int* seq_slot;
    const int* seq_start;
    const int* seq_end;
    const int* seq_row0;
    long long q_stride, k_stride, v_stride, state_stride;
    int H, G, kd, vd, cols, cp;  // cols: vd, or vd + 1 with a last column whose v is 1; cp: cols in whole tiles
    float q_scale;
};

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

// One block per (chunk, head, sequence): 2 048 tokens of 8 heads are 256 of them, two fit an SM.
template <bool DELTA, typename T, int KP>
__global__ void __launch_bounds__(NT, 2) chunk_prepare_kernel(ChunkArgs p) {
    constexpr int KS = KP + 4;
    constexpr int NQ = KP / 64;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                      // [C][KS]; later V [C][MS]
    float* Ks = Qs + C * KS;             // [C][KS]; later A K, then W, then U0 [C][MS]
    float* Ps = Ks + C * KS;             // [C][MS] D, then P
    float* Ts = Ps + C * MS;             // [C][MS] L, then T b (delta rule)
    float* av = Ts + (DELTA ? C * MS : 0);   // a_t
    float* bv = av + C;                  // b_t
    float* Av = bv + C;                  // A_t
    float* Dv = Av + C;                  // D(C, s)
    float* tmp = Dv + C;                 // [32][33] (delta rule)
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

    // tokens behind the sequence's end count as q = k = v = 0, a = 1: they change nothing
    if (tid < C) {
        const bool in = tid < count;
        av[tid] = !in ? 1.f : p.keep ? p.keep[(row0 + tid) * p.H + h] : p.head_decay[h];
        bv[tid] = !in ? 0.f : p.take ? p.take[(row0 + tid) * p.H + h] : 1.f;
    }
    const T* qp = (const T*)p.q + (size_t)g * p.kd;
    const T* kp = (const T*)p.k + (size_t)g * p.kd;
#pragma unroll 8
    for (int i = tid; i < C * KP; i += NT) {
        const int t = i / KP, d = i % KP;
        float qv = 0.f, kv = 0.f;
        if (t < count && d < p.kd) {
            qv = to_f32(qp[(row0 + t) * p.q_stride + d]) * p.q_scale;
            kv = to_f32(kp[(row0 + t) * p.k_stride + d]);
        }
        Qs[t * KS + d] = qv;
        Ks[t * KS + d] = kv;
    }
    __syncthreads();
    if (tid < C) {                       // a column of D each, by products alone
        float d = 1.f;
        Ps[tid * MS + tid] = 1.f;
        for (int t = tid + 1; t < C; ++t) {
            d *= av[t];
            Ps[t * MS + tid] = d;
        }
        Dv[tid] = d;
    } else if (tid == C) {
        float d = 1.f;
        for (int t = 0; t < C; ++t) {
            d *= av[t];
            Av[t] = d;
        }
        p.ac[row0 * p.H + h] = d;
    }
    __syncthreads();

    // P and L: 4 x 4 of their elements a thread, the 16 x 16 blocks on and below the diagonal
    const int rq = tid / 16, cq = tid % 16;
    {
        uint64_t qk[4][4], kk[4][4];
        clear(qk);
        clear(kk);
#pragma unroll 2
        for (int d = 0; d < KP; d += 4) {
            ulonglong2 kc[4], qr[4], kr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                kc[i] = pairs4(Ks + (cq + 16 * i) * KS + d);
                qr[i] = pairs4(Qs + (rq + 16 * i) * KS + d);
                if (DELTA) kr[i] = pairs4(Ks + (rq + 16 * i) * KS + d);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    fma2(qk[i][j], qr[i].x, kc[j].x);
                    fma2(qk[i][j], qr[i].y, kc[j].y);
                    if (DELTA) {
                        fma2(kk[i][j], kr[i].x, kc[j].x);
                        fma2(kk[i][j], kr[i].y, kc[j].y);
                    }
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = rq + 16 * i;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int s = cq + 16 * j;
                const float2 a = unpair(qk[i][j]), c = unpair(kk[i][j]);
                const bool seen = j <= i && s <= t;
                const float d = seen ? Ps[t * MS + s] : 0.f;
                Ps[t * MS + s] = seen ? d * (a.x + a.y) : 0.f;
                if (DELTA) Ts[t * MS + s] = seen && s < t ? bv[t] * d * (c.x + c.y) : 0.f;
            }
        }
    }
    __syncthreads();

    // Kd, and (delta rule) A K in its place; else Q' = A Q
#pragma unroll 4
    for (int i = tid; i < C * KP; i += NT) {
        const int t = i / KP, d = i % KP;
        const float kv = Ks[t * KS + d];
        const size_t at = ((row0 + t) * p.H + h) * KP + d;
        if (t < count) {
            p.kd_[at] = Dv[t] * kv;
            if (!DELTA) p.qd[at] = Av[t] * Qs[t * KS + d];
        }
        if (DELTA) Ks[t * KS + d] = Av[t] * kv;
    }
    if (DELTA) {
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
        uint64_t acc[4][2 * NQ];
        clear(acc);
        lower_product<NQ>(Ts, Ks, KS, rq, cq, acc);                  // W = (T b) (A K)
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const int t = rq + 16 * i, d = 4 * cq + 64 * j;
                const ulonglong2 v = make_ulonglong2(acc[i][2 * j], acc[i][2 * j + 1]);
                *reinterpret_cast<ulonglong2*>(Ks + t * KS + d) = v;
                if (t < count) *reinterpret_cast<ulonglong2*>(p.w + ((row0 + t) * p.H + h) * KP + d) = v;
            }
        __syncthreads();
        clear(acc);
        lower_product<NQ>(Ps, Ks, KS, rq, cq, acc);                  // Q' = A Q - P W
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const int t = rq + 16 * i, d = 4 * cq + 64 * j;
                const float4 q = *reinterpret_cast<const float4*>(Qs + t * KS + d);
                const float2 x = unpair(acc[i][2 * j]), y = unpair(acc[i][2 * j + 1]);
                const float A = Av[t];
                if (t < count)
                    *reinterpret_cast<float4*>(p.qd + ((row0 + t) * p.H + h) * KP + d) =
                        make_float4(A * q.x - x.x, A * q.y - x.y, A * q.z - y.x, A * q.w - y.y);
            }
    }

    // U0 and O0, 64 columns at a time
    float* Vs = Qs;
    float* Us = DELTA ? Ks : Qs;
    const T* vp = (const T*)p.v + (size_t)h * p.vd;
    for (int c0 = 0; c0 < p.cp; c0 += 64) {
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < C * 64; i += NT) {
            const int t = i / 64, col = c0 + i % 64;
            float v = 0.f;
            if (t < count) v = col < p.vd ? to_f32(vp[(row0 + t) * p.v_stride + col]) : col < p.cols ? 1.f : 0.f;
            if (!DELTA) {
                v *= bv[t];
                if (t < count && col < p.cp) p.u0[((row0 + t) * p.H + h) * p.cp + col] = v;
            }
            Vs[t * MS + i % 64] = v;
        }
        __syncthreads();
        uint64_t acc[4][2];
        if (DELTA) {
            clear(acc);
            lower_product<1>(Ts, Vs, MS, rq, cq, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = rq + 16 * i;
                const ulonglong2 v = make_ulonglong2(acc[i][0], acc[i][1]);
                *reinterpret_cast<ulonglong2*>(Us + t * MS + 4 * cq) = v;
                if (t < count && c0 + 4 * cq < p.cp)
                    *reinterpret_cast<ulonglong2*>(p.u0 + ((row0 + t) * p.H + h) * p.cp + c0 + 4 * cq) = v;
            }
            __syncthreads();
        }
        clear(acc);
        lower_product<1>(Ps, Us, MS, rq, cq, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = rq + 16 * i;
            const float2 x = unpair(acc[i][0]), y = unpair(acc[i][1]);
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

// One block per (16 columns, head, sequence) walks the chunks.  The matrix's 16 columns stay in
// registers (2 rows x 4 columns a thread) with a copy in shared memory for the products with
// them; Q' | W of the next chunk are copied while Kd^T U runs, Kd of this one while [Q' ; W] S does.
template <bool DELTA, int KP>
__global__ void __launch_bounds__(NT, 1) chunk_walk_kernel(ChunkArgs p) {
    constexpr int KS = KP + 4;
    constexpr int ROWS = DELTA ? 2 * C : C;
    constexpr int RI = ROWS / 64;                // rows of [Q' ; W] a thread works on
    constexpr int KI = KP / 64;                  // rows of the matrix a thread keeps
    extern __shared__ __align__(16) float sm[];
    float* QW = sm;                              // [ROWS][KS]
    float* Kd = QW + ROWS * KS;                  // [C][KP]
    float* U0 = Kd + C * KP;                     // [C][CB]
    float* U = U0 + C * CB;                      // [C][CB] (delta rule)
    float* S = U + (DELTA ? C * CB : 0);         // [KP][CB]
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = blockIdx.x * CB, h = blockIdx.y, b = blockIdx.z;
    const int slot = p.seq_slot[b];
    const size_t row0 = p.seq_row0[b];
    const int n = p.seq_end[b] - p.seq_start[b];
    const int chunks = (n + C - 1) / C;
    const int cq = 4 * (lane & 3), rl = lane >> 2;
    pdl_wait();

    auto copy_qw = [&](int c) {                  // Q' | W and (delta rule) U0
        const int t0 = c * C, count = min(C, n - t0);
#pragma unroll
        for (int i = 0; i < ROWS * KP / 4 / NT; ++i) {
            const int e = tid + NT * i, r = e / (KP / 4), d = 4 * (e % (KP / 4)), t = r % C;
            const float* src = (r < C ? p.qd : p.w) + ((row0 + t0 + min(t, count - 1)) * p.H + h) * KP + d;
            copy16(QW + r * KS + d, src, t < count);
        }
    };
    auto copy_u0 = [&](int c) {
        const int t0 = c * C, count = min(C, n - t0), t = tid / (CB / 4), d = 4 * (tid % (CB / 4));
        const float* src = p.u0 + ((row0 + t0 + min(t, count - 1)) * p.H + h) * p.cp + col0 + d;
        copy16(U0 + t * CB + d, src, t < count);
    };
    auto copy_kd = [&](int c) {
        const int t0 = c * C, count = min(C, n - t0);
#pragma unroll
        for (int i = 0; i < C * KP / 4 / NT; ++i) {
            const int e = tid + NT * i, t = e / (KP / 4), d = 4 * (e % (KP / 4));
            const float* src = p.kd_ + ((row0 + t0 + min(t, count - 1)) * p.H + h) * KP + d;
            copy16(Kd + t * KP + d, src, t < count);
        }
    };

    uint64_t s_reg[KI][2];
    const int k0 = warp * (KP / 8) + rl * KI;    // this thread's rows k0 .. k0 + KI - 1 of the matrix
    float* mine = slot >= 0 ? p.state + (size_t)slot * p.state_stride + ((size_t)h * p.cols + col0) * p.kd : nullptr;
#pragma unroll
    for (int e = 0; e < KI; ++e) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            v[j] = mine && col0 + cq + j < p.cols && k0 + e < p.kd ? mine[(size_t)(cq + j) * p.kd + k0 + e] : 0.f;
        *reinterpret_cast<float4*>(S + (k0 + e) * CB + cq) = make_float4(v[0], v[1], v[2], v[3]);
        const ulonglong2 two = pairs4(S + (k0 + e) * CB + cq);
        s_reg[e][0] = two.x;
        s_reg[e][1] = two.y;
    }
    if (chunks > 0) {
        copy_qw(0);
        if (DELTA) copy_u0(0);
        copies_commit();
    }
    for (int c = 0; c < chunks; ++c) {
        const int t0 = c * C, count = min(C, n - t0);
        const bool outputs = !DELTA || warp < 4;              // (the other half of the warps makes U)
        float o[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int t = (warp * (ROWS / 8) + rl + 8 * i) % C;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                o[i][j] = outputs && t < count && col0 + cq + j < p.cols
                              ? p.out[((row0 + t0 + t) * p.H + h) * p.cols + col0 + cq + j] : 0.f;
        }
        const float keep = p.ac[(row0 + t0) * p.H + h];
        copies_wait();
        __syncthreads();                                      // Q' | W and S are there; Kd is free
        copy_kd(c);
        if (!DELTA) copy_u0(c);
        copies_commit();
        uint64_t acc[RI][2], sum[RI][2];
#pragma unroll
        for (int i = 0; i < RI; ++i) acc[i][0] = acc[i][1] = sum[i][0] = sum[i][1] = 0ull;
        const float* rows = QW + (warp * (ROWS / 8) + rl) * KS;
#pragma unroll 4
        for (int k = 0; k < KP; k += 4) {
            if (k % 32 == 0 && k > 0) {              // (sums of 32, then of those: half the rounding of one long sum)
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        add2(sum[i][j], acc[i][j]);
                        acc[i][j] = 0ull;
                    }
            }
            float4 a[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(rows + 8 * i * KS + k);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const ulonglong2 s = pairs4(S + (k + e) * CB + cq);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const uint64_t x = pair_of(e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w);
                    fma2(acc[i][0], x, s.x);
                    fma2(acc[i][1], x, s.y);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int t = (warp * (ROWS / 8) + rl + 8 * i) % C;
            add2(sum[i][0], acc[i][0]);
            add2(sum[i][1], acc[i][1]);
            const float2 x = unpair(sum[i][0]), y = unpair(sum[i][1]);
            if (!outputs) {
                const float4 u = *reinterpret_cast<const float4*>(U0 + t * CB + cq);
                *reinterpret_cast<float4*>(U + t * CB + cq) = make_float4(u.x - x.x, u.y - x.y, u.z - y.x, u.w - y.y);
                continue;
            }
            const float v[4] = {o[i][0] + x.x, o[i][1] + x.y, o[i][2] + y.x, o[i][3] + y.y};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (t < count && col0 + cq + j < p.cols)
                    p.out[((row0 + t0 + t) * p.H + h) * p.cols + col0 + cq + j] = v[j];
        }
        copies_wait();
        __syncthreads();                                      // Kd and U are there; Q' | W and S are free
        if (c + 1 < chunks) {
            copy_qw(c + 1);
            if (DELTA) copy_u0(c + 1);
            copies_commit();
        }
        const uint64_t keep2 = pair_of(keep);
        const float* Uc = DELTA ? U : U0;
        uint64_t add[KI][2];
#pragma unroll
        for (int e = 0; e < KI; ++e) add[e][0] = add[e][1] = 0ull;
#pragma unroll 8
        for (int t = 0; t < C; ++t) {
            const ulonglong2 u = pairs4(Uc + t * CB + cq);
            float kv[KI];
            if (KI == 2) {
                const float2 two = *reinterpret_cast<const float2*>(Kd + t * KP + k0);
                kv[0] = two.x;
                kv[KI - 1] = two.y;
            } else {
                kv[0] = Kd[t * KP + k0];
            }
#pragma unroll
            for (int e = 0; e < KI; ++e) {
                const uint64_t x = pair_of(kv[e]);
                fma2(add[e][0], x, u.x);
                fma2(add[e][1], x, u.y);
            }
        }
#pragma unroll
        for (int e = 0; e < KI; ++e) {
            fma2(add[e][0], keep2, s_reg[e][0]);
            fma2(add[e][1], keep2, s_reg[e][1]);
            s_reg[e][0] = add[e][0];
            s_reg[e][1] = add[e][1];
            *reinterpret_cast<ulonglong2*>(S + (k0 + e) * CB + cq) = make_ulonglong2(add[e][0], add[e][1]);
        }
    }
    if (!mine) return;
#pragma unroll
    for (int e = 0; e < KI; ++e) {
        const float2 x = unpair(s_reg[e][0]), y = unpair(s_reg[e][1]);
        const float v[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col0 + cq + j < p.cols && k0 + e < p.kd) mine[(size_t)(cq + j) * p.kd + k0 + e] = v[j];
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
    T ri = from_f32<T>(0.f), rf = ri;
    auto fetch = [&](int t) {
        if (t < n) {
            ri = gi[(row0 + t) * p.stride];
            rf = gf[(row0 + t) * p.stride];
        }
    };
    fetch(lane);
    for (int t0 = 0; t0 < n; t0 += 32) {
        const int t = t0 + lane;
        float i = p.cap * tanhf((to_f32(ri) + bias_i) / p.cap);
        float f = p.cap * tanhf((to_f32(rf) + bias_f) / p.cap);
        f = -(fmaxf(-f, 0.f) + log1pf(expf(-fabsf(f))));      // log sigmoid
        if (t >= n) {
            i = -INFINITY;
            f = 0.f;
        }
        fetch(t + 32);
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
    if (cell && lane == 0) *cell = m;
}

template <bool DELTA, typename T, int KP>
int launch_chunks(const ChunkArgs& p, int n_seqs, int longest, cudaStream_t s) {
    const size_t prepare = ((size_t)2 * C * (KP + 4) + (DELTA ? 2 : 1) * C * MS + 4 * C + (DELTA ? 32 * 33 : 0)) * sizeof(float);
    const size_t walk = ((size_t)(DELTA ? 2 : 1) * C * (KP + 4) + C * KP + (DELTA ? 2 : 1) * C * CB + KP * CB) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(chunk_prepare_kernel<DELTA, T, KP>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prepare);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(chunk_walk_kernel<DELTA, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk);
    SIB_REQUIRE(e == cudaSuccess, "chunked_scan: %s", cudaGetErrorString(e));
    sib_launch_chained(chunk_prepare_kernel<DELTA, T, KP>, dim3((longest + C - 1) / C, p.H, n_seqs), dim3(NT),
                       prepare, s, p);
    const int rc = sib_check_launch("chunk_prepare");
    if (rc) return rc;
    sib_launch_chained(chunk_walk_kernel<DELTA, KP>, dim3(p.cp / CB, p.H, n_seqs), dim3(NT), walk, s, p);
    return sib_check_launch("chunk_walk");
}

template <bool DELTA, typename T>
int launch_chunks(ChunkArgs p, float* scratch, long long rows, int n_seqs, int longest, cudaStream_t s) {
    const int KP = p.kd <= 64 ? 64 : 128;
    p.cp = (p.cols + CB - 1) / CB * CB;
    const long long units = rows * p.H;
    p.qd = scratch;
    p.kd_ = p.qd + units * KP;
    p.w = p.kd_ + units * KP;
    p.u0 = p.w + (DELTA ? units * KP : 0);
    p.ac = p.u0 + units * p.cp;
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
SIB_EXPORT long long sib_chunked_scan_floats(long long rows, int H, int kd, int cols, int delta, int memory) {
    if (kd <= 0 || kd > 128 || rows <= 0 || H <= 0 || cols <= 0) return 0;
    const int KP = kd <= 64 ? 64 : 128, cp = (cols + CB - 1) / CB * CB;
    // (whole groups of 4 floats in front, so that every part begins on a 16-byte boundary)
    return rows * H * ((delta ? 3 : 2) * KP + cp + 1 + (memory ? 2 : 0)) + 4;
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
    float* keep = scratch + sib_chunked_scan_floats(rows, H, kd, vd + 1, 0, 0) - 4;
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
