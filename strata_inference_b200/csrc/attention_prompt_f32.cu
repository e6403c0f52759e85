// Attention of packed 32-bit prompts that start at position 0 over their own keys and values, in 32-bit
// arithmetic throughout: the mathematics of attention_rows.cu (scale, soft cap, causal, window, chunk and
// kept first positions, sink, softmax, weighted sum), in tiles.
//
// attention_rows.cu gives every (row, head) a warp that reads every key and value it sees by itself:
// two prompts of 301 and 700 rows, 8 heads of 256 on 4 kv heads, took 711 us, 3.5 TFLOP/s, waiting for L2 (here: 162).
// Here a block of four warps takes 32 (row, query head) pairs of one kv head and walks the keys 32 at a time:
//
// * scores: 8 pairs x 4 keys a thread, 12 words of shared memory for 32 FMAs.  One warp covers the 32 x 32 scores, so the
//   four warps take a quarter of the head's dimensions each and their parts are added by the softmax;
// * weighted sum: 8 pairs a warp, every lane its own columns, the weights read by the whole warp at once;
// * K and V share one buffer, so that two blocks fit an SM at 256 dimensions: V is copied (cp.async) during
//   the softmax, K of the next tile once the weighted sum is done with V.  Neither copy hides behind its own
//   block's products; the other resident block's do that.
//
// The longest blocks start first.  FMAs would bound it: 1.2 G of them for the prompts above, 33 us at the rate of
// all SMs; with two warps a scheduler it is the latencies of shared memory and of the exposed copies.  A key
// that a row may not see is left out of its sum, not multiplied by zero.
//
// Plain counterpart: tests/plain_gemma2.py attention().
#include "common.cuh"

namespace {

constexpr int PAIRS = 32, KEYS = 32, THREADS = 128, SS = KEYS + 4;

struct PromptF32Args {
    const float* q;          // row r, head h at q + r * stride + h * head_dim
    const float* k;          // row r, kv head g at k + r * stride + g * head_dim
    const float* v;
    float* out;              // [rows, n_heads * head_dim]
    const int* seq_start;
    const int* seq_end;
    const int* seq_row0;
    int q_stride, kv_stride, n_heads, n_kv, head_dim;
    float scale, softcap;
    int window, chunk, keep;
    const float* sink;       // [n_heads] or null
    int n_seqs, tiles;       // tiles of rows of the longest sequence
};

__device__ __forceinline__ uint64_t pair_of(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void mul2(uint64_t& d, uint64_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = in ? 16 : 0;               // 0: the 16 bytes are set to zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// HDP: head size rounded up to 64, 128 or 256; the dimensions beyond head_dim are zeros.
template <int HDP>
__global__ void __launch_bounds__(THREADS, 2) attention_prompt_f32_kernel(PromptF32Args p) {
    constexpr int KS = HDP + 4;                  // row stride of Q and K
    constexpr int CPL = HDP / 32;                // columns of the output a lane owns
    constexpr int DW = HDP / 4;                  // dimensions of a warp's part of the scores
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                              // [PAIRS][KS]
    float* Ks = Qs + PAIRS * KS;                 // [KEYS][KS], then
    float* Vs = Ks;                              // [KEYS][KS]
    float* Sp = Ks + KEYS * KS;                  // [4][PAIRS][SS]: the warps' parts; part 0 becomes the weights
    float* corr_sm = Sp + 4 * PAIRS * SS;        // [PAIRS]
    float* inv_sm = corr_sm + PAIRS;             // [PAIRS]
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.n_heads / p.n_kv, rows_per = PAIRS / G;
    // (kv heads next to each other, then sequences, tiles from the last on: the longest blocks first)
    const int g = (int)(blockIdx.x % p.n_kv), b = (int)((blockIdx.x / p.n_kv) % p.n_seqs);
    const int n = p.seq_end[b] - p.seq_start[b];
    const int r0 = (p.tiles - 1 - (int)(blockIdx.x / ((unsigned)p.n_kv * p.n_seqs))) * rows_per;
    if (r0 >= n) return;
    const size_t row0 = p.seq_row0[b];
    const int last = min(r0 + rows_per, n) - 1;          // the tile's last row: it sees keys up to itself
    const int lo_tile = first_visible(r0, p.window, p.chunk);
    auto seen_tile = [&](int t) { return t * KEYS + KEYS - 1 >= lo_tile || t * KEYS < p.keep; };
    auto next_tile = [&](int t) {
        while (t * KEYS <= last && !seen_tile(t)) ++t;
        return t;
    };
    pdl_wait();

    const int hd4 = p.head_dim / 4;
    auto copy_rows = [&](const float* src, int t) {       // keys t * KEYS .. of K or V
        for (int e = tid; e < KEYS * (HDP / 4); e += THREADS) {
            const int key = e / (HDP / 4), d = e % (HDP / 4), j = t * KEYS + key;
            const bool in = j < n && d < hd4;
            copy16(Ks + key * KS + 4 * d, src + (row0 + (in ? j : 0)) * p.kv_stride + (size_t)g * p.head_dim + (in ? 4 * d : 0), in);
        }
    };
    for (int e = tid; e < PAIRS * (HDP / 4); e += THREADS) {
        const int i = e / (HDP / 4), d = e % (HDP / 4), row = r0 + i / G;
        const bool in = i < rows_per * G && row <= last && d < hd4;
        copy16(Qs + i * KS + 4 * d,
               p.q + (row0 + (in ? row : 0)) * p.q_stride + (size_t)(g * G + (in ? i % G : 0)) * p.head_dim + (in ? 4 * d : 0), in);
    }
    int t = next_tile(0);
    copy_rows(p.k, t);
    copies_commit();

    uint64_t acc[8][CPL / 2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < CPL / 2; ++c) acc[i][c] = 0ull;
    // softmax: four threads a pair, 8 keys each (quads sub and sub + 4)
    const int mine = tid >> 2, sub = tid & 3;
    const int my_row = r0 + mine / G;
    const bool my_live = mine < rows_per * G && my_row <= last;
    const int my_lo = first_visible(my_row, p.window, p.chunk), my_kept = kept_before(my_lo, p.keep);
    float m = -INFINITY, l = 0.f;

    while (t * KEYS <= last) {
        copies_wait();
        __syncthreads();                                  // K is there
        // ---- scores: this warp's dimensions of all 32 x 32 ----
        {
            const int rg = lane >> 3, kg = lane & 7;      // pairs rg + 4 i, keys kg + 8 j
            // (the even and the odd dimensions of 16 as two sums, then the sums' sum: as a single sum of 64 products
            // scores were further from 64 bits than the general kernel's, which adds 8 a lane and then by pairs)
            float sum[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[i][j] = 0.f;
            const float* qb = Qs + rg * KS + warp * DW;
            const float* kb = Ks + kg * KS + warp * DW;
#pragma unroll 1
            for (int d0 = 0; d0 < DW; d0 += 16) {
                uint64_t s[8][4];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = 0ull;
#pragma unroll
                for (int d = d0; d < d0 + 16; d += 4) {
                    ulonglong2 q[8], k[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(kb + 8 * j * KS + d);
#pragma unroll
                    for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const ulonglong2*>(qb + 4 * i * KS + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            fma2(s[i][j], q[i].x, k[j].x);
                            fma2(s[i][j], q[i].y, k[j].y);
                        }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 x = unpair(s[i][j]);
                        sum[i][j] += x.x + x.y;
                    }
            }
            float* part = Sp + warp * PAIRS * SS;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[(rg + 4 * i) * SS + kg + 8 * j] = sum[i][j];
        }
        __syncthreads();                                  // the parts are there; K is free
        copy_rows(p.v, t);
        copies_commit();
        // ---- softmax ----
        {
            float s[8], mx = -INFINITY;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int at = mine * SS + 4 * (sub + 4 * u);
                float4 x = *reinterpret_cast<const float4*>(Sp + at);
#pragma unroll
                for (int w = 1; w < 4; ++w) {
                    const float4 y = *reinterpret_cast<const float4*>(Sp + w * PAIRS * SS + at);
                    x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
                }
                const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = t * KEYS + 4 * (sub + 4 * u) + e;
                    const bool seen = my_live && j <= my_row && (j >= my_lo || j < my_kept);
                    float z = v[e] * p.scale;
                    if (p.softcap > 0.f) z = p.softcap * tanhf(z / p.softcap);
                    s[4 * u + e] = seen ? z : -INFINITY;
                    mx = fmaxf(mx, s[4 * u + e]);
                }
            }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float now = fmaxf(m, mx);
            const float corr = m == -INFINITY ? 0.f : expf(m - now);
            float sum = 0.f;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float w[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    w[e] = s[4 * u + e] == -INFINITY ? 0.f : expf(s[4 * u + e] - now);
                    sum += w[e];
                }
                *reinterpret_cast<float4*>(Sp + mine * SS + 4 * (sub + 4 * u)) = make_float4(w[0], w[1], w[2], w[3]);
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l = l * corr + sum;
            m = now;
            if (sub == 0) corr_sm[mine] = corr;
        }
        copies_wait();
        __syncthreads();                                  // V and the weights are there
        // ---- weighted sum: pairs 8 warp .. 8 warp + 7 ----
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t c = pair_of(corr_sm[8 * warp + i]);
#pragma unroll
            for (int x = 0; x < CPL / 2; ++x) mul2(acc[i][x], c);
        }
        auto value = [&](int key, uint64_t (&x)[CPL / 2]) {
            const float* vp = Vs + key * KS;
            if constexpr (CPL == 2) {
                x[0] = *reinterpret_cast<const uint64_t*>(vp + 2 * lane);
            } else {
#pragma unroll
                for (int c = 0; c < CPL / 4; ++c) {
                    const ulonglong2 two = *reinterpret_cast<const ulonglong2*>(vp + 128 * c + 4 * lane);
                    x[2 * c] = two.x;
                    x[2 * c + 1] = two.y;
                }
            }
        };
        // (whole where every pair of the tile sees every key of it)
        const bool whole = t * KEYS + KEYS - 1 <= r0 && (t * KEYS >= first_visible(last, p.window, p.chunk)) && last - r0 + 1 == rows_per;
        // A weight of 0 does no harm unless it meets an infinity (or NaN) in a value that its row must not
        // see, so such a tile is looked through first.
        bool by_key = false;
        if (!whole) {
            bool bad = false;
            for (int e = tid; e < KEYS * (HDP / 4); e += THREADS) {
                const float4 x = *reinterpret_cast<const float4*>(Vs + (e / (HDP / 4)) * KS + 4 * (e % (HDP / 4)));
                bad |= !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w));
            }
            by_key = __syncthreads_or(bad);
        }
        if (!by_key) {
#pragma unroll 2
            for (int key = 0; key < KEYS; key += 4) {
                float4 w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = *reinterpret_cast<const float4*>(Sp + (8 * warp + i) * SS + key);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    uint64_t x[CPL / 2];
                    value(key + e, x);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint64_t a = pair_of(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
#pragma unroll
                        for (int c = 0; c < CPL / 2; ++c) fma2(acc[i][c], a, x[c]);
                    }
                }
            }
        } else {
            int row[8], lo[8], kept[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                row[i] = r0 + (8 * warp + i) / G;
                if (8 * warp + i >= rows_per * G || row[i] > last) row[i] = -1;     // (sees nothing)
                lo[i] = first_visible(max(row[i], 0), p.window, p.chunk);
                kept[i] = kept_before(lo[i], p.keep);
            }
#pragma unroll 1
            for (int key = 0; key < KEYS; ++key) {
                const int j = t * KEYS + key;
                if (j > last) break;
                uint64_t x[CPL / 2];
                value(key, x);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (j <= row[i] && (j >= lo[i] || j < kept[i])) {
                        const uint64_t a = pair_of(Sp[(8 * warp + i) * SS + key]);
#pragma unroll
                        for (int c = 0; c < CPL / 2; ++c) fma2(acc[i][c], a, x[c]);
                    }
            }
        }
        t = next_tile(t + 1);
        __syncthreads();                                  // V and the weights are free
        if (t * KEYS <= last) {
            copy_rows(p.k, t);
            copies_commit();
        }
    }
    if (sub == 0) {
        float corr = 1.f;
        if (p.sink && my_live) {                          // one more term of the denominator
            const float sk = p.sink[g * G + mine % G], now = fmaxf(m, sk);
            corr = expf(m - now);
            l = l * corr + expf(sk - now);
        }
        corr_sm[mine] = corr;
        inv_sm[mine] = 1.0f / l;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int pair = 8 * warp + i, row = r0 + pair / G;
        if (pair >= rows_per * G || row > last) continue;
        const float f = corr_sm[pair] * inv_sm[pair];
        float* op = p.out + (row0 + row) * (size_t)p.n_heads * p.head_dim + (size_t)(g * G + pair % G) * p.head_dim;
#pragma unroll
        for (int c = 0; c < CPL / 2; ++c) {
            const int col = CPL == 2 ? 2 * lane : 128 * (c / 2) + 4 * lane + 2 * (c % 2);
            if (col < p.head_dim) {                       // (head_dim is even)
                const float2 x = unpair(acc[i][c]);
                *reinterpret_cast<float2*>(op + col) = make_float2(x.x * f, x.y * f);
            }
        }
    }
}

template <int HDP> int launch_prompt(PromptF32Args p, int longest, cudaStream_t s) {
    const size_t smem = ((size_t)(PAIRS + KEYS) * (HDP + 4) + 4 * PAIRS * SS + 2 * PAIRS) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(attention_prompt_f32_kernel<HDP>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    SIB_REQUIRE(e == cudaSuccess, "attention_prompt_f32: %s", cudaGetErrorString(e));
    const int rows_per = PAIRS / (p.n_heads / p.n_kv);
    p.tiles = (longest + rows_per - 1) / rows_per;
    const long long blocks = (long long)p.tiles * p.n_kv * p.n_seqs;
    SIB_REQUIRE(blocks < (1ll << 31), "attention_prompt_f32: too many rows (%d sequences of up to %d)", p.n_seqs, longest);
    sib_launch_chained(attention_prompt_f32_kernel<HDP>, dim3((unsigned)blocks), dim3(THREADS), smem, s, p);
    return sib_check_launch("attention_prompt_f32");
}

}  // namespace

// 1 if this kernel takes the shape (else the caller uses attention_rows).
SIB_EXPORT int sib_attention_prompt_f32_supports(int n_heads, int n_kv, int head_dim) {
    return n_kv > 0 && n_heads % n_kv == 0 && n_heads / n_kv <= PAIRS && head_dim > 0 &&
           head_dim % 4 == 0 && head_dim <= 256;
}

SIB_EXPORT int sib_attention_prompt_f32(const float* q, int q_stride, const float* k, const float* v, int kv_stride,
                                        const int* seq_start, const int* seq_end, const int* seq_row0, float* out,
                                        int n_seqs, int longest, int n_heads, int n_kv, int head_dim, float scale,
                                        float softcap, int window, int chunk, int keep, const float* sink,
                                        void* stream) {
    SIB_REQUIRE(sib_attention_prompt_f32_supports(n_heads, n_kv, head_dim),
                "attention_prompt_f32: heads=%d kv_heads=%d head_dim=%d", n_heads, n_kv, head_dim);
    SIB_REQUIRE(n_seqs > 0 && n_seqs < 65536 && longest > 0, "attention_prompt_f32: %d sequences of up to %d rows",
                n_seqs, longest);
    SIB_REQUIRE(window >= 0 && chunk >= 0 && (chunk == 0 || window == 0) && keep >= 0 && (keep == 0 || window > 0),
                "attention_prompt_f32: window=%d chunk=%d keep=%d (a chunk goes without a window, kept positions "
                "with one)", window, chunk, keep);
    SIB_REQUIRE(q_stride % 4 == 0 && kv_stride % 4 == 0 && ((uintptr_t)q % 16) == 0 && ((uintptr_t)k % 16) == 0 &&
                    ((uintptr_t)v % 16) == 0 && ((uintptr_t)out % 8) == 0,
                "attention_prompt_f32: rows must start on 16-byte boundaries");
    PromptF32Args p{q, k, v, out, seq_start, seq_end, seq_row0, q_stride, kv_stride, n_heads, n_kv, head_dim,
                    scale, softcap, window, chunk, keep, sink, n_seqs, 0};
    cudaStream_t s = (cudaStream_t)stream;
    return head_dim <= 64 ? launch_prompt<64>(p, longest, s)
           : head_dim <= 128 ? launch_prompt<128>(p, longest, s) : launch_prompt<256>(p, longest, s);
}
