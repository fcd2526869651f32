// Plain attention over the paged cache, one block per (token, query head),
// every step of the arithmetic in 32-bit.  It serves the 32-bit path for
// prefill and decode alike and any head size up to 256.
//
// The query at absolute position a sees key j iff j <= a and (window == 0 or
// a - j < window), or, with ``chunk`` > 0, iff j <= a and both lie in the same block of ``chunk`` positions; the first
// ``keep`` positions of a sequence are seen besides.  score = dot(q, k_j) / sqrt(hd) (divided after the product), or dot(q, k_j) * scale when a scale is
// given.  Values may have another size than keys (vd).  With ``sink`` the denominator holds one more term, exp(0 - max):
// a key of score zero that carries no value; with ``sink_vals`` the term is exp(sink_vals[head] - max), a number per head
// that is not scaled.  With ``softcap`` > 0 the scaled score s becomes softcap * tanh(s / softcap).  ``maps`` > 1: a key
// head's row in the cache holds that many keys side by side (hd numbers each) over one value; the query heads of a key
// head come map by map within each head, so query head h reads the key h % maps of key head h / (nh / nkv).  The result
// may be kept in float whatever the cache's type (TO), for a caller that goes on computing with it.
// Keys are walked in chunks of CHUNK positions aligned to absolute multiples of
// CHUNK with a running maximum and sum, so the order of every addition depends
// on the query's position alone: not on how the sequence was cut into steps,
// nor on what else is in the batch.
#include "common.cuh"

namespace {
constexpr int CHUNK = 256;
constexpr int THREADS = 128;
constexpr int MAX_HD = 256;

template <typename T, typename TO>
__global__ void __launch_bounds__(THREADS)
attn_simt_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                 TO* __restrict__ out, const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                 const int* __restrict__ block_table, int table_stride, int n_pages, int page, int nh, int nkv, int hd,
                 int vd, float scale, int sink, const float* __restrict__ sink_vals, int window, int chunk, int keep,
                 float softcap, int maps, int* __restrict__ status) {
    __shared__ float qs[MAX_HD];
    __shared__ float ps[CHUNK];
    __shared__ int pages[CHUNK];      // page id of each key of the chunk (or -1)
    __shared__ float scratch[33];
    const int n = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int seq = tok_seq[n], pos = tok_pos[n];
    const int kvh = h / (nh / nkv), map = h % maps;
    const VisibleKeys seen = visible_keys(pos, window, chunk, keep);
    const T* qrow = q + ((size_t)n * nh + h) * hd;
    for (int d = tid; d < hd; d += THREADS) qs[d] = to_f32(qrow[d]);
    const float root = sqrtf((float)hd);
    // the sink is a key of score zero (or of the head's own score) ahead of all others: the running maximum and sum start from it
    float m_run = sink ? (sink_vals ? sink_vals[h] : 0.f) : -INFINITY, l_run = sink ? 1.f : 0.f;
    float acc[MAX_HD / THREADS];
#pragma unroll
    for (int i = 0; i < MAX_HD / THREADS; i++) acc[i] = 0.f;
    __syncthreads();

    for (int c = seen.kept > 0 ? 0 : seen.lo / CHUNK; c <= pos / CHUNK; c++) {
        if (c * CHUNK >= seen.kept && c < seen.lo / CHUNK) c = seen.lo / CHUNK;     // nothing between the kept keys and the window
        const int j0 = c * CHUNK < seen.kept ? c * CHUNK : max(seen.lo, c * CHUNK), j1 = min(pos, c * CHUNK + CHUNK - 1);
        const int count = j1 - j0 + 1;
        // scores
        float local_max = -INFINITY;
        for (int t = tid; t < count; t += THREADS) {
            const int j = j0 + t;
            if (!seen.sees(j)) {                                     // a chunk that holds both kept keys and the window's first
                pages[t] = -1;
                ps[t] = -INFINITY;
                continue;
            }
            int pg = block_table[(size_t)seq * table_stride + j / page];
            if (pg < 0 || pg >= n_pages) {
                atomicOr(status, ESP_STATUS_BAD_INDEX);
                pg = -1;
            }
            pages[t] = pg;
            float s = -INFINITY;
            if (pg >= 0) {
                const T* krow = k_cache + ((((size_t)pg * nkv + kvh) * page + j % page) * maps + map) * hd;
                float dot = 0.f;
                for (int d = 0; d < hd; d++) dot = fmaf(qs[d], to_f32(krow[d]), dot);
                s = scale > 0.f ? dot * scale : dot / root;
                if (softcap > 0.f) s = softcap * tanhf(s / softcap);
            }
            ps[t] = s;
            local_max = fmaxf(local_max, s);
        }
        const float m_chunk = block_max(local_max, scratch);
        const float m_new = fmaxf(m_run, m_chunk);
        if (m_new == -INFINITY) continue;          // every key of the chunk was skipped as a bad index
        float local_sum = 0.f;
        for (int t = tid; t < count; t += THREADS) {
            const float p = expf(ps[t] - m_new);
            ps[t] = p;
            local_sum += p;
        }
        const float l_chunk = block_sum(local_sum, scratch);   // also orders the writes of ps before the reads below
        const float rescale = expf(m_run - m_new);
        l_run = l_run * rescale + l_chunk;
        m_run = m_new;
#pragma unroll
        for (int i = 0; i < MAX_HD / THREADS; i++) {
            const int d = tid + i * THREADS;
            if (d < vd) {
                float a = acc[i] * rescale;
                for (int t = 0; t < count; t++) {
                    const int pg = pages[t];
                    if (pg < 0) continue;
                    const int j = j0 + t;
                    a = fmaf(ps[t], to_f32(v_cache[(((size_t)pg * nkv + kvh) * page + j % page) * vd + d]), a);
                }
                acc[i] = a;
            }
        }
        __syncthreads();
    }
    TO* orow = out + ((size_t)n * nh + h) * vd;
#pragma unroll
    for (int i = 0; i < MAX_HD / THREADS; i++) {
        const int d = tid + i * THREADS;
        if (d < vd) orow[d] = from_f32<TO>(l_run > 0.f ? acc[i] / l_run : 0.f);
    }
}

// The same for the 32-bit cache with one key per value and heads of up to 128 channels (multiples of 4), with up to 16
// queries of a sequence at once.  The tokens are cut into windows of 16; a run (tokens of one sequence at consecutive positions)
// within a window is worked on by one block, run i of a window by the block with blockIdx.z = i modulo gridDim.z.  Keys and
// values pass through shared memory 64 at a time, from absolute multiples of 64 on, each read once for all queries of the run; the
// places of a chunk's keys in the cache are looked up once, while the chunk before it is worked on.  A thread makes 2 x 4
// scores, each a chain over the channels, and then 4 queries x 4 channels of the output, each a chain over the keys; runs of
// one or two tokens give a thread one score and one channel (the same chains, on all warps and not on one).  A key that a
// query does not see has the score -infinity, adds an exact zero to the sum of weights and is left out of the output, so a row
// depends on its own position alone: not on its run, nor on which of the two ways the run takes.
// The softmax takes 64 keys at a time where the kernel above takes 256, so the two differ in the order of their sums.
// Bound by the latency of a chunk's steps, two blocks an SM.  The kernel above takes a block per query, each thread a key of
// its own: every load of a warp touches 32 lines, and the queries of a prompt read the same keys again and again.
// 16 heads of 128, that kernel -> this: a prompt of 1,400 tokens 8,960 -> 558 us; a token each of sequences of about 3,000:
// one 1,936 -> 255, 65 2,850 -> 1,100, 256 8,670 -> 4,340.
constexpr int TQ = 16, TK = 64, P_LD = TQ + 4;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(THREADS, 2)
attn_simt_tile_kernel(const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                      float* __restrict__ out, const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                      const int* __restrict__ block_table, int table_stride, int n_pages, int page, int n_tokens, int nh, int nkv, int hd,
                      int vd, float scale, int sink, const float* __restrict__ sink_vals, int window, int chunk, int keep,
                      float softcap, int* __restrict__ status) {
    extern __shared__ __align__(16) float tile_smem[];
    __shared__ long long places[2][TK];                        // cache rows of a chunk's keys for this head, or -1, for two chunks in turn
    const int k_ld = hd + 4;                                   // rows 16 bytes apart in the banks
    float* ks = tile_smem;                                     // [TK][k_ld]
    float* vs = ks + TK * k_ld;                                // [TK][vd]
    float* qs = vs + TK * vd;                                  // [TQ][hd]
    float* ps = qs + TQ * hd;                                  // [TK][P_LD]: scores, then weights, of key x query
    float* factor = ps + TK * P_LD;                            // [TQ]: what the sums so far are multiplied with; at the end 1 / l
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid % 32, kvh = h / (nh / nkv);
    const int n0 = blockIdx.x * TQ, n_here = min(TQ, n_tokens - n0);
    // the window's tokens, a lane each, and where its runs begin: every warp finds them by itself
    const int tok_s = lane < n_here ? tok_seq[n0 + lane] : 0, tok_p = lane < n_here ? tok_pos[n0 + lane] : 0;
    const int before_s = __shfl_up_sync(0xffffffffu, tok_s, 1), before_p = __shfl_up_sync(0xffffffffu, tok_p, 1);
    unsigned starts = __ballot_sync(0xffffffffu, lane < n_here && (lane == 0 || tok_s != before_s || tok_p != before_p + 1));
    // this thread's part of a chunk's copy: 16 bytes of the keys first, first + step, ... (threads beyond whole rows rest)
    const int k_quads = hd / 4, k_first = tid / k_quads, k_step = THREADS / k_quads, k_at = tid % k_quads * 4;
    const int v_quads = vd / 4, v_first = tid / v_quads, v_step = THREADS / v_quads, v_at = tid % v_quads * 4;
    const float root = sqrtf((float)hd);
    for (int run = 0; starts; run++) {
        const int at = __ffs(starts) - 1;
        starts &= starts - 1;
        if (run % gridDim.z != blockIdx.z) continue;
        const int rows = (starts ? __ffs(starts) - 1 : n_here) - at, n = n0 + at;
        const int seq = __shfl_sync(0xffffffffu, tok_s, at), pos = __shfl_sync(0xffffffffu, tok_p, at);
        const bool few = rows <= 2;
        const int last = pos + rows - 1;
        const int lo = visible_keys(pos, window, chunk, keep).lo;
        const int lo_last = visible_keys(last, window, chunk, keep).lo, kept = visible_keys(last, window, chunk, keep).kept;
        auto next_chunk = [&](int c) { return c * TK >= kept && c < lo / TK ? lo / TK : c; };   // nothing between the kept keys and the window

        for (int i = tid; i < TQ * k_quads; i += THREADS) {
            const int r = i / k_quads, d = i % k_quads * 4;
            *reinterpret_cast<float4*>(qs + r * hd + d) =
                r < rows ? *reinterpret_cast<const float4*>(q + ((size_t)(n + r) * nh + h) * hd + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // a quarter of a warp per query: eight lanes, each with every eighth key of a chunk
        const int my_q = tid / 8, my_l = tid % 8;
        const VisibleKeys seen = visible_keys(pos + my_q, window, chunk, keep);
        float m_run = sink ? (sink_vals ? sink_vals[h] : 0.f) : -INFINITY, l_run = sink ? 1.f : 0.f;
        // scores: queries 2 sq, 2 sq + 1 and keys sk + 16 i; output: queries 4 oq .. 4 oq + 3, channels 4 od .. 4 od + 3.
        // few: scores of query tid / 64 and key tid % 64; output of both queries, channel tid, in acc[0][0] and acc[1][0]
        const int sq = tid / 16, sk = tid % 16, oq = tid / 32, od = tid % 32;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = 0.f;

        // key tid of chunk c (the first 64 threads): its page, and from that its place
        auto page_of = [&](int c) {
            const int j = c * TK + tid;
            return tid < TK && j <= last ? block_table[(size_t)seq * table_stride + j / page] : -1;
        };
        auto put_place = [&](int c, int pg, int buf) {
            if (tid < TK) places[buf][tid] = pg < 0 || pg >= n_pages ? -1ll : ((long long)pg * nkv + kvh) * page + (c * TK + tid) % page;
        };
        auto fetch = [&](const float* cache, float* dst, int ld, int width, int first, int step, int d, int buf) {
            if (first < step) {
#pragma unroll 4
                for (int t = first; t < TK; t += step) {
                    const long long row = places[buf][t];
                    copy16(dst + t * ld + d, row >= 0 ? cache + row * width + d : cache, row >= 0);
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        const int c_end = last / TK;
        int c = next_chunk(kept > 0 ? 0 : lo / TK), buf = 0;
        put_place(c, page_of(c), buf);
        __syncthreads();
        fetch(k_cache, ks, k_ld, hd, k_first, k_step, k_at, buf);
        fetch(v_cache, vs, vd, vd, v_first, v_step, v_at, buf);
        while (c <= c_end) {
            const int c_next = next_chunk(c + 1);
            const int page_next = c_next <= c_end ? page_of(c_next) : -1;      // arrives while the scores are made
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();                                       // the keys are there, and the queries
            auto put_score = [&](int t, int r, float dot) {
                float v = scale > 0.f ? dot * scale : dot / root;
                if (softcap > 0.f) v = softcap * tanhf(v / softcap);
                ps[t * P_LD + r] = v;
            };
            if (few) {
                if (tid / TK < rows) {
                    const float* a_row = qs + tid / TK * hd;
                    const float* b_row = ks + tid % TK * k_ld;
                    float s = 0.f;
#pragma unroll 8
                    for (int d = 0; d < hd; d += 4) {
                        const float4 a = *reinterpret_cast<const float4*>(a_row + d), b = *reinterpret_cast<const float4*>(b_row + d);
                        s = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
                    }
                    put_score(tid % TK, tid / TK, s);
                }
            } else if (2 * sq < rows) {
                float s[2][4];
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) s[i][j] = 0.f;
#pragma unroll 4
                for (int d = 0; d < hd; d += 4) {
                    float4 a[2], b[4];
#pragma unroll
                    for (int i = 0; i < 2; i++) a[i] = *reinterpret_cast<const float4*>(qs + (2 * sq + i) * hd + d);
#pragma unroll
                    for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4*>(ks + (sk + 16 * j) * k_ld + d);
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
                }
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) put_score(sk + 16 * j, 2 * sq + i, s[i][j]);
            }
            put_place(c_next, page_next, buf ^ 1);
            __syncthreads();                                       // the scores and the next places are there, and the keys read
            if (my_q < rows) {
                float p[TK / 8], best = -INFINITY;
#pragma unroll
                for (int i = 0; i < TK / 8; i++) {
                    const int t = my_l + 8 * i, j = c * TK + t;
                    const bool sees = j <= pos + my_q && seen.sees(j), bad = places[buf][t] < 0;
                    if (sees && bad) atomicOr(status, ESP_STATUS_BAD_INDEX);
                    p[i] = sees && !bad ? ps[t * P_LD + my_q] : -INFINITY;
                    best = fmaxf(best, p[i]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffu << (tid % 32 / 8 * 8), best, o));
                const float m_new = fmaxf(m_run, best);
                const float base = m_new == -INFINITY ? 0.f : m_new;      // nothing seen so far: every term is zero
                float sum = 0.f;
#pragma unroll
                for (int i = 0; i < TK / 8; i++) {
                    p[i] = expf(p[i] - base);
                    sum += p[i];
                    ps[(my_l + 8 * i) * P_LD + my_q] = p[i];
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffu << (tid % 32 / 8 * 8), sum, o);
                const float rescale = expf(m_run - base);
                l_run = l_run * rescale + sum;
                m_run = m_new;
                if (my_l == 0) factor[my_q] = rescale;
            } else {
#pragma unroll
                for (int i = 0; i < TK / 8; i++) ps[(my_l + 8 * i) * P_LD + my_q] = 0.f;
                if (my_l == 0) factor[my_q] = 0.f;
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();                                       // the values are there, the weights too, and this chunk's places are read
            if (c_next <= c_end) fetch(k_cache, ks, k_ld, hd, k_first, k_step, k_at, buf ^ 1);
            else asm volatile("cp.async.commit_group;\n" ::: "memory");
            const int count = min(TK, last - c * TK + 1);
            // a chunk that every query of the run sees whole, or (the same choice for a warp) key by key: a value that is not
            // finite must not reach the queries that do not see it
            const bool whole = c * TK + count - 1 <= pos && (c * TK >= lo_last || c * TK + TK <= kept);
            if (few) {
                if (tid < vd) {
                    float first = acc[0][0] * factor[0], second = acc[1][0] * factor[1];
                    const VisibleKeys of_first = visible_keys(pos, window, chunk, keep), of_second = visible_keys(pos + 1, window, chunk, keep);
#pragma unroll 8
                    for (int t = 0; t < count; t++) {
                        const float2 w = *reinterpret_cast<const float2*>(ps + t * P_LD);
                        const float v = vs[t * vd + tid];
                        const int j = c * TK + t;
                        if (whole || (j <= pos && of_first.sees(j))) first = fmaf(w.x, v, first);
                        if (whole || (j <= pos + 1 && of_second.sees(j))) second = fmaf(w.y, v, second);
                    }
                    acc[0][0] = first, acc[1][0] = second;
                }
            } else if (4 * oq < rows && 4 * od < vd) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] *= factor[4 * oq + i];
                auto add_key = [&](int t, auto seen_by) {
                    const float4 w = *reinterpret_cast<const float4*>(ps + t * P_LD + 4 * oq);
                    const float4 v = *reinterpret_cast<const float4*>(vs + t * vd + 4 * od);
                    const float we[4] = {w.x, w.y, w.z, w.w}, ve[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (!seen_by(i)) continue;
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(we[i], ve[j], acc[i][j]);
                    }
                };
                if (whole) {
#pragma unroll 4
                    for (int t = 0; t < count; t++) add_key(t, [](int) { return true; });
                } else {
                    VisibleKeys keys[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) keys[i] = visible_keys(pos + 4 * oq + i, window, chunk, keep);
                    for (int t = 0; t < count; t++)
                        add_key(t, [&](int i) { return c * TK + t <= pos + 4 * oq + i && keys[i].sees(c * TK + t); });
                }
            }
            __syncthreads();                                       // the values and weights are read
            if (c_next <= c_end) fetch(v_cache, vs, vd, vd, v_first, v_step, v_at, buf ^ 1);
            else asm volatile("cp.async.commit_group;\n" ::: "memory");
            c = c_next;
            buf ^= 1;
        }
        if (my_l == 0) factor[my_q] = l_run;
        __syncthreads();
        if (few) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                if (r >= rows || tid >= vd) continue;
                const float l = factor[r];
                out[((size_t)(n + r) * nh + h) * vd + tid] = l > 0.f ? acc[r][0] / l : 0.f;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = 4 * oq + i;
                if (r >= rows || 4 * od >= vd) continue;
                const float l = factor[r];
                float* orow = out + ((size_t)(n + r) * nh + h) * vd + 4 * od;
                *reinterpret_cast<float4*>(orow) = l > 0.f ? make_float4(acc[i][0] / l, acc[i][1] / l, acc[i][2] / l, acc[i][3] / l)
                                                           : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        __syncthreads();                                           // ``factor`` and the places are read before the next run begins
    }
}
}  // namespace

ESP_API int esp_attn_simt(const void* q, const void* k_cache, const void* v_cache, void* out, int is_bf16, int out_is_bf16,
                          const int* tok_seq, const int* tok_pos, const int* block_table, int table_stride, int n_pages,
                          int page, int n_tokens, int nh, int nkv, int hd, int vd, float scale, int sink,
                          const float* sink_vals, int window, int chunk, int keep, float softcap, int maps, int* status,
                          cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (vd <= 0) vd = hd;
    if (vd > MAX_HD || hd > MAX_HD || hd <= 0 || nkv <= 0 || nh % nkv != 0 || nh > 65535 || maps <= 0 || (nh / nkv) % maps != 0)
        return (int)cudaErrorInvalidValue;
    dim3 grid(n_tokens, nh);
    // by sizes and alignment alone, never by the number of tokens: a row has the same bits in a prompt and by itself
    const uintptr_t ends = (uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out;
    if (!is_bf16 && !out_is_bf16 && maps == 1 && hd % 4 == 0 && vd % 4 == 0 && hd <= 128 && vd <= 128 && ends % 16 == 0) {
        const int bytes = (TK * (hd + 4) + TK * vd + TQ * hd + TK * P_LD + TQ) * (int)sizeof(float);
        static bool raised[64] = {false};          // per device: the attribute belongs to the device's context
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return (int)cudaErrorInvalidDevice;
        if (!raised[device]) {
            const cudaError_t e = cudaFuncSetAttribute(attn_simt_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
            if (e != cudaSuccess) return (int)e;
            raised[device] = true;
        }
        // How many blocks share a window of 16 tokens: its runs are between one (a prompt) and 16 (a token of each sequence), which the
        // host does not know.  As many as it takes to fill the device four times over with two blocks an SM; those without a run
        // leave at once, and come last, as blockIdx.z varies slowest.
        const long long windows = (n_tokens + TQ - 1) / TQ * (long long)nh;
        const int sharing = (int)(windows >= 4 * 2 * 148 ? 1 : (4 * 2 * 148 + windows - 1) / windows);
        attn_simt_tile_kernel<<<dim3((n_tokens + TQ - 1) / TQ, nh, sharing < TQ ? sharing : TQ), THREADS, bytes, stream>>>(
            (const float*)q, (const float*)k_cache, (const float*)v_cache, (float*)out, tok_seq, tok_pos, block_table, table_stride, n_pages,
            page, n_tokens, nh, nkv, hd, vd, scale, sink, sink_vals, window, chunk, keep, softcap, status);
        return esp_launch_status();
    }
#define ESP_SIMT(T, TO)                                                                                                    \
    attn_simt_kernel<T, TO><<<grid, THREADS, 0, stream>>>((const T*)q, (const T*)k_cache, (const T*)v_cache, (TO*)out, tok_seq, \
                                                          tok_pos, block_table, table_stride, n_pages, page, nh, nkv, hd, vd, \
                                                          scale, sink, sink_vals, window, chunk, keep, softcap, maps, status)
    if (is_bf16 && out_is_bf16) ESP_SIMT(bf16, bf16);
    else if (is_bf16) ESP_SIMT(bf16, float);
    else if (!out_is_bf16) ESP_SIMT(float, float);
    else return (int)cudaErrorInvalidValue;
#undef ESP_SIMT
    return esp_launch_status();
}
