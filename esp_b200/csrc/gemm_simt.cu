// Matrix product on the CUDA cores with true 32-bit multiply-adds:
//   C[m, n] = (sum_k A[row(m), k] * W[g][n, k] + bias[n]) * row_scale[m]
// A and W may be float or bfloat16 (widened exactly), the sum is float, C is
// float or bfloat16.  Each output element adds its products in the order
// k = 0, 1, 2, ... whatever the kernel and the tile it falls in, so a row's
// result does not depend on how many other rows are in the call.  This is the
// 32-bit path of every projection and the fallback for weight dtypes that the
// fast kernels do not take.
//
// Grouped form: rows are sorted by group, group g owns rows
// [group_offsets[g], group_offsets[g+1]) and its own [N, K] slice of W.
//
// Two kernels share that order.  ``gemm_simt_kernel`` cuts the output into tiles and is bound by the multiply-add
// units; ``gemm_simt_few_kernel`` streams the weights past eight rows a block and is bound by memory or, for few columns, by
// the chain of K dependent additions.
#include "common.cuh"

namespace {
// acc.lo = a.lo * b.lo + acc.lo, acc.hi = a.hi * b.hi + acc.hi, each rounded as fmaf rounds
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

__device__ __forceinline__ float4 widen4(uint2 v) {
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&v.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
    const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
    return make_float4(a.x, a.y, b.x, b.y);
}
// Four values from p[k] as they lie in memory; those at K and beyond are zero.  ``wide``: p + k is aligned to four values
// and K a multiple of four.  They become floats only when they are asked for: a conversion beside the load would wait for it.
template <typename T> struct Loaded4;
template <> struct Loaded4<float> {
    float4 v;
    __device__ __forceinline__ void load(const float* p, int k, int K, bool wide) {
        v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!p) return;
        if (wide) {
            if (k < K) v = __ldg(reinterpret_cast<const float4*>(p + k));
        } else {
            if (k < K) v.x = p[k];
            if (k + 1 < K) v.y = p[k + 1];
            if (k + 2 < K) v.z = p[k + 2];
            if (k + 3 < K) v.w = p[k + 3];
        }
    }
    __device__ __forceinline__ float4 get(bool) const { return v; }
};
template <> struct Loaded4<bf16> {
    uint2 pairs;                         // wide
    unsigned short one[4];               // else
    __device__ __forceinline__ void load(const bf16* p, int k, int K, bool wide) {
        pairs = make_uint2(0u, 0u);
#pragma unroll
        for (int i = 0; i < 4; i++) one[i] = 0;
        if (!p) return;
        if (wide) {
            if (k < K) pairs = __ldg(reinterpret_cast<const uint2*>(p + k));
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (k + i < K) one[i] = __ldg(reinterpret_cast<const unsigned short*>(p) + k + i);
        }
    }
    __device__ __forceinline__ float4 get(bool wide) const {
        if (wide) return widen4(pairs);
        return make_float4(__uint_as_float((unsigned)one[0] << 16), __uint_as_float((unsigned)one[1] << 16),
                           __uint_as_float((unsigned)one[2] << 16), __uint_as_float((unsigned)one[3] << 16));
    }
};

struct SimtParams {
    const void* A;
    const int* a_rows;
    const void* W;
    const float* bias;
    const float* row_scale;
    void* C;
    const int* group_offsets;
    int groups, M, N, K;
    long long lda, ldc;
    int wide_a, wide_w;
};

// The row tile that block ``tile`` of a grouped product works on: groups have ceil(rows / BM) tiles each, in order.
// Every warp finds it by itself.  Returns false past the last tile.
template <int BM>
__device__ __forceinline__ bool group_tile(const SimtParams& p, int tile, int& group, int& m0, int& m_end) {
    constexpr int ROUNDS = 4;                                        // of 32 groups whose offsets are asked for at once
    const int lane = threadIdx.x & 31;
    int before = 0;
    bool found = false;
    for (int g0 = 0; g0 < p.groups; g0 += 32 * ROUNDS) {
        int begin[ROUNDS], end[ROUNDS];
#pragma unroll
        for (int r = 0; r < ROUNDS; r++) {
            const int g = g0 + 32 * r + lane;
            begin[r] = g < p.groups ? p.group_offsets[g] : 0;
            end[r] = g < p.groups ? p.group_offsets[g + 1] : 0;
        }
#pragma unroll
        for (int r = 0; r < ROUNDS; r++) {
            const int tiles = end[r] > begin[r] ? (end[r] - begin[r] + BM - 1) / BM : 0;
            int upto = tiles;                                        // tiles of the lanes up to this one
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const bool mine = tile >= before + upto - tiles && tile < before + upto;
            const unsigned hit = __ballot_sync(0xffffffffu, mine);
            if (hit) {                                               // of one round at most
                const int src = __ffs(hit) - 1;
                const int first = begin[r] + (tile - (before + upto - tiles)) * BM;
                group = g0 + 32 * r + src;
                m0 = __shfl_sync(0xffffffffu, first, src);
                m_end = __shfl_sync(0xffffffffu, end[r], src);
                found = true;
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (found) break;
    }
    return found;
}

template <typename TC>
__device__ __forceinline__ void store_out(const SimtParams& p, int m, int n, float v, float scale) {
    if (p.bias) v += p.bias[n];
    if (p.row_scale) v *= scale;
    reinterpret_cast<TC*>(p.C)[(size_t)m * p.ldc + n] = from_f32<TC>(v);
}

constexpr int BK = 16, TM = 8;

// One tile of BM x BN outputs per block of BM / 8 x BN / TN threads, each with 8 x TN of them in registers, so that one k
// takes (8 + TN) / 4 shared loads of 16 bytes for 8 TN multiply-adds, which go out two at a time (fma.rn.f32x2).  A warp
// whose rows all lie behind the group's end does not multiply, and the warps' roles turn with the block so that the idle
// ones do not always fall on the same quarter of the SM.  The next k tile travels through registers while this one is
// multiplied.  Bound by the multiply-add pipe (72.8 TFLOP/s at 1,925 MHz) and by the last wave of tiles: 1,400 rows,
// N = 11,264, K = 2,048 in 1.29 ms, 50 TFLOP/s (61 without the last wave); with tiles of 64 x 64, 4 x 4 outputs a thread
// and one buffer it was 2.58 ms.
template <typename TA, typename TW, typename TC, int BM, int BN, int TN, int MIN_BLOCKS>
__global__ void __launch_bounds__(BM / TM * (BN / TN), MIN_BLOCKS)
gemm_simt_kernel(SimtParams p, int m_tiles) {
    constexpr int THREADS = BM / TM * (BN / TN), TX = BN / TN, WARPS = THREADS / 32;
    constexpr int WARP_ROWS = 32 / TX * TM;
    constexpr int A_LD = BM + 4, W_LD = BN + 4;
    constexpr int A_LOADS = BM * BK / 4 / THREADS, W_LOADS = BN * BK / 4 / THREADS;
    static_assert(32 % TX == 0 && A_LOADS * THREADS * 4 == BM * BK && W_LOADS * THREADS * 4 == BN * BK, "whole loads");
    __shared__ __align__(16) float As[2][BK][A_LD];
    __shared__ __align__(16) float Ws[2][BK][W_LD];
    int m0, m_end = p.M, group = 0;
    const int m_tile = blockIdx.x % m_tiles, n0 = (blockIdx.x / m_tiles) * BN;     // row tiles vary fastest: a run of blocks shares its weights
    if (p.group_offsets) {
        if (!group_tile<BM>(p, m_tile, group, m0, m_end)) return;
    } else {
        m0 = m_tile * BM;
    }
    const TW* Wg = reinterpret_cast<const TW*>(p.W) + (size_t)group * p.N * p.K;
    const int tid = threadIdx.x;
    const int turned = (((tid >> 5) + blockIdx.x) % WARPS) * 32 + (tid & 31);
    const int ty = turned / TX, tx = turned % TX;
    const bool busy = m0 + turned / 32 * WARP_ROWS < m_end;           // the same for a whole warp

    // this thread's places in the two k tiles: rows tid / 4 + i * THREADS / 4, values (tid % 4) * 4 .. + 3
    const int lrow = tid / 4, lk = (tid % 4) * 4;
    const TA* a_src[A_LOADS];
    const TW* w_src[W_LOADS];
#pragma unroll
    for (int i = 0; i < A_LOADS; i++) {
        const int m = m0 + lrow + i * (THREADS / 4);
        a_src[i] = m < m_end ? reinterpret_cast<const TA*>(p.A) + (size_t)(p.a_rows ? p.a_rows[m] : m) * p.lda : nullptr;
    }
#pragma unroll
    for (int i = 0; i < W_LOADS; i++) {
        const int n = n0 + lrow + i * (THREADS / 4);
        w_src[i] = n < p.N ? Wg + (size_t)n * p.K : nullptr;
    }
    Loaded4<TA> a_next[A_LOADS];
    Loaded4<TW> w_next[W_LOADS];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < A_LOADS; i++) a_next[i].load(a_src[i], k0 + lk, p.K, p.wide_a);
#pragma unroll
        for (int i = 0; i < W_LOADS; i++) w_next[i].load(w_src[i], k0 + lk, p.K, p.wide_w);
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < A_LOADS; i++) {
            float* d = &As[buf][lk][lrow + i * (THREADS / 4)];
            const float4 v = a_next[i].get(p.wide_a);
            d[0] = v.x, d[A_LD] = v.y, d[2 * A_LD] = v.z, d[3 * A_LD] = v.w;
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; i++) {
            float* d = &Ws[buf][lk][lrow + i * (THREADS / 4)];
            const float4 v = w_next[i].get(p.wide_w);
            d[0] = v.x, d[W_LD] = v.y, d[2 * W_LD] = v.z, d[3 * W_LD] = v.w;
        }
    };

    // acc[i][j]: row ty * 8 + i of the columns c and c + 1, c = (j / 2) * (BN / (TN / 4)) + tx * 4 + j % 2 * 2
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;
    // what one k needs, read one k ahead
    struct Piece {
        float4 a[TM / 4];
        ulonglong2 w[TN / 4];
    };
    auto piece = [&](Piece& d, int buf, int kk) {
#pragma unroll
        for (int i = 0; i < TM / 4; i++) d.a[i] = *reinterpret_cast<const float4*>(&As[buf][kk][ty * TM + 4 * i]);
#pragma unroll
        for (int q = 0; q < TN / 4; q++) d.w[q] = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][q * (BN / (TN / 4)) + tx * 4]);
    };
    auto multiply = [&](const Piece& d) {
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const float4 v = d.a[i / 4];
            const float x = i % 4 == 0 ? v.x : i % 4 == 1 ? v.y : i % 4 == 2 ? v.z : v.w;
            const unsigned long long x2 = pack2(x, x);
#pragma unroll
            for (int q = 0; q < TN / 4; q++) {
                fma2(acc[i][2 * q], x2, d.w[q].x);
                fma2(acc[i][2 * q + 1], x2, d.w[q].y);
            }
        }
    };

    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < p.K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < p.K;
        if (more) fetch(k0 + BK);
        if (busy) {
            Piece one, two;
            piece(one, buf, 0);
#pragma unroll
            for (int kk = 0; kk < BK; kk += 2) {
                piece(two, buf, kk + 1);
                multiply(one);
                if (kk + 2 < BK) piece(one, buf, kk + 2);
                multiply(two);
            }
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + ty * TM + i;
        if (m >= m_end) continue;
        const float scale = p.row_scale ? p.row_scale[m] : 1.0f;
#pragma unroll
        for (int j = 0; j < TN / 2; j++) {
            const int n = n0 + (j / 2) * (BN / (TN / 4)) + tx * 4 + j % 2 * 2;
            const float2 v = unpack2(acc[i][j]);
            if (n < p.N) store_out<TC>(p, m, n, v.x, scale);
            if (n + 1 < p.N) store_out<TC>(p, m, n + 1, v.y, scale);
        }
    }
}

constexpr int FEW_ROWS = 8;

__device__ __forceinline__ void copy16(void* dst, const void* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ float4 read4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 read4(const bf16* p) { return widen4(*reinterpret_cast<const uint2*>(p)); }

// BN columns against up to eight rows; a thread has RT rows of CT columns.  Further rows are further blocks', which find the
// weights in L2: a block that took a group's rows eight by eight made 90 passes over them where 720 rows fell to one group.  The weights (and the rows) pass
// through a ring of FEW_STAGES pieces of FEW_K k in shared memory, filled by cp.async, so that the loads run ahead of the
// chains of additions.  The ring's size is known to the compiler (no dynamic shared memory): it then spends the registers
// that the ring leaves on reading several k ahead; without, 6 x 2,048 x 2,048 takes 28 us instead of 20.  Wants rows of A
// and W that start on 16 bytes and K a whole number of 16-byte pieces.  Six rows, K = 2,048, the tile kernel of before ->
// this one: N = 151,936 1,412 -> 249 us (5.0 TB/s), N = 6,144 180 -> 31, N = 2,048 179 -> 21 (the chain of 2,048
// additions is 4.3 of them).
template <typename TA, typename TW, typename TC, int BN, int RT, int CT, int FEW_K, int FEW_STAGES>
__global__ void __launch_bounds__(BN / CT * (FEW_ROWS / RT))
gemm_simt_few_kernel(SimtParams p, int chunks) {
    constexpr int TX = BN / CT, THREADS = TX * (FEW_ROWS / RT);
    constexpr int A_PIECE = 16 / sizeof(TA), W_PIECE = 16 / sizeof(TW);
    constexpr int A_LD = FEW_K + A_PIECE, W_LD = FEW_K + W_PIECE;      // 16 bytes apart in the banks from row to row
    __shared__ __align__(16) TA As[FEW_STAGES][FEW_ROWS][A_LD];
    __shared__ __align__(16) TW Ws[FEW_STAGES][BN][W_LD];
    // Dense: the eights of rows vary fastest, so that they share a read of their weights.  Groups: the columns do, as the
    // blocks behind the last eight have nothing to do and would leave the others unevenly spread over the SMs.
    int m0, m_end = p.M, group = 0, n0;
    if (p.group_offsets) {
        const int n_tiles = (p.N + BN - 1) / BN;
        n0 = blockIdx.x % n_tiles * BN;
        if (!group_tile<FEW_ROWS>(p, blockIdx.x / n_tiles, group, m0, m_end)) return;
    } else {
        n0 = blockIdx.x / chunks * BN;
        m0 = blockIdx.x % chunks * FEW_ROWS;
    }
    const int tid = threadIdx.x, col = tid % TX, r0 = tid / TX * RT;
    const int steps = (p.K + FEW_K - 1) / FEW_K, rows = min(FEW_ROWS, m_end - m0);
    // this thread's places in a stage: of the weights rows wr + j * W_ROWS at wk, of A rows ar + j * A_ROWS at ak
    constexpr int W_LINE = FEW_K / W_PIECE, W_ROWS = THREADS / W_LINE, W_COPIES = BN / W_ROWS;
    constexpr int A_LINE = FEW_K / A_PIECE, A_ROWS = THREADS / A_LINE, A_COPIES = (FEW_ROWS + A_ROWS - 1) / A_ROWS;
    static_assert(W_ROWS * W_LINE == THREADS && W_COPIES * W_ROWS == BN && A_ROWS * A_LINE == THREADS, "whole lines");
    const int wr = tid / W_LINE, wk = tid % W_LINE * W_PIECE, ar = tid / A_LINE, ak = tid % A_LINE * A_PIECE;
    const TW* const Wg = reinterpret_cast<const TW*>(p.W) + (size_t)group * p.N * p.K;
    const TW* const w_src = Wg + (size_t)(n0 + wr) * p.K + wk;
    const TA* a_src[A_COPIES];
#pragma unroll
    for (int j = 0; j < A_COPIES; j++) {
        const int r = ar + j * A_ROWS;
        a_src[j] = r < rows ? reinterpret_cast<const TA*>(p.A) + (size_t)(p.a_rows ? p.a_rows[m0 + r] : m0 + r) * p.lda + ak : nullptr;
    }
    auto fill = [&](int step) {
        if (step < steps) {
            const int k0 = step * FEW_K, s = step % FEW_STAGES;
#pragma unroll
            for (int j = 0; j < W_COPIES; j++) {
                const bool valid = n0 + wr + j * W_ROWS < p.N && k0 + wk < p.K;
                copy16(&Ws[s][wr + j * W_ROWS][wk], valid ? w_src + (size_t)j * W_ROWS * p.K + k0 : Wg, valid);
            }
#pragma unroll
            for (int j = 0; j < A_COPIES; j++)
                if (a_src[j] && k0 + ak < p.K) copy16(&As[s][ar + j * A_ROWS][ak], a_src[j] + k0, true);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int s = 0; s < FEW_STAGES - 1; s++) fill(s);
    float acc[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < CT; j++) acc[i][j] = 0.f;
    const bool busy = r0 < rows;
    for (int step = 0; step < steps; step++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(FEW_STAGES - 2) : "memory");
        __syncthreads();                                          // the stage is whole, and the one filled next is read out
        fill(step + FEW_STAGES - 1);
        if (!busy) continue;
        const int s = step % FEW_STAGES, left = p.K - step * FEW_K;
        auto four = [&](int k) {
            float4 av[RT], wv[CT];
#pragma unroll
            for (int j = 0; j < CT; j++) wv[j] = read4(&Ws[s][j * TX + col][k]);
#pragma unroll
            for (int i = 0; i < RT; i++) av[i] = read4(&As[s][r0 + i][k]);        // rows behind the last one: whatever is there, never stored
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < CT; j++)
                    acc[i][j] = fmaf(av[i].w, wv[j].w, fmaf(av[i].z, wv[j].z, fmaf(av[i].y, wv[j].y, fmaf(av[i].x, wv[j].x, acc[i][j]))));
        };
        if (left >= FEW_K) {
#pragma unroll
            for (int k = 0; k < FEW_K; k += 4) four(k);
        } else {
            for (int k = 0; k < left; k += 4) four(k);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < RT; i++) {
        if (r0 + i >= rows) continue;
        const int m = m0 + r0 + i;
        const float scale = p.row_scale ? p.row_scale[m] : 1.0f;
#pragma unroll
        for (int j = 0; j < CT; j++) {
            const int n = n0 + j * TX + col;
            if (n < p.N) store_out<TC>(p, m, n, acc[i][j], scale);
        }
    }
}

template <typename TA, typename TW, typename TC, int BN, int RT, int CT, int FEW_K, int FEW_STAGES>
int launch_few(const SimtParams& p, cudaStream_t stream) {
    // Eights of rows: of groups an upper bound, as a group that has rows has one and another for every eight behind its first
    const long long first = p.group_offsets ? min(p.M, p.groups) : 0;
    const long long chunks = first + (p.group_offsets ? (p.M - first) / FEW_ROWS : (p.M + FEW_ROWS - 1) / FEW_ROWS);
    const long long blocks = chunks * ((p.N + BN - 1) / BN);
    if (blocks > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    gemm_simt_few_kernel<TA, TW, TC, BN, RT, CT, FEW_K, FEW_STAGES>
        <<<(unsigned)blocks, BN / CT * (FEW_ROWS / RT), 0, stream>>>(p, (int)chunks);
    return esp_launch_status();
}

template <typename TA, typename TW, typename TC, int BM, int BN, int TN, int MIN_BLOCKS>
int launch_tiles(const SimtParams& p, cudaStream_t stream) {
    const long long m_tiles = (p.M + BM - 1) / BM + (p.group_offsets ? p.groups : 0);       // of groups: an upper bound
    const long long blocks = m_tiles * ((p.N + BN - 1) / BN);
    if (blocks > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    gemm_simt_kernel<TA, TW, TC, BM, BN, TN, MIN_BLOCKS><<<(unsigned)blocks, BM / TM * (BN / TN), 0, stream>>>(p, (int)m_tiles);
    return esp_launch_status();
}

template <typename TA, typename TW, typename TC>
int launch(SimtParams p, cudaStream_t stream) {
    auto wide = [&](const void* base, long long ld, int size, int values) {
        return (uintptr_t)base % (values * size) == 0 && ld % values == 0 && p.K % values == 0;
    };
    p.wide_a = wide(p.A, p.lda, sizeof(TA), 4);
    p.wide_w = wide(p.W, p.K, sizeof(TW), 4);
    const bool grouped = p.group_offsets != nullptr;
    const long long groups = grouped ? p.groups : 1;
    // Few rows: up to 24 pass the weights in eights, faster than a tile (N = 2,048: 24 rows 31 us against 110; N = 151,936: 24 rows
    // 533 against 711), and more of them while the eights' outputs of a row are at most 46,000 in all, a few waves of blocks
    // (N = 2,048: 64 rows 50 us against 113; N = 11,264: 32 rows 108 against 124, 40 rows 128 against 125; K = 5,632, N = 6,144: 64 rows
    // 311 against 297).  Of a group about 12 on average, however they are spread (60 groups, N = 2,816, 400 rows in all: even 254 us
    // against 388, all in one group 182 against 375 with the tiles of 64 x 64 of before; 720 rows 402 and 318 against 1,553 and 595).  Four by two outputs a thread read shared memory least; they want as many blocks
    // as the SMs hold at once (four each), below that two by one have the more warps (6 rows, N = 2,048: 21 us against 37).
    const bool few = grouped ? p.M <= 12 * groups : p.M <= 24 || (p.M + 7ll) / 8 * p.N <= 46000;
    if (few && wide(p.A, p.lda, sizeof(TA), 16 / sizeof(TA)) && wide(p.W, p.K, sizeof(TW), 16 / sizeof(TW))) {
        if ((p.N + 63) / 64 * groups >= 592) return launch_few<TA, TW, TC, 64, 4, 2, 64, 2>(p, stream);
        return launch_few<TA, TW, TC, 32, 2, 1, 64, 4>(p, stream);
    }
    // Tiles: the larger one multiplies faster, the smaller one leaves less of the last wave (and of a group's end) empty.
    // Dense: what the busiest SM multiplies, with the smaller tile's outputs at 0.87 of the larger one's rate, tells them apart
    // (1,400 rows: N = 11,264 1.29 ms against 1.46, N = 2,048 400 us against 304; 200 rows, N = 2,048 236 us against 104).
    // Grouped, 60 groups, N = 2,816: 5,600 rows 1.63 ms against 1.80 and 1.82 (32 rows a tile), 800 rows 1.26 ms against
    // 0.66 and 0.54.
    if (grouped && p.M < 24 * groups) return launch_tiles<TA, TW, TC, 32, 64, 4, 6>(p, stream);
    auto busiest = [&](long long bm, long long bn) {
        return (((p.M + bm - 1) / bm) * ((p.N + bn - 1) / bn) + 147) / 148 * bm * bn;
    };
    if (grouped ? p.M >= 64 * groups : 87 * busiest(128, 128) <= 100 * busiest(64, 64))
        return launch_tiles<TA, TW, TC, 128, 128, 16, 2>(p, stream);
    return launch_tiles<TA, TW, TC, 64, 64, 4, 4>(p, stream);
}
}  // namespace

// dtype codes: 0 = float, 1 = bfloat16.  M is the total number of rows (for the
// grouped form: the upper bound of any group's row count as well).
ESP_API int esp_gemm_simt(const void* A, int a_dtype, const int* a_rows, const void* W, int w_dtype, const float* bias,
                          const float* row_scale, void* C, int c_dtype, const int* group_offsets, int groups, int M,
                          int N, int K, long long lda, long long ldc, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if ((long long)((M + 63) / 64) > 65535 || groups > 65535) return (int)cudaErrorInvalidValue;
    const SimtParams p{A, a_rows, W, bias, row_scale, C, group_offsets, groups, M, N, K, lda, ldc, 0, 0};
    const int code = a_dtype * 4 + w_dtype * 2 + c_dtype;
#define ESP_CASE(code_, TA, TW, TC) case code_: return launch<TA, TW, TC>(p, stream);
    switch (code) {
        ESP_CASE(0, float, float, float)
        ESP_CASE(1, float, float, bf16)
        ESP_CASE(2, float, bf16, float)
        ESP_CASE(3, float, bf16, bf16)
        ESP_CASE(4, bf16, float, float)
        ESP_CASE(5, bf16, float, bf16)
        ESP_CASE(6, bf16, bf16, float)
        ESP_CASE(7, bf16, bf16, bf16)
    }
#undef ESP_CASE
    return (int)cudaErrorInvalidValue;
}
