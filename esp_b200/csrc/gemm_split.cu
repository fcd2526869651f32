// 32-bit matrix product on the 5th-generation tensor cores:
//   C[m, n] = (sum_k A[row(m), k] * W[g][n, k] + bias[n]) * row_scale[m],   A, W, C float.
//
// A float is the sum of three bfloat16 numbers exactly (8 + 8 + 8 bits of mantissa, each piece rounded to nearest; numbers below
// 2^-110, 1e-33, lose what is below 2^-133, bfloat16's smallest), and the product of two bfloat16 numbers is exact in 32 bits.  So
// with x = x1 + x2 + x3 the product a * w is made of
//   main = a1 w1,   c1 = a2 w1 + a1 w2 + a1 w3,   c2 = a3 w1 + a2 w2 + a2 w3,
// which are summed over k in three accumulators of their own in tensor memory; what is left out (a3 w2, a3 w3) is at most 2^-25 of a
// product (|a3| <= 2^-17 and |w2| <= 2^-8 of the powers of two that a and w start with).  The tensor core cuts its sums off instead of
// rounding them.  That error has one sign, so it grows with the number of additions and not with its root, most where one product or a
// growing sum outweighs what is added.  So main is read out every SUB stages, 128 k, and added up with ordinary rounded additions.  c1
// and c2 are 2^-8 of main and are read out a segment (256 to 1,024 k), whose value main + (c1 + c2) is added to the running sum.
// The order of everything depends on k alone, so a row's result has the same bits whatever other rows are in the call, whatever the
// tile's width, whichever group the rows lie in and however many CTAs share a tile.
// Error against 64 bits (2-norm), this kernel / a chain of multiply-adds, K = 1,024, 2,048, 5,632: normal operands 1.3e-7 / 5.8e-7,
// 1.3e-7 / 8.1e-7, 1.4e-7 / 1.35e-6; positive ones 1.7e-7 / 4.9e-7, 1.7e-7 / 7.0e-7, 1.7e-7 / 1.06e-6; one channel of the rows 300 times
// the others 2.9e-7 / 5.8 to 8.0e-7, 2.9e-7 / 0.8 to 1.2e-6, 2.9e-7 / 1.4 to 1.9e-6 where it stands in the first half.  That channel sets
// SUB: 128 k before the row's end, the place where a chain has least to add behind it, they are 2.8e-7 / 2.95e-7, and SUB twice as
// long doubles ours.  With main read out once a segment the three were 4.7e-7, 4.7e-7, 9.7e-7, 9.0e-7, 9.0e-7, 2.1e-6 and 1.07e-6, 1.06e-6,
// 2.1e-6 (1,400 rows of 11,264 x 2,048 489 us then, 520 now; SUB = 4 502).
//
// Layout: the weights are the 128-row side of the MMA, up to NT token rows its N side; accumulator D[feature, token],
// TMEM lane = feature, columns of n_tok each.  A ring of stages of 64 k: the weights come by TMA into shared
// memory as they are; two groups of four warps take the stages in turn, split a stage and store its pieces as the A operand in
// tensor memory (as shared-memory operands they would cost more of that memory's bandwidth than there is: the token rows' pieces
// alone make the MMAs read 55 bytes a cycle).  Six warps load, split and store the token rows in shared memory (K-major,
// 128-byte swizzle); a gather by a_rows costs nothing.  One thread issues the MMAs.  The pieces of the token rows lie
// one behind the other as N rows [a1 | a2 | a3]: one MMA of n columns multiplies w1 by a1, and three of 2 n columns, into [c1 | c2], w1 by
// [a2 | a3], w2 and w3 by [a1 | a2].  MMAs keep their order where accumulator and shape are the same, and here those that share an
// accumulator have one shape.  (Three MMAs of 3 n, 2 n and n columns into overlapping accumulators would be a seventh less work, but
// nothing says that the second adds to what the first has written.)  Eight warps read the accumulators out.
//
// Main has two sets of columns, so that its read-out runs beside the next MMAs; 64 token rows leave room for two stages of split weights
// then (2 x 64 + 128 + 2 x 96 of 512 columns).
//
// What bounds it, 64 token rows (1,400 rows, N = 11,264, K = 2,048: 520 us, 124 TFLOP/s, multiply-adds 1,251): a stage takes 1,750
// cycles, of which the tensor core works 840 to 900.  The warp that issues (clock64; 1,900 with it) spends 711 of them issuing, 366
// waiting for a stage, 333 for accumulators to be read out and 282 on commits; the warps that split are busy most of the time as well
// (0.66 of the SM's issue slots), so that neither eight warps for the token rows (539 us) nor pieces made before their slot is free
// (623) nor all eight weight warps on each stage (673) helped.  Short tiles: 1,200 to 1,500 cycles a stage; six rows, N = 151,936 in
// 234 us, 5.3 TB/s; one row, N = 11,264 / 6,144 / 2,048 26 to 30 / 18 / 10 us where multiply-adds take 21 / 17 / 14, K = 5,632, N = 2,048
// 17 and 34.
//
// Persistent: a CTA per SM walks the tiles with the grid's stride; loads run ahead over the ends of tiles.  Every wait is
// bounded, and begun behind pdl_wait() where it hangs on the token rows, so that it times this kernel and not those before it (one
// may start beside a scan of many milliseconds, two launches back): if one runs out the kernel raises ESP_STATUS_WAIT_EXPIRED, stops,
// waits for its own copies and MMAs, frees its tensor memory and returns.  The lanes of a warp leave a role together: tcgen05.ld and
// .st and the barriers behind them want whole warps.
//
// Elements whose result is not finite (an infinity or a number beyond bfloat16's range among the operands would spread through the
// pieces) are made again with a chain of fused multiply-adds, by all warps of a CTA when its tiles are done: in the read-out, where
// others wait for its warps, one such row of six took 4.3 times the whole product (N = 40,000, K = 2,048).  A row of A with a NaN is
// NaN as it is.
#include "tc05.cuh"

namespace {
using namespace tc05;

constexpr int BF = 128;                    // weight rows (features) of a tile
constexpr int KS = 64;                     // k of a stage: four 16-wide MMA steps, 128 bytes of a token row's piece
constexpr int A_COLS = 3 * KS / 2;         // TMEM columns of a stage of weights
constexpr int RAW_BYTES = BF * KS * 4;     // the same as it comes: [4 steps][128 rows][16 k] float
constexpr int MAX_GROUPS = 256;
constexpr int MAX_PARTS = 8;               // segments of a tile that several CTAs share
constexpr int SUB = 2;                     // stages whose main products are summed in the tensor core
// k of a segment, a multiple of SUB stages: 256, from K = 1,024 on 512, from K = 4,096 on 1,024
__host__ __device__ constexpr int segment_of(int K) { return K >= 4096 ? 1024 : K >= 1024 ? 512 : 256; }
constexpr int W_WARPS = 8, E_WARPS = 8, T_WARPS = 6;     // with the one that issues the copies and the one that issues the MMAs: 24 warps
constexpr int T_ROWS = T_WARPS * 4;        // token rows that the T_WARPS take at once, eight threads a row
constexpr int THREADS = (W_WARPS + E_WARPS + T_WARPS + 2) * 32;

struct SplitParams {
    const float* A;
    const int* a_rows;
    const float* W;
    const float* bias;
    const float* row_scale;
    float* C;
    const int* group_offsets;
    int groups, M, N, K;
    long long lda, ldc;
    int seg_stages, share;                 // stages of a segment; CTAs of a cluster that share a tile
    unsigned polls;                        // of a wait, at most
    int* status;
};

struct Tile {
    int group, m0, rows, n_tok, f0;        // n_tok: rows rounded up to 16
};

// A group that has rows, and the number of tiles of the groups before it.
struct Group {
    int group, begin, rows, before;
};
template <int NT> __device__ __forceinline__ int runs_of(int rows) { return (rows + NT - 1) / NT; }

// Lists the groups that have rows in shared memory (one warp).  Every role of a CTA walks this list, some several times: looked up in
// the offsets one by one, 60 groups took a role 2 us at the start of its first tile and again behind its last one.
template <int NT>
__device__ __forceinline__ void list_groups(const SplitParams& p, Group* list, int* count) {
    const int lane = threadIdx.x & 31, feat_tiles = (p.N + BF - 1) / BF;
    if (!p.group_offsets) {
        if (lane == 0) list[0] = Group{0, 0, p.M, 0}, *count = 1;
        return;
    }
    int at = 0, before = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 128) {
        int begin[4], rows[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int g = g0 + 32 * r + lane;
            begin[r] = g < p.groups ? p.group_offsets[g] : 0;
            rows[r] = g < p.groups ? min(p.M, p.group_offsets[g + 1]) - begin[r] : 0;
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const unsigned some = __ballot_sync(0xffffffffu, rows[r] > 0);
            const int tiles = rows[r] > 0 ? runs_of<NT>(rows[r]) * feat_tiles : 0;
            int upto = tiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (rows[r] > 0) list[at + __popc(some & ((1u << lane) - 1))] = Group{g0 + 32 * r + lane, begin[r], rows[r], before + upto - tiles};
            at += __popc(some);
            before += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (lane == 0) *count = at;
}

// Walks the tiles of a CTA (or of the ``share`` CTAs of a cluster) in order.  A group's rows are cut evenly into ceil(rows / NT)
// runs; its tiles are all runs of the first 128 features, then of the next (neighbours share their weights).
template <int NT>
struct Walk {
    const Group* list;
    int count, feat_tiles, tile, step, at;
    __device__ __forceinline__ Walk(const SplitParams& p, const Group* list_, int count_) : list(list_), count(count_), at(0) {
        feat_tiles = (p.N + BF - 1) / BF;
        step = gridDim.x / p.share;
        tile = (int)(blockIdx.x / p.share) - step;
    }
    __device__ __forceinline__ bool next(Tile& t) {
        tile += step;
        for (; at < count; at++) {
            const Group g = list[at];
            const int runs = runs_of<NT>(g.rows), i = tile - g.before;
            if (i >= runs * feat_tiles) continue;
            const int width = ((g.rows + runs - 1) / runs + 15) / 16 * 16, run = i % runs;
            t.group = g.group;
            t.m0 = g.begin + run * width;
            t.rows = min(width, g.rows - run * width);
            t.n_tok = (t.rows + 15) / 16 * 16;
            t.f0 = i / runs * BF;
            return true;
        }
        return false;
    }
};

// two floats, each rounded to bfloat16; the first in the low half
__device__ __forceinline__ unsigned round2(float lo, float hi) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// the next piece of two floats, packed; what is left of them stays (one subtraction for both)
__device__ __forceinline__ unsigned take2(float& x, float& y) {
    const unsigned q = round2(x, y);
    asm("{\n.reg .b64 a, b;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nsub.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(x), "+f"(y) : "f"(__uint_as_float(q << 16)), "f"(__uint_as_float(q & 0xFFFF0000u)));
    return q;
}
// 16 lanes x 16 columns: of each run of 8 columns this thread's first two words go to lane t / 4, columns 2 (t % 4) and the
// next, the other two eight lanes further
__device__ __forceinline__ void tc_st_16x256(unsigned taddr, const unsigned (&a)[2], const unsigned (&b)[2], const unsigned (&c)[2],
                                             const unsigned (&d)[2]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 ::"r"(taddr), "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]), "r"(c[0]), "r"(c[1]), "r"(d[0]), "r"(d[1]) : "memory");
}
// two times 16 consecutive float columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld16x2(unsigned ta, float (&a)[16], unsigned tb, float (&b)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=&f"(a[0]), "=&f"(a[1]), "=&f"(a[2]), "=&f"(a[3]), "=&f"(a[4]), "=&f"(a[5]), "=&f"(a[6]), "=&f"(a[7]), "=&f"(a[8]),
          "=&f"(a[9]), "=&f"(a[10]), "=&f"(a[11]), "=&f"(a[12]), "=&f"(a[13]), "=&f"(a[14]), "=&f"(a[15]), "=&f"(b[0]), "=&f"(b[1]),
          "=&f"(b[2]), "=&f"(b[3]), "=&f"(b[4]), "=&f"(b[5]), "=&f"(b[6]), "=&f"(b[7]), "=&f"(b[8]), "=&f"(b[9]), "=&f"(b[10]),
          "=&f"(b[11]), "=&f"(b[12]), "=&f"(b[13]), "=&f"(b[14]), "=&f"(b[15])
        : "r"(ta), "r"(tb) : "memory");
}
// one lane of a whole warp, always the same
__device__ __forceinline__ bool elect_one() {
    unsigned r;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}
// tc_mma_ta with the operand descriptor given as its two words
__device__ __forceinline__ void tc_mma_ta_lo(unsigned tmem_d, unsigned tmem_a, unsigned b_lo, unsigned b_hi, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 db;\n"
        "setp.ne.b32 p, %5, 0;\n"
        "mov.b64 db, {%2, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
// bfloat16 x bfloat16 -> float, B K-major (A in tensor memory), M = 128, N = n
__device__ __forceinline__ unsigned split_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(BF >> 4) << 24);
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// A value to the same place in the shared memory of another CTA of the cluster.
__device__ __forceinline__ void st_cluster(float* p, unsigned rank, float v) {
    unsigned there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(there) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(there), "f"(v) : "memory");
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }
__device__ __forceinline__ const float* a_row(const SplitParams& p, int m) { return p.A + (size_t)(p.a_rows ? p.a_rows[m] : m) * p.lda; }
// The element of row m (of the whole product) and feature n from its sum.
__device__ __forceinline__ void store(const SplitParams& p, int m, int n, float v) {
    if (p.bias) v += p.bias[n];
    if (p.row_scale) v *= p.row_scale[m];
    p.C[(size_t)m * p.ldc + n] = v;
}

// Makes the elements of a tile that are not finite again, each as a chain of fused multiply-adds.  A warp to a row; whole CTA.
__device__ __forceinline__ void chains(const SplitParams& p, const Tile& t) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < t.rows; r += THREADS / 32) {
        const int m = t.m0 + r;
        const float* a = a_row(p, m);
        unsigned odd = 0;
        for (int j = 0; j < BF / 32; j++) {
            const int n = t.f0 + 32 * j + lane;
            if (n < p.N && !finite(p.C[(size_t)m * p.ldc + n])) odd |= 1u << j;
        }
        if (!__any_sync(0xffffffffu, odd != 0)) continue;
        bool nan = false;
        for (int k = lane * 4; k < p.K; k += 128) {
            const float4 v = *reinterpret_cast<const float4*>(a + k);
            nan |= isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
        }
        if (__any_sync(0xffffffffu, nan)) continue;
        for (int j = 0; j < BF / 32; j++) {
            if (!(odd >> j & 1)) continue;
            const int n = t.f0 + 32 * j + lane;
            const float* w = p.W + ((size_t)t.group * p.N + n) * p.K;
            float s = 0.f;
#pragma unroll 4
            for (int k = 0; k < p.K; k += 4) {
                const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
                s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
            }
            store(p, m, n, s);
        }
    }
}

// NT: token rows of a tile at most; MD: sets of accumulators of main products, which the SUB stages take in turn, CD: of the corrections,
// which the segments take in turn; NS: stages of the ring of split operands, NR: of the ring of weights as they come.  SHARED: the
// CTAs of a cluster take a tile's segments in equal runs, and the first of them adds the segments' sums in order.
template <int NT, int MD, int CD, int NS, int NR, int G, bool SHARED>
__global__ void __launch_bounds__(THREADS, 1) gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, SplitParams p) {
    constexpr int C_COL = MD * NT, A_COL = C_COL + CD * 2 * NT;      // columns: [main sets][correction sets][stages of weights]
    constexpr int T_BYTES = 3 * NT * KS * 2;
    // G stages share their mbarriers.  A tile then has a whole number of them; stages behind K are zeros.
    constexpr int SLOTS = NS / G;
    static_assert(NS % G == 0, "whole slots");
    constexpr int RUNS = (NT / 16 + 1) / 2;                          // runs of 16 tokens that a warp reads out
    static_assert(2 * NT <= 256 && A_COL + NS * A_COLS <= 512, "tensor memory");
    static_assert(SUB % G == 0, "whole slots");
    // A group waits for every second stage.  A wait tells a phase from its neighbours only, so each group must have waited for the use of
    // the slot before this one, which an even ring gives.
    static_assert(NR % 2 == 0 && (G > 1 || NS % 2 == 0), "each slot belongs to one group, or to both");
    static_assert(NS <= NR, "the first stages are split before the weights' ring waits for its readers");
    static_assert(!SHARED || NT == 16, "a shared tile is one run of 16 tokens");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw = smem + NS * T_BYTES;
    // SHARED, first CTA: [segment][16 rows][128 features].  More than a run of tokens a warp: the running sums, [NT rows][128 features]
    float* parts = reinterpret_cast<float*>(raw + NR * RAW_BYTES);
    __shared__ __align__(8) unsigned long long full[SLOTS], empty[SLOTS], raw_full[NR], raw_empty[NR], main_full[MD], main_empty[MD], corr_empty[CD], drained;
    __shared__ unsigned tmem_slot;
    __shared__ __align__(16) Group groups[MAX_GROUPS];
    __shared__ int group_count;
    __shared__ volatile int abort_flag, odd_flag;                    // odd_flag: some element is not finite
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < SLOTS; i++) mbar_init(&full[i], G * (W_WARPS / 2 + T_WARPS)), mbar_init(&empty[i], 1);
        for (int i = 0; i < NR; i++) mbar_init(&raw_full[i], 1), mbar_init(&raw_empty[i], W_WARPS / 2);
        for (int i = 0; i < MD; i++) mbar_init(&main_full[i], 1), mbar_init(&main_empty[i], E_WARPS);
        for (int i = 0; i < CD; i++) mbar_init(&corr_empty[i], E_WARPS);
        mbar_init(&drained, 1);
        abort_flag = 0, odd_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == W_WARPS + E_WARPS + T_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    if (warp == 0) {
        if (p.group_offsets) pdl_wait();
        list_groups<NT>(p, groups, &group_count);
    }
    tc_fence_before();
    __syncthreads();
    const int n_groups = group_count;
    if (SHARED) cluster_sync();                                      // the first CTA runs before anything is written to its memory
    tc_fence_after();
    const unsigned tmem = tmem_slot;
    const int all_stages = (p.K + G * KS - 1) / (G * KS) * G, segments = (all_stages + p.seg_stages - 1) / p.seg_stages;
    const int rank = SHARED ? (int)(blockIdx.x % p.share) : 0;
    const int seg0 = SHARED ? rank * segments / p.share : 0, seg1 = SHARED ? (rank + 1) * segments / p.share : segments;
    const int stage0 = seg0 * p.seg_stages, stages = min(all_stages, seg1 * p.seg_stages) - stage0;      // of this CTA, of every tile
    bool ok = true;
    // for all lanes of a warp alike
    auto warp_wait = [&](void* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait_limited(bar, parity, p.polls) && !abort_flag) != 0; };

    if (warp < W_WARPS) {
        // weights into pieces.  A lane holds 4 k of rows 8 i + lane / 4 (i = 0..3) of two of the stage's four MMA steps at a time.
        const int quad = warp & 3, half = warp >> 2;                 // TMEM lanes 32 quad .. + 31; the group
        const unsigned lanes = tmem + ((unsigned)(quad * 32) << 16);
        const int from = (quad * 32 + (lane >> 2)) * 64 + (lane & 3) * 16;    // byte of the stage: eight lanes read 128 bytes in a row
        if (p.group_offsets) pdl_wait();
        Walk<NT> walk(p, groups, n_groups);
        Tile t;
        int end = 0;                                                 // stages of the tiles seen so far
        for (int it = half;; it += 2) {
            bool more = it < end;
            while (!more && walk.next(t)) more = it < (end += stages);
            if (!more) break;
            const int s = it % NS, use = it / G / SLOTS, slot = it / G % SLOTS, r = it % NR;
            if (it >= NS && it < NS + 2) pdl_wait();                 // once a group: from here on its waits hang on the MMAs
            ok = warp_wait(&raw_full[r], (it / NR) & 1);
            if (!ok) break;
            const unsigned char* stage = raw + r * RAW_BYTES + from;
            const unsigned at = lanes + A_COL + s * A_COLS;
#pragma unroll
            for (int two = 0; two < 2; two++) {
                float4 v[2][4];
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) v[j][i] = *reinterpret_cast<const float4*>(stage + (2 * two + j) * (BF * 64) + i * 512);
                if (two == 0) {
                    if (use > 0) ok = warp_wait(&empty[slot], (use - 1) & 1);     // its last contents have been multiplied
                    tc_fence_after();
                }
                if (!ok) break;
#pragma unroll
                for (int piece = 0; piece < 3; piece++) {
                    unsigned q[2][4][2];
#pragma unroll
                    for (int j = 0; j < 2; j++)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            q[j][i][0] = take2(v[j][i].x, v[j][i].y);
                            q[j][i][1] = take2(v[j][i].z, v[j][i].w);
                        }
                    const unsigned to = at + piece * (KS / 2) + two * 16;
                    tc_st_16x256(to, q[0][0], q[0][1], q[1][0], q[1][1]);
                    tc_st_16x256(to + (16u << 16), q[0][2], q[0][3], q[1][2], q[1][3]);
                }
            }
            if (!ok) break;
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[slot]);
                mbar_arrive(&raw_empty[r]);
            }
        }
    } else if (warp < W_WARPS + E_WARPS) {
        // the accumulators: a warp has a quarter of the lanes and every second run of 16 tokens
        const int quad = warp & 3, half = (warp - W_WARPS) >> 2;
        const unsigned lanes = tmem + ((unsigned)(quad * 32) << 16);
        pdl_wait();
        Walk<NT> walk(p, groups, n_groups);
        Tile o;
        int subs = 0, count = 0;                                     // SUB stages and segments read out so far
        float* mine = parts + quad * 32 + lane;
        const bool wide = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;      // a row's features start on 16 bytes
        while (ok && walk.next(o)) {
            float sum[RUNS][16], total[RUNS][16];
            for (int seg = seg0; seg < seg1; seg++, count++) {
                const int n_subs = (min(p.seg_stages, all_stages - seg * p.seg_stages) + SUB - 1) / SUB;
                for (int u = 0; u < n_subs; u++, subs++) {
                    ok = warp_wait(&main_full[subs % MD], (subs / MD) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    if (u == n_subs - 1) {                           // the corrections of the segment, before its last main sum
                        const unsigned at = lanes + C_COL + count % CD * 2 * NT;
#pragma unroll
                        for (int r = 0; r < RUNS; r++) {
                            const int c = (2 * r + half) * 16;
                            if (c >= o.n_tok) continue;              // the same for a whole warp
                            float c1[16], c2[16];
                            tc_ld16x2(at + c, c1, at + o.n_tok + c, c2);
#pragma unroll
                            for (int i = 0; i < 16; i++) sum[r][i] = u == 0 ? c1[i] + c2[i] : sum[r][i] + (c1[i] + c2[i]);
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&corr_empty[count % CD]);
                    }
                    const unsigned at = lanes + subs % MD * NT + half * 16;
                    float v[RUNS][16];
                    if (RUNS == 2) tc_ld16x2(at, v[0], at + 32, v[RUNS - 1]);    // (columns behind n_tok are read and not used)
                    else tc_ld16(at, v[0]);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&main_empty[subs % MD]);
#pragma unroll
                    for (int r = 0; r < RUNS; r++)
#pragma unroll
                        for (int i = 0; i < 16; i++) sum[r][i] = u == 0 && n_subs > 1 ? v[r][i] : sum[r][i] + v[r][i];
                }
                if (!ok) break;
#pragma unroll
                for (int r = 0; r < RUNS; r++) {
                    const int c = (2 * r + half) * 16;
                    if (c >= o.n_tok) continue;
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        if (SHARED) st_cluster(mine + (seg * 16 + i) * BF, 0, sum[r][i]);
                        else if (RUNS > 1) mine[(c + i) * BF] = seg == 0 ? sum[r][i] : mine[(c + i) * BF] + sum[r][i];
                        else total[r][i] = seg == 0 ? sum[r][i] : total[r][i] + sum[r][i];
                    }
                }
            }
            const int n = o.f0 + quad * 32 + lane;
            if (SHARED || !ok || n >= p.N) continue;
            const float b = p.bias ? p.bias[n] : 0.f;
            bool odd = false;
#pragma unroll
            for (int r = 0; r < RUNS; r++) {
                const int c = (2 * r + half) * 16, m = o.m0 + c;
                float* to = p.C + (size_t)m * p.ldc + n;
                auto put = [&](int i, float v) {
                    odd |= !finite(v);
                    if (p.bias) v += b;
                    if (p.row_scale) v *= p.row_scale[m + i];
                    *to = v;
                    to += p.ldc;
                };
                if (RUNS > 1) {
                    const int count = min(16, o.rows - c);
                    if (wide && o.f0 + BF <= p.N) {
                        // four rows at a time, eight lanes to the 32 features of one
                        __syncwarp();
                        const float* from = parts + c * BF + quad * 32 + (lane & 7) * 4;
                        const int n4 = o.f0 + quad * 32 + (lane & 7) * 4;
                        float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (p.bias) b4 = make_float4(p.bias[n4], p.bias[n4 + 1], p.bias[n4 + 2], p.bias[n4 + 3]);
#pragma unroll
                        for (int i0 = 0; i0 < 16; i0 += 4) {
                            const int i = i0 + (lane >> 3);
                            if (i >= count) continue;
                            float4 v = *reinterpret_cast<const float4*>(from + i * BF);
                            odd |= !finite(v.x) || !finite(v.y) || !finite(v.z) || !finite(v.w);
                            if (p.bias) v.x += b4.x, v.y += b4.y, v.z += b4.z, v.w += b4.w;
                            if (p.row_scale) {
                                const float f = p.row_scale[m + i];
                                v.x *= f, v.y *= f, v.z *= f, v.w *= f;
                            }
                            *reinterpret_cast<float4*>(p.C + (size_t)(m + i) * p.ldc + n4) = v;
                        }
                        __syncwarp();
                    } else {
#pragma unroll 4
                        for (int i = 0; i < count; i++) put(i, mine[(c + i) * BF]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c + i < o.rows) put(i, total[r][i]);
                }
            }
            if (odd) odd_flag = 1;
        }
    } else if (warp < W_WARPS + E_WARPS + T_WARPS) {
        // token rows: eight threads to a row, each with eight k of it
        const int tid = threadIdx.x - (W_WARPS + E_WARPS) * 32;
        const int r0 = tid >> 3, part = tid & 7;
        constexpr int PASSES = (NT + T_ROWS - 1) / T_ROWS;
        pdl_wait();
        Walk<NT> walk(p, groups, n_groups);
        Tile t;
        float4 next[PASSES][2];
        const float* src[PASSES];
        int n_tok = 0, n_next = 0, kb = stage0;
        bool have = walk.next(t);
        auto point = [&]() {
#pragma unroll
            for (int j = 0; j < PASSES; j++) {
                const int r = r0 + T_ROWS * j;
                src[j] = nullptr;
                if (have && r < t.rows) src[j] = a_row(p, t.m0 + r) + part * 8;
            }
            n_next = have ? t.n_tok : 0;
        };
        point();
        auto load = [&]() {
            const int k = kb * KS + part * 8;
#pragma unroll
            for (int j = 0; j < PASSES; j++) {
                next[j][0] = next[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (src[j] && k < p.K) next[j][0] = *reinterpret_cast<const float4*>(src[j] + kb * KS);
                if (src[j] && k + 4 < p.K) next[j][1] = *reinterpret_cast<const float4*>(src[j] + kb * KS + 4);
            }
            n_tok = n_next;
            if (have && ++kb == stage0 + stages) {
                kb = stage0;
                have = walk.next(t);
                point();
            }
        };
        load();
        for (int it = 0; n_tok > 0; it++) {
            const int s = it % NS, use = it / G / SLOTS, slot = it / G % SLOTS;
            if (it % G == 0 && use > 0) ok = warp_wait(&empty[slot], (use - 1) & 1);
            if (!ok) break;
            const int n = n_tok;
            unsigned char* base = smem + s * T_BYTES;
#pragma unroll
            for (int j = 0; j < PASSES; j++) {
                const int r = r0 + T_ROWS * j;
                if (r >= n) break;
                uint4 q1, q2, q3;
                auto take8 = [&](uint4& q) {
                    q.x = take2(next[j][0].x, next[j][0].y), q.y = take2(next[j][0].z, next[j][0].w);
                    q.z = take2(next[j][1].x, next[j][1].y), q.w = take2(next[j][1].z, next[j][1].w);
                };
                take8(q1), take8(q2), take8(q3);
                unsigned char* at = base + r * 128 + ((part ^ (r & 7)) << 4);
                *reinterpret_cast<uint4*>(at) = q1;
                *reinterpret_cast<uint4*>(at + n * 128) = q2;
                *reinterpret_cast<uint4*>(at + 2 * n * 128) = q3;
            }
            load();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[slot]);
        }
    } else if (warp == W_WARPS + E_WARPS + T_WARPS) {
        // weights as they come: four boxes of 128 rows x 16 k a stage, a lane each
        if (p.group_offsets) pdl_wait();                             // whose weights are read follows from the offsets; of a dense product they are never written
        Walk<NT> walk(p, groups, n_groups);
        Tile t;
        int it = 0;
        while (ok && walk.next(t)) {
            for (int st = 0; st < stages && ok; st++, it++) {
                const int r = it % NR, k = (stage0 + st) * KS + lane * 16;
                if (it == NR) pdl_wait();                            // its reader may be waiting for MMAs, these for the token rows
                if (it >= NR) ok = warp_wait(&raw_empty[r], (it / NR - 1) & 1);
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(&raw_full[r], RAW_BYTES);
                __syncwarp();
                if (lane < 4) tma_load_3d(raw + r * RAW_BYTES + lane * (BF * 64), &map_w, k, t.f0, t.group, &raw_full[r]);
            }
        }
        // its copies land before the shared memory is given up, whoever has stopped reading them
        for (int i = it > NR ? it - NR : 0; i < it; i++) mbar_wait(&raw_full[i % NR], (i / NR) & 1);
        pdl_wait();
    } else {
        // The MMAs.  The whole warp walks along, so that what an MMA is given is the same in all lanes and known to be; one lane issues.
        pdl_wait();
        if (lane == 0) pdl_trigger();                                // behind the wait: a dependent kernel may count on all before this one
        Walk<NT> walk(p, groups, n_groups);
        Tile t;
        const unsigned cols = __shfl_sync(0xffffffffu, tmem, 0);
        const unsigned long long desc0 = smem_desc(smem);
        const unsigned desc_hi = (unsigned)(desc0 >> 32), desc_lo = __shfl_sync(0xffffffffu, (unsigned)desc0, 0);
        int it = 0, subs = 0, count = 0;                             // subs, count: of the SUB stages and segments begun
        while (ok && walk.next(t)) {
            const int n = __shfl_sync(0xffffffffu, t.n_tok, 0);
            const unsigned d_two = split_idesc(2 * n), d_one = split_idesc(n), off = n * (KS * 2 >> 4);
            int in_seg = 0;
            for (int st = 0; st < stages; st += G, it += G) {
                const int use = it / G / SLOTS, slot = it / G % SLOTS;
                const bool new_sub = st % SUB == 0, new_seg = in_seg == 0;
                if (new_sub && subs >= MD) ok = warp_wait(&main_empty[subs % MD], (subs / MD - 1) & 1);
                if (ok) ok = warp_wait(&full[slot], use & 1);
                if (!ok) break;
                tc_fence_after();
                const unsigned main = cols + (subs - !new_sub) % MD * NT, corr = cols + C_COL + (count - !new_seg) % CD * 2 * NT;
                const unsigned a0 = cols + A_COL + slot * G * A_COLS, b0 = desc_lo + ((slot * G * T_BYTES) >> 4);
                subs += new_sub;
                const bool wait_corr = new_seg && count >= CD;
                count += new_seg;
                in_seg = in_seg + G == p.seg_stages ? 0 : in_seg + G;
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < G * KS / 16; i++) {
                        const int g = i / (KS / 16), j = i % (KS / 16);
                        tc_mma_ta_lo(main, a0 + g * A_COLS + 8 * j, b0 + ((g * T_BYTES) >> 4) + 2 * j, desc_hi, d_one, i == 0 && new_sub ? 0u : 1u);      // w1 a1
                    }
                }
                if (wait_corr) {
                    ok = warp_wait(&corr_empty[(count - 1) % CD], ((count - 1) / CD - 1) & 1);
                    if (!ok) break;
                    tc_fence_after();
                }
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < G * KS / 16; i++) {
                        const int g = i / (KS / 16), j = i % (KS / 16);
                        const unsigned a = a0 + g * A_COLS + 8 * j, b = b0 + ((g * T_BYTES) >> 4) + 2 * j;
                        tc_mma_ta_lo(corr, a, b + off, desc_hi, d_two, i == 0 && new_seg ? 0u : 1u);      // w1 a2 | w1 a3
                        tc_mma_ta_lo(corr, a + KS / 2, b, desc_hi, d_two, 1u);                            // w2 a1 | w2 a2
                        tc_mma_ta_lo(corr, a + KS, b, desc_hi, d_two, 1u);                                // w3 a1 | w3 a2
                    }
                    tc_commit(&empty[slot]);
                    if ((st + G) % SUB == 0 || st + G >= stages) tc_commit(&main_full[(subs - 1) % MD]);
                }
            }
        }
        if (elect_one()) tc_commit(&drained);                        // the MMAs end before their memory is given up
        mbar_wait(&drained, 0);
    }
    if (!ok && lane == 0) {
        atomicOr(p.status, ESP_STATUS_WAIT_EXPIRED);
        abort_flag = 1;
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (SHARED) {
        // the segments' sums are with the first CTA, which adds them in order
        cluster_sync();
        if (rank == 0 && !abort_flag) {
            Walk<NT> walk(p, groups, n_groups);
            Tile o;
            const bool have = walk.next(o);
            for (int i = threadIdx.x; have && i < o.rows * BF; i += THREADS) {
                const int n = o.f0 + i % BF;
                if (n >= p.N) continue;
                float v = parts[i];
                for (int seg = 1; seg < segments; seg++) v += parts[seg * 16 * BF + i];
                if (!finite(v)) odd_flag = 1;
                store(p, o.m0 + i / BF, n, v);
            }
        }
        __syncthreads();
    }
    if (odd_flag && rank == 0 && !abort_flag) {
        Walk<NT> walk(p, groups, n_groups);
        Tile o;
        while (walk.next(o)) chains(p, o);
    }
    if (warp == W_WARPS + E_WARPS + T_WARPS + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// W as [groups][N][K] float, boxes of 128 rows x 16 k, zeros out of bounds
int map_weights(CUtensorMap* map, const SplitParams& p) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess)
            return (int)cudaErrorNotSupported;
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    const cuuint64_t dims[3] = {(cuuint64_t)p.K, (cuuint64_t)p.N, (cuuint64_t)p.groups};
    const cuuint64_t strides[2] = {(cuuint64_t)p.K * 4, (cuuint64_t)p.K * p.N * 4};
    const cuuint32_t box[3] = {16, BF, 1}, elem[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p.W), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

// runs of at most ``nt`` rows; of groups an upper bound
long long row_runs(const SplitParams& p, int nt) {
    return p.group_offsets ? p.M / nt + (p.groups < p.M ? p.groups : p.M) : (p.M + nt - 1) / nt;
}

template <int NT, int MD, int CD, int NS, int NR, int G, bool SHARED>
int launch(SplitParams p, int sms, cudaStream_t stream) {
    constexpr int SMEM = NS * 3 * NT * KS * 2 + NR * RAW_BYTES + (SHARED ? MAX_PARTS * 16 * BF * 4 : NT > 32 ? NT * BF * 4 : 0) + 1024;
    static_assert(SMEM + 4096 + 512 <= 227 * 1024, "shared memory");
    CUtensorMap map;
    const int rc = map_weights(&map, p);
    if (rc) return rc;
    const auto kernel = gemm_split_kernel<NT, MD, CD, NS, NR, G, SHARED>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    const long long tiles = row_runs(p, NT) * ((p.N + BF - 1) / BF);
    if (tiles + sms > 0x3fffffffll) return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(SHARED ? tiles * p.share : tiles < sms ? tiles : sms));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = esp_pdl_enabled(ESP_PDL_DENSE) ? 1 : 0;
    if (SHARED) {
        cudaLaunchAttribute& cluster = attr[cfg.numAttrs++];
        cluster.id = cudaLaunchAttributeClusterDimension;
        cluster.val.clusterDim.x = p.share, cluster.val.clusterDim.y = 1, cluster.val.clusterDim.z = 1;
    }
    cudaLaunchKernelEx(&cfg, kernel, map, p);
    return esp_launch_status();
}
}  // namespace

// All float.  K, lda multiples of 4, A and W on 16 bytes, at most 256 groups.
ESP_API int esp_gemm_split(const void* A, const int* a_rows, const void* W, const float* bias, const float* row_scale, void* C,
                           const int* group_offsets, int groups, int M, int N, int K, long long lda, long long ldc, int polls, int* status,
                           cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 != 0 || lda % 4 != 0 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15) || groups < 1 || groups > MAX_GROUPS || polls < 0)
        return (int)cudaErrorInvalidValue;
    SplitParams p{(const float*)A, a_rows, (const float*)W, bias, row_scale, (float*)C, group_offsets, groups, M, N, K, lda, ldc,
                  segment_of(K) / KS, 1, (unsigned)polls, status};
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return (int)e;
    {
        // Few tiles of 16 rows: as many CTAs to each as there are SMs for (6 rows, K = 2,048: N = 2,048 24.5 us with a CTA a tile, 9.6 with
        // four; N = 6,144 24.8 and 17.5 with two.  64 rows: N = 2,048 18.5 us, tiles of 64 rows 35.8).  Clusters of eight did not all find room at once
        const long long tiles = row_runs(p, 16) * ((N + BF - 1) / BF);
        const int segments = ((K + KS - 1) / KS + p.seg_stages - 1) / p.seg_stages;
        const long long most = segments > MAX_PARTS ? 1 : min(min(6ll, (long long)segments), sms / tiles);
        if (most > 1) {
            const int each = (segments + (int)most - 1) / (int)most;     // segments of a CTA at most
            p.share = (segments + each - 1) / each;
        }
        if (p.share > 1) return launch<16, 2, 2, 4, 4, 1, true>(p, sms, stream);
    }
    // Few rows, of a group four on average: a short tile leaves tensor memory for two sets of accumulators.  A wait and a commit keep
    // the issuing warp some 300 and 90 cycles, a third of its time where the MMAs are short: groups, and a tile a CTA, have two stages
    // behind one of each (200 rows over 60 groups, N = 2,816, K = 2,048 255 -> 243 us, 16 rows, N = 2,048, K = 1,408 44.8 -> 40.9; one row,
    // N = 11,264 27.2 -> 25.6).  Many tiles a CTA of one matrix, which memory bounds, are better off with the finer ring (6 rows, N = 151,936:
    // 234 us against 242).
    if (M <= (group_offsets ? 4ll * groups : 16ll)) {
        if (group_offsets || (N + BF - 1) / BF <= sms) return launch<16, 2, 2, 4, 6, 2, false>(p, sms, stream);
        return launch<16, 2, 2, 4, 6, 1, false>(p, sms, stream);
    }
    return launch<64, 2, 1, 2, 4, 1, false>(p, sms, stream);
}
