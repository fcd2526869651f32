// Choosing the next token of each row of a logits matrix on the device.
//
// temperature == 0: the arg-max, lower id on ties.
// temperature  > 0: weights w_i = exp((l_i - max) / T) in 32-bit; the ids are
// ranked by descending weight, ties by ascending id; an optional nucleus cut
// keeps the shortest prefix of that ranking whose mass reaches top_p * total;
// one uniform draw u in [0, 1) from the row's splitmix64 stream picks the first
// id whose cumulative mass reaches u * (kept mass).  Exactly one draw per token.
//
// The ranking is never materialised: the crossing point is found by a radix
// selection over the weights' bits, summing the mass of every bucket.  Masses
// are 40-bit fixed point integers, so the sums are exact and do not depend on
// the order in which threads add them.
//
// What bounds it: a row is read once (0.6 MB at 151,936 ids); all else is latency.  So a row is spread over a cluster
// of eight blocks, each keeps its weights in shared memory for the later passes, and a search is three levels of the
// 29 bits that a weight of at least 2^-40 can have (11, 9 and 9: lighter ones have no mass and are skipped), one
// histogram over the cluster's shared memory per level.  Both searches, for the nucleus and for the draw, start from the
// same first level, and end at once where the first rank reaches the threshold alone.  Ids enter only where several
// weights are equal in all bits.  Eight rows of 151,936 ids, top_p 0.95: 65 us for normal logits, 16 us with one likely
// token, 7 us greedy; a block per row with eight passes over 64-bit keys and 64-bit atomics took 5,280, 795 and 10 us.
// 64 rows: 195, 43 and 12.5 us against 5,293, 802 and 10.5 us (and a launch of 6 us, the finite check, is part of it).
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {
constexpr int PICK_THREADS = 1024;
constexpr int PICK_WARPS = PICK_THREADS / 32;
constexpr int PICK_CLUSTER = 8;
constexpr float FIXED_ONE = 1099511627776.0f;   // 2^40
constexpr unsigned ONE_BITS = 0x3F800000u;
constexpr unsigned long long FIRST_MASS = 1ull << 40;      // of the first rank, whose weight is exp(0)
constexpr int L1_BINS = 2048, LX_BINS = 512;    // a first-level bin is 2^18 steps of the weight's bits: 1,281 are used
// Weights that a block keeps in shared memory: 96 KB beside its 28 KB of bins.  Two blocks fit an SM up to about 21,900 of them
// (175,000 ids), one from there on, which still draws faster than two that read the row anew in every pass (38 rows of 190,000
// ids, three settings: 117 to 176 us against 128 to 205; greedy rows, 64 of them, lose by it: 34 against 23).
constexpr int KEPT_MAX = 24576;

typedef unsigned long long u64;

__device__ __forceinline__ u64 splitmix_next(u64* state) {
    *state += 0x9E3779B97F4A7C15ull;
    u64 z = *state;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// mass of a weight in [0, 1]; 0 for anything else (rows with a NaN are refused by the finite check)
__device__ __forceinline__ u64 mass_of(float w) { return w > 0.f && w <= 1.f ? __float2ull_rd(w * FIXED_ONE) : 0ull; }

__device__ __forceinline__ void better(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

// What one block of the cluster holds.  A mass is kept in three words of 14 (the last: 13) bits and more, so that a bin
// is added up with 32-bit atomics: a block has fewer than 2^18 ids (else ``wide``: 64-bit atomics on the first two words).
template <int CS>
struct PickShared {
    union {
        unsigned hist[3][L1_BINS];
        u64 hist64[L1_BINS];
    };
    u64 cum1[L1_BINS / CS], cumx[LX_BINS / CS];      // this block's share of a level's bins: masses up to and with each
    u64 total1[CS], totalx[CS];                      // mass of every block's share
    u64 found_before[2];
    int found_bin[2];
    float best_v[CS];
    int best_i[CS];
    int heaviest, first[CS];                         // lowest id of weight 1: this block's, every block's
    u64 warp_u64[PICK_WARPS];
    float warp_v[PICK_WARPS];
    int warp_i[PICK_WARPS];
};

template <int CS>
struct Picker {
    PickShared<CS>& s;
    int rank, n;                 // this block's place in the cluster, its number of ids
    bool wide;                   // the same in every block: they read one another's bins
    int finds = 0;

    __device__ __forceinline__ PickShared<CS>* of(int r) const {
        if constexpr (CS == 1) return &s;
        else return cg::this_cluster().map_shared_rank(&s, r);
    }
    __device__ __forceinline__ void sync() const {
        if constexpr (CS == 1) __syncthreads();
        else cg::this_cluster().sync();
    }
    __device__ void clear(int bins) {
        for (int b = threadIdx.x; b < bins; b += PICK_THREADS) {
            if (wide) s.hist64[b] = 0;
            else s.hist[0][b] = s.hist[1][b] = s.hist[2][b] = 0;
        }
        __syncthreads();
    }
    // All lanes of a warp call this together; ``mass`` 0: nothing to add.  Lanes that mean the same bin add up first: a
    // warp with one bin (many equal weights) then costs one addition and not 32 in a row.
    __device__ __forceinline__ void add(unsigned bin, u64 mass) {
        const unsigned active = __ballot_sync(0xffffffffu, mass != 0);
        if (!active) return;
        unsigned w0 = (unsigned)(mass & 0x3fff), w1 = (unsigned)((mass >> 14) & 0x3fff), w2 = (unsigned)(mass >> 28);
        const int lead = __ffs(active) - 1;
        const unsigned first = __shfl_sync(0xffffffffu, bin, lead);
        bool mine = mass != 0;
        if (__all_sync(0xffffffffu, mass == 0 || bin == first)) {
            w0 = __reduce_add_sync(0xffffffffu, w0);
            w1 = __reduce_add_sync(0xffffffffu, w1);
            w2 = __reduce_add_sync(0xffffffffu, w2);
            mine = (threadIdx.x & 31) == lead;
        }
        if (!mine) return;
        if (wide) {
            atomicAdd(&s.hist64[bin], (u64)w0 + ((u64)w1 << 14) + ((u64)w2 << 28));
        } else {
            atomicAdd(&s.hist[0][bin], w0);
            atomicAdd(&s.hist[1][bin], w1);
            atomicAdd(&s.hist[2][bin], w2);
        }
    }
    __device__ __forceinline__ u64 bin_mass(const PickShared<CS>* p, int b) const {
        return wide ? p->hist64[b] : (u64)p->hist[0][b] + ((u64)p->hist[1][b] << 14) + ((u64)p->hist[2][b] << 28);
    }
    // After every block has filled its histogram: the running masses of this block's share of the bins, and the total of
    // every share, in every block.
    template <int BINS>
    __device__ void merge(u64* cum, bool first_level) {
        constexpr int SHARE = BINS / CS, PER = (SHARE + PICK_THREADS - 1) / PICK_THREADS;
        sync();
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        u64 m[PER], run = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            const int b = tid * PER + j;
            m[j] = 0;
            if (b < SHARE) {
#pragma unroll
                for (int c = 0; c < CS; c++) m[j] += bin_mass(of(c), rank * SHARE + b);
            }
            run += m[j];
        }
        u64 incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) s.warp_u64[warp] = incl;
        __syncthreads();
        u64 ahead = 0;
        for (int w = 0; w < warp; w++) ahead += s.warp_u64[w];
        u64 at = ahead + incl - run;
#pragma unroll
        for (int j = 0; j < PER; j++) {
            at += m[j];
            if (tid * PER + j < SHARE) cum[tid * PER + j] = at;
        }
        if (tid == PICK_THREADS - 1) {
#pragma unroll
            for (int c = 0; c < CS; c++) {
                (first_level ? of(c)->total1 : of(c)->totalx)[rank] = at;
                if (first_level) of(c)->first[rank] = s.heaviest;
            }
        }
        sync();
    }
    // The first bin with mass whose cumulative mass, ``base`` ahead of the level, reaches ``threshold``; ``before``: the
    // mass ahead of that bin.  The threshold is at most base + the level's mass.
    template <int BINS>
    __device__ int find(const u64* cum, const u64* totals, u64 base, u64 threshold, u64& before) {
        constexpr int SHARE = BINS / CS;
        const int buf = finds++ & 1;            // two results in turn: a block may still read the one before
        u64 run = base;
        int owner = -1;
        for (int c = 0; c < CS; c++) {
            if (totals[c] > 0 && run + totals[c] >= threshold) { owner = c; break; }
            run += totals[c];
        }
        if (owner == rank) {
            for (int b = threadIdx.x; b < SHARE; b += PICK_THREADS) {
                const u64 prev = b ? cum[b - 1] : 0;
                if (cum[b] > prev && run + cum[b] >= threshold && (prev == 0 || run + prev < threshold)) {
                    for (int c = 0; c < CS; c++) {
                        of(c)->found_bin[buf] = rank * SHARE + b;
                        of(c)->found_before[buf] = run + prev;
                    }
                }
            }
        }
        sync();
        if (owner < 0) { before = base; return 0; }
        before = s.found_before[buf];
        return s.found_bin[buf];
    }
};

template <int CS>
__global__ void __launch_bounds__(PICK_THREADS, 2)
pick_tokens_kernel(const float* __restrict__ logits, int vocab, int per_block, int keep, int vec,
                   const float* __restrict__ temperature, const float* __restrict__ top_p, u64* __restrict__ rng_state,
                   const int* __restrict__ row_slot, int* __restrict__ tokens, int* __restrict__ status) {
    pdl_trigger();
    pdl_wait();
    logits = behind_wait(logits);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PickShared<CS>& s = *reinterpret_cast<PickShared<CS>*>(smem_raw);
    float* weights = reinterpret_cast<float*>(smem_raw + (sizeof(PickShared<CS>) + 15) / 16 * 16);     // [per_block] if keep
    const int r = blockIdx.x / CS, rank = blockIdx.x % CS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = min(vocab, rank * per_block), n = min(vocab, i0 + per_block) - i0;
    const float* row = logits + (size_t)r * vocab + i0;
    const float temp = temperature ? temperature[r] : 0.f;
    Picker<CS> pick{s, rank, n, per_block >= (1 << 18)};

    // arg-max with the lower id on ties (also gives the maximum for the weights), and whether all values are finite
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    bool bad = false;
    auto look = [&](int i, float v) {
        bad |= (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u;
        if (v > bv) { bv = v; bi = i0 + i; }
    };
    if (vec) {
        for (int i = tid * 4; i < n; i += PICK_THREADS * 4) {          // n and i0 are multiples of 4
            const float4 v = *reinterpret_cast<const float4*>(row + i);
            look(i, v.x), look(i + 1, v.y), look(i + 2, v.z), look(i + 3, v.w);
            if (keep) *reinterpret_cast<float4*>(weights + i) = v;
        }
    } else {
        for (int i = tid; i < n; i += PICK_THREADS) {
            const float v = row[i];
            look(i, v);
            if (keep) weights[i] = v;
        }
    }
    if (status && __any_sync(0xffffffffu, bad) && lane == 0) atomicOr(status, ESP_STATUS_LOGITS_NONFINITE);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        better(bv, bi, __shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
    if (lane == 0) { s.warp_v[warp] = bv; s.warp_i[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        bv = s.warp_v[lane];
        bi = s.warp_i[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            better(bv, bi, __shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
    }
    // the stream's state is read by every block before the cluster's first barrier and written by one behind it
    u64 state = 0;
    if (temp > 0.f) state = rng_state[row_slot[r]];
    if constexpr (CS > 1) {
        // no block may write into another's shared memory before that one has started
        pick.sync();
        if (tid == 0)
            for (int c = 0; c < CS; c++) { pick.of(c)->best_v[rank] = bv; pick.of(c)->best_i[rank] = bi; }
    } else if (tid == 0) {
        s.best_v[0] = bv;
        s.best_i[0] = bi;
    }
    pick.sync();
    bv = s.best_v[0];
    bi = s.best_i[0];
#pragma unroll
    for (int c = 1; c < CS; c++) better(bv, bi, s.best_v[c], s.best_i[c]);
    if (bi == 0x7fffffff) bi = 0;
    const float mx = bv;
    if (!(temp > 0.f)) {
        if (rank == 0 && tid == 0) tokens[r] = bi;
        return;
    }
    const u64 z = splitmix_next(&state);
    if (rank == 0 && tid == 0) rng_state[row_slot[r]] = state;
    const float inv_t = 1.0f / temp;

    // first level, shared by both searches; the weights take the logits' place in shared memory.  The first rank is the
    // lowest id whose weight is 1: logits that differ can have that weight alike, so it need not be the arg-max.
    int heaviest = 0x7fffffff;
    if (tid == 0) s.heaviest = heaviest;
    pick.clear(L1_BINS);
    for (int at = 0; at < n; at += PICK_THREADS) {
        const int i = at + tid;
        float w = 0.f;
        if (i < n) {
            w = expf(((keep ? weights[i] : row[i]) - mx) * inv_t);
            if (keep) weights[i] = w;
        }
        const u64 m = mass_of(w);
        if (w == 1.f) heaviest = min(heaviest, i0 + i);
        pick.add((ONE_BITS - __float_as_uint(w)) >> 18 & (L1_BINS - 1), m);
    }
    if (heaviest != 0x7fffffff) atomicMin(&s.heaviest, heaviest);
    pick.template merge<L1_BINS>(s.cum1, true);
    u64 kept = 0;
    int first = 0x7fffffff;
#pragma unroll
    for (int c = 0; c < CS; c++) kept += s.total1[c], first = min(first, s.first[c]);
    if (kept < FIRST_MASS) {                 // no weight is a number (a temperature whose inverse overflows): the arg-max
        if (rank == 0 && tid == 0) tokens[r] = bi;
        return;
    }

    // the weight at which the cumulative mass reaches ``threshold``, as steps of its bits below 1; the mass ahead of it
    auto crossing = [&](u64 threshold, u64& before) {
        unsigned d = (unsigned)pick.template find<L1_BINS>(s.cum1, s.total1, 0, threshold, before);
#pragma unroll 1
        for (int shift = 9; shift >= 0; shift -= 9) {
            pick.clear(LX_BINS);
            for (int at = 0; at < n; at += PICK_THREADS) {
                const int i = at + tid;
                float w = 0.f;
                if (i < n) w = keep ? weights[i] : expf((row[i] - mx) * inv_t);
                const unsigned key = ONE_BITS - __float_as_uint(w);
                const u64 m = w > 0.f && key >> (shift + 9) == d ? mass_of(w) : 0ull;
                pick.add(key >> shift & (LX_BINS - 1), m);
            }
            pick.template merge<LX_BINS>(s.cumx, false);
            const u64 ahead = before;
            d = d << 9 | (unsigned)pick.template find<LX_BINS>(s.cumx, s.totalx, ahead, threshold, before);
        }
        return d;
    };
    // of the equal weights at the crossing, how many it takes (at least one) to reach the threshold
    auto taken = [](u64 threshold, u64 before, u64 m) { return threshold > before ? (threshold - before + m - 1) / m : 1ull; };

    const float tp = top_p ? top_p[r] : -1.f;
    if (tp >= 0.f) {
        const float c = fminf(fmaxf(tp, 0.f), 1.f);
        const u64 target = (u64)((double)kept * (double)c);
        if (target <= FIRST_MASS) {
            kept = FIRST_MASS;               // the first rank alone reaches it: its weight is 1
        } else if (target <= kept) {         // beyond it (the product rounds up): everything is kept
            u64 before;
            const unsigned d = crossing(target, before);
            const u64 m = mass_of(__uint_as_float(ONE_BITS - d));
            if (m) kept = before + taken(target, before, m) * m;
        }
    }
    // the uniform is rounded to 32-bit before it is scaled
    const float u = (float)((double)(z >> 11) * (1.0 / 9007199254740992.0));
    u64 threshold = (u64)((double)u * (double)kept);
    if (threshold > kept) threshold = kept;
    if (threshold <= FIRST_MASS) {
        if (rank == 0 && tid == 0) tokens[r] = first;
        return;
    }
    u64 before;
    const unsigned d = crossing(threshold, before);
    const u64 m = mass_of(__uint_as_float(ONE_BITS - d));
    // the blocks hold ascending runs of ids, and their last histograms tell how many equal weights each has
    u64 place = m ? taken(threshold, before, m) : 1;
    bool mine = m != 0;
    for (int c = 0; c < CS && mine; c++) {
        const u64 has = pick.bin_mass(pick.of(c), d & (LX_BINS - 1)) / m;
        if (c == rank) { mine = place <= has; break; }
        if (place <= has) mine = false;
        place -= has;
    }
    pick.sync();                             // no block leaves while another reads its histogram
    if (!mine) {
        if (m == 0 && rank == 0 && tid == 0) tokens[r] = first;
        return;
    }
    for (int at = 0; at < n; at += PICK_THREADS) {
        const int i = at + tid;
        float w = 0.f;
        if (i < n) w = keep ? weights[i] : expf((row[i] - mx) * inv_t);
        const bool equal = w > 0.f && ONE_BITS - __float_as_uint(w) == d;
        const u64 here = (u64)__syncthreads_count(equal);
        if (place > here) { place -= here; continue; }
        const unsigned lanes = __ballot_sync(0xffffffffu, equal);
        if (lane == 0) s.warp_i[warp] = __popc(lanes);
        __syncthreads();
        int ahead = 0;
        for (int w2 = 0; w2 < warp; w2++) ahead += s.warp_i[w2];
        if (equal && ahead + __popc(lanes & ((1u << lane) - 1)) + 1 == (int)place) tokens[r] = i0 + i;
        break;
    }
}

template <int CS>
int launch_pick(const float* logits, int n_rows, int vocab, const float* temperature, const float* top_p, u64* rng_state,
                const int* row_slot, int* tokens, int* status, cudaStream_t stream) {
    const int per_block = ((vocab + CS - 1) / CS + 3) / 4 * 4;
    const int keep = per_block <= KEPT_MAX;
    const int vec = vocab % 4 == 0 && reinterpret_cast<uintptr_t>(logits) % 16 == 0;
    const size_t smem = (sizeof(PickShared<CS>) + 15) / 16 * 16 + (keep ? (size_t)per_block * sizeof(float) : 0);
    constexpr int MOST = (int)(sizeof(PickShared<CS>) + 15) / 16 * 16 + KEPT_MAX * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(pick_tokens_kernel<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_rows * CS);
    cfg.blockDim = dim3(PICK_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = esp_pdl_enabled(ESP_PDL_SMALL) ? 2 : 1;
    cudaLaunchKernelEx(&cfg, pick_tokens_kernel<CS>, logits, vocab, per_block, keep, vec, temperature, top_p, rng_state, row_slot,
                       tokens, status);
    return esp_launch_status();
}
}  // namespace

// status: null, or a status word that gets the bit of non-finite logits where a row has any.
ESP_API int esp_pick_tokens(const float* logits, int n_rows, int vocab, const float* temperature, const float* top_p,
                            u64* rng_state, const int* row_slot, int* tokens, int* status, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    // A block alone takes a vocabulary that its threads read in eight steps: no barrier of a cluster is worth it there
    // (eight rows drawn from 8,192 ids by a block each 26 us, from 8,196 by clusters 37 us), and up to what it keeps in shared
    // memory where there are more than 32 rows, whose clusters no longer start at once (16,384 ids, 38 rows: greedy 8.4 us against
    // 12.2, drawn 31 against 53; 64 rows 8.3 against 13.1, 31 against 68; 32 rows by clusters 9.9 and 39; 24,576 ids, eight rows:
    // a block 38, a cluster 29).
    if (vocab <= 8192 || (vocab <= KEPT_MAX && n_rows > 32))
        return launch_pick<1>(logits, n_rows, vocab, temperature, top_p, rng_state, row_slot, tokens, status, stream);
    return launch_pick<PICK_CLUSTER>(logits, n_rows, vocab, temperature, top_p, rng_state, row_slot, tokens, status, stream);
}
