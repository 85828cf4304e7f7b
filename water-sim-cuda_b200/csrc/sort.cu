// Morton keys and the stable radix sort of the reference's particle order.
//
// The reference builds int keys with setKeys (kernels.cu:361-371) and sorts
// (key, 0..n-1) pairs with thrust::sort_by_key (engine.cu:98-99), a stable
// ascending sort on signed keys.  This file restates that contract with a
// least-significant-digit radix sort written for this engine: 8-bit digits,
// up to four passes, each pass a per-CTA histogram, a per-digit scan of the
// CTA counts, and a scatter that ranks each 2048-key tile in shared memory
// with warp match/ballot and writes runs of equal digits contiguously.
//
// A digit that all keys share orders nothing, and the keys of a grid of 2^k
// cells per axis use 3 k bits: the first histogram also collects which bits
// differ, and the kernels of a pass whose digit does not vary return at once
// (a 128^3 grid's keys take three passes, a 32^3 grid's two).  The passes that
// run read and write two buffers in turn; the first generates the values
// (input position) instead of reading them, the last writes only the
// permutation (and, for the engine, the inverse permutation and the gather
// index of the reordered state).  The Morton keys are computed inside the
// first histogram, and every launch is chained to the one before it.
// Measured at 2M keys of a 128^3 grid: kernels 135 -> 88 us, the whole call 162
// -> 85 us back to back and 600 -> 108 us alone (the scratch pool, engine.cu).
// The scatter (20 us a pass) is bound by the chain of a tile: load, match,
// eight counter updates, block scan, write.
#include <algorithm>

#include "kernels.h"
#include "launch.cuh"

namespace mpm {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;                   // keys per thread per tile
constexpr int kTile = kThreads * kItems;    // 2048 keys
constexpr int kRadix = 256;
constexpr int kPasses = 4;
constexpr int kMaxCtas = 4 * 148;           // four CTAs per SM of a B200

__device__ __forceinline__ uint32_t digit_of(int32_t key, int shift) {
    // Flipping the sign bit orders signed keys as unsigned.
    return ((static_cast<uint32_t>(key) ^ 0x80000000u) >> shift) & 0xFFu;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Inclusive block scan over 256 threads; *total gets the block sum.
__device__ __forceinline__ uint32_t block_scan_incl(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < kWarps; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kWarps) s_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t prefix = warp > 0 ? s_warp[warp - 1] : 0u;
    *total = s_warp[kWarps - 1];
    __syncthreads();
    return x + prefix;
}

// Which passes run (bits 0..3 of *active, written by the first pass's spine)
// and where a pass reads and writes.
struct Pass {
    bool run, first, last;
    int src;  // the buffer it reads: 0 / 1, or -1 = the input keys
};
__device__ __forceinline__ Pass pass_of(const uint32_t* __restrict__ active, int pass) {
    const uint32_t a = *active, before = a & ((1u << pass) - 1u);
    Pass r;
    r.run = (a >> pass) & 1u;
    r.first = before == 0u;
    r.last = (a >> (pass + 1)) == 0u;
    r.src = r.first ? -1 : (__popc(before) - 1) & 1;
    return r;
}

// Per-CTA digit histogram of the keys next(i), i in [begin, end):
// hist[d * nb + cta].  Integer shared-memory atomics; all threads.
template <typename Next>
__device__ __forceinline__ void count_digits(int begin, int end, int nb, int shift, uint32_t* __restrict__ hist, Next next) {
    __shared__ uint32_t s_hist[2][kRadix];  // two copies: half the warps each
    for (int t = threadIdx.x; t < 2 * kRadix; t += kThreads) (&s_hist[0][0])[t] = 0u;
    __syncthreads();
    uint32_t* h = s_hist[(threadIdx.x >> 5) & 1];
#pragma unroll 8
    for (int i = begin + threadIdx.x; i < end; i += kThreads) atomicAdd(h + digit_of(next(i), shift), 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < kRadix; d += kThreads) hist[(size_t)d * nb + blockIdx.x] = s_hist[0][d] + s_hist[1][d];
}

// The first pass's histogram; diff[cta] = the bits in which the CTA's keys
// differ from key 0.  kMorton: the keys are those of the positions, and are
// written to `keys`.
template <bool kMorton>
__global__ void __launch_bounds__(kThreads) radix_first_kernel(const float* __restrict__ px, const float* __restrict__ py,
                                                               const float* __restrict__ pz, int32_t* __restrict__ keys,
                                                               int n, int per_cta, int nb, uint32_t* __restrict__ hist,
                                                               uint32_t* __restrict__ diff) {
    pdl_wait();
    __shared__ uint32_t s_diff[kWarps];
    const int begin = blockIdx.x * per_cta, end = min(begin + per_cta, n);
    const int32_t key0 = kMorton ? morton_key(__ldg(px), __ldg(py), __ldg(pz)) : keys[0];
    uint32_t d = 0u;
    count_digits(begin, end, nb, 0, hist, [&](int i) {
        int32_t key;
        if constexpr (kMorton) {
            key = morton_key(__ldg(px + i), __ldg(py + i), __ldg(pz + i));
            keys[i] = key;
        } else {
            key = keys[i];
        }
        d |= (uint32_t)(key ^ key0);
        return key;
    });
    d = __reduce_or_sync(0xffffffffu, d);
    if ((threadIdx.x & 31) == 0) s_diff[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < kWarps; ++w) d |= s_diff[w];
        diff[blockIdx.x] = d;
    }
}

// The histogram of a later pass.
__global__ void __launch_bounds__(kThreads) radix_hist_kernel(const int32_t* __restrict__ keys, SortScratch s, int pass) {
    pdl_wait();
    const Pass ps = pass_of(s.active, pass);
    if (!ps.run) return;
    const int32_t* in = ps.src < 0 ? keys : (ps.src ? s.key_b : s.key_a);
    const int begin = blockIdx.x * s.per_cta, end = min(begin + s.per_cta, s.n);
    count_digits(begin, end, s.nb, 8 * pass, s.hist, [&](int i) { return __ldg(in + i); });
}

// One CTA per digit: exclusive scan of the digit's CTA counts in place.  In the
// first pass CTA 0 also turns the CTAs' differing bits into the active passes.
__global__ void __launch_bounds__(kThreads) radix_spine_kernel(SortScratch s, int pass) {
    pdl_wait();
    __shared__ uint32_t s_warp[kWarps];
    if (pass == 0) {
        if (blockIdx.x == 0) {
            uint32_t d = 0u;
            for (int i = threadIdx.x; i < s.nb; i += kThreads) d |= s.diff[i];
            d = __reduce_or_sync(0xffffffffu, d);
            if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = d;
            __syncthreads();
            if (threadIdx.x == 0) {
#pragma unroll
                for (int w = 1; w < kWarps; ++w) d |= s_warp[w];
                uint32_t a = 0u;
                for (int k = 0; k < kPasses; ++k) a |= (d >> (8 * k) & 0xFFu) ? 1u << k : 0u;
                // equal keys: one pass still writes the identity
                *s.active = a ? a : 1u;
            }
            __syncthreads();
        }
    } else if (!pass_of(s.active, pass).run) {
        return;
    }
    uint32_t* row = s.hist + (size_t)blockIdx.x * s.nb;
    uint32_t carry = 0;
    for (int base = 0; base < s.nb; base += kThreads) {
        const int idx = base + threadIdx.x;
        const uint32_t v = idx < s.nb ? row[idx] : 0u;
        uint32_t tot;
        const uint32_t incl = block_scan_incl(v, s_warp, &tot);
        if (idx < s.nb) row[idx] = carry + incl - v;
        carry += tot;
    }
    if (threadIdx.x == 0) s.totals[blockIdx.x] = carry;
}

// Stable scatter of one pass.  The first one's values are the input positions;
// the last one writes the permutation (and rank/gidx) instead of keys and
// values.
__global__ void __launch_bounds__(kThreads) radix_scatter_kernel(const int32_t* __restrict__ keys, SortScratch s, int pass,
                                                                 int32_t* __restrict__ sigma,
                                                                 int32_t* __restrict__ rank_out,
                                                                 const int32_t* __restrict__ rank_in,
                                                                 int32_t* __restrict__ gidx) {
    pdl_wait();
    const Pass ps = pass_of(s.active, pass);
    if (!ps.run) return;
    const int32_t* keys_in = ps.src < 0 ? keys : (ps.src ? s.key_b : s.key_a);
    const int32_t* vals_in = ps.src ? s.val_b : s.val_a;
    const int dst = ps.src < 0 ? 0 : 1 - ps.src;
    int32_t* keys_out = dst ? s.key_b : s.key_a;
    int32_t* vals_out = ps.last ? sigma : (dst ? s.val_b : s.val_a);
    const int n = s.n, per_cta = s.per_cta, nb = s.nb, shift = 8 * pass;
    const uint32_t* hist = s.hist;
    const uint32_t* totals = s.totals;
    __shared__ uint32_t s_base[kRadix];    // global position of this CTA's next key of each digit
    __shared__ uint32_t s_tstart[kRadix];  // tile-local start of each digit
    __shared__ uint32_t s_tcount[kRadix];
    __shared__ uint32_t s_whist[kWarps][kRadix];
    __shared__ int32_t s_keys[kTile];
    __shared__ int32_t s_vals[kTile];
    __shared__ uint32_t s_warp[kWarps];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const uint32_t tot = totals[tid];
        uint32_t all;
        const uint32_t incl = block_scan_incl(tot, s_warp, &all);
        s_base[tid] = incl - tot + hist[(size_t)tid * nb + blockIdx.x];
    }
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s_whist[w][tid] = 0u;
    __syncthreads();

    const int begin = blockIdx.x * per_cta;
    const int end = min(begin + per_cta, n);
    const uint32_t lt = lanemask_lt();
    for (int tile = begin; tile < end; tile += kTile) {
        const int tile_n = min(kTile, end - tile);
        // All of the thread's loads, then all of its matches, are in flight
        // before the counters, which go one item after the other.
        int32_t k[kItems], v[kItems];
        uint32_t r[kItems], peers[kItems];
        const int first = warp * (32 * kItems) + lane;
#pragma unroll
        for (int it = 0; it < kItems; ++it) k[it] = first + it * 32 < tile_n ? __ldg(keys_in + tile + first + it * 32) : 0;
#pragma unroll
        for (int it = 0; it < kItems; ++it)
            v[it] = ps.first ? tile + first + it * 32 : (first + it * 32 < tile_n ? __ldg(vals_in + tile + first + it * 32) : 0);
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const uint32_t vmask = __ballot_sync(0xffffffffu, first + it * 32 < tile_n);
            peers[it] = __match_any_sync(0xffffffffu, digit_of(k[it], shift)) & vmask;
        }
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            uint32_t* h = &s_whist[warp][digit_of(k[it], shift)];
            const uint32_t before = *h;
            __syncwarp();
            if (first + it * 32 < tile_n && lane == __ffs(peers[it]) - 1) *h = before + __popc(peers[it]);
            __syncwarp();
            r[it] = before + __popc(peers[it] & lt);
        }
        __syncthreads();
        {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = s_whist[w][tid];
                s_whist[w][tid] = run;
                run += c;
            }
            s_tcount[tid] = run;
            uint32_t all;
            const uint32_t incl = block_scan_incl(run, s_warp, &all);
            s_tstart[tid] = incl - run;
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const int local = warp * (32 * kItems) + it * 32 + lane;
            if (local < tile_n) {
                const uint32_t d = digit_of(k[it], shift);
                const uint32_t pos = s_tstart[d] + s_whist[warp][d] + r[it];
                s_keys[pos] = k[it];
                s_vals[pos] = v[it];
            }
        }
        __syncthreads();
        for (int q = tid; q < tile_n; q += kThreads) {
            const int32_t key = s_keys[q];
            const int32_t val = s_vals[q];
            const uint32_t d = digit_of(key, shift);
            const uint32_t g = s_base[d] + (uint32_t)q - s_tstart[d];
            vals_out[g] = val;
            if (ps.last) {
                if (rank_out) rank_out[val] = (int32_t)g;
                if (gidx) gidx[g] = rank_in ? __ldg(rank_in + val) : val;
            } else {
                keys_out[g] = key;
            }
        }
        __syncthreads();
        s_base[tid] += s_tcount[tid];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s_whist[w][tid] = 0u;
        __syncthreads();
    }
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

void plan(int n, int* nb, int* per_cta) {
    const int tiles = std::max(1, (n + kTile - 1) / kTile);
    const int tiles_per_cta = std::max(1, (tiles + kMaxCtas - 1) / kMaxCtas);
    *per_cta = tiles_per_cta * kTile;
    *nb = std::max(1, (n + *per_cta - 1) / *per_cta);
}

}  // namespace

size_t sort_scratch_bytes(int n) {
    int nb, per;
    plan(n, &nb, &per);
    const size_t kv = align256((size_t)std::max(n, 1) * sizeof(int32_t));
    return 4 * kv + align256((size_t)kRadix * nb * sizeof(uint32_t)) + align256(kRadix * sizeof(uint32_t)) +
           align256(((size_t)nb + 1) * sizeof(uint32_t));
}

void sort_scratch_carve(void* base, int n, SortScratch* s) {
    int nb, per;
    plan(n, &nb, &per);
    const size_t kv = align256((size_t)std::max(n, 1) * sizeof(int32_t));
    char* p = static_cast<char*>(base);
    s->key_a = reinterpret_cast<int32_t*>(p);
    s->val_a = reinterpret_cast<int32_t*>(p + kv);
    s->key_b = reinterpret_cast<int32_t*>(p + 2 * kv);
    s->val_b = reinterpret_cast<int32_t*>(p + 3 * kv);
    s->hist = reinterpret_cast<uint32_t*>(p + 4 * kv);
    s->totals = reinterpret_cast<uint32_t*>(p + 4 * kv + align256((size_t)kRadix * nb * sizeof(uint32_t)));
    s->diff = s->totals + align256(kRadix * sizeof(uint32_t)) / sizeof(uint32_t);
    s->active = s->diff + nb;
    s->n = n;
    s->nb = nb;
    s->per_cta = per;
}

namespace {
template <bool kMorton>
int sort_passes(const float* px, const float* py, const float* pz, int32_t* keys, const SortScratch& s, int32_t* sigma,
                int32_t* rank_out, const int32_t* rank_in, int32_t* gidx, cudaStream_t st) {
    for (int pass = 0; pass < kPasses; ++pass) {
        if (pass == 0)
            launch_dep(radix_first_kernel<kMorton>, s.nb, kThreads, 0, st, px, py, pz, keys, s.n, s.per_cta, s.nb, s.hist,
                       s.diff);
        else
            launch_dep(radix_hist_kernel, s.nb, kThreads, 0, st, keys, s, pass);
        launch_dep(radix_spine_kernel, kRadix, kThreads, 0, st, s, pass);
        launch_dep(radix_scatter_kernel, s.nb, kThreads, 0, st, keys, s, pass, sigma, rank_out, rank_in, gidx);
    }
    return 3 * kPasses;
}
}  // namespace

int launch_morton_sort(const float* px, const float* py, const float* pz, int32_t* keys, const SortScratch& s,
                       int32_t* sigma, cudaStream_t st) {
    if (s.n <= 0) return 0;
    return sort_passes<true>(px, py, pz, keys, s, sigma, nullptr, nullptr, nullptr, st);
}

int launch_radix_sort(const int32_t* keys, int n, const SortScratch& s, int32_t* sigma, int32_t* rank_out,
                      const int32_t* rank_in, int32_t* gidx, cudaStream_t st) {
    if (n <= 0) return 0;
    // the keys are only read (kMorton false)
    return sort_passes<false>(nullptr, nullptr, nullptr, const_cast<int32_t*>(keys), s, sigma, rank_out, rank_in, gidx, st);
}

}  // namespace mpm
