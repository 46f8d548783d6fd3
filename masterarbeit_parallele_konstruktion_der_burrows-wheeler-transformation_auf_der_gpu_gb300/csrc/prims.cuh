// prims.cuh -- device-wide scan and stable LSD radix sort (sm_103a).
//
// Scan: one pass over the input (decoupled look-back), with functor loads and
// stores so that flags, compaction and segmented heads are computed on the
// fly instead of being materialised.
//
// Radix sort: stable LSD passes over 8-bit digits.  A pass ranks keys inside each warp with __match_any_sync multisplit, reorders the
// tile in shared memory and writes each digit's run with consecutive
// addresses.  (Measured on GB300: for the stable ranking, match beats a
// ballot-per-bit multisplit, whose ALU cost exceeds the match pipe's.)
#pragma once
#include "gbwt_internal.cuh"

namespace gbwt {

constexpr int SC_THREADS = 256;

// Scan operators.  diff(inc, ex) returns a value v with op(ex, v) == inc:
// the item itself for sums, the inclusive prefix for maxima (the scan hands
// stores that v, see k_scan).
struct OpAdd {
    template <typename T> __device__ __forceinline__ T operator()(T a, T b) const { return a + b; }
    template <typename T> __device__ __forceinline__ T diff(T inc, T ex) const { return inc - ex; }
};
// Component-wise max of the two 32-bit halves of a 64-bit word.
struct OpMax2 {
    __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const {
        uint32_t ah = (uint32_t)(a >> 32), bh = (uint32_t)(b >> 32);
        uint32_t al = (uint32_t)a, bl = (uint32_t)b;
        return ((uint64_t)(ah > bh ? ah : bh) << 32) | (al > bl ? al : bl);
    }
    __device__ __forceinline__ uint64_t diff(uint64_t inc, uint64_t) const { return inc; }
};
// High half: max; low half: sum (a running head with a running count).
struct OpMaxAdd {
    __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const
    {
        const uint32_t ah = (uint32_t)(a >> 32), bh = (uint32_t)(b >> 32);
        return ((uint64_t)(ah > bh ? ah : bh) << 32) | (uint32_t)((uint32_t)a + (uint32_t)b);
    }
    __device__ __forceinline__ uint64_t diff(uint64_t inc, uint64_t ex) const
    {
        return (inc & 0xFFFFFFFF00000000ull) | (uint32_t)((uint32_t)inc - (uint32_t)ex);
    }
};

// Warp shuffles of values wider than 8 bytes go member by member.
template <typename T>
__device__ __forceinline__ T shfl_xor_any(T v, int o)
{
    if constexpr (sizeof(T) <= 8) return __shfl_xor_sync(0xFFFFFFFFu, v, o);
    else return v.shfl_xor(o);
}
template <typename T>
__device__ __forceinline__ T shfl_up_any(T v, int o)
{
    if constexpr (sizeof(T) <= 8) return __shfl_up_sync(0xFFFFFFFFu, v, o);
    else return v.shfl_up(o);
}

// Four sums scanned together.
struct Sum4 {
    uint32_t a, b, c, d;
    Sum4() = default;
    __device__ __forceinline__ explicit Sum4(int) : a(0), b(0), c(0), d(0) {}
    __device__ __forceinline__ Sum4(uint32_t a_, uint32_t b_, uint32_t c_, uint32_t d_) : a(a_), b(b_), c(c_), d(d_) {}
    __device__ __forceinline__ Sum4 operator+(const Sum4 &o) const { return {a + o.a, b + o.b, c + o.c, d + o.d}; }
    __device__ __forceinline__ Sum4 operator-(const Sum4 &o) const { return {a - o.a, b - o.b, c - o.c, d - o.d}; }
    __device__ __forceinline__ Sum4 shfl_xor(int m) const
    {
        return {__shfl_xor_sync(0xFFFFFFFFu, a, m), __shfl_xor_sync(0xFFFFFFFFu, b, m),
                __shfl_xor_sync(0xFFFFFFFFu, c, m), __shfl_xor_sync(0xFFFFFFFFu, d, m)};
    }
    __device__ __forceinline__ Sum4 shfl_up(int m) const
    {
        return {__shfl_up_sync(0xFFFFFFFFu, a, m), __shfl_up_sync(0xFFFFFFFFu, b, m),
                __shfl_up_sync(0xFFFFFFFFu, c, m), __shfl_up_sync(0xFFFFFFFFu, d, m)};
    }
};

// Block-wide exclusive scan (identity 0); `total` receives the block total.
template <typename T, typename Op>
__device__ __forceinline__ T block_excl_scan(T v, T &total, Op op, T *s_warp /*[32]*/)
{
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned nw = (blockDim.x + 31) >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = shfl_up_any(x, o);
        if (lane >= (unsigned)o) x = op(y, x);
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < nw ? s_warp[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = shfl_up_any(w, o);
            if (lane >= (unsigned)o) w = op(y, w);
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    T wp = warp ? s_warp[warp - 1] : T(0);
    total = s_warp[nw - 1];
    T xe = shfl_up_any(x, 1);
    if (lane == 0) xe = T(0);
    __syncthreads();
    return op(wp, xe);
}

// ---- single-pass scan -------------------------------------------------
// One kernel per scan: every tile publishes its total, looks back over the
// published totals of the tiles before it (a warp reads 32 at a time) and
// publishes its inclusive prefix (Merrill & Garland 2016, "Single-pass
// parallel prefix scan with decoupled look-back").  Against a reduce pass, a
// scan of the tile totals and a second pass over the input (three to five
// launches, every input loaded twice), the load functors -- often chains of
// random reads -- run once and small inputs pay for one launch: the 8 MiB DNA
// text takes 59 launches fewer and 1.15 instead of 1.30 ms, a batch of 24
// texts 1.09 instead of 1.24 ms; at 512 MiB the two forms are level.
//
// Tiles are numbered by a ticket in the order their CTAs start, so a tile
// only waits for tiles whose CTAs are already running and every wait ends.
// A status is one 64-bit word per 32 bits of the value, each word carrying
// the same tag (scan number << 2 | state) in its high half: words are read
// and written whole, and a reader takes a value only when all its tags agree,
// so no fence is needed.  The scan number differs from call to call, so old
// statuses need no clearing; the CTA holding the last ticket resets the
// ticket counter.
constexpr uint32_t LB_TOTAL = 1u, LB_PREFIX = 2u;      // states
constexpr uint32_t LB_MAX_POLLS = 1u << 22;            // seconds; a wait ends after microseconds

struct LookBack {
    uint64_t *status;       // word w of tile t at status[w * stride + t]
    uint32_t stride;
    uint32_t seq;           // number of this scan, 1 .. 2^30 - 1
    uint32_t *ticket;       // 0 between scans
    uint32_t *err;          // set to 1 when a wait gave up
};

// Status words for a pass of `tiles` tiles on the storage's stream.
inline LookBack look_back(Storage *st, size_t tiles, size_t words)
{
    const size_t bytes = tiles * words * sizeof(uint64_t);
    const bool fresh = st->slots[S_LOOKBACK].cap < (bytes < 256 ? 256 : bytes);
    uint64_t *status = slot<uint64_t>(st, S_LOOKBACK, tiles * words);
    if (fresh || st->lb_seq >= (1u << 30) - 1u) {
        check_cuda(cudaMemsetAsync(status, 0, st->slots[S_LOOKBACK].cap, st->stream));
        st->lb_seq = 0;
    }
    st->lb_seq++;
    return LookBack{status, (uint32_t)tiles, st->lb_seq, (uint32_t *)(st->d_scalars + 60), st->h_err};
}

__device__ __forceinline__ void lb_store(uint64_t *p, uint64_t v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t lb_load(const uint64_t *p)
{
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lb_load32(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
template <typename T>
__device__ __forceinline__ void lb_publish(const LookBack &lb, uint32_t tile, T v, uint32_t state)
{
    constexpr int NW = sizeof(T) / 4;
    uint32_t w[NW];
    memcpy(w, &v, sizeof(T));
    const uint64_t tag = (uint64_t)((lb.seq << 2) | state) << 32;
#pragma unroll
    for (int k = 0; k < NW; k++) lb_store(lb.status + (size_t)k * lb.stride + tile, tag | w[k]);
}
// State of a tile (0 = nothing usable yet) and its value.
template <typename T>
__device__ __forceinline__ uint32_t lb_read(const LookBack &lb, uint32_t tile, T &v)
{
    constexpr int NW = sizeof(T) / 4;
    uint64_t q[NW];
#pragma unroll
    for (int k = 0; k < NW; k++) q[k] = lb_load(lb.status + (size_t)k * lb.stride + tile);
    uint32_t w[NW];
    const uint32_t tag = (uint32_t)(q[0] >> 32);
    bool same = (tag >> 2) == lb.seq;
#pragma unroll
    for (int k = 0; k < NW; k++) {
        same = same && (uint32_t)(q[k] >> 32) == tag;
        w[k] = (uint32_t)q[k];
    }
    memcpy(&v, w, sizeof(T));
    return same ? tag & 3u : 0u;
}

// Prefix of all tiles before `tile` (> 0), by one warp; every Op used here
// commutes, so the lanes' values combine in any order.  A round reads
// LB_WIDE x 32 statuses.  Measured on GB300 (32-bit sums in place): 34 M
// items in 106 us with 1, 122 us with 4 and 156 us with 8; 3 M items in
// 16.7, 20.1 and 24.9 us: the polls of waiting tiles compete with the
// statuses being published, so fewer reads per round win.
constexpr int LB_WIDE = 1;
template <typename T, typename Op>
__device__ __forceinline__ T lb_prefix(const LookBack &lb, uint32_t tile)
{
    const uint32_t lane = threadIdx.x & 31u;
    Op op;
    T acc = T(0);                              // per lane, combined at the end
    int64_t top = (int64_t)tile - 1;           // nearest tile not yet included
    uint32_t polls = 0;
    bool found = false;
    while (top >= 0 && !found) {
        T v[LB_WIDE];
        uint32_t state[LB_WIDE];
#pragma unroll
        for (int k = 0; k < LB_WIDE; k++) {
            const int64_t i = top - (int64_t)(k * 32) - (int64_t)lane;
            v[k] = T(0);
            state[k] = LB_PREFIX;              // before the first tile: identity
            if (i >= 0) state[k] = lb_read<T>(lb, (uint32_t)i, v[k]);
        }
#pragma unroll
        for (int k = 0; k < LB_WIDE; k++) {
            const unsigned rm = __ballot_sync(0xFFFFFFFFu, state[k] != 0u);
            const unsigned pm = __ballot_sync(0xFFFFFFFFu, state[k] == LB_PREFIX);
            // lanes up to the nearest inclusive prefix, or all 32
            const unsigned need = pm ? (0xFFFFFFFFu >> (32 - __ffs(pm))) : 0xFFFFFFFFu;
            if ((rm & need) != need) {
                // never runs out: see above.  The host refuses the result if it does.
                if (++polls >= LB_MAX_POLLS) {
                    if (lane == 0) *(volatile uint32_t *)lb.err = 1u;
                    found = true;
                }
                break;
            }
            if ((need >> lane) & 1u) acc = op(acc, v[k]);
            if (pm) { found = true; break; }
            top -= 32;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = op(acc, shfl_xor_any(acc, o));
    return acc;
}

// Shared-memory slot of tile item i: one padding slot per 32 items, so the
// blocked accesses (thread t, items IT*t ..) hit distinct banks.
__device__ __forceinline__ uint32_t sc_pad(uint32_t i) { return i + (i >> 5); }

// Loads and stores run in striped order (consecutive threads on consecutive
// items, so both coalesce); the blocked prefixes go through shared memory.
// store(i, prefix, v) gets the exclusive (or inclusive) prefix and
// v = op.diff(inclusive, exclusive) -- the item's value for sums.
template <typename T, typename Op, int IT, typename Load, typename Store>
__global__ void __launch_bounds__(SC_THREADS) k_scan(Load load, Store store, size_t n, LookBack lb, bool inclusive,
                                                     T *total_out)
{
    constexpr int TILE = SC_THREADS * IT;
    __shared__ T s_tile[TILE + TILE / 32 + 1];
    __shared__ T s_warp[32];
    __shared__ uint32_t s_id;
    Op op;
    uint32_t tile = 0;
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) {
            s_id = atomicAdd(lb.ticket, 1u);
            if (s_id == gridDim.x - 1) *lb.ticket = 0;
        }
        __syncthreads();
        tile = s_id;
    }
    const size_t base = (size_t)tile * TILE;
#pragma unroll
    for (int j = 0; j < IT; j++) {
        const size_t i = base + (size_t)j * SC_THREADS + threadIdx.x;
        s_tile[sc_pad(j * SC_THREADS + threadIdx.x)] = i < n ? load(i) : T(0);
    }
    __syncthreads();
    T v[IT];
    T sum = T(0);
#pragma unroll
    for (int j = 0; j < IT; j++) {
        v[j] = s_tile[sc_pad(threadIdx.x * IT + j)];
        sum = op(sum, v[j]);
    }
    T total;
    T run = block_excl_scan<T, Op>(sum, total, op, s_warp);   // ends with a barrier: s_tile and s_warp are free
    if (gridDim.x > 1) {
        if (threadIdx.x < 32) {
            if (threadIdx.x == 0) lb_publish(lb, tile, total, tile ? LB_TOTAL : LB_PREFIX);
            if (tile) {
                const T pre = lb_prefix<T, Op>(lb, tile);
                if (threadIdx.x == 0) {
                    lb_publish(lb, tile, op(pre, total), LB_PREFIX);
                    s_warp[0] = pre;
                }
            } else if (threadIdx.x == 0) {
                s_warp[0] = T(0);
            }
        }
        __syncthreads();
        run = op(s_warp[0], run);
    }
    // exclusive prefixes of the tile's items (items past n add the identity)
#pragma unroll
    for (int j = 0; j < IT; j++) {
        s_tile[sc_pad(threadIdx.x * IT + j)] = run;
        run = op(run, v[j]);
    }
    if (threadIdx.x == SC_THREADS - 1) s_tile[sc_pad(TILE)] = run;
    __syncthreads();
#pragma unroll 4
    for (int j = 0; j < IT; j++) {
        const uint32_t li = (uint32_t)j * SC_THREADS + threadIdx.x;
        const size_t i = base + li;
        if (i < n) {
            const T exi = s_tile[sc_pad(li)], inc = s_tile[sc_pad(li + 1)];
            store(i, inclusive ? inc : exi, op.diff(inc, exi));
            if (total_out && i == n - 1) *total_out = inc;
        }
    }
}

template <typename T>
struct LoadArr {
    const T *a;
    __device__ __forceinline__ T operator()(size_t i) const { return a[i]; }
};
struct LoadPopc {                      // bits set in a word
    const uint32_t *w;
    __device__ __forceinline__ uint32_t operator()(size_t i) const { return (uint32_t)__popc(w[i]); }
};
template <typename T>
struct StoreArr {
    T *a;
    __device__ __forceinline__ void operator()(size_t i, T pre, T) const { a[i] = pre; }
};

// Scan of load(i), i in [0,n): store(i, prefix, value) is called with the
// exclusive (or inclusive) prefix.  The total is written to *total_dev when
// given (device pointer; left untouched for n == 0).  In-place scans are
// fine: a tile reads its items before it writes them and no other tile's.
// Inputs that give every SM fewer than eight such tiles take tiles of four
// items per thread, so that they spread over the SMs instead of running as
// one long chain of dependent loads; larger ones take as many as fit about 32
// KB of shared memory: fewer tiles for a prefix to travel over (130 M 32-bit
// items in 314 us with 32 per thread, 367 us with 16).  SMALL = 1 is for loads that
// loop themselves, LARGE for loads of several dependent reads, whose chain per
// thread counts more than the tiles (active test of a big group, 16 M items: 247 us
// with 32, 175 with 16, 161 with 8).
template <typename T, typename Op, int SMALL = 4, int LARGE = 0, typename Load, typename Store>
void device_scan(Storage *st, size_t n, Load load, Store store, bool inclusive, T *total_dev)
{
    if (n == 0) return;
    constexpr int BIG = LARGE ? LARGE : sizeof(T) == 4 ? 32 : sizeof(T) == 8 ? 16 : 8;
    const bool small = n <= (size_t)st->num_sms * 8 * SC_THREADS * SMALL;
    const size_t per = (size_t)SC_THREADS * (small ? SMALL : BIG);
    const size_t tiles = (n + per - 1) / per;
    const LookBack lb = look_back(st, tiles, sizeof(T) / 4);
    if (small) k_scan<T, Op, SMALL><<<(unsigned)tiles, SC_THREADS, 0, st->stream>>>(load, store, n, lb, inclusive, total_dev);
    else k_scan<T, Op, BIG><<<(unsigned)tiles, SC_THREADS, 0, st->stream>>>(load, store, n, lb, inclusive, total_dev);
    after_launch(st);
}

// Product modulo 2^61 - 1 of two values below it (phrase fingerprints).
constexpr uint64_t M61 = (1ull << 61) - 1ull;
__device__ __forceinline__ uint64_t mulmod61(uint64_t a, uint64_t b)
{
    uint64_t lo = a * b, hi = __umul64hi(a, b);
    uint64_t r = (lo & M61) + (lo >> 61) + (hi << 3);
    r = (r & M61) + (r >> 61);
    return r >= M61 ? r - M61 : r;
}

// ---------------------------------------------------------------------
// Stable LSD radix sort, in two forms.
//
// Up to two tiles per SM (one wave): one kernel counts the digits of every
// pass in one read of the keys, and each pass is one kernel in which a tile
// counts its digits, publishes the counts and looks back over the tiles before
// it, digit by digit (onesweep: Adinets & Merrill 2022, "Onesweep: a faster
// least significant digit radix sort for GPUs").  A single tile needs no
// counts either: one launch per pass.
//
// Above that: a tile histogram, a scan of all tile histograms and a scatter
// per pass.  The look-back then costs more than the launches: tiles of 4096
// keys leave at 40 to 80 a microsecond, and with an L2 read of about 0.7 us
// between the dies every digit walks back over tens of tiles.
//
// Measured, 40-bit keys with values in 5 passes, look-back / histograms: 1 M
// keys (20 to 100 tiles) 89..102 / 124 us, 168 tiles 135 / 163 us, 300 tiles 162
// / 165 us, 1500 tiles 569 / 557 us; per pass of 243 M 32-bit keys 1541 / 890 us.
// ---------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;

template <typename K>
__device__ __forceinline__ uint32_t rs_digit(K k, int shift, uint32_t mask)
{
    return (uint32_t)(k >> shift) & mask;
}

// Ranking can split its items between two warp multisplits so that both
// issue pipes work: __match_any_sync (one instruction, limited by its pipe)
// and one ballot per digit bit (ALU work); every BALLOT-th item uses ballots
// (template argument, 0 = never).  Measured on GB300 for the batched output
// sort (u32 keys, uniform 8-bit digits): 727 us per pass with match only,
// 595 us with BALLOT = 3, 580 us with BALLOT = 2.  The match instruction's
// cost grows with the number of distinct digits in a warp, so sorts whose
// warps see few distinct digits keep match only.

// Lanes of the warp holding the same digit d (< 2^BITS, or 0xFFFFFFFF for
// no key: those lanes form their own class).
template <int BITS>
__device__ __forceinline__ unsigned rs_peers_ballot(uint32_t d)
{
    const bool valid = d != 0xFFFFFFFFu;
    const unsigned vm = __ballot_sync(0xFFFFFFFFu, valid);
    unsigned m = valid ? vm : ~vm;
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const unsigned v = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
        m &= ((d >> b) & 1u) ? v : ~v;
    }
    return m;
}


// A segmented sort: the tiles are grouped into segments of whole tiles that
// are sorted on their own.
struct RsSegs {
    const uint2 *tseg = nullptr;      // per tile: {first tile, tiles} of its segment (null: one segment)
    const uint32_t *sid = nullptr;    // per tile: number of its segment
    uint32_t nseg = 1;
};

// Histogram slot of digit d for tile b.  Unsegmented: digit-major over all
// tiles.  Segmented (tseg[b] = {first tile, tiles} of b's segment, every
// segment a whole number of tiles): segment-major, then digit-major inside
// the segment, so one exclusive scan gives every tile its offsets inside its
// own segment and each pass sorts the segments independently.
__device__ __forceinline__ size_t rs_hist_index(const RsSegs &sg, uint32_t b, uint32_t d, uint32_t num_tiles, int D)
{
    if (!sg.tseg) return (size_t)d * num_tiles + b;
    const uint2 q = sg.tseg[b];
    return (size_t)q.x * D + (size_t)d * q.y + (b - q.x);
}

template <typename K, int BITS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const K *__restrict__ keys, uint32_t n, int shift,
                                                           uint32_t mask, uint32_t *__restrict__ tile_hist,
                                                           uint32_t num_tiles, RsSegs sg)
{
    constexpr int D = 1 << BITS;
    __shared__ uint32_t h[RS_WARPS * D];       // one histogram per warp
    for (int d = threadIdx.x; d < RS_WARPS * D; d += RS_THREADS) h[d] = 0;
    __syncthreads();
    uint32_t *wh = h + (threadIdx.x >> 5) * D;
    const size_t base = (size_t)blockIdx.x * RS_TILE;
    constexpr int KPV = 16 / (int)sizeof(K);          // keys per 16-byte load
    constexpr int NV = RS_ITEMS / KPV;
    if (base + RS_TILE <= n && (((uintptr_t)keys) & 15u) == 0) {
        // full tile: every load issued before any count (counting needs no order)
        uint4 v[NV];
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] = __ldg((const uint4 *)(keys + base) + (size_t)j * RS_THREADS + threadIdx.x);
#pragma unroll
        for (int j = 0; j < NV; j++) {
            K kk[KPV];
            memcpy(kk, &v[j], 16);
#pragma unroll
            for (int q = 0; q < KPV; q++) atomicAdd(&wh[rs_digit(kk[q], shift, mask)], 1u);
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < RS_ITEMS; j++) {
            size_t i = base + (size_t)j * RS_THREADS + threadIdx.x;
            if (i < n) atomicAdd(&wh[rs_digit(keys[i], shift, mask)], 1u);
        }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < D; d += RS_THREADS) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) sum += h[w * D + d];
        tile_hist[rs_hist_index(sg, blockIdx.x, d, num_tiles, D)] = sum;
    }
}

// Digit counts of all passes of a sort of few tiles, one CTA per tile (eight
// tiles a CTA took 24 us for the 168 tiles of an 8 MiB text's dictionary, one 12
// us): hist[(p * nseg + segment) * D + digit], added up from shared memory
// (several copies: the digits of a small alphabet repeat).
template <typename K, int BITS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const K *__restrict__ keys, uint32_t n, int begin_bit,
                                                        int end_bit, RsSegs sg, uint32_t *__restrict__ hist)
{
    constexpr int D = 1 << BITS;
    constexpr int PMAX = ((int)sizeof(K) * 8 + BITS - 1) / BITS;
    constexpr int FIT = 32768 / (PMAX * D * 4);
    constexpr int COPIES = FIT >= 4 ? 4 : FIT >= 2 ? 2 : 1;
    __shared__ uint32_t h[COPIES * PMAX * D];
    const int np = (end_bit - begin_bit + BITS - 1) / BITS;
    for (int c = 0; c < COPIES; c++)
        for (int i = threadIdx.x; i < np * D; i += RS_THREADS) h[c * (PMAX * D) + i] = 0;
    __syncthreads();
    uint32_t *mine = h + ((threadIdx.x >> 5) % COPIES) * (PMAX * D);
    const uint32_t base = blockIdx.x * (uint32_t)RS_TILE;
#pragma unroll
    for (int j = 0; j < RS_ITEMS; j++) {
        const uint32_t i = base + (uint32_t)j * RS_THREADS + threadIdx.x;
        if (i >= n) break;
        const K k = keys[i];
        for (int p = 0; p < np; p++) {
            const int shift = begin_bit + p * BITS;
            const int bits = end_bit - shift < BITS ? end_bit - shift : BITS;
            atomicAdd(&mine[p * D + rs_digit(k, shift, (1u << bits) - 1u)], 1u);
        }
    }
    __syncthreads();
    const uint32_t seg = sg.sid ? sg.sid[blockIdx.x] : 0u;
    for (int i = threadIdx.x; i < np * D; i += RS_THREADS) {
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < COPIES; k++) c += h[k * (PMAX * D) + i];
        if (c) atomicAdd(hist + ((size_t)(i / D) * sg.nseg + seg) * D + i % D, c);
    }
}

// Place of a digit's `cnt` keys (of one tile) among the n: `at`, unless they
// would reach past the end.  A wrong count is then an error code and not a write
// outside the buffers.  One compare per digit and tile: a compare per key took
// 1 % of the 512 MiB DNA text (14.45 -> 14.60 ms).
__device__ __forceinline__ uint32_t rs_checked(uint32_t at, uint32_t cnt, uint32_t n, uint32_t *flags)
{
    if (at <= n - cnt) return at;              // cnt <= n: the tile's keys are among them
    atomicOr(flags, ERR_INTERNAL);
    return n - cnt;
}

template <typename K, bool HAS_VAL, int BITS>
constexpr size_t rs_smem_bytes()
{
    return (size_t)RS_TILE * sizeof(K) + (HAS_VAL ? (size_t)RS_TILE * 4 : 0) + (size_t)RS_WARPS * (1 << BITS) * 4 +
           (size_t)(1 << BITS) * 4 * 2 + 32 * 8;
}

// Scatter of one pass, places from the scanned tile histograms.  The time of a
// tile is a chain of latencies (three or two CTAs an SM, DRAM and issue slots
// half idle), so the chain is kept short: the tile's offsets (num_tiles words
// apart) and all keys are in flight before the first barrier, every warp
// clears its own counters, a digit's start in the tile is folded into the
// counters and into its offset (one shared read per key less in both places).
// Passes of 512 MiB DNA: 243 M 32-bit keys 740 -> 542 us (offsets loaded after
// ranking and one barrier more: 667; offsets early: 604), 34 M 32-bit keys with
// values 204 -> 178 us, 26 M 64-bit keys with values 136 -> 111 us.  Three CTAs
// of 32-bit keys fit in 80 registers, more or wider keys would spill.
template <typename K, bool HAS_VAL, int BITS, int BALLOT>
__global__ void __launch_bounds__(RS_THREADS, sizeof(K) == 4 && !HAS_VAL ? 3 : 2)
k_rs_downsweep(const K *__restrict__ kin, K *__restrict__ kout, const uint32_t *__restrict__ vin,
               uint32_t *__restrict__ vout, uint32_t n, int shift, uint32_t mask,
               const uint32_t *tile_off, uint32_t num_tiles, RsSegs sg, uint32_t *flags)
{
    constexpr int D = 1 << BITS;
    constexpr int DPT = D / RS_THREADS;       // digits per thread in the per-digit phase
    extern __shared__ __align__(16) unsigned char rs_smem[];
    K *s_k = (K *)rs_smem;
    uint32_t *s_v = (uint32_t *)(s_k + RS_TILE);
    uint32_t *s_wh = HAS_VAL ? s_v + RS_TILE : s_v;
    uint32_t *s_goff = s_wh + RS_WARPS * D;
    uint32_t *s_scan = s_goff + D;

    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t off[DPT];                        // loaded early: num_tiles words apart
#pragma unroll
    for (int e = 0; e < DPT; e++)
        off[e] = lb_load32(tile_off + rs_hist_index(sg, blockIdx.x, threadIdx.x * DPT + e, num_tiles, D));
    const size_t tile_base = (size_t)blockIdx.x * RS_TILE;
    const size_t wbase = tile_base + (size_t)warp * (RS_ITEMS * 32);
    K k[RS_ITEMS];
    uint32_t v[RS_ITEMS];
    uint32_t rk[RS_ITEMS];
    uint32_t dg[RS_ITEMS];
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        size_t idx = wbase + (size_t)i * 32 + lane;
        bool valid = idx < n;
        k[i] = valid ? kin[idx] : K(0);
        if (HAS_VAL) v[i] = !vin ? (uint32_t)idx : valid ? vin[idx] : 0u;
        dg[i] = valid ? rs_digit(k[i], shift, mask) : 0xFFFFFFFFu;
    }
    uint32_t *wh = s_wh + warp * D;
    for (int i = lane; i < D; i += 32) wh[i] = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        // every lane reads its digit's counter (one bank access per digit, as
        // for one lane), then the lowest lane of the class advances it
        const uint32_t d = dg[i];
        const unsigned peers = (BALLOT > 0 && i % (BALLOT > 0 ? BALLOT : 1) == (BALLOT > 0 ? BALLOT - 1 : 0))
                                   ? rs_peers_ballot<BITS>(d)
                                   : __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t below = (uint32_t)__popc(peers & ((1u << lane) - 1u));
        const uint32_t prior = d != 0xFFFFFFFFu ? wh[d] : 0u;
        __syncwarp();
        if (below == 0 && d != 0xFFFFFFFFu) wh[d] = prior + (uint32_t)__popc(peers);
        rk[i] = prior + below;
        __syncwarp();
    }
    __syncthreads();
    {
        // thread t owns digits [t*DPT, t*DPT + DPT)
        uint32_t cnt[DPT];
        uint32_t sum = 0;
#pragma unroll
        for (int e = 0; e < DPT; e++) {
            const uint32_t d = threadIdx.x * DPT + e;
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) run += s_wh[w * D + d];
            cnt[e] = run;
            sum += run;
        }
        uint32_t total;
        uint32_t ex = block_excl_scan<uint32_t, OpAdd>(sum, total, OpAdd(), s_scan);
#pragma unroll
        for (int e = 0; e < DPT; e++) {
            const uint32_t d = threadIdx.x * DPT + e;
            s_goff[d] = rs_checked(off[e], cnt[e], n, flags) - ex;
            uint32_t run = ex;
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) {
                const uint32_t c = s_wh[w * D + d];
                s_wh[w * D + d] = run;
                run += c;
            }
            ex += cnt[e];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        if (dg[i] != 0xFFFFFFFFu) {
            uint32_t lp = wh[dg[i]] + rk[i];
            s_k[lp] = k[i];
            if (HAS_VAL) s_v[lp] = v[i];
        }
    }
    __syncthreads();
    const uint32_t tile_n = (uint32_t)(((size_t)n - tile_base) < (size_t)RS_TILE ? ((size_t)n - tile_base) : RS_TILE);
    for (uint32_t j = threadIdx.x; j < tile_n; j += RS_THREADS) {
        K kk = s_k[j];
        const uint32_t g = s_goff[rs_digit(kk, shift, mask)] + j;
        kout[g] = kk;
        if (HAS_VAL) vout[g] = s_v[j];
    }
}

// One pass by look-back.  status[tile * D + digit] is a look-back word: the
// tile's own count (LB_TOTAL) or the count up to and including the tile
// (LB_PREFIX).  Counts are published before the tile is reordered in shared
// memory, so most predecessors have theirs in place when the look-back
// starts.  A single tile needs neither counts nor look-back.
template <typename K, bool HAS_VAL, int BITS, int BALLOT>
__global__ void __launch_bounds__(RS_THREADS, 2)
k_rs_pass(const K *__restrict__ kin, K *__restrict__ kout, const uint32_t *__restrict__ vin,
          uint32_t *__restrict__ vout, uint32_t n, int shift, uint32_t mask, const uint32_t *hist, RsSegs sg,
          LookBack lb, uint32_t *flags)
{
    constexpr int D = 1 << BITS;
    constexpr int DPT = D / RS_THREADS;       // digits per thread in the per-digit phases
    extern __shared__ __align__(16) unsigned char rs_smem[];
    K *s_k = (K *)rs_smem;
    uint32_t *s_v = (uint32_t *)(s_k + RS_TILE);
    uint32_t *s_wh = HAS_VAL ? s_v + RS_TILE : s_v;
    uint32_t *s_dstart = s_wh + RS_WARPS * D;
    uint32_t *s_goff = s_dstart + D;
    uint64_t *s_scan = (uint64_t *)(s_goff + D);

    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t tile = 0;
    if (gridDim.x > 1 && threadIdx.x == 0) {
        tile = atomicAdd(lb.ticket, 1u);
        if (tile == gridDim.x - 1) *lb.ticket = 0;
        s_dstart[0] = tile;
    }
    uint32_t *wh = s_wh + warp * D;
    for (int i = lane; i < D; i += 32) wh[i] = 0;
    __syncthreads();
    if (gridDim.x > 1) tile = s_dstart[0];
    // Tiles of the segment (first, count) and its digit counts, loaded early.
    // Through a `const __restrict__` pointer some compiled instances (9-bit
    // digits, two tiles) summed other digits' counts.  Nothing writes the counts
    // while the kernel runs, so the qualifier was legal and the source does not
    // show the cause; relaxed loads are free of it in every instance.
    uint2 q = make_uint2(0u, gridDim.x);
    uint32_t seg = 0;
    if (sg.tseg) { q = sg.tseg[tile]; seg = sg.sid[tile]; }
    uint32_t hd[DPT];
#pragma unroll
    for (int e = 0; e < DPT; e++) hd[e] = q.y > 1 ? lb_load32(hist + (size_t)seg * D + threadIdx.x * DPT + e) : 0u;

    const size_t tile_base = (size_t)tile * RS_TILE;
    const size_t wbase = tile_base + (size_t)warp * (RS_ITEMS * 32);
    K k[RS_ITEMS];
    uint32_t v[RS_ITEMS];
    uint32_t rk[RS_ITEMS];
    uint32_t dg[RS_ITEMS];
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        size_t idx = wbase + (size_t)i * 32 + lane;
        bool valid = idx < n;
        k[i] = valid ? kin[idx] : K(0);
        if (HAS_VAL) v[i] = !vin ? (uint32_t)idx : valid ? vin[idx] : 0u;
        dg[i] = valid ? rs_digit(k[i], shift, mask) : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const uint32_t d = dg[i];           // ranked as in k_rs_downsweep
        const unsigned peers = (BALLOT > 0 && i % (BALLOT > 0 ? BALLOT : 1) == (BALLOT > 0 ? BALLOT - 1 : 0))
                                   ? rs_peers_ballot<BITS>(d)
                                   : __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t below = (uint32_t)__popc(peers & ((1u << lane) - 1u));
        const uint32_t prior = d != 0xFFFFFFFFu ? wh[d] : 0u;
        __syncwarp();
        if (below == 0 && d != 0xFFFFFFFFu) wh[d] = prior + (uint32_t)__popc(peers);
        rk[i] = prior + below;
        __syncwarp();
    }
    __syncthreads();
    // thread t owns digits [t*DPT, t*DPT + DPT): the tile's counts (low words)
    // and the segment's (high words) scanned together
    uint32_t cnt[DPT], gbase[DPT];
    {
        uint64_t both[DPT], sum = 0;
#pragma unroll
        for (int e = 0; e < DPT; e++) {
            const uint32_t d = threadIdx.x * DPT + e;
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) {
                uint32_t c = s_wh[w * D + d];
                s_wh[w * D + d] = run;
                run += c;
            }
            cnt[e] = run;
            if (q.y > 1) {
                lb_store(lb.status + (size_t)tile * D + d,
                         ((uint64_t)((lb.seq << 2) | (tile == q.x ? LB_PREFIX : LB_TOTAL)) << 32) | run);
                both[e] = ((uint64_t)hd[e] << 32) | run;
            } else {
                both[e] = ((uint64_t)run << 32) | run;       // alone in its segment
            }
            sum += both[e];
        }
        uint64_t total;
        uint64_t ex = block_excl_scan<uint64_t, OpAdd>(sum, total, OpAdd(), s_scan);
#pragma unroll
        for (int e = 0; e < DPT; e++) {
            s_dstart[threadIdx.x * DPT + e] = (uint32_t)ex;
            gbase[e] = q.x * (uint32_t)RS_TILE + (uint32_t)(ex >> 32);
            ex += both[e];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        if (dg[i] != 0xFFFFFFFFu) {
            uint32_t lp = s_dstart[dg[i]] + wh[dg[i]] + rk[i];
            s_k[lp] = k[i];
            if (HAS_VAL) s_v[lp] = v[i];
        }
    }
#pragma unroll
    for (int e = 0; e < DPT; e++) {
        const uint32_t d = threadIdx.x * DPT + e;
        uint32_t pre = 0;
        if (tile != q.x) {
            // four predecessors a step: all tiles run at once, and the last ones
            // walk far before a prefix meets them (168 tiles, 64-bit keys with
            // values: 15.0 -> 14.4 us a pass with the early loads)
            uint32_t p = tile, polls = 0;
            bool found = false;
            while (!found) {
                uint64_t w[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; j++)
                    w[j] = j < p - q.x ? lb_load(lb.status + (size_t)(p - 1u - j) * D + d) : 0u;
                const uint32_t from = p;
                bool go = true;
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) {
                    const uint32_t tag = (uint32_t)(w[j] >> 32);
                    go = go && (tag >> 2) == lb.seq;
                    if (go) {
                        pre += (uint32_t)w[j];
                        p--;
                        found = (tag & 3u) == LB_PREFIX;
                        go = !found;
                    }
                }
                // never runs out (tickets, see above); places only shrink, the host refuses the result
                if (p == from && ++polls >= LB_MAX_POLLS) { *(volatile uint32_t *)lb.err = 1u; break; }
            }
            lb_store(lb.status + (size_t)tile * D + d,
                     ((uint64_t)((lb.seq << 2) | LB_PREFIX) << 32) | (pre + cnt[e]));
        }
        s_goff[d] = rs_checked(gbase[e] + pre, cnt[e], n, flags) - s_dstart[d];
    }
    __syncthreads();
    const uint32_t tile_n = (uint32_t)(((size_t)n - tile_base) < (size_t)RS_TILE ? ((size_t)n - tile_base) : RS_TILE);
    for (uint32_t j = threadIdx.x; j < tile_n; j += RS_THREADS) {
        K kk = s_k[j];
        const uint32_t g = s_goff[rs_digit(kk, shift, mask)] + j;
        kout[g] = kk;
        if (HAS_VAL) vout[g] = s_v[j];
    }
}

static __global__ void k_iota(uint32_t *v, uint32_t n)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

// Sorts (keys, vals) stably by bits [begin_bit, end_bit) with BITS-bit digits
// (8: 256 buckets; 10: 1024 buckets, fewer passes for 17..20-bit keys).  On
// return `keys` and `vals` point at the sorted data (the *_alt buffers hold
// garbage).  With `iota` the values are the positions 0..n-1 (vals need not be
// filled).  With segments (n a multiple of RS_TILE) every segment is sorted on
// its own.
//
// Internal linkage: every source file has kernels of its own, and attr_set has
// to speak for those.  With one attr_set for the library, the first file to
// sort 64-bit keys with values (59 KB of shared memory) left the other's
// kernels at 48 KB and their launches failed.
template <typename K, bool HAS_VAL, int BITS = 8, int BALLOT = 0>
static void radix_sort(Storage *st, K *&keys, K *&keys_alt, uint32_t *&vals, uint32_t *&vals_alt, uint32_t n,
                int begin_bit, int end_bit, RsSegs sg = RsSegs(), bool iota = false)
{
    static_assert((1 << BITS) % RS_THREADS == 0, "digit count must be a multiple of the CTA size");
    if (n <= 1 || end_bit <= begin_bit) {
        if (iota && n) {
            k_iota<<<grid_for(n, 256), 256, 0, st->stream>>>(vals, n);
            after_launch(st);
        }
        return;
    }
    static bool attr_set = false;
    constexpr size_t smem = rs_smem_bytes<K, HAS_VAL, BITS>();
    if (!attr_set) {
        check_cuda(cudaFuncSetAttribute(k_rs_pass<K, HAS_VAL, BITS, BALLOT>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        check_cuda(cudaFuncSetAttribute(k_rs_downsweep<K, HAS_VAL, BITS, BALLOT>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
    }
    const uint32_t num_tiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
    const size_t D = (size_t)1 << BITS;
    const int np = (end_bit - begin_bit + BITS - 1) / BITS;
    uint32_t *hist = nullptr;
    const bool small = num_tiles <= 2u * (uint32_t)st->num_sms;
    if (!small) {
        hist = slot<uint32_t>(st, S_RSHIST, D * num_tiles);
    } else if (num_tiles > 1) {
        const size_t words = (size_t)np * sg.nseg * D;
        hist = slot<uint32_t>(st, S_RSHIST, words);
        check_cuda(cudaMemsetAsync(hist, 0, words * sizeof(uint32_t), st->stream));
        k_rs_hist<K, BITS><<<num_tiles, RS_THREADS, 0, st->stream>>>(keys, n, begin_bit, end_bit, sg, hist);
        after_launch(st);
    }
    for (int p = 0; p < np; p++) {
        const int shift = begin_bit + p * BITS;
        int bits = end_bit - shift < BITS ? end_bit - shift : BITS;
        uint32_t mask = (1u << bits) - 1u;
        LookBack lb{};
        if (!small) {
            k_rs_upsweep<K, BITS><<<num_tiles, RS_THREADS, 0, st->stream>>>(keys, n, shift, mask, hist, num_tiles, sg);
            after_launch(st);
            device_scan<uint32_t, OpAdd>(st, D * num_tiles, LoadArr<uint32_t>{hist}, StoreArr<uint32_t>{hist}, false,
                                         (uint32_t *)nullptr);
        } else if (num_tiles > 1) {
            lb = look_back(st, (size_t)num_tiles * D, 1);
        }
        probe_begin(st, GBWT_PROBE_RADIX_SCATTER);
        const uint32_t *vi = iota && p == 0 ? nullptr : vals;
        if (small)
            k_rs_pass<K, HAS_VAL, BITS, BALLOT><<<num_tiles, RS_THREADS, smem, st->stream>>>(
                keys, keys_alt, vi, vals_alt, n, shift, mask, hist ? hist + (size_t)p * sg.nseg * D : nullptr, sg, lb,
                st->d_flags);
        else
            k_rs_downsweep<K, HAS_VAL, BITS, BALLOT><<<num_tiles, RS_THREADS, smem, st->stream>>>(
                keys, keys_alt, vi, vals_alt, n, shift, mask, hist, num_tiles, sg, st->d_flags);
        probe_end(st, GBWT_PROBE_RADIX_SCATTER, (uint64_t)n * 2 * (sizeof(K) + (HAS_VAL ? 4 : 0)));
        after_launch(st);
        K *t = keys; keys = keys_alt; keys_alt = t;
        if (HAS_VAL) { uint32_t *u = vals; vals = vals_alt; vals_alt = u; }
    }
}

}  // namespace gbwt
