// pfp_unbwt.cu -- inverse BWT on the GPU (sm_103a).
//
// The reference declares libcubwt_unbwt but does not define it
// (libcubwt.cuh:101; its LF kernels are at libcubwt.cu:2453-2925).  Here:
//
//   rows   0..n of the BWT of T$; row 0 is the suffix "$".  Element e of the
//          input belongs to a row (UbIn): libcubwt's L lists the rows without
//          the '$' row; the PFP output O lists rows 1..n, with row 0's symbol
//          standing in the '$' row.  Both are read as they are.
//   LF     LF(r) = 1 + (position of row r in the stable sort of the non-'$'
//          rows by symbol), LF($ row) = 0.  One counting pass: tile
//          histograms, a digit-major scan, and a ranking pass (warp match
//          multisplit, as in the radix downsweep) that writes LF in row
//          order, so nothing is scattered.
//   walk   T[n-1-k] = B[LF^k(0)].  Blocks of 32 rows whose hash falls in 1/rate
//          are rulers (block 0 always); an LF entry whose target is a ruler
//          row holds bit 31 | the row's ruler number.  A lane follows LF from a
//          ruler row to the next one and records the distance; list ranking
//          over the chain of ruler rows gives each its distance from row 0; a
//          second walk writes every text byte.  The symbol of a row comes from
//          the bucket its LF value falls in, so a step reads one word.
//
// Neighbouring rows with the same symbol have neighbouring LF rows, and in a
// repetitive text they stay together for as long as the copies agree.  A warp
// walks from the 32 rows of one block, so its lanes read the same few sectors
// and mostly arrive together; rulers chosen row by row gave a warp 32 stretches
// of different lengths, and a sector per lane and step.
//
// The hash is a permutation of [0, 2^kb), 2^kb the power of two at or above the
// number of blocks, so a block's number is its hash over the rate and its place
// the inverse hash of that: no list of rulers, no search in it.  The chain is
// ranked through one ruler in 8 or 16 (the carriers): sequential hops between
// those, pointer jumping over them, and the hops again.  Which one is hashed too:
// between the copies of an exactly repeated text a walk keeps its row modulo the
// number of copies, and with the first of every 16 rulers as carrier one thread
// hopped over the chain of whole copies (16 copies: 8 MiB took 149 ms, now 16 MiB
// take 0.56 ms).
//
// 128 MiB of DNA copies, before / after on GB300, one row in 64 a ruler: LF 1.37 / 0.31
// ms, first walk 2.22 / 1.25, list ranking 1.11 / 0.18, second walk 3.46 / 1.75, in
// all 9.1 / 3.6 ms; one in 16, 32, 64, 128: 3.0, 3.0, 3.5, 4.3 ms (512 MiB: 12.2,
// 10.6, 10.7, 12.5; 64 MiB of random DNA: 3.0, 3.3, 3.7, 4.9, before 4.7 at best).
//
// In a long run of one symbol, and where the text repeats a short period, LF
// leads from row to row of one block: 31 of its 32 rulers end at the next row and
// the last one walks alone through all blocks up to the next ruler block.
// Stretches of 1024 rows and more of long runs therefore mark one target row in 32
// to 256 as a ruler of its own (numbers from `slots` on, rows in a list).  16 MiB of
// one symbol 2.36 -> 0.53 ms, of period 7 2.26 -> 0.56, half of it zeros 2.02 -> 0.65
// (with rulers row by row 1.10, 1.17, 1.27); 200 KB of each 0.34, 0.26, 0.39 -> 0.18, 0.18,
// 0.23 (0.22, 0.21, 0.23); 128 MiB of one symbol 13.1 -> 2.7 ms (5.6).  Fewer listed
// rows (an eighth of the rulers' density) than fit such texts best: a text of
// thousands of copies has such stretches too and its blocks walk well (Fibonacci
// word of 128 MiB 2.6 -> 3.2 ms, with four times as many 3.5).  DNA has none.
//
// LF is a permutation, so a walk ends at the latest at its own ruler; the input
// is a BWT exactly when the cycle of row 0 has all n + 1 rows.
#include "prims.cuh"

namespace gbwt {

constexpr uint32_t UB_RULER = 0x80000000u;
constexpr uint32_t UB_NIL = 0xFFFFFFFFu;
constexpr int UB_EXTRA_LOG2 = 3;          // one listed ruler in 2^(rate_log2 + UB_EXTRA_LOG2) rows of such a tile
constexpr int UB_LUT_LOG2 = 12;

// Permutation of [0, 2^kb): xor-shifts by at least half the bits undo
// themselves, odd factors have inverses modulo 2^32 (these two: any with mixed bits
// do).
constexpr uint32_t UB_MUL1 = 0x2C1B3C6Du, UB_MUL2 = 0x297A2D39u;
constexpr uint32_t ub_inverse(uint32_t a)
{
    uint32_t x = a;                        // correct to 3 bits; each step doubles them
    for (int i = 0; i < 5; i++) x *= 2u - a * x;
    return x;
}
constexpr uint32_t UB_INV1 = ub_inverse(UB_MUL1), UB_INV2 = ub_inverse(UB_MUL2);
static_assert(UB_MUL1 * UB_INV1 == 1u && UB_MUL2 * UB_INV2 == 1u, "inverses modulo 2^32");
struct UbHash {
    uint32_t mask;       // 2^kb - 1
    int half;            // ceil(kb / 2)
    int rate_log2;
    uint32_t rows;
    __device__ __forceinline__ uint32_t mix(uint32_t x) const
    {
        x ^= x >> half;
        x = (x * UB_MUL1) & mask;
        x ^= x >> half;
        x = (x * UB_MUL2) & mask;
        return x ^ (x >> half);
    }
    __device__ __forceinline__ uint32_t unmix(uint32_t x) const
    {
        x ^= x >> half;
        x = (x * UB_INV2) & mask;
        x ^= x >> half;
        x = (x * UB_INV1) & mask;
        return x ^ (x >> half);
    }
    // LF entry for target row t: t, or its ruler number with bit 31
    __device__ __forceinline__ uint32_t entry(uint32_t t) const
    {
        const uint32_t h = mix(t >> 5);
        return (h & ((1u << rate_log2) - 1u)) ? t : (UB_RULER | ((h >> rate_log2) << 5) | (t & 31u));
    }
    __device__ __forceinline__ uint32_t row_of(uint32_t ruler) const
    {
        return (unmix((ruler >> 5) << rate_log2) << 5) | (ruler & 31u);
    }
};

// All rulers: `slots` numbers of blocks, then the listed rows.
struct UbRulers {
    UbHash hash;
    uint32_t slots;
    uint32_t *extra;             // rows of the listed rulers
    uint32_t *extra_n;           // their number, at most extra_cap
    uint32_t extra_cap, extra_mask;
    int super_log2;              // one ruler in 2^super_log2 carries the list ranking
    __device__ __forceinline__ uint32_t count() const { return slots + min(*extra_n, extra_cap); }
    __device__ __forceinline__ uint32_t row_of(uint32_t j) const { return j < slots ? hash.row_of(j) : extra[j - slots]; }
    // The ruler of the s-th group that carries the list ranking; ruler 0 for s = 0.
    // The groups of a block pick alike: walks that keep their row modulo the
    // group's size move and stop together.
    __device__ __forceinline__ uint32_t carrier(uint32_t s) const
    {
        return (s << super_log2) | (((s >> (5 - super_log2)) * 0x9E3779B1u) >> (32 - super_log2));
    }
    __device__ __forceinline__ bool carries(uint32_t j) const { return j == carrier(j >> super_log2); }
};

// Where the input's elements belong.  PFP: element e is row e + 1, except
// element p, whose symbol is row 0's (its place is the '$' row).  libcubwt:
// element e is row e before the '$' row, e + 1 from there on.
struct UbIn {
    const uint8_t *L;
    uint32_t n;
    uint32_t dollar;     // '$' row
    uint32_t p;          // PFP: element of row 0; libcubwt: none (UB_NIL)
    __device__ __forceinline__ uint32_t row(uint32_t e) const { return p != UB_NIL ? e + 1u : (e < dollar ? e : e + 1u); }
};

// Symbol counts of every tile (element p left out), digit-major over the tiles; and
// for each of its eight parts (512 elements, 16 a thread) whether it holds long
// runs: at most one thread of the part's warp sees a change of symbol.
__global__ void __launch_bounds__(RS_THREADS) k_byte_hist(UbIn in, uint32_t *__restrict__ tile_hist, uint32_t num_tiles,
                                                          uint8_t *__restrict__ long_runs)
{
    constexpr int D = 256;
    __shared__ uint32_t h[RS_WARPS * D];       // one histogram per warp
    for (int d = threadIdx.x; d < RS_WARPS * D; d += RS_THREADS) h[d] = 0;
    __syncthreads();
    uint32_t *wh = h + (threadIdx.x >> 5) * D;
    const size_t base = (size_t)blockIdx.x * RS_TILE;
    bool change = false;
    if (base + RS_TILE <= in.n && (((uintptr_t)in.L) & 15u) == 0) {
        const uint4 v = __ldg((const uint4 *)(in.L + base) + threadIdx.x);       // 16 symbols per thread
        uint8_t kk[16];
        memcpy(kk, &v, 16);
#pragma unroll
        for (int q = 0; q < 16; q++) atomicAdd(&wh[kk[q]], 1u);
        change = v.x != __byte_perm(v.x, 0u, 0u) || v.x != v.y || v.x != v.z || v.x != v.w;
    } else {
        const size_t i0 = base + (size_t)threadIdx.x * RS_ITEMS;
        uint8_t first = i0 < in.n ? in.L[i0] : 0;
#pragma unroll 4
        for (int j = 0; j < RS_ITEMS; j++)
            if (i0 + j < in.n) {
                const uint8_t c = in.L[i0 + j];
                atomicAdd(&wh[c], 1u);
                change |= c != first;
            }
    }
    static_assert(RS_ITEMS == 16 && RS_WARPS == 8, "a part is a warp's 16 symbols a thread, a tile has eight");
    const bool runs = __popc(__ballot_sync(0xFFFFFFFFu, change)) <= 1;
    if ((threadIdx.x & 31u) == 0) long_runs[(size_t)blockIdx.x * RS_WARPS + (threadIdx.x >> 5)] = runs;
    __syncthreads();
    for (int d = threadIdx.x; d < D; d += RS_THREADS) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) sum += h[w * D + d];
        if (in.p != UB_NIL && in.p >= base && in.p < base + RS_TILE && in.L[in.p] == d) sum--;
        tile_hist[(size_t)d * num_tiles + blockIdx.x] = sum;
    }
}

// LF of every row (entries as UbHash::entry).  Row 0 precedes all rows of its
// symbol c0 in the sort: with PFP input its element is left out of the counts
// and every other position at or above c0's bucket moves up by one.
__global__ void __launch_bounds__(RS_THREADS) k_lf_rank(UbIn in, const uint32_t *tile_off, uint32_t num_tiles,
                                                        UbHash hash, uint32_t *__restrict__ LF, uint32_t *flags)
{
    constexpr int D = 256;
    __shared__ uint32_t s_wh[RS_WARPS * D];
    __shared__ uint32_t s_goff[D];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = threadIdx.x; q < RS_WARPS * D; q += RS_THREADS) s_wh[q] = 0;
    __syncthreads();
    const uint32_t c0 = in.p != UB_NIL ? in.L[in.p] : 256u;
    const size_t tile_base = (size_t)blockIdx.x * RS_TILE;
    const size_t wbase = tile_base + (size_t)warp * (RS_ITEMS * 32);
    uint32_t dg[RS_ITEMS], rk[RS_ITEMS];
    uint32_t *wh = s_wh + warp * D;
#pragma unroll
    for (int q = 0; q < RS_ITEMS; q++) {
        const size_t idx = wbase + (size_t)q * 32 + lane;
        dg[q] = idx < in.n && idx != in.p ? (uint32_t)in.L[idx] : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int q = 0; q < RS_ITEMS; q++) {
        // the lowest lane of each digit class reads and advances the warp's
        // counter; the others take the old value from it
        const uint32_t d = dg[q];
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
        const unsigned leader = (unsigned)(__ffs(peers) - 1);
        uint32_t prior = 0;
        if (lane == leader && d != 0xFFFFFFFFu) {
            prior = wh[d];
            wh[d] = prior + (uint32_t)__popc(peers);
        }
        prior = __shfl_sync(0xFFFFFFFFu, prior, leader);
        rk[q] = prior + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over the warps, and the tile's global offset
    {
        const uint32_t d = threadIdx.x;
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) {
            const uint32_t c = s_wh[w * D + d];
            s_wh[w * D + d] = run;
            run += c;
        }
        const uint32_t off = lb_load32(tile_off + (size_t)d * num_tiles + blockIdx.x);
        s_goff[d] = rs_checked(1u + off + (c0 <= d ? 1u : 0u), run, hash.rows, flags);     // the walks stay in the table
        // row 0 (PFP) and the '$' row, by the first tile
        if (blockIdx.x == 0 && d == c0) LF[0] = hash.entry(rs_checked(1u + off, 1u, hash.rows, flags));
        if (blockIdx.x == 0 && d == 0) LF[in.dollar] = UB_RULER;      // row 0 is ruler 0
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < RS_ITEMS; q++) {
        const uint32_t d = dg[q];
        if (d == 0xFFFFFFFFu) continue;
        LF[in.row((uint32_t)(wbase + (size_t)q * 32 + lane))] = hash.entry(s_goff[d] + s_wh[warp * D + d] + rk[q]);
    }
}

// Listed rulers: in parts of long runs every target row that is a multiple of
// 2^extra_log2, numbered with one atomic per tile.  A CTA looks at up to UB_XTILES
// tiles, one where there are few (a tile of long runs takes 4.5 us: 800 KB of one
// byte 36 us with eight tiles a CTA, 7 with one; 128 MiB of DNA 5 us with eight, 8 with
// four).
constexpr uint32_t UB_XTILES = 8;
//
// The first CTA also writes the cumulative symbol counts of all non-'$' rows from
// the scanned tile histograms (row 0's symbol added back for PFP input).
__global__ void __launch_bounds__(RS_THREADS) k_lf_extra(UbIn in, const uint64_t *__restrict__ long_runs,
                                                         uint32_t num_tiles, uint32_t per_cta, UbRulers ru, uint32_t *LF,
                                                         const uint32_t *tile_off, uint32_t *cum)
{
    __shared__ uint32_t s_warp[32], s_first;
    if (blockIdx.x == 0) {
        const uint32_t c = threadIdx.x, c0 = in.p != UB_NIL ? in.L[in.p] : 256u;
        cum[c] = tile_off[(size_t)c * num_tiles] + (c0 < c ? 1u : 0u);
        if (c == 0) cum[256] = in.n;
    }
    const uint32_t b0 = blockIdx.x * per_cta, b1 = min(b0 + per_cta, num_tiles);
    const bool set = threadIdx.x < b1 - b0 && long_runs[b0 + threadIdx.x];
    if (!__syncthreads_or(set)) return;
    for (uint32_t b = b0; b < b1; b++) {
        // a byte each; two neighbours at least (a single one comes up by chance: 64
        // copies that agree on the symbol before eight contexts in a row)
        uint64_t parts = long_runs[b];
        parts &= (parts >> 8) | (parts << 8);
        if (!parts) continue;
        uint32_t mine = 0, total;
#pragma unroll
        for (int q = 0; q < RS_ITEMS; q++) {
            const uint32_t i = q * RS_THREADS + threadIdx.x, e = b * RS_TILE + i;
            if (e >= in.n || e == in.p || !((parts >> (8u * (i / (32 * RS_ITEMS)))) & 1u)) continue;
            const uint32_t v = LF[in.row(e)];
            if (!(v & (UB_RULER | ru.extra_mask))) mine |= 1u << q;
        }
        uint32_t j = block_excl_scan<uint32_t, OpAdd>((uint32_t)__popc(mine), total, OpAdd(), s_warp);
        if (threadIdx.x == 0) s_first = atomicAdd(ru.extra_n, total);
        __syncthreads();
        j += s_first;
        for (uint32_t m = mine; m && j < ru.extra_cap; m &= m - 1u, j++) {
            const uint32_t r = in.row(b * RS_TILE + (uint32_t)(__ffs(m) - 1) * RS_THREADS + threadIdx.x);
            ru.extra[j] = LF[r];
            LF[r] = UB_RULER | (ru.slots + j);
        }
        __syncthreads();
    }
}

// First walk: the next ruler and the distance to it.  A warp takes block after
// block of 32 ruler rows.
__global__ void k_walk_count(const uint32_t *__restrict__ LF, UbRulers ru, uint32_t *succ, uint32_t *wt)
{
    const uint32_t step = gridDim.x * blockDim.x, count = ru.count(), rows = ru.hash.rows;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += step) {
        uint32_t r = ru.row_of(j), steps = 0, v = UB_NIL;
        if (r < rows) {               // else a hash value past the rows: no ruler
            do {
                v = __ldg(LF + r);
                r = v;
                steps++;
            } while (!(v & UB_RULER) && steps <= rows);
            v &= ~UB_RULER;
        }
        succ[j] = v;
        wt[j] = steps;
    }
}

// Hops between carriers: the next one and the distance.  The one whose next is
// ruler 0 ends the chain.
__global__ void k_super_hops(const uint32_t *succ, const uint32_t *wt, UbRulers ru, uint32_t supers, uint32_t *ssucc,
                             uint32_t *swt)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x, slots = ru.count();
    if (s >= supers) return;           // from an upper bound of the rulers: the last ones may not be there
    uint32_t j = ru.carrier(s), acc = 0, hops = 0;
    if (j >= slots || ru.row_of(j) >= ru.hash.rows) {
        ssucc[s] = UB_NIL;
        swt[s] = 0;
        return;
    }
    do {
        acc += wt[j];
        j = succ[j];
    } while (j < slots && !ru.carries(j) && ++hops < slots);
    ssucc[s] = j == 0 || j >= slots ? UB_NIL : j >> ru.super_log2;
    swt[s] = acc;
}

// Pointer jumping: after r rounds wt[s] is the distance over the next 2^r
// carriers (or to the chain's end).  Double-buffered.
__global__ void k_jump(const uint32_t *succ, const uint32_t *wt, uint32_t m, uint32_t *succ2, uint32_t *wt2)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= m) return;
    const uint32_t t = succ[s];
    succ2[s] = t == UB_NIL ? UB_NIL : succ[t];
    wt2[s] = wt[s] + (t == UB_NIL ? 0u : wt[t]);
}

// Distances from row 0 for every ruler: the hops again, from rows - (distance
// of the carrier to the end).
__global__ void k_ruler_off(const uint32_t *succ, const uint32_t *wt, UbRulers ru, const uint32_t *sdist, uint32_t *off)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x, slots = ru.count();
    uint32_t j = ru.carrier(s), hops = 0;
    if (j >= slots || ru.row_of(j) >= ru.hash.rows) return;
    uint32_t o = ru.hash.rows - sdist[s];
    do {
        off[j] = o;
        o += wt[j];
        j = succ[j];
    } while (j < slots && !ru.carries(j) && ++hops < slots);
}

// Second walk: every ruler writes the text bytes of its stretch, from high to
// low addresses, gathered into 8-byte words.  sym(row) is the bucket of
// LF(row) - 1 among the cumulative counts cum[0..256]: a table over the value's
// high bits gives the first candidate.  LISTED: there are listed rulers (a look at
// the list in the loop takes 2 % of texts that have none).
template <bool LISTED>
__device__ __forceinline__ void emit_stretches(const uint32_t *__restrict__ LF, const UbRulers &ru, const uint32_t *off,
                                               const uint32_t *s_cum, const uint8_t *s_lut, int lut_shift, uint32_t n,
                                               uint8_t *T)
{
    const uint32_t step = gridDim.x * blockDim.x, count = LISTED ? ru.count() : ru.slots;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += step) {
        uint32_t r = LISTED ? ru.row_of(j) : ru.hash.row_of(j);
        if (r >= ru.hash.rows) continue;
        uint32_t k = off[j], in_word = 0;    // bytes gathered in `word`
        uint64_t word = 0;
        for (bool last = false; !last; k++) {
            const uint32_t v = __ldg(LF + r);
            last = (v & UB_RULER) != 0;
            r = !last ? v : LISTED ? ru.row_of(v & ~UB_RULER) : ru.hash.row_of(v & ~UB_RULER);
            if (k >= n || r == 0) break;     // the '$' row: the stretch ends here
            uint32_t c = s_lut[(r - 1u) >> lut_shift];
            while (s_cum[c + 1] <= r - 1u) c++;
            uint8_t *p = T + (n - 1u - k);
            word = (word << 8) | c;          // bytes come from high to low addresses
            in_word++;
            if (last || ((uintptr_t)p & 7u) == 0) {
                if (in_word == 8u) *(uint64_t *)p = word;
                else for (uint32_t q = 0; q < in_word; q++) p[q] = (uint8_t)(word >> (8u * q));
                in_word = 0;
                word = 0;
            }
        }
        // bytes before the '$' row: the lowest is T[0]
        for (uint32_t q = 0; q < in_word; q++) T[q] = (uint8_t)(word >> (8u * q));
    }
}
__global__ void __launch_bounds__(256) k_walk_emit(const uint32_t *__restrict__ LF, UbRulers ru, const uint32_t *off,
                                                   const uint32_t *cum, int lut_shift, uint32_t n, uint8_t *T)
{
    __shared__ uint32_t s_cum[257];
    __shared__ uint8_t s_lut[1 << UB_LUT_LOG2];
    for (int c = threadIdx.x; c < 257; c += blockDim.x) s_cum[c] = cum[c];
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < (1u << UB_LUT_LOG2); q += blockDim.x) {
        const uint64_t first = (uint64_t)q << lut_shift;
        uint32_t lo = 0, hi = 255;           // last c with cum[c] <= first
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1u) >> 1;
            if (s_cum[mid] <= first) lo = mid; else hi = mid - 1u;
        }
        s_lut[q] = (uint8_t)lo;
    }
    __syncthreads();
    if (*ru.extra_n) emit_stretches<true>(LF, ru, off, s_cum, s_lut, lut_shift, n, T);
    else emit_stretches<false>(LF, ru, off, s_cum, s_lut, lut_shift, n, T);
}

// Inverse of the PFP output (p: its primary row, i unused) or of libcubwt's L
// (p = 0xFFFFFFFF, i its primary index in [1, n]).
void run_unbwt(Storage *st, const uint8_t *dL, uint32_t n, uint32_t i, uint32_t p, uint8_t *dT)
{
    const uint32_t rows = n + 1u;
    UbIn in{dL, n, p != UB_NIL ? p + 1u : i, p};
    // ~1/32 of the rows are rulers (tuning knob); small inputs use denser ones
    const uint32_t rate_max = 1u << tune_unbwt_rate_log2(st);
    uint32_t rate = 4;
    while (rate < rate_max && (uint64_t)rate * 65536u < rows) rate <<= 1;
    const int kb = bits_for((rows - 1u) >> 5);
    UbHash hash;
    hash.mask = (uint32_t)((1ull << kb) - 1ull);
    hash.half = (kb + 1) / 2;
    hash.rate_log2 = 0;
    while ((1u << hash.rate_log2) < rate && hash.rate_log2 < kb) hash.rate_log2++;
    hash.rows = rows;
    const uint32_t slots = (uint32_t)((1ull << kb) >> hash.rate_log2) << 5;
    const int extra_log2 = hash.rate_log2 + UB_EXTRA_LOG2;
    const uint32_t extra_cap = (rows >> extra_log2) + 1u, rulers = slots + extra_cap;       // upper bounds
    // 1 MiB of mutated copies 281 us with one in 16, 259 with one in 8 (shorter
    // hops), 3 MB 300 and 280; 22 MiB of versions 703 and 727, 128 MiB of DNA 3.26 and 3.28 ms
    // (one round of pointer jumping more, over twice the carriers)
    const int super_log2 = rows < (1u << 23) ? 3 : 4;
    const uint32_t supers = (rulers + (1u << super_log2) - 1u) >> super_log2;
    UbRulers ru{hash, slots, slot<uint32_t>(st, S_ACTX, extra_cap), st->d_flags + 56, extra_cap, (1u << extra_log2) - 1u,
                super_log2};
    // LF
    const uint32_t num_tiles = (uint32_t)(((size_t)n + RS_TILE - 1) / RS_TILE);
    uint32_t *hist = slot<uint32_t>(st, S_RSHIST, (size_t)256 * num_tiles);
    uint64_t *long_runs = slot<uint64_t>(st, S_ACTG, num_tiles);
    k_byte_hist<<<num_tiles, RS_THREADS, 0, st->stream>>>(in, hist, num_tiles, (uint8_t *)long_runs);
    after_launch(st);
    device_scan<uint32_t, OpAdd>(st, (size_t)256 * num_tiles, LoadArr<uint32_t>{hist}, StoreArr<uint32_t>{hist}, false,
                                 (uint32_t *)nullptr);
    uint32_t *LF = slot<uint32_t>(st, S_ISA, rows);
    k_lf_rank<<<num_tiles, RS_THREADS, 0, st->stream>>>(in, hist, num_tiles, hash, LF, st->d_flags);
    after_launch(st);
    uint32_t *cum = slot<uint32_t>(st, S_TMP2, 257);
    uint32_t xtiles = num_tiles / ((uint32_t)st->num_sms * 8u);
    xtiles = xtiles < 1u ? 1u : xtiles < UB_XTILES ? xtiles : UB_XTILES;
    k_lf_extra<<<grid_for(num_tiles, xtiles), RS_THREADS, 0, st->stream>>>(in, long_runs, num_tiles, xtiles, ru, LF,
                                                                               hist, cum);
    after_launch(st);
    // walk 1 and list ranking of the ruler chain
    uint32_t *succ = slot<uint32_t>(st, S_TMP0, rulers), *wt = slot<uint32_t>(st, S_TMP1, rulers);
    unsigned grid = grid_for(rulers, 256);
    const unsigned full = (unsigned)st->num_sms * 8u;          // 2048 threads per SM
    if (grid > full) grid = full;
    k_walk_count<<<grid, 256, 0, st->stream>>>(LF, ru, succ, wt);
    after_launch(st);
    uint32_t *ssucc = slot<uint32_t>(st, S_VAL0, supers), *ssucc2 = slot<uint32_t>(st, S_VAL1, supers);
    uint32_t *swt = slot<uint32_t>(st, S_KEY0, supers), *swt2 = slot<uint32_t>(st, S_KEY1, supers);
    k_super_hops<<<grid_for(supers, 128), 128, 0, st->stream>>>(succ, wt, ru, supers, ssucc, swt);
    after_launch(st);
    const int rounds = bits_for(supers);
    for (int r = 0; r < rounds; r++) {
        k_jump<<<grid_for(supers, 256), 256, 0, st->stream>>>(ssucc, swt, supers, ssucc2, swt2);
        after_launch(st);
        uint32_t *ts = ssucc; ssucc = ssucc2; ssucc2 = ts;
        uint32_t *tw = swt; swt = swt2; swt2 = tw;
    }
    // from ruler 0 the cycle must come back to row 0 after n+1 steps, its list closed
    check_cuda(cudaMemcpyAsync(st->h_scalars + 1, ssucc, 4, cudaMemcpyDeviceToHost, st->stream));
    check_cuda(cudaMemcpyAsync(st->h_scalars + 2, swt, 4, cudaMemcpyDeviceToHost, st->stream));
    sync_stream(st);
    if ((uint32_t)st->h_scalars[1] != UB_NIL || (uint32_t)st->h_scalars[2] != rows) throw Error{GBWT_BAD_PARAMETER};
    uint32_t *off = slot<uint32_t>(st, S_SA, rulers);
    k_ruler_off<<<grid_for(supers, 128), 128, 0, st->stream>>>(succ, wt, ru, swt, off);
    after_launch(st);
    const int lut_shift = kb + 5 > UB_LUT_LOG2 ? kb + 5 - UB_LUT_LOG2 : 0;
    k_walk_emit<<<grid, 256, 0, st->stream>>>(LF, ru, off, cum, lut_shift, n, dT);
    after_launch(st);
}

}  // namespace gbwt
