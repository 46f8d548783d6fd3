// pfp_phrases.cu -- phrase fingerprints, exact deduplication and the
// dictionary buffer (sm_103a).
//
// The reference gives equal phrases equal ids by sorting all z occurrences
// lexicographically and pointer-jumping over equal neighbours
// (Prefix_Free_Parsing_W=5_P=16_kommentiert.cu, "K", K:1990-2164 and
// K:616-691).  Here equal phrases are found without sorting: every
// occurrence is fingerprinted (polynomial hash mod 2^61-1 over a CTA-staged
// text window), inserted into an open-addressing table sized to stay in L2
// when the dictionary is small, and then compared byte for byte with its
// table representative (the occurrence that inserted the key), so ids are
// exact.  A fingerprint collision or table overflow is detected on the
// device and the stage is re-run with a new seed or a larger table.  Which
// occurrence wins an insert varies from run to run, so internal ids may too;
// nothing downstream depends on them (phrase order comes from the
// dictionary sort), and every output is deterministic.
#include "prims.cuh"

namespace gbwt {

constexpr int PH_THREADS = 256;
constexpr int PH_SPAN = 24576;
// More probes mean a table too full to go on.  Linear probing up to the limit of
// 0.75 of the slots takes at most 160 to 240 for tables of 2^20 to 2^24 slots (random
// keys, four runs each); the full-size table is at most half full and gets room
// to spare, since nothing larger follows it.  When a small table overflows, every
// thread in flight runs into the dense rest of it before the first CTA reports its
// count: 102 MB of versions, first attempt 703 -> 329 us with 2048 -> 256.
constexpr uint32_t PH_PROBES = 2048, PH_PROBES_SMALL = 256;

// Phrase k spans [start, end]: end = D[k]; start = D[k-1]-W+1 (consecutive
// phrases overlap by W, K:578-592).  In a batch of texts (xsep = the padded
// buffer, see pfp_batch.cu) a phrase whose predecessor ended on a sentinel byte
// is the first phrase of the next text and starts right after it.
__device__ __forceinline__ void phrase_span(const uint32_t *D, uint32_t k, int W, const uint8_t *xsep,
                                            uint32_t &start, uint32_t &end)
{
    end = D[k];
    if (!k) { start = 0; return; }
    const uint32_t p = D[k - 1];
    start = (xsep && xsep[p] == 1) ? p + 1u : p - (uint32_t)W + 1u;
}

// What keeping a batch's texts apart would cost: bytes of the distinct phrases
// and of the distinct (text, phrase) pairs, and whether the count of pairs was
// given up.  The texts are kept apart when that adds at most a quarter to the
// dictionary.
struct Parting {
    unsigned long long bytes, pair_bytes;
    uint32_t full, pad;
};
__host__ __device__ __forceinline__ bool part_texts(const Parting &p)
{
    return !p.full && p.pair_bytes * 4ull <= p.bytes * 5ull;
}
// Sum of v over the CTA, to one thread (the others 0); all threads take part.
__device__ __forceinline__ uint32_t block_sum(uint32_t v)
{
    __shared__ uint32_t s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    const uint32_t w = __reduce_add_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31u) == 0 && w) atomicAdd(&s_sum, w);
    __syncthreads();
    return threadIdx.x == 0 ? s_sum : 0u;
}

struct HashArgs {
    const uint8_t *T;
    uint32_t n;
    const uint32_t *D;
    uint32_t z;
    int W;
    uint64_t base;          // polynomial base, < 2^61
    unsigned long long *tkeys;
    uint32_t *tvals;
    uint32_t cmask;
    int logc;
    uint32_t limit;         // distinct keys allowed before ERR_TABLE_FULL
    uint32_t *slot_of;
    uint32_t *flags;
    const uint8_t *xsep;    // batch: padded text buffer, else null
    uint32_t probes;        // longest run
    uint32_t *full;         // set with ERR_TABLE_FULL: away from the counters that every insert updates
    unsigned long long *bytes;      // PART: sum of the distinct phrases' lengths
};

// Fingerprint of phrase k and its table slot.
__device__ __forceinline__ void phrase_insert(const HashArgs &a, uint32_t k, const uint8_t *s_txt, uint32_t a_al,
                                              bool staged, uint32_t &fresh)
{
    uint32_t start, end;
    phrase_span(a.D, k, a.W, a.xsep, start, end);
    const uint32_t len = end - start + 1u;
    // polynomial mod 2^61-1 over little-endian 7-byte chunks (56 bits, below
    // the modulus; the last one zero-padded)
    uint64_t h = 0;
    if (staged) {
        const uint32_t *w = (const uint32_t *)s_txt;
        for (uint32_t i = 0; i < len; i += 7) {
            const uint32_t p = start - a_al + i, q = p >> 2, sh = (p & 3u) * 8u;
            const uint32_t lo = __funnelshift_r(w[q], w[q + 1], sh), hi = __funnelshift_r(w[q + 1], w[q + 2], sh);
            uint64_t chunk = (((uint64_t)hi << 32) | lo) & 0x00FFFFFFFFFFFFFFull;
            if (len - i < 7) chunk &= (1ull << (8u * (len - i))) - 1ull;
            h = mulmod61(h, a.base) + chunk + 1u;
            if (h >= M61) h -= M61;
        }
    } else {
        // one thread reads the phrase, however long: the bytes of a chunk are loaded
        // together (2 MiB without a trigger: the call 155 -> 126 ms)
        for (uint32_t i = 0; i < len; i += 7) {
            uint64_t chunk = 0;
#pragma unroll
            for (uint32_t b = 0; b < 7; b++)
                chunk |= (uint64_t)(i + b < len ? text_at(a.T, a.n, start + i + b) : 0) << (8 * b);
            h = mulmod61(h, a.base) + chunk + 1u;
            if (h >= M61) h -= M61;
        }
    }
    uint64_t key = h ^ ((uint64_t)len * 0x9E3779B97F4A7C15ull);
    if (key == 0) key = 1;
    uint32_t pos = (uint32_t)((key * 0xD6E8FEB86659FD93ull) >> (64 - a.logc));
    bool ok = false;
    for (uint32_t probe = 0; probe <= a.cmask; probe++) {
        // a plain read first: in a repetitive text most occurrences find
        // their key already in place, and a load costs L2 less than a CAS
        // (keys are never removed, so a key seen once stays)
        unsigned long long cur = __ldcg(a.tkeys + pos);
        if (cur == 0ull) cur = atomicCAS(a.tkeys + pos, 0ull, (unsigned long long)key);
        if (cur == 0ull) {
            // the inserting occurrence is the slot's representative
            a.tvals[pos] = k;
            fresh = len;
            ok = true;
            break;
        }
        if (cur == key) { ok = true; break; }
        pos = (pos + 1u) & a.cmask;
        if (probe >= a.probes || ((probe & 7u) == 7u && *(volatile uint32_t *)a.full)) break;
    }
    if (!ok) {
        atomicOr(a.flags, ERR_TABLE_FULL);
        *a.full = 1u;
        a.slot_of[k] = 0;
        return;
    }
    a.slot_of[k] = pos;
}

// PART: a batch that may be kept apart by text; its distinct bytes are summed.
template <bool PART>
__global__ void __launch_bounds__(PH_THREADS) k_phrase_hash(HashArgs a)
{
    __shared__ __align__(16) uint8_t s_txt[PH_SPAN];
    __shared__ bool s_full;         // the table is full: the stage is run again with a larger one
    uint32_t flag0 = 0;             // loaded beside the text, kept for the barrier
    if (threadIdx.x == 0) flag0 = *(volatile uint32_t *)a.full;
    const uint32_t k0 = blockIdx.x * PH_THREADS;
    const uint32_t klast = min(k0 + PH_THREADS - 1u, a.z - 1u);
    const uint32_t sa = k0 ? a.D[k0 - 1] - (uint32_t)a.W + 1u : 0u;
    const uint32_t sb = a.D[klast];
    const uint32_t a_al = sa & ~15u;
    // +32: the word reads of the last chunk may touch 12 bytes past the span
    const bool staged = (size_t)(sb - a_al) + 32 <= PH_SPAN;
    if (staged) {
        const bool aligned = (((uintptr_t)a.T) & 15u) == 0;
        const uint32_t nvec = (sb - a_al) / 16 + 1;
        for (uint32_t v = threadIdx.x; v < nvec; v += PH_THREADS) {
            uint32_t p = a_al + v * 16;
            uint4 val;
            if (aligned && (size_t)p + 16 <= a.n) {
                val = __ldg((const uint4 *)(a.T + p));
            } else {
                uint8_t b[16];
#pragma unroll
                for (int j = 0; j < 16; j++) b[j] = text_at(a.T, a.n, p + j);
                memcpy(&val, b, 16);
            }
            *(uint4 *)(s_txt + v * 16) = val;
        }
    }
    if (threadIdx.x == 0) s_full = flag0 != 0;
    __syncthreads();
    const uint32_t k = k0 + threadIdx.x;
    uint32_t fresh = 0;             // length of a phrase first seen here
    if (k < a.z && !s_full) phrase_insert(a, k, s_txt, a_al, staged, fresh);
    // the inserts of a CTA are counted together: one atomic on the counter
    const uint32_t count = (uint32_t)__syncthreads_count(fresh != 0u);
    if (threadIdx.x == 0 && count && atomicAdd(a.flags + 1, count) + count > a.limit) {
        atomicOr(a.flags, ERR_TABLE_FULL);
        *a.full = 1u;
    }
    if constexpr (PART) {
        const uint32_t sum = block_sum(fresh);
        if (sum) atomicAdd(a.bytes, (unsigned long long)sum);
    }
}
// The distinct (text, content slot) pairs, exact keys: a pair's slot per phrase.
// A kernel of its own: inside the fingerprint kernel, which lives on shared
// memory, the second chain of random reads took 3.0 ms of a 4096-text batch,
// here 0.75 ms.  Sums go through one atomic per CTA (one per insert: 1.6 ms more).
constexpr uint32_t PAIR_PROBES = 128;      // a longer run means a table too full to go on
__global__ void k_pairs(const uint32_t *D, uint32_t z, int W, const uint8_t *xsep, const uint32_t *ptid,
                        const uint32_t *slot_of, const uint32_t *flags,
                        unsigned long long *pkeys, uint32_t *pvals, uint32_t pmask, uint32_t *pslot, Parting *part)
{
    __shared__ bool s_stop;
    if (threadIdx.x == 0) s_stop = (*flags & ERR_TABLE_FULL) || *(volatile uint32_t *)&part->full;
    __syncthreads();
    if (s_stop) return;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t fresh = 0;
    if (k < z) {
        const unsigned long long pair = ((unsigned long long)(ptid[k] + 1u) << 32) | slot_of[k];
        uint32_t q = (uint32_t)((pair * 0x9E3779B97F4A7C15ull) >> 32) & pmask;
        for (uint32_t probe = 0;; probe++, q = (q + 1u) & pmask) {
            unsigned long long cur = __ldcg(pkeys + q);
            if (cur == 0ull) cur = atomicCAS(pkeys + q, 0ull, pair);
            if (cur == 0ull) {
                pvals[q] = k;
                uint32_t s, e;
                phrase_span(D, k, W, xsep, s, e);
                fresh = e - s + 1u;
                break;
            }
            if (cur == pair) break;
            if (probe >= PAIR_PROBES) {
                part->full = 1u;
                break;
            }
        }
        pslot[k] = q;
    }
    const uint32_t sum = block_sum(fresh);
    // past the line the answer is known, and the CTAs to come need not look
    if (sum && (atomicAdd(&part->pair_bytes, (unsigned long long)sum) + sum) * 4ull > part->bytes * 5ull) part->full = 1u;
}

// 8 text bytes starting at T + p (any alignment): two aligned 8-byte loads
// and a shift.  The caller keeps T + p + 16 inside the buffer.
__device__ __forceinline__ uint64_t load8_any(const uint8_t *T, uint32_t p)
{
    const uintptr_t a = (uintptr_t)(T + p);
    const uint64_t *w = (const uint64_t *)(a & ~(uintptr_t)7);
    const uint32_t sh = (uint32_t)(a & 7u) * 8u;
    const uint64_t lo = __ldg(w), hi = __ldg(w + 1);
    return sh ? (lo >> sh) | (hi << (64u - sh)) : lo;
}

// Compares each occurrence with its representative; marks representatives.
// Where a batch's texts are kept apart, the pairs take the contents' place:
// their representatives and slots.
// Inside the text 8 bytes at a time; the tail and the sentinel run after
// the text byte by byte.
__global__ void k_phrase_verify(const uint8_t *T, uint32_t n, const uint32_t *D, uint32_t z, int W,
                                const uint32_t *tvals, uint32_t *slot_of, uint32_t *isrep, uint32_t *flags,
                                const uint8_t *xsep, const uint32_t *pvals, const uint32_t *pslot, const Parting *part)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= z) return;
    if (*(volatile uint32_t *)flags & ERR_TABLE_FULL) {          // the stage is run again; slots may be missing
        isrep[k] = 0;
        return;
    }
    const uint32_t rep = tvals[slot_of[k]];
    if (part && part_texts(*part)) {
        const uint32_t q = pslot[k];
        isrep[k] = pvals[q] == k;
        slot_of[k] = q;
    } else {
        isrep[k] = rep == k;
    }
    if (rep == k) return;
    if (rep >= z) { atomicOr(flags, ERR_COLLISION); return; }
    uint32_t s1, e1, s2, e2;
    phrase_span(D, k, W, xsep, s1, e1);
    phrase_span(D, rep, W, xsep, s2, e2);
    if (e1 - s1 != e2 - s2) { atomicOr(flags, ERR_COLLISION); return; }
    const uint32_t len = e1 - s1 + 1u;
    const uint32_t hi_start = s1 > s2 ? s1 : s2;
    // words only where both 16-byte load windows stay inside the n text bytes
    // (an 8-byte aligned text: the aligned loads never start before it)
    const uint32_t inside = (((uintptr_t)T & 7u) == 0 && n > hi_start + 16u) ? n - hi_start - 16u : 0u;
    const uint32_t wlen = (len < inside ? len : inside) & ~7u;
    uint32_t i = 0;
    for (; i < wlen; i += 8) {
        if (load8_any(T, s1 + i) != load8_any(T, s2 + i)) { atomicOr(flags, ERR_COLLISION); return; }
    }
    for (; i < len; i++) {
        if (text_at(T, n, s1 + i) != text_at(T, n, s2 + i)) { atomicOr(flags, ERR_COLLISION); return; }
    }
}

// Dense ids in first-occurrence order: id of representative k = prefix.
struct StoreDense {
    const uint32_t *D;
    const uint32_t *slot_of;
    uint32_t *tdense;
    uint32_t *dlen;
    uint32_t *dstart;
    int W;
    const uint8_t *xsep;
    const uint32_t *ptid;
    uint32_t *dtid;
    __device__ __forceinline__ void operator()(size_t k, uint32_t pre, uint32_t v) const
    {
        if (!v) return;
        if (dtid) dtid[pre] = ptid[k];
        uint32_t s, e;
        phrase_span(D, (uint32_t)k, W, xsep, s, e);
        tdense[slot_of[k]] = pre;
        dlen[pre] = e - s + 1u;
        dstart[pre] = s;
    }
};

// pid per occurrence; occurrence counts and the preceding bytes seen (byte c as
// c | (~c << 16), OR-ed) of every distinct phrase.
//
// Two reductions per occurrence: neighbouring occurrences rarely share a phrase,
// and a match per warp costs more than it saves.  Where they do share one, the
// reductions meet at one address, 0.6 ns each.  A warp whose 32 occurrences are of
// one phrase adds once (runs of one byte between others, 16 MiB: the call 20.8 ->
// 15.6 ms).  FEW: at most PH_FEW phrases of hundreds of occurrences each are counted in
// shared memory, a CTA many rows of occurrences: 16 MiB of one byte, the call 59.5 ->
// 36.8 ms (20.8 ms of it were this kernel), 200 texts of random DNA with W = 1, P = 1 (20 M
// occurrences of 20 phrases) 14.0 -> 7.9 ms.
constexpr uint32_t PH_FEW = 2048, PH_FEW_OCC = 256;
template <bool FEW>
__global__ void k_phrase_finalize(const uint8_t *T, uint32_t n, const uint32_t *D, uint32_t z, uint32_t d, int W,
                                  const uint32_t *slot_of, const uint32_t *tdense, uint32_t *pid, uint32_t *pidpc,
                                  uint2 *occpc, const uint8_t *xsep, const uint32_t *ptid, const uint8_t *lastb)
{
    __shared__ uint32_t s_occ[FEW ? PH_FEW : 1], s_seen[FEW ? PH_FEW : 1];
    if constexpr (FEW) {
        for (uint32_t q = threadIdx.x; q < d; q += blockDim.x) s_occ[q] = s_seen[q] = 0;
        __syncthreads();
    }
    // one row of occurrences per CTA, or (FEW) as many as there are
    for (uint32_t k0 = blockIdx.x * blockDim.x; k0 < z; k0 += gridDim.x * blockDim.x) {
        const uint32_t k = k0 + threadIdx.x;
        uint32_t id = 0xFFFFFFFFu, seen = 0;
        if (k < z) {
            id = tdense[slot_of[k]];
            pid[k] = id;
            uint32_t s, e, c;
            phrase_span(D, k, W, xsep, s, e);
            // the first phrase of a text is preceded by the text's last byte
            if (xsep && (k == 0 || xsep[D[k - 1]] == 1)) c = lastb[ptid[k]];
            else c = preceding_byte(T, n, s);
            if (pidpc) pidpc[k] = (id << 8) | c;     // only when ids fit 24 bits
            seen = c | ((c ^ 0xFFu) << 16);
        }
        const bool one = __all_sync(0xFFFFFFFFu, id == __shfl_sync(0xFFFFFFFFu, id, 0));
        if (one) seen = __reduce_or_sync(0xFFFFFFFFu, seen);
        if (k >= z || (one && (threadIdx.x & 31u))) continue;
        if constexpr (FEW) {
            atomicAdd(&s_occ[id], one ? 32u : 1u);
            if (seen & ~*(volatile uint32_t *)&s_seen[id]) atomicOr(&s_seen[id], seen);
        } else {
            atomicAdd(&occpc[id].x, one ? 32u : 1u);
            atomicOr(&occpc[id].y, seen);
        }
    }
    if constexpr (FEW) {
        __syncthreads();
        for (uint32_t q = threadIdx.x; q < d; q += blockDim.x)
            if (s_occ[q]) {
                atomicAdd(&occpc[q].x, s_occ[q]);
                atomicOr(&occpc[q].y, s_seen[q]);
            }
    }
}

struct LoadLen64 {
    const uint32_t *a;
    __device__ __forceinline__ uint64_t operator()(size_t i) const { return a[i]; }
};
struct StoreOff32 {
    uint32_t *a;
    size_t n;                   // a[n] = the total
    __device__ __forceinline__ void operator()(size_t i, uint64_t pre, uint64_t v) const
    {
        a[i] = (uint32_t)pre;
        if (i + 1 == n) a[n] = (uint32_t)(pre + v);
    }
};

// LANES lanes per distinct phrase: copy its bytes and tag positions with the id.
// A warp per phrase leaves most lanes idle on phrases of twenty bytes: eight
// lanes take 102 MB of versions (18 bytes on average) from 447 to 193 us and the
// 512 MiB DNA text (30) from 130 to 75 us.  Phrases of 64 bytes and more on average
// fill two rows of a warp and keep it (W=35: 160 bytes, 130 MB in 270 us).
template <int LANES>
__global__ void k_dict_copy(const uint8_t *T, uint32_t n, uint32_t d, const uint32_t *doff, const uint32_t *dlen,
                            const uint32_t *dstart, uint8_t *dict, uint32_t *dphr)
{
    const uint32_t id = (blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    if (id >= d) return;
    const uint32_t off = doff[id], len = dlen[id], st = dstart[id];
    for (uint32_t j = threadIdx.x % LANES; j < len; j += LANES) {
        dict[off + j] = text_at(T, n, st + j);
        dphr[off + j] = id;
    }
}

static uint32_t pow2_at_least(uint64_t v)
{
    uint64_t c = 1024;
    while (c < v) c <<= 1;
    return (uint32_t)c;
}

void run_phrases(Storage *st, const uint8_t *dT, uint32_t n, int W, Phrases &ph, const BatchText *bt, bool may_part)
{
    const uint32_t *ptid = may_part ? bt->ptid : nullptr;
    uint32_t *dtid = may_part ? slot<uint32_t>(st, S_DTID, ph.z) : nullptr;
    Parting *part = (Parting *)(st->d_scalars + 8);
    static_assert(sizeof(Parting) == 24, "three words of the device scalars");
    const uint8_t *xsep = bt ? dT : nullptr;
    const uint32_t z = ph.z;
    uint32_t *slot_of = slot<uint32_t>(st, S_SLOT, z);
    uint32_t *isrep = slot<uint32_t>(st, S_PID, z);     // reused for pid below
    const uint32_t full_c = pow2_at_least((uint64_t)z * 2);
    const uint32_t cap = 1u << tune_hash_log2(st);       // L2-sized table while the dictionary fits
    uint32_t c = full_c < cap ? full_c : cap;
    uint64_t seed = 0x2545F4914F6CDD1Dull;
    uint32_t d = 0;
    uint32_t *tdense = nullptr, *dlen = nullptr, *dstart = nullptr;
    int attempt = 0;
    for (;; attempt++) {
        if (attempt > 6) throw Error{GBWT_INTERNAL_ERROR};
        unsigned long long *tkeys = slot<unsigned long long>(st, S_TKEYS, c);
        uint32_t *tvals = slot<uint32_t>(st, S_TVALS, c);
        // pairs: twice the slots, so that a dictionary that just fits parts too
        const uint32_t c2 = may_part ? (full_c / 2 > c ? c * 2 : c) : 0u;
        unsigned long long *pkeys = may_part ? slot<unsigned long long>(st, S_PKEYS, c2) : nullptr;
        uint32_t *pvals = may_part ? slot<uint32_t>(st, S_PVALS, c2) : nullptr;
        uint32_t *pslot = may_part ? slot<uint32_t>(st, S_PSLOT, z) : nullptr;
        if (may_part) {
            check_cuda(cudaMemsetAsync(pkeys, 0, (size_t)c2 * 8, st->stream));
            check_cuda(cudaMemsetAsync(part, 0, sizeof(Parting), st->stream));
        }
        tdense = slot<uint32_t>(st, S_TDENSE, c2 > c ? c2 : c);
        dlen = slot<uint32_t>(st, S_DLEN, (size_t)z + 1);
        dstart = slot<uint32_t>(st, S_DSTART, (size_t)z + 1);
        check_cuda(cudaMemsetAsync(tkeys, 0, (size_t)c * 8, st->stream));
        check_cuda(cudaMemsetAsync(st->d_flags, 0, 8, st->stream));
        check_cuda(cudaMemsetAsync(st->d_flags + 48, 0, 4, st->stream));
        HashArgs a;
        a.full = st->d_flags + 48;
        a.T = dT; a.n = n; a.D = ph.D; a.z = z; a.W = W;
        a.base = (seed % (M61 - 1000)) + 257;
        a.tkeys = tkeys; a.tvals = tvals; a.cmask = c - 1;
        int logc = 0;
        while ((1u << logc) < c) logc++;
        a.logc = logc;
        a.limit = (uint32_t)(((uint64_t)c * 3) / 4);
        a.probes = c < full_c ? PH_PROBES_SMALL : PH_PROBES;
        a.slot_of = slot_of; a.flags = st->d_flags; a.xsep = xsep;
        a.bytes = may_part ? &part->bytes : nullptr;
        probe_begin(st, GBWT_PROBE_PHRASE_HASH);
        if (may_part) k_phrase_hash<true><<<grid_for(z, PH_THREADS), PH_THREADS, 0, st->stream>>>(a);
        else k_phrase_hash<false><<<grid_for(z, PH_THREADS), PH_THREADS, 0, st->stream>>>(a);
        // text bytes of all phrases (n + (W-1)(z-1) overlap) + D read + slot write
        probe_end(st, GBWT_PROBE_PHRASE_HASH, (uint64_t)n + (uint64_t)(W - 1) * (z - 1) + 8ull * z);
        after_launch(st);
        if (may_part) {
            k_pairs<<<grid_for(z, 256), 256, 0, st->stream>>>(ph.D, z, W, xsep, bt->ptid, slot_of, st->d_flags, pkeys,
                                                              pvals, c2 - 1u, pslot, part);
            after_launch(st);
        }
        k_phrase_verify<<<grid_for(z, 256), 256, 0, st->stream>>>(dT, n, ph.D, z, W, tvals, slot_of, isrep,
                                                                  st->d_flags, xsep, pvals, pslot, may_part ? part : nullptr);
        after_launch(st);
        device_scan<uint32_t, OpAdd>(st, z, LoadArr<uint32_t>{isrep}, StoreDense{ph.D, slot_of, tdense, dlen, dstart, W, xsep, ptid, dtid},
                                     false, st->d_flags + 6);
        check_cuda(cudaMemcpyAsync(st->h_scalars, st->d_flags, 32, cudaMemcpyDeviceToHost, st->stream));
        if (may_part)
            check_cuda(cudaMemcpyAsync(st->h_scalars + 4, part, sizeof(Parting), cudaMemcpyDeviceToHost, st->stream));
        sync_stream(st);
        const uint32_t flags = (uint32_t)st->h_scalars[0];
        d = (uint32_t)st->h_scalars[3];
        if (flags & ERR_TABLE_FULL) { c = full_c; st->stats.hash_retries++; continue; }
        if (flags & ERR_COLLISION) {
            seed = seed * 6364136223846793005ull + 1442695040888963407ull;
            st->stats.hash_retries++;
            continue;
        }
        break;
    }
    ph.d = d;
    Parting hp{};
    if (may_part) memcpy(&hp, st->h_scalars + 4, sizeof(hp));
    const bool parted = may_part && part_texts(hp);
    ph.dtid = parted ? dtid : nullptr;
    ph.texts = parted ? bt->k : 1u;
    uint32_t *pid = isrep;   // isrep is dead after the scan
    uint2 *occpc = slot<uint2>(st, S_OCC, d);
    check_cuda(cudaMemsetAsync(occpc, 0, (size_t)d * sizeof(uint2), st->stream));
    uint32_t *pidpc = d < (1u << 24) ? slot<uint32_t>(st, S_PIDPC, z) : nullptr;
    const bool few = d <= PH_FEW && z / d >= PH_FEW_OCC;
    unsigned fgrid = grid_for(z, 256);
    if (few && fgrid > (unsigned)st->num_sms * 8u) fgrid = (unsigned)st->num_sms * 8u;
    const uint32_t *ptids = bt ? bt->ptid : nullptr;
    const uint8_t *lastb = bt ? bt->lastb : nullptr;
    if (few)
        k_phrase_finalize<true><<<fgrid, 256, 0, st->stream>>>(dT, n, ph.D, z, d, W, slot_of, tdense, pid, pidpc, occpc,
                                                                xsep, ptids, lastb);
    else
        k_phrase_finalize<false><<<fgrid, 256, 0, st->stream>>>(dT, n, ph.D, z, d, W, slot_of, tdense, pid, pidpc, occpc,
                                                                 xsep, ptids, lastb);
    ph.pidpc = pidpc;
    after_launch(st);
    // dictionary offsets (64-bit scan, checked against 2^32)
    uint32_t *doff = slot<uint32_t>(st, S_DOFF, (size_t)d + 1);
    device_scan<uint64_t, OpAdd>(st, d, LoadLen64{dlen}, StoreOff32{doff, d}, false, (uint64_t *)st->d_scalars);
    if (ph.have_alpha)
        check_cuda(cudaMemcpyAsync(st->h_scalars + 4, st->d_flags + 8, sizeof(ph.alpha), cudaMemcpyDeviceToHost, st->stream));
    fetch_scalars(st, 1);
    if (ph.have_alpha) memcpy(ph.alpha, st->h_scalars + 4, sizeof(ph.alpha));
    const uint64_t dict_bytes = st->h_scalars[0];
    if (dict_bytes >= 0xFFFFFF00ull) throw Error{GBWT_UNSUPPORTED_INPUT};
    uint8_t *dict = slot<uint8_t>(st, S_DICT, dict_bytes + 16);
    uint32_t *dphr = slot<uint32_t>(st, S_DPHR, dict_bytes + 1);
    if (dict_bytes >= (uint64_t)d * 64u)
        k_dict_copy<32><<<grid_for((size_t)d * 32, 256), 256, 0, st->stream>>>(dT, n, d, doff, dlen, dstart, dict, dphr);
    else
        k_dict_copy<8><<<grid_for((size_t)d * 8, 256), 256, 0, st->stream>>>(dT, n, d, doff, dlen, dstart, dict, dphr);
    after_launch(st);
    ph.pid = pid; ph.dlen = dlen; ph.doff = doff; ph.occpc = occpc;
    ph.dict = dict; ph.dphr = dphr; ph.dict_bytes = dict_bytes;
}

}  // namespace gbwt
