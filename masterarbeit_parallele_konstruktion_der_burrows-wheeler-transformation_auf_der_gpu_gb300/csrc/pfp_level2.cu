// pfp_level2.cu -- suffix array of a large repetitive parse by parsing the
// parse (sm_103a).
//
// The reference sorts the parse by prefix doubling over all of its suffixes
// (Prefix_Free_Parsing_W=5_P=16_kommentiert.cu, "K": Sort_Suffix_Array
// K:2342-2412).  In a repetitive text almost every suffix of the parse stays
// tied for six or seven doublings, since the copies agree over hundreds of
// phrases, and every doubling reads and writes all of them.  The prefix-free
// parsing that shortened the text works on the parse just as well, with a
// phrase as the symbol and windows of one symbol:
//
//   symbols   V[i] = lexicographic rank of phrase i, plus 1; V[z] = 0 ends it
//   triggers  positions 1..z-1 whose symbol hashes below a threshold (one in
//             L2_RATE), and the end; phrase j of the second level spans
//             V[s_j .. s_{j+1}], both triggers included.  In a batch every text
//             starts a phrase, and the phrase before it ends with the symbol 0
//             instead: no phrase crosses a text, and suffixes of different
//             texts may tie, as in the plain batch parse
//   phrases   exact deduplication (hash table, then symbol by symbol), one
//             dictionary, sorted by the engine that sorts the first one
//   parse     suffix array of the second-level parse, L2_RATE times shorter
//   output    every first-level suffix i lies in one second-level phrase and
//             starts one of its suffixes of at least two symbols; no such
//             string is a proper prefix of another (a trigger is found only at
//             its end), so suffixes order by (group of that string, rank of
//             the next second-level suffix).  Emitting them in the order of
//             that rank and sorting stably by group leaves the suffix array.
//
// Parse stage before / after on GB300: 512 MiB DNA (z = 33.6 M) 8.45 / 4.2 ms, 256
// MiB of versions (11.7 M) 3.85 / 1.7 ms, 128 MiB DNA (8.4 M) 2.12 / 1.54 ms.
//
// Taken for parses of at least L2_MIN_Z phrases: its launches and host round
// trips are about 0.7 ms (z = 2.1 M: 0.70 ms plain, 0.92 ms here; 4.2 M: 1.23 and
// 1.15 ms).  And with at most one distinct phrase in L2_DISTINCT: a text of
// little repetition has few ties and a dictionary as long as the parse (one in
// 8: 1.09 ms plain, 1.82 ms here; one in 2.5: 1.36 and 1.92 ms; one in 18 to 75:
// as above).  L2_RATE: 4, 6, 8, 12 give 4.52, 4.19, 4.24, 4.66 ms on the DNA and
// 2.14, 1.85, 1.71, 1.62 ms on the versions.  It gives up, and the plain path
// runs, when a second-level phrase is longer than L2_MAXLEN symbols (a long run
// of one phrase: one thread reads it) or the dictionary exceeds half the parse.
#include "prims.cuh"

namespace gbwt {

constexpr uint32_t L2_RATE = 8;
constexpr uint32_t L2_MAXLEN = 4096;
constexpr uint32_t L2_MIN_Z = 1u << 22;
constexpr uint32_t L2_DISTINCT = 10;
constexpr int L2_TABLE_LOG2 = 22;

__device__ __forceinline__ bool l2_trigger(uint32_t v)
{
    // multiplicative hash of the symbol, high bits compared with 2^32 / L2_RATE
    uint32_t x = v * 0x9E3779B1u;
    x ^= x >> 15;
    x *= 0x85EBCA77u;
    return x < 0xFFFFFFFFu / L2_RATE;
}

// Symbols, start bits (triggers and text starts) and, with ptid (the text of
// every phrase), text-start bits.  Position 0 starts a phrase without a bit.
__global__ void k_l2_symbols(const uint32_t *pid, const uint32_t *lexrank, const uint32_t *ptid, uint32_t z, uint32_t *V,
                             uint32_t *bits, uint32_t *tstart)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool t = false, ts = false;
    if (i < z) {
        const uint32_t v = lexrank[pid[i]] + 1u;
        V[i] = v;
        ts = ptid && i > 0 && ptid[i] != ptid[i - 1];
        t = ts || (i > 0 && l2_trigger(v));
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, t), tm = __ballot_sync(0xFFFFFFFFu, ts);
    if ((threadIdx.x & 31u) == 0 && i < z) {
        bits[i >> 5] = m;
        if (tstart) tstart[i >> 5] = tm;
    }
}
// s[1 + j] = position of trigger j (s[0] = 0 and s[z2] = z are set apart).
struct StoreStarts {
    const uint32_t *w;
    uint32_t *s;
    uint32_t cap;               // the host gives up when there are more
    __device__ __forceinline__ void operator()(size_t i, uint32_t pre, uint32_t) const
    {
        for (uint32_t m = w[i]; m && pre < cap; m &= m - 1u)
            s[1u + pre++] = (uint32_t)i * 32u + (uint32_t)(__ffs(m) - 1);
    }
};
__global__ void k_l2_ends(uint32_t *s, uint32_t z2, uint32_t z)
{
    s[0] = 0;
    s[z2] = z;
}

// The symbols: V, and at a phrase's end e the trigger there or 0 at the end of
// a text.
struct L2Text {
    const uint32_t *V, *tstart;      // tstart: text-start bits of a batch, else null
    uint32_t z;
    __device__ __forceinline__ uint32_t inside(uint32_t i) const { return __ldg(V + i); }
    __device__ __forceinline__ uint32_t end(uint32_t e) const
    {
        if (e >= z || (tstart && ((tstart[e >> 5] >> (e & 31u)) & 1u))) return 0u;
        return __ldg(V + e);
    }
};

// Fingerprint (polynomial mod 2^61 - 1) and table slot of every phrase.
// give_up: [0] phrase too long or table full, [1] distinct phrases so far,
// [2] two phrases share a fingerprint.
__global__ void k_l2_hash(L2Text V, const uint32_t *s, uint32_t z2, uint64_t base,
                          unsigned long long *tkeys, uint32_t *tvals, int logc, uint32_t limit, uint32_t *slot_of,
                          uint32_t *give_up)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= z2) return;
    const uint32_t a = s[j], e = s[j + 1], len = e - a + 1u;
    slot_of[j] = 0;
    if (len > L2_MAXLEN) {
        give_up[0] = 1;
        return;
    }
    uint64_t h = len;
    for (uint32_t i = a; i <= e; i++) {
        h = mulmod61(h, base) + (i < e ? V.inside(i) : V.end(e)) + 1u;
        if (h >= M61) h -= M61;
    }
    const unsigned long long key = h + 1u;                       // 0 marks an empty slot
    const uint32_t cmask = (1u << logc) - 1u;
    uint32_t pos = (uint32_t)((key * 0xD6E8FEB86659FD93ull) >> (64 - logc));
    for (uint32_t probe = 0; probe <= cmask; probe++) {
        // a plain read first: most phrases of a repetitive parse are there already
        unsigned long long cur = __ldcg(tkeys + pos);
        if (cur == 0ull) cur = atomicCAS(tkeys + pos, 0ull, key);
        if (cur == 0ull) {
            tvals[pos] = j;                                       // the slot's representative
            if (atomicAdd(give_up + 1, 1u) >= limit) give_up[0] = 1;
            slot_of[j] = pos;
            return;
        }
        if (cur == key) {
            slot_of[j] = pos;
            return;
        }
        pos = (pos + 1u) & cmask;
        if ((probe & 7u) == 7u && *(volatile uint32_t *)give_up) return;
    }
    give_up[0] = 1;
}

// Every phrase against its representative, symbol by symbol.
__global__ void k_l2_verify(L2Text V, const uint32_t *s, uint32_t z2, const uint32_t *tvals,
                            const uint32_t *slot_of, uint32_t *isrep, uint32_t *give_up)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= z2) return;
    isrep[j] = 0;
    if (*(volatile uint32_t *)give_up) return;
    const uint32_t r = tvals[slot_of[j]];
    if (r == j) {
        isrep[j] = 1;
        return;
    }
    if (r >= z2) { give_up[2] = 1; return; }
    const uint32_t a = s[j], b = s[r], len = s[j + 1] - a;
    if (s[r + 1] - b != len) { give_up[2] = 1; return; }
    for (uint32_t i = 0; i < len; i++)
        if (V.inside(a + i) != V.inside(b + i)) { give_up[2] = 1; return; }
    if (V.end(a + len) != V.end(b + len)) give_up[2] = 1;
}

// Dense ids and dictionary offsets of the representatives in one scan:
// (symbols << 32) | phrases.
struct LoadRep {
    const uint32_t *isrep, *s;
    __device__ __forceinline__ uint64_t operator()(size_t j) const
    {
        return isrep[j] ? ((uint64_t)(s[j + 1] - s[j] + 1u) << 32) | 1u : 0ull;
    }
};
struct StoreRep {
    const uint32_t *s, *slot_of;
    uint32_t *tvals;            // the slot's representative -> its dense id
    uint32_t *dlen, *dstart, *doff;
    __device__ __forceinline__ void operator()(size_t j, uint64_t pre, uint64_t v) const
    {
        if (!v) return;
        const uint32_t id = (uint32_t)pre;
        tvals[slot_of[j]] = id;
        dlen[id] = (uint32_t)(v >> 32);
        dstart[id] = s[j];
        doff[id] = (uint32_t)(pre >> 32);
    }
};
__global__ void k_l2_ids(const uint32_t *slot_of, const uint32_t *dense, uint32_t z2, uint32_t *pid, uint32_t *occ)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= z2) return;
    const uint32_t id = dense[slot_of[j]];
    pid[j] = id;
    atomicAdd(occ + id, 1u);
}
// Eight lanes per distinct phrase (they average about ten symbols).
__global__ void k_l2_dict(L2Text V, uint32_t d, const uint32_t *doff, const uint32_t *dlen,
                          const uint32_t *dstart, uint32_t *dict, uint32_t *dphr)
{
    const uint32_t id = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    if (id >= d) return;
    const uint32_t off = doff[id], len = dlen[id], st = dstart[id];
    for (uint32_t i = threadIdx.x & 7u; i < len; i += 8u) {
        dict[off + i] = i + 1u < len ? V.inside(st + i) : V.end(st + i);
        dphr[off + i] = id;
    }
}
// First keys: the next h0 symbols plus 1 (0 = past the phrase end) and the bit
// "continues past h0", as in the first dictionary's keys; rem8[x] = min(rem, 255).
__global__ void k_l2_keys(const uint32_t *dict, uint32_t N, const uint32_t *dphr, const uint32_t *doff,
                          const uint32_t *dlen, int bps, int h0, uint64_t *keys, uint8_t *rem8)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    const uint32_t q = dphr[x], rem = doff[q] + dlen[q] - x;
    uint64_t key = 0;
    for (int i = 0; i < h0; i++) key = (key << bps) | ((uint32_t)i < rem ? (uint64_t)dict[x + i] + 1u : 0ull);
    keys[x] = (key << 1) | (rem > (uint32_t)h0 ? 1u : 0u);
    rem8[x] = (uint8_t)(rem < 255u ? rem : 255u);
}
// Groups of suffixes of at least two symbols, numbered in sorted order: mark
// their heads in a bit vector (N / 8 bytes), count, number.
__global__ void k_l2_heads(uint32_t N, const uint8_t *rem8, const uint32_t *isa, uint32_t *bits)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N || rem8[x] < 2) return;
    const uint32_t t = isa[x];
    const uint32_t b = 1u << (t & 31u);
    if (!(*(volatile uint32_t *)(bits + (t >> 5)) & b)) atomicOr(bits + (t >> 5), b);
}
__global__ void k_l2_groups(uint32_t N, const uint8_t *rem8, const uint32_t *isa, const uint32_t *bits,
                            const uint32_t *pre, uint32_t *grp)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N || rem8[x] < 2) return;
    const uint32_t t = isa[x];
    grp[x] = pre[t >> 5] + (uint32_t)__popc(bits[t >> 5] & ((1u << (t & 31u)) - 1u));
}

// Emission slots in the order of the next second-level suffix: the last phrase
// first, then the phrase before each suffix in suffix-array order (none before
// suffix 0).
__global__ void k_l2_slots(const uint32_t *psa, const uint32_t *pisa, const uint32_t *pid, const uint32_t *s,
                           const uint32_t *doff, uint32_t z2, uint32_t *from, uint32_t *to, uint32_t *cnt)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= z2) return;
    uint32_t j = z2 - 1u;
    if (t) j = psa[t - 1u < pisa[0] ? t - 1u : t] - 1u;
    from[t] = doff[pid[j]];
    to[t] = s[j];
    cnt[t] = s[j + 1] - s[j];
}
// Batch: the text of every second-level phrase, and one past each text's last.
__global__ void k_l2_texts(const uint32_t *s, uint32_t z2, const uint32_t *ptid, uint32_t *tid2, uint32_t *zend2)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= z2) return;
    const uint32_t t = ptid[s[j]];
    tid2[j] = t;
    if (j + 1u == z2 || ptid[s[j + 1]] != t) zend2[t] = j + 1u;
}
// Batch slots: every text's last phrase, then the phrase before each suffix in
// suffix-array order (an empty slot for a text's first).
__global__ void k_l2_slots_batch(const uint32_t *psa, const uint32_t *pid, const uint32_t *s, const uint32_t *doff,
                                 const uint32_t *tid2, const uint32_t *zend2, uint32_t k, uint32_t z2, uint32_t *from,
                                 uint32_t *to, uint32_t *cnt)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= k + z2) return;
    uint32_t j;
    if (t < k) {
        j = zend2[t] - 1u;
    } else {
        const uint32_t x = psa[t - k];
        if (x == 0 || tid2[x] != tid2[x - 1u]) {
            from[t] = 0;
            to[t] = 0;
            cnt[t] = 0;
            return;
        }
        j = x - 1u;
    }
    from[t] = doff[pid[j]];
    to[t] = s[j];
    cnt[t] = s[j + 1] - s[j];
}
// 256 slots per CTA; each thread walks EL_PER consecutive elements, staged so
// that consecutive threads write consecutive elements.
constexpr int EL_T = 256;
constexpr int EL_PER = 8;
__global__ void __launch_bounds__(EL_T) k_l2_emit(uint32_t z2, const uint32_t *eoff, const uint32_t *from,
                                                  const uint32_t *to, const uint32_t *grp, uint32_t z, uint32_t *keys,
                                                  uint32_t *vals, uint32_t *flags)
{
    __shared__ uint32_t s_off[EL_T + 1], s_from[EL_T], s_to[EL_T];
    __shared__ uint32_t s_key[EL_T * EL_PER + EL_T * EL_PER / 32], s_val[EL_T * EL_PER + EL_T * EL_PER / 32];
    const uint32_t t0 = blockIdx.x * EL_T;
    const uint32_t tn = min((uint32_t)EL_T, z2 - t0);
    if (threadIdx.x < tn) {
        s_off[threadIdx.x] = eoff[t0 + threadIdx.x];
        s_from[threadIdx.x] = from[t0 + threadIdx.x];
        s_to[threadIdx.x] = to[t0 + threadIdx.x];
    }
    if (threadIdx.x == 0) s_off[tn] = eoff[t0 + tn];
    __syncthreads();
    const uint32_t o0 = s_off[0], cnt = s_off[tn] - o0;
    if ((uint64_t)o0 + cnt > z) {
        if (threadIdx.x == 0) atomicOr(flags, ERR_INTERNAL);
        return;
    }
    for (uint32_t cb = 0; cb < cnt; cb += EL_T * EL_PER) {
        const uint32_t e0 = cb + threadIdx.x * EL_PER;
        if (e0 < cnt) {
            uint32_t lo = 0, hi = tn - 1u;            // last slot with s_off <= o0 + e0
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1u) >> 1;
                if (s_off[mid] <= o0 + e0) lo = mid; else hi = mid - 1u;
            }
#pragma unroll
            for (int q = 0; q < EL_PER; q++) {
                const uint32_t o = o0 + e0 + q;
                if (e0 + q >= cnt) break;
                while (s_off[lo + 1] <= o) lo++;
                const uint32_t k = sc_pad(threadIdx.x * EL_PER + q);
                s_key[k] = grp[s_from[lo] + (o - s_off[lo])];
                s_val[k] = s_to[lo] + (o - s_off[lo]);
            }
        }
        __syncthreads();
        const uint32_t m = min((uint32_t)(EL_T * EL_PER), cnt - cb);
        for (uint32_t i = threadIdx.x; i < m; i += EL_T) {
            keys[o0 + cb + i] = s_key[sc_pad(i)];
            vals[o0 + cb + i] = s_val[sc_pad(i)];
        }
        __syncthreads();
    }
}

// first[0], first[1]: ranks of suffixes 0 and 1.
__global__ void k_l2_first(const uint32_t *sa, uint32_t z, uint32_t *first)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < z && sa[r] < 2u) first[sa[r]] = r;
}

bool run_parse_sa_level2(Storage *st, Phrases &ph, DictOrder &dord, ParseOrder &pord, const BatchText *bt)
{
    const uint32_t z = ph.z;
    if (z < L2_MIN_Z || ph.d > z / L2_DISTINCT) return false;
    // symbols, triggers, phrase starts
    uint32_t *sym = slot<uint32_t>(st, S_2SYM, z);
    const size_t zw = ((size_t)z + 31) / 32;
    uint32_t *trig = slot<uint32_t>(st, S_2TRIG, zw);
    uint32_t *tstart = bt ? slot<uint32_t>(st, S_2TSTART, zw) : nullptr;
    k_l2_symbols<<<grid_for(z, 256), 256, 0, st->stream>>>(ph.pid, dord.lexrank, bt ? bt->ptid : nullptr, z, sym, trig,
                                                           tstart);
    after_launch(st);
    const L2Text V{sym, tstart, z};
    // starts are stored by the scan that counts them: room for one in three
    // positions, more means symbols that hash alike (or tiny texts) and no gain
    const uint32_t cap = z / 3u;
    uint32_t *s = slot<uint32_t>(st, S_2START, (size_t)cap + 2);
    device_scan<uint32_t, OpAdd>(st, zw, LoadPopc{trig}, StoreStarts{trig, s, cap}, false, (uint32_t *)st->d_scalars);
    fetch_scalars(st, 1);
    const uint32_t z2 = (uint32_t)st->h_scalars[0] + 1u;
    if (z2 > cap) return false;
    k_l2_ends<<<1, 1, 0, st->stream>>>(s, z2, z);
    after_launch(st);
    // distinct phrases
    const int logc = L2_TABLE_LOG2;
    const uint32_t c = 1u << logc;
    unsigned long long *tkeys = slot<unsigned long long>(st, S_TKEYS, c);
    uint32_t *tvals = slot<uint32_t>(st, S_TVALS, c);
    uint32_t *slot_of = slot<uint32_t>(st, S_2SLOT, z2);
    uint32_t *pid = slot<uint32_t>(st, S_2PID, z2);          // representative marks until the ids are known
    const uint32_t limit = c / 4u * 3u;
    const uint32_t dmax = z2 < limit ? z2 : limit;
    uint32_t *dlen = slot<uint32_t>(st, S_2DLEN, dmax), *dstart = slot<uint32_t>(st, S_2DSTART, dmax);
    uint32_t *doff = slot<uint32_t>(st, S_2DOFF, dmax);
    uint32_t *give_up = st->d_flags + 28;
    check_cuda(cudaMemsetAsync(tkeys, 0, (size_t)c * 8, st->stream));
    check_cuda(cudaMemsetAsync(give_up, 0, 3 * 4, st->stream));
    k_l2_hash<<<grid_for(z2, 256), 256, 0, st->stream>>>(V, s, z2, 0x0A5C3D1F2B4E6987ull, tkeys, tvals, logc, limit,
                                                         slot_of, give_up);
    after_launch(st);
    k_l2_verify<<<grid_for(z2, 256), 256, 0, st->stream>>>(V, s, z2, tvals, slot_of, pid, give_up);
    after_launch(st);
    check_cuda(cudaMemcpyAsync(st->h_scalars + 4, give_up, 3 * 4, cudaMemcpyDeviceToHost, st->stream));
    sync_stream(st);
    const uint32_t *g = (const uint32_t *)(st->h_scalars + 4);
    if (g[0] || g[2]) return false;
    device_scan<uint64_t, OpAdd>(st, z2, LoadRep{pid, s}, StoreRep{s, slot_of, tvals, dlen, dstart, doff}, false,
                                 (uint64_t *)st->d_scalars);
    fetch_scalars(st, 1);
    const uint32_t d = (uint32_t)st->h_scalars[0], N = (uint32_t)(st->h_scalars[0] >> 32);
    if (N > z / 2u) return false;
    uint32_t *occ = slot<uint32_t>(st, S_2OCC, d);
    check_cuda(cudaMemsetAsync(occ, 0, (size_t)d * 4, st->stream));
    k_l2_ids<<<grid_for(z2, 256), 256, 0, st->stream>>>(slot_of, tvals, z2, pid, occ);
    after_launch(st);
    // dictionary and its order
    uint32_t *dict = slot<uint32_t>(st, S_2DICT, N), *dphr = slot<uint32_t>(st, S_2DPHR, N);
    k_l2_dict<<<grid_for((size_t)d * 8, 256), 256, 0, st->stream>>>(V, d, doff, dlen, dstart, dict, dphr);
    after_launch(st);
    const int bps = bits_for((uint64_t)ph.d + 1u);
    const int h0 = 2;      // 1, 2 or 3 symbols in the first key: 4.45, 4.19, 4.26 ms (512 MiB DNA); 2 * bps < 64
    uint64_t *keys = slot<uint64_t>(st, S_KEY0, N);
    uint8_t *rem8 = slot<uint8_t>(st, S_2TRIG, N);          // the trigger bits are dead
    k_l2_keys<<<grid_for(N, 256), 256, 0, st->stream>>>(dict, N, dphr, doff, dlen, bps, h0, keys, rem8);
    after_launch(st);
    uint32_t *isa = slot<uint32_t>(st, S_2ISA, N), *sa = slot<uint32_t>(st, S_2SA, N);
    pord.rounds = sort_phrase_suffixes(st, N, h0 * bps + 1, (uint32_t)h0, dphr, doff, dlen, rem8, isa, sa);
    uint32_t *rank = slot<uint32_t>(st, S_2RANK, d);
    phrase_ranks(st, N, d, isa, doff, rank);
    // suffix array of the second-level parse
    uint32_t *pisa = slot<uint32_t>(st, S_2PISA, z2), *psa = slot<uint32_t>(st, S_2PSA, z2);
    uint32_t *tid2 = nullptr, *zend2 = nullptr;
    if (bt) {
        tid2 = slot<uint32_t>(st, S_2TID, z2);
        zend2 = slot<uint32_t>(st, S_2ZEND, bt->k);
        k_l2_texts<<<grid_for(z2, 256), 256, 0, st->stream>>>(s, z2, bt->ptid, tid2, zend2);
        after_launch(st);
        pord.rounds += parse_sa_batch(st, z2, d, pid, rank, tid2, zend2, bt->k, true, pisa, psa);
    } else {
        pord.rounds += parse_sa_buckets(st, z2, d, pid, rank, occ, 1, pisa, psa);
    }
    // group numbers per dictionary position (sa is dead: it takes them)
    const size_t nw = ((size_t)N + 31) / 32;
    uint32_t *bits = slot<uint32_t>(st, S_TMP0, nw), *pre = slot<uint32_t>(st, S_TMP1, nw);
    uint32_t *grp = sa;
    check_cuda(cudaMemsetAsync(bits, 0, nw * 4, st->stream));
    k_l2_heads<<<grid_for(N, 256), 256, 0, st->stream>>>(N, rem8, isa, bits);
    after_launch(st);
    device_scan<uint32_t, OpAdd>(st, nw, LoadPopc{bits}, StoreArr<uint32_t>{pre}, false, (uint32_t *)st->d_scalars);
    k_l2_groups<<<grid_for(N, 256), 256, 0, st->stream>>>(N, rem8, isa, bits, pre, grp);
    after_launch(st);
    // emission and the sort by group
    const uint32_t S = bt ? bt->k + z2 : z2;
    uint32_t *from = slot<uint32_t>(st, S_ACTX, S), *to = slot<uint32_t>(st, S_ACTG, S);
    uint32_t *cnt = slot<uint32_t>(st, S_ACTX2, (size_t)S + 1);
    if (bt)
        k_l2_slots_batch<<<grid_for(S, 256), 256, 0, st->stream>>>(psa, pid, s, doff, tid2, zend2, bt->k, z2, from, to,
                                                                   cnt);
    else
        k_l2_slots<<<grid_for(S, 256), 256, 0, st->stream>>>(psa, pisa, pid, s, doff, z2, from, to, cnt);
    after_launch(st);
    device_scan<uint32_t, OpAdd>(st, S, LoadArr<uint32_t>{cnt}, StoreArr<uint32_t>{cnt}, false, cnt + S);
    check_cuda(cudaMemcpyAsync(st->d_scalars + 1, cnt + S, 4, cudaMemcpyDeviceToDevice, st->stream));
    fetch_scalars(st, 2);
    const uint32_t G = (uint32_t)st->h_scalars[0];
    if (G == 0 || (uint32_t)st->h_scalars[1] != z) throw Error{GBWT_INTERNAL_ERROR};
    uint32_t *k = slot<uint32_t>(st, S_KEY0, z), *k_alt = slot<uint32_t>(st, S_KEY1, z);
    uint32_t *v = slot<uint32_t>(st, S_PSA, z), *v_alt = slot<uint32_t>(st, S_PISA, z);
    k_l2_emit<<<grid_for(S, EL_T), EL_T, 0, st->stream>>>(S, cnt, from, to, grp, z, k, v, st->d_flags);
    after_launch(st);
    radix_sort<uint32_t, true>(st, k, k_alt, v, v_alt, z, 0, bits_for(G - 1u));
    pord.sa = v;
    pord.isa = nullptr;
    if (bt) return true;
    uint32_t *first = st->d_flags + 32;
    k_l2_first<<<grid_for(z, 256), 256, 0, st->stream>>>(v, z, first);
    after_launch(st);
    pord.first = first;
    return true;
}

}  // namespace gbwt
