// pfp_assembly.cu -- BWT assembly from the dictionary order and the parse
// suffix array (sm_103a).
//
// The reference enumerates S (distinct phrase suffixes longer than W) from a
// colex sort of all occurrences, finds each entry's colex interval with a
// next-smaller-value search, writes one-byte blocks ("runs") directly and
// sorts the remaining ("mixed") blocks by the rank of the next parse suffix
// (Prefix_Free_Parsing_W=5_P=16_kommentiert.cu, "K": Compute_S1..S6
// K:2509-3369, bitonic block sorts K:3556-4248).
//
// Here S comes out of the dictionary suffix order directly: equal suffixes
// are one group of the prefix-doubling result, named by the sorted position
// of its first member.  For every group we add the occurrence counts of its
// phrases (block length) and check whether all preceding bytes agree (run).
// Runs are written one group per thread with 16-byte stores (long blocks one CTA
// each).  For mixed groups, every phrase occurrence -- visited in parse
// suffix-array order, which is exactly the "rank of the next parse suffix"
// order the reference sorts by -- emits one (group, byte) element per mixed
// suffix of its phrase; one stable radix sort by group then places every
// byte, and a coalesced scatter writes them into the output.
#include "prims.cuh"

namespace gbwt {

constexpr uint32_t PC_VAR = 0x100u;     // "byte preceding the occurrence"

struct PosInfo {
    const uint32_t *dphr, *doff, *dlen;
    __device__ __forceinline__ void get(uint32_t x, uint32_t &q, uint32_t &off, uint32_t &rem) const
    {
        q = dphr[x];
        off = x - doff[q];
        rem = dlen[q] - off;
    }
};

// ---- single text: groups by the sorted position of their head ----------
// stat[t] of the group whose head is sorted position t: x = block length, y =
// the preceding bytes seen, byte c as c | (~c << 16).  OR-ing members keeps a
// bit position clear in one half exactly when all bytes agree in it, so y's
// halves are disjoint in their low bytes iff the block is one run.
//
// One pass over dictionary positions in storage order (phrase tables read
// almost sequentially) with two reductions per long suffix into the 8-byte
// word of its group.  Random sectors bound it: one read and one write-back per
// suffix.  Numbering the groups first cost a byte scattered per suffix, a
// random read of the number, a sum, a stored byte and a second pass comparing
// the bytes (four random sectors per suffix).  All S-group kernels together:
// 512 MiB DNA, W=35 (N = 130 M) 13.9 -> 4.3 ms, of it 3.5 here; W=5 1.28 -> 0.73
// ms; 102 MB of versions 4.9 -> 1.7 ms.
__device__ __forceinline__ bool gs_mixed(uint32_t y) { return (y & (y >> 16) & 0xFFu) != 0; }

__global__ void k_group_stats(uint32_t N, PosInfo pi, uint32_t W, const uint32_t *isa, const uint8_t *dict,
                              const uint2 *occpc, uint2 *stat)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    uint32_t q, off, rem;
    pi.get(x, q, off, rem);
    if (rem <= W) return;
    const uint32_t t = isa[x];
    const uint2 oc = occpc[q];                  // a whole phrase: the bytes before its occurrences
    const uint32_t c = off ? dict[x - 1] : 0u;
    atomicAdd(&stat[t].x, oc.x);
    atomicOr(&stat[t].y, off ? c | ((c ^ 0xFFu) << 16) : oc.y);
}

// One scan of the block lengths turns the statistics into places: stat[t]
// becomes x = the output offset of t's block (for a position that heads no
// group: of the next block; stat[N].x = n), y = tag: the run's byte, GS_MIX, or
// GS_NONE.  Heads and mixed heads also go into bit vectors over sorted
// positions, so that the few mixed blocks are numbered by a scan over words
// (N / 32 items) instead of carrying three more sums through this one
// (512 MiB DNA, W=35, N = 130 M: 1.51 ms for a scan of four sums).
constexpr uint32_t GS_MIX = 0x80000000u, GS_NONE = 0x100u;
struct LoadGCount {
    const uint2 *stat;
    __device__ __forceinline__ uint32_t operator()(size_t t) const { return stat[t].x; }
};
struct StoreGroup {
    uint2 *stat;
    uint32_t N;
    uint32_t *heads, *mixed;
    // called for consecutive t by consecutive lanes, warps starting at multiples of 32
    __device__ __forceinline__ void operator()(size_t t, uint32_t pre, uint32_t v) const
    {
        const uint32_t y = stat[t].y;
        const bool head = v != 0, mix = gs_mixed(y);
        const uint32_t left = N - ((uint32_t)t & ~31u);          // lanes of this warp inside [0, N)
        const unsigned lanes = left >= 32u ? 0xFFFFFFFFu : (1u << left) - 1u;
        const unsigned hm = __ballot_sync(lanes, head), mm = __ballot_sync(lanes, mix);
        if (((uint32_t)t & 31u) == 0) {
            heads[t >> 5] = hm;
            mixed[t >> 5] = mm;
        }
        stat[t] = make_uint2(pre, mix ? GS_MIX : head ? (y & 0xFFu) : GS_NONE);
        if (t + 1 == N) stat[N] = make_uint2(pre + v, GS_NONE);
    }
};
// Per word of the bit vectors: bytes in mixed blocks, mixed blocks, groups.
struct LoadMixWord {
    const uint2 *stat;
    const uint32_t *heads, *mixed;
    __device__ __forceinline__ Sum4 operator()(size_t w) const
    {
        uint32_t m = mixed[w], bytes = 0;
        const uint32_t cnt = (uint32_t)__popc(m);
        for (; m; m &= m - 1u) {
            const size_t t = w * 32 + (size_t)(__ffs(m) - 1);
            bytes += stat[t + 1].x - stat[t].x;
        }
        return Sum4(bytes, cnt, (uint32_t)__popc(heads[w]), 0u);
    }
};
struct StoreMixWord {
    uint2 *stat;
    const uint32_t *mixed;
    uint32_t *delta;            // per mixed block: output offset minus its place among the mixed bytes
    __device__ __forceinline__ void operator()(size_t w, const Sum4 &pre, const Sum4 &) const
    {
        uint32_t place = pre.a, b = pre.b;
        for (uint32_t m = mixed[w]; m; m &= m - 1u, b++) {
            const size_t t = w * 32 + (size_t)(__ffs(m) - 1);
            const uint32_t o = stat[t].x;
            delta[b] = o - place;
            place += stat[t + 1].x - o;
            stat[t].y = GS_MIX | b;
        }
    }
};

// ---- batch: dense group numbers ------------------------------------------
// The batch sorts its output by group, so the numbers have to be dense: mark
// the sorted position isa[x] of every long suffix's group head, scan the
// marks, read each position's number back through isa[x].
__global__ void k_mark_sheads(uint32_t N, PosInfo pi, uint32_t W, const uint32_t *isa, uint8_t *mark)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    uint32_t q, off, rem;
    pi.get(x, q, off, rem);
    if (rem > W) mark[isa[x]] = 1;
}
struct LoadMark {
    const uint8_t *m;
    __device__ __forceinline__ uint32_t operator()(size_t t) const { return m[t]; }
};
struct StoreGid {
    uint32_t *gid;
    __device__ __forceinline__ void operator()(size_t t, uint32_t inc, uint32_t v) const
    {
        if (v) gid[t] = inc - 1u;
    }
};
__global__ void k_group_of(uint32_t N, PosInfo pi, uint32_t W, const uint32_t *isa, const uint32_t *gid,
                           uint32_t *grp_of)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N) return;
    uint32_t q, off, rem;
    pi.get(x, q, off, rem);
    if (rem > W) grp_of[x] = gid[isa[x]];
}

// Per-phrase lists of mixed suffixes, in dictionary (phrase, offset) order:
// one bit per dictionary position (looked up in the mixed-head vector, N / 8
// bytes that stay in L2), a scan of the words' counts, and a pass over the set
// bits.  One position per thread keeps many lookups in flight; as the load of
// a scan each thread ran a chain of them (512 MiB DNA, W=35: 2.9 ms for the
// scan, 1.5 ms for these passes).
__global__ void k_mix_flags(uint32_t N, PosInfo pi, uint32_t W, const uint32_t *isa, const uint32_t *mixed,
                            uint32_t *words)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    bool set = false;
    if (x < N) {
        uint32_t q, off, rem;
        pi.get(x, q, off, rem);
        if (rem > W) {
            const uint32_t t = isa[x];
            set = (mixed[t >> 5] >> (t & 31u)) & 1u;
        }
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, set);
    if ((threadIdx.x & 31u) == 0 && x < N) words[x >> 5] = m;
}
__device__ __forceinline__ uint32_t bits_before(const uint32_t *words, const uint32_t *pre, uint32_t x)
{
    return pre[x >> 5] + (uint32_t)__popc(words[x >> 5] & ((1u << (x & 31u)) - 1u));
}
__global__ void k_mix_offsets(uint32_t d, const uint32_t *doff, const uint32_t *words, const uint32_t *pre,
                              uint32_t *moff)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < d) moff[q] = bits_before(words, pre, doff[q]);
}
__global__ void k_mix_entries(uint32_t N, const uint32_t *dphr, const uint32_t *doff, const uint8_t *dict,
                              const uint32_t *isa, const uint2 *stat, const uint32_t *words, const uint32_t *pre,
                              uint32_t *mb, uint16_t *mc)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= N || !((words[x >> 5] >> (x & 31u)) & 1u)) return;
    const uint32_t e = bits_before(words, pre, x);
    mb[e] = stat[isa[x]].y & ~GS_MIX;
    mc[e] = (uint16_t)(x != doff[dphr[x]] ? dict[x - 1] : PC_VAR);
}

// Emission order: the last phrase first (its next-suffix rank is -1,
// K:787-807), then the phrase before each parse suffix in suffix-array order.
struct Emit {
    const uint32_t *psa, *first, *pid, *moff, *D;     // first[0]: rank of parse suffix 0
    uint32_t z;
    __device__ __forceinline__ uint32_t occ_at(size_t t) const
    {
        if (t == 0) return z - 1u;
        const uint32_t pos0 = first[0];
        const uint32_t r = (uint32_t)t - 1u < pos0 ? (uint32_t)t - 1u : (uint32_t)t;
        return psa[r] - 1u;
    }
};

// Per emission slot t: phrase id, number of mixed elements and the byte
// preceding the occurrence (the random gathers happen once, here).
__global__ void k_emit_prep(Emit e, const uint32_t *pidpc, const uint8_t *T, uint32_t n, int W, const uint32_t *ptid,
                            const uint8_t *lastb, uint32_t *emq, uint8_t *emp, uint32_t *ecnt)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= e.z) return;
    const uint32_t k = e.occ_at(t);
    uint32_t q, prev;
    if (pidpc) {                      // one gather: id and preceding byte packed
        const uint32_t v = pidpc[k];
        q = v >> 8;
        prev = v & 0xFFu;
    } else {
        q = e.pid[k];
        if (ptid && (k == 0 || T[e.D[k - 1]] == 1)) {
            prev = lastb[ptid[k]];            // a text's first phrase follows the text's last byte
        } else {
            const uint32_t start = k ? e.D[k - 1] - (uint32_t)W + 1u : 0u;
            prev = preceding_byte(T, n, start);
        }
    }
    emq[t] = q;
    emp[t] = (uint8_t)prev;
    ecnt[t] = e.moff[q + 1] - e.moff[q];
}

// 256 emission slots per CTA; the CTA writes its contiguous output range
// with consecutive threads on consecutive elements.
constexpr int EM_T = 256;
constexpr int EM_PER = 8;          // consecutive elements per thread and chunk
template <typename E>
__global__ void __launch_bounds__(EM_T) k_emit(uint32_t z, const uint32_t *eoff, const uint32_t *emq,
                                               const uint8_t *emp, const uint32_t *moff, const uint32_t *mb,
                                               const uint16_t *mc, E *elem, uint32_t cap, uint32_t *flags)
{
    __shared__ uint32_t s_off[EM_T + 1];
    __shared__ uint32_t s_base[EM_T];
    __shared__ uint8_t s_prev[EM_T];
    __shared__ E s_out[EM_T * EM_PER + EM_T * EM_PER / 32];     // sc_pad layout (bank-conflict free)
    const uint32_t t0 = blockIdx.x * EM_T;
    const uint32_t tn = min((uint32_t)EM_T, z - t0);
    if (threadIdx.x < tn) {
        const uint32_t t = t0 + threadIdx.x;
        s_off[threadIdx.x] = eoff[t];
        s_base[threadIdx.x] = moff[emq[t]];
        s_prev[threadIdx.x] = emp[t];
    }
    if (threadIdx.x == 0) s_off[tn] = eoff[t0 + tn];
    __syncthreads();
    const uint32_t o0 = s_off[0], cnt = s_off[tn] - o0;
    if ((uint64_t)o0 + cnt > cap) {
        if (threadIdx.x == 0) atomicOr(flags, ERR_INTERNAL);
        return;
    }
    // chunks of EM_T * EM_PER elements: each thread finds the slot of its
    // first element once and walks forward; the chunk is staged in shared
    // memory and written with consecutive threads on consecutive elements
    for (uint32_t cb = 0; cb < cnt; cb += EM_T * EM_PER) {
        const uint32_t e0 = cb + threadIdx.x * EM_PER;
        if (e0 < cnt) {
            const uint32_t o = o0 + e0;
            uint32_t lo = 0, hi = tn - 1u;            // last slot with s_off <= o
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1u) >> 1;
                if (s_off[mid] <= o) lo = mid; else hi = mid - 1u;
            }
#pragma unroll
            for (int q = 0; q < EM_PER; q++) {
                const uint32_t e = e0 + q;
                if (e >= cnt) break;
                while (s_off[lo + 1] <= o0 + e) lo++;
                const uint32_t j = s_base[lo] + (o0 + e - s_off[lo]);
                uint32_t c = mc[j];
                if (c == PC_VAR) c = s_prev[lo];
                s_out[sc_pad(threadIdx.x * EM_PER + q)] = ((E)mb[j] << 8) | (E)c;
            }
        }
        __syncthreads();
        const uint32_t m = min((uint32_t)(EM_T * EM_PER), cnt - cb);
        for (uint32_t i = threadIdx.x; i < m; i += EM_T) elem[o0 + cb + i] = s_out[sc_pad(i)];
        __syncthreads();
    }
}

// 4 sorted elements per thread; consecutive elements of one block land on
// consecutive output bytes.
template <typename E>
__global__ void k_mixed_scatter(const E *elem, uint32_t M, const uint32_t *delta, uint32_t B, uint8_t *out,
                                uint32_t n, uint32_t *flags)
{
    const uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4u;
    if (i0 >= M) return;
    E v[4];
    if (i0 + 4u <= M) {                 // one (or two) 16-byte loads
        if constexpr (sizeof(E) == 4) {
            const uint4 w = *(const uint4 *)(elem + i0);
            memcpy(v, &w, 16);
        } else {
            const ulonglong2 w0 = *(const ulonglong2 *)(elem + i0);
            const ulonglong2 w1 = *(const ulonglong2 *)(elem + i0 + 2);
            memcpy(v, &w0, 16);
            memcpy((char *)v + 16, &w1, 16);
        }
    } else {
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) v[j] = i0 + j < M ? elem[i0 + j] : (E)0;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const uint32_t i = i0 + j;
        if (i >= M) break;
        const E e = v[j];
        const uint32_t b = (uint32_t)(e >> 8);
        const uint32_t p = b < B ? i + delta[b] : 0xFFFFFFFFu;
        if (p < n) out[p] = (uint8_t)(e & 0xFFu);
        else atomicOr(flags, ERR_INTERNAL);
    }
}

// Run fill, one thread per sorted position: the block of a run group is one
// byte repeated, written in pieces of 1, 2, 4 and 8 bytes up to a 16-byte
// boundary, 16-byte stores, and pieces again (neighbouring threads' edges meet
// in L2).  Runs average tens of bytes, so their edges are most of the stores:
// pieces take at most eight where bytes took up to thirty (512 MiB DNA: 342 ->
// 187 us, 256 MiB of versions: 377 -> 134 us).  Mixed groups are skipped: the
// mixed scatter writes every byte of theirs.  Blocks longer than RF_LONG bytes
// are listed and filled by one CTA each, so no thread carries a long block.
constexpr uint32_t RF_LONG = 512;

__device__ __forceinline__ void fill_run(uint8_t *out, uint32_t b0, uint32_t b1, uint8_t c)
{
    const uint32_t w = (uint32_t)c * 0x01010101u;
    const uint64_t w2 = ((uint64_t)w << 32) | w;
    uint8_t *p = out + b0;
    uint32_t r = b1 - b0;
    // a piece is skipped only when fewer bytes are left, so p stays aligned
    // to every smaller piece
    if (((uintptr_t)p & 1u) && r >= 1u) { *p = c; p += 1; r -= 1; }
    if (((uintptr_t)p & 2u) && r >= 2u) { *(uint16_t *)p = (uint16_t)w; p += 2; r -= 2; }
    if (((uintptr_t)p & 4u) && r >= 4u) { *(uint32_t *)p = w; p += 4; r -= 4; }
    if (((uintptr_t)p & 8u) && r >= 8u) { *(uint64_t *)p = w2; p += 8; r -= 8; }
    for (; r >= 16u; p += 16, r -= 16) *(uint4 *)p = make_uint4(w, w, w, w);
    if (r & 8u) { *(uint64_t *)p = w2; p += 8; }
    if (r & 4u) { *(uint32_t *)p = w; p += 4; }
    if (r & 2u) { *(uint16_t *)p = (uint16_t)w; p += 2; }
    if (r & 1u) *p = c;
}

__global__ void k_run_fill_groups(uint8_t *out, uint32_t n, const uint2 *stat, uint32_t N, uint32_t *longs,
                                  uint32_t long_cap, uint32_t *flags)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N) return;
    const uint2 s = stat[t];
    if (s.y > 0xFFu) return;                  // mixed, or no group's head
    const uint32_t b0 = s.x, b1 = t + 1u < N ? stat[t + 1u].x : n;
    if (b1 < b0 || b1 > n) { atomicOr(flags, ERR_INTERNAL); return; }
    if (b1 - b0 > RF_LONG) {
        const uint32_t i = atomicAdd(flags + 5, 1u);
        if (i < long_cap) longs[i] = t;
        else atomicOr(flags, ERR_INTERNAL);
        return;
    }
    fill_run(out, b0, b1, (uint8_t)s.y);
}

// One CTA per listed long run (the count is read on the device: no host sync).
__global__ void k_run_fill_long(uint8_t *out, uint32_t n, const uint2 *stat, uint32_t N, const uint32_t *longs,
                                const uint32_t *nlong, uint32_t long_cap)
{
    const uint32_t cnt = min(*nlong, long_cap);
    for (uint32_t i = blockIdx.x; i < cnt; i += gridDim.x) {
        const uint32_t t = longs[i];
        const uint32_t b0 = stat[t].x, b1 = t + 1u < N ? stat[t + 1u].x : n;
        const uint8_t c = (uint8_t)stat[t].y;
        // head bytes to the first 16-byte boundary, then striped 16-byte stores
        uint32_t a0 = b0;
        while (a0 < b1 && (((uintptr_t)(out + a0)) & 15u)) a0++;
        if (threadIdx.x < a0 - b0) out[b0 + threadIdx.x] = c;
        const uint32_t nv = (b1 - a0) / 16u;
        const uint32_t w = (uint32_t)c * 0x01010101u;
        const uint4 v = make_uint4(w, w, w, w);
        for (uint32_t j = threadIdx.x; j < nv; j += blockDim.x) *(uint4 *)(out + a0 + 16u * j) = v;
        const uint32_t t0 = a0 + 16u * nv;
        if (threadIdx.x < b1 - t0) out[t0 + threadIdx.x] = c;
    }
}

// Output row of the suffix starting at text position 0 (the "primary index"):
// its block is the group g0 of phrase 0 taken whole; inside a block the rows
// follow the rank of the next parse suffix (last phrase: -1, K:787-807).
// counter = goff[g0] + the occurrences of g0's string ranked before text
// position 0's.  Pass 1 (text order, tables read in sequence) marks, in a bit
// vector over parse positions, the suffixes that follow the other occurrences;
// pass 2 (suffix-array order) counts the marked ones before suffix 1.  An
// occurrence that ends the parse comes first.  The inverse of the parse
// suffix array is not needed.
struct PrimaryArgs {
    const uint32_t *pid, *doff, *dlen, *isa;
    const uint2 *stat;
    uint32_t z;
    uint32_t *marks;
    uint32_t *counter;
};
__global__ void k_primary_marks(PrimaryArgs a)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t q0 = a.pid[0], len0 = a.dlen[q0];
    const uint32_t g0 = a.isa[a.doff[q0]];
    bool same = false;
    if (k < a.z && k != 0) {
        const uint32_t q = a.pid[k], lq = a.dlen[q];
        same = lq >= len0 && a.isa[a.doff[q] + lq - len0] == g0;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, same);
    if ((threadIdx.x & 31u) == 0 && k < a.z) a.marks[k >> 5] = m;
    if (k == 0) atomicAdd(a.counter, a.stat[g0].x);
    if (same && k + 1u == a.z) atomicAdd(a.counter, 1u);
}
__global__ void k_primary_count(const uint32_t *sa, const uint32_t *first, uint32_t z, const uint32_t *marks,
                                uint32_t *counter)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (z < 2u || blockIdx.x * blockDim.x >= first[1]) return;
    bool before = false;
    if (r < first[1]) {
        const uint32_t x = sa[r];            // the suffix after occurrence x - 1
        before = x > 1u && ((marks[(x - 1u) >> 5] >> ((x - 1u) & 31u)) & 1u);
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, before);
    if ((threadIdx.x & 31u) == 0 && m) atomicAdd(counter, (uint32_t)__popc(m));
}

template <typename E>
static void mixed_blocks(Storage *st, const uint8_t *dT, uint32_t n, int W, Phrases &ph, ParseOrder &pord,
                         const uint32_t *moff, const uint32_t *mb, const uint16_t *mc, const uint32_t *delta,
                         uint32_t B, uint32_t M, uint8_t *dOut, uint32_t n_out, const BatchText *bt)
{
    E *elem = slot<E>(st, S_ELEM0, M);
    E *elem_alt = slot<E>(st, S_ELEM1, M);
    const uint32_t z = ph.z;
    Emit e{pord.sa, pord.first, ph.pid, moff, ph.D, z};
    uint32_t *emq = slot<uint32_t>(st, S_TMP0, z);
    uint32_t *ecnt = slot<uint32_t>(st, S_TMP1, (size_t)z + 1);
    uint8_t *emp = (uint8_t *)slot<uint32_t>(st, S_TMP2, z / 4 + 1);
    k_emit_prep<<<grid_for(z, 256), 256, 0, st->stream>>>(e, ph.pidpc, dT, n, W, bt ? bt->ptid : nullptr,
                                                            bt ? bt->lastb : nullptr, emq, emp, ecnt);
    after_launch(st);
    // in-place exclusive scan of the counts; ecnt[z] = total
    device_scan<uint32_t, OpAdd>(st, z, LoadArr<uint32_t>{ecnt}, StoreArr<uint32_t>{ecnt}, false, ecnt + z);
    k_emit<E><<<grid_for(z, EM_T), EM_T, 0, st->stream>>>(z, ecnt, emq, emp, moff, mb, mc, elem, M, st->d_flags);
    after_launch(st);
    uint32_t *nv = nullptr, *nv2 = nullptr;
    // sort by block id; 8-bit digits unless the tuning asks for 10 (fewer
    // passes, larger tile histograms)
    if (st->tuning.mixed_radix_bits == 10) radix_sort<E, false, 10>(st, elem, elem_alt, nv, nv2, M, 8, 8 + bits_for(B - 1));
    else radix_sort<E, false, 8>(st, elem, elem_alt, nv, nv2, M, 8, 8 + bits_for(B - 1));
    probe_begin(st, GBWT_PROBE_MIXED_SCATTER);
    k_mixed_scatter<E><<<grid_for((M + 3) / 4, 256), 256, 0, st->stream>>>(elem, M, delta, B, dOut, n_out, st->d_flags);
    probe_end(st, GBWT_PROBE_MIXED_SCATTER, (uint64_t)M * (sizeof(E) + 1));
    after_launch(st);
}

uint32_t run_group_index(Storage *st, Phrases &ph, DictOrder &dord, int W, uint32_t *&grp_of)
{
    const uint32_t N = (uint32_t)ph.dict_bytes;
    PosInfo pi{ph.dphr, ph.doff, ph.dlen};
    uint8_t *mark = slot<uint8_t>(st, S_MB, N);
    uint32_t *gid = slot<uint32_t>(st, S_TMP0, N);
    check_cuda(cudaMemsetAsync(mark, 0, N, st->stream));
    k_mark_sheads<<<grid_for(N, 256), 256, 0, st->stream>>>(N, pi, (uint32_t)W, dord.isa, mark);
    after_launch(st);
    device_scan<uint32_t, OpAdd>(st, N, LoadMark{mark}, StoreGid{gid}, true, (uint32_t *)st->d_scalars);
    fetch_scalars(st, 1);
    const uint32_t G = (uint32_t)st->h_scalars[0];
    grp_of = slot<uint32_t>(st, S_GRP, N);
    k_group_of<<<grid_for(N, 256), 256, 0, st->stream>>>(N, pi, (uint32_t)W, dord.isa, gid, grp_of);
    after_launch(st);
    return G;
}

void run_assembly(Storage *st, const uint8_t *dT, uint32_t n, int W, Phrases &ph, DictOrder &dord, ParseOrder &pord,
                  uint8_t *dOut, uint32_t n_out, const BatchText *bt)
{
    const uint32_t N = (uint32_t)ph.dict_bytes;
    PosInfo pi{ph.dphr, ph.doff, ph.dlen};
    uint2 *stat = slot<uint2>(st, S_GCOUNT, (size_t)N + 1);
    check_cuda(cudaMemsetAsync(stat, 0, (size_t)N * sizeof(uint2), st->stream));
    k_group_stats<<<grid_for(N, 256), 256, 0, st->stream>>>(N, pi, (uint32_t)W, dord.isa, ph.dict, ph.occpc, stat);
    after_launch(st);
    const size_t nw = ((size_t)N + 31) / 32;
    uint32_t *heads = slot<uint32_t>(st, S_TMP0, nw), *mixed = slot<uint32_t>(st, S_TMP1, nw);
    device_scan<uint32_t, OpAdd>(st, N, LoadGCount{stat}, StoreGroup{stat, N, heads, mixed}, false,
                                 (uint32_t *)st->d_scalars);
    // a mixed block has at least two bytes
    uint32_t *delta = slot<uint32_t>(st, S_DELTA, (size_t)(N < n_out / 2 ? N : n_out / 2) + 1);
    device_scan<Sum4, OpAdd, 1>(st, nw, LoadMixWord{stat, heads, mixed}, StoreMixWord{stat, mixed, delta}, false,
                             (Sum4 *)(st->d_scalars + 1));
    fetch_scalars(st, 3);
    const uint32_t total = (uint32_t)st->h_scalars[0], M = (uint32_t)st->h_scalars[1];
    const uint32_t B = (uint32_t)(st->h_scalars[1] >> 32), G = (uint32_t)st->h_scalars[2];
    if (total != n_out || G == 0) throw Error{GBWT_INTERNAL_ERROR};
    st->stats.s = G;
    st->stats.mixed_blocks = B;
    st->stats.mixed_elems = M;
    stage_mark(st, 4);

    if (!bt) {
        uint32_t *marks = slot<uint32_t>(st, S_TMP2, ((size_t)ph.z + 31) / 32);
        k_primary_marks<<<grid_for(ph.z, 256), 256, 0, st->stream>>>(
            PrimaryArgs{ph.pid, ph.doff, ph.dlen, dord.isa, stat, ph.z, marks, st->d_flags + 2});
        after_launch(st);
        k_primary_count<<<grid_for(ph.z, 256), 256, 0, st->stream>>>(pord.sa, pord.first, ph.z, marks, st->d_flags + 2);
        after_launch(st);
    }
    const uint32_t long_cap = n_out / RF_LONG + 1u;
    uint32_t *longs = slot<uint32_t>(st, S_TILEG, long_cap);
    probe_begin(st, GBWT_PROBE_RUN_FILL);
    k_run_fill_groups<<<grid_for(N, 256), 256, 0, st->stream>>>(dOut, n_out, stat, N, longs, long_cap, st->d_flags);
    probe_end(st, GBWT_PROBE_RUN_FILL, (uint64_t)(n_out - M) + 8ull * N);
    after_launch(st);
    k_run_fill_long<<<st->num_sms * 4, 256, 0, st->stream>>>(dOut, n_out, stat, N, longs, st->d_flags + 5, long_cap);
    after_launch(st);
    stage_mark(st, 5);
    if (B == 0) return;

    // per-phrase mixed-suffix lists
    uint32_t *moff = slot<uint32_t>(st, S_MOFF, (size_t)ph.d + 1);
    uint32_t *mb = slot<uint32_t>(st, S_MB, N);
    uint16_t *mc = slot<uint16_t>(st, S_MC, N);
    uint32_t *words = slot<uint32_t>(st, S_TMP2, nw), *pre = heads;      // heads are counted
    k_mix_flags<<<grid_for(N, 256), 256, 0, st->stream>>>(N, pi, (uint32_t)W, dord.isa, mixed, words);
    after_launch(st);
    device_scan<uint32_t, OpAdd>(st, nw, LoadPopc{words}, StoreArr<uint32_t>{pre}, false, moff + ph.d);
    k_mix_offsets<<<grid_for(ph.d, 256), 256, 0, st->stream>>>(ph.d, ph.doff, words, pre, moff);
    after_launch(st);
    k_mix_entries<<<grid_for(N, 256), 256, 0, st->stream>>>(N, ph.dphr, ph.doff, ph.dict, dord.isa, stat, words, pre,
                                                            mb, mc);
    after_launch(st);
    if (B < (1u << 24)) mixed_blocks<uint32_t>(st, dT, n, W, ph, pord, moff, mb, mc, delta, B, M, dOut, n_out, bt);
    else mixed_blocks<uint64_t>(st, dT, n, W, ph, pord, moff, mb, mc, delta, B, M, dOut, n_out, bt);
}

}  // namespace gbwt
