// Radix scatters with right and with wrong digit counts: the stable order, and
// an error bit in place of stores past the keys.  The buffers are four times
// as long as the keys, so a store past the keys lands in bytes that are checked.
#include "prims.cuh"
#include <algorithm>
#include <stdio.h>
#include <vector>
using namespace gbwt;

static int failures = 0;
static void expect(bool ok, const char *what, const char *kind, int bits)
{
    if (!ok) { printf("%s: %s, %d-bit digits\n", what, kind, bits); failures++; }
}

template <typename T> static T *device(const std::vector<T> &h)
{
    T *p = nullptr;
    check_cuda(cudaMalloc(&p, h.size() * sizeof(T)));
    check_cuda(cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return p;
}
template <typename T> static std::vector<T> host(const T *p, size_t n)
{
    std::vector<T> h(n);
    check_cuda(cudaMemcpy(h.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost));
    return h;
}

template <typename K, bool HAS_VAL, int BITS, int BALLOT> static void run(uint32_t n, bool look_back_form, bool wrong)
{
    constexpr uint32_t D = 1u << BITS;
    const uint32_t tiles = (n + RS_TILE - 1) / RS_TILE, room = 4 * n, mask = D - 1u;
    const int shift = 3;
    const char *kind = look_back_form ? "look-back" : "histograms";
    std::vector<K> keys(room, (K)0);
    std::vector<uint32_t> vals(room, 0u);
    uint64_t x = 88172645463325252ull + n;
    for (uint32_t i = 0; i < n; i++) {
        x ^= x << 13; x ^= x >> 7; x ^= x << 17;
        keys[i] = (K)x;
        vals[i] = i;
    }
    auto digit = [&](K k) { return (uint32_t)(k >> shift) & mask; };
    // counts: per digit (look-back), or offsets per digit and tile (histograms)
    std::vector<uint32_t> counts(look_back_form ? D : D * tiles, 0u);
    for (uint32_t i = 0; i < n; i++) counts[look_back_form ? digit(keys[i]) : digit(keys[i]) * tiles + i / RS_TILE]++;
    if (!look_back_form) {
        uint32_t run = 0;
        for (uint32_t &c : counts) { const uint32_t q = c; c = run; run += q; }
    }
    if (wrong) {                                     // what comes after the middle digit moves past the keys
        if (look_back_form) counts[D / 2] += n;
        else for (uint32_t i = D / 2 * tiles + 1; i < D * tiles; i++) counts[i] += n;
    }
    K *kin = device(keys), *kout = device(std::vector<K>(room, (K)~(K)0));
    uint32_t *vin = device(vals), *vout = device(std::vector<uint32_t>(room, ~0u));
    uint32_t *dc = device(counts), *words = device(std::vector<uint32_t>(8, 0u));
    uint64_t *status = device(std::vector<uint64_t>((size_t)tiles * D, 0ull));
    const size_t smem = rs_smem_bytes<K, HAS_VAL, BITS>();
    if (look_back_form) {
        check_cuda(cudaFuncSetAttribute(k_rs_pass<K, HAS_VAL, BITS, BALLOT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const LookBack lb{status, tiles, 1u, words + 2, words + 4};
        k_rs_pass<K, HAS_VAL, BITS, BALLOT><<<tiles, RS_THREADS, smem>>>(kin, kout, vin, vout, n, shift, mask, dc,
                                                                        RsSegs(), lb, words);
    } else {
        check_cuda(cudaFuncSetAttribute(k_rs_downsweep<K, HAS_VAL, BITS, BALLOT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_rs_downsweep<K, HAS_VAL, BITS, BALLOT><<<tiles, RS_THREADS, smem>>>(kin, kout, vin, vout, n, shift, mask, dc,
                                                                             tiles, RsSegs(), words);
    }
    check_cuda(cudaGetLastError());
    check_cuda(cudaDeviceSynchronize());
    const std::vector<uint32_t> w = host(words, 8);
    const std::vector<K> ko = host(kout, room);
    const std::vector<uint32_t> vo = host(vout, room);
    bool outside = false;
    for (uint32_t i = n; i < room; i++) outside = outside || ko[i] != (K)~(K)0 || vo[i] != ~0u;
    expect(!outside, "a store past the keys", kind, BITS);
    expect(w[4] == 0, "a wait gave up", kind, BITS);
    expect(w[0] == (wrong ? (uint32_t)ERR_INTERNAL : 0u), wrong ? "no error bit" : "an error bit", kind, BITS);
    std::vector<uint32_t> order(vals.begin(), vals.begin() + n);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return digit(keys[a]) < digit(keys[b]); });
    bool same = true;
    for (uint32_t i = 0; i < n; i++) {
        if (wrong && digit(keys[order[i]]) >= D / 2) break;
        same = same && ko[i] == keys[order[i]] && (!HAS_VAL || vo[i] == order[i]);
    }
    expect(same, "wrong order", kind, BITS);
    cudaFree(kin); cudaFree(kout); cudaFree(vin); cudaFree(vout); cudaFree(dc); cudaFree(words); cudaFree(status);
}

template <typename K, bool HAS_VAL, int BITS, int BALLOT> static void all()
{
    for (uint32_t n : {4097u, 8192u, 9005u, 70001u})
        for (bool form : {true, false})
            for (bool wrong : {false, true}) run<K, HAS_VAL, BITS, BALLOT>(n, form, wrong);
}

int main()
{
    try {
        all<uint32_t, false, 8, 0>();
        all<uint32_t, false, 8, 2>();
        all<uint32_t, false, 8, 3>();
        all<uint32_t, false, 9, 0>();
        all<uint32_t, false, 9, 2>();
        all<uint32_t, false, 9, 3>();
        all<uint32_t, false, 10, 0>();
        all<uint64_t, false, 8, 3>();
        all<uint64_t, false, 9, 3>();
        all<uint32_t, true, 8, 0>();
        all<uint64_t, true, 8, 0>();
    } catch (const Error &e) {
        printf("CUDA error\n");
        return 2;
    }
    printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
