// level2_taken FILE W P: whether the parse of the text is parsed again (1) or the
// plain suffix sort runs (0).
#include "gbwt_internal.cuh"
#include <stdio.h>
#include <stdlib.h>
#include <vector>
using namespace gbwt;

int main(int argc, char **argv)
{
    if (argc != 4) return 2;
    FILE *f = fopen(argv[1], "rb");
    if (!f) return 2;
    std::vector<uint8_t> t(1 << 25);
    t.resize(fread(t.data(), 1, t.size(), f));
    fclose(f);
    const uint32_t n = (uint32_t)t.size();
    const int W = atoi(argv[2]), P = atoi(argv[3]);
    void *p = nullptr;
    if (gbwt_allocate_device_storage(&p, 0) != GBWT_NO_ERROR) return 2;
    Storage *st = (Storage *)p;
    try {
        uint8_t *dT = nullptr;
        check_cuda(cudaMalloc(&dT, (size_t)n + 16));
        check_cuda(cudaMemcpy(dT, t.data(), n, cudaMemcpyHostToDevice));
        check_cuda(cudaMemsetAsync(st->d_flags, 0, 64 * sizeof(uint32_t), st->stream));
        uint32_t *D = nullptr;
        Phrases ph;
        ph.z = run_trigger_scan(st, dT, n, W, P, false, D);
        ph.D = D;
        run_phrases(st, dT, n, W, ph);
        DictOrder dord;
        run_dict_sort(st, ph, W, false, dord);
        ParseOrder pord;
        st->round_words = 42;
        const bool taken = run_parse_sa_level2(st, ph, dord, pord, nullptr);
        sync_stream(st);
        printf("%d z %u d %u\n", taken ? 1 : 0, ph.z, ph.d);
        cudaFree(dT);
    } catch (const Error &e) {
        printf("error %lld\n", (long long)e.code);
        return 2;
    }
    return gbwt_free_device_storage(p) == GBWT_NO_ERROR ? 0 : 2;
}
