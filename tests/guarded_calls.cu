// guarded(): what a failed call leaves behind.  A wait that gave up in work that
// the call had queued belongs to that call, however it ended, and must not fail
// the next one.  Runs without a GPU (no stream, the word in host memory).
#include "gbwt_api.cu"

int main()
{
    Storage st;
    uint32_t word = 0;
    st.h_err = &word;
    int failures = 0;
    auto expect = [&](bool ok, const char *what) {
        if (!ok) { printf("%s\n", what); failures++; }
    };
    int64_t rc = guarded(&st, [&]() -> int64_t { word = 1; throw Error{GBWT_GPU_NOT_ENOUGH_MEMORY}; });
    expect(rc == GBWT_GPU_NOT_ENOUGH_MEMORY, "code of a thrown error");
    expect(word == 0, "given-up wait kept after a thrown error");
    rc = guarded(&st, [&]() -> int64_t { word = 1; throw std::bad_alloc(); });
    expect(rc == GBWT_NOT_ENOUGH_MEMORY && word == 0, "given-up wait kept after a failed host allocation");
    rc = guarded(&st, [&]() -> int64_t { word = 1; return GBWT_BAD_PARAMETER; });
    expect(rc == GBWT_BAD_PARAMETER && word == 0, "given-up wait kept after a returned error");
    rc = guarded(&st, [&]() -> int64_t { return 17; });
    expect(rc == 17, "result");
    st.h_err = nullptr;                    // the storage failed before it had the word
    rc = guarded(&st, [&]() -> int64_t { throw Error{GBWT_GPU_ERROR}; });
    expect(rc == GBWT_GPU_ERROR, "error without the word");
    printf("%d failures\n", failures);
    return failures ? 1 : 0;
}
