"""Host logic around an entry point's work (csrc/guard.h), on the CPU with a fake runtime."""
import fake_util

FAKES = r"""
#include <stdio.h>
#include <string.h>
#include <stdexcept>
#include <string>
#include "guard.h"
std::string events;
static void ev(const char* x) { events += x; events += ' '; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { ev(s == (cudaStream_t)1 ? "sync-main" : "sync-copy"); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)2; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaMallocHost(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); ev("clear"); return cudaSuccess; }
namespace fgss { void set_thread_error(const std::string&) {} }
using namespace fgss;
fgss_ctx ctx;
"""


def test_blocks_are_given_back_after_the_copies_into_them(tmp_path):
    """A failed call waits for both streams before what it had allocated for the caller is freed."""
    out = fake_util.run(tmp_path, FAKES + r"""
int main() {
    ctx.c.stream = (cudaStream_t)1;
    ctx.c.copy_stream = (cudaStream_t)2;
    for (int kind = 0; kind < 3; kind++) {
        events.clear();
        const fgss_status st = guard(&ctx, [&] {
            or_undo(ctx.c, [&] {
                ev("copy");
                if (kind == 0) fail(FGSS_ERR_NOMEM, "second copy");
                if (kind == 1) throw std::bad_alloc();
                throw std::runtime_error("x");
            }, [&] { ev("free"); });
        });
        printf("%d %s\n", (int)st, events.c_str());
    }
    events.clear();
    const fgss_status st = guard(&ctx, [&] { or_undo(ctx.c, [&] { ev("copy"); }, [&] { ev("free"); }); });
    printf("%d %s\n", (int)st, events.c_str());
}
""").splitlines()
    for line, status in zip(out[:3], ("3", "3", "2")):
        st, *events = line.split()
        assert st == status
        assert events[:4] == ["copy", "sync-main", "sync-copy", "free"], line
    assert out[3].split() == ["0", "copy"]


def test_a_wait_that_gave_up_fails_its_call_only(tmp_path):
    """The word that a device wait sets stops the call at its next wait, before anything read back is
    used, and is clear for the next call whatever the failed one ended with."""
    out = fake_util.run(tmp_path, FAKES + r"""
int main() {
    uint32_t word = 0;
    ctx.c.stream = (cudaStream_t)1;
    ctx.c.err_host = &word;
    auto good = [&] { return (int)guard(&ctx, [&] { ctx.c.sync(); }); };
    int used = 0;
    int st = guard(&ctx, [&] { word = 1; ctx.c.sync(); used = 1; });
    printf("at a wait %d used %d word %u next %d\n", st, used, word, good());
    st = guard(&ctx, [&] { word = 1; });
    printf("at the end %d word %u next %d\n", st, word, good());
    st = guard(&ctx, [&] { word = 1; fail(FGSS_ERR_NOMEM, "other"); });
    printf("other reason %d word %u next %d\n", st, word, good());
    st = guard(&ctx, [&] { word = 1; throw std::bad_alloc(); });
    printf("host memory %d word %u next %d\n", st, word, good());
    printf("message '%s'\n", ctx.c.last_error.c_str());
}
""")
    assert out.splitlines() == ["at a wait 7 used 0 word 0 next 0", "at the end 7 word 0 next 0",
                                "other reason 3 word 0 next 0", "host memory 3 word 0 next 0", "message ''"]


def test_training_runs_under_the_guard():
    """fgss_model_train joins on the device like the joins' own entry points."""
    import os
    src = open(os.path.join(fake_util.CSRC, "model_api.cu")).read()
    body = src[src.index("fgss_status fgss_model_train("):src.index("int fgss_model_num_params")]
    assert "return guard(ctx," in body
