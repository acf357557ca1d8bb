// guard.h -- what an entry point does around its work: the library's internal
// errors become a status, and nothing that a failed call queued outlives it.
#pragma once

#include <new>

#include "ctx.h"

namespace fgss {

// Message for fgss_last_error(NULL) (api.cu).
void set_thread_error(const std::string& msg);

// Waits for everything the context has queued: copies from or to the caller's
// page-locked arrays, and to blocks that are about to be given back.
inline void settle(Ctx& c) {
    if (c.stream && cudaStreamSynchronize(c.stream) != cudaSuccess) (void)cudaGetLastError();
    if (c.copy_stream && cudaStreamSynchronize(c.copy_stream) != cudaSuccess) (void)cudaGetLastError();
}

// Runs f.  Where it throws, waits for what it queued, then runs undo, which gives
// back what f had allocated for the caller (a block of the page-locked pool may
// be another thread's the moment it is given back), and throws on.
template <typename F, typename U>
void or_undo(Ctx& c, F&& f, U&& undo) {
    try {
        f();
    } catch (...) {
        settle(c);
        undo();
        throw;
    }
}

// Runs f and returns its status.  A wait of a scan or sort that gave up is looked
// at wherever the call waits for the stream (Ctx::sync), before anything read back
// is used, and here once more; every failed call, whatever its reason, leaves the
// words clear for the next one.
template <typename F>
fgss_status guard(fgss_ctx* ctx, F&& f) {
    fgss_status st = FGSS_ERR_CUDA;
    std::string msg;
    try {
        f();
        if (ctx) ctx->c.check_waits();
        if (ctx) ctx->c.last_error.clear();
        return FGSS_OK;
    } catch (const Error& e) {
        st = e.st;
        msg = e.msg;
        set_thread_error(e.msg);
    } catch (const std::bad_alloc&) {
        st = FGSS_ERR_NOMEM;
        msg = "host allocation failed";
    } catch (...) {
        msg = "unknown error";
    }
    if (ctx) {
        settle(ctx->c);
        ctx->c.clear_waits();
        ctx->c.last_error = msg;
    }
    return st;
}

}  // namespace fgss
