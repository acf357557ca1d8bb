// tokenize.h -- GPU tokenizer (tokenize.cu).
#pragma once

#include "ctx.h"

namespace fgss {

struct TokParams {
    int q;
    int mode;      // 0 q-grams, 1 canonical k-mers
    int pad;
    int pad_char;
    int suffix;
    int lower;
};

// The caller's options (null: the defaults).  Every mode but FGSS_TOK_QGRAM is k-mers:
// the kernels and the limits on q tell the two apart by 0 and 1 alone.
inline TokParams tok_params(const fgss_tok_opts* opts) {
    fgss_tok_opts o;
    fgss_tok_opts_default(&o);
    if (opts) o = *opts;
    return {o.q, o.mode == FGSS_TOK_QGRAM ? 0 : 1, o.pad, o.pad_char, o.suffix, o.lower};
}

// Text -> sets in MEMORY order (host arrays malloc'd into *out).
void tokenize_device(Ctx& c, const char* text, uint64_t n_bytes, const TokParams& p, fgss_sets* out);

}  // namespace fgss
