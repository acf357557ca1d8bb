// join.cu -- host driver of the self-join stages (see join_kernels.cuh for
// the device side and the reference file:line of each stage).
#include <string.h>

#include <algorithm>

#include "join.h"
#include "pinned.h"
#include "prims.cuh"

namespace fgss {

namespace {

template <typename T>
void upload(Ctx& c, T* dst, const std::vector<T>& v) {
    FGSS_CK(cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, c.stream));
}

}  // namespace

int bits_for(uint64_t v) {
    int b = 1;
    while (b < 64 && (1ull << b) < v) b++;
    return b;
}

DevBounds device_bounds(Ctx& c, float t, int mode) {
    uint32_t bits;
    memcpy(&bits, &t, 4);
    std::string k = "lut." + std::to_string(bits) + "." + std::to_string(mode) + ".";
    const size_t L = kMaxLen + 1, S = 2 * (size_t)kMaxLen + 1;
    bool fresh = c.bufs.find(k + "probe") == c.bufs.end();
    DevBounds d;
    d.probe = c.devT<uint16_t>(k + "probe", L);
    d.index = c.devT<uint16_t>(k + "index", L);
    d.minsz = c.devT<uint32_t>(k + "minsz", L);
    d.maxsz = c.devT<uint32_t>(k + "maxsz", L);
    d.lmin = c.devT<uint32_t>(k + "lmin", L);
    d.cand_min = c.devT<uint32_t>(k + "cand", S);
    d.inter_min = c.devT<uint32_t>(k + "inter", S);
    d.need = c.devT<uint32_t>(k + "need", S);
    d.smin = c.devT<uint4>(k + "smin", S);
    if (fresh) {
        BoundTables b;
        compute_bounds(t, mode, b);
        std::vector<uint16_t>& pm = c.probe_max[k];
        pm = b.probe;
        for (size_t i = 1; i < pm.size(); i++) pm[i] = std::max(pm[i], pm[i - 1]);
        upload(c, d.probe, b.probe);
        upload(c, d.index, b.index);
        upload(c, d.minsz, b.minsz);
        upload(c, d.maxsz, b.maxsz);
        upload(c, d.lmin, b.lmin);
        upload(c, d.cand_min, b.cand_min);
        upload(c, d.inter_min, b.inter_min);
        upload(c, d.need, b.need);
        std::vector<uint4> sm(S);
        for (size_t i = 0; i < S; i++) sm[i] = make_uint4(b.cand_min[i], b.inter_min[i], b.need[i], 0u);
        upload(c, d.smin, sm);
        c.sync();  // the host vectors go out of scope
    }
    d.probe_max = c.probe_max[k].data();
    return d;
}

fgss_sets_view sets_to_device(Ctx& c, const std::string& name, const fgss_sets_view& v) {
    const uint32_t* host[4] = {v.id, v.pos, v.len, v.tokens};
    const uint64_t bytes[4] = {v.id ? v.n_sets * 4 : 0, v.n_sets * 4, v.n_sets * 4, v.n_tokens * 4};
    uint64_t off[4], total = 0;
    uintptr_t lo = UINTPTR_MAX, hi = 0;
    for (int k = 0; k < 4; k++) {
        off[k] = total;
        total += (bytes[k] + 4 + 255) & ~uint64_t(255);
        if (bytes[k] == 0) continue;
        lo = std::min(lo, (uintptr_t)host[k]);
        hi = std::max(hi, (uintptr_t)host[k] + bytes[k]);
    }
    // Columns side by side in one page-locked block (the library's own token sets): one copy of
    // their span instead of four (48 joins of titles 7.7 -> 7.0 ms, 1,000 titles 289 -> 272 us).
    const bool one = hi > lo && hi - lo <= total + 1024 && pinned_holds((const void*)lo, hi - lo);
    char* d = (char*)c.dev(name, std::max<uint64_t>(total, one ? hi - lo : 0) + 256);
    if (one) {
        FGSS_CK(cudaMemcpyAsync(d, (const void*)lo, hi - lo, cudaMemcpyHostToDevice, c.stream));
        for (int k = 0; k < 4; k++)
            if (bytes[k]) off[k] = (uintptr_t)host[k] - lo;
    } else {
        for (int k = 1; k <= 4; k++)
            if (bytes[k % 4])
                FGSS_CK(cudaMemcpyAsync(d + off[k % 4], host[k % 4], bytes[k % 4], cudaMemcpyHostToDevice, c.stream));
    }
    fgss_sets_view w = v;
    w.id = v.id ? (const uint32_t*)(d + off[0]) : nullptr;
    w.pos = (const uint32_t*)(d + off[1]);
    w.len = (const uint32_t*)(d + off[2]);
    w.tokens = (const uint32_t*)(d + off[3]);
    w.on_device = 1;
    return w;
}

void join_setup_host(Ctx& c, JoinState& J, const fgss_sets_view& v, const fgss_join_opts& o, int slot) {
    J.slot = slot;
    J.t = o.threshold;
    J.res_cap_user = o.result_capacity;
    J.bounds = o.bounds;
    J.filter = o.filter;
    if (o.filter < FGSS_FILTER_AUTO || o.filter > FGSS_FILTER_GLOBAL) fail(FGSS_ERR_INVALID, "unknown filter strategy");
    if (!(o.threshold > 0.0f && o.threshold < 1.0f))
        fail(FGSS_ERR_INVALID, "threshold must be in (0, 1) (fgssjoin_cli.cu:31-35)");
    if (v.n_sets >= 0xffffffffull) fail(FGSS_ERR_UNSUPPORTED, "more than 2^32-1 records");
    if (v.n_tokens >= 0xffffffffull) fail(FGSS_ERR_UNSUPPORTED, "more than 2^32-1 tokens");
    const uint64_t n = v.n_sets;
    J.in = v.on_device ? v : sets_to_device(c, J.pfx("in"), v);
    J.id = J.in.id;
    J.lut = device_bounds(c, J.t, J.bounds);

    JoinArgs& a = J.args;
    memset(&a, 0, sizeof a);
    a.pos = J.in.pos;
    a.len = J.in.len;
    a.tok = J.in.tokens;
    a.n = (uint32_t)n;
    a.n_terms = v.n_terms;
    a.n_tokens = v.n_tokens;
    a.probe = J.lut.probe;
    a.index = J.lut.index;
    a.minsz = J.lut.minsz;
    a.maxsz = J.lut.maxsz;
    a.cand_min = J.lut.cand_min;
    a.inter_min = J.lut.inter_min;
    a.need = J.lut.need;
    a.lmin = J.lut.lmin;
    a.id = J.id;
    a.thr = J.t;
    a.side = J.side;
    a.heavy_cap = (uint32_t)n;
    a.join_id = (uint32_t)slot;
    a.heavy_min_qp = 0xffffffffu;  // set by the batched method's launch shape
    if (o.query_end > o.query_begin) {
        if (o.query_end > n) fail(FGSS_ERR_INVALID, "query_end beyond the number of records");
        a.q_lo = (uint32_t)o.query_begin;
        a.q_hi = (uint32_t)o.query_end;
    } else {
        a.q_lo = 0;
        a.q_hi = (uint32_t)n;
    }
}

void check_input_status(uint32_t st) {
    if (st & ST_BAD_OFFSETS) fail(FGSS_ERR_FORMAT, "a record's pos + len exceeds n_tokens");
    if (st & ST_TOO_LONG) fail(FGSS_ERR_UNSUPPORTED, "a record has more than 65535 tokens");
    if (st & ST_BAD_TOKENS)
        fail(FGSS_ERR_FORMAT, "tokens must be strictly ascending inside each record and below n_terms");
}

void apply_status(JoinState& J, uint32_t st, const unsigned long long* stats) {
    J.status_host = st;
    memcpy(J.stats_host, stats, sizeof(J.stats_host));
    if (J.status_host & ST_TOO_LONG) fail(FGSS_ERR_UNSUPPORTED, "a record has more than 65535 tokens");
    if (J.status_host & ST_BAD_TOKENS)
        fail(FGSS_ERR_FORMAT, "tokens must be strictly ascending inside each record and below n_terms");
    if (J.status_host & (ST_HASH_FULL | ST_HEAVY_OVERFLOW))
        fail(FGSS_ERR_CUDA, "internal table overflow in the filter (status " + std::to_string(J.status_host) + ")");
}

HeavyScratch heavy_scratch(Ctx& c, const std::string& prefix, uint64_t n, uint32_t slots, bool capture) {
    HeavyScratch h;
    h.zero_words = (2 * n + 63) & ~63ull;
    h.aux_words = (2 * n + 65536 + 65537 + 63) & ~63ull;
    const std::string zn = prefix + "heavy.zero";
    auto it = c.bufs.find(zn);
    const size_t need = h.zero_words * slots * 4;
    const bool grow = it == c.bufs.end() || it->second.bytes < need;
    if (grow && capture) fail(FGSS_ERR_CUDA, "heavy scratch would grow inside a graph capture");
    h.zero = (uint32_t*)c.dev(zn, need);
    if (grow) FGSS_CK(cudaMemsetAsync(h.zero, 0, c.bufs[zn].bytes, c.stream));
    h.aux = c.devT<uint32_t>(prefix + "heavy.aux", h.aux_words * slots);
    return h;
}

void join_output(Ctx& c, JoinState& J, uint64_t* keys, uint32_t* vals, const uint64_t* d_n, uint64_t n_cap) {
    const uint64_t n = J.in.n_sets;
    J.out_col = out_column(n_cap);
    J.oq = c.devT<uint32_t>(J.pfx("o"), 6 * J.out_col);
    J.os = J.oq + J.out_col;
    J.oidq = J.oq + 2 * J.out_col;
    J.oids = J.oq + 3 * J.out_col;
    J.oo = J.oq + 4 * J.out_col;
    J.osim = reinterpret_cast<float*>(J.oq + 5 * J.out_col);
    if (n_cap == 0) return;
    const int qb = bits_for(n);  // keys are q << qb | s
    radix_sort<uint64_t, uint32_t>(c, keys, vals, n_cap, d_n, 0, 2 * qb, J.pfx("rsort").c_str());
    k_result_out<<<grid_for(n_cap, 256, c.num_sms * 32), 256, 0, c.stream>>>(
        keys, vals, d_n, (uint32_t)qb, J.id, J.in.len, J.oq, J.os, J.oidq, J.oids, J.oo, J.osim, c.err_dev);
    FGSS_LAUNCH_CK();
}

}  // namespace fgss
