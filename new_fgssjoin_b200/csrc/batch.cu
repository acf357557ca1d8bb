// batch.cu -- the batched method: every join of a batch in one launch per
// stage (per-record counts, index, windows, bitmaps; where they are needed
// features, learned estimates, work-item costs, items, chunk splits; one
// filter+verify launch per class of queries, one global-accumulator launch,
// result keys, sort, output), presized result buffers with an exact re-run on
// overflow; and the plain method's filter and verification of one join.
#include <string.h>

#include <algorithm>
#include <cmath>

#include "batch_kernels.cuh"
#include "join.h"
#include "model.h"
#include "prims.cuh"

namespace fgss {

static_assert(kFeatures == kFeat, "model feature rows");

// Warp per record: the learned model's features of one join (training rows,
// model_api.cu), the same as the batch's k_features_mj.
__global__ void k_features(JoinArgs a, float* __restrict__ feat) {
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < a.n; q += warps)
        features_record(a, q, feat + (uint64_t)q * kFeatures);
}

// (By an order that a sort gave up on, the items stay as they are.)
__global__ void k_permute_items(const uint4* __restrict__ items, const uint32_t* __restrict__ order, uint64_t n,
                                uint4* __restrict__ out, const uint32_t* __restrict__ err) {
    const bool as_is = gave_up(err);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = items[as_is ? i : order[i]];
}

template <int NT, int HLOG, int RT>
static int resident_ctas(Ctx& c) {
    int occ = 0;
    FGSS_CK(cudaFuncSetAttribute(k_fused<NT, HLOG, RT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)FusedLayout<HLOG>::bytes));
    FGSS_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fused<NT, HLOG, RT, false>, NT,
                                                          FusedLayout<HLOG>::bytes));
    return std::max(occ, 1) * c.num_sms;
}

int fused_resident_ctas(Ctx& c, const TuneEntry& te) {
#define FGSS_R(NT, HL, RT) \
    if (te.threads == NT && te.hash_log2 == HL && te.regs_rt == RT) return resident_ctas<NT, HL, RT>(c);
    FGSS_R(32, 8, 1024)
    FGSS_R(32, 9, 1024)
    FGSS_R(64, 9, 1024)
    FGSS_R(64, 9, 768)
    FGSS_R(64, 10, 1024)
    FGSS_R(128, 9, 1024)
    FGSS_R(128, 10, 1024)
    FGSS_R(128, 10, 768)
    FGSS_R(128, 11, 768)
    FGSS_R(128, 11, 896)
    FGSS_R(256, 11, 768)
    FGSS_R(256, 12, 768)
#undef FGSS_R
    return resident_ctas<64, 9, 768>(c);
}

template <int NT, int HLOG, int RT, bool SIDED>
static void launch_fused(Ctx& c, const JoinArgs* d_args, const FusedArgs* d_fargs, const uint4* items,
                         uint32_t n_items, uint32_t* counter, int ctas_per_sm) {
    static bool attr = false;
    const size_t smem = FusedLayout<HLOG>::bytes;
    if (!attr) {
        FGSS_CK(cudaFuncSetAttribute(k_fused<NT, HLOG, RT, SIDED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
        attr = true;
    }
    int occ = 0;
    FGSS_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fused<NT, HLOG, RT, SIDED>, NT, smem));
    if (occ < 1) occ = 1;
    const int per = ctas_per_sm > 0 ? std::min(occ, ctas_per_sm) : occ;
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)per * c.num_sms, std::max<uint32_t>(n_items, 1));
    k_fused<NT, HLOG, RT, SIDED><<<grid, NT, smem, c.stream>>>(d_args, d_fargs, items, n_items, counter);
    FGSS_LAUNCH_CK();
}

// Launch shapes the autotuner chooses from: CTA size, slot-table log2 size,
// resident threads per SM the register budget is sized for.
extern const int kFusedShapes[][3] = {{32, 8, 1024},  {32, 9, 1024},  {64, 9, 1024},   {64, 9, 768},
                                      {64, 10, 1024}, {128, 9, 1024}, {128, 10, 1024}, {128, 10, 768},
                                      {128, 11, 768}, {256, 11, 768},  {256, 12, 768}, {128, 11, 896}};
extern const int kNumFusedShapes = 12;

// The launch shape that stands for a requested filter strategy.
TuneEntry filter_entry(int filter) {
    TuneEntry te;
    te.threads = filter == FGSS_FILTER_WARP ? 32 : 128;
    te.hash_log2 = filter == FGSS_FILTER_WARP ? 9 : 11;
    te.regs_rt = filter == FGSS_FILTER_WARP ? 1024 : 768;
    te.ctas_per_sm = 0;
    te.heavy_min_probe = filter == FGSS_FILTER_GLOBAL ? 1 : 0;
    return te;
}

// The strategy a tuned entry amounts to (the claim kernels: a CTA per query, but for few entries).
int filter_of(const TuneEntry& te) {
    return te.heavy_min_probe == 1 ? FGSS_FILTER_GLOBAL : te.threads == 32 ? FGSS_FILTER_WARP : FGSS_FILTER_CTA;
}

// sided: the batch is an R-S join (its records carry a side byte)
void fused_launch(Ctx& c, const TuneEntry& te, const JoinArgs* d_args, const FusedArgs* d_fargs, const uint4* items,
                  uint32_t n_items, uint32_t* counter, bool sided) {
#define FGSS_F(NT, HL, RT)                                                                               \
    if (te.threads == NT && te.hash_log2 == HL && te.regs_rt == RT) {                                    \
        if (sided) launch_fused<NT, HL, RT, true>(c, d_args, d_fargs, items, n_items, counter, te.ctas_per_sm); \
        else launch_fused<NT, HL, RT, false>(c, d_args, d_fargs, items, n_items, counter, te.ctas_per_sm);      \
        return;                                                                                          \
    }
    FGSS_F(32, 8, 1024)
    FGSS_F(32, 9, 1024)
    FGSS_F(64, 9, 1024)
    FGSS_F(64, 9, 768)
    FGSS_F(64, 10, 1024)
    FGSS_F(128, 9, 1024)
    FGSS_F(128, 10, 1024)
    FGSS_F(128, 10, 768)
    FGSS_F(128, 11, 768)
    FGSS_F(128, 11, 896)
    FGSS_F(256, 11, 768)
    FGSS_F(256, 12, 768)
#undef FGSS_F
    if (sided) launch_fused<64, 9, 768, true>(c, d_args, d_fargs, items, n_items, counter, te.ctas_per_sm);
    else launch_fused<64, 9, 768, false>(c, d_args, d_fargs, items, n_items, counter, te.ctas_per_sm);
}

namespace {

// k_claim's shapes: 256 consumer threads, 8192 claim slots, 6 entries a thread or 8
// (wide), 3 CTAs per SM (53 and 59 KB of shared memory each: at 66 KB and more the L1
// that is left costs 10 %).  The wide shape has fewer steps, the other
// less to lay out for a short one and fewer spills (80 bytes stored and 88 loaded a thread, the
// wide one 116 and 96; 92 and 108, 128 and 116 with sides).  6 / 8 entries, kernel time: 1,000,000
// heavy-tailed records at t = 0.7 (5,350 window entries a query) 99.9 / 94.9 ms;
// 100,000 titles at t = 0.5 (3,356) 4.14 / 4.24; R-S of 2 x 60,000 titles at t = 0.6
// 3.44 / 3.47; 150,000 heavy-tailed records at t = 0.85 (86) 0.54 / 0.58; 100,000 titles
// at t = 0.7, plain 1.53 / 1.83.  (5 entries: 104.7, 4.14, 3.36, 0.52, 1.55; 4096 slots: 103.0,
// 4.40, 3.46, 0.56, 1.58 with 6; 4 CTAs of 56 registers lose everywhere.)
using Claim = ClaimShape<256, 6, 13>;
using ClaimWide = ClaimShape<256, 8, 13>;
constexpr int kClaimCtas = 3;
// Average cost (k_cost_mj) of k_claim's queries from which it is wide: between the averages
// 3,356 and 5,350 above, nothing nearer was timed.  Without costs (a light call, the plain
// method) it is narrow.
constexpr uint64_t kClaimWideCost = 4096;

template <class Shape, int MODE, bool SIDED>
void claim_launch_as(Ctx& c, const JoinArgs* d_args, const FusedArgs* d_fargs, const ClaimItems& items,
                     uint32_t* counter) {
    FGSS_CK(cudaFuncSetAttribute(k_claim<Shape, kClaimCtas, MODE, SIDED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Shape::bytes));
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)kClaimCtas * c.num_sms, items.n);
    k_claim<Shape, kClaimCtas, MODE, SIDED><<<grid, Shape::NT, Shape::bytes, c.stream>>>(d_args, d_fargs, items, counter);
    FGSS_LAUNCH_CK();
}

template <int MODE, class Shape = Claim>
void claim_launch(Ctx& c, const JoinArgs* d_args, const FusedArgs* d_fargs, const ClaimItems& items, uint32_t* counter,
                  bool sided) {
    if (sided) claim_launch_as<Shape, MODE, true>(c, d_args, d_fargs, items, counter);
    else claim_launch_as<Shape, MODE, false>(c, d_args, d_fargs, items, counter);
}

// m in tiles small enough to make at least `want` of them, but not below `low` records.
TileMap tiles_for(const TileMap& m, uint64_t want, uint32_t low) {
    uint32_t tile = m.tile;
    while (tile > low && (uint64_t)m.ntiles * (m.tile / tile) < want) tile >>= 1;
    return finer_tiles(m, tile);
}

// Tiles of the warp-per-record stages.  Records come in descending size, so a tile of
// the longest ones is the stage's critical path: small enough to give every resident CTA
// (8 of 8 warps on an SM) 4 tiles, as long as a warp still has a record (500 titles: k_windows_mj 40 -> 4.1 us,
// k_bitmaps_mj 32 -> 3.3, k_index_entries_mj 21 -> 2.9 with tiles of 8 instead of 256).
TileMap warp_tiles(Ctx& c, const TileMap& m) { return tiles_for(m, (uint64_t)32 * c.num_sms, 8); }

// Items of the records in order: about 128 per CTA.  Of one join, its query range
// only: an item costs a CTA an atomic and its records' classes even where it has no
// query (one query of 100,000 records: k_claim 237 us over all of them).
ClaimItems items_in_order(Ctx& c, const Batch& B) {
    const uint64_t want = (uint64_t)128 * kClaimCtas * c.num_sms;
    if (B.js.size() > 1) {
        const TileMap t = tiles_for(B.rec, want, 1);
        return {nullptr, t, 0, t.ntiles};
    }
    const JoinArgs& a = B.js[0]->args;
    uint32_t tile = B.rec.tile;
    while (tile > 1 && (a.q_hi - a.q_lo) / tile < want) tile >>= 1;
    const uint32_t first = a.q_lo / tile, end = (uint32_t)(((uint64_t)a.q_hi + tile - 1) / tile);
    return {nullptr, finer_tiles(B.rec, tile), first, end - first};
}

template <int MODE>
void tiny_launch(Ctx& c, const JoinArgs* d_args, const FusedArgs* d_fargs, const TileMap& m, bool sided) {
    // 4 tiles for each of the 16 CTAs an SM is given, down to a record per warp: the first
    // tiles hold the longest records (150,000 heavy-tailed ones 450 us at half a tile each,
    // 330 at 4, 315 at 8, where 500,000 reads lose: 765 -> 825; more CTAs lose everywhere)
    const TileMap t = tiles_for(finer_tiles(m, 32), (uint64_t)64 * c.num_sms, kTinyWarps);
    const unsigned grid = std::min<unsigned>(t.ntiles, (unsigned)c.num_sms * 16);
    if (sided) k_tiny<MODE, true><<<grid, kTinyWarps * 32, 0, c.stream>>>(d_args, d_fargs, t);
    else k_tiny<MODE, false><<<grid, kTinyWarps * 32, 0, c.stream>>>(d_args, d_fargs, t);
    FGSS_LAUNCH_CK();
}

constexpr uint32_t kRecTile = 256;  // records per tile of the per-record stages (thread per record in the MLP)

// Uploads the tile map of joins [off[j], off[j+1]) in tiles of `tile` to the
// device buffer `name` (through a pinned buffer of its own, so a captured
// graph's copy node always reads this map).
TileMap upload_tiles(Ctx& c, const std::string& name, const std::vector<uint64_t>& off, uint32_t tile) {
    const size_t nj = off.size() - 1;
    const size_t bytes = (nj + 1) * 12;
    char* h = (char*)c.pinned(name + ".h", bytes);
    uint64_t* ho = reinterpret_cast<uint64_t*>(h);
    uint32_t* ht = reinterpret_cast<uint32_t*>(h + (nj + 1) * 8);
    uint64_t t = 0;
    for (size_t j = 0; j < nj; j++) {
        ho[j] = off[j];
        ht[j] = (uint32_t)t;
        t += (off[j + 1] - off[j] + tile - 1) / tile;
    }
    ho[nj] = off[nj];
    if (t >= 0xffffffffull) fail(FGSS_ERR_UNSUPPORTED, "too many tiles in one batch");
    ht[nj] = (uint32_t)t;
    char* d = (char*)c.dev(name, bytes);
    FGSS_CK(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, c.stream));
    TileMap m;
    m.roff = reinterpret_cast<const uint64_t*>(d);
    m.tile_off = reinterpret_cast<const uint32_t*>(d + (nj + 1) * 8);
    m.nj = (uint32_t)nj;
    m.tile = tile;
    m.ntiles = (uint32_t)t;
    m.split = 1;
    return m;
}

// Every join's JoinArgs to the device, through the pinned buffer `name`.
void upload_args(Ctx& c, Batch& B, const std::string& name) {
    const size_t nj = B.js.size();
    JoinArgs* h = c.pinnedT<JoinArgs>(name, nj);
    for (size_t j = 0; j < nj; j++) h[j] = B.js[j]->args;
    FGSS_CK(cudaMemcpyAsync(B.d_args, h, nj * sizeof(JoinArgs), cudaMemcpyHostToDevice, c.stream));
}

unsigned tile_grid(Ctx& c, const TileMap& m, unsigned per_sm = 16) {
    return std::max<unsigned>(1, std::min<unsigned>(m.ntiles, (unsigned)c.num_sms * per_sm));
}

template <typename K>
void index_sort(Ctx& c, Batch& B, uint64_t E_cap, int tbits, int jbits, const uint64_t* d_E, const uint64_t* d_loff,
                uint32_t* list, const uint64_t* d_toff, uint32_t* tab, uint2* ent) {
    const std::string& p = c.bpfx;
    K* key = c.devT<K>(p + "b.ix.key", E_cap + 1);
    uint64_t* val = c.devT<uint64_t>(p + "b.ix.val", E_cap + 1);
    const TileMap wt = warp_tiles(c, B.rec);
    k_index_entries_mj<K><<<tile_grid(c, wt), 256, 0, c.stream>>>(B.d_args, wt, B.ioff, (uint32_t)tbits, key, val);
    FGSS_LAUNCH_CK();
    radix_sort<K, uint64_t>(c, key, val, E_cap, d_E, 0, tbits + jbits, (p + "b.ixsort").c_str());
    k_index_lists_mj<K><<<grid_for(E_cap, 256, c.num_sms * 32), 256, 0, c.stream>>>(
        B.d_args, key, val, d_E, (uint32_t)tbits, d_loff, list, d_toff, tab, ent, c.err_dev);
    FGSS_LAUNCH_CK();
}

// The batch's pre-pass, first part (index built): windows of every probe
// token (exact per-query work), the class of every query (pc: windows_query), the learned model's estimates (model) and the work-item costs
// (k_cost_mj).  d_sums: k_cost_mj's 2 nj + 4 sums, then the joins' predicted
// results (nj) and candidates (nj).
struct Prepass {
    uint2* win = nullptr;
    uint32_t* wpre = nullptr;
    uint32_t* wtot = nullptr;
    uint4* meta = nullptr;
    uint32_t* pred = nullptr;       // null without the model
    uint64_t* cost[2] = {};         // class QC_KEYED, QC_CLAIM
    uint64_t* d_sums = nullptr;
    size_t n_sums = 0;
};

// light: the windows and classes only.
Prepass batch_prepass(Ctx& c, Batch& B, uint32_t cap_entries, uint64_t P_cap, bool model, uint32_t pc, bool light = false) {
    const size_t nj = B.js.size();
    const std::string& p = c.bpfx;
    const uint64_t R = B.R;
    Prepass pp;
    pp.win = c.devT<uint2>(p + "b.win", P_cap + 1);
    pp.wpre = c.devT<uint32_t>(p + "b.wpre", P_cap + 1);
    pp.wtot = c.devT<uint32_t>(p + "b.wtot", R + 1);
    pp.meta = c.devT<uint4>(p + "b.meta", R + 1);
    const TileMap wt = warp_tiles(c, B.rec);
    const unsigned wg = tile_grid(c, wt);
    if (light) {
        if (R) {
            k_windows_mj<<<wg, 256, 0, c.stream>>>(B.d_args, wt, B.poff, pp.win, pp.wpre, pp.wtot, pp.meta, pc);
            FGSS_LAUNCH_CK();
        }
        return pp;
    }
    float* feat = c.devT<float>(p + "b.feat", (R + 1) * kFeatures);
    uint32_t* pred = c.devT<uint32_t>(p + "b.pred", R + 1);
    pp.cost[0] = c.devT<uint64_t>(p + "b.cost0", R + 1);
    pp.cost[1] = c.devT<uint64_t>(p + "b.cost1", R + 1);
    pp.n_sums = 4 * nj + 4;
    pp.d_sums = c.devT<uint64_t>(p + "b.sums", pp.n_sums);
    FGSS_CK(cudaMemsetAsync(pp.d_sums, 0, pp.n_sums * 8, c.stream));
    if (R == 0) return pp;
    k_windows_mj<<<wg, 256, 0, c.stream>>>(B.d_args, wt, B.poff, pp.win, pp.wpre, pp.wtot, pp.meta, pc);
    FGSS_LAUNCH_CK();
    if (model) {
        pp.pred = pred;
        k_features_mj<<<wg, 256, 0, c.stream>>>(B.d_args, wt, feat);
        FGSS_LAUNCH_CK();
        model_predict_tiles(c, feat, B.rec, pred, pp.d_sums + 2 * nj + 4, pp.d_sums + 3 * nj + 4);
    }
    k_cost_mj<<<tile_grid(c, B.rec), 256, 0, c.stream>>>(B.d_args, B.rec, pp.meta, pp.pred, cap_entries, pp.cost[0], pp.cost[1],
                                       (unsigned long long*)pp.d_sums);
    FGSS_LAUNCH_CK();
    return pp;
}

// Work items of one class, K[j] of join j, longest first (on the device).
uint4* batch_items(Ctx& c, Batch& B, const Prepass& pp, int cls, const std::vector<uint32_t>& K, uint64_t nitems) {
    const size_t nj = B.js.size();
    const std::string p = c.bpfx + "b.i" + std::to_string(cls) + ".";
    uint64_t* cpre = c.devT<uint64_t>(p + "cpre", B.R + 1);
    exclusive_scan<uint64_t>(c, pp.cost[cls], cpre, B.R, nullptr, cpre + B.R, (p + "scan").c_str());
    uint32_t* hk = c.pinnedT<uint32_t>(p + "hkoff", nj + 1);
    hk[0] = 0;
    for (size_t i = 0; i < nj; i++) hk[i + 1] = hk[i] + K[i];
    uint32_t* d_koff = c.devT<uint32_t>(p + "koff", nj + 1);
    FGSS_CK(cudaMemcpyAsync(d_koff, hk, (nj + 1) * 4, cudaMemcpyHostToDevice, c.stream));
    uint4* items = c.devT<uint4>(p + "items", nitems + 1);
    uint32_t* ikey = c.devT<uint32_t>(p + "key", nitems + 1);
    uint32_t* ival = c.devT<uint32_t>(p + "val", nitems + 1);
    k_items_mj<<<grid_for(nitems, 128), 128, 0, c.stream>>>(B.rec.roff, d_koff, (uint32_t)nj, (uint32_t)nitems, cpre,
                                                             pp.d_sums + cls * nj, items, ikey, ival);
    FGSS_LAUNCH_CK();
    if (nitems > 1) {
        // longest-processing-time order: sort items by descending cost
        uint4* sorted = c.devT<uint4>(p + "items2", nitems + 1);
        radix_sort<uint32_t, uint32_t>(c, ikey, ival, nitems, nullptr, 0, 16, (p + "sort").c_str());
        k_permute_items<<<grid_for(nitems, 128), 128, 0, c.stream>>>(items, ival, nitems, sorted, c.err_dev);
        FGSS_LAUNCH_CK();
        items = sorted;
    }
    return items;
}

// Second part: every record's token bitmap and the chunk splits of the
// queries whose windows exceed cap_entries, into a boundary buffer of
// cbuf_cap words (a query that finds it full is bisected by the fused kernel
// instead); returns the fused kernel's per-join arguments on the device.
FusedArgs* batch_filters(Ctx& c, Batch& B, const Prepass& pp, uint32_t cap_entries, uint64_t cbuf_cap, bool chunks) {
    const size_t nj = B.js.size();
    const std::string& p = c.bpfx;
    const uint64_t R = B.R;
    uint2* qchunk = c.devT<uint2>(p + "b.qchunk", R + 1);
    uint32_t* cbuf = c.devT<uint32_t>(p + "b.cbuf", cbuf_cap + 1);
    std::vector<uint64_t> boff(nj + 1, 0);
    std::vector<uint32_t> bmw(nj);
    for (size_t j = 0; j < nj; j++) {
        bmw[j] = bitmap_words(B.js[j]->in.n_tokens, B.js[j]->in.n_sets);
        boff[j + 1] = boff[j] + (uint64_t)bmw[j] * B.js[j]->in.n_sets;
    }
    uint4* bmap = c.devT<uint4>(p + "b.bmap", boff[nj] + 4);
    FusedArgs* hf = c.pinnedT<FusedArgs>(p + "b.hf", nj);
    for (size_t j = 0; j < nj; j++) {
        FusedArgs& f = hf[j];
        f.poff = B.poff + B.roff[j];
        f.win = pp.win;
        f.wpre = pp.wpre;
        f.smin = B.js[j]->lut.smin;
        f.meta = pp.meta + B.roff[j];
        f.qchunk = qchunk + B.roff[j];
        f.cbuf = cbuf;
        f.bmap = bmap + boff[j];
        f.bmw = bmw[j];
    }
    FusedArgs* d_fargs = c.devT<FusedArgs>(p + "b.fargs", nj);
    FGSS_CK(cudaMemcpyAsync(d_fargs, hf, nj * sizeof(FusedArgs), cudaMemcpyHostToDevice, c.stream));
    unsigned long long* cused = c.devT<unsigned long long>(p + "b.cused", 1);
    if (R == 0) return d_fargs;
    const TileMap wt = warp_tiles(c, B.rec);
    const unsigned g = tile_grid(c, wt);
    k_bitmaps_mj<<<g, 256, 0, c.stream>>>(B.d_args, d_fargs, wt);
    FGSS_LAUNCH_CK();
    if (!chunks) return d_fargs;  // no query for k_fused
    FGSS_CK(cudaMemsetAsync(cused, 0, 8, c.stream));
    k_chunks_mj<<<g, 256, 0, c.stream>>>(B.d_args, d_fargs, wt, pp.wtot, cap_entries, cbuf, cbuf_cap, cused);
    FGSS_LAUNCH_CK();
    return d_fargs;
}

// The batch's launch shape: the tuned shape of its most expensive join (the
// lowest threshold, then the most records), or the one of a requested strategy.
// A request for the strategy that the autotuner reported for the workload class runs
// the entry it had timed (*as_tuned), which may be the claim kernels: 20,000 titles at
// t = 0.5 0.36 ms, the keyed shape of that strategy 0.63 ms.
TuneEntry batch_shape(Ctx& c, const Batch& B, bool* as_tuned = nullptr) {
    if (as_tuned) *as_tuned = false;
    if (c.tune_force) return *c.tune_force;
    size_t lead = 0;
    for (size_t i = 1; i < B.js.size(); i++)
        if (B.js[i]->t < B.js[lead]->t || (B.js[i]->t == B.js[lead]->t && B.js[i]->in.n_sets > B.js[lead]->in.n_sets))
            lead = i;
    const JoinState& L = *B.js[lead];
    const std::string key = tune_key(L.in.n_sets, L.in.n_tokens, L.t);
    if (L.filter != FGSS_FILTER_AUTO) {
        const auto it = c.tune.find(key);
        if (it == c.tune.end() || filter_of(it->second) != L.filter) return filter_entry(L.filter);
        if (as_tuned) *as_tuned = true;
    }
    return tune_lookup(c, key);
}

}  // namespace

void batch_prep(Ctx& c, Batch& B, const std::vector<JoinState*>& js, const fgss_sets_view* views,
                const fgss_join_opts* opts) {
    const size_t nj = js.size();
    const std::string& p = c.bpfx;
    B.js = js;
    B.roff.assign(nj + 1, 0);
    B.n_max = 0;
    B.terms_max = 0;
    uint64_t T = 0;
    for (size_t j = 0; j < nj; j++) {
        JoinState& J = *js[j];
        fgss_sets_view v = views[j];
        if (!v.on_device) {
            // the same host arrays as an earlier join of the batch: copied to the device once
            for (size_t k = 0; k < j; k++) {
                const fgss_sets_view& w = views[k];
                if (!w.on_device && w.id == v.id && w.pos == v.pos && w.len == v.len && w.tokens == v.tokens &&
                    w.n_sets == v.n_sets && w.n_tokens == v.n_tokens) {
                    v = js[k]->in;
                    v.n_terms = views[j].n_terms;
                    break;
                }
            }
        }
        join_setup_host(c, J, v, opts[j], J.slot);
        B.roff[j + 1] = B.roff[j] + J.in.n_sets;
        B.n_max = std::max<uint32_t>(B.n_max, (uint32_t)J.in.n_sets);
        B.terms_max = std::max<uint32_t>(B.terms_max, J.in.n_terms);
        T += J.in.n_tokens;
    }
    B.R = B.roff[nj];
    // per-record offsets are 32-bit: the caller splits larger batches
    if (T >= 0xffffffffull || B.R >= 0xffffffffull) fail(FGSS_ERR_UNSUPPORTED, "a batch of 2^32 or more tokens");
    // one block, cleared and read back as one
    B.words = (nj * (4 + SS_N + 2) + 2) * 8;
    uint64_t* words = c.devT<uint64_t>(p + "b.words", B.words / 8);
    B.status = reinterpret_cast<uint32_t*>(words);
    B.stats = reinterpret_cast<unsigned long long*>(words + nj * 4);
    B.d_e = words + nj * (4 + SS_N);
    B.tot = B.d_e + nj * 2;
    B.icnt = c.devT<uint32_t>(p + "b.icnt", B.R + 1);
    B.pcnt = c.devT<uint32_t>(p + "b.pcnt", B.R + 1);
    B.ioff = c.devT<uint32_t>(p + "b.ioff", B.R + 1);
    B.poff = c.devT<uint32_t>(p + "b.poff", B.R + 1);
    B.send = c.devT<uint32_t>(p + "b.send", nj * 65537);
    B.heavy_q = c.devT<uint32_t>(p + "b.heavy_q", B.R + 1);
    B.d_args = c.devT<JoinArgs>(p + "b.args", nj);
    FGSS_CK(cudaMemsetAsync(words, 0, B.words, c.stream));
    for (size_t j = 0; j < nj; j++) {
        JoinState& J = *js[j];
        J.status = B.status + 8 * j;
        J.stats = B.stats + SS_N * j;
        J.d_e = B.d_e + 2 * j;
        JoinArgs& a = J.args;
        a.status = J.status;
        a.stats = J.stats;
        a.send = B.send + 65537ull * j;
        a.heavy_q = B.heavy_q + B.roff[j];
        a.heavy_count = J.status + 2;
        a.res_count = J.status + 3;
    }
    B.rec = upload_tiles(c, p + "b.rec", B.roff, kRecTile);
    upload_args(c, B, p + "b.ha0");
    if (B.R) {
        const TileMap t = warp_tiles(c, B.rec);
        k_prep_mj<<<tile_grid(c, t, 8), 256, 0, c.stream>>>(B.d_args, t, B.icnt, B.pcnt);
        FGSS_LAUNCH_CK();
        k_send_mj<<<grid_for((uint64_t)nj << 16, 256, c.num_sms * 32), 256, 0, c.stream>>>(B.d_args, (uint32_t)nj,
                                                                                          B.send);
        FGSS_LAUNCH_CK();
        exclusive_scan<uint32_t>(c, B.icnt, B.ioff, B.R, nullptr, B.ioff + B.R, (p + "b.scan.i").c_str());
        exclusive_scan<uint32_t>(c, B.pcnt, B.poff, B.R, nullptr, B.poff + B.R, (p + "b.scan.p").c_str());
        k_join_totals<<<grid_for(nj, 128), 128, 0, c.stream>>>(B.d_args, B.rec.roff, (uint32_t)nj, B.ioff, B.poff, B.d_e,
                                                               B.tot);
        FGSS_LAUNCH_CK();
    } else {
        FGSS_CK(cudaMemsetAsync(B.ioff, 0, 4, c.stream));
        FGSS_CK(cudaMemsetAsync(B.poff, 0, 4, c.stream));
    }
    // one wait for the whole batch: no kernel reads tokens through caller
    // offsets before they are validated
    const uint32_t* h = batch_read_status(c, B);
    const uint64_t* tot = reinterpret_cast<const uint64_t*>(h) + (B.tot - words);
    B.E = tot[0];
    B.P = tot[1];
    B.len_max = 0;
    B.keyed_possible = false;
    B.status_host = nullptr;  // of the filter, not yet read
    for (size_t j = 0; j < nj; j++) {
        if (js[j]->in.n_sets) check_input_status(h[8 * j]);
        B.len_max = std::max(B.len_max, h[8 * j + 1]);
        B.keyed_possible |= js[j]->lut.probe_max[std::min<uint32_t>(h[8 * j + 1], kMaxLen)] > kClaimPC;
    }
}

void batch_index(Ctx& c, Batch& B, uint64_t E_cap) {
    const size_t nj = B.js.size();
    const std::string& p = c.bpfx;
    if (E_cap < B.E) fail(FGSS_ERR_CUDA, "index buffers below the batch's entry count");
    const int tbits = bits_for((uint64_t)B.terms_max + 1);
    const int jbits = bits_for(nj);
    // join j's list offsets: n_terms + 1 entries from loff[j], positions in
    // the batch's entry arrays; its block table, n_terms nb + 1 entries from
    // toff[j].  A join of at most kBlockIds records has one block and its list
    // offsets are the table; one whose table would hold more words than a
    // quarter of its tokens (k-mers: millions of terms with short lists) has none.
    uint64_t* hl = c.pinnedT<uint64_t>(p + "b.hloff", 2 * nj + 2);
    uint64_t* ht = hl + nj + 1;
    hl[0] = ht[0] = 0;
    for (size_t j = 0; j < nj; j++) {
        const fgss_sets_view& in = B.js[j]->in;
        JoinArgs& a = B.js[j]->args;
        hl[j + 1] = hl[j] + in.n_terms + 1;
        const uint64_t nb = (in.n_sets + kBlockIds - 1) / kBlockIds;
        a.nb = nb <= 1 ? (uint32_t)nb : nb * in.n_terms <= in.n_tokens / 4 + 65536 ? (uint32_t)nb : 0u;
        ht[j + 1] = ht[j] + (a.nb > 1 ? nb * in.n_terms + 1 : 0);
    }
    const uint64_t L = hl[nj], TB = ht[nj];
    uint64_t* d_loff = c.devT<uint64_t>(p + "b.loff", 2 * nj + 2);
    const uint64_t* d_toff = d_loff + nj + 1;
    FGSS_CK(cudaMemcpyAsync(d_loff, hl, (2 * nj + 2) * 8, cudaMemcpyHostToDevice, c.stream));
    uint32_t* list = c.devT<uint32_t>(p + "b.list", L + 1);
    uint32_t* tab = c.devT<uint32_t>(p + "b.tab", TB + 1);
    uint2* ent = c.devT<uint2>(p + "b.ent", E_cap + 1);
    for (size_t j = 0; j < nj; j++) {
        JoinArgs& a = B.js[j]->args;
        a.list_off = list + hl[j];
        a.tab = a.nb > 1 ? tab + ht[j] : a.list_off;
        a.ent = ent;
    }
    upload_args(c, B, p + "b.ha1");
    // a join without entries keeps these zero offsets (empty lists)
    FGSS_CK(cudaMemsetAsync(list, 0, L * 4, c.stream));
    if (TB) FGSS_CK(cudaMemsetAsync(tab, 0, TB * 4, c.stream));
    if (B.R) {
        if (tbits + jbits <= 32) index_sort<uint32_t>(c, B, E_cap, tbits, jbits, B.tot, d_loff, list, d_toff, tab, ent);
        else index_sort<uint64_t>(c, B, E_cap, tbits, jbits, B.tot, d_loff, list, d_toff, tab, ent);
    }
}

void batch_query_costs(Ctx& c, Batch& B, bool use_model, uint64_t* out) {
    if (B.R == 0) return;
    const TuneEntry te = batch_shape(c, B);
    const Prepass pp = batch_prepass(c, B, (1u << te.hash_log2) / 4 * 3, B.P, use_model && c.model, 0);
    k_query_costs_mj<<<tile_grid(c, B.rec), 256, 0, c.stream>>>(B.d_args, B.rec, pp.wtot, pp.pred, pp.cost[0]);
    FGSS_LAUNCH_CK();
    FGSS_CK(cudaMemcpyAsync(out, pp.cost[0], B.R * 8, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
}

// Runs the fused filter+verify over every join of the batch (index built).
//
// With a plan in record mode the host-side decisions of this run (launch
// shape, buffer sizes, work items per join, result capacities, heavy-path
// slots) are kept; in capture mode (plan->capture) the same device work is
// issued with those decisions and without any host synchronization, so the
// stream can be captured into a CUDA graph and replayed on later calls.
void batched_filter_verify(Ctx& c, Batch& B, bool use_model, BatchPlan* plan) {
    const size_t nj = B.js.size();
    std::vector<JoinState*>& joins = B.js;
    const bool capture = plan && plan->capture;
    const std::string& p = c.bpfx;
    bool as_tuned = false;
    const TuneEntry te = capture ? plan->te : batch_shape(c, B, &as_tuned);
    if (capture) as_tuned = plan->as_tuned;
    else if (plan) plan->as_tuned = as_tuned;
    const uint32_t cap_entries = (1u << te.hash_log2) / 4 * 3;  // chunk capacity of the chosen kernel shape
    const uint64_t P_cap = plan ? plan->P_cap : B.P;
    if (P_cap < B.P) fail(FGSS_ERR_CUDA, "window buffers below the batch's probe-token count");
    const bool model = use_model && c.model;
    // the caller's own choice of a strategy, a tuned keyed shape and the global accumulator take every query
    bool classes = te.heavy_min_probe == 0 && !te.keyed;
    for (size_t i = 0; i < nj; i++)
        classes &= joins[i]->filter == FGSS_FILTER_AUTO || (as_tuned && joins[i]->filter == filter_of(te));
    // light: no query can be k_fused's and there is no learned estimate to order them by, so
    // k_claim takes the records in order and the costs, items and their sort, and the wait
    // for their counts, are left out (1,000 titles: 60 us of 450)
    const bool light = capture ? plan->light : classes && !model && !B.keyed_possible && B.R != 0;
    if (plan && !capture) plan->light = light;
    const Prepass pp = batch_prepass(c, B, cap_entries, P_cap, model, classes ? kClaimPC : 0, light);

    // work items per class of k_fused and k_claim: ~256 per resident CTA over
    // the whole batch (a few queries per item at 100k records), split by cost
    // share and handed out longest first, so the dynamic queue ends with short
    // items.  A class without queries gets none, or under a plan (whose graph
    // may be replayed on other data) a few.
    std::vector<uint32_t> K[2] = {std::vector<uint32_t>(nj, 0), std::vector<uint32_t>(nj, 0)};
    uint64_t nitems[2] = {0, 0};
    bool tiny = classes && B.R != 0;
    bool wide = capture && plan->wide;  // (light: the costs are not known)
    uint64_t* hsum = c.pinnedT<uint64_t>(p + "b.hsum", std::max<size_t>(pp.n_sums, 1));
    if (light) {
        // nothing to read back
    } else if (capture) {
        for (int k = 0; k < 2; k++) {
            K[k] = plan->K[k];
            nitems[k] = plan->nitems[k];
        }
    } else {
        FGSS_CK(cudaMemcpyAsync(hsum, pp.d_sums, pp.n_sums * 8, cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        for (size_t i = 0; i < nj; i++) {
            if (!model || joins[i]->res_cap_hint) continue;
            joins[i]->pred_results = hsum[2 * nj + 4 + i];
            joins[i]->pred_candidates = hsum[3 * nj + 4 + i];
        }
        const uint64_t* count = hsum + 2 * nj;  // queries per class
        for (int k = 0; k < 2; k++) {
            if (k == QC_CLAIM && !classes) continue;
            if (k == QC_CLAIM) {
                uint64_t cost = 0;
                for (size_t i = 0; i < nj; i++) cost += hsum[nj + i];
                wide = count[k] != 0 && cost / count[k] >= kClaimWideCost;
            }
            if (count[k] == 0 && !plan) continue;
            uint64_t grand = 0;
            for (size_t i = 0; i < nj; i++) grand += hsum[k * nj + i];
            const uint64_t ctas = k == QC_CLAIM ? (uint64_t)kClaimCtas * c.num_sms : fused_resident_ctas(c, te);
            const uint64_t want = (count[k] ? 256 : 4) * ctas;
            for (size_t i = 0; i < nj; i++) {
                const uint64_t n = joins[i]->in.n_sets;
                if (n == 0) continue;
                uint64_t v = grand ? (want * hsum[k * nj + i] + grand - 1) / grand : 1;
                v = std::max<uint64_t>(1, std::min<uint64_t>(v, n));
                K[k][i] = (uint32_t)v;
                nitems[k] += v;
            }
        }
        if (!plan) tiny &= count[QC_TINY] != 0;
    }
    if (nitems[0] >= 0xffffffffull || nitems[1] >= 0xffffffffull) fail(FGSS_ERR_UNSUPPORTED, "too many work items");
    // chunk boundaries: exactly the words the splits take (the plan's size in
    // a capture; a replay on other data that needs more bisects instead)
    const uint64_t cbuf_cap = light ? 0 : capture ? plan->cbuf_cap : std::min<uint64_t>(hsum[2 * nj + 3], 0xfffffff0ull);
    if (plan && !capture) plan->cbuf_cap = cbuf_cap;
    FusedArgs* d_fargs = batch_filters(c, B, pp, cap_entries, cbuf_cap, nitems[QC_KEYED] != 0);
    const uint4* items[2] = {nullptr, nullptr};
    for (int k = 0; k < 2; k++)
        if (nitems[k]) items[k] = batch_items(c, B, pp, k, K[k], nitems[k]);
    const ClaimItems claims = light ? items_in_order(c, B)
                                    : ClaimItems{items[QC_CLAIM], B.rec, 0, (uint32_t)nitems[QC_CLAIM]};

    bool sided = false;
    for (size_t i = 0; i < nj; i++) sided |= joins[i]->args.side != nullptr;
    uint32_t* counter = c.devT<uint32_t>(p + "b.counter", 4 + nj);
    uint32_t* hst = c.pinnedT<uint32_t>(p + "b.hst", nj * 8);
    std::vector<uint64_t> cap(nj, 0);
    uint32_t slots = 0;
    // (inside a capture the events must be external record nodes to be timed at replay)
    const unsigned rec_flags = capture ? cudaEventRecordExternal : 0u;
    for (int attempt = 0;; attempt++) {
        // result buffers: the caller's size, the learned estimate (x1.5 +
        // slack), the last size seen for this slot, or the exact count after
        // an overflow
        std::vector<uint64_t> capoff(nj + 1, 0);
        for (size_t i = 0; i < nj; i++) {
            JoinState& J = *joins[i];
            if (capture) {
                cap[i] = plan->res_cap[i];
            } else {
                auto itc = c.tune.find(J.pfx("rescap"));
                const uint64_t last = itc != c.tune.end() ? (uint64_t)itc->second.ctas_per_sm : 0;
                uint64_t v;
                if (J.res_cap_hint) v = J.res_cap_hint;
                else if (J.res_cap_user) v = J.res_cap_user;
                else if (model) v = std::max<uint64_t>((uint64_t)((double)hsum[2 * nj + 4 + i] * 1.5) + 4096, last);
                else v = std::max<uint64_t>(J.in.n_sets + 4096, last);
                cap[i] = std::min<uint64_t>(v, 0xfffffff0ull);
                if (model && !J.res_cap_hint && !J.res_cap_user && cap[i] > (1ull << 26)) {
                    // a wild estimate must not take the device's memory (about 48 bytes a
                    // slot): too small a buffer only costs an exact re-run
                    size_t free_b = 0, total_b = 0;
                    FGSS_CK(cudaMemGetInfo(&free_b, &total_b));
                    cap[i] = std::min<uint64_t>(cap[i], std::max<uint64_t>({J.in.n_sets + 4096, last, free_b / 256}));
                }
            }
            capoff[i + 1] = capoff[i] + cap[i];
        }
        uint32_t* res_q = c.devT<uint32_t>(p + "b.res.q", capoff[nj] + 1);
        uint32_t* res_s = c.devT<uint32_t>(p + "b.res.s", capoff[nj] + 1);
        uint32_t* res_o = c.devT<uint32_t>(p + "b.res.o", capoff[nj] + 1);
        for (size_t i = 0; i < nj; i++) {
            JoinArgs& a = joins[i]->args;
            a.res_cap = (uint32_t)cap[i];
            a.heavy_min_qp = te.heavy_min_probe > 0 ? (uint32_t)te.heavy_min_probe : 0xffffffffu;
            a.res_q = res_q + capoff[i];
            a.res_s = res_s + capoff[i];
            a.res_o = res_o + capoff[i];
        }
        upload_args(c, B, p + "b.ha2");
        FGSS_CK(cudaMemsetAsync(counter, 0, (4 + nj) * 4, c.stream));
        FGSS_CK(cudaEventRecordWithFlags(c.ev[4], c.stream, rec_flags));
        if (claims.n && wide) claim_launch<MODE_FUSED, ClaimWide>(c, B.d_args, d_fargs, claims, counter + 1, sided);
        else if (claims.n) claim_launch<MODE_FUSED>(c, B.d_args, d_fargs, claims, counter + 1, sided);
        if (nitems[QC_KEYED])
            fused_launch(c, te, B.d_args, d_fargs, items[QC_KEYED], (uint32_t)nitems[QC_KEYED], counter, sided);
        if (tiny) tiny_launch<MODE_FUSED>(c, B.d_args, d_fargs, B.rec, sided);
        FGSS_CK(cudaEventRecordWithFlags(c.ev[5], c.stream, rec_flags));
        c.probe_timed = true;
        // queries deferred to the global-memory accumulator: one persistent
        // launch for every join.  Eagerly only when some were queued; under a
        // plan always, with scratch for a fixed slot count (a launch whose
        // queues are empty returns at once).
        uint32_t max_nh = 0;
        if (!capture && !plan && nitems[QC_KEYED]) {  // only k_fused defers queries
            FGSS_CK(cudaMemcpyAsync(hst, B.status, nj * 32, cudaMemcpyDeviceToHost, c.stream));
            c.sync();
            for (size_t i = 0; i < nj; i++) max_nh = std::max(max_nh, hst[8 * i + 2]);
        }
        const uint32_t all_slots = std::min<uint32_t>(std::max<uint32_t>(B.n_max, 1), (uint32_t)c.num_sms);
        slots = light ? 0 : capture ? plan->heavy_slots : plan ? all_slots : std::min<uint32_t>(max_nh, (uint32_t)c.num_sms);
        if (slots) {
            const HeavyScratch hs = heavy_scratch(c, p, B.n_max, slots, capture);
            FGSS_CK(cudaEventRecordWithFlags(c.ev[6], c.stream, rec_flags));
            k_probe_heavy<MODE_FUSED, 512><<<slots, 512, 0, c.stream>>>(B.d_args, 0, (uint32_t)nj, hs.zero,
                                                                        hs.zero_words, hs.aux, hs.aux_words,
                                                                        counter + 4);
            FGSS_LAUNCH_CK();
            FGSS_CK(cudaEventRecordWithFlags(c.ev[7], c.stream, rec_flags));
            c.heavy_timed = true;
        }
        if (capture) break;
        const uint32_t* st = batch_read_status(c, B);
        bool over = false;
        for (size_t i = 0; i < nj; i++) {
            JoinState& J = *joins[i];
            const uint32_t got = st[8 * i + 3];
            if (got > cap[i]) {
                // The learned (or remembered) capacity was too small: the kernel
                // kept counting, so the batch re-runs with the exact size.  A
                // plan keeps that exact size for the captured batch.
                J.res_cap_hint = got;
                J.overflow_retries++;
                over = true;
            }
        }
        if (!over) break;
        if (attempt) fail(FGSS_ERR_CUDA, "result buffers overflowed at their exact size");
        k_clear_filter_state_mj<<<(unsigned)std::min<size_t>(nj, 1024), 32, 0, c.stream>>>(B.d_args, (uint32_t)nj);
        FGSS_LAUNCH_CK();
    }
    if (plan && !capture) {
        plan->te = te;
        plan->wide = wide;
        for (int k = 0; k < 2; k++) plan->K[k] = K[k];
        for (int k = 0; k < 2; k++) plan->nitems[k] = nitems[k];
        plan->heavy_slots = slots;
        plan->res_cap = cap;
    }

    // results: join j's in the output columns from out_off[j] (its result
    // count eagerly, its capacity under a plan, so a captured graph finds
    // every buffer at the size it has now)
    std::vector<uint64_t> rcap(nj);
    for (size_t i = 0; i < nj; i++) {
        JoinState& J = *joins[i];
        if (capture) {
            rcap[i] = cap[i];
            continue;
        }
        const uint32_t got = B.status_host[8 * i + 3];
        J.n_res = got;
        J.res_cap_hint = 0;
        // remember a sufficient capacity for the next call on this slot
        c.tune[J.pfx("rescap")].ctas_per_sm = (int)std::min<uint64_t>((uint64_t)got + got / 4 + 1024, 0x7fffffff);
        rcap[i] = plan ? cap[i] : got;
    }
    B.out_off.assign(nj + 1, 0);
    for (size_t i = 0; i < nj; i++) B.out_off[i + 1] = B.out_off[i] + rcap[i];
    B.out_cap = B.out_off[nj];
    const uint64_t oc = B.out_cap;
    B.out_col = out_column(oc);
    uint32_t* o6 = c.devT<uint32_t>(p + "b.o", 6 * B.out_col);
    B.oq = o6;
    B.os = o6 + B.out_col;
    B.oidq = o6 + 2 * B.out_col;
    B.oids = o6 + 3 * B.out_col;
    B.oo = o6 + 4 * B.out_col;
    B.osim = reinterpret_cast<float*>(o6 + 5 * B.out_col);
    for (size_t i = 0; i < nj; i++) {
        JoinState& J = *joins[i];
        const uint64_t o = B.out_off[i];
        J.out_col = B.out_col;
        J.oq = B.oq + o;
        J.os = B.os + o;
        J.oidq = B.oidq + o;
        J.oids = B.oids + o;
        J.oo = B.oo + o;
        J.osim = B.osim + o;
    }
    if (oc == 0) return;
    const TileMap rt = upload_tiles(c, p + "b.rt", B.out_off, 256);
    uint64_t* resoff = c.devT<uint64_t>(p + "b.resoff", nj + 2);
    uint64_t* d_n = resoff + nj + 1;
    k_result_offsets<<<1, 1024, 0, c.stream>>>(B.d_args, (uint32_t)nj, resoff, d_n);
    FGSS_LAUNCH_CK();
    // sort keys join << 2qb | q << qb | s: only the bits that vary
    const int qb = bits_for(B.n_max), jb = bits_for(nj);
    if (2 * qb + jb > 64) fail(FGSS_ERR_UNSUPPORTED, "result keys of more than 64 bits");
    uint64_t* key = c.devT<uint64_t>(p + "b.rkey", oc + 1);
    uint32_t* val = c.devT<uint32_t>(p + "b.rval", oc + 1);
    k_result_keys_mj<<<tile_grid(c, rt), 256, 0, c.stream>>>(B.d_args, rt, resoff, (uint32_t)qb, key, val);
    FGSS_LAUNCH_CK();
    radix_sort<uint64_t, uint32_t>(c, key, val, oc, d_n, 0, 2 * qb + jb, (p + "b.rsort").c_str());
    k_result_out_mj<<<grid_for(oc, 256, c.num_sms * 32), 256, 0, c.stream>>>(
        B.d_args, key, val, d_n, resoff, rt.roff, (uint32_t)qb, B.oq, B.os, B.oidq, B.oids, B.oo, B.osim, c.err_dev);
    FGSS_LAUNCH_CK();
}

namespace {

__global__ void k_sum_u32(const uint32_t* __restrict__ in, uint64_t n, unsigned long long* out) {
    unsigned long long s = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        s += in[i];
    s = warp_sum(s);
    if (lane_id() == 0 && s) atomicAdd(out, s);
}

template <int MODE, int NT, int HLOG>
void probe_launch(Ctx& c, const JoinArgs* d_args, uint64_t n, cudaStream_t stream) {
    FGSS_CK(cudaFuncSetAttribute(k_probe<MODE, NT, HLOG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)ProbeLayout<MODE, HLOG>::bytes));
    k_probe<MODE, NT, HLOG><<<(unsigned)n, NT, ProbeLayout<MODE, HLOG>::bytes, stream>>>(d_args);
    FGSS_LAUNCH_CK();
}

// Probe tokens up to which a query of a join that runs k_probe anyway is k_claim's.  A
// step of k_claim costs its producer two bounds for every probe token, so from about
// 400 of them on the consumers wait for it and k_probe is the faster one.  Calls with
// the line at 640 / 384 / 256 (k_probe beside k_claim): 2,100 records of 700 to 1,400
// tokens at t = 0.5 4.69 / 3.48 / 3.47 ms, 6,000 of 200 to 1,800 17.4 / 16.2 / 16.3;
// 20,000 of 100 to 700 and 20 longer ones 46 / 46 / 57.
constexpr uint32_t kPlainPC = 384;

// k_probe on the copies' stream, beside the claim kernels, whose queries are others:
// both leave the chip idle at their ends, together less (with the line at 384, 2,100
// records as above 3.64 -> 3.48 ms, 6,000 of 900 to 1,800 38.9 -> 35.7).  The context's
// stream goes on behind both.
template <int MODE, typename F>
void probe_beside(Ctx& c, const JoinArgs* d_args, uint64_t n, bool keyed, F&& claims) {
    if (!keyed) return claims();
    c.copy_lane();
    FGSS_CK(cudaEventRecord(c.copy_ev[0], c.stream));
    FGSS_CK(cudaStreamWaitEvent(c.copy_stream, c.copy_ev[0], 0));
    probe_launch<MODE, 256, 12>(c, d_args, n, c.copy_stream);
    FGSS_CK(cudaEventRecord(c.copy_ev[1], c.copy_stream));
    claims();
    FGSS_CK(cudaStreamWaitEvent(c.stream, c.copy_ev[1], 0));
}

}  // namespace

void plain_filter_verify(Ctx& c, Batch& B, bool want_cand) {
    JoinState& J = *B.js[0];
    const uint64_t n = J.in.n_sets;
    JoinArgs& a = J.args;
    J.n_res = 0;
    if (n == 0) return;
    const std::string& p = c.bpfx;
    // ---- pre-pass: windows and classes of the queries; k_claim takes the records in order
    const bool keyed = B.keyed_possible, sided = a.side != nullptr;
    const Prepass pp = batch_prepass(c, B, 1u << 30, B.P, false, keyed ? kPlainPC : kClaimPC, true);
    const ClaimItems claims = items_in_order(c, B);
    FusedArgs* d_fargs = batch_filters(c, B, pp, 1u << 30, 0, false);
    const FusedArgs& fa = c.pinnedT<FusedArgs>(p + "b.hf", 1)[0];
    a.meta = pp.meta;
    a.vcnt = c.devT<uint32_t>(J.pfx("vcnt"), n + 1);
    a.ccnt = c.devT<uint32_t>(J.pfx("ccnt"), n + 1);
    a.wcnt = c.devT<uint32_t>(J.pfx("wcnt"), n + 1);
    uint32_t* voff = c.devT<uint32_t>(J.pfx("voff"), n + 1);
    a.voff = voff;
    uint32_t* hcnt = c.pinnedT<uint32_t>(J.pfx("h.cnt"), 8);
    // words: candidates, results (64-bit, the scans write the low halves), then per pass
    // the counters of the work items and of the queue of the global accumulator
    uint32_t* ctr = c.devT<uint32_t>(J.pfx("words"), 8);
    uint64_t* d_nc = reinterpret_cast<uint64_t*>(ctr);
    J.d_nres = d_nc + 1;
    ctr += 4;
    FGSS_CK(cudaMemsetAsync(a.vcnt, 0, n * 4, c.stream));
    FGSS_CK(cudaMemsetAsync(d_nc, 0, 32, c.stream));
    // ---- count pass
    upload_args(c, B, p + "b.ha2");
    if (keyed) {
        FGSS_CK(cudaMemsetAsync(a.ccnt, 0, n * 4, c.stream));
        FGSS_CK(cudaMemsetAsync(a.wcnt, 0, n * 4, c.stream));
        FGSS_CK(cudaMemsetAsync(a.heavy_count, 0, 4, c.stream));
    }
    probe_beside<MODE_COUNT>(c, B.d_args, n, keyed, [&] {
        claim_launch<MODE_COUNT>(c, B.d_args, d_fargs, claims, ctr, sided);
        tiny_launch<MODE_COUNT>(c, B.d_args, d_fargs, B.rec, sided);
    });
    HeavyScratch hs;
    uint32_t hslots = 0;
    if (keyed) {
        // probe prefixes beyond k_probe's shared memory: the global accumulator
        FGSS_CK(cudaMemcpyAsync(hcnt, a.heavy_count, 4, cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        hslots = std::min<uint32_t>(hcnt[0], (uint32_t)c.num_sms);
        if (hslots) {
            hs = heavy_scratch(c, "", n, hslots, false);
            k_probe_heavy<MODE_COUNT, 512><<<hslots, 512, 0, c.stream>>>(B.d_args, 0, 1, hs.zero, hs.zero_words, hs.aux,
                                                                         hs.aux_words, ctr + 1);
            FGSS_LAUNCH_CK();
        }
        k_sum_u32<<<grid_for(n, 256, c.num_sms * 8), 256, 0, c.stream>>>(a.ccnt, n, &J.stats[SS_CANDIDATES]);
        FGSS_LAUNCH_CK();
        k_sum_u32<<<grid_for(n, 256, c.num_sms * 8), 256, 0, c.stream>>>(a.wcnt, n, &J.stats[SS_WINDOW]);
        FGSS_LAUNCH_CK();
    }
    exclusive_scan<uint32_t>(c, a.vcnt, voff, n, nullptr, reinterpret_cast<uint32_t*>(d_nc), J.pfx("scan.v").c_str());
    FGSS_CK(cudaMemcpyAsync(hcnt, d_nc, 4, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    const uint64_t C = hcnt[0];
    // ---- fill pass
    uint4* cand = c.devT<uint4>(J.pfx("cand"), C + 1);
    a.cand = cand;
    if (C) {
        FGSS_CK(cudaMemsetAsync(a.ccnt, 0, n * 4, c.stream));
        ctr += 2;
        if (keyed) FGSS_CK(cudaMemsetAsync(a.heavy_count, 0, 4, c.stream));
        upload_args(c, B, p + "b.ha2");
        probe_beside<MODE_FILL>(c, B.d_args, n, keyed, [&] {
            claim_launch<MODE_FILL>(c, B.d_args, d_fargs, claims, ctr, sided);
            tiny_launch<MODE_FILL>(c, B.d_args, d_fargs, B.rec, sided);
        });
        if (hslots) {
            k_probe_heavy<MODE_FILL, 512><<<hslots, 512, 0, c.stream>>>(B.d_args, 0, 1, hs.zero, hs.zero_words, hs.aux,
                                                                        hs.aux_words, ctr + 1);
            FGSS_LAUNCH_CK();
        }
    }
    if (want_cand) {
        std::vector<uint4> hc(C);
        if (C) FGSS_CK(cudaMemcpyAsync(hc.data(), cand, C * 16, cudaMemcpyDeviceToHost, c.stream));
        c.sync();
        J.cand_host.resize(3 * C);
        for (uint64_t i = 0; i < C; i++) {
            J.cand_host[3 * i] = hc[i].x;
            J.cand_host[3 * i + 1] = hc[i].y;
            J.cand_host[3 * i + 2] = hc[i].z;
        }
    }
    if (C == 0) return;
    // ---- verification (thread-per-candidate merge in the reference; see k_verify)
    uint32_t* ov = c.devT<uint32_t>(J.pfx("ov"), C + 1);
    uint32_t per = 32;
    while (per > 1 && C < (uint64_t)per * 64 * c.num_sms) per >>= 1;
    // groups from the length on at which they gained: calls with records of up to 250 tokens lose 1 to
    // 4 % by them, of 500 and more gain up to 40 %.  Where a warp has fewer than 32 records the bound's
    // loads do not matter and every record is a group: 1,500 records of 1,500 to 4,000 tokens at
    // t = 0.8 1.65 ms in groups of 4, 1.52 of 1
    // Beyond 64 rounds of all warps a warp's share of the runs evens out and only the loads are left:
    // 200,000 heavy-tailed records at t = 0.8 (17 rounds) 5.09 ms without groups, 3.97 with, at 0.7 (54)
    // 11.52 and 11.37; 500,000 at 0.8 (97) 13.6 and 14.0, 1,000,000 at 0.7 (1,190) 177 and 185.
    const unsigned blocks = grid_for((C + per - 1) / per * 32, 256, c.num_sms * 32);
    const bool spread = B.len_max > 256 && C / 64 <= (uint64_t)blocks * 256;
    const uint32_t group = !spread ? per : per == 32 ? 4u : 1u;
    k_verify<<<blocks, 256, 0, c.stream>>>(a, cand, d_nc, per, group, ov, fa.bmap, fa.bmw);
    FGSS_LAUNCH_CK();
    // ---- compaction of the verified pairs: count -> scan -> fill
    uint32_t* flag = c.devT<uint32_t>(J.pfx("flag"), C + 1);
    uint32_t* off = c.devT<uint32_t>(J.pfx("off"), C + 1);
    k_result_flags<<<grid_for(C, 256, c.num_sms * 32), 256, 0, c.stream>>>(a, cand, ov, d_nc, flag);
    FGSS_LAUNCH_CK();
    exclusive_scan<uint32_t>(c, flag, off, C, nullptr, reinterpret_cast<uint32_t*>(J.d_nres),
                             J.pfx("scan.r").c_str());
    // up to 65,536 candidates the buffers and grids are theirs and the number of results
    // is read back at the end: a wait here costs more than the launches it would shrink
    FGSS_CK(cudaMemcpyAsync(hcnt + 2, J.d_nres, 4, cudaMemcpyDeviceToHost, c.stream));
    const bool wait = C > 65536;
    if (wait) c.sync();
    const uint64_t R = wait ? hcnt[2] : C;
    uint64_t* keys = c.devT<uint64_t>(J.pfx("rkey"), R + 1);
    uint32_t* vals = c.devT<uint32_t>(J.pfx("rval"), R + 1);
    if (R) {
        k_result_fill<<<grid_for(C, 256, c.num_sms * 32), 256, 0, c.stream>>>(
            cand, ov, flag, off, d_nc, (uint32_t)bits_for(n), keys, vals, c.err_dev);
        FGSS_LAUNCH_CK();
    }
    join_output(c, J, keys, vals, J.d_nres, R);
    batch_read_status(c, B);
    J.n_res = hcnt[2];
}

const uint32_t* batch_read_status(Ctx& c, Batch& B) {
    uint32_t* h = c.pinnedT<uint32_t>(c.bpfx + "b.hwords", B.words / 4);
    FGSS_CK(cudaMemcpyAsync(h, B.status, B.words, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    B.status_host = h;
    return h;
}

void batch_finish_status(Ctx& c, Batch& B) {
    const size_t nj = B.js.size();
    const uint32_t* h = B.status_host ? B.status_host : batch_read_status(c, B);
    const uint64_t* w = reinterpret_cast<const uint64_t*>(h);
    const unsigned long long* hs = reinterpret_cast<const unsigned long long*>(w + nj * 4);
    const uint64_t* he = w + (B.d_e - reinterpret_cast<const uint64_t*>(B.status));
    for (size_t j = 0; j < nj; j++) {
        B.js[j]->n_entries = he[2 * j];
        B.js[j]->n_res = h[8 * j + 3];
        apply_status(*B.js[j], h[8 * j], hs + SS_N * j);
    }
}

}  // namespace fgss
