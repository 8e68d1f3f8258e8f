// fmha_fwd / batch prefill / paged prefill / multi-token split-KV on the tcgen05 kernel (fmha_fwd_sm100.cuh): which calls it
// takes, the device parameters of a call, and the choice of the instance.
#include <atomic>

#include "fmha_fwd_sm100.cuh"

namespace fck {

namespace sm100 {

#define FCK_EXTERN(T, E, V, S, H) extern FCK_SM100_INST(T, E, V, S, H)
#define FCK_EXTERN_SPLIT(T, S, E) extern FCK_SM100_INST_SPLIT(T, S, E)
FCK_SM100_PLAIN(FCK_EXTERN, __half) FCK_SM100_PLAIN(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_HDIM64(FCK_EXTERN, __half) FCK_SM100_HDIM64(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_EXTRA(FCK_EXTERN, __half) FCK_SM100_EXTRA(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_EXTRA64(FCK_EXTERN, __half) FCK_SM100_EXTRA64(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_BIAS(FCK_EXTERN, __half) FCK_SM100_BIAS(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_TMA_BIAS(FCK_EXTERN, __half) FCK_SM100_TMA_BIAS(FCK_EXTERN, __nv_bfloat16)
FCK_SM100_FP8(FCK_EXTERN, f8e4m3_t) FCK_SM100_FP8(FCK_EXTERN, f8e5m2_t)
FCK_SM100_SPLIT(FCK_EXTERN_SPLIT, __half) FCK_SM100_SPLIT(FCK_EXTERN_SPLIT, __nv_bfloat16)

}  // namespace sm100

using namespace sm100;

namespace {

// With the packed f16x2 exp2 the threshold also bounds the rounding of the arguments (f16 spacing grows with the
// magnitude): 2 keeps an argument above the running max within 2^-11, at the price of a few more O rescales in the
// first tiles of a row.  Instance parameter "rescale_log2_x100".
std::atomic<int64_t> g_rescale_half_x100{200};

std::atomic<int64_t> g_use_sm100{1};
std::atomic<int64_t> g_use_sm100_bias{1};    // elementwise bias tensors (hdim 128, contiguous) on the tcgen05 instance (0: general)
std::atomic<int64_t> g_last_bias_form{-1};   // how the last bias tensor of this process came: 1 by TMA, 0 by the threads ("last_bias_form", read-only)
std::atomic<int64_t> g_use_sm100_fp8{1};     // 8-bit prefill (hdim 128, contiguous) on the tcgen05 instance (0: general)
std::atomic<int64_t> g_use_sm100_hdim64{1};  // hdim-64 prefill on the tcgen05 instance (0: on the general one)
// exponentials of the softmax (template parameter EXPM of the kernel): 0 fp32 on the exp2 unit, 1 packed f16x2 on the
// exp2 unit, 11 / 12 / 13 fp32 with 1 / 2 / 3 of every 8 column pairs on an FMA-pipe polynomial
// (measured on B200, BASELINE config 2, bf16: 0 -> 962 TFLOP/s; 1 -> 915 at a rescale threshold of 4 and up, 866 at 2,
// with the LSE of a row that one late key dominates off by up to 9.7e-4; 11 / 12 / 13 -> 934 / 916 / 883: the unpacking
// of the packed results and the polynomial both cost the softmax warps more issue slots than the exp2 unit gives back)
std::atomic<int64_t> g_exp_mode{0};
std::atomic<int64_t> g_exp_mode_splitkv{0};
std::atomic<int64_t> g_use_sm100_splitkv{1};  // multi-token split-KV on the tcgen05 instance
std::atomic<int64_t> g_split_item_cost{kItemCostDefault};
std::atomic<int64_t> g_split_min_piece_tiles{8};  // instance parameter "split_min_piece_tiles": at least 1024 keys per work item

int64_t split_cap_tiles(const SplitKVParams& p) {  // key tiles of the longest sequence the cache can hold
    const int64_t cap = p.block_table ? p.bt_stride * p.page : p.seqlen_k_cap;
    return (cap + BN - 1) / BN;
}
// At most 64 packed rows and room for two splits per piece: the rows are duplicated (kernel mode 2).
bool split_duplicates_rows(const SplitKVParams& p) {
    return p.max_seqlen_q * (p.hq / p.hkv) <= 64 && p.num_splits >= 2;
}

}  // namespace

bool fwd_sm100_supported(const FwdParams& p) {
    if (!g_use_sm100.load()) return false;
    if (p.d != p.dv || (p.d != 128 && p.d != 64)) return false;
    if (p.d == 64 && !g_use_sm100_hdim64.load()) return false;
    if (p.dtype == FLASHCK_DTYPE_FLOAT8 || p.dtype == FLASHCK_DTYPE_BFLOAT8) {
        // the 8-bit instances: hdim 128, contiguous K/V, no score additions
        if (!g_use_sm100_fp8.load() || p.d != 128 || p.bias || p.logits_soft_cap > 0.f || p.block_table || p.kv_indptr) return false;
    }
    if (p.bias && p.bias_type == 1) {
        // an elementwise bias tensor: the BIAS instances (hdim 128, contiguous K/V of the stated length, 16-bit elements)
        if (!g_use_sm100_bias.load() || p.d != 128 || p.block_table || p.kv_indptr || p.bias_rank > 2) return false;
        if (p.bias_rank == 2 && p.seqstart_q) return false;
    }
    if (p.bias && p.bias_type == 2 && p.bias_rank > 1) return false;
    const bool paged = p.block_table || p.kv_indptr;
    if (paged) {
        // pages of 16 .. 128 tokens that divide a 128-key tile, or whole multiples of it
        if (p.page < 16 || !((BN % p.page == 0) || (p.page % BN == 0))) return false;
        if (p.seqlen_k64 || p.seqstart_k) return false;
        if (p.kv_indptr && (!p.kv_page_indices || !p.kv_last_page_len || p.cache_batch_idx)) return false;
    } else {
        if (p.cache_batch_idx || p.seqlen_k64 || p.seqlen_k32) return false;
        if ((p.seqstart_q == nullptr) != (p.seqstart_k == nullptr)) return false;
    }
    if (p.mask_type > 3) return false;
    if (p.wl >= (1ll << 30) || p.wr >= (1ll << 30)) return false;
    if (p.batch > kMaxBatch || (p.max_seqlen_q + BM - 1) / BM > kMaxLevels) return false;  // on-chip schedule
    if (p.hq > 1023) return false;
    {   // work items per CTA, bounded from the longest sequence: the on-chip work list holds kMaxRounds
        const bool pair = (p.hq / p.hkv) % 2 == 0;
        const int64_t rows_per_block = pair ? BM : 2 * BM;
        const int64_t items = p.batch * ((p.max_seqlen_q + rows_per_block - 1) / rows_per_block) * (pair ? p.hq / 2 : p.hq);
        if ((items + sm_count() - 1) / sm_count() > kMaxRounds) return false;
    }
    if (p.total_q >= (1ll << 31) || (!paged && p.batch * p.seqlen_k >= (1ll << 31))) return false;
    if (paged && p.num_pages * p.page >= (1ll << 31)) return false;  // token rows of the pools are 31-bit coordinates
    if (p.batch * std::max<int64_t>(p.seqlen_q, 1) >= (1ll << 31)) return false;
    return true;
}

// An elementwise bias by TMA: its rows start on 16-byte boundaries (a whole number of 8 keys, an aligned buffer), a row holds at
// least one box, and a sequence's block starts at a row's first key (batch mode: in the packed form it starts anywhere, and a
// copy must start on a 16-byte boundary).  Everything else is fetched by the softmax threads.  us by the threads / by TMA: 2 x 2048 tokens
// of 16 heads, a plane per head 216 / 109, causal 116 / 58, one plane 208 / 88; a plane per batch, 4 x 1024, 116 / 53; one plane behind a
// window of 511, 4096 tokens, 150 / 107; 8 x 64 tokens 9.8 / 9.0; 16 x 72, 8 heads 10.0 / 10.0.
static bool bias_by_tma(const FwdParams& p) {
    return !p.seqstart_q && p.seqlen_k >= 64 && p.seqlen_k % 8 == 0 && (reinterpret_cast<uintptr_t>(p.bias) & 15u) == 0 &&
           p.seqlen_q < (1ll << 31) && p.seqlen_k < (1ll << 31);
}

int launch_fwd_sm100(const FwdParams& p, cudaStream_t stream) {
    int* status = device_status_ptr();
    if (!status) return FLASHCK_ERR_CUDA;
    Sm100Dev dev{};
    dev.o = p.o; dev.lse = p.lse; dev.seqstart_q = p.seqstart_q; dev.seqstart_k = p.seqstart_k; dev.status = status;
    dev.batch = (int)p.batch; dev.seqlen_q = (int)p.seqlen_q; dev.seqlen_k = (int)p.seqlen_k;
    dev.hq = (int)p.hq; dev.hkv = (int)p.hkv; dev.total_q = (int)p.total_q;
    dev.v = p.v;
    dev.page_ids = p.kv_indptr ? p.kv_page_indices : p.block_table;
    dev.kv_indptr = p.kv_indptr; dev.kv_last_page_len = p.kv_last_page_len; dev.seqlen_k32 = p.seqlen_k32;
    dev.cache_batch_idx = p.cache_batch_idx;
    dev.page = (p.block_table || p.kv_indptr) ? (int)p.page : 0;
    dev.bt_stride = (int)p.bt_stride;
    dev.causal = p.mask_type;
    dev.wl = p.wl < 0 ? -1 : (int)p.wl;
    dev.wr = p.wr < 0 ? -1 : (int)p.wr;
    dev.pair_heads = ((p.hq / p.hkv) % 2 == 0) ? 1 : 0;
    dev.num_levels = (int)((p.max_seqlen_q + (dev.pair_heads ? BM : 2 * BM) - 1) / (dev.pair_heads ? BM : 2 * BM));
    {   // the work list (see the schedule in the kernel)
        const auto inverse = [](int64_t d) { return d > 1 ? (uint32_t)(((1ll << 32) + d - 1) / d) : 0u; };
        dev.uniform = !p.seqstart_q && !p.seqstart_k && !p.kv_indptr && !p.seqlen_k32;
        // (without a pair of heads a block is two row tiles: an odd number of tiles leaves a last block of one)
        dev.light = !dev.pair_heads && ((p.max_seqlen_q + BM - 1) / BM) % 2 != 0 ? 1 : 0;
        dev.inv_per_group = inverse(dev.pair_heads ? p.hq / 2 : p.hq);
        dev.inv_inner = inverse(p.mask_type != 0 || (p.bias && p.bias_type == 1) ? p.batch : dev.num_levels - dev.light);
    }
    dev.scale_log2 = p.scale * 1.4426950408889634f;
    const bool bf16 = p.dtype == FLASHCK_DTYPE_BFLOAT16;
    const bool window = p.mask_type != 0 && !(p.wl < 0 && p.wr == 0);
    const bool ebias = p.bias && p.bias_type == 1;
    const bool extra = (p.bias && p.bias_type == 2) || p.logits_soft_cap > 0.f;
    const int expm = extra ? 0 : (int)g_exp_mode.load();
    dev.rescale_thr = expm == 1 ? 0.01f * (float)g_rescale_half_x100.load() : kRescaleThreshold;
    dev.soft_cap = p.logits_soft_cap;
    if (p.logits_soft_cap > 0.f) {
        const float k = p.scale * (1.f / p.logits_soft_cap), c0 = dev.scale_log2;
        SoftCap& s = dev.cap;
        // The coefficients carry powers of k up to the eighth, so that the raw score itself is the variable.  Where the last
        // one leaves the range in which products keep 24 bits (a scale of 0.0884 with caps above 2000, say), the score is
        // multiplied by k first instead, in the branch that has both forms.
        const auto last = [&](float kk) { return 0.017135002f * (c0 * (kk * kk) * (kk * kk)); };
        const float l = fabsf(last(k * k));
        const bool powers = fabsf(k) < 1e3f && l > 1e-36f && l < 1e36f;
        const float kk = powers ? k * k : 1.f;
        s.lim = 0.5f / fabsf(k); s.lim_all = powers ? s.lim : -1.f; s.k = k;
        s.c0 = c0; s.c1 = -0.33333069f * (c0 * kk); s.c2 = 0.13324779f * (c0 * kk * kk);
        s.c3 = -0.052986056f * (c0 * kk * kk * kk); s.c4 = last(kk);
        s.k2e = 2.885390081777927f * k; s.c = copysignf(p.logits_soft_cap * kLog2e, k); s.m2c = -2.f * s.c;
    }
    dev.alibi = (p.bias && p.bias_type == 2) ? (const float*)p.bias : nullptr; dev.alibi_rank = p.bias_rank;
    if (p.dtype == FLASHCK_DTYPE_FLOAT8 || p.dtype == FLASHCK_DTYPE_BFLOAT8) {
        // The running max may lag the row max by `thr` (P up to 2^thr) only as far as P * scale_p stays inside the 8-bit
        // format: thr = log2(largest finite value / scale_p), at most the 16-bit instances' threshold, at least 0 (the
        // max then follows every increase).  scale_p = 256: 0.8 for E4M3 (max 448), 7.8 for E5M2 (max 57344).
        {
            const float fmt_max = p.dtype == FLASHCK_DTYPE_FLOAT8 ? 448.f : 57344.f;
            const float thr = log2f(fmt_max / p.scale_p);
            dev.rescale_thr = thr < 0.f ? 0.f : (thr > kRescaleThreshold ? kRescaleThreshold : thr);
        }
        dev.scale_p = p.scale_p; dev.scale_o = p.scale_o; dev.out_dtype = p.out_dtype;
        const bool e4 = p.dtype == FLASHCK_DTYPE_FLOAT8;
        if (window) return e4 ? launch_t<f8e4m3_t, 0, 1, 0>(p, dev, stream) : launch_t<f8e5m2_t, 0, 1, 0>(p, dev, stream);
        return e4 ? launch_t<f8e4m3_t, 0, 0, 0>(p, dev, stream) : launch_t<f8e5m2_t, 0, 0, 0>(p, dev, stream);
    }
    if (ebias) {  // (an elementwise bias: fp32 exponentials on the exp2 unit, with or without a second mask bound)
        dev.rescale_thr = kRescaleThreshold;
        dev.bias_el = p.bias; dev.bias_el_rank = p.bias_rank;
        dev.bias_sk = p.seqlen_k; dev.bias_sq = p.seqstart_q ? p.total_q : p.seqlen_q;
        g_last_bias_form = bias_by_tma(p) ? 1 : 0;
        if (bias_by_tma(p)) {
            if (window) return bf16 ? launch_t<__nv_bfloat16, 0, 13, 0>(p, dev, stream) : launch_t<__half, 0, 13, 0>(p, dev, stream);
            return bf16 ? launch_t<__nv_bfloat16, 0, 12, 0>(p, dev, stream) : launch_t<__half, 0, 12, 0>(p, dev, stream);
        }
        if (window) return bf16 ? launch_t<__nv_bfloat16, 0, 5, 0>(p, dev, stream) : launch_t<__half, 0, 5, 0>(p, dev, stream);
        return bf16 ? launch_t<__nv_bfloat16, 0, 4, 0>(p, dev, stream) : launch_t<__half, 0, 4, 0>(p, dev, stream);
    }
#define FCK_SM100_LAUNCH(E, V) \
    return bf16 ? launch_t<__nv_bfloat16, E, V, 0>(p, dev, stream) : launch_t<__half, E, V, 0>(p, dev, stream)
    if (p.d == 64) {  // the hdim-64 instances: fp32 exponentials on the exp2 unit, every mask and score addition
        dev.rescale_thr = kRescaleThreshold;
        switch ((window ? 1 : 0) | (extra ? 2 : 0)) {
            case 0: return bf16 ? launch_t<__nv_bfloat16, 0, 0, 0, 64>(p, dev, stream) : launch_t<__half, 0, 0, 0, 64>(p, dev, stream);
            case 1: return bf16 ? launch_t<__nv_bfloat16, 0, 1, 0, 64>(p, dev, stream) : launch_t<__half, 0, 1, 0, 64>(p, dev, stream);
            case 2: return bf16 ? launch_t<__nv_bfloat16, 0, 2, 0, 64>(p, dev, stream) : launch_t<__half, 0, 2, 0, 64>(p, dev, stream);
            default: return bf16 ? launch_t<__nv_bfloat16, 0, 3, 0, 64>(p, dev, stream) : launch_t<__half, 0, 3, 0, 64>(p, dev, stream);
        }
    }
    if (extra) {  // (the score-addition instances take their exponentials in fp32 on the exp2 unit)
        if (window) { FCK_SM100_LAUNCH(0, 3); }
        FCK_SM100_LAUNCH(0, 2);
    }
    if (window) {  // (the window instances come with the two exp2-unit forms only)
        if (expm == 1) { FCK_SM100_LAUNCH(1, 1); }
        FCK_SM100_LAUNCH(0, 1);
    }
    switch (expm) {
        case 1: FCK_SM100_LAUNCH(1, 0);
        case 11: FCK_SM100_LAUNCH(11, 0);
        case 12: FCK_SM100_LAUNCH(12, 0);
        case 13: FCK_SM100_LAUNCH(13, 0);
        default: FCK_SM100_LAUNCH(0, 0);
    }
#undef FCK_SM100_LAUNCH
}

bool splitkv_sm100_supported(const SplitKVParams& p) {
    if (!g_use_sm100_splitkv.load()) return false;
    if (p.alibi_slopes) return false;  // ALiBi runs on the mma.sync decode kernel
    if (p.d != HD || p.dv != HD || p.batch <= 0 || p.batch > kMaxBatch || p.hq > 1023) return false;
    const int64_t group = p.hq / p.hkv;
    if (group > BM || BM % group != 0) return false;
    // one 16-row tile of (token, group head) rows is what the mma.sync decode kernel serves at the HBM rate
    if (p.max_seqlen_q * group <= 16) return false;
    if ((p.max_seqlen_q * group + BM - 1) / BM > 16) return false;
    if (p.seqstart_k) return false;                           // paged or [rows, seqlen_k, hkv, d] caches
    if (p.mask_type > 2 || (p.mask_type != 0 && !(p.wl < 0 && p.wr == 0))) return false;  // none or causal
    if (p.block_table) {
        if (p.page < 16 || !((BN % p.page == 0) || (p.page % BN == 0)) || p.cache_batch_idx) return false;
    } else if (p.seqlen_k_cap <= 0 || p.cache_batch_idx) {
        return false;  // (with cache_batch_idx the number of cache rows is not known here: see the K/V maps)
    }
    if (p.num_splits > 1 && !p.lse_acc) return false;
    if (p.num_splits > 255) return false;  // the split index of a work item has 8 bits
    // The work line (see kItemCostDefault) is indexed with 31 bits, and a CTA's work list holds kSplitItems items: a CTA's
    // piece of w units reaches into at most w / item_cost + 2 streams, and w is at most the larger of the line's
    // 148th, the shortest piece, and what keeps the longest possible stream within the workspace's splits.
    const int64_t cap_tiles = split_cap_tiles(p);
    const int64_t streams = p.batch * p.hkv * ((p.max_seqlen_q * group + BM - 1) / BM);
    const int64_t item_cost = g_split_item_cost.load(), min_piece = g_split_min_piece_tiles.load();
    const int64_t line = streams * (cap_tiles + item_cost);
    if (line >= (1ll << 31)) return false;
    const int64_t max_pieces = std::max<int64_t>(1, split_duplicates_rows(p) ? p.num_splits / 2 : p.num_splits);
    int64_t w_max = std::max<int64_t>(line / sm_count() + 1, min_piece + item_cost);
    if (max_pieces >= 2) w_max = std::max(w_max, cap_tiles / (max_pieces - 1) + 1);
    if (std::min(streams, w_max / item_cost + 2) > kSplitItems) return false;
    const int64_t tokens = p.seqstart_q ? p.total_q : p.batch * p.seqlen_q;
    if (tokens >= (1ll << 31) || (!p.block_table && p.batch * p.seqlen_k_cap >= (1ll << 31))) return false;
    if (p.block_table && p.num_pages * p.page >= (1ll << 31)) return false;
    return true;
}

int launch_splitkv_sm100(const SplitKVParams& p, cudaStream_t stream) {
    int* status = device_status_ptr();
    if (!status) return FLASHCK_ERR_CUDA;
    if (p.batch == 0 || p.max_seqlen_q == 0) return FLASHCK_OK;
    Sm100Dev dev{};
    dev.o = nullptr; dev.lse = nullptr; dev.seqstart_q = p.seqstart_q; dev.seqstart_k = nullptr; dev.status = status;
    dev.batch = (int)p.batch; dev.seqlen_q = (int)p.seqlen_q; dev.seqlen_k = (int)p.seqlen_k_cap;
    dev.hq = (int)p.hq; dev.hkv = (int)p.hkv; dev.total_q = (int)p.total_q;
    dev.v = p.v;
    dev.page_ids = p.block_table; dev.seqlen_k32 = p.seqlen_k; dev.cache_batch_idx = p.cache_batch_idx;
    // a contiguous cache goes through the chunked loader too (chunk = 128 tokens): the rows behind a sequence's end
    // are uninitialised cache, which the loader keeps out of V
    dev.page = p.block_table ? (int)p.page : BN;
    dev.bt_stride = (int)p.bt_stride;
    dev.o_acc = p.o_acc; dev.lse_acc = p.lse_acc; dev.num_splits = (int)p.num_splits;
    dev.piece_tiles = (int)g_split_min_piece_tiles.load();
    dev.item_cost = (int)g_split_item_cost.load();
    dev.group = (int)(p.hq / p.hkv);
    dev.sq_cap = (int)p.seqlen_q;
    dev.causal = p.mask_type; dev.wl = -1; dev.wr = p.mask_type ? 0 : -1;
    dev.pair_heads = 0; dev.num_levels = 1;
    dev.scale_log2 = p.scale * 1.4426950408889634f;
    const bool bf16 = p.dtype == FLASHCK_DTYPE_BFLOAT16;
    const bool hexp = g_exp_mode_splitkv.load() == 1;
    dev.rescale_thr = hexp ? 0.01f * (float)g_rescale_half_x100.load() : kRescaleThreshold;
    if (split_duplicates_rows(p)) {
        if (hexp) return bf16 ? launch_split_t<__nv_bfloat16, 2, 1>(p, dev, stream) : launch_split_t<__half, 2, 1>(p, dev, stream);
        return bf16 ? launch_split_t<__nv_bfloat16, 2, 0>(p, dev, stream) : launch_split_t<__half, 2, 0>(p, dev, stream);
    }
    if (hexp) return bf16 ? launch_split_t<__nv_bfloat16, 1, 1>(p, dev, stream) : launch_split_t<__half, 1, 1>(p, dev, stream);
    return bf16 ? launch_split_t<__nv_bfloat16, 1, 0>(p, dev, stream) : launch_split_t<__half, 1, 0>(p, dev, stream);
}

static bool valid_exp_mode(int64_t v) { return v == 0 || v == 1 || (v >= 11 && v <= 13); }

int fwd_set_param(const char* key, int64_t value) {
    if (!strcmp(key, "use_sm100")) { g_use_sm100 = value; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_hdim64")) { g_use_sm100_hdim64 = value; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_fp8")) { g_use_sm100_fp8 = value; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_bias")) { g_use_sm100_bias = value; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_splitkv")) { g_use_sm100_splitkv = value; return FLASHCK_OK; }
    if (!strcmp(key, "exp_mode")) {
        if (!valid_exp_mode(value)) return FLASHCK_ERR_INVALID_ARGUMENT;
        g_exp_mode = value;
        return FLASHCK_OK;
    }
    if (!strcmp(key, "exp_mode_splitkv")) {
        if (value != 0 && value != 1) return FLASHCK_ERR_INVALID_ARGUMENT;
        g_exp_mode_splitkv = value;
        return FLASHCK_OK;
    }
    if (!strcmp(key, "split_item_cost")) {
        if (value < 1 || value > 64) return FLASHCK_ERR_INVALID_ARGUMENT;
        g_split_item_cost = value;
        return FLASHCK_OK;
    }
    if (!strcmp(key, "split_min_piece_tiles")) {
        if (value < 1 || value > 4096) return FLASHCK_ERR_INVALID_ARGUMENT;
        g_split_min_piece_tiles = value;
        return FLASHCK_OK;
    }
    if (!strcmp(key, "rescale_log2_x100")) {
        if (value < 0 || value > 1400) return FLASHCK_ERR_INVALID_ARGUMENT;  // f16 holds 2^15; P < 2^14 leaves headroom
        g_rescale_half_x100 = value;
        return FLASHCK_OK;
    }
    if (!strcmp(key, "poly8")) {  // older spelling: the polynomial share alone (0 = exp2 unit in fp32)
        if (value < 0 || value > 3) return FLASHCK_ERR_INVALID_ARGUMENT;
        g_exp_mode = value ? 10 + value : 0;
        return FLASHCK_OK;
    }
    return FLASHCK_ERR_INVALID_ARGUMENT;
}
int fwd_get_param(const char* key, int64_t* value) {
    if (!strcmp(key, "use_sm100")) { *value = g_use_sm100; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_hdim64")) { *value = g_use_sm100_hdim64; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_fp8")) { *value = g_use_sm100_fp8; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_bias")) { *value = g_use_sm100_bias; return FLASHCK_OK; }
    if (!strcmp(key, "last_bias_form")) { *value = g_last_bias_form; return FLASHCK_OK; }
    if (!strcmp(key, "use_sm100_splitkv")) { *value = g_use_sm100_splitkv; return FLASHCK_OK; }
    if (!strcmp(key, "exp_mode")) { *value = g_exp_mode; return FLASHCK_OK; }
    if (!strcmp(key, "exp_mode_splitkv")) { *value = g_exp_mode_splitkv; return FLASHCK_OK; }
    if (!strcmp(key, "rescale_log2_x100")) { *value = g_rescale_half_x100; return FLASHCK_OK; }
    if (!strcmp(key, "split_item_cost")) { *value = g_split_item_cost; return FLASHCK_OK; }
    if (!strcmp(key, "split_min_piece_tiles")) { *value = g_split_min_piece_tiles; return FLASHCK_OK; }
    if (!strcmp(key, "poly8")) { const int64_t m = g_exp_mode; *value = m >= 11 ? m - 10 : 0; return FLASHCK_OK; }
    return FLASHCK_ERR_INVALID_ARGUMENT;
}

}  // namespace fck
