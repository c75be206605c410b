// Host side of the tensor-core convolution: which load mode, tile and shared-memory plan a geometry takes, the tensor maps, and
// the launch.  The kernel is in conv_tc_kernel.cuh, its instances in the object files of conv_tc_inst.cu.
#include "conv_tc_kernel.cuh"

#include <cudaTypedefs.h>

#include <algorithm>

namespace tsb {
namespace tc {

#define TSB_TC_EXTERN(BN_, BK_, SWAP_, MODE_, EPI_, DUAL_)                                                                         \
    extern template int launch<BN_, BK_, SWAP_, MODE_, EPI_, DUAL_>(const Config &, const CUtensorMap &, const CUtensorMap &,     \
                                                              const CUtensorMap &, const CUtensorMap &, const CUtensorMap &, \
                                                              const KernelParams &, const EpiParams &, cudaStream_t,         \
                                                              const std::conditional_t<DUAL_, DualParams, NoDual> &);
TSB_TC_ALL(TSB_TC_EXTERN)
#undef TSB_TC_EXTERN

namespace {

#ifdef TSB_ENABLE_TRACE
unsigned long long *g_trace = nullptr;  // set through set_trace_buffer()
#endif
PFN_cuTensorMapEncodeTiled_v12000 g_encode_tiled = nullptr;
PFN_cuTensorMapEncodeIm2col_v12000 g_encode_im2col = nullptr;

int load_driver() {
    if (g_encode_tiled && g_encode_im2col) return TSB_OK;
    cudaDriverEntryPointQueryResult q;
    void *fn = nullptr;
    TSB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !fn) return fail(TSB_ERR_UNSUPPORTED, "driver lacks cuTensorMapEncodeTiled");
    g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    TSB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !fn) return fail(TSB_ERR_UNSUPPORTED, "driver lacks cuTensorMapEncodeIm2col");
    g_encode_im2col = reinterpret_cast<PFN_cuTensorMapEncodeIm2col_v12000>(fn);
    return TSB_OK;
}

CUtensorMapSwizzle swizzle_for(int bk) {
    return bk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (bk == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

}  // namespace

#ifdef TSB_ENABLE_TRACE
void set_trace_buffer(unsigned long long *device_buffer) { g_trace = device_buffer; }
#endif

bool make_view(const ConvGeom &g, const Tuning &tune, View *view, const char **why) {
    *why = "";
    View v;
    v.real = g;
    v.g = g;
    if (g.pad_value != 0) { *why = "non-zero padding_value"; return false; }
    if (g.C <= 16) {
        // fold the filter row into the channel dimension
        const int cpix = (g.C <= 8 && g.sw % 2 == 0) ? 8 : 16;
        const int span = (g.KW - 1) * g.dw + 1;
        const int bkf = round_up(span * cpix, 64);
        if (bkf > 128) { *why = "filter row too wide to fold into one K block"; return false; }
        const int unit = 32 / cpix;  // pixels per 32 bytes: rows of the staging are whole 32-byte units (what one thread of
                                     // the staging quantize writes)
        const int need = std::max(g.W + g.pad_l, (g.OW - 1) * g.sw + bkf / cpix);
        v.fold = 1;
        v.cpix = cpix;
        v.Wp = round_up(need, unit);
        v.g.C = bkf; v.g.Cp = bkf; v.g.W = g.OW; v.g.KW = 1; v.g.sw = 1; v.g.dw = 1; v.g.pad_l = 0;
        v.stride_w = (uint64_t)g.sw * cpix;
        v.stride_h = (uint64_t)v.Wp * cpix;
        v.stride_n = v.stride_h * g.H;
        v.stage_bytes = (size_t)v.stride_n * g.N;
        // raw-row mode: pixel stride of exactly one 16-byte unit, every output row meets at least one input row, and
        // output rows long enough to fill most of a 128-pixel tile (tune.rows forces it on/off where it is possible)
        bool rows_ok = v.stride_w == 16 && (size_t)g.KH * bkf * std::min(round_up(g.O, 64), 256) <= 96 * 1024 &&
                       (size_t)(g.KH - 1) * g.dh * v.stride_h + (size_t)ceil_div(g.OW, kBM) * kBM * 16 + 2048 <= 48 * 1024;
        for (int oh = 0; oh < g.OH && rows_ok; ++oh) {
            bool any = false;
            for (int kh = 0; kh < g.KH; ++kh) {
                const int ih = oh * g.sh - g.pad_t + kh * g.dh;
                any = any || (ih >= 0 && ih < g.H);
            }
            rows_ok = any;
        }
        const int segs = ceil_div(g.OW, kBM);
        const bool rows_pay = (double)g.OW / (double)(segs * kBM) >= 0.75;
        if (rows_ok && (tune.rows ? tune.rows == 2 : rows_pay)) {
            v.rows = 1;
            v.rows_segs = segs;
            v.stage_bytes += (size_t)kBM * 16 + 256;   // the copy under the last tile of the last row runs past the row's end
        }
    } else {
        if (g.Cp % 64 != 0) { *why = "channel padding is not a multiple of 64"; return false; }
        v.stride_w = (uint64_t)g.Cp;
        v.stride_h = (uint64_t)g.Cp * g.W;
        v.stride_n = v.stride_h * g.H;
        v.stage_bytes = (size_t)v.stride_n * g.N;
    }
    v.a_tiled = (!v.fold && g.KH == 1 && g.KW == 1 && g.sh == 1 && g.sw == 1 && g.pad_t == 0 && g.pad_l == 0 &&
                 g.OH == g.H && g.OW == g.W) ? 1 : 0;
    if (!v.fold && !v.a_tiled && g.KH * g.KW > 1 && tune.patch != 1) {
        if (g.sh == 1 && g.sw == 1 && (g.KW - 1) * g.dw + 8 <= 256 && (g.KH - 1) * g.dh + 32 <= 256) v.patch = 1;
        // (stride 2 over 64 padded channels: 297 rows of 128 bytes a tile instead of the 1152 im2col rows of 64 bytes, at some 4.5 cycles a row;
        // CSPDarknet53, whose 32 -> 64 and 64 -> 128 layers at 608 and 304 take it, 16 images 2.37 -> 2.21 ms, one image 0.511 -> 0.501)
        else if (g.sh == 2 && g.sw == 2 && g.dh == 1 && g.dw == 1 && g.Cp == 64 && g.W % 2 == 0 && g.KW <= 128 && g.KH <= 128) v.patch = 2;
    }
    const ConvGeom &t = v.g;
    v.weight_bytes = (size_t)t.O * t.KH * t.KW * t.Cp;
    // im2col tensor maps take box corners in [-128,127], filter offsets in [0,255] and traversal strides up to 8
    const int up_w = (t.OW - 1) * t.sw - t.pad_l - (t.W - 1);
    const int up_h = (t.OH - 1) * t.sh - t.pad_t - (t.H - 1);
    if (t.pad_t > 128 || t.pad_l > 128 || t.pad_t < 0 || t.pad_l < 0 || up_w < -128 || up_w > 127 || up_h < -128 || up_h > 127) {
        *why = "padding beyond the im2col corner range";
        return false;
    }
    if ((t.KW - 1) * t.dw > 255 || (t.KH - 1) * t.dh > 255) { *why = "filter extent beyond the im2col offset range"; return false; }
    if (t.sh > 8 || t.sw > 8) { *why = "stride beyond the traversal-stride range"; return false; }
    if ((int64_t)t.N * t.OH * t.OW > INT32_MAX - 256) { *why = "too many output pixels"; return false; }
    if ((int64_t)t.N * t.O * t.OH * t.OW > UINT32_MAX) { *why = "output too large for 32-bit indexing"; return false; }
    if (v.stage_bytes > (size_t)INT32_MAX) { *why = "staged input too large"; return false; }
    *view = v;
    return true;
}

bool wants_staging(const View &v, const EpiParams &epi) {
    const ConvGeom &g = v.real;
    if (epi.out_acc) return false;
    const bool per_sample = epi.nscales > 1 && epi.nscales == g.N && epi.group_len == (uint32_t)(g.O * g.OH * g.OW);
    if (epi.out_i8 && !(epi.i8_nhwc && (epi.nscales == 1 || per_sample))) return false;
    if (epi.out_i8 && reinterpret_cast<uintptr_t>(epi.out_i8) % 16) return false;
    const bool f32_tiles = (epi.out_f32 || epi.residual) && epi.f32_nhwc;
    if (f32_tiles) {
        // tensor maps over [pixels][O] fp32: rows must be whole 16-byte units, the tensors 16-byte aligned and distinct
        if (g.O % 4 != 0 || (const void *)epi.residual == (const void *)epi.out_f32) return false;
        if ((reinterpret_cast<uintptr_t>(epi.out_f32) | reinterpret_cast<uintptr_t>(epi.residual)) % 16) return false;
        return true;
    }
    // fp32 NCHW output, or int8 NHWC_PAD alone: the direct paths (a thread's 32 int8 channels are one 32-byte sector,
    // which two 16-byte stores write as well as a tile store would)
    return false;
}

// Shared memory of the staged epilogue: per quad `tiles` fp32 tiles and an int8 tile.
static uint32_t staged_bytes(int tiles) { return tiles ? kQuads * ((uint32_t)tiles * kStageF32Bytes + kStageI8Bytes) : 0u; }

// bytes of K from which on a layer of few tiles is split
constexpr int kSplitMinK = 2048;

// tiles_per_quad: fp32 tiles per quad of the staged epilogue, 0: not staged
static Config plan_config(const View &v, const Tuning &tune, int sm_count, int orientation, int tiles_per_quad) {
    const ConvGeom &g = v.g;
    Config c;
    c.bk = (g.Cp % 128 == 0) ? 128 : 64;
    const int64_t M = (int64_t)g.N * g.OH * g.OW;
    uint32_t stg_bytes = staged_bytes(tiles_per_quad), budget = kSmemBudget - stg_bytes;
    // An MMA instruction costs the issuing warp 77-115 cycles whatever its N (the tensor core 128 at N = 256, 64 at 128, 48 at 64), so N should
    // be 256 whenever possible.
    // Normal orientation: 128 pixels on M, up to 256 output channels on N.  Swapped orientation: channels on M,
    // 256 (or 128) pixels on N -- it halves the MMA count of narrow layers but its epilogue (one channel per thread)
    // is dearer, so it is taken where it measured faster: multi-tap filters with at most 64 output channels.
    // patch mode under a given tile shape: most of each 8 x (pix/8) tile inside the image, and the whole weight tile
    // in shared memory beside at least two patches (tune.patch == 2 drops the first condition)
    // (extent of a patch in pixels or pixel pairs; a row of it in bytes)
    auto patch_extent = [&](int pix, int *pw, int *ph) {
        const int th = pix / 8;
        if (v.patch == 2) {
            *pw = 8 + (g.KW - 1 - g.pad_l >= 0 ? (g.KW - 1 - g.pad_l) / 2 : -((g.pad_l - g.KW + 2) / 2)) + (g.pad_l + 1) / 2;
            *ph = (th - 1) * 2 + g.KH;
        } else {
            *pw = 8 + (g.KW - 1) * g.dw;
            *ph = th + (g.KH - 1) * g.dh;
        }
    };
    const int patch_row = v.patch == 2 ? 128 : c.bk;
    auto patch_fits = [&](int pix, int ch) {
        if (!v.patch) return false;
        // (the swapped kernel has no fast path for pixel-major fp32 tensors in patch mode, which is what the swapped plan is kept for)
        if (v.patch == 2 && c.swap && tune.patch != 2) return false;
        const int th = pix / 8;
        const int tiles_w = ceil_div(g.OW, 8), tiles_h = ceil_div(g.OH, th);
        int pw, ph;
        patch_extent(pix, &pw, &ph);
        const double eff = (double)(g.OH * g.OW) / ((double)tiles_w * tiles_h * pix);
        const uint64_t patch_bytes = (uint64_t)round_up(pw * ph * patch_row, 1024);
        const uint64_t w_all = (uint64_t)g.KH * g.KW * g.Cp * (uint64_t)ch;
        return (eff >= 0.7 || tune.patch == 2) && w_all + 2 * patch_bytes <= budget;
    };
    const int bn_normal = g.O > 128 ? 256 : (g.O > 64 ? 128 : 64);
    // Split-K where clusters of kSplit CTAs, one per 128 x 128 tile, fit the GPU at once and a tile has K enough to pay for the exchange of
    // the partial sums (some 3 us with the cluster's launch).  Measured alone, cold, split against whole: 3x3 512 -> 512 at 7 x 7, 8 images,
    // 11.5 / 16 us; 3x3 512 -> 512 at 19 x 19, one image, 15 / 19 us; 3x3 256 -> 256 at 38 x 38 13.4 / 14.5; 1x1 1024 -> 256 at 14 x 14,
    // 8 images, 10 / 8.  Patch mode, which loads an activation once and not once per tap, stays ahead where it fits (256 -> 256 at 14 x 14,
    // 8 images, 9.5 / 10.5).  CSPDarknet53 of one image 0.535 -> 0.519 ms, ResNet-50 of 8 images 0.398 -> 0.395.
    const bool split = orientation < 0 && tune.orientation != 2 && tune.patch != 2 && !v.fold && g.KH * g.KW * g.Cp >= kSplitMinK &&
                       ceil_div64(M, kBM) * ceil_div(g.O, 128) * kSplit <= sm_count - sm_count / 8;
    if (v.rows || split) c.swap = 0;
    else if (orientation >= 0) c.swap = orientation;
    else if (tune.orientation) c.swap = tune.orientation == 2 && g.O <= 128;
    // narrow multi-tap layers: swapped fills the MMA's N, but where patch mode applies the normal orientation with its
    // cheaper epilogue (16 warps, 16-byte stores) measured faster
    else c.swap = g.O <= 64 && g.KH * g.KW >= 9 && !v.fold && !patch_fits(kBM, bn_normal);
    if (c.swap) {
        c.ch = kBM;
        c.bn = 256;
        if (ceil_div64(M, 256) < sm_count && ceil_div64(M, 128) > ceil_div64(M, 256)) c.bn = 128;  // few pixels: more, smaller tiles
        c.pix = c.bn;
    } else {
        c.bn = g.O > 128 ? 256 : (g.O > 64 ? 128 : 64);
        // the staged block epilogue over plain [pixels][channels] tiles (the 1x1 expansions of residual blocks) measured 3-5 %
        // faster with four 128-channel accumulators, one tile per epilogue quad, than with two 256-channel ones
        if (tiles_per_quad && v.a_tiled && c.bn == 256) c.bn = 128;
        const int m_tiles128 = (int)ceil_div64(M, kBM);
        // a narrower N tile when the wide one leaves most SMs idle or the last wave nearly empty
        while (c.bn > 64) {
            const int64_t tiles = (int64_t)m_tiles128 * ceil_div(g.O, c.bn);
            const int64_t waves = ceil_div64(tiles, sm_count);
            const double eff = (double)tiles / (double)(waves * sm_count);
            if (eff >= 0.8) break;
            const int64_t tiles2 = (int64_t)m_tiles128 * ceil_div(g.O, c.bn / 2);
            const double eff2 = (double)tiles2 / (double)(ceil_div64(tiles2, sm_count) * sm_count);
            if (eff2 <= eff) break;
            c.bn /= 2;
        }
        c.pix = kBM;
        c.ch = c.bn;
    }
    if (split && !patch_fits(c.pix, c.ch)) {
        c.split = 1;
        c.bn = c.ch = 128;
    }
    c.num_m_tiles = v.rows ? g.N * g.OH * v.rows_segs : (int)ceil_div64(M, c.pix);
    c.num_n_tiles = ceil_div(g.O, c.ch);
    if (!c.split && patch_fits(c.pix, c.ch)) {
        const int th = c.pix / 8;
        c.patch = v.patch;
        c.patch_tiles_w = ceil_div(g.OW, 8); c.patch_tiles_h = ceil_div(g.OH, th);
        patch_extent(c.pix, &c.patch_pw, &c.patch_ph);
        c.num_m_tiles = g.N * c.patch_tiles_w * c.patch_tiles_h;
    }
    const int64_t tiles = (int64_t)c.num_m_tiles * c.num_n_tiles;
    c.grid = c.split ? (int)tiles * kSplit : (int)(tiles < sm_count ? tiles : sm_count);
    if (c.split) budget = kSmemBudget - (stg_bytes = staged_bytes(1));   // the partial sums of the other CTAs arrive in the quads' fp32 tiles
    // shared-memory plan: keep the CTA's whole weight tile resident when it is small enough to leave room for
    // at least four activation stages; otherwise stream activations and weights together
    // raw-row mode stages, per output row, the KH staged image rows under all its segments of 128 sliding windows
    // (127 pixel strides of 16 bytes plus one window in the last segment)
    const uint32_t p_bytes = c.patch ? (uint32_t)round_up(c.patch_pw * c.patch_ph * patch_row, 1024) : v.rows ? (uint32_t)round_up((g.KH - 1) * g.dh * (int)v.stride_h + (v.rows_segs - 1) * kBM * 16 + (kBM - 1) * 16 + c.bk, 128)
                                    : (uint32_t)c.pix * c.bk;
    const uint32_t w_bytes = (uint32_t)c.ch * c.bk;
    const uint32_t k_iters = (uint32_t)g.KH * g.KW * (g.Cp / c.bk);
    const uint32_t w_total = k_iters * w_bytes;
    const bool want_resident = v.rows || c.patch || (tiles > c.grid && !c.split);  // pays off only when a CTA runs several tiles
    // (raw-row mode always keeps its weights resident; make_view admitted it only where two row stages fit beside them)
    const uint32_t min_stages = v.rows ? 2 : 4;
    // K blocks per stage (im2col / tiled loads only): the MMA issuer pays a barrier wait and a commit per stage, which
    // costs it more than the MMAs of one K block take when N is small, so short K blocks are grouped -- as long as the
    // group divides the K blocks of a tile, stays within 48 KB and leaves at least three stages.
    auto group_for = [&](uint32_t unit, uint32_t room) {
        if (c.patch || v.rows || c.split) return 1;
        for (int gsz = 4; gsz >= 2; gsz /= 2)
            if (k_iters % (uint32_t)gsz == 0 && (uint32_t)gsz * unit <= 48 * 1024 && room / ((uint32_t)gsz * unit) >= 3) return gsz;
        return 1;
    };
    if (c.patch || (want_resident && w_total <= 128 * 1024 && w_total < budget && (budget - w_total) / p_bytes >= min_stages)) {
        c.b_resident = 1;
        c.unit_bytes = p_bytes;
        c.kgroup = group_for(p_bytes, budget - w_total);
        c.stage_bytes = (uint32_t)c.kgroup * p_bytes;
        c.stages = std::min<int>(kMaxStages, (int)((budget - w_total) / c.stage_bytes));
        c.b_off = (uint32_t)c.stages * c.stage_bytes;
        c.bar_off = c.b_off + w_total;
    } else {
        c.b_resident = 0;
        c.unit_bytes = p_bytes + w_bytes;
        c.kgroup = group_for(c.unit_bytes, budget);
        c.stage_bytes = (uint32_t)c.kgroup * c.unit_bytes;
        c.stages = std::min<int>(kMaxStages, (int)(budget / c.stage_bytes));
        c.b_off = 0;
        c.bar_off = (uint32_t)c.stages * c.stage_bytes;
    }
    // the staged epilogue's tiles (1024-byte aligned for the 128B swizzle) sit between the pipeline and the barriers
    c.staging = c.swap ? 0 : (c.split ? std::min(tiles_per_quad, 1) : tiles_per_quad);
    // The more of a group's quads work on one tile, the closer together the CTA's copies lie in memory; but a quad needs a
    // chunk of its own (32 channels), and the tiles of a deep K come too slowly for one group to wait for each in turn.
    c.stg_groups = v.a_tiled ? (c.bn >= 128 ? 1 : 2) : (c.bn >= 128 ? 2 : 4);
    if (c.split) c.stg_groups = 1;
    if (c.staging || c.split) {
        c.stg_off = (c.bar_off + 1023u) & ~1023u;
        c.bar_off = c.stg_off + stg_bytes;
    }
    const uint32_t tables = ((c.bar_off + 8 * num_barriers(c.stages) + 8 + 15) & ~15u) + kMaxAccBufs * 2 * (uint32_t)c.bn * 4 +
                            (c.patch ? 4 * (uint32_t)(g.KH * g.KW) : 0);   // epilogue tables, then patch mode's tap table
    c.dyn_smem = tables + 1024;  // slack to align the tiles to 1024 bytes
    return c;
}

// Two fp32 tiles per quad for plain [pixels][channels] tiles (1x1 layers, which the copies bound) as long as two K blocks are left in
// flight, even where the weights then have to be streamed; one for filters of several taps, whose pipeline is worth more than
// the second tile.  Measured, two tiles against one, residual + fp32 + int8, 64 images: 128 -> 512 at 28 x 28 46 / 55 us,
// 256 -> 1024 at 14 x 14 26 / 34 us; 16 images, 3x3 64 -> 64 at 152 x 152 94 / 52 us, 128 -> 128 at 76 x 76 40 / 35 us.
Config choose_config(const View &v, const Tuning &tune, int sm_count, int orientation, bool staging) {
    if (staging && v.a_tiled) {
        const Config two = plan_config(v, tune, sm_count, orientation, 2);
        if (two.staging && two.stages >= 2) return two;
    }
    return plan_config(v, tune, sm_count, orientation, staging ? 1 : 0);
}

bool dual_supported(const View &v, const View &sc, const char **why) {
    const ConvGeom &g = v.g, &s = sc.g;
    *why = "";
    if (v.fold || v.rows || sc.fold || sc.rows) { *why = "folded inputs (at most 16 channels)"; return false; }
    if (s.KH != 1 || s.KW != 1 || s.pad_t != 0 || s.pad_l != 0) { *why = "the projection must be a 1x1 convolution without padding"; return false; }
    if (s.N != g.N || s.O != g.O || s.OH != g.OH || s.OW != g.OW) { *why = "the projection's output shape differs"; return false; }
    if ((s.H - 1) / s.sh + 1 != s.OH || (s.W - 1) / s.sw + 1 != s.OW) { *why = "the projection's padding is not zero on every side"; return false; }
    if (g.O % 4 != 0) { *why = "output channels not a multiple of 4"; return false; }
    return true;
}

static Config plan_config_dual(const View &v, const View &sc, int sm_count, int bn, bool concat, int tiles_per_quad) {
    const ConvGeom &g = v.g, &s = sc.g;
    Config c;
    c.bk = (g.Cp % 128 == 0 && s.Cp % 128 == 0) ? 128 : 64;
    c.swap = 0;
    // 128 channels per tile: four accumulator buffers hold two tiles, so the MMAs of one tile run under the epilogue of
    // the other (256 would fill tensor memory with a single tile; measured 10-25 % slower on the ResNet-50 shapes)
    c.bn = bn == 128 || bn == 256 ? bn : 128;
    if (concat && bn == 0 && g.O <= 64) c.bn = 64;      // one accumulator per tile: a narrow layer keeps its narrow tile
    c.pix = kBM;
    c.ch = c.bn;
    const int64_t M = (int64_t)g.N * g.OH * g.OW;
    c.num_m_tiles = (int)ceil_div64(M, c.pix);
    c.num_n_tiles = ceil_div(g.O, c.ch);
    const int64_t tiles = (int64_t)c.num_m_tiles * c.num_n_tiles;
    c.grid = (int)(tiles < sm_count ? tiles : sm_count);
    const uint32_t stg_bytes = staged_bytes(tiles_per_quad), budget = kSmemBudget - stg_bytes;
    const uint32_t p_bytes = (uint32_t)c.pix * c.bk, w_bytes = (uint32_t)c.ch * c.bk;
    const uint32_t k1 = (uint32_t)g.KH * g.KW * (g.Cp / c.bk), k2 = (uint32_t)(s.Cp / c.bk);
    const uint32_t w_total = (k1 + k2) * w_bytes;
    // K blocks per stage: a stage never mixes the two convolutions, so the group divides both block counts
    auto group_for = [&](uint32_t unit, uint32_t room) {
        for (int gsz = 4; gsz >= 2; gsz /= 2)
            if (k1 % (uint32_t)gsz == 0 && k2 % (uint32_t)gsz == 0 && (uint32_t)gsz * unit <= 48 * 1024 && room / ((uint32_t)gsz * unit) >= 3) return gsz;
        return 1;
    };
    if (tiles > c.grid && w_total <= 128 * 1024 && w_total < budget && (budget - w_total) / p_bytes >= 4) {
        c.b_resident = 1;
        c.unit_bytes = p_bytes;
        c.kgroup = group_for(p_bytes, budget - w_total);
        c.stage_bytes = (uint32_t)c.kgroup * p_bytes;
        c.stages = std::min<int>(kMaxStages, (int)((budget - w_total) / c.stage_bytes));
        c.b_off = (uint32_t)c.stages * c.stage_bytes;
        c.bar_off = c.b_off + w_total;
    } else {
        c.b_resident = 0;
        c.unit_bytes = p_bytes + w_bytes;
        c.kgroup = group_for(c.unit_bytes, budget);
        c.stage_bytes = (uint32_t)c.kgroup * c.unit_bytes;
        c.stages = std::min<int>(kMaxStages, (int)(budget / c.stage_bytes));
        c.b_off = 0;
        c.bar_off = (uint32_t)c.stages * c.stage_bytes;
    }
    c.staging = tiles_per_quad;
    c.stg_groups = 1;
    c.stg_off = (c.bar_off + 1023u) & ~1023u;
    c.bar_off = c.stg_off + stg_bytes;
    const uint32_t tables = ((c.bar_off + 8 * num_barriers(c.stages) + 8 + 15) & ~15u) + kMaxAccBufs * 2 * (uint32_t)c.bn * 4;
    c.dyn_smem = tables + 1024;
    return c;
}

// (Measured, two tiles per quad against one: 64 + 64 -> 256 at 56 x 56, 64 images, whose weights stay resident either way, 67 / 73 us;
// where the second tile evicts them, 128 + 256 -> 512 at 28 x 28 46 / 44 us and 256 + 512 -> 1024 at 14 x 14 33 / 28 us.)
Config choose_config_dual(const View &v, const View &sc, int sm_count, int bn, bool concat, bool staging) {
    const Config one = plan_config_dual(v, sc, sm_count, bn, concat, staging ? 1 : 0);
    if (!staging) return one;
    const Config two = plan_config_dual(v, sc, sm_count, bn, concat, 2);
    return two.b_resident == one.b_resident && two.stages >= 2 ? two : one;
}

int encode_weight_map(const View &v, const Config &cfg, const int8_t *w_packed, CUtensorMap *map) {
    int st = load_driver();
    if (st != TSB_OK) return st;
    const ConvGeom &g = v.g;
    const cuuint64_t ktot = (cuuint64_t)g.KH * g.KW * g.Cp;
    cuuint64_t dims[2] = {ktot, (cuuint64_t)g.O};
    cuuint64_t strides[1] = {ktot};
    cuuint32_t box[2] = {(cuuint32_t)cfg.bk, (cuuint32_t)cfg.ch};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(w_packed), dims, strides, box,
                                estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cfg.bk),
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TSB_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled(weights) failed with %d", (int)r);
    return TSB_OK;
}

int encode_activation_map(const View &v, const Config &cfg, const int8_t *x, CUtensorMap *map) {
    int st = load_driver();
    if (st != TSB_OK) return st;
    if (reinterpret_cast<uintptr_t>(x) % 16) return fail(TSB_ERR_INVALID_ARGUMENT, "staged activations must be 16-byte aligned");
    const ConvGeom &g = v.g;
    if (cfg.patch) {
        const cuuint64_t pair = cfg.patch == 2 ? 2 : 1;      // pixels per row of the patch
        cuuint64_t dims4[4] = {(cuuint64_t)g.Cp * pair, (cuuint64_t)g.W / pair, (cuuint64_t)g.H, (cuuint64_t)g.N};
        cuuint64_t strides4[3] = {v.stride_w * pair, v.stride_h, v.stride_n};
        cuuint32_t box4[4] = {(cuuint32_t)(cfg.bk * pair), (cuuint32_t)cfg.patch_pw, (cuuint32_t)cfg.patch_ph, 1};
        cuuint32_t estr4[4] = {1, 1, 1, 1};
        CUresult r4 = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t *>(x), dims4, strides4, box4,
                                     estr4, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for((int)(cfg.bk * pair)),
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r4 != CUDA_SUCCESS) return fail(TSB_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled(activation patches) failed with %d", (int)r4);
        return TSB_OK;
    }
    if (v.a_tiled) {
        cuuint64_t dims2[2] = {(cuuint64_t)g.Cp, (cuuint64_t)g.N * g.H * g.W};
        cuuint64_t strides2[1] = {(cuuint64_t)g.Cp};
        cuuint32_t box2[2] = {(cuuint32_t)cfg.bk, (cuuint32_t)cfg.pix};
        cuuint32_t estr2[2] = {1, 1};
        CUresult r2 = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(x), dims2, strides2, box2,
                                     estr2, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(cfg.bk),
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r2 != CUDA_SUCCESS) return fail(TSB_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled(activations) failed with %d", (int)r2);
        return TSB_OK;
    }
    cuuint64_t dims[4] = {(cuuint64_t)g.Cp, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.N};
    cuuint64_t strides[3] = {v.stride_w, v.stride_h, v.stride_n};
    // The box of base pixels: from -pad to the last position a filter can start at.  The far corner is chosen so
    // that exactly OW x OH positions are visited with the traversal stride (floor semantics of the operator).
    int lower[2] = {-g.pad_l, -g.pad_t};
    int upper[2] = {(g.OW - 1) * g.sw - g.pad_l - (g.W - 1), (g.OH - 1) * g.sh - g.pad_t - (g.H - 1)};
    cuuint32_t estr[4] = {1, (cuuint32_t)g.sw, (cuuint32_t)g.sh, 1};
    CUresult r = g_encode_im2col(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t *>(x), dims, strides, lower,
                                 upper, (cuuint32_t)cfg.bk, (cuuint32_t)cfg.pix, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 swizzle_for(cfg.bk), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TSB_ERR_UNSUPPORTED, "cuTensorMapEncodeIm2col failed with %d", (int)r);
    // Tensors under 128 KiB: drivers up to 13.1 set a descriptor bit that makes im2col loads of such small tensors
    // misbehave; clearing it is the documented remedy used by NVIDIA's open-source templates.
    int driver = 0;
    cudaDriverGetVersion(&driver);
    if (driver <= 13010 && v.stage_bytes < 131072)
        reinterpret_cast<uint64_t *>(map)[1] &= ~(1ull << 21);
    return TSB_OK;
}

namespace {

// [O][C][KH][KW] -> [O][KH][KW][Cp], padding channels zero
__global__ void pack_weights_kernel(const int8_t *__restrict__ w, int8_t *__restrict__ wp, int O, int C, int Cp, int taps) {
    const int64_t total = (int64_t)O * taps * Cp;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % Cp);
        const int t = (int)((i / Cp) % taps);
        const int o = (int)(i / ((int64_t)Cp * taps));
        wp[i] = c < C ? w[((int64_t)o * C + c) * taps + t] : (int8_t)0;
    }
}

// [O][C][KH][KW] -> [O][KH][bkf]: byte j of a filter row belongs to pixel offset j / cpix and channel j % cpix
__global__ void pack_weights_folded_kernel(const int8_t *__restrict__ w, int8_t *__restrict__ wp, int O, int C, int KH,
                                           int KW, int dw, int cpix, int bkf) {
    const int64_t total = (int64_t)O * KH * bkf;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(i % bkf);
        const int kh = (int)((i / bkf) % KH);
        const int o = (int)(i / ((int64_t)bkf * KH));
        const int pj = j / cpix, c = j % cpix;
        int8_t val = 0;
        if (c < C && pj % dw == 0 && pj / dw < KW) val = w[(((int64_t)o * C + c) * KH + kh) * KW + pj / dw];
        wp[i] = val;
    }
}

// int8 [N][C][H][W] (or NHWC_PAD [N][H][W][Cp]) -> [N][H][Wp][cpix]; one thread writes 16 bytes
__global__ void stage_folded_kernel(const int8_t *__restrict__ x, int x_nhwc, int Cp, int8_t *__restrict__ y, int N, int C,
                                    int H, int W, int Wp, int cpix, int pad_l) {
    const int units_per_row = Wp * cpix / 16;
    const int64_t total = (int64_t)N * H * units_per_row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int u = (int)(i % units_per_row);
        const int h = (int)((i / units_per_row) % H);
        const int n = (int)(i / ((int64_t)units_per_row * H));
        uint32_t word[4] = {0, 0, 0, 0};
#pragma unroll
        for (int b = 0; b < 16; ++b) {
            const int byte = u * 16 + b;
            const int wp = byte / cpix, c = byte % cpix;
            const int wi = wp - pad_l;
            int8_t v = 0;
            if (c < C && wi >= 0 && wi < W)
                v = x_nhwc ? x[(((int64_t)n * H + h) * W + wi) * Cp + c] : x[(((int64_t)n * C + c) * H + h) * W + wi];
            word[b >> 2] |= (uint32_t)(uint8_t)v << (8 * (b & 3));
        }
        *reinterpret_cast<int4 *>(y + i * 16) = make_int4(word[0], word[1], word[2], word[3]);
    }
}

}  // namespace

int pack_weights(const View &v, const int8_t *w_oihw, int8_t *w_packed, cudaStream_t stream) {
    const ConvGeom &r = v.real;
    const int64_t total = (int64_t)v.weight_bytes;
    const int blocks = (int)std::min<int64_t>(ceil_div64(total, 256), 148 * 8);
    if (v.fold) {
        pack_weights_folded_kernel<<<blocks, 256, 0, stream>>>(w_oihw, w_packed, r.O, r.C, r.KH, r.KW, r.dw, v.cpix, v.g.Cp);
        TSB_LAUNCHED("pack_weights_folded_kernel");
    } else {
        pack_weights_kernel<<<blocks, 256, 0, stream>>>(w_oihw, w_packed, r.O, r.C, r.Cp, r.KH * r.KW);
        TSB_LAUNCHED("pack_weights_kernel");
    }
    return TSB_OK;
}

int stage_folded(const View &v, const int8_t *x, int x_nhwc, int8_t *staged, cudaStream_t stream) {
    const ConvGeom &r = v.real;
    const int64_t total = (int64_t)v.stage_bytes / 16;
    const int blocks = (int)std::min<int64_t>(ceil_div64(total, 256), 148 * 16);
    stage_folded_kernel<<<blocks, 256, 0, stream>>>(x, x_nhwc, r.Cp, staged, r.N, r.C, r.H, r.W, v.Wp, v.cpix, r.pad_l);
    TSB_LAUNCHED("stage_folded_kernel");
    return TSB_OK;
}

int launch_conv_tc(const View &v, const Config &cfg, const CUtensorMap &map_a, const CUtensorMap &map_b,
                   const int8_t *x_staged, const EpiParams &epi, int *status_word, cudaStream_t stream, const DualArgs *dual) {
    const ConvGeom &g = v.g;
    if (dual) {
        // the projected-shortcut kernels exist for the staged block epilogue only
        const bool i8_ok = !epi.out_i8 || (epi.i8_nhwc && reinterpret_cast<uintptr_t>(epi.out_i8) % 16 == 0 &&
                                           (epi.nscales == 1 || (epi.nscales == g.N && epi.group_len == (uint32_t)(g.O * g.OH * g.OW))));
        const bool f32_ok = !epi.out_f32 || (epi.f32_nhwc && reinterpret_cast<uintptr_t>(epi.out_f32) % 16 == 0);
        if (epi.out_acc || epi.residual || !i8_ok || !f32_ok || g.O % 4 != 0 || cfg.swap || cfg.patch || v.rows || v.fold || (!cfg.staging && dual->dq))
            return fail(TSB_ERR_UNSUPPORTED, "projected shortcut: needs pixel-major fp32 / NHWC_PAD int8 outputs, no residual tensor, O %% 4 == 0");
    }
    KernelParams kp;
    kp.M_total = g.N * g.OH * g.OW;
    kp.OW = g.OW;
    kp.P = g.OH * g.OW;
    kp.KH = g.KH; kp.KW = g.KW;
    kp.sh = g.sh; kp.sw = g.sw; kp.dh = g.dh; kp.dw = g.dw; kp.pad_t = g.pad_t; kp.pad_l = g.pad_l;
    kp.Cp = g.Cp;
    kp.num_m_tiles = cfg.num_m_tiles;
    kp.num_n_tiles = cfg.num_n_tiles;
    kp.d_P = FastDiv((uint32_t)kp.P); kp.d_OW = FastDiv((uint32_t)kp.OW);
    kp.d_m_tiles = FastDiv((uint32_t)cfg.num_m_tiles); kp.d_n_tiles = FastDiv((uint32_t)cfg.num_n_tiles);
    kp.d_segs = FastDiv((uint32_t)std::max(1, v.rows_segs)); kp.d_OH = FastDiv((uint32_t)g.OH); kp.d_dh = FastDiv((uint32_t)g.dh);
    const bool per_sample = epi.nscales > 1 && epi.nscales == g.N && epi.group_len == (uint32_t)(g.O * g.OH * g.OW);    // scale index = image index
    kp.status = status_word;
#ifdef TSB_ENABLE_TRACE
    kp.trace = g_trace;
#else
    kp.trace = nullptr;
#endif
    kp.a_tiled = v.a_tiled;
    kp.stages = cfg.stages; kp.stage_bytes = cfg.stage_bytes; kp.b_resident = cfg.b_resident;
    kp.kgroup = cfg.kgroup; kp.unit_bytes = cfg.unit_bytes;
    kp.b_off = cfg.b_off; kp.bar_off = cfg.bar_off;
    kp.rows_segs = 0; kp.rows_OH = g.OH; kp.rows_H = g.H; kp.rows_bytes = 0; kp.rows_stride_h = 0; kp.rows_stride_n = 0;
    kp.rows_x = nullptr;
    kp.patch = cfg.patch; kp.OH = g.OH;
    kp.patch_tiles_w = std::max(1, cfg.patch_tiles_w); kp.patch_tiles_hw = std::max(1, cfg.patch_tiles_w * cfg.patch_tiles_h);
    kp.patch_pw = cfg.patch_pw; kp.patch_bytes = (uint32_t)(cfg.patch_pw * cfg.patch_ph * (cfg.patch == 2 ? 128 : cfg.bk));
    kp.patch_left = cfg.patch == 2 ? (g.pad_l + 1) / 2 : g.pad_l;
    kp.d_tiles_w = FastDiv((uint32_t)kp.patch_tiles_w); kp.d_tiles_hw = FastDiv((uint32_t)kp.patch_tiles_hw);
    if (cfg.patch && !cfg.b_resident) return fail(TSB_ERR_UNSUPPORTED, "patch mode needs resident weights");
    if (v.rows) {
        if (cfg.swap || !cfg.b_resident || !x_staged) return fail(TSB_ERR_UNSUPPORTED, "raw-row mode needs the normal orientation and resident weights");
        kp.rows_segs = v.rows_segs;
        kp.rows_bytes = (uint32_t)round_up((kBM - 1) * 16 + cfg.bk, 16);
        kp.rows_stride_h = (long long)v.stride_h;
        kp.rows_stride_n = (long long)v.stride_n;
        kp.rows_x = x_staged;
    }
    if (cfg.dyn_smem > kMaxDynamicSmem) return fail(TSB_ERR_UNSUPPORTED, "shared-memory plan of %u bytes does not fit", cfg.dyn_smem);
    const bool plain = !epi.out_acc && !epi.residual;
    int epi_mode = kEpiGeneric;      // which epilogue class the outputs take
    if (plain && epi.out_f32 && !epi.f32_nhwc && !epi.out_i8) epi_mode = kEpiF32Nchw;
    // ... and with an fp32 NCHW residual (a shortcut folded into the convolution by the graph rewrite), where a thread owns a pixel
    if (!cfg.swap && !epi.out_acc && epi.residual && epi.out_f32 && !epi.f32_nhwc && !epi.out_i8 && (const void *)epi.residual != (const void *)epi.out_f32)
        epi_mode = kEpiF32Nchw;
    const bool i8_fast = !epi.out_i8 || (epi.i8_nhwc && (epi.nscales == 1 || per_sample));
    if (plain && epi.out_i8 && !epi.out_f32 && i8_fast) epi_mode = kEpiI8Nhwc;
    // pixel-major fp32 tensors (block outputs and residuals of a network) where a thread owns a channel; where it owns a pixel they
    // take the staged class, below, or, in raw rows without room for it, 16-byte accesses
    const bool nhwc_rows = v.rows && g.O % 4 == 0 && ((reinterpret_cast<uintptr_t>(epi.out_f32) | reinterpret_cast<uintptr_t>(epi.residual)) & 15) == 0;
    if (!epi.out_acc && (epi.out_f32 || epi.residual) && epi.f32_nhwc && i8_fast && (const void *)epi.residual != (const void *)epi.out_f32 &&
        ((cfg.swap && !cfg.patch) || nhwc_rows))
        epi_mode = kEpiNhwc;
    const int mode = cfg.patch ? kModePatch : (v.rows ? kModeRows : (cfg.split ? kModeSplit : kModeGeneral));
    // Pixel-major fp32 residual (the shortcut of a residual block, as large as the output): a tensor map over it lets the
    // epilogue prefetch the boxes it is about to read into L2.  The map is not used for loads, so a failure to encode one
    // only switches the prefetch off.
    CUtensorMap map_r = map_b;
    kp.res_prefetch = 0;
    if (epi_mode == kEpiNhwc && epi.residual && mode == kModeGeneral && g.O % 4 == 0 && reinterpret_cast<uintptr_t>(epi.residual) % 16 == 0 &&
        load_driver() == TSB_OK) {
        cuuint64_t dims[2] = {(cuuint64_t)g.O, (cuuint64_t)kp.M_total};
        cuuint64_t strides[1] = {(cuuint64_t)g.O * 4};
        cuuint32_t box[2] = {(cuuint32_t)std::min(g.O, kBM), 32u};
        cuuint32_t estr[2] = {1, 1};
        if (g_encode_tiled(&map_r, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(epi.residual), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
            kp.res_prefetch = 1;
        else
            map_r = map_b;
    }
    // Staged epilogue (normal orientation, shared memory set aside by the configuration): tensor maps over the residual,
    // the fp32 output and the int8 output whose boxes are one quad's tile -- 32 channels x the tile's 128 pixels, shaped
    // like the pixel tile of the load mode (a run of pixels, a run inside one output row, or an 8 x 16 block).
    CUtensorMap map_of = map_b, map_oi = map_b;
    kp.stg_off = cfg.stg_off;
    kp.stg_tiles = cfg.staging;
    kp.stg_groups = cfg.stg_groups;
    // (a projection needs the staged epilogue, whose fp32 tile receives its result; a concatenation takes whatever epilogue
    // its outputs would take in a plain run -- int8 alone goes out through the direct path, which is faster for it)
    const bool dual_concat = dual && dual->dq == nullptr;
    const bool want_staging = (dual && !dual_concat) || wants_staging(v, epi);
    if (want_staging && cfg.staging && load_driver() == TSB_OK) {
        const ConvGeom &r = v.real;
        auto encode = [&](CUtensorMap *map, const void *ptr, bool is_f32, uint64_t channels) -> bool {
            const uint64_t es = is_f32 ? 4 : 1;
            const CUtensorMapDataType dt = is_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
            const CUtensorMapSwizzle sw = is_f32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE;
            cuuint32_t estr[4] = {1, 1, 1, 1};
            CUresult rc;
            if (mode == kModePatch) {
                cuuint64_t dims[4] = {channels, (cuuint64_t)r.OW, (cuuint64_t)r.OH, (cuuint64_t)r.N};
                cuuint64_t strides[3] = {channels * es, channels * es * r.OW, channels * es * r.OW * r.OH};
                cuuint32_t box[4] = {32, 8, (cuuint32_t)(kBM / 8), 1};
                rc = g_encode_tiled(map, dt, 4, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            } else if (mode == kModeRows) {
                cuuint64_t dims[3] = {channels, (cuuint64_t)r.OW, (cuuint64_t)r.N * r.OH};
                cuuint64_t strides[2] = {channels * es, channels * es * r.OW};
                cuuint32_t box[3] = {32, (cuuint32_t)kBM, 1};
                rc = g_encode_tiled(map, dt, 3, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            } else {
                cuuint64_t dims[2] = {channels, (cuuint64_t)kp.M_total};
                cuuint64_t strides[1] = {channels * es};
                cuuint32_t box[2] = {32, (cuuint32_t)kBM};
                rc = g_encode_tiled(map, dt, 2, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            }
            return rc == CUDA_SUCCESS;
        };
        bool ok_maps = true;
        if (epi.residual) ok_maps = ok_maps && encode(&map_r, epi.residual, true, (uint64_t)r.O);
        if (epi.out_f32) ok_maps = ok_maps && encode(&map_of, epi.out_f32, true, (uint64_t)r.O);
        if (epi.out_i8) ok_maps = ok_maps && encode(&map_oi, epi.out_i8, false, (uint64_t)epi.out_cp);
        if (ok_maps) {
            epi_mode = epi.res_after ? kEpiStagedAfter : kEpiStaged;
            kp.res_prefetch = 0;
        }
    }
    if (dual) {
        if (!dual_concat && !is_staged(epi_mode)) return fail(TSB_ERR_UNSUPPORTED, "projected shortcut: the output tensor maps could not be encoded");
        if (dual_concat && !is_staged(epi_mode) && epi_mode != kEpiI8Nhwc)
            return fail(TSB_ERR_UNSUPPORTED, "concatenated input: outputs must be pixel-major fp32 and / or NHWC_PAD int8");
        const ConvGeom &s = dual->view->g;
        DualParams dp;
        dp.map_a2 = dual->map_a; dp.map_b2 = dual->map_b;
        dp.dq2 = dual->dq; dp.bias2 = dual->bias;
        dp.concat = dual->dq == nullptr ? 1 : 0;
        dp.k2_iters = s.Cp / cfg.bk; dp.Cp2 = s.Cp; dp.a2_tiled = dual->view->a_tiled; dp.sh2 = s.sh; dp.sw2 = s.sw;
#define TSB_TC_CASE(BN_, BK_, SWAP_, MODE_, EPI_, DUAL_)                                                                     \
    if constexpr (DUAL_)                                                                                                     \
        if (cfg.bn == BN_ && cfg.bk == BK_ && epi_mode == EPI_ && (BN_ > 64 || dual_concat))                                 \
            return launch<BN_, BK_, SWAP_, MODE_, EPI_, true>(cfg, map_a, map_b, map_r, map_of, map_oi, kp, epi, stream, dp);
        TSB_TC_PART_9(TSB_TC_CASE)
#undef TSB_TC_CASE
        return fail(TSB_ERR_UNSUPPORTED, "no projected-shortcut kernel for tile %dx%d", cfg.bn, cfg.bk);
    }
#define TSB_TC_CASE(BN_, BK_, SWAP_, MODE_, EPI_, DUAL_)                                                                           \
    if constexpr (!DUAL_)                                                                                                    \
        if (cfg.bn == BN_ && cfg.bk == BK_ && (cfg.swap != 0) == SWAP_ && mode == MODE_ && epi_mode == EPI_)                 \
            return launch<BN_, BK_, SWAP_, MODE_, EPI_, false>(cfg, map_a, map_b, map_r, map_of, map_oi, kp, epi, stream, NoDual());
    TSB_TC_ALL(TSB_TC_CASE)
#undef TSB_TC_CASE
    return fail(TSB_ERR_UNSUPPORTED, "no tcgen05 kernel for tile %dx%d", cfg.bn, cfg.bk);
}

}  // namespace tc
}  // namespace tsb
