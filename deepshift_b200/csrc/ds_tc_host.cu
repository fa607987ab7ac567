// Tensor-core path: geometry, tile choice and the ds_tc_* entry points.  Kernels: ds_tc.cu.
#include "ds_tc.cuh"

#include <algorithm>

namespace ds {

int* bounds_status_ptr();
unsigned tc_wait_ns();

namespace {

constexpr int kSms = 148;

constexpr unsigned kWaitNs = 2000000000u;  // two seconds; correct runs stay below a third of one
unsigned g_wait_ns = kWaitNs;              // changed by ds_tc_debug_waits only
int g_hold = 0;

long long round16(long long v) { return (v + 15) & ~15ll; }

FastDiv fast_div(unsigned d)
{
    int l = 0;
    while (l < 31 && (1u << l) < d) ++l;
    if (l == 0) return {0u, 0};
    return {unsigned(((1ull << (31 + l)) + d - 1) / d), l - 1};
}

// Bytes per pixel and plane, and the groups per window row that follow.  The (kw, c) run of one window row
// is contiguous (KW * Cp bytes), so only its end is padded to 16; Cp a multiple of 4, 8 or 16 decides how
// wide the loads are.  Fewest groups first, then the widest loads.  Of a folded window an item holds one pixel's channels.
void choose_pixel(TcGeom& g, int fold)
{
    int best_j = 1 << 30;
    for (int a = 16; a >= 4; a >>= 1) {
        const int cp = (g.C + a - 1) / a * a;
        const int j = ((fold > 1 ? 1 : g.KW) * cp + 15) / 16;
        if (j < best_j) {
            best_j = j;
            g.Cp = cp;
        }
    }
    g.fold = fold;
    g.J = best_j;
    g.G = g.KH * g.J;
    g.align = 16;
    // offsets are sums of multiples of Cp * sw, of the row pitch Wp * Cp and of 16
    while (g.align > 4 && ((g.Cp * g.sw) % g.align || ((long long)g.Wp * g.Cp) % g.align)) g.align >>= 1;
    g.RW = fold > 1 ? g.W : g.OW;
    g.lanes = fold > 1 && 32 % g.W ? 30 : 32;
    g.rows = (long long)g.B * g.OH * g.RW;
}

// Clock cycles of one (group, 128 rows) item: the MMAs at 192 and 128 columns (768 and 512), the producers below.  For the
// choice of a tile and a split only: on 16 folded layers (one image to 4096) it is within 2 % of the best width; tile_cycles
// has the widths' own pace.
double item_cycles(int bn, bool wide)
{
    if (wide) return 1000;
    return bn == 192 ? 800 : bn == 128 ? 700 : bn == 64 ? 520 : 480;
}

const int kTiles[2][3] = {{128, 64, 32}, {192, 96, 48}};  // columns: plain, folded

// Whether a tile of bn columns is one for this layer: not half of it empty.
bool tile_fits(const TcGeom& g, int bn)
{
    return g.wide ? bn == 64 : bn == kTiles[g.fold > 1][2] || g.N > bn / g.fold / 2;
}

// Cycles of one tile in a long run: its items, and what of the epilogue they don't hide.  Fitted to 3x3 layers of 3 to 96
// channels (1 to 18 items of a folded tile, 3 to 54 of a plain one) and 256 images of 14 x 14 and 7 x 7; within 10 %.
double tile_cycles(int bn, double items)
{
    switch (bn) {
        case 32: return 520 * items + 1500;
        case 64: return 540 * items + 2100;
        case 128: return 540 * items + 3000;
        case 48: return 650 * items + 1400;
        case 96: return std::max(390 * items + 3600, 600 * items + 1700);  // the epilogue's pace, the producers'
        default: return std::max(600 * items + 4200, 780 * items + 2000);  // 192: the epilogue's, the MMAs'
    }
}

// Cycles that 128 rows of a long run take with the best tile, and the packing of as many pixels beyond what each layer has.
double cycles_per_block(const TcGeom& g)
{
    double best = 1e30;
    for (int bn : kTiles[g.fold > 1]) {
        if (!tile_fits(g, bn)) continue;
        const int ch = bn / g.fold;
        const double c = double((g.N + ch - 1) / ch) * tile_cycles(bn, g.G) * 32 / g.lanes;
        if (c < best) best = c;
    }
    return best + 30.0 * g.Cp;
}

// Tile and split with the smallest estimated time: waves of units over the SMs, a unit being the longer of
// its MMAs and its epilogue (HBM share of an SM: 23 bytes per cycle), plus one epilogue that nothing hides.
void choose_tile(TcGeom& g)
{
    double best = 1e30;
    for (int bn : kTiles[g.fold > 1]) {
        if (!tile_fits(g, bn)) continue;
        const int ch = bn / g.fold;
        const long long gm = (g.rows + 4ll * g.lanes - 1) / (4 * g.lanes), gn = (g.N + ch - 1) / ch;
        const double epi = TC_ROWS * (double)ch * 4 / 23;
        for (int sp = 1; sp <= 16; ++sp) {
            const int gps = (g.G + sp - 1) / sp;
            if (sp > 1 && (gps < 4 || (g.G + gps - 1) / gps != sp)) continue;
            if (sp > 1 && gm * gn >= 2 * kSms) break;
            const long long units = gm * gn * sp;
            const double waves = double((units + kSms - 1) / kSms);
            const double main = gps * item_cycles(bn, g.wide) + 300;
            double cost = waves * (main > epi ? main : epi) + (main > epi ? epi : main) + 3000;  // ... and the pipeline's fill
            if (sp > 1) cost += 3000 + 800.0 * sp * (bn / 32);  // the last CTA reads all partial sums
            if (cost < best) {
                best = cost;
                g.BN = bn;
                g.grid_m = int(gm);
                g.grid_n = int(gn);
                g.splits = sp;
                g.gps = gps;
            }
        }
    }
}

// Fills the geometry; DS_ERR_UNSUPPORTED when 32-bit offsets do not reach.
int tc_geometry(TcGeom& g, int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits,
                bool wide)
{
    if (B < 0 || C <= 0 || H <= 0 || W <= 0 || OC <= 0 || KH <= 0 || KW <= 0 || sh <= 0 || sw <= 0 || ph < 0 || pw < 0)
        return DS_ERR_BAD_ARG;
    if (KH > 31 || KW > 31) return DS_ERR_UNSUPPORTED;
    if ((long long)H + 2ll * ph < KH || (long long)W + 2ll * pw < KW) return DS_ERR_BAD_ARG;
    if (B == 0) return DS_ERR_UNSUPPORTED;
    g = TcGeom{};
    g.wide = wide;
    if (wide && !(H == 1 && W == 1 && KH == 1 && KW == 1 && ph == 0 && pw == 0)) return DS_ERR_UNSUPPORTED;  // linear layers
    g.B = B; g.C = C; g.H = H; g.W = W; g.OC = OC; g.KH = KH; g.KW = KW; g.sh = sh; g.sw = sw; g.ph = ph; g.pw = pw;
    long long hp = (long long)H + 2ll * ph, wp = (long long)W + 2ll * pw;
    const long long oh = (hp - KH) / sh + 1, ow = (wp - KW) / sw + 1;
    g.sub_h = g.sub_w = 1;
    if (KH == 1 && KW == 1 && ph == 0 && pw == 0) {
        // a strided 1x1 window reads only these pixels (256 x 64 x 56 x 56, stride 2: 252 us with all packed)
        g.sub_h = sh;
        g.sub_w = sw;
        g.sh = g.sw = 1;
        hp = oh;
        wp = ow;
    }
    if (hp > (1 << 20) || wp > (1 << 20) || (long long)C * KH * KW > (1ll << 30)) return DS_ERR_UNSUPPORTED;
    const long long M = B * oh * ow, K = (long long)C * KH * KW;
    // what ds_conv2d_ex refuses with DS_ERR_RANGE stays with it
    if ((long long)C * H * W >= (1ll << 29) || K * KH * KW >= (1ll << 32)) return DS_ERR_UNSUPPORTED;
    const long long limit = 0x7FFFFFFFll - (1 << 20);
    const long long pixels = B * hp * wp;
    if (pixels > limit || M > limit) return DS_ERR_UNSUPPORTED;
    g.Hp = int(hp); g.Wp = int(wp); g.OH = int(oh); g.OW = int(ow);
    g.M = int(M); g.K = int(K); g.N = OC; g.P = int(oh * ow);
    choose_pixel(g, 1);
    // A folded window's rows are the pixels of an image row, its outputs W + 2 pw - 2 of them, so in a long run the times of
    // all rows are compared; in one wave the longest unit counts, and a folded one has a third of the items.  A layer's
    // weights have up to three layouts of either form, whatever the batches.  Measured, us, plain -> folded, padding 1:
    // 64 channels 56 x 56, 256 images 447 -> 278, one 14.8 -> 10.8; 32 channels 16 x 16, 4096 images 314 -> 160; 16 channels
    // 32 x 32 679 -> 313; 256 channels 14 x 14, 256 images 268 -> 258, 64 images 95 -> 74 (finer units), one 18.2 -> 14.8;
    // 512 channels 7 x 7 263 -> 253, 96 -> 83, 22.9 -> 19.0.  128 channels 28 x 28: 257 -> 264, 78 -> 76, 14.9 -> 12.8; layers
    // that one plain tile of 128 columns covers stay plain.  Few items, 64 images of 56 x 56, with the packing: 5 -> 20
    // channels 32 -> 39, 8 -> 64 37 -> 51, 16 -> 144 111 -> 121, 17 -> 48 65 -> 62, 32 -> 160 161 -> 149, 96 -> 256 428 -> 444;
    // 24 -> 144 140 -> 152, but 14 x 14, 256 images 51 -> 47.  One wave: 96 -> 256, 28 x 28, 16 images 59 -> 39, 24 -> 144, 14 x
    // 14, eight 12.0 -> 10.4.  Without padding, 64 images: 512 channels 7 x 7 72 -> 133, 14 x 14 203 -> 233, 256 channels 14 x
    // 14 60 -> 89, 28 x 28 258 -> 286, 64 channels 56 x 56 152 -> 100; one wave, 1024 images of 64 channels, 3 x 3 14.3 -> 12.8,
    // 256 channels 7 x 7 33.1 -> 32.5; two, 256 channels 10 x 10 44 -> 57.
    if (KW == TC_FOLD && g.sw == 1 && pw <= 1 && (OC <= 64 || OC > 128)) {
        TcGeom f = g;
        choose_pixel(f, TC_FOLD);
        const bool wave = (f.rows + 4ll * f.lanes - 1) / (4 * f.lanes) * ((OC + 63) / 64) <= kSms;
        const bool faster = wave ? f.G < g.G
                                 : cycles_per_block(f) * double(f.rows) < 1.05 * cycles_per_block(g) * double(g.rows);
        if (f.rows <= limit && pixels * f.Cp <= limit && OC <= 65535 * 16 && faster) g = f;
    }
    choose_tile(g);
    if (pixels * g.Cp > limit) return DS_ERR_UNSUPPORTED;
    g.plane = round16(pixels * g.Cp + 16);  // the last group of a window row may read up to 15 bytes beyond it
    const long long tiles = (long long)g.grid_m * g.grid_n;
    if (tiles * g.splits > limit || g.grid_n > 65535) return DS_ERR_UNSUPPORTED;
    if (g.splits > 1 && tiles > TC_MAX_SPLIT_TILES) return DS_ERR_UNSUPPORTED;
    g.planes_off = TC_HEADER + (g.splits > 1 ? tiles * g.splits * TC_ROWS * g.BN * 4 : 0);
    g.act_bytes = g.planes_off + (wide ? 3 : 2) * g.plane;
    g.colc_off = (long long)g.grid_n * g.G * g.BN * (wide ? TC_PLANES_WIDE : TC_PLANES) * TC_KG;
    g.state_off = g.colc_off + round16(4ll * g.fold * g.N + 4);  // the word behind: a shift of 16..31 exists (wide)
    g.words_off = g.state_off + 16;
    const int num = 32 / (bits + 1);
    g.weight_bytes = g.words_off + round16(4ll * g.N * ((g.K + num - 1) / num));
    if ((long long)g.grid_n * (g.G + TC_COLC_BLOCKS) > limit) return DS_ERR_UNSUPPORTED;  // blocks of the expansion
    return DS_OK;
}

enum { TC_NO = 0, TC_DIRECT, TC_GATED };

// Whether the activations of this call are known to fit 16 bits (TC_DIRECT), may fit (TC_GATED: measured on
// the device while packing, the integer path stands behind) or cannot be served.  LinearShift's entry conversion
// does not clamp, so its codes pass 16 bits as soon as |x| >= 2^(15-F): they take the 24-bit form.
int tc_mode(const ds_fuse_t& f, int bits, int base)
{
    if (base != 0 || bits < 1 || bits > 7) return TC_NO;
    const int I = f.act_integer_bits, F = f.act_fraction_bits;
    const int code_bits = I == 1 ? F + 2 : I + F;
    switch (f.in_kind) {
        case DS_IN_I32:
            if (f.act_bits == DS_ACT_BITS_AUTO) return TC_GATED;
            return f.act_bits >= 1 && f.act_bits <= 15 ? TC_DIRECT : TC_NO;  // 16 promises |x| <= 2^15, one too many
        case DS_IN_F32_CONV:
        case DS_IN_I32_CLAMP: return I >= 1 && F >= 0 && code_bits <= 16 ? TC_DIRECT : TC_NO;
        case DS_IN_F32_LINEAR: return F >= 0 && F <= 30 ? TC_GATED : TC_NO;
        default: return TC_NO;
    }
}

// int32 codes with a promise: the FP32-pipe path takes one launch and splits K while nothing is fused, so a call
// costs it 20 us of host time or 8 us and 0.09 us per 10^6 products of its 64 x 128 tiles.  Here the weights are
// expanded per call: three launches, 28 us, or 22 us, 5 us per 1000 of K (the column constants) and 6.5 us per 10^6
// weights.  Measured, us, that path -> this one: 128 x 2048 -> 1000 32 -> 47, 256 x 2048 -> 1000 57 -> 51, 512 x 700 ->
// 1000 43 -> 35, 512 x 2048 -> 256 32 -> 37, 1024 x 2048 -> 256 57 -> 43, 65 x 256 -> 10 19 -> 28; the 15 % keep calls at
// the crossing where they were.
bool promised_linear(const TcGeom& g)
{
    const double eff = (double)((g.M + 63) / 64 * 64) * g.K * ((g.N + 127) / 128 * 128);
    const double there = 8 + 0.09e-6 * eff, here = 22 + 0.005 * g.K + 6.5e-6 * g.N * (double)g.K;
    return there > 1.15 * (here > 28.5 ? here : 28.5);
}

// Whether the tensor cores beat the other paths, packing included.  Measured, us, other path -> this one:
//   linear, fp32 input (weights kept): 64 x 784 -> 512 120 -> 19, 17 x 512 -> 512 83 -> 18, 1024 x 500 -> 10 80 -> 19:
//     the integer path behind it runs one CTA per 64 x 128 outputs over all of K, 0.16 us per k, so the GPU times meet
//     near K = 150, with the host's four launches (about 45 us a call) near 300.  That is one wave of CTAs: with many
//     rows and columns this path also wins below (8192 x 256 -> 256 88 -> 30), which the rule leaves out.  Up to 16
//     rows the small-batch kernel takes 10 to 15.
//   linear, int32 input without a promise (expanded per call): 256 x 512 -> 1000 86 -> 28, 1024 x 800 -> 500 108 -> 37;
//     up to 64 rows the integer path splits K and is faster (64 x 784 -> 512 21 -> 26).  With the launch of the
//     expansion the two meet near K = 200.
//   linear, int32 input with a promise: promised_linear; with a fused epilogue the other path does not split K, 0.1 us
//     per k, and the two meet at K = 400 (quantised fp32 input, 320: 43 -> 51, 512: 62 -> 51).
//   convolution: 128 -> 128 channels, 28 x 28, one image 103 -> 19; 1x1 stride 2, 64 -> 128, one image 32 -> 12:
//     few 256-row tiles leave the other path's SMs idle.  With many tiles it pays from about 2^26 shift-accumulates
//     (16 -> 16 channels, 32 x 32, 64 images 40 -> 24), and not where most of the padded product is padding
//     (1 -> 20 channels, 5x5: a tenth is live, 110 -> 135).
bool worthwhile(const TcGeom& g, const ds_fuse_t& f)
{
    const int in_kind = f.in_kind;
    const double ops = (double)g.M * g.N * g.K;
    if (g.H == 1 && g.W == 1 && g.KH == 1 && g.KW == 1) {
        if (in_kind == DS_IN_F32_LINEAR) return g.M > 16 && g.K >= 320;
        if (g.M <= 64 || g.K < 256) return false;
        if (in_kind != DS_IN_I32 || f.act_bits < 1) return true;
        const bool plain = f.out_kind == DS_OUT_I32 && !f.relu && !f.requant && !f.round_f32 && !f.residual;
        return plain ? promised_linear(g) : g.K >= 400;
    }
    const long long tiles = ((g.M + 255ll) / 256) * ((g.N + 127) / 128);
    if (in_kind == DS_IN_I32) {
        // Weights expanded per call: five launches, 45 us of host time.  The other path takes about 20 us and 0.23 us
        // per k and wave of 256 x 128 tiles (0.13 at 64 columns), up to four CTAs sharing a tile along K: 37 images of
        // 45 channels, 31 x 29, stride 2, -> 70: 85 -> 45; one image, 64 channels, 56 x 56 stays.
        const double waves = tiles >= kSms ? double((tiles + kSms - 1) / kSms) : tiles * 4 >= kSms ? (double)tiles / kSms : 0.25;
        if (waves * g.K * (g.N > 64 ? 0.23 : 0.13) < 20) return false;
    }
    auto padded = [](const TcGeom& t) { return (double)t.grid_m * TC_ROWS * t.grid_n * t.BN * t.G * TC_KG; };
    double least = padded(g);
    if (g.fold > 1) {  // chosen because it takes less time, often with more padding: never a reason to refuse
        TcGeom h = g;
        choose_pixel(h, 1);
        choose_tile(h);
        if (padded(h) < least) least = padded(h);
    }
    return tiles <= 16 ? ops >= 6e6 : ops >= double(1 << 26) && ops * 5 >= least;
}

}  // namespace

unsigned tc_wait_ns() { return g_wait_ns; }
int tc_hold() { return g_hold; }

}  // namespace ds

using namespace ds;

extern "C" int ds_tc_bytes(int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits,
                           int base, const ds_fuse_t* fuse, int any_size, long long* act_bytes, long long* weight_bytes)
{
    if (!fuse || !act_bytes || !weight_bytes) return DS_ERR_BAD_ARG;
    *act_bytes = *weight_bytes = 0;
    if (tc_mode(*fuse, bits, base) == TC_NO) return DS_OK;
    TcGeom g;
    const int rc = tc_geometry(g, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, fuse->in_kind == DS_IN_F32_LINEAR);
    if (rc == DS_ERR_UNSUPPORTED) return DS_OK;
    if (rc) return rc;
    if (!any_size && !worthwhile(g, *fuse)) return DS_OK;
    *act_bytes = g.act_bytes;
    *weight_bytes = g.weight_bytes;
    return DS_OK;
}

extern "C" int ds_tc_columns(int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits,
                             int base, const ds_fuse_t* fuse)
{
    TcGeom g;
    if (!fuse || tc_mode(*fuse, bits, base) == TC_NO ||
        tc_geometry(g, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, fuse->in_kind == DS_IN_F32_LINEAR) != DS_OK)
        return 0;
    return g.BN;  // the folded widths are none of the plain ones
}

namespace ds {
namespace {

TcExpand expand_params(const TcGeom& g, const int32_t* packed, int bits, void* weights)
{
    TcExpand p = {};
    p.packed = packed;
    p.wexp = static_cast<unsigned char*>(weights);
    p.colc = reinterpret_cast<int*>(p.wexp + g.colc_off);
    p.state = reinterpret_cast<int*>(p.wexp + g.state_off);
    p.words = reinterpret_cast<int*>(p.wexp + g.words_off);
    p.total = g.grid_n * (g.G + TC_COLC_BLOCKS);
    p.dec.bits = bits;
    p.dec.fw = bits + 1;
    p.dec.num = 32 / (bits + 1);
    p.dec.base = 0;
    p.dec.row_len = (g.K + p.dec.num - 1) / p.dec.num;
    p.C = g.C; p.KH = g.KH; p.KW = g.KW; p.Cp = g.Cp; p.J = g.J; p.G = g.G; p.N = g.N; p.K = g.K; p.BN = g.BN;
    p.fold = g.fold;
    p.wide = g.wide;
    p.nwords = (long long)g.N * p.dec.row_len;
    p.chk_w_bytes = p.nwords * 4;
    p.chk_status = bounds_status_ptr();
    return p;
}

}  // namespace
}  // namespace ds

extern "C" int ds_tc_expand(const int32_t* packed, int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw,
                            int ph, int pw, int bits, int base, const ds_fuse_t* fuse, void* weights,
                            long long weight_bytes, void* stream)
{
    if (!packed || !weights || !fuse) return DS_ERR_BAD_ARG;
    if (base != 0 || bits < 1 || bits > 7) return DS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(weights) & 15u) return DS_ERR_ALIGN;
    TcGeom g;
    const int rc = tc_geometry(g, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, fuse->in_kind == DS_IN_F32_LINEAR);
    if (rc) return rc;
    if (weight_bytes < g.weight_bytes) return DS_ERR_SCRATCH;
    return tc_launch_expand(expand_params(g, packed, bits, weights), static_cast<cudaStream_t>(stream));
}

namespace ds {
namespace {

// A ds_planes_t whose extent fits the 32-bit offsets of the kernels; its plane size in bytes, 0 if malformed.
long long planes_plane(const ds_planes_t* t)
{
    if (!t || t->B <= 0 || t->H <= 0 || t->W <= 0 || t->C <= 0 || t->C % 16 || t->halo < 0 || t->halo > 31) return 0;
    const long long px = t->B * (t->H + 2ll * t->halo) * (t->W + 2ll * t->halo);
    if (t->H > (1 << 20) || t->W > (1 << 20) || px > 0x7FFFFFFFll / t->C - 64) return 0;
    return round16(px * t->C + 16);
}

TcPack pack_params(const GemmParams& q, const void* x, unsigned char* act, long long plane, int B, int C, int H, int W,
                   int ph, int pw, int Hp, int Wp, int Cp, int sub_h, int sub_w)
{
    TcPack pk = {};
    pk.x = x;
    pk.act = act;
    pk.plane = plane;
    pk.B = B; pk.C = C; pk.H = H; pk.W = W; pk.ph = ph; pk.pw = pw; pk.Hp = Hp; pk.Wp = Wp; pk.Cp = Cp;
    pk.sub_h = sub_h; pk.sub_w = sub_w;
    pk.Q = (long long)B * pk.Hp * pk.Wp;
    pk.row_bytes = unsigned(Cp);
    pk.group_bytes = 16;
    pk.in_kind = q.in_kind;
    pk.q = q.q;
    pk.rq_lo = q.rq_lo; pk.rq_hi = q.rq_hi; pk.rq_mul = q.rq_mul; pk.rq_add = q.rq_add;
    pk.chk_act = act;
    pk.chk_act_bytes = (q.in_kind == DS_IN_F32_LINEAR ? 3 : 2) * plane;
    pk.chk_x_bytes = (long long)B * C * H * W * 4 - check_shrink_x();
    pk.chk_status = bounds_status_ptr();
    return pk;
}

}  // namespace
}  // namespace ds

extern "C" long long ds_planes_bytes(int B, int H, int W, int C, int halo)
{
    const ds_planes_t t = {nullptr, B, H, W, C, halo};
    const long long plane = planes_plane(&t);
    return plane ? 2 * plane : -1;
}

extern "C" int ds_planes_pack(const void* x, int in_kind, int I, int F, const ds_planes_t* dst, void* stream)
{
    const long long plane = planes_plane(dst);
    if (!x || !plane || !dst->data) return DS_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(dst->data) & 15u) return DS_ERR_ALIGN;
    ds_fuse_t f = {};
    f.in_kind = in_kind;
    f.act_integer_bits = I;
    f.act_fraction_bits = F;
    if ((in_kind != DS_IN_F32_CONV && in_kind != DS_IN_I32_CLAMP) || tc_mode(f, 1, 0) != TC_DIRECT) return DS_ERR_UNSUPPORTED;
    GemmParams q = {};
    bool fp = false;
    q.K = 1;
    const int rc = setup_common(q, 1, 0, &f, fp);
    if (rc) return rc;
    return tc_launch_pack(pack_params(q, x, static_cast<unsigned char*>(dst->data), plane, dst->B, dst->C, dst->H, dst->W,
                                      dst->halo, dst->halo, dst->H + 2 * dst->halo, dst->W + 2 * dst->halo, dst->C, 1, 1),
                          nullptr, false, static_cast<cudaStream_t>(stream));
}

namespace ds {
namespace {

// What `weights` is: scratch of this call; a buffer to be kept, with nothing in it yet; one that an earlier call
// has filled, from whatever words `packed` held then; tiles of these packed words.
enum { TILES_SCRATCH = 0, TILES_FRESH, TILES_KEPT, TILES_READY };

int tc_conv2d(const void* x, const ds_planes_t* xp, const int32_t* packed, const int32_t* bias, void* out,
              const ds_planes_t* next, int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw,
              int bits, int base, const ds_fuse_t* fuse, void* act, long long act_bytes, void* weights,
              long long weight_bytes, int tiles, cudaStream_t st)
{
    if ((!x && !xp) || (!out && !next) || !packed || !fuse || !act || !weights) return DS_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(act) | reinterpret_cast<uintptr_t>(weights)) & 15u)
        return DS_ERR_ALIGN;
    if (base != 0) return DS_ERR_UNSUPPORTED;
    const int mode = xp ? TC_DIRECT : tc_mode(*fuse, bits, base);
    if (mode == TC_NO || (mode == TC_GATED && next) || (xp && fuse->in_kind == DS_IN_F32_LINEAR)) return DS_ERR_UNSUPPORTED;
    TcGeom g;
    const bool wide = !xp && fuse->in_kind == DS_IN_F32_LINEAR;
    int rc = tc_geometry(g, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, wide);
    if (rc) return rc;
    if (act_bytes < g.act_bytes || weight_bytes < g.weight_bytes) return DS_ERR_SCRATCH;
    // the quantiser and clamp constants, checked as for every other path
    GemmParams q = {};
    bool fp = false;
    q.K = g.K;
    rc = setup_common(q, bits, base, fuse, fp);
    if (rc) return rc;
    if (fuse->residual && (reinterpret_cast<uintptr_t>(fuse->residual) & 3u)) return DS_ERR_ALIGN;
    unsigned char* a = static_cast<unsigned char*>(act);
    int* counters = static_cast<int*>(act) + 4;
    // the range flag, in this call's own scratch: other calls may enqueue launches of theirs between these
    int* flag = static_cast<int*>(act);

    const bool rows = !xp && H == 1 && W == 1 && g.Hp == 1 && g.Wp == 1;  // a matrix: its planes lie group by group
    std::optional<GateLock> lock;
    TcRun p = {};
    int Hp = g.Hp, Wp = g.Wp, step_h = g.sh, step_w = g.sw;
    if (xp) {
        const long long plane = planes_plane(xp);
        if (!plane || !xp->data || xp->B != B || xp->C != C || xp->H != H || xp->W != W || xp->halo < ph || xp->halo < pw)
            return DS_ERR_BAD_ARG;
        if (reinterpret_cast<uintptr_t>(xp->data) & 15u) return DS_ERR_ALIGN;
        Hp = H + 2 * xp->halo;
        Wp = W + 2 * xp->halo;
        step_h = sh;
        step_w = sw;
        p.act = static_cast<const unsigned char*>(xp->data) + ((long long)(xp->halo - ph) * Wp + (xp->halo - pw)) * C;
        p.plane = plane;
        p.chk_act = static_cast<const unsigned char*>(xp->data);
        p.chk_act_bytes = 2 * plane;
    } else {
        p.act = a + g.planes_off;
        p.plane = g.plane;
        p.chk_act = p.act;
        p.chk_act_bytes = (wide ? 3 : 2) * g.plane;
        TcPack pk = pack_params(q, x, a + g.planes_off, g.plane, B, C, H, W, ph, pw, g.Hp, g.Wp, g.Cp, g.sub_h, g.sub_w);
        if (rows) {
            pk.row_bytes = 16;
            pk.group_bytes = 16u * unsigned(g.M);
        }
        pk.counters = g.splits > 1 ? counters : nullptr;
        pk.ncounters = g.splits > 1 ? g.grid_m * g.grid_n : 0;
        if (mode == TC_GATED) {
            p.gate = pk.flag = flag;
            if (!wide) p.report = workspace_gate_word(fuse);  // what DS_ACT_BITS_AUTO promises
            if (p.report) lock.emplace(p.report);
        }
        if (pk.flag && cudaMemsetAsync(flag, 0, sizeof(int), st) != cudaSuccess) return DS_ERR_CUDA;
        const bool kept = tiles == TILES_FRESH || tiles == TILES_KEPT;
        TcExpand e = expand_params(g, packed, bits, weights);
        e.fresh = tiles == TILES_FRESH;
        e.range_flag = pk.flag;
        if (e.fresh && cudaMemsetAsync(e.state, 0, 16, st) != cudaSuccess) return DS_ERR_CUDA;
        if (tiles == TILES_SCRATCH) rc = tc_launch_expand(e, st);
        if (rc) return rc;
        if (wide) pk.refuse = e.colc + g.N;
        rc = tc_launch_pack(pk, kept ? &e : nullptr, wide, st);
        if (rc) return rc;
    }
    p.wexp = static_cast<const unsigned char*>(weights);
    p.colc = reinterpret_cast<const int*>(p.wexp + g.colc_off);
    p.bias = bias;
    p.residual = fuse->residual;
    p.out = out;
    p.M = g.M; p.N = g.N; p.P = g.P; p.OC = g.OC; p.OW = g.OW; p.G = g.G; p.J = g.J; p.align = g.align;
    p.rows = int(g.rows); p.RW = g.RW; p.lanes = g.lanes; p.pw1 = pw - 1;
    p.image = g.OH * g.RW;
    p.by_image = fast_div(unsigned(p.image));
    p.by_row = fast_div(unsigned(g.RW));
    if (g.fold > 1) p.act += (long long)pw * g.Cp;  // rows are pixels, not windows
    p.kh_step = unsigned(Wp) * unsigned(g.Cp);
    p.img_bytes = rows ? 16u : unsigned(Hp) * p.kh_step;
    p.j_step = rows ? 16u * unsigned(g.M) : 16u;
    p.row_step = unsigned(step_h) * p.kh_step;
    p.col_step = unsigned(step_w) * unsigned(g.Cp);
    if (next) {
        const long long plane = planes_plane(next);
        if (!plane || !next->data || next->B != B || next->C != OC || next->H != g.OH || next->W != g.OW) return DS_ERR_BAD_ARG;
        if (reinterpret_cast<uintptr_t>(next->data) & 15u) return DS_ERR_ALIGN;
        const int I = fuse->act_integer_bits, F = fuse->act_fraction_bits;
        if (I < 2 || F < 0 || I + F > 16 || fuse->out_kind != DS_OUT_I32) return DS_ERR_UNSUPPORTED;
        const unsigned nw = unsigned(next->W + 2 * next->halo), nh = unsigned(next->H + 2 * next->halo);
        p.next_px = unsigned(OC);
        p.next_row = nw * unsigned(OC);
        p.next_img = nh * p.next_row;
        p.next = static_cast<unsigned char*>(next->data) + ((long long)next->halo * nw + next->halo) * OC;
        p.next_plane = plane;
        p.chk_next = static_cast<const unsigned char*>(next->data);
        p.chk_next_bytes = 2 * plane;
        p.next_lo = -(1 << (I - 1 + F));
        p.next_hi = ((1 << (I - 1)) - 1) * (1 << F);
    }
    p.grid_m = g.grid_m; p.grid_n = g.grid_n; p.splits = g.splits; p.gps = g.gps;
    p.units = g.grid_m * g.grid_n * g.splits;
    // neighbouring CTAs share the smaller operand's tiles through L2: rows fastest when the weights are the
    // larger one
    p.m_fast = g.colc_off > 2 * g.plane;
    p.by_splits = fast_div(unsigned(g.splits));
    p.by_tile = fast_div(unsigned(p.m_fast ? g.grid_m : g.grid_n));
    p.counters = counters;
    p.partials = reinterpret_cast<int*>(a + TC_HEADER);
    p.out_kind = q.out_kind; p.relu = q.relu; p.requant = q.requant; p.round_f32 = q.round_f32;
    p.rq_lo = q.rq_lo; p.rq_hi = q.rq_hi; p.rq_mul = q.rq_mul; p.rq_add = q.rq_add;
    p.inv_scale = q.inv_scale;
    p.gate_want = 0;
    p.wait_ns = g_wait_ns;
    p.hold = g_hold;
    p.chk_o_bytes = (long long)g.M * g.N * 4;
    p.chk_status = bounds_status_ptr();
    rc = tc_launch_run(p, g.BN, wide, st);
    if (rc || mode != TC_GATED) return rc;
    return launch_gated_int(x, packed, bias, out, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, base, fuse, flag, 1, false, st);
}

}  // namespace
}  // namespace ds

extern "C" int ds_tc_conv2d_ex(const void* x, const ds_planes_t* xp, const int32_t* packed, const int32_t* bias, void* out,
                               const ds_planes_t* next, int B, int C, int H, int W, int OC, int KH, int KW, int sh, int sw,
                               int ph, int pw, int bits, int base, const ds_fuse_t* fuse, void* act, long long act_bytes,
                               const void* weights, long long weight_bytes, void* stream)
{
    return tc_conv2d(x, xp, packed, bias, out, next, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, base, fuse, act,
                     act_bytes, const_cast<void*>(weights), weight_bytes, TILES_READY, static_cast<cudaStream_t>(stream));
}

extern "C" int ds_tc_conv2d_packed(const void* x, const int32_t* packed, const int32_t* bias, void* out, int B, int C, int H,
                                   int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits, int base,
                                   const ds_fuse_t* fuse, void* act, long long act_bytes, void* weights,
                                   long long weight_bytes, int kept, void* stream)
{
    if (!x || !out || kept < TILES_SCRATCH || kept > TILES_KEPT) return DS_ERR_BAD_ARG;
    return tc_conv2d(x, nullptr, packed, bias, out, nullptr, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, base, fuse, act,
                     act_bytes, weights, weight_bytes, kept, static_cast<cudaStream_t>(stream));
}

extern "C" int ds_tc_conv2d(const void* x, const int32_t* packed, const int32_t* bias, void* out, int B, int C, int H,
                            int W, int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits, int base,
                            const ds_fuse_t* fuse, void* act, long long act_bytes, const void* weights,
                            long long weight_bytes, void* stream)
{
    if (!x || !out) return DS_ERR_BAD_ARG;
    return ds_tc_conv2d_ex(x, nullptr, packed, bias, out, nullptr, B, C, H, W, OC, KH, KW, sh, sw, ph, pw, bits, base, fuse,
                           act, act_bytes, weights, weight_bytes, stream);
}

// Checked build only: limit of the kernel's waits in nanoseconds (0 restores the normal one) and the parts of it that
// do not do their work, so that a test can watch waits run out.  DS_ERR_UNSUPPORTED in a normal build.
extern "C" int ds_tc_debug_waits(long long limit_ns, int hold)
{
#ifdef DS_BOUNDS_CHECK
    if (limit_ns < 0 || limit_ns > kWaitNs || hold < 0 || hold > 7) return DS_ERR_BAD_ARG;
    ds::g_wait_ns = limit_ns ? unsigned(limit_ns) : kWaitNs;
    ds::g_hold = hold;
    return DS_OK;
#else
    (void)limit_ns;
    (void)hold;
    return DS_ERR_UNSUPPORTED;
#endif
}
