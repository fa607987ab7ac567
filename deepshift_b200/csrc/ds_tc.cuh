// Tensor-core path: declarations shared by ds_tc.cu (kernels, launches) and ds_tc_host.cu (entry points).
//
// The arithmetic.  out[m,n] = sum_k s[n,k] * (x[m,k] >> r[n,k]) is not a matrix product, because the
// shift rounds every term.  For 16-bit codes and r in 0..15 it becomes one after widening K sixteenfold:
// x >> r, as a function of x, lies in the span of sixteen byte-valued functions f_0..f_15 of x with
// integer coefficients of at most 127, so
//
//     sum_k s * (x >> r)  =  sum_k sum_p f_p(x[m,k]) * (s[n,k] * c_p(r[n,k]))  +  const[n]
//
// is a u8 x s8 product with int32 accumulation, exact modulo 2^32 like the reference's sum.  With
// y = x + 2^15 = 256 h + l (unsigned, so that x >> r = (y >> r) - 2^(15-r); the second part is const[n]):
//
//     f_0 = (l & 127) + (l >> 7) + 2 (h & 1)     y >> 0 = f_0 + 127 (f_7 + f_8 + f_15) + 4 f_9
//     f_1 = (l >> 1) & 63                        y >> 1 = f_1 + 64 (f_7 + f_8 + f_15)
//     f_r = l >> r           (r = 2..6)          y >> r = f_r + 2^(8-r) f_8
//     f_7 = h + (l >> 7) - (h >> 7)              y >> 7 = f_7 + f_8 + f_15
//     f_r = h >> (r - 8)     (r = 8..15)         y >> r = f_r
//
// Sixteen is the least possible: the sixteen functions x >> r are linearly independent.  The coefficient
// 256 of the high byte (r = 0) does not fit an s8 operand; f_0, f_7 and f_9 are chosen so that two nearly
// equal high-byte functions carry 127 each.  r in 16..31 equals r = 15 for 16-bit x, r >= 32 is a zero
// weight.
//
// Wider codes (linear layers with unclamped activations): for |x| < 2^23, y = x + 2^23 has a third byte t and
//     y >> r = ((256 h + l) >> r) + 2^(16-r) t       (r = 0..15),
// so two more products with plane t go into the same sum (r >= 9: coefficients up to 128 as 64 + 64) and four
// into a second accumulator of weight 2^8 (r <= 8: up to 256 as four times 64).
#pragma once
#include <optional>

#include "ds_gemm_common.cuh"

namespace ds {

constexpr int TC_ROWS = 128;    // rows (TMEM lanes) of one MMA
constexpr int TC_PLANES = 16;   // functions f_p per value
constexpr int TC_PLANES_WIDE = 22;  // ... of one 24-bit value: planes 16-21 are copies of t
constexpr int TC_KG = 16;       // values of k per group: one 16-byte run of each plane
constexpr int TC_COLC_BLOCKS = 16;  // expansion blocks per column tile that compute const[n]
// Scratch header: the range flag, then the arrival counters of split tiles (K is split only below 2 x 148
// tiles).  At a fixed place, so that calls of different geometry may share a scratch buffer: the counters are
// zero before and after every call.
constexpr int TC_HEADER = 2048;
constexpr int TC_MAX_SPLIT_TILES = (TC_HEADER - 16) / 4;

// Division of n < 2^31 by a constant of the call: (n * mul >> 32) >> sh, mul = ceil(2^(31 + l) / d), l = ceil(log2 d).
// Exact, since n (mul d - 2^(31 + l)) < 2^31 * 2^l.  mul = 0 stands for d = 1.
struct FastDiv {
    unsigned mul;
    int sh;
};

// Folded windows.  A convolution whose columns move by one pixel (stride 1 along W) may multiply a pixel's channels by
// the weights of all KW window columns at once: KW times as many columns, a KW-th of the items, and out[x] is the sum of
// column block kw at pixel x + kw - (KW - 1) / 2, which the epilogue fetches from the neighbouring lanes.  An item costs
// the producers 177 ALU instructions per scheduler whatever the columns are, so below 128 columns this is what counts.
constexpr int TC_FOLD = 3;

// Geometry and tiling of one call; a pure function of its arguments (weights expanded for a geometry
// fit every later call of the same geometry).
struct TcGeom {
    int B, C, H, W, OC, KH, KW, sh, sw, ph, pw, OH, OW;
    int M, N, K, P;
    int sub_h, sub_w;    // packing takes every sub-th pixel: the strides of a 1x1 window, else 1
    int Hp, Wp, Cp;      // padded image and bytes per pixel of one byte plane (l or h) of the activations
    int J, G;            // groups per window row: ceil(KW * Cp / 16); groups in all: KH * J
    int align;           // every load starts at a multiple of this: 16, 8 or 4
    long long plane;     // bytes of one byte plane
    int wide;            // 24-bit codes: three byte planes
    int fold;            // window columns side by side in a tile: 1, or KW for a folded window
    int BN;              // tile: 128 rows, BN columns = fold * channels
    int RW;              // pixels along W that rows stand for: OW, or W for a folded window
    int lanes;           // rows of a warp that own outputs: 32, or 30 where a warp's first and last only lend theirs
    long long rows;      // B * OH * RW
    int grid_m, grid_n, splits, gps;  // gps: groups per split
    long long act_bytes;      // scratch of one call: header, partial sums, both planes
    long long planes_off;
    long long weight_bytes;   // expanded weights, the column constants, then what a kept buffer is checked by:
    long long colc_off, state_off, words_off;  // two state words and a copy of the packed words
};

struct TcRun {
    const unsigned char* act;   // pixel (0, -ph, -pw) of the l plane
    long long plane;
    const unsigned char* wexp;
    const int* colc;
    const int* bias;
    const int* residual;
    void* out;
    int M, N, P, OC, OW, G, J, align;
    int rows, RW, lanes, pw1;  // as in TcGeom; pw - 1 of a folded window
    int image;                 // OH * RW
    FastDiv by_image, by_row;  // image, RW
    FastDiv by_splits, by_tile;  // splits; grid_m (m_fast) or grid_n
    unsigned img_bytes, row_step, col_step, kh_step, j_step;  // byte offsets inside a plane
    int grid_m, grid_n, splits, gps, units, m_fast;
    // byte planes of the layer that reads this output (null: none); `next` is the pixel (0, 0, 0) of the l plane
    unsigned char* next;
    long long next_plane;
    unsigned next_img, next_row, next_px;  // byte steps of an image, a row, a pixel
    int next_lo, next_hi;                  // clamp of that layer's quantiser
    int* counters;
    int* partials;
    int out_kind, relu, requant, round_f32;
    int rq_lo, rq_hi, rq_mul, rq_add;
    float inv_scale;
    const int* gate;
    int gate_want;
    int* report;         // receives *gate: the workspace's word, for who wants to know which path served; null = none
    unsigned wait_ns;    // limit of every wait
    int hold;            // checked build: see ds_tc_debug_waits
    int* err_flag;
    // checked build: extents of the output, of the planes read and of the planes written
    long long chk_o_bytes;
    const unsigned char *chk_act, *chk_next;
    long long chk_act_bytes, chk_next_bytes;
    int* chk_status;
};

struct TcPack {
    const void* x;
    unsigned char* act;
    long long plane;
    int B, C, H, W, ph, pw, Hp, Wp, Cp;
    int sub_h, sub_w;    // source pixel of (h, w): (h * sub_h, w * sub_w)
    long long Q;         // padded pixels
    unsigned row_bytes, group_bytes;  // tc_pack_rows: from one row, or group of 16 values, to the next
    int in_kind;
    Quant q;
    int rq_lo, rq_hi, rq_mul, rq_add;
    int* flag;           // set to 1 when a code does not fit 16 (24) bits; null = no check
    const int* refuse;   // wide: not zero when the weights hold a shift of 16..31; null = no such word
    int* counters;       // zeroed here for the launch behind
    int ncounters;
    long long chk_x_bytes;
    const unsigned char* chk_act;  // checked build: the planes
    long long chk_act_bytes;
    int* chk_status;
};

struct TcExpand {
    const int* packed;
    unsigned char* wexp;
    int* colc;
    Decode dec;
    int C, KH, KW, Cp, J, G, N, K, BN, fold;
    int wide;            // 22 planes; colc[N] is set when a weight has a shift of 16..31
    int total;           // blocks of work: (G + TC_COLC_BLOCKS) per column tile
    // A kept buffer, looked after by blocks of the packing launch (tc_keep_*):
    int* words;          // copy of the packed words that its tiles were made from
    int* state;          // three words, zero between calls: words differ; comparing, expanding blocks that are done
    long long nwords;
    int fresh;           // nothing is in the buffer yet
    int cmp_blocks;      // the first blocks of the launch compare, the last `exp_blocks` make stale tiles again
    int exp_blocks;
    int* range_flag;     // set with colc[N]; null = none
    int* err_flag;
    long long chk_w_bytes;
    int* chk_status;
};

// ds_gemm.cu: the checks and constants every path shares; the integer path gated on *gate == want; bytes
// taken off the declared extent of x (checked build).
int setup_common(GemmParams& p, int bits, int base, const ds_fuse_t* fuse, bool& use_fp);
int launch_gated_int(const void* x, const int32_t* packed, const int32_t* bias, void* out, int B, int C, int H, int W,
                     int OC, int KH, int KW, int sh, int sw, int ph, int pw, int bits, int base, const ds_fuse_t* fuse,
                     const int* gate, int want, bool zeroed, cudaStream_t st);
long long check_shrink_x();
int* workspace_gate_word(const ds_fuse_t* fuse);  // null without a workspace
// Held while the launches of a call with a measured range are enqueued: two threads on one stream share its workspace.  Calls
// with other workspaces (streams, devices) don't wait for one another.  Allocates nothing: the lock is its own list node.
class GateLock {
public:
    explicit GateLock(const int* word);  // the workspace's gate word
    ~GateLock();
    GateLock(const GateLock&) = delete;
    GateLock& operator=(const GateLock&) = delete;

private:
    const int* word_;
    GateLock* next_;
};
unsigned tc_wait_ns();  // limit of the tensor-core kernels' waits
int tc_hold();          // checked build: see ds_tc_debug_waits

// `e` (may be null): a kept buffer of expanded weights to look after in the same launch.
int tc_launch_pack(const TcPack& p, const TcExpand* e, bool wide, cudaStream_t st);
int tc_launch_expand(const TcExpand& p, cudaStream_t st);
int tc_launch_run(const TcRun& p, int BN, bool wide, cudaStream_t st);

}  // namespace ds
