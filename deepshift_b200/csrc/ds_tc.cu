// Tensor-core shift GEMM / convolution (tcgen05, kind::i8).  The arithmetic is described in ds_tc.cuh.
//
// Three kernels:
//   tc_pack_*     x (int32 or fp32, quantised here) -> two byte planes l and h, pixel-major with a physical
//                 zero border.  One pass over x; from here on a filter tap is an address offset.
//   tc_expand     packed weights -> s8 operand tiles in the order the MMA reads them, and const[n].  Once per
//                 layer for callers that keep it and never change the weights; where they may change, tc_pack looks
//                 after a kept buffer.
//   tc_run        the product.  Persistent, one CTA per SM, warp-specialised:
//                   warps 0-     two or three producer warpgroups, thread = output row = TMEM lane.  A thread loads 16
//                                values (16 bytes of l, 16 of h) and turns them into the sixteen planes with
//                                byte-parallel shifts and masks: 132 instructions per 16 values, then two
//                                32-column tcgen05.st.  The operand A never exists in shared memory.
//                   next four    epilogue: tcgen05.ld, constants, residual / ReLU / rounding, store.
//                   next         one thread issues the MMAs: 128 x BN x 32 bytes, A from TMEM, B from shared memory.
//                   last         one thread fetches weight tiles with cp.async.bulk into a ring.
//                 TMEM: a ring of BN-column accumulator slots, so that the epilogue of a tile overlaps the next tile's
//                 MMAs, and one A slot per producer warpgroup (sixteen planes x 16 bytes x 128 rows), two up to 64 columns and
//                 in the two-warpgroup form of 128.
//
// What bounds it: the s8 MMA rate, 16 byte-products per shift-accumulate (8192 per SM and clock: 144 T
// shift-op/s at 1.9 GHz).  A takes N / 2 cycles per MMA from tensor memory, whatever N; from shared memory 40 + N / 8
// up to 128 columns, which could not carry both operands.  At 128 and 192 columns 74 to 85 % of the rate are in use (8192 x
// 4096 x 4096: 1124 us = 122 T; 3x3 on 256 images, 64 channels 278 us = 106 T, 128 to 512 channels 253 to 257 us = 115 T).
// Narrower tiles are bound by the producers, 177 ALU instructions per item and scheduler on a pipe that takes one every
// other cycle (550 cycles per item of a plain tile of 64 columns, whose MMAs take 256): hence the folded windows.  Folded
// tiles of 16 channels: 4096 images of 32 x 32, 309 us, 371 with residuals and codes; 2650 cycles for three items, of
// which the MMAs take 576 and the ALU pipe 1440.
#include "ds_tc_ptx.cuh"

namespace ds {

namespace {

// Per column width: WG producer warpgroups, each with A slots of its own (64 columns: sixteen planes x 16
// bytes; a slot shared between warpgroups could not be guarded by a phase parity, since a warpgroup may be two
// phases away from it), and as many accumulator slots as the remaining columns hold: at least two, so
// that the epilogue of a tile overlaps the next tile's MMAs.  Tiles of 192, 96 and 48 columns are 64, 32 and 16 channels of
// a folded window.
template <int BN, bool WIDE, bool SHORT>
struct TcTile {
    static constexpr int FOLD = BN % 3 == 0 ? TC_FOLD : 1;
    static constexpr int CH = BN / FOLD;             // channels
    static constexpr int WG = WIDE || SHORT || BN == 192 || BN == 48 ? 2 : 3;
    // Epilogue warpgroups, which take the tiles in turn: a folded tile of 16 channels may have three items only (4096
    // images, 32 x 32, with residual and codes: 498 -> 396 us; three and two warpgroups leave 80 registers, 819 us).
    static constexpr int EWG = BN == 48 ? 2 : 1;
    static constexpr int PLANES = WIDE ? TC_PLANES_WIDE : TC_PLANES;
    static constexpr int ASTRIDE = WIDE ? 96 : 64;   // columns from one A slot to the next
    static constexpr int ACC = WIDE ? 2 * BN : BN;   // columns of an accumulator slot (wide: sums of weight 2^8 behind)
    static constexpr int THREADS = (4 * WG + 4 * EWG + 2) * 32;  // + MMA warp + loader warp
    static constexpr int MMA_WARP = 4 * WG + 4 * EWG;
    // A slots, handed out round robin: item i fills slot i % SLOTS
    static constexpr int SLOTS = (WIDE || (BN >= 96 && !SHORT) ? 1 : 2) * WG;
    static constexpr int ACC_COLS = TC_TMEM_COLS - ASTRIDE * SLOTS;
    static constexpr int NACC = ACC_COLS / ACC < 4 ? ACC_COLS / ACC : 4;
    static constexpr int STAGE = BN * PLANES * TC_KG;
    // weight tiles in shared memory, more than A slots
    static constexpr int STAGES = BN == 192 ? 4 : BN == 128 ? 6 : WIDE || BN == 96 ? 8 : 12;
    static_assert(NACC >= 2 && NACC % EWG == 0 && STAGES > SLOTS, "slots");
};

template <int BN, bool WIDE, bool SHORT>
struct TcSmem {
    alignas(128) unsigned char b[TcTile<BN, WIDE, SHORT>::STAGES][TcTile<BN, WIDE, SHORT>::STAGE];
    alignas(8) unsigned long long bfull[TcTile<BN, WIDE, SHORT>::STAGES];
    unsigned long long full[TcTile<BN, WIDE, SHORT>::SLOTS];   // both operands of the item in this slot are there
    unsigned long long empty[TcTile<BN, WIDE, SHORT>::SLOTS];  // its MMAs are done
    unsigned long long accfull[6];
    unsigned long long accempty[6];
    unsigned long long done;
    unsigned tmem;
    int err;
    int last_flag[2];
    alignas(16) int colc[TcTile<BN, WIDE, SHORT>::EWG][2][BN];
};

__device__ __forceinline__ unsigned fdiv(unsigned n, FastDiv d) { return d.mul ? __umulhi(n, d.mul) >> d.sh : n; }

struct Unit {
    int tile, sp, mt, n0, nt, g0, g1;
};

template <int CH>
__device__ __forceinline__ Unit unit_of(const TcRun& p, int u)
{
    Unit r;
    r.tile = int(fdiv(u, p.by_splits));
    r.sp = u - r.tile * p.splits;
    if (p.m_fast) {
        r.nt = int(fdiv(r.tile, p.by_tile));
        r.mt = r.tile - r.nt * p.grid_m;
    } else {
        r.mt = int(fdiv(r.tile, p.by_tile));
        r.nt = r.tile - r.mt * p.grid_n;
    }
    r.n0 = r.nt * CH;
    r.g0 = r.sp * p.gps;
    r.g1 = min(p.G, r.g0 + p.gps);
    return r;
}

// The pixel that a thread's row stands for.
struct Pixel {
    int b, y, x;
    bool in;  // else the pixel is the first or last one, and the row owns no output
};

template <int FOLD>
__device__ __forceinline__ Pixel pixel_of(const TcRun& p, int mt, int row)
{
    // a folded row of pixels that does not end with the warp: 30 of its 32 rows own outputs, the first and last one
    // are their neighbours' (no exchange between warps; 32 of 32 where 32 is a multiple of W)
    const int lane = row & 31;
    int q = FOLD == 1 ? mt * TC_ROWS + row : (mt * 4 + (row >> 5)) * p.lanes + lane - (p.lanes < 32 ? 1 : 0);
    Pixel r;
    r.in = unsigned(q) < unsigned(p.rows) && (FOLD == 1 || p.lanes == 32 || (lane > 0 && lane < 31));
    q = min(max(q, 0), p.rows - 1);
    r.b = int(fdiv(q, p.by_image));
    const int t = q - r.b * p.image;
    r.y = int(fdiv(t, p.by_row));
    r.x = t - r.y * p.RW;
    return r;
}

// Groups of unit u.
__device__ __forceinline__ int unit_groups(const TcRun& p, int u)
{
    if (p.splits == 1) return p.G;
    const int g0 = u % p.splits * p.gps;
    return min(p.G, g0 + p.gps) - g0;
}

__device__ __forceinline__ void epi_bar(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }

// Epilogue of CC columns of one row, in steps: each step's condition is tested once for all columns (with the conditions
// inside the loop over the columns the epilogue of a 1x1 layer took longer than its MMAs).

// The residual of channels h..h+15 of those at `o0`, `live` of which exist.
__device__ __forceinline__ void load_residual(const TcRun& p, int (&r)[16], int h, int live, long long o0)
{
    const int* q = p.residual + o0 + (long long)h * p.P;
#pragma unroll
    for (int c = 0; c < 16; ++c, q += p.P) r[c] = (h + c < live && DS_O_OK(p, p.residual, q, 4)) ? *q : 0;
}

// v: the finished sums, residual included, at the row's outputs.  NEXT: the codes also (or only, when p.out is null) go
// into the byte planes of the next layer -- CC channels of one pixel, CC contiguous bytes per plane and thread.
template <bool NEXT, int CC>
__device__ __forceinline__ void tc_store(const TcRun& p, int (&v)[CC], int n, int live, long long o0, unsigned nextoff)
{
    int* oi = static_cast<int*>(p.out);
    if (p.relu) {
#pragma unroll
        for (int c = 0; c < CC; ++c) v[c] = max(v[c], 0);
    }
    if (p.requant) {
#pragma unroll
        for (int c = 0; c < CC; ++c) v[c] = min(max(v[c], p.rq_lo), p.rq_hi) * p.rq_mul + p.rq_add;
    }
    if (p.round_f32) {
#pragma unroll
        for (int c = 0; c < CC; ++c) v[c] = __float2int_rn(__int2float_rn(v[c]));
    }
    if (p.out) {
        if (p.out_kind == DS_OUT_F32) {
#pragma unroll
            for (int c = 0; c < CC; ++c) v[c] = __float_as_int(__int2float_rn(v[c]) * p.inv_scale);
        }
        if (p.P == 1 && (p.N & 3) == 0) {
#pragma unroll
            for (int c = 0; c < CC; c += 4)
                if (c < live && DS_O_OK(p, oi, oi + o0 + c, 16))
                    *reinterpret_cast<int4*>(oi + o0 + c) = make_int4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        } else {
            int* o = oi + o0;
#pragma unroll
            for (int c = 0; c < CC; ++c, o += p.P)
                if (c < live && DS_O_OK(p, oi, o, 4)) *o = v[c];
        }
    }
    if (NEXT) {
        unsigned char* nx = p.next + (nextoff + unsigned(n));
#pragma unroll
        for (int h = 0; h < CC; h += 16) {
            if (h >= live) break;  // N is a multiple of 16 here
            unsigned lw[4], hw[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                unsigned c[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) c[e] = unsigned(min(max(v[h + 4 * q + e], p.next_lo), p.next_hi)) + 32768u;
                const unsigned x = __byte_perm(c[0], c[1], 0x5140), y = __byte_perm(c[2], c[3], 0x5140);
                lw[q] = __byte_perm(x, y, 0x5410);
                hw[q] = __byte_perm(x, y, 0x7632);
            }
            if (DS_N_OK(p, nx + h, 16)) *reinterpret_cast<uint4*>(nx + h) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            if (DS_N_OK(p, nx + p.next_plane + h, 16))
                *reinterpret_cast<uint4*>(nx + p.next_plane + h) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        }
    }
}

template <int CC>
__device__ __forceinline__ void add_residual(int (&v)[CC], const int (&r)[16], int h)
{
#pragma unroll
    for (int c = 0; c < 16; ++c) v[h + c] = __float2int_rn(__int2float_rn(v[h + c]) + __int2float_rn(r[c]));
}

// Adds a row's partial sums of all splits into those of the first, 32 loads in flight.  A pass of its own: with the loads in
// the epilogue's own loop every tile paid for their registers (16 channels, 4096 images of 32 x 32: 313 -> 384 us).
template <int BN>
__device__ __forceinline__ void add_partials(int* first, int splits)
{
#pragma unroll 1
    for (int c = 0; c < BN; c += 8) {
        int v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
        for (int k = 0; k < splits; k += 4) {
            int t[4][8];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    t[j][q] = k + j < splits ? __ldcg(first + (long long)(k + j) * (BN * TC_ROWS) + (c + q) * TC_ROWS) : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] += t[j][q];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) __stcg(first + (c + q) * TC_ROWS, v[q]);
    }
}

// CC channels' sums of one row: `acc(col, v)` gives the raw sums of CC columns.  colc: the constants of the tile's
// channels; for a folded window those of all three columns together, then minus those of the left and right one, which
// stand in where the row's neighbour is not part of the image.
template <int CH, int FOLD, int CC, class Acc>
__device__ __forceinline__ void row_sums(int (&v)[CC], const int* colc, int c, bool left, bool right, Acc acc)
{
    acc(FOLD == 1 ? c : CH + c, v);
#pragma unroll
    for (int q = 0; q < CC; q += 4) {
        const int4 k = *reinterpret_cast<const int4*>(colc + c + q);
        v[q] += k.x;
        v[q + 1] += k.y;
        v[q + 2] += k.z;
        v[q + 3] += k.w;
    }
    if (FOLD > 1) {
        int t[CC];
        acc(c, t);
#pragma unroll
        for (int q = 0; q < CC; q += 4) {
            const int4 k = *reinterpret_cast<const int4*>(colc + CH + c + q);
            const int z[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int n = __shfl_up_sync(0xFFFFFFFFu, t[q + e], 1);
                v[q + e] += left ? n : z[e];
            }
        }
        acc(2 * CH + c, t);
#pragma unroll
        for (int q = 0; q < CC; q += 4) {
            const int4 k = *reinterpret_cast<const int4*>(colc + 2 * CH + c + q);
            const int z[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int n = __shfl_down_sync(0xFFFFFFFFu, t[q + e], 1);
                v[q + e] += right ? n : z[e];
            }
        }
    }
}

template <int BN, bool NEXT, bool WIDE, bool SHORT>
__global__ void __launch_bounds__(TcTile<BN, WIDE, SHORT>::THREADS, 1) tc_run_kernel(const TcRun p)
{
    using T = TcTile<BN, WIDE, SHORT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    TcSmem<BN, WIDE, SHORT>& s = *reinterpret_cast<TcSmem<BN, WIDE, SHORT>*>(smem_raw);
    if (p.gate) {
        const int found = *p.gate;
        if (p.report && blockIdx.x == 0 && threadIdx.x == 0) *p.report = found;
        if (found != p.gate_want) return;  // the other arithmetic path serves this input
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* err = &s.err;

    if (threadIdx.x == 0) {
        s.err = 0;
        for (int i = 0; i < T::STAGES; ++i) bar_init(&s.bfull[i], 1);
        for (int i = 0; i < T::SLOTS; ++i) {
            bar_init(&s.full[i], 5);  // four producer warps and the loader
            bar_init(&s.empty[i], 1);
        }
        for (int i = 0; i < T::NACC; ++i) {
            bar_init(&s.accfull[i], 1);
            bar_init(&s.accempty[i], 4);
        }
        bar_init(&s.done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == T::MMA_WARP) {
        tmem_alloc(&s.tmem);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // All 512 columns belong to this CTA, so its columns start at 0: as a constant the MMA operands' addresses
    // are immediates.
    constexpr unsigned tmem = 0;
    constexpr unsigned tmem_a = tmem + T::ACC_COLS;
    if (threadIdx.x == 0 && s.tmem != 0) s.err = 1;

    if (warp < 4 * T::WG) {
        // ---- producers: expand activations into TMEM -------------------------------------------------
        const int wg = warp >> 2;
        const int row = threadIdx.x & 127;
        const unsigned lane_base = unsigned(warp & 3) << 21;  // TMEM lane (warp % 4) * 32 in bits 16-31
        unsigned roff = 0;
        int u = blockIdx.x, g = 0, g1 = 0, j = 0, kh = 0;
        // Unit u, `skip` groups in; units too short for that are passed over.
        auto enter = [&](int skip) {
            for (; u < p.units; u += gridDim.x) {
                const Unit un = unit_of<T::CH>(p, u);
                g = un.g0 + skip;
                g1 = un.g1;
                if (g < g1) {
                    kh = g / p.J;
                    j = g - kh * p.J;
                    const Pixel px = pixel_of<T::FOLD>(p, un.mt, row);
                    roff = unsigned(px.b) * p.img_bytes + unsigned(px.y) * p.row_step + unsigned(px.x) * p.col_step;
                    return;
                }
                skip = g - g1;
            }
        };
        // this warpgroup's next item
        auto step = [&]() {
            g += T::WG;
            if (g >= g1) {
                u += gridDim.x;
                enter(g - g1);
            } else {
                j += T::WG;
                while (j >= p.J) {
                    j -= p.J;
                    ++kh;
                }
            }
        };
        uint4 nl = make_uint4(0, 0, 0, 0), nh = nl, nt = nl;
        auto fetch = [&]() {
            const unsigned char* a = p.act + (roff + unsigned(kh) * p.kh_step + unsigned(j) * p.j_step);
            if (DS_A_OK(p, a, 16)) nl = ld16(a, p.align);
            if (DS_A_OK(p, a + p.plane, 16)) nh = ld16(a + p.plane, p.align);
            if (WIDE && DS_A_OK(p, a + 2 * p.plane, 16)) nt = ld16(a + 2 * p.plane, p.align);
        };
        enter(wg);
        if (u < p.units) fetch();
        for (unsigned round = 0; u < p.units;) {
            const uint4 l = nl, h = nh, t = nt;
            step();
            if (u < p.units) fetch();
            constexpr int PER = T::SLOTS / T::WG;  // slots of this warpgroup, used in turn
            const unsigned slot = wg + T::WG * (round % PER), use = round / PER;
            const unsigned at = tmem_a + lane_base + slot * T::ASTRIDE;
            ++round;
            unsigned v[64];
            planes_low(l.x, h.x, v, 0);
            planes_low(l.y, h.y, v, 1);
            planes_low(l.z, h.z, v, 2);
            planes_low(l.w, h.w, v, 3);
            planes_high(h.x, v + 32, 0);
            planes_high(h.y, v + 32, 1);
            planes_high(h.z, v + 32, 2);
            planes_high(h.w, v + 32, 3);
            // One hand-shake per 16 values (two, a slot per eight planes, cost a third of the rate at 128 columns),
            // and nothing but the stores between the slot's release and its hand-over.
            const bool ok = use == 0 || bar_wait(&s.empty[slot], (use - 1) & 1u, err, p.wait_ns);
            if (!__all_sync(0xFFFFFFFFu, ok) || TC_HELD(p, 2)) break;  // the whole warp, or none of it
            tc_fence_after();
            tmem_st32(at, v);
            tmem_st32(at + 32, v + 32);
            if (WIDE) {
                const unsigned w[16] = {t.x, t.y, t.z, t.w, t.x, t.y, t.z, t.w, t.x, t.y, t.z, t.w, t.x, t.y, t.z, t.w};
                tmem_st16(at + 64, w);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(&s.full[slot]);
        }
    } else if (warp < T::MMA_WARP) {
        // ---- epilogue ----------------------------------------------------------------------------------
        // Channels at a time.  16 of a folded window: their sums, a neighbour's, and residuals fetched ahead.  32 of a plain
        // tile, with one wait for tensor memory and, at its end, for the residuals (16 at a time and fetched ahead: 36
        // images of 5 channels, 82 x 82 -> 162 119 -> 147 us).
        constexpr int CC = T::FOLD > 1 ? 16 : 32;
        const int row = threadIdx.x & 127;
        const unsigned lane_base = unsigned(warp & 3) << 21;
        const int eg = (warp - 4 * T::WG) >> 2;  // this epilogue warpgroup
        unsigned acc = unsigned(eg);             // units of this CTA before this one
        int par = 0, nt = -1;
        // A warp whose wait gives up walks on without the unit's sums: the named barriers below need all four.
        for (int u = blockIdx.x + eg * gridDim.x; u < p.units; u += T::EWG * gridDim.x, acc += T::EWG) {
            const Unit un = unit_of<T::CH>(p, u);
            if (un.nt != nt) {
                // column constants of these channels; two copies, so a slow warp still reads the previous ones
                nt = un.nt;
                par ^= 1;
                if (row < T::CH) {
                    const int n = un.n0 + row;
                    int c = 0, l = 0, r = 0;
                    if (n < p.N) {
                        c = __ldg(p.colc + n) + (p.bias ? __ldg(p.bias + n) : 0);
                        if (T::FOLD > 1) {
                            l = __ldg(p.colc + p.N + n);
                            r = __ldg(p.colc + 2 * p.N + n);
                        }
                    }
                    s.colc[eg][par][row] = c;
                    if (T::FOLD > 1) {
                        s.colc[eg][par][T::CH + row] = l;
                        s.colc[eg][par][2 * T::CH + row] = r;
                    }
                }
                epi_bar(eg);
            }
            const Pixel px = pixel_of<T::FOLD>(p, un.mt, row);
            const int ox = T::FOLD > 1 ? px.x + p.pw1 : px.x;
            const bool in = px.in && (T::FOLD == 1 || unsigned(ox) < unsigned(p.OW));
            const bool left = px.x > 0, right = px.x + 1 < p.RW;
            const long long rowoff = (long long)px.b * p.OC * p.P + px.y * p.OW + ox;
            const unsigned nextoff = NEXT ? unsigned(px.b) * p.next_img + unsigned(px.y) * p.next_row + unsigned(ox) * p.next_px : 0u;
            const unsigned slot = acc % T::NACC;
            int res[16];
            // the residual is fetched ahead: of the first columns while the sums are still being made
            auto fetch = [&](int c) {
                const int n = un.n0 + c;
                if (T::FOLD > 1 && p.residual && in && n < p.N) load_residual(p, res, 0, p.N - n, rowoff + (long long)n * p.P);
            };
            auto finish = [&](int c, auto get) {
                int v[CC];
                row_sums<T::CH, T::FOLD>(v, s.colc[eg][par], c, left, right, get);
                const int n = un.n0 + c;
                if (T::FOLD > 1) {
                    if (p.residual) add_residual(v, res, 0);
                    if (c + CC < T::CH) fetch(c + CC);
                } else if (p.residual && in && n < p.N) {
#pragma unroll
                    for (int h = 0; h < CC; h += 16) {
                        load_residual(p, res, h, p.N - n, rowoff + (long long)n * p.P);
                        add_residual(v, res, h);
                    }
                }
                if (in && n < p.N) tc_store<NEXT>(p, v, n, p.N - n, rowoff + (long long)n * p.P, nextoff);
            };
            if (p.splits == 1) fetch(0);
            if (__all_sync(0xFFFFFFFFu, bar_wait(&s.accfull[slot], (acc / T::NACC) & 1u, err, p.wait_ns))) {
                tc_fence_after();
                const unsigned base = tmem + lane_base + slot * T::ACC;
                auto sums = [&](int c, int (&v)[CC]) {
                    tmem_ld(base + c, v);
                    if (WIDE) {
                        int w[CC];
                        tmem_ld(base + BN + c, w);
#pragma unroll
                        for (int q = 0; q < CC; ++q) v[q] += int(unsigned(w[q]) << 8);
                    }
                };
                auto release = [&]() {  // the accumulators have been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && !TC_HELD(p, 4)) bar_arrive(&s.accempty[slot]);
                };
                if (p.splits == 1) {
#pragma unroll 1
                    for (int c = 0; c < T::CH; c += CC)
                        finish(c, [&](int col, int (&v)[CC]) {
                            sums(col, v);
                            if (col + CC == BN) release();
                        });
                } else {
#pragma unroll 1
                    for (int c = 0; c < BN; c += CC) {
                        int v[CC];
                        sums(c, v);
                        if (c + CC == BN) release();
                        int* dst = p.partials + (long long)(un.tile * p.splits + un.sp) * (BN * TC_ROWS) + c * TC_ROWS + row;
#pragma unroll
                        for (int q = 0; q < CC; ++q) __stcg(dst + q * TC_ROWS, v[q]);
                    }
                }
            }
            if (p.splits > 1) {
                // the split that arrives last adds all partial sums in order and applies the epilogue
                __threadfence();
                epi_bar(eg);
                if (row == 0) s.last_flag[eg] = atomicAdd(p.counters + un.tile, 1) == p.splits - 1;
                epi_bar(eg);
                if (s.last_flag[eg]) {
                    __threadfence();
                    if (row == 0) p.counters[un.tile] = 0;  // for the next launch
                    int* all = p.partials + (long long)un.tile * p.splits * (BN * TC_ROWS) + row;
                    if (T::FOLD > 1) add_partials<BN>(all, p.splits);
                    fetch(0);
#pragma unroll 1
                    for (int c = 0; c < T::CH; c += CC)
                        finish(c, [&](int col, int (&v)[CC]) {
#pragma unroll
                            for (int q = 0; q < CC; ++q) v[q] = __ldcg(all + (col + q) * TC_ROWS);
                            if (T::FOLD == 1)
#pragma unroll 1
                                for (int k = 1; k < p.splits; ++k) {
                                    const int* src = all + (long long)k * (BN * TC_ROWS) + col * TC_ROWS;
#pragma unroll
                                    for (int q = 0; q < CC; ++q) v[q] += __ldcg(src + q * TC_ROWS);
                                }
                        });
                }
                epi_bar(eg);  // last_flag is read by all before the next unit writes it
            }
        }
    } else if (warp == T::MMA_WARP) {
        // ---- MMA issue ---------------------------------------------------------------------------------
        // One elected lane walks the whole loop.  Its instructions are in one queue with the MMAs and, on its
        // scheduler, with the producers' stores to tensor memory: a wait costs 150 to 300 cycles even when what it
        // waits for is there (64 columns, MMAs alone 256 cycles per item: two waits, two commits and an election per
        // item 620 cycles, one wait of which the answer is asked for before the previous item's MMAs 367).  So an item
        // has one barrier for both operands, asked ahead, and one commit.
        // A wait that gives up does not leave the loop: the error word makes all later ones return at once,
        // and every access stays inside shared and tensor memory.
        // D s32, A u8, B s8, both K-major, N = BN, M = 128
        constexpr unsigned idesc = (2u << 4) | (0u << 7) | (1u << 10) | (unsigned(BN / 8) << 17) | (8u << 24);
        // B: no swizzle, core matrices of 8 columns x 16 bytes; 128 bytes from one to the next along N, one
        // plane (BN * 16 bytes) along K
        const unsigned long long desc0 =
            (1ull << 46) | (8ull << 32) | ((unsigned long long)BN << 16) | (s32(&s.b[0][0]) >> 4);
        if (elect_one()) {
            unsigned slot = 0, ph = 0, st = 0, aslot = 0, accph = 1;
            bool ready = false, acc_ready = true;  // the first round finds the accumulator slots free
            for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
                const unsigned d = tmem + aslot * T::ACC;
                if (!acc_ready) bar_wait(&s.accempty[aslot], accph, err, p.wait_ns);
                unsigned long long* accfull = &s.accfull[aslot];
                if (++aslot == unsigned(T::NACC)) {
                    aslot = 0;
                    accph ^= 1u;
                }
                unsigned more = 0;  // the first MMA of a unit overwrites the accumulator
                for (int left = unit_groups(p, u); left > 0; --left) {
                    if (!ready) bar_wait(&s.full[slot], ph, err, p.wait_ns);
                    const unsigned cur = slot;
                    if (++slot == unsigned(T::SLOTS)) {
                        slot = 0;
                        ph ^= 1u;
                    }
                    ready = bar_test(&s.full[slot], ph);
                    if (left == 1) acc_ready = bar_test(&s.accempty[aslot], accph);
                    const unsigned long long bdesc = desc0 + st * unsigned(T::STAGE >> 4);
                    const unsigned at = tmem_a + cur * T::ASTRIDE;
                    tc_fence_after();
#pragma unroll
                    for (int q = 0; q < 8; ++q) tc_mma_i8(d, at + q * 8, bdesc + q * (2 * BN), idesc, q == 0 ? more : 1u);
                    if (WIDE) {
                        tc_mma_i8(d, at + 64, bdesc + 8 * (2 * BN), idesc, 1u);
                        tc_mma_i8(d + BN, at + 64, bdesc + 9 * (2 * BN), idesc, more);
                        tc_mma_i8(d + BN, at + 72, bdesc + 10 * (2 * BN), idesc, 1u);
                    }
                    tc_commit(&s.empty[cur]);
                    more = 1;
                    if (++st == unsigned(T::STAGES)) st = 0;
                }
                tc_commit(accfull);
            }
            tc_commit(&s.done);  // nothing of this CTA is in flight when the columns go back
            if (!bar_drain(&s.done, 0)) *err = 1;
        }
        __syncwarp();
    } else {
        // ---- weight tiles: one thread ------------------------------------------------------------------
        // It keeps STAGES tiles in flight or in use, and takes part in each item's barrier once its tile has landed:
        // the stage of item i is free again when item i's MMAs are done, which is also when slot i % SLOTS is.
        if (lane == 0) {
            int lu = blockIdx.x, lleft = 0;  // what to fetch next
            const unsigned char* src = nullptr;
            unsigned lst = 0, issued = 0;
            auto fetch = [&]() {
                while (lleft == 0) {
                    if (lu >= p.units || TC_HELD(p, 1)) return;
                    const Unit un = unit_of<T::CH>(p, lu);
                    src = p.wexp + ((long long)un.nt * p.G + un.g0) * T::STAGE;
                    lleft = un.g1 - un.g0;
                    lu += gridDim.x;
                }
                bulk_load(s32(&s.b[lst][0]), src, T::STAGE, &s.bfull[lst]);
                src += T::STAGE;
                --lleft;
                ++issued;
                if (++lst == unsigned(T::STAGES)) lst = 0;
            };
            for (int i = 0; i < T::STAGES; ++i) fetch();
            unsigned i = 0, st = 0, bph = 0, slot = 0, ph = 1;
            for (; i < issued; ++i) {
                if (i >= unsigned(T::SLOTS)) {
                    if (!bar_wait(&s.empty[slot], ph, err, p.wait_ns)) break;
                    fetch();
                }
                if (!bar_wait(&s.bfull[st], bph, err, p.wait_ns)) break;
                bar_arrive(&s.full[slot]);
                if (++slot == unsigned(T::SLOTS)) {
                    slot = 0;
                    ph ^= 1u;
                }
                if (++st == unsigned(T::STAGES)) {
                    st = 0;
                    bph ^= 1u;
                }
            }
            // Every copy has landed before the CTA ends, also when a wait gave up.
            for (; i < issued; ++i) {
                if (!bar_drain(&s.bfull[st], bph)) *err = 1;
                if (++st == unsigned(T::STAGES)) {
                    st = 0;
                    bph ^= 1u;
                }
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == T::MMA_WARP)
        tmem_dealloc();
    if (threadIdx.x == 0 && s.err) *p.err_flag = 1;
}

// ---- weights -> operand tiles -------------------------------------------------------------------------
// Packed field of weight (n, k): r in 0..15 with bit 4 for a negative weight, or 32 for a zero weight.
__device__ __forceinline__ int tc_code(const TcExpand& p, unsigned field)
{
    const int r = int(field & ((1u << p.dec.bits) - 1u));
    if (r >= 32) return 32;
    return min(r, 15) | (((field >> p.dec.bits) & 1u) ? 0 : 16);
}

constexpr int TC_KEEP_WAIT = 1 << 22;  // rounds of at least 64 ns

struct ExpandSmem {
    unsigned lut[6][33];
    int stale;
    alignas(16) unsigned char codes[192 * 16];
};

// A lane's share of -sum s 2^(15-r) over the weights of channel n.
template <bool FOLD>
__device__ __forceinline__ void column_sums(const TcExpand& p, int n, int lane, unsigned& sum, unsigned& first, unsigned& last,
                                            bool& far)
{
    const unsigned fmask = (1u << p.dec.fw) - 1u;
    const int* src = p.packed + (long long)n * p.dec.row_len;
    for (int w = lane; w < p.dec.row_len; w += 32) {
        unsigned word = DS_W_OK(p, src + w, 4) ? unsigned(__ldg(src + w)) : 0u;
        const int k = w * p.dec.num;
        int kw = FOLD ? k % p.KW : 1;
        for (int i = 0; i < p.dec.num && k + i < p.K; ++i, word >>= p.dec.fw) {
            const int c = tc_code(p, word & fmask);
            if (c < 32) {
                if (p.wide) far |= (word & fmask & ((1u << p.dec.bits) - 1u)) >= 16u;
                const unsigned v = 1u << ((p.wide ? 23 : 15) - (c & 15)), s = (c & 16) ? v : 0u - v;
                sum += s;
                if (FOLD && kw == 0) first += s;
                if (FOLD && kw == 2) last += s;
            }
            if (FOLD && ++kw == p.KW) kw = 0;
        }
    }
}

// Block (nt, g): the operand tile of group g, columns nt * BN.. -- [16 planes][BN][16 bytes].  A thread makes
// four planes of one column: 16 table words (four planes each, sign applied), transposed 4 x 4 bytes.
// Blocks g = G.. compute the column constants -sum s 2^(15-r).
// FOLD apart: as branches it cost the plain form a fifth (4096 x 4096 weights 92 -> 111 us).
template <bool FOLD>
__device__ __forceinline__ void expand_form(const TcExpand& p, int nt, int g, ExpandSmem& sm)
{
    const int ch = FOLD ? p.BN / TC_FOLD : p.BN, n0 = nt * ch;
    const unsigned fmask = (1u << p.dec.fw) - 1u;
    if (g >= p.G) {
        // 1, 2, 4 or 8 channels, one per warp
        const int per = ch / TC_COLC_BLOCKS;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int n = n0 + (g - p.G) * per + warp;
        if (warp >= per || n >= p.N) return;
        unsigned sum = 0, first = 0, last = 0;  // folded: those of the window's first and last column apart
        bool far = false;
        column_sums<FOLD>(p, n, lane, sum, first, last, far);
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        if (FOLD) {
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                first += __shfl_xor_sync(0xFFFFFFFFu, first, o);
                last += __shfl_xor_sync(0xFFFFFFFFu, last, o);
            }
            if (lane == 0) {
                p.colc[p.N + n] = -int(first);
                p.colc[2 * p.N + n] = -int(last);
            }
        }
        if (p.wide && __any_sync(0xFFFFFFFFu, far) && lane == 0) {
            p.colc[p.N] = 1;
            if (p.range_flag) *p.range_flag = 1;
        }
        if (lane == 0) p.colc[n] = int(sum);
        return;
    }
    for (int i = threadIdx.x; i < 6 * 33; i += 256) (&sm.lut[0][0])[i] = g_tc_lut.w[i];
    // a thread keeps its place in the group (and with it the word and the bit position) and walks the columns
    const int kh = g / p.J, j = g - kh * p.J;
    const int t = 16 * j + (threadIdx.x & 15);  // byte of the window row: (kw, c), or c of a folded window
    const int nl0 = threadIdx.x >> 4;
#pragma unroll
    for (int f = 0; f < (FOLD ? TC_FOLD : 1); ++f) {
        const int kw = FOLD ? f : t / p.Cp, c = FOLD ? t : t - kw * p.Cp;
        const bool live = kw < p.KW && c < p.C;
        const int k = (c * p.KH + kh) * p.KW + kw;
        const int w = k / p.dec.num, at = (k - w * p.dec.num) * p.dec.fw;
        const int* src = p.packed + (long long)(n0 + nl0) * p.dec.row_len + w;
#pragma unroll 8
        for (int nl = nl0; nl < ch; nl += 16, src += 16ll * p.dec.row_len) {
            int code = 32;
            if (live && n0 + nl < p.N && DS_W_OK(p, src, 4)) code = tc_code(p, (unsigned(__ldg(src)) >> at) & fmask);
            sm.codes[(f * ch + nl) * 16 + (threadIdx.x & 15)] = (unsigned char)code;
        }
    }
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(p.wexp + ((long long)nt * p.G + g) * (p.BN * (p.wide ? TC_PLANES_WIDE : TC_PLANES) * TC_KG));
    for (int i = threadIdx.x; i < p.BN * (p.wide ? 6 : 4); i += 256) {
        const int q = i / p.BN, n = FOLD ? i - q * p.BN : i & (p.BN - 1);
        const uint4 cw = *reinterpret_cast<const uint4*>(sm.codes + n * 16);
        const unsigned cws[4] = {cw.x, cw.y, cw.z, cw.w};
        unsigned o[4][4];  // [plane][word]
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            unsigned a[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] = sm.lut[q][(cws[w] >> (8 * e)) & 255u];
            transpose4(a[0], a[1], a[2], a[3], o[0][w], o[1][w], o[2][w], o[3][w]);
        }
#pragma unroll
        for (int f = 0; f < 4; ++f)
            if (4 * q + f < TC_PLANES_WIDE) out[(4 * q + f) * p.BN + n] = make_uint4(o[f][0], o[f][1], o[f][2], o[f][3]);
    }
}

__device__ __forceinline__ void expand_block(const TcExpand& p, int nt, int g, ExpandSmem& sm)
{
    if (p.fold > 1) expand_form<true>(p, nt, g, sm);
    else expand_form<false>(p, nt, g, sm);
}

template <bool FOLD>
__global__ void __launch_bounds__(256) tc_expand_kernel(const TcExpand p)
{
    __shared__ ExpandSmem sm;
    expand_form<FOLD>(p, blockIdx.y, blockIdx.x, sm);
}

// Kept buffers.  The tiles stay with the packed words they were made from, and the packing launch of every call looks
// after them: its first blocks compare the copy with the words of the moment (4096 x 4096 weights: 34 MB, 9 us; a
// convolution's disappear in the packing pass), its last ones wait for those and make the tiles again if a word
// differs.  Weights changed by any means take effect with the next call, and no launch is added for it (comparing
// tile by tile inside the expansion took 45 us for 4096 x 4096, a launch of its own 5 us per layer).
__device__ __forceinline__ void keep_compare(const TcExpand& p, unsigned block)
{
    const long long i0 = block * 256ll + threadIdx.x, step = p.cmp_blocks * 256ll;
    const long long n4 = (reinterpret_cast<uintptr_t>(p.packed) & 15u) == 0 ? p.nwords / 4 : 0;
    bool differs = p.fresh != 0;
#pragma unroll 2
    for (long long i = i0; i < n4; i += step) {
        const int4* src = reinterpret_cast<const int4*>(p.packed) + i;
        int4* dst = reinterpret_cast<int4*>(p.words) + i;
        if (!DS_W_OK(p, src, 16)) continue;
        const int4 a = __ldg(src), b = __ldcg(dst);
        if (p.fresh || ((a.x ^ b.x) | (a.y ^ b.y) | (a.z ^ b.z) | (a.w ^ b.w)) != 0) {
            *dst = a;
            differs = true;
        }
    }
    for (long long i = 4 * n4 + i0; i < p.nwords; i += step) {
        if (!DS_W_OK(p, p.packed + i, 4)) continue;
        const int a = __ldg(p.packed + i);
        if (p.fresh || a != __ldcg(p.words + i)) {
            p.words[i] = a;
            differs = true;
        }
    }
    if (differs) {
        if (p.wide) p.colc[p.N] = 0;  // found again, if it holds, when the tiles are made
        p.state[0] = 1;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(p.state + 1, 1);
}

// The wait ends: the blocks waited for depend on nothing and come first in the launch, and exp_blocks, an eighth of
// what is resident, never fill the GPU.  (Bounded all the same.)
__device__ __forceinline__ void keep_expand(const TcExpand& p, int block, ExpandSmem& sm)
{
    if (threadIdx.x == 0) {
        int done = 0;
        for (int i = 0; i < TC_KEEP_WAIT && !done; ++i) {
            done = *(volatile const int*)(p.state + 1) >= p.cmp_blocks;
            if (!done) __nanosleep(64);
        }
        if (!done) *p.err_flag = 1;
        __threadfence();
        sm.stale = *(volatile const int*)p.state;
    }
    __syncthreads();
    if (sm.stale) {
        const int per_tile = p.G + TC_COLC_BLOCKS;
        for (int b = block; b < p.total; b += p.exp_blocks) {
            const int nt = b / per_tile;
            expand_block(p, nt, b - nt * per_tile, sm);
            __syncthreads();
        }
    }
    if (threadIdx.x == 0 && atomicAdd(p.state + 2, 1) == p.exp_blocks - 1) {
        // all others have read the state
        p.state[0] = 0;
        p.state[1] = 0;
        p.state[2] = 0;
    }
}

// Blocks of a packing launch that look after the weights; false for the others, whose index among themselves goes
// to `block`.
__device__ __forceinline__ bool keep_weights(const TcExpand& p, unsigned& block, ExpandSmem& sm)
{
    if (blockIdx.x < unsigned(p.cmp_blocks)) {
        keep_compare(p, blockIdx.x);
        return true;
    }
    const int left = int(gridDim.x - blockIdx.x);
    if (left <= p.exp_blocks) {
        keep_expand(p, left - 1, sm);
        return true;
    }
    block = blockIdx.x - unsigned(p.cmp_blocks);
    return false;
}

// ---- activations -> byte planes -----------------------------------------------------------------------
// Code of the raw word `v` of x, as operand_of defines it for the integer path.
template <int INK>
__device__ __forceinline__ int pack_code(const TcPack& p, int v)
{
    if (INK == INK_I32) return v;
    if (INK == INK_I32_CLAMP) return min(max(v, p.rq_lo), p.rq_hi) * p.rq_mul + p.rq_add;
    if (p.in_kind == DS_IN_F32_CONV) return __float2int_rz(quant_conv_f(__int_as_float(v), p.q));
    return __float2int_rz(truncf(__int_as_float(v) * p.q.scale));
}

// NCHW -> pixel-major planes.  A block takes 1024 / CW padded pixels x 4 CW channels: lanes run over pixels
// when reading (coalesced in x), over channels when writing (coalesced in the planes).  HBM-bound: 4 bytes
// read and 2 written per value.  `nx` blocks side by side along the pixels, one row of them per 4 CW channels.
// KEPT: further blocks look after the weights; eight blocks per SM as without them (at the 40 registers the
// expansion would like, 64 x 64 x 56 x 56 takes 34 us instead of 29).
template <int INK, bool KEPT>
__global__ void __launch_bounds__(256, 8) tc_pack_nchw_kernel(const TcPack p, const TcExpand e, int cw_log, unsigned nx)
{
    __shared__ __align__(16) unsigned words[2][2048];
    unsigned block = blockIdx.x;
    if (KEPT && keep_weights(e, block, *reinterpret_cast<ExpandSmem*>(&words[0][0]))) return;
    unsigned *sl = words[0], *sh = words[1];
    const unsigned by = block / nx, bx = block - by * nx;
    const int CW = 1 << cw_log, PIX = 1024 >> cw_log;
    const long long q0 = (long long)bx * PIX;
    const int cw0 = int(by << cw_log);
    if (p.counters && by == 0)
        for (long long i = bx * 256ll + threadIdx.x; i < p.ncounters; i += nx * 256ll) p.counters[i] = 0;
    const long long hw = (long long)p.H * p.W;
    const int* x = static_cast<const int*>(p.x);
    bool over = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = threadIdx.x + 256 * k;
        const int pix = i & (PIX - 1), cw = i >> (10 - cw_log);
        const long long q = q0 + pix;
        int c4[4] = {0, 0, 0, 0};
        if (q < p.Q) {
            const unsigned qi = unsigned(q);
            const unsigned rowi = qi / unsigned(p.Wp);
            const int w = (int(qi - rowi * unsigned(p.Wp)) - p.pw) * p.sub_w;
            const unsigned b = rowi / unsigned(p.Hp);
            const int h = (int(rowi - b * unsigned(p.Hp)) - p.ph) * p.sub_h;
            if (unsigned(h) < unsigned(p.H) && unsigned(w) < unsigned(p.W)) {
                const int c = 4 * (cw0 + cw);
                const int* src = x + ((long long)b * p.C + c) * hw + (long long)h * p.W + w;
                int raw[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) raw[e] = (c + e < p.C && DS_X_OK(p, src + e * hw, 4)) ? __ldg(src + e * hw) : 0;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < p.C) c4[e] = pack_code<INK>(p, raw[e]);
            }
        }
        unsigned l, h;
        pack4(c4, l, h, over);
        sl[pix * (CW + 1) + cw] = l;
        sh[pix * (CW + 1) + cw] = h;
    }
    if (over && p.flag) *p.flag = 1;
    __syncthreads();
    const int cwords = p.Cp >> 2;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = threadIdx.x + 256 * k;
        const int cw = i & (CW - 1), pix = i >> cw_log;
        const long long q = q0 + pix;
        if (q < p.Q && cw0 + cw < cwords) {
            unsigned* dst = reinterpret_cast<unsigned*>(p.act + q * p.Cp) + cw0 + cw;
            unsigned* dsth = reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(dst) + p.plane);
            if (DS_A_OK(p, dst, 4)) *dst = sl[pix * (CW + 1) + cw];
            if (DS_A_OK(p, dsth, 4)) *dsth = sh[pix * (CW + 1) + cw];
        }
    }
}

// Rows of a matrix [Q, C]: 4 values of a row per thread, 16 values of 8 rows per warp.  The planes come out pixel-major
// (row_bytes = Cp, group_bytes = 16) or, for the product behind, as [16 values][row]: its threads are rows, and 16 bytes
// at the row's pitch from each cost the load unit a wavefront per thread.  KEPT as above.
template <int INK, bool WIDE, bool KEPT>
__global__ void __launch_bounds__(256, 8) tc_pack_rows_kernel(const TcPack p, const TcExpand e)
{
    unsigned block = blockIdx.x, blocks = gridDim.x;
    if constexpr (KEPT) {
        __shared__ ExpandSmem sm;
        if (keep_weights(e, block, sm)) return;
        blocks -= unsigned(e.cmp_blocks + e.exp_blocks);
    }
    const unsigned groups = (unsigned(p.Cp) + 15u) >> 4;
    const unsigned total = (unsigned(p.Q) + 7u) / 8u * groups * 32u;  // checked by the launch
    const bool vec = p.C % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0;
    const unsigned i0 = block * 256u + threadIdx.x;
    if (p.counters)
        for (unsigned i = i0; i < unsigned(p.ncounters); i += blocks * 256u) p.counters[i] = 0;
    bool over = i0 == 0 && p.refuse && *p.refuse;
    for (unsigned i = i0; i < total; i += blocks * 256u) {
        const unsigned t = i >> 5, mb = t / groups, j = t - mb * groups;
        const unsigned m = 8 * mb + ((i >> 2) & 7u);
        const int k = int(16 * j + 4 * (i & 3u));
        if (m >= unsigned(p.Q) || k >= p.Cp) continue;
        const int* src = static_cast<const int*>(p.x) + (long long)m * p.C + k;
        int raw[4] = {0, 0, 0, 0}, c4[4];
        if (vec && k + 4 <= p.C) {
            if (DS_X_OK(p, src, 16)) {
                const int4 v = __ldg(reinterpret_cast<const int4*>(src));
                raw[0] = v.x; raw[1] = v.y; raw[2] = v.z; raw[3] = v.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k + e < p.C && DS_X_OK(p, src + e, 4)) raw[e] = __ldg(src + e);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) c4[e] = k + e < p.C ? pack_code<INK>(p, raw[e]) : 0;
        unsigned l, h;
        unsigned* dst = reinterpret_cast<unsigned*>(p.act + (m * p.row_bytes + j * p.group_bytes + 4 * (i & 3u)));
        if (WIDE) {
            unsigned y[4], t = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[e] = unsigned(c4[e]) + (1u << 23);
                over |= y[e] >> 24 != 0;
                t |= ((y[e] >> 16) & 255u) << (8 * e);
                c4[e] = int(y[e] & 0xFFFFu) - 32768;
            }
            unsigned* dstt = reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(dst) + 2 * p.plane);
            if (DS_A_OK(p, dstt, 4)) *dstt = t;
        }
        pack4(c4, l, h, over);
        unsigned* dsth = reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(dst) + p.plane);
        if (DS_A_OK(p, dst, 4)) *dst = l;
        if (DS_A_OK(p, dsth, 4)) *dsth = h;
    }
    if (over && p.flag) *p.flag = 1;
}

template <int BN, bool NEXT, bool WIDE, bool SHORT = false>
int run_cfg(const TcRun& p0, cudaStream_t st)
{
    TcRun p = p0;
    p.err_flag = kernel_error_flag();
    const int dev = device_slot();
    if (!p.err_flag || dev < 0) return DS_ERR_CUDA;
    auto kern = tc_run_kernel<BN, NEXT, WIDE, SHORT>;
    const size_t smem = sizeof(TcSmem<BN, WIDE, SHORT>);
    static bool done[kMaxDevices];  // per instantiation and device
    static int sms[kMaxDevices];
    if (!done[dev]) {
        int n = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess ||
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
            cudaGetLastError();
            return DS_ERR_CUDA;
        }
        sms[dev] = n;
        done[dev] = true;
    }
    const int grid = p.units < sms[dev] ? p.units : sms[dev];
    kern<<<grid, TcTile<BN, WIDE, SHORT>::THREADS, smem, st>>>(p);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? DS_OK : DS_ERR_CUDA;
}

}  // namespace

int tc_launch_pack(const TcPack& p, const TcExpand* e0, bool wide, cudaStream_t st)
{
    TcExpand e = e0 ? *e0 : TcExpand{};
    if (e0) {
        e.err_flag = kernel_error_flag();
        if (!e.err_flag) return DS_ERR_CUDA;
        const long long want = (e.nwords + 2047) / 2048;
        e.cmp_blocks = int(want > 148 * 4 ? 148 * 4 : want);
        e.exp_blocks = e.total < 148 ? e.total : 148;
    }
    const unsigned more = unsigned(e.cmp_blocks + e.exp_blocks);
    auto rows = [&](auto ink) {
        const long long want = ((p.Q + 7) / 8 * ((p.Cp + 15) / 16) * 32 + 255) / 256;
        const unsigned grid = unsigned(want > 148 * 64 ? 148 * 64 : want) + more;
        constexpr int K = decltype(ink)::value;
        if (wide && e0) tc_pack_rows_kernel<K, true, true><<<grid, 256, 0, st>>>(p, e);
        else if (wide) tc_pack_rows_kernel<K, true, false><<<grid, 256, 0, st>>>(p, e);
        else if (e0) tc_pack_rows_kernel<K, false, true><<<grid, 256, 0, st>>>(p, e);
        else tc_pack_rows_kernel<K, false, false><<<grid, 256, 0, st>>>(p, e);
    };
    auto nchw = [&](auto ink) {
        int lg = 0;
        while (lg < 4 && (4 << lg) < p.Cp) ++lg;
        const int pix = 1024 >> lg;
        const unsigned nx = unsigned((p.Q + pix - 1) / pix);
        const unsigned grid = nx * unsigned((p.Cp / 4 + (1 << lg) - 1) >> lg) + more;
        constexpr int K = decltype(ink)::value;
        if (e0) tc_pack_nchw_kernel<K, true><<<grid, 256, 0, st>>>(p, e, lg, nx);
        else tc_pack_nchw_kernel<K, false><<<grid, 256, 0, st>>>(p, e, lg, nx);
    };
    auto go = [&](auto ink) {
        if (p.Hp == 1 && p.Wp == 1 && p.H == 1 && p.W == 1) rows(ink);
        else nchw(ink);
    };
    if (p.in_kind == DS_IN_I32) go(std::integral_constant<int, INK_I32>());
    else if (p.in_kind == DS_IN_I32_CLAMP) go(std::integral_constant<int, INK_I32_CLAMP>());
    else go(std::integral_constant<int, INK_F32>());
    note_launch();
    return cudaGetLastError() == cudaSuccess ? DS_OK : DS_ERR_CUDA;
}

int tc_launch_expand(const TcExpand& p, cudaStream_t st)
{
    if (p.wide && cudaMemsetAsync(p.colc + p.N, 0, sizeof(int), st) != cudaSuccess) return DS_ERR_CUDA;
    const dim3 grid(unsigned(p.G + TC_COLC_BLOCKS), unsigned(p.total / (p.G + TC_COLC_BLOCKS)));
    if (p.fold > 1) tc_expand_kernel<true><<<grid, 256, 0, st>>>(p);
    else tc_expand_kernel<false><<<grid, 256, 0, st>>>(p);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? DS_OK : DS_ERR_CUDA;
}

template <bool NEXT>
static int launch_run(const TcRun& p, int BN, cudaStream_t st)
{
    switch (BN) {
        case 192: return run_cfg<192, NEXT, false>(p, st);
        case 128:
            // Where K is shared, or several column tiles of few items each, the epilogue sets the pace, and two producer
            // warpgroups leave it more of the schedulers; elsewhere three are faster.  Measured, us, three -> two.  K shared:
            // 7936 x 891 -> 377 102 -> 85, 700 x 4096 -> 500 46 -> 36, 16 images of 256 channels, 14 x 14, 3x3 -> 128 37 -> 28,
            // 1000 x 2048 -> 1000 34 -> 35.  1x1 on 36 images of 82 x 82: -> 162 channels, six items 109 -> 103, eight 127 -> 119,
            // nine 126 -> 119, ten 132 -> 137; -> 256, eight 127 -> 118, nine 121 -> 128, ten 129 -> 147; -> 128 (one column
            // tile), six 52 -> 54, nine 64 -> 70, ten 69 -> 80.  28 x 28, 256 images -> 128, fourteen 72 -> 88, 36 (3x3) 134 -> 152.
            return p.splits > 1 || (p.grid_n > 1 && p.G <= 8) ? run_cfg<128, NEXT, false, true>(p, st) : run_cfg<128, NEXT, false>(p, st);
        case 96: return run_cfg<96, NEXT, false>(p, st);
        case 64: return run_cfg<64, NEXT, false>(p, st);
        case 48: return run_cfg<48, NEXT, false>(p, st);
        default: return run_cfg<32, NEXT, false>(p, st);
    }
}

int tc_launch_run(const TcRun& p, int BN, bool wide, cudaStream_t st)
{
    if (wide) return run_cfg<64, false, true>(p, st);
    return p.next ? launch_run<true>(p, BN, st) : launch_run<false>(p, BN, st);
}

}  // namespace ds
