// Linear layers with few rows on the tensor cores (tcgen05, kind::i8): the weights are expanded inside the kernel.
//
// tc_run (ds_tc.cu) reads weights that were expanded to sixteen bytes each, which pays for itself over many rows or many
// calls.  Here the operands change places: the rows of the MMA are 128 output columns, whose packed words a producer
// thread decodes straight into tensor memory (A, s8), and the columns are rows of x, as planes f_0..f_15 that a first pass
// has made from the codes (B, u8: 256 bytes per value and 16 rows, fetched with cp.async.bulk).
//
//   few_pack     x (int32) -> [row tile][group][16 planes][BN rows][16 bytes], every code's range noted, and the output
//                zeroed where K is shared.  A group is the weights of whole packed words, 16 at most.
//   few_run      persistent, one CTA per SM, warp-specialised: three producer warpgroups, four epilogue warps, one
//                issuing lane, one loading lane; the hand-shake is tc_run's.
//
// The last column of a tile is a row of zeros (code 0).  Its sum is what the offset 2^15 of the planes adds up to in the
// others, so no column constants are needed: out = D[n][m] - D[n][last].  Words past the end of K, whatever they
// decode to, meet code 0 in every column and cancel as well.
//
// Expanding a weight: its packed field is the index into a table of sixteen signed coefficients in shared memory (one
// 16-byte read), and four weights' planes are transposed 4 x 4 bytes.  Eight copies of the table, one per lane of a
// quarter warp, each in banks of its own, so that no two reads of one phase collide.
//
// What bounds it: at 80 columns the producers, 64 x 4096 -> 4096 29.7 us = 830 cycles per item, of which the MMAs take 320 and the
// ALU pipe 350; the rest is waiting for the packed words, 16 bytes per thread at the rows' pitch (78 % of the sectors
// come from L1; a prefetch into L1 changed nothing).  The whole call 41 us, 136 on the integer path.  At 144 columns the
// MMAs (576 cycles per item).
#include "ds_tc_ptx.cuh"

#include <algorithm>

namespace ds {

int* bounds_status_ptr();

namespace {

constexpr int FEW_WG = 3;                             // producer warpgroups, one A slot each
constexpr int FEW_THREADS = (4 * FEW_WG + 6) * 32;    // + epilogue warpgroup, MMA warp, loader warp
constexpr int FEW_NACC = 2;
constexpr int FEW_FLAGS = 1024;                       // blocks of few_pack, each with a range flag of its own
constexpr int FEW_HEADER = 4 * (FEW_FLAGS + 4);       // the flag of the whole call, then the blocks'

// 160 bytes.  What a launch costs the host depends on this size in no obvious way: three launches of a call 12.3 us at 128
// bytes, 12.3 at 136 and 144, 10.9 at 160, 11.4 at 168, 12.2 at 176, 12.9 at 192.
struct FewParams {
    const int* x;
    const int* packed;
    const int* bias;
    int* out;
    int* flag;           // whole call; the blocks' flags at flag + 4
    int* report;         // as in TcRun
    unsigned char* planes;
    int M, K, N, row_len, G, kpg;
    int grid_m, grid_n, splits, gps, units, rpt;  // rpt: rows of x per tile, the last column is the row of zeros
    int blocks;          // of few_pack
    int gated;           // the range is measured
    int zero_out;
    unsigned wait_ns;
    int* err_flag;
    long long chk_x_bytes, chk_w_bytes, chk_o_bytes;
    int* chk_status;
#ifdef DS_BOUNDS_CHECK
    const unsigned char* chk_act;  // the whole scratch
    long long chk_act_bytes;
    int hold;                      // see ds_tc_debug_waits
#endif
};

template <int BN>
struct FewTile {
    static constexpr int STAGE = BN * TC_PLANES * TC_KG;
    static constexpr int STAGES = BN == 144 ? 4 : 6;
    static constexpr int ACC_COLS = TC_TMEM_COLS - 64 * FEW_WG;
    static_assert(FEW_NACC * BN <= ACC_COLS && STAGES > FEW_WG, "slots");
};

template <int BN, int FW>
struct FewSmem {
    alignas(128) unsigned char b[FewTile<BN>::STAGES][FewTile<BN>::STAGE];
    alignas(128) uint4 lut[1 << FW][8];
    alignas(8) unsigned long long bfull[FewTile<BN>::STAGES];
    unsigned long long full[FEW_WG];
    unsigned long long empty[FEW_WG];
    unsigned long long accfull[FEW_NACC];
    unsigned long long accempty[FEW_NACC];
    unsigned long long done;
    unsigned tmem;
    int err;
};

// One thread: the 16 planes of one group of one row.
template <int BN>
__global__ void __launch_bounds__(256) few_pack_kernel(const FewParams p)
{
    const unsigned rows = unsigned(p.grid_m) * BN;
    const unsigned total = rows * unsigned(p.G);  // checked by the entry point
    const bool vec = p.K % 4 == 0 && p.kpg % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0;
    bool over = false;
    for (unsigned i = blockIdx.x * 256u + threadIdx.x; i < total; i += gridDim.x * 256u) {
        const unsigned tg = i / BN, r = i - tg * BN, mt = tg / unsigned(p.G), g = tg - mt * unsigned(p.G);
        const int m = int(mt) * p.rpt + int(r);
        const int k0 = int(g) * p.kpg;
        const bool live = int(r) < p.rpt && m < p.M;
        const int* src = p.x + (long long)m * p.K + k0;
        unsigned v[64];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int c[4] = {0, 0, 0, 0};
            if (live) {
                if (vec) {
                    if (4 * q < p.kpg && k0 + 4 * q < p.K && DS_X_OK(p, src + 4 * q, 16)) {
                        const int4 t = __ldg(reinterpret_cast<const int4*>(src) + q);
                        c[0] = t.x; c[1] = t.y; c[2] = t.z; c[3] = t.w;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (4 * q + e < p.kpg && k0 + 4 * q + e < p.K && DS_X_OK(p, src + 4 * q + e, 4)) c[e] = __ldg(src + 4 * q + e);
                }
            }
            unsigned l, h;
            pack4(c, l, h, over);
            planes_low(l, h, v, q);
            planes_high(h, v + 32, q);
        }
        uint4* dst = reinterpret_cast<uint4*>(p.planes) + ((long long)tg * TC_PLANES * BN + r);
#pragma unroll
        for (int f = 0; f < TC_PLANES; ++f)
            if (DS_A_OK(p, dst + f * BN, 16)) dst[f * BN] = make_uint4(v[4 * f], v[4 * f + 1], v[4 * f + 2], v[4 * f + 3]);
    }
    if (p.zero_out) {
        const long long n = (long long)p.M * p.N;
        for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll)
            if (DS_O_OK(p, p.out, p.out + i, 4)) p.out[i] = 0;
    }
    // a flag per block, written whatever it is: none has to be cleared by a launch before
    const int any = __syncthreads_or(over);
    if (threadIdx.x == 0) p.flag[4 + blockIdx.x] = any;
}

struct FewUnit {
    int mt, nt, sp, g0, g1;
};

// Neighbouring CTAs share a tile of planes.
__device__ __forceinline__ FewUnit few_unit(const FewParams& p, int u)
{
    FewUnit r;
    const int t = u / p.grid_n;
    r.nt = u - t * p.grid_n;
    r.mt = t / p.splits;
    r.sp = t - r.mt * p.splits;
    r.g0 = r.sp * p.gps;
    r.g1 = min(p.G, r.g0 + p.gps);
    return r;
}

template <int BN, int FW>
__global__ void __launch_bounds__(FEW_THREADS, 1) few_run_kernel(const FewParams p)
{
    using T = FewTile<BN>;
    constexpr int NUM = 32 / FW, WPG = 16 / NUM, KPG = NUM * WPG;  // weights per word, words and weights per group
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FewSmem<BN, FW>& s = *reinterpret_cast<FewSmem<BN, FW>*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (p.gated) {
        int over = 0;
        for (int i = threadIdx.x; i < p.blocks; i += FEW_THREADS) over |= __ldg(p.flag + 4 + i);
        over = __syncthreads_or(over);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *p.flag = over;  // for the integer path behind
            if (p.report) *p.report = over;
        }
        if (over) return;
    }
    volatile int* err = &s.err;
    for (int i = threadIdx.x; i < (8 << FW); i += FEW_THREADS) {
        const int field = i >> 3, r = field & ((1 << (FW - 1)) - 1);
        const int code = r >= 32 ? 32 : min(r, 15) | ((field >> (FW - 1)) ? 0 : 16);
        s.lut[field][i & 7] = make_uint4(g_tc_lut.w[code], g_tc_lut.w[33 + code], g_tc_lut.w[66 + code], g_tc_lut.w[99 + code]);
    }
    if (threadIdx.x == 0) {
        s.err = 0;
        for (int i = 0; i < T::STAGES; ++i) bar_init(&s.bfull[i], 1);
        for (int i = 0; i < FEW_WG; ++i) {
            bar_init(&s.full[i], 5);  // four producer warps and the loader
            bar_init(&s.empty[i], 1);
        }
        for (int i = 0; i < FEW_NACC; ++i) {
            bar_init(&s.accfull[i], 1);
            bar_init(&s.accempty[i], 4);
        }
        bar_init(&s.done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 * FEW_WG + 4) tmem_alloc(&s.tmem);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr unsigned tmem_a = T::ACC_COLS;  // all columns are this CTA's: they start at 0
    if (threadIdx.x == 0 && s.tmem != 0) s.err = 1;

    if (warp < 4 * FEW_WG) {
        // ---- producers: expand weights into TMEM -----------------------------------------------------------
        const int wg = warp >> 2, row = threadIdx.x & 127;
        const unsigned at = tmem_a + (unsigned(warp & 3) << 21) + wg * 64;
        const unsigned lut = s32(&s.lut[0][lane & 7]);
        const bool vec = WPG > 1 && p.row_len % WPG == 0 && (reinterpret_cast<uintptr_t>(p.packed) & (4 * WPG - 1)) == 0;
        int u = blockIdx.x, g = 0, g1 = 0;
        const int* wrow = p.packed;
        auto enter = [&](int skip) {
            for (; u < p.units; u += gridDim.x) {
                const FewUnit un = few_unit(p, u);
                g = un.g0 + skip;
                g1 = un.g1;
                if (g < g1) {
                    wrow = p.packed + (long long)min(un.nt * TC_ROWS + row, p.N - 1) * p.row_len;
                    return;
                }
                skip = g - g1;
            }
        };
        auto step = [&]() {
            g += FEW_WG;
            if (g >= g1) {
                u += gridDim.x;
                enter(g - g1);
            }
        };
        unsigned nw[WPG];
#pragma unroll
        for (int i = 0; i < WPG; ++i) nw[i] = 0;
        auto fetch = [&]() {
            const int w = g * WPG;
            const int* a = wrow + w;
            if (vec && WPG == 4) {
                if (DS_W_OK(p, a, 16)) {
                    const uint4 t = __ldg(reinterpret_cast<const uint4*>(a));
                    nw[0] = t.x; nw[WPG > 1 ? 1 : 0] = t.y; nw[WPG > 2 ? 2 : 0] = t.z; nw[WPG > 3 ? 3 : 0] = t.w;
                }
            } else if (vec && WPG == 2) {
                if (DS_W_OK(p, a, 8)) {
                    const uint2 t = __ldg(reinterpret_cast<const uint2*>(a));
                    nw[0] = t.x; nw[WPG > 1 ? 1 : 0] = t.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < WPG; ++i) nw[i] = (w + i < p.row_len && DS_W_OK(p, a + i, 4)) ? unsigned(__ldg(a + i)) : 0u;
            }
        };
        enter(wg);
        if (u < p.units) fetch();
        for (unsigned use = 0; u < p.units; ++use) {
            unsigned w[WPG];
#pragma unroll
            for (int i = 0; i < WPG; ++i) w[i] = nw[i];
            step();
            if (u < p.units) fetch();
            unsigned v[64];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 a[4];  // coefficients of four weights
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int k = 4 * q + e;
                    a[e] = make_uint4(0, 0, 0, 0);
                    if (k < KPG) {
                        const unsigned word = w[k / NUM];
                        const int sh = k % NUM * FW - 7;  // the field, times the 128 bytes of a table row
                        const unsigned off = (sh < 0 ? word << (sh < 0 ? -sh : 0) : word >> (sh < 0 ? 0 : sh)) & (((1u << FW) - 1u) << 7);
                        a[e] = lds128(lut + off);
                    }
                }
                transpose4(a[0].x, a[1].x, a[2].x, a[3].x, v[q], v[4 + q], v[8 + q], v[12 + q]);
                transpose4(a[0].y, a[1].y, a[2].y, a[3].y, v[16 + q], v[20 + q], v[24 + q], v[28 + q]);
                transpose4(a[0].z, a[1].z, a[2].z, a[3].z, v[32 + q], v[36 + q], v[40 + q], v[44 + q]);
                transpose4(a[0].w, a[1].w, a[2].w, a[3].w, v[48 + q], v[52 + q], v[56 + q], v[60 + q]);
            }
            const bool ok = use == 0 || bar_wait(&s.empty[wg], (use - 1) & 1u, err, p.wait_ns);
            if (!__all_sync(0xFFFFFFFFu, ok) || TC_HELD(p, 2)) break;  // the whole warp, or none of it
            tc_fence_after();
            tmem_st32(at, v);
            tmem_st32(at + 32, v + 32);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(&s.full[wg]);
        }
    } else if (warp < 4 * FEW_WG + 4) {
        // ---- epilogue: a thread is an output column, its columns are rows of x ------------------------------
        const int row = threadIdx.x & 127;
        const unsigned lane_base = unsigned(warp & 3) << 21;
        unsigned acc = 0;
        for (int u = blockIdx.x; u < p.units; u += gridDim.x, ++acc) {
            const FewUnit un = few_unit(p, u);
            const int n = un.nt * TC_ROWS + row;
            const int b = p.bias && un.sp == 0 && n < p.N ? __ldg(p.bias + n) : 0;
            const unsigned slot = acc % FEW_NACC;
            if (!__all_sync(0xFFFFFFFFu, bar_wait(&s.accfull[slot], (acc / FEW_NACC) & 1u, err, p.wait_ns))) continue;
            tc_fence_after();
            const unsigned base = lane_base + slot * BN;
            const int m0 = un.mt * p.rpt, rows = min(p.rpt, p.M - m0);
            int v[16];
            tmem_ld(base + BN - 16, v);
            const int zero = b - v[15];
            int* o = p.out + (long long)m0 * p.N + n;
#pragma unroll 1
            for (int c = 0; c < rows; c += 16) {
                tmem_ld(base + c, v);
#pragma unroll
                for (int q = 0; q < 16; ++q, o += p.N)
                    if (c + q < rows && n < p.N && DS_O_OK(p, p.out, o, 4)) {
                        if (p.splits > 1) atomicAdd(o, v[q] + zero);
                        else *o = v[q] + zero;
                    }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && !TC_HELD(p, 4)) bar_arrive(&s.accempty[slot]);
        }
    } else if (warp == 4 * FEW_WG + 4) {
        // ---- MMA issue: one lane, one wait and one commit per item, asked ahead (ds_tc.cu) -------------------
        // D s32, A s8, B u8, both K-major, N = BN, M = 128
        constexpr unsigned idesc = (2u << 4) | (1u << 7) | (0u << 10) | (unsigned(BN / 8) << 17) | (8u << 24);
        const unsigned long long desc0 =
            (1ull << 46) | (8ull << 32) | ((unsigned long long)BN << 16) | (s32(&s.b[0][0]) >> 4);
        if (elect_one()) {
            unsigned slot = 0, ph = 0, st = 0, aslot = 0, accph = 1;
            bool ready = false;
            for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
                const FewUnit un = few_unit(p, u);
                bar_wait(&s.accempty[aslot], accph, err, p.wait_ns);  // the first round finds the slots free
                const unsigned d = aslot * BN;
                unsigned more = 0;
                for (int g = un.g0; g < un.g1; ++g) {
                    if (!ready) bar_wait(&s.full[slot], ph, err, p.wait_ns);
                    const unsigned cur = slot;
                    if (++slot == unsigned(FEW_WG)) {
                        slot = 0;
                        ph ^= 1u;
                    }
                    ready = bar_test(&s.full[slot], ph);
                    const unsigned long long bdesc = desc0 + st * unsigned(T::STAGE >> 4);
                    tc_fence_after();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        tc_mma_i8(d, tmem_a + cur * 64 + q * 8, bdesc + q * (2 * BN), idesc, q == 0 ? more : 1u);
                    tc_commit(&s.empty[cur]);
                    more = 1;
                    if (++st == unsigned(T::STAGES)) st = 0;
                }
                tc_commit(&s.accfull[aslot]);
                if (++aslot == unsigned(FEW_NACC)) {
                    aslot = 0;
                    accph ^= 1u;
                }
            }
            tc_commit(&s.done);  // nothing of this CTA is in flight when the columns go back
            if (!bar_drain(&s.done, 0)) *err = 1;
        }
        __syncwarp();
    } else {
        // ---- tiles of planes: one thread, as in ds_tc.cu ----------------------------------------------------
        if (lane == 0) {
            int lu = blockIdx.x, lleft = 0;
            const unsigned char* src = nullptr;
            unsigned lst = 0, issued = 0;
            auto fetch = [&]() {
                while (lleft == 0) {
                    if (lu >= p.units || TC_HELD(p, 1)) return;
                    const FewUnit un = few_unit(p, lu);
                    src = p.planes + ((long long)un.mt * p.G + un.g0) * T::STAGE;
                    lleft = un.g1 - un.g0;
                    lu += gridDim.x;
                }
                if (DS_A_OK(p, src, T::STAGE)) bulk_load(s32(&s.b[lst][0]), src, T::STAGE, &s.bfull[lst]);
                else bar_arrive(&s.bfull[lst]);
                src += T::STAGE;
                --lleft;
                ++issued;
                if (++lst == unsigned(T::STAGES)) lst = 0;
            };
            for (int i = 0; i < T::STAGES; ++i) fetch();
            unsigned i = 0, st = 0, bph = 0, slot = 0, ph = 1;
            auto next = [&]() {
                if (++st == unsigned(T::STAGES)) {
                    st = 0;
                    bph ^= 1u;
                }
            };
            for (; i < issued; ++i, next()) {
                if (i >= unsigned(FEW_WG)) {
                    if (!bar_wait(&s.empty[slot], ph, err, p.wait_ns)) break;
                    fetch();
                }
                if (!bar_wait(&s.bfull[st], bph, err, p.wait_ns)) break;
                bar_arrive(&s.full[slot]);
                if (++slot == unsigned(FEW_WG)) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
            for (; i < issued; ++i, next())  // every copy has landed before the CTA ends
                if (!bar_drain(&s.bfull[st], bph)) *err = 1;
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 4 * FEW_WG + 4) tmem_dealloc();
    if (threadIdx.x == 0 && s.err) *p.err_flag = 1;
}

template <int BN, int FW>
int few_cfg(const FewParams& p, cudaStream_t st)
{
    const int dev = device_slot();
    if (dev < 0) return DS_ERR_CUDA;
    auto kern = few_run_kernel<BN, FW>;
    const size_t smem = sizeof(FewSmem<BN, FW>);
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
    few_pack_kernel<BN><<<p.blocks, 256, 0, st>>>(p);
    note_launch();
    kern<<<p.units < sms[dev] ? p.units : sms[dev], FEW_THREADS, smem, st>>>(p);
    note_launch();
    return cudaGetLastError() == cudaSuccess ? DS_OK : DS_ERR_CUDA;
}

template <int BN>
int few_launch(const FewParams& p, int fw, cudaStream_t st)
{
    switch (fw) {
        case 2: return few_cfg<BN, 2>(p, st);
        case 3: return few_cfg<BN, 3>(p, st);
        case 4: return few_cfg<BN, 4>(p, st);
        case 5: return few_cfg<BN, 5>(p, st);
        case 6: return few_cfg<BN, 6>(p, st);
        case 7: return few_cfg<BN, 7>(p, st);
        case 8: return few_cfg<BN, 8>(p, st);
        default: return DS_ERR_UNSUPPORTED;
    }
}

struct FewGeom {
    int BN, rpt, grid_m, grid_n, G, wpg, kpg, row_len, splits, gps, blocks;
    long long act_bytes;
    double run_us;  // estimated time of few_run
};

// Which calls: int32 codes that are promised or measured to fit 16 bits, right shifts, nothing fused.
int few_mode(const ds_fuse_t& f, int bits, int base)
{
    if (base != 0 || bits < 1 || bits > 7 || f.in_kind != DS_IN_I32) return 0;
    if (f.out_kind != DS_OUT_I32 || f.relu || f.requant || f.round_f32 || f.residual) return 0;
    return f.act_bits == DS_ACT_BITS_AUTO ? 2 : f.act_bits >= 1 && f.act_bits <= 15 ? 1 : 0;
}

bool few_geometry(FewGeom& g, int M, int K, int N, int bits)
{
    const int num = 32 / (bits + 1);
    g.row_len = (K + num - 1) / num;
    g.wpg = 16 / num;
    g.kpg = g.wpg * num;
    g.G = (g.row_len + g.wpg - 1) / g.wpg;
    g.BN = M <= 79 ? 80 : 144;
    g.grid_m = (M + g.BN - 2) / (g.BN - 1);
    g.rpt = (M + g.grid_m - 1) / g.grid_m;
    g.grid_n = (N + TC_ROWS - 1) / TC_ROWS;
    const long long bytes = (long long)g.grid_m * g.G * g.BN * (TC_PLANES * TC_KG);
    if (bytes > (1ll << 31) || (long long)M * N > 0x7FFFFFFFll || (long long)M * K > 0x7FFFFFFFll) return false;
    g.act_bytes = FEW_HEADER + bytes;
    const long long want = ((long long)g.grid_m * g.G * g.BN + 255) / 256;
    g.blocks = int(want > FEW_FLAGS ? FEW_FLAGS : want);
    // K is shared until the units fill the SMs evenly; an item is 16 weights of 128 columns.  The cycles are what a short unit's
    // items cost beyond its 1500: an item of a long one takes 700 (80 columns) and 880 (144), start and end of the launch 12000
    // in all.  The choice is what they are for: on 14 shapes (17 to 512 rows, 1024 to 8192 x 512 to 11008) it is within 2 % of
    // the best of all splits; and with the 10 us of few_worthwhile, the calls that take this path.
    const double item = g.BN == 144 ? 600 : 420;
    g.run_us = 1e30;
    for (int sp = 1; sp <= 64; ++sp) {
        const int gps = (g.G + sp - 1) / sp;
        if (sp > 1 && (gps < 4 || (g.G + gps - 1) / gps != sp)) continue;
        const double waves = double(((long long)g.grid_m * g.grid_n * sp + 147) / 148);
        const double us = (waves * (gps * item + 1500) + 6000) / 1900;
        if (us < g.run_us) {
            g.run_us = us;
            g.splits = sp;
            g.gps = gps;
        }
    }
    return (long long)g.grid_m * g.grid_n * g.splits <= 0x7FFFFFFFll - 4096;
}

// Whether this path beats the others.  Measured, us a call, range measured, other path (integer up to 64 rows, expanded
// weights above) -> this one: 17 x 4096 -> 4096 133 -> 39, 64 x 4096 -> 4096 138 -> 42, 64 x 1024 -> 4096 46 -> 35, 64 x 1024 ->
// 1024 20 -> 24, 64 x 2048 -> 1024 28 -> 35, 128 x 4096 -> 4096 175 -> 51, 256 x 1024 -> 1024 42 -> 28, 512 x 4096 -> 4096 203 -> 134,
// 1024 x 4096 -> 4096 324 -> 284, 2000 x 4096 -> 4096 439 -> 473.  With a promise 64 x 4096 -> 4096 98 -> 38, 64 x 1024 -> 1024 18 -> 22;
// above 64 rows the other path is then the FP32 pipe in one launch (ds_tc_host.cu, promised_linear): 80 x 1500 -> 400 23 -> 28,
// 200 x 1216 -> 256 23 -> 28, 65 x 4096 -> 10 31 -> 29, 128 x 2048 -> 1000 31 -> 28, 128 x 4096 -> 1000 52 -> 29.
// The 15 % keep calls at the crossing where they were.
bool few_worthwhile(const FewGeom& g, int M, int K, int N, int mode)
{
    if (M <= 16 || K < 256) return false;
    const double here = g.run_us + 10 + 1e-6 * M * (double)K * 20;  // packing, gaps between the launches
    const double weights = (double)N * K;
    double there;
    if (M <= 64) there = 6 + 64 * weights / (mode == 2 ? 7.9e6 : 11.6e6);
    else there = 22 + 0.005 * K + 6.5e-6 * weights + (double)((M + 127) / 128 * 128) * weights / 100e6;
    if (M > 64 && mode == 1) {
        const double pipe = 8 + 0.09e-6 * ((M + 63) / 64 * 64) * (double)K * ((N + 127) / 128 * 128), depth = 1 + 0.0072 * K;
        there = std::min(there, std::max({21.0, pipe, depth}));
    }
    return (here > 26 ? here : 26) < 0.85 * there;
}

}  // namespace
}  // namespace ds

using namespace ds;

extern "C" int ds_tc_few_bytes(int M, int K, int N, int bits, int base, const ds_fuse_t* fuse, int any_size, long long* act_bytes)
{
    if (!fuse || !act_bytes) return DS_ERR_BAD_ARG;
    *act_bytes = 0;
    if (M < 1 || K < 1 || N < 1) return DS_ERR_BAD_ARG;
    const int mode = few_mode(*fuse, bits, base);
    FewGeom g;
    if (!mode || !few_geometry(g, M, K, N, bits)) return DS_OK;
    if (!any_size && !few_worthwhile(g, M, K, N, mode)) return DS_OK;
    *act_bytes = g.act_bytes;
    return DS_OK;
}

extern "C" int ds_tc_linear_few(const int32_t* x, const int32_t* packed, const int32_t* bias, int32_t* out, int M, int K, int N,
                                int bits, int base, const ds_fuse_t* fuse, void* act, long long act_bytes, void* stream)
{
    if (!x || !packed || !out || !fuse || !act || M < 1 || K < 1 || N < 1) return DS_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(act)) & 15u) return DS_ERR_ALIGN;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(bias)) & 3u) return DS_ERR_ALIGN;
    const int mode = few_mode(*fuse, bits, base);
    FewGeom g;
    if (!mode || !few_geometry(g, M, K, N, bits)) return DS_ERR_UNSUPPORTED;
    if (act_bytes < g.act_bytes) return DS_ERR_SCRATCH;
    FewParams p = {};
    p.x = x; p.packed = packed; p.bias = bias; p.out = out;
    p.flag = static_cast<int*>(act);
    p.planes = static_cast<unsigned char*>(act) + FEW_HEADER;
    p.M = M; p.K = K; p.N = N; p.row_len = g.row_len; p.G = g.G; p.kpg = g.kpg;
    p.grid_m = g.grid_m; p.grid_n = g.grid_n; p.splits = g.splits; p.gps = g.gps; p.rpt = g.rpt;
    p.units = g.grid_m * g.grid_n * g.splits;
    p.blocks = g.blocks;
    p.gated = mode == 2;
    std::optional<GateLock> lock;
    if (p.gated && (p.report = workspace_gate_word(fuse)) != nullptr) lock.emplace(p.report);
    p.zero_out = g.splits > 1 || p.gated;  // the integer path behind may share K as well
    p.wait_ns = tc_wait_ns();
    p.err_flag = kernel_error_flag();
    if (!p.err_flag) return DS_ERR_CUDA;
    p.chk_x_bytes = (long long)M * K * 4 - check_shrink_x();
    p.chk_w_bytes = (long long)N * g.row_len * 4;
    p.chk_o_bytes = (long long)M * N * 4;
    p.chk_status = bounds_status_ptr();
#ifdef DS_BOUNDS_CHECK
    p.chk_act = static_cast<const unsigned char*>(act);
    p.chk_act_bytes = g.act_bytes;
    p.hold = tc_hold();
#endif
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int rc = g.BN == 144 ? few_launch<144>(p, bits + 1, st) : few_launch<80>(p, bits + 1, st);
    if (rc || !p.gated) return rc;
    return launch_gated_int(x, packed, bias, out, M, K, 1, 1, N, 1, 1, 1, 1, 0, 0, bits, base, fuse, p.flag, 1, true, st);
}
