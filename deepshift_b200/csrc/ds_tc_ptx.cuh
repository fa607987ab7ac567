// Tensor-core path: what its kernels share on the device -- barriers, tcgen05, the planes of a value and the table of
// coefficients.  The arithmetic is described in ds_tc.cuh.
#pragma once
#include "ds_tc.cuh"

namespace ds {

int* kernel_error_flag();

namespace {

constexpr int TC_TMEM_COLS = 512;

constexpr int TC_WAIT_ROUNDS = 1 << 22;    // rounds of one wait, each up to TC_WAIT_NS
constexpr unsigned TC_WAIT_NS = 1000000;   // suspend hint of one round
constexpr unsigned long long TC_DRAIN_NS = 2000000000ull;  // limit on what a CTA has in flight when it ends

// Checked build: parts of the kernels that ds_tc_debug_waits keeps from doing their work, so that waits run out.
#ifdef DS_BOUNDS_CHECK
#define TC_HELD(p, bit) (((p).hold & (bit)) != 0)
#else
#define TC_HELD(p, bit) false
#endif

__device__ __forceinline__ unsigned s32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(unsigned long long* b, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void bar_arrive(unsigned long long* b)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(s32(b)) : "memory");
}

__device__ __forceinline__ bool bar_try(unsigned long long* b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool bar_try_long(unsigned long long* b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s32(b)), "r"(parity), "r"(TC_WAIT_NS)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool bar_test(unsigned long long* b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait of at most limit_ns; whoever gives up sets the CTA's error word, and every wait that finds it set and its
// barrier not ready returns at once.  The longest wait of a correct run is the epilogue's for one unit of K: planes
// stay below 2^31 bytes and tiles in 180 GB, which leaves at most 2^19 groups of half a microsecond.
// The first rounds carry no suspend hint: with one, a wait between warps of the main loop wakes up later
// (7 % of the whole kernel).
__device__ __forceinline__ bool bar_wait(unsigned long long* b, unsigned parity, volatile int* err, unsigned limit_ns)
{
    if (bar_test(b, parity)) return true;
    for (int i = 0; i < 32; ++i) {
        if (*err) return false;
        if (bar_try(b, parity)) return true;
    }
    const unsigned long long t0 = now_ns();
    for (int i = 0; i < TC_WAIT_ROUNDS; ++i) {
        if (bar_try_long(b, parity)) return true;
        if (*err) return false;
        if (now_ns() - t0 > limit_ns) break;
    }
    *err = 1;
    return false;
}

// Wait for this CTA's own copies or MMAs in flight, error or not.
__device__ __forceinline__ bool bar_drain(unsigned long long* b, unsigned parity)
{
    if (bar_try(b, parity)) return true;
    const unsigned long long t0 = now_ns();
    for (int i = 0; i < TC_WAIT_ROUNDS; ++i) {
        if (bar_try_long(b, parity)) return true;
        if (now_ns() - t0 > TC_DRAIN_NS) break;
    }
    return false;
}

// One copy of `bytes` (a multiple of 16) into shared memory; its arrival completes the barrier's phase.
__device__ __forceinline__ void bulk_load(unsigned dst, const unsigned char* src, unsigned bytes, unsigned long long* bar)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(s32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                 "r"(bytes), "r"(s32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_alloc(unsigned* at)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(at)), "n"(TC_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_dealloc()
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(0), "n"(TC_TMEM_COLS));
}

__device__ __forceinline__ void tc_commit(unsigned long long* b)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(b)) : "memory");
}

__device__ __forceinline__ void tc_mma_i8(unsigned d, unsigned a, unsigned long long bdesc, unsigned idesc, unsigned acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

// True in one lane of the (converged) warp, always the same one.
__device__ __forceinline__ bool elect_one()
{
    unsigned e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e)::"memory");
    return e != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

#define TC_R4(v, i) "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3])
#define TC_W4(v, i) "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3])

__device__ __forceinline__ void tmem_st32(unsigned addr, const unsigned* v)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
        TC_R4(v, 0), TC_R4(v, 4), TC_R4(v, 8), TC_R4(v, 12), TC_R4(v, 16), TC_R4(v, 20), TC_R4(v, 24), TC_R4(v, 28)
        : "memory");
}

__device__ __forceinline__ void tmem_ld(unsigned addr, int (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
        : TC_W4(v, 0), TC_W4(v, 4), TC_W4(v, 8), TC_W4(v, 12), TC_W4(v, 16), TC_W4(v, 20), TC_W4(v, 24), TC_W4(v, 28)
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld(unsigned addr, int (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : TC_W4(v, 0), TC_W4(v, 4), TC_W4(v, 8), TC_W4(v, 12)
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tmem_st16(unsigned addr, const unsigned* v)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
        TC_R4(v, 0), TC_R4(v, 4), TC_R4(v, 8), TC_R4(v, 12)
        : "memory");
}

// 16 bytes from an address aligned to `align` (16, 8 or 4).
__device__ __forceinline__ uint4 ld16(const unsigned char* a, int align)
{
    if (align == 16) return __ldg(reinterpret_cast<const uint4*>(a));
    uint4 v;
    if (align == 8) {
        const uint2 x = __ldg(reinterpret_cast<const uint2*>(a)), y = __ldg(reinterpret_cast<const uint2*>(a) + 1);
        v = make_uint4(x.x, x.y, y.x, y.y);
    } else {
        const unsigned* w = reinterpret_cast<const unsigned*>(a);
        v = make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
    }
    return v;
}

// Planes 0-7 of four values (one byte each of l and h): word q of each plane.
__device__ __forceinline__ void planes_low(unsigned l, unsigned h, unsigned* v, int q)
{
    const unsigned b7 = (l >> 7) & 0x01010101u, b15 = (h >> 7) & 0x01010101u;
    v[q] = (l & 0x7F7F7F7Fu) + b7 + 2u * (h & 0x01010101u);  // <= 130: no carry between bytes
    v[4 + q] = (l >> 1) & 0x3F3F3F3Fu;
    v[8 + q] = (l >> 2) & 0x3F3F3F3Fu;
    v[12 + q] = (l >> 3) & 0x1F1F1F1Fu;
    v[16 + q] = (l >> 4) & 0x0F0F0F0Fu;
    v[20 + q] = (l >> 5) & 0x07070707u;
    v[24 + q] = (l >> 6) & 0x03030303u;
    v[28 + q] = (h - b15) + b7;                               // 0..255: b15 set means h >= 128
}

__device__ __forceinline__ void planes_high(unsigned h, unsigned* v, int q)
{
    v[q] = h;
    v[4 + q] = (h >> 1) & 0x7F7F7F7Fu;
    v[8 + q] = (h >> 2) & 0x3F3F3F3Fu;
    v[12 + q] = (h >> 3) & 0x1F1F1F1Fu;
    v[16 + q] = (h >> 4) & 0x0F0F0F0Fu;
    v[20 + q] = (h >> 5) & 0x07070707u;
    v[24 + q] = (h >> 6) & 0x03030303u;
    v[28 + q] = (h >> 7) & 0x01010101u;
}

// Bytes l and h of four codes; notes a code that does not fit 16 bits.
__device__ __forceinline__ void pack4(const int (&c)[4], unsigned& l, unsigned& h, bool& over)
{
    unsigned y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        y[e] = unsigned(c[e]) + 32768u;
        over |= y[e] > 65535u;
    }
    const unsigned a = __byte_perm(y[0], y[1], 0x5140), b = __byte_perm(y[2], y[3], 0x5140);  // l0 l1 h0 h1
    l = __byte_perm(a, b, 0x5410);
    h = __byte_perm(a, b, 0x7632);
}

__device__ __forceinline__ uint4 lds128(unsigned addr)
{
    uint4 v;
    asm("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// Byte f of the four words a, as word f.
__device__ __forceinline__ void transpose4(unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned& o0, unsigned& o1,
                                           unsigned& o2, unsigned& o3)
{
    const unsigned x01 = __byte_perm(a0, a1, 0x5140), y01 = __byte_perm(a0, a1, 0x7362);
    const unsigned x23 = __byte_perm(a2, a3, 0x5140), y23 = __byte_perm(a2, a3, 0x7362);
    o0 = __byte_perm(x01, x23, 0x5410);
    o1 = __byte_perm(x01, x23, 0x7632);
    o2 = __byte_perm(y01, y23, 0x5410);
    o3 = __byte_perm(y01, y23, 0x7632);
}

// Coefficient of plane f for a right shift r in 0..15 (ds_tc.cuh).
constexpr int tc_coef(int r, int f)
{
    if (r == 0) return f == 0 ? 1 : (f == 7 || f == 8 || f == 15) ? 127 : f == 9 ? 4 : 0;
    if (r == 1) return f == 1 ? 1 : (f == 7 || f == 8 || f == 15) ? 64 : 0;
    if (r <= 6) return f == r ? 1 : f == 8 ? 1 << (8 - r) : 0;
    if (r == 7) return (f == 7 || f == 8 || f == 15) ? 1 : 0;
    return f == r ? 1 : 0;
}

// Planes 16-21 of a 24-bit value, all copies of t: 2^(16-r) for r >= 9 in planes 16 and 17, 2^(8-r) in planes
// 18-21 (the accumulator of weight 2^8) for r <= 8.
constexpr int tc_coef_t(int r, int f)
{
    if (f >= 22) return 0;
    if (f == 16) return r == 9 ? 64 : r > 9 ? 1 << (16 - r) : 0;
    if (f == 17) return r == 9 ? 64 : 0;
    if (r == 0) return 64;
    if (r == 1) return f <= 19 ? 64 : 0;
    return f == 18 && r <= 8 ? 1 << (8 - r) : 0;
}

// [four planes][code]: the signed coefficients of four planes as the bytes of a word; code 32 is a zero weight.
struct TcLut {
    unsigned w[6 * 33];
};
constexpr TcLut tc_make_lut()
{
    TcLut t = {};
    for (int q = 0; q < 6; ++q)
        for (int c = 0; c < 33; ++c)
            for (int e = 0; e < 4; ++e) {
                const int v = c == 32 ? 0 : (c & 16 ? -1 : 1) * (q < 4 ? tc_coef(c & 15, 4 * q + e) : tc_coef_t(c & 15, 4 * q + e));
                t.w[q * 33 + c] |= (unsigned(v) & 255u) << (8 * e);
            }
    return t;
}
__constant__ TcLut g_tc_lut = tc_make_lut();

}  // namespace
}  // namespace ds
