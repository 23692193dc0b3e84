// BCQ product for several activation rows on the tensor cores (tcgen05), sm_100a.
//
//   y[m][n] = sum_b sum_k (+-alpha_b[k][n]) * x[m][k]
//
// The planes are never summed up to a weight: every plane is an operand of its own, whose elements are the fp16 scale
// with the plane's bit as its sign.  Such an element is exact, its product with an fp16 activation is exact in fp32, and
// all planes and all of K are summed in the fp32 accumulators of the tensor core.  Forming an element pair costs one
// shift and one three-input logic operation: bits t and t + 16 of a packed word are moved to the two sign bits of a
// 32-bit register that holds the (negated) scale twice.  Features are therefore paired (t, t + 16) along K, and the
// activations are staged in the same order.
//
// The tables of the one-row kernel (sal_lutgemm.cu) do not amortise over rows: every row looks every byte up again.  Here
// the work on the planes is done once for up to 256 rows, and the rows only add tensor-core time.
//
// The operands are written to tensor memory, from where the tensor core reads operand A at full rate (32 clocks for 128 columns x 16
// features x 64 rows, 10 for 16 rows); through shared memory an instruction takes 39 clocks at least, and the writes come on top.
//
// Roles of a CTA (128 output columns at a time, one CTA per SM, 23 warps):
//   warps 0-15  operand warps: lane = output column.  Words of the planes from the ring -> sign/scale operands (operand A); they
//               also read the accumulators back and write the result
//   warps 16-19 reorder the activations of a unit in place (a fence between plain stores and the tensor core waits for the
//               thread's outstanding loads, so these warps load nothing from global memory)
//   warp 20     planes and scales from global memory into the ring, up to twelve units ahead, by tiled TMA (4-byte
//               asynchronous copies where their rows are not aligned for it).  Neither depends on the kernel in front, so this
//               starts before griddepcontrol.wait
//   warp 21     issues tcgen05.mma (M = 128 output columns, N = rows, K = 16) and commits
//   warp 22     activations by tiled TMA into 128-byte-swizzled shared memory (operand B)
//
// Work split: the launch's (output tile, 128-feature unit) pairs in tile-major order are dealt to the CTAs in contiguous runs: whole
// numbers of CTAs per tile where that fills most of the SMs (whole_shares), else equal runs that may end inside a tile.  A tile that several CTAs
// share is summed by the last of them to arrive, in ascending order of K (deterministic), from fp32 partial sums in the scratch buffer.
//
// What bounds it: a unit takes 0.66 / 0.9 / 1.1 us for 2 / 3 / 4 planes up to 64 rows, against 0.13 to 0.26 us that its planes take to
// arrive.  About half of that the MMA warp waits for activations and the operand warps for the stages it frees; the operands
// themselves (32 logic operations per word and plane, tensor-memory stores) are some 900 clocks.  At 256 rows the tensor core (128
// clocks per instruction, 8 per plane and unit) and the same wait.  Measured in us, before (tables, a pass
// per pair of rows or per row) and here: 4096 x 11008, 4 planes, 8 rows 31 -> 27, 64 rows 174 -> 36; 11008 x 4096, 3 planes, 16 rows
// 42 -> 25; 28672 x 8192, 2 planes, 64 rows 540 -> 82; block layout, 11008 x 4096, 3 planes, 128 rows 959 -> 49.  Steps on the way: the
// scales by TMA instead of by plain loads in the staging warps; sixteen operand warps instead of eight; the activations by TMA and
// reordered in place (a proxy fence behind plain loads waits for them: 256 rows 301 -> 199 us at 28672 x 8192); the MMA behind
// elect.sync instead of `lane == 0` (34 -> 24 us at 11008 x 4096, 1 to 16 rows).  Operands through shared memory instead of tensor
// memory gained nothing (38 us there, before the last step).
//
// Every wait on a barrier is bounded (about a second) and not repeated: a thread that gave up once runs through to its end.  It is recorded
// as SAL_E_TIMEOUT in the header of the scratch buffer (a launch without one has no place for it).  The limit covers this launch's own
// pipeline only: a warp whose progress depends on the activations executes griddepcontrol.wait, which takes as long as the kernel in front
// does, before its first such wait.  The warps that issue copies and matrix instructions stop copying once they gave up, and wait (once more
// bounded) for what they have in flight before the CTA ends; in a launch that ran as it should that has long been consumed.
#include <cuda_fp16.h>
#include <float.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "sal_decode_ops.h"
#include "sal_launch.h"
#include "sal_mma.h"

namespace sal_mma {
namespace {

constexpr int TILE_N = 128;          // output columns of a tile = lanes of tensor memory
constexpr int UNIT_WORDS = 4;        // a unit is 4 packed words = 128 features of K
constexpr int OP_WARPS = 16;         // four per quarter of the lanes, one for each word of a unit
constexpr int STG_WARPS = 4;
constexpr int W_WARP = OP_WARPS + STG_WARPS;
constexpr int MMA_WARP = W_WARP + 1;
constexpr int X_WARP = MMA_WARP + 1;
constexpr int THREADS = (X_WARP + 1) * 32;
constexpr int MAX_X_UNITS = 4;       // units of activations in flight
// bytes of a staged row of scales.  By TMA: ROW 128 columns, BLOCK a tile's eight groups; by 4-byte copies with one value more in front
constexpr int S_PITCH_ROW = 272, S_PITCH_ROW_TMA = 256, S_PITCH_BLOCK = 32, S_PITCH_BLOCK_TMA = 16;
constexpr int TMEM_COLS = 512;
constexpr int MAX_MT = 256;          // rows of a row tile
constexpr size_t WS_HEADER = 256, WS_PARTIALS = 16384;
constexpr int MAX_CTAS = 148;        // one per SM
constexpr int MAX_COUNTERS = (int)(WS_PARTIALS - WS_HEADER) / 4;

template <int Q>
struct Cfg {
    static constexpr int W_BYTES = UNIT_WORDS * Q * TILE_N * 4;   // planes of a unit
    static constexpr int A_COLS = 32 * Q;                         // tensor-memory columns of the operand of 64 features
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, int *status) {
    uint64_t t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 256; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > 1000000000ull) break;
    }
    if (status) atomicExch(status, SAL_E_TIMEOUT);
    return false;
}
// `live` goes false with the first wait that runs out; later waits of the thread return at once.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, int *status, bool &live) {
    if (mbar_try_wait(bar, parity)) return;
    if (live) live = mbar_wait_slow(bar, parity, status);
}
// The same for a warp that runs ahead of the dependency wait: a barrier that has to be waited for may depend on the kernel in front, so
// that kernel is waited for first.
__device__ __forceinline__ void mbar_wait_behind(uint32_t bar, uint32_t parity, int *status, bool &live, bool &waited) {
    if (mbar_try_wait(bar, parity)) return;
    if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
    waited = true;
    if (live) live = mbar_wait_slow(bar, parity, status);
}
// Waits for the last fill of every slot of a ring: `next` is the slot that would be filled next, `empty_parity` the parity its producer
// would wait for (1 in the first round).
__device__ __forceinline__ void land(uint32_t full, int slots, int next, uint32_t empty_parity, int *status) {
    bool live = true;
    // a slot in front of `next` was last filled in this round, the others in the one before (in the first round: not at all, and a
    // fresh barrier passes a wait for the phase before its first)
    for (int i = 0; i < slots; ++i) mbar_wait(full + 8 * i, i < next ? empty_parity ^ 1u : empty_parity, status, live);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t selector) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
    return d;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_store16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_load4(uint32_t addr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
// D[128 columns][rows] (+)= A (tensor memory, fp16, K-major) * B (shared memory, fp16, K-major)
__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// One lane of a converged warp, known to the compiler as such: the same instructions behind `lane == 0` take 52 clocks each to issue
// (their operands must be uniform registers), behind this 10.
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// Shared-memory descriptor of a K-major operand in 128-byte swizzle: rows of 128 bytes (64 fp16), eight rows to a
// 1024-byte atom; start address and strides in units of 16 bytes, descriptor version 1, swizzle mode 2.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// The 4-byte word `w` of `count` scales from element e0 on, into shared memory.  `alpha` is 4-byte aligned; a run that starts at an odd
// element is copied with the element in front of it, and one that ends in the middle of a word is cut there.
__device__ __forceinline__ void copy_scales(uint32_t dst, const unsigned short *alpha, size_t e0, int count, int w) {
    const int odd = (int)(e0 & 1), bytes = min(4, 2 * (count + odd - 2 * w));
    if (bytes > 0) asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * w), "l"(alpha + e0 - odd + 2 * w), "r"(bytes) : "memory");
}

// A run of units inside one output tile.
struct Segment {
    int pi, n0, m0, rows, tile;   // problem, first column, first row, rows, output tile of the launch
    int k0, k1;                   // units of K
    int tile_unit;                // the tile's first unit in the launch's sequence
};

__device__ __forceinline__ int run_begin(const Params &P, int cta, int grid) { return (int)(((long long)cta * P.total_units) / grid); }
// the CTA whose run holds unit u
__device__ __forceinline__ int run_of(const Params &P, int u, int grid) { return (int)(((long long)(u + 1) * grid - 1) / P.total_units); }

__device__ __forceinline__ void cta_range(const Params &P, int &u, int &u_end) {
    if (P.whole_tiles) {
        int pi = 0;
        while (pi + 1 < P.count && (int)blockIdx.x >= P.p[pi + 1].tile_begin) ++pi;
        u = P.p[pi].unit_begin + ((int)blockIdx.x - P.p[pi].tile_begin) * P.p[pi].ku;
        u_end = u + P.p[pi].ku;
    } else {
        u = run_begin(P, blockIdx.x, gridDim.x);
        u_end = run_begin(P, blockIdx.x + 1, gridDim.x);
    }
}
// Next segment of the run [u, u_end); advances u.
__device__ __forceinline__ bool next_segment(const Params &P, int &u, int u_end, Segment &s) {
    if (u >= u_end) return false;
    int pi = 0;
    while (pi + 1 < P.count && u >= P.p[pi + 1].unit_begin) ++pi;
    const Problem &pr = P.p[pi];
    const int t = (u - pr.unit_begin) / pr.ku;
    s.pi = pi;
    s.tile = pr.tile_begin + t;
    s.tile_unit = pr.unit_begin + t * pr.ku;
    s.n0 = (t / P.mtiles) * TILE_N;
    s.m0 = (t % P.mtiles) * P.mt;
    s.rows = min(P.mt, P.M - s.m0);
    s.k0 = u - s.tile_unit;
    s.k1 = min(pr.ku, u_end - s.tile_unit);
    u = s.tile_unit + s.k1;
    return true;
}

template <int Q>
__device__ float scaled_sums(const Params &P, const Problem &pr, int m, int n) {
    const __half *x = reinterpret_cast<const __half *>(pr.x) + (size_t)m * pr.K;
    float acc = 0.f;
    for (int k = 0; k < pr.K / 32; k += pr.run)
        for (int b = 0; b < Q; ++b) {
            float sum = 0.f;
            for (int r = 0; r < pr.run; ++r) {
                const unsigned w = pr.bw[((size_t)(k + r) * Q + b) * pr.N + n];
                for (int t = 0; t < 32; ++t) {
                    const float v = __half2float(x[(k + r) * 32 + t]);
                    sum += (w >> t) & 1u ? v : -v;
                    if (P.layout != ROW && (t & 7) == 7) {   // a scale per eight features
                        acc += __half2float(__ushort_as_half(pr.alpha[((size_t)(k * 4 + t / 8) * Q + b) * pr.ngroups + n / pr.gs])) * sum;
                        sum = 0.f;
                    }
                }
            }
            if (P.layout == ROW) acc += __half2float(__ushort_as_half(pr.alpha[((size_t)(k / pr.gw) * Q + b) * pr.N + n])) * sum;
        }
    return acc;
}

// A scale that is infinite: the sum of (+-inf) * x over a group is NaN, while the table kernels, which multiply the signed sum of a group's
// activations, give an infinity (NaN only if a column's infinite scales disagree).  All elements of such a column are no finite numbers, so a
// CTA looks at one row's, and if one of them (for this or another reason) is none, goes over its tiles' scales and forms the elements of such
// columns again in the tables' way.
// `summed`: the tiles at the begin (bit 0) and end (bit 1) of the CTA's run that it was the last to arrive at.
template <int Q>
__device__ __noinline__ void infinite_columns(const Params &P, int summed) {
    if (P.layout == BLOCK_U16) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int u, u_end;
    cta_range(P, u, u_end);
    Segment sg;
    while (next_segment(P, u, u_end, sg)) {
        const Problem &pr = P.p[sg.pi];
        if (!(sg.k0 == 0 && sg.k1 == pr.ku) && !(summed & (sg.k0 == 0 ? 2 : 1))) continue;
        const int rows = (P.layout == ROW ? pr.ngroups : pr.K / 8) * Q, pitch = P.layout == ROW ? pr.N : pr.ngroups;
        for (int n = sg.n0 + warp; n < min(sg.n0 + TILE_N, pr.N); n += THREADS / 32) {
            const unsigned short *scale = pr.alpha + (P.layout == ROW ? n : n / pr.gs);
            bool any = false;
#pragma unroll 8
            for (int r = lane; r < rows; r += 32) any |= (scale[(size_t)r * pitch] & 0x7fffu) == 0x7c00u;
            if (!__any_sync(0xffffffffu, any)) continue;
            for (int m = sg.m0 + lane; m < sg.m0 + sg.rows; m += 32)   // no finite number, so bias and a finite y in place do not show
                reinterpret_cast<__half *>(pr.y)[(size_t)m * pr.N + n] = __float2half_rn(scaled_sums<Q>(P, pr, m, n));
        }
    }
}

template <int Q>
__global__ void __launch_bounds__(THREADS, 1) bcq_mma_kernel(const __grid_constant__ Params P) {
    using C = Cfg<Q>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last, s_summed, s_infinite;   // of the CTA's cut tiles: which it has summed; is an element no finite number?
    __shared__ __align__(8) uint64_t bars[2 * 16 + 3 * MAX_X_UNITS + 2 * 4 + 2];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int x_bytes = P.mpad * 128;               // 64 features of every row; a multiple of 1024 (mpad is one of 16)
    const uint32_t xs = smem0, ws = xs + P.x_units * 2 * x_bytes;
    const int w_stage = C::W_BYTES + P.s_bytes;     // a unit's planes, then its scales
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * 16, x_raw = w_empty + 8 * 16, x_full = x_raw + 8 * MAX_X_UNITS,
                   x_empty = x_full + 8 * MAX_X_UNITS, a_full = x_empty + 8 * MAX_X_UNITS, a_empty = a_full + 8 * 4, d_full = a_empty + 8 * 4, d_empty = d_full + 8;
    const int d_cols = (P.mpad + 31) & ~31;
    bool live = true;

    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        fence_before();
    }
    if (tid == 0) {
        s_summed = s_infinite = 0;
        for (int i = 0; i < P.w_stages; ++i) {
            // one arrival with the byte count of the TMA loads, and one per lane when its 4-byte copies have landed
            mbar_init(w_full + 8 * i, (P.use_tma ? 1 : 0) + (P.tma_scales ? 0 : 32));
            mbar_init(w_empty + 8 * i, OP_WARPS);
        }
        for (int i = 0; i < P.x_units; ++i) mbar_init(x_raw + 8 * i, 1), mbar_init(x_full + 8 * i, STG_WARPS), mbar_init(x_empty + 8 * i, 1);
        for (int i = 0; i < P.a_stages; ++i) mbar_init(a_full + 8 * i, OP_WARPS / 2), mbar_init(a_empty + 8 * i, 1);   // two words
        mbar_init(d_full, 1);
        mbar_init(d_empty, OP_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = s_tmem;
    int u, u_end;
    cta_range(P, u, u_end);
    Segment sg;

    if (warp == W_WARP) {
        // ------------------------------------------- planes and scales -------------------------------------------
        int st = 0;
        uint32_t ph = 1;   // a fresh barrier passes a wait for the phase before its first
        bool waited = false;
        while (next_segment(P, u, u_end, sg)) {
            const Problem &pr = P.p[sg.pi];
            const int cols = min(TILE_N, pr.N - sg.n0);
            const int gfirst = P.layout == ROW ? 0 : sg.n0 / pr.gs;   // BLOCK: the tile's groups
            const int bgroups = P.layout == ROW ? 0 : min((sg.n0 + TILE_N - 1) / pr.gs, pr.ngroups - 1) - gfirst + 1;
            for (int k = sg.k0; k < sg.k1 && live; ++k) {
                mbar_wait_behind(w_empty + 8 * st, ph, P.status, live, waited);
                live = __all_sync(0xffffffffu, live);   // the warp stops as one
                if (!live) break;
                const uint32_t dst = ws + st * w_stage, bar = w_full + 8 * st;
                const uint32_t sdst = dst + C::W_BYTES;
                const int g0 = pr.gshift >= 0 ? (k * UNIT_WORDS) >> pr.gshift : (k * UNIT_WORDS) / pr.gw;   // ROW: first group of the unit
                if (P.use_tma) {
                    if (elect_one()) {   // words past K / 32 and columns past N are zero-filled and counted
                        mbar_expect_tx(bar, C::W_BYTES + (P.tma_scales ? pr.s_tx : 0));
                        asm volatile(
                            "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                            "l"(reinterpret_cast<uint64_t>(&pr.tmap)), "r"(sg.n0), "r"(0), "r"(k * UNIT_WORDS), "r"(bar)
                            : "memory");
                        if (P.tma_scales)   // (group, plane) or (chunk, plane) rows; those past the last one are zero-filled and counted
                            asm volatile(
                                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(sdst),
                                "l"(reinterpret_cast<uint64_t>(&pr.smap)), "r"(P.layout == ROW ? sg.n0 : gfirst), "r"(P.layout == ROW ? g0 * Q : k * 16 * Q), "r"(bar)
                                : "memory");
                    }
                    __syncwarp();
                } else {
                    const int words = pr.K / 32;
                    const bool pairs = (pr.N & 1) == 0 && (reinterpret_cast<uintptr_t>(pr.bw) & 7) == 0;
#pragma unroll 2
                    for (int r = 0; r < UNIT_WORDS * Q; ++r) {
                        const int kk = k * UNIT_WORDS + r / Q;
                        const bool row_ok = kk < words;
                        const uint32_t *src = pr.bw + ((size_t)(row_ok ? kk : 0) * Q + r % Q) * pr.N;
                        if (pairs) {
#pragma unroll
                            for (int c = 0; c < TILE_N; c += 64) {
                                const int n = sg.n0 + c + 2 * lane;
                                const bool ok = row_ok && n < pr.N;
                                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + (uint32_t)(r * TILE_N + c + 2 * lane) * 4),
                                             "l"(src + (ok ? n : 0)), "r"(ok ? 8 : 0)
                                             : "memory");
                            }
                            continue;
                        }
#pragma unroll
                        for (int c = 0; c < TILE_N; c += 32) {
                            const int n = sg.n0 + c + lane;
                            const bool ok = row_ok && n < pr.N;
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + (uint32_t)(r * TILE_N + c + lane) * 4),
                                         "l"(src + (ok ? n : 0)), "r"(ok ? 4 : 0)
                                         : "memory");
                        }
                    }
                }
                if (!P.tma_scales) {
                    if (P.layout == ROW) {
                        const int ng = (pr.gshift >= 0 ? (k * UNIT_WORDS + UNIT_WORDS - 1) >> pr.gshift : (k * UNIT_WORDS + UNIT_WORDS - 1) / pr.gw) - g0 + 1;
#pragma unroll 1
                        for (int r = 0; r < ng * Q; ++r) {
                            const size_t e0 = (size_t)min(g0 * Q + r, pr.ngroups * Q - 1) * pr.N + sg.n0;
                            copy_scales(sdst + r * S_PITCH_ROW, pr.alpha, e0, cols, lane);
                            copy_scales(sdst + r * S_PITCH_ROW, pr.alpha, e0, cols, lane + 32);
                            if (lane == 0) copy_scales(sdst + r * S_PITCH_ROW, pr.alpha, e0, cols, 64);
                        }
                    } else {   // (chunk, plane) rows of the unit's groups
                        const int last = pr.K / 8 * Q - 1;
#pragma unroll
                        for (int i = 0; i < (16 * Q * 5 + 31) / 32; ++i) {
                            const int r = (lane + 32 * i) / 5, w = (lane + 32 * i) % 5;
                            if (r < 16 * Q) copy_scales(sdst + r * S_PITCH_BLOCK, pr.alpha, (size_t)min(k * 16 * Q + r, last) * pr.ngroups + gfirst, bgroups, w);
                        }
                    }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
                }
                if (++st == P.w_stages) st = 0, ph ^= 1u;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        land(w_full, P.w_stages, st, ph, P.status);
    } else if (warp == MMA_WARP) {
        // ------------------------------------------- tensor core -------------------------------------------
        // fp32 accumulators, fp16 operands, both K-major, N = mpad, M = 128
        const uint32_t idesc = (1u << 4) | ((uint32_t)(P.mpad >> 3) << 17) | ((TILE_N >> 4) << 24);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int xst = 0, ast = 0;
        uint32_t xph = 0, aph = 0, dph = 1;
        bool any = false;
        while (next_segment(P, u, u_end, sg)) {
            mbar_wait(d_empty, dph, P.status, live);
            dph ^= 1u;
            fence_after();
            for (int step = 2 * sg.k0; step < 2 * sg.k1; ++step) {
                if (!(step & 1)) mbar_wait(x_full + 8 * xst, xph, P.status, live);
                mbar_wait(a_full + 8 * ast, aph, P.status, live);
                fence_after();
                const uint64_t bdesc = smem_desc(xs + (2 * xst + (step & 1)) * x_bytes);
                const uint32_t a = tmem + d_cols + ast * C::A_COLS, more = step > 2 * sg.k0;
                if (elect_one()) {
#pragma unroll
                    for (int b = 0; b < Q; ++b)
#pragma unroll
                        for (int k = 0; k < 4; ++k) mma_f16(tmem, a + b * 32 + k * 8, bdesc + 2 * k, idesc, b + k ? 1u : more);
                    mma_commit(a_empty + 8 * ast);
                    if (step & 1) mma_commit(x_empty + 8 * xst);
                    if (step == 2 * sg.k1 - 1) mma_commit(d_full);
                }
                __syncwarp();
                if (++ast == P.a_stages) ast = 0, aph ^= 1u;
                if ((step & 1) && ++xst == P.x_units) xst = 0, xph ^= 1u;
            }
            any = true;
        }
        bool once = true;
        if (any) mbar_wait(d_full, dph, P.status, once);   // the last segment's commit
    } else if (warp == X_WARP) {
        // ------------------------------------------- activations: fetch -------------------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int xst = 0;
        uint32_t xph = 1;
        while (next_segment(P, u, u_end, sg)) {
            const Problem &pr = P.p[sg.pi];
            for (int k = sg.k0; k < sg.k1 && live; ++k) {
                mbar_wait(x_empty + 8 * xst, xph, P.status, live);
                live = __all_sync(0xffffffffu, live);   // the warp stops as one
                if (!live) break;
                if (elect_one()) {   // rows past M and features past K are zero-filled and counted
                    const uint32_t bar = x_raw + 8 * xst, dst = xs + 2 * xst * x_bytes;
                    mbar_expect_tx(bar, 2 * x_bytes);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst + h * x_bytes),
                            "l"(reinterpret_cast<uint64_t>(&pr.xmap)), "r"(k * 128 + h * 64), "r"(sg.m0), "r"(bar)
                            : "memory");
                }
                __syncwarp();
                if (++xst == P.x_units) xst = 0, xph ^= 1u;
            }
        }
        land(x_raw, P.x_units, xst, xph, P.status);
    } else if (warp >= OP_WARPS) {
        // ------------------------------------------- activations: reorder -------------------------------------------
        // A warp takes one word (32 features, 64 bytes) of every row; a lane's row is read and written in place, features t and t + 16
        // side by side.  Eight neighbouring rows lie in eight different bank groups (the swizzle), so both sides are conflict-free.
        const int word = warp - OP_WARPS;
        const uint32_t c0 = (uint32_t)(word & 1) * 4, sw = (uint32_t)(lane & 7);   // 32 rows on, the swizzle is the same
        const uint32_t o0 = ((c0 + 0) ^ sw) << 4, o1 = ((c0 + 1) ^ sw) << 4, o2 = ((c0 + 2) ^ sw) << 4, o3 = ((c0 + 3) ^ sw) << 4;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int xst = 0;
        uint32_t xph = 0;
        while (next_segment(P, u, u_end, sg)) {
            for (int k = sg.k0; k < sg.k1; ++k) {
                mbar_wait(x_raw + 8 * xst, xph, P.status, live);
                const uint32_t x0 = xs + (2 * xst + (word >> 1)) * x_bytes + lane * 128;
#pragma unroll 2
                for (int row = lane; row < sg.rows; row += 32) {
                    const uint32_t rb = x0 + (row - lane) * 128;
                    const uint4 l0 = lds128(rb + o0), l1 = lds128(rb + o1), h0 = lds128(rb + o2), h1 = lds128(rb + o3);   // features 0-7, 8-15, 16-23, 24-31
                    sts128(rb + o0, prmt(l0.x, h0.x, 0x5410), prmt(l0.x, h0.x, 0x7632), prmt(l0.y, h0.y, 0x5410), prmt(l0.y, h0.y, 0x7632));
                    sts128(rb + o1, prmt(l0.z, h0.z, 0x5410), prmt(l0.z, h0.z, 0x7632), prmt(l0.w, h0.w, 0x5410), prmt(l0.w, h0.w, 0x7632));
                    sts128(rb + o2, prmt(l1.x, h1.x, 0x5410), prmt(l1.x, h1.x, 0x7632), prmt(l1.y, h1.y, 0x5410), prmt(l1.y, h1.y, 0x7632));
                    sts128(rb + o3, prmt(l1.z, h1.z, 0x5410), prmt(l1.z, h1.z, 0x7632), prmt(l1.w, h1.w, 0x5410), prmt(l1.w, h1.w, 0x7632));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(x_full + 8 * xst);
                if (++xst == P.x_units) xst = 0, xph ^= 1u;
            }
        }
    } else {
        // ------------------------------------------- operands and results -------------------------------------------
        const int quarter = warp & 3, wi = warp >> 2;              // this warp's lanes and its word of every unit
        const int col = quarter * 32 + lane;                       // output column of the tile = lane of tensor memory
        const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16);
        int wst = 0, ast = wi >> 1;                                // words 0, 1: the first 64 features of a unit, 2, 3: the second
        uint32_t wph = 0, aph = 1, dph = 0;
        bool waited = false, finite = true;
        while (next_segment(P, u, u_end, sg)) {
            const Problem &pr = P.p[sg.pi];
            const int gw = pr.gw, gshift = pr.gshift;
            // BLOCK: the column's group within the tile (columns past N take the last one: their results are not stored)
            const int gfirst = P.layout == ROW ? 0 : sg.n0 / pr.gs;
            const int gi = P.layout == ROW ? 0 : min(sg.n0 + col, pr.N - 1) / pr.gs - gfirst;
            for (int k = sg.k0; k < sg.k1; ++k) {
                mbar_wait(w_full + 8 * wst, wph, P.status, live);
                const uint32_t wbase = ws + wst * w_stage, sbase = wbase + C::W_BYTES;
                uint32_t w[Q], sa[Q], sb[Q];
#pragma unroll
                for (int b = 0; b < Q; ++b) w[b] = lds32(wbase + (uint32_t)((wi * Q + b) * TILE_N + col) * 4);
                if (P.layout == ROW) {
                    const int kk = k * UNIT_WORDS, g0 = gshift >= 0 ? kk >> gshift : kk / gw;
                    const int j = (gshift >= 0 ? (kk + wi) >> gshift : (kk + wi) / gw) - g0;
                    // a row of scales that starts at an odd element lies one further on
#pragma unroll
                    for (int b = 0; b < Q; ++b) {
                        const uint32_t a = lds16(sbase + (uint32_t)((j * Q + b) * P.s_pitch + (col + (min((g0 + j) * Q + b, pr.ngroups * Q - 1) & pr.N & 1)) * 2));
                        sa[b] = sb[b] = prmt(a, a, 0x1010) ^ 0x80008000u;
                    }
                } else {
                    // chunks 0..3 of the word: features 0-7 pair with 16-23 (chunks 0, 2), 8-15 with 24-31 (chunks 1, 3)
#pragma unroll
                    for (int b = 0; b < Q; ++b) {
                        uint32_t a[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int c = 4 * wi + j, e = min((k * 16 + c) * Q + b, pr.K / 8 * Q - 1);   // row of the scales, as it was copied
                            a[j] = lds16(sbase + (uint32_t)((c * Q + b) * P.s_pitch + (gi + (((e & pr.ngroups) ^ gfirst) & 1)) * 2));
                            if (P.layout == BLOCK_U16)   // 2^a + 2^b + 2^c with exponents 0..7: at most 384, exact in fp16
                                a[j] = __half_as_ushort(__int2half_rn((1 << (a[j] & 7)) + (1 << ((a[j] >> 3) & 7)) + (1 << ((a[j] >> 6) & 7))));
                        }
                        sa[b] = prmt(a[0], a[2], 0x5410) ^ 0x80008000u;
                        sb[b] = prmt(a[1], a[3], 0x5410) ^ 0x80008000u;
                    }
                }
                mbar_wait_behind(a_empty + 8 * ast, aph, P.status, live, waited);
                fence_after();
                const uint32_t dst = tlane + d_cols + ast * C::A_COLS + (wi & 1) * 16;
#pragma unroll
                for (int b = 0; b < Q; ++b) {
                    uint32_t r[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) r[i] = ((w[b] << (15 - i)) & 0x80008000u) ^ (i < 8 ? sa[b] : sb[b]);
                    tmem_store16(dst + b * 32, r);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(w_empty + 8 * wst);   // the ring's words and scales are in registers
                    mbar_arrive(a_full + 8 * ast);
                }
                ast += 2;   // the other two words take the stage in between
                if (ast >= P.a_stages) ast -= P.a_stages, aph ^= 1u;
                if (++wst == P.w_stages) wst = 0, wph ^= 1u;
            }
            // ---- the segment's accumulators
            if (!waited) {   // results and scratch may still be in use by the kernel in front
                asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            }
            mbar_wait(d_full, dph, P.status, live);
            dph ^= 1u;
            fence_after();
            const bool whole = sg.k0 == 0 && sg.k1 == pr.ku;
            const int n = sg.n0 + col;
            const float bias = (pr.bias && n < pr.N) ? __half2float(__ushort_as_half(pr.bias[n])) : 0.f;
            const int mh = P.mpad / 4, m_lo = wi * mh, m_hi = min(m_lo + mh, sg.rows);   // a quarter of the rows per warp of these lanes
            __half *ycol = reinterpret_cast<__half *>(pr.y) + (size_t)sg.m0 * pr.N + n;
            // a CTA's first segment has its slot 2 c, one that follows (the begin of a tile shared with later CTAs) 2 c + 1
            const int tile_first = whole ? 0 : run_of(P, sg.tile_unit, gridDim.x);
            const int first_slot = whole ? 0 : 2 * tile_first + (run_begin(P, tile_first, gridDim.x) < sg.tile_unit ? 1 : 0);
            float *part = whole ? nullptr : P.partials + (size_t)((int)blockIdx.x == tile_first ? first_slot : 2 * (int)blockIdx.x) * P.mt * TILE_N + col;
            for (int m = m_lo; m < m_hi; m += 4) {
                float v[4];
                tmem_load4(tlane + m, v);
                if (m == 0 && whole && n < pr.N) finite = finite && fabsf(v[0]) <= FLT_MAX;   // one row shows it
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (m + i < m_hi) {
                        if (!whole) __stcg(part + (size_t)(m + i) * TILE_N, v[i]);
                        else if (n < pr.N) {
                            float r = v[i] + bias;
                            __half *yp = ycol + (size_t)(m + i) * pr.N;
                            if (P.accumulate) r += __half2float(*yp);
                            *yp = __float2half_rn(r);
                        }
                    }
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty);
            if (!whole) {
                // one acquire-release add per CTA behind a barrier of the operand warps (release: covers the other threads'
                // partial sums; acquire: those of the CTAs that arrived earlier, behind the second barrier)
                asm volatile("bar.sync 1, %0;" ::"n"(OP_WARPS * 32) : "memory");
                const int tile_last = run_of(P, sg.tile_unit + pr.ku - 1, gridDim.x), shares = tile_last - tile_first + 1;
                if (tid == 0) {
                    unsigned old;
                    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(P.counters + sg.tile) : "memory");
                    s_last = old == (unsigned)(shares - 1);
                    if (s_last) P.counters[sg.tile] = 0u;   // ready for the next launch
                }
                asm volatile("bar.sync 1, %0;" ::"n"(OP_WARPS * 32) : "memory");
                if (s_last) {
                    // a warp takes every sixteenth row, a lane four columns; the loads of four shares and two rows are in flight together
                    const int nc = sg.n0 + 4 * lane;
                    const size_t row4 = TILE_N / 4, slot4 = (size_t)P.mt * row4;
                    const float4 *p0 = reinterpret_cast<const float4 *>(P.partials) + (size_t)first_slot * slot4 + lane;
                    const float4 *p1 = reinterpret_cast<const float4 *>(P.partials) + (size_t)(2 * tile_first) * slot4 + lane;
                    for (int m = warp; m < sg.rows; m += 2 * OP_WARPS) {
                        float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
                        for (int c0 = 0; c0 < shares; c0 += 4) {
                            float4 t[4][2];
#pragma unroll
                            for (int c = 0; c < 4; ++c)
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    const int mm = m + i * OP_WARPS;
                                    const float4 *src = c0 + c == 0 ? p0 : p1 + (size_t)(2 * (c0 + c)) * slot4;
                                    t[c][i] = c0 + c < shares && mm < sg.rows ? __ldcg(src + (size_t)mm * row4) : make_float4(0.f, 0.f, 0.f, 0.f);
                                }
#pragma unroll
                            for (int c = 0; c < 4; ++c)
#pragma unroll
                                for (int i = 0; i < 2; ++i) v[i].x += t[c][i].x, v[i].y += t[c][i].y, v[i].z += t[c][i].z, v[i].w += t[c][i].w;
                        }
                        if (m == 0) {   // columns past N have whatever scales the ring held
                            const float r0[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) finite = finite && (nc + e >= pr.N || fabsf(r0[e]) <= FLT_MAX);
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int mm = m + i * OP_WARPS;
                            if (mm >= sg.rows) continue;
                            const float r4[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
                            __half *yp = reinterpret_cast<__half *>(pr.y) + (size_t)(sg.m0 + mm) * pr.N + nc;
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (nc + e < pr.N) {
                                    float r = r4[e] + (pr.bias ? __half2float(__ushort_as_half(pr.bias[nc + e])) : 0.f);
                                    if (P.accumulate) r += __half2float(yp[e]);
                                    yp[e] = __float2half_rn(r);
                                }
                        }
                    }
                    if (tid == 0) s_summed |= sg.k0 == 0 ? 2 : 1;
                }
            }
        }
        if (!finite) s_infinite = 1;
        fence_before();
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
    if (s_infinite) infinite_columns<Q>(P, s_summed);
}

template <int Q>
cudaError_t launch_q(const Built &b, const Params &P, cudaStream_t stream) {
    static std::atomic<bool> configured[64];
    const cudaError_t e = sal_allow_shared_memory(bcq_mma_kernel<Q>, configured);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)b.ctas);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)b.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (b.flags & SAL_PDL) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, bcq_mma_kernel<Q>, P);
}

// CTAs per tile where all CTAs have the same number of them (0: runs of units are cut anywhere).
// Where whole numbers of shares per tile fill most of the SMs, runs are cut at tile borders (run_begin does so by itself): every
// CTA has one segment instead of two, and a tile fewer shares to sum, which for many rows costs as much as the product.  At least
// four units per share, or eight shares.  us with 148 CTAs / with whole shares, for 64 and 256 rows: 4096 x 4096, 3 planes 20.3 / 17.3
// and 43.3 / 36.2 (128 CTAs), 4096 x 1024 15.3 / 13.5 and 45.4 / 32.3 (64), 2048 x 2048 14.8 / 11.2 and 37.7 / 29.2 (128), 8192 x 8192,
// 2 planes 32.7 / 32.0 and 70.2 / 73.1 (128); with 86 of 148 (4096 x 11008) 36.7 / 45.8, hence the line at 86 %.
// Not where rows are copied by plain instructions: a unit takes three times as long there (2080 x 1378, 3 rows: 18.4 / 20.5).
int whole_shares(int tiles, int ku, int sms) {
    if (tiles > sms) return 0;
    const int most = ku / 4 > 8 ? ku / 4 : 8;
    int shares = sms / tiles;
    const bool enough = shares > most;
    if (shares > most) shares = most;
    if (shares > ku) shares = ku;
    return enough || shares * tiles * 100 >= 86 * sms ? shares : 0;
}

// Can the scales be fetched by TMA?  Rows of a multiple of 16 bytes; ROW: groups that make a unit or that a unit is made of, BLOCK: eight
// groups per tile.
bool scales_by_tma(const sal_problem &sp, AlphaLayout layout) {
    const int gw = layout == ROW ? sp.K / sp.num_groups / 32 : 0;
    return (layout == ROW ? sp.N : sp.num_groups) % 8 == 0 && (reinterpret_cast<uintptr_t>(sp.alpha) & 15) == 0 &&
           (layout == ROW ? gw % UNIT_WORDS == 0 || UNIT_WORDS % gw == 0 : sp.N / sp.num_groups == 16);
}
bool planes_by_tma(const sal_problem &sp) { return sp.N % 4 == 0 && (reinterpret_cast<uintptr_t>(sp.bw) & 15) == 0; }

}  // namespace

double block_us(const sal_problem &sp, AlphaLayout layout, int sms) {
    if (sms > MAX_CTAS) sms = MAX_CTAS;
    const int ku = (sp.K + 127) / 128, tiles = (sp.N + TILE_N - 1) / TILE_N * ((sp.M + MAX_MT - 1) / MAX_MT), i = sp.q - 1;
    const bool tma = planes_by_tma(sp) && scales_by_tma(sp, layout);
    const int shares = tma ? whole_shares(tiles, ku, sms) : 0, ctas = shares ? shares * tiles : (sms < tiles * ku ? sms : tiles * ku);
    static const double by_tma[4] = {0.45, 0.72, 1.03, 1.28}, by_copies[4] = {0.7, 1.0, 1.38, 1.56};
    double unit = tma ? by_tma[i] * (shares ? 1.0 : tiles > sms ? 1.06 : 1.2) : by_copies[i];
    if (layout == BLOCK_U16) unit *= tma ? 1.3 : 1.1;   // decoding the exponents
    return (tma ? 8.2 : 11.0) + unit * ((tiles * ku + ctas - 1) / ctas) + 0.06 * shares + (sp.M > 16 ? 0.06 * (sp.M - 16) : 0.0);
}

bool eligible(const void *bw, const void *alpha, const void *x, int M, int K, int N, int q, int num_groups, AlphaLayout layout) {
    if (M < 1 || M > MAX_ROWS || q < 1 || q > 4 || K < 32 || K % 32 || N < 1 || num_groups < 1) return false;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(bw) & 3) || (reinterpret_cast<uintptr_t>(alpha) & 3)) return false;
    if (layout == ROW) return K % num_groups == 0 && (K / num_groups) % 32 == 0;
    return N % num_groups == 0 && (N / num_groups) % 16 == 0;   // at most nine groups meet a tile of 128 columns
}

size_t full_scratch_bytes(int M) {
    const int mt = M < 1 ? 1 : (M > MAX_MT ? MAX_MT : M);
    return WS_PARTIALS + (size_t)MAX_CTAS * 2 * TILE_N * mt * sizeof(float);
}

int build(const sal_problem *problems, int count, AlphaLayout layout, unsigned flags, size_t ws_bytes, int sms, Built *out, bool encode) {
    Built &b = *out;
    b = Built{};
    Params &P = b.P;
    b.q = problems[0].q;
    b.flags = flags;
    b.count = P.count = count;
    P.M = problems[0].M;
    P.mtiles = (P.M + MAX_MT - 1) / MAX_MT;
    P.mt = (P.M + P.mtiles - 1) / P.mtiles;
    if (P.mtiles > 1) P.mt = (P.mt + 15) / 16 * 16;
    P.mpad = (P.mt + 15) / 16 * 16;
    P.accumulate = (flags & SAL_ACCUMULATE) ? 1 : 0;
    P.layout = layout;
    bool tma = true;
    for (int i = 0; i < count; ++i) tma = tma && planes_by_tma(problems[i]);
    P.use_tma = tma;
    bool tma_scales = tma;
    for (int i = 0; i < count; ++i) tma_scales = tma_scales && scales_by_tma(problems[i], layout);
    P.tma_scales = tma_scales;
    P.s_pitch = layout == ROW ? (tma_scales ? S_PITCH_ROW_TMA : S_PITCH_ROW) : (tma_scales ? S_PITCH_BLOCK_TMA : S_PITCH_BLOCK);
    int units = 0, tiles = 0;
    long long total = 0;
    for (int i = 0; i < count; ++i) {
        const sal_problem &sp = problems[i];
        Problem &p = P.p[i];
        p.bw = reinterpret_cast<const unsigned *>(sp.bw);
        p.alpha = reinterpret_cast<const unsigned short *>(sp.alpha);
        p.bias = reinterpret_cast<const unsigned short *>(sp.bias);
        p.x = reinterpret_cast<const unsigned short *>(sp.x);
        p.y = reinterpret_cast<unsigned short *>(sp.y);
        p.K = sp.K, p.N = sp.N;
        p.ku = (sp.K + 127) / 128;
        p.unit_begin = units;
        p.tile_begin = tiles;
        p.ntiles = (sp.N + TILE_N - 1) / TILE_N * P.mtiles;
        total += (long long)p.ntiles * p.ku;
        if (total > 0x3fffffff) return SAL_E_UNSUPPORTED;
        units += p.ntiles * p.ku;
        tiles += p.ntiles;
        p.ngroups = sp.num_groups;
        p.gw = 1, p.gshift = 0, p.gs = 1, p.run = 1;
        if (layout == ROW) {
            p.gw = sp.K / sp.num_groups / 32;
            p.run = sp.K % 256 == 0 && sp.N % 8 == 0 && p.gw % 4 == 0 ? 4 : 1;   // the tiled table kernel's shapes, else the generic one's
            // groups that a unit of four words can meet: one if they are whole units
            const int ng = p.gw % UNIT_WORDS == 0 ? 1 : (UNIT_WORDS - 2) / p.gw + 2;
            if (ng * b.q * P.s_pitch > P.s_bytes) P.s_bytes = ng * b.q * P.s_pitch;
            p.gshift = -1;
            for (int s = 0; s < 31; ++s)
                if (p.gw == 1 << s) p.gshift = s;
        } else {
            p.gs = sp.N / sp.num_groups;
            P.s_bytes = 16 * b.q * P.s_pitch;
        }
        if (tma_scales) {
            const int rows = layout == ROW ? (p.gw < UNIT_WORDS ? UNIT_WORDS / p.gw : 1) * b.q : 16 * b.q;
            p.s_tx = rows * P.s_pitch;
            const int rc = !encode ? SAL_OK : sal_encode_rows(&p.smap, sp.alpha, layout == ROW ? sp.N : sp.num_groups, layout == ROW ? sp.num_groups * b.q : sp.K / 8 * b.q,
                                           P.s_pitch / 2, rows, 0);
            if (rc != SAL_OK) return rc;
        }
        if (tma && encode) {
            const int rc = sal_encode_planes(&p.tmap, sp.bw, sp.K, sp.N, sp.q, TILE_N, sp.q, UNIT_WORDS);
            if (rc != SAL_OK) return rc;
        }
        if (!sp.x_mul && encode) {
            const int rc = sal_encode_rows(&p.xmap, sp.x, sp.K, P.M, 64, P.mpad, 1);
            if (rc != SAL_OK) return rc;
        }
        b.gate[i] = sp.x_mul ? sp.x : nullptr;
        b.up[i] = sp.x_mul;
        if (sp.x_mul) b.act_bytes += ((size_t)P.M * sp.K * 2 + 255) & ~(size_t)255;
    }
    P.total_units = units;
    // CTAs: one per SM, as far as there are units and the scratch buffer holds their partial sums (two slots of mt x 128
    // floats each; the documented size holds them all, so that the split and with it the last bits follow from the shape alone);
    // without scratch, or with so little that it would leave SMs idle, one per output tile
    const size_t slot_bytes = (size_t)2 * P.mt * TILE_N * sizeof(float);
    if (sms > MAX_CTAS) sms = MAX_CTAS;
    bool same_k = true;
    for (int i = 1; i < count; ++i) same_k = same_k && P.p[i].ku == P.p[0].ku;
    const int shares = same_k && tma_scales ? whole_shares(tiles, P.p[0].ku, sms) : 0;
    long long ctas = shares ? (long long)shares * tiles : (sms < units ? sms : units);
    if (ws_bytes < WS_PARTIALS + b.act_bytes) {
        if (b.act_bytes) return SAL_E_WORKSPACE;
        ctas = 0;
    } else {
        const long long fit = (long long)((ws_bytes - WS_PARTIALS - b.act_bytes) / slot_bytes);
        if (ctas > fit) ctas = fit;
    }
    if (tiles > MAX_COUNTERS) ctas = 0;
    P.whole_tiles = ctas < (tiles < sms ? tiles : sms);   // of what the scratch buffer leaves
    b.ctas = P.whole_tiles ? tiles : (int)ctas;
    b.ws_need = P.whole_tiles ? 0 : WS_PARTIALS + (size_t)b.ctas * slot_bytes;
    const int d_cols = (P.mpad + 31) & ~31, a_cols = 32 * b.q;
    P.s_bytes = (P.s_bytes + 127) & ~127;   // a stage begins where TMA may write
    const int w_bytes = UNIT_WORDS * b.q * TILE_N * 4 + P.s_bytes;
    P.a_stages = (TMEM_COLS - d_cols) / a_cols;
    if (P.a_stages > 4) P.a_stages = 4;
    P.x_units = P.mpad <= 32 ? 4 : P.mpad <= 64 ? 3 : 2;
    const int fixed = 1024 + P.x_units * P.mpad * 256;
    P.w_stages = (224 * 1024 - fixed) / w_bytes;
    if (P.w_stages > 12) P.w_stages = 12;
    b.smem = fixed + P.w_stages * w_bytes;
    return SAL_OK;
}

size_t scratch_bytes(const Built &b) {
    if (b.ws_need + b.act_bytes == 0) return 0;
    return (b.ws_need ? b.ws_need : WS_PARTIALS) + b.act_bytes;
}

int launch(const Built &b, void *workspace, size_t ws_bytes, cudaStream_t stream) {
    const size_t need = scratch_bytes(b);
    if (need > 0 && (!workspace || ws_bytes < need)) return SAL_E_WORKSPACE;
    std::shared_mutex &order = sal_scratch_order(workspace);
    std::unique_lock<std::shared_mutex> alone(order, std::defer_lock);
    std::shared_lock<std::shared_mutex> shared(order, std::defer_lock);
    if (b.act_bytes) alone.lock();
    else shared.lock();
    Params P = b.P;
    char *base = reinterpret_cast<char *>(workspace);
    P.status = reinterpret_cast<int *>(workspace);
    if (!P.whole_tiles) {
        P.counters = reinterpret_cast<unsigned *>(base + WS_HEADER);
        P.partials = reinterpret_cast<float *>(base + WS_PARTIALS);
    }
    size_t off = b.ws_need ? b.ws_need : WS_PARTIALS;
    for (int i = 0; i < b.count; ++i) {
        if (!b.up[i]) continue;
        // silu(x) * x_mul, formed once in front of the product (every column tile reads it)
        const int rc = sal_silu_mul_f16(b.gate[i], b.up[i], base + off, P.M * P.p[i].K, stream);
        if (rc != SAL_OK) return rc;
        P.p[i].x = reinterpret_cast<const unsigned short *>(base + off);
        const int erc = sal_encode_rows(&P.p[i].xmap, base + off, P.p[i].K, P.M, 64, P.mpad, 1);
        if (erc != SAL_OK) return erc;
        off += ((size_t)P.M * P.p[i].K * 2 + 255) & ~(size_t)255;
    }
    cudaError_t e;
    switch (b.q) {
        case 1: e = launch_q<1>(b, P, stream); break;
        case 2: e = launch_q<2>(b, P, stream); break;
        case 3: e = launch_q<3>(b, P, stream); break;
        default: e = launch_q<4>(b, P, stream); break;
    }
    return e == cudaSuccess ? SAL_OK : SAL_E_LAUNCH;
}

}  // namespace sal_mma
