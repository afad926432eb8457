// Correlation on the tensor cores (tcgen05) in BF16 or FP16 with FP32
// accumulation: the reduced-precision form of custom::Correlation (the
// legacy = 0 layout of correlation.cc:45-143 / correlation_cuda.cu:97-175).
//
// For one row y of the output and a segment of kTcM = 128 pixels starting at
// x0, and one displacement row dy, the 2 md + 1 correlations of every pixel
// are a band of the product
//     D_dy[m][n] = sum_c f1[c][y][x0 + m] * f2[c][y + dy][x0 - md + n],
// m < 128, n < kTcN = 144 (>= 128 + 2 md): pixel m's value for displacement
// dx is D_dy[m][m + dx + md].  Each D_dy is one M = 128, N = 144 MMA chain
// over K = channels (padded to a multiple of 16 with zeros), accumulated in
// Tensor Memory; both operands come from shared memory, staged by one 5-D TMA
// load each from the features in a "chunked" layout
//     [n][y][c / cw][x][c % cw]  (16-bit elements, channels padded to Cp),
// cw = 64, 32 or 16, the largest that divides Cp, which the TMA box {cw,
// pixels, Cp / cw} with the swizzle of 2 cw bytes turns directly into the
// K-major operand layout of that swizzle: one chunk plane of pixels x 2 cw
// bytes (one K step is 32 bytes along a row).  The TMA works through a box by
// its rows: a 144-pixel row of 64 channels is 144 rows of 128 bytes, not 576 of 32.
// A work item is R adjacent output rows: each of the R + 2 md f2 rows it needs
// is loaded once and multiplied with up to R f1 rows.
// Rows y + dy and columns outside the map are zero-filled by the TMA, which
// is the operator's zero outside.
// The epilogue reads each warp's 32 lanes x 48 columns of D_dy out of Tensor
// Memory, stages them in shared memory and picks the diagonal band.
//
// Per-level scaling: each operand is multiplied by a power of two 2^k chosen
// from its largest magnitude (|f| 2^k in [2^13, 2^14)) before the 16-bit
// conversion, which keeps FP16 clear of overflow and of its subnormal range;
// the sums are multiplied by 2^-(k1 + k2) afterwards (exact).
#include "vsc_device.h"
#include "vsc_internal.h"
#include "vsc_math.cuh"
#include "vsc_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <functional>

namespace vsc {
namespace {

constexpr int kTcM = 128;        // pixels per tile (MMA M, TMEM lanes)
constexpr int kTcN = 144;        // f2 window per displacement row (MMA N)
constexpr int kTcCols = 48;      // TMEM columns one warp reads per row: 32 + 2 md
constexpr int kTcPitch = 52;     // staging row pitch (floats): 53 * lane spreads the diagonal over all banks
// warps: 0 TMA producer, 1 MMA issuer + Tensor Memory owner, then 1..3
// epilogue groups of four warps (one per 32 TMEM lanes); group g drains the
// accumulators of rows u with u % groups == g
constexpr int kMaxEpiGroups = 3;
constexpr int kMaxStagesA = 2, kMaxStagesB = 4, kStagesD = 3;
constexpr uint32_t kTmemCols = 512;    // three accumulators
constexpr uint32_t kDStride = 160;     // TMEM columns between accumulators (>= kTcN, multiple of 32)
constexpr int kTcWaitSpins = 1 << 22;  // bounded mbarrier waits (about a second)
constexpr int kTcGroupStageBytes = 4 * 32 * kTcPitch * 4;  // one epilogue group's staging
constexpr int kTcBarBytes = 256;
constexpr int kTcSmemLimit = 232448;   // dynamic shared memory per CTA on sm_103
// at least this much dynamic shared memory, so that one CTA (and one
// 512-column Tensor Memory allocation) occupies an SM
constexpr int kTcMinSmem = 120 * 1024;
static_assert(kTcN >= kTcM + 2 * kTcMaxMd && kTcN % 16 == 0 && kTcN <= 256, "MMA N");
static_assert(32 * 3 + kTcCols <= kTcN, "epilogue columns inside the accumulator");
static_assert(kTcCols >= 32 + 2 * kTcMaxMd, "epilogue columns cover the band");
static_assert((kStagesD - 1) * kDStride + kTcN <= kTmemCols, "accumulators inside the allocation");

__host__ __device__ constexpr uint32_t align1k(uint32_t v) { return (v + 1023u) & ~1023u; }

struct TcPlan {
    int rows, stages_a, stages_b, groups;  // output rows of an item; sets of f1 rows, f2 rows, epilogue groups
    uint32_t smem;
};

__host__ uint32_t tc_smem_need(int cp, int rows, int sa, int sb, int g)
{
    return 1024 + sa * rows * align1k(kTcM * cp * 2) + sb * align1k(kTcN * cp * 2) + g * kTcGroupStageBytes +
           kTcBarBytes;
}

// Buffers that fit in shared memory for Cp channels: three epilogue groups,
// two sets of f1 rows and four f2 rows when they fit; f2 rows, then f1 sets,
// then epilogue groups are given up in that order (208 channels: 1, 2, 2).
__host__ TcPlan tc_plan(int cp, int rows)
{
    TcPlan p{rows, kMaxStagesA, kMaxStagesB, kMaxEpiGroups, 0};
    while (tc_smem_need(cp, rows, p.stages_a, p.stages_b, p.groups) > static_cast<uint32_t>(kTcSmemLimit)) {
        if (p.stages_b > 2)
            --p.stages_b;
        else if (p.stages_a > 1)
            --p.stages_a;
        else if (p.groups > 1)
            --p.groups;
        else
            break;
    }
    p.smem = std::max<uint32_t>(tc_smem_need(cp, rows, p.stages_a, p.stages_b, p.groups), kTcMinSmem);
    return p;
}

// Base + stride, not arrays of pointers: indexed by run-time stage numbers,
// arrays would live in local memory and every access would wait on it.
struct TcShared {
    unsigned char* a;  // f1 row r of set i at a + (i * rows + r) * a_stride
    unsigned char* b;
    uint32_t a_stride, b_stride;
    float* stage;
    uint64_t *full_a, *empty_a, *full_b, *empty_b, *full_d, *empty_d;
    uint32_t* tmem_slot;
    volatile int* abort;
};

// Bounded wait that also gives up when another role has aborted; a wait that
// runs out raises the abort for everyone.  The polling loop is a function of its
// own: inlined at every wait it made the roles' loops miss the instruction cache.
__device__ __noinline__ bool tc_poll(uint64_t* bar, uint32_t parity, volatile int* abort)
{
#pragma unroll 1
    for (int i = 0; i < kTcWaitSpins; ++i) {
        if (ptx::mbar_try_wait(bar, parity))
            return true;
        if ((i & 63) == 63 && *abort)
            return false;
        if (i > 256)  // hand-offs are short: poll first, then back off
            __nanosleep(64);
    }
    *abort = 1;
    return false;
}

__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    return ptx::mbar_try_wait(bar, parity) || tc_poll(bar, parity, abort);
}

// One work item: `rows` output rows from y0 (fewer at the map's end) of a
// 128-pixel segment, displacement rows d0 .. d1 - 1.
struct TcItem {
    int prob, n, seg, y0, ny, d0, d1;
};

// A ring's next slot and its phase, stepped rather than divided out of a count:
// a division by a run-time number is some 100 cycles of the one thread that
// issues everything.
struct TcRing {
    int i = 0, n;
    uint32_t phase = 0;
    __device__ explicit TcRing(int slots) : n(slots) {}
    __device__ void next()
    {
        if (++i == n) {
            i = 0;
            phase ^= 1;
        }
    }
};

// Persistent, warp-specialised: every CTA walks items blockIdx.x, +gridDim.x,
// ...  An item's f2 rows stream in order of y; f2 row b meets output row y0 + r
// as its displacement row d = b - y0 - r + md.  Rings: sets of f1 rows (producer
// -> MMA, freed by the MMA's commit after the item's last product), f2 rows
// (freed by the commit of the last MMA that read them), accumulators in Tensor
// Memory (MMA -> epilogue, freed by the four epilogue warps as soon as their
// columns are in registers, before the shared-memory and global part of the
// epilogue).
// What bounds it is the one thread that issues the MMAs: a product's three
// waits, its MMAs (four for 64 channels, about 75 cycles each) and commits take it
// about 1000 cycles, the epilogue's three groups about 300 a product, the loads
// less.  So the issuing branches are elect.sync ones (a branch on the lane
// number made every MMA cost 150 cycles), rings are stepped, and the polling is
// out of line: 2 x 64 x 136 x 240 36 us before these three, 19 with them.
__global__ void __launch_bounds__((2 + 4 * kMaxEpiGroups) * 32, 1)
    corr_tc_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
        float* __restrict__ out, const __grid_constant__ CUtensorMap mA2, const __grid_constant__ CUtensorMap mB2,
        float* __restrict__ out2, int nprob, const float* __restrict__ scales, int N, int H, int W, int Cp, int cw,
        int md, uint32_t idesc, int rows, int stages_a, int stages_b, int groups, int ndyg,
        int* __restrict__ timeout_flag)
{
    extern __shared__ unsigned char smem_raw[];
    const uint32_t bytesA = kTcM * Cp * 2;
    const uint32_t bytesB = kTcN * Cp * 2;
    TcShared sh;
    {
        unsigned char* p = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                            ~static_cast<uintptr_t>(1023));
        sh.a_stride = align1k(bytesA);
        sh.b_stride = align1k(bytesB);
        sh.a = p;
        p += stages_a * rows * sh.a_stride;
        sh.b = p;
        p += stages_b * sh.b_stride;
        sh.stage = reinterpret_cast<float*>(p);
        uint64_t* bars = reinterpret_cast<uint64_t*>(p + groups * kTcGroupStageBytes);
        sh.full_a = bars;
        sh.empty_a = bars + 2;
        sh.full_b = bars + 4;
        sh.empty_b = bars + 8;
        sh.full_d = bars + 12;
        sh.empty_d = bars + 15;
        sh.tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
        sh.abort = reinterpret_cast<volatile int*>(bars + 19);
    }
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (uniform)
    const int P = 2 * md + 1;
    const int nseg = (W + kTcM - 1) / kTcM;
    const int nyb = (H + rows - 1) / rows;
    // small maps (rows = 1) split the 2 md + 1 displacement rows over ndyg items
    // to fill the GPU
    const int rpg = (P + ndyg - 1) / ndyg;
    // nprob independent correlations of the same shape (the flow's two
    // directions) share the launch: item it belongs to problem it / items_per
    const int items_per = N * nyb * nseg * ndyg;
    const int items = items_per * nprob;
    auto item = [&](int it) {
        TcItem t;
        t.prob = it / items_per;
        int r = it - t.prob * items_per;
        const int dyg = r % ndyg;
        r /= ndyg;
        t.y0 = (r % nyb) * rows;
        t.ny = min(rows, H - t.y0);
        r /= nyb;
        t.seg = r % nseg;
        t.n = r / nseg;
        t.d0 = dyg * rpg;
        t.d1 = min(P, t.d0 + rpg);
        return t;
    };

    if (warp == 1) {
        ptx::tmem_alloc(sh.tmem_slot, kTmemCols);
        ptx::tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        *sh.abort = 0;
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&sh.full_a[i], 1);
            ptx::mbar_init(&sh.empty_a[i], 1);
        }
        for (int i = 0; i < 4; ++i) {
            ptx::mbar_init(&sh.full_b[i], 1);
            ptx::mbar_init(&sh.empty_b[i], 1);
        }
        for (int i = 0; i < kStagesD; ++i) {
            ptx::mbar_init(&sh.full_d[i], 1);
            ptx::mbar_init(&sh.empty_d[i], 4);  // one arrival per epilogue warp
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *sh.tmem_slot;
    // the setup above (Tensor Memory, barriers) overlaps the previous
    // kernel's tail; its outputs (this launch's operands) are read from here
    pdl_enter();

    if (warp == 0) {
        // ---- TMA producer ------------------------------------------------------
        if (ptx::elect_one()) {
            int ua = 0, ub = 0;
            TcRing ra(stages_a), rb(stages_b);
            bool ok = true;
            for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
                const TcItem t = item(it);
                const CUtensorMap* ma = t.prob ? &mA2 : &mA;
                const CUtensorMap* mb = t.prob ? &mB2 : &mB;
                const int x0 = t.seg * kTcM;
                if (!(ok = tc_wait(&sh.empty_a[ra.i], ra.phase ^ 1, sh.abort)))
                    break;
                ptx::mbar_expect_tx(&sh.full_a[ra.i], t.ny * bytesA);
                for (int r = 0; r < t.ny; ++r)
                    ptx::tma_load_5d(sh.a + (ra.i * rows + r) * sh.a_stride, ma, 0, x0, 0, t.y0 + r, t.n,
                        &sh.full_a[ra.i]);
                ++ua;
                ra.next();
                for (int b = t.d0; b < t.ny - 1 + t.d1; ++b) {  // f2 row y0 + b - md
                    if (!(ok = tc_wait(&sh.empty_b[rb.i], rb.phase ^ 1, sh.abort)))
                        break;
                    ptx::mbar_expect_tx(&sh.full_b[rb.i], bytesB);
                    ptx::tma_load_5d(sh.b + rb.i * sh.b_stride, mb, 0, x0 - md, 0, t.y0 + b - md, t.n,
                        &sh.full_b[rb.i]);
                    ++ub;
                    rb.next();
                }
            }
            if (*sh.abort) {  // let every copy issued land before the CTA exits
                for (int i = 0; i < stages_a && i < ua; ++i) {
                    const int u = ua - 1 - i;
                    ptx::mbar_wait_bounded(&sh.full_a[u % stages_a], (u / stages_a) & 1, kTcWaitSpins);
                }
                for (int i = 0; i < stages_b && i < ub; ++i) {
                    const int u = ub - 1 - i;
                    ptx::mbar_wait_bounded(&sh.full_b[u % stages_b], (u / stages_b) & 1, kTcWaitSpins);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----------------------------------------------------------
        if (ptx::elect_one()) {
            int last = -1, last_phase = 0;
            TcRing ra(stages_a), rb(stages_b), rd(kStagesD);
            bool ok = true;
            // an MMA's K is 32 bytes of a chunk plane's rows
            const int row = 2 * cw;
            const uint64_t a0 = ptx::umma_desc_kmajor_swizzled(ptx::smem_u32(sh.a), row);
            const uint64_t b0 = ptx::umma_desc_kmajor_swizzled(ptx::smem_u32(sh.b), row);
            for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
                const TcItem t = item(it);
                if (!(ok = tc_wait(&sh.full_a[ra.i], ra.phase, sh.abort)))
                    break;
                for (int b = t.d0; ok && b < t.ny - 1 + t.d1; ++b) {
                    if (!(ok = tc_wait(&sh.full_b[rb.i], rb.phase, sh.abort)))
                        break;
                    for (int r = max(0, b - t.d1 + 1); r <= min(t.ny - 1, b - t.d0); ++r) {
                        if (!(ok = tc_wait(&sh.empty_d[rd.i], rd.phase ^ 1, sh.abort)))
                            break;
                        ptx::tc_fence_after();
                        uint64_t ad = a0 + (((ra.i * rows + r) * sh.a_stride) >> 4);
                        uint64_t bd = b0 + ((rb.i * sh.b_stride) >> 4);
                        const uint32_t dcol = tmem + rd.i * kDStride;
                        for (int c = 0; c < Cp; c += cw) {
                            ptx::umma_f16(dcol, ad, bd, idesc, c > 0);
                            for (int k = 1; k < cw >> 4; ++k)
                                ptx::umma_f16(dcol, ad + 2 * k, bd + 2 * k, idesc, true);
                            ad += (kTcM * row) >> 4;
                            bd += (kTcN * row) >> 4;
                        }
                        ptx::umma_commit(&sh.full_d[rd.i]);  // accumulator ready
                        last = rd.i;
                        last_phase = rd.phase;
                        rd.next();
                    }
                    if (!ok)
                        break;
                    ptx::umma_commit(&sh.empty_b[rb.i]);  // f2 row read
                    rb.next();
                }
                if (!ok)
                    break;
                ptx::umma_commit(&sh.empty_a[ra.i]);  // f1 rows read by every product of the item
                ra.next();
            }
            if (*sh.abort && last >= 0)  // the MMAs still in flight finish before Tensor Memory is freed
                ptx::mbar_wait_bounded(&sh.full_d[last], last_phase, kTcWaitSpins);
        }
    } else {
        // ---- epilogue: TMEM -> registers -> shared (diagonal) -> global -----------
        const int q = warp & 3;          // this warp's 32 TMEM lanes (the warp's rank in its warpgroup)
        const int grp = (warp - 2) >> 2;  // epilogue group
        const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
        float* st = sh.stage + (warp - 2) * 32 * kTcPitch;
        const float inv_scale = 1.0f / (scales[0] * scales[1]);  // powers of two: exact
        const int64_t HW = static_cast<int64_t>(H) * W;
        int turn = 0;  // the group whose product is next
        TcRing rd(kStagesD);
        bool ok = true;
        for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
            const TcItem t = item(it);
            const int x = t.seg * kTcM + q * 32 + lane;
            float* obase =
                (t.prob ? out2 : out) + static_cast<int64_t>(t.n) * P * P * HW + static_cast<int64_t>(t.y0) * W + x;
            for (int b = t.d0; ok && b < t.ny - 1 + t.d1; ++b) {
                for (int r = max(0, b - t.d1 + 1); r <= min(t.ny - 1, b - t.d0); ++r) {
                    const bool mine = turn == grp;
                    const int sd = rd.i;
                    const uint32_t phase = rd.phase;
                    turn = turn + 1 == groups ? 0 : turn + 1;
                    rd.next();
                    if (!mine)
                        continue;
                    // One lane polls: twelve warps of 32 polling lanes kept the shared
                    // memory pipe so full that each wait of the issuing thread cost 330
                    // cycles.  Warp-uniform outcome: the loads below are warp-collective.
                    ok = __shfl_sync(0xffffffffu, lane == 0 ? tc_wait(&sh.full_d[sd], phase, sh.abort) : 0, 0);
                    if (!ok)
                        break;
                    __syncwarp();  // orders the other lanes' loads after lane 0's wait (a shuffle does not)
                    ptx::tc_fence_after();
                    uint32_t v0[32], v1[16];
                    const uint32_t ta = tmem + lane_base + sd * kDStride + q * 32;
                    ptx::tmem_ld32(ta, v0);
                    ptx::tmem_ld16(ta + 32, v1);
                    ptx::tmem_ld_wait();
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        ptx::mbar_arrive(&sh.empty_d[sd]);  // the accumulator may be overwritten
                    float4* row = reinterpret_cast<float4*>(st + lane * kTcPitch);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        row[j] = make_float4(__uint_as_float(v0[4 * j]), __uint_as_float(v0[4 * j + 1]),
                            __uint_as_float(v0[4 * j + 2]), __uint_as_float(v0[4 * j + 3]));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        row[8 + j] = make_float4(__uint_as_float(v1[4 * j]), __uint_as_float(v1[4 * j + 1]),
                            __uint_as_float(v1[4 * j + 2]), __uint_as_float(v1[4 * j + 3]));
                    __syncwarp();
                    if (x < W) {
                        float* o = obase + static_cast<int64_t>(b - r) * P * HW + static_cast<int64_t>(r) * W;
                        const float* srow = st + lane * kTcPitch + lane;
                        for (int k0 = 0; k0 < P; k0 += 9) {  // (the staging row has kTcPitch columns)
                            float v[9];
#pragma unroll
                            for (int k = 0; k < 9; ++k)
                                v[k] = srow[k0 + k];
#pragma unroll
                            for (int k = 0; k < 9; ++k)
                                if (k0 + k < P)
                                    o[(k0 + k) * HW] = v[k] * inv_scale;
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, kTmemCols);
    }
    if (threadIdx.x == 0 && *sh.abort)
        atomicExch(timeout_flag, 1);
}

// ---- operand preparation ---------------------------------------------------------
// scale = 2^k with m * 2^k in [2^13, 2^14); 1 for a zero or non-finite m.
__device__ __forceinline__ float tc_scale(float m)
{
    float s = 1.0f;
    if (m > 0.0f && m <= 3.4e38f) {
        int e;
        frexpf(m, &e);  // m = f 2^e, f in [0.5, 1)
        s = ldexpf(1.0f, min(60, max(-60, 14 - e)));
    }
    return s;
}

// max of m over the block (256 threads), in every thread
__device__ __forceinline__ float block_max(float m, float* wm)
{
    for (int o = 16; o > 0; o >>= 1)
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0)
        wm[threadIdx.x >> 5] = m;
    __syncthreads();
    m = wm[0];
    for (int i = 1; i < 8; ++i)
        m = fmaxf(m, wm[i]);
    __syncthreads();
    return m;
}

// max |a| of both operands (blockIdx.y), one partial maximum a block in
// part[blockIdx.y * gridDim.x + blockIdx.x].
__global__ void __launch_bounds__(256) absmax2_kernel(const float* __restrict__ a, const float* __restrict__ b,
    int64_t n, int vec, float* __restrict__ part)
{
    pdl_enter();
    __shared__ float wm[8];
    const float* src = blockIdx.y ? b : a;
    float m = 0.0f;
    const int64_t i0 = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    int64_t done = 0;
    if (vec) {
        const float4* s4 = reinterpret_cast<const float4*>(src);
        done = n / 4 * 4;
#pragma unroll 4
        for (int64_t i = i0; i < n / 4; i += step) {
            const float4 v = s4[i];
            m = fmaxf(fmaxf(fmaxf(m, fabsf(v.x)), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
    }
    for (int64_t i = done + i0; i < n; i += step)
        m = fmaxf(m, fabsf(src[i]));
    m = block_max(m, wm);
    if (threadIdx.x == 0)
        part[blockIdx.y * gridDim.x + blockIdx.x] = m;
}

// The chunked 16-bit layout [n][y][c / cw][x][c % cw]: a thread that packs the 8
// channels 8 q ... of row (n, y) of the map writes the uint4 at this index.
__device__ __forceinline__ int64_t chunked_index(int64_t row, int q, int x, int W, int chunks8, int cw)
{
    const int per = cw >> 3;
    return ((row * (chunks8 / per) + q / per) * W + x) * per + q % per;
}

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float a, float b)
{
    if (kBf16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    } else {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
}

// Both operands, NCHW float -> chunked 16-bit, scaled, zero-padded to Cp
// channels.  Each block first reduces absmax2_kernel's partial maxima to the two
// scales (the first one stores them for the correlation), then walks (operand,
// batch, chunk, pixels) items: a chunk of kPx = 64 pixels (128 of the narrowest
// chunk) is read coalesced along x, packed in shared memory (pixels 16 bytes
// further apart than they are long, which spreads them over the banks) and
// written out whole, 16 bytes a thread side by side.  2 x 64 x 136 x 240 take 11.4 us,
// and 13.4 when the reading threads stored their 32 bytes of every pixel
// themselves; the loads of the first item do not wait for the scales.  A thread of
// the narrowest chunk has one 16-byte piece and stores it itself, the next item's
// loads on their way, without barriers.
template <bool kBf16, int kCw>
__global__ void __launch_bounds__(256) to_chunked2_kernel(const float* __restrict__ f1, const float* __restrict__ f2,
    uint4* __restrict__ c1, uint4* __restrict__ c2, const float* __restrict__ part, int nparts,
    float* __restrict__ scales, int N, int C, int H, int W, int Cp)
{
    constexpr int kPer = kCw / 8;                  // 16-byte pieces of a pixel
    constexpr int kPx = kCw == 16 ? 128 : 64;      // pixels of an item
    constexpr int kCh = kCw * kPx / 256;           // channels a thread reads
    constexpr int kPitch = kPer + 1;
    __shared__ uint4 tile[kCw == 16 ? 1 : kPx * kPitch];
    __shared__ float wm[8];
    pdl_enter();
    const unsigned HW = static_cast<unsigned>(H) * W;  // < 2^30
    const unsigned npb = (HW + kPx - 1) / kPx, nq = Cp / kCw;
    const unsigned items = 2u * N * nq * npb;  // (an item is 1 KB of the workspace or more: < 2^31)
    const int px = threadIdx.x % kPx, part_of = threadIdx.x / kPx;
    unsigned pb;
    int q, n, t;
    float v[kCh];
    auto fetch = [&](unsigned it) {
        pb = it % npb * kPx;
        unsigned r = it / npb;
        q = static_cast<int>(r % nq);
        r /= nq;
        n = static_cast<int>(r % N);
        t = static_cast<int>(r / N);
        const int c0 = q * kCw + part_of * kCh;
        const float* src = (t ? f2 : f1) + (static_cast<int64_t>(n) * C + c0) * HW + pb + px;
#pragma unroll
        for (int j = 0; j < kCh; ++j)
            v[j] = pb + px < HW && c0 + j < C ? src[static_cast<int64_t>(j) * HW] : 0.0f;
    };
    fetch(blockIdx.x);  // the grid is no larger than the items
    float m1 = 0.0f, m2 = 0.0f;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        m1 = fmaxf(m1, part[i]);
        m2 = fmaxf(m2, part[nparts + i]);
    }
    const float s1 = tc_scale(block_max(m1, wm)), s2 = tc_scale(block_max(m2, wm));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        scales[0] = s1;
        scales[1] = s2;
    }
    for (unsigned it = blockIdx.x;;) {
        const float sc = t ? s2 : s1;
        if constexpr (kCw == 16) {
            static_assert(kCw != 16 || kCh == 8, "a piece a thread");
            const uint4 packed = make_uint4(pack2<kBf16>(v[0] * sc, v[1] * sc), pack2<kBf16>(v[2] * sc, v[3] * sc),
                pack2<kBf16>(v[4] * sc, v[5] * sc), pack2<kBf16>(v[6] * sc, v[7] * sc));
            const unsigned p = pb + px, y = p / W, x = p - y * W;
            uint4* const dst = (t ? c2 : c1) + ((static_cast<int64_t>(n) * H + y) * nq + q) * W * kPer + x * kPer + part_of;
            const bool in = p < HW;
            it += gridDim.x;
            if (it < items)
                fetch(it);
            if (in)
                *dst = packed;
            if (it >= items)
                break;
            continue;
        }
#pragma unroll
        for (int h = 0; h < kCh / 8; ++h)
            tile[px * kPitch + part_of * (kCh / 8) + h] =
                make_uint4(pack2<kBf16>(v[8 * h] * sc, v[8 * h + 1] * sc),
                    pack2<kBf16>(v[8 * h + 2] * sc, v[8 * h + 3] * sc),
                    pack2<kBf16>(v[8 * h + 4] * sc, v[8 * h + 5] * sc),
                    pack2<kBf16>(v[8 * h + 6] * sc, v[8 * h + 7] * sc));
        __syncthreads();
        uint4* dst = t ? c2 : c1;
#pragma unroll
        for (int i = threadIdx.x; i < kPx * kPer; i += 256) {
            const unsigned p = pb + i / kPer;
            if (p < HW) {
                const unsigned y = p / W, x = p - y * W;
                dst[((static_cast<int64_t>(n) * H + y) * nq + q) * W * kPer + x * kPer + i % kPer] =
                    tile[i / kPer * kPitch + i % kPer];
            }
        }
        it += gridDim.x;
        if (it >= items)
            break;
        fetch(it);
        __syncthreads();
    }
}

// The same for the five levels of a feature pyramid (N = 1, a given scale, 8
// channels a thread) in one launch: a flat list of (128-pixel block, chunk) pairs, level after level.
constexpr int kChunkLevelsMax = 5;
struct ChunkLevels {
    const float* in[kChunkLevelsMax];
    uint4* out[kChunkLevelsMax];
    int C[kChunkLevelsMax], H[kChunkLevelsMax], W[kChunkLevelsMax], chunks[kChunkLevelsMax], cw[kChunkLevelsMax];
    int block0[kChunkLevelsMax + 1];
    int count;
};

template <bool kBf16>
__global__ void to_chunked_levels_kernel(const __grid_constant__ ChunkLevels cl, const float* __restrict__ scale)
{
    pdl_enter();
    int l = 0;
    while (l + 1 < cl.count && static_cast<int>(blockIdx.x) >= cl.block0[l + 1])
        ++l;
    const int W = cl.W[l], H = cl.H[l], C = cl.C[l], chunks = cl.chunks[l];
    const int HW = H * W, nhw = (HW + 127) / 128;
    const int b = blockIdx.x - cl.block0[l];
    const int p = (b % nhw) * 128 + threadIdx.x, q = b / nhw;
    if (p >= HW)
        return;
    const int y = p / W, x = p - y * W;
    const float s = *scale;
    const float* src = cl.in[l] + p;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = q * 8 + j;
        v[j] = c < C ? src[static_cast<int64_t>(c) * HW] * s : 0.0f;
    }
    cl.out[l][chunked_index(y, q, x, W, chunks, cl.cw[l])] = make_uint4(pack2<kBf16>(v[0], v[1]),
        pack2<kBf16>(v[2], v[3]), pack2<kBf16>(v[4], v[5]), pack2<kBf16>(v[6], v[7]));
}

// custom::Warp (the single-precision arithmetic of warp_op_kernel) writing
// the chunked 16-bit operand layout directly, scaled by *scale: the warped
// second-frame features of the flow estimator go straight to the tensor-core
// correlation.  One thread per pixel and chunk of 8 channels.  kUp: `flow`
// is the estimator's coarser cw x chh level, upsampled 2x here (up2_sample)
// instead of read from an upsampled copy.
template <bool kBf16, bool kUp>
__global__ void warp_to_chunked_kernel(const float* __restrict__ in, const float* __restrict__ flow,
    uint4* __restrict__ out, const float* __restrict__ scale, int C, int H, int W, int chunks, int chunk_w,
    int64_t sin, int64_t sfl, int64_t sout, int cw, int chh)
{
    pdl_enter();
    const int64_t HW = static_cast<int64_t>(H) * W;
    const int64_t p = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (p >= HW)
        return;
    const int q = blockIdx.y, n = blockIdx.z;
    // 32-bit division where the plane allows (a 64-bit one is a software routine)
    const int y = HW < (int64_t(1) << 31) ? static_cast<int>(p) / W : static_cast<int>(p / W);
    const int x = static_cast<int>(p - static_cast<int64_t>(y) * W);
    const float* fl = flow + n * sfl;
    const float xf = static_cast<float>(x) + (kUp ? up2_sample(fl, cw, chh, x, y, 0) : __ldg(fl + p));
    const float yf = static_cast<float>(y) + (kUp ? up2_sample(fl, cw, chh, x, y, 1) : __ldg(fl + HW + p));
    const float fxl = floorf(xf), fyt = floorf(yf);
    const float a = xf - fxl, b = yf - fyt;
    const float xR = fxl + 1.0f, yB = fyt + 1.0f;
    const bool mL = (0.0f <= fxl && fxl <= static_cast<float>(W - 1));
    const bool mR = (0.0f <= xR && xR <= static_cast<float>(W - 1));
    const bool mT = (0.0f <= fyt && fyt <= static_cast<float>(H - 1));
    const bool mB = (0.0f <= yB && yB <= static_cast<float>(H - 1));
    const float ia = 1.0f - a, ib = 1.0f - b;
    const float wTL = ia * ib, wTR = a * ib, wBL = ia * b, wBR = a * b;
    const bool tl = mT && mL, tr = mT && mR, bl = mB && mL, br = mB && mR;
    float mask = 0.0f;
    mask += tl ? wTL : 0.0f;
    mask += tr ? wTR : 0.0f;
    mask += bl ? wBL : 0.0f;
    mask += br ? wBR : 0.0f;
    const bool take = mask > 0.999f;
    const int xl = take ? static_cast<int>(fxl) : 0;
    const int yt = take ? static_cast<int>(fyt) : 0;
    const int64_t oTL = static_cast<int64_t>(yt) * W + xl;
    const float s = *scale;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = q * 8 + j;
        float val = 0.0f;
        if (take && c < C) {
            const float* src = in + n * sin + static_cast<int64_t>(c) * HW;
            val += tl ? wTL * __ldg(src + oTL) : 0.0f;
            val += tr ? wTR * __ldg(src + oTL + 1) : 0.0f;
            val += bl ? wBL * __ldg(src + oTL + W) : 0.0f;
            val += br ? wBR * __ldg(src + oTL + W + 1) : 0.0f;
        }
        v[j] = val * s;
    }
    out[n * sout + chunked_index(y, q, x, W, chunks, chunk_w)] =
        make_uint4(pack2<kBf16>(v[0], v[1]), pack2<kBf16>(v[2], v[3]), pack2<kBf16>(v[4], v[5]), pack2<kBf16>(v[6], v[7]));
}

// 5-D map over a chunked tensor: {c % cw, x, c / cw, y, n}, box {cw, pixels, cp /
// cw, 1, 1}, swizzled by the box's 2 cw-byte rows: the tile lands in the operand
// layout umma_desc_kmajor_swizzled describes.
bool encode_chunked_map(CUtensorMap* m, const void* base, int N, int H, int W, int cp, int box_pixels)
{
    EncodeTiledFn fn = tensor_map_encoder();
    if (!fn)
        return false;
    const int w = tc_chunk_channels(cp);
    const cuuint64_t row = static_cast<cuuint64_t>(w) * 2;
    const cuuint64_t q = static_cast<cuuint64_t>(cp / w);
    const cuuint64_t dims[5] = {static_cast<cuuint64_t>(w), static_cast<cuuint64_t>(W), q, static_cast<cuuint64_t>(H),
        static_cast<cuuint64_t>(N)};
    const cuuint64_t strides[4] = {row, static_cast<cuuint64_t>(W) * row, q * W * row,
        static_cast<cuuint64_t>(H) * q * W * row};
    const cuuint32_t box[5] = {static_cast<cuuint32_t>(w), static_cast<cuuint32_t>(box_pixels),
        static_cast<cuuint32_t>(q), 1, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 5, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE,
               w == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : w == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The dynamic shared memory opt-in is a per-device function attribute; the
// persistent grid is sized by the device's SM count.
cudaError_t tc_prepare_device(int* sms)
{
    static PerDevice<int> device;
    return device.get(
        [](int* count) {
            cudaError_t e =
                cudaFuncSetAttribute(corr_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemLimit);
            int dev = 0;
            if (e == cudaSuccess)
                e = cudaGetDevice(&dev);
            return e != cudaSuccess ? e : cudaDeviceGetAttribute(count, cudaDevAttrMultiProcessorCount, dev);
        },
        sms);
}

}  // namespace

int tc_padded_channels(int C) { return (C + 15) / 16 * 16; }
int tc_chunk_channels(int cp) { return cp % 64 == 0 ? 64 : cp % 32 == 0 ? 32 : 16; }

size_t corr_tc_workspace_bytes(int N, int C, int H, int W)
{
    const size_t chunked = static_cast<size_t>(N) * H * W * tc_padded_channels(C) * 2;
    return 256 + 2 * ((chunked + 255) / 256 * 256);
}

cudaError_t launch_corr_tc_chunked(const void* f1c, const void* f2c, float* out, const float* scales, int N, int Cp,
    int H, int W, int md, bool bf16, cudaStream_t st)
{
    return launch_corr_tc_chunked2(f1c, f2c, out, nullptr, nullptr, nullptr, scales, N, Cp, H, W, md, bf16, st);
}

cudaError_t launch_corr_tc_chunked2(const void* f1c, const void* f2c, float* out, const void* g1c, const void* g2c,
    float* out2, const float* scales, int N, int Cp, int H, int W, int md, bool bf16, cudaStream_t st)
{
    const int nprob = g1c ? 2 : 1;
    if (Cp % 16 != 0 || Cp > kTcMaxChannelsPadded || md < 0 || md > kTcMaxMd)
        return cudaErrorInvalidValue;
    int sms = 0;
    cudaError_t e = tc_prepare_device(&sms);
    if (e != cudaSuccess)
        return e;
    int* flag = nullptr;
    if ((e = device_timeout_flag(&flag)) != cudaSuccess)
        return e;
    CUtensorMap mA, mB, mA2, mB2;
    if (!encode_chunked_map(&mA, f1c, N, H, W, Cp, kTcM) || !encode_chunked_map(&mB, f2c, N, H, W, Cp, kTcN))
        return cudaErrorInvalidValue;
    if (nprob == 2 &&
        (!encode_chunked_map(&mA2, g1c, N, H, W, Cp, kTcM) || !encode_chunked_map(&mB2, g2c, N, H, W, Cp, kTcN)))
        return cudaErrorInvalidValue;
    if (nprob == 1) {
        mA2 = mA;
        mB2 = mB;
    }
    const int P = 2 * md + 1;
    const int nseg = (W + kTcM - 1) / kTcM;
    auto items_of = [&](int rows) { return nprob * N * ((H + rows - 1) / rows) * nseg; };
    // Output rows of an item: as many as shared memory holds two sets of beside
    // four f2 rows (4 rows of 32 channels, 2 of 64), fewer when the items would
    // leave an eighth of the SMs or more idle.  On 2 x 64 x 136 x 240 19.2 us
    // with two rows and 21.7 with one; 32 x 272 x 480 29.4 with four, 37.4 with one.
    int rows = Cp <= 32 ? 4 : Cp <= 64 ? 2 : 1;
    while (rows > 1 && 8 * items_of(rows) < 7 * sms)
        rows /= 2;
    const TcPlan plan = tc_plan(Cp, rows);
    int ndyg = 1;  // split the displacement rows until there are two items per SM
    while (rows == 1 && ndyg < P && items_of(1) * ndyg < 2 * sms)
        ++ndyg;
    const int items = items_of(rows) * ndyg;
    const cudaError_t el = launch_pdl(corr_tc_kernel, dim3(std::min(items, sms)), dim3((2 + 4 * plan.groups) * 32),
        plan.smem, st, mA, mB, out, mA2, mB2, nprob == 2 ? out2 : out, nprob, scales, N, H, W, Cp,
        tc_chunk_channels(Cp), md, ptx::umma_idesc_f16(bf16, kTcM, kTcN), plan.rows, plan.stages_a, plan.stages_b,
        plan.groups, ndyg, flag);
    return el != cudaSuccess ? el : cudaGetLastError();
}

cudaError_t launch_to_chunked_levels(const float* const* in, void* const* out, const int* C, const int* H,
    const int* W, int n, const float* scale, bool bf16, cudaStream_t st)
{
    if (n < 1 || n > kChunkLevelsMax)
        return cudaErrorInvalidValue;
    ChunkLevels cl{};
    cl.count = n;
    cl.block0[0] = 0;
    for (int l = 0; l < n; ++l) {
        if (static_cast<int64_t>(H[l]) * W[l] >= (int64_t(1) << 31))
            return cudaErrorInvalidValue;
        cl.in[l] = in[l];
        cl.out[l] = static_cast<uint4*>(out[l]);
        cl.C[l] = C[l];
        cl.H[l] = H[l];
        cl.W[l] = W[l];
        cl.chunks[l] = tc_padded_channels(C[l]) / 8;
        cl.cw[l] = tc_chunk_channels(tc_padded_channels(C[l]));
        cl.block0[l + 1] = cl.block0[l] + ((H[l] * W[l] + 127) / 128) * cl.chunks[l];
    }
    const cudaError_t e = launch_pdl(bf16 ? to_chunked_levels_kernel<true> : to_chunked_levels_kernel<false>,
        dim3(cl.block0[n]), dim3(128), 0, st, cl, scale);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_warp_to_chunked(const float* in, const float* flow, void* out, const float* scale, int N, int C,
    int H, int W, int64_t sin, int64_t sfl, int64_t sout_bytes, bool bf16, cudaStream_t st, int cw, int chh)
{
    const int chunks = tc_padded_channels(C) / 8;
    const int64_t HW = static_cast<int64_t>(H) * W;
    const dim3 g(static_cast<unsigned>((HW + 255) / 256), chunks, N);
    const int64_t so = sout_bytes / 16;
    const bool up = cw > 0 && chh > 0;
    auto k = bf16 ? (up ? warp_to_chunked_kernel<true, true> : warp_to_chunked_kernel<true, false>)
                  : (up ? warp_to_chunked_kernel<false, true> : warp_to_chunked_kernel<false, false>);
    const cudaError_t e = launch_pdl(k, g, dim3(256), 0, st, in, flow, static_cast<uint4*>(out), scale, C, H, W,
        chunks, tc_chunk_channels(chunks * 8), sin, sfl, so, cw, chh);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_corr_tc(const float* f1, const float* f2, float* out, int N, int C, int H, int W, int md,
    bool bf16, void* workspace, cudaStream_t st)
{
    const int cp = tc_padded_channels(C);
    const size_t chunked = static_cast<size_t>(N) * H * W * cp * 2;
    const size_t chunked_al = (chunked + 255) / 256 * 256;
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    float* scales = reinterpret_cast<float*>(ws);
    uint4* c1 = reinterpret_cast<uint4*>(ws + 256);
    uint4* c2 = reinterpret_cast<uint4*>(ws + 256 + chunked_al);
    int sms = 0;
    cudaError_t e = tc_prepare_device(&sms);
    if (e != cudaSuccess)
        return e;
    // Three launches: partial maxima (kept at the front of `out`, which the
    // correlation overwrites; behind the scales when it has no 64 elements or shares
    // memory with an operand), both operands' conversion with the scales
    // worked out by every block, the correlation.  (A memset, a maximum and a
    // conversion per operand and a launch for the scales, with the correlation of
    // that time: 2 x 64 x 136 x 240 67.7 us a call, now 38.7; 130 x 34 x 60 on one
    // pair of operands 29 and 14.)
    const int64_t total = static_cast<int64_t>(N) * C * H * W;
    const int64_t outs = static_cast<int64_t>(N) * (2 * md + 1) * (2 * md + 1) * H * W;
    auto apart = [&](const float* f) { return std::less_equal<const float*>()(f + total, out) ||
                                              std::less_equal<const float*>()(out + outs, f); };
    const bool in_out = outs >= 64 && apart(f1) && apart(f2);
    float* part = in_out ? out : scales + 8;
    const int64_t want = std::min<int64_t>((total / 4 + 1023) / 1024, 4 * sms);  // 4+ vectors a thread, every SM full
    const unsigned parts = static_cast<unsigned>(
        std::max<int64_t>(1, std::min<int64_t>(want, in_out ? outs / 2 : 28)));
    auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    e = launch_pdl(absmax2_kernel, dim3(parts, 2), dim3(256), 0, st, f1, f2, total, a16(f1) && a16(f2) ? 1 : 0, part);
    if (e != cudaSuccess)
        return e;
    const int cw = tc_chunk_channels(cp), px = cw == 16 ? 128 : 64;
    const int64_t items = 2 * static_cast<int64_t>(N) * (cp / cw) * ((static_cast<int64_t>(H) * W + px - 1) / px);
    const unsigned blocks = static_cast<unsigned>(std::min<int64_t>(items, 16 * sms));
    auto kernel = cw == 64   ? (bf16 ? to_chunked2_kernel<true, 64> : to_chunked2_kernel<false, 64>)
                  : cw == 32 ? (bf16 ? to_chunked2_kernel<true, 32> : to_chunked2_kernel<false, 32>)
                             : (bf16 ? to_chunked2_kernel<true, 16> : to_chunked2_kernel<false, 16>);
    e = launch_pdl(kernel, dim3(blocks), dim3(256), 0, st, f1, f2, c1, c2, static_cast<const float*>(part),
        static_cast<int>(parts), scales, N, C, H, W, cp);
    return e != cudaSuccess ? e : launch_corr_tc_chunked(c1, c2, out, scales, N, cp, H, W, md, bf16, st);
}

}  // namespace vsc
