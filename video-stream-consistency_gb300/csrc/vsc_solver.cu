// The blend solver of the stabilization pass (reference: kernel_consist_out
// and get_consist_out, src/stabilization/flowconsistency.cu:193-258, :350-374).
//
// Differences from the reference's schedule (results are the CPU
// restatement's, bit for bit except that a zero may carry the other sign,
// see jacobi_px):
//   - Jacobi iteration: the reference updates consisOut in place
//     (flowconsistency.cu:370), so neighbours read a timing-dependent mix of
//     old and new values; here every pixel reads the previous iterate;
//   - the Laplacian of the processed image, which the reference recomputes in
//     every iteration, is computed once per solve (same expression, same bits);
//   - several iterations per launch on register-resident tiles (temporal
//     blocking) instead of one launch per iteration.
#include "vsc_internal.h"
#include "vsc_math.cuh"

#include <cuda.h>  // CUtensorMap (the encoder is fetched from the driver at run time)

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace vsc {
namespace {

inline dim3 grid2d(int w, int h, dim3 b) { return dim3((w + b.x - 1) / b.x, (h + b.y - 1) / b.y); }

// ---- kernel_consist_out (flowconsistency.cu:193-258) ------------------------
// Laplacian of the processed image with the reference's neighbour rule and
// summation order (right, left, bottom, top, then - cnt * centre).
__global__ void lap_pr_kernel(const float* __restrict__ P, float* __restrict__ L, int w, int h)
{
    pdl_enter();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h)
        return;
    const int64_t i0 = pix_index(x, y, w) * 3;
    const int64_t rs = static_cast<int64_t>(w) * 3;
    for (int c = 0; c < 3; ++c) {
        const int64_t i = i0 + c;
        int cnt = 0;
        float lap = 0.0f;
        if ((x + 1) < (w - 1)) {
            lap += P[i + 3];
            cnt += 1;
        }
        if ((x - 1) >= 0) {
            lap += P[i - 3];
            cnt += 1;
        }
        if ((y + 1) < (h - 1)) {
            lap += P[i + rs];
            cnt += 1;
        }
        if ((y - 1) >= 0) {
            lap += P[i - rs];
            cnt += 1;
        }
        lap -= static_cast<float>(cnt) * P[i];
        L[i] = lap;
    }
}

// ---- temporally blocked solver --------------------------------------------
// kTbT Jacobi iterations per launch on a kTbEX x kTbEY extended tile; the
// interior (the tile minus a kTbT-wide ring) is exact after kTbT iterations
// and is written back.  Each of the 512 threads owns a 2x2 pixel block and
// keeps its state (O, U) and the per-pixel constants (lap P, A, consWt) in
// registers; O is published to shared memory (double-buffered) for the rows
// of the neighbouring warps, and horizontal neighbours travel by warp
// shuffle (one warp spans the full tile width).  Tiles away from the image
// border skip the reference's neighbour-validity selects.  The result equals
// the one-iteration-per-launch Jacobi bit for bit.
constexpr int kTbEX = 64;
constexpr int kTbEY = 32;
constexpr int kTbPX = kTbEX + 4;               // shared row pitch (2-column apron each side)
constexpr int kTbPlane = kTbPX * (kTbEY + 2);  // one colour plane with a 1-row apron
constexpr int kTbSmem = 2 * 3 * kTbPlane * static_cast<int>(sizeof(float));
static_assert(2 * kTbT < kTbEY, "tile too small for the iteration count");

// One Jacobi step of one pixel (kernel_consist_out's expression).  With kAll
// every neighbour is valid (cnt = 4) and the validity selects are skipped.
template <bool kAll>
__device__ __forceinline__ float jacobi_px(float o, float& u, float a, float wt, float lp, float right, float left,
    float down, float up, bool vr, bool vl, bool vd, bool vu, float cnt, float step, float mom, bool mom_on)
{
    // The reference sums the neighbours onto 0.0f; starting from the first
    // term drops one addition per pixel and channel.  0 + x equals x except
    // for x = -0 (0 + -0 = +0), so the two sums differ at most in the sign of
    // a zero, and no later operation of the pass (sums, products, squares,
    // fabs, comparisons) turns a zero's sign into a different non-zero value
    // or output byte.
    float lap;
    if (kAll) {
        lap = right + left;
        lap += down;
        lap += up;
    } else {
        lap = vr ? right : 0.0f;
        lap += vl ? left : 0.0f;
        lap += vd ? down : 0.0f;
        lap += vu ? up : 0.0f;
    }
    // with every neighbour valid cnt is 4 and 4 * o is exact (|o| < 2^125),
    // so one fused multiply-add rounds as the reference's multiply, subtract
    if (kAll)
        lap = __fmaf_rn(-4.0f, o, lap);
    else
        lap -= cnt * o;
    const float tmp_1 = wt * (o - a);
    const float tmp_2 = lap - lp;
    const float sg = step * (tmp_2 - tmp_1);
    float out = o + sg;
    if (mom_on)
        out = out + mom * u;
    u = sg;
    return out;
}

struct TbState {
    float o[4][3], u[4][3], a[4][3], wt[4][3], lp[4][3];  // [pixel q = 2*row + col][channel]
};

// One Jacobi step of a thread's 2x2 block, all three channels: reads the
// previous iterate from shared buffer `cur` (vertical neighbours) and the
// neighbouring lanes (horizontal ones), publishes the new one to `cur ^ 1`.
template <bool kAll>
__device__ __forceinline__ void tb_step(TbState& s, const bool (&vr)[4], const bool (&vl)[4], const bool (&vd)[4],
    const bool (&vu)[4], const float (&cnt)[4], float* smem, int cur, bool mom_on, float step, float mom, int px0,
    int py0)
{
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const float* S = smem + (cur * 3 + ch) * kTbPlane;
        const float2 up = *reinterpret_cast<const float2*>(&S[py0 * kTbPX + px0 + 2]);
        const float2 dn = *reinterpret_cast<const float2*>(&S[(py0 + 3) * kTbPX + px0 + 2]);
        const float o0 = s.o[0][ch], o1 = s.o[1][ch], o2 = s.o[2][ch], o3 = s.o[3][ch];
        const float l0 = __shfl_up_sync(0xffffffffu, o1, 1);
        const float l1 = __shfl_up_sync(0xffffffffu, o3, 1);
        const float r0 = __shfl_down_sync(0xffffffffu, o0, 1);
        const float r1 = __shfl_down_sync(0xffffffffu, o2, 1);
        const float n0 = jacobi_px<kAll>(o0, s.u[0][ch], s.a[0][ch], s.wt[0][ch], s.lp[0][ch], o1, l0, o2, up.x,
            vr[0], vl[0], vd[0], vu[0], cnt[0], step, mom, mom_on);
        const float n1 = jacobi_px<kAll>(o1, s.u[1][ch], s.a[1][ch], s.wt[1][ch], s.lp[1][ch], r0, o0, o3, up.y,
            vr[1], vl[1], vd[1], vu[1], cnt[1], step, mom, mom_on);
        const float n2 = jacobi_px<kAll>(o2, s.u[2][ch], s.a[2][ch], s.wt[2][ch], s.lp[2][ch], o3, l1, dn.x, o0,
            vr[2], vl[2], vd[2], vu[2], cnt[2], step, mom, mom_on);
        const float n3 = jacobi_px<kAll>(o3, s.u[3][ch], s.a[3][ch], s.wt[3][ch], s.lp[3][ch], r1, o2, dn.y, o1,
            vr[3], vl[3], vd[3], vu[3], cnt[3], step, mom, mom_on);
        s.o[0][ch] = n0;
        s.o[1][ch] = n1;
        s.o[2][ch] = n2;
        s.o[3][ch] = n3;
        float* D = smem + ((cur ^ 1) * 3 + ch) * kTbPlane;
        *reinterpret_cast<float2*>(&D[(py0 + 1) * kTbPX + px0 + 2]) = make_float2(n0, n1);
        *reinterpret_cast<float2*>(&D[(py0 + 2) * kTbPX + px0 + 2]) = make_float2(n2, n3);
    }
}

// `ring` is the width of the ring around the rows written back (the rows
// [ring, kTbEY - ring) are exact after the T iterations).  Iteration k only
// has to be right on rows [ring - T + k + 1, kTbEY - ring + T - k - 1), one
// row fewer on each side per iteration, so a warp (two rows) whose rows all
// lie outside skips it: the rows it would have published are read only by
// rows that are themselves outside the next iteration's range.  A launch of
// the full kTbT iterations after the first step of the solve (momentum on
// throughout) runs fully unrolled; others take the general loop.
template <bool kAll>
__device__ __forceinline__ void tb_iterate(TbState& s, const bool (&vr)[4], const bool (&vl)[4],
    const bool (&vd)[4], const bool (&vu)[4], const float (&cnt)[4], float* smem, int T, int ring, int k0,
    float step, float mom, int px0, int py0)
{
    if (T == kTbT && ring == kTbT) {
        // full launches, unrolled; momentum is off only in the first step of a solve
        const bool later = k0 > 0;
#pragma unroll
        for (int k = 0; k < kTbT; ++k) {
            const int lo = k + 1, hi = kTbEY - k - 1;  // the general bounds with ring == T == kTbT
            if (!(py0 + 1 < lo || py0 >= hi))  // warp-uniform: py0 = 2 * threadIdx.y
                tb_step<kAll>(s, vr, vl, vd, vu, cnt, smem, k & 1, k > 0 || later, step, mom, px0, py0);
            __syncthreads();
        }
        return;
    }
    for (int k = 0; k < T; ++k) {
        const int lo = ring - T + k + 1, hi = kTbEY - ring + T - k - 1;
        if (!(py0 + 1 < lo || py0 >= hi))
            tb_step<kAll>(s, vr, vl, vd, vu, cnt, smem, k & 1, (k0 + k) > 0, step, mom, px0, py0);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kTbEX / 2 * kTbEY / 2, 1)
    solver_tb_kernel(const float* __restrict__ Oin, float* __restrict__ Oout, const float* __restrict__ Uin,
        float* __restrict__ Uout, const float* __restrict__ L, const float* __restrict__ A,
        const float* __restrict__ Wt, int w, int h, int T, int k0, float step, float mom, uint8_t* __restrict__ rgba)
{
    extern __shared__ __align__(16) float smem[];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * 32 + tx;
    const int ox = blockIdx.x * (kTbEX - 2 * T) - T;
    const int oy = blockIdx.y * (kTbEY - 2 * T) - T;
    const int px0 = 2 * tx, py0 = 2 * ty;

    // both buffers start at zero, aprons included (apron cells are only read
    // by pixels of the outermost ring, whose results are never written back)
    for (int i = tid; i < 2 * 3 * kTbPlane; i += blockDim.x * blockDim.y)
        smem[i] = 0.0f;
    __syncthreads();

    TbState s;
    float cnt[4];
    bool vr[4], vl[4], vd[4], vu[4], inimg[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int gx = ox + px0 + (q & 1);
        const int gy = oy + py0 + (q >> 1);
        inimg[q] = gx >= 0 && gx < w && gy >= 0 && gy < h;
        vr[q] = (gx + 1) < (w - 1);
        vl[q] = (gx - 1) >= 0;
        vd[q] = (gy + 1) < (h - 1);
        vu[q] = (gy - 1) >= 0;
        cnt[q] = static_cast<float>(static_cast<int>(vr[q]) + static_cast<int>(vl[q]) + static_cast<int>(vd[q]) +
                                    static_cast<int>(vu[q]));
        const int64_t idx = inimg[q] ? pix_index(gx, gy, w) * 3 : 0;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            s.o[q][ch] = inimg[q] ? Oin[idx + ch] : 0.0f;
            s.u[q][ch] = inimg[q] ? Uin[idx + ch] : 0.0f;
            s.a[q][ch] = inimg[q] ? A[idx + ch] : 0.0f;
            s.wt[q][ch] = inimg[q] ? Wt[idx + ch] : 0.0f;
            s.lp[q][ch] = inimg[q] ? L[idx + ch] : 0.0f;
        }
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        float* S = smem + ch * kTbPlane;
        *reinterpret_cast<float2*>(&S[(py0 + 1) * kTbPX + px0 + 2]) = make_float2(s.o[0][ch], s.o[1][ch]);
        *reinterpret_cast<float2*>(&S[(py0 + 2) * kTbPX + px0 + 2]) = make_float2(s.o[2][ch], s.o[3][ch]);
    }
    __syncthreads();

    // tiles whose every pixel has all four neighbours skip the validity selects
    const bool interior = ox >= 1 && oy >= 1 && ox + kTbEX - 1 <= w - 3 && oy + kTbEY - 1 <= h - 3;
    if (interior)
        tb_iterate<true>(s, vr, vl, vd, vu, cnt, smem, T, T, k0, step, mom, px0, py0);
    else
        tb_iterate<false>(s, vr, vl, vd, vu, cnt, smem, T, T, k0, step, mom, px0, py0);

#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = q >> 1, c = q & 1;
        const int px = px0 + c, py = py0 + r;
        if (!inimg[q] || px < T || px >= kTbEX - T || py < T || py >= kTbEY - T)
            continue;
        const int64_t p = pix_index(ox + px, oy + py, w);
        float ov[3];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            ov[ch] = s.o[q][ch];
            Oout[p * 3 + ch] = ov[ch];
            Uout[p * 3 + ch] = s.u[q][ch];
        }
        if (rgba)
            reinterpret_cast<uint32_t*>(rgba)[p] = pack_rgba(ov[0], ov[1], ov[2]);
    }
}

// ---- persistent, TMA-fed solver ----------------------------------------------
// Same tile, same per-pixel arithmetic as solver_tb_kernel, but one CTA per
// SM walks a list of tiles and the five input tiles (O, U, A, consWt, lap P:
// 32 rows x 192 floats of the interleaved images each) of its NEXT tile are
// fetched by TMA into shared memory while the current tile iterates, so
// global-memory latency no longer serialises with the compute.  The tile
// origin is fixed by the 8-pixel ring (kTbT), whatever the iteration count
// of the launch, which keeps the TMA x coordinate (3 * origin floats) on the
// 16-byte grid.  Needs width % 4 == 0 (16-byte row pitch) and 16-byte
// aligned images; other sizes use solver_tb_kernel.
constexpr int kIW = kTbEX - 2 * kTbT;                  // interior width  (48)
constexpr int kIH = kTbEY - 2 * kTbT;                  // interior height (16)
constexpr int kStageFloats = kTbEY * kTbEX * 3;        // one input tile
constexpr int kStageBytes = kStageFloats * static_cast<int>(sizeof(float));
constexpr int kPsSmem = 5 * kStageBytes + kTbSmem + 16;
constexpr int kWaitSpins = 1 << 22;                    // bounded mbarrier wait (about a second)
static_assert((3 * kTbT) % 4 == 0 && (3 * kIW) % 4 == 0, "TMA x coordinates must be 16-byte aligned");

__device__ int g_device_timeout;  // set by a kernel whose bounded wait gave up

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Spins at most `spins` polls (with back-off); false if the phase never completed.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int spins)
{
    for (int i = 0; i < spins; ++i) {
        if (mbar_try_wait(bar, parity))
            return true;
        if (i > 32)
            __nanosleep(256);
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// Programmatic dependent launch: a solver launch may start while the previous
// one drains (its CTAs set up shared memory and barriers meanwhile); before
// the first read of the previous launch's O and U, and before any write to
// the images it was reading, every thread waits for that launch to complete.
// The previous launch lets the next one start once each of its CTAs is on
// its last tile.  Without the launch attribute both are no-ops.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependent_launch() { asm volatile("griddepcontrol.launch_dependents;" :::); }

// TMA tensor store (shared -> global) of one box; elements outside the image are clipped
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* src)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
        "r"(x), "r"(y), "r"(smem_u32(src))
        : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// this thread's bulk stores have read their shared-memory source
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// this thread's bulk stores are complete
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// The interior of a tile (after the T-pixel ring) leaves through shared memory
// and two TMA stores, one per image, instead of scalar stores of 12-byte
// pixels: `so` / `su` hold rows of 3 * kIW floats, filled by every thread,
// then one thread issues the stores; the staging is reusable after
// bulk_wait_read and a barrier.
__device__ __forceinline__ void store_interior(const CUtensorMap* mOo, const CUtensorMap* mUo, int ox, int oy,
    const float* so, const float* su)
{
    tma_store_2d(mOo, 3 * (ox + kTbT), oy + kTbT, so);
    tma_store_2d(mUo, 3 * (ox + kTbT), oy + kTbT, su);
    bulk_commit();
}

// The images of one solve, in the order of a problem's tensor maps: the five
// loaded per tile (O, U, A, consWt, lap P; tile box) and the two stored
// (O, U; interior box).
enum { kMapO, kMapU, kMapA, kMapW, kMapL, kMapOo, kMapUo, kMaps };

constexpr int kGroupMax = 16;  // images of a grouped solve's launch

// One launch of a persistent kernel on interleaved images, kN of any sizes (one
// per video of a grouped solve): each one's tensor maps, size and first tile in
// the launch's list.  Passed by value as a __grid_constant__ parameter, so the
// maps stay in parameter memory, where TMA reads them.
template <int kN>
struct SolverLaunch {
    CUtensorMap map[kN][kMaps];
    int w[kN], h[kN], tiles_x[kN];
    int tile0[kN + 1];  // first tile of image p; tile0[count] = tiles in all
    uint8_t* rgba[kN];  // RGBA8 output of the last launch, or null
    int count;
};

struct TileLoc {
    int p;       // image
    int ox, oy;  // tile origin (ring included)
};

template <int kRows, int kN>
__device__ __forceinline__ TileLoc locate(const SolverLaunch<kN>& g, int tile)
{
    int p = 0;
    if (kN > 1) {
#pragma unroll 1
        while (p + 1 < g.count && tile >= g.tile0[p + 1])
            ++p;
    }
    const int t = tile - g.tile0[p];
    return TileLoc{p, (t % g.tiles_x[p]) * kIW - kTbT, (t / g.tiles_x[p]) * kRows - kTbT};
}

// input tiles first .. last - 1 (map order) of a tile at (ox, oy), into consecutive stages
__device__ __forceinline__ void issue_tile_loads(float* stage, const CUtensorMap* m, int ox, int oy, int stage_floats,
    int first, int last, uint64_t* bar)
{
    for (int i = first; i < last; ++i)
        tma_load_2d(stage + i * stage_floats, m + i, 3 * ox, oy, bar);
}

// the five input tiles of a tile at (ox, oy), `bytes` each, into consecutive stages
__device__ __forceinline__ void issue_loads(float* stage, const CUtensorMap* m, int ox, int oy, int stage_floats,
    uint32_t bytes, uint64_t* bar)
{
    mbar_expect_tx(bar, 5 * bytes);
    issue_tile_loads(stage, m, ox, oy, stage_floats, kMapO, kMapL + 1, bar);
}

// The first tile of a launch.  A, consWt and lap P are not written by solver
// launches, so a launch after the first of a solve (k0 > 0: its predecessor
// is the previous solver launch, which itself waited for the kernels that
// wrote them) fetches them before waiting for the predecessor to complete;
// O and U, which the predecessor writes, after.
__device__ __forceinline__ void issue_first_loads(float* stage, const CUtensorMap* m, int ox, int oy,
    int stage_floats, uint32_t bytes, uint64_t* bar, bool early)
{
    if (early) {
        mbar_expect_tx(bar, 5 * bytes);
        issue_tile_loads(stage, m, ox, oy, stage_floats, kMapA, kMapL + 1, bar);
    }
    grid_dependency_wait();
    if (early)
        issue_tile_loads(stage, m, ox, oy, stage_floats, kMapO, kMapU + 1, bar);
    else
        issue_loads(stage, m, ox, oy, stage_floats, bytes, bar);
}

template <int kN>
__global__ void __launch_bounds__(kTbEX / 2 * kTbEY / 2, 1)
    solver_persistent_kernel(const __grid_constant__ SolverLaunch<kN> g, int T, int k0, float step, float mom)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* stage = reinterpret_cast<float*>(smem_raw);
    float* obuf = stage + 5 * kStageFloats;
    uint64_t* bar = reinterpret_cast<uint64_t*>(obuf + 2 * 3 * kTbPlane);
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * 32 + tx;
    const int px0 = 2 * tx, py0 = 2 * ty;

    for (int i = tid; i < 2 * 3 * kTbPlane; i += blockDim.x * blockDim.y)
        obuf[i] = 0.0f;
    if (tid == 0)
        mbar_init(bar, 1);
    __syncthreads();
    const int ntiles = g.tile0[g.count];
    int tile = blockIdx.x;
    if (tid == 0 && tile < ntiles) {
        const TileLoc n = locate<kIH>(g, tile);
        issue_first_loads(stage, g.map[n.p], n.ox, n.oy, kStageFloats, kStageBytes, bar, k0 > 0);
    }
    grid_dependency_wait();
    uint32_t parity = 0;
    for (; tile < ntiles; tile += gridDim.x) {
        if (tile + static_cast<int>(gridDim.x) >= ntiles)
            allow_dependent_launch();
        const TileLoc c = locate<kIH>(g, tile);
        const int ox = c.ox, oy = c.oy, w = g.w[c.p], h = g.h[c.p];
        if (!mbar_wait_bounded(bar, parity, kWaitSpins)) {
            // the outputs are invalid and vsc_check_device reports VSC_ETIMEOUT; the
            // second bounded wait gives copies still in flight a chance to land
            // before the CTA exits
            if (tid == 0) {
                atomicExch(&g_device_timeout, 1);
                bulk_wait_all();
            }
            mbar_wait_bounded(bar, parity, kWaitSpins);
            return;
        }
        parity ^= 1;

        TbState s;
        float cnt[4];
        bool vr[4], vl[4], vd[4], vu[4], inimg[4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = py0 + r;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int q = 2 * r + c;
                const int gx = ox + px0 + c, gy = oy + row;
                inimg[q] = gx >= 0 && gx < w && gy >= 0 && gy < h;
                vr[q] = (gx + 1) < (w - 1);
                vl[q] = (gx - 1) >= 0;
                vd[q] = (gy + 1) < (h - 1);
                vu[q] = (gy - 1) >= 0;
                cnt[q] = static_cast<float>(static_cast<int>(vr[q]) + static_cast<int>(vl[q]) +
                                            static_cast<int>(vd[q]) + static_cast<int>(vu[q]));
            }
            // six consecutive floats: both pixels' RGB (TMA zero-fills outside the image)
            float(*dst[5])[3] = {s.o, s.u, s.a, s.wt, s.lp};
#pragma unroll
            for (int arr = 0; arr < 5; ++arr) {
                const float* src = stage + arr * kStageFloats + row * (3 * kTbEX) + 3 * px0;
                const float2 v01 = *reinterpret_cast<const float2*>(src);
                const float2 v23 = *reinterpret_cast<const float2*>(src + 2);
                const float2 v45 = *reinterpret_cast<const float2*>(src + 4);
                float* p0 = dst[arr][2 * r];
                float* p1 = dst[arr][2 * r + 1];
                p0[0] = v01.x;
                p0[1] = v01.y;
                p0[2] = v23.x;
                p1[0] = v23.y;
                p1[1] = v45.x;
                p1[2] = v45.y;
            }
        }
        if (tid == 0)
            bulk_wait_read();  // the previous tile's TMA stores have read the staging
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int ch = 0; ch < 3; ++ch)
                *reinterpret_cast<float2*>(&obuf[ch * kTbPlane + (py0 + r + 1) * kTbPX + px0 + 2]) =
                    make_float2(s.o[2 * r][ch], s.o[2 * r + 1][ch]);
        __syncthreads();  // staging consumed, O published
        if (tid == 0 && tile + static_cast<int>(gridDim.x) < ntiles) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const TileLoc n = locate<kIH>(g, tile + gridDim.x);
            issue_loads(stage, g.map[n.p], n.ox, n.oy, kStageFloats, kStageBytes, bar);
        }

        const bool interior = ox >= 1 && oy >= 1 && ox + kTbEX - 1 <= w - 3 && oy + kTbEY - 1 <= h - 3;
        if (interior)
            tb_iterate<true>(s, vr, vl, vd, vu, cnt, obuf, T, kTbT, k0, step, mom, px0, py0);
        else
            tb_iterate<false>(s, vr, vl, vd, vu, cnt, obuf, T, kTbT, k0, step, mom, px0, py0);

        // interior out: the edge-row buffers are idle until the next tile's publish;
        // a thread's two pixels of a row are six consecutive floats
        float* so = obuf;
        float* su = obuf + kIH * 3 * kIW;
        {
            const int ix = px0 - kTbT;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int iy = py0 + r - kTbT;
                if (ix < 0 || ix >= kIW || iy < 0 || iy >= kIH)
                    continue;
                float2* o2 = reinterpret_cast<float2*>(so + iy * 3 * kIW + 3 * ix);
                float2* u2 = reinterpret_cast<float2*>(su + iy * 3 * kIW + 3 * ix);
                const float* a = s.o[2 * r];
                const float* b = s.o[2 * r + 1];
                o2[0] = make_float2(a[0], a[1]);
                o2[1] = make_float2(a[2], b[0]);
                o2[2] = make_float2(b[1], b[2]);
                const float* c = s.u[2 * r];
                const float* d = s.u[2 * r + 1];
                u2[0] = make_float2(c[0], c[1]);
                u2[1] = make_float2(c[2], d[0]);
                u2[2] = make_float2(d[1], d[2]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0)
            store_interior(g.map[c.p] + kMapOo, g.map[c.p] + kMapUo, ox, oy, so, su);
        if (uint8_t* rgba = g.rgba[c.p]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int px = px0 + (q & 1), py = py0 + (q >> 1);
                if (!inimg[q] || px < kTbT || px >= kTbEX - kTbT || py < kTbT || py >= kTbEY - kTbT)
                    continue;
                reinterpret_cast<uint32_t*>(rgba)[pix_index(ox + px, oy + py, w)] =
                    pack_rgba(s.o[q][0], s.o[q][1], s.o[q][2]);
            }
        }
        // the TMA stores read the staging while the next tile's copies land
    }
    if (tid == 0)
        bulk_wait_all();
}

// ---- persistent, TMA-fed solver on 64 x 48 tiles of 2 x 4 pixel blocks -------------
// Same per-pixel arithmetic as the kernels above, on a taller tile: 12 warps,
// each thread a 2-column x 4-row block (its vertical neighbours inside the
// block are its own registers), so 48 rows fit in the register budget of
// 384 threads and the interior after the 8-pixel ring is 48 x 32 (50 % of
// the tile instead of 37.5 %).  Only the top and bottom row of each warp
// are read by other warps; they are published to a compact double-buffered
// array of "slots" (slot w + 1 holds warp w's two edge rows, slots 0 and 13
// are zero aprons).  Half the shared-memory traffic per pixel of the 2 x 2
// blocking, the same shuffles per pixel.
constexpr int kPWarps = 12;
constexpr int kPThreads = 32 * kPWarps;
constexpr int kPEY = 4 * kPWarps;            // 48 tile rows
constexpr int kPIH = kPEY - 2 * kTbT;        // 32 interior rows
constexpr int kPStageFloats = kPEY * kTbEX * 3;
constexpr int kPStageBytes = kPStageFloats * static_cast<int>(sizeof(float));
constexpr int kPSlots = kPWarps + 2;
constexpr int kPPlane = kPSlots * 2 * kTbPX;  // one channel of one buffer
constexpr int kPObuf = 2 * 3 * kPPlane;
constexpr int kPSmem = 5 * kPStageBytes + kPObuf * static_cast<int>(sizeof(float)) + 16;
static_assert(kPSmem <= 232448, "dynamic shared memory per CTA");
static_assert(kPObuf >= 2 * kPIH * 3 * kIW && 2 * 3 * kTbPlane >= 2 * kIH * 3 * kIW,
    "the edge-row buffers hold a tile's interior O and U");
static_assert((kPIH * 3 * kIW * 4) % 128 == 0 && (kIH * 3 * kIW * 4) % 128 == 0 &&
    (5 * kPStageBytes) % 128 == 0 && (5 * kStageBytes) % 128 == 0, "TMA store sources on the 128-byte grid");
static_assert(2 * kTbT < kPEY, "tile too small for the iteration count");

struct P8State {
    float o[8][3], u[8][3], a[8][3], wt[8][3], lp[8][3];  // [pixel q = 2 * row + col][channel]
};

// validity of a pixel's four neighbours in the reference's rule (border tiles only)
struct Nb {
    bool vr, vl, vd, vu;
    float cnt;
};
__device__ __forceinline__ Nb nb_of(int gx, int gy, int w, int h)
{
    Nb n;
    n.vr = (gx + 1) < (w - 1);
    n.vl = (gx - 1) >= 0;
    n.vd = (gy + 1) < (h - 1);
    n.vu = (gy - 1) >= 0;
    n.cnt = static_cast<float>(static_cast<int>(n.vr) + static_cast<int>(n.vl) + static_cast<int>(n.vd) +
                               static_cast<int>(n.vu));
    return n;
}

template <bool kAll>
__device__ __forceinline__ void p8_step(P8State& s, float* obuf, int cur, bool mom_on, float step, float mom, int px0,
    int warp, int gx0, int gy0, int w, int h)
{
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const float* S = obuf + (cur * 3 + ch) * kPPlane;
        const float2 up = *reinterpret_cast<const float2*>(&S[(warp * 2 + 1) * kTbPX + px0 + 2]);   // slot w, row 1
        const float2 dn = *reinterpret_cast<const float2*>(&S[((warp + 2) * 2) * kTbPX + px0 + 2]);  // slot w+2, row 0
        float ol[4], orr[4], L[4], R[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            ol[r] = s.o[2 * r][ch];
            orr[r] = s.o[2 * r + 1][ch];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            L[r] = __shfl_up_sync(0xffffffffu, orr[r], 1);
            R[r] = __shfl_down_sync(0xffffffffu, ol[r], 1);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float ul = r == 0 ? up.x : ol[r - 1], ur = r == 0 ? up.y : orr[r - 1];
            const float dl = r == 3 ? dn.x : ol[r + 1], dr = r == 3 ? dn.y : orr[r + 1];
            Nb a{true, true, true, true, 4.0f}, b{true, true, true, true, 4.0f};
            if (!kAll) {
                a = nb_of(gx0, gy0 + r, w, h);
                b = nb_of(gx0 + 1, gy0 + r, w, h);
            }
            const int ql = 2 * r, qr = 2 * r + 1;
            s.o[ql][ch] = jacobi_px<kAll>(ol[r], s.u[ql][ch], s.a[ql][ch], s.wt[ql][ch], s.lp[ql][ch], orr[r], L[r], dl,
                ul, a.vr, a.vl, a.vd, a.vu, a.cnt, step, mom, mom_on);
            s.o[qr][ch] = jacobi_px<kAll>(orr[r], s.u[qr][ch], s.a[qr][ch], s.wt[qr][ch], s.lp[qr][ch], R[r], ol[r],
                dr, ur, b.vr, b.vl, b.vd, b.vu, b.cnt, step, mom, mom_on);
        }
        float* D = obuf + ((cur ^ 1) * 3 + ch) * kPPlane + ((warp + 1) * 2) * kTbPX + px0 + 2;
        *reinterpret_cast<float2*>(D) = make_float2(s.o[0][ch], s.o[1][ch]);            // top row
        *reinterpret_cast<float2*>(D + kTbPX) = make_float2(s.o[6][ch], s.o[7][ch]);    // bottom row
    }
}

// Iteration k is needed on rows [ring - T + k + 1, kPEY - ring + T - k - 1);
// a warp (four rows) outside that range skips it (the argument of tb_iterate).
template <bool kAll>
__device__ __forceinline__ void p8_iterate(P8State& s, float* obuf, int T, int k0, float step, float mom, int px0,
    int warp, int gx0, int gy0, int w, int h)
{
    const int r0 = 4 * warp;
    if (T == kTbT) {
        // full launches, unrolled; momentum is off only in the first step of a solve
        const bool later = k0 > 0;
#pragma unroll
        for (int k = 0; k < kTbT; ++k) {
            if (!(r0 + 3 < k + 1 || r0 >= kPEY - k - 1))
                p8_step<kAll>(s, obuf, k & 1, k > 0 || later, step, mom, px0, warp, gx0, gy0, w, h);
            __syncthreads();
        }
        return;
    }
    for (int k = 0; k < T; ++k) {
        const int lo = kTbT - T + k + 1, hi = kPEY - kTbT + T - k - 1;
        if (!(r0 + 3 < lo || r0 >= hi))
            p8_step<kAll>(s, obuf, k & 1, (k0 + k) > 0, step, mom, px0, warp, gx0, gy0, w, h);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kPThreads, 1)
    solver_tall_kernel(const __grid_constant__ SolverLaunch<1> g, int T, int k0, float step, float mom)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* stage = reinterpret_cast<float*>(smem_raw);
    float* obuf = stage + 5 * kPStageFloats;
    uint64_t* bar = reinterpret_cast<uint64_t*>(obuf + kPObuf);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int px0 = 2 * lane, py0 = 4 * warp;

    for (int i = threadIdx.x; i < kPObuf; i += kPThreads)
        obuf[i] = 0.0f;  // the apron slots stay zero
    if (threadIdx.x == 0)
        mbar_init(bar, 1);
    __syncthreads();
    const int ntiles = g.tile0[g.count];
    int tile = blockIdx.x;
    if (threadIdx.x == 0 && tile < ntiles) {
        const TileLoc n = locate<kPIH>(g, tile);
        issue_first_loads(stage, g.map[n.p], n.ox, n.oy, kPStageFloats, kPStageBytes, bar, k0 > 0);
    }
    grid_dependency_wait();
    uint32_t parity = 0;
    for (; tile < ntiles; tile += gridDim.x) {
        if (tile + static_cast<int>(gridDim.x) >= ntiles)
            allow_dependent_launch();
        const TileLoc c = locate<kPIH>(g, tile);
        const int ox = c.ox, oy = c.oy, w = g.w[c.p], h = g.h[c.p];
        if (!mbar_wait_bounded(bar, parity, kWaitSpins)) {
            // the outputs are invalid and vsc_check_device reports VSC_ETIMEOUT; the
            // second bounded wait gives copies still in flight a chance to land
            // before the CTA exits
            if (threadIdx.x == 0) {
                atomicExch(&g_device_timeout, 1);
                bulk_wait_all();
            }
            mbar_wait_bounded(bar, parity, kWaitSpins);
            return;
        }
        parity ^= 1;

        P8State s;
        float(*dst[5])[3] = {s.o, s.u, s.a, s.wt, s.lp};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            // six consecutive floats: both pixels' RGB (TMA zero-fills outside the image)
#pragma unroll
            for (int arr = 0; arr < 5; ++arr) {
                const float* src = stage + arr * kPStageFloats + (py0 + r) * (3 * kTbEX) + 3 * px0;
                const float2 v01 = *reinterpret_cast<const float2*>(src);
                const float2 v23 = *reinterpret_cast<const float2*>(src + 2);
                const float2 v45 = *reinterpret_cast<const float2*>(src + 4);
                float* p0 = dst[arr][2 * r];
                float* p1 = dst[arr][2 * r + 1];
                p0[0] = v01.x;
                p0[1] = v01.y;
                p0[2] = v23.x;
                p1[0] = v23.y;
                p1[1] = v45.x;
                p1[2] = v45.y;
            }
        }
        if (threadIdx.x == 0)
            bulk_wait_read();  // the previous tile's TMA stores have read the staging
        __syncthreads();
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            float* D = obuf + ch * kPPlane + ((warp + 1) * 2) * kTbPX + px0 + 2;  // buffer 0
            *reinterpret_cast<float2*>(D) = make_float2(s.o[0][ch], s.o[1][ch]);
            *reinterpret_cast<float2*>(D + kTbPX) = make_float2(s.o[6][ch], s.o[7][ch]);
        }
        __syncthreads();  // staging consumed, edge rows published
        if (threadIdx.x == 0 && tile + static_cast<int>(gridDim.x) < ntiles) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const TileLoc n = locate<kPIH>(g, tile + gridDim.x);
            issue_loads(stage, g.map[n.p], n.ox, n.oy, kPStageFloats, kPStageBytes, bar);
        }

        const int gx0 = ox + px0, gy0 = oy + py0;
        const bool interior = ox >= 1 && oy >= 1 && ox + kTbEX - 1 <= w - 3 && oy + kPEY - 1 <= h - 3;
        if (interior)
            p8_iterate<true>(s, obuf, T, k0, step, mom, px0, warp, gx0, gy0, w, h);
        else
            p8_iterate<false>(s, obuf, T, k0, step, mom, px0, warp, gx0, gy0, w, h);

        // interior out: the edge-row slots are idle until the next tile's publish;
        // a thread's two pixels of a row are six consecutive floats (the
        // interior starts at an even column, so both or neither are inside)
        float* so = obuf;
        float* su = obuf + kPIH * 3 * kIW;
        {
            const int ix = px0 - kTbT;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int iy = py0 + r - kTbT;
                if (ix < 0 || ix >= kIW || iy < 0 || iy >= kPIH)
                    continue;
                float2* o2 = reinterpret_cast<float2*>(so + iy * 3 * kIW + 3 * ix);
                float2* u2 = reinterpret_cast<float2*>(su + iy * 3 * kIW + 3 * ix);
                const float* a = s.o[2 * r];
                const float* b = s.o[2 * r + 1];
                o2[0] = make_float2(a[0], a[1]);
                o2[1] = make_float2(a[2], b[0]);
                o2[2] = make_float2(b[1], b[2]);
                const float* c = s.u[2 * r];
                const float* d = s.u[2 * r + 1];
                u2[0] = make_float2(c[0], c[1]);
                u2[1] = make_float2(c[2], d[0]);
                u2[2] = make_float2(d[1], d[2]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0)
            store_interior(g.map[c.p] + kMapOo, g.map[c.p] + kMapUo, ox, oy, so, su);
        if (uint8_t* rgba = g.rgba[c.p]) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int px = px0 + (q & 1), py = py0 + (q >> 1);
                const int gx = ox + px, gy = oy + py;
                if (gx < 0 || gx >= w || gy < 0 || gy >= h || px < kTbT || px >= kTbEX - kTbT || py < kTbT ||
                    py >= kPEY - kTbT)
                    continue;
                reinterpret_cast<uint32_t*>(rgba)[pix_index(gx, gy, w)] =
                    pack_rgba(s.o[q][0], s.o[q][1], s.o[q][2]);
            }
        }
        // the TMA stores read the staging while the next tile's copies land; the
        // next tile waits for those reads before it publishes its edge rows
    }
    if (threadIdx.x == 0)
        bulk_wait_all();
}

// ---- FMA form of the solver ---------------------------------------------------
// kernel_consist_out's step, g = (lap O - lap P) - w (O - A), O' = O + s g
// (+ m U), U' = s g, regrouped around two per-pixel constants computed once
// per solve (solver_prep_kernel):
//   Cs = s * fma(w, A, -lap P),   nK = -(s * (cnt + w))   (cnt = valid neighbours),
// so that one step is
//   S = (left + right) + (up + down),  g = fma(nK, O, fma(s, S, Cs)),
//   O' = O + g, then O' = fma(m, U, O') after the first step,  U' = g,
// with invalid neighbours read as +0: seven FP32 operations per pixel and
// channel against twelve in the reference expression.  The rounding differs
// from the reference form's, so results agree with it within a tolerance
// (and with the restatement's FMA form, vo_consist_out_fma, bit for bit).
//
// The three colour channels of the step never interact, so the form solves
// each channel as its own image: the workspace holds O, U, Cs and nK as
// planes (channel-major, planar_group_kernel converts O at the ends of a
// solve).  A tile is 128 x 72 pixels of one plane: each of 256 threads keeps a
// 4-column x 9-row block of O, U, Cs and nK in registers (144 floats), a warp
// spans the tile's width, so the 8-pixel ring of the temporal blocking leaves
// a 112 x 56 interior (68 % of the tile), horizontal neighbours cost two
// shuffles per row for four pixels, and each warp publishes its top and
// bottom row as two 16-byte stores per thread.

// Cs = step * fma(wt, A, -lap P) and nK = -(step * (cnt + wt)) as planes
// (lap P, cnt as lap_pr_kernel computes them); with O non-null, also O as
// planes into Op, or with Oc non-null the cw x ch image Oc upsampled to w x h
// as kernel_bilinear does (bilinear_px: the pyramid's initial solution of
// this level, written straight into the planes); with cnt non-null, the ncnt
// solve counters zeroed.  The exact form's constants: lap P in Cs, wt in nK, A
// in Ap.
template <int kForm>
__global__ void solver_prep_kernel(const float* __restrict__ P, const float* __restrict__ A,
    const float* __restrict__ Wt, const float* __restrict__ O, float* __restrict__ Cs, float* __restrict__ nK,
    float* __restrict__ Ap, float* __restrict__ Op, int w, int h, int pitch, float step, unsigned* __restrict__ cnt, int ncnt,
    const float* __restrict__ Oc, int cw, int ch)
{
    pdl_enter();
    if (cnt && blockIdx.x == 0 && blockIdx.y == 0)  // the solve kernel's counters start at zero
        for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < ncnt; i += blockDim.x * blockDim.y)
            cnt[i] = 0;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h)
        return;
    const int64_t i0 = pix_index(x, y, w) * 3;
    const int64_t rs = static_cast<int64_t>(w) * 3;
    const int64_t plane = static_cast<int64_t>(pitch) * h;
    const int64_t q = pix_index(x, y, pitch);
    float up[3];
    if (Oc)
        bilinear_px(Oc, cw, ch, w, h, 3, x, y, up);
    for (int c = 0; c < 3; ++c) {
        const int64_t i = i0 + c;
        int cnt = 0;
        float lap = 0.0f;
        if ((x + 1) < (w - 1)) {
            lap += P[i + 3];
            cnt += 1;
        }
        if ((x - 1) >= 0) {
            lap += P[i - 3];
            cnt += 1;
        }
        if ((y + 1) < (h - 1)) {
            lap += P[i + rs];
            cnt += 1;
        }
        if ((y - 1) >= 0) {
            lap += P[i - rs];
            cnt += 1;
        }
        lap = __fsub_rn(lap, __fmul_rn(static_cast<float>(cnt), P[i]));
        const float wt = Wt[i];
        if (kForm == kSolverFma) {
            Cs[c * plane + q] = __fmul_rn(step, __fmaf_rn(wt, A[i], -lap));
            nK[c * plane + q] = -__fmul_rn(step, __fadd_rn(static_cast<float>(cnt), wt));
        } else {
            Cs[c * plane + q] = lap;
            nK[c * plane + q] = wt;
            Ap[c * plane + q] = A[i];
        }
        if (Oc)
            Op[c * plane + q] = up[c];
        else if (O)
            Op[c * plane + q] = O[i];
    }
}

// Interleaved <-> planar copies of the images of up to kPlanarGroupMax solves
// (one launch per level of a multi-stream step): to_planar = 1 reads the
// interleaved src and writes dst as planes of `pitch`-float rows; 0 the reverse, and writes the
// RGBA8 copy when rgba is non-null.
constexpr int kPlanarGroupMax = 16;
struct PlanarGroup {
    const float* src[kPlanarGroupMax];
    float* dst[kPlanarGroupMax];
    uint8_t* rgba[kPlanarGroupMax];
    unsigned* cnt[kPlanarGroupMax];  // solve counters zeroed on the way in, or null
    int ncnt[kPlanarGroupMax];
    int64_t npix[kPlanarGroupMax];
    int w[kPlanarGroupMax], pitch[kPlanarGroupMax];  // of an image row, of a plane's row
    int64_t plane[kPlanarGroupMax];                  // floats of a plane
    int block0[kPlanarGroupMax + 1];
    int count;
};

__global__ void __launch_bounds__(256) planar_group_kernel(const __grid_constant__ PlanarGroup g, int to_planar)
{
    pdl_enter();
    int p = 0;
    while (p + 1 < g.count && static_cast<int>(blockIdx.x) >= g.block0[p + 1])
        ++p;
    if (g.cnt[p] && static_cast<int>(blockIdx.x) == g.block0[p])
        for (int k = threadIdx.x; k < g.ncnt[p]; k += blockDim.x)
            g.cnt[p][k] = 0;
    const int64_t i = static_cast<int64_t>(blockIdx.x - g.block0[p]) * blockDim.x + threadIdx.x;
    const int64_t n = g.npix[p];
    if (i >= n)
        return;
    const int64_t pl = g.plane[p];
    int64_t q = i;  // the pixel's place in a plane
    if (g.pitch[p] != g.w[p])
        q += (n < (int64_t{1} << 31) ? static_cast<int>(i) / g.w[p] : i / g.w[p]) * (g.pitch[p] - g.w[p]);
    if (to_planar) {
        const float* s = g.src[p] + i * 3;
        g.dst[p][q] = s[0];
        g.dst[p][pl + q] = s[1];
        g.dst[p][2 * pl + q] = s[2];
        return;
    }
    const float r = g.src[p][q], gg = g.src[p][pl + q], b = g.src[p][2 * pl + q];
    float* d = g.dst[p] + i * 3;
    d[0] = r;
    d[1] = gg;
    d[2] = b;
    if (g.rgba[p])
        reinterpret_cast<uint32_t*>(g.rgba[p])[i] = pack_rgba(r, gg, b);
}

template <int kCfg>
struct PlState {
    static constexpr int kR = PlGeo<kCfg>::kRPT;
    float4 o[kR], u[kR], c[kR], nk[kR];  // [row] = (column 0 .. 3); exact form: c = lap P, nk = consWt
    float4 a[!PlGeo<kCfg>::kFma ? kR : 1];
};

__device__ __forceinline__ float& f4(float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }
__device__ __forceinline__ float f4c(const float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

// The columns left and right of a thread's block, from the neighbouring lanes
// (the outer lanes keep their own value: the tile's outer columns never reach
// the interior).
template <int kCfg>
struct PlSides {
    float l[PlGeo<kCfg>::kRPT], r[PlGeo<kCfg>::kRPT];
};

// One step of row r of a thread's block: the new row in `on`, U in place;
// then the lanes exchange the new row's end columns for the next step.
template <int kCfg, int kMode>
__device__ __forceinline__ void pl_row(PlState<kCfg>& s, PlSides<kCfg>& x, float4* on, int r, float4 up, float4 dn,
    float step, float mom, const PlPlace& t)
{
    using G = PlGeo<kCfg>;
    const float4 o = s.o[r];
    float4 u = r == 0 ? up : s.o[r - 1];
    float4 d = r == G::kRPT - 1 ? dn : s.o[r + 1];
    constexpr bool kFixed = kMode == kPlLanes || kMode == kPlCols;
    float cnt_rows = 4.0f;  // exact form: left, right and the valid ones of up and down
    if ((kFixed && r == G::kTopRow && t.zt) || (kMode == kPlEvery && r == t.top)) {
        u = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        cnt_rows -= 1.0f;
    }
    if ((kFixed && ((r == G::kBot2Row && t.zb2) || (r == G::kBot1Row && t.zb1))) || (kMode == kPlEvery && r >= t.bot)) {
        d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        cnt_rows -= 1.0f;
    }
    float lft = x.l[r], rgt = x.r[r], o3 = o.w;  // left of column 0, right of columns 3 and 2
    if (kMode != kPlAll)
        lft = t.zl ? 0.0f : lft;
    if (kMode == kPlLanes) {
        rgt = t.zr ? 0.0f : rgt;
        o3 = t.zr ? 0.0f : o3;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float left = j == 0 ? lft : f4c(o, j - 1);
        float right = j == 3 ? rgt : (j == 2 ? o3 : f4c(o, j + 1));
        if (kMode == kPlCols || kMode == kPlEvery)
            right = j < t.xlim ? right : 0.0f;
        const float oj = f4c(o, j);
        float g;
        if (G::kFma) {
            g = __fmaf_rn(f4c(s.nk[r], j), oj,
                __fmaf_rn(step, __fadd_rn(__fadd_rn(left, right), __fadd_rn(f4c(u, j), f4c(d, j))), f4c(s.c[r], j)));
            f4(on[r], j) = __fmaf_rn(mom, f4c(s.u[r], j), __fadd_rn(oj, g));
        } else {
            // jacobi_px's expression; where a neighbour is read as +0, cnt of the
            // valid ones times o is rounded before the subtraction, as there
            float lap = __fadd_rn(__fadd_rn(__fadd_rn(right, left), f4c(d, j)), f4c(u, j));
            if (kMode == kPlAll) {
                lap = __fmaf_rn(-4.0f, oj, lap);
            } else {
                const bool vr = kMode == kPlLanes ? !(j >= 2 && t.zr) : j < t.xlim;
                const float cnt = cnt_rows - (vr ? 0.0f : 1.0f) - (j == 0 && t.zl ? 1.0f : 0.0f);
                lap = __fsub_rn(lap, __fmul_rn(cnt, oj));
            }
            const float d1 = __fmul_rn(f4c(s.nk[r], j), __fsub_rn(oj, f4c(s.a[r], j)));
            g = __fmul_rn(step, __fsub_rn(__fsub_rn(lap, f4c(s.c[r], j)), d1));
            f4(on[r], j) = __fadd_rn(__fadd_rn(oj, g), __fmul_rn(mom, f4c(s.u[r], j)));
        }
        f4(s.u[r], j) = g;
    }
    x.l[r] = __shfl_up_sync(0xffffffffu, on[r].w, 1);
    x.r[r] = __shfl_down_sync(0xffffffffu, on[r].x, 1);
}

// One step of a thread's block; `up` and `dn` are the previous iterate's rows
// above and below it.  The rows between go first, while those two arrive; each
// row's shuffles for the next step run beside the following rows' arithmetic.
template <int kCfg, int kMode>
__device__ __forceinline__ void pl_step(PlState<kCfg>& s, PlSides<kCfg>& x, float4 up, float4 dn, float step,
    float mom, const PlPlace& t)
{
    constexpr int kR = PlGeo<kCfg>::kRPT;
    float4 on[kR];
#pragma unroll
    for (int q = 0; q < kR; ++q)
        pl_row<kCfg, kMode>(s, x, on, q < kR - 2 ? q + 1 : (q == kR - 2 ? 0 : kR - 1), up, dn, step, mom, t);
#pragma unroll
    for (int r = 0; r < kR; ++r)
        s.o[r] = on[r];
}

// The steps of one tile's round.  After each step a warp publishes its top and
// bottom row to a slot buffer (slot w + 1 is warp w's; even steps write buffer
// 0 and odd ones buffer 1) and bar() joins the warps; `up` and `dn` are the
// rows above and below the thread's block in the initial iterate.
//
// The steps of a full round are a loop of two: unrolled to eight, its code (24
// KB a test mode) missed the instruction cache for 10 % of the warps' time,
// and with a condition in it (momentum off in a solve's first step, steps left
// out) the two steps' registers meet in moves.  A solve's first step has U = +0
// and takes mom = -0: fma(-0, +0, n) is n, whatever n is.
template <int kCfg, int kMode, class Bar>
__device__ __forceinline__ void pl_steps(PlState<kCfg>& s, float4 up, float4 dn, float* slots, int T, int k0,
    float step, float mom, int lane, int warp, const PlPlace& t, Bar&& bar)
{
    using G = PlGeo<kCfg>;
    PlSides<kCfg> x;
#pragma unroll
    for (int r = 0; r < G::kRPT; ++r) {
        x.l[r] = __shfl_up_sync(0xffffffffu, s.o[r].w, 1);
        x.r[r] = __shfl_down_sync(0xffffffffu, s.o[r].x, 1);
    }
    float* const top = slots + ((warp + 1) * 2) * kPlW + 4 * lane;  // slot of this warp: top row, bottom row
    auto exchange = [&](float* b) {
        *reinterpret_cast<float4*>(b) = s.o[0];
        *reinterpret_cast<float4*>(b + kPlW) = s.o[G::kRPT - 1];
        bar();
        up = *reinterpret_cast<const float4*>(b - kPlW);      // slot w, bottom row
        dn = *reinterpret_cast<const float4*>(b + 2 * kPlW);  // slot w + 2, top row
    };
    float m = k0 > 0 ? mom : -0.0f;
#pragma unroll 1
    for (int k = 0; k + 1 < T; k += 2) {
        pl_step<kCfg, kMode>(s, x, up, dn, step, m, t);
        exchange(top);
        pl_step<kCfg, kMode>(s, x, up, dn, step, mom, t);
        exchange(top + G::kSlots);
        m = mom;
    }
    if (T & 1)  // a short last round
        pl_step<kCfg, kMode>(s, x, up, dn, step, m, t);
}

template <int kCfg, class Bar>
__device__ __forceinline__ void pl_round(int mode, PlState<kCfg>& s, float4 up, float4 dn, float* slots, int T,
    int k0, float step, float mom, int lane, int warp, const PlPlace& t, Bar&& bar)
{
    if (mode == kPlAll)
        pl_steps<kCfg, kPlAll>(s, up, dn, slots, T, k0, step, mom, lane, warp, t, bar);
    else if (mode == kPlLanes)
        pl_steps<kCfg, kPlLanes>(s, up, dn, slots, T, k0, step, mom, lane, warp, t, bar);
    else if (mode == kPlCols)
        pl_steps<kCfg, kPlCols>(s, up, dn, slots, T, k0, step, mom, lane, warp, t, bar);
    else
        pl_steps<kCfg, kPlEvery>(s, up, dn, slots, T, k0, step, mom, lane, warp, t, bar);
}

// A thread's block out of the staged tile, with the O rows above and below it
// (zero outside the tile: values the ring never passes on to the interior).
template <int kCfg>
__device__ __forceinline__ void pl_take(PlState<kCfg>& s, float4& up, float4& dn, const float* stage, int k0, int lane,
    int warp)
{
    using G = PlGeo<kCfg>;
    const float* base = stage + PlGeo<kCfg>::kRPT * warp * kPlW + 4 * lane;
#pragma unroll
    for (int r = 0; r < PlGeo<kCfg>::kRPT; ++r) {
        const float* row = base + r * kPlW;
        s.o[r] = *reinterpret_cast<const float4*>(row);
        s.u[r] = *reinterpret_cast<const float4*>(row + G::kStage);
        s.nk[r] = *reinterpret_cast<const float4*>(row + 2 * G::kStage);
        s.c[r] = *reinterpret_cast<const float4*>(row + 3 * G::kStage);
        if constexpr (!PlGeo<kCfg>::kFma)
            s.a[r] = *reinterpret_cast<const float4*>(row + 4 * G::kStage);
    }
    if (k0 == 0)  // no U yet
#pragma unroll
        for (int r = 0; r < PlGeo<kCfg>::kRPT; ++r)
            s.u[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    up = dn = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (warp > 0)
        up = *reinterpret_cast<const float4*>(base - kPlW);
    if (warp < G::kWarps - 1)
        dn = *reinterpret_cast<const float4*>(base + PlGeo<kCfg>::kRPT * kPlW);
}

// A thread's interior pixels of O and U into the out staging.
template <int kCfg>
__device__ __forceinline__ void pl_put(const PlState<kCfg>& s, float* so, float* su, int lane, int warp)
{
    using G = PlGeo<kCfg>;
    const int ix = 4 * lane - G::kT;
    if (ix < 0 || ix >= G::kIW)
        return;
#pragma unroll
    for (int r = 0; r < PlGeo<kCfg>::kRPT; ++r) {
        const int iy = PlGeo<kCfg>::kRPT * warp + r - G::kT;
        if (iy < 0 || iy >= PlGeo<kCfg>::kIRows)
            continue;
        *reinterpret_cast<float4*>(so + iy * G::kIW + ix) = s.o[r];
        *reinterpret_cast<float4*>(su + iy * G::kIW + ix) = s.u[r];
    }
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int x, int y, int z, const void* src)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
        "r"(x), "r"(y), "r"(z), "r"(smem_u32(src))
        : "memory");
}

// The planes of one solve for the plain-load form of the kernel (widths that
// are not a multiple of 4, or planes off the 16-byte grid).
struct PlPlain {
    const float *O, *U, *K, *C;
    float *Oo, *Uo;  // (Uo: null in the last round)
    int w, h, tiles_x, ntiles;
};

// Stage <- tile (c, ox, oy) of the four planes, zero outside the image; U (not read
// in a solve's first round) from round 1 on.  Copied asynchronously, 4 bytes at a
// time: through registers, four elements ahead, the eight warps had too few loads
// in flight (854x480, 75 steps 296 us, twelve ahead 271, and 239 so; twelve warps
// of the kernel before, four ahead, 280).
__device__ __forceinline__ void pl_plain_load(float* stage, const PlPlain& p, int c, int ox, int oy, bool with_u)
{
    using G = PlGeo<kSolverFma>;
    const float* src[4] = {p.O, p.U, p.K, p.C};
    const int64_t base = static_cast<int64_t>(c) * p.w * p.h;
#pragma unroll 4
    for (int i = threadIdx.x; i < G::kStage; i += 32 * G::kWarps) {
        const int row = i / kPlW, col = i - row * kPlW;
        const int gy = oy + row, gx = ox + col;
        const bool in = gx >= 0 && gx < p.w && gy >= 0 && gy < p.h;
        const int64_t idx = in ? base + pix_index(gx, gy, p.w) : 0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
            if (a != 1 || with_u)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(stage + a * G::kStage + i)),
                    "l"(src[a] + idx), "r"(in ? 4 : 0)
                    : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The plain-load form (widths that are not a multiple of 4 in a caller's
// workspace, whose planes then have no room for a 16-byte row pitch): one
// launch per round of up to G::kT steps, each CTA walking the round's tiles
// with plain loads and stores.
__global__ void __launch_bounds__(32 * PlGeo<kSolverFma>::kWarps, 1)
    solver_fma_plain_kernel(const __grid_constant__ PlPlain pl, int T, int k0, float step, float mom)
{
    using G = PlGeo<kSolverFma>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* stage = reinterpret_cast<float*>(smem_raw);
    float* slots = stage + 4 * G::kStage;
    float* so = slots + 2 * G::kSlots;
    float* su = so + G::kOut;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    for (int i = threadIdx.x; i < 2 * G::kSlots; i += blockDim.x)
        slots[i] = 0.0f;  // the apron slots stay zero
    grid_dependency_wait();
    const int per_plane = pl.ntiles / 3;
    for (int tile = blockIdx.x; tile < pl.ntiles; tile += gridDim.x) {
        if (tile + static_cast<int>(gridDim.x) >= pl.ntiles)
            allow_dependent_launch();
        const int c = tile / per_plane, r = tile - c * per_plane;
        const int ox = (r % pl.tiles_x) * G::kIW - G::kT, oy = (r / pl.tiles_x) * G::kIRows - G::kT;
        const int w = pl.w, h = pl.h;
        __syncthreads();  // the previous tile has left the staging
        pl_plain_load(stage, pl, c, ox, oy, k0 > 0);
        __syncthreads();
        PlState<kSolverFma> s;
        float4 up, dn;
        pl_take<kSolverFma>(s, up, dn, stage, k0, lane, warp);
        const bool interior = ox >= 1 && oy >= 1 && ox + kPlW - 1 <= w - 3 && oy + G::kRows - 1 <= h - 3;
        pl_round<kSolverFma>(interior ? kPlAll : kPlEvery, s, up, dn, slots, T, k0, step, mom, lane, warp,
            pl_place<kSolverFma>(ox, oy, w, h, lane, warp), [] { __syncthreads(); });
        pl_put<kSolverFma>(s, so, su, lane, warp);
        __syncthreads();
        const int64_t base = static_cast<int64_t>(c) * w * h;
#pragma unroll 4
        for (int i = threadIdx.x; i < G::kOut; i += 32 * G::kWarps) {
            const int iy = i / G::kIW, ix = i - iy * G::kIW;
            const int gy = oy + G::kT + iy, gx = ox + G::kT + ix;
            if (gx < w && gy < h) {
                const int64_t idx = base + pix_index(gx, gy, w);
                pl.Oo[idx] = so[i];
                if (pl.Uo)
                    pl.Uo[idx] = su[i];
            }
        }
    }
}

// ---- a solve in one persistent launch -------------------------------------------
// A solve of L launches' worth of 8-step rounds over N tiles is one kernel:
// each CTA takes (round k, tile t) tickets in order from a global counter
// (k = ticket / N, t = ticket % N), waits until the tile's 3x3 neighbourhood
// has finished round k - 1 (per-tile counters of finished rounds, released
// after the tile's TMA stores complete), runs the tile's steps and signals
// its counter.  Round k reads O[k & 1], U[k & 1] and writes O[(k + 1) & 1],
// U[(k + 1) & 1]; waiting for the neighbours' round k - 1 orders both the
// reads of round k after those writes and the writes of round k after the
// neighbours' round-(k - 1) reads of the same buffer region.  A ticket only
// waits for earlier tickets, whose CTAs already run, so the order cannot
// deadlock whatever else occupies the GPU; every wait is bounded all the
// same.  Rounds overlap: a CTA moves on to round k + 1 while the last tiles of
// round k finish elsewhere, which removes the per-launch tail (1,080 tiles
// per round at 1920x1080 leave the eighth of eight rounds 11 % full) and the
// launch boundaries.
//
// The compute warps only run steps: they wait for a tile's data, take it into
// registers, hand the staging back, iterate, and put the interior into the
// out staging.  Two control warps do the rest, overlapping it with the steps.
// One takes and decodes tickets, watches the neighbours' counters (nine lanes,
// one look per L2 round trip), and loads the next tile as soon as the staging
// is free and its neighbours are done.  The other stores a finished interior
// and publishes its round when the stores are complete.  With that work in a
// compute warp's idle steps the counters were looked at three times a tile, a
// tile whose neighbours were late was loaded only after the tile before it,
// its nine counters read one after the other, and a finished tile was
// published at the end of the next one.
//
// An FMA tile takes 4.6 us at 1920x1080: 6,500 cycles of steps (4,030 of FP32
// issue; the exchange between warps and two warps a scheduler the rest), 2,100
// of moving 147 KB out of the staging and 50 KB into the other, 700 of waits.
// Microseconds per 8 steps before (12 warps of 4 x 6 blocks, unrolled steps, the
// bookkeeping in warp 0) and now: 3840x2160 144 -> 122, 1920x1080 38.2 -> 32.3,
// 1280x720 21.5 -> 14.2, 960x540 13.9 -> 9.5, 640x360 12.3 -> 6.3.  Two CTAs of
// 6 warps on 64 x 72 tiles an SM, tried in place of this: 41.3 at 1920x1080.
// The exact form, before (a launch a round on interleaved images) and now:
// 3840x2160 256 -> 171, 1920x1080 75.5 -> 45.7, 1280x720 40.3 -> 20.3, 960x540
// 27.1 -> 12.9, 640x360 18.3 -> 10.2.
enum { kPmO0, kPmO1, kPmU0, kPmU1, kPmK, kPmC, kPmA, kPmOo0, kPmOo1, kPmUo0, kPmUo1, kPlMaps };

template <int kN>
struct PlSolve {
    CUtensorMap map[kN][kPlMaps];
    unsigned* done[kN];  // per problem and tile: rounds finished (zeroed before the launch)
    int w[kN], h[kN], tiles_x[kN];
    int tile0[kN + 1];   // first tile of problem p in a round's tile list; tile0[count] = N
    int count, num_iter;
    int round0, nround;  // this launch's rounds: round0 .. round0 + nround - 1
    unsigned* ticket;    // the next ticket (zeroed before the launch)
};

struct PlJob {
    int k;                    // round
    int p, local, per_plane;  // problem, tile index within it, its tiles of a plane
    int w, h;
    PlTileAt t;
};

template <int kCfg, int kN>
__device__ __forceinline__ PlJob pl_job(const PlSolve<kN>& g, int ticket)
{
    using G = PlGeo<kCfg>;
    const int N = g.tile0[g.count];
    PlJob j;
    const int round = ticket / N;
    j.k = g.round0 + round;
    const int tile = ticket - round * N;
    int p = 0;
    if (kN > 1) {
        // the last problem whose first tile is <= tile (binary search)
        int hi = g.count - 1;
#pragma unroll 1
        while (p < hi) {
            const int mid = (p + hi + 1) >> 1;
            if (g.tile0[mid] <= tile)
                p = mid;
            else
                hi = mid - 1;
        }
    }
    j.p = p;
    j.local = tile - g.tile0[p];
    j.w = g.w[p];
    j.h = g.h[p];
    j.per_plane = (g.tile0[p + 1] - g.tile0[p]) / 3;
    j.t = pl_tile<kCfg>(j.h, g.tiles_x[p], j.per_plane, j.local);
    return j;
}

// A tile's constant planes, which no round writes, and its O and U for its
// round, after its neighbours' stores; both on one full barrier.
template <int kCfg, int kN>
__device__ __forceinline__ void pl_load_constants(float* stage, const PlSolve<kN>& g, const PlJob& j, uint64_t* bar)
{
    using G = PlGeo<kCfg>;
    const CUtensorMap* m = g.map[j.p];
    tma_load_3d(stage + 2 * G::kStage, m + kPmK, j.t.ox, j.t.oy, j.t.c, bar);
    tma_load_3d(stage + 3 * G::kStage, m + kPmC, j.t.ox, j.t.oy, j.t.c, bar);
    if (!G::kFma)
        tma_load_3d(stage + 4 * G::kStage, m + kPmA, j.t.ox, j.t.oy, j.t.c, bar);
}

// The first round has no U to load, and the last one's U is not stored: 3840x2160,
// FMA form, 1 step 250 -> 236 us, 8 steps 292 -> 271.
template <int kCfg, int kN>
__device__ __forceinline__ void pl_load_iterate(float* stage, const PlSolve<kN>& g, const PlJob& j, uint64_t* bar)
{
    using G = PlGeo<kCfg>;
    asm volatile("fence.proxy.async.global;" ::: "memory");  // the acquired stores, before the async-proxy reads
    const CUtensorMap* m = g.map[j.p];
    const int par = j.k & 1;
    tma_load_3d(stage, m + (par ? kPmO1 : kPmO0), j.t.ox, j.t.oy, j.t.c, bar);
    if (j.k > 0)  // (there is no U before the first round)
        tma_load_3d(stage + G::kStage, m + (par ? kPmU1 : kPmU0), j.t.ox, j.t.oy, j.t.c, bar);
}

// Lane i of the loading warp watches the counter of the job's watched tile i (null:
// none to watch).
template <int kCfg, int kN>
__device__ __forceinline__ const unsigned* pl_watched(const PlSolve<kN>& g, const PlJob& j, int lane)
{
    if (j.k == 0)
        return nullptr;
    const int tile = pl_watched_tile<kCfg>(j.h, g.tiles_x[j.p], j.t, lane);
    return tile >= 0 ? g.done[j.p] + j.t.c * j.per_plane + tile : nullptr;
}

// One look by the whole warp, an L2 round trip: the acquiring loads and the
// warp barrier order the counters' published stores before the warp's later
// accesses (lane 0's TMA loads).
__device__ __forceinline__ bool pl_look(const unsigned* f, int k)
{
    unsigned v = ~0u;
    if (f)
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
    const bool ok = __all_sync(0xffffffffu, v >= static_cast<unsigned>(k));
    __syncwarp();
    return ok;
}

__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// one look at a phase, without waiting
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// What the loading warp tells the others of a tile (visible to the compute
// warps with its full_in barrier, to the storing warp with its full_out).
struct PlTile {
    int ox, oy, w, h, k0, T, mode;
    int k, p, c, local;
    int valid;  // 0: no more tiles
};

// Bounded wait that also gives up once another role has aborted; a wait that
// runs out raises the abort for everyone.
__device__ __forceinline__ bool pl_wait(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    for (int i = 0; i < kWaitSpins; ++i) {
        if (mbar_try_wait(bar, parity))
            return true;
        if ((i & 63) == 63 && *abort)
            return false;
        if (i > 64)
            __nanosleep(64);
    }
    *abort = 1;
    return false;
}

// The block: the compute warps and one warpgroup whose first two warps control
// (registers are handed out per warpgroup).  All start with 168 registers a
// thread; the control group gives up what the compute warps need beyond that
// (setmaxnreg: 256 x 216 + 128 x 72 = 256 x 224 + 128 x 56 = 384 x 168).
constexpr int kPlStartRegs = 168;

template <int kCfg, int kN>
__global__ void __launch_bounds__(32 * (PlGeo<kCfg>::kWarps + 4), 1)
    solver_solve_kernel(const __grid_constant__ PlSolve<kN> g, float step, float mom)
{
    using G = PlGeo<kCfg>;
    static_assert(G::kWarps % 4 == 0 &&
            G::kWarps * G::kComputeRegs + 4 * G::kControlRegs <= (G::kWarps + 4) * kPlStartRegs &&
            32 * (G::kWarps + 4) * kPlStartRegs <= 65536,
        "the warpgroups' registers within the block's");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* stage = reinterpret_cast<float*>(smem_raw);
    float* slots = stage + G::kPlanes * G::kStage;
    float* so = slots + 2 * G::kSlots;
    float* su = so + G::kOut;
    uint64_t* full_in = reinterpret_cast<uint64_t*>(su + G::kOut);  // the tile's data is staged
    uint64_t* empty_in = full_in + 1;   // every compute warp has taken it
    uint64_t* full_out = full_in + 2;   // every compute warp has put its interior
    uint64_t* empty_out = full_in + 3;  // the out staging has been stored
    // Tile i's entry is i % 4: entry i is written again for tile i + 4, whose
    // load follows the taking of tile i + 3, the putting of tile i + 2 and so
    // the storing of tile i + 1.
    __shared__ PlTile s_tile[4];
    __shared__ volatile int s_abort;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    for (int i = threadIdx.x; i < 2 * G::kSlots; i += blockDim.x)
        slots[i] = 0.0f;  // the apron slots stay zero
    if (threadIdx.x == 0) {
        mbar_init(full_in, 1);
        mbar_init(empty_in, G::kWarps);
        mbar_init(full_out, G::kWarps);
        mbar_init(empty_out, 1);
        s_abort = 0;
    }
    __syncthreads();
    grid_dependency_wait();

    if (warp >= G::kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(G::kControlRegs));
        if (warp == G::kWarps) {
            // ---- loading warp ---------------------------------------------------------
            const int total = g.tile0[g.count] * g.nround;  // (pl_launch_rounds: far below 2^31)
            int ticket = 0, phases = 0;  // full_in phases armed
            if (lane == 0)
                ticket = static_cast<int>(atomicAdd(g.ticket, 1u));
            for (int i = 0;; ++i) {
                ticket = __shfl_sync(0xffffffffu, ticket, 0);
                const bool valid = ticket < total;
                PlJob j{};
                const unsigned* watched = nullptr;
                bool ready = true;
                if (valid) {
                    j = pl_job<kCfg>(g, ticket);
                    // look at the neighbours until they are done or the staging is free
                    watched = pl_watched<kCfg>(g, j, lane);
                    ready = pl_look(watched, j.k);
                    for (int spins = 0; !ready && spins < kWaitSpins && !s_abort; ++spins) {
                        const bool free = i == 0 || mbar_test(empty_in, (i - 1) & 1);
                        if (__shfl_sync(0xffffffffu, static_cast<int>(free), 0))
                            break;
                        ready = pl_look(watched, j.k);
                    }
                }
                if (lane == 0) {
                    if (i > 0)
                        pl_wait(empty_in, (i - 1) & 1, &s_abort);
                    PlTile t{};
                    if (valid) {
                        t.ox = j.t.ox;
                        t.oy = j.t.oy;
                        t.w = j.w;
                        t.h = j.h;
                        t.k0 = j.k * G::kT;
                        t.T = min(G::kT, g.num_iter - t.k0);
                        t.mode = pl_mode<kCfg>(j.t.ox, j.t.oy, j.w, j.h);
                        t.k = j.k;
                        t.p = j.p;
                        t.c = j.t.c;
                        t.local = j.local;
                        t.valid = !s_abort;
                    }
                    s_tile[i & 3] = t;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    ++phases;
                    if (t.valid) {
                        mbar_expect_tx(full_in, (G::kPlanes - (j.k == 0 ? 1 : 0)) * G::kStageBytes);
                        if (ready)
                            pl_load_iterate<kCfg>(stage, g, j, full_in);
                        pl_load_constants<kCfg>(stage, g, j, full_in);
                    } else {
                        mbar_arrive(full_in);
                    }
                }
                __syncwarp();
                if (!valid || s_abort)
                    break;
                if (!ready) {
                    // late neighbours: the constants are on their way meanwhile
                    for (int spins = 0; !ready && spins < kWaitSpins && !s_abort; ++spins)
                        ready = pl_look(watched, j.k);
                    if (lane == 0) {
                        if (!ready)
                            s_abort = 1;
                        pl_load_iterate<kCfg>(stage, g, j, full_in);  // also when giving up: the phase completes
                    }
                    __syncwarp();
                }
                if (lane == 0)
                    ticket = static_cast<int>(atomicAdd(g.ticket, 1u));
                if (!valid || s_abort)
                    break;
            }
            if (s_abort && lane == 0) {
                // the outputs are invalid and vsc_check_device reports VSC_ETIMEOUT; let
                // the copies in flight land before the CTA exits
                atomicExch(&g_device_timeout, 1);
                mbar_wait_bounded(full_in, (phases - 1) & 1, kWaitSpins);
            }
        } else if (warp == G::kWarps + 1 && lane == 0) {
            // ---- storing warp ---------------------------------------------------------
            for (int i = 0; pl_wait(full_out, i & 1, &s_abort); ++i) {
                const PlTile t = s_tile[i & 3];
                if (!t.valid || s_abort)
                    break;
                const CUtensorMap* m = g.map[t.p];
                const int par = (t.k + 1) & 1;
                tma_store_3d(m + (par ? kPmOo1 : kPmOo0), t.ox + G::kT, t.oy + G::kT, t.c, so);
                if (t.k0 + t.T < g.num_iter)  // (nor is U read after the last)
                    tma_store_3d(m + (par ? kPmUo1 : kPmUo0), t.ox + G::kT, t.oy + G::kT, t.c, su);
                bulk_commit();
                // publish: the release store orders the completed async-proxy writes,
                // brought into the generic proxy by the proxy fence, before the counter
                bulk_wait_all();
                asm volatile("fence.proxy.async.global;" ::: "memory");
                st_release_u32(g.done[t.p] + t.local, static_cast<unsigned>(t.k + 1));
                mbar_arrive(empty_out);
            }
        }
        return;
    }

    // ---- compute warps --------------------------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(G::kComputeRegs));
    bool ok = true;
    for (int i = 0;; ++i) {
        ok = pl_wait(full_in, i & 1, &s_abort) && ok;
        // the warps leave together: one whose wait gave up takes the others with it
        int any;
        asm volatile(
            "{\n"
            " .reg .pred p, q;\n"
            " setp.ne.s32 p, %1, 0;\n"
            " barrier.cta.red.or.pred q, 1, %2, p;\n"
            " selp.s32 %0, 1, 0, q;\n"
            "}\n"
            : "=r"(any)
            : "r"(ok ? 0 : 1), "n"(32 * G::kWarps)
            : "memory");
        const PlTile& t = s_tile[i & 3];
        if (any || !t.valid) {
            __syncwarp();
            if (lane == 0)
                mbar_arrive(full_out);  // the storing warp leaves, too
            break;
        }
        const int T = t.T, k0 = t.k0, mode = t.mode;
        const PlPlace place = pl_place<kCfg>(t.ox, t.oy, t.w, t.h, lane, warp);
        PlState<kCfg> s;
        float4 up, dn;
        pl_take<kCfg>(s, up, dn, stage, k0, lane, warp);
        __syncwarp();
        if (lane == 0)
            mbar_arrive(empty_in);
        pl_round<kCfg>(mode, s, up, dn, slots, T, k0, step, mom, lane, warp, place,
            [] { asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * G::kWarps) : "memory"); });
        if (i > 0)
            ok = pl_wait(empty_out, (i - 1) & 1, &s_abort);
        pl_put<kCfg>(s, so, su, lane, warp);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0)
            mbar_arrive(full_out);
    }
}

// An mbarrier nobody arrives on, waited for with a bounded spin: exercises
// the timeout path of the bounded waits (sets g_device_timeout, returns).
__global__ void bounded_wait_selftest_kernel(int spins)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0)
        mbar_init(&bar, 1);
    __syncthreads();
    if (!mbar_wait_bounded(&bar, 0, spins) && threadIdx.x == 0)
        atomicExch(&g_device_timeout, 1);
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// 2D map over an interleaved w x h x 3 float image: x = float index in a row.
bool encode_image_map(CUtensorMap* m, const float* base, int w, int h, int box_rows, int box_cols = 3 * kTbEX)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn)
        return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(w) * 3, static_cast<cuuint64_t>(h)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(w) * 3 * sizeof(float)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int kN>
bool set_group_smem()
{
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    return cudaFuncSetAttribute(solver_solve_kernel<kSolverFma, kN>, kAttr, PlGeo<kSolverFma>::kSmem) == cudaSuccess &&
           cudaFuncSetAttribute(solver_solve_kernel<kSolverExact, kN>, kAttr, PlGeo<kSolverExact>::kSmem) == cudaSuccess &&
           cudaFuncSetAttribute(solver_persistent_kernel<kN>, kAttr, kPsSmem) == cudaSuccess;
}

struct DeviceInfo {
    int sms = 0;
    bool tb_smem = false, ps_smem = false;
};

// The solver kernels need more than 48 KB of dynamic shared memory; the
// opt-in is a per-device function attribute, set once per device together
// with the SM count the persistent kernel sizes its grid by.
cudaError_t device_info(DeviceInfo** out)
{
    static std::mutex mu;
    static DeviceInfo info[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    DeviceInfo& d = info[dev];
    if (!d.sms) {
        if ((e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
            return e;
        if ((e = cudaFuncSetAttribute(solver_tb_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTbSmem)) !=
            cudaSuccess)
            return e;
        constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
        auto single = [](auto c) {
            return cudaFuncSetAttribute(solver_solve_kernel<decltype(c)::value, 1>, kAttr,
                       PlGeo<decltype(c)::value>::kSmem) == cudaSuccess;
        };
        d.ps_smem = single(std::integral_constant<int, kSolverFma | kPlLong>{}) &&
                    single(std::integral_constant<int, kSolverFma | kPlMid>{}) &&
                    single(std::integral_constant<int, kSolverExact | kPlLong>{}) &&
                    single(std::integral_constant<int, kSolverExact | kPlMid>{}) &&
                    cudaFuncSetAttribute(solver_tall_kernel, kAttr, kPSmem) == cudaSuccess &&
                    set_group_smem<1>() && set_group_smem<4>() && set_group_smem<kGroupMax>() &&
                    cudaFuncSetAttribute(solver_fma_plain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                        PlGeo<kSolverFma>::kSmem) == cudaSuccess;
        cudaGetLastError();
    }
    *out = &d;
    return cudaSuccess;
}

bool aligned16p(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---- tile-shape autotuner ------------------------------------------------------------
// The two persistent kernels of the exact form on interleaved images (64 x 32
// and 64 x 48 tiles) give the same results bit for bit; which is faster depends
// on how their tiles fill the waves of one tile per SM.  solver_autotune times
// both on scratch images of a size and keeps the faster per (device, form,
// size); sizes never tuned use a wave model: a 64 x 48 tile costs about 1.91
// times a 64 x 32 one (GB300, 1920x1080 and 960x540).  The FMA form has one
// shape, 128 x 72 pixels of one channel plane.
struct ShapeTable {
    std::mutex mu;
    std::map<std::tuple<int, int, int, int>, int> rows;  // {device, form, w, h} -> tile rows
    bool enabled = true;
};
ShapeTable& shape_table()
{
    static ShapeTable t;
    return t;
}

int tiles_of(int w, int h, int ir) { return ((w + kIW - 1) / kIW) * ((h + ir - 1) / ir); }

int model_rows(int w, int h, int sms, int form)
{
    if (form == kSolverFma)
        return PlGeo<kSolverFma>::kRows;
    const int n_short = tiles_of(w, h, kIH), n_tall = tiles_of(w, h, kPIH);
    return 1.91 * ((n_tall + sms - 1) / sms) < 1.0 * ((n_short + sms - 1) / sms) ? kPEY : kTbEY;
}

// the tile rows a launch at this size uses on the current device: tuned, else the model
int chosen_rows(int dev, int w, int h, int sms, int form, bool* tuned = nullptr)
{
    ShapeTable& t = shape_table();
    std::lock_guard<std::mutex> lock(t.mu);
    auto it = t.rows.find({dev, form, w, h});
    if (tuned)
        *tuned = it != t.rows.end();
    return it != t.rows.end() ? it->second : model_rows(w, h, sms, form);
}

int interior_rows(int rows) { return rows - 2 * kTbT; }

// The tensor maps of one image's solve for both ping-pong phases: O[c] / U[c]
// with the tile box (loads), Oo[c] / Uo[c] with the interior box (stores).
struct SolveMaps {
    CUtensorMap O[2], U[2], A, W, L, Oo[2], Uo[2];
};

bool encode_solve(SolveMaps* m, float* const O[2], float* const U[2], const float* A, const float* Wt,
    const float* L, int w, int h, int rows)
{
    const int ir = interior_rows(rows);
    bool ok = encode_image_map(&m->A, A, w, h, rows) && encode_image_map(&m->W, Wt, w, h, rows) &&
              encode_image_map(&m->L, L, w, h, rows);
    for (int c = 0; c < 2 && ok; ++c)
        ok = encode_image_map(&m->O[c], O[c], w, h, rows) && encode_image_map(&m->U[c], U[c], w, h, rows) &&
             encode_image_map(&m->Oo[c], O[c], w, h, ir, 3 * kIW) &&
             encode_image_map(&m->Uo[c], U[c], w, h, ir, 3 * kIW);
    return ok;
}

// 3D map over the three w x h planes of a planar image (x, y, channel) of
// `pitch`-float rows (a multiple of 4).
bool encode_plane_map(CUtensorMap* m, const float* base, int w, int h, int pitch, int box_w, int box_h)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn)
        return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(w), static_cast<cuuint64_t>(h), 3};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(pitch) * sizeof(float),
        static_cast<cuuint64_t>(pitch) * h * sizeof(float)};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(box_w), static_cast<cuuint32_t>(box_h), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// rounds of a solve
int solve_launches(int num_iter, int steps = kTbT) { return num_iter > 0 ? (num_iter - 1) / steps + 1 : 0; }

// One image of a solve in rounds on interleaved images; c0: the buffer of O that the
// first round reads.
struct RoundsImage {
    SolveMaps maps;
    int w, h, c0;
    uint8_t* rgba;
};

// Steps k_first .. num_iter - 1 of a solve of n images in launches of T <= kTbT
// steps of a persistent kernel (`rows`-row tiles; the tall one takes one image)
// with programmatic dependent launch, kN images a launch.  Round li reads O[c0 ^
// (li & 1)] and U[li & 1] and writes the others.
template <int kN>
cudaError_t launch_rounds(const RoundsImage* im, int n, int rows, int num_iter, float step, float mom, int sms,
    cudaStream_t st, int* nl, int k_first = 0)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int nlaunch = solve_launches(num_iter - k_first);
    cudaError_t e = cudaSuccess;
    SolverLaunch<kN> g{};
    int k0 = k_first;
    for (int li = 0; li < nlaunch && e == cudaSuccess; ++li) {
        const int T = std::min(kTbT, num_iter - k0);
        for (int b0 = 0; b0 < n && e == cudaSuccess; b0 += kN) {  // (a round of one group in the tail of another's)
            g.count = std::min(n - b0, kN);
            for (int p = 0; p < g.count; ++p) {
                const RoundsImage& m = im[b0 + p];
                const int c = m.c0 ^ (li & 1);
                g.map[p][kMapO] = m.maps.O[c];
                g.map[p][kMapU] = m.maps.U[li & 1];
                g.map[p][kMapA] = m.maps.A;
                g.map[p][kMapW] = m.maps.W;
                g.map[p][kMapL] = m.maps.L;
                g.map[p][kMapOo] = m.maps.Oo[c ^ 1];
                g.map[p][kMapUo] = m.maps.Uo[(li + 1) & 1];
                g.w[p] = m.w;
                g.h[p] = m.h;
                g.tiles_x[p] = (m.w + kIW - 1) / kIW;
                g.tile0[p + 1] = g.tile0[p] + tiles_of(m.w, m.h, interior_rows(rows));
                g.rgba[p] = li == nlaunch - 1 ? m.rgba : nullptr;
            }
            cfg.gridDim = dim3(std::min(g.tile0[g.count], sms));
            if constexpr (kN == 1) {
                if (rows == kPEY) {
                    cfg.blockDim = dim3(kPThreads);
                    cfg.dynamicSmemBytes = kPSmem;
                    e = cudaLaunchKernelEx(&cfg, solver_tall_kernel, g, T, k0, step, mom);
                }
            }
            if (rows != kPEY) {
                cfg.blockDim = dim3(32, kTbEY / 2);
                cfg.dynamicSmemBytes = kPsSmem;
                e = cudaLaunchKernelEx(&cfg, solver_persistent_kernel<kN>, g, T, k0, step, mom);
            }
            ++*nl;
        }
        k0 += T;
    }
    return e;
}

}  // namespace

void solver_set_autotune(bool on)
{
    ShapeTable& t = shape_table();
    std::lock_guard<std::mutex> lock(t.mu);
    t.enabled = on;
    if (!on)
        t.rows.clear();
}

int solver_tile_rows(int w, int h, bool* tuned, int form)
{
    int dev = 0;
    DeviceInfo* di = nullptr;
    if (cudaGetDevice(&dev) != cudaSuccess || device_info(&di) != cudaSuccess)
        return 0;
    return chosen_rows(dev, w, h, di->sms, form, tuned);
}

bool solver_one_wave(int w, int h)
{
    DeviceInfo* di = nullptr;
    return device_info(&di) == cudaSuccess && tiles_of(w, h, kPIH) <= di->sms;
}

cudaError_t solver_autotune(int w, int h, cudaStream_t st, int* rows_out, int form)
{
    DeviceInfo* di = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = device_info(&di);
    if (e != cudaSuccess)
        return e;
    // the FMA form has one shape
    const bool eligible = di->ps_smem && form != kSolverFma && w % 4 == 0 && w >= 1 && h >= 1;
    const size_t total = static_cast<size_t>(w) * h * 3;
    ShapeTable& t = shape_table();
    const std::tuple<int, int, int, int> key{dev, form, w, h};
    {
        std::lock_guard<std::mutex> lock(t.mu);
        auto it = t.rows.find(key);
        if (it != t.rows.end() || !t.enabled || !eligible) {
            if (rows_out)
                *rows_out = it != t.rows.end() ? it->second : model_rows(w, h, di->sms, form);
            return cudaSuccess;
        }
    }
    // scratch images (zeros; the kernels have no data-dependent control flow):
    // O, O2, U0, U1, A, Wt, lap P
    float* buf = nullptr;
    if ((e = cudaMalloc(&buf, 7 * total * sizeof(float))) != cudaSuccess)
        return e;
    // Five rounds, the shapes alternating within each, one warm-up launch per
    // shape and four timed 8-step launches; each shape's best round counts (the
    // first launches after the allocation and a clock still ramping up would
    // otherwise favour whichever shape is timed last; where the shapes are
    // close, more rounds keep the choice from flipping between runs).
    cudaEvent_t ev[2] = {};
    float best_ms[2] = {1e30f, 1e30f};
    const int shapes[2] = {kTbEY, kPEY};
    SolveMaps maps[2];
    e = cudaMemsetAsync(buf, 0, 7 * total * sizeof(float), st);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i)
        e = cudaEventCreate(&ev[i]);
    for (int s = 0; s < 2 && e == cudaSuccess; ++s) {
        float* const O[2] = {buf, buf + total};
        float* const U[2] = {buf + 2 * total, buf + 3 * total};
        if (!encode_solve(&maps[s], O, U, buf + 4 * total, buf + 5 * total, buf + 6 * total, w, h, shapes[s]))
            e = cudaErrorInvalidValue;
    }
    auto launch = [&](int s, int num_iter, int* nl) {
        const RoundsImage im{maps[s], w, h, 0, nullptr};
        return launch_rounds<1>(&im, 1, shapes[s], num_iter, 0.15f, 0.15f, di->sms, st, nl, kTbT);
    };
    for (int round = 0; round < 5 && e == cudaSuccess; ++round) {
        for (int s = 0; s < 2 && e == cudaSuccess; ++s) {
            int nl = 0;
            // a warm-up launch, then four timed ones, all of kTbT steps with momentum
            e = launch(s, 2 * kTbT, &nl);
            if (e == cudaSuccess)
                e = cudaEventRecord(ev[0], st);
            if (e == cudaSuccess)
                e = launch(s, 5 * kTbT, &nl);
            float ms = 0.0f;
            if (e == cudaSuccess)
                e = cudaEventRecord(ev[1], st);
            if (e == cudaSuccess)
                e = cudaEventSynchronize(ev[1]);
            if (e == cudaSuccess)
                e = cudaEventElapsedTime(&ms, ev[0], ev[1]);
            if (e == cudaSuccess)
                best_ms[s] = std::min(best_ms[s], ms);
        }
    }
    for (cudaEvent_t x : ev)
        if (x)
            cudaEventDestroy(x);
    cudaFree(buf);
    if (e != cudaSuccess)
        return e;
    const int best = best_ms[1] < best_ms[0] ? shapes[1] : shapes[0];
    {
        std::lock_guard<std::mutex> lock(t.mu);
        if (t.enabled)
            t.rows[key] = best;
    }
    if (rows_out)
        *rows_out = best;
    return cudaSuccess;
}

// A workspace of planes ends in the solve kernel's counters: the ticket,
// padding to 64 bytes, one finished-round counter per tile; rounded up to
// 256 bytes so that a workspace placed after it stays aligned.
int pl_tiles_of(int w, int h, int cfg)
{
    switch (cfg) {
        case kSolverFma: return pl_tiles<kSolverFma>(w, h);
        case kSolverFma | kPlLong: return pl_tiles<kSolverFma | kPlLong>(w, h);
        case kSolverFma | kPlMid: return pl_tiles<kSolverFma | kPlMid>(w, h);
        case kSolverExact | kPlLong: return pl_tiles<kSolverExact | kPlLong>(w, h);
        case kSolverExact | kPlMid: return pl_tiles<kSolverExact | kPlMid>(w, h);
        default: return pl_tiles<kSolverExact>(w, h);
    }
}
int pl_counter_floats(int w, int h, int cfg) { return (16 + pl_tiles_of(w, h, cfg) + 63) / 64 * 64; }

// A plane's row in floats where the workspace has room for rows on the 16-byte
// grid (TMA's), whatever the width.
// 854x480, FMA form, 150 steps: 162 us; with plain loads, which a tile's steps
// wait for, and a launch a round 454 us.
int pl_pitch(int w) { return (w + 3) & ~3; }

// planes-images of a form: O, U (two each) and its constants
constexpr int pl_images(int form) { return form == kSolverFma ? 6 : 7; }

size_t solver_workspace_floats(int w, int h, int form)
{
    const size_t img = static_cast<size_t>(w) * h * 3;
    return form == kSolverFma ? 6 * img + pl_counter_floats(w, h, form) : 4 * img;
}

size_t solver_workspace_full_floats(int w, int h, int form)
{
    return pl_images(form) * static_cast<size_t>(pl_pitch(w)) * h * 3 + pl_counter_floats(w, h, form | kPlLong);
}

size_t solver_workspace_any_floats(int w, int h)
{
    return std::max(solver_workspace_full_floats(w, h, kSolverExact), solver_workspace_full_floats(w, h, kSolverFma));
}

int solver_steps_per_launch() { return kTbT; }

namespace {

// Rounds of one launch of the solve kernel at `tiles` tiles a round.  A launch
// counts its tickets, tiles x rounds, in 32 bits, and nothing bounds a caller's
// num_iter: a solve of more than 2^20 tickets (1920x1080, exact form: 6,752 steps,
// 39 ms) is several launches, each of whole rounds.
constexpr int kLaunchTickets = 1 << 20;
int pl_launch_rounds(int tiles, int nround) { return std::min(nround, std::max(1, kLaunchTickets / tiles)); }

struct WsView {
    float *L, *U0, *U1, *O2;
};
WsView ws_view(float* ws, int w, int h)
{
    const size_t n = static_cast<size_t>(w) * h * 3;
    return WsView{ws, ws + n, ws + 2 * n, ws + 3 * n};
}

// A form's workspace of planes: its planar images (three planes of h rows of
// `pitch` floats each; A: the exact form's only), then the solve kernel's counters.
struct PlWs {
    float *C, *K, *U[2], *O[2], *A;
    unsigned* cnt;
    int ncnt, pitch;
};
PlWs pl_view(float* ws, int w, int h, int pitch, int cfg)
{
    const int form = cfg & 1;
    const size_t n = static_cast<size_t>(pitch) * h * 3;
    return PlWs{ws, ws + n, {ws + 2 * n, ws + 3 * n}, {ws + 4 * n, ws + 5 * n}, ws + 6 * n,
        reinterpret_cast<unsigned*>(ws + pl_images(form) * n), pl_counter_floats(w, h, cfg), pitch};
}

bool tma_eligible(const DeviceInfo* di, int w, const float* O, const WsView& v, const float* A, const float* Wt)
{
    return di->ps_smem && (w % 4) == 0 && aligned16p(O) && aligned16p(v.O2) && aligned16p(v.U0) &&
           aligned16p(v.U1) && aligned16p(A) && aligned16p(Wt) && aligned16p(v.L);
}

// A solve in planes of rows on the 16-byte grid: a 16-byte aligned workspace with
// room for them and for the counters of cfg's tiles.
bool pl_fits(int w, int h, size_t ws_floats, int cfg)
{
    const size_t planes = pl_images(cfg & 1) * static_cast<size_t>(pl_pitch(w)) * h * 3;
    return ws_floats >= planes + pl_counter_floats(w, h, cfg);
}
bool pl_tma_eligible(const DeviceInfo* di, int w, int h, const float* ws, size_t ws_floats, int cfg)
{
    return di->ps_smem && aligned16p(ws) && pl_fits(w, h, ws_floats, cfg);
}

// The rounds of a solve: 8, 12 or 16 steps.  Where an SM has few tiles a round
// is a chain of waits (for the neighbours' stores, counters and loads: about 5 us)
// and its steps, and long rounds need fewer of them; where it has many, a round
// is its tiles' work, and a ring of 16 pixels leaves 42 % of an FMA tile as
// interior (exact form 37 %), one of 12 54 (51) and one of 8 68 (66).  A round's
// time, measured at 17 sizes from 320x180 to 1280x720, is the larger of `least`
// and base + tile * (tiles per SM) within a tenth, so longer rounds are taken
// where their estimate is a tenth below that of 8.  They are not where three
// 8-step tiles an SM or more make a round work alone (1920x1080, 150 steps in
// rounds of 8 and 12: FMA 657 and 711 us, exact 913 and 1,009), nor, beyond the
// smallest frames, for a few rounds, whose first loads nothing hides (exact
// 854x480, 12 steps: 36 us in two rounds of 8, 42 in one of 12).  150 steps in
// us, 8, 12 and 16 a round: FMA 320x180 147, 126, 109; 640x360 177, 145, 131;
// 854x480 196, 163, 177; 960x540 195, 211, 217; 1280x720 290, 324, 385; exact
// 480x270 189, 162, 167; 560x316 202, 170, 156; 640x360 204, 174, 199; 800x450
// 220, 227, 277 (calls in place, back to back on one image; on another image each
// time, its start copied, the 854x480 FMA call takes 172).  Of the rounds that a
// workspace of ws_floats has counters for: a smaller one may have them for 12 steps
// and not for 16.
int pl_rounds_cfg(int sms, int w, int h, int num_iter, int form, size_t ws_floats)
{
    struct Cost {
        int cfg;
        float least, base, tile;  // us
    };
    static constexpr Cost kCost[2][3] = {
        {{0, 10.5f, 2.8f, 5.3f}, {kPlMid, 12.8f, 5.5f, 6.2f}, {kPlLong, 14.5f, 5.0f, 8.4f}},
        {{0, 9.4f, 5.6f, 2.9f}, {kPlMid, 11.2f, 2.6f, 5.5f}, {kPlLong, 12.5f, 3.0f, 7.0f}}};
    const int tiles8 = pl_tiles_of(w, h, form);
    if (tiles8 > 3 * sms || (num_iter < 4 * kTbT && 5 * tiles8 > 3 * sms))
        return form;
    int best = form;
    float limit = 0.0f;
    for (const Cost& c : kCost[form == kSolverFma]) {
        if (c.cfg != 0 && !pl_fits(w, h, ws_floats, form | c.cfg))
            continue;
        const float tiles = static_cast<float>(pl_tiles_of(w, h, form | c.cfg)) / static_cast<float>(sms);
        const float us = static_cast<float>(solve_launches(num_iter, pl_round_steps(c.cfg))) *
                         std::max(c.least, c.base + c.tile * tiles);
        if (c.cfg == 0) {
            limit = 0.9f * us;
        } else if (us < limit) {
            best = form | c.cfg;
            limit = us;
        }
    }
    return best;
}

// The exact form on interleaved images, a launch a round, where one wave of its
// 64 x 32 tiles is the image (75 steps: 320x180 71 us against 75 in planes,
// 240x135 70 against 86), one of the 64 x 48 tiles for two rounds at most
// (600x338, 16 steps: 28 us against 32), or where a few steps do not pay for the
// planes' conversions: of a large image, and where the eight images of a solve
// stay in L2 (100 of its 129 MB) and eleven do not (us, interleaved and in planes:
// 1120x630 1 step 27 and 24; 1280x720 1 step 29 and 32, 3 steps 35 and 37, 4 steps 39
// and 38; 1440x810 1 step 47 and 42; 1600x900 1 step 57 and 53; 1760x990 3 steps 59
// and 67, 5 steps 70 and 72, 6 steps 77 and 75; 1920x1080 1 step 62 and 75, 6 steps 85
// and 89, 7 steps 93 and 94, 8 steps 107 and 98; 3840x2160 2 steps 210 and 288, 6
// steps 298 and 309, 7 steps 326 and 320).
bool exact_interleaved(int sms, int w, int h, int num_iter)
{
    const int tall = tiles_of(w, h, kPIH);
    const int64_t image = int64_t{12} * w * h, l2 = 100 << 20;  // bytes
    return tiles_of(w, h, kIH) <= sms || (num_iter <= 2 * kTbT && tall <= sms) ||
           (num_iter <= 3 && 8 * image <= l2 && 11 * image > l2) ||
           (num_iter <= 6 && tall > 7 * sms);
}

// The same for a level of a step, where planes save a launch (the start is
// upsampled in the setup) and, with fewer blocks, leave room for other streams'
// steps: more than two rounds of one wave's frames stay on planes unless a row of
// their tiles in rounds of 16 steps takes the per-row tests, which cost a round a
// quarter.  Exact frames of 150 steps, us a frame of one video and of three at a
// time, interleaved and in planes: 320x180 321, 327; 144, 128; 400x224 337, 359;
// 188, 170; with row tests 128x72 301, 335; 104, 115; 256x144 313, 357; 122, 127;
// 416x240 336, 363; 198, 199.
bool step_interleaved(int sms, int w, int h, int num_iter)
{
    return exact_interleaved(sms, w, h, num_iter) &&
           (num_iter <= 2 * kTbT || tiles_of(w, h, kIH) > sms || pl_row_tests<kSolverExact | kPlLong>(w, h));
}

struct PlanarCopy {
    const float* src;
    float* dst;
    uint8_t* rgba;
    int w, h, pitch;
    unsigned* cnt = nullptr;  // solve counters to zero on the way in
    int ncnt = 0;
};

// Interleaved <-> planar copies of n images, kPlanarGroupMax per launch.
cudaError_t launch_planar(const PlanarCopy* c, int n, int to_planar, cudaStream_t st, int* nl)
{
    for (int b0 = 0; b0 < n; b0 += kPlanarGroupMax) {
        PlanarGroup g{};
        g.count = std::min(n - b0, kPlanarGroupMax);
        g.block0[0] = 0;
        for (int p = 0; p < g.count; ++p) {
            g.src[p] = c[b0 + p].src;
            g.dst[p] = c[b0 + p].dst;
            g.rgba[p] = c[b0 + p].rgba;
            g.cnt[p] = c[b0 + p].cnt;
            g.ncnt[p] = c[b0 + p].ncnt;
            g.npix[p] = static_cast<int64_t>(c[b0 + p].w) * c[b0 + p].h;
            g.w[p] = c[b0 + p].w;
            g.pitch[p] = c[b0 + p].pitch;
            g.plane[p] = static_cast<int64_t>(c[b0 + p].pitch) * c[b0 + p].h;
            g.block0[p + 1] = g.block0[p] + static_cast<int>((g.npix[p] + 255) / 256);
        }
        const cudaError_t e = launch_pdl(planar_group_kernel, dim3(g.block0[g.count]), dim3(256), 0, st, g, to_planar);
        if (e != cudaSuccess)
            return e;
        ++*nl;
    }
    return cudaGetLastError();
}

// The solve kernel over n members, kN a launch (each member's counters zeroed
// beforehand; the first member's ticket serves the launch).  The tiles' counters
// run on from launch to launch of a long solve, the ticket starts again.
template <int kCfg, int kN>
cudaError_t launch_solve(const std::vector<PlWs>& v, const int* w, const int* h, int n, int num_iter, float step,
    float mom, int sms, cudaStream_t st, int* nl)
{
    using G = PlGeo<kCfg>;
    const int nround = solve_launches(num_iter, G::kT);
    for (int b0 = 0; b0 < n; b0 += kN) {
        PlSolve<kN> g{};
        g.count = std::min(n - b0, kN);
        g.tile0[0] = 0;
        for (int p = 0; p < g.count; ++p) {
            const PlWs& m = v[b0 + p];
            const int W = w[b0 + p], H = h[b0 + p];
            CUtensorMap* mp = g.map[p];
            bool ok = true;
            for (int c = 0; c < 2 && ok; ++c)
                ok = encode_plane_map(&mp[c ? kPmO1 : kPmO0], m.O[c], W, H, m.pitch, kPlW, G::kRows) &&
                     encode_plane_map(&mp[c ? kPmU1 : kPmU0], m.U[c], W, H, m.pitch, kPlW, G::kRows) &&
                     encode_plane_map(&mp[c ? kPmOo1 : kPmOo0], m.O[c], W, H, m.pitch, G::kIW, G::kIRows) &&
                     encode_plane_map(&mp[c ? kPmUo1 : kPmUo0], m.U[c], W, H, m.pitch, G::kIW, G::kIRows);
            if (!ok || !encode_plane_map(&mp[kPmK], m.K, W, H, m.pitch, kPlW, G::kRows) ||
                !encode_plane_map(&mp[kPmC], m.C, W, H, m.pitch, kPlW, G::kRows) ||
                (!G::kFma && !encode_plane_map(&mp[kPmA], m.A, W, H, m.pitch, kPlW, G::kRows)))
                return cudaErrorInvalidValue;
            g.done[p] = m.cnt + 16;
            g.w[p] = W;
            g.h[p] = H;
            g.tiles_x[p] = pl_tiles_x<kCfg>(W);
            g.tile0[p + 1] = g.tile0[p] + pl_tiles<kCfg>(W, H);
        }
        g.num_iter = num_iter;
        g.ticket = v[b0].cnt;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        // no more CTAs than a round has tiles: a CTA more could only start on the next
        // round and would wait, holding an SM that another stream's kernel could use
        // (three 640x360 videos at a time, exact form: 353 -> 303 us a frame; one: the same)
        cfg.gridDim = dim3(std::min(g.tile0[g.count], sms));
        cfg.blockDim = dim3(32 * (G::kWarps + 4));
        cfg.dynamicSmemBytes = G::kSmem;
        const int per = pl_launch_rounds(g.tile0[g.count], nround);
        for (int r0 = 0; r0 < nround; r0 += per) {
            g.round0 = r0;
            g.nround = std::min(per, nround - r0);
            cudaError_t e = r0 > 0 ? cudaMemsetAsync(g.ticket, 0, sizeof(unsigned), st) : cudaSuccess;
            if (e == cudaSuccess)
                e = cudaLaunchKernelEx(&cfg, solver_solve_kernel<kCfg, kN>, g, step, mom);
            if (e != cudaSuccess)
                return e;
            ++*nl;
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_prep(int form, const float* P, const float* A, const float* Wt, const float* O, const PlWs& v,
    float* Op, int w, int h, float step, unsigned* cnt, int ncnt, const float* Oc, int cw, int ch, cudaStream_t st)
{
    const dim3 b(32, 8);
    auto k = form == kSolverFma ? solver_prep_kernel<kSolverFma> : solver_prep_kernel<kSolverExact>;
    return launch_pdl(k, grid2d(w, h, b), b, 0, st, P, A, Wt, O, v.C, v.K, v.A, Op, w, h, v.pitch, step, cnt, ncnt, Oc,
        cw, ch);
}

// run_solver in planes: constants, the planes of the start Oi (or of the
// coarse solution Oc upsampled) and zeroed counters, the solve (one launch; for
// the FMA form in a smaller workspace a launch a round with plain loads), O
// (and the RGBA8 copy) back from its planes.
cudaError_t run_solver_planes(const DeviceInfo* di, int form, const float* P, const float* A, const float* Wt,
    const float* Oi, float* O, int w, int h, int num_iter, float step, float mom, float* workspace, size_t ws_floats,
    cudaStream_t st, int* nl, uint8_t* rgba_out, const float* Oc, int cw, int ch)
{
    const bool tma = pl_tma_eligible(di, w, h, workspace, ws_floats, form);
    const int cfg = tma ? pl_rounds_cfg(di->sms, w, h, num_iter, form, ws_floats) : form;
    const PlWs v = pl_view(workspace, w, h, tma ? pl_pitch(w) : w, cfg);
    cudaError_t e = launch_prep(form, P, A, Wt, Oi, v, v.O[0], w, h, step, v.cnt, v.ncnt, Oc, cw, ch, st);
    ++*nl;
    const int nlaunch = solve_launches(num_iter, pl_round_steps(cfg));
    if (e == cudaSuccess && tma) {
        const std::vector<PlWs> one(1, v);
        auto solve = [&](auto c) {
            return launch_solve<decltype(c)::value, 1>(one, &w, &h, 1, num_iter, step, mom, di->sms, st, nl);
        };
        switch (cfg) {
            case kSolverFma: e = solve(std::integral_constant<int, kSolverFma>{}); break;
            case kSolverFma | kPlLong: e = solve(std::integral_constant<int, kSolverFma | kPlLong>{}); break;
            case kSolverFma | kPlMid: e = solve(std::integral_constant<int, kSolverFma | kPlMid>{}); break;
            case kSolverExact | kPlLong: e = solve(std::integral_constant<int, kSolverExact | kPlLong>{}); break;
            case kSolverExact | kPlMid: e = solve(std::integral_constant<int, kSolverExact | kPlMid>{}); break;
            default: e = solve(std::integral_constant<int, kSolverExact>{}); break;
        }
    } else if (e == cudaSuccess) {
        // plain loads and stores
        const int tx = pl_tiles_x<kSolverFma>(w), nt = pl_tiles<kSolverFma>(w, h);
        int k0 = 0;
        for (int li = 0; li < nlaunch && e == cudaSuccess; ++li) {
            const int T = std::min(kTbT, num_iter - k0);
            const PlPlain pl{v.O[li & 1], v.U[li & 1], v.K, v.C, v.O[(li + 1) & 1],
                li + 1 < nlaunch ? v.U[(li + 1) & 1] : nullptr, w, h, tx, nt};
            e = launch_pdl(solver_fma_plain_kernel, dim3(std::min(nt, di->sms)), dim3(32 * PlGeo<kSolverFma>::kWarps),
                PlGeo<kSolverFma>::kSmem, st, pl, T, k0, step, mom);
            ++*nl;
            k0 += T;
        }
    }
    if (e == cudaSuccess) {
        const PlanarCopy back{v.O[nlaunch & 1], O, rgba_out, w, h, v.pitch};
        e = launch_planar(&back, 1, 0, st, nl);
    }
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

bool solver_tma_supported()
{
    DeviceInfo* di = nullptr;
    return device_info(&di) == cudaSuccess && di->ps_smem;
}

bool solver_group_interleaved(const int* w, const int* h, int n, int form)
{
    DeviceInfo* di = nullptr;
    if (form != kSolverExact || device_info(&di) != cudaSuccess || !di->ps_smem)
        return false;
    for (int b0 = 0; b0 < n; b0 += kGroupMax) {
        int64_t tiles = 0;
        for (int i = b0; i < std::min(n, b0 + kGroupMax); ++i) {
            if (w[i] % 4 != 0)
                return false;
            tiles += tiles_of(w[i], h[i], kIH);
        }
        if (tiles > di->sms)
            return false;
    }
    return true;
}

float* solver_group_start(float* O, float* workspace, int w, int h, int num_iter, bool interleaved)
{
    return interleaved && solve_launches(num_iter) % 2 == 1 ? ws_view(workspace, w, h).O2 : O;
}

cudaError_t solver_prep(int form, const float* P, const float* A, const float* Wt, int w, int h, float step,
    float* workspace, bool interleaved, cudaStream_t st)
{
    if (interleaved) {
        const dim3 b(32, 8);
        const cudaError_t e = launch_pdl(lap_pr_kernel, grid2d(w, h, b), b, 0, st, P, ws_view(workspace, w, h).L, w, h);
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    const PlWs v = pl_view(workspace, w, h, pl_pitch(w), form);
    const cudaError_t e = launch_prep(form, P, A, Wt, nullptr, v, nullptr, w, h, step, nullptr, 0, nullptr, 0, 0, st);
    return e != cudaSuccess ? e : cudaGetLastError();
}

bool solver_planes_fit(int form, int w, int h, size_t ws_floats) { return pl_fits(w, h, ws_floats, form); }

bool solver_step_interleaved(int form, const float* A, const float* Wt, const float* O, int w, int h, int num_iter,
    float* workspace)
{
    DeviceInfo* di = nullptr;
    if (form != kSolverExact || device_info(&di) != cudaSuccess ||
        !tma_eligible(di, w, O, ws_view(workspace, w, h), A, Wt))
        return false;
    return step_interleaved(di->sms, w, h, num_iter);
}

cudaError_t solver_plan(int w, int h, int num_iter, int form, size_t ws_floats, int sms, SolverPlan* out)
{
    if (sms <= 0) {
        DeviceInfo* di = nullptr;
        const cudaError_t e = device_info(&di);
        if (e != cudaSuccess)
            return e;
        sms = di->sms;
    }
    SolverPlan p{};
    const bool inter = form == kSolverExact && w % 4 == 0 && exact_interleaved(sms, w, h, num_iter);
    p.planes = form == kSolverFma || (!inter && pl_fits(w, h, ws_floats, form));
    const bool one_launch = p.planes && pl_fits(w, h, ws_floats, form);
    const int cfg = one_launch ? pl_rounds_cfg(sms, w, h, num_iter, form, ws_floats) : form;
    p.steps = pl_round_steps(cfg);
    p.rounds = solve_launches(num_iter, p.steps);
    if (p.planes) {
        p.tiles = pl_tiles_of(w, h, cfg);
    } else {
        const int T = std::min(num_iter, kTbT);  // (solver_tb_kernel's ring is its launch's steps)
        p.tiles = w % 4 == 0 ? tiles_of(w, h, interior_rows(model_rows(w, h, sms, form)))
                             : ((w - 1) / (kTbEX - 2 * T) + 1) * ((h - 1) / (kTbEY - 2 * T) + 1);
    }
    p.rounds_per_launch = one_launch ? pl_launch_rounds(p.tiles, p.rounds) : std::min(1, p.rounds);
    *out = p;
    return cudaSuccess;
}

cudaError_t run_solver_group(const SolverImage* im, int n, int num_iter, float step, float mom, cudaStream_t st,
    int* launches, int form, bool interleaved)
{
    DeviceInfo* di = nullptr;
    cudaError_t e = device_info(&di);
    if (e != cudaSuccess)
        return e;
    if (n < 1 || !di->ps_smem)
        return cudaErrorInvalidValue;
    int nl = 0;
    if (num_iter <= 0) {
        for (int i = 0; i < n && e == cudaSuccess; ++i)
            if (im[i].rgba) {
                e = launch_float_to_rgba(im[i].O, im[i].rgba, static_cast<int64_t>(im[i].w) * im[i].h, st);
                ++nl;
            }
        if (launches)
            *launches += nl;
        return e;
    }
    if (interleaved) {
        std::vector<RoundsImage> ri(n);
        for (int i = 0; i < n; ++i) {
            const WsView v = ws_view(im[i].workspace, im[i].w, im[i].h);
            float* const O[2] = {im[i].O, v.O2};
            float* const U[2] = {v.U0, v.U1};
            if (!tma_eligible(di, im[i].w, im[i].O, v, im[i].A, im[i].Wt) ||
                !encode_solve(&ri[i].maps, O, U, im[i].A, im[i].Wt, v.L, im[i].w, im[i].h, kTbEY))
                return cudaErrorInvalidValue;
            ri[i].w = im[i].w;
            ri[i].h = im[i].h;
            ri[i].c0 = solve_launches(num_iter) % 2;
            ri[i].rgba = im[i].rgba;
        }
        e = n <= 4 ? launch_rounds<4>(ri.data(), n, kTbEY, num_iter, step, mom, di->sms, st, &nl)
                   : launch_rounds<kGroupMax>(ri.data(), n, kTbEY, num_iter, step, mom, di->sms, st, &nl);
        if (launches)
            *launches += nl;
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    // O into planes (counters zeroed), one solve launch per 16 images, O back
    std::vector<int> ws(n), hs(n);
    std::vector<PlWs> v(n);
    std::vector<PlanarCopy> to(n), back(n);
    for (int i = 0; i < n; ++i) {
        const int w = ws[i] = im[i].w, h = hs[i] = im[i].h;
        v[i] = pl_view(im[i].workspace, w, h, pl_pitch(w), form);
        if (!aligned16p(im[i].workspace))
            return cudaErrorInvalidValue;
        to[i] = PlanarCopy{im[i].O, v[i].O[0], nullptr, w, h, v[i].pitch, v[i].cnt, v[i].ncnt};
        back[i] = PlanarCopy{v[i].O[solve_launches(num_iter) & 1], im[i].O, im[i].rgba, w, h, v[i].pitch};
    }
    e = launch_planar(to.data(), n, 1, st, &nl);
    auto solve = [&](auto f, auto group) {
        return launch_solve<decltype(f)::value, decltype(group)::value>(v, ws.data(), hs.data(), n, num_iter, step, mom,
            di->sms, st, &nl);
    };
    using Fma = std::integral_constant<int, kSolverFma>;
    using Exact = std::integral_constant<int, kSolverExact>;
    using Few = std::integral_constant<int, 4>;
    using Many = std::integral_constant<int, kGroupMax>;
    if (e == cudaSuccess)
        e = form == kSolverFma ? (n <= 4 ? solve(Fma{}, Few{}) : solve(Fma{}, Many{}))
                               : (n <= 4 ? solve(Exact{}, Few{}) : solve(Exact{}, Many{}));
    if (e == cudaSuccess)
        e = launch_planar(back.data(), n, 0, st, &nl);
    if (launches)
        *launches += nl;
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t run_solver_planes(int form, const float* P, const float* A, const float* Wt, const float* Oi, float* O,
    int w, int h, const float* Oc, int cw, int ch, int num_iter, float step, float mom, float* workspace,
    size_t ws_floats, cudaStream_t st, int* launches, uint8_t* rgba_out)
{
    if (num_iter <= 0 || !(Oi || (Oc && cw > 0 && ch > 0)))
        return cudaErrorInvalidValue;
    DeviceInfo* di = nullptr;
    cudaError_t e = device_info(&di);
    if (e != cudaSuccess)
        return e;
    if (!di->ps_smem || !pl_tma_eligible(di, w, h, workspace, ws_floats, form))
        return cudaErrorNotSupported;
    int nl = 0;
    e = run_solver_planes(di, form, P, A, Wt, Oi, O, w, h, num_iter, step, mom, workspace, ws_floats, st, &nl, rgba_out,
        Oc, cw, ch);
    if (launches)
        *launches += nl;
    return e;
}

cudaError_t run_solver(const float* P, const float* A, const float* Wt, float* O, int w, int h, int num_iter,
    float step, float mom, float* workspace, size_t ws_floats, cudaStream_t st, int* launches, uint8_t* rgba_out, int form)
{
    const size_t n = static_cast<size_t>(w) * h * 3;
    const WsView v = ws_view(workspace, w, h);
    int nl = 0;
    if (num_iter <= 0) {
        if (rgba_out) {
            cudaError_t e = launch_float_to_rgba(O, rgba_out, static_cast<int64_t>(w) * h, st);
            if (launches)
                *launches += 1;
            return e;
        }
        return cudaSuccess;
    }
    DeviceInfo* di = nullptr;
    cudaError_t e0 = device_info(&di);
    if (e0 != cudaSuccess)
        return e0;
    if (form == kSolverFma && !di->ps_smem)
        return cudaErrorNotSupported;
    const bool interleaved = tma_eligible(di, w, O, v, A, Wt) && exact_interleaved(di->sms, w, h, num_iter);
    if (form == kSolverFma || (!interleaved && pl_tma_eligible(di, w, h, workspace, ws_floats, form))) {
        const cudaError_t e = run_solver_planes(di, form, P, A, Wt, O, O, w, h, num_iter, step, mom, workspace,
            ws_floats, st, &nl, rgba_out, nullptr, 0, 0);
        if (launches)
            *launches += nl;
        return e;
    }
    const dim3 b(32, 8);
    if ((e0 = launch_pdl(lap_pr_kernel, grid2d(w, h, b), b, 0, st, P, v.L, w, h)) != cudaSuccess)
        return e0;
    ++nl;
    // Launches of up to kTbT iterations; ping-pong O between O and O2 and U
    // between its two buffers so that the last launch writes O.
    const int nlaunch = solve_launches(num_iter);
    float* cur = nlaunch % 2 == 0 ? O : v.O2;
    if (cur != O) {
        cudaError_t e = cudaMemcpyAsync(v.O2, O, n * sizeof(float), cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess)
            return e;
    }
    // TMA path: 16-byte row pitch and aligned images; the tile shape is the
    // autotuned one for this size, else the wave model's
    int dev = 0;
    if ((e0 = cudaGetDevice(&dev)) != cudaSuccess)
        return e0;
    const int rows = chosen_rows(dev, w, h, di->sms, kSolverExact);
    SolveMaps m;
    bool tma = tma_eligible(di, w, O, v, A, Wt);
    if (tma) {
        float* const Ob[2] = {O, v.O2};
        float* const Ub[2] = {v.U0, v.U1};
        tma = encode_solve(&m, Ob, Ub, A, Wt, v.L, w, h, rows);
    }
    if (tma) {
        const RoundsImage im{m, w, h, cur == O ? 0 : 1, rgba_out};
        cudaError_t e = launch_rounds<1>(&im, 1, rows, num_iter, step, mom, di->sms, st, &nl);
        if (launches)
            *launches += nl;
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    float* U[2] = {v.U0, v.U1};
    int k0 = 0;
    for (int li = 0; li < nlaunch; ++li) {
        const int T = std::min(kTbT, num_iter - k0);
        float* nxt = (cur == O) ? v.O2 : O;
        uint8_t* rg = (li == nlaunch - 1) ? rgba_out : nullptr;
        const dim3 grid((w + (kTbEX - 2 * T) - 1) / (kTbEX - 2 * T), (h + (kTbEY - 2 * T) - 1) / (kTbEY - 2 * T));
        solver_tb_kernel<<<grid, dim3(32, kTbEY / 2), kTbSmem, st>>>(cur, nxt, U[li & 1], U[(li + 1) & 1], v.L, A,
            Wt, w, h, T, k0, step, mom, rg);
        ++nl;
        k0 += T;
        cur = nxt;
    }
    if (launches)
        *launches += nl;
    return cudaGetLastError();
}

// ---- device addresses of file-scope device arrays -----------------------------
// In host code a __device__ variable's name is only a stand-in symbol, not a
// device address.  Its address is looked up with cudaGetSymbolAddress, with
// the device current, once per device and context: the address belongs to
// the module loaded into the context, so after a device reset (a new primary
// context) it is looked up again.  The context is told apart by its id
// (cuCtxGetId, fetched from the driver at run time); without that entry
// point every call looks the address up.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

bool current_context_id(unsigned long long* id)
{
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<CtxGetCurrentFn>(p);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<CtxGetIdFn>(p);
    });
    CUcontext ctx = nullptr;
    return get_current && get_id && get_current(&ctx) == CUDA_SUCCESS && ctx && get_id(ctx, id) == CUDA_SUCCESS;
}

struct SymbolCache {
    std::mutex mu;
    void* addr[64] = {};
    unsigned long long ctx[64] = {};
};

cudaError_t symbol_address(SymbolCache& c, const void* symbol, void** out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= 64)
        return cudaErrorInvalidDevice;
    unsigned long long id = 0;
    std::lock_guard<std::mutex> lock(c.mu);
    if (!c.addr[dev] || !current_context_id(&id) || c.ctx[dev] != id) {
        void* p = nullptr;
        if ((e = cudaGetSymbolAddress(&p, symbol)) != cudaSuccess)
            return e;
        // the lookup made the device's context current
        c.addr[dev] = p;
        c.ctx[dev] = current_context_id(&id) ? id : 0;
    }
    *out = c.addr[dev];
    return cudaSuccess;
}

// ---- solver workspace for callers that cannot allocate ------------------------
// A file-scope device array (every GPU that loads the library holds it until
// the process exits), handed to the kernels by its device address
// (symbol_address: looked up once per device and context).
static __device__ __align__(256) float g_noalloc_ws[kNoAllocWorkspaceFloats];

cudaError_t noalloc_workspace(float** out)
{
    static SymbolCache cache;
    return symbol_address(cache, g_noalloc_ws, reinterpret_cast<void**>(out));
}

cudaError_t run_solver_noalloc(const float* P, const float* A, const float* Wt, float* O, int w, int h, int num_iter,
    float step, float mom, cudaStream_t st)
{
    float* ws = nullptr;
    cudaError_t e = noalloc_workspace(&ws);
    if (e != cudaSuccess)
        return e;
    // Every workspace element (lap P, both momentum images, the second Jacobi
    // buffer) is written before it is read, so nothing is cleared.
    // On interleaved images even where the array has room for planes: the solve on
    // planes waits for counters in its workspace, and of two calls that overlap (a
    // race on the shared array that costs their results) the setup of one would
    // zero the counters that the other's blocks wait for.
    return run_solver(P, A, Wt, O, w, h, num_iter, step, mom, ws, solver_workspace_floats(w, h, kSolverExact), st,
        nullptr, nullptr, kSolverExact);
}

cudaError_t device_timeout_flag(int** flag)
{
    static SymbolCache cache;
    return symbol_address(cache, &g_device_timeout, reinterpret_cast<void**>(flag));
}

cudaError_t check_device_timeout(int* flagged)
{
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_device_timeout, sizeof(int));
    if (e != cudaSuccess)
        return e;
    if (v) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_device_timeout, &zero, sizeof(int));
    }
    *flagged = v;
    return e;
}

cudaError_t launch_bounded_wait_selftest(int spins, cudaStream_t st)
{
    bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(spins);
    return cudaGetLastError();
}

}  // namespace vsc
