// ppf_nn_conv.cu -- 3x3x3 convolutions of the surrogate network as
// implicit GEMMs on the fifth-generation tensor cores (tcgen05, BF16 in,
// FP32 accumulation in TMEM).
//
// conv_kernel<CI, CO, EPI>: out[v] = sum over the 27 taps of W_tap * in[v + tap].
//   One tile = 128 consecutive voxels of one x row (M = 128), N = 3 CO (the
//   three dy taps), K = 9 (dz, dx) taps x CI.  A work item is a column of
//   tiles marching in y (rows y0..y1-1 of one z plane and x segment).  An
//   input "segment" is 130 voxels (the tile plus one each side) of one input
//   row, moved into shared memory by 1-D bulk copies, one per 8-channel
//   plane.  A ring of RING row slots (3 segments each, z-1..z+1) holds the
//   rows while the next ones load, so every input row is fetched once per
//   work item.  The A operand of tap (dz, dx) is its segment started dx+1
//   voxels (16 bytes each) in; the B operand is that tap's CI x 3 CO block of
//   the weight image, loaded once per CTA.
//   Warp roles: three producer threads (one per z plane), two MMA-issuing
//   threads (alternate rows; the first one's warp owns the TMEM
//   allocation), and two or three epilogue groups of four warps that take
//   the output rows in turn from a ring of five TMEM tiles.
//   What bounds it: with N = 96 an MMA reads 7 KB of operands from shared
//   memory, 56 cycles at 128 bytes a clock (measured; the mathematics is
//   48), so a row of 18 takes 1008 cycles; at 256^3, 32 -> 32 channels, that
//   is 0.49 ms.  Measured 0.65 ms (0.82 ms before): one producer thread
//   issued a row's 12 copies in about 1400 cycles, one MMA thread spends
//   about 500 on a row's waits and descriptors, and every row's halo voxel in
//   x sent its warp through the eight-image loop.
//
// wgrad_kernel<CX, CZ>: dW[tap][co][ci] = sum over voxels u of
//   X[u][ci] * dZ[u - tap][co] (periodic).  The reduction runs over voxels
//   (K), both operands are channel-contiguous (MN-major).  A CTA marches
//   columns of 128-voxel rows in y.  A row r of X comes as its three z planes
//   (M = 128: three slots of CX channels and zeros), a row y of dZ three times,
//   shifted by dx = -1, 0, 1 (N = 3 CZ); row r meets dZ rows r+1, r, r-1, one
//   accumulator per dy.  dW stays in TMEM over all the CTA's rows and is
//   written once at the end.
//   What bounds it: 24 MMAs a row, 56 cycles each (N = 96), 1344 cycles a row;
//   loading nine X segments for every tile (40 copies) and 72 MMAs of N = 32
//   (40 cycles each) it took about 5200 (146 us for 32 -> 32 channels on
//   64 x 128 x 128; now 68 us, a third of it the ramp and the write-out).
//
// Every mbarrier wait is bounded by a time limit; on expiry the CTA sets
// the error word, stops issuing work, drains its own copies and MMAs
// (bounded) and exits.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ppf_nn.h"
#include "ppf_pair.h"
#include "ppf_ptx.h"

namespace ppf {
namespace nn {

using namespace ppf::ptx;

namespace {

// bounded wait that also gives up when another role flagged an abort
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, unsigned long long limit_ns,
                                              volatile int *abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = globaltimer();
    for (uint32_t it = 0;; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 31u) == 31u) {
            if (*abort_flag) return false;
            if (globaltimer() - t0 > limit_ns) return false;
        }
    }
}

// the same with a short sleep between polls: for the many epilogue warps,
// whose spinning would otherwise take issue slots from the MMA thread
__device__ __forceinline__ bool wait_backoff(uint32_t bar, uint32_t parity, unsigned long long limit_ns,
                                             volatile int *abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = globaltimer();
    for (uint32_t it = 0;; ++it) {
        __nanosleep(64);
        if (mbar_try(bar, parity)) return true;
        if ((it & 7u) == 7u) {
            if (*abort_flag) return false;
            if (globaltimer() - t0 > limit_ns) return false;
        }
    }
}

// Programmatic dependent launch: a convolution or weight-gradient kernel starts
// while the CTAs of the one before finish, sets itself up, and waits here until
// that one is complete and its results are visible.  The next kernel may start
// only after grid_release, so at most two are in flight.  A CTA calls that behind
// the barrier that follows its TMEM allocation: earlier, a CTA of the next kernel
// could take the columns first and wait for this grid, which waits for the
// columns.  (64 x 128 x 128, width 32: 1186 us a training step, 1232 us without
// the overlap on the same machine.)
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// launch with that attribute
template <typename Args>
cudaError_t launch_pdl(void (*kern)(Args), int grid, int block, int smem, const Args &a, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

__device__ __forceinline__ void fail(volatile int *abort_flag, int *err, int code) {
    *abort_flag = 1;
    atomicOr(err, code);
}

// the halo image of interior coordinate x, or kNone (periodic: x=0 -> n,
// x=n-1 -> -1; no-flux: x=0 -> -1, x=n-1 -> n); needs n >= 2
constexpr int kNone = -0x40000000;
__device__ __forceinline__ int image_of(int x, int n, int bc) {
    return x == 0 ? (bc == 0 ? n : -1) : x == n - 1 ? (bc == 0 ? -1 : n) : kNone;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ uint4 pack8(const V2<float> *f) {
    return make_uint4(pack_bf16x2(f[0].x(), f[0].y()), pack_bf16x2(f[1].x(), f[1].y()),
                      pack_bf16x2(f[2].x(), f[2].y()), pack_bf16x2(f[3].x(), f[3].y()));
}

__device__ __forceinline__ void unpack8(uint4 q, V2<float> *f) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = V2<float>(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
}

// logistic function: sigma(z) = (1 + tanh(z/2)) / 2 with the hardware
// tanh (tanh.approx.f32, relative error about 2^-11, well below the BF16
// rounding of every value it feeds)
__device__ __forceinline__ V2<float> sigmoid2(V2<float> z) {
    const V2<float> h = splat(0.5f) * z;
    float t, u;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h.x()));
    asm("tanh.approx.f32 %0, %1;" : "=f"(u) : "f"(h.y()));
    return fma2(splat(0.5f), V2<float>(t, u), splat(0.5f));
}

// the halo images of voxel (x, y, z) in y and z (and their images in x); v[j]
// is the voxel in channel plane j
template <int NP>
__device__ __noinline__ void store_images(const NNGeom &g, uint4 *base, int x, int y, int z, const uint4 (&v)[NP]) {
    const int ax = image_of(x, g.nx, g.bc), ay = image_of(y, g.ny, g.bc), az = image_of(z, g.nz, g.bc);
    for (int k = 2; k < 8; ++k) {
        const int xx = (k & 1) ? ax : x, yy = (k & 2) ? ay : y, zz = (k & 4) ? az : z;
        if (xx == kNone || yy == kNone || zz == kNone) continue;
        const int64_t p = g.p(xx, yy, zz);
#pragma unroll
        for (int j = 0; j < NP; ++j) base[(int64_t)j * g.Pst + p] = v[j];
    }
}


template <int CI, int CO>
struct ConvCfg {
    static constexpr int RING = 6;                       // input-row slots in shared memory
    static constexpr int ND = 5;                         // TMEM tiles (one per input row)
    static constexpr int NCOL = 3 * CO;                  // one tile: contributions to rows y+1, y, y-1
    static constexpr int SEGB = (CI / 8) * kSegPlane;    // one segment, all channel planes
    static constexpr int ROWB = 3 * SEGB;                // one slot: segments at z-1, z, z+1
    static constexpr int WB = 27 * CI * CO * 2;          // weight image
    static constexpr int OFF_W = RING * ROWB;
    static constexpr int OFF_BAR = OFF_W + WB;
    static constexpr int NBAR = 2 * RING + 2 * ND + 3;   // full, empty, dfull, dempty, wbar, drain x2
    static constexpr int OFF_SLOT = OFF_BAR + NBAR * 8;  // TMEM base, abort flag
    static constexpr int OFF_RED = OFF_SLOT + 16;        // [16][CO + 1] floats
    static constexpr int OFF_BIAS = (OFF_RED + 16 * (CO + 1) * 4 + 15) / 16 * 16;   // CO floats
    static constexpr int OFF_REDD = OFF_BIAS + CO * 4;   // [16] doubles
    static constexpr int SMEM = OFF_REDD + 16 * 8;
    static constexpr int TMEM_COLS = ND * NCOL <= 256 ? 256 : 512;
    // CTAs per SM: shared memory (228 KB per SM, 1 KB reserved per CTA), TMEM (512 columns per SM)
    static constexpr int BY_SMEM = 233472 / (SMEM + 1024), BY_TMEM = 512 / TMEM_COLS;
    static constexpr int CTAS = BY_SMEM < BY_TMEM ? BY_SMEM : BY_TMEM;
    static_assert(CTAS >= 1, "one CTA fits");
    // what a launch asks for: enough that no more CTAs than that share an SM
    // (a CTA beyond the TMEM of an SM would sit there until another one ends)
    static constexpr int LAUNCH_SMEM = CTAS == 1 && BY_SMEM > 1 ? 233472 / 2 : SMEM;
    // epilogue groups of four warps: as many as the registers of the CTAs hold
    // and as help (32 -> 32 channels at 256^3: 2 groups 652 us, 3 645, 4 672)
    static constexpr int groups(int epi) { return CTAS > 1 || epi == EPI_DGRAD ? 2 : 3; }
    // warps: a producer, an MMA issuer, the epilogue's, two more producers, another MMA issuer
    static constexpr int producer2(int epi) { return 2 + 4 * groups(epi); }
    static constexpr int mma2(int epi) { return producer2(epi) + 2; }
    static constexpr int threads(int epi) { return 32 * (mma2(epi) + 1); }
    // A parity wait is sound only if the phase before the awaited one is known to
    // be complete; otherwise it returns at once.  The MMA issuers take alternate
    // rows, so with an even RING the row that used a slot before is the issuer's
    // own, whose data it has waited for; with RING = 5 it was the other issuer's,
    // and an issuer could start on a row that had not arrived when an earlier
    // row's copies were late by three rows.  For the epilogue's waits, items have
    // at least two rows: over items of one row, three groups in turn lie nine
    // tiles apart, more than the ND the tile ring remembers.
    static_assert(RING % 2 == 0, "a slot's rows belong to one MMA issuer");
    static_assert(CI % 16 == 0 && CO % 16 == 0 && CO <= 32, "channel counts");
    static_assert(ND * NCOL <= 512 && NCOL <= 256, "TMEM / MMA N");
    static_assert(OFF_W % 16 == 0 && OFF_BAR % 8 == 0, "alignment");
};

struct Item {
    int z, x0, y0, y1;
};

__device__ __forceinline__ Item item_of(const NNGeom &g, int nyc, int it) {
    const int nxt = g.nx / kTileX;
    Item r;
    const int xt = it % nxt;
    const int rest = it / nxt;
    const int yi = rest % nyc;
    r.z = rest / nyc;
    r.x0 = xt * kTileX;
    r.y0 = yi * g.ny / nyc;
    r.y1 = (yi + 1) * g.ny / nyc;
    return r;
}

// Work order inside a CTA: items in turn, and in an item the input rows
// y0-1 .. y1 in order; input row number q (counted over the CTA's items)
// owns shared-memory slot q % RING and TMEM tile q % ND.  The MMAs of row q
// compute, for the 128 voxels of the tile and all three dy at once
// (N = 3 CO), D_q[v][(dy, co)] = sum over (dz, dx, ci) of
// W[dz][dy][dx][co][ci] in[z+dz][row q][x+dx][ci]; output row y is
// D_{y-1}[dy=-1] + D_y[dy=0] + D_{y+1}[dy=+1], summed by the epilogue.
template <int CI, int CO, int EPI>
__global__ void __launch_bounds__(ConvCfg<CI, CO>::threads(EPI), ConvCfg<CI, CO>::CTAS) conv_kernel(const __grid_constant__ ConvArgs a) {
    using C = ConvCfg<CI, CO>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sb = smem_u32(smem);
    const uint32_t ring = sb, wsm = sb + C::OFF_W, bars = sb + C::OFF_BAR;
    const uint32_t wbar = bars + 8 * (2 * C::RING + 2 * C::ND), dbar = wbar + 8;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + C::OFF_SLOT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::OFF_SLOT + 4);
    float *red = reinterpret_cast<float *>(smem + C::OFF_RED);
    float *sbias = reinterpret_cast<float *>(smem + C::OFF_BIAS);
    auto full = [&](uint32_t s) { return bars + 8 * s; };
    auto empty = [&](uint32_t s) { return bars + 8 * (C::RING + s); };
    auto dfull = [&](uint32_t s) { return bars + 8 * (2 * C::RING + s); };
    auto dempty = [&](uint32_t s) { return bars + 8 * (2 * C::RING + C::ND + s); };
    const NNGeom &g = a.g;

    if (tid < CO) sbias[tid] = a.bias[tid];
    if (tid == 0) {
        for (int s = 0; s < C::RING; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int s = 0; s < C::ND; ++s) {
            mbar_init(dfull(s), 1);
            mbar_init(dempty(s), 3 * 4);         // three output rows read a tile, four warps each
        }
        mbar_init(wbar, 1);
        mbar_init(dbar, 1);
        mbar_init(dbar + 8, 1);
        *abort_flag = 0;
        mbar_init_fence();
        mbar_expect_tx(wbar, C::WB);
        bulk_load(wsm, a.wimg, C::WB, wbar);
    }
    if (warp == 1) tmem_alloc(smem_u32(tslot), C::TMEM_COLS);
    // Everything above reads parameters only, which no kernel of the same pass
    // writes: it may run while the kernel before still does.
    grid_wait();
    tc_fence_before();
    __syncthreads();
    grid_release();
    tc_fence_after();
    const uint32_t tbase = *reinterpret_cast<volatile uint32_t *>(tslot);

    if (warp == 0 || (warp >= C::producer2(EPI) && warp < C::mma2(EPI))) {
        // ---------------- producers: bulk copies of input rows.  Issuing a copy
        // takes one thread 115-150 cycles, so three threads share a row's, one
        // per z plane; the first one also announces the row's bytes (copies that
        // complete before that leave the phase open: its one arrival is the
        // announcement) ----------------
        if (lane == 0) {
            const int dz = warp == 0 ? 0 : warp - C::producer2(EPI) + 1;
            uint32_t issued_q[C::RING];
#pragma unroll
            for (int s = 0; s < C::RING; ++s) issued_q[s] = 0xFFFFFFFFu;
            uint32_t q = 0;
            bool ok = true;
            for (int it = blockIdx.x; ok && it < a.items; it += gridDim.x) {
                const Item w = item_of(g, a.nyc, it);
                const unsigned char *src = reinterpret_cast<const unsigned char *>(a.x) +
                                           g.p(w.x0 - 1, w.y0 - 1, w.z + dz - 1) * 16;
                for (int r = w.y0 - 1; r <= w.y1; ++r, ++q, src += (int64_t)g.X * 16) {
                    const uint32_t s = q % C::RING;
                    // the producers run ahead of the MMAs: their waits for a free slot
                    // sleep between polls instead of taking issue slots
                    if (q >= (uint32_t)C::RING &&
                        !wait_backoff(empty(s), ((q / C::RING) + 1) & 1, a.limit_ns, abort_flag)) {
                        fail(abort_flag, a.err, 1);
                        ok = false;
                        break;
                    }
                    // test hook: the second row's barrier expects 16 bytes that never come
                    if (dz == 0)
                        mbar_expect_tx(full(s), 3 * (CI / 8) * kSegBytes + ((a.inject_stall && q == 1) ? 16u : 0u));
#pragma unroll
                    for (int k = 0; k < C::RING; ++k)
                        if (k == (int)s) issued_q[k] = q;
                    const uint32_t dst = ring + s * C::ROWB + dz * C::SEGB;
#pragma unroll
                    for (int j = 0; j < CI / 8; ++j)
                        bulk_load(dst + j * kSegPlane, src + (int64_t)j * g.Pst * 16, kSegBytes, full(s));
                }
            }
            // drain: every issued copy has landed before the CTA may exit
#pragma unroll
            for (int s = 0; s < C::RING; ++s)
                if (issued_q[s] != 0xFFFFFFFFu && !mbar_wait(full(s), (issued_q[s] / C::RING) & 1, a.limit_ns))
                    atomicOr(a.err, 4);
            if (dz == 0 && !mbar_wait(wbar, 0, a.limit_ns)) atomicOr(a.err, 4);
        }
    } else if (warp == 1 || warp == C::mma2(EPI)) {
        // ---------------- MMA issuers: one D tile per input row; one thread takes
        // the even rows, another the odd ones, so that one's waits and
        // bookkeeping (about 500 cycles a row) overlap the other's MMAs ----------
        if (lane == 0) {
            constexpr int NM = 9 * (CI / 16);              // MMAs of a row
            const uint32_t mine = warp == 1 ? 0u : 1u;
            const uint32_t idesc = idesc_bf16(128, C::NCOL, false, false);
            // descriptors of slot 0 and of the weight image; every operand
            // below is one of these plus a byte offset / 16 (no carry: all
            // shared addresses stay below 2^18).  Weight image rows for
            // (dz, dx, 8-channel group j) are (dy, co): N = 3 CO rows.
            const uint64_t a0 = smem_desc(ring, kSegPlane, 128);
            const uint64_t b0 = smem_desc(wsm, C::NCOL * 16, 128);
            bool ok = wait_or_abort(wbar, 0, a.limit_ns, abort_flag);
            if (!ok) fail(abort_flag, a.err, 1);
            uint32_t total = 0;                            // input rows of the CTA's items
            for (int it = blockIdx.x; it < a.items; it += gridDim.x) {
                const Item w = item_of(g, a.nyc, it);
                total += (uint32_t)(w.y1 - w.y0) + 2;
            }
            for (uint32_t q = mine; ok && q < total; q += 2) {
                const uint32_t sl = q % C::RING, ds = q % C::ND;
                if (!wait_or_abort(full(sl), (q / C::RING) & 1, a.limit_ns, abort_flag) ||
                    (q >= (uint32_t)C::ND &&
                     !wait_or_abort(dempty(ds), ((q / C::ND) + 1) & 1, a.limit_ns, abort_flag))) {
                    fail(abort_flag, a.err, 1);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tbase + ds * C::NCOL;
                const uint64_t ab = a0 + ((sl * C::ROWB) >> 4);
#pragma unroll
                for (int k = 0; k < NM; ++k) {             // (dz, dx, channel half)
                    const int tap = k / (CI / 16), kk = k % (CI / 16), dz = tap / 3, dx = tap % 3;
                    const uint64_t ad = ab + ((dz * C::SEGB + dx * 16 + kk * 2 * kSegPlane) >> 4);
                    const uint64_t bd = b0 + (((tap * (CI / 8) + 2 * kk) * C::NCOL * 16) >> 4);
                    mma_bf16(d, ad, bd, idesc, k ? 1u : 0u);
                }
                mma_commit(empty(sl));
                mma_commit(dfull(ds));
            }
            // drain: all issued MMAs complete before TMEM is released
            const uint32_t mydbar = dbar + 8 * mine;
            mma_commit(mydbar);
            if (!mbar_wait(mydbar, 0, a.limit_ns)) atomicOr(a.err, 4);
        }
    } else {
        // ---------------- epilogue: groups of four warps take the output rows in
        // turn (counted over the CTA's items), a warp the voxels of its TMEM lane
        // quarter, warp % 4, with all channels ----
        constexpr uint32_t NG = C::groups(EPI);
        constexpr int NEW = 4 * NG;                        // epilogue warps
        const int ew = warp - 2;
        const uint32_t grp = (uint32_t)ew >> 2;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16);
        constexpr bool STATE_OUT = EPI == EPI_STATE || EPI == EPI_LOSS;
        constexpr int CH = STATE_OUT ? 4 : 16;             // channels loaded at a time
        constexpr int NCH = STATE_OUT ? 1 : CO / 16;
        constexpr int NSUM = EPI == EPI_DGRAD ? CO / 2 : EPI == EPI_LOSS ? 2 : 1;
        V2<float> sums[NSUM];                              // per channel pair (EPI_DGRAD, EPI_LOSS)
        float lsum = 0.f;                                  // the loss
#pragma unroll
        for (int c = 0; c < NSUM; ++c) sums[c] = splat(0.f);
        Mass1 msum;
        uint32_t q = 0, rows = 0;
        bool ok = true;
        auto wait_d = [&](uint32_t t) {
            return wait_backoff(dfull(t % C::ND), (t / C::ND) & 1, a.limit_ns, abort_flag);
        };
        for (int it = blockIdx.x; ok && it < a.items; it += gridDim.x) {
            const Item w = item_of(g, a.nyc, it);
            const uint32_t qb = q, n = (uint32_t)(w.y1 - w.y0);  // input row y0 - 1; output rows
            q += n + 2;
            const int x = w.x0 + row, z = w.z;
            // halo images: one in x is a second store; those in y and z (edge rows and
            // planes) are left to store_images
            const bool xedge = x == 0 || x == g.nx - 1, zedge = z == 0 || z == g.nz - 1;
            const int dxi = xedge ? image_of(x, g.nx, g.bc) - x : 0;
            const int64_t p0 = g.p(x, w.y0, z);
            const int64_t s0 = STATE_OUT ? a.sg.at(x, w.y0, z) : 0;
            for (uint32_t i = (grp + NG - rows % NG) % NG; i < n; i += NG) {
                const int y = w.y0 + (int)i;
                const uint32_t qy = qb + i + 1;            // input row y
                const int64_t p = p0 + (int64_t)i * g.X;
                // loads that do not depend on the accumulators go first
                uint4 zl[EPI == EPI_DGRAD ? CO / 8 : 1];
                float s0v[3], s1v[3];
                const int64_t sa = s0 + (int64_t)i * a.sg.P;
                if (EPI == EPI_DGRAD) {
#pragma unroll
                    for (int j = 0; j < CO / 8; ++j)
                        zl[j] = reinterpret_cast<const uint4 *>(a.zlow)[(int64_t)j * g.Pst + p];
                }
                if (STATE_OUT) {
                    s0v[0] = a.s0.eS[sa];
                    s0v[1] = a.s0.eL[sa];
                    s0v[2] = a.s0.c[sa];
                    if (EPI == EPI_LOSS) {
                        s1v[0] = a.s1.eS[sa];
                        s1v[1] = a.s1.eL[sa];
                        s1v[2] = a.s1.c[sa];
                    }
                }
                if (!wait_d(qy - 1) || !wait_d(qy) || !wait_d(qy + 1)) {
                    fail(abort_flag, a.err, 1);
                    ok = false;
                    break;
                }
                __syncwarp();
                tc_fence_after();
                // out[y] = sum_dy W_dy in[y + dy]: the dy = -1 block of
                // D_{y-1}, the dy = 0 block of D_y, the dy = +1 block of D_{y+1}
                const uint32_t t0 = tl + ((qy - 1) % C::ND) * C::NCOL;
                const uint32_t t1 = tl + (qy % C::ND) * C::NCOL + CO;
                const uint32_t t2 = tl + ((qy + 1) % C::ND) * C::NCOL + 2 * CO;
#pragma unroll
                for (int ch = 0; ch < NCH; ++ch) {
                    uint32_t u0[CH], u1[CH], u2[CH];
                    tmem_ld(t0 + CH * ch, u0);
                    tmem_ld(t1 + CH * ch, u1);
                    tmem_ld(t2 + CH * ch, u2);
                    tmem_wait_ld(u0, u1, u2);
                    if (ch == NCH - 1) {
                        // Every tile is released by three arrivals per thread: one from
                        // each row that reads it, and at the item's ends, where fewer
                        // rows do, the missing ones from the first that does.
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(dempty((qy - 1) % C::ND), i == 0 ? 3u : 1u);
                            mbar_arrive(dempty(qy % C::ND), i == 0 ? (n > 1 ? 2u : 3u) : 1u);
                            mbar_arrive(dempty((qy + 1) % C::ND), i + 1 == n ? 3u : i + 2 == n ? 2u : 1u);
                        }
                    }
                    auto pr = [](const uint32_t(&u)[CH], int k) {
                        return V2<float>(__uint_as_float(u[2 * k]), __uint_as_float(u[2 * k + 1]));
                    };
                    V2<float> v[CH / 2];
#pragma unroll
                    for (int k = 0; k < CH / 2; ++k) v[k] = (pr(u0, k) + pr(u1, k)) + pr(u2, k);
                    if (EPI == EPI_ACT || EPI == EPI_ACT_TRAIN) {
                        uint4 o[2], zz[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            V2<float> h[4], sv[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                h[k] = v[4 * j + k] + ld2(sbias + 16 * ch + 8 * j + 2 * k);
                                sv[k] = h[k] * sigmoid2(h[k]);
                            }
                            o[j] = pack8(sv);
                            zz[j] = pack8(h);
                        }
                        uint4 *ob = reinterpret_cast<uint4 *>(a.out) + (int64_t)(2 * ch) * g.Pst;
                        ob[p] = o[0];
                        ob[g.Pst + p] = o[1];
                        if (xedge) {
                            ob[p + dxi] = o[0];
                            ob[g.Pst + p + dxi] = o[1];
                        }
                        if (zedge || y == 0 || y == g.ny - 1) store_images<2>(g, ob, x, y, z, o);
                        if (EPI == EPI_ACT_TRAIN) {
                            uint4 *zb = reinterpret_cast<uint4 *>(a.zout) + (int64_t)(2 * ch) * g.Pst;
                            zb[p] = zz[0];
                            zb[g.Pst + p] = zz[1];
                        }
                    } else if (EPI == EPI_DGRAD) {
                        uint4 o[2];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            V2<float> zi[4], dd[4];
                            unpack8(zl[2 * ch + j], zi);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const V2<float> sg = sigmoid2(zi[k]);
                                dd[k] = v[4 * j + k] * sg * fma2(zi[k], splat(1.0f) - sg, splat(1.0f));
                                sums[(8 * ch + 4 * j + k) % NSUM] = sums[(8 * ch + 4 * j + k) % NSUM] + dd[k];
                            }
                            o[j] = pack8(dd);
                        }
                        uint4 *ob = reinterpret_cast<uint4 *>(a.out) + (int64_t)(2 * ch) * g.Pst;
                        ob[p] = o[0];
                        ob[g.Pst + p] = o[1];
                        if (xedge) {
                            ob[p + dxi] = o[0];
                            ob[g.Pst + p + dxi] = o[1];
                        }
                        if (zedge || y == 0 || y == g.ny - 1) store_images<2>(g, ob, x, y, z, o);
                    } else if (EPI == EPI_STATE) {
                        const Geom &sg = a.sg;
                        const float nv[3] = {s0v[0] + a.oscale[0] * (v[0].x() + sbias[0]),
                                             s0v[1] + a.oscale[1] * (v[0].y() + sbias[1]),
                                             s0v[2] + a.oscale[2] * (v[1].x() + sbias[2])};
                        auto put = [&](int64_t b) {
                            a.s1.eS[b] = nv[0];
                            a.s1.eL[b] = nv[1];
                            a.s1.c[b] = nv[2];
                        };
                        put(sa);
                        msum.add(nv[2]);
                        // the stencil's face ghosts: written by the cell they mirror
                        if (xedge) put(sa + dxi);
                        if (zedge || y == 0 || y == g.ny - 1) {
                            const int ay = image_of(y, sg.ny, sg.bc), az = image_of(z, sg.nz, sg.bc);
                            if (ay != kNone) put(sg.at(x, ay, z));
                            if (az != kNone) put(sg.at(x, y, az));
                        }
                    } else if (EPI == EPI_LOSS) {
                        const float vv[3] = {v[0].x(), v[0].y(), v[1].x()};
                        float gr[3];
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float tg = (s1v[c] - s0v[c]) / a.oscale[c];
                            const float diff = vv[c] + sbias[c] - tg;
                            lsum += a.lw[c] * diff * diff;
                            gr[c] = 2.0f * a.lw[c] * diff;
                        }
                        const V2<float> gp[4] = {V2<float>(gr[0], gr[1]), V2<float>(gr[2], 0.f), splat(0.f), splat(0.f)};
                        sums[0] = sums[0] + gp[0];
                        sums[1 % NSUM] = sums[1 % NSUM] + gp[1];
                        const uint4 o[1] = {pack8(gp)};
                        uint4 *ob = reinterpret_cast<uint4 *>(a.out);
                        ob[p] = o[0];
                        if (xedge) ob[p + dxi] = o[0];
                        if (zedge || y == 0 || y == g.ny - 1) store_images<1>(g, ob, x, y, z, o);
                    }
                }
            }
            rows += n;
        }
        if (EPI == EPI_STATE) {
            // deterministic per-CTA FP64 sum of the new c
            double *redd = reinterpret_cast<double *>(smem + C::OFF_REDD);
            double mass = msum.get();
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
            if (lane == 0) redd[ew] = mass;
            asm volatile("bar.sync 1, %0;" ::"r"(32 * NEW) : "memory");
            if (ew == 0 && lane == 0 && a.mass_part) {
                double t = 0;
                for (int k = 0; k < NEW; ++k) t += redd[k];
                a.mass_part[blockIdx.x] = t;
            }
        }
        if (EPI == EPI_DGRAD || EPI == EPI_LOSS) {
            // deterministic per-CTA sums: warp shuffle, then the warps in order
#pragma unroll
            for (int c = 0; c < 2 * NSUM; ++c) {
                float sv = (c & 1) ? sums[c / 2].y() : sums[c / 2].x();
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sv += __shfl_xor_sync(0xffffffffu, sv, o);
                if (lane == 0) red[ew * (CO + 1) + c] = sv;
            }
            if (lane == 0)
                for (int c = 2 * NSUM; c < CO; ++c) red[ew * (CO + 1) + c] = 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
            if (lane == 0) red[ew * (CO + 1) + CO] = lsum;
            asm volatile("bar.sync 1, %0;" ::"r"(32 * NEW) : "memory");
            if (ew == 0) {
                float *dst = a.partials + (int64_t)blockIdx.x * (CO + 1);
                for (int c = lane; c <= CO; c += 32) {
                    float t = 0.f;
                    for (int k = 0; k < NEW; ++k) t += red[k * (CO + 1) + c];
                    dst[c] = t;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tbase, C::TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------

template <int CX, int CZ>
struct WgCfg {
    static constexpr int PL = kTileX * 16;                // one 8-channel plane of a row
    static constexpr int NX = 3, NZ = 5;                  // rows of X, of dZ in shared memory
    static constexpr int XSEG = (CX / 8) * PL;            // one z plane of a row of X
    static constexpr int XB = 16 * PL;                    // M = 128 channels: three planes, then zeros
    static constexpr int ZSEG = (CZ / 8) * PL, ZB = 3 * ZSEG;
    static constexpr int OFF_Z = NX * XB;
    static constexpr int OFF_BAR = OFF_Z + NZ * ZB;
    static constexpr int NBAR = 2 * NX + 1;
    static constexpr int OFF_SLOT = OFF_BAR + NBAR * 8;
    static constexpr int SMEM = OFF_SLOT + 16;
    static constexpr int NCOL = 3 * CZ;                   // one accumulator: dx, co
    static constexpr int TMEM_COLS = 3 * NCOL <= 256 ? 256 : 512;
    static_assert(3 * NCOL <= 512 && 3 * XSEG <= XB, "TMEM columns, M");
};

// A CTA's rows t0 .. t1-1 (y fastest, then x tile, then z) in columns: rows
// ya .. yb-1 of one column at a time.
struct WgCol {
    int x0, z, ya, yb;
};

__device__ __forceinline__ WgCol wg_col(const NNGeom &g, int t, int t1) {
    const int nxt = g.nx / kTileX, col = t / g.ny;
    WgCol c;
    c.ya = t - col * g.ny;
    c.yb = min(g.ny, c.ya + (t1 - t));
    c.x0 = (col % nxt) * kTileX;
    c.z = col / nxt;
    return c;
}

template <int CX, int CZ>
__global__ void __launch_bounds__(256, 1) wgrad_kernel(const __grid_constant__ WgradArgs a) {
    using C = WgCfg<CX, CZ>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sb = smem_u32(smem), bars = sb + C::OFF_BAR;
    auto full = [&](uint32_t s) { return bars + 8 * s; };
    auto empty = [&](uint32_t s) { return bars + 8 * (C::NX + s); };
    const uint32_t dbar = bars + 8 * (2 * C::NX);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + C::OFF_SLOT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::OFF_SLOT + 4);
    const NNGeom &g = a.g;
    const int t0 = (int)((int64_t)a.ntiles * blockIdx.x / gridDim.x);
    const int t1 = (int)((int64_t)a.ntiles * (blockIdx.x + 1) / gridDim.x);

    // the channels of M past the three z planes read as zeros
    for (int st = 0; st < C::NX; ++st)
        for (int i = tid; i < (C::XB - 3 * C::XSEG) / 16; i += blockDim.x)
            reinterpret_cast<uint4 *>(smem + st * C::XB + 3 * C::XSEG)[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
    if (tid == 0) {
        for (int s = 0; s < C::NX; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(dbar, 1);
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(smem_u32(tslot), C::TMEM_COLS);
    grid_wait();
    tc_fence_before();
    __syncthreads();
    grid_release();
    tc_fence_after();
    const uint32_t tbase = *reinterpret_cast<volatile uint32_t *>(tslot);

    // Unit n (counted over the CTA's columns) is a row r of X, ya - 1 .. yb, in
    // X slot n % NX, and with it row r + 1 of dZ, the z-th of the CTA's, in dZ
    // slot z % NZ.  A dZ row is last used by the second unit after the one that
    // loads it, so when unit n - NX is done, the dZ slot is free too (NZ = NX + 2).
    if (warp == 0 || warp >= 6) {
        // ---- producers: thread k loads z plane k - 1 of X and the dZ row shifted by
        // 1 - k; the first one announces the unit's bytes ----
        if (lane == 0) {
            const int k = warp == 0 ? 0 : warp - 5;
            uint32_t n = 0, zr = 0;
            bool ok = true;
            for (int t = t0; ok && t < t1;) {
                const WgCol c = wg_col(g, t, t1);
                for (int r = c.ya - 1; r <= c.yb; ++r, ++n) {
                    const uint32_t st = n % C::NX;
                    if (n >= (uint32_t)C::NX &&
                        !wait_backoff(empty(st), ((n / C::NX) + 1) & 1, a.limit_ns, abort_flag)) {
                        fail(abort_flag, a.err, 1);
                        ok = false;
                        break;
                    }
                    const bool z = r + 1 < c.yb;
                    if (k == 0) mbar_expect_tx(full(st), 3 * C::XSEG + (z ? C::ZB : 0));
                    const unsigned char *xs = reinterpret_cast<const unsigned char *>(a.x) + g.p(c.x0, r, c.z + k - 1) * 16;
#pragma unroll
                    for (int j = 0; j < CX / 8; ++j)
                        bulk_load(sb + st * C::XB + k * C::XSEG + j * C::PL, xs + (int64_t)j * g.Pst * 16, C::PL, full(st));
                    if (z) {
                        const unsigned char *zs = reinterpret_cast<const unsigned char *>(a.dz) +
                                                  g.p(c.x0 + 1 - k, r + 1, c.z) * 16;
                        const uint32_t dst = sb + C::OFF_Z + (zr % C::NZ) * C::ZB + k * C::ZSEG;
#pragma unroll
                        for (int j = 0; j < CZ / 8; ++j)
                            bulk_load(dst + j * C::PL, zs + (int64_t)j * g.Pst * 16, C::PL, full(st));
                        ++zr;
                    }
                }
                t += c.yb - c.ya;
            }
            // drain the copies of the last units
            for (uint32_t i = n > (uint32_t)C::NX ? n - C::NX : 0; i < n; ++i)
                if (!mbar_wait(full(i % C::NX), (i / C::NX) & 1, a.limit_ns)) atomicOr(a.err, 4);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(128, C::NCOL, true, true);
            // MN-major operands: LBO = stride of 8-voxel K groups (128 B), SBO =
            // stride of 8-channel groups (a plane)
            const uint64_t a0 = smem_desc(sb, 128, C::PL);
            const uint64_t b0 = smem_desc(sb + C::OFF_Z, 128, C::PL);
            uint32_t n = 0, zr = 0;                        // units; dZ rows of earlier columns
            uint32_t begun = 0;                            // accumulators written so far (bits)
            bool ok = true;
            auto ready = [&](uint32_t u) {
                if (ok && !wait_or_abort(full(u % C::NX), (u / C::NX) & 1, a.limit_ns, abort_flag)) {
                    fail(abort_flag, a.err, 1);
                    ok = false;
                }
            };
            if (t0 < t1) ready(0);
            for (int t = t0; ok && t < t1;) {
                const WgCol c = wg_col(g, t, t1);
                t += c.yb - c.ya;
                for (int r = c.ya - 1; ok && r <= c.yb; ++r, ++n) {
                    tc_fence_after();
                    const uint64_t ax = a0 + (((n % C::NX) * C::XB) >> 4);
#pragma unroll
                    for (int dy = 0; dy < 3; ++dy) {       // X row r meets dZ row y = r - (dy - 1)
                        const int y = r + 1 - dy;
                        // before the last MMAs of a unit, wait for the next one, so that its
                        // MMAs follow at once
                        if (dy == 2 && (r < c.yb || t < t1)) ready(n + 1);
                        if (y < c.ya || y >= c.yb) continue;
                        const uint64_t bz = b0 + ((((zr + (uint32_t)(y - c.ya)) % C::NZ) * C::ZB) >> 4);
                        const uint32_t d = tbase + dy * C::NCOL;
                        const uint32_t more = (begun >> dy) & 1u;
#pragma unroll
                        for (int kb = 0; kb < kTileX / 16; ++kb)
                            mma_bf16(d, ax + kb * 16, bz + kb * 16, idesc, kb ? 1u : more);
                        begun |= 1u << dy;
                    }
                    mma_commit(empty(n % C::NX));
                }
                zr += (uint32_t)(c.yb - c.ya);
            }
            mma_commit(dbar);
        }
    }
    // epilogue: all four lane quarters; wait for the last MMA
    if (warp >= 2 && warp < 6) {
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const bool have = t1 > t0;
        bool ok = true;
        if (!wait_or_abort(dbar, 0, a.limit_ns, abort_flag)) {
            fail(abort_flag, a.err, 1);
            ok = false;
        }
        __syncwarp();
        tc_fence_after();
        float *out = a.partials + (int64_t)blockIdx.x * 27 * CZ * CX;
        const int dz = row / CX, ci = row % CX;
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int c16 = 0; c16 < C::NCOL / 16; ++c16) {
                float v[16];
                tmem_ld16(tbase + ((uint32_t)(quarter * 32) << 16) + dy * C::NCOL + 16 * c16, v);
                if (dz < 3) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int dx = (16 * c16 + i) / CZ, co = (16 * c16 + i) % CZ;
                        out[((int64_t)(dz * 9 + dy * 3 + dx) * CZ + co) * CX + ci] = (ok && have) ? v[i] : 0.f;
                    }
                }
            }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        // make sure no MMA is still running on an aborted CTA
        if (lane == 0 && !mbar_wait(dbar, 0, a.limit_ns)) atomicOr(a.err, 4);
        __syncwarp();
        tmem_dealloc(tbase, C::TMEM_COLS);
    }
}

template <int CI, int CO, int EPI>
cudaError_t conv_launch(const ConvArgs &a, int grid, cudaStream_t s) {
    using C = ConvCfg<CI, CO>;
    return launch_pdl(conv_kernel<CI, CO, EPI>, grid, C::threads(EPI), C::LAUNCH_SMEM, a, s);
}

template <int CI, int CO>
cudaError_t conv_launch_epi(int epi, const ConvArgs &a, int grid, cudaStream_t s) {
    switch (epi) {
        case EPI_ACT: return conv_launch<CI, CO, EPI_ACT>(a, grid, s);
        case EPI_ACT_TRAIN: return conv_launch<CI, CO, EPI_ACT_TRAIN>(a, grid, s);
        case EPI_DGRAD: return conv_launch<CI, CO, EPI_DGRAD>(a, grid, s);
        case EPI_STATE: return CO == 16 ? conv_launch<CI, 16, EPI_STATE>(a, grid, s) : cudaErrorInvalidValue;
        case EPI_LOSS: return CO == 16 ? conv_launch<CI, 16, EPI_LOSS>(a, grid, s) : cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
    }
}

template <int CI, int CO, int EPI>
cudaError_t conv_attr() {
    return cudaFuncSetAttribute(conv_kernel<CI, CO, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                ConvCfg<CI, CO>::LAUNCH_SMEM);
}

template <int CI, int CO>
cudaError_t conv_attr_all() {
    cudaError_t e;
    if ((e = conv_attr<CI, CO, EPI_ACT>()) != cudaSuccess) return e;
    if ((e = conv_attr<CI, CO, EPI_ACT_TRAIN>()) != cudaSuccess) return e;
    if ((e = conv_attr<CI, CO, EPI_DGRAD>()) != cudaSuccess) return e;
    if (CO == 16) {
        if ((e = conv_attr<CI, 16, EPI_STATE>()) != cudaSuccess) return e;
        if ((e = conv_attr<CI, 16, EPI_LOSS>()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int CX, int CZ>
cudaError_t wgrad_attr() {
    return cudaFuncSetAttribute(wgrad_kernel<CX, CZ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                WgCfg<CX, CZ>::SMEM);
}

}  // namespace

template <int CI, int CO>
int conv_per_sm() {
    return ConvCfg<CI, CO>::CTAS;
}

int conv_ctas_per_sm(int ci, int co) {
    if (ci == 16 && co == 16) return conv_per_sm<16, 16>();
    if (ci == 16 && co == 32) return conv_per_sm<16, 32>();
    if (ci == 32 && co == 16) return conv_per_sm<32, 16>();
    if (ci == 32 && co == 32) return conv_per_sm<32, 32>();
    return 1;
}

cudaError_t conv_setup(int max_smem_optin) {
    if (WgCfg<32, 32>::SMEM > max_smem_optin || ConvCfg<32, 32>::SMEM > max_smem_optin) return cudaErrorInvalidValue;
    cudaError_t e;
    if ((e = conv_attr_all<16, 16>()) != cudaSuccess) return e;
    if ((e = conv_attr_all<16, 32>()) != cudaSuccess) return e;
    if ((e = conv_attr_all<32, 16>()) != cudaSuccess) return e;
    if ((e = conv_attr_all<32, 32>()) != cudaSuccess) return e;
    if ((e = wgrad_attr<16, 16>()) != cudaSuccess) return e;
    if ((e = wgrad_attr<16, 32>()) != cudaSuccess) return e;
    if ((e = wgrad_attr<32, 16>()) != cudaSuccess) return e;
    return wgrad_attr<32, 32>();
}

cudaError_t launch_conv(int ci, int co, int epi, const ConvArgs &a, int grid, cudaStream_t s) {
    if (ci == 16 && co == 16) return conv_launch_epi<16, 16>(epi, a, grid, s);
    if (ci == 16 && co == 32) return conv_launch_epi<16, 32>(epi, a, grid, s);
    if (ci == 32 && co == 16) return conv_launch_epi<32, 16>(epi, a, grid, s);
    if (ci == 32 && co == 32) return conv_launch_epi<32, 32>(epi, a, grid, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_wgrad(int cx, int cz, const WgradArgs &a, int grid, cudaStream_t s) {
    if (cx == 16 && cz == 16) return launch_pdl(wgrad_kernel<16, 16>, grid, 256, WgCfg<16, 16>::SMEM, a, s);
    if (cx == 16 && cz == 32) return launch_pdl(wgrad_kernel<16, 32>, grid, 256, WgCfg<16, 32>::SMEM, a, s);
    if (cx == 32 && cz == 16) return launch_pdl(wgrad_kernel<32, 16>, grid, 256, WgCfg<32, 16>::SMEM, a, s);
    if (cx == 32 && cz == 32) return launch_pdl(wgrad_kernel<32, 32>, grid, 256, WgCfg<32, 32>::SMEM, a, s);
    return cudaErrorInvalidValue;
}

}  // namespace nn
}  // namespace ppf
