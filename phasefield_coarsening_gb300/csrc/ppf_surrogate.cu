// ppf_surrogate.cu -- the learned time-stepping surrogate (a 3-D
// convolutional network that advances an FP32 state by k explicit steps in
// one call), its training on the device, and the FP64 solute-mass
// projection.  No counterpart in the reference: the reference only has
// the explicit step (phasefield.c:301-476) that this network stands in for
// and that trains it, corrects it and measures its error.
//
// Network: six 3x3x3 convolutions, 16 -> W -> W -> W -> W -> W -> 16
// channels (W = 16 or 32), SiLU after the first five, residual output:
//   state(t + k dt) = state(t) + out_scale * net(features(state(t)))
// for the three fields (etaS, etaL, c); output channels 3..15 and input
// channels 5..15 are zero padding that keeps every GEMM K and N a multiple
// of 16.  Input features: etaS, etaL, (c - c_eq(h)) * in_scale_c with
// h = etaS^2 / (etaS^2 + etaL^2) (the reference's interpolation,
// phasefield.c:331) and c_eq(h) = h c_solid + (1-h) c_liquid, so the
// composition enters as its (small) departure from local equilibrium,
// which BF16 represents to 2^-8 relative; then 256 (etaS - bf16(etaS)) and
// 256 (etaL - bf16(etaL)), the part of each phase field BF16 drops.
//
// After every call the solute mass sum(c) is projected back, in FP64, to
// its value before the call: the deficit is spread over the cells as whole
// units of 2^-24 (one FP32 ulp on [0.5, 1)) by a Bresenham rule, so the
// FP32 sum lands on the target to within about one ulp; a second pass
// removes what rounding at other binades left.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "ppf.h"
#include "ppf_ctx.h"
#include "ppf_internal.h"
#include "ppf_nn.h"
#include "ppf_pair.h"

using namespace ppf;
using namespace ppf::nn;

namespace {

constexpr int kLayers = 6;
constexpr int kNT = 256;

int serr(int code, const char *fmt, ...) {
    char buf[400];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    return set_last_error(code, buf);
}

#define SCU(x)                                                                                   \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess) return serr(PPF_ECUDA, "%s: %s", #x, cudaGetErrorString(e_));     \
    } while (0)

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// the halo image of interior coordinate x, or kNone (periodic: x=0 -> n,
// x=n-1 -> -1; no-flux: x=0 -> -1, x=n-1 -> n)
constexpr int kNone = -0x40000000;
__device__ __forceinline__ int image_of(int x, int n, int bc) {
    return x == 0 ? (bc == 0 ? n : -1) : x == n - 1 ? (bc == 0 ? -1 : n) : kNone;
}

__device__ __forceinline__ void block_sum_to(double s, double *out) {
    __shared__ double red[kNT / 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < kNT / 32; ++w) t += red[w];
        *out = t;
    }
}

// state (FP32, stencil layout) -> first channel plane of the 16-channel
// BF16 features (etaS, etaL, composition feature; channels 8..15 live in
// the second plane, zero from allocation and never written), with every
// halo image; also the per-CTA FP64 sum of c (the mass before the call).
// Bound by HBM: 12 bytes read and 16 written per cell.  A warp takes 128
// voxels of a row, lane after lane, so that each 16-byte store instruction
// fills whole lines; images are stored only by the rows and voxels that have
// them, and the mass is summed in three floats per thread: a conversion and
// an addition in FP64 per cell took longer than the memory traffic.  256^3:
// 78 us, was 152 us.
__global__ void __launch_bounds__(kNT) features_kernel(Geom sg, Fields<const float> s, NNGeom g, uint16_t *act,
                                                       float cS, float cL, float kc, double *mass_part) {
    Mass<float> m;
    uint4 *out = reinterpret_cast<uint4 *>(act);
    const int lane = threadIdx.x & 31;
    const int per = g.nx / kTileX;
    const int nw = g.nz * g.ny * per;
    for (int w = blockIdx.x * (kNT / 32) + (threadIdx.x >> 5); w < nw; w += gridDim.x * (kNT / 32)) {
        const int row = w / per, x0 = (w - row * per) * kTileX + lane;
        const int z = row / g.ny, y = row - z * g.ny;
        const int64_t a0 = sg.at(x0, y, z);
        float eS[4], eL[4], c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            eS[k] = s.eS[a0 + 32 * k];
            eL[k] = s.eL[a0 + 32 * k];
            c[k] = s.c[a0 + 32 * k];
        }
        m.add(V2<float>(c[0], c[1]));
        m.add(V2<float>(c[2], c[3]));
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float s2 = eS[k] * eS[k], l2 = eL[k] * eL[k];
            const float h = s2 / fmaxf(s2 + l2, 1e-30f);
            const float f2 = (c[k] - (cL + (cS - cL) * h)) * kc;
            // what BF16 drops of etaS and etaL, scaled into range: with
            // channels 0-1 the network sees both fields to ~16 bits
            const uint32_t hi = pack2(eS[k], eL[k]);
            const float rS = (eS[k] - __uint_as_float(hi << 16)) * 256.0f;
            const float rL = (eL[k] - __uint_as_float(hi & 0xFFFF0000u)) * 256.0f;
            v[k] = make_uint4(hi, pack2(f2, rS), pack2(rL, 0.f), 0u);
        }
        const int ay = image_of(y, g.ny, g.bc), az = image_of(z, g.nz, g.bc);
        for (int q = 0; q < 4; ++q) {
            const int yy = (q & 1) ? ay : y, zz = (q & 2) ? az : z;
            if (yy == kNone || zz == kNone) continue;
            uint4 *o = out + g.p(0, yy, zz);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = x0 + 32 * k;
                o[x] = v[k];
                const int ax = image_of(x, g.nx, g.bc);
                if (ax != kNone) o[ax] = v[k];
            }
        }
    }
    block_sum_to(m.get(), mass_part + blockIdx.x);
}

// The projection moves sum(c) by R = round((target - sum) / 2^-24) units of
// 2^-24: every cell by `base` units and `rem` cells by one more, where
// base = floor(R / n), rem = R - base n in [0, n); the extra unit goes to
// the cells i where floor(i rem / n) steps up, (i rem mod n) + rem >= n,
// evenly spread.
struct MassPlan {
    double target, sum;
};

struct Shift {
    long long base, rem;
};

__device__ __forceinline__ Shift shift_of(const MassPlan &mp, long long n) {
    const double d = (mp.target - mp.sum) * 16777216.0;     // in units of 2^-24
    long long R = 0;
    if (fabs(d) < 4.0e18) R = llrint(d);                     // non-finite or absurd: leave c alone
    Shift s{R / n, R % n};
    if (s.rem < 0) {
        s.rem += n;
        s.base -= 1;
    }
    return s;
}

constexpr float kUnit = 5.9604644775390625e-08f;             // 2^-24

// (a call, so that its FP64 operations are not predicated into the loop: at
// 1/64 of the FP32 rate they cost the same whether they take effect or not)
__device__ __noinline__ float add_wide(float v, long long base) {
    return (float)((double)v + (double)base * (double)kUnit);
}

// One pass over the rows of c, a warp per row and four cells per lane:
// APPLY adds each cell its `base` units of 2^-24 and then, rounded by itself,
// the extra one (both exact in FP32 up to 2^24 units), SUM leaves the per-CTA FP64 sums
// of the resulting c, three floats per thread (more than an FP64 running sum
// keeps).  Bound by memory, mostly the L2, which holds the 67 MB of c at
// 256^3: 41 us with both, 6 us adding few units.  A pass of its own for the
// sum (79 us: an FP64 conversion and addition per cell), one over all cells
// for `base` (21 us) and one scattered over `rem` cells (58 us) did the same
// before.  Products of 64 bits: rows x rem stays below 2^63 for any domain
// that fits in memory.  N holds a cell's i rem mod n plus rem: 32 bits below
// 2^31 cells.
template <typename N, bool APPLY, bool SUM>
__global__ void __launch_bounds__(kNT) mass_kernel(Geom sg, float *c, const MassPlan *mp, double *partials) {
    __shared__ Shift sh;
    const long long n = (long long)sg.nx * sg.ny * sg.nz;
    Shift s{0, 0};
    if (APPLY) {
        if (threadIdx.x == 0) sh = shift_of(*mp, n);
        __syncthreads();
        s = sh;
        if (!SUM && s.base == 0 && s.rem == 0) return;
    }
    const bool narrow = s.base >= -(1 << 24) && s.base <= (1 << 24);
    const float add = (float)s.base * kUnit;
    const int lane = threadIdx.x & 31, nwarps = gridDim.x * (kNT / 32);
    const int nrows = sg.ny * sg.nz, row0 = blockIdx.x * (kNT / 32) + (threadIdx.x >> 5);
    // i rem mod n of the thread's next row, kept by additions, and its
    // advances: the next row's, 128 cells'
    const N nn = (N)n, rem = (N)s.rem;
    auto mod_add = [&](N &u, N d) {
        u += d;
        const bool over = u >= nn;
        if (over) u -= nn;
        return over;
    };
    N trow = 0, rrow = 0, r128 = 0;
    if (APPLY) {
        const long long per_row = sg.nx * s.rem % n;
        trow = (N)(row0 * per_row % n);
        mod_add(trow, (N)(4 * lane * s.rem % n));
        rrow = (N)(nwarps * per_row % n);
        r128 = (N)(128 * s.rem % n);
    }
    Mass<float> m;
    for (int row = row0; row < nrows; row += nwarps) {
        const int z = row / sg.ny, y = row - z * sg.ny;
        const int64_t a0 = sg.at(0, y, z);
        const int ay = image_of(y, sg.ny, sg.bc), az = image_of(z, sg.nz, sg.bc);
        N t = trow;
        mod_add(trow, rrow);
        for (int x = 4 * lane; x < sg.nx; x += 128) {
            unsigned extra = 0;                              // bit k: cell x + k takes one unit more
            if (APPLY) {
                N u = t;
#pragma unroll
                for (int k = 0; k < 4; ++k) extra |= (unsigned)mod_add(u, rem) << k;
                mod_add(t, r128);
                if (!SUM && s.base == 0 && !extra) continue;
            }
            // rows start on 32 bytes and are padded to 8 cells past the last
            // halo cell: the load stays inside the row
            const float4 q = *reinterpret_cast<const float4 *>(c + a0 + x);
            float v[4] = {q.x, q.y, q.z, q.w};
            const int nk = min(4, sg.nx - x);
            if (APPLY) {
                if (narrow) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] += add;
                } else {
                    for (int k = 0; k < 4; ++k) v[k] = add_wide(v[k], s.base);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] += extra >> k & 1 ? kUnit : 0.f;
                auto put = [&](int64_t a) {
                    if (nk == 4) {
                        *reinterpret_cast<float4 *>(c + a) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
                        for (int k = 0; k < nk; ++k) c[a + k] = v[k];
                    }
                };
                put(a0 + x);
                if (ay != kNone) put(sg.at(x, ay, z));
                if (az != kNone) put(sg.at(x, y, az));
                if (x == 0) c[sg.at(image_of(0, sg.nx, sg.bc), y, z)] = v[0];
                if (x + nk == sg.nx && sg.nx > 1) c[sg.at(image_of(sg.nx - 1, sg.nx, sg.bc), y, z)] = v[nk - 1];
            }
            if (SUM) {
                m.add(V2<float>(v[0], nk > 1 ? v[1] : 0.f));
                m.add(V2<float>(nk > 2 ? v[2] : 0.f, nk > 3 ? v[3] : 0.f));
            }
        }
    }
    if (SUM) block_sum_to(m.get(), partials + blockIdx.x);
}

// The partial sums of a training step: per job, out[i] = sum_b
// part[b * stride + i] for i < n, in a fixed order; job 0 also has the loss
// behind its n values.  Blocks first[j] .. first[j + 1] - 1 have job j.
constexpr int kJobs = 2 * kLayers;
struct ReduceJobs {
    const float *part[kJobs];
    float *out[kJobs];
    int nb[kJobs], stride[kJobs], n[kJobs], first[kJobs + 1];
    double *loss;
};

// the plain FP64 sum, for sums that floats do not hold
__device__ __noinline__ double wide_sum(const float *part, int nb, int stride) {
    double s = 0;
    for (int b = 0; b < nb; ++b) s += (double)part[(int64_t)b * stride];
    return s;
}

// A block takes 32 values, its eight warps an eighth of the partial sums each:
// independent loads in flight instead of one thread's chain (21 us for 152
// partials of 27 x 32 x 32 weights), and sums in three floats (about 72 bits,
// more than an FP64 sum keeps) instead of FP64, whose conversions and additions
// alone would take 14 us; one that overflows or holds no number is summed in
// FP64 after all.  All jobs of a step in one launch: 33 us for the 84 MB of a
// width-32 network (62 us in twelve launches; 42 us with the eight parts of a
// value put together by one lane; 24 us in two floats, 48 bits).
__global__ void __launch_bounds__(kNT) reduce_kernel(const __grid_constant__ ReduceJobs q) {
    __shared__ Mass1 red[kNT / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int j = 0;
    while ((int)blockIdx.x >= q.first[j + 1]) ++j;
    const int nb = q.nb[j], n = q.n[j];
    const int nv = n + (j == 0 ? 1 : 0);
    const int b0 = nb * warp / (kNT / 32), b1 = nb * (warp + 1) / (kNT / 32);
    const int i = ((int)blockIdx.x - q.first[j]) * 32 + lane;
    const float *part = q.part[j] + i;
    Mass1 s;
    if (i < nv) {
#pragma unroll 8
        for (int b = b0; b < b1; ++b) s.add(part[(int64_t)b * q.stride[j]]);
    }
    red[warp][lane] = s;
    __syncthreads();
    // eight lanes per value now
    static_assert(kNT == 256, "32 values of eight parts");
    const int v = i - lane + ((int)threadIdx.x >> 3);
    s = red[threadIdx.x & 7][threadIdx.x >> 3];
#pragma unroll
    for (int d = 1; d < 8; d *= 2) {
        const float hi = __shfl_xor_sync(0xffffffffu, s.hi, d), mid = __shfl_xor_sync(0xffffffffu, s.mid, d);
        const float lo = __shfl_xor_sync(0xffffffffu, s.lo, d);
        s.add(hi);
        s.add(mid);
        s.lo += lo;
    }
    if ((threadIdx.x & 7) == 0 && v < nv) {
        double t = s.get();
        if (!isfinite(t)) t = wide_sum(q.part[j] + v, nb, q.stride[j]);
        if (v < n) q.out[j][v] = (float)t;
        else *q.loss = t;
    }
}

// Where a layer's weights stand among the parameters, and their BF16 images.
struct PackTable {
    int64_t n;                   // parameters
    int64_t woff[kLayers];
    int ci[kLayers], co[kLayers];
    uint16_t *wf[kLayers], *wb[kLayers];
};

// W[27][co][ci] (FP32, tap = 9 dz + 3 dy + dx over 0..2) -> the BF16
// B-operand images of the convolution kernel, [dz][dx][ci/8][dy][co][8]
// (one MMA's N = 3 co rows are the three dy taps), forward and for the
// input-gradient convolution (taps reversed, ci and co swapped).
__device__ __forceinline__ void pack_weight(const PackTable &t, int64_t p, float w) {
    int l = kLayers - 1;
    while (p < t.woff[l]) --l;
    const int i = (int)(p - t.woff[l]), ci = t.ci[l], co = t.co[l];
    if (i >= 27 * ci * co) return;                           // a bias
    const int c_in = i % ci, c_out = (i / ci) % co, tap = i / (ci * co);
    const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
    const __nv_bfloat16 h = __float2bfloat16_rn(w);
    const uint16_t u = *reinterpret_cast<const uint16_t *>(&h);
    t.wf[l][((((int64_t)(dz * 3 + dx) * (ci / 8) + c_in / 8) * 3 + dy) * co + c_out) * 8 + (c_in & 7)] = u;
    const int rz = 2 - dz, ry = 2 - dy, rx = 2 - dx;
    t.wb[l][((((int64_t)(rz * 3 + rx) * (co / 8) + c_out / 8) * 3 + ry) * ci + c_in) * 8 + (c_out & 7)] = u;
}

__global__ void __launch_bounds__(kNT) pack_kernel(const __grid_constant__ PackTable t, const float *p) {
    for (int64_t i = blockIdx.x * (int64_t)kNT + threadIdx.x; i < t.n; i += (int64_t)gridDim.x * kNT) pack_weight(t, i, p[i]);
}

__global__ void __launch_bounds__(kNT) adam_kernel(const __grid_constant__ PackTable t, float *p, const float *g, float *m,
                                                   float *v, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int64_t i = blockIdx.x * (int64_t)kNT + threadIdx.x; i < t.n; i += (int64_t)gridDim.x * kNT) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = w;
        pack_weight(t, i, w);
    }
}

}  // namespace

struct ppf_surrogate {
    ppf_surrogate_config cfg;
    int W = 0;
    int dev = 0, num_sms = 0;
    int ci[kLayers], co[kLayers];
    int64_t woff[kLayers], boff[kLayers], nparams = 0;
    float *params = nullptr, *grads = nullptr, *mom1 = nullptr, *mom2 = nullptr;
    uint16_t *wf[kLayers] = {}, *wb[kLayers] = {};
    int64_t adam_t = 0;
    // workspace for one domain shape
    int wz = 0, wy = 0, wx = 0, wbc = -1;
    NNGeom g{};
    uint16_t *feat = nullptr, *act[5] = {}, *zp[5] = {}, *g16 = nullptr, *gw[2] = {};
    bool train_ready = false;    // g16, gw, zp allocated for the current shape
    // per-CTA sums of all layers (training): weight gradients, bias gradients
    // and the loss, summed up in one launch at the end of the backward pass
    float *wpart = nullptr, *bpart = nullptr;
    double *mpart = nullptr;     // per-CTA sums of c after a call (output layer)
    double *dscal = nullptr;     // [0] loss
    float *scratch = nullptr;    // predictions: zero state + output state
    double *stage = nullptr;
    size_t scratch_elems = 0;
    int conv_grid[2][2] = {}, wgrad_grid = 0;
    int nyc[2][2] = {};          // work items per column of the current shape
    int inject = 0;              // test hook: the next convolution's wait runs out
};

namespace {

void free_train(ppf_surrogate *s) {
    for (auto &p : s->zp) cudaFree(p), p = nullptr;
    for (auto &p : s->gw) cudaFree(p), p = nullptr;
    cudaFree(s->g16);
    s->g16 = nullptr;
    s->train_ready = false;
}

// buffers may still be in use by work queued on any context's stream: the
// whole device is synchronised before anything is freed
void free_ws(ppf_surrogate *s) {
    cudaDeviceSynchronize();
    free_train(s);
    cudaFree(s->feat);
    for (auto &p : s->act) cudaFree(p), p = nullptr;
    cudaFree(s->scratch);
    cudaFree(s->stage);
    s->feat = nullptr;
    s->scratch = nullptr;
    s->stage = nullptr;
    s->scratch_elems = 0;
    s->wz = s->wy = s->wx = 0;
    s->wbc = -1;
}

int alloc_zero(void **p, size_t bytes, cudaStream_t st) {
    SCU(cudaMalloc(p, bytes));
    SCU(cudaMemsetAsync(*p, 0, bytes, st));
    return PPF_OK;
}

int check_ctx(ppf_ctx *c) {
    if (!c) return serr(PPF_EINVAL, "null context");
    if (c->prec != PPF_F32) return serr(PPF_EINVAL, "the surrogate runs on FP32 contexts");
    if (c->nx % kTileX != 0) return serr(PPF_EINVAL, "the surrogate needs an x edge that is a multiple of %d", kTileX);
    if (c->ny < 2 || c->nz < 2) return serr(PPF_EINVAL, "the surrogate needs y and z edges of at least 2");
    if (!c->uploaded) return serr(PPF_ESTATE, "no state uploaded");
    return PPF_OK;
}

// Work items per column of ny rows, of at least two rows each: a CTA's rows
// are its items' plus two halo rows each, so a count that gives the busiest CTA
// few of them (64 x 128 x 128 on 152 CTAs: items of 18-19 rows, 63 in all,
// where 4-row items made 84); of counts within 2 % the largest, whose CTAs stay
// closer together in z and share more of their input rows through the L2
// (256^3: 32 rows 45.9 ms a cycle of ten calls, 128 rows 46.9 ms).
int pick_nyc(const NNGeom &g, int grid) {
    const int64_t cols = (int64_t)g.nz * (g.nx / kTileX);
    auto rows = [&](int k) { return (cols * k + grid - 1) / grid * ((g.ny + k - 1) / k + 2); };
    int64_t least = rows(1);
    for (int k = 2; k <= g.ny / 2; ++k) least = std::min(least, rows(k));
    for (int k = g.ny / 2;; --k)
        if (rows(k) * 50 <= least * 51) return k;
}

int ensure_ws(ppf_surrogate *s, ppf_ctx *c, bool train) {
    int rc = check_ctx(c);
    if (rc) return rc;
    if (c->dev != s->dev) return serr(PPF_EINVAL, "context and surrogate on different devices");
    if (s->wz != c->nz || s->wy != c->ny || s->wx != c->nx || s->wbc != c->bc) {
        free_ws(s);
        s->g = make_nngeom(c->nz, c->ny, c->nx, c->bc);
        if ((rc = alloc_zero((void **)&s->feat, act_bytes(s->g, 16), c->stream))) return rc;
        for (auto &p : s->act)
            if ((rc = alloc_zero((void **)&p, act_bytes(s->g, s->W), c->stream))) return rc;
        for (int p = 0; p < 2; ++p)
            for (int q = 0; q < 2; ++q) s->nyc[p][q] = pick_nyc(s->g, s->conv_grid[p][q]);
        s->wz = c->nz;
        s->wy = c->ny;
        s->wx = c->nx;
        s->wbc = c->bc;
    }
    if (train && !s->train_ready) {
        // all or nothing: a failure leaves no half-allocated training set
        rc = alloc_zero((void **)&s->g16, act_bytes(s->g, 16), c->stream);
        for (auto &p : s->gw)
            if (!rc) rc = alloc_zero((void **)&p, act_bytes(s->g, s->W), c->stream);
        for (auto &p : s->zp)
            if (!rc) rc = alloc_zero((void **)&p, act_bytes(s->g, s->W), c->stream);
        if (!rc && !s->wpart && cudaMalloc(&s->wpart, (size_t)s->wgrad_grid * s->nparams * sizeof(float)) != cudaSuccess)
            rc = serr(PPF_ENOMEM, "no memory for the weight gradients' partial sums");
        if (rc) {
            cudaDeviceSynchronize();
            free_train(s);
            return rc;
        }
        s->train_ready = true;
    }
    return PPF_OK;
}

Fields<const float> cur_fields(ppf_ctx *c) {
    return {(const float *)c->fld[c->cur_eta][0], (const float *)c->fld[c->cur_eta][1],
            (const float *)c->fld[c->cur_c][2]};
}

ConvArgs conv_args(ppf_surrogate *s, ppf_ctx *c, int layer, const uint16_t *x, const uint16_t *wimg) {
    ConvArgs a{};
    a.g = s->g;
    a.x = x;
    a.wimg = wimg;
    a.bias = s->params + s->boff[layer];
    a.sg = c->g;
    a.nyc = s->nyc[s->ci[layer] == 32][s->co[layer] == 32];
    a.items = s->g.nz * a.nyc * (s->g.nx / kTileX);
    a.err = c->derr;
    a.limit_ns = c->wait_limit_ns;
    for (int k = 0; k < 3; ++k) {
        a.oscale[k] = (float)s->cfg.out_scale[k];
        a.lw[k] = (float)(s->cfg.loss_weight[k] / (3.0 * (double)c->nz * c->ny * c->nx));
    }
    return a;
}

int run_conv(ppf_surrogate *s, ppf_ctx *c, int ci, int co, int epi, const ConvArgs &a) {
    const int grid = s->conv_grid[ci == 32][co == 32];
    ConvArgs b = a;
    b.inject_stall = s->inject;
    s->inject = 0;
    SCU(launch_conv(ci, co, epi, b, grid, c->stream));
    return PPF_OK;
}

MassPlan *plan_of(ppf_ctx *c) { return reinterpret_cast<MassPlan *>(c->dres + 16); }

// blocks of the kernels that take a warp per row
int row_blocks(const ppf_ctx *c) {
    return (int)std::min<int64_t>(((int64_t)c->ny * c->nz + kNT / 32 - 1) / (kNT / 32), 8LL * c->num_sms);
}

// features of the current state; the mass before the call goes to the plan's target
int features(ppf_surrogate *s, ppf_ctx *c) {
    const int nb = row_blocks(c);
    int rc = ensure_partials(c, nb);
    if (rc) return rc;
    features_kernel<<<nb, kNT, 0, c->stream>>>(c->g, cur_fields(c), s->g, s->feat, (float)s->cfg.c_solid,
                                               (float)s->cfg.c_liquid, (float)s->cfg.in_scale_c, c->partials);
    SCU(cudaGetLastError());
    SCU(launch_final_sum(c->partials, nb, 1, 1, &plan_of(c)->target, c->stream));
    return PPF_OK;
}

// features + hidden layers 0..4 (train: keep pre-activations)
int forward_hidden(ppf_surrogate *s, ppf_ctx *c, bool train) {
    int rc = features(s, c);
    if (rc) return rc;
    for (int l = 0; l < 5; ++l) {
        ConvArgs a = conv_args(s, c, l, l == 0 ? s->feat : s->act[l - 1], s->wf[l]);
        a.out = s->act[l];
        a.zout = train ? s->zp[l] : nullptr;
        if ((rc = run_conv(s, c, s->ci[l], s->co[l], train ? EPI_ACT_TRAIN : EPI_ACT, a))) return rc;
    }
    return PPF_OK;
}

// per-CTA sums of a layer's weight gradients, and of its bias gradients (CO + 1 per CTA)
float *wpart_of(ppf_surrogate *s, int layer) { return s->wpart + s->wgrad_grid * s->woff[layer]; }
float *bpart_of(ppf_surrogate *s, int layer) { return s->bpart + (size_t)layer * 2 * s->num_sms * 33; }

int wgrad(ppf_surrogate *s, ppf_ctx *c, int layer, const uint16_t *x, const uint16_t *dz) {
    WgradArgs w{};
    w.g = s->g;
    w.x = x;
    w.dz = dz;
    w.partials = wpart_of(s, layer);
    w.ntiles = s->g.nz * s->g.ny * (s->g.nx / kTileX);
    w.err = c->derr;
    w.limit_ns = c->wait_limit_ns;
    SCU(launch_wgrad(s->ci[layer], s->co[layer], w, s->wgrad_grid, c->stream));
    return PPF_OK;
}

int reduce_all(ppf_surrogate *s, ppf_ctx *c, const int (&bias_grid)[kLayers]) {
    ReduceJobs q{};
    q.loss = s->dscal;
    int blocks = 0, j = 0;
    auto job = [&](const float *part, float *out, int nb, int stride, int n) {
        q.part[j] = part;
        q.out[j] = out;
        q.nb[j] = nb;
        q.stride[j] = stride;
        q.n[j] = n;
        q.first[j] = blocks;
        blocks += (n + (j == 0 ? 1 : 0) + 31) / 32;
        q.first[++j] = blocks;
    };
    for (int l = kLayers - 1; l >= 0; --l) job(bpart_of(s, l), s->grads + s->boff[l], bias_grid[l], s->co[l] + 1, s->co[l]);
    for (int l = 0; l < kLayers; ++l) {
        const int n = 27 * s->ci[l] * s->co[l];
        job(wpart_of(s, l), s->grads + s->woff[l], s->wgrad_grid, n, n);
    }
    reduce_kernel<<<blocks, kNT, 0, c->stream>>>(q);
    SCU(cudaGetLastError());
    return PPF_OK;
}

// loss and gradients of all parameters for one (input, target) pair
int loss_grad(ppf_surrogate *s, ppf_ctx *in, ppf_ctx *tg) {
    int rc = ensure_ws(s, in, true);
    if (rc) return rc;
    if ((rc = check_ctx(tg))) return rc;
    if (tg->nz != in->nz || tg->ny != in->ny || tg->nx != in->nx)
        return serr(PPF_EINVAL, "input and target shapes differ");
    if (in->bc != PPF_BC_PERIODIC) return serr(PPF_EINVAL, "training runs on periodic domains");
    if (tg->stream != in->stream) SCU(cudaStreamSynchronize(tg->stream));
    if ((rc = forward_hidden(s, in, true))) return rc;
    int bias_grid[kLayers];      // CTAs that sum a layer's bias gradients
    // output layer + loss: dZ5 -> g16
    {
        ConvArgs a = conv_args(s, in, 5, s->act[4], s->wf[5]);
        a.out = s->g16;
        a.partials = bpart_of(s, 5);
        a.s0 = cur_fields(in);
        Fields<const float> t = cur_fields(tg);
        a.s1 = {const_cast<float *>(t.eS), const_cast<float *>(t.eL), const_cast<float *>(t.c)};
        if ((rc = run_conv(s, in, s->ci[5], 16, EPI_LOSS, a))) return rc;
        bias_grid[5] = s->conv_grid[s->ci[5] == 32][0];
    }
    if ((rc = wgrad(s, in, 5, s->act[4], s->g16))) return rc;
    const uint16_t *cur = s->g16;
    for (int l = 5; l >= 1; --l) {
        // dZ_{l-1} = conv^T(dZ_l, W_l) * silu'(z_{l-1}); bias gradient of layer l-1
        uint16_t *out = s->gw[(5 - l) % 2];
        ConvArgs a = conv_args(s, in, l, cur, s->wb[l]);
        a.out = out;
        a.zlow = s->zp[l - 1];
        a.partials = bpart_of(s, l - 1);
        const int ci = s->co[l], co = s->ci[l];
        if ((rc = run_conv(s, in, ci, co, EPI_DGRAD, a))) return rc;
        bias_grid[l - 1] = s->conv_grid[ci == 32][co == 32];
        if ((rc = wgrad(s, in, l - 1, l - 1 == 0 ? s->feat : s->act[l - 2], out))) return rc;
        cur = out;
    }
    return reduce_all(s, in, bias_grid);
}

PackTable pack_table(const ppf_surrogate *s) {
    PackTable t{};
    t.n = s->nparams;
    for (int l = 0; l < kLayers; ++l) {
        t.woff[l] = s->woff[l];
        t.ci[l] = s->ci[l];
        t.co[l] = s->co[l];
        t.wf[l] = s->wf[l];
        t.wb[l] = s->wb[l];
    }
    return t;
}

int param_blocks(const ppf_surrogate *s) { return (int)std::min<int64_t>((s->nparams + kNT - 1) / kNT, 4LL * s->num_sms); }

int pack_all(ppf_surrogate *s, cudaStream_t st) {
    pack_kernel<<<param_blocks(s), kNT, 0, st>>>(pack_table(s), s->params);
    SCU(cudaGetLastError());
    return PPF_OK;
}

// move sum(c) onto the plan's target; `have_sum`: the plan's sum is already
// that of the current state
template <typename N>
int project_n(ppf_ctx *c, bool have_sum) {
    MassPlan *mp = plan_of(c);
    float *cc = (float *)c->fld[c->cur_c][2];
    const int nb = row_blocks(c);
    int rc = ensure_partials(c, nb);
    if (rc) return rc;
    if (!have_sum) {
        mass_kernel<N, false, true><<<nb, kNT, 0, c->stream>>>(c->g, cc, mp, c->partials);
        SCU(cudaGetLastError());
        SCU(launch_final_sum(c->partials, nb, 1, 1, &mp->sum, c->stream));
    }
    mass_kernel<N, true, true><<<nb, kNT, 0, c->stream>>>(c->g, cc, mp, c->partials);
    SCU(cudaGetLastError());
    SCU(launch_final_sum(c->partials, nb, 1, 1, &mp->sum, c->stream));
    mass_kernel<N, true, false><<<nb, kNT, 0, c->stream>>>(c->g, cc, mp, nullptr);
    SCU(cudaGetLastError());
    return PPF_OK;
}

int project(ppf_ctx *c, bool have_sum) {
    const long long n = (long long)c->nz * c->ny * c->nx;
    return n < (1LL << 31) ? project_n<unsigned>(c, have_sum) : project_n<unsigned long long>(c, have_sum);
}

}  // namespace

// ---------------------------------------------------------------- C-ABI --

extern "C" void ppf_surrogate_config_default(ppf_surrogate_config *cfg) {
    if (!cfg) return;
    std::memset(cfg, 0, sizeof *cfg);
    cfg->width = 32;
    cfg->k_steps = 50;
    cfg->c_solid = 0.47603;
    cfg->c_liquid = 0.99903;
    cfg->in_scale_c = 1000.0;
    cfg->out_scale[0] = cfg->out_scale[1] = 1e-2;
    cfg->out_scale[2] = 1e-3;
    cfg->loss_weight[0] = cfg->loss_weight[1] = cfg->loss_weight[2] = 1.0;
}

extern "C" int ppf_surrogate_create(const ppf_surrogate_config *cfg, ppf_surrogate **out) {
    if (!cfg || !out) return serr(PPF_EINVAL, "null argument");
    *out = nullptr;
    if (cfg->width != 16 && cfg->width != 32) return serr(PPF_EINVAL, "width must be 16 or 32");
    if (cfg->k_steps < 1) return serr(PPF_EINVAL, "k_steps must be positive");
    for (int k = 0; k < 3; ++k)
        if (!(cfg->out_scale[k] > 0)) return serr(PPF_EINVAL, "out_scale must be positive");
    ppf_surrogate *s = new ppf_surrogate();
    s->cfg = *cfg;
    s->W = cfg->width;
    if (cudaGetDevice(&s->dev) != cudaSuccess) {
        delete s;
        return serr(PPF_ECUDA, "no CUDA device");
    }
    int optin = 0, major = 0;
    cudaDeviceGetAttribute(&s->num_sms, cudaDevAttrMultiProcessorCount, s->dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->dev);
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, s->dev);
    if (major < 10) {
        delete s;
        return serr(PPF_ECUDA, "the surrogate's kernels need a Blackwell (sm_10x) GPU");
    }
    cudaError_t e = conv_setup(optin);
    if (e != cudaSuccess) {
        delete s;
        return serr(PPF_ECUDA, "convolution set-up failed: %s", cudaGetErrorString(e));
    }
    const int chans[kLayers + 1] = {16, s->W, s->W, s->W, s->W, s->W, 16};
    int64_t off = 0;
    for (int l = 0; l < kLayers; ++l) {
        s->ci[l] = chans[l];
        s->co[l] = chans[l + 1];
        s->woff[l] = off;
        off += 27LL * s->ci[l] * s->co[l];
        s->boff[l] = off;
        off += s->co[l];
    }
    s->nparams = off;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b) s->conv_grid[a][b] = conv_ctas_per_sm(a ? 32 : 16, b ? 32 : 16) * s->num_sms;
    s->wgrad_grid = s->num_sms;
    const size_t pb = (size_t)s->nparams * sizeof(float);
    bool ok = cudaMalloc(&s->params, pb) == cudaSuccess && cudaMalloc(&s->grads, pb) == cudaSuccess &&
              cudaMalloc(&s->mom1, pb) == cudaSuccess && cudaMalloc(&s->mom2, pb) == cudaSuccess &&
              cudaMalloc(&s->bpart, (size_t)kLayers * 2 * s->num_sms * 33 * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&s->mpart, (size_t)2 * s->num_sms * sizeof(double)) == cudaSuccess &&
              cudaMalloc(&s->dscal, 8 * sizeof(double)) == cudaSuccess;
    for (int l = 0; ok && l < kLayers; ++l)
        ok = cudaMalloc(&s->wf[l], 27 * s->ci[l] * s->co[l] * 2) == cudaSuccess &&
             cudaMalloc(&s->wb[l], 27 * s->ci[l] * s->co[l] * 2) == cudaSuccess;
    if (ok)
        ok = cudaMemset(s->params, 0, pb) == cudaSuccess && cudaMemset(s->grads, 0, pb) == cudaSuccess &&
             cudaMemset(s->mom1, 0, pb) == cudaSuccess && cudaMemset(s->mom2, 0, pb) == cudaSuccess &&
             cudaMemset(s->dscal, 0, 8 * sizeof(double)) == cudaSuccess;
    if (ok) ok = pack_all(s, 0) == PPF_OK && cudaDeviceSynchronize() == cudaSuccess;
    if (!ok) {
        ppf_surrogate_destroy(s);
        return serr(PPF_ENOMEM, "surrogate allocation failed");
    }
    *out = s;
    return PPF_OK;
}

extern "C" int ppf_surrogate_destroy(ppf_surrogate *s) {
    if (!s) return PPF_OK;
    cudaDeviceSynchronize();
    free_ws(s);
    for (int l = 0; l < kLayers; ++l) {
        cudaFree(s->wf[l]);
        cudaFree(s->wb[l]);
    }
    cudaFree(s->params);
    cudaFree(s->grads);
    cudaFree(s->mom1);
    cudaFree(s->mom2);
    cudaFree(s->wpart);
    cudaFree(s->bpart);
    cudaFree(s->mpart);
    cudaFree(s->dscal);
    delete s;
    return PPF_OK;
}

extern "C" int64_t ppf_surrogate_num_params(const ppf_surrogate *s) { return s ? s->nparams : -1; }

extern "C" int ppf_surrogate_get_config(const ppf_surrogate *s, ppf_surrogate_config *cfg) {
    if (!s || !cfg) return serr(PPF_EINVAL, "null argument");
    *cfg = s->cfg;
    return PPF_OK;
}

extern "C" int ppf_surrogate_set_params(ppf_surrogate *s, const float *host, int64_t n) {
    if (!s || !host) return serr(PPF_EINVAL, "null argument");
    if (n != s->nparams) return serr(PPF_EINVAL, "expected %lld parameters", (long long)s->nparams);
    SCU(cudaMemcpy(s->params, host, n * sizeof(float), cudaMemcpyHostToDevice));
    SCU(cudaMemset(s->mom1, 0, n * sizeof(float)));
    SCU(cudaMemset(s->mom2, 0, n * sizeof(float)));
    s->adam_t = 0;
    int rc = pack_all(s, 0);
    if (rc) return rc;
    SCU(cudaDeviceSynchronize());
    return PPF_OK;
}

extern "C" int ppf_surrogate_get_params(ppf_surrogate *s, float *host, int64_t n) {
    if (!s || !host) return serr(PPF_EINVAL, "null argument");
    if (n != s->nparams) return serr(PPF_EINVAL, "expected %lld parameters", (long long)s->nparams);
    SCU(cudaDeviceSynchronize());
    SCU(cudaMemcpy(host, s->params, n * sizeof(float), cudaMemcpyDeviceToHost));
    return PPF_OK;
}

extern "C" int ppf_surrogate_loss_grad(ppf_surrogate *s, ppf_ctx *input, ppf_ctx *target, double *loss,
                                       float *grad, int64_t n) {
    if (!s) return serr(PPF_EINVAL, "null surrogate");
    if (grad && n != s->nparams) return serr(PPF_EINVAL, "expected %lld gradient entries", (long long)s->nparams);
    int rc = loss_grad(s, input, target);
    if (rc) return rc;
    double l = 0;
    SCU(cudaMemcpyAsync(&l, s->dscal, sizeof(double), cudaMemcpyDeviceToHost, input->stream));
    if (grad)
        SCU(cudaMemcpyAsync(grad, s->grads, s->nparams * sizeof(float), cudaMemcpyDeviceToHost, input->stream));
    SCU(cudaStreamSynchronize(input->stream));
    if ((rc = check_device_error(input))) return rc;
    if (loss) *loss = l;
    return PPF_OK;
}

extern "C" int ppf_surrogate_train_step(ppf_surrogate *s, ppf_ctx *input, ppf_ctx *target, double lr,
                                        double *loss) {
    if (!s) return serr(PPF_EINVAL, "null surrogate");
    if (!(lr >= 0)) return serr(PPF_EINVAL, "learning rate must be non-negative");
    int rc = loss_grad(s, input, target);
    if (rc) return rc;
    s->adam_t++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)s->adam_t), c2 = 1.f - powf(b2, (float)s->adam_t);
    adam_kernel<<<param_blocks(s), kNT, 0, input->stream>>>(pack_table(s), s->params, s->grads, s->mom1, s->mom2, (float)lr,
                                                            b1, b2, 1e-8f, c1, c2);
    SCU(cudaGetLastError());
    if (loss) {
        SCU(cudaMemcpyAsync(loss, s->dscal, sizeof(double), cudaMemcpyDeviceToHost, input->stream));
        SCU(cudaStreamSynchronize(input->stream));
        return check_device_error(input);
    }
    return PPF_OK;
}

extern "C" int ppf_surrogate_predict(ppf_surrogate *s, ppf_ctx *c, double *out3) {
    if (!s || !out3) return serr(PPF_EINVAL, "null argument");
    int rc = ensure_ws(s, c, false);
    if (rc) return rc;
    const size_t elems = (size_t)c->g.total * 3;
    if (s->scratch_elems != elems) {
        cudaDeviceSynchronize();
        cudaFree(s->scratch);
        cudaFree(s->stage);
        s->scratch = nullptr;
        s->stage = nullptr;
        s->scratch_elems = 0;
        if ((rc = alloc_zero((void **)&s->scratch, 2 * elems * sizeof(float), c->stream))) return rc;
        SCU(cudaMalloc(&s->stage, (size_t)3 * c->nz * c->ny * c->nx * sizeof(double)));
        s->scratch_elems = elems;
    }
    if ((rc = forward_hidden(s, c, false))) return rc;
    const int64_t T = c->g.total;
    float *z0 = s->scratch, *o = s->scratch + elems;
    ConvArgs a = conv_args(s, c, 5, s->act[4], s->wf[5]);
    a.s0 = {z0, z0 + T, z0 + 2 * T};
    a.s1 = {o, o + T, o + 2 * T};
    a.mass_part = s->mpart;
    if ((rc = run_conv(s, c, s->ci[5], 16, EPI_STATE, a))) return rc;
    const size_t cells = (size_t)c->nz * c->ny * c->nx;
    double *const st3[3] = {s->stage, s->stage + cells, s->stage + 2 * cells};
    SCU(launch_unpack<float>(c->g, Fields<const float>{o, o + T, o + 2 * T}, st3, c->stream));
    SCU(cudaMemcpyAsync(out3, s->stage, (size_t)3 * c->nz * c->ny * c->nx * sizeof(double), cudaMemcpyDeviceToHost,
                        c->stream));
    SCU(cudaStreamSynchronize(c->stream));
    return check_device_error(c);
}

extern "C" int ppf_surrogate_advance(ppf_surrogate *s, ppf_ctx *c, int ncalls) {
    if (!s) return serr(PPF_EINVAL, "null surrogate");
    if (ncalls < 0) return serr(PPF_EINVAL, "negative call count");
    int rc = ensure_ws(s, c, false);
    if (rc) return rc;
    for (int k = 0; k < ncalls; ++k) {
        if ((rc = forward_hidden(s, c, false))) return rc;     // features: mass before the call
        const int ie = c->cur_eta, ic = c->cur_c;
        ConvArgs a = conv_args(s, c, 5, s->act[4], s->wf[5]);
        a.s0 = cur_fields(c);
        a.s1 = {(float *)c->fld[1 - ie][0], (float *)c->fld[1 - ie][1], (float *)c->fld[1 - ic][2]};
        a.mass_part = s->mpart;
        if ((rc = run_conv(s, c, s->ci[5], 16, EPI_STATE, a))) return rc;
        SCU(launch_final_sum(s->mpart, s->conv_grid[s->ci[5] == 32][0], 1, 1, &plan_of(c)->sum, c->stream));
        c->cur_eta = 1 - ie;
        c->cur_c = 1 - ic;
        c->steps += s->cfg.k_steps;
        if ((rc = project(c, true))) return rc;
    }
    return PPF_OK;
}

extern "C" int ppf_surrogate_debug_inject(ppf_surrogate *s, int fault) {
    if (!s) return serr(PPF_EINVAL, "null surrogate");
    if (fault != PPF_INJECT_NONE && fault != PPF_INJECT_STALL_WAIT) return serr(PPF_EINVAL, "unknown fault");
    s->inject = fault == PPF_INJECT_STALL_WAIT;
    return PPF_OK;
}

extern "C" int ppf_mass_project(ppf_ctx *c, double target_mass) {
    if (!c) return serr(PPF_EINVAL, "null context");
    if (c->prec != PPF_F32) return serr(PPF_EINVAL, "mass projection applies to FP32 contexts");
    if (!c->uploaded) return serr(PPF_ESTATE, "no state uploaded");
    if (!std::isfinite(target_mass)) return serr(PPF_EINVAL, "target mass must be finite");
    SCU(cudaMemcpyAsync(&plan_of(c)->target, &target_mass, sizeof(double), cudaMemcpyHostToDevice, c->stream));
    int rc = project(c, false);
    if (rc) return rc;
    SCU(cudaStreamSynchronize(c->stream));
    return check_device_error(c);
}

extern "C" int ppf_copy_state(ppf_ctx *dst, ppf_ctx *src) {
    if (!dst || !src) return serr(PPF_EINVAL, "null context");
    if (dst->nz != src->nz || dst->ny != src->ny || dst->nx != src->nx || dst->prec != src->prec ||
        dst->bc != src->bc)
        return serr(PPF_EINVAL, "contexts differ in shape, precision or boundary condition");
    if (!src->uploaded) return serr(PPF_ESTATE, "no state uploaded");
    if (dst == src) return PPF_OK;
    const size_t bytes = (size_t)src->g.total * (src->prec == PPF_F32 ? 4 : 8);
    SCU(cudaStreamSynchronize(src->stream));
    for (int k = 0; k < 3; ++k)
        SCU(cudaMemcpyAsync(dst->fld[0][k], src->fld[k < 2 ? src->cur_eta : src->cur_c][k], bytes,
                            cudaMemcpyDeviceToDevice, dst->stream));
    dst->cur_eta = dst->cur_c = 0;
    dst->uploaded = 1;
    dst->steps = src->steps;
    return recheck_box(dst);   // (the contexts' parameters, and so their boxes, may differ)
}
