// ppf_state.cu -- state movement and reductions around the fused step:
// pack/unpack between the caller's compact [z][y][x] double arrays and the
// padded ghosted device layout (the BC fill of phasefield.c:207-211 is done
// on pack), the observables reduction and the
// deterministic final sum of per-CTA partials.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "ppf_fx.h"
#include "ppf_internal.h"
#include "ppf_pair.h"

namespace ppf {

// Face-ghost targets of an interior index i in [0, n): the ghost that the
// BC fill would copy this cell into (-2 = none).
__device__ __forceinline__ void ghost_targets(int i, int n, int bc, int &g0, int &g1) {
    g0 = -2;
    g1 = -2;
    if (i == 0) g0 = (bc == 0) ? n : -1;          // periodic: ghost n = cell 0; no-flux: ghost -1
    if (i == n - 1) g1 = (bc == 0) ? -1 : n;      // periodic: ghost -1 = cell n-1
}

template <typename T>
__device__ __forceinline__ void store3(const Geom &g, Fields<T> out, int x, int y, int z, T s, T l, T c,
                                       bool c_only) {
    int64_t i = g.at(x, y, z);
    if (!c_only) {
        out.eS[i] = s;
        out.eL[i] = l;
    }
    out.c[i] = c;
}

template <typename T>
__device__ __forceinline__ void store_with_ghosts(const Geom &g, Fields<T> out, int x, int y, int z, T s,
                                                  T l, T c, bool c_only) {
    store3(g, out, x, y, z, s, l, c, c_only);
    int a, b;
    ghost_targets(x, g.nx, g.bc, a, b);
    if (a != -2) store3(g, out, a, y, z, s, l, c, c_only);
    if (b != -2) store3(g, out, b, y, z, s, l, c, c_only);
    ghost_targets(y, g.ny, g.bc, a, b);
    if (a != -2) store3(g, out, x, a, z, s, l, c, c_only);
    if (b != -2) store3(g, out, x, b, z, s, l, c, c_only);
    ghost_targets(z, g.nz, g.bc, a, b);
    if (a != -2) store3(g, out, x, y, a, s, l, c, c_only);
    if (b != -2) store3(g, out, x, y, b, s, l, c, c_only);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide sum of NV doubles per thread; thread 0 writes partials[NV*b+i].
template <int NT, int NV>
__device__ __forceinline__ void block_sum_store(double (&v)[NV], double *partials, int b) {
    __shared__ double red[NT / 32][NV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = warp_sum(v[i]);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) red[w][i] = v[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double s = 0;
            for (int q = 0; q < NT / 32; ++q) s += red[q][i];
            partials[(int64_t)NV * b + i] = s;
        }
    }
}

// ------------------------------------------------------- pack / unpack ----
//
// Bound by HBM: 24 bytes of float64 per cell on the caller's side and 12 or
// 24 in the state.  One warp per x row, so that a row's y, z and ghost rows
// are worked out once and a lane only adds x (no 64-bit divisions per cell).
// The caller's three arrays are read and written in place when they are
// device memory of this device; host arrays pass through the staging array.
// A lane loads four of its accesses before it stores one, by predicate, so that
// rows that end inside them wait for memory as often as whole ones do.
// Whole download, FP32: 256^3 109 us (117 with a loop the compiler unrolled by
// four, whose remainder went one access at a time), 250^3 107 (152), 251^3 106
// (224), 512^3 798 (938); through the staging array with one thread per cell
// 256^3 took 106 us and 126 us of copies.

constexpr int kRowWarps = 8;   // rows per block and pass

__device__ __forceinline__ bool out_of_box(double s, double l, double c, unsigned cmax) {
    return !fx::in_box_eta((unsigned)__double2hiint(s) & 0x7fffffffu, (unsigned)__double2hiint(l) & 0x7fffffffu) ||
           !fx::in_box_c((unsigned)__double2hiint(c), cmax);
}

template <typename T>
__device__ __forceinline__ void pack_rows(const Geom &g, const double *__restrict__ s0, const double *__restrict__ s1,
                                          const double *__restrict__ s2, const Fields<T> &dst, BoxCheck box) {
    bool bad = false;
    const int lane = threadIdx.x & 31;
    const int nrows = g.ny * g.nz;
    for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < nrows; r += gridDim.x * kRowWarps) {
        const int z = r / g.ny, y = r - z * g.ny;
        const int64_t i0 = (int64_t)r * g.nx;
        const bool inner = y > 0 && y < g.ny - 1 && z > 0 && z < g.nz - 1;   // feeds x ghosts only
        const int64_t a0 = g.at(0, y, z);
        for (int x0 = lane; x0 < g.nx; x0 += 128) {
            double v[4][3];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (x0 + 32 * k < g.nx) {
                    const int64_t i = i0 + x0 + 32 * k;
                    v[k][0] = s0[i];
                    v[k][1] = s1[i];
                    v[k][2] = s2[i];
                }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = x0 + 32 * k;
                if (x >= g.nx) continue;
                const T s = (T)v[k][0], l = (T)v[k][1], c = (T)v[k][2];
                if (std::is_same<T, double>::value && box.word)
                    bad = bad || out_of_box(s, l, c, box.cmax);
                if (inner && x > 0 && x < g.nx - 1) {
                    dst.eS[a0 + x] = s;
                    dst.eL[a0 + x] = l;
                    dst.c[a0 + x] = c;
                } else {
                    store_with_ghosts(g, dst, x, y, z, s, l, c, false);
                }
            }
        }
    }
    if (bad) *box.word = 1;
}

// A float as a double.  The conversion instruction runs at the FP64 rate,
// 1/64 of the FP32 rate here, and bounded the FP32 unpack (three per cell);
// for normal numbers and zeros the double's bits are the float's, shifted,
// with the exponent rebased.
__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v), m = b & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u || m == 0u) {
        const unsigned hi = (m >> 3) + (m ? 0x38000000u : 0u);
        return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)(b << 29));
    }
    // denormals, infinities, NaN (volatile: not evaluated ahead of the test)
    double d;
    asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ double widen(double v) { return v; }

template <typename T>
__device__ __forceinline__ void unpack_rows(const Geom &g, const T *__restrict__ eS, const T *__restrict__ eL,
                                            const T *__restrict__ c, double *__restrict__ d0, double *__restrict__ d1,
                                            double *__restrict__ d2) {
    const int lane = threadIdx.x & 31;
    const int nrows = g.ny * g.nz;
    // rows that start on 16 bytes everywhere: two cells per lane and access
    const bool two = (g.nx & 1) == 0 && (((uintptr_t)d0 | (uintptr_t)d1 | (uintptr_t)d2) & 15) == 0;
    for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < nrows; r += gridDim.x * kRowWarps) {
        const int z = r / g.ny, y = r - z * g.ny;
        const int64_t i0 = (int64_t)r * g.nx, a0 = g.at(0, y, z);
        if (two) {
            for (int x0 = 2 * lane; x0 < g.nx; x0 += 256) {
                V2<T> s[4], l[4], q[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 64 * k < g.nx) {
                        const int64_t a = a0 + x0 + 64 * k;
                        s[k] = ld2(eS + a);
                        l[k] = ld2(eL + a);
                        q[k] = ld2(c + a);
                    }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 64 * k < g.nx) {
                        const int64_t i = i0 + x0 + 64 * k;
                        st2(d0 + i, V2<double>(widen(s[k].x()), widen(s[k].y())));
                        st2(d1 + i, V2<double>(widen(l[k].x()), widen(l[k].y())));
                        st2(d2 + i, V2<double>(widen(q[k].x()), widen(q[k].y())));
                    }
            }
        } else {
            for (int x0 = lane; x0 < g.nx; x0 += 128) {
                T s[4], l[4], q[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 32 * k < g.nx) {
                        const int64_t a = a0 + x0 + 32 * k;
                        s[k] = eS[a];
                        l[k] = eL[a];
                        q[k] = c[a];
                    }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 32 * k < g.nx) {
                        const int64_t i = i0 + x0 + 32 * k;
                        d0[i] = widen(s[k]);
                        d1[i] = widen(l[k]);
                        d2[i] = widen(q[k]);
                    }
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(32 * kRowWarps) pack_kernel(Geom g, const double *s0, const double *s1,
                                                              const double *s2, Fields<T> dst, BoxCheck box) {
    pack_rows<T>(g, s0, s1, s2, dst, box);
}

template <typename T>
__global__ void __launch_bounds__(32 * kRowWarps) unpack_kernel(Geom g, Fields<const T> src, double *d0, double *d1,
                                                                double *d2) {
    unpack_rows<T>(g, src.eS, src.eL, src.c, d0, d1, d2);
}

template <typename T>
__global__ void __launch_bounds__(32 * kRowWarps, 3) pack_multi_kernel(const IoDesc *__restrict__ table) {
    const IoDesc &d = table[blockIdx.y];
    const Geom g = d.g;
    const Fields<T> dst = {(T *)d.fld[0][0], (T *)d.fld[0][1], (T *)d.fld[0][2]};
    if (blockIdx.x == 0 && threadIdx.x < 3) d.dres[threadIdx.x] = 0.0;
    const int64_t n = (int64_t)g.nx * g.ny * g.nz;
    pack_rows<T>(g, d.staging, d.staging + n, d.staging + 2 * n, dst, d.box);
}

template <typename T>
__global__ void __launch_bounds__(32 * kRowWarps, 3) unpack_multi_kernel(const IoDesc *__restrict__ table, int buf) {
    const IoDesc &d = table[blockIdx.y];
    const Geom g = d.g;
    const int64_t n = (int64_t)g.nx * g.ny * g.nz;
    unpack_rows<T>(g, (const T *)d.fld[buf][0], (const T *)d.fld[buf][1], (const T *)d.fld[buf][2], d.staging,
                   d.staging + n, d.staging + 2 * n);
}

static int row_grid(int64_t nrows) {
    const int64_t b = (nrows + kRowWarps - 1) / kRowWarps;
    return (int)(b < 152 * 8 ? b : 152 * 8);
}

template <typename T>
cudaError_t launch_pack_multi(const IoDesc *table, int n, int64_t max_rows, cudaStream_t s) {
    pack_multi_kernel<T><<<dim3((unsigned)row_grid(max_rows), (unsigned)n), 32 * kRowWarps, 0, s>>>(table);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_unpack_multi(const IoDesc *table, int n, int64_t max_rows, int buf, cudaStream_t s) {
    unpack_multi_kernel<T><<<dim3((unsigned)row_grid(max_rows), (unsigned)n), 32 * kRowWarps, 0, s>>>(table, buf);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_pack(const Geom &g, const double *const src[3], Fields<T> dst, BoxCheck box, cudaStream_t s) {
    pack_kernel<T><<<row_grid((int64_t)g.ny * g.nz), 32 * kRowWarps, 0, s>>>(g, src[0], src[1], src[2], dst, box);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(32 * kRowWarps) box_check_kernel(Geom g, Fields<const double> f, BoxCheck box) {
    const int lane = threadIdx.x & 31, nrows = g.ny * g.nz;
    bool bad = false;
    for (int r = blockIdx.x * kRowWarps + (threadIdx.x >> 5); r < nrows; r += gridDim.x * kRowWarps) {
        const int z = r / g.ny, y = r - z * g.ny;
        const int64_t a = g.at(0, y, z);
        for (int x = lane; x < g.nx; x += 32) bad = bad || out_of_box(f.eS[a + x], f.eL[a + x], f.c[a + x], box.cmax);
    }
    if (bad) *box.word = 1;
}

cudaError_t launch_box_check(const Geom &g, Fields<const double> f, BoxCheck box, cudaStream_t s) {
    box_check_kernel<<<row_grid((int64_t)g.ny * g.nz), 32 * kRowWarps, 0, s>>>(g, f, box);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_unpack(const Geom &g, Fields<const T> src, double *const dst[3], cudaStream_t s) {
    unpack_kernel<T><<<row_grid((int64_t)g.ny * g.nz), 32 * kRowWarps, 0, s>>>(g, src, dst[0], dst[1], dst[2]);
    return cudaGetLastError();
}

// ----------------------------------------------------------- observables --
// Free energy density (no counterpart in the reference; its variational
// derivative is the bracket of phasefield.c:360-373):
//   m f0(etaS, etaL) + kappa/2 |grad eta|^2 (forward differences) + hS fS + (1-hS) fL.
// By the KKS identity AS (cS-cS0) = AL (cL-cL0) = mu the chemical part is
//   AS AL / (2 (AS + (AL-AS) hS)) w^2 + CL + hS (CS-CL),  w = c - cL0 + (cL0-cS0) hS,
// so that only w^2 is summed per cell and the constants CS, CL (orders of
// magnitude above the rest) enter once per block, through the cell count and
// the sum of hS.
//
// Each thread owns 16 bytes of cells in x and marches up z, so that a
// plane's upper neighbours are the next plane's own cells; an FP32 thread
// evaluates its four cells as two packed pairs.  FP32 state: the solid
// fraction and the energy terms are compensated float sums per thread
// (about 48 bits), the solute mass a float sum in three parts (about 72
// bits: more than an FP64 running sum keeps), FP64 beyond the thread.  FP64
// accumulation per cell is what bounded the FP32 form (one conversion and
// one addition per cell, each 1/64 of the FP32 rate); the FP64 state's form
// in FP64 arithmetic is bound by the FP64 pipe, so it has few operations
// (about 32 per cell; ObsFx below has fewer).  256^3 FP32: 56 us (186 us with
// one cell per thread and FP64 sums of the solute mass); 64^3: 7 us (33 us).

// a / b of a pair, as accurate as a division: the quotient by the hardware's
// reciprocal estimate (about 1 ulp), and its residual times the estimate
__device__ __forceinline__ V2<float> ratio(V2<float> a, V2<float> b) {
    float y0, y1;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(b.x()));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(b.y()));
    const V2<float> y(y0, y1), q = a * y;
    return fma2(fma2(splat(0.f) - b, q, a), y, q);
}
// The FP64 estimate has 20 bits: one third-order Newton step y (1 + e + e^2),
// e = 1 - b y, first.
__device__ __forceinline__ double ratio(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ V2<double> ratio(V2<double> a, V2<double> b) {
    return V2<double>(ratio(a.x(), b.x()), ratio(a.y(), b.y()));
}

// whether a^2 + b^2 and its reciprocal lie inside the normal range, as these
// estimates need them: the larger one in [2^-63, 2^62), [2^-480, 2^480) (NaN and
// infinities are not)
__device__ __forceinline__ bool invertible(float a, float b) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(fabsf(a)), "f"(fabsf(b)));
    return __float_as_uint(m) - 0x20000000u < 0x3e800000u;
}
__device__ __forceinline__ bool invertible(double a, double b) {
    const unsigned m = max((unsigned)__double2hiint(a) & 0x7fffffffu, (unsigned)__double2hiint(b) & 0x7fffffffu);
    return m - 0x21f00000u < 0x3c000000u;
}

// a / b of a pair whose values are alike, for anything
template <typename T>
__device__ __noinline__ T divide1(T a, T b) { return a / b; }
template <typename T>
__device__ __forceinline__ V2<T> divide(V2<T> a, V2<T> b) { return splat(divide1<T>(a.x(), b.x())); }

// finite, and above one half, without FP64 instructions
__device__ __forceinline__ bool finite_(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite_(double v) {
    return ((unsigned)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u;
}
__device__ __forceinline__ bool above_half(float v) { return v > 0.5f; }
__device__ __forceinline__ bool above_half(double v) { return __double_as_longlong(v) > 0x3fe0000000000000ll; }

template <typename T>
struct ObsCoef {
    T cL0, dc0, AS, dA, m, kg, g;
    int eq;                       // AS == AL: w^2 is summed without its denominator
    double hA, CL, dC, vol;       // hA = AS AL / 2 (AS / 2 when eq)
};

template <typename T>
struct ObsAcc {
    Mass<T> mass;
    Sum<T> h, w, f;      // solid fraction, chemical energy, m f0 + gradient energy
    int n = 0, solid = 0, bad = 0;

    // A pair of finite cells (own values and the +x, +y, +z neighbours), of
    // which the first nv count.  DIV: etaS^2 + etaL^2 and AS + (AL - AS) h may be
    // anything; else both are invertible.
    template <bool DIV = false>
    __device__ __forceinline__ void pair(const ObsCoef<T> &k, V2<T> eS, V2<T> eL, V2<T> c, V2<T> sx, V2<T> lx,
                                         V2<T> sy, V2<T> ly, V2<T> sz, V2<T> lz, int nv = 2) {
        const V2<T> S2 = eS * eS, L2 = eL * eL, s2 = fma2(eL, eL, S2);
        const V2<T> hh = DIV ? divide(S2, s2) : ratio(S2, s2);
        const V2<T> ww = fma2(hh, splat(k.dc0), c - splat(k.cL0));
        V2<T> ch = ww * ww;
        if (!k.eq) {
            const V2<T> den = fma2(hh, splat(k.dA), splat(k.AS));
            ch = DIV ? divide(ch, den) : ratio(ch, den);
        }
        // f0 = S2 (S2/4 - 1/2 + gamma L2) + L2 (L2/4 - 1/2) + 1/4
        const V2<T> q = splat(T(0.25)), hf = splat(T(-0.5));
        const V2<T> f0 = fma2(S2, fma2(S2, q, fma2(splat(k.g), L2, hf)), fma2(L2, fma2(L2, q, hf), q));
        V2<T> d = sx - eS;
        V2<T> gr = d * d;
        d = lx - eL;
        gr = fma2(d, d, gr);
        d = sy - eS;
        gr = fma2(d, d, gr);
        d = ly - eL;
        gr = fma2(d, d, gr);
        d = sz - eS;
        gr = fma2(d, d, gr);
        d = lz - eL;
        gr = fma2(d, d, gr);
        auto in = [&](V2<T> v) { return V2<T>(nv > 0 ? v.x() : T(0), nv > 1 ? v.y() : T(0)); };
        mass.add(in(c));
        h.add(in(hh));
        w.add(in(ch));
        // (each on its own: they can differ by orders of magnitude)
        f.add(in(splat(k.m) * f0));
        f.add(in(splat(k.kg) * gr));
    }
};

// Sums of fixed-point numbers: exact (low words and high words apart).
struct FxSum {
    unsigned long long lo = 0;
    long long hi = 0;
    __device__ __forceinline__ void add(fx::i64 v) {
        lo += (unsigned)v;
        hi += v >> 32;
    }
    __device__ __forceinline__ double get(double scale) const {
        return scale * ((double)hi * 4294967296.0 + (double)lo);
    }
};

// Squares of fixed-point numbers below 3.5 2^59, taken to 2^4 units: exact for
// 2^14 of them (128 bits).
struct FxSquares {
    unsigned long long lo = 0, hi = 0;
    __device__ __forceinline__ void add(fx::i64 v) {
        const fx::i64 a = (v + 8) >> 4;
        const unsigned long long p = (unsigned long long)a * (unsigned long long)a;
        lo += p;
        hi += (unsigned long long)__mul64hi(a, a) + (lo < p);
    }
    __device__ __forceinline__ double get(double scale) const {
        return scale * ((double)hi * 18446744073709551616.0 + (double)lo) * scale;
    }
};

// Cells of an FP64 state in fixed-point arithmetic (ppf_fx.h) as far as its
// absolute errors are below those of float64: w and the sum of its squares
// (exact, w to 2^-56), the reciprocal, the well energy, and the solute mass where c
// has no bits below 2^-59.  What float64 holds relative to its own size stays
// float64: smaller values of c, the solid fraction of states that have little
// of it, the gradient's differences and squares.  Fourteen of about 32
// operations a cell are left for the FP64 pipe, which runs beside the integer
// pipes.  256^3: 0.58 ms; 1.24 ms with all of it in FP64, 0.49 with all but the
// gradient in fixed point.
struct ObsFx {
    FxSum f0, c;
    FxSquares w;
    double mass = 0, h = 0, gr = 0;
    __device__ __forceinline__ void cell(const fx::FxCoef &k, int cbias, double eS, double eL, double c, double sx,
                                         double lx, double sy, double ly, double sz, double lz) {
        fx::i64 C, W, R, f;
        fx::observe(k, eS, eL, c, cbias, C, W, R, f);
        // cmax is the high word of 2^(ec + 1)
        if (((unsigned)__double2hiint(c) & 0x7fffffffu) >= k.cmax - (7u << 20)) this->c.add(C);
        else mass += c;
        h = fma(eS * eS, fx::unit60(R), h);
        w.add(W);
        f0.add(f);
        double d = sx - eS;
        gr = fma(d, d, gr);
        d = lx - eL;
        gr = fma(d, d, gr);
        d = sy - eS;
        gr = fma(d, d, gr);
        d = ly - eL;
        gr = fma(d, d, gr);
        d = sz - eS;
        gr = fma(d, d, gr);
        d = lz - eL;
        gr = fma(d, d, gr);
    }
};

// The solute mass of a thread's finite cells in FP64, for FP32 compositions so
// large that their sum in floats is none (FP64 holds any such sum).
template <typename T>
__device__ __noinline__ double column_mass(const Geom &g, const Fields<const T> &f, int64_t j, int nz, int cells) {
    double m = 0;
    for (int z = 0; z < nz; ++z, j += g.PS)
        for (int i = 0; i < cells; ++i)
            if (finite_(f.eS[j + i]) && finite_(f.eL[j + i]) && finite_(f.c[j + i])) m += (double)f.c[j + i];
    return m;
}

// FX: an FP64 state whose parameters fit the fixed-point step; cells outside
// its box take the FP64 path.  MASK: the rows' last groups hold fewer cells than
// the others; a warp with such a group counts its cells by mask, all lanes alike
// (250^3 FP32, whole reduction: 72 us, 115 us with those cells taken one by one;
// 128 x 128 x 135 FP64: 118 and 152 us).  A kernel of its own, since the masks cost
// the others 3 %.
template <typename T, bool FX, bool MASK>
__global__ void __launch_bounds__(256, FX ? 2 : 3) observe_kernel(Geom g, ObsCoef<T> k, Fields<const T> fl, int nq, int zc,
                                                      double *partials, fx::FxCoef kx) {
    constexpr int Q = 16 / (int)sizeof(T), NP = Q / 2;   // cells and pairs per thread
    ObsAcc<T> acc;
    ObsFx ax;
    const int cbias = FX ? fx::c_bias(kx.ec) : 0;
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int y = (int)(t / nq), x0 = (int)(t - (int64_t)y * nq) * Q;
    // (a test at run time also where it always holds: without it the compiler
    // orders the loads so that registers run out, 695 us at 512^3 instead of 520)
    const bool whole = x0 + Q <= g.nx;
    const int cells = MASK && y < g.ny ? min(Q, g.nx - x0) : Q;
    const bool masked = MASK && __any_sync(0xffffffffu, cells < Q);
    if (y < g.ny) {
        const int z0 = blockIdx.y * zc, z1 = min(g.nz, z0 + zc);
        int64_t j = g.at(x0, y, z0);        // rows start on a sector: 16-byte aligned
        T s[Q], l[Q];
        auto load = [](const T *p, T (&v)[Q]) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                const V2<T> w = ld2(p + 2 * i);
                v[2 * i] = w.x();
                v[2 * i + 1] = w.y();
            }
        };
        load(fl.eS + j, s);
        load(fl.eL + j, l);
        for (int z = z0; z < z1; ++z, j += g.PS) {
            T c[Q], sy[Q], ly[Q], sz[Q], lz[Q];
            load(fl.c + j, c);
            load(fl.eS + j + g.P, sy);
            load(fl.eL + j + g.P, ly);
            load(fl.eS + j + g.PS, sz);
            load(fl.eL + j + g.PS, lz);
            // the cell after the last one (a ghost at the domain's end)
            const T sx = whole ? fl.eS[j + Q] : T(0), lx = whole ? fl.eL[j + Q] : T(0);
            bool fine = MASK || whole;
            // (bitwise: a chain of branches made the loop a third slower)
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                if constexpr (FX) fine = fine && (i >= cells || !out_of_box(s[i], l[i], c[i], kx.cmax));
                else fine = fine & ((i >= cells) | (invertible(s[i], l[i]) & finite_(c[i])));
            }
            if (fine) {
                acc.n += cells;
#pragma unroll
                for (int i = 0; i < Q; ++i) acc.solid += i < cells && above_half(s[i]) ? 1 : 0;
                if constexpr (FX) {
#pragma unroll
                    for (int i = 0; i < Q; ++i)
                        if (i < cells)
                            ax.cell(kx, cbias, s[i], l[i], c[i], i == Q - 1 ? sx : s[(i + 1) % Q],
                                    i == Q - 1 ? lx : l[(i + 1) % Q], sy[i], ly[i], sz[i], lz[i]);
                } else {
                    auto pairs = [&](int n) {
#pragma unroll
                        for (int i = 0; i < NP; ++i) {
                            const int a = 2 * i, b = a + 1;
                            const bool e = b == Q - 1;
                            acc.pair(k, V2<T>(s[a], s[b]), V2<T>(l[a], l[b]), V2<T>(c[a], c[b]),
                                     V2<T>(s[b], e ? sx : s[(b + 1) % Q]), V2<T>(l[b], e ? lx : l[(b + 1) % Q]),
                                     V2<T>(sy[a], sy[b]), V2<T>(ly[a], ly[b]), V2<T>(sz[a], sz[b]),
                                     V2<T>(lz[a], lz[b]), n - a);
                        }
                    };
                    if (masked) pairs(cells);
                    else pairs(Q);
                }
            } else {
                // non-finite cells (counted and left out), or cells outside the box or
                // the reciprocal's range: cell by cell, twice the same cell in a pair
                for (int i = 0; i < Q && x0 + i < g.nx; ++i) {
                    const int64_t a = j + i;
                    const T S = fl.eS[a], L = fl.eL[a], C = fl.c[a];
                    if (!finite_(S) || !finite_(L) || !finite_(C)) {
                        ++acc.bad;
                        continue;
                    }
                    ++acc.n;
                    acc.solid += above_half(S) ? 1 : 0;
                    acc.template pair<true>(k, splat(S), splat(L), splat(C), splat(fl.eS[a + 1]), splat(fl.eL[a + 1]),
                             splat(fl.eS[a + g.P]), splat(fl.eL[a + g.P]), splat(fl.eS[a + g.PS]),
                             splat(fl.eL[a + g.PS]), 1);
                }
            }
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                s[i] = sz[i];
                l[i] = lz[i];
            }
        }
    }
    // Four sums over the warp: each exchange halves the sums a lane carries
    // (six FP64 additions a thread instead of twenty; with a few dozen cells a
    // thread the reduction itself would otherwise fill the FP64 pipe), and
    // lanes 0, 8, 16, 24 end with mass, h, w and f.
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[4] = {acc.mass.get(), acc.h.get(), acc.w.get(), acc.f.get()};
    if constexpr (!std::is_same<T, double>::value) {
        if (!finite_(v[0])) {
            const int z0 = blockIdx.y * zc;
            v[0] = column_mass<T>(g, fl, g.at(x0, y, z0), min(g.nz - z0, zc), min(Q, g.nx - x0));
        }
    }
    if constexpr (FX) {
        v[0] += ax.c.get(kx.sc) + ax.mass;
        v[1] += ax.h;
        v[2] += ax.w.get(16.0 * kx.sc);
        v[3] += fma(k.kg, ax.gr, k.m * ax.f0.get(6.9388939039072284e-18));         // 2^-57
    }
    const bool up = lane & 16, up2 = lane & 8;
    double a0 = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
    const double a1 = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
    a0 = (up2 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up2 ? a0 : a1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    __shared__ double red[8][4];
    __shared__ int cnt[8][3];
    if ((lane & 7) == 0) red[warp][lane >> 3] = a0;
    const int n = __reduce_add_sync(0xffffffffu, acc.n), ns = __reduce_add_sync(0xffffffffu, acc.solid),
              nb = __reduce_add_sync(0xffffffffu, acc.bad);
    if (lane == 0) {
        cnt[warp][0] = n;
        cnt[warp][1] = ns;
        cnt[warp][2] = nb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[4] = {0, 0, 0, 0};
        int64_t u[3] = {0, 0, 0};
        for (int q = 0; q < 8; ++q) {
            for (int i = 0; i < 4; ++i) t[i] += red[q][i];
            for (int i = 0; i < 3; ++i) u[i] += cnt[q][i];
        }
        double *o = partials + 5 * ((int64_t)blockIdx.x + (int64_t)gridDim.x * blockIdx.y);
        o[0] = t[0];
        o[1] = t[1];
        o[2] = (double)u[1];
        o[3] = k.vol * (t[3] + k.hA * t[2] + (double)u[0] * k.CL + k.dC * t[1]);
        o[4] = (double)u[2];
    }
}

// Blocks of the observables reduction: 256 groups of 16 bytes of cells, in
// z chunks that give about three blocks per SM, what the registers let
// reside at once (each chunk reads one plane more than it owns).
static void observe_shape(const Geom &g, int group, int num_sms, int *nq, int *bx, int *zc, int *bz) {
    *nq = (g.nx + group - 1) / group;
    *bx = (int)(((int64_t)*nq * g.ny + 255) / 256);
    int chunks = 3 * num_sms / *bx;
    chunks = chunks < 1 ? 1 : chunks > g.nz ? g.nz : chunks;
    *zc = (g.nz + chunks - 1) / chunks;
    *bz = (g.nz + *zc - 1) / *zc;
}

template <typename T>
int observe_blocks(const Geom &g, int num_sms) {
    int nq, bx, zc, bz;
    observe_shape(g, 16 / (int)sizeof(T), num_sms, &nq, &bx, &zc, &bz);
    return bx * bz;
}

template <typename T>
cudaError_t launch_observe(const Geom &g, const CoefD &k, const fx::FxCoef *kx, Fields<const T> f, double *partials,
                           int num_sms, cudaStream_t s) {
    int nq, bx, zc, bz;
    observe_shape(g, 16 / (int)sizeof(T), num_sms, &nq, &bx, &zc, &bz);
    ObsCoef<T> o;
    o.cL0 = (T)k.cL0;
    o.dc0 = (T)(k.cL0 - k.cS0);
    o.AS = (T)k.AS;
    o.dA = (T)k.dA;
    o.m = (T)k.m;
    o.kg = (T)k.kappa_h2_half;
    o.g = (T)k.gamma;
    o.eq = k.AS == k.AL;
    o.hA = 0.5 * k.AS * (o.eq ? 1.0 : k.AL);
    o.CL = k.CL;
    o.dC = k.CS - k.CL;
    o.vol = k.vol;
    const dim3 grid((unsigned)bx, (unsigned)bz);
    const bool ragged = g.nx % (16 / (int)sizeof(T)) != 0;
    if constexpr (std::is_same<T, double>::value) {
        if (kx) {
            if (ragged) observe_kernel<T, true, true><<<grid, 256, 0, s>>>(g, o, f, nq, zc, partials, *kx);
            else observe_kernel<T, true, false><<<grid, 256, 0, s>>>(g, o, f, nq, zc, partials, *kx);
            return cudaGetLastError();
        }
    }
    if (ragged) observe_kernel<T, false, true><<<grid, 256, 0, s>>>(g, o, f, nq, zc, partials, fx::FxCoef());
    else observe_kernel<T, false, false><<<grid, 256, 0, s>>>(g, o, f, nq, zc, partials, fx::FxCoef());
    return cudaGetLastError();
}

// one block per value: four independent chains of loads per thread, then a
// fixed tree (the order depends only on the number of partial sums)
__global__ void __launch_bounds__(256) final_sum_kernel(const double *__restrict__ partials, int nblocks, int stride,
                                                        double *out) {
    const double *p = partials + blockIdx.x;
    double a[4] = {0, 0, 0, 0};
    int b = threadIdx.x;
    for (; b + 768 < nblocks; b += 1024)
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] += p[(int64_t)stride * (b + 256 * q)];
    for (; b < nblocks; b += 256) a[0] += p[(int64_t)stride * b];
    double s[1] = {(a[0] + a[1]) + (a[2] + a[3])};
    block_sum_store<256, 1>(s, out, blockIdx.x);
}

cudaError_t launch_final_sum(const double *partials, int nblocks, int stride, int nvals, double *out,
                             cudaStream_t s) {
    final_sum_kernel<<<nvals, 256, 0, s>>>(partials, nblocks, stride, out);
    return cudaGetLastError();
}

// explicit instantiations
template cudaError_t launch_pack<float>(const Geom &, const double *const[3], Fields<float>, BoxCheck, cudaStream_t);
template cudaError_t launch_pack<double>(const Geom &, const double *const[3], Fields<double>, BoxCheck, cudaStream_t);
template cudaError_t launch_unpack<float>(const Geom &, Fields<const float>, double *const[3], cudaStream_t);
template cudaError_t launch_unpack<double>(const Geom &, Fields<const double>, double *const[3], cudaStream_t);
template cudaError_t launch_pack_multi<float>(const IoDesc *, int, int64_t, cudaStream_t);
template cudaError_t launch_pack_multi<double>(const IoDesc *, int, int64_t, cudaStream_t);
template cudaError_t launch_unpack_multi<float>(const IoDesc *, int, int64_t, int, cudaStream_t);
template cudaError_t launch_unpack_multi<double>(const IoDesc *, int, int64_t, int, cudaStream_t);
template cudaError_t launch_observe<float>(const Geom &, const CoefD &, const fx::FxCoef *, Fields<const float>, double *, int,
                                           cudaStream_t);
template cudaError_t launch_observe<double>(const Geom &, const CoefD &, const fx::FxCoef *, Fields<const double>, double *, int,
                                            cudaStream_t);

template int observe_blocks<float>(const Geom &, int);
template int observe_blocks<double>(const Geom &, int);

}  // namespace ppf
