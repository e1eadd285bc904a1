// ppf_particles.cu -- particle analysis of a state on the GPU: connected
// components of the solid (etaS > threshold, 6-connected, wrapping across
// periodic faces), their volumes, equivalent-sphere radii, the mean radius
// R-bar, and the solid/liquid interface area.  The reference does this
// analysis outside the program (README.md:26: MATLAB post-processing); here
// it runs on the device state between steps.
//
// The cells are first reduced to one bit each (the only pass over the field:
// 2 MB of words at 256^3, which stay in the L2); everything else works on
// runs, the stretches of solid cells inside a 32-cell word of an x row.  A
// run is named by its first cell and has a label and a volume there.
// Labelling is a lock-free union-find over the runs: a run starts as its own
// root; runs that touch (in the next word, row or plane: one union per
// stretch of common bits) have their roots joined by hooking the larger
// root onto the smaller with a compare-and-swap.  Parent labels therefore
// strictly decrease along every path, so each find terminates; retry loops
// are additionally capped and report PPF_ETIMEOUT if the cap is ever
// reached.  The interface area is a population count of differing bits.
//
// What bounds it is the latency of the label chains in the L2.  Labels per
// cell, with 64-bit divisions for every cell's place, took 0.80 ms at 256^3
// (merge 443 us, volumes 232 us); see launch_particles for the run form.
#include <cuda_runtime.h>

#include <cstdint>

#include "ppf_internal.h"
#include "ppf_particles.h"

namespace ppf {

namespace {

constexpr int kNT = 256;
constexpr int kMaxRetry = 1 << 20;

// Label reads and the halving writes bypass L1 (other SMs change labels
// through L2 while the merge runs).
__device__ __forceinline__ int find_root(int *lab, int i) {
    // path halving: each visited cell points two levels up (still an ancestor)
    for (int it = 0; it < kMaxRetry; ++it) {
        const int p = __ldcg(lab + i);
        if (p == i) return i;
        const int gp = __ldcg(lab + p);
        if (gp != p) __stcg(lab + i, gp);
        i = gp;
    }
    return -1;
}

__device__ __forceinline__ bool unite(int *lab, int a, int b) {
    for (int it = 0; it < kMaxRetry; ++it) {
        a = find_root(lab, a);
        b = find_root(lab, b);
        if (a < 0 || b < 0) return false;
        if (a == b) return true;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(lab + a, a, b);   // hook root a under b < a
        if (old == a) return true;
        a = old;                                     // a was hooked meanwhile: retry from there
    }
    return false;
}

// The words of a grid: nw per x row, rows in [z][y] order.
struct Words {
    int nx, ny, nz, nw, bc;
    int64_t count;   // nw ny nz
};

// One warp per x row: the row's words, and label and volume of every run.
template <typename T>
__global__ void __launch_bounds__(kNT) find_runs(Geom g, Words q, const T *__restrict__ eS, T thr,
                                                 unsigned *__restrict__ bits, int *__restrict__ lab,
                                                 int *__restrict__ vol) {
    const int lane = threadIdx.x & 31;
    const int nrows = q.ny * q.nz;
    for (int r = blockIdx.x * (kNT / 32) + (threadIdx.x >> 5); r < nrows; r += gridDim.x * (kNT / 32)) {
        const int z = r / q.ny, y = r - z * q.ny;
        const T *row = eS + g.at(0, y, z);
        for (int w0 = 0; w0 < q.nw; w0 += 8) {
            bool s[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int x = 32 * (w0 + k) + lane;
                s[k] = x < q.nx && row[x] > thr;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const unsigned m = __ballot_sync(0xffffffffu, s[k]);
                if (w0 + k < q.nw && lane == k) bits[(int64_t)r * q.nw + w0 + k] = m;
                if (s[k] && !((m << 1 >> lane) & 1u)) {      // the cell before is not solid, or in another word
                    const int i = r * q.nx + 32 * (w0 + k) + lane;
                    lab[i] = i;
                    vol[i] = 0;
                }
            }
        }
    }
}

// first bit of the run of `m` that holds bit p
__device__ __forceinline__ int run_start(unsigned m, int p) {
    const unsigned below = ~m & ((1u << p) - 1u);
    return below ? 32 - __clz(below) : 0;
}

__device__ __forceinline__ bool unite_common(int *lab, unsigned a, int ia, unsigned b, int ib) {
    bool ok = true;
    const unsigned m = a & b;
    for (unsigned s = m & ~(m << 1); s; s &= s - 1) {
        const int p = __ffs((int)s) - 1;
        ok = unite(lab, ia + run_start(a, p), ib + run_start(b, p)) && ok;
    }
    return ok;
}

// One thread per word: joins its runs with the touching runs of the next
// word, row and plane (wrapping for periodic boundaries); counts the
// solid/liquid faces to them (interface area).
__global__ void __launch_bounds__(kNT) merge_runs(Words q, const unsigned *__restrict__ bits, int *lab,
                                                  double *__restrict__ partials, int *__restrict__ err) {
    int64_t faces = 0;
    bool ok = true;
    for (int64_t i = blockIdx.x * (int64_t)kNT + threadIdx.x; i < q.count; i += (int64_t)gridDim.x * kNT) {
        const int r = (int)(i / q.nw), w = (int)(i - (int64_t)r * q.nw);
        const int z = r / q.ny, y = r - z * q.ny;
        const int n = min(32, q.nx - 32 * w);                // cells of the word
        const unsigned all = n == 32 ? 0xffffffffu : (1u << n) - 1u;
        const unsigned a = bits[i];
        const int cell = r * q.nx + 32 * w;                  // the word's first cell
        const bool last = w == q.nw - 1;
        // the next cell in x: inside the word, then the next word's (or the row's) first
        unsigned in = a ^ (a >> 1);
        in &= all >> 1;
        faces += __popc(in);
        if (!last || q.bc == 0) {
            const unsigned b = last ? bits[i - w] : bits[i + 1];
            const bool sa = (a >> (n - 1)) & 1u, sb = b & 1u;
            faces += sa != sb;
            if (sa && sb) ok = unite(lab, cell + run_start(a, n - 1), last ? r * q.nx : cell + 32) && ok;
        }
        if (y + 1 < q.ny || q.bc == 0) {
            const int r2 = y + 1 < q.ny ? r + 1 : r - y;
            const unsigned b = bits[(int64_t)r2 * q.nw + w];
            faces += __popc(a ^ b);
            ok = unite_common(lab, a, cell, b, r2 * q.nx + 32 * w) && ok;
        }
        if (z + 1 < q.nz || q.bc == 0) {
            const int r2 = z + 1 < q.nz ? r + q.ny : y;
            const unsigned b = bits[(int64_t)r2 * q.nw + w];
            faces += __popc(a ^ b);
            ok = unite_common(lab, a, cell, b, r2 * q.nx + 32 * w) && ok;
        }
    }
    if (!ok) atomicOr(err, 2);
    // block sum of the face count
    __shared__ int64_t red[kNT / 32];
    for (int o = 16; o > 0; o >>= 1) faces += __shfl_xor_sync(0xffffffffu, faces, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = faces;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int k = 0; k < kNT / 32; ++k) s += red[k];
        partials[blockIdx.x] = (double)s;
    }
}

// One thread per word: every run's cells are added to its root's volume (the
// lanes of a warp that hold the same root add once).
__global__ void __launch_bounds__(kNT) count_volumes(Words q, const unsigned *__restrict__ bits, int *lab,
                                                     int *__restrict__ vol, int *__restrict__ err) {
    const int64_t step = (int64_t)gridDim.x * kNT;
    for (int64_t i0 = blockIdx.x * (int64_t)kNT; i0 < q.count; i0 += step) {
        const int64_t i = i0 + threadIdx.x;
        unsigned m = 0;
        int cell = 0;
        if (i < q.count) {
            m = bits[i];
            const int r = (int)(i / q.nw), w = (int)(i - (int64_t)r * q.nw);
            cell = r * q.nx + 32 * w;
        }
        while (__any_sync(0xffffffffu, m != 0)) {
            int root = -1, len = 0;
            if (m) {
                const int p = __ffs((int)m) - 1;
                const unsigned up = ~(m >> p);               // the run's first zero
                len = up ? __ffs((int)up) - 1 : 32;          // (bits shifted in at the top are zero: never past the word)
                m = p + len >= 32 ? 0u : m >> (p + len) << (p + len);
                root = find_root(lab, cell + p);
                if (root < 0) atomicOr(err, 2);
                else if (root != cell + p) lab[cell + p] = root;
            }
            const unsigned peers = __match_any_sync(0xffffffffu, root);
            const int sum = __reduce_add_sync(peers, len);
            if (root >= 0 && (threadIdx.x & 31) == __ffs((int)peers) - 1) atomicAdd(vol + root, sum);
        }
    }
}

// per root: count, sum of equivalent radii, sum of volumes, largest volume;
// optionally the list of volumes
__global__ void __launch_bounds__(kNT) root_stats(Words q, const unsigned *__restrict__ bits, const int *__restrict__ lab,
                                                  const int *__restrict__ vol, double dx3,
                                                  double *__restrict__ partials, int64_t *__restrict__ list,
                                                  int64_t cap, unsigned long long *__restrict__ nlist) {
    double cnt = 0, rsum = 0, vsum = 0, vmax = 0;
    const double k = 3.0 / (4.0 * 3.14159265358979323846);
    for (int64_t i = blockIdx.x * (int64_t)kNT + threadIdx.x; i < q.count; i += (int64_t)gridDim.x * kNT) {
        const unsigned m = bits[i];
        const int r = (int)(i / q.nw), w = (int)(i - (int64_t)r * q.nw);
        for (unsigned s = m & ~(m << 1); s; s &= s - 1) {
            const int c = r * q.nx + 32 * w + __ffs((int)s) - 1;
            if (lab[c] != c) continue;
            const double v = (double)vol[c];
            cnt += 1.0;
            rsum += cbrt(k * v * dx3);
            vsum += v;
            vmax = v > vmax ? v : vmax;
            if (list) {
                const unsigned long long slot = atomicAdd(nlist, 1ull);
                if ((int64_t)slot < cap) list[slot] = (int64_t)vol[c];
            }
        }
    }
    __shared__ double red[kNT / 32][4];
    double v4[4] = {cnt, rsum, vsum, vmax};
    for (int q = 0; q < 4; ++q) {
        double a = v4[q];
        for (int o = 16; o > 0; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = q == 3 ? (b > a ? b : a) : a + b;
        }
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s[4] = {0, 0, 0, 0};
        for (int w = 0; w < kNT / 32; ++w) {
            s[0] += red[w][0];
            s[1] += red[w][1];
            s[2] += red[w][2];
            s[3] = red[w][3] > s[3] ? red[w][3] : s[3];
        }
        for (int q = 0; q < 4; ++q) partials[(int64_t)blockIdx.x * 4 + q] = s[q];
    }
}

// one block per value of count, rsum, vsum, vmax, faces
__global__ void __launch_bounds__(kNT) finish_stats(const double *__restrict__ faces, const double *__restrict__ rs,
                                                    int nb, double *__restrict__ out) {
    __shared__ double red[kNT];
    const int q = blockIdx.x;
    double a = 0.0;
    for (int b = threadIdx.x; b < nb; b += kNT) {
        const double v = q < 4 ? rs[(int64_t)b * 4 + q] : faces[b];
        a = q == 3 ? (v > a ? v : a) : a + v;
    }
    red[threadIdx.x] = a;
    __syncthreads();
    for (int h = kNT / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) {
            const double o = red[threadIdx.x + h];
            red[threadIdx.x] = q == 3 ? (o > red[threadIdx.x] ? o : red[threadIdx.x]) : red[threadIdx.x] + o;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[q] = red[0];
}

}  // namespace

int64_t particle_words(const Geom &g) { return (int64_t)((g.nx + 31) / 32) * g.ny * g.nz; }

template <typename T>
cudaError_t launch_particles(const Geom &g, const T *etaS, double threshold, int *lab, int *vol, unsigned *bits,
                             double *partials, int nblocks, double dx, double *out, int64_t *list, int64_t cap,
                             unsigned long long *nlist, int *err, cudaStream_t s) {
    const Words q = {g.nx, g.ny, g.nz, (g.nx + 31) / 32, g.bc, particle_words(g)};
    const T thr = (T)threshold;
    find_runs<T><<<nblocks, kNT, 0, s>>>(g, q, etaS, thr, bits, lab, vol);
    merge_runs<<<nblocks, kNT, 0, s>>>(q, bits, lab, partials, err);
    count_volumes<<<nblocks, kNT, 0, s>>>(q, bits, lab, vol, err);
    if (list) cudaMemsetAsync(nlist, 0, sizeof(unsigned long long), s);
    root_stats<<<nblocks, kNT, 0, s>>>(q, bits, lab, vol, dx * dx * dx, partials + nblocks, list, cap, nlist);
    finish_stats<<<5, kNT, 0, s>>>(partials, partials + nblocks, nblocks, out);
    return cudaGetLastError();
}

template cudaError_t launch_particles<float>(const Geom &, const float *, double, int *, int *, unsigned *, double *, int, double,
                                             double *, int64_t *, int64_t, unsigned long long *, int *, cudaStream_t);
template cudaError_t launch_particles<double>(const Geom &, const double *, double, int *, int *, unsigned *, double *, int,
                                              double, double *, int64_t *, int64_t, unsigned long long *, int *,
                                              cudaStream_t);

}  // namespace ppf
