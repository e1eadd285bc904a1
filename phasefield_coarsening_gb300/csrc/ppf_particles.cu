// ppf_particles.cu -- particle analysis of a state on the GPU: connected
// components of the solid (etaS > threshold, 6-connected, wrapping across
// periodic faces), their volumes, equivalent-sphere radii, the mean radius
// R-bar, and the solid/liquid interface area.  The reference does this
// analysis outside the program (README.md:26: MATLAB post-processing); here
// it runs on the device state between steps.
//
// The cells are first reduced to one bit each (the only pass over the field);
// everything else works on runs, the stretches of solid cells inside a
// 32-cell word of an x row.  A run is a node of a lock-free union-find: it
// starts as its own root; runs that touch (in the next word, row or plane:
// one union per stretch of common bits) have their roots joined by hooking the
// larger root onto the smaller with a compare-and-swap.  Parent labels
// therefore strictly decrease along every path, so each find terminates;
// retry loops are additionally capped and report PPF_ETIMEOUT if the cap is
// ever reached.  The interface area is a population count of differing bits.
//
// What bounds a union-find is the latency of its label chains.  A block labels
// a brick of 512 words in shared memory, counts its components' cells there
// and hands out one node per component (and the labels of the runs on its
// faces); only the unions across bricks, about a tenth of all, go through the
// L2, and the passes over volumes and roots see the bricks' components (about
// three per particle) instead of every run.  With all unions and every run's
// count in global memory the analysis took 0.21 ms of kernels at 256^3 and
// 1.00 ms at 512^3 (merge 121 and 491 us, volumes and roots 50 and 240); now
// 0.08 and 0.36.  The volumes are sorted here too: 57,000 of them are in order
// and on the host after 0.09 ms (the host's sort alone took 0.5).
#include <cuda_runtime.h>

#include <cstdint>

#include "ppf_internal.h"
#include "ppf_particles.h"

namespace ppf {

namespace {

constexpr int kNT = 256;
constexpr int kMaxRetry = 1 << 20;

// Labels in global memory: reads and the halving writes bypass L1 (other SMs
// change labels through L2 while unions run).
struct GlobalLabels {
    int *lab;
    __device__ __forceinline__ int get(int i) const { return __ldcg(lab + i); }
    __device__ __forceinline__ void set(int i, int v) const { __stcg(lab + i, v); }
    __device__ __forceinline__ int cas(int i, int v) const { return atomicCAS(lab + i, i, v); }
};

// Labels of a brick in shared memory.
struct BrickLabels {
    int *lab;
    __device__ __forceinline__ int get(int i) const { return *(volatile int *)(lab + i); }
    __device__ __forceinline__ void set(int i, int v) const { *(volatile int *)(lab + i) = v; }
    __device__ __forceinline__ int cas(int i, int v) const { return atomicCAS(lab + i, i, v); }
};

template <typename L>
__device__ __forceinline__ int find_root(L lab, int i) {
    // path halving: each visited node points two levels up (still an ancestor)
    for (int it = 0; it < kMaxRetry; ++it) {
        const int p = lab.get(i);
        if (p == i) return i;
        const int gp = lab.get(p);
        if (gp != p) lab.set(i, gp);
        i = gp;
    }
    return -1;
}

// the root without halving, for labels that nobody changes any more
__device__ __forceinline__ int climb(BrickLabels lab, int i) {
    for (int it = 0; it < kMaxRetry; ++it) {
        const int p = lab.get(i);
        if (p == i) return i;
        i = p;
    }
    return -1;
}

// Climbs from both nodes at once (two loads in flight), halving both paths.
template <typename L>
__device__ __forceinline__ bool unite(L lab, int a, int b) {
    for (int it = 0; it < kMaxRetry; ++it) {
        const int pa = lab.get(a), pb = lab.get(b);
        if (pa == pb) return true;
        if (pa == a && pb == b) {
            const int hi = max(a, b), lo = min(a, b);
            const int old = lab.cas(hi, lo);         // hook the larger root under the smaller
            if (old == hi) return true;
            a = old;                                 // it was hooked meanwhile: retry from there
            b = lo;
        } else {
            const int ga = lab.get(pa), gb = lab.get(pb);
            if (ga != pa) lab.set(a, ga);
            if (gb != pb) lab.set(b, gb);
            a = ga;
            b = gb;
        }
    }
    return false;
}

// The words of a grid (nw per x row, rows in [z][y] order), its nodes (the
// k-th run of word w of row r is node r npr + 16 w + k) and its bricks of 2^lbw
// words, kBrickY rows and 2^lbz planes.
constexpr int kBrickNT = 512, kBrickY = 16;
struct Words {
    int nx, ny, nz, nw, bc, npr, lbw, lbz, nbx, nby, nbz;
};

__device__ __forceinline__ int run_count(unsigned m) { return __popc(m & ~(m << 1)); }
// which run of `m` holds bit p
__device__ __forceinline__ int run_of(unsigned m, int p) { return __popc(m & ~(m << 1) & ((2u << p) - 1u)) - 1; }
// takes the first run off `m` and returns its length (bits shifted in at the
// top are zero: never past the word)
__device__ __forceinline__ int take_run(unsigned &m) {
    const int p = __ffs((int)m) - 1;
    const unsigned up = ~(m >> p);
    const int len = up ? __ffs((int)up) - 1 : 32;
    m = p + len >= 32 ? 0u : m >> (p + len) << (p + len);
    return len;
}

// joins the runs of word a (node ia + k step) with those of b that touch them
template <typename L>
__device__ __forceinline__ bool unite_common(L lab, unsigned a, int ia, unsigned b, int ib, int step) {
    bool ok = true;
    const unsigned m = a & b;
    for (unsigned s = m & ~(m << 1); s; s &= s - 1) {
        const int p = __ffs((int)s) - 1;
        ok = unite(lab, ia + run_of(a, p) * step, ib + run_of(b, p) * step) && ok;
    }
    return ok;
}

// the block's sum of face counts
__device__ __forceinline__ void put_faces(int64_t faces, double *out) {
    __shared__ int64_t red[32];
    for (int o = 16; o > 0; o >>= 1) faces += __shfl_xor_sync(0xffffffffu, faces, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = faces;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t s = 0;
        for (int k = 0; k < (int)blockDim.x / 32; ++k) s += red[k];
        *out = (double)s;
    }
}

// which of the n cells (four at most) at p are solid
__device__ __forceinline__ unsigned four_bits(const float *p, float thr, int n) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    const unsigned m = (v.x > thr) | (v.y > thr) << 1 | (v.z > thr) << 2 | (v.w > thr) << 3;
    return n < 4 ? m & ((1u << n) - 1u) : m;
}
__device__ __forceinline__ unsigned four_bits(const double *p, double thr, int n) {
    const double2 v = reinterpret_cast<const double2 *>(p)[0], w = reinterpret_cast<const double2 *>(p)[1];
    const unsigned m = (v.x > thr) | (v.y > thr) << 1 | (w.x > thr) << 2 | (w.y > thr) << 3;
    return n < 4 ? m & ((1u << n) - 1u) : m;
}

struct BrickSmem {
    int lab[16 * kBrickNT];        // run k of word t: k kBrickNT + t (lanes in different banks)
    int vol[16 * kBrickNT];
    unsigned bits[kBrickNT];
    int added, base;
};

// One block per brick, a thread per word: the field's bits, the brick's
// components, their volumes and the faces inside the brick.  Writes every
// word's bits, label, volume and list entry of every component's root, and the
// labels of the runs on the brick's faces.
template <typename T>
__global__ void __launch_bounds__(kBrickNT, 3) label_bricks(Geom g, Words q, const T *__restrict__ eS, T thr,
                                                            unsigned *__restrict__ bits, int *__restrict__ lab,
                                                            int *__restrict__ vol, int *__restrict__ list,
                                                            int *__restrict__ nlist, double *__restrict__ partials,
                                                            int *__restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BrickSmem &sm = *reinterpret_cast<BrickSmem *>(smem_raw);
    const BrickLabels L{sm.lab};
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int bw = 1 << q.lbw, bz = 1 << q.lbz;
    const int nbricks = q.nbx * q.nby * q.nbz;
    int64_t faces = 0;
    bool ok = true;
    for (int br = blockIdx.x; br < nbricks; br += gridDim.x) {
        const int jx = br % q.nbx, rest = br / q.nbx, jy = rest % q.nby, jz = rest / q.nby;
        const int w0 = jx << q.lbw, y0 = jy * kBrickY, z0 = jz << q.lbz;
        auto word_of = [&](int i, int &w, int &y, int &z) {
            w = w0 + (i & (bw - 1));
            y = y0 + ((i >> q.lbw) & (kBrickY - 1));
            z = z0 + (i >> q.lbw) / kBrickY;
            return w < q.nw && y < q.ny && z < q.nz;
        };
        // a warp reads the 32 words of its threads, four at a time: eight lanes
        // a word, four cells a lane (rows start on 32 bytes and are padded to
        // whole 32 bytes behind the last halo cell)
        unsigned part[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            int w, y, z;
            const bool in = word_of(32 * warp + 4 * k + (lane >> 3), w, y, z);
            const int x = 32 * w + 4 * (lane & 7);
            part[k] = 0;
            if (in && x < q.nx) part[k] = four_bits(eS + g.at(x, y, z), thr, q.nx - x) << (4 * (lane & 7));
        }
        unsigned a = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            unsigned m = part[k];
            m |= __shfl_xor_sync(0xffffffffu, m, 1);
            m |= __shfl_xor_sync(0xffffffffu, m, 2);
            m |= __shfl_xor_sync(0xffffffffu, m, 4);
            m = __shfl_sync(0xffffffffu, m, 8 * (lane & 3));
            if (lane >> 2 == k) a = m;
        }
        int w, y, z;
        const bool in = word_of(t, w, y, z);
        const int lx = w - w0, ly = y - y0, lz = z - z0;
        const int row = z * q.ny + y;
        if (in) bits[(int64_t)row * q.nw + w] = a;
        sm.bits[t] = a;
        const int nruns = run_count(a);
        unsigned m = a;
        for (int k = 0; k < nruns; ++k) {
            sm.lab[k * kBrickNT + t] = k * kBrickNT + t;
            sm.vol[k * kBrickNT + t] = take_run(m);
        }
        if (t == 0) sm.added = 0;
        __syncthreads();

        if (in) {
            const int n = min(32, q.nx - 32 * w);            // cells of the word
            const unsigned all = n == 32 ? 0xffffffffu : (1u << n) - 1u;
            faces += __popc((a ^ (a >> 1)) & (all >> 1));
            if (lx + 1 < bw && w + 1 < q.nw) {
                const unsigned b = sm.bits[t + 1];
                const bool sa = a >> 31, sb = b & 1u;
                faces += sa != sb;
                if (sa && sb) ok = unite(L, (nruns - 1) * kBrickNT + t, t + 1) && ok;
            }
            if (ly + 1 < kBrickY && y + 1 < q.ny) {
                const unsigned b = sm.bits[t + bw];
                faces += __popc(a ^ b);
                ok = unite_common(L, a, t, b, t + bw, kBrickNT) && ok;
            }
            if (lz + 1 < bz && z + 1 < q.nz) {
                const unsigned b = sm.bits[t + bw * kBrickY];
                faces += __popc(a ^ b);
                ok = unite_common(L, a, t, b, t + bw * kBrickY, kBrickNT) && ok;
            }
        }
        __syncthreads();

        // labels become roots; cells are added to the root's volume
        int own = 0;
        for (int k = 0; k < nruns; ++k) {
            const int i = k * kBrickNT + t, r = find_root(L, i);
            if (r < 0) ok = false;
            if (r == i) ++own;
            else if (r >= 0) {
                L.set(i, r);
                atomicAdd(&sm.vol[r], sm.vol[i]);            // (no one adds to vol[i]: i is no root)
            }
        }
        // places for the roots in the list
        int before = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        int wbase = 0;
        if (lane == 31 && before) wbase = atomicAdd(&sm.added, before);
        wbase = __shfl_sync(0xffffffffu, wbase, 31);
        __syncthreads();
        if (t == 0) sm.base = sm.added ? atomicAdd(nlist, sm.added) : 0;
        __syncthreads();
        int at = sm.base + wbase + before - own;
        const bool face = lx == 0 || lx == bw - 1 || w == q.nw - 1 || ly == 0 || ly == kBrickY - 1 || y == q.ny - 1 ||
                          lz == 0 || lz == bz - 1 || z == q.nz - 1;
        for (int k = 0; k < nruns; ++k) {
            // (the label may be short of the root again: another thread's halving,
            // begun before the root was set, can have put an ancestor there)
            const int i = k * kBrickNT + t, r = climb(L, i), node = row * q.npr + 16 * w + k;
            if (r == i) {
                lab[node] = node;
                vol[node] = sm.vol[i];
                list[at++] = node;
            } else if (face && r >= 0) {
                int rw, ry, rz;
                word_of(r & (kBrickNT - 1), rw, ry, rz);
                lab[node] = (rz * q.ny + ry) * q.npr + 16 * rw + r / kBrickNT;
            }
        }
        __syncthreads();                                     // the next brick reuses the arrays
    }
    if (!ok) atomicOr(err, 2);
    put_faces(faces, partials + blockIdx.x);
}

// The unions and faces across bricks (wrapping for periodic boundaries), a
// thread per word on a brick's upper x, y or z side.
__global__ void __launch_bounds__(kNT) merge_bricks(Words q, const unsigned *__restrict__ bits, int *lab,
                                                    double *__restrict__ partials, int *__restrict__ err) {
    const GlobalLabels L{lab};
    const int64_t first = blockIdx.x * (int64_t)kNT + threadIdx.x, step = (int64_t)gridDim.x * kNT;
    int64_t faces = 0;
    bool ok = true;
    auto across = [&](int r, int r2, int w) {
        const unsigned a = bits[(int64_t)r * q.nw + w], b = bits[(int64_t)r2 * q.nw + w];
        faces += __popc(a ^ b);
        ok = unite_common(L, a, r * q.npr + 16 * w, b, r2 * q.npr + 16 * w, 1) && ok;
    };
    const int64_t cx = (int64_t)q.ny * q.nz * q.nbx, cy = (int64_t)q.nw * q.nz * q.nby, cz = (int64_t)q.nw * q.ny * q.nbz;
    for (int64_t j = first; j < cx + cy + cz; j += step) {
        int64_t i = j;
        if (i >= cx) {
            i -= cx;
            const int w = (int)((i < cy ? i : i - cy) % q.nw), rest = (int)((i < cy ? i : i - cy) / q.nw);
            if (i < cy) {
                const int jy = rest % q.nby, z = rest / q.nby, y = min((jy + 1) * kBrickY, q.ny) - 1;
                if (y + 1 < q.ny || q.bc == 0) across(z * q.ny + y, z * q.ny + (y + 1 < q.ny ? y + 1 : 0), w);
            } else {
                const int y = rest % q.ny, jz = rest / q.ny, z = min((jz + 1) << q.lbz, q.nz) - 1;
                if (z + 1 < q.nz || q.bc == 0) across(z * q.ny + y, (z + 1 < q.nz ? z + 1 : 0) * q.ny + y, w);
            }
            continue;
        }
        const int r = (int)(i / q.nbx), w = min((((int)(i - (int64_t)r * q.nbx) + 1) << q.lbw), q.nw) - 1;
        const bool last = w == q.nw - 1;
        if (last && q.bc != 0) continue;
        const int n = min(32, q.nx - 32 * w), w2 = last ? 0 : w + 1;
        const unsigned a = bits[(int64_t)r * q.nw + w], b = bits[(int64_t)r * q.nw + w2];
        const bool sa = (a >> (n - 1)) & 1u, sb = b & 1u;
        faces += sa != sb;
        if (sa && sb) ok = unite(L, r * q.npr + 16 * w + run_count(a) - 1, r * q.npr + 16 * w2) && ok;
    }
    if (!ok) atomicOr(err, 2);
    put_faces(faces, partials + blockIdx.x);
}

// Every brick component's volume is added to its root's (the lanes of a warp
// that hold the same root add once).
__global__ void __launch_bounds__(kNT) add_volumes(const int *__restrict__ list, const int *__restrict__ nlist, int *lab,
                                                   int *vol, int *__restrict__ err) {
    const GlobalLabels L{lab};
    const int n = *nlist, step = gridDim.x * kNT;
    for (int i0 = blockIdx.x * kNT; i0 < n; i0 += step) {
        const int i = i0 + (int)threadIdx.x;
        int root = -1, v = 0;
        if (i < n) {
            const int node = list[i];
            root = find_root(L, node);
            if (root < 0) atomicOr(err, 2);
            if (root == node) root = -1;                     // its volume is already there
            else v = vol[node];
        }
        const unsigned peers = __match_any_sync(0xffffffffu, root);
        const int sum = __reduce_add_sync(peers, v);
        if (root >= 0 && (threadIdx.x & 31) == __ffs((int)peers) - 1) atomicAdd(vol + root, sum);
        if (n - i0 <= step) break;                           // (i0 + step could pass 2^31)
    }
}

// Radii are summed exactly, in units of 2^-53 cells (any two words of a sum apart,
// the low one's carries left in it): the list is in no order, and a rounded
// sum's last bits would depend on it.
struct RadiusSum {
    unsigned long long lo = 0, hi = 0;
    __device__ __forceinline__ void add(double r) {               // 0.6 <= r < 801: volumes below 2^31
        const unsigned long long v = (unsigned long long)__double2ll_rn(r * 9007199254740992.0);
        lo += (unsigned)v;
        hi += v >> 32;
    }
    __device__ __forceinline__ void add(const RadiusSum &o) {
        lo += o.lo;
        hi += o.hi;
    }
    __device__ __forceinline__ void add_lane(int d) {             // that of the lane at distance d (xor)
        lo += __shfl_xor_sync(0xffffffffu, lo, d);
        hi += __shfl_xor_sync(0xffffffffu, hi, d);
    }
    __device__ __forceinline__ double get() const {
        return ((double)(hi + (lo >> 32)) * 4294967296.0 + (double)(unsigned)lo) * 1.1102230246251565e-16;
    }
};

// per root: count, sum of equivalent radii, sum of volumes, largest volume;
// optionally the volumes themselves, in no order.  partials: count, volumes,
// largest volume, then the radius sum's two words.
__global__ void __launch_bounds__(kNT) root_stats(const int *__restrict__ list, const int *__restrict__ nlist,
                                                  const int *__restrict__ lab, const int *__restrict__ vol,
                                                  double *__restrict__ partials, int *__restrict__ volumes, int64_t cap,
                                                  int *__restrict__ nvolumes) {
    double cnt = 0, vsum = 0, vmax = 0;
    RadiusSum rsum;
    const double k = 3.0 / (4.0 * 3.14159265358979323846);
    const int n = *nlist, step = gridDim.x * kNT, lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * kNT; i0 < n; i0 += step) {
        const int i = i0 + (int)threadIdx.x;
        const int c = i < n ? list[i] : -1;
        const bool root = c >= 0 && lab[c] == c;
        const int iv = root ? vol[c] : 0;
        if (root) {
            const double v = (double)iv;
            cnt += 1.0;
            rsum.add(cbrt(k * v));
            vsum += v;
            vmax = v > vmax ? v : vmax;
        }
        if (volumes) {
            const unsigned roots = __ballot_sync(0xffffffffu, root);
            int at = 0;
            if (lane == 0 && roots) at = atomicAdd(nvolumes, __popc(roots));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(roots & ((1u << lane) - 1u));
            if (root && at < cap) volumes[at] = iv;
        }
        if (n - i0 <= step) break;
    }
    __shared__ double red[kNT / 32][3];
    __shared__ unsigned long long rred[kNT / 32][2];
    double v3[3] = {cnt, vsum, vmax};
    for (int q = 0; q < 3; ++q) {
        double a = v3[q];
        for (int o = 16; o > 0; o >>= 1) {
            const double b = __shfl_xor_sync(0xffffffffu, a, o);
            a = q == 2 ? (b > a ? b : a) : a + b;
        }
        if (lane == 0) red[threadIdx.x >> 5][q] = a;
    }
    for (int o = 16; o > 0; o >>= 1) rsum.add_lane(o);
    if (lane == 0) {
        rred[threadIdx.x >> 5][0] = rsum.lo;
        rred[threadIdx.x >> 5][1] = rsum.hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s[3] = {0, 0, 0};
        unsigned long long u[2] = {0, 0};
        for (int w = 0; w < kNT / 32; ++w) {
            s[0] += red[w][0];
            s[1] += red[w][1];
            s[2] = red[w][2] > s[2] ? red[w][2] : s[2];
            u[0] += rred[w][0];
            u[1] += rred[w][1];
        }
        double *p = partials + (int64_t)blockIdx.x * 5;
        for (int q = 0; q < 3; ++q) p[q] = s[q];
        for (int q = 0; q < 2; ++q) p[3 + q] = __longlong_as_double((long long)u[q]);
    }
}

// ---- sorting the volumes: a radix sort from the low digits up, stable, a
// segment of the keys per warp.  hist[digit][warp] is counted, summed up
// exclusively in that order, and tells each warp where its keys go.

constexpr int kSortBits = 9, kSortWarps = 512;

__global__ void __launch_bounds__(kNT) sort_count(const int *__restrict__ keys, int64_t n, int64_t seg, int nwarps,
                                                  int shift, int bins, int *__restrict__ hist) {
    __shared__ int cnt[kNT / 32][1 << kSortBits];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, w = blockIdx.x * (kNT / 32) + wl;
    for (int b = lane; b < bins; b += 32) cnt[wl][b] = 0;
    __syncwarp();
    if (w >= nwarps) return;
    const int64_t end = min(n, (w + 1) * seg);
    for (int64_t i = w * seg + lane; i < end; i += 32) atomicAdd(&cnt[wl][(keys[i] >> shift) & (bins - 1)], 1);
    __syncwarp();
    for (int b = lane; b < bins; b += 32) hist[b * nwarps + w] = cnt[wl][b];
}

__global__ void __launch_bounds__(1024) sort_scan(int *hist, int n) {
    __shared__ int sums[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int carry = 0;
    for (int i0 = 0; i0 < n; i0 += 4096) {
        int v[4], s = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + 4 * t + k;
            v[k] = i < n ? hist[i] : 0;
            s += v[k];
        }
        int up = s;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, up, o);
            if (lane >= o) up += u;
        }
        if (lane == 31) sums[warp] = up;
        __syncthreads();
        int below = 0, total = 0;
        for (int k = 0; k < 32; ++k) {
            if (k < warp) below += sums[k];
            total += sums[k];
        }
        int at = carry + below + up - s;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + 4 * t + k;
            if (i < n) hist[i] = at;
            at += v[k];
        }
        carry += total;
        __syncthreads();
    }
}

template <typename O>
__global__ void __launch_bounds__(kNT) sort_scatter(const int *__restrict__ keys, int64_t n, int64_t seg, int nwarps,
                                                    int shift, int bins, const int *__restrict__ hist,
                                                    O *__restrict__ out) {
    __shared__ int next[kNT / 32][1 << kSortBits];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, w = blockIdx.x * (kNT / 32) + wl;
    if (w >= nwarps) return;
    for (int b = lane; b < bins; b += 32) next[wl][b] = hist[b * nwarps + w];
    __syncwarp();
    const int64_t end = min(n, (w + 1) * seg);
    for (int64_t i0 = w * seg; i0 < end; i0 += 32) {
        const int64_t i = i0 + lane;
        const int key = i < end ? keys[i] : 0;
        const int d = i < end ? (key >> shift) & (bins - 1) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        const int at = d >= 0 ? next[wl][d] + rank : 0;
        __syncwarp();
        if (d >= 0 && rank == 0) next[wl][d] += __popc(peers);
        __syncwarp();
        if (d >= 0) out[at] = key;
    }
}

// Up to kSmallSort keys in one block and launch, in shared memory, five bits a
// pass: 17 us for 3900 keys of 18 bits, 25 in six launches of the kernels above.
constexpr int kSmallSort = 8192;

struct SmallSort {
    int buf[2][kSmallSort];
    int cnt[32 * 32];              // digit, warp
    int sums[32];
};

__global__ void __launch_bounds__(1024) sort_small(const int *__restrict__ keys, int n, int bits,
                                                   int64_t *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSort &sm = *reinterpret_cast<SmallSort *>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int seg = ((n + 31) / 32 + 31) / 32 * 32, begin = warp * seg, end = min(n, begin + seg);
    for (int i = t; i < n; i += 1024) sm.buf[0][i] = keys[i];
    int src = 0;
    for (int shift = 0; shift < bits; shift += 5, src ^= 1) {
        sm.cnt[t] = 0;
        __syncthreads();
        for (int i = begin + lane; i < end; i += 32) atomicAdd(&sm.cnt[((sm.buf[src][i] >> shift) & 31) * 32 + warp], 1);
        __syncthreads();
        const int own = sm.cnt[t];
        int up = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, up, o);
            if (lane >= o) up += u;
        }
        if (lane == 31) sm.sums[warp] = up;
        __syncthreads();
        const int below = __reduce_add_sync(0xffffffffu, lane < warp ? sm.sums[lane] : 0);
        sm.cnt[t] = below + up - own;
        __syncthreads();
        for (int i0 = begin; i0 < end; i0 += 32) {
            const int i = i0 + lane;
            const int key = i < end ? sm.buf[src][i] : 0;
            const int d = i < end ? (key >> shift) & 31 : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, d);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            const int at = d >= 0 ? sm.cnt[d * 32 + warp] + rank : 0;
            __syncwarp();
            if (d >= 0 && rank == 0) sm.cnt[d * 32 + warp] += __popc(peers);
            __syncwarp();
            if (d >= 0) sm.buf[src ^ 1][at] = key;
        }
        __syncthreads();
    }
    for (int i = t; i < n; i += 1024) out[i] = sm.buf[src][i];
}

// one block per value of count, rsum, vsum, vmax, faces
__global__ void __launch_bounds__(kNT) finish_stats(const double *__restrict__ faces, int nf,
                                                    const double *__restrict__ rs, int nb, double *__restrict__ out) {
    __shared__ double red[kNT];
    const int q = blockIdx.x;
    if (q == 1) {
        __shared__ RadiusSum rred[kNT];
        RadiusSum s;
        for (int b = threadIdx.x; b < nb; b += kNT) {
            s.lo += (unsigned long long)__double_as_longlong(rs[(int64_t)b * 5 + 3]);
            s.hi += (unsigned long long)__double_as_longlong(rs[(int64_t)b * 5 + 4]);
        }
        rred[threadIdx.x] = s;
        __syncthreads();
        for (int h = kNT / 2; h > 0; h >>= 1) {
            if ((int)threadIdx.x < h) rred[threadIdx.x].add(rred[threadIdx.x + h]);
            __syncthreads();
        }
        if (threadIdx.x == 0) out[q] = rred[0].get();
        return;
    }
    double a = 0.0;
    for (int b = threadIdx.x; b < (q < 4 ? nb : nf); b += kNT) {
        const double v = q < 4 ? rs[(int64_t)b * 5 + (q == 0 ? 0 : q - 1)] : faces[b];
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

static Words words_of(const Geom &g) {
    Words q;
    q.nx = g.nx;
    q.ny = g.ny;
    q.nz = g.nz;
    q.bc = g.bc;
    q.nw = (g.nx + 31) / 32;
    q.npr = 16 * (q.nw - 1) + (g.nx - 32 * (q.nw - 1) + 1) / 2;
    q.lbw = q.nw >= 3 ? 2 : q.nw - 1;
    q.lbz = 5 - q.lbw;
    q.nbx = (q.nw + (1 << q.lbw) - 1) >> q.lbw;
    q.nby = (g.ny + kBrickY - 1) / kBrickY;
    q.nbz = (g.nz + (1 << q.lbz) - 1) >> q.lbz;
    return q;
}
static_assert((4 * kBrickY) << 3 == kBrickNT, "a thread per word of a brick");

ParticleScratch particle_scratch(const Geom &g, int *mem) {
    const Words q = words_of(g);
    const int64_t rows = (int64_t)g.ny * g.nz, nodes = rows * q.npr, words = rows * q.nw;
    ParticleScratch p;
    p.nodes = nodes;
    p.lab = mem;
    p.vol = mem + nodes;
    p.list = mem + 2 * nodes;
    p.bits = (unsigned *)(mem + 3 * nodes);
    p.hist = mem + 3 * nodes + words;
    p.counts = p.hist + (kSortWarps << kSortBits);
    p.ints = 3 * nodes + words + (kSortWarps << kSortBits) + 2;
    return p;
}

template <typename T>
cudaError_t launch_particles(const Geom &g, const T *etaS, double threshold, const ParticleScratch &p, double *partials,
                             int nblocks, int num_sms, double *out, int *volumes, int64_t cap, int *err,
                             cudaStream_t s) {
    const Words q = words_of(g);
    cudaError_t e =
        cudaFuncSetAttribute(label_bricks<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BrickSmem));
    if (e == cudaSuccess) e = cudaMemsetAsync(p.counts, 0, 2 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    // (FP64 sums over every block: no more blocks than SMs)
    const int nb4 = nblocks < num_sms ? nblocks : num_sms;
    const int64_t bricks = (int64_t)q.nbx * q.nby * q.nbz;
    const int nb1 = (int)(bricks < 3 * num_sms ? bricks : 3 * num_sms);
    double *const stats = partials + nb1 + nblocks;
    label_bricks<T><<<nb1, kBrickNT, sizeof(BrickSmem), s>>>(g, q, etaS, (T)threshold, p.bits, p.lab, p.vol, p.list,
                                                              p.counts, partials, err);
    merge_bricks<<<nblocks, kNT, 0, s>>>(q, p.bits, p.lab, partials + nb1, err);
    add_volumes<<<nblocks, kNT, 0, s>>>(p.list, p.counts, p.lab, p.vol, err);
    root_stats<<<nb4, kNT, 0, s>>>(p.list, p.counts, p.lab, p.vol, stats, volumes, cap, p.counts + 1);
    finish_stats<<<5, kNT, 0, s>>>(partials, nb1 + nblocks, stats, nb4, out);
    return cudaGetLastError();
}

cudaError_t launch_sort_volumes(int *keys, int *spare, int64_t n, int64_t largest, const ParticleScratch &p,
                                int64_t **sorted, cudaStream_t s) {
    int bits = 1;
    while (bits < 31 && (largest >> bits)) ++bits;
    const int passes = (bits + kSortBits - 1) / kSortBits, d = (bits + passes - 1) / passes;
    const int nwarps = (int)(n < 256 ? 1 : n / 256 < kSortWarps ? n / 256 : kSortWarps);
    const int64_t seg = ((n + nwarps - 1) / nwarps + 31) / 32 * 32;
    const int blocks = (nwarps + kNT / 32 - 1) / (kNT / 32);
    *sorted = reinterpret_cast<int64_t *>(p.lab);            // labels and volumes are done with: 2 nodes >= 2 n ints
    if (n <= kSmallSort) {
        const cudaError_t e =
            cudaFuncSetAttribute(sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSort));
        if (e != cudaSuccess) return e;
        sort_small<<<1, 1024, sizeof(SmallSort), s>>>(keys, (int)n, bits, *sorted);
        return cudaGetLastError();
    }
    for (int k = 0; k < passes; ++k) {
        sort_count<<<blocks, kNT, 0, s>>>(keys, n, seg, nwarps, k * d, 1 << d, p.hist);
        sort_scan<<<1, 1024, 0, s>>>(p.hist, nwarps << d);
        if (k + 1 < passes)
            sort_scatter<int><<<blocks, kNT, 0, s>>>(keys, n, seg, nwarps, k * d, 1 << d, p.hist, spare);
        else
            sort_scatter<int64_t><<<blocks, kNT, 0, s>>>(keys, n, seg, nwarps, k * d, 1 << d, p.hist, *sorted);
        int *const t = keys;
        keys = spare;
        spare = t;
    }
    return cudaGetLastError();
}

template cudaError_t launch_particles<float>(const Geom &, const float *, double, const ParticleScratch &, double *, int,
                                             int, double *, int *, int64_t, int *, cudaStream_t);
template cudaError_t launch_particles<double>(const Geom &, const double *, double, const ParticleScratch &, double *,
                                              int, int, double *, int *, int64_t, int *, cudaStream_t);

}  // namespace ppf
