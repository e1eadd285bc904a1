// ppf_step_fx.cu -- the float64 step (phasefield.c:301-476) in 64-bit
// fixed-point arithmetic (ppf_fx.h), for states and parameters that fit.
//
// What bounded the float64 step was the FP64 pipe: about 75 operations per
// cell-step at 2 lanes per clock and SM, 2.2 ms at 256^3 against 0.12 ms for
// its memory traffic.  Here a cell has twelve: nine for the increment of its
// smaller phase field, which keeps float64's relative precision however small
// the value is (ppf_fx.h), one conversion of the larger one, two for c.
// 0.61 ms at 256^3, 18 us at 64^3 (56 us).  What bounds it are dependency waits
// at sixteen warps an SM: the FP64 pipe is busy 53 % of the time, 54 % of the
// issue slots are taken (780 instructions a cell), the ALU 46 %.  With both
// fields' increments in fixed point (six operations, small values lost) it took
// 0.64 ms, with both in float64 0.90; two additions in place of each conversion
// instruction, 0.78 against 0.70; rates in the halo planes too, 20.6 us at 64^3.
//
// The data flow is that of ppf_step_tma.cuh: work items (z chunk, 32 x 16
// tile) marched up z, etaS/etaL/c boxes streamed by TMA, pass A once per
// loaded cell into a three-plane shared ring that now holds four integers
// per cell (etaS, etaL, w, M'), pass B + C one plane behind.  Three stages of
// raw planes (one in flight) leave room for the wider ring with two CTAs per
// SM; the arithmetic per plane is long against a load.  Faces are oriented
// from low to high, so that both cells of a face use the same number.
#include "ppf_step_tma.cuh"

#include "ppf_step_fx.h"

namespace ppf {

using fx::FxCoef;
using fx::i64;

namespace {

using G = TmaGeo<double, 0>;
constexpr int kStages = 3;
// Two cells per thread interleave two chains of arithmetic; one cell and twice
// the warps needs more than its 64 registers, and an unrolled plane loop more
// than 128 (0.78 and 0.76 ms at 256^3 where this form took 0.67).
constexpr int kCells = 2;                      // cells per thread, stacked in y
constexpr int kThreads = G::TX * G::TY / kCells;

struct alignas(128) FxSmem {
    double raw[kStages][3][G::BOX_PAD];   // etaS, etaL, c boxes per stage
    i64 nb[3][4][G::BOX];                 // etaS, etaL, w, M' of three consecutive planes
    unsigned long long bar[kStages];
};
constexpr size_t kSmemBytes = sizeof(FxSmem) + 128;

// What a launch needs beyond the tables.
struct FxArgs {
    Geom g;
    Coef<double> k;
    FxCoef kx;
    Fields<const double> in;
    Fields<double> out;
    Tiles tiles;
    ZSplit zs;
    double *partials;
    int *err;
    unsigned long long limit_ns;
    const DomainDesc *table;
    int ndom, nitems, parity, set, second, inject_stall;
    int *sched, *box;
};

template <bool MULTI>
__device__ __forceinline__ Item fx_item(const FxArgs &a, int item) {
    if (a.set == SET_WHOLE) return item_at<MULTI, SET_WHOLE>(item, a.tiles, a.zs, a.g.nz, a.table, a.ndom);
    if (a.set == SET_EDGE) return item_at<MULTI, SET_EDGE>(item, a.tiles, a.zs, a.g.nz, a.table, a.ndom);
    return item_at<MULTI, SET_ALL>(item, a.tiles, a.zs, a.g.nz, a.table, a.ndom);
}

// mu and M' of a cell in float64, as the general kernel computes them
__device__ __forceinline__ void mu_m(const Coef<double> &k, double eS, double eL, double c, double &mu, double &M,
                                     double &rs) {
    const double S2 = __dmul_rn(eS, eS), s2 = fma(eL, eL, S2);
    rs = __drcp_rn(s2);
    const double h = __dmul_rn(S2, rs);
    mu = __dmul_rn(k.A, fma(h, k.dc0, c - k.cL0));
    M = fma(h, k.Mt1, k.Mt0);
}

// One item of a step whose input has left the box, in float64 with the
// general kernel's operations in its order: mu and M' once per cell, in the
// ring of three shared planes (`mm`, next slot `mb`), everything else straight
// from global memory.  A domain that leaves the box stays on this path until
// its next upload, so it has to keep the general kernel's rate; FP64 operations
// bound both: 2.66 ms at 256^3, 0.28 ms at 96 x 128 x 128 (general 2.22 and 0.24;
// cell by cell, with mu and M' of all seven cells, 4.37 and 0.44).
template <bool C_ONLY>
__device__ __noinline__ void slow_item(const Coef<double> &k, const Geom &g, const Fields<const double> &in,
                                       const Fields<double> &out, const Item &it, double (*mm)[2][G::BOX], int &mb,
                                       double *inc) {
    constexpr int TX = G::TX, TY = G::TY, XH = G::XH, BX = G::BX;
    const int tid = threadIdx.x, tx = tid & 31, ty0 = (tid >> 5) * kCells;
    const int x = it.bx * TX + tx, y = it.by * TY + ty0, ob = (ty0 + 1) * BX + tx + XH;
    // this thread's ring cell, tile coordinates (the last threads: the rows -1
    // and TY, then the columns -1 and TX)
    const int rt = tid - (kThreads - G::RING);
    const int rx = rt < 2 * TX ? rt % TX : rt < 2 * TX + TY ? -1 : TX;
    const int ry = rt < TX ? -1 : rt < 2 * TX ? TY : (rt - 2 * TX) % TY;
    const bool ring = rt >= 0 && it.bx * TX + rx <= g.nx && it.by * TY + ry <= g.ny;
    double mu[kCells], M[kCells], rs[kCells], mq[kCells], Mq[kCells], rq[kCells], mz[kCells], Mz[kCells];
#pragma unroll
    for (int j = 0; j < kCells; ++j) mu[j] = M[j] = rs[j] = mq[j] = Mq[j] = rq[j] = mz[j] = Mz[j] = 0;
    int prev = mb;
    for (int pz = it.z0 - 1; pz <= it.z1; ++pz) {
#pragma unroll
        for (int j = 0; j < kCells; ++j)
            if (x <= g.nx && y + j <= g.ny) {      // (with the ghosts that cells of this tile see)
                const int64_t i = g.at(x, y + j, pz);
                mu_m(k, in.eS[i], in.eL[i], in.c[i], mu[j], M[j], rs[j]);
                mm[mb][0][ob + j * BX] = mu[j];
                mm[mb][1][ob + j * BX] = M[j];
            }
        if (ring) {
            const int64_t i = g.at(it.bx * TX + rx, it.by * TY + ry, pz);
            const int o = (ry + 1) * BX + rx + XH;
            double r;
            mu_m(k, in.eS[i], in.eL[i], in.c[i], mm[mb][0][o], mm[mb][1][o], r);
        }
        __syncthreads();
        const int q = pz - 1;
#pragma unroll
        for (int j = 0; j < kCells; ++j) {
            if (q < it.z0 || x >= g.nx || y + j >= g.ny) continue;
            const int64_t i = g.at(x, y + j, q);
            const int o = ob + j * BX;
            const double *pm = mm[prev][0], *pM = mm[prev][1];
            double fl = __dmul_rn(M[j] + Mq[j], mu[j] - mq[j]);
            fl = fma(Mz[j] + Mq[j], mz[j] - mq[j], fl);
            fl = fma(pM[o + BX] + Mq[j], pm[o + BX] - mq[j], fl);
            fl = fma(pM[o - BX] + Mq[j], pm[o - BX] - mq[j], fl);
            fl = fma(pM[o + 1] + Mq[j], pm[o + 1] - mq[j], fl);
            fl = fma(pM[o - 1] + Mq[j], pm[o - 1] - mq[j], fl);
            const double eS = in.eS[i], eL = in.eL[i], cn = __dadd_rn(in.c[i], fl);
            double Sn = eS, Ln = eL;
            inc[0] += fl * fl;
            if (!C_ONLY) {
                // z+, z-, then y+, y-, x+, x-, each added in turn
                auto six = [&](const double *f) {
                    double s = __dadd_rn(f[i + g.PS], f[i - g.PS]);
                    s = __dadd_rn(s, f[i + g.P]);
                    s = __dadd_rn(s, f[i - g.P]);
                    s = __dadd_rn(s, f[i + 1]);
                    return __dadd_rn(s, f[i - 1]);
                };
                const double D = fma(mq[j], -k.q1, k.dC);
                const double dmu = __dmul_rn(__dmul_rn(__dmul_rn(k.dm2, __dmul_rn(eS, eL)), __dmul_rn(rq[j], rq[j])), D);
                const double S2 = __dmul_rn(eS, eS), L2 = __dmul_rn(eL, eL);
                const double lapS = fma(-6.0, eS, six(in.eS)), lapL = fma(-6.0, eL, six(in.eL));
                const double dS = fma(__dmul_rn(k.mt, eS), fma(k.tg, L2, __dadd_rn(S2, -1.0)),
                                      fma(-k.kt, lapS, __dmul_rn(eL, dmu)));
                const double dL = fma(__dmul_rn(k.mt, eL), fma(k.tg, S2, __dadd_rn(L2, -1.0)),
                                      fma(-k.kt, lapL, __dadd_rn(0.0, -__dmul_rn(eS, dmu))));
                Sn = __dadd_rn(eS, dS);
                Ln = __dadd_rn(eL, dL);
                inc[1] += dS * dS;
                inc[2] += dL * dL;
            }
            auto put = [&](int64_t a) { put_ghost<double, C_ONLY>(out, a, Sn, Ln, cn); };
            put(i);
            const bool per = g.bc == 0;
            if (x == 0) put(per ? i + g.nx : i - 1);
            if (x == g.nx - 1) put(per ? i - g.nx : i + 1);
            if (y + j == 0) put(per ? i + g.ny * g.P : i - g.P);
            if (y + j == g.ny - 1) put(per ? i - g.ny * g.P : i + g.P);
            if (q == 0) put(per ? i + g.nz * g.PS : i - g.PS);
            if (q == g.nz - 1) put(per ? i - g.nz * g.PS : i + g.PS);
        }
#pragma unroll
        for (int j = 0; j < kCells; ++j) {
            mz[j] = mq[j];
            Mz[j] = Mq[j];
            mq[j] = mu[j];
            Mq[j] = M[j];
            rq[j] = rs[j];
        }
        prev = mb;
        mb = mb + 1 == 3 ? 0 : mb + 1;
    }
}

// which of a cell's fields is the smaller one: 0 etaS, 1 etaL
__device__ __forceinline__ int smaller(double eS, double eL) {
    return ((unsigned)__double2hiint(eL) & 0x7fffffffu) < ((unsigned)__double2hiint(eS) & 0x7fffffffu) ? 1 : 0;
}

// sum of three doubles over the CTA, in a fixed order, to partials[3 item ..]
__device__ __forceinline__ void put_sums(const double (&acc)[3], double *partials, int item) {
    __shared__ double ired[kThreads / 32][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double v = acc[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) ired[warp][i] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int i = 0; i < 3; ++i) {
            double s = 0;
            for (int w = 0; w < kThreads / 32; ++w) s += ired[w][i];
            partials[(int64_t)item * 3 + i] = s;
        }
}

// FULL: every tile of the launch lies inside its domain.  STATS: the increments'
// sums of squares go to a.partials, the larger field's increments computed once
// more for them with a precision of their own (a kernel of its own: their code
// costs the others 4 % in registers; 256^3 0.61 and 0.89 ms, 0.70 with the
// increments that are added).
template <bool C_ONLY, bool FULL, bool MULTI, bool STATS>
__global__ void __launch_bounds__(kThreads, 2)
    step_fx_kernel(const __grid_constant__ CUtensorMap mapS, const __grid_constant__ CUtensorMap mapL,
                   const __grid_constant__ CUtensorMap mapC, const __grid_constant__ FxArgs a) {
    constexpr int TX = G::TX, TY = G::TY, XH = G::XH, BX = G::BX, BY = G::BY, NT = kThreads, S = kStages;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    const uint32_t pad = (128u - (smem_u32(smem_dyn) & 127u)) & 127u;
    FxSmem &sm = *reinterpret_cast<FxSmem *>(smem_dyn + pad);
    const FxCoef &kx = a.kx;

    // programmatic dependent launch: as in step_tma_kernel
    if (!a.second) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane, ty0 = warp * kCells;
    const int ob = (ty0 + 1) * BX + tx + XH;          // own first cell in a box
    const int nitems = a.nitems;
    __shared__ int s_next[2];

    // domains whose input has left the box
    auto left_box = [&](int dom) -> bool {
        const int *b = MULTI ? a.table[dom].box : a.box;
        return *reinterpret_cast<const volatile int *>(b + a.parity) != 0;
    };
    bool any = false;
    if (MULTI) {
        for (int d = tid; d < a.ndom; d += NT) any = any || left_box(d);
        any = __syncthreads_or(any) != 0;
    } else {
        any = left_box(0);
    }
    if (any) {
        // their items in float64, and their outputs stay marked
        int mb = 0;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            const Item it = fx_item<MULTI>(a, item);
            if (MULTI && !left_box(it.dom)) continue;
            const Geom g = MULTI ? a.table[it.dom].g : a.g;
            Fields<const double> in = a.in;
            Fields<double> out = a.out;
            if (MULTI) {
                const DomainDesc &d = a.table[it.dom];
                in = {(const double *)d.fld[a.parity][0], (const double *)d.fld[a.parity][1],
                      (const double *)d.fld[a.parity][2]};
                out = {(double *)d.fld[1 - a.parity][0], (double *)d.fld[1 - a.parity][1],
                       (double *)d.fld[1 - a.parity][2]};
            }
            double inc[3] = {0, 0, 0};
            slow_item<C_ONLY>(a.k, g, in, out, it, reinterpret_cast<double(*)[2][G::BOX]>(sm.nb), mb, inc);
            if (tid == 0) (MULTI ? a.table[it.dom].box : a.box)[1 - a.parity] = 1;
            if (STATS) put_sums(inc, a.partials, item);
        }
    }
    if ((MULTI || !any) && (a.sched || (int)blockIdx.x < nitems)) {
        if (tid == 0) {
            for (int s = 0; s < S; ++s) mbar_init(smem_u32(&sm.bar[s]), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        // producer (thread 0): the CTA's items and their planes, S-2 loads ahead
        // (see step_tma_kernel); items of domains that left the box are passed over
        int p_item = 0, p_pz = 0, p_xs = 0, p_ys = 0, p_seq = 0, p_round = 0;
        bool p_done = a.sched == nullptr;
        Item p_it;
        auto take = [&]() {
            int v;
            do {
                if (a.sched) {
                    v = p_round == 0 ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(&a.sched[0], 1);
                    if (v >= nitems) {
                        v = nitems;
                        if (atomicAdd(&a.sched[1], 1) == (int)gridDim.x - 1) {
                            atomicExch(&a.sched[0], 0);
                            atomicExch(&a.sched[1], 0);
                        }
                        p_done = true;
                    }
                } else {
                    v = min(nitems, (int)blockIdx.x + p_round * (int)gridDim.x);
                }
                ++p_round;
                if (v < nitems) p_it = fx_item<MULTI>(a, v);
            } while (MULTI && any && v < nitems && left_box(p_it.dom));
            s_next[p_seq & 1] = v;
            ++p_seq;
            p_item = v;
        };
        const CUtensorMap *p_mS = &mapS, *p_mL = &mapL, *p_mC = &mapC;
        auto p_set = [&]() {
            if (p_item < nitems) {
                p_pz = p_it.z0 - 1;
                const int xoff = MULTI ? a.table[p_it.dom].g.xoff : a.g.xoff;
                p_xs = p_it.bx * TX + xoff - XH;
                p_ys = p_it.by * TY;
                if (MULTI) {
                    p_mS = &a.table[p_it.dom].maps[a.parity][0];
                    p_mL = &a.table[p_it.dom].maps[a.parity][1];
                    p_mC = &a.table[p_it.dom].maps[a.parity][2];
                }
            }
        };
        int ist = 0, issued = 0;
        auto issue = [&]() {
            const uint32_t bar = smem_u32(&sm.bar[ist]);
            uint32_t bytes = 3u * (uint32_t)G::BOX_BYTES;
            if (a.inject_stall && issued == 1) bytes += 16u;   // test hook: this phase can never complete
            mbar_expect_tx(bar, bytes);
            tma_load_3d(smem_u32(sm.raw[ist][0]), p_mS, p_xs, p_ys, p_pz + 1, bar);
            tma_load_3d(smem_u32(sm.raw[ist][1]), p_mL, p_xs, p_ys, p_pz + 1, bar);
            tma_load_3d(smem_u32(sm.raw[ist][2]), p_mC, p_xs, p_ys, p_pz + 1, bar);
            if (++p_pz > p_it.z1) {
                take();
                p_set();
            }
            ist = ist + 1 == S ? 0 : ist + 1;
            ++issued;
        };
        if (tid == 0) {
            take();
            p_set();
            for (int l = 0; l < S - 2 && p_item < nitems; ++l) issue();
        }
        __syncthreads();

        // ring cell of this thread: the last 96 threads take the top and bottom
        // rows, then the left and right columns
        const int rt = tid - (NT - G::RING);
        int ro = 0;
        if (rt >= 0) {
            if (rt < TX) ro = XH + rt;
            else if (rt < 2 * TX) ro = (BY - 1) * BX + XH + rt - TX;
            else if (rt < 2 * TX + TY) ro = (rt - 2 * TX + 1) * BX + XH - 1;
            else ro = (rt - 2 * TX - TY + 1) * BX + XH + TX;
        }
        const int cbias = fx::c_bias(kx.ec);

        // Registers between planes: of the plane below, which field is the smaller
        // one, the two rates (its other values are in the shared planes) and the
        // flux through the lower face; of the plane below that, the larger field's
        // value in fixed point and the smaller one's.
        int small[kCells];
        i64 rb[kCells], rs[kCells], Fz[kCells], zb[kCells];
        double zs[kCells];
        fx::Nb Xn[kCells];
#pragma unroll
        for (int j = 0; j < kCells; ++j) {
            small[j] = 0;
            rb[j] = rs[j] = Fz[j] = zb[j] = 0;
            zs[j] = 0;
        }
        double acc[3] = {0, 0, 0};
        int st = 0, mb = 0, st_prev = 0, mb_prev = 0, consumed = 0;
        uint32_t par = 0;
        bool dead = false;
        for (int seq = 0; !dead; ++seq) {
            const int item = s_next[seq & 1];
            if (item >= nitems) break;
            const Item it = fx_item<MULTI>(a, item);
            // (an ensemble's stays in memory: its copy would spill 160 bytes, and 16
            // domains of 64^3 take 230 instead of 221 us)
            const std::conditional_t<MULTI, const Geom &, Geom> g = MULTI ? a.table[it.dom].g : a.g;
            Fields<double> out = a.out;
            int *box = a.box;
            if (MULTI) {
                const DomainDesc &d = a.table[it.dom];
                out = {(double *)d.fld[1 - a.parity][0], (double *)d.fld[1 - a.parity][1],
                       (double *)d.fld[1 - a.parity][2]};
                box = d.box;
            }
            const int z0 = it.z0, z1 = it.z1, x = it.bx * TX + tx, y = it.by * TY + ty0;
            bool vj[kCells];
#pragma unroll
            for (int j = 0; j < kCells; ++j) vj[j] = FULL || (x < g.nx && y + j < g.ny);
            const uint32_t col = (uint32_t)((y + 1) * (int)g.P + x + g.xoff);
            for (int pz = z0 - 1; pz <= z1; ++pz) {
                const bool late = !mbar_wait(smem_u32(&sm.bar[st]), par, a.limit_ns);
                if (late) atomicOr(a.err, 1);
                const double *rS = sm.raw[st][0], *rL = sm.raw[st][1], *rC = sm.raw[st][2];
                fx::Own X[kCells] = {};
                int sm_new[kCells];
                i64(*nb)[G::BOX] = sm.nb[mb];
                auto put_nb = [&](int o, const fx::Nb &n) {
                    if (!C_ONLY) {
                        nb[0][o] = n.S;
                        nb[1][o] = n.L;
                    }
                    nb[2][o] = n.W;
                    nb[3][o] = n.M;
                };
                auto own_cells = [&](bool rates) {
#pragma unroll
                    for (int j = 0; j < kCells; ++j) {
                        const int o = ob + j * BX;
                        fx::pass_a<C_ONLY>(kx, rS[o], rL[o], rC[o], cbias, Xn[j], X[j], rates);
                        put_nb(o, Xn[j]);
                        if (!C_ONLY) sm_new[j] = smaller(rS[o], rL[o]);
                    }
                };
                if (C_ONLY || (pz >= z0 && pz < z1)) own_cells(true);
                else own_cells(false);             // a halo plane
                if (rt >= 0) {
                    fx::Nb n;
                    fx::Own unused;
                    fx::pass_a<C_ONLY>(kx, rS[ro], rL[ro], rC[ro], cbias, n, unused, false);
                    put_nb(ro, n);
                }
                // the plane barrier also tells every thread whether any wait ran out
                if (__syncthreads_or(late)) {
                    dead = true;
                    break;
                }
                if (tid == 0 && p_item < nitems) issue();   // refill the stage freed two planes ago

                const int q = pz - 1;
                const i64 *nW = sm.nb[mb_prev][2], *nM = sm.nb[mb_prev][3];
                i64 W[kCells], M[kCells], Fu[kCells];
#pragma unroll
                for (int j = 0; j < kCells; ++j) {
                    W[j] = nW[ob + j * BX];            // (the first plane of an item: left from the last item, unused)
                    M[j] = nM[ob + j * BX];
                    Fu[j] = fx::face(Xn[j].M, M[j], Xn[j].W, W[j]);
                }
                if (q >= z0) {
                    const uint32_t base = col + (uint32_t)(q + 1) * (uint32_t)g.PS, sink = base - col;
                    double gS[kCells], gL[kCells], gC[kCells];
                    bool bad = false;
                    i64 Fy = fx::face(M[0], nM[ob - BX], W[0], nW[ob - BX]);
#pragma unroll
                    for (int j = 0; j < kCells; ++j) {
                        const int o = ob + j * BX;
                        const i64 Fyu = fx::face(nM[o + BX], M[j], nW[o + BX], W[j]);
                        const i64 fl = (fx::face(nM[o + 1], M[j], nW[o + 1], W[j]) -
                                        fx::face(M[j], nM[o - 1], W[j], nW[o - 1])) +
                                       (Fyu - Fy) + (Fu[j] - Fz[j]);
                        Fy = Fyu;
                        const double c = sm.raw[st_prev][2][o];
                        const double df = (double)fl;
                        gC[j] = fma(df, kx.sc, c);
                        if (!C_ONLY) {
                            const int f = small[j];
                            const i64 *nB = sm.nb[mb_prev][1 - f];
                            const i64 b6 = (nB[o + 1] + nB[o - 1]) + (nB[o + BX] + nB[o - BX]) + (sm.nb[mb][1 - f][o] + zb[j]);
                            const i64 ib = fx::eta_inc(kx, rb[j], nB[o], b6);
                            const double gb = fx::eta_large(kx, nB[o], ib);
                            const double *ps = sm.raw[st_prev][f];
                            const double s6 = (ps[o + 1] + ps[o - 1]) + (ps[o + BX] + ps[o - BX]) + (sm.raw[st][f][o] + zs[j]);
                            const double ds = fx::eta_inc(kx, rs[j], ps[o], s6);
                            const double gs = fma(ds, kx.su, ps[o]);
                            gS[j] = f ? gb : gs;
                            gL[j] = f ? gs : gb;
                            if (STATS && vj[j]) {
                                const double db = fx::eta_inc_large(kx, sm.raw[st_prev][1 - f][o], ps[o], nB[o], sm.nb[mb_prev][f][o], W[j],
                                                                    b6 - 6 * nB[o], f);
                                const double iS = f ? db : ds, iL = f ? ds : db;
                                acc[1] = fma(iS, iS, acc[1]);
                                acc[2] = fma(iL, iL, acc[2]);
                            }
                            bad = bad || (vj[j] && !fx::in_box_eta((unsigned)__double2hiint(gS[j]) & 0x7fffffffu,
                                                                   (unsigned)__double2hiint(gL[j]) & 0x7fffffffu));
                        }
                        bad = bad || (vj[j] && !fx::in_box_c((unsigned)__double2hiint(gC[j]), kx.cmax));
                        if (STATS && vj[j]) acc[0] = fma(df, df, acc[0]);
                        // a cell outside the domain stores to padding that nothing reads
                        const uint32_t at = vj[j] ? base + (uint32_t)j * (uint32_t)g.P : sink;
                        put_ghost<double, C_ONLY, uint32_t>(out, at, gS[j], gL[j], gC[j]);
                    }
                    if (bad) box[1 - a.parity] = 1;
                    // face ghosts: as in step_tma_kernel
                    const bool per = g.bc == 0;
                    auto put_row = [&](int j, uint32_t d) {
                        if (vj[j])
                            put_ghost<double, C_ONLY, uint32_t>(out, base + (uint32_t)j * (uint32_t)g.P + d, gS[j],
                                                                gL[j], gC[j]);
                    };
#pragma unroll
                    for (int j = 0; j < kCells; ++j) {
                        if (x == 0) put_row(j, per ? (uint32_t)g.nx : (uint32_t)-1);
                        if (x == g.nx - 1) put_row(j, per ? (uint32_t)-g.nx : 1u);
                        if (y + j == 0) put_row(j, per ? (uint32_t)g.ny * (uint32_t)g.P : (uint32_t)-g.P);
                        if (y + j == g.ny - 1) put_row(j, per ? (uint32_t)(-g.ny) * (uint32_t)g.P : (uint32_t)g.P);
                        if (q == 0) put_row(j, per ? (uint32_t)g.nz * (uint32_t)g.PS : (uint32_t)-g.PS);
                        if (q == g.nz - 1) put_row(j, per ? (uint32_t)(-g.nz) * (uint32_t)g.PS : (uint32_t)g.PS);
                    }
                }
#pragma unroll
                for (int j = 0; j < kCells; ++j) {
                    Fz[j] = Fu[j];
                    if (!C_ONLY) {
                        const int f = sm_new[j], o = ob + j * BX;
                        small[j] = f;
                        rb[j] = f ? X[j].bS : X[j].bL;
                        rs[j] = f ? X[j].bL : X[j].bS;
                        zb[j] = sm.nb[mb_prev][1 - f][o];
                        zs[j] = sm.raw[st_prev][f][o];
                    }
                }
                st_prev = st;
                mb_prev = mb;
                if (++st == S) {
                    st = 0;
                    par ^= 1u;
                }
                mb = mb + 1 == 3 ? 0 : mb + 1;
                ++consumed;
            }
            if (STATS && !dead) {
                // (sums of squares in the increments' units until here)
                acc[0] = acc[0] * kx.sc * kx.sc;
                acc[1] = acc[1] * kx.su * kx.su;
                acc[2] = acc[2] * kx.su * kx.su;
                put_sums(acc, a.partials, item);
                acc[0] = acc[1] = acc[2] = 0;
            }
        }
        if (dead && tid == 0) {
            // drain this CTA's copies still in flight (bounded), stop taking items
            for (int d = 0; d < issued - consumed; ++d)
                (void)mbar_wait(smem_u32(&sm.bar[(st + d) % S]), par ^ (uint32_t)(((st + d) / S) & 1), a.limit_ns);
            if (!p_done && atomicAdd(&a.sched[1], 1) == (int)gridDim.x - 1) {
                atomicExch(&a.sched[0], 0);
                atomicExch(&a.sched[1], 0);
            }
        }
    }
    if (a.second) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <bool C_ONLY, bool FULL, bool MULTI>
cudaError_t attr() {
    const cudaError_t e = cudaFuncSetAttribute(step_fx_kernel<C_ONLY, FULL, MULTI, false>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(step_fx_kernel<C_ONLY, FULL, MULTI, true>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
}

void launch(const CUtensorMap *maps, const FxArgs &a, bool c_only, bool multi, int grid, bool pdl, cudaStream_t s) {
    if (a.nitems < grid) grid = a.nitems;
    const bool full = a.set == SET_WHOLE;
#define PPF_FX_LAUNCH(CO, FU, MU)                                                                                      \
    {                                                                                                                  \
        if (a.partials)                                                                                                \
            launch_step_ex(pdl, step_fx_kernel<CO, FU, MU, true>, grid, kThreads, kSmemBytes, s, maps[0], maps[1],     \
                           maps[2], a);                                                                                \
        else                                                                                                           \
            launch_step_ex(pdl, step_fx_kernel<CO, FU, MU, false>, grid, kThreads, kSmemBytes, s, maps[0], maps[1],    \
                           maps[2], a);                                                                                \
    }
    if (multi) { if (full) PPF_FX_LAUNCH(false, true, true) else PPF_FX_LAUNCH(false, false, true) }
    else if (c_only) { if (full) PPF_FX_LAUNCH(true, true, false) else PPF_FX_LAUNCH(true, false, false) }
    else { if (full) PPF_FX_LAUNCH(false, true, false) else PPF_FX_LAUNCH(false, false, false) }
#undef PPF_FX_LAUNCH
}

// the launches of a step: one over the whole tiles when there are no others
// or over every tile, or the whole tiles and the edge tiles
void launch_sets(const CUtensorMap *maps, FxArgs a, const int *items, bool c_only, bool multi, int grid, bool pdl,
                 bool split, cudaStream_t s) {
    const int ne = items[0], nw = items[1], na = items[2];
    if (ne == 0 || (split && nw > 0)) {
        a.set = SET_WHOLE;
        a.nitems = nw;
        launch(maps, a, c_only, multi, grid, pdl, s);
        if (ne == 0) return;
        a.set = SET_EDGE;
        a.nitems = ne;
        a.second = 1;
        a.inject_stall = 0;
        if (a.partials) a.partials += 3 * (int64_t)nw;
        if (a.sched) a.sched += 2;
    } else {
        a.set = SET_ALL;
        a.nitems = na;
    }
    launch(maps, a, c_only, multi, grid, pdl, s);
}

}  // namespace

int fx_occupancy(bool multi) {
    static int occ_of[64][2];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int &occ = occ_of[dev][multi];
    if (!occ) {
        cudaError_t e = multi ? attr<false, true, true>() : attr<false, true, false>();
        if (e == cudaSuccess) e = multi ? attr<false, false, true>() : attr<false, false, false>();
        if (!multi && e == cudaSuccess) e = attr<true, true, false>();
        if (!multi && e == cudaSuccess) e = attr<true, false, false>();
        int o = 0;
        if (e == cudaSuccess)
            e = multi ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, step_fx_kernel<false, true, true, true>, kThreads, kSmemBytes)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, step_fx_kernel<false, true, false, true>, kThreads, kSmemBytes);
        if (e != cudaSuccess || o < 1) return 0;
        occ = o;
    }
    return occ;
}

cudaError_t launch_step_fx(const Geom &g, const Coef<double> &k, const FxCoef &kx, const CUtensorMap *maps,
                           Fields<const double> in, Fields<double> out, bool c_only, double *partials,
                           const StepTune &tune, int *err, unsigned long long limit_ns, int inject_stall, int *sched,
                           int *box, int parity, cudaStream_t s) {
    FxArgs a;
    memset(&a, 0, sizeof a);
    a.g = g;
    a.k = k;
    a.kx = kx;
    a.in = in;
    a.out = out;
    a.tiles = tiles_of<double>(g, 0);
    a.zs = zsplit(g, tune);
    a.partials = partials;
    a.err = err;
    a.limit_ns = limit_ns;
    a.parity = parity;
    a.inject_stall = inject_stall;
    a.sched = tune.sched ? sched : nullptr;
    a.box = box;
    const int64_t chunks = tma_items<double>(g, tune) / ((int64_t)a.tiles.ntx * a.tiles.nty);
    const int items[3] = {(int)(chunks * tiles_in_set(a.tiles, SET_EDGE)), (int)(chunks * tiles_in_set(a.tiles, SET_WHOLE)),
                          (int)(chunks * tiles_in_set(a.tiles, SET_ALL))};
    launch_sets(maps, a, items, c_only, false, tune.grid, tune.pdl != 0, tune.split != 0, s);
    return cudaGetLastError();
}

cudaError_t launch_step_fx_multi(const DomainDesc *table, int ndom, const int *items, const Coef<double> &k,
                                 const FxCoef &kx, int parity, double *partials, int grid, bool pdl, bool split,
                                 int *err, unsigned long long limit_ns, int *sched, cudaStream_t s) {
    FxArgs a;
    memset(&a, 0, sizeof a);
    a.k = k;
    a.kx = kx;
    a.tiles = {1, 1, 1, 1};
    a.zs = {1, 1, 1};
    a.partials = partials;
    a.err = err;
    a.limit_ns = limit_ns;
    a.table = table;
    a.ndom = ndom;
    a.parity = parity;
    a.sched = sched;
    CUtensorMap none[3];
    memset(none, 0, sizeof none);
    launch_sets(none, a, items, false, true, grid, pdl, split, s);
    return cudaGetLastError();
}

}  // namespace ppf
