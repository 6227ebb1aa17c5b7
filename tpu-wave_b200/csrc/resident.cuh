// On-chip runs of the elastic and acoustic steps: many steps in one cooperative launch, each CTA keeping one
// tile of the grid in shared memory, for grids that fit on the chip's SMs (FP32: elastic up to
// about 1.1 million cells, acoustic 1.15 million).
//
// Such a grid is bound by latency, not by bytes: one launch a step leaves the machine idle
// between launches, and a launch's first loads and its boundary strips are a serial chain of some
// 30 us whatever the grid's size. Here the state never leaves the SMs between steps. What limits
// a step is the exchange of tile edges (about a microsecond: one store and one load through L2)
// and the instructions of the largest tile. Us a step, one launch a step -> here (B200, FP32, energy
// off): 48 x 40 29.1 -> 2.4, 200 x 150 27.2 -> 2.5, 509 x 317 28.9 -> 3.4, 700 x 700 30.7 -> 7.4, 1024 x 1024
// 38.1 -> 15.7; with the energy 509 x 317 33.9 -> 4.8; FP64 509 x 317 30.9 -> 5.0, 700 x 700 32.7 -> 13.1;
// '6C' 509 x 317 32.9 -> 3.9. Acoustic FP32 (two launches and the receivers' before): periodic 256 x 256
// 5.3 -> 1.8, 512 x 512 7.5 -> 2.3, 1000 x 1000 16.3 -> 4.6; free surface 512 x 512 8.5 -> 2.5.
//
// A tile owns rows [x0, x1) and columns [y0, y1) (the last tiles also the N-type row Mx and column
// My). It holds the stresses with a halo of 3 points on each side and the velocities with 2, which
// it recomputes itself, so one exchange of stresses a step suffices:
//   V: velocities of the tile and of its halo from the stresses (they read nothing the
//      neighbour's own velocities need, so both compute the same values);
//   S: stresses of the tile from the velocities; the points within 3 of an edge also go to the
//      exchange buffer;
//   X: the halo points of the neighbours' stresses are read from the exchange buffer.
// An exchanged value travels as 64-bit words of 32 value bits and a 32-bit tag, the number of the
// step in the handle's life: a reader polls the word itself until the tag is the one it waits
// for, so there is no flag, fence or barrier between CTAs. Words alternate between two buffers by
// the tag's parity: a CTA can be at most one step ahead of its neighbours, since it needs their
// words of the step before. Every poll is bounded; a CTA that gives up raises FLAG_TIMEOUT and
// leaves, and so in turn do the CTAs that wait for it.
//
// Thread layout: an item is one row of 16 bytes' worth of columns (4 FP32, 2 FP64), items are
// dealt to the threads row by row. Per point the arithmetic and the order of the right-hand-side
// terms are those of step_kernels.cu: results are bit-identical.
#pragma once
#include "kernels.h"
#include "stepper.cuh"
#include "vec.cuh"

namespace tw {

namespace {


// the closure and penalty weights of the x ends in shared memory, as Vec weights (read there with
// one broadcast load; indexed by the row they would come from the parameter bank one by one)
template <class C>
struct XEnds {
    using W = typename Vec<C>::W;
    W dn[6][5], dm[8][5];   // M-type rows 0..2, Mx-3..Mx-1; N-type rows 0..3, Mx-3..Mx
    W satM[6], satN[2], pM[6];
};
template <class C>
__device__ __forceinline__ void load_ends(XEnds<C> &x, const Ops<C> &o, int tid)
{
    if (tid < 15) { x.dn[tid / 5][tid % 5] = wt(o.dnL[tid / 5][tid % 5]); x.dn[3 + tid / 5][tid % 5] = wt(o.dnR[tid / 5][tid % 5]); }
    if (tid < 20) { x.dm[tid / 5][tid % 5] = wt(o.dmL[tid / 5][tid % 5]); x.dm[4 + tid / 5][tid % 5] = wt(o.dmR[tid / 5][tid % 5]); }
    if (tid < 3) { x.satM[tid] = wt(o.satML[tid]); x.satM[3 + tid] = wt(o.satMR[tid]); x.pM[tid] = wt(o.pML[tid]); x.pM[3 + tid] = wt(o.pMR[tid]); }
    if (tid == 0) { x.satN[0] = wt(o.satNL); x.satN[1] = wt(o.satNR); }
}

// x derivative of an M-type row ix next to an x end (get(r): the N-type neighbour's vector at row r)
template <class C, class G>
__device__ __forceinline__ Vec<C> vdxN_end(const XEnds<C> &o, const St<C> &s, int Mx, int ix, G get)
{
    const bool L = ix < 3;
    const auto *c = o.dn[L ? ix : ix - (Mx - 6)];
    const int r0 = L ? 0 : Mx - 4;
    Vec<C> v = vzero(C(0));
#pragma unroll
    for (int w = 0; w < 5; w++) v = s.add(v, mulw(get(r0 + w), c[w]));
    return v;
}
// the same of an N-type row from its M-type neighbour
template <class C, class G>
__device__ __forceinline__ Vec<C> vdxM_end(const XEnds<C> &o, const St<C> &s, int Mx, int ix, G get)
{
    const bool L = ix < 4;
    const auto *c = o.dm[L ? ix : ix - (Mx - 7)];
    const int r0 = L ? 0 : Mx - 5;
    Vec<C> v = vzero(C(0));
#pragma unroll
    for (int w = 0; w < 5; w++) v = s.add(v, mulw(get(r0 + w), c[w]));
    return v;
}

template <int CPST, class C>
__device__ __forceinline__ void vupdate(const St<C> &t_, Vec<C> &s, Vec<C> &r, Vec<C> &c)
{
    if constexpr (CPST == 0) {
        s = t_.add(s, r);
    } else if constexpr (CPST == 1 || CPST == 3) {
        const Vec<C> y = t_.add(r, c), t = t_.add(s, y);
        c = t_.sub(y, t_.sub(t, s));
        s = t;
    } else if constexpr (CPST == 2 || CPST == 4) {
        const Vec<C> t = t_.add(s, r);
        r = t_.sub(r, t_.sub(t, s));
        s = t;
    } else {
        const Vec<C> b = (CPST == 5) ? t_.add(r, c) : r;
        const Vec<C> t = t_.add(s, b);
        const Vec<C> pa = t_.sub(t, b), pb = t_.sub(t, pa);
        const Vec<C> d = t_.add(t_.sub(s, pa), t_.sub(b, pb));
        s = t;
        if constexpr (CPST == 5) c = d; else r = d;
    }
}

// ---- exchange words: 32 value bits and the tag (an FP64 value is two words)
__device__ __forceinline__ u64 xword(unsigned v, unsigned tag)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(v), "r"(tag));
    return r;
}
__device__ __forceinline__ void xst(u64 *p, float v, unsigned tag)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(xword(__float_as_uint(v), tag)) : "memory");
}
// two words at once (each word is written whole)
__device__ __forceinline__ void xst2(u64 *p, u64 x, u64 y)
{
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void xst(u64 *p, double v, unsigned tag)
{
    xst2(p, xword((unsigned)__double2loint(v), tag), xword((unsigned)__double2hiint(v), tag));
}
__device__ __forceinline__ void xstv(u64 *p, const float (&e)[4], unsigned tag)
{
    xst2(p, xword(__float_as_uint(e[0]), tag), xword(__float_as_uint(e[1]), tag));
    xst2(p + 2, xword(__float_as_uint(e[2]), tag), xword(__float_as_uint(e[3]), tag));
}
__device__ __forceinline__ void xstv(u64 *p, const double (&e)[2], unsigned tag)
{
    xst(p, e[0], tag);
    xst(p + 2, e[1], tag);
}
__device__ __forceinline__ u64 xld(const u64 *p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// one exchanged value: loaded, and whether it is the step's
template <class C> struct XV;
template <> struct XV<float> {
    u64 x;
    __device__ __forceinline__ void load(const u64 *p) { x = xld(p); }
    __device__ __forceinline__ bool ok(unsigned tag) const { return (unsigned)(x >> 32) == tag; }
    __device__ __forceinline__ float get() const { return __uint_as_float((unsigned)x); }
};
template <> struct XV<double> {
    u64 x, y;
    __device__ __forceinline__ void load(const u64 *p)
    {
        x = xld(p);
        y = xld(p + 1);
    }
    __device__ __forceinline__ bool ok(unsigned tag) const { return (unsigned)(x >> 32) == tag && (unsigned)(y >> 32) == tag; }
    __device__ __forceinline__ double get() const { return __hiloint2double((int)(unsigned)y, (int)(unsigned)x); }
};

}  // namespace

// one tile's shared memory: rows of NF x RES_P values (the five fields, then their residuals under a
// compensation code, then with CS the coefficients), so that every neighbour of a point is at a
// compile-time distance from it. A row's vectors belong to LANES threads; a thread keeps its column
// and walks down the rows, RES_THREADS / LANES rows apart (tall tiles: two rows at a time).
// PHYS: RES_ELASTIC, or acoustic (MN, NM and the pressure in MM0; only the pressure is exchanged, its halo
// is a cross, nothing reads beyond an N-type seam): RES_AC_FREE the x free surfaces, RES_AC_PER
// periodic x, whose halo rows are the rows at the other end.
// blk: this CTA's tile, of nblk
// DUMP: the state after every step goes to a.dump (the adjoint's recomputed segments)
template <class C, int CPST, bool ENERGY, bool CS, int PHYS, bool DUMP = false>
__device__ __forceinline__ void resident_run(const ResArgs<C> &a, int blk, int nblk)
{
    constexpr bool KR = Cpst<CPST>::keep_r, KC = Cpst<CPST>::keep_c, RES = KR || KC;
    constexpr int N = Vec<C>::N, H = RES_PAD, P = RES_P, LANES = RES_LANES_COLS / N;
    constexpr bool EL = PHYS == RES_ELASTIC, PERX = PHYS == RES_AC_PER;
    constexpr int NB = EL ? 5 : 3;                         // fields
    constexpr int NF = NB + (RES ? NB : 0) + (CS ? NB : 0), RS = NF * P;
    constexpr int iNN = 0, iMN = EL ? 1 : 0, iNM = iMN + 1, iM0 = iNM + 1, iM1 = EL ? iM0 + 1 : iM0;   // (acoustic: syy is p)
    constexpr int o_r = NB * P, o_c = (RES ? 2 : 1) * NB * P;   // residual and coefficient rows
    constexpr int XW = sizeof(C) / 4;                      // exchange words of a value
    using V = Vec<C>;
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ double red[2][3][RES_THREADS / 32];
    __shared__ int bad_s;
    __shared__ XEnds<C> ends;
    const int tid = threadIdx.x;
    const int Mx = a.Mx, My = a.My;
    const int tx = blk / a.nty, ty = blk - tx * a.nty;
    const int x0 = (int)((long)tx * Mx / a.ntx), x1 = (int)((long)(tx + 1) * Mx / a.ntx);
    const int nq4 = (My + 4) / 4;   // column quads of the grid (My + 1 columns)
    const int y0 = 4 * (int)((long)ty * nq4 / a.nty);
    const bool lastx = tx == a.ntx - 1, lasty = ty == a.nty - 1;
    const int y1 = lasty ? My : 4 * (int)((long)(ty + 1) * nq4 / a.nty);   // M-type columns end here
    const int R = x1 - x0, W = y1 - y0;             // owned M-type rows and columns
    const int RN = R + (lastx ? 1 : 0), WN = W + (lasty ? 1 : 0);
    C *sm = reinterpret_cast<C *>(res_smem);
    C *altL = sm + (size_t)a.rows_s * RS, *altR = altL + a.rows_s;
    auto at = [&](int i, int r, int c) { return sm + (r + H) * RS + i * P + c + H; };   // i: iNN .. iM1
    auto slot_of = [](int i) { return EL ? i : (i == iM0 ? (int)F_MM0 : i + F_MN); };
    auto index_of = [](int f) { return EL ? f : (f == F_MM0 ? iM0 : f - F_MN); };
    auto ntypeY = [](int f) { return f == F_NN || f == F_MN; };
    auto rows_of = [&](int f) { return (f == F_NN || f == F_NM) ? Mx + 1 : Mx; };
    auto phys = [&](bool ntype, int c) {   // physical column of the tile's column c
        int g = y0 + c;
        if (g < 0) g += My;
        else if (ntype ? g > My : g >= My) g -= My;
        return g;
    };
    auto physr = [&](bool ntype, int g) {   // physical row of grid row g (periodic x)
        if (PERX) {
            if (g < 0) g += Mx;
            else if (ntype ? g > Mx : g >= Mx) g -= Mx;
        }
        return g;
    };
    const int it0 = *a.step;
    if (tid == 0) bad_s = 0;
    load_ends<C>(ends, a.op, tid);

    // ---- load the tile with its halo
    for (int k = tid; k < a.rows_s * P; k += RES_THREADS) {
        const int r = k / P - H, c = k - (r + H) * P - H, g = x0 + r;
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const int f = slot_of(i), gr = physr(f == F_NN || f == F_NM, g);
            const bool in = gr >= 0 && gr < rows_of(f) && r < RN + 3 && r >= -3 && c >= -3 && c < WN + 3;
            const long o = in ? (long)gr * a.pitch + phys(ntypeY(f), c) : 0;
            C *q = at(i, r, c);
            q[0] = in ? a.in[f][o] : C(0);
            if constexpr (RES) q[o_r] = in ? a.rin[f][o] : C(0);
            if constexpr (CS) q[o_c] = in ? a.coef[f][o] : C(0);
        }
    }
    // the N-type seam: an M-type point left of column 0 reads column My where this tile holds
    // column 0, one right of column My - 1 reads column 0 where it holds column My
    for (int k = tid; EL && k < a.rows_s; k += RES_THREADS) {
        const int g = x0 + k - H;
        const bool in = g >= 0 && g <= Mx && k - H < RN + 3;
        altL[k] = in && ty == 0 ? a.in[F_NN][(long)g * a.pitch + My] : C(0);
        altR[k] = in && lasty ? a.in[F_NN][(long)g * a.pitch] : C(0);
    }
    const int rb = a.rcv_off[blk], re = a.rcv_off[blk + 1];
    const St<C> st(a.op.st, a.n > 0);
    const bool multi = a.ntx * a.nty > 1;
    const int lc = W;   // (last tile of a row) the local column of My

    // ---- this thread's column and rows: V on rows [va, vb) and columns -4 .. WN + 1, S on the owned
    // points. Tiles of few rows give the two kinds of point of a phase to the two halves of the CTA.
    constexpr int SLOTS = RES_THREADS / LANES;
    const int va = PERX ? -1 : max(-2, -x0), vb = PERX ? R + 2 : min(R + 2, Mx + 1 - x0);
    const int c = (tid % LANES) * N - 4;
    const bool split = vb - va <= SLOTS / 2;
    const int slot = split ? (tid / LANES) % (SLOTS / 2) : tid / LANES, dslot = split ? SLOTS / 2 : SLOTS;
    const bool first = !split || tid < RES_THREADS / 2, second = !split || tid >= RES_THREADS / 2;
    const bool vcol = c < WN + 2, scol = c >= 0 && c < WN;
    const int ownN = scol ? min(N, WN - c) : 0, ownM = scol ? max(0, min(N, W - c)) : 0;
    const bool vpair = !ENERGY && vb - va > SLOTS;   // (the energy's registers leave no room for two rows)
    const bool seamL = ty == 0 && c == -N, seamR = lasty && c + N > lc && c <= lc + 1;
    const bool bcol = c < 4 || c + N > WN - 4;   // columns the neighbours (or the seam) read
    int sq = -1;                                 // the source's column among this thread's
    if (a.src_grid >= 0)
        for (int q = 0; q < N; q++)
            if (c + q >= -3 && c + q < WN + 3 && phys(a.src_grid == G_NN || a.src_grid == G_MN, c + q) == a.src_iy) sq = q;
    auto own_row = [&](int g) { return g == a.src_grid ? a.src_ix - x0 : -(1 << 20); };
    const int srcMN = own_row(G_MN), srcNM = own_row(G_NM), srcNN = own_row(G_NN), srcMM = own_row(G_MM);
    // (periodic x: the halo rows hold the points of the other end)
    auto is_srcNM = [&](int r) { return PERX ? a.src_grid == G_NM && physr(true, x0 + r) == a.src_ix : r == srcNM; };

    // ---- this thread's halo words: 3 rows above and below over columns [-3, WN + 3), 3 columns on
    // each side, the seam columns of the V rows
    constexpr int XI = 3;   // (RES_THREADS x XI covers the largest tile: resident_plan)
    int xs[XI], xm[XI], xg[XI], xh[XI];   // shared index of NN, of MM0 (-1: none), words of NN, of MM0
    {
        // (acoustic: the pressure's rows and columns, M type)
        const int Rh = EL ? RN : R, Wh = EL ? WN : W, hw = Wh + 6, ht = PERX || tx > 0 ? 3 : 0, hb = PERX || !lastx ? 3 : 0;
        const int nvr = EL ? vb - va : 0;
        const int n1 = (ht + hb) * hw, n2 = n1 + Rh * 6, n3 = n2 + (ty == 0 ? nvr : 0), n4 = n3 + (lasty ? nvr : 0);
#pragma unroll
        for (int m = 0; m < XI; m++) {
            const int h = tid + m * RES_THREADS;
            xs[m] = xm[m] = -1;
            xg[m] = xh[m] = 0;
            if (!multi || h >= n4) continue;
            if (h < n2) {
                int r, cc;
                if (h < n1) {
                    const int q = h / hw;
                    cc = h - q * hw - 3;
                    r = q < ht ? q - 3 : Rh + (q - ht);
                } else {
                    r = (h - n1) / 6;
                    cc = h - n1 - 6 * r;
                    cc = cc < 3 ? cc - 3 : Wh + cc - 3;
                }
                const int g = physr(false, x0 + r);
                if constexpr (EL) {
                    const int cm = (lasty && cc >= WN) ? cc - 1 : cc;   // (M-type halos start at W)
                    xs[m] = (int)(at(iNN, r, cc) - sm);
                    xg[m] = (g * a.xcols + phys(true, cc)) * XW;
                    if (g < Mx) {
                        xm[m] = (int)(at(iM0, r, cm) - sm);
                        xh[m] = (g * a.xcols + phys(false, cm)) * XW;
                    }
                } else {
                    xs[m] = (int)(at(iM0, r, cc) - sm);
                    xg[m] = (g * a.xcols + phys(false, cc)) * XW;
                }
            } else {
                const bool left = h < n3;
                const int r = va + (left ? h - n2 : h - n3);
                xs[m] = (int)((left ? altL : altR) + r + H - sm);
                xg[m] = ((x0 + r) * a.xcols + (left ? My : 0)) * XW;
            }
        }
    }
    double ep_prev = 0.;
    __syncthreads();

    for (int k = 0; k < a.n; k++) {
        const int it = it0 + k;
        const bool last = k == a.n - 1;
        double ek = 0., ep0 = 0., ep1 = 0.;
        auto source = [&](V &v) {
            if (sq >= 0) {
                const double inc = a.src_inc[it];
                C e[N];
                vget(v, e);
#pragma unroll
                for (int q = 0; q < N; q++)
                    if (q == sq) e[q] = (C)add((double)e[q], inc);
                v = vset(e);
            }
        };
        // an owned row's new values into the state this step leaves
        auto dump = [&](int f, int r, int own, const V &v) {
            if constexpr (DUMP) {
                if (last || own <= 0) return;   // (the last state is the run's result)
                C *o = a.dump[f] + (long)k * a.dump_stride + (long)(x0 + r) * a.pitch + y0 + c;
                if (own >= N) {
                    vst(o, v);
                } else {
                    C e[N];
                    vget(v, e);
#pragma unroll
                    for (int q = 0; q < N - 1; q++)
                        if (q < own) o[q] = e[q];
                }
            }
        };
        // the energy weights of this thread's points of a row (loaded before the points are computed)
        struct WV { double w[N]; };
        auto weights = [&](int f, int r, bool own) {
            WV v;
            const double2 *p = reinterpret_cast<const double2 *>(a.w[f] + (long)(x0 + r) * a.pitch + y0 + c);
#pragma unroll
            for (int q = 0; q < N; q += 2) {
                const double2 x = own ? __ldg(p + q / 2) : make_double2(0., 0.);
                v.w[q] = x.x;
                v.w[q + 1] = x.y;
            }
            return v;
        };
        // ---- V: velocities
        // one row; ld(f, o): this column's vector of field f, o rows on
        auto vrow = [&](int r, C *q, auto ld) {
                const int j = x0 + r;
                [[maybe_unused]] const bool orow = r >= 0 && r < RN;
                auto coefv = [&](int f) -> V {
                    if constexpr (CS) return vld(q + index_of(f) * P + o_c);
                    else return vldg(a.coefx[f - F_MN] + (long)physr(f == F_NM, j) * a.xpitch + y0 + c + 4);
                };
                const V nnj = EL ? ld(iNN, 0) : vzero(C(0));
                if (first && (EL ? j < Mx : r >= 0 && r < R)) {   // MN: x from NN, y from MM syy
                    [[maybe_unused]] WV wv;
                    if constexpr (ENERGY) wv = weights(F_MN, r, orow && ownN > 0);
                    const V P_ = coefv(F_MN);
                    V r_ = vzero(C(0)), cc = r_, vx;
                    if constexpr (KR) r_ = vld(q + iMN * P + o_r);
                    if constexpr (KC) cc = vld(q + iMN * P + o_r);
                    if constexpr (!EL) {   // (no shear: the y derivative alone)
                    } else if (j >= 3 && j < Mx - 3) {
                        vx = taps<C>(st, ld(iNN, -1), nnj, ld(iNN, 1), ld(iNN, 2));
                        r_ = st.add(r_, mul(vx, P_));
                    } else {   // closure and SAT
                        vx = vdxN_end<C>(ends, st, Mx, j, [&](int g) { return vld(at(iNN, g - x0, c)); });
                        r_ = st.add(r_, mul(vx, P_));
                        const bool L = j < 3;
                        const V send = mulw(vld(at(iNN, L ? -x0 : Mx - x0, c)), wt(a.op.pN));
                        r_ = st.add(r_, mul(mulw(send, ends.satM[L ? j : j - (Mx - 6)]), P_));
                    }
                    r_ = st.add(r_, mul(dyN(st, q + iM1 * P, vld(q + iM1 * P)), P_));
                    V s = vld(q + iMN * P);
                    vupdate<CPST, C>(st, s, r_, cc);
                    if (r == srcMN) source(s);
                    vst(q + iMN * P, s);
                    if (orow) dump(F_MN, r, ownN, s);
                    if constexpr (RES) vst(q + iMN * P + o_r, KR ? r_ : cc);
                    if constexpr (ENERGY) {
                        C e[N];
                        vget(s, e);
#pragma unroll
                        for (int i = 0; i < N; i++)
                            if (orow && i < ownN) ek = add(ek, mul(mul((double)e[i], wv.w[i]), (double)e[i]));
                    }
                }
                if (second) {   // NM: x from MM sxx, y from NN
                    [[maybe_unused]] WV wv;
                    if constexpr (ENERGY) wv = weights(F_NM, r, orow && ownM > 0);
                    const V P_ = coefv(F_NM);
                    V r_ = vzero(C(0)), cc = r_, vx;
                    if constexpr (KR) r_ = vld(q + iNM * P + o_r);
                    if constexpr (KC) cc = vld(q + iNM * P + o_r);
                    if (PERX || (j >= 4 && j < Mx - 3)) {
                        vx = taps<C>(st, ld(iM0, -2), ld(iM0, -1), ld(iM0, 0), ld(iM0, 1));
                        r_ = st.add(r_, mul(vx, P_));
                    } else {
                        vx = vdxM_end<C>(ends, st, Mx, j, [&](int g) { return vld(at(iM0, g - x0, c)); });
                        r_ = st.add(r_, mul(vx, P_));
                        if (j == 0 || j == Mx) {   // SAT
                            const bool L = j == 0;
                            V send = vzero(C(0));
#pragma unroll
                            for (int w = 0; w < 3; w++)
                                send = st.add(send, mulw(vld(at(iM0, (L ? w : Mx - 3 + w) - x0, c)), ends.pM[(L ? 0 : 3) + w]));
                            r_ = st.add(r_, mul(mulw(send, ends.satN[L ? 0 : 1]), P_));
                        }
                    }
                    if constexpr (EL) {
                    // (left of column 0 the next column is My, not the tile's column 0)
                    V vy = dyM(st, q + iNN * P, nnj, seamL, altL + r + H);
                    if (seamR) {   // the columns from My on: the one there is column 0
                        const C *p = at(iNN, r, lc);
                        const C z = altR[r + H], p1 = p[1], p2 = p[2];
                        auto tap4 = [&](C t0, C t1, C t2, C t3) {
                            C v = mul(t0, a.op.st[0]);
                            v = add(v, mul(t1, a.op.st[1]));
                            v = add(v, mul(t2, a.op.st[2]));
                            return add(v, mul(t3, a.op.st[3]));
                        };
                        const C w0 = tap4(p[-1], z, p1, p2), w1 = tap4(z, p1, p2, p[3]);
                        C e[N];
                        vget(vy, e);
#pragma unroll
                        for (int i = 0; i < N; i++) e[i] = c + i == lc ? w0 : (c + i == lc + 1 ? w1 : e[i]);
                        vy = vset(e);
                    }
                    r_ = st.add(r_, mul(vy, P_));
                    }
                    V s = vld(q + iNM * P);
                    vupdate<CPST, C>(st, s, r_, cc);
                    if (is_srcNM(r)) source(s);
                    vst(q + iNM * P, s);
                    if (orow) dump(F_NM, r, ownM, s);
                    if constexpr (RES) vst(q + iNM * P + o_r, KR ? r_ : cc);
                    if constexpr (ENERGY) {
                        C e[N];
                        vget(s, e);
#pragma unroll
                        for (int i = 0; i < N; i++)
                            if (orow && i < ownM) ek = add(ek, mul(mul((double)e[i], wv.w[i]), (double)e[i]));
                    }
                }
        };
        if (vcol) {
            if (vpair) {   // two rows at a time: their x stencils share all but one row
                for (int r = va + 2 * slot; r < vb; r += 2 * SLOTS) {
                    C *q = at(0, r, c);
                    V nn[5], m0[5];
#pragma unroll
                    for (int w = 0; w < 5; w++) {
                        nn[w] = EL ? vld(q + iNN * P + (w - 1) * RS) : vzero(C(0));
                        m0[w] = vld(q + iM0 * P + (w - 2) * RS);
                    }
                    vrow(r, q, [&](int f, int o) { return EL && f == iNN ? nn[o + 1] : m0[o + 2]; });
                    if (r + 1 < vb) vrow(r + 1, q + RS, [&](int f, int o) { return EL && f == iNN ? nn[o + 2] : m0[o + 3]; });
                }
            } else {
                for (int r = va + slot; r < vb; r += dslot) {
                    C *q = at(0, r, c);
                    vrow(r, q, [&](int f, int o) { return vld(q + f * P + o * RS); });
                }
            }
        }
        __syncthreads();
        for (int q = rb + tid; q < re; q += RES_THREADS) {   // velocity receivers (the velocities rest during S)
            const int *e = a.rcv + 4 * q;
            if (e[0] == F_MN || e[0] == F_NM)
                a.traces[(long)e[3] * a.max_steps + it] = (double)*at(index_of(e[0]), e[1] - x0, e[2] - y0);
        }
        // ---- S: stresses of the owned points; those near an edge also to the exchange words
        const unsigned tag = a.tag0 + (unsigned)k + 1u;
        u64 *xb = a.xbuf + (size_t)(tag & 1u) * (EL ? 3 : 1) * a.xarr;
        auto send = [&](int r, int own, int f3, const V &v) {
            C e[N];
            vget(v, e);
            u64 *p = xb + f3 * a.xarr + ((x0 + r) * a.xcols + y0 + c) * XW;
            if (own >= N) {
                xstv(p, e, tag);
            } else {
#pragma unroll
                for (int q = 0; q < N - 1; q++)
                    if (q < own) xst(p + q * XW, e[q], tag);
            }
        };
        auto srow = [&](int r, C *q, auto ld) {
                const int i = x0 + r;
                [[maybe_unused]] const long go = (long)i * a.pitch + y0 + c;
                auto coefv = [&](int f) -> V {
                    if constexpr (CS) return vld(q + index_of(f) * P + o_c);
                    else return vldg(a.coef[f] + go);
                };
                const bool border = !last && multi && (bcol || r < 3 || r >= R - 3);
                if constexpr (EL) {
                if (first) {   // NN: x from MN, y from NM
                    [[maybe_unused]] WV wv;
                    if constexpr (ENERGY) wv = weights(F_NN, r, true);
                    const V P_ = coefv(F_NN);
                    V r_ = vzero(C(0)), cc = r_, vx;
                    if constexpr (KR) r_ = vld(q + iNN * P + o_r);
                    if constexpr (KC) cc = vld(q + iNN * P + o_r);
                    if (i >= 4 && i < Mx - 3)
                        vx = taps<C>(st, ld(iMN, -2), ld(iMN, -1), ld(iMN, 0), ld(iMN, 1));
                    else
                        vx = vdxM_end<C>(ends, st, Mx, i, [&](int g) { return vld(at(iMN, g - x0, c)); });
                    r_ = st.add(r_, mul(vx, P_));
                    r_ = st.add(r_, mul(dyN(st, q + iNM * P, ld(iNM, 0)), P_));
                    const V old = vld(q + iNN * P);
                    V s = old;
                    vupdate<CPST, C>(st, s, r_, cc);
                    if (r == srcNN) source(s);
                    vst(q + iNN * P, s);
                    dump(F_NN, r, ownN, s);
                    if constexpr (RES) vst(q + iNN * P + o_r, KR ? r_ : cc);
                    if (border) send(r, ownN, 0, s);
                    if constexpr (ENERGY) {
                        C e[N], o[N];
                        vget(s, e);
                        vget(old, o);
#pragma unroll
                        for (int m = 0; m < N; m++)
                            if (m < ownN) {
                                if (k == 0) ep0 = add(ep0, mul(mul((double)o[m], wv.w[m]), (double)o[m]));
                                ep1 = add(ep1, mul(mul((double)e[m], wv.w[m]), (double)e[m]));
                            }
                    }
                }
                if (second && r < R && ownM > 0) {   // MM: x from NM, y from MN
                    [[maybe_unused]] WV wv3, wv4;
                    if constexpr (ENERGY) { wv3 = weights(F_MM0, r, true); wv4 = weights(F_MM1, r, true); }
                    const V L = coefv(F_MM0), M2 = coefv(F_MM1);
                    V r0 = vzero(C(0)), r1 = r0, k0 = r0, k1 = r0, vx;
                    if constexpr (KR) { r0 = vld(q + iM0 * P + o_r); r1 = vld(q + iM1 * P + o_r); }
                    if constexpr (KC) { k0 = vld(q + iM0 * P + o_r); k1 = vld(q + iM1 * P + o_r); }
                    if (i >= 3 && i < Mx - 3)
                        vx = taps<C>(st, ld(iNM, -1), ld(iNM, 0), ld(iNM, 1), ld(iNM, 2));
                    else
                        vx = vdxN_end<C>(ends, st, Mx, i, [&](int g) { return vld(at(iNM, g - x0, c)); });
                    r0 = st.add(r0, mul(vx, L));
                    r1 = st.add(r1, mul(vx, L));
                    r0 = st.add(r0, mul(vx, M2));
                    const V vy = dyM(st, q + iMN * P, ld(iMN, 0), false, nullptr);
                    r0 = st.add(r0, mul(vy, L));
                    r1 = st.add(r1, mul(vy, L));
                    r1 = st.add(r1, mul(vy, M2));
                    const V o0 = vld(q + iM0 * P), o1 = vld(q + iM1 * P);
                    V s0 = o0, s1 = o1;
                    vupdate<CPST, C>(st, s0, r0, k0);
                    vupdate<CPST, C>(st, s1, r1, k1);
                    if (r == srcMM) {
                        source(s0);
                        source(s1);
                    }
                    vst(q + iM0 * P, s0);
                    vst(q + iM1 * P, s1);
                    dump(F_MM0, r, ownM, s0);
                    dump(F_MM1, r, ownM, s1);
                    if constexpr (RES) {
                        vst(q + iM0 * P + o_r, KR ? r0 : k0);
                        vst(q + iM1 * P + o_r, KR ? r1 : k1);
                    }
                    if (border) {
                        send(r, ownM, 1, s0);
                        send(r, ownM, 2, s1);
                    }
                    if constexpr (ENERGY) {
                        C e0[N], e1[N], p0[N], p1[N];
                        vget(s0, e0);
                        vget(s1, e1);
                        vget(o0, p0);
                        vget(o1, p1);
#pragma unroll
                        for (int m = 0; m < N; m++)
                            if (m < ownM) {
                                const double w3 = wv3.w[m], w4 = wv4.w[m];
                                auto pot = [&](double b0, double b1, double &E) {
                                    E = add(E, mul(mul(b0, w3), b0));
                                    E = add(E, mul(mul(b1, w3), b1));
                                    E = add(E, mul(mul(b0, w4), b1));
                                };
                                if (k == 0) pot((double)p0[m], (double)p1[m], ep0);
                                pot((double)e0[m], (double)e1[m], ep1);
                            }
                    }
                }
                } else {
                if (r < R && ownM > 0 && (!split || (r & 1) == (second ? 1 : 0))) {   // pressure: x from NM, y from MN
                    const V K_ = coefv(F_MM0);
                    V r_ = vzero(C(0)), cc = r_, vx;
                    if constexpr (KR) r_ = vld(q + iM0 * P + o_r);
                    if constexpr (KC) cc = vld(q + iM0 * P + o_r);
                    if (PERX || (i >= 3 && i < Mx - 3))
                        vx = taps<C>(st, ld(iNM, -1), ld(iNM, 0), ld(iNM, 1), ld(iNM, 2));
                    else
                        vx = vdxN_end<C>(ends, st, Mx, i, [&](int g) { return vld(at(iNM, g - x0, c)); });
                    r_ = st.add(r_, mul(vx, K_));
                    const C *mnp = q + iMN * P;
                    r_ = st.add(r_, mul(dyM(st, mnp, vld(mnp), false, nullptr), K_));
                    V s = vld(q + iM0 * P);
                    vupdate<CPST, C>(st, s, r_, cc);
                    if (r == srcMM) source(s);
                    vst(q + iM0 * P, s);
                    if constexpr (RES) vst(q + iM0 * P + o_r, KR ? r_ : cc);
                    if (border) send(r, ownM, 0, s);
                }
                }
        };
        if (scol) {
            if (vpair) {
                for (int r = 2 * slot; r < RN; r += 2 * SLOTS) {
                    C *q = at(0, r, c);
                    V mn[5], nm[5];
#pragma unroll
                    for (int w = 0; w < 5; w++) {
                        mn[w] = EL ? vld(q + iMN * P + (w - 2) * RS) : vzero(C(0));
                        nm[w] = vld(q + iNM * P + (w - 1) * RS);
                    }
                    srow(r, q, [&](int f, int o) { return EL && f == iMN ? mn[o + 2] : nm[o + 1]; });
                    if (r + 1 < RN) srow(r + 1, q + RS, [&](int f, int o) { return EL && f == iMN ? mn[o + 3] : nm[o + 2]; });
                }
            } else {
                for (int r = slot; r < RN; r += dslot) {
                    C *q = at(0, r, c);
                    srow(r, q, [&](int f, int o) { return vld(q + f * P + o * RS); });
                }
            }
        }
        if constexpr (ENERGY) {   // each warp's sums (side by side); the CTA's are added up after the barrier
            double v3[3] = {ek, ep1, ep0};
            const int nv = k == 0 ? 3 : 2;   // (the stresses before a later step are those after the one before it)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (q < nv) v3[q] += __shfl_down_sync(0xffffffffu, v3[q], o);
            if ((tid & 31) == 0)
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (q < nv) red[k & 1][q][tid >> 5] = v3[q];
        }
        __syncthreads();
        for (int q = rb + tid; q < re; q += RES_THREADS) {   // stress receivers (the owned stresses rest until S)
            const int *e = a.rcv + 4 * q;
            if (e[0] != F_MN && e[0] != F_NM)
                a.traces[(long)e[3] * a.max_steps + it] = (double)*at(index_of(e[0]), e[1] - x0, e[2] - y0);
        }
        if constexpr (ENERGY) {
            constexpr int NW = RES_THREADS / 32;
            if (tid >> 5 == NW - 1) {   // the last warp
                const int l = tid & 31;
                double v[3];
#pragma unroll
                for (int q = 0; q < 3; q++) v[q] = l < NW && (q < 2 || k == 0) ? red[k & 1][q][l] : 0.;
#pragma unroll
                for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int q = 0; q < 3; q++) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
                if (k > 0) v[2] = ep_prev;
                ep_prev = v[1];
                if (l == 0 && it < a.max_steps) {   // records: E_p0, E_k, E_p1
                    if (v[2] != 0.) atomicAdd(a.energy + it, 0.5 * v[2]);
                    if (v[0] != 0.) atomicAdd(a.energy + (long)a.max_steps + it, 0.5 * v[0]);
                    if (v[1] != 0.) atomicAdd(a.energy + 2L * a.max_steps + it, 0.5 * v[1]);
                }
            }
        }
        if (last) break;
        // ---- X: the halo's stresses
        if (multi) {
            // a thread's words are polled together: one round trip when the neighbours are done (an
            // item at a time in FP64 and with the energy on, where the registers are short)
            constexpr int B = sizeof(C) == 8 || ENERGY ? 1 : XI;
            bool ok = true;
#pragma unroll
            for (int b = 0; b < XI; b += B) {
                if (!ok || xs[b] < 0) break;
                XV<C> v[B][3];
                ok = false;
                for (int n = 0; n < a.polls && !ok; n++) {
#pragma unroll
                    for (int m = 0; m < B; m++) {
                        if (xs[b + m] >= 0) v[m][0].load(xb + xg[b + m]);
                        if (EL && xm[b + m] >= 0) {
                            v[m][1].load(xb + a.xarr + xh[b + m]);
                            v[m][2].load(xb + 2 * a.xarr + xh[b + m]);
                        }
                    }
                    ok = true;
#pragma unroll
                    for (int m = 0; m < B; m++) {
                        if (xs[b + m] >= 0) ok = ok && v[m][0].ok(tag);
                        if (EL && xm[b + m] >= 0) ok = ok && v[m][1].ok(tag) && v[m][2].ok(tag);
                    }
                }
                if (ok) {
#pragma unroll
                    for (int m = 0; m < B; m++) {
                        if (xs[b + m] >= 0) sm[xs[b + m]] = v[m][0].get();
                        if (EL && xm[b + m] >= 0) {
                            sm[xm[b + m]] = v[m][1].get();
                            sm[xm[b + m] + P] = v[m][2].get();
                        }
                    }
                }
            }
            if (!ok) bad_s = 1;
        } else if constexpr (EL) {   // one tile: the periodic columns from the tile itself
            for (int idx = tid; idx < RN * 6; idx += RES_THREADS) {
                const int r = idx / 6, q = idx - 6 * r;
                const int cn = q < 3 ? q - 3 : WN + q - 3, cm = cn >= WN ? cn - 1 : cn;
                *at(iNN, r, cn) = *at(iNN, r, phys(true, cn));
                if (r < R) {
                    *at(iM0, r, cm) = *at(iM0, r, phys(false, cm));
                    *at(iM1, r, cm) = *at(iM1, r, phys(false, cm));
                }
            }
            for (int r = tid; r < RN; r += RES_THREADS) {
                altL[r + H] = *at(iNN, r, lc);
                altR[r + H] = *at(iNN, r, 0);
            }
        } else {
            for (int idx = tid; idx < R * 6 + (PERX ? W * 6 : 0); idx += RES_THREADS) {
                const bool col = idx < R * 6;
                const int h = col ? idx : idx - R * 6, r = h / 6, q = h - 6 * r, e = q < 3 ? q - 3 : (col ? W : R) + q - 3;
                if (col) *at(iM0, r, e) = *at(iM0, r, phys(false, e));
                else *at(iM0, e, r) = *at(iM0, physr(false, e), r);
            }
        }
        __syncthreads();
        if (bad_s) break;
    }
    // ---- the state after the run. (A value that stopped being finite at any step has stayed so: an
    // update adds to it.)
    C nf = C(0);   // stays 0 until a value is not finite (v * 0 is NaN then)
    for (int i = 0; i < NB; i++) {
        const int f = slot_of(i);
        const int rows = f == F_NN || f == F_NM ? RN : R, cols = ntypeY(f) ? WN : W;
        for (int k = tid; k < rows * RES_LANES_COLS; k += RES_THREADS) {
            const int r = k / RES_LANES_COLS, cc = k - r * RES_LANES_COLS;
            if (cc >= cols) continue;
            const C *q = at(i, r, cc);
            const long o = (long)(x0 + r) * a.pitch + y0 + cc;
            nf = nf + q[0] * C(0);
            a.out[f][o] = q[0];
            if constexpr (RES) a.rout[f][o] = q[o_r];
        }
    }
    if (tid == 0 && bad_s) atomicOr(a.flags, FLAG_TIMEOUT);
    if (nf != C(0)) atomicOr(a.flags, FLAG_NONFINITE);
    // the last CTA advances the step counter, after every CTA has read it
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(a.done, 1) == nblk - 1) {
            *a.done = 0;
            *a.step_w = it0 + a.n;
            __threadfence();
        }
    }
}

template <class C, int CPST, bool ENERGY, bool CS, int PHYS, bool DUMP = false>
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(const __grid_constant__ ResArgs<C> a)
{
    resident_run<C, CPST, ENERGY, CS, PHYS, DUMP>(a, blockIdx.x, gridDim.x);
}

// several shots side by side: shot k's tiles are the CTAs [first[k], first[k + 1]). A small shot alone
// pays a step's latency whatever its size; several share it. 24 periodic FP32 shots of 256^2 to 1024^2 (8.9
// million cells): 119 us a step by the batch kernels, 68 here.
template <class C, int CPST, bool CS, int PHYS>
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident_shots(const ResArgs<C> *shots, const int *first, int n)
{
    __shared__ ResArgs<C> a;
    int k = 0;
    while (k + 1 < n && first[k + 1] <= (int)blockIdx.x) k++;
    const int *src = reinterpret_cast<const int *>(shots + k);
    for (int i = threadIdx.x; i < (int)(sizeof(a) / sizeof(int)); i += RES_THREADS) reinterpret_cast<int *>(&a)[i] = src[i];
    __syncthreads();
    resident_run<C, CPST, false, CS, PHYS>(a, (int)blockIdx.x - first[k], first[k + 1] - first[k]);
}

// ------------------------------------------------------------------------------- launcher
// codes 1 / 3 and 2 / 4 are the same update; coefficients stay in L2 for the plain update only
template <class C, int PHYS, bool ENERGY, class F>
cudaError_t resident_code(int cpst, bool cs, F f)
{
    if (cpst == 0) return cs ? f(k_resident<C, 0, ENERGY, true, PHYS>) : f(k_resident<C, 0, ENERGY, false, PHYS>);
    if (cpst == 2 || cpst == 4) return f(k_resident<C, 4, ENERGY, true, PHYS>);
    if (cpst == 6) return f(k_resident<C, 6, ENERGY, true, PHYS>);
    if constexpr (PHYS != RES_AC_PER) {   // (the periodic tree has '0', '3' and '6')
        if (cpst == 1 || cpst == 3) return f(k_resident<C, 3, ENERGY, true, PHYS>);
        return f(k_resident<C, 5, ENERGY, true, PHYS>);
    }
    return cudaErrorInvalidValue;
}
template <class C, int PHYS, class F>
cudaError_t resident_kernel(int cpst, bool energy, bool cs, F f)
{
    if constexpr (PHYS == RES_ELASTIC)   // (acoustic energies: the per-point kernels)
        if (energy) return resident_code<C, PHYS, true>(cpst, cs, f);
    return resident_code<C, PHYS, false>(cpst, cs, f);
}

// (the opt-in is the kernel's, not a handle's: always the most a plan may ask for)
template <class C, int PHYS>
cudaError_t prepare_resident(int cpst, bool energy, const ResPlan &p, int smem_max)
{
    if constexpr (PHYS == RES_ELASTIC)
        if (cpst == 0) {
            const auto k = p.cs ? k_resident<C, 0, false, true, PHYS, true> : k_resident<C, 0, false, false, PHYS, true>;
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
            if (e != cudaSuccess) return e;
            if (energy) {   // the gradient's sweeps without the energy
                const cudaError_t e2 = resident_kernel<C, PHYS>(0, false, p.cs, [&](auto q) {
                    return cudaFuncSetAttribute(q, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
                });
                if (e2 != cudaSuccess) return e2;
            }
        }
    return resident_kernel<C, PHYS>(cpst, energy, p.cs, [&](auto k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
    });
}

// (a.dump set: elastic, plain update, no energies)
template <class C, int PHYS>
cudaError_t launch_resident(const ResArgs<C> &a, int cpst, bool energy, const ResPlan &p, cudaStream_t st)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.ntx * p.nty);
    cfg.blockDim = dim3(RES_THREADS);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];   // CTAs poll their neighbours' words: all must be resident
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = p.ntx * p.nty > 1 ? 1 : 0;
    if constexpr (PHYS == RES_ELASTIC)
        if (a.dump[0]) {
            const auto k = p.cs ? k_resident<C, 0, false, true, PHYS, true> : k_resident<C, 0, false, false, PHYS, true>;
            return cudaLaunchKernelEx(&cfg, k, a);
        }
    return resident_kernel<C, PHYS>(cpst, energy, p.cs, [&](auto k) { return cudaLaunchKernelEx(&cfg, k, a); });
}

// the shots of a group (acoustic, the single-core tree's codes): f with the kernel's pointer
template <class C, int PHYS, class F>
cudaError_t resident_shots_kernel(int cpst, bool cs, F f)
{
    if (cpst == 0) return cs ? f(k_resident_shots<C, 0, true, PHYS>) : f(k_resident_shots<C, 0, false, PHYS>);
    if (cpst == 4) return f(k_resident_shots<C, 4, true, PHYS>);
    return f(k_resident_shots<C, 6, true, PHYS>);
}
template <class C, int PHYS>
cudaError_t prepare_resident_shots(int cpst, bool cs, int smem_max)
{
    return resident_shots_kernel<C, PHYS>(cpst, cs, [&](auto k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
    });
}
template <class C, int PHYS>
cudaError_t launch_resident_shots(const ResArgs<C> *shots, const int *first, int n, int ctas, size_t smem, int cpst, bool cs,
                                  cudaStream_t st)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(RES_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return resident_shots_kernel<C, PHYS>(cpst, cs, [&](auto k) { return cudaLaunchKernelEx(&cfg, k, shots, first, n); });
}

}  // namespace tw
