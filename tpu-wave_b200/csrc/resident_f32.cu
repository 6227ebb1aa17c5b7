// On-chip runs of the elastic step (resident.cuh) for FP32 fields, and the tiling of both types.
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<float, RES_ELASTIC>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_ELASTIC>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);

ResPlan resident_plan(long Mx, long My, int esize, int fields, bool comp, int n_sm, size_t smem_max, bool shared)
{
    ResPlan best;
    double best_cost = 1e30;
    const int N = 16 / esize, nq4 = (int)((My + 4) / 4);
    auto pin = [](const char *name) { const char *v = std::getenv(name); return v ? std::atoi(v) : 0; };
    const int pin_x = pin("TW_RES_NTX"), pin_y = pin("TW_RES_NTY");
    std::vector<int> widest(n_sm + 1, 0);   // by nty: most columns of a tile (the last one with column My), 0: too few
    for (int nty = 1; nty <= n_sm; nty++) {
        int wmin = 1 << 30;
        for (int t = 0; t < nty; t++) {
            const int b = 4 * (int)((long)t * nq4 / nty);
            const int e = t == nty - 1 ? (int)My : 4 * (int)((long)(t + 1) * nq4 / nty);
            wmin = std::min(wmin, e - b);
            widest[nty] = std::max(widest[nty], e - b + (t == nty - 1 ? 1 : 0));
        }
        if (wmin >= RES_MIN) continue;
        widest[nty] = 0;
        break;   // (narrower still from here on)
    }
    for (int ntx = 1; ntx <= n_sm && Mx / ntx >= RES_MIN; ntx++)
        for (int nty = 1; ntx * nty <= n_sm && widest[nty]; nty++) {
            if ((pin_x && ntx != pin_x) || (pin_y && nty != pin_y)) continue;
            const int wmax = widest[nty];
            if (wmax > RES_W) continue;
            const int R = (int)((Mx + ntx - 1) / ntx);
            // halo words (k_resident: XI), the elastic grids' seam columns among them
            if (6 * (wmax + 6) + (fields == 3 ? 6 : (nty > 1 ? 7 : 8)) * (R + 1) + 8 > 3 * RES_THREADS) continue;
            const int rows_s = R + 1 + 2 * RES_PAD;
            const size_t one = (size_t)rows_s * RES_P * esize, alt = (size_t)2 * rows_s * esize;
            const size_t base = one * (fields + (comp ? fields : 0)) + alt;
            bool cs = base + fields * one <= smem_max;
            if (!cs && (comp || base > smem_max)) continue;
            // modelled cost in rounds of about 0.5 us (within 10 % of the best of a sweep of tilings at 48 x 40
            // to 1024 x 1024): rounds of the CTA's rows in the two phases (short tiles split a phase's two kinds of
            // point over the CTA's halves), the exchange about a round and a half
            const int slots = RES_THREADS * N / RES_LANES_COLS;
            auto rounds = [&](int rows) { return rows <= slots / 2 ? 0.7 : (rows <= slots ? 1.0 : 0.75 * ((rows + 1) / 2 + slots - 1) / slots * 2); };
            const double rv = rounds(R + 4), rs = rounds(R + 1);
            const double step = 0.3 + rv + 1.2 * rs + (ntx * nty > 1 ? 1.5 + (6.0 * R + 6.0 * wmax) / RES_THREADS / 4 : 0.0) + (cs ? 0.0 : 0.2 * (rv + rs)) + 1e-4 * ntx * nty;
            const double cost = shared ? step * ntx * nty : step;
            if (cost < best_cost) {
                best_cost = cost;
                best.ntx = ntx;
                best.nty = nty;
                best.rows_s = rows_s;
                best.cs = cs;
                best.smem = base + (cs ? fields * one : 0);
            }
        }
    return best;
}

int resident_tile(const ResPlan &p, long Mx, long My, int row, int col)
{
    const int nq4 = (int)((My + 4) / 4);
    int tx = 0, ty = 0;
    while (tx + 1 < p.ntx && (long)(tx + 1) * Mx / p.ntx <= row) tx++;
    while (ty + 1 < p.nty && 4 * (int)((long)(ty + 1) * nq4 / p.nty) <= col) ty++;
    return tx * p.nty + ty;
}

template <class C>
__global__ void k_pad_columns(const C *in, long pitch, C *out, long xpitch, int rows, int My, int n_type)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (c >= My + 13) return;
    int g = c - 4;
    if (g < 0) g += My;
    else if (n_type ? g > My : g >= My) g -= My;
    out[(long)r * xpitch + c] = in[(long)r * pitch + g];
}

template <class C>
void launch_pad_columns(const C *in, long pitch, C *out, long xpitch, int rows, int My, int n_type, cudaStream_t st)
{
    k_pad_columns<C><<<dim3((My + 13 + 255) / 256, rows), 256, 0, st>>>(in, pitch, out, xpitch, rows, My, n_type);
}
template void launch_pad_columns<float>(const float *, long, float *, long, int, int, int, cudaStream_t);
template void launch_pad_columns<double>(const double *, long, double *, long, int, int, int, cudaStream_t);
}  // namespace tw
