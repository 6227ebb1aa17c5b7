// On-chip runs of the elastic step (resident.cuh) for FP32 fields, and the tiling of both types.
#include <algorithm>
#include <array>
#include <cstdlib>
#include <map>
#include <vector>

#include "resident.cuh"

namespace tw {
template cudaError_t prepare_resident<float, RES_ELASTIC>(int, bool, const ResPlan &, int);
template cudaError_t launch_resident<float, RES_ELASTIC>(const ResArgs<float> &, int, bool, const ResPlan &, cudaStream_t);

// f(plan, modelled step) for every tiling of a grid over at most n_sm SMs with smem_max bytes each
template <class F>
static void each_tiling(long Mx, long My, int esize, int fields, bool comp, int n_sm, size_t smem_max, F f)
{
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
            ResPlan p;
            p.ntx = ntx;
            p.nty = nty;
            p.rows_s = R + 1 + 2 * RES_PAD;
            const size_t one = (size_t)p.rows_s * RES_P * esize, alt = (size_t)2 * p.rows_s * esize;
            const size_t base = one * (fields + (comp ? fields : 0)) + alt;
            p.cs = base + fields * one <= smem_max;
            if (!p.cs && (comp || base > smem_max)) continue;
            p.smem = base + (p.cs ? fields * one : 0);
            // modelled cost in rounds of about 0.5 us (within 10 % of the best of a sweep of tilings at 48 x 40
            // to 1024 x 1024): rounds of the CTA's rows in the two phases (short tiles split a phase's two kinds of
            // point over the CTA's halves), the exchange about a round and a half
            const int slots = RES_THREADS * N / RES_LANES_COLS;
            auto rounds = [&](int rows) { return rows <= slots / 2 ? 0.7 : (rows <= slots ? 1.0 : 0.75 * ((rows + 1) / 2 + slots - 1) / slots * 2); };
            const double rv = rounds(R + 4), rs = rounds(R + 1);
            f(p, 0.3 + rv + 1.2 * rs + (ntx * nty > 1 ? 1.5 + (6.0 * R + 6.0 * wmax) / RES_THREADS / 4 : 0.0) + (p.cs ? 0.0 : 0.2 * (rv + rs)) + 1e-4 * ntx * nty);
        }
}

ResPlan resident_plan(long Mx, long My, int esize, int fields, bool comp, int n_sm, size_t smem_max)
{
    ResPlan best;
    double best_step = 1e30;
    each_tiling(Mx, My, esize, fields, comp, n_sm, smem_max, [&](const ResPlan &p, double step) {
        if (step >= best_step) return;
        best_step = step;
        best = p;
    });
    return best;
}

// the tilings of one shot from the fewest CTAs to the shortest step, each faster than the ones with fewer CTAs
struct Tiling {
    ResPlan p;
    double step;
};
static std::vector<Tiling> frontier(long Mx, long My, int esize, int fields, bool comp, int n_sm, size_t smem_max)
{
    std::vector<Tiling> by(n_sm + 1, Tiling{ResPlan{}, 1e30});
    each_tiling(Mx, My, esize, fields, comp, n_sm, smem_max, [&](const ResPlan &p, double step) {
        if (step < by[p.ntx * p.nty].step) by[p.ntx * p.nty] = {p, step};
    });
    std::vector<Tiling> out;
    for (const Tiling &t : by)
        if (t.p.ntx > 0 && (out.empty() || t.step < out.back().step)) out.push_back(t);
    return out;
}

// (us a step of FP32 periodic shots, each with the tiling of least SM time and the SMs left over idle -> here, and
// the same shots stepped one after another: 1 x 256^2 5.8 -> 2.2 (2.0), 3 x 256^2 6.2 -> 2.9 (5.5), 8 x 128^2 6.9 ->
// 3.6 (15.3), 2 x 512^2 6.0 -> 4.0 (4.7), 4 x 512^2 11.9 -> 9.4 (9.2), 8 x 512^2 18.4 / 18.8 (18.5), 24 x 512^2 50.5 / 50.2
// (55.5), 4 x 1000^2 22.9 / 23.2 (19.4))
ResShots resident_shots_plan(const std::vector<std::array<long, 2>> &grids, int esize, int fields, bool comp, int n_sm, size_t smem_max)
{
    const int n = (int)grids.size();
    std::map<std::array<long, 2>, std::vector<Tiling>> known;
    std::vector<const std::vector<Tiling> *> shot(n);
    std::vector<double> steps;   // a group's step is its slowest shot's: the steps to try
    for (int k = 0; k < n; k++) {
        auto it = known.find(grids[k]);
        if (it == known.end()) {
            it = known.emplace(grids[k], frontier(grids[k][0], grids[k][1], esize, fields, comp, n_sm, smem_max)).first;
            for (const Tiling &t : it->second) steps.push_back(t.step);
        }
        if (it->second.empty()) return {};
        shot[k] = &it->second;
    }
    std::sort(steps.begin(), steps.end());
    steps.erase(std::unique(steps.begin(), steps.end()), steps.end());
    constexpr size_t TRIES = 64;
    auto ctas = [](const Tiling &t) { return t.p.ntx * t.p.nty; };
    struct Group {
        std::vector<int> shots;
        int ctas;
        bool cs;
    };
    ResShots best;
    double best_cost = 1e30;
    std::vector<int> use(n), by(n);   // the tiling of each shot; shots by CTAs
    for (size_t i = 0; i < std::min(steps.size(), TRIES); i++) {
        const double target = steps.size() <= TRIES ? steps[i] : steps[i * (steps.size() - 1) / (TRIES - 1)];
        // every shot with the fewest CTAs that reach the target (or its fastest tiling), the largest first,
        // each into the first group with room
        for (int k = 0; k < n; k++) {
            int &u = use[k];
            for (u = 0; u + 1 < (int)shot[k]->size() && (*shot[k])[u].step > target;) u++;
            by[k] = k;
        }
        std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return ctas((*shot[x])[use[x]]) > ctas((*shot[y])[use[y]]); });
        std::vector<Group> groups;
        for (int k : by) {
            const Tiling &t = (*shot[k])[use[k]];
            size_t g = 0;
            while (g < groups.size() && (groups[g].ctas + ctas(t) > n_sm || groups[g].cs != t.p.cs)) g++;
            if (g == groups.size()) groups.push_back(Group{{}, 0, t.p.cs});
            groups[g].shots.push_back(k);
            groups[g].ctas += ctas(t);
        }
        // the SMs a group leaves go to its slowest shot, as long as they make that faster
        double cost = 0.;
        for (Group &g : groups) {
            for (;;) {
                int slow = g.shots[0];
                for (int k : g.shots)
                    if ((*shot[k])[use[k]].step > (*shot[slow])[use[slow]].step) slow = k;
                const std::vector<Tiling> &f = *shot[slow];
                int v = use[slow] + 1;
                while (v < (int)f.size() && f[v].p.cs != g.cs) v++;
                if (v == (int)f.size() || g.ctas + ctas(f[v]) - ctas(f[use[slow]]) > n_sm) {
                    cost += f[use[slow]].step + 1.;   // (a group's launch and its tiles' loads: some 25 us a call)
                    break;
                }
                g.ctas += ctas(f[v]) - ctas(f[use[slow]]);
                use[slow] = v;
            }
        }
        if (cost >= best_cost) continue;
        best_cost = cost;
        best.groups.clear();
        best.plans.resize(n);
        for (const Group &g : groups) best.groups.push_back(g.shots);
        for (int k = 0; k < n; k++) best.plans[k] = (*shot[k])[use[k]].p;
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
