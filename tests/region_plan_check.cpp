// Checks psdm::plan_regions and psdm::region_loads on the CPU (see
// tests/test_region_plan.py).  Prints: fits, regions, live cells not covered
// exactly once, ring cells that a packet exchange leaves wrong, regions over
// the shared-memory limit, injection or receiver entries that name another
// cell, packets received more than once.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "rtm_internal.h"

using namespace psdm;

int main(int argc, char** argv) {
    const int ny = atoi(argv[1]), nx = atoi(argv[2]), dPML = atoi(argv[3]), fs = atoi(argv[4]),
              max_regions = atoi(argv[5]);
    const size_t max_floats = (size_t)atol(argv[6]);
    const Grid g = make_grid(dPML, ny, nx);
    RegPlan plan;
    if (!plan_regions(g, fs, max_regions, max_floats, &plan)) {
        printf("0\n");
        return 0;
    }
    const int n = (int)plan.blocks.size();
    auto id = [&](int z, int x) { return 1.0 + (double)x * g.ldz + z; };
    std::vector<int> cover((size_t)g.nxt * g.ldz, 0), owner((size_t)g.nxt * g.ldz, -1);
    std::vector<std::vector<double>> lv(n), phi(n);
    int over = 0;
    for (int b = 0; b < n; ++b) {
        const RegBlock& r = plan.blocks[b];
        lv[b].assign((size_t)r.P * (r.ns + 6), 0.0);
        if (r.type == kRegCorner) {  // phi with its slow ring
            phi[b].assign((size_t)r.Q * (r.ns + 6), 0.0);
            for (int s = 0; s < r.ns; ++s)
                for (int f = 0; f < r.nf; ++f) phi[b][(size_t)(s + 3) * r.Q + f] = id(r.z0 + f, r.x0 + s);
        }
        for (int s = 0; s < r.ns; ++s)
            for (int f = 0; f < r.nf; ++f) {
                const int z = r.z0 + (r.fastx ? s : f), x = r.x0 + (r.fastx ? f : s);
                ++cover[(size_t)x * g.ldz + z];
                owner[(size_t)x * g.ldz + z] = b;
                lv[b][(size_t)(s + 3) * r.P + f + 4] = id(z, x);
            }
        const size_t per = (size_t)2 * r.P * (r.ns + 6) +
                           (size_t)r.Q * r.ns * (r.type == kRegInterior ? 1 : r.type == kRegStrip ? 4 : 7);
        over += per > max_floats || plan.floats > max_floats;
        over += r.nq > kRegMaxQuads || r.nf < 3 || r.ns < 3;
    }
    long wrong_cover = 0;
    for (int x = 0; x < g.nxt; ++x)
        for (int z = 0; z < g.ldz; ++z) {
            const int lz = z - g.zoff;
            const bool live = lz >= (fs ? g.dn : 0) && lz < g.nyt;
            wrong_cover += cover[(size_t)x * g.ldz + z] != (live ? 1 : 0);
        }
    // one exchange
    std::vector<double> board((size_t)plan.npk * 3, -1.0);
    std::vector<int> written(plan.npk, 0), read(plan.npk, 0);
    for (int b = 0; b < n; ++b) {
        const RegBlock& r = plan.blocks[b];
        for (int k = 0; k < r.npub; ++k) {
            const RegPair d = plan.pub[r.pub0 + k];
            const int off = d.y & kRegOffMask, st = (d.y & kRegPhi) ? r.Q : (d.y & kRegSlow) ? r.P : 1;
            for (int c = 0; c < 3; ++c) board[(size_t)d.x * 3 + c] = ((d.y & kRegPhi) ? phi : lv)[b].at(off + c * st);
            ++written[d.x];
        }
    }
    for (int b = 0; b < n; ++b) {
        const RegBlock& r = plan.blocks[b];
        for (int k = 0; k < r.nrcv; ++k) {
            const int d = plan.rcv[r.rcv0 + k];
            const int off = d & kRegOffMask, st = (d & kRegPhi) ? r.Q : (d & kRegSlow) ? r.P : 1;
            for (int c = 0; c < 3; ++c)
                ((d & kRegPhi) ? phi : lv)[b].at(off + c * st) = board[(size_t)(r.rcv_first + k) * 3 + c];
            ++read[r.rcv_first + k];
        }
    }
    long wrong_ring = 0, twice = 0;
    for (int k = 0; k < plan.npk; ++k) twice += written[k] != 1 || read[k] != 1;
    for (int b = 0; b < n; ++b) {
        const RegBlock& r = plan.blocks[b];
        for (int s = -3; s < r.ns + 3; ++s)
            for (int f = -3; f < r.nf + 3; ++f) {
                const bool inf = f >= 0 && f < r.nf, ins = s >= 0 && s < r.ns;
                if (!inf && !ins) continue;  // diagonal cells are in no stencil
                const int z = r.z0 + (r.fastx ? s : f), x = r.x0 + (r.fastx ? f : s);
                double want = 0.0;
                if (z >= 0 && z < g.ldz && x >= 0 && x < g.nxt && owner[(size_t)x * g.ldz + z] >= 0) want = id(z, x);
                wrong_ring += lv[b][(size_t)(s + 3) * r.P + f + 4] != want;
            }
    }
    // a corner region's phi ring: the columns beside it that lie in the corner
    for (int b = 0; b < n; ++b) {
        const RegBlock& r = plan.blocks[b];
        if (r.type != kRegCorner) continue;
        for (int s = -3; s < r.ns + 3; ++s)
            for (int f = 0; f < r.nf; ++f) {
                const bool in = r.soff + s >= 0 && r.soff + s < g.dn;
                wrong_ring += phi[b][(size_t)(s + 3) * r.Q + f] != (in ? id(r.z0 + f, r.x0 + s) : 0.0);
            }
    }
    // inner cells are updated before the ring arrives: their stencils, clamped at the grid's edge and (phi)
    // at the strip's edges, end inside the region
    auto inside = [](int c, int n) { return c - 3 >= 0 && c + 3 < n; };
    auto clamp = [](int v, int lo, int hi) { return v < lo ? lo : v > hi ? hi : v; };
    for (const RegBlock& r : plan.blocks) {
        const bool corner = r.type == kRegCorner, strip = r.type == kRegStrip;
        const int fa = corner ? r.fa : 4 * r.qa, fb = corner ? r.fb : 4 * r.qb;
        for (int s = r.sa; s < r.sb; ++s)
            for (int f = fa; f < fb; ++f) {
                const int sg = s + (corner ? r.soff : 0);  // within the strip or corner
                const int cs = corner ? (r.low ? std::max(sg, 3) : std::min(sg, g.dn - 4)) - r.soff : s;
                const int cp = strip || corner ? clamp(sg, 3, g.dn - 4) - (corner ? r.soff : 0) : s;
                const int cz = corner ? (r.lowf ? std::max(f, 3) : std::min(f, r.nf - 4)) : f;
                const bool grid_top = !corner && f < 3 && fa == 0, grid_end = !corner && f + 3 >= r.nf && fb >= r.nf;
                over += !inside(cs, r.ns) || !inside(cp, r.ns) || (!grid_top && !grid_end && !inside(cz, r.nf));
            }
    }
    // injection points on two rows (every other column) and receivers anywhere
    std::vector<int> cell, trace, rec;
    for (int x = g.dn; x < g.dn + nx; x += 2)
        for (int z : {0, ny - 1}) {
            cell.push_back(x * g.ldz + z + g.dn + g.zoff);
            trace.push_back((int)trace.size() * 3);
        }
    for (int x = 0; x < g.nxt; x += 3) rec.push_back(x * g.ldz + g.zoff + (x * 7) % g.nyt);
    RegLists L;
    long wrong_list = 0;
    if (region_loads(plan, g, max_floats, (int)cell.size(), cell.data(), trace.data(), (int)rec.size(), rec.data(), &L)) {
        std::map<int, int> want;
        for (size_t j = 0; j < cell.size(); ++j) want[cell[j]] = trace[j];
        size_t ninj = 0, nrec = 0, live = 0;
        for (int c : rec) live += owner[c] >= 0;
        for (int b = 0; b < n; ++b) {
            const RegBlock& r = plan.blocks[b];
            const RegLoad& l = L.loads[b];
            for (int j = 0; j < l.ninj; ++j) {
                const RegPair d = L.inj[l.inj0 + j];
                const int q4 = d.x / 4 / r.ns, s = d.x / 4 % r.ns;
                int q = 0;
                while (q < r.nq && L.slots[l.slot0 + q] != q4) ++q;
                const int c = (r.x0 + s) * g.ldz + r.z0 + 4 * q + d.x % 4;
                wrong_list += q == r.nq || want.count(c) == 0 || want[c] != d.y;
            }
            ninj += l.ninj;
            for (int j = 0; j < l.nrec; ++j) {
                const RegPair d = L.rec[l.rec0 + j];
                const int s = d.y / r.P - 3, f = d.y % r.P - 4;
                const int c = (r.x0 + (r.fastx ? f : s)) * g.ldz + r.z0 + (r.fastx ? s : f);
                wrong_list += rec[d.x] != c;
            }
            nrec += l.nrec;
        }
        wrong_list += ninj != cell.size() || nrec != live;
    }
    printf("1 %d %ld %ld %d %ld %ld\n", n, wrong_cover, wrong_ring, over, wrong_list, twice);
    if (argc > 7)
        for (const RegBlock& r : plan.blocks)
            printf("type %d fastx %d z0 %d x0 %d nf %d ns %d C %d items %d pub %d\n", r.type, r.fastx, r.z0, r.x0, r.nf,
                   r.ns, r.C, r.items, r.npub);
    if (argc > 7) printf("cost %.0f floats %zu npk %d\n", plan.cost, plan.floats, plan.npk);
    return 0;
}
