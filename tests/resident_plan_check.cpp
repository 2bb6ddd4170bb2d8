// Checks fomo::resident_plan and the exchange's index arithmetic on the host:
// prints one line per grid that breaks a rule, and the counts of layouts seen.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "../fomo_julia_b200/csrc/resident_launch.h"

using namespace fomo;

static int bad = 0;
static void rule(bool ok, const char* what, int nx, int nz, int M, int b, int fs) {
    if (ok) return;
    ++bad;
    if (bad < 40) std::printf("BAD %s: grid %dx%d M=%d nbc=%d fs=%d\n", what, nx, nz, M, b, fs);
}

template <int M>
static void exchange(const ResidentLayout& L, int nx, int nz, int b, int fs) {
    const int box = resident_mail_items(M, L.h_max) / 2;
    for (int r = 0; r < L.rows; ++r)
        for (int s = 0; s < L.strips; ++s) {
            const int h = L.z_edge[r + 1] - L.z_edge[r], w = L.x_edge[s + 1] - L.x_edge[s];
            std::set<int> cells;
            for (int idx = 0; idx < 2 * M * h + 2 * M * kRW; ++idx) {
                const MailItem m = resident_mail_item<M>(h, w, L.h_max, idx);
                if (m.col >= w) continue;
                const int s2 = s + (m.dir == 1) - (m.dir == 0), r2 = r + (m.dir == 3) - (m.dir == 2);
                if (s2 < 0 || s2 >= L.strips || r2 < 0 || r2 >= L.rows) continue;
                rule(m.slot >= 0 && m.slot < box, "slot in the mailbox", nx, nz, M, b, fs);
                rule(m.col >= 0 && m.row >= 0 && m.row < h, "border cell in the region", nx, nz, M, b, fs);
                const int hc = m.halo_col(M), hr = m.halo_row(M);
                rule(hc >= -resident_hx(M) && hc < kRW + resident_hx(M) && hr >= -M && hr < h + M, "halo cell in the plane", nx, nz, M, b, fs);
                rule(cells.insert(hr * 4096 + hc).second, "one message per halo cell", nx, nz, M, b, fs);
                // the neighbour's item with the same grid cell lands in the slot we read the halo cell from
                const int h2 = L.z_edge[r2 + 1] - L.z_edge[r2], w2 = L.x_edge[s2 + 1] - L.x_edge[s2];
                bool found = false;
                for (int back = m.dir < 2 ? (1 - m.dir) * M * h2 : 2 * M * h2 + (3 - m.dir) * M * kRW, n = 0; n < (m.dir < 2 ? M * h2 : M * kRW); ++n) {
                    const MailItem o = resident_mail_item<M>(h2, w2, L.h_max, back + n);
                    if (o.col >= w2 || o.peer_slot(M, L.h_max) != m.slot) continue;
                    found = L.x_edge[s2] + o.col == L.x_edge[s] + hc && L.z_edge[r2] + o.row == L.z_edge[r] + hr && o.dir == (m.dir ^ 1);
                }
                rule(found, "sender and receiver agree", nx, nz, M, b, fs);
            }
        }
}

int main() {
    int seen = 0, fit = 0;
    unsigned rng = 12345;
    auto rnd = [&](int lo, int hi) { rng = rng * 1664525u + 1013904223u; return lo + (int)((rng >> 8) % (unsigned)(hi - lo + 1)); };
    for (int n = 0; n < 60000; ++n) {
        const int M = rnd(1, 6), b = rnd(1, 64), fs = rnd(0, 3) > 0, iso = rnd(0, 1);
        const int pad = b + M, span = 1 << rnd(4, 11);
        const int nx = 2 * pad + rnd(2, span), nz = 2 * pad + rnd(2, span);
        if (nx < 2 * b + 3 || nz < 2 * b + 2) continue;
        const int slots = rnd(0, 1) ? 148 : rnd(1, 148);
        ++seen;
        const ResidentPlan p = resident_plan(nx, nz, M, b, fs, iso, slots);
        if (!p.ok) continue;
        ++fit;
        const ResidentLayout& L = p.L;
        rule(L.strips * L.rows <= slots, "blocks within the slots", nx, nz, M, b, fs);
        rule(L.x_edge[0] == 0 && L.x_edge[L.strips] == nx && L.z_edge[0] == 0 && L.z_edge[L.rows] == nz, "cover", nx, nz, M, b, fs);
        for (int s = 0; s < L.strips; ++s) {
            const int w = L.x_edge[s + 1] - L.x_edge[s];
            rule(w <= kRW && (L.strips == 1 || w >= M) && L.x_edge[s] % 4 == 0, "strip width", nx, nz, M, b, fs);
        }
        for (int r = 0; r < L.rows; ++r) {
            const int h = L.z_edge[r + 1] - L.z_edge[r];
            rule((L.rows == 1 || h >= M) && h <= L.h_max, "region height", nx, nz, M, b, fs);
            const size_t need = sizeof(float) * resident_smem_floats(M, b, h, r == L.rows - 1, r == 0 && !fs, false, iso);
            rule(need <= p.smem && p.smem == sizeof(float) * (size_t)L.smem_floats && p.smem <= 227 * 1024 - 256, "shared memory", nx, nz, M, b, fs);
        }
        rule(nx - 2 * b - 1 >= 4, "no four columns of both side bands", nx, nz, M, b, fs);
        rule(resident_plane(M, L.h_max) < 65536, "plane offsets in 16 bits", nx, nz, M, b, fs);
        rule(L.x_edge[1] >= b + 2, "left band and the column after it in the first strip", nx, nz, M, b, fs);
        rule(L.x_edge[L.strips - 1] <= nx - b - 2, "right band and the column before it in the last strip", nx, nz, M, b, fs);
        rule(L.z_edge[L.rows - 1] <= nz - b - 2, "bottom band and the row above it in the last row", nx, nz, M, b, fs);
        if (!fs) rule(L.z_edge[1] >= b + 2, "top band and the row below it in the first row", nx, nz, M, b, fs);
        if (n % 200 == 0) switch (M) {
            case 1: exchange<1>(L, nx, nz, b, fs); break;
            case 2: exchange<2>(L, nx, nz, b, fs); break;
            case 3: exchange<3>(L, nx, nz, b, fs); break;
            case 4: exchange<4>(L, nx, nz, b, fs); break;
            case 5: exchange<5>(L, nx, nz, b, fs); break;
            case 6: exchange<6>(L, nx, nz, b, fs); break;
        }
    }
    std::printf("%d grids, %d resident, %d broken rules\n", seen, fit, bad);
    return bad || fit < 1000;
}
