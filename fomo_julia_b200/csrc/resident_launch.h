// resident_launch.h -- host side of the resident kernel (step_resident.cuh):
// the layout of a grid over the blocks, and the launch entry points of the
// per-order translation units (resident_m<M>.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <vector>

namespace fomo {

struct StepParams;

constexpr int kRW = 64;           // most columns of a block's region (16 lanes x 4)
constexpr int kRThreads = 512;
constexpr int kRMaxEdges = 160;   // strips + 1, rows of blocks + 1
constexpr int kRMaxSteps = 256;   // time steps of one launch
constexpr int kRRecCap = 512;     // receivers a block keeps listed in shared memory
constexpr int kErrResidentTimeout = 4;
constexpr int kRRowsOne = 64;     // regions up to this many rows: one row per thread and pass, taller ones two

// Layout of one grid: block (strip, row) owns columns [x_edge[strip],
// x_edge[strip+1]) and rows [z_edge[row], z_edge[row+1]).
struct ResidentLayout {
    int strips, rows;
    int h_max;        // tallest region (sizes the mailboxes)
    int smem_floats;  // shared memory of a block: one whose region leaves room keeps its medium there too
    short x_edge[kRMaxEdges], z_edge[kRMaxEdges];
};

// Launch-wide parameters besides StepParams.
struct ResidentArgs {
    ResidentLayout L;
    const float* b[4];   // buoyancy dtx/rho_vx, dtz/rho_vx, dtx/rho_vz, dtz/rho_vz
    int iso;
    int* status;
    ulonglong2* mail;    // mailboxes of the launch's blocks (resident_mail_items each)
    uint32_t tag0;       // step s of the launch (0-based) marks its messages tag0 + s
    int n_steps, k0;     // steps to run; 1-based number of the first
    float wav[kRMaxSteps];  // source samples of the steps
};

// x halo of a region, as Geo<M>::HX.
__host__ __device__ constexpr int resident_hx(int M) { return 4 * ((M + 3) / 4); }
__host__ __device__ constexpr int resident_pitch(int M) { return kRW + 2 * resident_hx(M); }

// 16-byte messages of one block's mailbox: two kinds (v, tau) of two sides
// (M columns x h_max rows) and two row neighbours (M rows x kRW columns).
__host__ __device__ constexpr int resident_mail_items(int M, int h_max) { return 2 * (2 * M * h_max + 2 * M * kRW); }

// Shared-memory floats of a region of h rows: five field planes, the bottom
// band's scratch (step-start values of its b rows and the row above; x terms of
// the corners), the top
// band's (no free surface: values before the band rule of rows 0..b+1, one
// row of step-start values; results), the medium where it fits, the receiver
// list, the exchange's table, the weight tables and a few words.
__host__ __device__ constexpr size_t resident_plane(int M, int h) { return (size_t)(h + 2 * M + 1) * resident_pitch(M); }
__host__ __device__ constexpr size_t resident_bottom_floats(int b) { return (size_t)3 * (2 * b + 1) * kRW; }
__host__ __device__ constexpr size_t resident_top_floats(int b) { return (size_t)3 * (2 * b + 3) * kRW; }
__host__ __device__ constexpr size_t resident_tail_floats(int b) { return (size_t)3 * kRW + 3 * (b + 2) + 2 * kRRecCap + 16; }
__host__ __device__ constexpr size_t resident_table_floats(int M, int h) { return 2 * (size_t)(2 * M * h + 2 * M * kRW); }
__host__ __device__ constexpr size_t resident_med_floats(int h, bool iso) { return (size_t)(iso ? 5 : 7) * h * kRW; }
__host__ __device__ constexpr size_t resident_smem_floats(int M, int b, int h, bool bottom, bool top, bool med, bool iso) {
    return 5 * resident_plane(M, h) + (bottom ? resident_bottom_floats(b) : 0) + (top ? resident_top_floats(b) : 0) +
           (med ? resident_med_floats(h, iso) : 0) + resident_table_floats(M, h) + resident_tail_floats(b);
}

// Item `idx` of the messages a region of h rows and w columns exchanges
// (idx < 2 M h + 2 M kRW; columns past w have none): direction 0 left, 1
// right, 2 up, 3 down, its slot among a mailbox's messages of one kind when
// it comes from that direction, and the region's border cell it carries when
// it goes there.
struct MailItem {
    int dir, slot, col, row;
    // the slot it lands in at the neighbour, which receives it from the opposite direction
    __host__ __device__ int peer_slot(int M, int h_max) const {
        return slot + (dir < 2 ? (1 - 2 * dir) * M * h_max : (5 - 2 * dir) * M * kRW);
    }
    // the halo cell that a message received from the direction fills
    __host__ __device__ int halo_col(int M) const { return dir == 0 ? col - M : dir == 1 ? col + M : col; }
    __host__ __device__ int halo_row(int M) const { return dir == 2 ? row - M : dir == 3 ? row + M : row; }
};
template <int M>
__host__ __device__ inline MailItem resident_mail_item(int h, int w, int h_max, int idx) {
    MailItem m;
    const int side = M * h;
    if (idx < 2 * side) {
        m.dir = idx >= side;
        const int r = idx - m.dir * side;
        m.row = r / M;
        const int c = r - m.row * M;
        m.slot = m.dir * M * h_max + r;
        m.col = m.dir ? w - M + c : c;
    } else {
        const int v = idx - 2 * side, d = v >= M * kRW;
        m.dir = 2 + d;
        const int r = v - d * M * kRW, k = r / kRW;
        m.col = r & (kRW - 1);
        m.slot = 2 * M * h_max + v;
        m.row = d ? h - M + k : k;
    }
    return m;
}

// Layout of a grid over at most `slots` resident blocks, !ok if its fields do
// not fit their shared memory or a boundary rule would cross blocks.
struct ResidentPlan {
    bool ok = false;
    size_t smem = 0;
    ResidentLayout L;
};

constexpr size_t kSmemLimit = 227 * 1024 - 256;  // dynamic shared memory of a block, less the kernel's static words

inline ResidentPlan resident_plan(int nx, int nz, int M, int nbc, bool fs, bool iso, int slots) {
    ResidentPlan p;
    std::memset(&p.L, 0, sizeof(p.L));
    // Columns, in groups of 4: an even split into strips of at most kRW, the
    // first and last wide enough for the side band and the columns it reads.
    const int G = (nx + 3) / 4, per = kRW / 4, S = (G + per - 1) / per;
    if (S > slots || S >= kRMaxEdges) return p;
    if (nx - 2 * nbc - 1 < 4) return p;  // a thread's four columns hold one band's at most
    std::vector<int> g(S);
    for (int s = 0; s < S; ++s) g[s] = (int)((long)G * (s + 1) / S - (long)G * s / S);
    if (S > 1) {
        const int need_l = (nbc + 2 + 3) / 4, need_r = (nbc + 2 + 4 * G - nx + 3) / 4;
        g[0] = std::max(g[0], need_l);
        g[S - 1] = std::max(g[S - 1], need_r);
        const int rest = G - g[0] - g[S - 1], n = S - 2;
        if (g[0] > per || g[S - 1] > per || rest < n * ((M + 3) / 4) || (n == 0 && rest < 0)) return p;
        if (n == 0) g[0] += rest;
        for (int s = 0; s < n; ++s) g[1 + s] = (int)((long)rest * (s + 1) / n - (long)rest * s / n);
        if (g[0] > per) return p;
    }
    for (int s = 0, x = 0; s < S; ++s) {
        x += 4 * g[s];
        p.L.x_edge[s + 1] = (short)std::min(x, nx);
    }
    p.L.strips = S;
    // Rows: as many blocks as there are slots, none under h_min rows; the
    // bottom block holds the bottom band (its recurrence costs about as much
    // as nbc/2 rows) and the row above it, the top block the top band and the
    // row below it when there is no free surface.
    auto fits = [&](int h, bool bottom, bool top, bool med) {
        return resident_smem_floats(M, nbc, h, bottom, top, med, iso) * sizeof(float) <= kSmemLimit;
    };
    const int h_min = std::max(M, 8), band = std::max(nbc + 2, M);
    for (int C = std::min(slots / S, kRMaxEdges - 1); C >= 1; --C) {
        std::vector<int> h(C);
        if (C == 1) {
            h[0] = nz;
        } else {
            const int even = (nz + C - 1) / C;
            int hb = std::max(band, even - nbc / 2), ht = fs ? 0 : std::max(band, even - nbc / 2);
            while (hb > band && !fits(hb, true, false, false)) --hb;
            while (ht > band && !fits(ht, false, true, false)) --ht;
            const int n = C - 1 - (fs ? 0 : 1);
            if (n == 0) hb = nz - ht;
            const int rest = nz - hb - ht;
            if (hb < band || rest < n * h_min) continue;
            h[C - 1] = hb;
            if (!fs) h[0] = ht;
            for (int c = 0; c < n; ++c) h[c + (fs ? 0 : 1)] = (int)((long)rest * (c + 1) / n - (long)rest * c / n);
        }
        p.L.rows = C;
        for (int c = 0; c < C; ++c) {
            const bool bottom = c == C - 1, top = c == 0 && !fs;
            if (!fits(h[c], bottom, top, false)) return p;
            p.L.z_edge[c + 1] = (short)(p.L.z_edge[c] + h[c]);
            p.L.h_max = std::max(p.L.h_max, h[c]);
            p.L.smem_floats = std::max(p.L.smem_floats, (int)resident_smem_floats(M, nbc, h[c], bottom, top,
                                                                                  fits(h[c], bottom, top, true), iso));
        }
        p.smem = sizeof(float) * (size_t)p.L.smem_floats;
        p.ok = true;
        return p;
    }
    return p;
}

// Launches the resident kernel cooperatively: strips x rows blocks of
// kRThreads threads.
template <int M>
cudaError_t resident_launch(int blocks, size_t smem, cudaStream_t st, const StepParams& P, const ResidentArgs& A);
template <int M>
const void* resident_kernel_fn(int h_max);

#define FOMO_RESIDENT_DECLARE(M)                                                                                    \
    template <>                                                                                                     \
    cudaError_t resident_launch<M>(int, size_t, cudaStream_t, const StepParams&, const ResidentArgs&);              \
    template <>                                                                                                     \
    const void* resident_kernel_fn<M>(int);
FOMO_RESIDENT_DECLARE(1)
FOMO_RESIDENT_DECLARE(2)
FOMO_RESIDENT_DECLARE(3)
FOMO_RESIDENT_DECLARE(4)
FOMO_RESIDENT_DECLARE(5)
FOMO_RESIDENT_DECLARE(6)
#undef FOMO_RESIDENT_DECLARE

}  // namespace fomo
