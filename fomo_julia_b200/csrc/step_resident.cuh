// step_resident.cuh -- many time steps of one shot in one launch, for grids
// whose five fields fit the chip's shared memory.
//
// What bounds small grids is latency, not bytes: a step of the split launches
// is four dependent launches, each of them one or two waves of tiles that
// load, compute and store once.  Here each block owns a region of the grid
// (up to 64 columns, any number of rows) and keeps its five fields, with an
// M-cell halo, in shared memory for all the steps of the launch.  A half step
// reads and writes shared memory only; the blocks then exchange the M border
// columns and rows of the fields the next half step differentiates through
// mailboxes in global memory (L2), and nothing else crosses the chip.  The
// launch is cooperative, since neighbouring blocks wait for each other.
//
// Exchange.  A message is 16 bytes: two values, each in one 64-bit word with
// the step's tag.  The receiver polls the words themselves until they carry
// the tag it waits for, so an exchange costs one store and one load latency
// and needs no fence or flag.  One mailbox per kind (v after the velocity
// half step, tau after the stress half step) is enough: a block writes its
// next message of a kind only after it has received its neighbours' messages
// of the other kind, which they send after reading the previous one.  Waits
// are bounded: a block that gives up sets the status word and leaves, and so
// do its neighbours.
//
// Regions.  The first and last strip hold the side HABC bands and the columns
// their rules read, the bottom row of blocks holds the whole bottom band and
// the row above it, and without a free surface the top row of blocks holds
// the whole top band and the row below, so no boundary rule crosses a block.
//   sides   a thread's neighbours in x are in the same half warp, so the side
//           rules run on registers and shuffles;
//   bottom  the recurrence along j (boundary.jl:88-132) runs in the plane,
//           a column per lane, with the step-start values in a scratch;
//   top     pointwise on values before the band rule, kept in a scratch.
// The source is added in the plane right after a step's stresses are final
// (before they are sent), the values before it are kept beside for the HABC
// and the receivers (source_receiver.jl:18-30, boundary.jl:20-56).
#pragma once

#include "mailbox.cuh"
#include "resident_launch.h"
#include "step_tiled.cuh"

namespace fomo {

// z-derivatives of RT consecutive rows from a (2M + RT - 1)-row window:
// d[rr] = sum_l a_l (w[rr+M+l-1] - w[rr+M-l]), column pairs.
template <int M, int RT>
__device__ __forceinline__ void zpairs(const StepParams& P, const float4 (&w)[2 * M + RT - 1], float2 (&lo)[RT],
                                       float2 (&hi)[RT]) {
#pragma unroll
    for (int rr = 0; rr < RT; ++rr) {
        float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll
        for (int l = 1; l <= M; ++l) {
            const float2 al = make_float2(P.a[l - 1], P.a[l - 1]);
            a = add2(mul2(P, al, sub2(lo2(w[rr + M + l - 1]), lo2(w[rr + M - l]))), a);
            b = add2(mul2(P, al, sub2(hi2(w[rr + M + l - 1]), hi2(w[rr + M - l]))), b);
        }
        lo[rr] = a;
        hi[rr] = b;
    }
}

// Rows j .. j+n-1 hold a row of the side bands (a warp's rows: uniform).
__device__ __forceinline__ bool side_rows(const StepParams& P, int j, int n) {
    return j + n > (P.fs ? P.nbc : 1) && j <= P.nz - P.nbc - 2;
}

// What a block knows of its region.
struct Region {
    int x0, x1, z0, z1, h;
    bool left, right, bottom, top, rim;
    int si, sj;        // source, in region coordinates; sj < 0: not here
    float* plane;      // five planes of `psize` floats, row pitch PITCH, cell (x0, z0) at M rows + HX columns
    size_t psize;
    float *old, *sx;   // bottom band: step-start values [3][b+1][kRW], row 0 the row above the band; x terms [3][b][kRW]
    float *e, *fin;    // top band: [3][b+3][kRW] (row b+2: step-start values of row b+1), [3][b][kRW]
    float* tab;        // weights of vx, vz, tau by distance, b + 2 each
    float* wcol;       // and of the region's columns, kRW each (rows below the top band)
    float* src;        // txx, tzz of the source cell before the source was added
};

template <int M>
__device__ __forceinline__ float* cell_at(const Region& R, int q, int col, int row) {
    return R.plane + q * R.psize + (size_t)(row + M) * resident_pitch(M) + col + resident_hx(M);
}

// Where a row's values go after the side rules.
__device__ __forceinline__ bool in_top_rows(const StepParams& P, int j) { return !P.fs && j >= 1 && j <= P.nbc; }

// Weights of columns x..x+3 of row j from table `t` (0 vx, 1 vz, 2 tau), every
// row above the bottom band: below the top band they depend on the column
// only and come as one 16-byte load.
__device__ __forceinline__ float4 region_weights(const StepParams& P, const Region& R, int t, int x, int j) {
    if (P.fs || j > P.nbc) return lds4(R.wcol + t * kRW + (x - R.x0));
    return side_weights(P, R.tab + t * (P.nbc + 2), x, j);
}

// Four columns of a row of the bottom band (row jb of field f): the values
// before the HABC go to the plane, the step-start values to R.old and, in a
// block at a corner, the x terms of the corner columns to R.sx (side_rules'
// sums; other columns hold whatever comes out).  All lanes of the half warp
// that share the row call it.
__device__ __forceinline__ void put_band_row(const StepParams& P, const Region& R, int f, float* p, int col, int jb,
                                             const float4& n, const float4& o, bool on) {
    constexpr unsigned FULL = 0xffffffffu;
    const int b = P.nbc;
    if (R.left || R.right) {
        const float2 nq = make_float2(-P.qx, -P.qx), qt = make_float2(P.qt_x, P.qt_x), qxt = make_float2(P.qxt, P.qxt);
        const float2 tl = mul2(P, qt, lo2(o)), th = mul2(P, qt, hi2(o));
        float2 nl, nh, ol, oh;  // the neighbours towards the interior: i+1 on the left, i-1 on the right
        const bool l = R.left && R.x0 + col <= b;  // a block on both sides: by group of columns
        const float nu = __shfl_up_sync(FULL, n.w, 1, 16), ou = __shfl_up_sync(FULL, o.w, 1, 16);
        const float nd = __shfl_down_sync(FULL, n.x, 1, 16), od = __shfl_down_sync(FULL, o.x, 1, 16);
        if (l) {
            nl = make_float2(n.y, n.z), nh = make_float2(n.w, nd);
            ol = make_float2(o.y, o.z), oh = make_float2(o.w, od);
        } else {
            nl = make_float2(nu, n.x), nh = make_float2(n.y, n.z);
            ol = make_float2(ou, o.x), oh = make_float2(o.y, o.z);
        }
        const float2 sl = sub2(sub2(mul2(P, nq, nl), tl), mul2(P, qxt, ol));
        const float2 sh = sub2(sub2(mul2(P, nq, nh), th), mul2(P, qxt, oh));
        if (on) *reinterpret_cast<float4*>(R.sx + (f * b + jb) * kRW + col) = make_float4(sl.x, sl.y, sh.x, sh.y);
    }
    if (on) {
        *reinterpret_cast<float4*>(p) = n;
        *reinterpret_cast<float4*>(R.old + (f * (b + 1) + jb + 1) * kRW + col) = o;
    }
}

// Stores four columns of field f (of the half step; plane q) of row j above
// the bottom band: to the plane; rows of the top band to its scratch, their
// plane keeps the step-start values.
template <int M>
__device__ __forceinline__ void put_row(const StepParams& P, const Region& R, int f, int q, int col, int row, const float4& n,
                                        const float4& o, bool zero, bool src_row) {
    const int b = P.nbc, j = R.z0 + row;
    float* p = cell_at<M>(R, q, col, row);
    if (R.top) {
        if (in_top_rows(P, j)) {
            *reinterpret_cast<float4*>(R.e + (f * (b + 3) + j) * kRW + col) = n;
            if (src_row) *reinterpret_cast<float4*>(p) = o;  // the band rule reads step-start values here
            return;
        }
        if (j == b + 1) {
            *reinterpret_cast<float4*>(R.e + (f * (b + 3) + b + 1) * kRW + col) = n;
            *reinterpret_cast<float4*>(R.e + (f * (b + 3) + b + 2) * kRW + col) = o;
        }
    }
    if (R.bottom && j == P.nz - b - 2) *reinterpret_cast<float4*>(R.old + f * (b + 1) * kRW + col) = o;
    *reinterpret_cast<float4*>(p) = zero ? make_float4(0.f, 0.f, 0.f, 0.f) : n;
}

// Whether a warp's rows j .. j+n-1 hold rows of the bottom band.
__device__ __forceinline__ bool band_rows(const StepParams& P, int j, int n) { return j + n > P.nz - P.nbc - 1 && j <= P.nz - 2; }

// Medium of the region: global memory or its copy in shared memory.
struct MedView {
    const float *b0, *b1, *b2, *b3, *lam, *mu, *mxz;  // at the region's first cell
    int pitch;
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Stencil update and side rules of the region's velocities.
template <int M, int RT>
__device__ __forceinline__ void resident_velocity(const StepParams& P, const Region& R, const MedView& D) {
    constexpr int PITCH = resident_pitch(M), HX = resident_hx(M), ROWS = kRThreads / 16 * RT;
    const int col = 4 * (threadIdx.x & 15), x = R.x0 + col;
#pragma unroll 1
    for (int base = 0; base < R.h; base += ROWS) {
        const int row = base + (threadIdx.x >> 4) * RT;
        const bool on = row < R.h && x < R.x1;
        float4 ox[RT], oz[RT], nx[RT], nz[RT];
        if (on) {
            const int mo = row * D.pitch + col;
            float4 b0[RT], b1[RT], b2[RT], b3[RT];
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const int m = mo + (row + rr < R.h ? rr : 0) * D.pitch;
                b0[rr] = ld4(D.b0 + m);
                b2[rr] = ld4(D.b2 + m);
                b1[rr] = D.b1 == D.b0 ? b0[rr] : ld4(D.b1 + m);
                b3[rr] = D.b3 == D.b2 ? b2[rr] : ld4(D.b3 + m);
            }
            const float* xx = cell_at<M>(R, TXX, col, row) - HX;  // windows start HX columns to the left
            const float* zz = cell_at<M>(R, TZZ, col, row);
            const float* xz = cell_at<M>(R, TXZ, col, row);
            float d1[RT][4], d3[RT][4];
            float2 d2lo[RT], d2hi[RT], d4lo[RT], d4hi[RT];
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                float w[4 * Geo<M>::NQ];
                load_xwin<M>(xx + rr * PITCH, w);
                xderiv<M, 0>(P, w, d1[rr]);  // dtxx/dx
                load_xwin<M>(xz - HX + rr * PITCH, w);
                xderiv<M, 1>(P, w, d3[rr]);  // dtxz/dx
            }
            {
                float4 w[2 * M + RT - 1];
#pragma unroll
                for (int k = 0; k < 2 * M + RT - 1; ++k) w[k] = lds4(xz + (k - M) * PITCH);
                zpairs<M, RT>(P, w, d2lo, d2hi);  // dtxz/dz
#pragma unroll
                for (int k = 0; k < 2 * M + RT - 1; ++k) w[k] = lds4(zz + (k - M + 1) * PITCH);
                zpairs<M, RT>(P, w, d4lo, d4hi);  // dtzz/dz
            }
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const float4 vx = lds4(cell_at<M>(R, VX, col, row + rr)), vz = lds4(cell_at<M>(R, VZ, col, row + rr));
                const float2 xl = add2(lo2(vx), add2(mul2(P, lo2(b0[rr]), make_float2(d1[rr][0], d1[rr][1])), mul2(P, lo2(b1[rr]), d2lo[rr])));
                const float2 xh = add2(hi2(vx), add2(mul2(P, hi2(b0[rr]), make_float2(d1[rr][2], d1[rr][3])), mul2(P, hi2(b1[rr]), d2hi[rr])));
                const float2 zl = add2(lo2(vz), add2(mul2(P, lo2(b2[rr]), make_float2(d3[rr][0], d3[rr][1])), mul2(P, lo2(b3[rr]), d4lo[rr])));
                const float2 zh = add2(hi2(vz), add2(mul2(P, hi2(b2[rr]), make_float2(d3[rr][2], d3[rr][3])), mul2(P, hi2(b3[rr]), d4hi[rr])));
                nx[rr] = make_float4(xl.x, xl.y, xh.x, xh.y);
                nz[rr] = make_float4(zl.x, zl.y, zh.x, zh.y);
                ox[rr] = vx;
                oz[rr] = vz;
                if (R.rim) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (!in_stencil(P, x + c, R.z0 + row + rr)) {
                            set_comp(nx[rr], c, comp(vx, c));
                            set_comp(nz[rr], c, comp(vz, c));
                        }
                }
            }
        } else {
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) ox[rr] = oz[rr] = nx[rr] = nz[rr] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if ((R.left || R.right) && side_rows(P, R.z0 + base + (threadIdx.x >> 5) * 2 * RT, 2 * RT)) {
            __syncwarp();
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const int j = R.z0 + row + rr;
                const float4 w[2] = {region_weights(P, R, 0, x, j), region_weights(P, R, 1, x, j)}, o[2] = {ox[rr], oz[rr]};
                float4 n[2] = {nx[rr], nz[rr]};
                side_rules(P, R.left, R.right, w, x, j, n, o);
                nx[rr] = n[0];
                nz[rr] = n[1];
            }
        }
        const bool band = R.bottom && band_rows(P, R.z0 + base + (threadIdx.x >> 5) * 2 * RT, 2 * RT);
#pragma unroll
        for (int rr = 0; rr < RT; ++rr) {
            const int jb = R.z0 + row + rr - (P.nz - P.nbc - 1);
            const bool here = on && row + rr < R.h, in_band = jb >= 0 && jb < P.nbc;
            if (band) {
                const int jc = min(max(jb, 0), P.nbc - 1);
                put_band_row(P, R, 0, cell_at<M>(R, VX, col, row + rr), col, jc, nx[rr], ox[rr], here && in_band);
                put_band_row(P, R, 1, cell_at<M>(R, VZ, col, row + rr), col, jc, nz[rr], oz[rr], here && in_band);
            }
            if (here && !in_band) {
                put_row<M>(P, R, 0, VX, col, row + rr, nx[rr], ox[rr], false, false);
                put_row<M>(P, R, 1, VZ, col, row + rr, nz[rr], oz[rr], false, false);
            }
        }
    }
}

// Stencil update and side rules of the region's stresses.  The planes hold
// the source already; step-start values are those before it.
template <int M, int RT>
__device__ __forceinline__ void resident_stress(const StepParams& P, const Region& R, const MedView& D) {
    constexpr int PITCH = resident_pitch(M), HX = resident_hx(M), ROWS = kRThreads / 16 * RT;
    const int col = 4 * (threadIdx.x & 15), x = R.x0 + col;
    const float2 dtx2 = make_float2(P.dtx, P.dtx), dtz2 = make_float2(P.dtz, P.dtz), two = make_float2(2.f, 2.f);
#pragma unroll 1
    for (int base = 0; base < R.h; base += ROWS) {
        const int row = base + (threadIdx.x >> 4) * RT;
        const bool on = row < R.h && x < R.x1;
        float4 o0[RT], o1[RT], o2[RT], n0[RT], n1[RT], n2[RT];
        if (on) {
            const int mo = row * D.pitch + col;
            float4 lam[RT], mu[RT], mxz[RT];
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const int m = mo + (row + rr < R.h ? rr : 0) * D.pitch;
                lam[rr] = ld4(D.lam + m);
                mu[rr] = ld4(D.mu + m);
                mxz[rr] = ld4(D.mxz + m);
            }
            const float* vx = cell_at<M>(R, VX, col, row);
            const float* vz = cell_at<M>(R, VZ, col, row);
            float dxx[RT][4], dzx[RT][4];
            float2 dzzlo[RT], dzzhi[RT], dxzlo[RT], dxzhi[RT];
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                float w[4 * Geo<M>::NQ];
                load_xwin<M>(vx - HX + rr * PITCH, w);
                xderiv<M, 1>(P, w, dxx[rr]);  // dvx/dx
                load_xwin<M>(vz - HX + rr * PITCH, w);
                xderiv<M, 0>(P, w, dzx[rr]);  // dvz/dx
            }
            {
                float4 w[2 * M + RT - 1];
#pragma unroll
                for (int k = 0; k < 2 * M + RT - 1; ++k) w[k] = lds4(vz + (k - M) * PITCH);
                zpairs<M, RT>(P, w, dzzlo, dzzhi);  // dvz/dz
#pragma unroll
                for (int k = 0; k < 2 * M + RT - 1; ++k) w[k] = lds4(vx + (k - M + 1) * PITCH);
                zpairs<M, RT>(P, w, dxzlo, dxzhi);  // dvx/dz
            }
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const float4 txx = lds4(cell_at<M>(R, TXX, col, row + rr)), tzz = lds4(cell_at<M>(R, TZZ, col, row + rr));
                const float4 txz = lds4(cell_at<M>(R, TXZ, col, row + rr));
                float2 r0[2], r1[2], r2[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 lv = h ? hi2(lam[rr]) : lo2(lam[rr]), mv = h ? hi2(mu[rr]) : lo2(mu[rr]);
                    const float2 l2m = add2(lv, mul2(P, two, mv));
                    const float2 ex = mul2(P, make_float2(dxx[rr][2 * h], dxx[rr][2 * h + 1]), dtx2);
                    const float2 ez = mul2(P, h ? dzzhi[rr] : dzzlo[rr], dtz2);
                    r0[h] = add2(h ? hi2(txx) : lo2(txx), add2(mul2(P, l2m, ex), mul2(P, lv, ez)));
                    r1[h] = add2(h ? hi2(tzz) : lo2(tzz), add2(mul2(P, lv, ex), mul2(P, l2m, ez)));
                    const float2 sh = add2(mul2(P, h ? dxzhi[rr] : dxzlo[rr], dtz2),
                                           mul2(P, make_float2(dzx[rr][2 * h], dzx[rr][2 * h + 1]), dtx2));
                    r2[h] = add2(h ? hi2(txz) : lo2(txz), mul2(P, h ? hi2(mxz[rr]) : lo2(mxz[rr]), sh));
                }
                n0[rr] = make_float4(r0[0].x, r0[0].y, r0[1].x, r0[1].y);
                n1[rr] = make_float4(r1[0].x, r1[0].y, r1[1].x, r1[1].y);
                n2[rr] = make_float4(r2[0].x, r2[0].y, r2[1].x, r2[1].y);
                o0[rr] = txx;
                o1[rr] = tzz;
                o2[rr] = txz;
                if (R.rim) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (!in_stencil(P, x + c, R.z0 + row + rr)) {
                            set_comp(n0[rr], c, comp(txx, c));
                            set_comp(n1[rr], c, comp(tzz, c));
                            set_comp(n2[rr], c, comp(txz, c));
                        }
                }
                if (row + rr == R.sj && R.si >= col && R.si < col + 4) {
                    set_comp(o0[rr], R.si - col, R.src[0]);
                    set_comp(o1[rr], R.si - col, R.src[1]);
                }
            }
        } else {
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                o0[rr] = o1[rr] = o2[rr] = make_float4(0.f, 0.f, 0.f, 0.f);
                n0[rr] = n1[rr] = n2[rr] = o0[rr];
            }
        }
        if ((R.left || R.right) && side_rows(P, R.z0 + base + (threadIdx.x >> 5) * 2 * RT, 2 * RT)) {
            __syncwarp();
#pragma unroll
            for (int rr = 0; rr < RT; ++rr) {
                const int j = R.z0 + row + rr;
                const float4 wt = region_weights(P, R, 2, x, j), w[3] = {wt, wt, wt}, o[3] = {o0[rr], o1[rr], o2[rr]};
                float4 n[3] = {n0[rr], n1[rr], n2[rr]};
                side_rules(P, R.left, R.right, w, x, j, n, o);
                n0[rr] = n[0];
                n1[rr] = n[1];
                n2[rr] = n[2];
            }
        }
        const bool band = R.bottom && band_rows(P, R.z0 + base + (threadIdx.x >> 5) * 2 * RT, 2 * RT);
#pragma unroll
        for (int rr = 0; rr < RT; ++rr) {
            const int jb = R.z0 + row + rr - (P.nz - P.nbc - 1);
            const bool here = on && row + rr < R.h, in_band = jb >= 0 && jb < P.nbc;
            if (band) {
                const int jc = min(max(jb, 0), P.nbc - 1);
                put_band_row(P, R, 0, cell_at<M>(R, TXX, col, row + rr), col, jc, n0[rr], o0[rr], here && in_band);
                put_band_row(P, R, 1, cell_at<M>(R, TZZ, col, row + rr), col, jc, n1[rr], o1[rr], here && in_band);
                put_band_row(P, R, 2, cell_at<M>(R, TXZ, col, row + rr), col, jc, n2[rr], o2[rr], here && in_band);
            }
            if (here && !in_band) {
                const bool zero = in_free_surface_rows(P, R.z0 + row + rr);
                const bool src = row + rr == R.sj && R.si >= col && R.si < col + 4;
                put_row<M>(P, R, 0, TXX, col, row + rr, n0[rr], o0[rr], false, src);
                put_row<M>(P, R, 1, TZZ, col, row + rr, n1[rr], o1[rr], zero, src);
                put_row<M>(P, R, 2, TXZ, col, row + rr, n2[rr], o2[rr], zero, false);
            }
        }
    }
}

// Bottom band (rows nz-nbc-1 .. nz-2) of the block's columns for n_fields
// fields from plane q0: the recurrence band_march runs,
//   f = A + W (sx + ((-qz f' - qt_z ov) - qxt ov')),  A = w pv,
// a column per lane, in the plane itself; put_band_row left pv in the plane, ov
// in R.old (row 0: the row above the band) and sx in R.sx, so a column reads
// its own values only.  A few warps alone on their SM run at the latency of
// what they wait for and at one instruction a cycle at best, so a row is kept
// to its loads, four or five products and the chain of six operations, with the
// next four rows loaded ahead of it (past the band's end too: shared memory
// follows).  In a block at a corner one more warp holds the columns of all
// fields that read their neighbour's final value (the last bottom-left column
// and the bottom-right chunk starts), kBandStage rows behind the others.
// Cycles for 50 rows of three fields on one SM: neighbours by shuffle inside
// the chain 13,900 at a corner and 3,300 on the edge; x terms read from the
// plane by two warps that meet once a group 8,250; this form 5,100 and 3,000.
constexpr int kBandStage = 8;

struct BandRows {  // four rows as loaded
    float pv[4], ov[4], w[4], s[4];
};

// KIND 0: edge columns only; 1: near a corner; 2: columns that read their
// neighbour's final value (dn columns away).
template <int PITCH, int KIND>
struct BandMarch {
    const StepParams& P;
    const float* tab;
    float* p;
    const float *old, *sx;
    int dx, dn;
    float h;
    bool corner, store;
    float fp, op;

    __device__ __forceinline__ void load(BandRows& o, int j) const {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            o.pv[r] = p[(j + r) * PITCH];
            o.ov[r] = old[(j + r + 1) * kRW];
            o.w[r] = tab[KIND ? min(dx, P.nbc - j - r) : P.nbc - j - r];
            if (KIND == 1) o.s[r] = corner ? sx[(j + r) * kRW] : -0.f;
            if (KIND == 2) o.s[r] = fmul(P.qxt, old[(j + r + 1) * kRW + dn]);
        }
    }
    // KIND 2: the x terms, from the neighbour's final values
    __device__ __forceinline__ void finals(BandRows& o, int j) const {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            o.s[r] = fsub(fsub(fmul(-P.qx, p[(j + r) * PITCH + dn]), fmul(P.qt_x, o.ov[r])), o.s[r]);
    }
    __device__ __forceinline__ void march(const BandRows& o, int j) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float A = fmul(o.w[r], o.pv[r]), w1 = fsub(1.f, o.w[r]), W = KIND ? fmul(w1, h) : w1;
            const float z = fsub(fsub(fmul(-P.qz, fp), fmul(P.qt_z, o.ov[r])), fmul(P.qxt, op));
            op = o.ov[r];
            fp = fadd(A, fmul(W, KIND ? fadd(o.s[r], z) : z));
            if (store && j + r < P.nbc) p[(j + r) * PITCH] = fp;
        }
    }
};

template <int M>
__device__ __forceinline__ void resident_bottom(const StepParams& P, const Region& R, int n_fields, int q0, const float* tab0,
                                                int tab_step) {
    constexpr int PITCH = resident_pitch(M);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = P.nbc, nx = P.nx, r0 = nx - b - 1;
    const bool corners = R.left || R.right, second = corners && warp == 2 * n_fields;
    if (warp >= 2 * n_fields && !second) return;
    // the lane's column: of the region, or of the columns that read a final value (at most 9 a field)
    const int nr = R.right ? (b + 7) / 8 : 0, per = nr + (R.left ? 1 : 0);
    const int f = second ? min(lane / per, n_fields - 1) : warp >> 1, c = lane - f * per;
    const int i = !second ? R.x0 + 32 * (warp & 1) + lane : lane >= per * n_fields ? R.x0 + 1 : c < nr ? r0 + 8 * c : b;
    const int col = i - R.x0;
    const bool lc = i >= 1 && i <= b, rc = i >= r0 && i <= nx - 2;
    const bool redo = (lc && i == b) || (rc && right_chunk_start(nx, b, i));
    const float* tab = tab0 + f * tab_step;
    float* p = cell_at<M>(R, q0 + f, col, P.nz - b - 1 - R.z0);
    const float* old = R.old + f * (b + 1) * kRW + col;
    const float *sx = R.sx + f * b * kRW + col;
    const int dx = max(min(min(i, nx - 1 - i), b + 1), 0);
    const float h = lc || rc ? 0.5f : 1.f;
    BandRows X, Y;
    if (!corners) {
        BandMarch<PITCH, 0> B{P, tab, p, old, sx, dx, 0, h, false, i < R.x1, p[-PITCH], old[0]};
        B.load(X, 0);
#pragma unroll 1
        for (int j = 0; j < b; j += 8) {
            B.load(Y, j + 4);
            B.march(X, j);
            B.load(X, j + 8);
            B.march(Y, j + 4);
        }
        return;
    }
    auto sync = [&] { asm volatile("bar.sync 1, %0;" ::"r"(32 * (2 * n_fields + 1)) : "memory"); };
    static_assert(kBandStage == 8, "two groups of four rows");
    if (!second) {
        BandMarch<PITCH, 1> B{P, tab, p, old, sx, dx, 0, h, lc || rc, i < min(R.x1, nx - 1) && i >= 1 && !redo, p[-PITCH], old[0]};
        B.load(X, 0);
#pragma unroll 1
        for (int j = 0; j < b; j += kBandStage) {
            B.load(Y, j + 4);
            B.march(X, j);
            B.load(X, j + 8);
            B.march(Y, j + 4);
            sync();
        }
    } else {
        BandMarch<PITCH, 2> B{P, tab, p, old, sx, dx, lc ? 1 : -1, h, true, lane < per * n_fields, p[-PITCH], old[0]};
#pragma unroll 1
        for (int j = 0; j < b; j += kBandStage) {
            sync();
            B.load(X, j);
            B.load(Y, j + 4);
            B.finals(X, j);
            B.finals(Y, j + 4);
            B.march(X, j);
            B.march(Y, j + 4);
        }
    }
}

// Top band (no free surface; rows 1 .. nbc) for n_fields fields from plane q0:
// a row of a field per warp, two columns per lane.  Every value is one of the
// top edge's or, in a corner, its blend with the x term; the columns that read
// their neighbour's final value (the last top-left column and the top-right
// chunk starts) take it from beside them and blend again.  Results go to a
// scratch, since the rows below and the neighbours read what is here, and from
// there to the plane.  A cell per thread with every rule spelled out took 4.9
// us for two fields in a corner block at nbc 30 (909 x 463: 20.3 us a step), this
// form 2.2 (14.0).
template <int M>
__device__ __forceinline__ void resident_top(const StepParams& P, const Region& R, int n_fields, int q0, const float* tab0,
                                             int tab_step) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int PITCH = resident_pitch(M);
    const int warp = threadIdx.x >> 5, col = 2 * (threadIdx.x & 31), i = R.x0 + col;
    const int b = P.nbc, nx = P.nx, r0 = nx - b - 1;
    const bool corners = R.left || R.right;
    bool lc[2], rc[2], rim[2], redo[2];
    int dx[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        lc[c] = i + c >= 1 && i + c <= b;
        rc[c] = i + c >= r0 && i + c <= nx - 2;
        rim[c] = i + c < 1 || i + c > nx - 2;
        redo[c] = i + c == b || (rc[c] && ((i + c - r0) & (kChunk - 1)) == 0);
        dx[c] = max(min(min(i + c, nx - 1 - i - c), b + 1), 0);
    }
#pragma unroll 1
    for (int fr = warp; fr < n_fields * b; fr += kRThreads / 32) {
        const int f = (fr >= b) + (fr >= 2 * b), j = fr - f * b + 1;
        const float* tab = tab0 + f * tab_step;
        const float* ep = R.e + (f * (b + 3) + j) * kRW + col;
        const float* op = cell_at<M>(R, q0 + f, col, j - R.z0);
        const float2 e = *reinterpret_cast<const float2*>(ep), ed = *reinterpret_cast<const float2*>(ep + kRW);
        const float2 o = *reinterpret_cast<const float2*>(op);
        const float2 od = *reinterpret_cast<const float2*>(j == b ? ep + 2 * kRW : op + PITCH);
        const int dj = min(j, P.nz - 1 - j);
        const float w0 = tab[min(dx[0], dj)], w1 = tab[min(dx[1], dj)];
        const float sz0 = edge_sum(P.qz, P.qt_z, P.qxt, ed.x, o.x, od.x), sz1 = edge_sum(P.qz, P.qt_z, P.qxt, ed.y, o.y, od.y);
        float v0 = blend_edge(w0, e.x, sz0), v1 = blend_edge(w1, e.y, sz1);
        if (corners) {
            const float el = __shfl_up_sync(FULL, e.y, 1), er = __shfl_down_sync(FULL, e.x, 1);
            const float ol = __shfl_up_sync(FULL, o.y, 1), orr = __shfl_down_sync(FULL, o.x, 1);
            const float n0 = lc[0] ? e.y : el, n1 = lc[1] ? er : e.x, o0 = lc[0] ? o.y : ol, o1 = lc[1] ? orr : o.x;
            if (lc[0] || rc[0]) v0 = blend_corner(w0, e.x, edge_sum(P.qx, P.qt_x, P.qxt, n0, o.x, o0), sz0);
            if (lc[1] || rc[1]) v1 = blend_corner(w1, e.y, edge_sum(P.qx, P.qt_x, P.qxt, n1, o.y, o1), sz1);
            const float vl = __shfl_up_sync(FULL, v1, 1), vr = __shfl_down_sync(FULL, v0, 1);
            const float u0 = blend_corner(w0, e.x, edge_sum(P.qx, P.qt_x, P.qxt, lc[0] ? v1 : vl, o.x, o0), sz0);
            const float u1 = blend_corner(w1, e.y, edge_sum(P.qx, P.qt_x, P.qxt, lc[1] ? vr : v0, o.y, o1), sz1);
            v0 = redo[0] ? u0 : v0;
            v1 = redo[1] ? u1 : v1;
        }
        *reinterpret_cast<float2*>(R.fin + fr * kRW + col) = make_float2(rim[0] ? e.x : v0, rim[1] ? e.y : v1);
    }
    __syncthreads();
#pragma unroll 1
    for (int fr = warp; fr < n_fields * b; fr += kRThreads / 32) {
        const int f = (fr >= b) + (fr >= 2 * b), j = fr - f * b + 1;
        if (i < R.x1)
            *reinterpret_cast<float2*>(cell_at<M>(R, q0 + f, col, j - R.z0)) = *reinterpret_cast<const float2*>(R.fin + fr * kRW + col);
    }
}

template <int M, int RT>
__global__ void __launch_bounds__(kRThreads, 1)
    resident_kernel(const __grid_constant__ StepParams P, const __grid_constant__ ResidentArgs A) {
    extern __shared__ __align__(128) float smem[];
    __shared__ int s_nrec, s_abort;
    __shared__ float s_src[2];
    constexpr int PITCH = resident_pitch(M), HX = resident_hx(M);
    const ResidentLayout& L = A.L;
    const int strip = blockIdx.x % L.strips, brow = blockIdx.x / L.strips;
    const int b = P.nbc, nx = P.nx, nz = P.nz;
    Region R;
    R.x0 = L.x_edge[strip];
    R.x1 = L.x_edge[strip + 1];
    R.z0 = L.z_edge[brow];
    R.z1 = L.z_edge[brow + 1];
    R.h = R.z1 - R.z0;
    R.left = strip == 0;
    R.right = strip == L.strips - 1;
    R.bottom = brow == L.rows - 1;
    R.top = brow == 0 && !P.fs;
    R.rim = R.left || R.right || R.z0 < M || R.z1 > nz - M;
    const bool src_here = P.src_i >= R.x0 && P.src_i < R.x1 && P.src_j >= R.z0 && P.src_j < R.z1;
    R.si = P.src_i - R.x0;
    R.sj = src_here ? P.src_j - R.z0 : -1;
    R.psize = resident_plane(M, R.h);
    R.plane = smem;
    float* next = smem + 5 * R.psize;
    R.old = next;
    R.sx = next + 3 * (b + 1) * kRW;
    if (R.bottom) next += resident_bottom_floats(b);
    R.e = next;
    R.fin = next + 3 * (b + 3) * kRW;
    if (R.top) next += resident_top_floats(b);
    float* med = next;
    const bool med_smem = resident_smem_floats(M, b, R.h, R.bottom, R.top, true, A.iso != 0) <= (size_t)L.smem_floats;
    if (med_smem) next += resident_med_floats(R.h, A.iso != 0);
    int2* rec = reinterpret_cast<int2*>(next);  // receivers of the region: plane offset, number
    next += 2 * kRRecCap;
    int2* mail_tab = reinterpret_cast<int2*>(next);
    next += resident_table_floats(M, R.h);
    R.wcol = next;
    next += 3 * kRW;
    R.tab = next;
    R.src = s_src;

    // ------------------------------------------------ load the region
    // (several rows of loads in flight: a call of ten steps is a quarter loading and storing; 218 -> 196 us on 1108 x 508)
    if (threadIdx.x == 0) s_nrec = s_abort = 0;
#pragma unroll 1
    for (int d = threadIdx.x; d < 3 * (b + 2); d += kRThreads) R.tab[d] = __ldg(w_table(P, d / (b + 2)) + d % (b + 2));
    if (threadIdx.x < 3 * kRW) {
        const int i = R.x0 + (threadIdx.x & (kRW - 1));
        R.wcol[threadIdx.x] = __ldg(w_table(P, threadIdx.x / kRW) + max(min(min(i, nx - 1 - i), b + 1), 0));
    }
    {
        const int rows = R.h + 2 * M + 1, n4 = PITCH / 4;
#pragma unroll 1
        for (int q = 0; q < 5; ++q) {
            const float* in = in_field(P, q);
#pragma unroll 4
            for (int idx = threadIdx.x; idx < rows * n4; idx += kRThreads) {
                const int r = idx / n4, c4 = idx - r * n4;
                const int j = R.z0 - M + r, i = R.x0 - HX + 4 * c4;
                const bool in_grid = j >= 0 && j < nz && i >= 0 && i < nx;  // x edges and row pitch are multiples of 4
                float4 v = in_grid ? ldg4(in + cell(P, i, j)) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (i + 3 >= nx)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (i + c >= nx) set_comp(v, c, 0.f);
                *reinterpret_cast<float4*>(R.plane + q * R.psize + (size_t)r * PITCH + 4 * c4) = v;
            }
        }
    }
    MedView D;
    {
        const size_t g = cell(P, R.x0, R.z0);
        const float* src[7] = {A.b[0] + g, A.b[2] + g, P.lam + g, P.mu_txx + g, P.mu_txz + g, A.b[1] + g, A.b[3] + g};
        if (med_smem) {
            const int n = A.iso ? 5 : 7, per = R.h * (kRW / 4);
#pragma unroll 1
            for (int q = 0; q < n; ++q)
#pragma unroll 4
                for (int idx = threadIdx.x; idx < per; idx += kRThreads) {
                    const int r = idx / (kRW / 4), c = 4 * (idx - r * (kRW / 4));
                    const float* s = q == 0 ? src[0] : q == 1 ? src[1] : q == 2 ? src[2] : q == 3 ? src[3] : q == 4 ? src[4] : q == 5 ? src[5] : src[6];
                    if (R.x0 + c < R.x1)
                        *reinterpret_cast<float4*>(med + (size_t)q * R.h * kRW + r * kRW + c) = ldg4(s + (size_t)r * P.pitch + c);
                }
            const size_t m = (size_t)R.h * kRW;
            D = MedView{med, A.iso ? med : med + 5 * m, med + m, A.iso ? med + m : med + 6 * m, med + 2 * m, med + 3 * m, med + 4 * m, kRW};
        } else {
            D = MedView{src[0], A.iso ? src[0] : src[5], src[1], A.iso ? src[1] : src[6], src[2], src[3], src[4], P.pitch};
        }
    }
    __syncthreads();
    // the first step's source, in this plane's copy of its cell (halo cells too)
    if (threadIdx.x < 2) {
        const int c = P.src_i - R.x0 + HX, r = P.src_j - R.z0 + M;
        if (c >= 0 && c < PITCH && r >= 0 && r < R.h + 2 * M) {
            float* p = R.plane + (TXX + threadIdx.x) * R.psize + r * PITCH + c;
            if (src_here) s_src[threadIdx.x] = *p;
            *p = fadd(*p, A.wav[0]);
        }
    }
    // receivers of the region
#pragma unroll 1
    for (int r = threadIdx.x; r < P.n_rec; r += kRThreads) {
        const int c = __ldg(P.rec_cell + r), j = c / P.pitch, i = c - j * P.pitch;
        if (i >= R.x0 && i < R.x1 && j >= R.z0 && j < R.z1) {
            const int at = atomicAdd(&s_nrec, 1);
            if (at < kRRecCap) rec[at] = make_int2((int)((j - R.z0 + M) * PITCH + i - R.x0 + HX), r);
        }
    }
    __syncthreads();
    const int n_rec = s_nrec;
    auto record = [&](int k) {  // receivers of step k from the planes
        auto put = [&](int off, int r) {
            const float* p = R.plane + off;
            float v;
            if (P.rec_kind == 0) v = p[VZ * R.psize];
            else if (P.rec_kind == 1) v = p[VX * R.psize];
            else v = fmul(fadd(p[TXX * R.psize], p[TZZ * R.psize]), 0.5f);
            P.gather[(size_t)(k - 1) + (size_t)r * P.nt] = v;
        };
        if (n_rec <= kRRecCap) {
#pragma unroll 1
            for (int q = threadIdx.x; q < n_rec; q += kRThreads) put(rec[q].x, rec[q].y);
        } else {  // more than the list holds: look through all of them
#pragma unroll 1
            for (int r = threadIdx.x; r < P.n_rec; r += kRThreads) {
                const int c = __ldg(P.rec_cell + r), j = c / P.pitch, i = c - j * P.pitch;
                if (i >= R.x0 && i < R.x1 && j >= R.z0 && j < R.z1) put((j - R.z0 + M) * PITCH + i - R.x0 + HX, r);
            }
        }
    };

    // ------------------------------------------------ exchange
    const int box = resident_mail_items(M, L.h_max);
    auto neighbour = [&](int dir) {
        if (dir == 0) return R.left ? -1 : (int)blockIdx.x - 1;
        if (dir == 1) return R.right ? -1 : (int)blockIdx.x + 1;
        if (dir == 2) return brow == 0 ? -1 : (int)blockIdx.x - L.strips;
        return R.bottom ? -1 : (int)blockIdx.x + L.strips;
    };
    const int n_side = M * R.h, n_items = 2 * n_side + 2 * M * kRW;
    const int w = R.x1 - R.x0;
    // every item's border and halo cell (plane offsets) and the message it goes to (-1: none), worked out once
    for (int idx = threadIdx.x; idx < n_items; idx += kRThreads) {
        const MailItem m = resident_mail_item<M>(R.h, w, L.h_max, idx);
        const int to = neighbour(m.dir);
        const unsigned src = (m.row + M) * PITCH + m.col + HX, dst = (m.halo_row(M) + M) * PITCH + m.halo_col(M) + HX;
        mail_tab[idx] = make_int2((int)(src | dst << 16), to < 0 || m.col >= w ? -1 : to * box + m.peer_slot(M, L.h_max));
    }
    __syncthreads();
    // kind 0: vx, vz to every side; kind 1: txx, txz to the sides, tzz, txz up and down
    auto send = [&](int kind, uint32_t tag) {
        ulonglong2* out = A.mail + kind * (box / 2);
        const float* pb = R.plane + (kind == 0 ? VZ : TXZ) * R.psize;
#pragma unroll 1
        for (int idx = threadIdx.x; idx < n_items; idx += kRThreads) {
            const int2 m = mail_tab[idx];
            const float* pa = R.plane + (kind == 0 ? VX : idx < 2 * n_side ? TXX : TZZ) * R.psize;
            if (m.y >= 0) mail_put(out + m.y, pa[m.x & 0xffff], pb[m.x & 0xffff], tag);
        }
    };
    auto receive = [&](int kind, uint32_t tag) {
        constexpr int Q = 4;
        const ulonglong2* mine = A.mail + (size_t)blockIdx.x * box + kind * (box / 2);
        float* pb = R.plane + (kind == 0 ? VZ : TXZ) * R.psize;
        const int gap = M * (L.h_max - R.h);  // mailboxes are laid out for h_max rows
#pragma unroll 1
        for (int base = threadIdx.x; base < n_items; base += Q * kRThreads) {
            unsigned dst[Q], todo = 0;
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int idx = base + q * kRThreads;
                const int2 m = idx < n_items ? mail_tab[idx] : make_int2(0, -1);
                dst[q] = (unsigned)m.x >> 16;
                todo |= m.y >= 0 ? 1u << q : 0;
            }
#pragma unroll 1
            for (int it = 0; todo; ++it) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (todo >> q & 1) {
                        const int idx = base + q * kRThreads;
                        const ulonglong2 v = mail_get(mine + idx + (idx < n_side ? 0 : idx < 2 * n_side ? gap : 2 * gap));
                        if ((uint32_t)(v.x >> 32) == tag && (uint32_t)(v.y >> 32) == tag) {
                            float* pa = R.plane + (kind == 0 ? VX : idx < 2 * n_side ? TXX : TZZ) * R.psize;
                            pa[dst[q]] = __uint_as_float((uint32_t)v.x);
                            pb[dst[q]] = __uint_as_float((uint32_t)v.y);
                            todo &= ~(1u << q);
                        }
                    }
                if (todo && mail_check_due(it) && mail_gives_up(it, kMailPolls, A.status)) {
                    s_abort = 1;
                    todo = 0;
                }
            }
        }
    };

    // ------------------------------------------------ the steps
    // One pass of the loop is a half step (kind 0 velocity, 1 stress), so that
    // the code of the bands and of the exchange is there once.
#pragma unroll 1
    for (int hs = 0; hs < 2 * A.n_steps; ++hs) {
        const int kind = hs & 1, s = hs >> 1;
        if (kind == 0) resident_velocity<M, RT>(P, R, D);
        else resident_stress<M, RT>(P, R, D);
        __syncthreads();
        if (R.bottom || R.top) {
            const int nf = 2 + kind, q0 = kind ? TXX : VX, step = kind ? 0 : b + 2;
            const float* tab = R.tab + (kind ? 2 * (b + 2) : 0);
            if (R.bottom) resident_bottom<M>(P, R, nf, q0, tab, step);
            if (R.top) resident_top<M>(P, R, nf, q0, tab, step);
            __syncthreads();
        }
        const bool rec_now = (P.rec_kind == 2) == (kind == 1);  // vx, vz after the velocity half step, p after the stress
        if (kind == 1) {
            if (rec_now) record(A.k0 + s);
            if (s + 1 == A.n_steps) break;
            if (src_here) {  // the next step's source, before the stresses are sent
                __syncthreads();
                if (threadIdx.x < 2) {
                    float* p = cell_at<M>(R, threadIdx.x == 0 ? TXX : TZZ, R.si, R.sj);
                    s_src[threadIdx.x] = *p;
                    *p = fadd(*p, A.wav[s + 1]);
                }
                __syncthreads();
            }
        }
        send(kind, A.tag0 + s);
        if (kind == 0 && rec_now) record(A.k0 + s);
        receive(kind, A.tag0 + s);
        __syncthreads();
        if (s_abort) return;
    }

    // ------------------------------------------------ store the region
#pragma unroll 1
    for (int q = 0; q < 5; ++q) {
        float* out = out_field(P, q);
#pragma unroll 4
        for (int idx = threadIdx.x; idx < R.h * (kRW / 4); idx += kRThreads) {
            const int r = idx / (kRW / 4), c = 4 * (idx - r * (kRW / 4));
            if (R.x0 + c < R.x1) stg4(out + cell(P, R.x0 + c, R.z0 + r), lds4(cell_at<M>(R, q, c, r)));
        }
    }
}

}  // namespace fomo
