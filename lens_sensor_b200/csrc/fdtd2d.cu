// 2D TE / TM CPML Yee step for sm_100a, with source, PEC and epilogues fused.
//
// One step = H half step (one launch) + E half step (one launch; TE also runs
// the epilogue there, TM needs node averages of the new E and runs it in a
// third, light launch).  Each thread owns one node (i, j); a block covers 8
// rows x 32 contiguous columns so every global access is a coalesced 128-byte
// row segment.
//
// Arithmetic follows planar_beads/boundaries.py:164-274 term by term:
//   TE  psi_Hxy = b*psi + c*dEz/dy;  Hx -= Ch*(dEz/dy/kappa + psi)      (:186-194)
//       psi_Hyx likewise along x;    Hy += Ch*(dEz/dx/kappa + psi)
//       Ez = CeE*Ez + CeH*(dHy/dx/kx + psi_x - dHx/dy/ky - psi_y)       (:196-205)
//   TM  Hz -= Ch*((dEy/dx/kx + psi) - (dEx/dy/ky + psi))                (:240-247)
//       E <- D*E (loss, fdtd2d_core.py:796-797), Ex += Ca_ex*(...),
//       Ey += -Ca_ey*(...)                                               (:249-258)
// then the Huygens source (vcsel.py:151-156) and the PEC termination
// (boundaries.py:207-215, 260-268) in the reference order (inject, then PEC).
#include <algorithm>
#include <cmath>
#include <initializer_list>

#include "lens_common.cuh"

namespace {

constexpr int BX = 32;  // columns (contiguous j) per block
constexpr int BY = 8;   // rows (i) per block

__device__ __forceinline__ float src_term(const LensSource &s, const LensStepTable &tab, int n,
                                          int i, int j) {
    // vcsel.py:151-156: F[ix] += env*sin(wt + ph1)*amp ; F[ix+1] -= env*sin(wt + ph2)*amp
    const int k = n - tab.t0;
    if (i == s.ix) return (tab.env[k] * sinf(tab.wt[k] + s.ph1[j])) * s.amp[j];
    return -((tab.env[k] * sinf(tab.wt[k] + s.ph2[j])) * s.amp[j]);
}

// Compensated complex sum of v e^{-iwt} (lens_common.cuh's kahan_add with its first product
// fused, written out so that every kernel rounds alike).
__device__ __forceinline__ void kahan_node(float *p, size_t o, float v, float pr, float pi) {
    float4 a = reinterpret_cast<float4 *>(p)[o];
    float y = __fmaf_rn(v, pr, -a.z), t = __fadd_rn(a.x, y);
    a.z = __fsub_rn(__fsub_rn(t, a.x), y);
    a.x = t;
    y = __fmaf_rn(v, pi, -a.w);
    t = __fadd_rn(a.y, y);
    a.w = __fsub_rn(__fsub_rn(t, a.y), y);
    a.y = t;
    reinterpret_cast<float4 *>(p)[o] = a;
}

// Epilogue on one node: detector boxes (FP64), compensated DFTs, intensity average.
// Every lane of the warp must call it (the box sums use warp shuffles).
__device__ __forceinline__ void epilogue_node(const LensEpi2D &ep, const LensStepTable &tab,
                                              int n, int i, int j, bool valid, size_t o,
                                              float field, float inten, float exn) {
    if (ep.nbox > 0) {
        const int bi0 = blockIdx.y * BY, bj0 = blockIdx.x * BX;
        for (int b = 0; b < ep.nbox; ++b) {
            const int *bx = ep.box[b];
            // block-uniform test: does this block touch box b at all?
            if (bx[1] <= bi0 || bx[0] >= bi0 + BY || bx[3] <= bj0 || bx[2] >= bj0 + BX) continue;
            const bool in = valid && i >= bx[0] && i < bx[1] && j >= bx[2] && j < bx[3];
            warp_atomic_add(ep.box_acc + b, in ? (double)inten : 0.0);
        }
    }
    if (!valid) return;
    const int k = n - tab.t0;
    if (n >= ep.dft_n0 && n < ep.dft_n1) {
        const float pr = tab.pe[2 * k], pi = tab.pe[2 * k + 1];
        if (ep.dft) kahan_node(ep.dft, o, field, pr, pi);
        if (ep.dft_ex) kahan_node(ep.dft_ex, o, exn, pr, pi);
    }
    if (ep.dft_prev && n >= ep.prev_n0 && n < ep.prev_n1) {
        const float pr = tab.pe[2 * k], pi = tab.pe[2 * k + 1];
        kahan_node(ep.dft_prev, o, field, pr, pi);
    }
    if (ep.iavg && n >= ep.iavg_n0) ep.iavg[o] = __fadd_rn(ep.iavg[o], inten);
}

// Plane DFT for the Poynting flux (flux.py:28-41): E on the plane, H averaged.
__device__ __forceinline__ void plane_node(const LensEpi2D &ep, const LensStepTable &tab, int n,
                                           int p, int pitch, int j, float e, float h) {
    const int k = n - tab.t0;
    double *a = ep.plane_acc + (size_t)p * 4 * pitch + j;
    const double er = tab.pe[2 * k], ei = tab.pe[2 * k + 1];
    const double hr = tab.ph[2 * k], hi = tab.ph[2 * k + 1];
    a[0] += (double)e * er;
    a[pitch] += (double)e * ei;
    a[2 * pitch] += (double)h * hr;
    a[3 * pitch] += (double)h * hi;
}

// Time-domain Poynting term of one plane cell (fdtd2d_core.py:489-497): the
// FP32 product of E and H averaged onto the E plane, summed in FP64.
__device__ __forceinline__ void sx_node(const LensEpi2D &ep, int p, int pitch, int j, float e, float h0, float h1) {
    const float h = __fmul_rn(0.5f, __fadd_rn(h0, h1));
    ep.sx_acc[(size_t)p * pitch + j] += (double)__fmul_rn(e, h);
}

__device__ __forceinline__ bool in_window(const LensEpi2D &ep, int n) {
    return n >= ep.dft_n0 && n < ep.dft_n1;
}

// Stitch drive of one cell of the driven component (rows i < d.nplanes):
// w * (env * Re(D e^{iwt})) in FP64 plus (1 - w) * E in FP32, rounded to FP32.
__device__ __forceinline__ float drive2(const LensDrive2D &d, const LensStepTable &tab, int n, int i,
                                        size_t o, float e) {
    const double *t = d.tab + 3 * (size_t)(n - tab.t0);
    const float2 D = reinterpret_cast<const float2 *>(d.hand)[o];
    const double re = __dsub_rn(__dmul_rn((double)D.x, t[1]), __dmul_rn((double)D.y, t[2]));
    const double din = __dmul_rn(t[0], re);
    const float w = d.taper[i];
    return (float)__dadd_rn(__dmul_rn((double)w, din), (double)__fmul_rn(__fsub_rn(1.0f, w), e));
}

// ------------------------------------------------------------------ TE
__global__ void __launch_bounds__(BX *BY) te2d_h(const LensTE2D g) {
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    if (i >= g.nx || j >= g.ny) return;
    const int P = g.pitch;
    const size_t o = (size_t)i * P + j;
    const float ez = g.ez[o];
    if (j < g.ny - 1) {
        const float d = g.ez[o + 1] - ez;
        float p = 0.f;
        const int s = strip_of(j, g.ay.h.lo, g.ay.h.hi, g.ay.h.n);
        if (s >= 0) {
            float *q = g.psi_hxy + (size_t)i * (g.ay.h.lo + g.ay.h.hi) + s;
            p = g.ay.h.b[j] * (*q) + g.ay.h.c[j] * d;
            *q = p;
        }
        g.hx[o] = g.hx[o] - g.ch * (d * g.ay.h.ik[j] + p);
    }
    if (i < g.nx - 1) {
        const float d = g.ez[o + P] - ez;
        float p = 0.f;
        const int s = strip_of(i, g.ax.h.lo, g.ax.h.hi, g.ax.h.n);
        if (s >= 0) {
            float *q = g.psi_hyx + (size_t)s * P + j;
            p = g.ax.h.b[i] * (*q) + g.ax.h.c[i] * d;
            *q = p;
        }
        g.hy[o] = g.hy[o] + g.ch * (d * g.ax.h.ik[i] + p);
    }
}

__global__ void __launch_bounds__(BX *BY)
    te2d_e(const LensTE2D g, const LensStepTable tab, const LensEpi2D ep, int n, const LensDrive2D d) {
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    const bool valid = i < g.nx && j < g.ny;
    const int P = g.pitch;
    const size_t o = (size_t)i * P + j;
    float ez = 0.f;
    if (valid) {
        ez = g.ez[o];
        if (i > 0 && i < g.nx - 1 && j > 0 && j < g.ny - 1) {
            const float dhy = g.hy[o] - g.hy[o - P];
            const float dhx = g.hx[o] - g.hx[o - 1];
            float qx = 0.f, qy = 0.f;
            int s = strip_of(i, g.ax.e.lo, g.ax.e.hi, g.ax.e.n);
            if (s >= 0) {
                float *q = g.psi_ezx + (size_t)s * P + j;
                qx = g.ax.e.b[i] * (*q) + g.ax.e.c[i] * dhy;
                *q = qx;
            }
            s = strip_of(j, g.ay.e.lo, g.ay.e.hi, g.ay.e.n);
            if (s >= 0) {
                float *q = g.psi_ezy + (size_t)i * (g.ay.e.lo + g.ay.e.hi) + s;
                qy = g.ay.e.b[j] * (*q) + g.ay.e.c[j] * dhx;
                *q = qy;
            }
            ez = g.ce_e[o] * ez +
                 g.ce_h[o] * (dhy * g.ax.e.ik[i] + qx - dhx * g.ay.e.ik[j] - qy);
        }
        if (g.src.ix >= 0 && (i == g.src.ix || i == g.src.ix + 1) && j < g.src.nj)
            ez += src_term(g.src, tab, n, i, j);
        if (i < d.nplanes) ez = drive2(d, tab, n, i, o, ez);
        if ((g.pec[0] && i == 0) || (g.pec[1] && i == g.nx - 1) || (g.pec[2] && j == 0) ||
            (g.pec[3] && j == g.ny - 1))
            ez = 0.f;
        g.ez[o] = ez;
        if (ep.nplane > 0 && in_window(ep, n)) {
            for (int p = 0; p < ep.nplane; ++p)
                if (i == ep.plane[p])
                    plane_node(ep, tab, n, p, P, j, ez, 0.5f * (g.hy[o - P] + g.hy[o]));
        }
        for (int p = 0; p < ep.nsx; ++p)
            if (i == ep.sx_plane[p]) sx_node(ep, p, P, j, ez, g.hy[o - P], g.hy[o]);
    }
    epilogue_node(ep, tab, n, i, j, valid, o, ez, __fmul_rn(ez, ez), 0.f);
}

// ------------------------------------------------------------------ TM
__global__ void __launch_bounds__(BX *BY) tm2d_h(const LensTM2D g) {
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    if (i >= g.nx - 1 || j >= g.ny - 1) return;
    const int P = g.pitch;
    const size_t o = (size_t)i * P + j;
    const float dyx = g.ey[o + P] - g.ey[o];
    const float dxy = g.ex[o + 1] - g.ex[o];
    float px = 0.f, py = 0.f;
    int s = strip_of(i, g.ax.h.lo, g.ax.h.hi, g.ax.h.n);
    if (s >= 0) {
        float *q = g.psi_hzx + (size_t)s * P + j;
        px = g.ax.h.b[i] * (*q) + g.ax.h.c[i] * dyx;
        *q = px;
    }
    s = strip_of(j, g.ay.h.lo, g.ay.h.hi, g.ay.h.n);
    if (s >= 0) {
        float *q = g.psi_hzy + (size_t)i * (g.ay.h.lo + g.ay.h.hi) + s;
        py = g.ay.h.b[j] * (*q) + g.ay.h.c[j] * dxy;
        *q = py;
    }
    g.hz[o] = g.hz[o] - g.ch * ((dyx * g.ax.h.ik[i] + px) - (dxy * g.ay.h.ik[j] + py));
}

__global__ void __launch_bounds__(BX *BY)
    tm2d_e(const LensTM2D g, const LensStepTable tab, int n, const LensDrive2D d) {
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    const int P = g.pitch;
    const size_t o = (size_t)i * P + j;
    if (i < g.nx - 1 && j < g.ny) {  // Ex at (i+1/2, j)
        float e = g.ex[o];
        if (g.da_x) e = e * g.da_x[o];
        if (j > 0 && j < g.ny - 1) {
            const float d = g.hz[o] - g.hz[o - 1];
            float p = 0.f;
            const int s = strip_of(j, g.ay.e.lo, g.ay.e.hi, g.ay.e.n);
            if (s >= 0) {
                float *q = g.psi_exy + (size_t)i * (g.ay.e.lo + g.ay.e.hi) + s;
                p = g.ay.e.b[j] * (*q) + g.ay.e.c[j] * d;
                *q = p;
            }
            e = e + g.ca_x[o] * (d * g.ay.e.ik[j] + p);
        }
        if ((g.pec[2] && j == 0) || (g.pec[3] && j == g.ny - 1)) e = 0.f;
        g.ex[o] = e;
    }
    if (i < g.nx && j < g.ny - 1) {  // Ey at (i, j+1/2)
        float e = g.ey[o];
        if (g.da_y) e = e * g.da_y[o];
        if (i > 0 && i < g.nx - 1) {
            const float d = g.hz[o] - g.hz[o - P];
            float p = 0.f;
            const int s = strip_of(i, g.ax.e.lo, g.ax.e.hi, g.ax.e.n);
            if (s >= 0) {
                float *q = g.psi_eyx + (size_t)s * P + j;
                p = g.ax.e.b[i] * (*q) + g.ax.e.c[i] * d;
                *q = p;
            }
            e = e + (-g.ca_y[o]) * (d * g.ax.e.ik[i] + p);
        }
        if (g.src.ix >= 0 && (i == g.src.ix || i == g.src.ix + 1) && j < g.src.nj)
            e += src_term(g.src, tab, n, i, j);
        if (i < d.nplanes) e = drive2(d, tab, n, i, o, e);
        if ((g.pec[0] && i == 0) || (g.pec[1] && i == g.nx - 1)) e = 0.f;
        g.ey[o] = e;
    }
}

// Node averages of the new TM fields (fdtd2d_core.py:458-486) and the epilogue.
__global__ void __launch_bounds__(BX *BY)
    tm2d_epi(const LensTM2D g, const LensStepTable tab, const LensEpi2D ep, int n) {
    const int j = blockIdx.x * BX + threadIdx.x;
    const int i = blockIdx.y * BY + threadIdx.y;
    const bool valid = i < g.nx && j < g.ny;
    const int P = g.pitch;
    const size_t o = (size_t)i * P + j;
    float field = 0.f, inten = 0.f, exn = 0.f;
    if (valid) {
        const int ny = g.ny, nx = g.nx;
        const float *ey = g.ey + (size_t)i * P;
        field = (j == 0) ? ey[0] : (j == ny - 1) ? ey[ny - 2] : 0.5f * (ey[j - 1] + ey[j]);
        float s2;
        if (i == 0) {
            const float a = g.ex[j];
            s2 = a * a;
            exn = a;
        } else if (i == nx - 1) {
            const float a = g.ex[(size_t)(nx - 2) * P + j];
            s2 = a * a;
            exn = a;
        } else {
            const float a = g.ex[o - P], b = g.ex[o];
            s2 = 0.5f * __fmaf_rn(a, a, __fmul_rn(b, b));
            exn = 0.5f * (a + b);
        }
        inten = __fmaf_rn(field, field, s2);
        if (in_window(ep, n)) {  // stitch: Ey on its own grid, Ex^2 on the nodes
            if (ep.dft_raw && j < ny - 1) {
                const int k = n - tab.t0;
                const float v = g.ey[o];
                kahan_add(reinterpret_cast<float4 *>(ep.dft_raw) + o, v * tab.pe[2 * k], v * tab.pe[2 * k + 1]);
            }
            if (ep.ex2) ep.ex2[o] += s2;
        }
        if (ep.nplane > 0 && in_window(ep, n) && j < ny - 1) {
            for (int p = 0; p < ep.nplane; ++p)
                if (i == ep.plane[p])
                    plane_node(ep, tab, n, p, P, j, g.ey[o], 0.5f * (g.hz[o - P] + g.hz[o]));
        }
        if (j < ny - 1)
            for (int p = 0; p < ep.nsx; ++p)
                if (i == ep.sx_plane[p]) sx_node(ep, p, P, j, g.ey[o], g.hz[o - P], g.hz[o]);
    }
    epilogue_node(ep, tab, n, i, j, valid, o, field, inten, exn);
}

// ------------------------------------------------------------------ wide passes
// H and E passes of grids too large for the chip (grid2d_resident.cuh): a thread updates
// WV = 4 columns of WR = 2 rows, all of its 16-byte loads issued before the arithmetic.
// They stream: 16 B (H) and 20 B (E) a cell for TM, 20 and 16 for TE, plus the
// coefficients, whose rows a layered grid repeats: rowref names the row to read, so a
// repeated row comes from the caches (NULL: every row its own).  Memory latency bounds
// them: 16000 x 700 cells with boxes, us a step TM / TE: 298 / 290 at one cell a thread (the
// kernels above, kept for the forms and sizes that the rules below leave to them), 106 / 95 here
// with 32 warps an SM, 110 / 98 in blocks of 8 warps, 139 / 122 without the register cap, 137 / 111
// with 3 rows, 125 / 112 with one row and 48 warps.  Warps clear of strips, faces and source rows run
// without tests (without that form: 178 / 165).
// The multiply-adds are written out and round as those kernels do, and as
// grid2d_resident.cuh.
constexpr int WV = 4, WR = 2, WT = 4;   // columns, rows of a thread; warps of a block (along x)
constexpr int WB = 8;                   // blocks of an SM: 64 registers

__device__ __forceinline__ float psi_w(const LensProfile &p, int m, float *q, float d) {
    const float v = __fmaf_rn(__ldg(p.b + m), *q, __fmul_rn(__ldg(p.c + m), d));
    *q = v;
    return v;
}

__device__ __forceinline__ void ld4(float (&v)[WV], const float *p, bool on) {
    const float4 t = on ? *reinterpret_cast<const float4 *>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}

__device__ __forceinline__ void st4(float *p, const float (&v)[WV]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// First row and column of this thread; rows of the last block may lie beyond nx (no
// return before the shuffles below: whole warps share their rows).
__device__ __forceinline__ int wide_i0() { return (blockIdx.y * WT + threadIdx.y) * WR; }
__device__ __forceinline__ int wide_j0() { return (blockIdx.x * BX + threadIdx.x) * WV; }

// Value of the column after (up) / before (dn) a lane's four; the warp's last / first lane loads it.
__device__ __forceinline__ float wide_up(const float (&v)[WV], const float *row, int j0, bool on) {
    const float u = __shfl_down_sync(0xffffffffu, v[0], 1);
    return threadIdx.x == 31 ? (on ? row[j0 + WV] : 0.f) : u;
}
__device__ __forceinline__ float wide_dn(const float (&v)[WV], const float *row, int j0, bool on) {
    const float u = __shfl_up_sync(0xffffffffu, v[WV - 1], 1);
    return threadIdx.x == 0 ? (on ? row[j0 - 1] : 0.f) : u;
}

// Rows i0 .. i0+WR-1 and columns j0 .. j0+WV-1 clear of a profile pair's strips, of the faces
// (lo: the first row and column that update) and of the source rows.
__device__ __forceinline__ bool wide_clear(const LensProfile &x, const LensProfile &y, int i0, int j0, int nx, int ny,
                                           int lo, int six) {
    return i0 >= max(x.lo, lo) && i0 + WR <= min(x.n - x.hi, nx - 1) && j0 >= max(y.lo, lo) &&
           j0 + WV <= min(y.n - y.hi, ny - 1) && (six < 0 || six + 1 < i0 || six >= i0 + WR);
}

__device__ __forceinline__ void ik4(float (&v)[WV], const float *p) {  // profile values of four columns
#pragma unroll
    for (int c = 0; c < WV; ++c) v[c] = __ldg(p + c);
}

__global__ void __launch_bounds__(32 * WT, WB) te2d_h_wide(const LensTE2D g) {
    const int i0 = wide_i0(), j0 = wide_j0(), nx = g.nx, ny = g.ny, P = g.pitch;
    if (i0 >= nx) return;
    const bool col = j0 < ny;  // the four columns lie inside the row pitch then
    const size_t o = (size_t)i0 * P + j0;
    float ez[WR + 1][WV], hx[WR][WV], hy[WR][WV], up[WR];
#pragma unroll
    for (int r = 0; r <= WR; ++r) ld4(ez[r], g.ez + o + (size_t)r * P, col && i0 + r < nx);
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const bool in = col && i0 + r < nx;
        ld4(hx[r], g.hx + o + (size_t)r * P, in);
        ld4(hy[r], g.hy + o + (size_t)r * P, in);
        up[r] = wide_up(ez[r], g.ez + (size_t)(i0 + r) * P, j0, in && j0 + WV < ny);
    }
    if (__all_sync(0xffffffffu, wide_clear(g.ax.h, g.ay.h, i0, j0, nx, ny, 0, -1))) {  // no psi, every cell updates
        float ky[WV];
        ik4(ky, g.ay.h.ik + j0);
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            const float kx = __ldg(g.ax.h.ik + i0 + r);
#pragma unroll
            for (int c = 0; c < WV; ++c) {
                const float d = (c + 1 < WV ? ez[r][c + 1 < WV ? c + 1 : 0] : up[r]) - ez[r][c];
                hx[r][c] = __fmaf_rn(-g.ch, __fmul_rn(d, ky[c]), hx[r][c]);
                hy[r][c] = __fmaf_rn(g.ch, __fmul_rn(ez[r + 1][c] - ez[r][c], kx), hy[r][c]);
            }
            st4(g.hx + o + (size_t)r * P, hx[r]);
            st4(g.hy + o + (size_t)r * P, hy[r]);
        }
        return;
    }
    if (!col) return;
    const int wy = g.ay.h.lo + g.ay.h.hi;
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        if (i >= nx) break;
        const int s = i < nx - 1 ? strip_of(i, g.ax.h.lo, g.ax.h.hi, g.ax.h.n) : -1;
        const float kx = i < nx - 1 ? __ldg(g.ax.h.ik + i) : 0.f;
#pragma unroll
        for (int c = 0; c < WV; ++c) {
            const int j = j0 + c;
            if (j < ny - 1) {
                const float d = (c + 1 < WV ? ez[r][c + 1 < WV ? c + 1 : 0] : up[r]) - ez[r][c];
                const int sj = strip_of(j, g.ay.h.lo, g.ay.h.hi, g.ay.h.n);
                const float p = sj >= 0 ? psi_w(g.ay.h, j, g.psi_hxy + (size_t)i * wy + sj, d) : 0.f;
                hx[r][c] = __fmaf_rn(-g.ch, __fmaf_rn(d, __ldg(g.ay.h.ik + j), p), hx[r][c]);
            }
            if (i < nx - 1 && j < ny) {
                const float d = ez[r + 1][c] - ez[r][c];
                const float p = s >= 0 ? psi_w(g.ax.h, i, g.psi_hyx + (size_t)s * P + j, d) : 0.f;
                hy[r][c] = __fmaf_rn(g.ch, __fmaf_rn(d, kx, p), hy[r][c]);
            }
        }
        st4(g.hx + o + (size_t)r * P, hx[r]);
        if (i < nx - 1) st4(g.hy + o + (size_t)r * P, hy[r]);
    }
}

__global__ void __launch_bounds__(32 * WT, WB) te2d_e_wide(const LensTE2D g, const int *rowref, const LensStepTable tab, int n) {
    const int i0 = wide_i0(), j0 = wide_j0(), nx = g.nx, ny = g.ny, P = g.pitch;
    if (i0 >= nx) return;
    const bool col = j0 < ny;
    const size_t o = (size_t)i0 * P + j0;
    float hy[WR + 1][WV], hx[WR][WV], ez[WR][WV], c0[WR][WV], c1[WR][WV], dn[WR];
#pragma unroll
    for (int r = 0; r <= WR; ++r)  // hy[r] = Hy(i0 + r - 1)
        ld4(hy[r], g.hy + o + (size_t)r * P - P, col && i0 + r >= 1 && i0 + r - 1 < nx);
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        const bool in = col && i < nx;
        const size_t oc = (size_t)(in && rowref ? __ldg(rowref + i) : i) * P + j0;
        ld4(hx[r], g.hx + o + (size_t)r * P, in);
        ld4(ez[r], g.ez + o + (size_t)r * P, in);
        ld4(c0[r], g.ce_e + oc, in);
        ld4(c1[r], g.ce_h + oc, in);
        dn[r] = wide_dn(hx[r], g.hx + (size_t)i * P, j0, in && j0 > 0);
    }
    if (__all_sync(0xffffffffu, wide_clear(g.ax.e, g.ay.e, i0, j0, nx, ny, 1, g.src.ix))) {
        float ky[WV];
        ik4(ky, g.ay.e.ik + j0);
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            const float kx = __ldg(g.ax.e.ik + i0 + r);
#pragma unroll
            for (int c = 0; c < WV; ++c) {
                const float dhy = hy[r + 1][c] - hy[r][c], dhx = hx[r][c] - (c > 0 ? hx[r][c > 0 ? c - 1 : 0] : dn[r]);
                const float t = __fmaf_rn(-dhx, ky[c], __fmul_rn(dhy, kx));
                ez[r][c] = __fmaf_rn(c0[r][c], ez[r][c], __fmul_rn(c1[r][c], t));
            }
            st4(g.ez + o + (size_t)r * P, ez[r]);
        }
        return;
    }
    if (!col) return;
    const int wy = g.ay.e.lo + g.ay.e.hi;
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        if (i >= nx) break;
        const bool xin = i > 0 && i < nx - 1, xsrc = g.src.ix >= 0 && (i == g.src.ix || i == g.src.ix + 1);
        const int s = xin ? strip_of(i, g.ax.e.lo, g.ax.e.hi, g.ax.e.n) : -1;
        const float kx = __ldg(g.ax.e.ik + i);
#pragma unroll
        for (int c = 0; c < WV; ++c) {
            const int j = j0 + c;
            if (j >= ny) continue;
            float v = ez[r][c];
            if (xin && j > 0 && j < ny - 1) {
                const float dhy = hy[r + 1][c] - hy[r][c], dhx = hx[r][c] - (c > 0 ? hx[r][c > 0 ? c - 1 : 0] : dn[r]);
                const int sj = strip_of(j, g.ay.e.lo, g.ay.e.hi, g.ay.e.n);
                const float qx = s >= 0 ? psi_w(g.ax.e, i, g.psi_ezx + (size_t)s * P + j, dhy) : 0.f;
                const float qy = sj >= 0 ? psi_w(g.ay.e, j, g.psi_ezy + (size_t)i * wy + sj, dhx) : 0.f;
                const float t = __fsub_rn(__fmaf_rn(-dhx, __ldg(g.ay.e.ik + j), __fmaf_rn(dhy, kx, qx)), qy);
                v = __fmaf_rn(c0[r][c], v, __fmul_rn(c1[r][c], t));
            }
            if (xsrc && j < g.src.nj) v = __fadd_rn(v, src_term(g.src, tab, n, i, j));
            if ((g.pec[0] && i == 0) || (g.pec[1] && i == nx - 1) || (g.pec[2] && j == 0) || (g.pec[3] && j == ny - 1)) v = 0.f;
            ez[r][c] = v;
        }
        st4(g.ez + o + (size_t)r * P, ez[r]);
    }
}

__global__ void __launch_bounds__(32 * WT, WB) tm2d_h_wide(const LensTM2D g) {
    const int i0 = wide_i0(), j0 = wide_j0(), nx = g.nx, ny = g.ny, P = g.pitch;
    if (i0 >= nx - 1) return;
    const bool col = j0 < ny;
    const size_t o = (size_t)i0 * P + j0;
    float ey[WR + 1][WV], ex[WR][WV], hz[WR][WV], up[WR];
#pragma unroll
    for (int r = 0; r <= WR; ++r) ld4(ey[r], g.ey + o + (size_t)r * P, col && i0 + r < nx);
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const bool in = col && i0 + r < nx - 1;
        ld4(ex[r], g.ex + o + (size_t)r * P, in);
        ld4(hz[r], g.hz + o + (size_t)r * P, in);
        up[r] = wide_up(ex[r], g.ex + (size_t)(i0 + r) * P, j0, in && j0 + WV < ny);
    }
    if (__all_sync(0xffffffffu, wide_clear(g.ax.h, g.ay.h, i0, j0, nx, ny, 0, -1))) {
        float ky[WV];
        ik4(ky, g.ay.h.ik + j0);
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            const float kx = __ldg(g.ax.h.ik + i0 + r);
#pragma unroll
            for (int c = 0; c < WV; ++c) {
                const float dyx = ey[r + 1][c] - ey[r][c],
                            dxy = (c + 1 < WV ? ex[r][c + 1 < WV ? c + 1 : 0] : up[r]) - ex[r][c];
                hz[r][c] = __fmaf_rn(-g.ch, __fsub_rn(__fmul_rn(dyx, kx), __fmul_rn(dxy, ky[c])), hz[r][c]);
            }
            st4(g.hz + o + (size_t)r * P, hz[r]);
        }
        return;
    }
    if (!col) return;
    const int wy = g.ay.h.lo + g.ay.h.hi;
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        if (i >= nx - 1) break;
        const int s = strip_of(i, g.ax.h.lo, g.ax.h.hi, g.ax.h.n);
        const float kx = __ldg(g.ax.h.ik + i);
#pragma unroll
        for (int c = 0; c < WV; ++c) {
            const int j = j0 + c;
            if (j >= ny - 1) continue;
            const float dyx = ey[r + 1][c] - ey[r][c], dxy = (c + 1 < WV ? ex[r][c + 1 < WV ? c + 1 : 0] : up[r]) - ex[r][c];
            const int sj = strip_of(j, g.ay.h.lo, g.ay.h.hi, g.ay.h.n);
            const float px = s >= 0 ? psi_w(g.ax.h, i, g.psi_hzx + (size_t)s * P + j, dyx) : 0.f;
            const float py = sj >= 0 ? psi_w(g.ay.h, j, g.psi_hzy + (size_t)i * wy + sj, dxy) : 0.f;
            const float t = __fsub_rn(__fmaf_rn(dyx, kx, px), __fmaf_rn(dxy, __ldg(g.ay.h.ik + j), py));
            hz[r][c] = __fmaf_rn(-g.ch, t, hz[r][c]);
        }
        st4(g.hz + o + (size_t)r * P, hz[r]);
    }
}

__global__ void __launch_bounds__(32 * WT, WB) tm2d_e_wide(const LensTM2D g, const int *rowref, const LensStepTable tab, int n) {
    const int i0 = wide_i0(), j0 = wide_j0(), nx = g.nx, ny = g.ny, P = g.pitch;
    if (i0 >= nx) return;
    const bool col = j0 < ny, lossy = g.da_x != nullptr;
    const size_t o = (size_t)i0 * P + j0;
    float hz[WR + 1][WV], ex[WR][WV], ey[WR][WV], dn[WR];
#pragma unroll
    for (int r = 0; r <= WR; ++r)  // hz[r] = Hz(i0 + r - 1)
        ld4(hz[r], g.hz + o + (size_t)r * P - P, col && i0 + r >= 1 && i0 + r - 1 < nx - 1);
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        const bool inx = col && i < nx - 1, iny = col && i < nx;
        ld4(ex[r], g.ex + o + (size_t)r * P, inx);
        ld4(ey[r], g.ey + o + (size_t)r * P, iny);
        dn[r] = wide_dn(hz[r + 1], g.hz + (size_t)i * P, j0, inx && j0 > 0);
    }
    if (__all_sync(0xffffffffu, wide_clear(g.ax.e, g.ay.e, i0, j0, nx, ny, 1, g.src.ix))) {
        float ky[WV];
        ik4(ky, g.ay.e.ik + j0);
#pragma unroll
        for (int r = 0; r < WR; ++r) {
            const int i = i0 + r;
            const size_t oc = (size_t)(rowref ? __ldg(rowref + i) : i) * P + j0;
            float ca[WV], cb[WV], da[WV], db[WV];
            ld4(ca, g.ca_x + oc, true);
            ld4(cb, g.ca_y + oc, true);
            if (lossy) {
                ld4(da, g.da_x + oc, true);
                ld4(db, g.da_y + oc, true);
            }
            const float kx = __ldg(g.ax.e.ik + i);
#pragma unroll
            for (int c = 0; c < WV; ++c) {
                const float d = hz[r + 1][c] - (c > 0 ? hz[r + 1][c > 0 ? c - 1 : 0] : dn[r]), d2 = hz[r + 1][c] - hz[r][c];
                const float e = lossy ? __fmul_rn(ex[r][c], da[c]) : ex[r][c], e2 = lossy ? __fmul_rn(ey[r][c], db[c]) : ey[r][c];
                ex[r][c] = __fmaf_rn(ca[c], __fmul_rn(d, ky[c]), e);
                ey[r][c] = __fmaf_rn(-cb[c], __fmul_rn(d2, kx), e2);
            }
            st4(g.ex + o + (size_t)r * P, ex[r]);
            st4(g.ey + o + (size_t)r * P, ey[r]);
        }
        return;
    }
    if (!col) return;
    const int wy = g.ay.e.lo + g.ay.e.hi;
#pragma unroll
    for (int r = 0; r < WR; ++r) {
        const int i = i0 + r;
        if (i >= nx) break;
        const size_t oc = (size_t)(rowref ? __ldg(rowref + i) : i) * P + j0;
        const size_t ox = i < nx - 1 ? oc : 0;  // the last row has no Ex (and no coefficients of it)
        float ca[WV], cb[WV], da[WV], db[WV];
        ld4(ca, g.ca_x + ox, true);
        ld4(cb, g.ca_y + oc, true);
        if (lossy) {
            ld4(da, g.da_x + ox, true);
            ld4(db, g.da_y + oc, true);
        }
        const bool xin = i > 0 && i < nx - 1, xsrc = g.src.ix >= 0 && (i == g.src.ix || i == g.src.ix + 1);
        const int s = xin ? strip_of(i, g.ax.e.lo, g.ax.e.hi, g.ax.e.n) : -1;
        const float kx = __ldg(g.ax.e.ik + i);
#pragma unroll
        for (int c = 0; c < WV; ++c) {
            const int j = j0 + c;
            if (i < nx - 1 && j < ny) {  // Ex at (i+1/2, j)
                float e = ex[r][c];
                if (lossy) e = __fmul_rn(e, da[c]);
                if (j > 0 && j < ny - 1) {
                    const float d = hz[r + 1][c] - (c > 0 ? hz[r + 1][c > 0 ? c - 1 : 0] : dn[r]);
                    const int sj = strip_of(j, g.ay.e.lo, g.ay.e.hi, g.ay.e.n);
                    const float p = sj >= 0 ? psi_w(g.ay.e, j, g.psi_exy + (size_t)i * wy + sj, d) : 0.f;
                    e = __fmaf_rn(ca[c], __fmaf_rn(d, __ldg(g.ay.e.ik + j), p), e);
                }
                if ((g.pec[2] && j == 0) || (g.pec[3] && j == ny - 1)) e = 0.f;
                ex[r][c] = e;
            }
            if (j < ny - 1) {  // Ey at (i, j+1/2)
                float e = ey[r][c];
                if (lossy) e = __fmul_rn(e, db[c]);
                if (xin) {
                    const float d = hz[r + 1][c] - hz[r][c];
                    const float p = s >= 0 ? psi_w(g.ax.e, i, g.psi_eyx + (size_t)s * P + j, d) : 0.f;
                    e = __fmaf_rn(-cb[c], __fmaf_rn(d, kx, p), e);
                }
                if (xsrc && j < g.src.nj) e = __fadd_rn(e, src_term(g.src, tab, n, i, j));
                if ((g.pec[0] && i == 0) || (g.pec[1] && i == nx - 1)) e = 0.f;
                ey[r][c] = e;
            }
        }
        if (i < nx - 1) st4(g.ex + o + (size_t)r * P, ex[r]);
        st4(g.ey + o + (size_t)r * P, ey[r]);
    }
}

// ---- coefficient rows that repeat
// For every row the first row of the run of rows it lies in that hold the same bits in
// every coefficient array.  Formed anew by each call that steps with it, from the
// coefficients as they are then: nothing of it outlives the call.
struct RowArrays {
    const float *a[4];
    int rows[4];  // rows that the array's component has (the last one of an x component is never compared)
    int n;
};
constexpr int RRB = 8, RRT = 128;  // rows, threads of a block

// ref[i] = i where row i differs from the row before, else 0.  Reads every coefficient
// once (and one row in eight again, from the caches): bound by memory, 47 us for the four
// arrays of 16000 x 700 TM cells between steps (179 MB, 3.8 TB/s).  Called over and over, part
// of them in the L2, 35 us, and 42 / 38 at 4 / 16 rows a block, 39 at 256 threads.
__global__ void __launch_bounds__(RRT) row_heads(const RowArrays v, int nx, int ny, int P, int *ref) {
    const int i0 = blockIdx.x * RRB, q4 = (ny + 3) / 4;
    unsigned diff = 0;
    for (int m = threadIdx.x; m < v.n * q4; m += RRT) {
        const int q = m / q4, rows = v.rows[q];
        const float *a = v.a[q] + 4 * (m - q * q4);
        int4 b[RRB + 1];
#pragma unroll
        for (int r = 0; r <= RRB; ++r)  // rows beyond the array: its last again
            b[r] = __ldg(reinterpret_cast<const int4 *>(a + (size_t)min(max(i0 + r - 1, 0), rows - 1) * P));
#pragma unroll
        for (int r = 0; r < RRB; ++r)
            diff |= (((b[r].x ^ b[r + 1].x) | (b[r].y ^ b[r + 1].y) | (b[r].z ^ b[r + 1].z) | (b[r].w ^ b[r + 1].w)) != 0 ? 1u : 0u) << r;
    }
    __shared__ unsigned all;
    if (threadIdx.x == 0) all = 0;
    __syncthreads();
    diff = __reduce_or_sync(0xffffffffu, diff);
    if ((threadIdx.x & 31) == 0 && diff) atomicOr(&all, diff);
    __syncthreads();
    const int r = threadIdx.x;
    if (r < RRB && i0 + r < nx) ref[i0 + r] = (all >> r & 1u) ? i0 + r : 0;
}

// The last row at or before each that row_heads marked, in place: one block, a warp 32
// rows at a time (a ballot names their heads), its RRN groups loaded before any is looked at.
// Bound by one SM's latency: 16000 rows 14.7 us with RRN neighbouring rows a thread, 5.1 here.
constexpr int RRS = 1024, RRN = 16;
__global__ void __launch_bounds__(RRS) row_runs(int *ref, int nx) {
    __shared__ int part[RRS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x / 32;
    int before = 0;  // last head of the rounds before
    for (int base = 0; base < nx; base += RRS * RRN) {
        const int i0 = base + w * 32 * RRN;
        int v[RRN], last = -1;  // last head of this warp's rows
#pragma unroll
        for (int q = 0; q < RRN; ++q) v[q] = i0 + 32 * q + lane < nx ? ref[i0 + 32 * q + lane] : 0;
#pragma unroll
        for (int q = 0; q < RRN; ++q) {
            const unsigned heads = __ballot_sync(0xffffffffu, v[q] != 0), m = heads & (0xffffffffu >> (31 - lane));
            v[q] = m ? i0 + 32 * q + 31 - __clz(m) : last;
            if (heads) last = i0 + 32 * q + 31 - __clz(heads);
        }
        if (lane == 0) part[w] = last;
        __syncthreads();
        int run = before;
#pragma unroll
        for (int q = 0; q < RRS / 32; ++q) {
            if (q < w) run = max(run, part[q]);
            before = max(before, part[q]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < RRN; ++q)
            if (i0 + 32 * q + lane < nx) ref[i0 + 32 * q + lane] = v[q] >= 0 ? v[q] : run;
    }
}

// Intensity on node (i, j) (fdtd2d_core.py:477-486), as the epilogues form it.
__device__ __forceinline__ float node_inten(const LensTE2D &g, int i, int j) {
    const float v = g.ez[(size_t)i * g.pitch + j];
    return __fmul_rn(v, v);
}

__device__ __forceinline__ float node_inten(const LensTM2D &g, int i, int j) {
    const float *ey = g.ey + (size_t)i * g.pitch, *ex = g.ex + (size_t)i * g.pitch + j;
    const float f = j == 0 ? ey[0] : (j == g.ny - 1 ? ey[g.ny - 2] : 0.5f * (ey[j - 1] + ey[j]));
    const float a = i > 0 ? ex[-g.pitch] : ex[0], b = i < g.nx - 1 ? ex[0] : a;
    const float s2 = i == 0 || i == g.nx - 1 ? __fmul_rn(a, a) : 0.5f * __fmaf_rn(a, a, __fmul_rn(b, b));
    return __fmaf_rn(f, f, s2);
}

// Detector boxes of a wide step that has no other epilogue: one launch for every box (z),
// a block a tile of BX columns by 4 BY rows and one FP64 addition (the epilogue's one per
// warp over two launches took 11 us each on boxes of 1600 x 80 nodes).
constexpr int BOXR = 4;
template <class G>
__global__ void __launch_bounds__(BX *BY) box2d(const G g, const LensEpi2D ep) {
    const int *bx = ep.box[blockIdx.z];
    const int j = max(0, bx[2]) + blockIdx.x * BX + threadIdx.x, j1 = min(g.ny, bx[3]);
    const int i0 = max(0, bx[0]) + (blockIdx.y * BY + threadIdx.y) * BOXR, i1 = min(g.nx, bx[1]);
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < BOXR; ++r)
        if (j < j1 && i0 + r < i1) v += (double)node_inten(g, i0 + r, j);
    __shared__ double red[BY];
    v = warp_sum(v);
    if (threadIdx.x == 0) red[threadIdx.y] = v;
    __syncthreads();
    if (threadIdx.y == 0) {
        v = warp_sum(threadIdx.x < BY ? red[threadIdx.x] : 0.0);
        if (threadIdx.x == 0 && v != 0.0) atomicAdd(ep.box_acc + blockIdx.z, v);
    }
}

// Does the epilogue do more at step n than sum its boxes?
bool epi2d_beyond_boxes(const LensEpi2D *ep, int n) {
    if (!ep) return false;
    if (ep->nsx > 0) return true;
    if ((ep->dft || ep->dft_ex || ep->dft_raw || ep->ex2 || ep->nplane > 0) && n >= ep->dft_n0 && n < ep->dft_n1)
        return true;
    if (ep->dft_prev && n >= ep->prev_n0 && n < ep->prev_n1) return true;
    return ep->iavg && n >= ep->iavg_n0;
}

bool epi2d_active(const LensEpi2D *ep, int n) { return epi2d_beyond_boxes(ep, n) || (ep && ep->nbox > 0); }

bool epi2d_ok(const LensEpi2D *ep, const LensStepTable *t, int nx) {
    if (!ep) return true;
    if (ep->nbox < 0 || ep->nbox > LENS_MAX_BOX || (ep->nbox > 0 && !ep->box_acc)) return false;
    if (ep->nplane < 0 || ep->nplane > LENS_MAX_PLANE || (ep->nplane > 0 && !ep->plane_acc))
        return false;
    for (int p = 0; p < ep->nplane; ++p)  // H is averaged over rows il-1 and il
        if (ep->plane[p] < 1 || ep->plane[p] > nx - 2) return false;
    if (ep->nsx < 0 || ep->nsx > LENS_MAX_PLANE || (ep->nsx > 0 && !ep->sx_acc)) return false;
    for (int p = 0; p < ep->nsx; ++p)
        if (ep->sx_plane[p] < 1 || ep->sx_plane[p] > nx - 2) return false;
    const bool dft = ep->dft || ep->dft_ex || ep->dft_prev || ep->dft_raw || ep->nplane > 0;
    return !dft || (t->pe && t->ph);
}

template <class G>
bool grid2d_ok(const G *g) {
    return g && g->nx >= 3 && g->ny >= 3 && g->pitch >= g->ny && (g->pitch % 32) == 0 &&
           lens_profile_ok(g->ax.e, g->nx) && lens_profile_ok(g->ax.h, g->nx - 1) &&
           lens_profile_ok(g->ay.e, g->ny) && lens_profile_ok(g->ay.h, g->ny - 1) &&
           (g->src.ix < 0 || (g->src.amp && g->src.ph1 && g->src.ph2 && g->src.ix + 1 < g->nx));
}

// psi arrays of the strips each kernel updates (te2d_h/te2d_e, tm2d_h/tm2d_e)
bool psi2d_ok(const LensTE2D *g) {
    return lens_psi_ok(g->ay.h, g->psi_hxy) && lens_psi_ok(g->ax.h, g->psi_hyx) &&
           lens_psi_ok(g->ax.e, g->psi_ezx) && lens_psi_ok(g->ay.e, g->psi_ezy);
}

bool psi2d_ok(const LensTM2D *g) {
    return lens_psi_ok(g->ax.h, g->psi_hzx) && lens_psi_ok(g->ay.h, g->psi_hzy) &&
           lens_psi_ok(g->ay.e, g->psi_exy) && lens_psi_ok(g->ax.e, g->psi_eyx);
}

LensEpi2D empty_epi() {
    LensEpi2D e{};
    e.dft_n0 = e.dft_n1 = 0;
    e.prev_n0 = e.prev_n1 = 0;
    e.iavg_n0 = 1 << 30;
    return e;
}

// A drive table must cover the steps run, its amplitudes the driven rows.
bool drive2d_ok(const LensDrive2D *d, const LensStepTable *tab, int nx) {
    return !d || d->nplanes == 0 || (d->nplanes > 0 && d->nplanes <= nx && d->taper && d->hand && d->tab &&
                                     (reinterpret_cast<uintptr_t>(d->hand) & 7) == 0 && tab);
}

// The wide passes carry every plain step whose arrays start on 16-byte boundaries; the
// stitch drive, the stitch sums and the pulse planes stay with one cell a thread.  They take
// 1024 cells a block, whole column blocks, and their warps at a y face run with tests: a
// grid has to be large, and more so a narrow one, whose last block is mostly idle.  us a
// step, one cell a thread / wide: TM 26.9 / 26.6 on 4251 x 400, 31.0 / 31.0 on 8595 x 256, 45.3 /
// 46.7 on 16923 x 130, 67.9 / 63.1 on 23075 x 130, 106.9 / 118.9 on 78123 x 64, 119 / 240 on 166667
// x 30; TE 22.6 / 25.1 on 5003 x 200 and 26.9 / 26.8 on 6499 x 200, 53.5 / 61.5 on 46875 x 64, 107 /
// 102 on 78123 x 64, 121 / 207 on 166667 x 30.  (By cells alone, from 0.7 M TM and 1.1 M TE, steps
// took up to 1.5 and 1.9 times the one-cell passes': 12000 x 64 TM, 40000 x 30 TE.)
bool wide_tm(double cells, int ny) {
    const int cb = (ny + BX * WV - 1) / (BX * WV);
    const double pad = (double)cb * BX * WV / ny;
    if (cb > 3) return cells >= 1.5e6;
    return pad <= 2.0 && cells >= 2.2e6 * std::sqrt(pad) * (cb == 1 && pad > 1.5 ? 2.3 : 1.0);
}

// TM inside its windows, whose sums are a launch of their own either way: the one-cell passes stay in
// front while fields, coefficients and sums lie in the L2.  us a step, one cell a thread / wide: 44.0 /
// 47.4 on 7500 x 200 with the DFT's sums (74 MB), 77.9 / 76.5 with every sum and loss (134 MB); 67.8 /
// 63.5 on 14800 x 100 with the DFTs' and loss (113 MB); 3600 x 400 38.8 / 38.9 (66 MB) and 45.2 / 43.8 (78).
bool wide_tm_sums(double cells, int ny, double bytes) {
    const int cb = (ny + BX * WV - 1) / (BX * WV);
    return wide_tm(cells, ny) || (cells >= 1.4e6 && 2.0 * cb * BX * WV <= 3.0 * ny && bytes >= (cb > 2 ? 70e6 : 110e6));
}

// Bytes a node of the sums that step n adds to.
int sum_bytes(const LensEpi2D &e, int n) {
    const bool win = n >= e.dft_n0 && n < e.dft_n1;
    return (win && e.dft ? 16 : 0) + (win && e.dft_ex ? 16 : 0) + (e.dft_prev && n >= e.prev_n0 && n < e.prev_n1 ? 16 : 0) +
           (e.iavg && n >= e.iavg_n0 ? 4 : 0);
}

bool wide_te(double cells, int ny) {
    const int cb = (ny + BX * WV - 1) / (BX * WV);
    const double pad = (double)cb * BX * WV / ny;
    return pad <= 2.0 && cells >= (cb == 1 && pad > 1.5 ? 5e6 : 1.1e6);
}

// TE grids whose wide passes gain whatever a step's epilogue.  Below, the one-cell E pass, which
// sums small boxes while it holds the field (32 us a million nodes), is faster than the wide passes and
// a launch of the boxes (4 us): 26.1 / 30.3 us a step on 5075 x 256 with boxes of 4000 nodes, 31.0 /
// 30.9 on 6643 x 256, 26.9 / 26.8 on 4331 x 300; and a step with sums keeps its H pass too: 41.2 / 43.2
// on 5075 x 256, 51.7 / 52.0 on 6643 x 256, 53.5 / 53.5 on 4251 x 400.
bool firm_te(double cells, int ny) { return cells >= (ny > 2 * BX * WV ? 1.2e6 : 1.8e6); }

// A TE step with sums has a wide H and the one-cell E pass, which adds to them while it holds the
// field: one cell / wide with the sums in a launch of their own / this: 79.6 / 88.1 / 78.2 us a step
// on 11003 x 200, 353 / 332 / 313 on 14283 x 700.
// TM's sums are a launch of their own either way, and its boxes have one (box2d, not the epilogue
// over the whole grid) from TM_BOX cells, whatever the passes: 33.2 -> 24.7 us a step on 5387 x 130.
constexpr double TM_BOX = 0.7e6;

double box_nodes(const LensEpi2D &e) {
    double nodes = 0.0;
    for (int b = 0; b < e.nbox; ++b)
        nodes += (double)std::max(0, e.box[b][1] - e.box[b][0]) * std::max(0, e.box[b][3] - e.box[b][2]);
    return nodes;
}

bool wide_ok(const LensEpi2D &e, const LensDrive2D *dr, std::initializer_list<const void *> arrays) {
    if (dr || e.nsx > 0 || e.dft_raw || e.ex2) return false;
    for (const void *p : arrays)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

// A span forms a row table where the coefficients come from memory, not from the L2 (126
// MB): by the bytes of fields, coefficients and the sums that TM's steps add to (TE's read every
// row, in their one-cell E pass).  us a step without / with the table: TM 1600 x
// 480 to 4000 x 448 cells (50 MB) the same within 0.5 %, 4000 x 700 (79 MB) 36.1 / 33.3, 16000 x
// 200 (100 MB) 61.9 / 51.3, 8000 x 700 (158 MB) 69.9 / 49.9, 16000 x 700 (315 MB) 122.8 / 105.7;
// TE 16000 x 200 (72 MB) 47.0 / 46.6, 8000 x 700 (113 MB) 51.9 / 43.1, 16000 x 700 (225 MB) 102.4
// / 95.0; TM inside its windows, every sum and loss, one cell a thread without: 3600 x 400 (120 MB)
// 64.0 / 57.5, 14800 x 100 80.1 / 75.1, 9000 x 130 63.0 / 58.9.  Forming it takes 19 to 52 us, two to four steps' gain; a grid without repeated
// rows loses that, 5 % of the shortest span that forms one.  (Formed once with the grid and
// kept, the table went stale when the coefficients were written past its check.)
constexpr double ROW_BYTES = 90e6;
constexpr int ROW_STEPS = 8;

bool row_table_pays(int nx, int P, int arrays, double sums, int nsteps) {
    return nsteps >= ROW_STEPS && (4.0 * arrays + sums) * nx * P >= ROW_BYTES;
}

// Bytes a node of the sums that a step of [n0, n0 + nsteps) adds to, on average.
double span_sum_bytes(const LensEpi2D &e, int n0, int nsteps) {
    auto met = [&](long a, long b) { return (double)std::max(0L, std::min(b, (long)n0 + nsteps) - std::max(a, (long)n0)); };
    const double k = met(e.dft_n0, e.dft_n1) * ((e.dft ? 16 : 0) + (e.dft_ex ? 16 : 0)) +
                     (e.dft_prev ? 16 * met(e.prev_n0, e.prev_n1) : 0.0) + (e.iavg ? 4 * met(e.iavg_n0, 1L << 40) : 0.0);
    return k / std::max(nsteps, 1);
}

// TM spans that read a table: the passes are wide inside the windows too (the one-cell E pass reads
// every row), where repeated rows leave the L2 to the sums.
bool table_tm(double cells, int ny, double sums) {
    const int cb = (ny + BX * WV - 1) / (BX * WV);
    const double pad = (double)cb * BX * WV / ny;
    return wide_tm(cells, ny) || (sums > 0.0 && cells >= 1.1e6 && pad <= 2.0 && (cb > 1 || pad <= 1.5));
}

int row_table(const RowArrays &v, int nx, int ny, int P, int *rowref, void *stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    row_heads<<<(nx + RRB - 1) / RRB, RRT, 0, s>>>(v, nx, ny, P, rowref);
    row_runs<<<1, RRS, 0, s>>>(rowref, nx);
    return lens_cuda_status();
}

// Grid of box2d: the largest extents of the boxes, clipped to the grid (z: the box).
dim3 box_grid(const LensEpi2D &e, int nx, int ny) {
    int w = 0, h = 0;
    for (int b = 0; b < e.nbox; ++b) {
        h = std::max(h, std::min(nx, e.box[b][1]) - std::max(0, e.box[b][0]));
        w = std::max(w, std::min(ny, e.box[b][3]) - std::max(0, e.box[b][2]));
    }
    return w > 0 && h > 0 ? dim3((w + BX - 1) / BX, (h + BY * BOXR - 1) / (BY * BOXR), e.nbox) : dim3(0, 1, 1);
}

// The launches of a span, made or (dry) only counted.
struct Launch {
    int *count;  // or NULL
    bool dry;
    template <class F>
    void operator()(F launch) const {
        if (count) ++*count;
        if (!dry) launch();
    }
};

int te2d_run(const LensTE2D *g, const LensStepTable *tab, const LensEpi2D *ep, const LensDrive2D *dr, int n0,
             int nsteps, void *stream, const int *rowref = nullptr, int *count = nullptr,
             bool dry = false) {
    if (!grid2d_ok(g) || !psi2d_ok(g) || !g->ez || !g->hx || !g->hy || !g->ce_e || !g->ce_h || nsteps < 0 ||
        !lens_table_ok(tab, n0, nsteps) || !epi2d_ok(ep, tab, g->nx) || !drive2d_ok(dr, tab, g->nx))
        return LENS_ERR_ARG;
    LensEpi2D e = ep ? *ep : empty_epi();
    lens_clip_boxes(e, g->nx, g->ny);
    const LensDrive2D d = dr ? *dr : LensDrive2D{};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Launch go{count, dry};
    const dim3 blk(BX, BY), grd((g->ny + BX - 1) / BX, (g->nx + BY - 1) / BY);
    const double cells = (double)g->nx * g->ny;
    if (wide_te(cells, g->ny) && wide_ok(e, dr, {g->ez, g->hx, g->hy, g->ce_e, g->ce_h})) {
        const dim3 wb(BX, WT), wg((g->ny + BX * WV - 1) / (BX * WV), (g->nx + WT * WR - 1) / (WT * WR)), bg = box_grid(e, g->nx, g->ny);
        const double nodes = box_nodes(e);
        const bool firm = firm_te(cells, g->ny), wide = firm || nodes == 0.0 || nodes >= 0.12e6;
        for (int n = n0; n < n0 + nsteps; ++n) {
            const bool sums = epi2d_beyond_boxes(&e, n);
            if (sums ? firm : wide) go([&] { te2d_h_wide<<<wg, wb, 0, s>>>(*g); });
            else go([&] { te2d_h<<<grd, blk, 0, s>>>(*g); });
            if (sums || !wide) {
                go([&] { te2d_e<<<grd, blk, 0, s>>>(*g, *tab, e, n, d); });
                continue;
            }
            go([&] { te2d_e_wide<<<wg, wb, 0, s>>>(*g, rowref, *tab, n); });
            if (bg.x > 0) go([&] { box2d<<<bg, blk, 0, s>>>(*g, e); });
        }
        return dry ? LENS_OK : lens_cuda_status();
    }
    for (int n = n0; n < n0 + nsteps; ++n) {
        go([&] { te2d_h<<<grd, blk, 0, s>>>(*g); });
        go([&] { te2d_e<<<grd, blk, 0, s>>>(*g, *tab, e, n, d); });
    }
    return dry ? LENS_OK : lens_cuda_status();
}

int tm2d_run(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep, const LensDrive2D *dr, int n0,
             int nsteps, void *stream, const int *rowref = nullptr, int *count = nullptr,
             bool dry = false) {
    if (!grid2d_ok(g) || !psi2d_ok(g) || !g->ex || !g->ey || !g->hz || !g->ca_x || !g->ca_y ||
        (!g->da_x) != (!g->da_y) || nsteps < 0 || !lens_table_ok(tab, n0, nsteps) ||
        !epi2d_ok(ep, tab, g->nx) || !drive2d_ok(dr, tab, g->nx))
        return LENS_ERR_ARG;
    LensEpi2D e = ep ? *ep : empty_epi();
    lens_clip_boxes(e, g->nx, g->ny);
    const LensDrive2D d = dr ? *dr : LensDrive2D{};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Launch go{count, dry};
    const dim3 blk(BX, BY), grd((g->ny + BX - 1) / BX, (g->nx + BY - 1) / BY);
    const double cells = (double)g->nx * g->ny;
    const bool ok = wide_ok(e, dr, {g->ex, g->ey, g->hz, g->ca_x, g->ca_y, g->da_x, g->da_y}), wide = ok && wide_tm(cells, g->ny);
    const double state = (double)g->nx * g->pitch;
    if (wide || (ok && cells >= TM_BOX)) {
        const dim3 wb(BX, WT), wg((g->ny + BX * WV - 1) / (BX * WV), (g->nx + WT * WR - 1) / (WT * WR)), bg = box_grid(e, g->nx, g->ny);
        for (int n = n0; n < n0 + nsteps; ++n) {
            const bool sums = epi2d_beyond_boxes(&e, n);
            if (sums ? rowref || wide_tm_sums(cells, g->ny, state * (4 * (g->da_x ? 7 : 5) + sum_bytes(e, n))) : wide) {
                go([&] { tm2d_h_wide<<<wg, wb, 0, s>>>(*g); });
                go([&] { tm2d_e_wide<<<wg, wb, 0, s>>>(*g, rowref, *tab, n); });
            } else {
                go([&] { tm2d_h<<<grd, blk, 0, s>>>(*g); });
                go([&] { tm2d_e<<<grd, blk, 0, s>>>(*g, *tab, n, d); });
            }
            if (sums) go([&] { tm2d_epi<<<grd, blk, 0, s>>>(*g, *tab, e, n); });
            else if (bg.x > 0) go([&] { box2d<<<bg, blk, 0, s>>>(*g, e); });
        }
        return dry ? LENS_OK : lens_cuda_status();
    }
    for (int n = n0; n < n0 + nsteps; ++n) {
        go([&] { tm2d_h<<<grd, blk, 0, s>>>(*g); });
        go([&] { tm2d_e<<<grd, blk, 0, s>>>(*g, *tab, n, d); });
        if (epi2d_active(&e, n)) go([&] { tm2d_epi<<<grd, blk, 0, s>>>(*g, *tab, e, n); });
    }
    return dry ? LENS_OK : lens_cuda_status();
}

}  // namespace

extern "C" int lens_te2d_step(const LensTE2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                              int n0, int nsteps, void *stream) {
    return te2d_run(g, tab, ep, nullptr, n0, nsteps, stream);
}

extern "C" int lens_tm2d_step(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                              int n0, int nsteps, void *stream) {
    return tm2d_run(g, tab, ep, nullptr, n0, nsteps, stream);
}

extern "C" int lens_te2d_step_rows(const LensTE2D *g, const int *rowref, const LensStepTable *tab, const LensEpi2D *ep,
                                   int n0, int nsteps, void *stream) {
    return te2d_run(g, tab, ep, nullptr, n0, nsteps, stream, rowref);
}

extern "C" int lens_tm2d_step_rows(const LensTM2D *g, const int *rowref, const LensStepTable *tab, const LensEpi2D *ep,
                                   int n0, int nsteps, void *stream) {
    return tm2d_run(g, tab, ep, nullptr, n0, nsteps, stream, rowref);
}

extern "C" int lens_te2d_step_counted(const LensTE2D *g, const int *rowref, const LensStepTable *tab, const LensEpi2D *ep,
                                      const LensDrive2D *drive, int n0, int nsteps, int *launches, void *stream) {
    return te2d_run(g, tab, ep, drive, n0, nsteps, stream, rowref, launches);
}

extern "C" int lens_te2d_step_launches(const LensTE2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                                       const LensDrive2D *drive, int n0, int nsteps) {
    int n = 0;
    const int st = te2d_run(g, tab, ep, drive, n0, nsteps, nullptr, nullptr, &n, true);
    return st == LENS_OK ? n : st;
}

extern "C" int lens_tm2d_step_counted(const LensTM2D *g, const int *rowref, const LensStepTable *tab, const LensEpi2D *ep,
                                      const LensDrive2D *drive, int n0, int nsteps, int *launches, void *stream) {
    return tm2d_run(g, tab, ep, drive, n0, nsteps, stream, rowref, launches);
}

extern "C" int lens_tm2d_step_launches(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                                       const LensDrive2D *drive, int n0, int nsteps) {
    int n = 0;
    const int st = tm2d_run(g, tab, ep, drive, n0, nsteps, nullptr, nullptr, &n, true);
    return st == LENS_OK ? n : st;
}

extern "C" int lens_te2d_row_table(const LensTE2D *g, const LensEpi2D *ep, int n0, int nsteps, int *rowref, void *stream) {
    if (!rowref) return LENS_ERR_ARG;
    if (!grid2d_ok(g) || !g->ce_e || !g->ce_h || !row_table_pays(g->nx, g->pitch, 5, 0.0, nsteps) ||
        !wide_te((double)g->nx * g->ny, g->ny) || !wide_ok(ep ? *ep : empty_epi(), nullptr, {g->ez, g->hx, g->hy, g->ce_e, g->ce_h}))
        return LENS_ERR_SIZE;
    if (ep && span_sum_bytes(*ep, n0, nsteps) >= 8.0) return LENS_ERR_SIZE;  // half of the steps or more read every row
    return row_table(RowArrays{{g->ce_e, g->ce_h}, {g->nx, g->nx}, 2}, g->nx, g->ny, g->pitch, rowref, stream);
}

extern "C" int lens_tm2d_row_table(const LensTM2D *g, const LensEpi2D *ep, int n0, int nsteps, int *rowref, void *stream) {
    if (!rowref) return LENS_ERR_ARG;
    const double sums = ep && nsteps > 0 ? span_sum_bytes(*ep, n0, nsteps) : 0.0;
    if (!grid2d_ok(g) || !g->ca_x || !g->ca_y || (!g->da_x) != (!g->da_y) ||
        !row_table_pays(g->nx, g->pitch, g->da_x ? 7 : 5, sums, nsteps) || !table_tm((double)g->nx * g->ny, g->ny, sums) ||
        !wide_ok(ep ? *ep : empty_epi(), nullptr, {g->ex, g->ey, g->hz, g->ca_x, g->ca_y, g->da_x, g->da_y}))
        return LENS_ERR_SIZE;
    return row_table(RowArrays{{g->ca_x, g->ca_y, g->da_x, g->da_y}, {g->nx - 1, g->nx, g->nx - 1, g->nx}, g->da_x ? 4 : 2},
                     g->nx, g->ny, g->pitch, rowref, stream);
}

extern "C" int lens_te2d_step_driven(const LensTE2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                                     const LensDrive2D *drive, int n0, int nsteps, void *stream) {
    if (!drive) return LENS_ERR_ARG;
    return te2d_run(g, tab, ep, drive, n0, nsteps, stream);
}

extern "C" int lens_tm2d_step_driven(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep,
                                     const LensDrive2D *drive, int n0, int nsteps, void *stream) {
    if (!drive) return LENS_ERR_ARG;
    return tm2d_run(g, tab, ep, drive, n0, nsteps, stream);
}
