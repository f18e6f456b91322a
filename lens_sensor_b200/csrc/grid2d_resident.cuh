#pragma once
// Resident 2D grid steps for sm_100a: a single-grid solve (lens_te2d_step /
// lens_tm2d_step with its epilogue) whose state fits on the chip advances any number of
// steps in ONE cooperative launch, the fields held in registers in between.
//
// A CTA owns a band of consecutive x rows and every y column of it: a thread holds
// columns j = 64*warp + 2*lane and j + 1 of each of the band's rows in registers (three
// field arrays of RM column pairs).  Per step:
//   H phase: neighbour terms along y from the pair itself, the next lane (one
//            shuffle a pair) or, for lane 31, lane 0 of the next warp (shared
//            memory); along x from the thread's own next row, and for the band's
//            last row from the next band's first row (its E field of the previous
//            step);
//   E phase: the same towards -y / -x; the H of the row before the band (the ghost
//            row lo-1) is computed here too, from the previous band's last E row;
//   epilogue: detector boxes, node DFTs, time averages and flux planes of the new
//            fields, as fdtd2d.cu's.
// Bands exchange those single E rows through L2 only, once per step: a thread
// publishes its columns of the row as 64-bit words {value, step tag} (each stored
// whole, no fence and no flag) at the start of the E phase, and the neighbour's
// thread of the same columns polls them at the end of its next H phase until the
// tag of the step it needs appears, so that the hop passes under the rest of both
// phases.  Every poll is bounded; a wait that runs out sets *err, and all CTAs
// leave the step loop at their next CTA barrier (or when they see *err), write NaN
// to their rows of the fields and sums and end.  Each slot of the halo rows is double-buffered by step
// parity; a band publishes step n+1 only after it has read both neighbours' step n,
// which they published after reading its step n-1, the slot's last content.
//
// What bounds it: the halo hop (an L2 store and the neighbour's polls) with two CTA
// barriers, about 1 us a step, and the latency of a row's dependent instructions in the
// warps at the y faces, about 0.1 us a row.  The step by step launches (two or three a
// step, one cell a thread) took 8.2 us a step on 140 x 96 cells (launches), 18.3 on 1600 x
// 480 (L2 latency) and 27.7 on 1201 x 431 absorbing TM cells with every epilogue on; this
// kernel takes 1.5, 3.3 and 13.4 (the last bound by the compensated sums' traffic in L2
// and shared memory: 16 bytes a node and DFT, read and written each step).
// A row is instantiated in four forms, each warp taking the least that its rows and
// columns need:
//   plain     a band clear of x strips, source rows and x faces whose rows repeat one
//             coefficient row, in a warp clear of the y faces and y strips:
//             coefficients in registers, no psi, no column tests;
//   V_N       rows with coefficients of their own (a bead): read from shared memory;
//   V_N|V_Y   columns at a y face or in a y strip: psi slots, selects;
//   V_N|V_Y|V_X  rows of an x strip, source row or x face (and bands much shorter
//             than the row template): row flags, x psi.
// Every multiply-add is written out and rounds as the step by step kernels' (fdtd2d.cu)
// do, so a solve may change between the two at any step and keep its bits.  The band's
// coefficient rows and the CPML psi of its strip cells live in shared memory for the
// launch.
#include "lens_cell2d.cuh"

namespace {

constexpr int RS_MAXW = 12;                  // warps per CTA, 64 columns each: ny <= 768
constexpr int RS_MAXWY = 64;                 // psi strip width of one y staggering (lo + hi)
constexpr unsigned RS_TRIES = 1u << 22;    // polls per wait (each an L2 round trip, >= 0.3 us)
constexpr unsigned FULL = 0xffffffffu;

constexpr int RS_MAXCTA = 512;                // bands per launch
struct GPlan {
    LensInst2D g;                     // the grid's arrays (no DFT of its own: ep holds them)
    LensEpi2D ep;
    int nbands, nc;                   // bands; coefficients per row held in shared memory
    int ncol;                         // row pitch of the shared arrays (a multiple of 32, every column)
    int hold;                         // the node DFT's sums sit in shared memory for the launch
    short lo[RS_MAXCTA];              // first row of each band (a band ends where the next begins)
    unsigned tries;                   // polls per wait
    int wd_cta;                       // watchdog self-test: this band withholds its E row of step 1 (-1: none)
};

// Row flags (RowC.flags): the row exists in the band, i < nx-1 (TE Hy / TM Hz
// and Ex rows), 0 < i < nx-1 (E curl rows), source rows ix (+) / ix+1 (-), PEC
// x face, psi of an x strip (H / E).
enum : unsigned { R_REAL = 1u, R_HOK = 2u, R_IN = 4u, R_SRCP = 8u, R_SRCM = 16u, R_XPEC = 32u, R_XH = 64u, R_XE = 128u };
constexpr unsigned R_LEAN = R_REAL | R_HOK | R_IN;
// Band flags
enum : unsigned { B_PREV = 1u, B_NEXT = 2u, B_LOSSY = 4u };

// Row constants of a band (shared memory): x profile values and strip indices.
struct __align__(16) RowC {
    float kxh, kxe, bxh, cxh, bxe, cxe;
    int sxh_sxe;         // x-strip index of the H psi (low 16 bits) and E psi (high 16 bits)
    unsigned flags;
};
static_assert(sizeof(RowC) % 16 == 0 && alignof(RowC) == 16, "row constants: whole 16-byte vectors");

// Band constants (shared memory).
struct Band {
    float *f[3];
    float *pxh, *pxe, *pyh, *pye;  // psi by role: x strips (w, pitch), y strips (nx, w)
    const float *amp, *ph1, *ph2;
    int nx, ny, P, lo, R, wyh, wye, snj;
    unsigned flags;
    float ch;
};

// The halo words of a thread's two columns: a 64-bit {tag, value} word each, written
// and read whole, the second columns' words `half` words after the first columns'.
__device__ __forceinline__ void put_tag(unsigned long long *p, int half, float2 v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(t | __float_as_uint(v.x)) : "memory");
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p + half), "l"(t | __float_as_uint(v.y)) : "memory");
}

// Halo words of both neighbours (NULL: none) once every tag is `tag`; false if the
// wait ran out or another CTA reported an error.  Each round asks for all that is
// missing at once.
__device__ __forceinline__ bool get_tags(const unsigned long long *pn, const unsigned long long *pp, int half, unsigned tag,
                                         const int *err, float2 &vn, float2 &vp, unsigned tries) {
    bool nn = pn != nullptr, np = pp != nullptr;
    for (unsigned t = 0; nn || np; ++t) {
        unsigned long long a0 = 0, a1 = 0, b0 = 0, b1 = 0;
        if (nn) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a0) : "l"(pn) : "memory");
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a1) : "l"(pn + half) : "memory");
        }
        if (np) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b0) : "l"(pp) : "memory");
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b1) : "l"(pp + half) : "memory");
        }
        if (nn && (unsigned)(a0 >> 32) == tag && (unsigned)(a1 >> 32) == tag) {
            vn = make_float2(__uint_as_float((unsigned)a0), __uint_as_float((unsigned)a1));
            nn = false;
        }
        if (np && (unsigned)(b0 >> 32) == tag && (unsigned)(b1 >> 32) == tag) {
            vp = make_float2(__uint_as_float((unsigned)b0), __uint_as_float((unsigned)b1));
            np = false;
        }
        if (!nn && !np) break;
        if (t >= tries) return false;
        if ((t & 255) == 255 && *reinterpret_cast<const volatile int *>(err)) return false;
    }
    return true;
}

// Band constants, row constants and the band's coefficient rows of CTA `cta`
// into shared memory.
template <int RM, int POL>
__device__ __forceinline__ void band_setup(const LensInst2D *gp, const GPlan &pl, int cta, int NS, Band &B, RowC *rowc,
                                           float *ypc, float *cs) {
    const int lane = threadIdx.x, w = threadIdx.y;
    const int nx = gp->nx, ny = gp->ny, P = gp->pitch;
    const int lo = pl.lo[cta], hi = cta + 1 < pl.nbands ? pl.lo[cta + 1] : nx;
    const int six = gp->src.ix;
    const bool lossy = POL == 1 && gp->c[2] != nullptr;
    if (w == 0 && lane == 0) {
        for (int k = 0; k < 3; ++k) B.f[k] = static_cast<float *>(gp->f[k]);
        B.pxh = gp->psi[POL ? 0 : 1];
        B.pxe = gp->psi[POL ? 3 : 2];
        B.pyh = gp->psi[POL ? 1 : 0];
        B.pye = gp->psi[POL ? 2 : 3];
        B.amp = gp->src.amp;
        B.ph1 = gp->src.ph1;
        B.ph2 = gp->src.ph2;
        B.snj = gp->src.nj;
        B.nx = nx;
        B.ny = ny;
        B.P = P;
        B.lo = lo;
        B.R = hi - lo;
        B.wyh = gp->ay.h.lo + gp->ay.h.hi;
        B.wye = gp->ay.e.lo + gp->ay.e.hi;
        B.flags = (cta > 0 ? B_PREV : 0u) | (hi < nx ? B_NEXT : 0u) | (lossy ? B_LOSSY : 0u);
        B.ch = gp->ch;
    }
    if (w == 0 && lane <= RM) {  // RM < 32; entry RM: the ghost row lo-1
        const int r = lane, i = r < RM ? lo + r : lo - 1;
        const LensProfile xh = gp->ax.h, xe = gp->ax.e;
        RowC rc;
        rc.kxh = rc.kxe = rc.bxh = rc.cxh = rc.bxe = rc.cxe = 0.f;
        int sh = -1, se = -1;
        unsigned f = 0;
        if (i >= 0 && i < hi) {
            f = R_REAL;
            if (i < nx - 1) {
                f |= R_HOK;
                rc.kxh = __ldg(xh.ik + i);
                sh = strip_of(i, xh.lo, xh.hi, xh.n);
                if (sh >= 0) {
                    rc.bxh = __ldg(xh.b + i);
                    rc.cxh = __ldg(xh.c + i);
                    f |= R_XH;
                }
            }
            rc.kxe = __ldg(xe.ik + i);
            if (i > 0 && i < nx - 1) {
                f |= R_IN;
                se = strip_of(i, xe.lo, xe.hi, xe.n);
                if (se >= 0) {
                    rc.bxe = __ldg(xe.b + i);
                    rc.cxe = __ldg(xe.c + i);
                    f |= R_XE;
                }
            }
            if (six >= 0 && i == six) f |= R_SRCP;
            if (six >= 0 && i == six + 1) f |= R_SRCM;
            if ((gp->pec[0] && i == 0) || (gp->pec[1] && i == nx - 1)) f |= R_XPEC;
        }
        rc.sxh_sxe = (sh & 0xffff) | (se << 16);
        rc.flags = f;
        rowc[r] = rc;
    }
    // y profile values of the strip columns: ypc[0..3][sj] = b_h, c_h, b_e, c_e
    const LensProfile yh = gp->ay.h, ye = gp->ay.e;
    // the band's coefficient rows: cs[(r * nc + k) * NS + j]
    const int nci = POL == 0 ? 2 : (lossy ? 4 : 2);
    for (int c = 0; c < 2; ++c) {
        const int j = w * 64 + 2 * lane + c;
        const int sjh = (j < ny - 1) ? strip_of(j, yh.lo, yh.hi, yh.n) : -1;
        const int sje = (j > 0 && j < ny - 1) ? strip_of(j, ye.lo, ye.hi, ye.n) : -1;
        if (sjh >= 0) {
            ypc[sjh] = __ldg(yh.b + j);
            ypc[RS_MAXWY + sjh] = __ldg(yh.c + j);
        }
        if (sje >= 0) {
            ypc[2 * RS_MAXWY + sje] = __ldg(ye.b + j);
            ypc[3 * RS_MAXWY + sje] = __ldg(ye.c + j);
        }
        for (int r = 0; r < RM && j < NS; ++r) {
            const int i = lo + r;
            for (int k = 0; k < pl.nc; ++k) {
                float v = k < 2 ? 0.f : 1.f;  // no damping array: a factor of one
                if (i < hi && j < ny && k < nci) v = __ldg(gp->c[k] + (size_t)i * P + j);
                cs[(r * pl.nc + k) * NS + j] = v;
            }
        }
    }
}

// Forms of a row (see the top of the file).
enum : unsigned { V_N = 1u, V_Y = 2u, V_X = 4u };
constexpr unsigned V_GEN = V_N | V_Y | V_X;

// Floats of one warp's edge column: rows 0..RM-1 and the ghost row RM.
constexpr int rs_edge(int rm) { return (rm + 1 + 3) / 4 * 4; }

// Row pitch of the y psi in shared memory: a slot pair for every thread's columns that
// meet a strip (a strip end may split a pair at either side), then a pair per lane for
// columns outside the strips, whose psi stays 0.
constexpr int RS_YD = RS_MAXWY + 4, RS_YP = RS_YD + 64;

// Slot pair of columns j, j + 1 (j even): st, strip indices of the two.
__device__ __forceinline__ int rs_yslot(const int (&st)[2], const LensProfile &p, int j, int lane) {
    if (st[0] < 0 && st[1] < 0) return RS_YD + 2 * lane;
    return j < p.lo ? j : (p.lo + 1) / 2 * 2 + j - (p.n - p.hi) / 2 * 2;
}

// Rows of a phase.  A band of the lean forms fills its template or lacks up to
// RS_SPARE rows (tested for); the general form tests every row, which keeps the rows'
// latency chains one after another (the y-strip warps of a 12-row band took 0.8 us a
// phase that way, on a step of 3.3 us).
constexpr int RS_SPARE = 2;
template <int RM, unsigned V>
constexpr bool row_sure(int r) { return !(V & V_X) && r + RS_SPARE < RM; }

// Everything a thread keeps across the steps of a launch.
template <int RM>
struct Th {
    float2 a[RM], b[RM], c[RM];      // TE Ez, Hx, Hy / TM Ex, Ey, Hz
    float2 ga, gc;                   // ghost row lo-1: TM Ex; TE Hy / TM Hz
    float2 gpx, gph, gpe;            // its psi: x strip (H), TM y strip (H, E)
    float2 gk0, gk2;                 // its coefficients: TM Ca_x, D_x
    float2 k0, k1, k2, k3;           // coefficients of the band's repeated row: TE c0, c1 / TM Ca_x, -Ca_y, D_x, D_y
    float2 kyh, kye, byh, cyh, bye, cye;
    float kxh, kxe;                  // plain form: the 1/kappa_x of every row
    float ch;
    int lane, w, nc, R;
    bool lossy;
    // column tests as bit masks: j < ny-1, j < ny, 0 < j < ny-1, zero after the E update
    // (TE: a PEC face or beyond ny; TM Ex: a PEC face); source column
    unsigned hx0, hx1, lt0, lt1, in0, in1, ze0, ze1;
    unsigned sh0, sh1, se0, se1;     // columns of a y strip (H, E)
    bool sr0, sr1;
    const float *cs;                 // coefficient rows, at this thread's columns
    float *xh, *xe;                  // x psi rows, at this thread's columns
    float *yh, *ye;                  // y psi slots of row 0 (rows RS_YP apart)
    const RowC *rowc;                // rows 0..RM-1 and the ghost row RM
    int NS, xs;                      // row pitch of the shared arrays; of the x psi rows (0: a column beyond them)
};

__device__ __forceinline__ float bsel(unsigned m, float a, float b) {  // m all ones: a, zero: b
    return __uint_as_float((__float_as_uint(a) & m) | (__float_as_uint(b) & ~m));
}
__device__ __forceinline__ float2 bsel2(unsigned m0, unsigned m1, float2 a, float2 b) {
    return make_float2(bsel(m0, a.x, b.x), bsel(m1, a.y, b.y));
}

// Edge column of the next / previous warp: every lane reads it, lane 31 / 0 uses it.
template <int RM>
__device__ __forceinline__ void edge_in(float (&v)[rs_edge(RM)], const float *edge, int w, bool on) {
#pragma unroll
    for (int r = 0; r < rs_edge(RM); r += 4) {
        const float4 t = on ? *reinterpret_cast<const float4 *>(edge + w * rs_edge(RM) + r) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[r] = t.x; v[r + 1] = t.y; v[r + 2] = t.z; v[r + 3] = t.w;
    }
}

template <int RM, bool HI>
__device__ __forceinline__ void edge_out(float *edge, int w, const float2 (&f)[RM], float2 ghost) {
    float v[rs_edge(RM)];
#pragma unroll
    for (int r = 0; r < rs_edge(RM); ++r) {
        const float2 p = r < RM ? f[r < RM ? r : 0] : ghost;
        v[r] = HI ? p.y : p.x;
    }
#pragma unroll
    for (int r = 0; r < rs_edge(RM); r += 4)
        *reinterpret_cast<float4 *>(edge + w * rs_edge(RM) + r) = make_float4(v[r], v[r + 1], v[r + 2], v[r + 3]);
}

// Neighbour pair one column up / down: the pair's other half and one value from the next lane.
__device__ __forceinline__ float2 pair_up(float2 v, int lane, float edge) {
    const float u = __shfl_down_sync(FULL, v.x, 1);
    return make_float2(v.y, lane == 31 ? edge : u);
}
__device__ __forceinline__ float2 pair_dn(float2 v, int lane, float edge) {
    const float u = __shfl_up_sync(FULL, v.y, 1);
    return make_float2(lane == 0 ? edge : u, v.x);
}

__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void st2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
// The caller's arrays, once per launch: no alignment beyond a float's is asked of them.
__device__ __forceinline__ float2 in2(const float *p) { return make_float2(p[0], p[1]); }
__device__ __forceinline__ void out2(float *p, float2 v) {
    p[0] = v.x;
    p[1] = v.y;
}

// What a row reads from shared memory and, the psi, gives back.  The rows of a group
// load theirs before any of them computes: behind a psi store the compiler keeps every
// later load in place, which made each row wait for its own (an LDS and four dependent
// FP32 latencies a row: 7 cycles per instruction in the y-strip warps).
struct RowIn {
    float2 y, x;                     // y and x psi
    float2 k0, k1, k2, k3;           // coefficients
    float kx, bx, cx;                // x profile values
    unsigned f;                      // row flags
    float2 s;                        // source term (rows of the pair)
};

template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_load(const Th<RM> &t, int r, RowIn &n) {
    n.f = R_LEAN;
    n.kx = t.kxh;
    if (V & V_X) {
        const RowC &rc = t.rowc[r];
        n.f = rc.flags;
        n.kx = rc.kxh;
        n.bx = rc.bxh;
        n.cx = rc.cxh;
        n.x = ld2(t.xh + r * t.xs);
    } else if (V & V_N) {
        n.kx = t.rowc[r].kxh;
    }
    if (V & V_Y) n.y = ld2(t.yh + r * RS_YP);
}

template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_store(const Th<RM> &t, int r, const RowIn &n) {
    if (V & V_X) st2(t.xh + r * t.xs, n.x);
    if (V & V_Y) st2(t.yh + r * RS_YP, n.y);
}

// Kept in a column or row of a strip, 0 outside, where psi is 0 whatever d: c = 0 alone would
// make it NaN of an infinite d, and the slot that the columns outside share with it.  Of the
// products (as here), of d and of psi, the y mask cost the warps at the y faces 0.7, 0.6 and
// 1.1 % over 36 sizes, their psi in slot pairs (5 % as single slots, the masks then needed
// registers that there were not).
__device__ __forceinline__ float2 in_strip(unsigned m0, unsigned m1, float2 v) { return bsel2(m0, m1, v, f2(0.f)); }

// psi' kept where the masks say, d * kx + psi' returned.  strip: the row lies in its strip.
__device__ __forceinline__ float2 psi_x(RowIn &n, float2 d, unsigned m0, unsigned m1, bool strip) {
    const unsigned s = strip ? ~0u : 0u;
    const float2 p = in_strip(s, s, cell_psi(f2(n.bx), n.x, f2(n.cx), d));
    n.x = bsel2(m0, m1, p, n.x);
    return fma2(d, f2(n.kx), p);
}

// H of row r, the band's last row excepted (TE: Hx of that row too).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_row(Th<RM> &t, int r, float edge, RowIn &n) {
    const float2 nch = f2(-t.ch);
    const bool hok = row_sure<RM, V>(r + 1) || (r + 1 < t.R && (!(V & V_X) || (n.f & R_HOK)));
    const int rn = r + 1 < RM ? r + 1 : r;
    if (POL == 0) {
        const float2 ez = t.a[r], d = sub2(pair_up(ez, t.lane, edge), ez);
        float2 u;
        if (V & V_Y) {
            n.y = fma2(t.byh, n.y, in_strip(t.sh0, t.sh1, mul2(t.cyh, d)));
            u = fma2(d, t.kyh, n.y);
        } else {
            u = mul2(d, t.kyh);
        }
        const float2 hx = fma2(nch, u, t.b[r]);
        t.b[r] = (V & V_Y) ? bsel2(t.hx0, t.hx1, hx, t.b[r]) : hx;
        if (r + 1 < RM) {
            const float2 e = sub2(t.a[rn], ez);
            const unsigned m0 = hok ? t.lt0 : 0u, m1 = hok ? t.lt1 : 0u;
            const float2 v = (V & V_X) ? psi_x(n, e, m0, m1, n.f & R_XH) : mul2(e, f2(n.kx));
            const float2 hy = fma2(f2(t.ch), v, t.c[r]);
            if (V & V_Y) t.c[r] = bsel2(m0, m1, hy, t.c[r]);
            else t.c[r] = sel2(hok, hok, hy, t.c[r]);
        }
    } else if (r + 1 < RM) {
        const float2 ex = t.a[r], dyx = sub2(t.b[rn], t.b[r]), dxy = sub2(pair_up(ex, t.lane, edge), ex);
        const unsigned m0 = hok ? t.hx0 : 0u, m1 = hok ? t.hx1 : 0u;
        const float2 u = (V & V_X) ? psi_x(n, dyx, m0, m1, n.f & R_XH) : mul2(dyx, f2(n.kx));
        float2 v;
        if (V & V_Y) {
            const float2 py = fma2(t.byh, n.y, in_strip(t.sh0, t.sh1, mul2(t.cyh, dxy)));
            n.y = sel2(hok, hok, py, n.y);
            v = fma2(dxy, t.kyh, py);
        } else {
            v = mul2(dxy, t.kyh);
        }
        const float2 hz = fma2(nch, sub2(u, v), t.c[r]);
        if (V & V_Y) t.c[r] = bsel2(m0, m1, hz, t.c[r]);
        else t.c[r] = sel2(hok, hok, hz, t.c[r]);
    }
}

// The band's last row (TE Hy, TM Hz) from en: the E field of row i+1 (TE Ez, TM Ey).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_last(Th<RM> &t, int r, float2 en, float edge) {
    RowIn n;
    h_load<RM, POL, V>(t, r, n);
    const bool hok = !(V & V_X) || (n.f & R_HOK);
    const float2 d = sub2(en, POL == 0 ? t.a[r] : t.b[r]);
    const unsigned m0 = hok ? (POL == 0 ? t.lt0 : t.hx0) : 0u, m1 = hok ? (POL == 0 ? t.lt1 : t.hx1) : 0u;
    const float2 u = (V & V_X) ? psi_x(n, d, m0, m1, n.f & R_XH) : mul2(d, f2(n.kx));
    float2 h;
    if (POL == 0) {
        h = fma2(f2(t.ch), u, t.c[r]);
    } else {
        const float2 ex = t.a[r], dxy = sub2(pair_up(ex, t.lane, edge), ex);
        float2 v;
        if (V & V_Y) {
            const float2 py = fma2(t.byh, n.y, in_strip(t.sh0, t.sh1, mul2(t.cyh, dxy)));
            n.y = sel2(hok, hok, py, n.y);
            v = fma2(dxy, t.kyh, py);
        } else {
            v = mul2(dxy, t.kyh);
        }
        h = fma2(f2(-t.ch), sub2(u, v), t.c[r]);
    }
    t.c[r] = (V & V_Y) ? bsel2(m0, m1, h, t.c[r]) : h;
    if (POL == 1) h_store<RM, POL, V>(t, r, n);
    else if (V & V_X) st2(t.xh + r * t.xs, n.x);
}

// H of the ghost row lo-1 (TE Hy, TM Hz) from ep: its E field (TE Ez, TM Ey).  The
// row may lie in an x strip whatever the band's form (b = c = 0 elsewhere).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_ghost(Th<RM> &t, float2 ep, float edge) {
    const RowC &rc = t.rowc[RM];
    const unsigned s = rc.flags & R_XH ? ~0u : 0u;
    const float2 d = sub2(POL == 0 ? t.a[0] : t.b[0], ep), px = in_strip(s, s, cell_psi(f2(rc.bxh), t.gpx, f2(rc.cxh), d));
    const float2 u = fma2(d, f2(rc.kxh), px);
    const unsigned m0 = POL == 0 ? t.lt0 : t.hx0, m1 = POL == 0 ? t.lt1 : t.hx1;
    float2 h;
    if (POL == 0) {
        h = fma2(f2(t.ch), u, t.gc);
    } else {
        const float2 dxy = sub2(pair_up(t.ga, t.lane, edge), t.ga);
        float2 v;
        if (V & V_Y) {
            t.gph = fma2(t.byh, t.gph, in_strip(t.sh0, t.sh1, mul2(t.cyh, dxy)));
            v = fma2(dxy, t.kyh, t.gph);
        } else {
            v = mul2(dxy, t.kyh);
        }
        h = fma2(f2(-t.ch), sub2(u, v), t.gc);
    }
    t.gpx = (V & V_Y) ? bsel2(m0, m1, px, t.gpx) : px;
    t.gc = (V & V_Y) ? bsel2(m0, m1, h, t.gc) : h;
}

// TM Ex of the ghost row lo-1.
template <int RM, unsigned V>
__device__ __forceinline__ void e_ghost(Th<RM> &t, float edge) {
    const float2 d = sub2(t.gc, pair_dn(t.gc, t.lane, edge));
    float2 u;
    if (V & V_Y) {
        t.gpe = fma2(t.bye, t.gpe, in_strip(t.se0, t.se1, mul2(t.cye, d)));
        u = fma2(d, t.kye, t.gpe);
    } else {
        u = mul2(d, t.kye);
    }
    float2 e = t.lossy ? mul2(t.ga, t.gk2) : t.ga;
    const float2 en = fma2(t.gk0, u, e);
    if (V & V_Y) {
        e = bsel2(t.in0, t.in1, en, e);
        e = bsel2(t.ze0, t.ze1, f2(0.f), e);
        t.ga = bsel2(t.lt0, t.lt1, e, t.ga);
    } else {
        t.ga = en;
    }
}

// Source term of the columns j, j + 1 for row flags rf at table row k (vcsel.py:151-156).
__device__ __forceinline__ float2 src_term(const Band &B, const LensStepTable &tab, unsigned rf, int j, bool on0, bool on1,
                                           int k) {
    const float env = __ldg(tab.env + k), wt = __ldg(tab.wt + k);
    const float *ph = (rf & R_SRCP) ? B.ph1 : B.ph2;
    float2 s = f2(0.f);
    if (on0) s.x = (env * sinf(wt + __ldg(ph + j))) * __ldg(B.amp + j);
    if (on1) s.y = (env * sinf(wt + __ldg(ph + j + 1))) * __ldg(B.amp + j + 1);
    return (rf & R_SRCP) ? s : neg2(s);
}

template <int RM, int POL, unsigned V>
__device__ __forceinline__ void e_load(const Th<RM> &t, int r, RowIn &n) {
    n.f = R_LEAN;
    n.kx = t.kxe;
    if (V & V_X) {
        const RowC &rc = t.rowc[r];
        n.f = rc.flags;
        n.kx = rc.kxe;
        n.bx = rc.bxe;
        n.cx = rc.cxe;
        n.x = ld2(t.xe + r * t.xs);
    } else if (V & V_N) {
        n.kx = t.rowc[r].kxe;
    }
    if (V & V_Y) n.y = ld2(t.ye + r * RS_YP);
    n.k0 = t.k0;
    n.k1 = t.k1;
    n.k2 = t.k2;
    n.k3 = t.k3;
    if (V & V_N) {
        const float *c = t.cs + r * t.nc * t.NS;
        n.k0 = ld2(c);
        n.k1 = POL == 0 ? ld2(c + t.NS) : neg2(ld2(c + t.NS));
        if (POL == 1 && t.lossy) {
            n.k2 = ld2(c + 2 * t.NS);
            n.k3 = ld2(c + 3 * t.NS);
        }
    }
}

template <int RM, int POL, unsigned V>
__device__ __forceinline__ void e_store(const Th<RM> &t, int r, const RowIn &n) {
    if (V & V_X) st2(t.xe + r * t.xs, n.x);
    if (V & V_Y) st2(t.ye + r * RS_YP, n.y);
}

// E of row r at table row k; hm: the H field of row i-1 (TE Hy, TM Hz).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void e_row(Th<RM> &t, int r, float2 hm, float edge, RowIn &n) {
    const unsigned rf = n.f;
    const bool rin = rf & R_IN;
    if (POL == 0) {
        const float2 hx = t.b[r], dhy = sub2(t.c[r], hm), dhx = sub2(hx, pair_dn(hx, t.lane, edge));
        float2 u = (V & V_X) ? psi_x(n, dhy, t.in0, t.in1, rf & R_XE) : mul2(dhy, f2(n.kx));
        u = fma2(neg2(dhx), t.kye, u);
        if (V & V_Y) {
            const float2 py = fma2(t.bye, n.y, in_strip(t.se0, t.se1, mul2(t.cye, dhx)));
            n.y = sel2(rin, rin, py, n.y);
            u = sub2(u, py);
        }
        float2 v = fma2(n.k0, t.a[r], mul2(n.k1, u));
        if (V & V_Y) v = bsel2(rin ? t.in0 : 0u, rin ? t.in1 : 0u, v, t.a[r]);
        if ((V & V_X) && (rf & (R_SRCP | R_SRCM))) {
            v.x += n.s.x;
            v.y += n.s.y;
        }
        if (V & V_Y) v = bsel2((rf & R_XPEC) ? ~0u : t.ze0, (rf & R_XPEC) ? ~0u : t.ze1, f2(0.f), v);
        t.a[r] = v;
    } else {
        const float2 hz = t.c[r], d = sub2(hz, pair_dn(hz, t.lane, edge)), d2 = sub2(hz, hm);
        float2 u;
        if (V & V_Y) {
            const float2 py = fma2(t.bye, n.y, in_strip(t.se0, t.se1, mul2(t.cye, d)));
            const bool on = rf & R_HOK;
            n.y = sel2(on, on, py, n.y);
            u = fma2(d, t.kye, py);
        } else {
            u = mul2(d, t.kye);
        }
        const float2 v = (V & V_X) ? psi_x(n, d2, t.hx0, t.hx1, rf & R_XE) : mul2(d2, f2(n.kx));
        // Ex at (i+1/2, j) (boundaries.py:249-258)
        float2 e = t.lossy ? mul2(t.a[r], n.k2) : t.a[r];
        const float2 en = fma2(n.k0, u, e);
        if (V & V_Y) {
            e = bsel2(t.in0, t.in1, en, e);
            e = bsel2(t.ze0, t.ze1, f2(0.f), e);
            t.a[r] = bsel2((rf & R_HOK) ? t.lt0 : 0u, (rf & R_HOK) ? t.lt1 : 0u, e, t.a[r]);
        } else {
            t.a[r] = en;
        }
        // Ey at (i, j+1/2) (:259-268)
        float2 e2 = t.lossy ? mul2(t.b[r], n.k3) : t.b[r];
        const float2 e2n = fma2(n.k1, v, e2);
        if (V & V_X) {
            e2 = sel2(rin, rin, e2n, e2);
            if (rf & (R_SRCP | R_SRCM)) {
                e2.x += n.s.x;
                e2.y += n.s.y;
            }
            e2 = sel2(rf & R_XPEC, rf & R_XPEC, f2(0.f), e2);
        } else {
            e2 = e2n;
        }
        t.b[r] = (V & V_Y) ? bsel2(t.hx0, t.hx1, e2, t.b[r]) : e2;
    }
}

// Rows that load together.
constexpr int rs_group(int pol, bool e) { return pol == 1 && e ? 2 : 4; }

// The H phase before the halo rows are needed: every row but the last (TE: its Hx too).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_phase(Th<RM> &t, const float (&z)[rs_edge(RM)]) {
    constexpr int G = rs_group(POL, false);
#pragma unroll
    for (int r0 = 0; r0 < RM; r0 += G) {
        RowIn n[G];
#pragma unroll
        for (int q = 0; q < G; ++q)
            if (r0 + q < RM) h_load<RM, POL, V>(t, r0 + q, n[q]);
#pragma unroll
        for (int q = 0; q < G; ++q)
            if (r0 + q < RM && (row_sure<RM, V>(r0 + q) || r0 + q < t.R)) {
                h_row<RM, POL, V>(t, r0 + q < RM ? r0 + q : 0, z[r0 + q < RM ? r0 + q : 0], n[q]);
                h_store<RM, POL, V>(t, r0 + q, n[q]);
            }
    }
}

// The first row the band's last row can be.
template <int RM, unsigned V>
constexpr int last_from() { return (V & V_X) || RM <= RS_SPARE ? 0 : RM - 1 - RS_SPARE; }

// The H phase after the halo rows en (the next band's first E row) and ep (the
// previous band's last) have arrived.
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void h_edges(Th<RM> &t, float2 en, float2 ep, bool prev, const float (&z)[rs_edge(RM)]) {
#pragma unroll
    for (int r = last_from<RM, V>(); r < RM; ++r)
        if (r == t.R - 1) h_last<RM, POL, V>(t, r, en, z[r]);
    if (prev) h_ghost<RM, POL, V>(t, ep, z[RM]);
}

// The E phase's rows that the neighbouring bands wait for, published at once (first /
// last: this thread's halo words for them, NULL without that neighbour).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void e_edges(Th<RM> &t, bool prev, const float (&x)[rs_edge(RM)], const float2 (&src)[RM],
                                        unsigned long long *first, unsigned long long *last, int half, unsigned tag) {
    constexpr int r1 = last_from<RM, V>() > 0 ? last_from<RM, V>() : 1, G = RM - r1;
    RowIn n0, n[G > 0 ? G : 1];
    e_load<RM, POL, V>(t, 0, n0);
#pragma unroll
    for (int q = 0; q < G; ++q) e_load<RM, POL, V>(t, r1 + q, n[q]);
    if (POL == 1 && prev) e_ghost<RM, V>(t, x[RM]);
    n0.s = src[0];
    e_row<RM, POL, V>(t, 0, t.gc, x[0], n0);
    if (first) put_tag(first, half, POL == 0 ? t.a[0] : t.b[0], tag);
    if (last && t.R == 1) put_tag(last, half, POL == 0 ? t.a[0] : t.b[0], tag);
    e_store<RM, POL, V>(t, 0, n0);
#pragma unroll
    for (int q = 0; q < G; ++q) {
        const int r = r1 + q;
        if (row_sure<RM, V>(r) || r < t.R) {
            n[q].s = src[r];
            e_row<RM, POL, V>(t, r, t.c[r - 1], x[r], n[q]);
            if (last && r == t.R - 1) put_tag(last, half, POL == 0 ? t.a[r] : t.b[r], tag);
            e_store<RM, POL, V>(t, r, n[q]);
        }
    }
}

// The rows e_edges left (the general form: none).
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void e_phase(Th<RM> &t, const float (&x)[rs_edge(RM)]) {
    constexpr int r1 = (V & V_X) ? 0 : last_from<RM, V>(), G = rs_group(POL, true);
#pragma unroll
    for (int r0 = 1; r0 < r1; r0 += G) {
        RowIn n[G];
#pragma unroll
        for (int q = 0; q < G; ++q)
            if (r0 + q < r1) e_load<RM, POL, V>(t, r0 + q, n[q]);
#pragma unroll
        for (int q = 0; q < G; ++q)
            if (r0 + q < r1) {
                const int r = r0 + q < RM ? r0 + q : 1;
                e_row<RM, POL, V>(t, r, t.c[r - 1], x[r], n[q]);
                e_store<RM, POL, V>(t, r, n[q]);
            }
    }
}

// ---------------------------------------------------------------- epilogue
// Which parts of the epilogue step n runs (uniform over the launch).
enum : unsigned { EP_DFT = 1u, EP_EX = 2u, EP_PREV = 4u, EP_IAVG = 8u, EP_PLANE = 16u };

__device__ __forceinline__ unsigned epi_parts(const LensEpi2D &ep, int n) {
    const bool win = n >= ep.dft_n0 && n < ep.dft_n1;
    return (win && ep.dft ? EP_DFT : 0u) | (win && ep.dft_ex ? EP_EX : 0u) | (win && ep.nplane > 0 ? EP_PLANE : 0u) |
           (ep.dft_prev && n >= ep.prev_n0 && n < ep.prev_n1 ? EP_PREV : 0u) | (ep.iavg && n >= ep.iavg_n0 ? EP_IAVG : 0u);
}

// Compensated complex sum (lens_common.cuh's kahan_add, its first product fused as
// there), real and imaginary part at once: a = (sum, carry), np = minus the phase.
// With m = carry - v phase = -y, the sum is t = sum - m and the carry (t - sum) + m.
__device__ __forceinline__ void kahan_pair(float4 &a, float v, float2 np) {
    const float2 s = make_float2(a.x, a.y), m = fma2(f2(v), np, make_float2(a.z, a.w)), t = sub2(s, m);
    const float2 c = __fadd2_rn(sub2(t, s), m);
    a = make_float4(t.x, t.y, c.x, c.y);
}

// Rows whose sums travel together.
constexpr int EPI_G = 4;

// Node value of row r: 0 the driven field, 1 (TM) Ex on the nodes, 2 the intensity
// (fdtd2d_core.py:458-486).  y: TM, the Ey of the column before each warp's first.
// Rows at an x face are the general form's, columns at a y face the V_Y form's.
template <int RM, int POL, unsigned V>
__device__ __forceinline__ float2 node_value(const Th<RM> &t, const Band &B, int r, int what, float y) {
    if (POL == 0) return what == 2 ? mul2(t.a[r], t.a[r]) : t.a[r];
    const float2 ey = t.b[r], lo = pair_dn(ey, t.lane, y);
    float2 F = mul2(f2(0.5f), make_float2(lo.x + ey.x, lo.y + ey.y));
    if (V & V_Y) {
        const int j = t.w * 64 + 2 * t.lane, ny = B.ny;
        F.x = j == 0 ? ey.x : (j == ny - 1 ? lo.x : F.x);
        F.y = j + 1 == ny - 1 ? lo.y : F.y;
    }
    if (what == 0) return F;
    const float2 p = r > 0 ? t.a[r > 0 ? r - 1 : 0] : t.ga, c = t.a[r];  // Ex of rows i-1 and i
    float2 X = mul2(f2(0.5f), make_float2(p.x + c.x, p.y + c.y)), s2 = mul2(f2(0.5f), fma2(p, p, mul2(c, c)));
    if (V & V_X) {
        const int i = B.lo + r;
        const bool first = i == 0, last = i == B.nx - 1;
        const float2 e = sel2(last, last, p, c);
        X = sel2(first || last, first || last, e, X);
        s2 = sel2(first || last, first || last, mul2(e, e), s2);
    }
    const float2 I = fma2(F, F, s2);
    return sel2(what == 1, what == 1, X, I);
}

// The epilogue of one step on a thread's cells.  box: this band meets a detector box.
// Loops over the sums stay loops: unrolled for every sum, box and row the code ran from
// beyond the instruction caches in each of the four row forms and cost 4.8 us a step
// whatever it had to do.
template <int RM, int POL, unsigned V>
__device__ __forceinline__ void epilogue(const Th<RM> &t, const Band &B, const LensEpi2D &ep, const LensStepTable &tab,
                                         int k, unsigned parts, bool box, const float (&y)[rs_edge(RM)], bool hold,
                                         float *sdft, double *bacc) {
    const int j = t.w * 64 + 2 * t.lane, ny = B.ny;
    const bool on0 = !(V & V_Y) || j < ny, on1 = !(V & V_Y) || j + 1 < ny;
    const size_t o = (size_t)B.lo * B.P + j;
    if (parts & (EP_DFT | EP_EX | EP_PREV)) {
        const float2 np = make_float2(-__ldg(tab.pe + 2 * k), -__ldg(tab.pe + 2 * k + 1));
#pragma unroll 1
        for (int a = 0; a < (POL == 1 ? 3 : 2); ++a) {  // compensated sums: DFT, comparison window, TM Ex
            if (!(parts & (a == 0 ? EP_DFT : (a == 1 ? EP_PREV : EP_EX)))) continue;
            float4 *d = reinterpret_cast<float4 *>(a == 0 ? ep.dft : (a == 1 ? ep.dft_prev : ep.dft_ex)) + o;
            int P = B.P;
            if (a == 0 && hold) {
                d = reinterpret_cast<float4 *>(sdft);
                P = t.NS;
            }
#pragma unroll
            for (int r0 = 0; r0 < RM; r0 += EPI_G) {
                float4 s[2 * EPI_G];
#pragma unroll
                for (int q = 0; q < EPI_G; ++q)
                    if (r0 + q < RM && r0 + q < t.R) {
                        if (on0) s[2 * q] = d[(size_t)(r0 + q) * P];
                        if (on1) s[2 * q + 1] = d[(size_t)(r0 + q) * P + 1];
                    }
#pragma unroll
                for (int q = 0; q < EPI_G; ++q) {
                    const int r = r0 + q < RM ? r0 + q : 0;
                    if (r0 + q >= RM) continue;
                    const float2 v = node_value<RM, POL, V>(t, B, r, a == 2 ? 1 : 0, y[r]);
                    if (r >= t.R) continue;
                    kahan_pair(s[2 * q], v.x, np);
                    kahan_pair(s[2 * q + 1], v.y, np);
                    if (on0) d[(size_t)r * P] = s[2 * q];
                    if (on1) d[(size_t)r * P + 1] = s[2 * q + 1];
                }
            }
        }
    }
    if (parts & EP_IAVG) {
        float *a = ep.iavg + o;
#pragma unroll
        for (int r0 = 0; r0 < RM; r0 += EPI_G) {
            float2 s[EPI_G];
#pragma unroll
            for (int q = 0; q < EPI_G; ++q)
                if (r0 + q < RM && r0 + q < t.R) {
                    if (on0) s[q].x = a[(size_t)(r0 + q) * B.P];
                    if (on1) s[q].y = a[(size_t)(r0 + q) * B.P + 1];
                }
#pragma unroll
            for (int q = 0; q < EPI_G; ++q) {
                const int r = r0 + q < RM ? r0 + q : 0;
                if (r0 + q >= RM) continue;
                const float2 I = node_value<RM, POL, V>(t, B, r, 2, y[r]);
                if (r >= t.R) continue;
                if (on0) a[(size_t)r * B.P] = __fadd_rn(s[q].x, I.x);
                if (on1) a[(size_t)r * B.P + 1] = __fadd_rn(s[q].y, I.y);
            }
        }
    }
    if (box) {
#pragma unroll 1
        for (int b = 0; b < ep.nbox; ++b) {
            const int lo = ep.box[b][0] - B.lo, hi = min(ep.box[b][1] - B.lo, t.R);
            const bool c0 = on0 && j >= ep.box[b][2] && j < ep.box[b][3],
                       c1 = on1 && j + 1 >= ep.box[b][2] && j + 1 < ep.box[b][3];
            if (hi <= lo || hi <= 0 || !__any_sync(FULL, c0 || c1)) continue;
            double v[4] = {0.0, 0.0, 0.0, 0.0};  // four chains of FP64 additions
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const float2 I = node_value<RM, POL, V>(t, B, r, 2, y[r]);
                const bool in = r >= lo && r < hi;
                v[r % 2 * 2] += (double)(in && c0 ? I.x : 0.f);
                v[r % 2 * 2 + 1] += (double)(in && c1 ? I.y : 0.f);
            }
            bacc[b * 32 * blockDim.y] += (v[0] + v[1]) + (v[2] + v[3]);
        }
    }
    if (parts & EP_PLANE) {
        // Poynting plane DFTs (flux.py:28-41): E on the plane, H averaged over rows il-1 and il
#pragma unroll 1
        for (int p = 0; p < ep.nplane; ++p) {
            const int rr = ep.plane[p] - B.lo;
            if (rr < 0 || rr >= t.R) continue;
            const double er = __ldg(tab.pe + 2 * k), ei = __ldg(tab.pe + 2 * k + 1), hr = __ldg(tab.ph + 2 * k),
                         hi = __ldg(tab.ph + 2 * k + 1);
            float2 e = f2(0.f), h = f2(0.f), hm = t.gc;
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const unsigned m = r == rr ? ~0u : 0u, mm = r + 1 == rr ? ~0u : 0u;
                e = bsel2(m, m, POL == 0 ? t.a[r] : t.b[r], e);
                h = bsel2(m, m, t.c[r], h);
                hm = bsel2(mm, mm, t.c[r], hm);
            }
            const int jn = POL == 0 ? ny : ny - 1;
            double *a = ep.plane_acc + (size_t)p * 4 * B.P + j;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (j + c >= jn) continue;
                const double ev = c ? e.y : e.x, hv = 0.5f * (c ? hm.y + h.y : hm.x + h.x);
                a[c] += ev * er;
                a[c + B.P] += ev * ei;
                a[c + 2 * B.P] += hv * hr;
                a[c + 3 * B.P] += hv * hi;
            }
        }
    }
}

// The steps of one launch in one row form.  Each warp runs the loop of its own form
// (the CTA barriers are the same ones): no choice is left inside a step.
template <int RM, int POL, unsigned V>
__device__ __forceinline__ bool rs_loop(Th<RM> &t, const Band &B, const GPlan &pl, const LensStepTable &tab, int n0,
                                        int nsteps, unsigned long long *halo, int *err, bool prev, bool next, bool box,
                                        float *zb, bool hold, float *sdft, double *bacc) {
    constexpr int EP = rs_edge(RM);
    const int lane = t.lane, w = t.w, W = blockDim.y, j = w * 64 + 2 * lane;
    float *xb = zb + W * EP, *eb = xb + W * EP;
    // halo words: [cta][kind 0: first E row, 1: last E row][slot][column of the pair][thread];
    // the rows of the state before step u carry tag u + 1
    const int half = 32 * W, hq = 4 * half;
    unsigned long long *h_my = halo + (size_t)(blockIdx.x * 2 * hq + w * 32 + lane);
    bool bad = false;
    for (int u = 0; u < nsteps; ++u) {
        const int k = n0 + u - tab.t0, slot = (u & 1) * 2 * half;
        // ------------------------------------------------------------ H phase
        float z[EP];
        edge_in<RM>(z, zb, w + 1, w + 1 < W);
        h_phase<RM, POL, V>(t, z);
        float2 src[RM];  // the step's source terms, before the wait that they need not follow
        if (V & V_X) {
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                src[r] = f2(0.f);
                const unsigned rf = t.rowc[r].flags;
                if (rf & (R_SRCP | R_SRCM)) src[r] = src_term(B, tab, rf, j, t.sr0, t.sr1, k);
            }
        }
        float2 en = f2(0.f), ep = f2(0.f);
        if (!bad)
            bad = !get_tags(next ? h_my + 2 * hq + slot : nullptr, prev ? h_my - hq + slot : nullptr, half,
                            (unsigned)(u + 1), err, en, ep, pl.tries);
        h_edges<RM, POL, V>(t, en, ep, prev, z);
        if (lane == 31) {
            if (POL == 0) edge_out<RM, true>(xb, w, t.b, f2(0.f));
            else edge_out<RM, true>(xb, w, t.c, t.gc);
        }
        if (__syncthreads_or(bad)) break;

        // ------------------------------------------------------------ E phase
        float x[EP];
        edge_in<RM>(x, xb, w - 1, w > 0);
        unsigned long long *h_pub = h_my + (2 * half - slot);
        const bool first = prev && !((int)blockIdx.x == pl.wd_cta && u == 1);
        e_edges<RM, POL, V>(t, prev, x, src, first ? h_pub : nullptr, next ? h_pub + hq : nullptr, half,
                            (unsigned)(u + 2));
        e_phase<RM, POL, V>(t, x);
        const unsigned parts = epi_parts(pl.ep, n0 + u);
        if (lane == 0) edge_out<RM, false>(zb, w, t.a, t.ga);
        if (POL == 1 && (parts || box) && lane == 31) edge_out<RM, true>(eb, w, t.b, f2(0.f));
        __syncthreads();  // a wait that ran out above leaves the loop at the next barrier
        if (parts || box) {
            float y[EP];
            if (POL == 1) edge_in<RM>(y, eb, w - 1, w > 0);
            epilogue<RM, POL, V>(t, B, pl.ep, tab, k, parts, box, y, hold, sdft, bacc);
        }
    }
    return bad;
}

// Columns j, j + 1 of a band whose results are invalid: NaN in the fields' own cells (what lies
// beyond them stays as it is) and in every sum that the band feeds.  Apart from the band's code:
// within it the steps' registers came out otherwise (TE 1201 x 431 in its windows 6.62 us a step
// against 6.29).
template <int POL>
__device__ __noinline__ void rs_invalid(const GPlan &pl, const Band &B, int j, int *err) {
    const float nan = __int_as_float(0x7fc00000);
    const LensEpi2D &ep = pl.ep;
    atomicOr(err, 1);
    for (int r = 0; r < B.R; ++r) {
        const int i = B.lo + r;
        for (int c = j; c < j + 2 && c < B.ny; ++c) {
            const size_t o = (size_t)i * B.P + c;
            const bool h = i < B.nx - 1, v = c < B.ny - 1;
            if (POL == 0 || h) B.f[0][o] = nan;
            if (v) B.f[1][o] = nan;
            if (h && (POL == 0 || v)) B.f[2][o] = nan;
            float *const sum[3] = {ep.dft, ep.dft_ex, ep.dft_prev};
            for (int q = 0; q < 3; ++q)
                if (sum[q]) reinterpret_cast<float4 *>(sum[q])[o] = make_float4(nan, nan, nan, nan);
            if (ep.iavg) ep.iavg[o] = nan;
            for (int p = 0; p < ep.nplane; ++p)
                for (int q = 0; q < 4; ++q)
                    if (ep.plane[p] == i) ep.plane_acc[((size_t)p * 4 + q) * B.P + c] = nan;
        }
    }
    for (int b = 0; b < ep.nbox; ++b)
        if (ep.box[b][0] < B.lo + B.R && ep.box[b][1] > B.lo) atomicAdd(ep.box_acc + b, (double)nan);
}

// One band.  GEN: every warp in the general form (at most RM rows), else the lean forms.
template <int RM, int POL, bool GEN>
__device__ __forceinline__ void rs_band(const GPlan &pl, const LensStepTable &tab, int n0, int nsteps,
                                        unsigned long long *halo, int *err, unsigned char *smem) {
    constexpr int EP = rs_edge(RM);
    Th<RM> t;
    const int lane = t.lane = threadIdx.x, w = t.w = threadIdx.y, W = blockDim.y, NS = t.NS = pl.ncol;
    const int j = w * 64 + 2 * lane, tid = w * 32 + lane;
    const int cta = blockIdx.x;
    const int NC = t.nc = pl.nc;
    const LensInst2D *gp = &pl.g;

    // shared memory: box sums [nbox][threads] (double), coefficient rows [RM][NC][NS], the
    // node DFT's sums [RM][NS][4] when held, x-strip psi
    // (H, E; general form) [RM][NS] and a pair per lane for the x psi of the last warp's
    // columns beyond NS [64], y-strip psi (H, E) [RM][RS_YP], edge columns of the
    // warps zb / xb / eb [W][EP], y profile values of the strip columns [4][RS_MAXWY], row
    // constants [RM + 1], band constants
    double *bacc = reinterpret_cast<double *>(smem) + tid;
    float *cs = reinterpret_cast<float *>(smem + (size_t)pl.ep.nbox * 32 * W * sizeof(double));
    float *dac = cs + RM * NC * NS;
    float *xps_h = dac + (pl.hold ? RM * NS * 4 : 0);
    float *xps_e = xps_h + (GEN ? RM * NS : 0);
    float *out = xps_e + (GEN ? RM * NS : 0);  // stays 0 (those columns update nothing)
    float *yps_h = out + 64;
    float *yps_e = yps_h + RM * RS_YP;
    float *zb = yps_e + RM * RS_YP;      // lane 0 of each warp: E field read at j+1 (TE Ez, TM Ex)
    // xb = zb + W EP, lane 31: H field read at j-1 (TE Hx, TM Hz); eb = xb + W EP, lane 31: TM Ey
    float *ypc = zb + 3 * W * EP;
    RowC *rowc = reinterpret_cast<RowC *>(ypc + 4 * RS_MAXWY);
    Band &B = *reinterpret_cast<Band *>(rowc + RM + 1);
    for (int v = tid; v < (GEN ? 2 * RM * NS : 0) + 64 + 2 * RM * RS_YP; v += 32 * W) xps_h[v] = 0.f;
    for (int b = 0; b < pl.ep.nbox; ++b) bacc[b * 32 * W] = 0.0;
    band_setup<RM, POL>(gp, pl, cta, NS, B, rowc, ypc, cs);
    __syncthreads();

    const int ny = B.ny, R = t.R = B.R;
    const unsigned bf = B.flags;
    const bool prev = bf & B_PREV, next = bf & B_NEXT;
    t.ch = B.ch;
    t.lossy = bf & B_LOSSY;
    t.rowc = rowc;
    const bool held = j < NS;  // the last warp's upper lanes may lie beyond the shared rows
    t.cs = cs + (held ? j : 0);
    t.xh = held ? xps_h + j : out + 2 * lane;
    t.xe = held ? xps_e + j : out + 2 * lane;
    t.xs = held ? NS : 0;
    // per column: tests, 1/kappa_y, y-psi slot and its profile values
    bool hx[2], lt[2], in[2], pe[2], sr[2];
    float kyh[2], kye[2], bh[2], chh[2], be[2], ce[2];
    int sjh[2], sje[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int jc = j + c;
        hx[c] = jc < ny - 1;
        lt[c] = jc < ny;
        in[c] = jc > 0 && jc < ny - 1;
        pe[c] = (gp->pec[2] && jc == 0) || (gp->pec[3] && jc == ny - 1);
        sr[c] = jc < B.snj;
        sjh[c] = hx[c] ? strip_of(jc, gp->ay.h.lo, gp->ay.h.hi, ny - 1) : -1;
        sje[c] = in[c] ? strip_of(jc, gp->ay.e.lo, gp->ay.e.hi, ny) : -1;
        kyh[c] = hx[c] ? __ldg(gp->ay.h.ik + jc) : 0.f;
        kye[c] = lt[c] ? __ldg(gp->ay.e.ik + jc) : 0.f;
        bh[c] = sjh[c] >= 0 ? ypc[sjh[c]] : 0.f;
        chh[c] = sjh[c] >= 0 ? ypc[RS_MAXWY + sjh[c]] : 0.f;
        be[c] = sje[c] >= 0 ? ypc[2 * RS_MAXWY + sje[c]] : 0.f;
        ce[c] = sje[c] >= 0 ? ypc[3 * RS_MAXWY + sje[c]] : 0.f;
    }
    t.kyh = make_float2(kyh[0], kyh[1]); t.kye = make_float2(kye[0], kye[1]);
    t.byh = make_float2(bh[0], bh[1]); t.cyh = make_float2(chh[0], chh[1]);
    t.bye = make_float2(be[0], be[1]); t.cye = make_float2(ce[0], ce[1]);
    t.yh = yps_h + rs_yslot(sjh, gp->ay.h, j, lane);
    t.ye = yps_e + rs_yslot(sje, gp->ay.e, j, lane);
    auto mask = [](bool v) { return v ? ~0u : 0u; };
    t.hx0 = mask(hx[0]); t.hx1 = mask(hx[1]); t.lt0 = mask(lt[0]); t.lt1 = mask(lt[1]);
    t.in0 = mask(in[0]); t.in1 = mask(in[1]);
    t.ze0 = mask(pe[0] || (POL == 0 && !lt[0])); t.ze1 = mask(pe[1] || (POL == 0 && !lt[1]));
    t.sr0 = sr[0]; t.sr1 = sr[1];
    t.sh0 = mask(sjh[0] >= 0); t.sh1 = mask(sjh[1] >= 0); t.se0 = mask(sje[0] >= 0); t.se1 = mask(sje[1] >= 0);
    // the row form of this warp
    bool same = !GEN;
    const RowC r0 = rowc[0];
#pragma unroll
    for (int r = 0; r < RM; ++r) {
        const RowC rc = rowc[r];
        if (!GEN && r < R) {
            same = same && rc.kxh == r0.kxh && rc.kxe == r0.kxe;
            for (int k = 0; k < NC; ++k) {
                const float2 u = ld2(t.cs + k * NS), v = ld2(t.cs + (r * NC + k) * NS);
                same = same && u.x == v.x && u.y == v.y;
            }
        }
    }
    const bool edge_w = __any_sync(FULL, !in[0] || !in[1] || sjh[0] >= 0 || sjh[1] >= 0 || sje[0] >= 0 || sje[1] >= 0);
    same = __all_sync(FULL, same);
    const unsigned form = edge_w ? (V_N | V_Y) : (same ? 0u : V_N);
    t.kxh = r0.kxh;
    t.kxe = r0.kxe;
    t.k0 = ld2(t.cs);
    t.k1 = POL == 0 ? ld2(t.cs + NS) : neg2(ld2(t.cs + NS));
    t.k2 = t.lossy ? ld2(t.cs + 2 * NS) : f2(1.f);
    t.k3 = t.lossy ? ld2(t.cs + 3 * NS) : f2(1.f);

    // ---- state in: fields (registers), psi strips (shared memory).  j is even and the
    // pitch a multiple of 32, so a pair whose first column exists lies inside its row.
#pragma unroll
    for (int r = 0; r < RM; ++r) {
        const bool on = r < R && lt[0];
        const size_t o = (size_t)(B.lo + r) * B.P + j;
        t.a[r] = on ? in2(B.f[0] + o) : f2(0.f);
        t.b[r] = on ? in2(B.f[1] + o) : f2(0.f);
        t.c[r] = on ? in2(B.f[2] + o) : f2(0.f);
        if (r < R) {
            const RowC &rc = rowc[r];
            const int sh = (int)(short)(rc.sxh_sxe & 0xffff), se = rc.sxh_sxe >> 16;
            if (GEN && sh >= 0 && on) st2(t.xh + r * NS, in2(B.pxh + (size_t)sh * B.P + j));
            if (GEN && se >= 0 && on) st2(t.xe + r * NS, in2(B.pxe + (size_t)se * B.P + j));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (sjh[c] >= 0) t.yh[r * RS_YP + c] = B.pyh[(size_t)(B.lo + r) * B.wyh + sjh[c]];
                if (sje[c] >= 0) t.ye[r * RS_YP + c] = B.pye[(size_t)(B.lo + r) * B.wye + sje[c]];
            }
        }
    }
    // the ghost row lo-1: its H (and TM Ex) advances here with the previous band's bits
    t.ga = t.gc = t.gpx = t.gph = t.gpe = t.gk0 = f2(0.f);
    t.gk2 = f2(1.f);
    if (prev && lt[0]) {
        const int i = B.lo - 1, sh = (int)(short)(rowc[RM].sxh_sxe & 0xffff);
        const size_t o = (size_t)i * B.P + j;
        t.gc = in2(B.f[2] + o);
        if (sh >= 0) t.gpx = in2(B.pxh + (size_t)sh * B.P + j);
        if (POL == 1) {
            t.ga = in2(B.f[0] + o);
            if (sjh[0] >= 0) t.gph.x = B.pyh[(size_t)i * B.wyh + sjh[0]];
            if (sjh[1] >= 0) t.gph.y = B.pyh[(size_t)i * B.wyh + sjh[1]];
            if (sje[0] >= 0) t.gpe.x = B.pye[(size_t)i * B.wye + sje[0]];
            if (sje[1] >= 0) t.gpe.y = B.pye[(size_t)i * B.wye + sje[1]];
            t.gk0 = in2(gp->c[0] + o);
            if (t.lossy) t.gk2 = in2(gp->c[2] + o);
        }
    }
    if (lane == 0) edge_out<RM, false>(zb, w, t.a, t.ga);
    // the node DFT's sums of the launch's window steps in shared memory where they fit
    const bool hold = pl.hold && pl.ep.dft && pl.ep.dft_n0 < n0 + nsteps && pl.ep.dft_n1 > n0;
    float *sdft = dac + 4 * (held ? j : 0);
    float4 *gdft = reinterpret_cast<float4 *>(pl.ep.dft) + (size_t)B.lo * B.P + j;
    if (hold && lt[0])
        for (int r = 0; r < R; ++r) {
            float4 *l = reinterpret_cast<float4 *>(sdft) + (size_t)r * NS;
            l[0] = gdft[(size_t)r * B.P];
            if (lt[1]) l[1] = gdft[(size_t)r * B.P + 1];
        }
    bool box = false;  // does this band meet a detector box?
    for (int b = 0; b < pl.ep.nbox; ++b) box = box || (pl.ep.box[b][0] < B.lo + R && pl.ep.box[b][1] > B.lo);
    // a neighbour that has seen this band's first words may end and write its rows
    // back: the rows read here are read before (fence)
    __threadfence();
    __syncthreads();
    const int half = 32 * W;
    unsigned long long *h_my = halo + (size_t)(cta * 8 * half + tid);
    if (prev) put_tag(h_my, half, POL == 0 ? t.a[0] : t.b[0], 1u);
    if (next)
        put_tag(h_my + 4 * half, half, lt[0] ? in2(B.f[POL == 0 ? 0 : 1] + (size_t)(B.lo + R - 1) * B.P + j) : f2(0.f), 1u);

    bool bad;
    if (GEN) bad = rs_loop<RM, POL, V_GEN>(t, B, pl, tab, n0, nsteps, halo, err, prev, next, box, zb, hold, sdft, bacc);
    else if (form == 0u) bad = rs_loop<RM, POL, 0u>(t, B, pl, tab, n0, nsteps, halo, err, prev, next, box, zb, hold, sdft, bacc);
    else if (form == V_N) bad = rs_loop<RM, POL, V_N>(t, B, pl, tab, n0, nsteps, halo, err, prev, next, box, zb, hold, sdft, bacc);
    else bad = rs_loop<RM, POL, V_N | V_Y>(t, B, pl, tab, n0, nsteps, halo, err, prev, next, box, zb, hold, sdft, bacc);
    if (__syncthreads_or(bad)) {  // one thread's wait ran out: the whole band's results are invalid
        rs_invalid<POL>(pl, B, j, err);
        return;
    }

    // ---- state out
    if (hold && lt[0])
        for (int r = 0; r < R; ++r) {
            const float4 *l = reinterpret_cast<const float4 *>(sdft) + (size_t)r * NS;
            gdft[(size_t)r * B.P] = l[0];
            if (lt[1]) gdft[(size_t)r * B.P + 1] = l[1];
        }
    for (int b = 0; b < pl.ep.nbox; ++b) {
        const double v = warp_sum(bacc[b * 32 * W]);
        if (lane == 0 && v != 0.0) atomicAdd(pl.ep.box_acc + b, v);
    }
#pragma unroll
    for (int r = 0; r < RM; ++r) {
        if (r < R && lt[0]) {
            const size_t o = (size_t)(B.lo + r) * B.P + j;
            out2(B.f[0] + o, t.a[r]);
            out2(B.f[1] + o, t.b[r]);
            out2(B.f[2] + o, t.c[r]);
        }
        if (r < R) {
            const RowC &rc = rowc[r];
            const int sh = (int)(short)(rc.sxh_sxe & 0xffff), se = rc.sxh_sxe >> 16;
            if (GEN && sh >= 0 && lt[0]) out2(B.pxh + (size_t)sh * B.P + j, ld2(t.xh + r * NS));
            if (GEN && se >= 0 && lt[0]) out2(B.pxe + (size_t)se * B.P + j, ld2(t.xe + r * NS));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (sjh[c] >= 0) B.pyh[(size_t)(B.lo + r) * B.wyh + sjh[c]] = t.yh[r * RS_YP + c];
                if (sje[c] >= 0) B.pye[(size_t)(B.lo + r) * B.wye + sje[c]] = t.ye[r * RS_YP + c];
            }
        }
    }
}

// Is row i special: an x strip (H or E psi), a source row or an x face?
__host__ __device__ inline bool row_special(const LensInst2D &g, int i) {
    if (i <= 0 || i >= g.nx - 1) return true;  // faces (and the row without Hy / Hz)
    if (g.src.ix >= 0 && (i == g.src.ix || i == g.src.ix + 1)) return true;
    const LensProfile &h = g.ax.h, &e = g.ax.e;
    return i < h.lo || i >= h.n - h.hi || i < e.lo || i >= e.n - e.hi;
}

// NT: the most threads of a CTA.  The register file is split over the SM's four
// schedulers, so 8 warps (NT = 256) leave a thread 255 registers and 12 (NT = 384: ny >
// 512, or more CTAs on an SM) 168.  Two CTAs of 8 warps (128 registers, bands half as
// long) spilled: 2.75 us per step on 1600 x 480 cells against 2.58 for one.  RX: the most
// rows of a band in the general form.
template <int RM, int NT, int RX>
__global__ void __launch_bounds__(NT, 1)
    grid2d_rs(const __grid_constant__ GPlan pl, const LensStepTable tab, int n0, int nsteps, unsigned long long *halo,
              int *err) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cta = blockIdx.x, lo = pl.lo[cta], hi = cta + 1 < pl.nbands ? pl.lo[cta + 1] : pl.g.nx;
    bool gen = hi - lo < RM - RS_SPARE;
    for (int i = lo; i < hi; ++i) gen = gen || row_special(pl.g, i);
    if (gen) {
        if (pl.g.pol == 0) rs_band<RX, 0, true>(pl, tab, n0, nsteps, halo, err, smem);
        else rs_band<RX, 1, true>(pl, tab, n0, nsteps, halo, err, smem);
    } else {
        if (pl.g.pol == 0) rs_band<RM, 0, false>(pl, tab, n0, nsteps, halo, err, smem);
        else rs_band<RM, 1, false>(pl, tab, n0, nsteps, halo, err, smem);
    }
}

}  // namespace
