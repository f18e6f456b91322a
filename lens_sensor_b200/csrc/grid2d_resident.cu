// Resident 2D grid steps: the band plan and the launches of grid2d_resident.cuh's kernel.
#include <algorithm>
#include <exception>
#include <vector>

#include "grid2d_resident.cuh"

// Kernel of a row template (grid2d_resident_k.cu); wide: the 384-thread split.
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k2(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k4(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k6(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k8(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k10(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k12(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k14(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k16(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k18(bool wide);
__attribute__((visibility("hidden"))) const void *lens_grid2d_rs_k20(bool wide);

namespace {

// Row templates, every second count: a band of the lean forms fills its template or
// lacks up to RS_SPARE rows.
struct RsForm {
    int rm, rx;  // most rows of a lean band, of a band in the general form
    const void *(*kernel)(bool wide);
};
constexpr int RS_NRM = 10;
const RsForm RS_FORMS[RS_NRM] = {{2, 1, lens_grid2d_rs_k2},   {4, 2, lens_grid2d_rs_k4},   {6, 2, lens_grid2d_rs_k6},
                                 {8, 2, lens_grid2d_rs_k8},   {10, 2, lens_grid2d_rs_k10}, {12, 2, lens_grid2d_rs_k12},
                                 {14, 2, lens_grid2d_rs_k14}, {16, 2, lens_grid2d_rs_k16}, {18, 2, lens_grid2d_rs_k18},
                                 {20, 2, lens_grid2d_rs_k20}};

// Shared memory of a CTA; hold: the node DFT's sums in it.
size_t rs_smem(const RsForm &f, int ncol, int nc, int nbox, bool hold) {
    const int W = (ncol + 63) / 64;
    auto bytes = [&](int rm, bool gen) {
        return (size_t)nbox * 32 * W * sizeof(double) +
               (size_t)(rm * (nc + (hold ? 4 : 0) + (gen ? 2 : 0)) * ncol + 64 + 2 * rm * RS_YP + 3 * W * rs_edge(rm) +
                        4 * RS_MAXWY) * sizeof(float) + (rm + 1) * sizeof(RowC) + sizeof(Band);
    };
    return std::max(bytes(f.rm, false), bytes(f.rx, true));
}

// Relative cost of a row and, in percent of its bands' cost, what a further CTA on an SM
// adds to a step: CTAs on an SM overlap one's halo wait with another's rows, so two bands of
// half the rows cost more than one of them and less than both in turn.  Neither is critical:
// us a step of 36 grids (140 x 96 to 1848 x 300 and 5000 x 128, inside their windows and not)
// on average, against 34 and 30: special rows at 20, 27 and 44 0.996, 1.003 and 1.006, shares
// of 0, 15 and 60 0.998, 1.002 and 1.002.
constexpr int RS_COST_LEAN = 10, RS_COST_SPECIAL = 34, RS_SHARE = 30;

// Runs of special and of other rows of a grid, in order.
struct Run {
    int len;
    bool special;
};

std::vector<Run> rs_runs(const LensInst2D &g) {
    std::vector<Run> v;
    for (int i = 0; i < g.nx; ++i) {
        const bool sp = row_special(g, i);
        if (v.empty() || v.back().special != sp) v.push_back(Run{0, sp});
        ++v.back().len;
    }
    return v;
}

// Bands of a grid with cost at most T, lean ones of at most rm rows and others of at
// most rx; their first rows into lo (when not NULL).  Every run is cut into bands of
// equal length to within a row; one that leaves the row template emptier than the lean
// forms take runs in the general form.
int rs_bands(const std::vector<Run> &runs, int T, int rm, int rx, short *lo) {
    int n = 0, i = 0;
    for (const Run &u : runs) {
        int nb = 0;
        if (!u.special) {
            const int m = std::min(rm, std::max(1, T / RS_COST_LEAN));
            nb = (u.len + m - 1) / m;
            if (u.len / nb < rm - RS_SPARE) nb = 0;
        }
        if (nb == 0) {
            const int m = std::min(rx, std::max(1, T / RS_COST_SPECIAL));
            nb = (u.len + m - 1) / m;
        }
        if (lo)
            for (int b = 0; b < nb; ++b) lo[n + b] = (short)(i + (int)((long)u.len * b / nb));
        n += nb;
        i += u.len;
    }
    return n;
}

// The least band cost T with which the bands number at most avail; -1 when none does.
int rs_threshold(const std::vector<Run> &runs, int avail, int rm, int rx) {
    int hi_t = rm * RS_COST_SPECIAL;  // every band as long as it may be
    if (avail < 1 || rs_bands(runs, hi_t, rm, rx, nullptr) > avail) return -1;
    int lo_t = RS_COST_LEAN - 1;        // one lean row per band is the least
    while (hi_t - lo_t > 1) {
        const int mid = (lo_t + hi_t) / 2;
        if (rs_bands(runs, mid, rm, rx, nullptr) <= avail) hi_t = mid;
        else lo_t = mid;
    }
    return hi_t;
}

bool rs_inst_ok(const LensInst2D &g) {
    if (g.nx < 3 || g.ny < 3 || g.nx > 32767 || g.pitch < g.ny || (g.pitch % 32)) return false;
    if (!g.f[0] || !g.f[1] || !g.f[2] || !g.c[0] || !g.c[1] || (!g.c[2]) != (!g.c[3])) return false;
    if (!lens_profile_ok(g.ax.e, g.nx) || !lens_profile_ok(g.ax.h, g.nx - 1) || !lens_profile_ok(g.ay.e, g.ny) ||
        !lens_profile_ok(g.ay.h, g.ny - 1))
        return false;
    if (g.src.ix >= 0 && (!g.src.amp || !g.src.ph1 || !g.src.ph2 || g.src.ix + 1 >= g.nx)) return false;
    const LensProfile *strip[2][4] = {{&g.ay.h, &g.ax.h, &g.ax.e, &g.ay.e}, {&g.ax.h, &g.ay.h, &g.ay.e, &g.ax.e}};
    for (int q = 0; q < 4; ++q)
        if (!lens_psi_ok(*strip[g.pol][q], g.psi[q])) return false;
    return true;
}

LensInst2D inst_of(const LensTE2D &g) {
    LensInst2D v{};
    v.pol = 0; v.nx = g.nx; v.ny = g.ny; v.pitch = g.pitch;
    v.f[0] = g.ez; v.f[1] = g.hx; v.f[2] = g.hy;
    v.c[0] = g.ce_e; v.c[1] = g.ce_h;
    v.ch = g.ch; v.ax = g.ax; v.ay = g.ay;
    v.psi[0] = g.psi_hxy; v.psi[1] = g.psi_hyx; v.psi[2] = g.psi_ezx; v.psi[3] = g.psi_ezy;
    for (int q = 0; q < 4; ++q) v.pec[q] = g.pec[q];
    v.src = g.src;
    v.src.nj = std::min(v.src.nj, g.ny);
    return v;
}

LensInst2D inst_of(const LensTM2D &g) {
    LensInst2D v{};
    v.pol = 1; v.nx = g.nx; v.ny = g.ny; v.pitch = g.pitch;
    v.f[0] = g.ex; v.f[1] = g.ey; v.f[2] = g.hz;
    v.c[0] = g.ca_x; v.c[1] = g.ca_y; v.c[2] = g.da_x; v.c[3] = g.da_y;
    v.ch = g.ch; v.ax = g.ax; v.ay = g.ay;
    v.psi[0] = g.psi_hzx; v.psi[1] = g.psi_hzy; v.psi[2] = g.psi_exy; v.psi[3] = g.psi_eyx;
    for (int q = 0; q < 4; ++q) v.pec[q] = g.pec[q];
    v.src = g.src;
    v.src.nj = std::min(v.src.nj, g.ny - 1);
    return v;
}

struct Plan {
    const RsForm *form;
    bool wide;
    int nbands, ncol, nc;
};

// Let a kernel's launches ask for any dynamic shared memory the device has.  The limit
// belongs to the kernel, whichever thread launches it: every call sets the same one, so no
// call takes from another thread's plan what it was made with.
bool rs_allow(const void *kernel, int smax) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smax) == cudaSuccess;
}

// Band plan of a grid on this device: the row template and register split, the CTA count
// and (when lo is not NULL) the first row of every band.  The bands minimise the largest
// band cost, weighed by the CTAs that share an SM.  LENS_ERR_SIZE when the grid does not
// fit on the chip.  nbox: detector boxes of the epilogue.
int plan_(const LensInst2D &g, int nbox, Plan &p, short *lo) {
    if (!rs_inst_ok(g)) return LENS_ERR_SIZE;  // the step by step entries name what is wrong
    if (g.ny > 64 * RS_MAXW || g.ay.e.lo + g.ay.e.hi > RS_MAXWY || g.ay.h.lo + g.ay.h.hi > RS_MAXWY) return LENS_ERR_SIZE;
    p.nc = g.c[2] ? 4 : 2;
    p.ncol = (g.ny + 31) / 32 * 32;
    const int W = (p.ncol + 63) / 64;
    int dev = 0, nsm = 0, smax = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess)
        return LENS_ERR_CUDA;
    if (!coop) return LENS_ERR_SIZE;
    const std::vector<Run> runs = rs_runs(g);
    // every (template, split, CTAs per SM) by its cost, the cheapest that is resident wins;
    // only kernels on the way there are asked for (a first question loads the kernel)
    struct Cand {
        long cost;
        int f, wide, c, T;
    };
    std::vector<Cand> cand;
    for (int t = 0; t < RS_NRM; ++t) {
        const RsForm &f = RS_FORMS[t];
        if (rs_smem(f, p.ncol, p.nc, nbox, false) > (size_t)smax) continue;
        for (int c = 1; c <= 16 / W || c == 1; ++c) {
            const int avail = (int)std::min((long)c * nsm, (long)RS_MAXCTA);
            const int T = rs_threshold(runs, avail, f.rm, f.rx);
            for (int wd = W > 8 ? 1 : 0; T > 0 && wd < 2; ++wd)
                cand.push_back(Cand{(long)T * (100 + RS_SHARE * (c - 1)), t, wd, c, T});
            if ((long)c * nsm >= RS_MAXCTA) break;
        }
    }
    std::stable_sort(cand.begin(), cand.end(), [](const Cand &a, const Cand &b) { return a.cost < b.cost; });
    for (const Cand &c : cand) {
        const RsForm &f = RS_FORMS[c.f];
        const void *k = f.kernel(c.wide);
        const size_t sm = rs_smem(f, p.ncol, p.nc, nbox, false);
        int per = 0;
        if (!rs_allow(k, smax) ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, 32 * W, sm) != cudaSuccess)
            return LENS_ERR_CUDA;
        if (per < c.c) continue;
        p.form = &f;
        p.wide = c.wide;
        p.nbands = rs_bands(runs, c.T, f.rm, f.rx, lo);
        return LENS_OK;
    }
    return LENS_ERR_SIZE;
}

// No exception passes a C entry: host memory that ran out is a size that does not fit.
int plan(const LensInst2D &g, int nbox, Plan &p, short *lo) {
    try {
        const int st = plan_(g, nbox, p, lo);
        if (st != LENS_OK) cudaGetLastError();
        return st;
    } catch (const std::exception &) {
        return LENS_ERR_SIZE;
    }
}

size_t scratch_bytes(const Plan &p) { return (size_t)p.nbands * 4 * ((p.ncol + 63) / 64 * 64) * sizeof(unsigned long long); }

// The most scratch a call may need.  A call's plan depends on its boxes, whose sums take
// shared memory: with fewer of them more CTAs may share an SM, with more and shorter bands.
size_t most_scratch(const LensInst2D &g) {
    size_t most = 0;
    for (int nbox = 0; nbox <= LENS_MAX_BOX; ++nbox) {
        Plan p{};
        if (plan(g, nbox, p, nullptr) == LENS_OK) most = std::max(most, scratch_bytes(p));
    }
    return most;
}

int rows_of(const LensInst2D &g, int nbox, int *rows, int *threads, int *bands) {
    if (nbox < 0 || nbox > LENS_MAX_BOX || !rows || !threads || !bands) return LENS_ERR_ARG;
    Plan p{};
    const int st = plan(g, nbox, p, nullptr);
    if (st != LENS_OK) return st;
    *rows = p.form->rm;
    *threads = p.wide ? 384 : 256;
    *bands = p.nbands;
    return LENS_OK;
}

int run(const LensInst2D &g, const LensEpi2D *ep, const LensStepTable *tab, int n0, int nsteps, void *scratch, size_t bytes,
        int *err, void *stream, unsigned tries, int wd) {
    if (!scratch || !err || nsteps < 1 || !lens_table_ok(tab, n0, nsteps)) return LENS_ERR_SIZE;
    GPlan pl{};
    pl.g = g;
    pl.ep.iavg_n0 = 1 << 30;
    if (ep) pl.ep = *ep;
    const LensEpi2D &e = pl.ep;
    // what the step by step kernels alone carry, and what they refuse
    if (e.dft_raw || e.ex2 || e.nsx != 0 || e.nbox < 0 || e.nbox > LENS_MAX_BOX || (e.nbox > 0 && !e.box_acc) ||
        e.nplane < 0 || e.nplane > LENS_MAX_PLANE || (e.nplane > 0 && !e.plane_acc) || (e.dft_ex && g.pol == 0))
        return LENS_ERR_SIZE;
    lens_clip_boxes(pl.ep, g.nx, g.ny);
    for (int q = 0; q < e.nplane; ++q)
        if (e.plane[q] < 1 || e.plane[q] > g.nx - 2) return LENS_ERR_SIZE;
    if ((e.dft || e.dft_ex || e.dft_prev || e.nplane > 0) && (!tab->pe || !tab->ph)) return LENS_ERR_SIZE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return LENS_ERR_SIZE;  // a captured span stays a sequence of plain launches
    }
    Plan p{};
    int st = plan(g, e.nbox, p, pl.lo);
    if (st != LENS_OK) return st;
    if (bytes < scratch_bytes(p)) return LENS_ERR_SIZE;
    const int W = (p.ncol + 63) / 64;
    pl.nbands = p.nbands;
    pl.nc = p.nc;
    pl.ncol = p.ncol;
    pl.tries = tries;
    pl.wd_cta = -1;
    if (wd) {
        if (p.nbands < 2 || nsteps < 3) return LENS_ERR_ARG;
        pl.wd_cta = 1;
    }
    // the node DFT's sums sit in shared memory where that leaves every CTA resident
    const void *kern = p.form->kernel(p.wide);
    size_t sm = rs_smem(*p.form, p.ncol, p.nc, e.nbox, false);
    // (not where another sum runs on the same array: that one is added to in global memory)
    if (e.dft && e.dft != e.dft_prev && e.dft != e.dft_ex && e.dft_n0 < n0 + nsteps && e.dft_n1 > n0) {
        int dev = 0, smax = 0, nsm = 0, per = 0;
        const size_t smd = rs_smem(*p.form, p.ncol, p.nc, e.nbox, true);
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && smd <= (size_t)smax &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 32 * W, smd) == cudaSuccess &&
            (long)per * nsm >= p.nbands) {
            pl.hold = 1;
            sm = smd;
        }
    }
    if (cudaMemsetAsync(scratch, 0, scratch_bytes(p), s) != cudaSuccess) return LENS_ERR_CUDA;
    LensStepTable t = *tab;
    unsigned long long *halo = static_cast<unsigned long long *>(scratch);
    void *args[] = {(void *)&pl, (void *)&t, (void *)&n0, (void *)&nsteps, (void *)&halo, (void *)&err};
    if (cudaLaunchCooperativeKernel(kern, dim3(p.nbands), dim3(32, W), args, sm, s) != cudaSuccess) {
        cudaGetLastError();
        return LENS_ERR_CUDA;
    }
    return lens_cuda_status();
}

}  // namespace

extern "C" int lens_te2d_resident_rows(const LensTE2D *g, int nbox, int *rows, int *threads, int *bands) {
    return g ? rows_of(inst_of(*g), nbox, rows, threads, bands) : LENS_ERR_ARG;
}

extern "C" int lens_tm2d_resident_rows(const LensTM2D *g, int nbox, int *rows, int *threads, int *bands) {
    return g ? rows_of(inst_of(*g), nbox, rows, threads, bands) : LENS_ERR_ARG;
}

extern "C" size_t lens_te2d_resident_bytes(const LensTE2D *g) { return g ? most_scratch(inst_of(*g)) : 0; }

extern "C" size_t lens_tm2d_resident_bytes(const LensTM2D *g) { return g ? most_scratch(inst_of(*g)) : 0; }

extern "C" int lens_te2d_resident(const LensTE2D *g, const LensStepTable *tab, const LensEpi2D *ep, int n0, int nsteps,
                                  void *scratch, size_t bytes, int *err, void *stream) {
    return g ? run(inst_of(*g), ep, tab, n0, nsteps, scratch, bytes, err, stream, RS_TRIES, 0) : LENS_ERR_ARG;
}

extern "C" int lens_tm2d_resident(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep, int n0, int nsteps,
                                  void *scratch, size_t bytes, int *err, void *stream) {
    return g ? run(inst_of(*g), ep, tab, n0, nsteps, scratch, bytes, err, stream, RS_TRIES, 0) : LENS_ERR_ARG;
}

extern "C" int lens_te2d_resident_watchdog_test(const LensTE2D *g, const LensStepTable *tab, int n0, int nsteps,
                                                void *scratch, size_t bytes, int *err, void *stream) {
    return g ? run(inst_of(*g), nullptr, tab, n0, nsteps, scratch, bytes, err, stream, 1024, 1) : LENS_ERR_ARG;
}

extern "C" int lens_tm2d_resident_watchdog_test(const LensTM2D *g, const LensStepTable *tab, const LensEpi2D *ep, int n0,
                                                int nsteps, void *scratch, size_t bytes, int *err, void *stream) {
    return g ? run(inst_of(*g), ep, tab, n0, nsteps, scratch, bytes, err, stream, 1024, 1) : LENS_ERR_ARG;
}
