// C ABI of odtbrain_gb300 (declared in include/odtbrain_gb300.h).
//
// Plan creation turns the FP64 host constants of the reference
// (odtbrain/_alg3d_bpp.py:317-437; _alg3d_bppt.py:680-820) into the FP32
// device tables the stage kernels read, and sizes the angle batches.
// Execution runs, per batch of angles, the filter stages into coefficient
// slabs and then the resampling/accumulation stage.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/odtbrain_gb300.h"
#include "odt_internal.cuh"

using odt::FilterTables;
using odt::RotParams;
using odt::StageParams;

namespace {

thread_local std::string g_last_error;

odt_status fail(odt_status st, const std::string &msg)
{
    g_last_error = msg;
    return st;
}

odt_status cuda_fail(cudaError_t e, const char *where)
{
    return fail(ODT_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

// Test hook (odt_debug_set_table_alloc_limit): plan creation refuses table
// allocations above this many bytes (0: no limit).
uint64_t g_table_alloc_limit = 0;
std::mutex g_debug_mutex;

constexpr uint64_t kDefaultWorkspace = 16ull << 30;   // 16 GiB of slabs, chunk buffers etc.
// Column-stage output chunk: planes and bytes at most.  Large chunks mean few
// launches with full waves.  Step with 256 / 512 / 1024 / 2048 / 4096 planes:
// 256^3 from 200 views 28.6 / 27.8 / 27.0 / 26.6 / 26.6 ms, 128^3 from 90
// 2.15 / 2.03 / 1.88 / 1.82 / 1.92 ms.
constexpr size_t kMaxJobs = 2048;
constexpr uint64_t kPlaneBudget = 2048ull << 20;
constexpr size_t kAlign = 256;

size_t align_up(size_t v) { return (v + kAlign - 1) / kAlign * kAlign; }

// The sampled centred B-spline of order 2..5, t[0] + t[1] (z + 1/z) +
// t[2] (z^2 + 1/z^2): [1 6 1]/8, [1 4 1]/6, [1 76 230 76 1]/384,
// [1 26 66 26 1]/120 (the kernel scipy.ndimage's prefilter inverts).
struct SplineTaps {
    double t[3];
    int npoles;  // 1 for orders 2, 3; 2 for orders 4, 5
};
SplineTaps spline_taps(int order)
{
    switch (order) {
    case 2: return {{6.0 / 8.0, 1.0 / 8.0, 0.0}, 1};
    case 3: return {{4.0 / 6.0, 1.0 / 6.0, 0.0}, 1};
    case 4: return {{230.0 / 384.0, 76.0 / 384.0, 1.0 / 384.0}, 2};
    default: return {{66.0 / 120.0, 26.0 / 120.0, 1.0 / 120.0}, 2};
    }
}

// Transfer function Bhat(w) of the sampled B-spline.
double spline_bhat(int order, double w)
{
    const SplineTaps T = spline_taps(order);
    return T.t[0] + 2.0 * T.t[1] * std::cos(w) + 2.0 * T.t[2] * std::cos(2.0 * w);
}

// Poles of the prefilter (the roots of the kernel's polynomial inside the
// unit circle), largest magnitude first.
int spline_poles(int order, double *z)
{
    const SplineTaps T = spline_taps(order);
    if (T.npoles == 1) {
        // t1 z^2 + t0 z + t1 = 0
        z[0] = (-T.t[0] + std::sqrt(T.t[0] * T.t[0] - 4.0 * T.t[1] * T.t[1])) / (2.0 * T.t[1]);
        return 1;
    }
    // with s = z + 1/z: t2 s^2 + t1 s + (t0 - 2 t2) = 0, then z^2 - s z + 1 = 0;
    // the root inside the unit circle as 2 / (s - sqrt(s^2 - 4)) (s < -2)
    const double disc = std::sqrt(T.t[1] * T.t[1] - 4.0 * T.t[2] * (T.t[0] - 2.0 * T.t[2]));
    const double s1 = (-T.t[1] + disc) / (2.0 * T.t[2]), s2 = (-T.t[1] - disc) / (2.0 * T.t[2]);
    z[0] = 2.0 / (s1 - std::sqrt(s1 * s1 - 4.0));
    z[1] = 2.0 / (s2 - std::sqrt(s2 * s2 - 4.0));
    return 2;
}

// Boundary solve of the prefilter folded into the transforms.  A line of n
// samples whose Fourier components were divided by Bhat (the particular
// solution c_p, known also beyond the line's ends) becomes scipy's
// mirror-boundary prefiltered line c = c_p + h with
//   h[k] = sum_i A_i z_i^k + B_i z_i^(n-1-k),
// where the coefficients follow from the kernel's equations at the first
// and last npoles samples, written with mirrored neighbours:
//   (A_1..A_np, B_1..B_np) = K (d_1L..d_npL, d_1R..d_npR),
//   d_mL = c_p[m] - c_p[-m],   d_mR = c_p[n-1-m] - c_p[n-1+m].
// K (row-major, 2np x 2np) is returned; false if the system is singular.
bool boundary_matrix(int order, int n, double *K)
{
    const SplineTaps T = spline_taps(order);
    double z[2];
    const int np = spline_poles(order, z), n2 = 2 * np;
    double M[4][4] = {}, R[4][4] = {};
    auto mirror = [&](int m) {
        if (n == 1)
            return 0;
        const int P = 2 * n - 2;
        m = std::abs(m) % P;
        return m < n ? m : P - m;
    };
    auto add_h = [&](int eq, double t, int k) {  // t * h[k]
        for (int i = 0; i < np; ++i) {
            M[eq][i] += t * std::pow(z[i], k);
            M[eq][np + i] += t * std::pow(z[i], n - 1 - k);
        }
    };
    int eq = 0;
    for (int q = 0; q < np; ++q, ++eq) {  // samples q (left) ...
        for (int k = -np; k <= np; ++k) {
            const int m = q + k;
            add_h(eq, T.t[std::abs(k)], mirror(m));
            if (m < 0)
                R[eq][-m - 1] -= T.t[std::abs(k)];
        }
    }
    for (int q = 0; q < np; ++q, ++eq) {  // ... and n-1-q (right)
        for (int k = -np; k <= np; ++k) {
            const int m = n - 1 - q + k;
            add_h(eq, T.t[std::abs(k)], mirror(m));
            if (m > n - 1)
                R[eq][np + (m - (n - 1)) - 1] -= T.t[std::abs(k)];
        }
    }
    // K = M^-1 R by Gauss-Jordan elimination with partial pivoting
    for (int c = 0; c < n2; ++c) {
        int piv = c;
        for (int r = c + 1; r < n2; ++r)
            if (std::fabs(M[r][c]) > std::fabs(M[piv][c]))
                piv = r;
        if (!(std::fabs(M[piv][c]) > 1e-300))
            return false;
        for (int j = 0; j < n2; ++j) {
            std::swap(M[c][j], M[piv][j]);
            std::swap(R[c][j], R[piv][j]);
        }
        const double inv = 1.0 / M[c][c];
        for (int j = 0; j < n2; ++j) {
            M[c][j] *= inv;
            R[c][j] *= inv;
        }
        for (int r = 0; r < n2; ++r) {
            if (r == c)
                continue;
            const double f = M[r][c];
            for (int j = 0; j < n2; ++j) {
                M[r][j] -= f * M[c][j];
                R[r][j] -= f * R[c][j];
            }
        }
    }
    for (int r = 0; r < n2; ++r)
        for (int j = 0; j < n2; ++j) {
            K[r * n2 + j] = R[r][j];
            if (!std::isfinite(R[r][j]))
                return false;
        }
    return true;
}

// Coefficients of the one-pole boundary solve in the form the adjoint
// kernels use: with d0 = u[-1] - u[1] and d1 = u[n] - u[n-2], the
// correction A z^k + B z^(n-1-k) has A = ca*d0 + cb*d1 and B = ca*d1 + cb*d0.
void boundary_solve(double z, int n, double *ca, double *cb)
{
    const double a = z - 1.0 / z;
    const double b = std::pow(z, n - 2) - std::pow(z, n);
    const double det = a * a - b * b;
    *ca = a / det;
    *cb = -b / det;
}

double fftfreq_rad(int k, int n)
{
    // 2*pi*numpy.fft.fftfreq(n)[k]
    const int half = (n - 1) / 2;
    const int m = k <= half ? k : k - n;
    return 2.0 * M_PI * (double)m / (double)n;
}

}  // namespace

int odt::set_error(int status, const char *msg)
{
    return (int)fail((odt_status)status, msg ? msg : "");
}

namespace {
// Batching and workspace of an execution over `units` slabs.
struct Layout {
    int units, batch;  // slabs (angles, or units of opposite views), slabs per batch
    int spu;           // spectrum slots per slab: 1, or 2 with opposite views
    int jobs;          // (slab, plane) jobs per column/row launch
    size_t off_spec, off_T, off_Tab, off_slab, off_comp, off_rot, ws_bytes;
    size_t off_Qg, off_W, off_Pg, off_vT, adj_ws_bytes;  // adjoint-only regions after ws_bytes
};
}  // namespace

struct odt_bpp3d_plan {
    odt_bpp3d_desc d;
    int device;      // CUDA device the tables, events and stream belong to
    int nz;
    int even;        // filter and propagator phase are even in kx (opposite views can be paired)
    Layout lay;      // one angle per slab
    double bx_ca, bx_cb, by_ca, by_cb;  // one-pole solve in the adjoint's form
    int npoles;                         // prefilter poles: 0, 1 or 2
    float kx_solve[16], ky_solve[16];   // boundary_matrix of x and y lines
    int kx_zero_lo, kx_zero_hi;  // all-zero spectrum columns [lo, hi)
    int ky_zero_lo, ky_zero_hi;  // all-zero spectrum rows [lo, hi)
    int col_slots;               // resident column-stage CTAs (occupancy x SMs)
    // device tables (one allocation)
    void *d_tables;
    FilterTables tab, tabt;
    int *d_status;
};

namespace {

// The plan's device must be the current one: its tables, events and second
// stream belong to that device.
odt_status check_device(const odt_bpp3d_plan *plan)
{
    int dev = -1;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaGetDevice");
    if (dev != plan->device) {
        char buf[128];
        snprintf(buf, sizeof buf, "plan was created on CUDA device %d but device %d is current", plan->device,
                 dev);
        return fail(ODT_ERR_INVALID_ARGUMENT, buf);
    }
    return ODT_OK;
}

StageParams stage_params(const odt_bpp3d_plan *p)
{
    StageParams P;
    const odt_bpp3d_desc &d = p->d;
    P.A = d.num_angles;
    P.ny = d.ny;
    P.nx = d.nx;
    P.nz = p->nz;
    P.lNy = d.pad_ny;
    P.lNx = d.pad_nx;
    P.padyl = d.pad_y_left;
    P.padxl = d.pad_x_left;
    P.pad_mode = d.pad_mode;
    P.padval = make_float2((float)d.padval_re, (float)d.padval_im);
    P.order = d.intp_order;
    P.tilted = d.geometry == ODT_GEOM_AFFINE3D;
    P.in_c128 = d.input_dtype == ODT_INPUT_C128;
    P.kx_zero_lo = p->kx_zero_lo;
    P.kx_zero_hi = p->kx_zero_hi;
    P.ky_zero_lo = p->ky_zero_lo;
    P.ky_zero_hi = p->ky_zero_hi;
    P.bx_ca = (float)p->bx_ca;
    P.bx_cb = (float)p->bx_cb;
    P.by_ca = (float)p->by_ca;
    P.by_cb = (float)p->by_cb;
    P.npoles = p->npoles;
    for (int i = 0; i < 16; ++i) {
        P.kxs[i] = p->kx_solve[i];
        P.kys[i] = p->ky_solve[i];
    }
    P.ypitch = odt::yaxis_slab_pitch(d.ny);
    P.col_slots = p->col_slots;
    P.zshift = (float)d.z_shift;
    P.tab = p->tab;
    P.tabt = p->tabt;
    P.gain = nullptr;
    P.again = nullptr;
    P.status = p->d_status;
    P.units = nullptr;
    P.trow0 = P.trows = 0;
    return P;
}

// Spectrum slots per batch: the spectrum, boundary and padding kernels have them
// on a grid's y or z extent.
constexpr int kMaxSlots = 65535;

// The largest batch of slabs (and column-stage chunk) whose workspace fits
// the plan's limit; one slab per batch with a shrunken chunk where none does.
Layout make_layout(const odt_bpp3d_plan *p, int units, int spu)
{
    const odt_bpp3d_desc &d = p->d;
    const int lNy = d.pad_ny, lNx = d.pad_nx, nz = p->nz, np = p->npoles;
    const bool tilted = d.geometry == ODT_GEOM_AFFINE3D;
    // one job's column-stage output: transposed [row][lNy] in the forward
    // execution, [y][lNx] in the adjoint
    const size_t plane_row_bytes =
        std::max((size_t)odt::transposed(stage_params(p)).trows * lNy, (size_t)d.ny * lNx) * 8;
    const size_t spec_bytes = (size_t)spu * lNy * lNx * 8;           // one slab's spectra
    // one coefficient slab [z][x][ypitch] (the adjoint's slab gradients
    // [y][z][x] fit too).  The row spectra, dead before the slab is written,
    // share its place.
    const size_t slab_bytes = std::max((size_t)nz * odt::yaxis_slab_pitch(d.ny) * d.nx * 8, spec_bytes);
    // one slab's z-boundary rows (not transposed for single-row planes)
    const size_t tab_bytes = (size_t)2 * np * std::max((size_t)d.nx * lNy, (size_t)d.ny * lNx) * 8;
    const size_t vol_bytes = (size_t)nz * d.ny * d.nx * 8;           // compensation buffer
    const uint64_t limit = d.workspace_limit ? d.workspace_limit : kDefaultWorkspace;
    // the chunk buffer takes at most a quarter of the limit, so tight limits
    // (save_memory) keep room for a batch of slabs.  A quarter against an eighth:
    // 64^3 from 60 single views within 16 / 64 MiB 4.17 -> 2.19 / 1.00 -> 0.71 ms,
    // 256^3 from 100 within 1 GiB 34.4 -> 33.1 ms.
    const uint64_t plane_budget = std::min<uint64_t>(kPlaneBudget, limit / 4);
    const size_t jobs_cap = std::max<size_t>(16, std::min<size_t>(kMaxJobs, plane_budget / plane_row_bytes));
    auto layout = [&](int batch, size_t jobs) -> Layout {
        Layout y{};
        y.units = units;
        y.batch = batch;
        y.spu = spu;
        y.jobs = (int)jobs;
        const int nbatches = (units + batch - 1) / batch;
        size_t w = 0;
        y.off_spec = w; w = align_up(w + (size_t)batch * spec_bytes);
        y.off_T = w; w = align_up(w + jobs * plane_row_bytes);
        y.off_Tab = w; w = align_up(w + (size_t)batch * tab_bytes);
        y.off_slab = w; w = align_up(w + (size_t)batch * slab_bytes);
        y.off_comp = w; w = align_up(w + (nbatches > 1 ? vol_bytes : 0));
        y.off_rot = w;
        w = align_up(w + odt::rotate_scratch_bytes(batch, d.ny, d.nx, nz, tilted ? 1 : 0));
        y.ws_bytes = w;
        const size_t spec_b = (size_t)batch * spec_bytes;
        y.off_Qg = w; w = align_up(w + spec_b);
        y.off_W = w; w = align_up(w + spec_b);
        y.off_Pg = w; w = align_up(w + spec_b);
        // the volume gradient in the [z][x][y] order (y-axis adjoint)
        y.off_vT = w; w = align_up(w + vol_bytes);
        y.adj_ws_bytes = w;
        return y;
    };
    auto jobs_for = [&](int batch) {
        size_t jobs = std::min((size_t)batch * nz, jobs_cap);
        return jobs >= 16 ? jobs / 16 * 16 : jobs;
    };
    const int most = std::min(units, kMaxSlots / spu);
    int best = 0;
    for (int lo = 1, hi = most; lo <= hi;) {  // ws grows with the batch
        const int mid = lo + (hi - lo) / 2;
        if (layout(mid, jobs_for(mid)).ws_bytes <= limit) {
            best = mid;
            lo = mid + 1;
        } else {
            hi = mid - 1;
        }
    }
    // a single batch needs no compensation buffer, so it can fit when a
    // slightly smaller batch does not
    if (best < units && most == units && layout(units, jobs_for(units)).ws_bytes <= limit)
        best = units;
    if (best > 0)
        return layout(best, jobs_for(best));
    // one slab per batch; shrink the column-stage chunk toward the limit, to
    // two planes (launches of one plane are twice as many: 256^3 from 100 views
    // within 256 MiB 516 ms with one, 276 with two)
    size_t jobs = jobs_for(1);
    while (jobs > 2 && layout(1, jobs).ws_bytes > limit)
        jobs = jobs > 16 ? jobs - 16 : jobs - 1;
    return layout(1, jobs);
}

// The layout of an execution over units of opposite views; an error when the
// plan cannot pair views.
odt_status pair_layout(const odt_bpp3d_plan *plan, int num_units, Layout *y)
{
    if (!plan->even)
        return fail(ODT_ERR_UNSUPPORTED, "opposite views need the rotation about y and tables even in kx");
    // Nearest neighbour jumps where a coordinate is a half integer, and the
    // views' coordinates c and n-1-c round such halves (multiples of 30
    // degrees at odd widths, of 45 degrees at even ones) to different samples:
    // with the first view's samples for both, 9e-3 rel-L2 at 33^3 from 12 views.
    if (plan->d.intp_order == 0)
        return fail(ODT_ERR_UNSUPPORTED, "opposite views need spline order 1 or more");
    if (num_units < 1 || num_units > plan->d.num_angles)
        return fail(ODT_ERR_INVALID_ARGUMENT, "need 1 <= num_units <= num_angles");
    *y = make_layout(plan, num_units, 2);
    const uint64_t limit = plan->d.workspace_limit ? plan->d.workspace_limit : kDefaultWorkspace;
    if (y->ws_bytes > limit)
        return fail(ODT_ERR_UNSUPPORTED, "the workspace limit holds no unit of opposite views");
    return ODT_OK;
}

odt_status validate(const odt_bpp3d_desc *d)
{
    if (!d)
        return fail(ODT_ERR_INVALID_ARGUMENT, "descriptor is NULL");
    if (d->num_angles < 1 || d->ny < 1 || d->nx < 2)
        return fail(ODT_ERR_INVALID_ARGUMENT, "need num_angles >= 1, ny >= 1, nx >= 2");
    if (d->pad_ny < d->ny || d->pad_nx < d->nx || d->pad_y_left < 0 || d->pad_x_left < 0 ||
        d->pad_y_left + d->ny > d->pad_ny || d->pad_x_left + d->nx > d->pad_nx)
        return fail(ODT_ERR_INVALID_ARGUMENT, "inconsistent padding geometry");
    if (d->pad_mode < ODT_PAD_NONE || d->pad_mode > ODT_PAD_RAMP)
        return fail(ODT_ERR_INVALID_ARGUMENT, "unknown pad_mode");
    if (d->pad_mode == ODT_PAD_NONE && (d->pad_ny != d->ny || d->pad_nx != d->nx))
        return fail(ODT_ERR_INVALID_ARGUMENT, "pad_mode NONE needs unpadded sizes");
    if (d->geometry != ODT_GEOM_Y_AXIS && d->geometry != ODT_GEOM_AFFINE3D)
        return fail(ODT_ERR_INVALID_ARGUMENT, "unknown geometry");
    if (d->input_dtype != ODT_INPUT_C64 && d->input_dtype != ODT_INPUT_C128)
        return fail(ODT_ERR_INVALID_ARGUMENT, "unknown input dtype");
    if (d->intp_order < 0 || d->intp_order > 5)
        return fail(ODT_ERR_INVALID_ARGUMENT, "intp_order must be in 0..5");
    if (d->intp_order >= 4 && (d->nx < 4 || (d->geometry == ODT_GEOM_AFFINE3D && d->ny > 1 && d->ny < 4)))
        return fail(ODT_ERR_UNSUPPORTED, "spline orders 4 and 5 need lines of at least 4 samples");
    if (!std::isfinite(d->z_shift) || std::fabs(d->z_shift) > 1.0 || 2.0 * d->z_shift != std::rint(2.0 * d->z_shift))
        return fail(ODT_ERR_INVALID_ARGUMENT, "z_shift must be 0, +-0.5 or +-1");
    if (!odt::line_size_supported(d->pad_nx) || !odt::line_size_supported(d->pad_ny))
        return fail(ODT_ERR_UNSUPPORTED,
                    "FFT length must be a power of two in [64, 4096] or any length <= 1024");
    if (!d->filter || !d->kz_phase)
        return fail(ODT_ERR_INVALID_ARGUMENT, "filter and kz_phase tables are required");
    // the resampling kernels address one angle's slab [z][x][y pitch] with
    // 32-bit element offsets
    if ((long long)d->nx * d->nx * odt::yaxis_slab_pitch(d->ny) >= (1ll << 31))
        return fail(ODT_ERR_UNSUPPORTED, "one angle's coefficient slab must hold fewer than 2^31 elements");
    return ODT_OK;
}

}  // namespace

extern "C" {

const char *odt_status_string(odt_status s)
{
    switch (s) {
    case ODT_OK: return "ok";
    case ODT_ERR_INVALID_ARGUMENT: return "invalid argument";
    case ODT_ERR_UNSUPPORTED: return "unsupported";
    case ODT_ERR_CUDA: return "CUDA error";
    case ODT_ERR_OUT_OF_MEMORY: return "out of memory";
    case ODT_ERR_DEVICE_CHECK: return "device-side check failed";
    }
    return "unknown status";
}

const char *odt_last_error(void) { return g_last_error.c_str(); }

odt_status odt_bpp3d_plan_create(const odt_bpp3d_desc *desc, odt_bpp3d_plan **out)
{
    if (!out)
        return fail(ODT_ERR_INVALID_ARGUMENT, "plan output pointer is NULL");
    *out = nullptr;
    odt_status st = validate(desc);
    if (st != ODT_OK)
        return st;
    odt_bpp3d_plan *p = new (std::nothrow) odt_bpp3d_plan();
    if (!p)
        return fail(ODT_ERR_OUT_OF_MEMORY, "host allocation failed");
    p->d = *desc;
    p->d.filter = nullptr;
    p->d.kz_phase = nullptr;
    const odt_bpp3d_desc &d = p->d;
    const int lNy = d.pad_ny, lNx = d.pad_nx, nz = d.nx;
    p->nz = nz;
    const int order = d.intp_order;
    const bool pf = order >= 2;
    const bool tilted = d.geometry == ODT_GEOM_AFFINE3D;
    const size_t K = (size_t)lNy * lNx;

    // ---- FP64 host tables -> FP32 device tables
    // prefilter (order >= 2): npoles poles; per pole the z-boundary tables
    // alpha_i, beta_i (planes) and the powers z_i^m
    double zpole[2] = {0.0, 0.0};
    const int np = pf ? spline_poles(order, zpole) : 0;
    p->npoles = np;
    std::vector<float2> G(K), W(K), S(K), AL((size_t)2 * K), BE((size_t)2 * K), twx(lNx), twy(lNy);
    std::vector<float> zp((size_t)2 * odt::ZPOW_N, 0.f);
    double Kz[16] = {0}, Kx[16] = {0}, Ky[16] = {0};
    std::memset(p->kx_solve, 0, sizeof p->kx_solve);
    std::memset(p->ky_solve, 0, sizeof p->ky_solve);
    if (pf) {
        bool ok = boundary_matrix(order, nz, Kz) && boundary_matrix(order, d.nx, Kx);
        if (d.ny >= 2)
            ok = ok && boundary_matrix(order, d.ny, Ky);
        if (!ok) {
            delete p;
            return fail(ODT_ERR_UNSUPPORTED, "the spline prefilter's boundary system is singular for these sizes");
        }
        for (int i = 0; i < 16; ++i) {
            p->kx_solve[i] = (float)Kx[i];
            p->ky_solve[i] = (float)Ky[i];
        }
        if (np == 1) {
            // the adjoint kernels' form of the one-pole solve
            boundary_solve(zpole[0], d.nx, &p->bx_ca, &p->bx_cb);
            if (d.ny >= 2)
                boundary_solve(zpole[0], d.ny, &p->by_ca, &p->by_cb);
        }
        for (int i = 0; i < np; ++i) {
            double zz = 1.0;
            for (int m = 0; m < odt::ZPOW_N; ++m) {
                zp[(size_t)i * odt::ZPOW_N + m] = (float)zz;
                zz *= zpole[i];
            }
        }
    }
    // positions of the first and last planes (the z-prefilter boundary terms
    // are per-frequency functions of them)
    const double z_first = 0.0 - 0.5 * nz + d.z_shift, z_last = (double)(nz - 1) - 0.5 * nz + d.z_shift;
    for (int ky = 0; ky < lNy; ++ky) {
        // (scipy leaves an axis of length 1 unfiltered: no y prefilter, and
        // its boundary coefficients stay zero, for a single detector row)
        const double iby = (pf && tilted && d.ny >= 2) ? 1.0 / spline_bhat(order, fftfreq_rad(ky, lNy)) : 1.0;
        for (int kx = 0; kx < lNx; ++kx) {
            const size_t k = (size_t)ky * lNx + kx;
            const double ibx = pf ? 1.0 / spline_bhat(order, fftfreq_rad(kx, lNx)) : 1.0;
            const double w = desc->kz_phase[k];
            const double ibw = pf ? 1.0 / spline_bhat(order, w) : 1.0;
            const double sc = ibx * iby * ibw;
            G[k] = make_float2((float)(desc->filter[2 * k] * sc), (float)(desc->filter[2 * k + 1] * sc));
            const double wpi = w / M_PI;
            const float whi = (float)wpi;
            W[k] = make_float2(whi, (float)(wpi - (double)whi));
            S[k] = make_float2((float)std::cos(w), (float)std::sin(w));
            for (int i = 0; i < 2; ++i) {
                AL[(size_t)i * K + k] = make_float2(0.f, 0.f);
                BE[(size_t)i * K + k] = make_float2(0.f, 0.f);
            }
            if (pf) {
                // along z the particular solution of plane p is exp(i w z_p):
                // d_mL = e(z_first) 2i sin(m w), d_mR = -e(z_last) 2i sin(m w)
                const std::complex<double> I(0.0, 1.0);
                const std::complex<double> e0 = std::exp(I * (w * z_first));
                const std::complex<double> en = std::exp(I * (w * z_last));
                std::complex<double> dv[4];
                for (int m = 1; m <= np; ++m) {
                    dv[m - 1] = e0 * (2.0 * std::sin(m * w)) * I;
                    dv[np + m - 1] = en * (-2.0 * std::sin(m * w)) * I;
                }
                const int n2 = 2 * np;
                for (int r = 0; r < n2; ++r) {
                    std::complex<double> c = 0.0;
                    for (int j = 0; j < n2; ++j)
                        c += Kz[r * n2 + j] * dv[j];
                    const float2 cf = make_float2((float)c.real(), (float)c.imag());
                    if (r < np)
                        AL[(size_t)r * K + k] = cf;
                    else
                        BE[(size_t)(r - np) * K + k] = cf;
                }
            }
        }
    }
    // largest runs of all-zero filter columns and rows around the Nyquist
    // frequency (outside the |k| < km disc): neither computed nor read
    auto zero_run = [](int n, auto &&zero, int *lo, int *hi) {
        *lo = *hi = n / 2;
        if (!zero(n / 2))
            return;
        *hi = n / 2 + 1;
        while (*lo > 0 && zero(*lo - 1))
            --*lo;
        while (*hi < n && zero(*hi))
            ++*hi;
    };
    auto zero_at = [&](int ky, int kx) {
        const size_t k = (size_t)ky * lNx + kx;
        return desc->filter[2 * k] == 0.0 && desc->filter[2 * k + 1] == 0.0;
    };
    zero_run(lNx, [&](int kx) {
        for (int ky = 0; ky < lNy; ++ky)
            if (!zero_at(ky, kx))
                return false;
        return true;
    }, &p->kx_zero_lo, &p->kx_zero_hi);
    zero_run(lNy, [&](int ky) {
        for (int kx = 0; kx < lNx; ++kx)
            if (!zero_at(ky, kx))
                return false;
        return true;
    }, &p->ky_zero_lo, &p->ky_zero_hi);
    for (int m = 0; m < lNx; ++m)
        twx[m] = make_float2((float)std::cos(-2.0 * M_PI * m / lNx), (float)std::sin(-2.0 * M_PI * m / lNx));
    for (int m = 0; m < lNy; ++m)
        twy[m] = make_float2((float)std::cos(-2.0 * M_PI * m / lNy), (float)std::sin(-2.0 * M_PI * m / lNy));

    size_t o = 0;
    const size_t oG = o; o = align_up(o + K * 8);
    const size_t oW = o; o = align_up(o + K * 8);
    const size_t oS = o; o = align_up(o + K * 8);
    const size_t oA = o; o = align_up(o + 2 * K * 8);
    const size_t oB = o; o = align_up(o + 2 * K * 8);
    // the propagator and boundary tables in the transposed order
    const size_t oWt = o; o = align_up(o + K * 8);
    const size_t oSt_ = o; o = align_up(o + K * 8);
    const size_t oAt = o; o = align_up(o + 2 * K * 8);
    const size_t oBt = o; o = align_up(o + 2 * K * 8);
    const size_t oTx = o; o = align_up(o + (size_t)lNx * 8);
    const size_t oTy = o; o = align_up(o + (size_t)lNy * 8);
    const size_t oZ = o; o = align_up(o + 2 * odt::ZPOW_N * 4);
    const size_t oSt = o; o = align_up(o + 16);
    {
        std::lock_guard<std::mutex> lock(g_debug_mutex);
        if (g_table_alloc_limit && o > g_table_alloc_limit) {
            delete p;
            return fail(ODT_ERR_OUT_OF_MEMORY, "plan tables exceed the allocation limit set by "
                                               "odt_debug_set_table_alloc_limit");
        }
    }
    cudaError_t e = cudaGetDevice(&p->device);
    if (e != cudaSuccess) {
        delete p;
        return cuda_fail(e, "cudaGetDevice");
    }
    e = cudaMalloc(&p->d_tables, o);
    if (e != cudaSuccess) {
        delete p;
        return e == cudaErrorMemoryAllocation ? fail(ODT_ERR_OUT_OF_MEMORY, "cudaMalloc of plan tables failed")
                                              : cuda_fail(e, "cudaMalloc");
    }
    char *base = (char *)p->d_tables;
    auto transpose = [&](const std::vector<float2> &src) {
        std::vector<float2> t(src.size());
        for (size_t i = 0; i < src.size(); i += K)
            for (int ky = 0; ky < lNy; ++ky)
                for (int kx = 0; kx < lNx; ++kx)
                    t[i + (size_t)kx * lNy + ky] = src[i + (size_t)ky * lNx + kx];
        return t;
    };
    const std::vector<float2> Wt = transpose(W), Stt = transpose(S), ALt = transpose(AL), BEt = transpose(BE);
    struct Up { size_t off; const void *src; size_t n; } ups[] = {
        {oG, G.data(), K * 8}, {oW, W.data(), K * 8}, {oS, S.data(), K * 8}, {oA, AL.data(), 2 * K * 8},
        {oB, BE.data(), 2 * K * 8}, {oTx, twx.data(), (size_t)lNx * 8}, {oTy, twy.data(), (size_t)lNy * 8},
        {oZ, zp.data(), 2 * odt::ZPOW_N * 4}, {oWt, Wt.data(), K * 8}, {oSt_, Stt.data(), K * 8},
        {oAt, ALt.data(), 2 * K * 8}, {oBt, BEt.data(), 2 * K * 8}};
    for (const Up &u : ups) {
        e = cudaMemcpy(base + u.off, u.src, u.n, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(p->d_tables);
            delete p;
            return cuda_fail(e, "cudaMemcpy of plan tables");
        }
    }
    e = cudaMemset(base + oSt, 0, 16);
    if (e != cudaSuccess) {
        cudaFree(p->d_tables);
        delete p;
        return cuda_fail(e, "cudaMemset");
    }
    p->tab.G = (const float2 *)(base + oG);
    p->tab.wsplit = (const float2 *)(base + oW);
    p->tab.step = (const float2 *)(base + oS);
    p->tab.alpha = (const float2 *)(base + oA);
    p->tab.beta = (const float2 *)(base + oB);
    p->tab.twx = (const float2 *)(base + oTx);
    p->tab.twy = (const float2 *)(base + oTy);
    p->tab.zpow = (const float *)(base + oZ);
    p->tabt = p->tab;
    p->tabt.G = nullptr;
    p->tabt.wsplit = (const float2 *)(base + oWt);
    p->tabt.step = (const float2 *)(base + oSt_);
    p->tabt.alpha = (const float2 *)(base + oAt);
    p->tabt.beta = (const float2 *)(base + oBt);
    std::swap(p->tabt.twx, p->tabt.twy);
    p->d_status = (int *)(base + oSt);

    p->lay = make_layout(p, d.num_angles, 1);

    // opposite views share a slab through the mirrored spectrum, which needs
    // tables even in kx (true of the reference's filters about y)
    p->even = tilted ? 0 : 1;
    for (int ky = 0; p->even && ky < lNy; ++ky)
        for (int kx = 1; kx < lNx - kx; ++kx) {
            const size_t k = (size_t)ky * lNx + kx, m = (size_t)ky * lNx + (lNx - kx);
            if (desc->kz_phase[k] != desc->kz_phase[m] || desc->filter[2 * k] != desc->filter[2 * m] ||
                desc->filter[2 * k + 1] != desc->filter[2 * m + 1]) {
                p->even = 0;
                break;
            }
        }

    p->col_slots = 0;
    StageParams P = stage_params(p);
    e = odt::configure_kernels(P);
    if (e == cudaSuccess) {
        p->col_slots = odt::columns_slots(odt::transposed(P));
        P.col_slots = p->col_slots;
    P.zshift = (float)d.z_shift;
    }
    if (e == cudaSuccess && !tilted)
        e = odt::configure_rotate_kernels();
    if (e == cudaSuccess)
        e = odt::configure_adjoint_kernels(P);
    if (e == cudaSuccess && !tilted)
        e = odt::configure_rotate_adjoint_kernels();
    if (e != cudaSuccess) {
        cudaFree(p->d_tables);
        delete p;
        return cuda_fail(e, "kernel configuration");
    }
    *out = p;
    return ODT_OK;
}

odt_status odt_bpp3d_workspace_size(const odt_bpp3d_plan *plan, uint64_t *bytes)
{
    if (!plan || !bytes)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    *bytes = plan->lay.ws_bytes;
    return ODT_OK;
}

odt_status odt_bpp3d_angle_batch(const odt_bpp3d_plan *plan, int32_t *batch)
{
    if (!plan || !batch)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    *batch = plan->lay.batch;
    return ODT_OK;
}

}  // extern "C"

namespace {

// Event pair around one launch, summed into a stage slot after the run.
struct LaunchTimer {
    odt_stage_timing *t;
    cudaStream_t s;
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> ev;
    explicit LaunchTimer(odt_stage_timing *timing, cudaStream_t stream) : t(timing), s(stream) {}
    void begin(int stage)
    {
        if (!t)
            return;
        cudaEvent_t a, b;
        cudaEventCreate(&a);
        cudaEventCreate(&b);
        cudaEventRecord(a, s);
        ev.push_back({stage, {a, b}});
    }
    void end(double bytes)
    {
        if (!t)
            return;
        cudaEventRecord(ev.back().second.second, s);
        t->launches[ev.back().first] += 1;
        t->bytes[ev.back().first] += bytes;
    }
    cudaError_t finish()
    {
        if (!t)
            return cudaSuccess;
        cudaError_t e = cudaStreamSynchronize(s);
        for (auto &x : ev) {
            float ms = 0.f;
            if (e == cudaSuccess)
                e = cudaEventElapsedTime(&ms, x.second.first, x.second.second);
            t->ms[x.first] += ms;
            cudaEventDestroy(x.second.first);
            cudaEventDestroy(x.second.second);
        }
        ev.clear();
        return e;
    }
};

// One execution: `units` NULL is one angle per slab (geometry per angle),
// otherwise the device list of opposite views with one geometry per unit.
odt_status run_plan(const odt_bpp3d_plan *plan, const Layout &lay, const int2 *units, const void *sino,
                    const double *weights, const double *geometry, const float *gain, const void *again,
                    void *volume, void *workspace, void *stream, odt_stage_timing *timing)
{
    if (!sino || !geometry || !volume || (!workspace && lay.ws_bytes))
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    if (((uintptr_t)workspace % kAlign) != 0)
        return fail(ODT_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    const odt_status dst = check_device(plan);
    if (dst != ODT_OK)
        return dst;
    const odt_bpp3d_desc &d = plan->d;
    cudaStream_t s = (cudaStream_t)stream;
    StageParams P = stage_params(plan);
    P.gain = gain;
    const size_t spec_elems = (size_t)plan->d.pad_ny * plan->d.pad_nx;
    char *ws = (char *)workspace;
    float2 *fspec = (float2 *)(ws + lay.off_spec);
    float2 *T = (float2 *)(ws + lay.off_T);
    float2 *Tab = (float2 *)(ws + lay.off_Tab);
    float2 *slab = (float2 *)(ws + lay.off_slab);
    float2 *comp = (float2 *)(ws + lay.off_comp);
    // row spectra: in the slab's place, in place of the filtered spectra for
    // single-row planes
    float2 *rowspec = odt::single_row_plan(P) ? fspec : slab;
    void *rot_scratch = ws + lay.off_rot;
    const size_t in_elem = d.input_dtype == ODT_INPUT_C128 ? 16 : 8;
    const int geo_stride = d.geometry == ODT_GEOM_AFFINE3D ? 12 : 6;
    const int nbatches = (lay.units + lay.batch - 1) / lay.batch;
    const double plane_in = (double)d.ny * d.nx, spec = (double)d.pad_ny * d.pad_nx;
    const double vol = (double)plan->nz * d.ny * d.nx;
    const double out_elem = d.onlyreal ? 4.0 : 8.0;
    if (timing)
        std::memset(timing, 0, sizeof(*timing));
    LaunchTimer lt(timing, s);
    cudaError_t e;
    for (int b = 0; b < nbatches; ++b) {
        const int a0 = b * lay.batch;  // first slab of the batch
        const int nb = std::min(lay.batch, lay.units - a0);
        const int ns = nb * lay.spu;   // spectrum slots
        const char *sino_b = (const char *)sino;
        const double *w_b = weights;
        if (units) {
            P.units = units + a0;
            P.again = (const float2 *)again;
        } else {
            sino_b += (size_t)a0 * d.ny * d.nx * in_elem;
            w_b = weights ? weights + a0 : nullptr;
            P.again = again ? (const float2 *)again + (size_t)a0 * spec_elems : nullptr;
        }
        lt.begin(ODT_STAGE_ROWS_FORWARD);
        e = odt::launch_rows_forward(P, sino_b, w_b, ns, rowspec, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "rows_forward launch");
        lt.end(ns * (plane_in * in_elem + spec * 8.0));
        const int total = nb * plan->nz;
        lt.begin(ODT_STAGE_COLUMNS_PROPAGATE);
        if (odt::single_row_plan(P))
            e = odt::launch_spectrum_line(P, fspec, Tab, nb, s);
        else
            e = odt::launch_columns_spectrum(P, rowspec, fspec, ns, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "columns_spectrum launch");
        lt.end(0.0);
        if (odt::single_row_plan(P)) {
            // single-row planes: the column stage is the identity and runs
            // inside the row stage, one launch over the batch's jobs
            lt.begin(ODT_STAGE_ROWS_INVERSE);
            e = odt::launch_rows_line(P, fspec, Tab, slab, 0, total, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "rows_line launch");
            lt.end(ns * spec * 8.0 + (double)total * plane_in * 8.0);
        } else {
            const StageParams Pt = odt::transposed(P);
            if (d.intp_order >= 2) {
                lt.begin(ODT_STAGE_COLUMNS_PROPAGATE);
                e = odt::launch_columns_boundary(Pt, fspec, Tab, nb, s);
                if (e != cudaSuccess)
                    return cuda_fail(e, "columns_boundary launch");
                lt.end(0.0);
            }
            // column and row stage of a chunk one after the other.  Running
            // the row stage of one chunk beside the column stage of the next
            // (two chunk buffers, a second stream) gained 1-2 % on small
            // planes and lost up to 16 % at 256^3 (step 28.3 ms like this,
            // 28.7 to 33.0 ms overlapped): a column launch is one wave of
            // long CTAs, and row CTAs that take its slots stretch it.
            // (chunks of equal size, so that the last one fills its waves too)
            const int nchunks = (total + lay.jobs - 1) / lay.jobs, chunk = (total + nchunks - 1) / nchunks;
            for (int q0 = 0; q0 < total; q0 += chunk) {
                const int qn = std::min(chunk, total - q0);
                lt.begin(ODT_STAGE_COLUMNS_PROPAGATE);
                e = odt::launch_columns_propagate(Pt, fspec, T, q0, qn, s);
                if (e != cudaSuccess)
                    return cuda_fail(e, "columns_propagate launch");
                lt.end((double)qn / plan->nz * lay.spu * spec * 8.0);
                lt.begin(ODT_STAGE_ROWS_INVERSE);
                e = odt::launch_rows_inverse(Pt, T, Tab, slab, q0, qn, s);
                if (e != cudaSuccess)
                    return cuda_fail(e, "rows_inverse launch");
                lt.end((double)qn * plane_in * 8.0);
            }
        }
        RotParams R;
        R.ny = d.ny;
        R.nx = d.nx;
        R.nz = plan->nz;
        R.ypitch = P.ypitch;
        R.nbatch_angles = nb;
        R.first_pass = b == 0;
        R.last_pass = b == nbatches - 1;
        R.onlyreal = d.onlyreal;
        R.status = plan->d_status;
        // the column stage's output is dead here: room for partial sums
        R.part = (float4 *)T;
        R.part_bytes = lay.off_Tab - lay.off_T;
        lt.begin(ODT_STAGE_ROTATE);
        e = odt::launch_rotate(R, d.intp_order, d.geometry == ODT_GEOM_AFFINE3D, slab,
                               geometry + (size_t)a0 * geo_stride, volume, comp, rot_scratch, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "rotate launch");
        double rb = nb * vol * 8.0 + vol * out_elem;
        if (!R.first_pass)
            rb += vol * (out_elem + 8.0);
        if (!R.last_pass)
            rb += vol * 8.0;
        lt.end(rb);
    }
    e = lt.finish();
    if (e != cudaSuccess)
        return cuda_fail(e, "timing");
    return ODT_OK;
}

}  // namespace

extern "C" {

odt_status odt_bpp3d_execute(const odt_bpp3d_plan *plan, const void *sino, const double *weights,
                             const double *geometry, void *volume, void *workspace, void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    return run_plan(plan, plan->lay, nullptr, sino, weights, geometry, nullptr, nullptr, volume, workspace, stream,
                    nullptr);
}

odt_status odt_bpp3d_execute_gain(const odt_bpp3d_plan *plan, const void *sino, const double *weights,
                                  const double *geometry, const float *gain, const void *angle_gain,
                                  void *volume, void *workspace, void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    return run_plan(plan, plan->lay, nullptr, sino, weights, geometry, gain, angle_gain, volume, workspace, stream,
                    nullptr);
}

odt_status odt_bpp3d_pair_workspace_size(const odt_bpp3d_plan *plan, int32_t num_units, uint64_t *bytes,
                                         uint64_t *adjoint_bytes)
{
    if (!plan || !bytes)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    Layout y;
    const odt_status st = pair_layout(plan, num_units, &y);
    if (st != ODT_OK)
        return st;
    *bytes = y.ws_bytes;
    if (adjoint_bytes)
        *adjoint_bytes = y.adj_ws_bytes;
    return ODT_OK;
}

odt_status odt_bpp3d_execute_pairs(const odt_bpp3d_plan *plan, const odt_bpp3d_units *units, const void *sino,
                                   const double *weights, const float *gain, const void *angle_gain, void *volume,
                                   void *workspace, void *stream, odt_stage_timing *timing)
{
    if (!plan || !units || !units->views)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    Layout y;
    const odt_status st = pair_layout(plan, units->num_units, &y);
    if (st != ODT_OK)
        return st;
    return run_plan(plan, y, (const int2 *)units->views, sino, weights, units->geometry, gain, angle_gain, volume,
                    workspace, stream, timing);
}

odt_status odt_bpp3d_adjoint_workspace_size(const odt_bpp3d_plan *plan, uint64_t *bytes)
{
    if (!plan || !bytes)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (plan->d.intp_order > 3)
        return fail(ODT_ERR_UNSUPPORTED, "the adjoint is implemented for spline orders 0..3");
    *bytes = plan->lay.adj_ws_bytes;
    return ODT_OK;
}

static odt_status run_adjoint(const odt_bpp3d_plan *plan, const Layout &lay, const int2 *units, const void *sino,
                              const double *weights, const double *geometry, const float *gain,
                              const void *angle_gain, const void *vol_grad, void *sino_grad, float *gain_grad,
                              void *angle_gain_grad, void *workspace, void *stream)
{
    if (!geometry || !vol_grad || !workspace)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    if (!sino_grad && !gain_grad && !angle_gain_grad)
        return ODT_OK;
    if ((gain_grad || angle_gain_grad) && !sino)
        return fail(ODT_ERR_INVALID_ARGUMENT, "the gain gradient needs the sinogram");
    if (((uintptr_t)workspace % kAlign) != 0)
        return fail(ODT_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    const odt_status dst = check_device(plan);
    if (dst != ODT_OK)
        return dst;
    const odt_bpp3d_desc &d = plan->d;
    const bool tilted = d.geometry == ODT_GEOM_AFFINE3D;
    const int geo_stride = tilted ? 12 : 6;
    if (d.onlyreal)
        return fail(ODT_ERR_UNSUPPORTED, "the adjoint needs a complex (onlyreal=0) plan");
    if (d.intp_order > 3)
        return fail(ODT_ERR_UNSUPPORTED, "the adjoint is implemented for spline orders 0..3");
    cudaStream_t s = (cudaStream_t)stream;
    StageParams P = stage_params(plan);
    P.gain = gain;
    char *ws = (char *)workspace;
    float2 *rowspec = (float2 *)(ws + lay.off_spec);
    float2 *T = (float2 *)(ws + lay.off_T);
    float2 *slab = (float2 *)(ws + lay.off_slab);
    float2 *Qg = (float2 *)(ws + lay.off_Qg);
    float2 *W = (float2 *)(ws + lay.off_W);
    float2 *Pg = (float2 *)(ws + lay.off_Pg);
    const size_t in_elem = d.input_dtype == ODT_INPUT_C128 ? 16 : 8;
    const size_t spec = (size_t)d.pad_ny * d.pad_nx;
    const int nbatches = (lay.units + lay.batch - 1) / lay.batch;
    cudaError_t e;
    const float2 *vg = (const float2 *)vol_grad;
    if (!tilted) {
        float2 *vT = (float2 *)(ws + lay.off_vT);
        e = odt::launch_volume_zxy(vg, vT, plan->nz, d.ny, d.nx, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "volume transpose launch");
        vg = vT;
    }
    if (gain_grad) {
        e = cudaMemsetAsync(gain_grad, 0, spec * sizeof(float), s);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMemsetAsync");
    }
    for (int b = 0; b < nbatches; ++b) {
        const int u0 = b * lay.batch;  // first slab of the batch
        const int nb = std::min(lay.batch, lay.units - u0);
        const int ns = nb * lay.spu;   // spectrum slots
        const int a0 = units ? 0 : u0; // angle that the per-angle arrays start at
        P.units = units ? units + u0 : nullptr;
        P.again = angle_gain ? (const float2 *)angle_gain + (size_t)a0 * spec : nullptr;
        RotParams R;
        R.ny = d.ny;
        R.nx = d.nx;
        R.nz = plan->nz;
        R.ypitch = P.ypitch;
        R.nbatch_angles = nb;
        R.first_pass = 1;
        R.last_pass = 1;
        R.onlyreal = 0;
        R.status = plan->d_status;
        R.part = nullptr;
        R.splits = 1;
        e = odt::launch_rotate_adjoint(R, d.intp_order, tilted ? 1 : 0, vg,
                                       geometry + (size_t)u0 * geo_stride, slab, ws + lay.off_rot, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "rotate_adjoint launch");
        if (gain_grad || angle_gain_grad) {
            const char *sino_b = (const char *)sino + (size_t)a0 * d.ny * d.nx * in_elem;
            e = odt::launch_rows_forward(P, sino_b, weights ? weights + a0 : nullptr, ns, rowspec, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "rows_forward launch");
        }
        e = cudaMemsetAsync(Qg, 0, (size_t)ns * spec * sizeof(float2), s);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMemsetAsync");
        const int total = nb * plan->nz;
        for (int q0 = 0; q0 < total; q0 += lay.jobs) {
            const int qn = std::min(lay.jobs, total - q0);
            e = odt::launch_adj_rows(P, slab, T, q0, qn, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "adj_rows launch");
            e = odt::launch_adj_columns(P, T, Qg, q0, qn, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "adj_columns launch");
        }
        e = odt::launch_adj_spectrum(P, rowspec, Qg, gain_grad,
                                     angle_gain_grad ? (float2 *)angle_gain_grad + (size_t)a0 * spec : nullptr, W,
                                     ns, s);
        if (e != cudaSuccess)
            return cuda_fail(e, "adj_spectrum launch");
        if (sino_grad) {
            e = odt::launch_adj_rows_full(P, W, Pg, ns, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "adj_rows_full launch");
            e = odt::launch_adj_pad(P, Pg, weights ? weights + a0 : nullptr, ns,
                                    (float2 *)sino_grad + (size_t)a0 * d.ny * d.nx, s);
            if (e != cudaSuccess)
                return cuda_fail(e, "adj_pad launch");
        }
    }
    return ODT_OK;
}

odt_status odt_bpp3d_adjoint(const odt_bpp3d_plan *plan, const void *sino, const double *weights,
                             const double *geometry, const float *gain, const void *angle_gain,
                             const void *vol_grad, void *sino_grad, float *gain_grad, void *angle_gain_grad,
                             void *workspace, void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    return run_adjoint(plan, plan->lay, nullptr, sino, weights, geometry, gain, angle_gain, vol_grad, sino_grad,
                       gain_grad, angle_gain_grad, workspace, stream);
}

odt_status odt_bpp3d_adjoint_pairs(const odt_bpp3d_plan *plan, const odt_bpp3d_units *units, const void *sino,
                                   const double *weights, const float *gain, const void *angle_gain,
                                   const void *vol_grad, void *sino_grad, float *gain_grad, void *angle_gain_grad,
                                   void *workspace, void *stream)
{
    if (!plan || !units || !units->views)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    Layout y;
    const odt_status st = pair_layout(plan, units->num_units, &y);
    if (st != ODT_OK)
        return st;
    return run_adjoint(plan, y, (const int2 *)units->views, sino, weights, units->geometry, gain, angle_gain,
                       vol_grad, sino_grad, gain_grad, angle_gain_grad, workspace, stream);
}

odt_status odt_bpp3d_execute_timed(const odt_bpp3d_plan *plan, const void *sino, const double *weights,
                                   const double *geometry, void *volume, void *workspace, void *stream,
                                   odt_stage_timing *timing)
{
    if (!timing)
        return fail(ODT_ERR_INVALID_ARGUMENT, "timing is NULL");
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL pointer argument");
    return run_plan(plan, plan->lay, nullptr, sino, weights, geometry, nullptr, nullptr, volume, workspace, stream,
                    timing);
}

static int64_t count_launches(const odt_bpp3d_plan *plan, const Layout &lay)
{
    int64_t n = 0;
    for (int b = 0; b * lay.batch < lay.units; ++b) {
        const int64_t total = (int64_t)std::min(lay.batch, lay.units - b * lay.batch) * plan->nz;
        if (odt::single_row_plan(stage_params(plan)))
            n += 4;  // row spectra, filtered spectra, fused column + row stage, resampling
        else
            n += 3 + (plan->d.intp_order >= 2) + 2 * ((total + lay.jobs - 1) / lay.jobs);
        if (plan->d.geometry == ODT_GEOM_Y_AXIS)
            n += 1;  // per-(slab, tile) geometry setup
    }
    return n;
}

odt_status odt_bpp3d_launch_count(const odt_bpp3d_plan *plan, int64_t *launches)
{
    if (!plan || !launches)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    *launches = count_launches(plan, plan->lay);
    return ODT_OK;
}

odt_status odt_bpp3d_pair_launch_count(const odt_bpp3d_plan *plan, int32_t num_units, int64_t *launches)
{
    if (!plan || !launches)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL argument");
    Layout y;
    const odt_status st = pair_layout(plan, num_units, &y);
    if (st == ODT_OK)
        *launches = count_launches(plan, y);
    return st;
}

odt_status odt_bpp3d_read_status(const odt_bpp3d_plan *plan, void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL plan");
    const odt_status dst = check_device(plan);
    if (dst != ODT_OK)
        return dst;
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, plan->d_status, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess)
        return cuda_fail(e, "status read");
    if (h != 0) {
        // cleared synchronously, so a failed clear is reported here and not
        // by some later call
        e = cudaMemset(plan->d_status, 0, sizeof(int));
        if (e != cudaSuccess)
            return cuda_fail(e, "status clear");
        char buf[96];
        snprintf(buf, sizeof buf, "device check failed (bits 0x%x)", h);
        return fail(ODT_ERR_DEVICE_CHECK, buf);
    }
    return ODT_OK;
}

odt_status odt_debug_inject_status(const odt_bpp3d_plan *plan, int32_t bits, void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL plan");
    if (bits < 0 || bits > 255)
        return fail(ODT_ERR_INVALID_ARGUMENT, "status bits must be in 0..255");
    const odt_status dst = check_device(plan);
    if (dst != ODT_OK)
        return dst;
    // the word's low byte (little-endian), stream-ordered like a kernel's
    // report; the upper bytes are cleared
    cudaError_t e = cudaMemsetAsync(plan->d_status, 0, sizeof(int), (cudaStream_t)stream);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(plan->d_status, bits, 1, (cudaStream_t)stream);
    if (e != cudaSuccess)
        return cuda_fail(e, "status injection");
    return ODT_OK;
}

odt_status odt_debug_set_table_alloc_limit(uint64_t bytes)
{
    std::lock_guard<std::mutex> lock(g_debug_mutex);
    g_table_alloc_limit = bytes;
    return ODT_OK;
}

odt_status odt_bpp3d_plan_destroy(odt_bpp3d_plan *plan)
{
    if (!plan)
        return ODT_OK;
    cudaError_t e = cudaFree(plan->d_tables);
    delete plan;
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaFree");
    return ODT_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Execution without allocation.
//
// Some callers cannot allocate device memory when they run a
// reconstruction: code inside a region where a cudaMalloc would stall the
// device or is not allowed (a latency-critical acquisition loop, a stream
// that is being captured, a framework that owns every byte of device
// memory and only hands out pointers to its own tensors).  For them the
// execution below takes its scratch space from a fixed array that is part of
// the library's device image instead of a caller-provided workspace.
//
// * The array is ODT_NOALLOC_SCRATCH_BYTES (64 MiB) per device; every device
//   on which the library's device code is loaded holds it until the process
//   exits.  Plans whose workspace is larger are rejected: create the plan
//   with desc.workspace_limit <= ODT_NOALLOC_SCRATCH_BYTES.
// * The first call on a device looks up the array's device address
//   (cudaGetSymbolAddress) with that device current, once; make that first
//   call before any stream capture.
// * Every call on a device uses the same array and leaves its contents
//   behind; nothing in it has to start at zero (each stage writes what the
//   next reads).  Calls whose executions overlap on the GPU race on it: run
//   them on one stream, or order them.
static __device__ __align__(256) unsigned char g_noalloc_scratch[ODT_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void *g_noalloc_addr[kMaxDevices];
}  // namespace

extern "C" odt_status odt_bpp3d_execute_noalloc(const odt_bpp3d_plan *plan, const void *sino,
                                                const double *weights, const double *geometry, void *volume,
                                                void *stream)
{
    if (!plan)
        return fail(ODT_ERR_INVALID_ARGUMENT, "NULL plan");
    if (plan->lay.ws_bytes > ODT_NOALLOC_SCRATCH_BYTES) {
        char buf[200];
        snprintf(buf, sizeof buf,
                 "plan needs %llu bytes of scratch, the static scratch holds %llu; create the plan with "
                 "workspace_limit <= %llu",
                 (unsigned long long)plan->lay.ws_bytes, (unsigned long long)ODT_NOALLOC_SCRATCH_BYTES,
                 (unsigned long long)ODT_NOALLOC_SCRATCH_BYTES);
        return fail(ODT_ERR_INVALID_ARGUMENT, buf);
    }
    // the scratch of the plan's device, which must be current
    const odt_status dst = check_device(plan);
    if (dst != ODT_OK)
        return dst;
    const int dev = plan->device;
    cudaError_t e = cudaSuccess;
    if (dev < 0 || dev >= kMaxDevices)
        return fail(ODT_ERR_UNSUPPORTED, "device ordinal beyond the static scratch table");
    void *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_addr[dev]) {
            e = cudaGetSymbolAddress(&g_noalloc_addr[dev], g_noalloc_scratch);
            if (e != cudaSuccess) {
                g_noalloc_addr[dev] = nullptr;
                return cuda_fail(e, "cudaGetSymbolAddress of the static scratch");
            }
        }
        scratch = g_noalloc_addr[dev];
    }
    return run_plan(plan, plan->lay, nullptr, sino, weights, geometry, nullptr, nullptr, volume, scratch, stream,
                    nullptr);
}
