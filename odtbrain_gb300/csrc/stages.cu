// Filter stages (a) and (b) of the 3D backpropagation on sm_103a.
//
// Reference loop body (odtbrain/_alg3d_bpp.py:492-528, _alg3d_bppt.py:
// 865-898), per angle:
//   pad -> forward 2D FFT -> *prefactor/(lNx*lNy) -> for every z plane p:
//   *exp(i km (M-1) z_p) -> unnormalised backward 2D FFT -> crop.
//
// GB300 decomposition (all lines in registers):
//   rows_forward       padded+weighted rows, forward FFT along x
//   columns_spectrum   forward FFT along y, filter multiply -> filtered
//                      spectrum, stored transposed [kx][ky]
//   columns_boundary   z-prefilter boundary rows (once per slab)
//   columns_propagate  for a run of z planes: propagator (exact anchor +
//                      complex recurrence), backward FFT along x, crop in x
//   rows_inverse       backward FFT along y, crop in y -> coefficient slab
//
// The last three work on the transposed plane (launched with the StageParams
// of transposed()): their "columns" run along x and their "rows" along y, so
// that a finished row lies along the slab's innermost axis and is stored from
// registers, contiguously.  With the rows along x every row group had to be
// transposed through shared memory behind three barriers and stored in runs
// of 32 bytes: row stage of 256^3 from 200 views 10.4 -> 8.4 ms (whole step
// 28.3 -> 27.0 ms), tilted 200^3 19.6 -> 16.1 ms.
//
// The B-spline prefilter that scipy.ndimage applies before resampling
// (mirror boundaries, along z and x of every plane; along all three axes on
// the tilted path) is folded into these stages exactly: each Fourier
// component exp(i k n) of a cropped line has the prefiltered form
// exp(i k n)/Bhat(k) + A z^n + B z^(N-1-n) (z the spline pole, Bhat the
// sampled B-spline's transfer function), where A and B follow from the two
// mirror conditions.  So the spectrum is divided by Bhat along every
// prefiltered axis (folded into the filter table G), z gets per-frequency
// boundary terms (alpha, beta tables), and x (and y) get per-line boundary
// terms computed from four samples just outside the crop.
//
// Opposite views.  Rotating by phi + pi is rotating the slab by pi about y
// and then by phi, and a rotation by pi maps the slab grid onto itself: plane
// p to nz-1-p, column x to nx-1-x.  So two views phi and phi + pi (a "unit")
// share one slab: with the second view's padded rows mirrored about the
// crop's centre (columns m -> 2 padxl + nx-1 - m, modulo lNx) its spectrum X'
// is the one of the mirrored view, and with z_(nz-1-p) = 2 zshift - 1 - z_p
// plane p of the shared slab is the backward transform of
//   G X e^(i w z_p) + G X' e^(i w (2 zshift - 1 - z_p)).
// Both terms are formed before the transforms, so one backward 2D transform
// per plane and one resampling serve two views.  256^3 from 200 views of a
// full circle: step 54.2 -> 36.2 ms.
#include <algorithm>
#include <type_traits>

#include "odt_fft.cuh"
#include "odt_internal.cuh"
#include "odt_stage_util.cuh"

namespace odt {

// Column stage of half-crop plans: keep the propagator step exp(i w) of a
// thread's elements in registers instead of shared memory, and read the
// third radix-8 pass's twiddles from the per-thread-class table (256^3
// workload: 25.7 ms without either, 25.7 / 26.0 ms with one of them,
// 24.1 ms with both).
constexpr bool kColumnStepRegs = true;
constexpr bool kColumnTw2 = true;
// Planes between exact propagator anchors within a column CTA's run, at most
// (anchor_planes has the rule).
constexpr int kReanchorPlanes = 32;
// Column CTAs that run through up to 256 planes of an angle, re-anchoring
// the propagator on the way: power-of-two columns in CTAs of at most 256
// threads, with the steps in registers (64 to 512 points).  256^3 from 200
// single views, cap on the planes per CTA against the column stage: 32 planes
// 24.1 ms, 64 22.8, 128 22.4, 256 22.2 ms.  The other column kernels keep runs
// of at most kReanchorPlanes planes.
template <class L, int KX>
constexpr bool long_runs()
{
    return pow2_len<L>() > 0 && kColumnStepRegs && KX * L::TPL <= 256;
}
// Column kernels that hold the propagator steps in registers and read the
// third pass's twiddles from the 64x7 table (N >= 512): the half-crop
// kernel, and for other crops power-of-two columns in CTAs of at most 256
// threads (with more threads per CTA, 64 registers per thread, the steps
// spill).
template <class L, int KX, bool HALF>
constexpr bool column_regs()
{
    return kColumnStepRegs && (HALF || (pow2_len<L>() > 0 && KX * L::TPL <= 256));
}

// ---------------------------------------------------------------------------
// (a) rows: pad + weight + forward FFT along x.
// rowspec[a][y][kx], a in the batch, y over the padded height.
// P.units: slot 2u is unit u's first view, slot 2u+1 its opposite view with
// the padded row mirrored (left unwritten when there is none).
template <class L, int LPC>
__global__ void __launch_bounds__(LPC * L::TPL) k_rows_forward(StageParams P, L line, const void *sino,
                                                               const double *weights, int nslots, float2 *rowspec)
{
    extern __shared__ float2 smem[];
    const int n = line.size();
    const int ls = xslots<false>(n);
    float2 *buf0 = smem, *buf1 = smem + LPC * ls, *tw = smem + 2 * LPC * ls;
    copy_twiddles<L>(tw, P.tab.twx, n);
    const int l = threadIdx.x / L::TPL, j = threadIdx.x % L::TPL;
    const int lid = (int)blockIdx.x * LPC + l;
    const int nlines = nslots * P.lNy;
    bool valid = lid < nlines;
    const int slot = valid ? lid / P.lNy : 0;
    const int y = valid ? lid - slot * P.lNy : 0;
    int a = slot;
    bool mirrored = false;
    if (P.units) {
        const int2 u = P.units[slot >> 1];
        mirrored = slot & 1;
        a = mirrored ? u.y : u.x;
        valid = valid && a >= 0;
    }
    const double w = (weights && valid) ? weights[a] : 1.0;
    const size_t arow = (size_t)(valid ? a : 0) * P.ny * P.nx;
    float2 v[L::SLOTS];
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        int x = j + r * L::TPL;
        const bool in = valid && x < n;
        if (mirrored) {
            x = 2 * P.padxl + P.nx - 1 - x;
            x += x < 0 ? n : 0;
            x -= x >= n ? n : 0;
        }
        v[r] = in ? padded_sample(P, sino, arow, w, y, x) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    int flip = 0;
    line.template run<-1>(v, j, buf0 + l * ls, buf1 + l * ls, 1, tw, flip);
    if (!valid)
        return;
    float2 *dst = rowspec + (size_t)lid * n;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int x = j + r * L::TPL;
        if (x < n)
            dst[x] = v[r];
    }
}

// ---------------------------------------------------------------------------
// Column helpers shared by the two column kernels.  A CTA owns KX adjacent
// spectrum columns kx; thread (c, j) holds rows ky = j + r*TPL of column c.

// The edge samples of a prefilter's boundary solve that thread j holds after a
// line's backward transform (crop of `len` samples from `pad`): bit 8 r + e
// is set when slot r holds the sample of edge slot e (the same for every line
// of the CTA, so it is computed once).  Power-of-two lines (8 slots).
template <class L, int NP>
__device__ __forceinline__ unsigned long long edge_holdings(int pad, int len, int n, int j)
{
    unsigned long long m = 0;
#pragma unroll
    for (int e = 0; e < EDGE_SLOTS; ++e) {
        if (edge_used(e, NP)) {
            const int pos = (pad + edge_offset(e, len) + 2 * n) % n;
            if (pos % L::TPL == j)
                m |= 1ull << (8 * (pos / L::TPL) + e);
        }
    }
    return m;
}

// Backward FFT along the column of v, then the prefilter boundary terms (YF
// poles) and the cropped store dst[yy * lNx] for yy < ny.
template <class L, int KX, int YF>
__device__ __forceinline__ void column_inverse_store(const StageParams &P, const L &line, float2 (&v)[L::SLOTS],
                                                     int c, int j, bool colok, float2 *buf0, float2 *buf1,
                                                     const float2 *tw, float2 *edge, int &flip, float2 *dst)
{
    const int n = line.size();
    const int ny = P.ny, padyl = P.padyl;
    line.template run<1, true>(v, j, buf0 + c, buf1 + c, KX, tw, flip);
    // u around the crop's ends (periodic over the padded height)
#pragma unroll
    for (int e = 0; e < EDGE_SLOTS; ++e) {
        float2 t;
        if (edge_used(e, YF) && held<L>(v, j, (padyl + edge_offset(e, ny) + 2 * n) % n, t))
            edge[c * EDGE_SLOTS + e] = t;
    }
    __syncthreads();
    float2 cf[2 * YF];
    pf_coefs<YF>(P.kys, edge + c * EDGE_SLOTS, cf);
    if (!colok)
        return;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int yy = j + r * L::TPL - padyl;
        if (yy >= 0 && yy < ny)
            dst[(size_t)yy * P.lNx] = pf_apply<YF>(P, cf, yy, ny, v[r]);
    }
}

// ---------------------------------------------------------------------------
// (a2) filtered spectra, once per slot: forward FFT along y of the row
// spectra times the filter and the gains, stored transposed [kx][ky] (zero for
// a unit without opposite view).  The column kernel used to redo this
// transform at the head of every run of planes and keep its result in shared
// memory for the re-anchoring; read from here (16 bytes per element and 32
// planes) that shared memory is free.
template <class L, int KX>
__global__ void __launch_bounds__(KX * L::TPL) k_columns_spectrum(StageParams P, L line, const float2 *rowspec,
                                                                  float2 *spec)
{
    extern __shared__ float2 smem[];
    const int n = line.size();
    const int ls = xslots<true>(n);
    float2 *buf0 = smem, *buf1 = smem + KX * ls, *tw = smem + 2 * KX * ls;
    const int c = threadIdx.x % KX, j = threadIdx.x / KX;
    const int kx = blockIdx.x * KX + c;
    const bool colok = kx < P.lNx;
    const int slot = blockIdx.y;
    const size_t K = (size_t)P.lNy * P.lNx;
    int a = slot, kg = kx;
    if (P.units) {
        const int2 u = P.units[slot >> 1];
        a = (slot & 1) ? u.y : u.x;
        if ((slot & 1) && kx)
            kg = P.lNx - kx;  // the gains' column of a mirrored view
    }
    float2 v[L::SLOTS];
    // (the early cases are uniform over the CTA)
    if (a < 0 || !group_active<KX>(P, blockIdx.x * KX)) {
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r)
            v[r] = make_float2(0.f, 0.f);
    } else {
        copy_twiddles<L>(tw, P.tab.twy, n);
        const float2 *src = rowspec + slot * K;
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            v[r] = (colok && ky < n) ? src[(size_t)ky * P.lNx + kx] : make_float2(0.f, 0.f);
        }
        __syncthreads();
        int flip = 0;
        line.template run<-1, true>(v, j, buf0 + c, buf1 + c, KX, tw, flip);
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            if (colok && ky < n) {
                const size_t row = (size_t)ky * P.lNx;
                // (the zero band's row spectra do not reach the result)
                v[r] = column_active(P, kx) ? cmul(v[r], P.tab.G[row + kx]) : make_float2(0.f, 0.f);
                if (P.gain)
                    v[r] = cscale(v[r], P.gain[row + kg]);
                if (P.again)
                    v[r] = cmul(v[r], P.again[a * K + row + kg]);
            }
        }
    }
    if (!colok)
        return;
    float2 *dst = spec + slot * K + (size_t)kx * n;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int ky = j + r * L::TPL;
        if (ky < n)
            dst[ky] = v[r];
    }
}

// (b0) z-prefilter boundary rows, once per slab (order >= 2).  The
// prefiltered propagator of plane p is E_p + alpha z^p + beta z^(nz-1-p); by
// linearity the alpha and beta parts are transformed once here (Tab[u][0] =
// column transform of G X alpha, Tab[u][1] of G X beta) and the row stage adds
// z^p Tab[u][0] + z^(nz-1-p) Tab[u][1] to the first and last planes' rows.
// The opposite view of a unit (PAIR) enters with alpha and beta exchanged:
// its plane p is plane nz-1-p of its own slab.
template <class L, int KX, int YF, bool PAIR>
__global__ void __launch_bounds__(KX * L::TPL) k_columns_boundary(StageParams P, L line, const float2 *spec,
                                                                  float2 *Tab)
{
    if (!group_active<KX>(P, blockIdx.x * KX))
        return;  // all-zero columns: the row stage never reads them
    extern __shared__ float2 smem[];
    const int n = line.size();
    const int ls = xslots<true>(n);
    float2 *buf0 = smem, *buf1 = smem + KX * ls, *tw = smem + 2 * KX * ls, *edge = tw + tw_slots(n);
    copy_twiddles<L>(tw, P.tab.twy, n);
    const int c = threadIdx.x % KX, j = threadIdx.x / KX;
    const int kx = blockIdx.x * KX + c;
    const bool colok = kx < P.lNx;
    const int u = blockIdx.y;
    const size_t K = (size_t)P.lNy * P.lNx;
    __syncthreads();
    int flip = 0;
    const float2 *su = spec + (size_t)(PAIR ? 2 * u : u) * K + kx;
    const int np = P.npoles;
#pragma unroll 1
    for (int t = 0; t < 2 * np; ++t) {
        const int i = t < np ? t : t - np;
        const float2 *tab = (t < np ? P.tab.alpha : P.tab.beta) + i * K + kx;
        const float2 *opp = (t < np ? P.tab.beta : P.tab.alpha) + i * K + kx;
        float2 v[L::SLOTS];
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            v[r] = make_float2(0.f, 0.f);
            if (colok && ky < n) {
                const size_t k = (size_t)ky * P.lNx;
                v[r] = cmul(su[k], tab[k]);
                if (PAIR)
                    v[r] = cfma(su[K + k], opp[k], v[r]);
            }
        }
        column_inverse_store<L, KX, YF>(P, line, v, c, j, colok, buf0, buf1, tw, edge, flip,
                                        Tab + ((size_t)(u * 2 * np + t) * P.ny) * P.lNx + kx);
    }
}

// (b1) columns: for the z planes of jobs q in [q0, q0+qn) (q = u*nz + p):
// the filtered spectrum times the propagator (exact anchor, then a complex
// recurrence), backward FFT along the column, crop.  PAIR: the unit's opposite
// view is added with its own propagator (the header comment), which the
// conjugate step advances.
// Output T[q-q0][row][kx], the P.trows rows from padded row P.trow0 on: the
// crop and, from order 2, the npoles samples before and after it, from which
// the row stage solves the column axis' prefilter boundary terms.  (Adding
// them here needs samples that a few other threads hold, a barrier per plane:
// tilted 200^3 columns 30.4 ms against 24.8 ms.)
// HALF (half_crop plans): the crop is slots 2..5 of every thread, without
// predicates.
template <class L, int KX, bool HALF, bool PAIR>
__global__ void __launch_bounds__(KX * L::TPL, (KX * L::TPL <= 256) ? 3 : ((KX * L::TPL <= 512) ? 2 : 1))
    k_columns_propagate(StageParams P, L line, const float2 *spec, float2 *T, int q0, int qn, int ppc, int anchor)
{
    if (!group_active<KX>(P, blockIdx.x * KX))
        return;  // all-zero columns: the row stage never reads them
    // power-of-two columns: the per-element propagator step lives in
    // registers and (N >= 512) the third radix-8 pass reads
    // per-thread-class twiddles (with long runs, tilted 200^3 step 72.1 ->
    // 70.6 ms; same box)
    constexpr bool STEP_REGS = column_regs<L, KX, HALF>();
    constexpr bool TW2 = STEP_REGS && kColumnTw2 && pow2_len<L>() >= 512;
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNy
    const int ls = xslots<true>(n);
    float2 *buf0 = smem, *buf1 = smem + KX * ls, *tw = smem + 2 * KX * ls;
    float2 *stp = tw + (TW2 ? tw_slots2(n) : tw_slots(n));  // [n][KX] propagator step (not STEP_REGS)
    if constexpr (TW2)
        copy_twiddles2<L>(tw, P.tab.twy, n);
    else
        copy_twiddles<L>(tw, P.tab.twy, n);
    const int c = threadIdx.x % KX, j = threadIdx.x / KX;
    const int kx = blockIdx.x * KX + c;
    const bool colok = kx < P.lNx;
    const int lNx = P.lNx, nz = P.nz;
    const size_t K = (size_t)n * lNx;
    const int qb = q0 + blockIdx.y * ppc;
    const int qe = min(q0 + qn, qb + ppc);
    float2 St[L::SLOTS];  // STEP_REGS: exp(i w) of this thread's elements
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {  // (columns beyond lNx: never stored)
        const int ky = j + r * L::TPL;
        const float2 t = (colok && ky < n) ? P.tab.step[(size_t)ky * lNx + kx] : make_float2(1.f, 0.f);
        if constexpr (STEP_REGS)
            St[r] = t;
        else if (ky < n)
            stp[ky * KX + c] = t;  // read back only by this thread
    }
    __syncthreads();

    float2 V[L::SLOTS];                    // G X exp(i w z_p) for this thread's elements
    float2 W[PAIR ? L::SLOTS : 1];         // the opposite view's
    int flip = 0;
    int cur_u = -1;
    int since = 0;  // planes advanced by the recurrence since the last exact anchor
    int u = qb / nz, p = qb % nz;
    const long long tstep = (long long)P.trows * lNx;  // T elements per plane
    float2 *d = T + (qb - q0) * tstep + (long long)(j - P.trow0) * lNx + kx;
    const int t0 = j - P.trow0;
    for (int q = qb; q < qe; ++q, ++p, d += tstep) {
        if (p == nz) {
            p = 0;
            ++u;
        }
        if (u != cur_u || since == anchor) {
            // exact anchor at the first plane of a unit, and again every
            // `anchor` planes: the FP32 recurrence drifts by about one
            // rounding per plane (measured on the 256^3 workload: rel-L2 to
            // the FP64 oracle 3.5e-7 with anchors every 32 planes, 1.6e-6
            // with one anchor per 256-plane run)
            const float zp = (float)p - 0.5f * (float)nz + P.zshift;
            const float zo = 2.f * P.zshift - 1.f - zp;  // the opposite view's plane
            const float2 *su = spec + (size_t)(PAIR ? 2 * u : u) * K;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int ky = j + r * L::TPL;
                V[r] = make_float2(0.f, 0.f);
                if (PAIR)
                    W[r] = make_float2(0.f, 0.f);
                if (colok && ky < n) {
                    const size_t k = (size_t)ky * lNx + kx;
                    const float2 w = P.tab.wsplit[k];
                    V[r] = cmul(su[k], expi_phase(w, zp));
                    if (PAIR)
                        W[r] = cmul(su[K + k], expi_phase(w, zo));
                }
            }
            cur_u = u;
            since = 0;
        }
        ++since;
        float2 v[L::SLOTS];
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            v[r] = PAIR ? V[r] + W[r] : V[r];
            if (STEP_REGS || HALF || ky < n) {  // (power-of-two lines: ky < n)
                float2 st;
                if constexpr (STEP_REGS)
                    st = St[r];
                else
                    st = stp[ky * KX + c];
                V[r] = cmul(V[r], st);
                if (PAIR)
                    W[r] = cmul_conj(W[r], st);
            }
        }
        line.template run<1, true, TW2>(v, j, buf0 + c, buf1 + c, KX, tw, flip);
        if constexpr (HALF) {
            constexpr int N = L::N, TPL = L::TPL;  // lNx is N too
            const int np = P.npoles;
#pragma unroll
            for (int r = 2; r <= 5; ++r)
                d[r * TPL * N] = v[r];
            if (j >= TPL - np)
                d[1 * TPL * N] = v[1];
            if (j < np)
                d[6 * TPL * N] = v[6];
        } else if (colok) {
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r)
                if ((unsigned)(t0 + r * L::TPL) < (unsigned)P.trows)
                    d[r * L::TPL * lNx] = v[r];
        }
    }
}

// ---------------------------------------------------------------------------
// (b2) rows: (+ the column axis' prefilter terms, + z-boundary rows), backward
// FFT along the row, the row axis' prefilter terms (ROWPF: tilted path), crop
// -> slab [a][z][x][y] (y innermost, pitch P.ypitch: a multiple of 32, or 1 for
// single-row planes).  P is transposed(): rows run along y, one per x, so
// a row's crop is contiguous in the slab and is stored straight from
// registers.  A CTA owns RG consecutive rows of one plane (job) and transforms
// them in groups of LPC lines (one line per TPL threads); the T values of the
// next group are loaded (evict-first) while the current one is transformed.
// When a line is whole warps, its FFT exchanges sync only its own warps
// (named barrier) and the lines never wait for each other.
// HALF (half_crop plans): the cropped outputs are slots 2..5 of every
// thread and the edge samples sit at compile-time slots.
// NP: prefilter poles (0 below order 2).
template <int LPC>
constexpr int rows_per_cta()
{
    // 16 rows share the CTA's set-up (twiddle table, boundary weights; 256^3
    // row stage with 8 / 16 / 32 rows, before it stored rows directly: 21.7 /
    // 20.9 / 21.2 ms for 200 single views)
    return LPC >= 16 ? LPC : 16;
}

// The column stage leaves its axis' prefilter boundary terms to this stage
// (order >= 2).  A CTA with rows within ZPOW_N of either end of the crop
// solves each column's coefficients once, from the job's samples around the
// crop's ends, into shared memory (lines of up to 2048; longer lines solve them per row),
// and those rows add the terms before the z-boundary rows.
template <class L>
constexpr bool ycoef_smem()
{
    return pow2_len<L>() == 0 || pow2_len<L>() <= 2048;
}
template <class L, int NP>
constexpr size_t smem_rows_y(int n)
{
    return (NP > 0 && ycoef_smem<L>()) ? (size_t)2 * NP * n * sizeof(float2) : 0;
}
template <class L, int LPC, int NP, bool ROWPF, bool HALF>
__global__ void __launch_bounds__(LPC * L::TPL, (LPC * L::TPL <= 256) ? 4 : 1)
    k_rows_inverse(StageParams P, L line, const float2 *T, const float2 *Tab, float2 *slab, int q0)
{
    constexpr int RG = rows_per_cta<LPC>(), G = RG / LPC;
    constexpr int NPA = NP > 0 ? NP : 1;  // array extents
    extern __shared__ float2 smem[];
    const int n = line.size();  // the row's padded length
    const int ls = xslots<false>(n);
    float2 *buf0 = smem, *buf1 = smem + LPC * ls, *tw = smem + 2 * LPC * ls;
    float2 *edge = tw + tw_slots(n);          // [LPC][EDGE_SLOTS]
    float2 *ycs = edge + EDGE_SLOTS * LPC;    // [2 NP][n] column-axis coefficients
    // (a third-pass twiddle table costs more to set up per CTA than its
    // conflict-free reads save here)
    copy_twiddles<L>(tw, P.tab.twx, n);
    // A direct transform's lines are interleaved, a warp holding 32 / LPC outputs
    // of each, so that fewer of its twiddle reads (their stride is the summation
    // index) meet on a bank, and its slots past the line are skipped.  41 views
    // of 33 x 256 unpadded: row stage 6.34 ms with the layout of the power-of-two
    // lines, 5.47 interleaved, 2.71 like this (the column stage, which had these
    // transforms before the stages were transposed, took 4.81).
    constexpr bool MIX = pow2_len<L>() == 0;
    const int l = MIX ? threadIdx.x % LPC : threadIdx.x / L::TPL, j = MIX ? threadIdx.x / LPC : threadIdx.x % L::TPL;
    constexpr int ES = MIX ? LPC : 1;
    float2 *line0 = buf0 + (MIX ? l : l * ls), *line1 = buf1 + (MIX ? l : l * ls);
    // lines of whole warps sync on named barrier 1 + l
    const int bar = (!MIX && L::TPL % 32 == 0 && LPC < 15) ? 1 + l : 0;
    const int ny = P.ny, nx = P.nx, nz = P.nz, padxl = P.padxl;
    const int cpj = (ny + RG - 1) / RG;  // CTAs per job
    // (last jobs first: their T rows are the ones still in L2)
    const int bid = (int)gridDim.x - 1 - (int)blockIdx.x;
    const int qrel = bid / cpj;
    const int ybase = (bid - qrel * cpj) * RG;
    const int GV = min(G, (ny - ybase + LPC - 1) / LPC);  // groups holding a row
    const int qq = q0 + qrel;  // the grid covers exactly the launch's jobs
    const int a = qq / nz, p = qq - a * nz;
    // z-boundary weights of this plane: z_i^p (alpha rows), z_i^(nz-1-p)
    // (beta rows), per pole
    float zl[NPA], zh[NPA];
    bool zb_any = false;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        zl[i] = p < ZPOW_N ? P.tab.zpow[i * ZPOW_N + p] : 0.f;
        zh[i] = nz - 1 - p < ZPOW_N ? P.tab.zpow[i * ZPOW_N + nz - 1 - p] : 0.f;
        zb_any = zb_any || zl[i] != 0.f || zh[i] != 0.f;
    }
    // a direct transform's slots past the line (uniform over the CTA)
    auto beyond = [&](int r) { return MIX && r * L::TPL >= n; };
    // slots of this thread in the all-zero column band or beyond the line
    unsigned zmask = 0;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        if (beyond(r))
            break;
        if (!column_active(P, j + r * L::TPL))
            zmask |= 1u << r;
    }
    unsigned long long eheld = 0;
    if constexpr (ROWPF && !HALF && L::SLOTS <= 8)
        eheld = edge_holdings<L, NPA>(padxl, nx, n, j);
    int epos[MIX && ROWPF ? EDGE_SLOTS : 1];
    if constexpr (MIX && ROWPF) {
#pragma unroll
        for (int e = 0; e < EDGE_SLOTS; ++e)
            epos[e] = edge_used(e, NPA) ? (padxl + edge_offset(e, nx) + 2 * n) % n : 0;
    }
    // the job's T rows; crop row y is row y + crop0
    const float2 *Tj = T + (size_t)qrel * P.trows * n;
    const int crop0 = P.padyl - P.trow0;
    const float2 *Tq = Tj + (size_t)crop0 * n + j;
    auto edge_sample = [&](int e, int x) {
        return Tj[(size_t)P.tedge[e] * n + x];
    };
    // this thread's T values of row y (zeros for y >= ny or zero columns)
    auto load_row = [&](int y, float2 (&v)[L::SLOTS]) {
        const bool valid = HALF || y < ny;
        const float2 *src = Tq + (size_t)(valid ? y : 0) * n;
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            if (beyond(r))
                break;
            v[r] = (valid && !((zmask >> r) & 1u)) ? __ldcs(src + r * L::TPL) : make_float2(0.f, 0.f);
        }
    };
    if constexpr (NP > 0 && ycoef_smem<L>()) {
        if (ybase < ZPOW_N || min(ybase + RG, ny) - 1 >= ny - ZPOW_N) {
            for (int x = threadIdx.x; x < n; x += LPC * L::TPL) {
                float2 cy[2 * NPA];
                if (column_active(P, x)) {
                    float2 ed[EDGE_SLOTS];
#pragma unroll
                    for (int e = 0; e < EDGE_SLOTS; ++e)
                        ed[e] = edge_used(e, NP) ? edge_sample(e, x) : make_float2(0.f, 0.f);
                    pf_coefs<NPA>(P.kys, ed, cy);
                } else {
#pragma unroll
                    for (int i = 0; i < 2 * NP; ++i)
                        cy[i] = make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 2 * NP; ++i)
                    ycs[i * n + x] = cy[i];
            }
        }
    }
    // (direct transforms read nothing ahead: they would spill)
    float2 v[L::SLOTS], vn[MIX ? 1 : L::SLOTS];
    if constexpr (!MIX)
        load_row(ybase + l, v);
    __syncthreads();  // twiddles (and the coefficient rows)
    // kept across groups: with an odd number of exchanges per transform the
    // next group starts in the other buffer
    int flip = 0;
#pragma unroll 1
    for (int g = 0; g < GV; ++g) {
        const int y = ybase + g * LPC + l;
        const bool valid = HALF || y < ny;
        if constexpr (MIX)
            load_row(y, v);
        else if (g + 1 < GV)
            load_row(y + LPC, vn);
        if constexpr (NP > 0) {
            if (valid && (y < ZPOW_N || ny - 1 - y < ZPOW_N)) {
#pragma unroll
                for (int r = 0; r < L::SLOTS; ++r) {
                    if (beyond(r))
                        break;
                    if (!((zmask >> r) & 1u)) {
                        const int x = j + r * L::TPL;
                        float2 cy[2 * NPA];
                        if constexpr (ycoef_smem<L>()) {
#pragma unroll
                            for (int i = 0; i < 2 * NP; ++i)
                                cy[i] = ycs[i * n + x];
                        } else {
                            float2 ed[EDGE_SLOTS];
#pragma unroll
                            for (int e = 0; e < EDGE_SLOTS; ++e)
                                ed[e] = edge_used(e, NP) ? edge_sample(e, x) : make_float2(0.f, 0.f);
                            pf_coefs<NPA>(P.kys, ed, cy);
                        }
                        v[r] = pf_apply<NPA>(P, cy, y, ny, v[r]);
                    }
                }
            }
            if (valid && zb_any) {
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const float2 *ta = Tab + ((size_t)(a * 2 * NP + i) * ny + y) * n + j;
                    const float2 *tb = Tab + ((size_t)(a * 2 * NP + NP + i) * ny + y) * n + j;
#pragma unroll
                    for (int r = 0; r < L::SLOTS; ++r) {
                        if (beyond(r))
                            break;
                        if (!((zmask >> r) & 1u)) {
                            const float2 u = ta[r * L::TPL], w = tb[r * L::TPL];
                            v[r] = make_float2(fmaf(zh[i], w.x, fmaf(zl[i], u.x, v[r].x)),
                                               fmaf(zh[i], w.y, fmaf(zl[i], u.y, v[r].y)));
                        }
                    }
                }
            }
        }
        line.template run<1>(v, j, line0, line1, ES, tw, flip, bar);
        float2 cf[2 * NPA];
        if constexpr (ROWPF) {
            // the samples around the crop's ends, each held by one thread
            // (its previous group's readers are past this transform's barriers)
            if constexpr (HALF) {
#pragma unroll
                for (int e = 0; e < EDGE_SLOTS; ++e) {
                    float2 t;
                    if (edge_used(e, NP) && held<L>(v, j, n / 4 + edge_offset(e, n / 2), t))
                        edge[l * EDGE_SLOTS + e] = t;
                }
            } else if constexpr (L::SLOTS <= 8) {
                if (eheld) {
#pragma unroll
                    for (int r = 0; r < L::SLOTS; ++r) {
                        if (beyond(r))
                            break;
                        const unsigned m = (unsigned)(eheld >> (8 * r)) & 0xffu;
                        if (m) {
#pragma unroll
                            for (int e = 0; e < EDGE_SLOTS; ++e)
                                if (edge_used(e, NP) && (m & (1u << e)))
                                    edge[l * EDGE_SLOTS + e] = v[r];
                        }
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < EDGE_SLOTS; ++e) {
                    // (v is in local memory: a run-time index)
                    if (edge_used(e, NP) && (epos[e] & (L::TPL - 1)) == j)
                        edge[l * EDGE_SLOTS + e] = v[epos[e] / L::TPL];
                }
            }
            if (bar > 0)
                line_sync(bar, L::TPL);
            else
                __syncthreads();
            pf_coefs<NPA>(P.kxs, edge + l * EDGE_SLOTS, cf);
        }
        if (valid) {
            float2 *dst = slab + (((size_t)a * nz + p) * ny + y) * P.ypitch;
            if constexpr (HALF) {
                dst += j;
#pragma unroll
                for (int r = 2; r <= 5; ++r) {
                    float2 o = v[r];
                    if constexpr (ROWPF)
                        o = pf_apply<NPA>(P, cf, j + L::TPL * (r - 2), n / 2, o);
                    __stcs(dst + (r - 2) * L::TPL, o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < L::SLOTS; ++r) {
                    if (beyond(r))
                        break;
                    const int xx = j + r * L::TPL - padxl;
                    if (xx >= 0 && xx < nx) {
                        float2 o = v[r];
                        if constexpr (ROWPF)
                            o = pf_apply<NPA>(P, cf, xx, nx, o);
                        __stcs(dst + xx, o);
                    }
                }
            }
        }
        if constexpr (!MIX) {
            if (g + 1 < GV) {
#pragma unroll
                for (int r = 0; r < L::SLOTS; ++r)
                    v[r] = vn[r];
            }
        }
    }
}

// (b1+b2) single-row planes (lNy == ny == 1, slab pitch 1: the 2D
// reconstruction): the column transforms are the identity, so a job's row
// is the filtered spectrum (k_spectrum_line) times the propagator of its
// plane, formed here instead of in a column stage (PAIR: plus the opposite
// view's, see the header comment).  A CTA takes RG
// consecutive jobs as groups of LPC lines (one job per line).  With one
// line per group the propagator is anchored exactly at the CTA's first job
// (and wherever the unit changes) and advanced plane by plane with the
// complex step exp(i w), as in k_columns_propagate; with several lines per
// group every line is anchored exactly.  Then per line the z-boundary rows
// of its plane, the backward FFT along x, the x-prefilter boundary terms,
// and the cropped row stored contiguously at slab[a][p][x].
template <int LPC>
constexpr int line_jobs_per_cta()
{
    return LPC >= 8 ? LPC : 8;
}
template <class L, int LPC, int NP, bool PAIR>
__global__ void __launch_bounds__(LPC * L::TPL, (LPC * L::TPL <= 256) ? 3 : 1)
    k_rows_line(StageParams P, L line, const float2 *spec, const float2 *Tab, float2 *slab, int q0, int qn)
{
    constexpr int RG = line_jobs_per_cta<LPC>(), G = RG / LPC;
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNx
    const int ls = xslots<false>(n);
    float2 *buf0 = smem, *buf1 = smem + LPC * ls, *tw = smem + 2 * LPC * ls;
    copy_twiddles<L>(tw, P.tab.twx, n);
    const int l = threadIdx.x / L::TPL, j = threadIdx.x % L::TPL;
    const int bar = (L::TPL % 32 == 0 && LPC < 15) ? 1 + l : 0;
    const int nx = P.nx, nz = P.nz, padxl = P.padxl;
    const bool pf = P.order >= 2;
    const int qbase = (int)blockIdx.x * RG;
    const int GV = min(G, (qn - qbase + LPC - 1) / LPC);  // groups holding a job
    // LPC == 1: the next plane's propagated spectrum, of the first and the
    // opposite view
    float2 V[L::SLOTS], W[PAIR ? L::SLOTS : 1];
    int cur_a = -1;
    __syncthreads();  // twiddles
#pragma unroll 1
    for (int g = 0; g < GV; ++g) {
        const int qrel = qbase + g * LPC + l;
        const bool valid = qrel < qn;
        const int q = q0 + (valid ? qrel : 0);
        const int a = q / nz, p = q - a * nz;
        float2 v[L::SLOTS];
        if (LPC > 1 || a != cur_a) {
            const float zp = (float)p - 0.5f * (float)nz + P.zshift;
            const float zo = 2.f * P.zshift - 1.f - zp;
            const float2 *su = spec + (size_t)(PAIR ? 2 * a : a) * n;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int x = j + r * L::TPL;
                V[r] = make_float2(0.f, 0.f);
                if (PAIR)
                    W[r] = make_float2(0.f, 0.f);
                if (valid && column_active(P, x)) {
                    const float2 w = P.tab.wsplit[x];
                    V[r] = cmul(su[x], expi_phase(w, zp));
                    if (PAIR)
                        W[r] = cmul(su[n + x], expi_phase(w, zo));
                }
            }
            cur_a = a;
        }
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int x = j + r * L::TPL;
            v[r] = PAIR ? V[r] + W[r] : V[r];
            if (LPC == 1 && column_active(P, x)) {
                const float2 st = P.tab.step[x];
                V[r] = cmul(V[r], st);
                if (PAIR)
                    W[r] = cmul_conj(W[r], st);
            }
        }
        if (valid && pf) {
            constexpr int np = NP;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float zl = (i < np && p < ZPOW_N) ? P.tab.zpow[i * ZPOW_N + p] : 0.f;
                const float zh = (i < np && nz - 1 - p < ZPOW_N) ? P.tab.zpow[i * ZPOW_N + nz - 1 - p] : 0.f;
                if (zl != 0.f || zh != 0.f) {
                    const float2 *ta = Tab + (size_t)(a * 2 * np + i) * n;
                    const float2 *tb = Tab + (size_t)(a * 2 * np + np + i) * n;
#pragma unroll
                    for (int r = 0; r < L::SLOTS; ++r) {
                        const int x = j + r * L::TPL;
                        if (column_active(P, x)) {
                            const float2 u = ta[x], w = tb[x];
                            v[r] = make_float2(fmaf(zh, w.x, fmaf(zl, u.x, v[r].x)),
                                               fmaf(zh, w.y, fmaf(zl, u.y, v[r].y)));
                        }
                    }
                }
            }
        }
        int flip = 0;
        line.template run<1>(v, j, buf0 + l * ls, buf1 + l * ls, 1, tw, flip, bar);
        float2 cf[2 * NP];
        if (pf) {
            // the line's samples at x0-1, x0+1, x1-1, x1+1 (periodic), through
            // the exchange buffer the FFT's last exchange did not use
            float2 *sc = (flip ? buf1 : buf0) + l * ls;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int x = j + r * L::TPL;
                if (x < n)
                    sc[x] = v[r];
            }
            if (bar > 0)
                line_sync(bar, L::TPL);
            else
                __syncthreads();
            float2 ed[EDGE_SLOTS];
#pragma unroll
            for (int e = 0; e < EDGE_SLOTS; ++e)
                ed[e] = edge_used(e, NP) ? sc[(padxl + edge_offset(e, nx) + 2 * n) % n] : make_float2(0.f, 0.f);
            pf_coefs<NP>(P.kxs, ed, cf);
        }
        if (valid) {
            float2 *dst = slab + ((size_t)a * nz + p) * nx;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int xx = j + r * L::TPL - padxl;
                if (xx >= 0 && xx < nx) {
                    float2 o = v[r];
                    if (pf)
                        o = pf_apply<NP>(P, cf, xx, nx, o);
                    __stcs(dst + xx, o);
                }
            }
        }
        // the edge reads of this group end before the next group's FFT
        // writes the exchange buffers
        if (g + 1 < GV) {
            if (bar > 0)
                line_sync(bar, L::TPL);
            else
                __syncthreads();
        }
    }
}

// (a2, b0) the filtered spectra (in place) and z-boundary rows of single-row
// planes, whose column transforms are the identity.  One thread per (unit, kx).
__global__ void __launch_bounds__(256) k_spectrum_line(StageParams P, float2 *rowspec, float2 *Tab, int nunits)
{
    const int lNx = P.lNx;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)nunits * lNx)
        return;
    const int u = (int)(id / lNx), kx = (int)(id - (long long)u * lNx);
    const int2 views = P.units ? P.units[u] : make_int2(u, -1);
    float2 *spec = rowspec + (size_t)(P.units ? 2 * u : u) * lNx + kx;
    auto filtered = [&](float2 x, int a, int kg) {
        x = cmul(x, P.tab.G[kx]);
        if (P.gain)
            x = cscale(x, P.gain[kg]);
        if (P.again)
            x = cmul(x, P.again[(size_t)a * lNx + kg]);
        return x;
    };
    const bool act = column_active(P, kx);
    const float2 zero = make_float2(0.f, 0.f);
    const float2 g = act ? filtered(spec[0], views.x, kx) : zero;
    const float2 h = (act && views.y >= 0) ? filtered(spec[lNx], views.y, kx ? lNx - kx : 0) : zero;
    spec[0] = g;
    if (P.units)
        spec[lNx] = h;
    const int np = P.npoles;
    for (int i = 0; i < np; ++i) {
        const float2 al = P.tab.alpha[(size_t)i * lNx + kx], be = P.tab.beta[(size_t)i * lNx + kx];
        float2 ta = cmul(g, al), tb = cmul(g, be);
        if (P.units) {
            ta = cfma(h, be, ta);
            tb = cfma(h, al, tb);
        }
        Tab[(size_t)(u * 2 * np + i) * lNx + kx] = ta;
        Tab[(size_t)(u * 2 * np + np + i) * lNx + kx] = tb;
    }
}

// ---------------------------------------------------------------------------
// Planes per column-stage CTA: the run length that takes the fewest plane
// times, whole waves of the resident CTAs over the active column groups, with
// a start-up (tables, exact anchor) counted as four planes.  At most 256 for
// long runs (long_runs), else at most kReanchorPlanes.
template <int KX>
static int active_groups(const StageParams &P)
{
    const int groups = (P.lNx + KX - 1) / KX;
    int active = 0;
    for (int g = 0; g < groups; ++g)
        if (!(g * KX >= P.kx_zero_lo && g * KX + KX <= P.kx_zero_hi))
            ++active;
    return active;
}
template <int KX>
static int planes_per_cta(const StageParams &P, int qn, bool long_run)
{
    const int active = active_groups<KX>(P);
    const int slots = std::max(1, P.col_slots), cap = std::min(long_run ? 256 : kReanchorPlanes, qn);
    int best = cap;
    long long least = -1;
    for (int ppc = cap; ppc >= std::min(4, cap); --ppc) {
        const long long ctas = (long long)active * ((qn + ppc - 1) / ppc);
        const long long t = (ctas + slots - 1) / slots * (ppc + 4);
        if (least < 0 || t < least) {
            least = t;
            best = ppc;
        }
    }
    return best;
}

// Planes between anchors: what one wave of up to 1024 planes gives a CTA, 4 to
// 32, in equal parts of a slab.  Few column groups make long runs of small
// planes, whose anchors cost little: 64^3 from 60 views with anchors every 32 /
// 16 / 8 planes 323 / 320 / 333 us at rel-L2 2.0 / 1.7 / 1.6e-7, 256^3 from 200
// views 26.6 / 27.3 / 28.7 ms at 2.6 / 2.4 / 2.4e-7.  Opposite views drift
// together from one anchor where single ones do so apart, so below 512 points,
// where that shows (128^3 2.71e-7 against 2.60e-7 for single views), units
// take three quarters of it.
template <int KX>
static int anchor_planes(const StageParams &P, int qn)
{
    const int slots = std::max(1, P.col_slots);
    const int wave = (std::min(qn, 1024) * active_groups<KX>(P) + slots - 1) / slots;
    int most = std::min(kReanchorPlanes, std::max(4, wave));
    if (P.units && P.lNy < 512)
        most = std::max(4, most * 3 / 4);
    const int parts = (P.nz + most - 1) / most;
    return (P.nz + parts - 1) / parts;
}

// Shared memory of the column kernel: the exchange buffers, the twiddle
// tables and, where the propagator steps are not in registers, the steps.
template <class L, bool HALF>
static size_t smem_cols_prop(int n)
{
    constexpr int KX = Cfg<L>::KX;
    constexpr bool regs = column_regs<L, KX, HALF>();
    const bool tw2 = regs && kColumnTw2 && pow2_len<L>() >= 512;
    return (size_t)(2 * KX * xslots<true>(n) + (tw2 ? tw_slots2(n) : tw_slots(n)) + (regs ? 0 : KX * n)) *
           sizeof(float2);
}

// Calls fn(std::integral_constant<int, V>) for V = v (one of 0, 1, 2), so a
// pole count chosen at run time selects a compile-time instantiation.
template <class F>
static cudaError_t with_poles(int v, F &&fn)
{
    switch (v) {
    case 0: return fn(std::integral_constant<int, 0>{});
    case 1: return fn(std::integral_constant<int, 1>{});
    case 2: return fn(std::integral_constant<int, 2>{});
    default: return cudaErrorInvalidValue;
    }
}
// Prefilter poles of the transposed stages (0 below order 2).
static int stage_poles(const StageParams &P)
{
    return P.order >= 2 ? P.npoles : 0;
}

template <class L>
static cudaError_t rows_forward_impl(const StageParams &P, L line, const void *sino, const double *w, int nslots,
                                     float2 *out, cudaStream_t s)
{
    constexpr int LPC = Cfg<L>::LPC;
    const long long lines = (long long)nslots * P.lNy;
    const unsigned grid = (unsigned)((lines + LPC - 1) / LPC);
    k_rows_forward<L, LPC><<<grid, LPC * L::TPL, smem_rows<L>(line.n), s>>>(P, line, sino, w, nslots, out);
    return cudaGetLastError();
}

template <class L>
static cudaError_t spectrum_impl(const StageParams &P, L line, const float2 *rowspec, float2 *spec, int nslots,
                                 cudaStream_t s)
{
    constexpr int KX = Cfg<L>::KX;
    dim3 grid((P.lNx + KX - 1) / KX, nslots);
    k_columns_spectrum<L, KX><<<grid, KX * L::TPL, smem_cols<L>(line.n), s>>>(P, line, rowspec, spec);
    return cudaGetLastError();
}

template <class L>
static cudaError_t boundary_impl(const StageParams &P, L line, const float2 *spec, float2 *Tab, int nunits,
                                 cudaStream_t s)
{
    constexpr int KX = Cfg<L>::KX;
    dim3 grid((P.lNx + KX - 1) / KX, nunits);
    return with_poles(stage_poles(P), [&](auto yf) {
        constexpr int YF = decltype(yf)::value;
        if constexpr (YF > 0) {
            if (P.units)
                k_columns_boundary<L, KX, YF, true>
                    <<<grid, KX * L::TPL, smem_cols<L>(line.n), s>>>(P, line, spec, Tab);
            else
                k_columns_boundary<L, KX, YF, false>
                    <<<grid, KX * L::TPL, smem_cols<L>(line.n), s>>>(P, line, spec, Tab);
            return cudaGetLastError();
        } else {
            return cudaErrorInvalidValue;
        }
    });
}

// Lines of the half-crop kernels.
template <class L>
constexpr bool half_line()
{
    return pow2_len<L>() > 0;
}
template <class L, bool HALF, bool PAIR>
static cudaError_t columns_launch(const StageParams &P, L line, const float2 *spec, float2 *T, int q0, int qn,
                                  cudaStream_t s)
{
    constexpr int KX = Cfg<L>::KX;
    const int ppc = planes_per_cta<KX>(P, qn, long_runs<L, KX>());
    dim3 grid((P.lNx + KX - 1) / KX, (qn + ppc - 1) / ppc);
    k_columns_propagate<L, KX, HALF, PAIR>
        <<<grid, KX * L::TPL, smem_cols_prop<L, HALF>(line.n), s>>>(P, line, spec, T, q0, qn, ppc, anchor_planes<KX>(P, qn));
    return cudaGetLastError();
}
template <class L>
static cudaError_t columns_impl(const StageParams &P, L line, const float2 *spec, float2 *T, int q0, int qn,
                                cudaStream_t s)
{
    if constexpr (half_line<L>()) {
        if (half_crop(P))
            return P.units ? columns_launch<L, true, true>(P, line, spec, T, q0, qn, s)
                           : columns_launch<L, true, false>(P, line, spec, T, q0, qn, s);
    }
    return P.units ? columns_launch<L, false, true>(P, line, spec, T, q0, qn, s)
                   : columns_launch<L, false, false>(P, line, spec, T, q0, qn, s);
}

template <class L, int NP>
static size_t smem_rows_inverse(int n)
{
    return smem_rows<L>(n) + smem_rows_y<L, NP>(n);
}
template <class L, int NP, bool ROWPF, bool HALF>
static cudaError_t rows_launch(const StageParams &P, L line, const float2 *T, const float2 *Tab, float2 *slab, int q0,
                               int qn, cudaStream_t s)
{
    constexpr int LPC = Cfg<L>::LPC, RG = rows_per_cta<LPC>();
    const unsigned grid = (unsigned)((long long)qn * ((P.ny + RG - 1) / RG));
    k_rows_inverse<L, LPC, NP, ROWPF, HALF>
        <<<grid, LPC * L::TPL, smem_rows_inverse<L, NP>(line.n), s>>>(P, line, T, Tab, slab, q0);
    return cudaGetLastError();
}
template <class L>
static cudaError_t rows_inverse_impl(const StageParams &P, L line, const float2 *T, const float2 *Tab,
                                     float2 *slab, int q0, int qn, cudaStream_t s)
{
    // scipy prefilters the row axis on the tilted path only, and leaves an
    // axis of length 1 alone
    return with_poles(stage_poles(P), [&](auto np) {
        constexpr int NP = decltype(np)::value;
        const bool rowpf = NP > 0 && P.tilted && P.nx >= 2;
        if constexpr (half_line<L>()) {
            if (half_crop(P)) {
                if constexpr (NP > 0) {
                    if (rowpf)
                        return rows_launch<L, NP, true, true>(P, line, T, Tab, slab, q0, qn, s);
                }
                return rows_launch<L, NP, false, true>(P, line, T, Tab, slab, q0, qn, s);
            }
        }
        if constexpr (NP > 0) {
            if (rowpf)
                return rows_launch<L, NP, true, false>(P, line, T, Tab, slab, q0, qn, s);
        }
        return rows_launch<L, NP, false, false>(P, line, T, Tab, slab, q0, qn, s);
    });
}

// The attribute is per kernel and process-wide, so it is always set to the
// largest size the instantiation can need (the generic line serves every
// length up to its maximum).
template <class F>
static cudaError_t allow_smem(F *kernel, size_t bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <class L, int NP, bool HALF>
static cudaError_t set_smem_attrs_crop(int n)
{
    constexpr int KX = Cfg<L>::KX, LPC = Cfg<L>::LPC;
    cudaError_t e = allow_smem(k_columns_propagate<L, KX, HALF, false>, smem_cols_prop<L, HALF>(n));
    if (e == cudaSuccess)
        e = allow_smem(k_columns_propagate<L, KX, HALF, true>, smem_cols_prop<L, HALF>(n));
    if (e == cudaSuccess)
        e = allow_smem(k_rows_inverse<L, LPC, NP, false, HALF>, smem_rows_inverse<L, NP>(n));
    if constexpr (NP > 0) {
        if (e == cudaSuccess)
            e = allow_smem(k_rows_inverse<L, LPC, NP, true, HALF>, smem_rows_inverse<L, NP>(n));
    }
    return e;
}
template <class L, int NP>
static cudaError_t set_smem_attrs_np(int n)
{
    constexpr int KX = Cfg<L>::KX, LPC = Cfg<L>::LPC;
    cudaError_t e = set_smem_attrs_crop<L, NP, false>(n);
    if constexpr (half_line<L>()) {
        if (e == cudaSuccess)
            e = set_smem_attrs_crop<L, NP, true>(n);
    }
    if constexpr (NP > 0) {
        if (e == cudaSuccess)
            e = allow_smem(k_rows_line<L, LPC, NP, false>, smem_rows<L>(n));
        if (e == cudaSuccess)
            e = allow_smem(k_rows_line<L, LPC, NP, true>, smem_rows<L>(n));
        if (e == cudaSuccess)
            e = allow_smem(k_columns_boundary<L, KX, NP, false>, smem_cols<L>(n));
        if (e == cudaSuccess)
            e = allow_smem(k_columns_boundary<L, KX, NP, true>, smem_cols<L>(n));
    }
    return e;
}

template <class L>
static cudaError_t set_smem_attrs(int n)
{
    if (std::is_same<L, GenericLine>::value)
        n = GenericLine::TPL * GenericLine::SLOTS;
    cudaError_t e;
    e = allow_smem(k_rows_forward<L, Cfg<L>::LPC>, smem_rows<L>(n));
    if (e == cudaSuccess)
        e = allow_smem(k_columns_spectrum<L, Cfg<L>::KX>, smem_cols<L>(n));
    if (e != cudaSuccess)
        return e;
    for (int np = 0; np <= 2; ++np) {
        e = with_poles(np, [&](auto v) { return set_smem_attrs_np<L, decltype(v)::value>(n); });
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

int columns_slots(const StageParams &P)
{
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const cudaError_t e = with_line(P.lNy, [&](auto line) {
        using L = decltype(line);
        constexpr int KX = Cfg<L>::KX;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_columns_propagate<L, KX, false, false>,
                                                             KX * L::TPL, smem_cols_prop<L, false>(line.n));
    });
    return e == cudaSuccess ? per * sms : 0;
}

bool line_size_supported(int n)
{
    switch (n) {
    case 64: case 128: case 256: case 512: case 1024: case 2048: case 4096: return true;
    default: return n >= 1 && n <= GenericLine::TPL * GenericLine::SLOTS;
    }
}

cudaError_t configure_kernels(const StageParams &P)
{
    cudaError_t e = with_line(P.lNx, [&](auto line) { return set_smem_attrs<decltype(line)>(line.n); });
    if (e != cudaSuccess)
        return e;
    return with_line(P.lNy, [&](auto line) { return set_smem_attrs<decltype(line)>(line.n); });
}

cudaError_t launch_rows_forward(const StageParams &P, const void *sino, const double *weights, int nslots,
                                float2 *rowspec, cudaStream_t s)
{
    return with_line(P.lNx, [&](auto line) {
        return rows_forward_impl(P, line, sino, weights, nslots, rowspec, s);
    });
}

cudaError_t launch_columns_propagate(const StageParams &P, const float2 *spec, float2 *T, int q0, int qn,
                                     cudaStream_t s)
{
    return with_line(P.lNy, [&](auto line) { return columns_impl(P, line, spec, T, q0, qn, s); });
}

bool half_crop(const StageParams &P)
{
    const int N = P.lNx;
    return P.lNy == N && N >= 64 && N <= 4096 && (N & (N - 1)) == 0 && 2 * P.ny == N && 2 * P.nx == N &&
           4 * P.padyl == N && 4 * P.padxl == N && P.nz == P.nx && P.ypitch == P.ny;
}

bool single_row_plan(const StageParams &P)
{
    return P.lNy == 1 && P.ny == 1 && P.padyl == 0 && P.ypitch == 1;
}

cudaError_t launch_rows_line(const StageParams &P, const float2 *spec, const float2 *Tab, float2 *slab, int q0,
                             int qn, cudaStream_t s)
{
    return with_line(P.lNx, [&](auto line) {
        using L = decltype(line);
        constexpr int LPC = Cfg<L>::LPC;
        const unsigned grid = (unsigned)((qn + line_jobs_per_cta<LPC>() - 1) / line_jobs_per_cta<LPC>());
        // (one pole's kernel also runs orders 0 and 1, without prefilter terms)
        return with_poles(std::max(1, stage_poles(P)), [&](auto np) {
            constexpr int NP = decltype(np)::value;
            if constexpr (NP >= 1) {
                if (P.units)
                    k_rows_line<L, LPC, NP, true>
                        <<<grid, LPC * L::TPL, smem_rows<L>(line.n), s>>>(P, line, spec, Tab, slab, q0, qn);
                else
                    k_rows_line<L, LPC, NP, false>
                        <<<grid, LPC * L::TPL, smem_rows<L>(line.n), s>>>(P, line, spec, Tab, slab, q0, qn);
                return cudaGetLastError();
            } else {
                return cudaErrorInvalidValue;
            }
        });
    });
}

cudaError_t launch_columns_spectrum(const StageParams &P, const float2 *rowspec, float2 *spec, int nslots,
                                    cudaStream_t s)
{
    return with_line(P.lNy, [&](auto line) { return spectrum_impl(P, line, rowspec, spec, nslots, s); });
}

cudaError_t launch_columns_boundary(const StageParams &P, const float2 *spec, float2 *Tab, int nunits, cudaStream_t s)
{
    return with_line(P.lNy, [&](auto line) { return boundary_impl(P, line, spec, Tab, nunits, s); });
}

cudaError_t launch_spectrum_line(const StageParams &P, float2 *spec, float2 *Tab, int nunits, cudaStream_t s)
{
    const long long n = (long long)nunits * P.lNx;
    k_spectrum_line<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(P, spec, Tab, nunits);
    return cudaGetLastError();
}

StageParams transposed(const StageParams &P)
{
    StageParams t = P;
    std::swap(t.ny, t.nx);
    std::swap(t.lNy, t.lNx);
    std::swap(t.padyl, t.padxl);
    std::swap(t.kx_zero_lo, t.ky_zero_lo);
    std::swap(t.kx_zero_hi, t.ky_zero_hi);
    std::swap(t.kxs, t.kys);
    t.tab = P.tabt;
    t.tabt = P.tab;
    // T rows: the crop and npoles samples on either side, or the whole column
    // where those would wrap around its ends
    t.trow0 = t.padyl - t.npoles;
    t.trows = t.ny + 2 * t.npoles;
    if (t.trow0 < 0 || t.trow0 + t.trows > t.lNy) {
        t.trow0 = 0;
        t.trows = t.lNy;
    }
    for (int e = 0; e < EDGE_SLOTS; ++e)
        t.tedge[e] = (t.padyl + edge_offset(e, t.ny) + 2 * t.lNy) % t.lNy - t.trow0;
    return t;
}

cudaError_t launch_rows_inverse(const StageParams &P, const float2 *T, const float2 *Tab, float2 *slab, int q0,
                                int qn, cudaStream_t s)
{
    return with_line(P.lNx, [&](auto line) { return rows_inverse_impl(P, line, T, Tab, slab, q0, qn, s); });
}

}  // namespace odt
