// Adjoint (vector-Jacobian product) of the filter stages, y-axis path.
//
// Forward, per angle a (stages.cu):
//   X  = FFT2(pad(w_a s_a))                          (rows, then columns)
//   V_p = G g X P_p,   P_p = exp(i w z_p) + zl_p alpha + zh_p beta
//   T_p = crop_y IFFT_y(V_p);  slab_p = L_x(T_p) = (crop_x + xfix) IFFT_x(T_p)
// with G the filter (prefilter particular factors folded in), g an optional
// real per-frequency gain, zl_p = pole^p, zh_p = pole^(nz-1-p).
//
// Adjoint, given slab_grad (from the transposed resampling, rotate.cu):
//   T_p_grad = FFT_x((crop_x + xfix)^T slab_grad_p)          k_adj_rows
//   Z_p      = FFT_y(crop_y^T T_p_grad)
//   Q        = sum_p conj(P_p) Z_p                            k_adj_columns
//   dg      += Re(conj(G X) Q)   (X recomputed)               k_adj_spectrum
//   X_grad   = conj(G g) Q;  W = IFFT_y(X_grad)               k_adj_spectrum
//   P_grad   = IFFT_x(W)                                      k_adj_rows_full
//   s_grad   = w_a pad^T(P_grad)                              k_adj_pad
// The adjoint of an unnormalised backward FFT is the unnormalised forward
// FFT and vice versa; the transpose of the x-prefilter boundary terms
// collects two weighted sums of the cotangent and scatters them onto the
// four samples outside the crop.
//
// Opposite views (units of two angles, see stages.cu): both views' spectra
// take their gradient from the shared slab's Z_p, the second one against the
// propagator of its own plane nz-1-p,
//   conj(e^(i w (c - z_p))) Z_p = conj(e^(i w c)) e^(i w z_p) Z_p,  c = 2 zshift - 1,
// so one propagator recurrence serves both and the constant factor is applied
// when the sum is complete.  The second view's row gradients are mirrored.
#include "odt_fft.cuh"
#include "odt_internal.cuh"
#include "odt_stage_util.cuh"

namespace odt {

// Rows: crop_x/xfix transpose + forward FFT along x.  A CTA transforms G
// groups of LPC consecutive rows: they share its twiddle table, and the next
// group's loads are in flight while the current one is transformed.  The
// boundary sums are formed with shuffles: shared-memory float atomics on one
// address are compare-and-swap loops, and 24 lanes of every line met on them
// (128^3 from 90 views: 1.13 ms with the atomics, 0.60 ms like this).
template <int LPC>
constexpr int adj_row_groups()
{
    return LPC >= 32 ? 1 : 32 / LPC;
}
template <class L, int LPC>
__global__ void __launch_bounds__(LPC * L::TPL, (LPC * L::TPL <= 256) ? 4 : 1)
    k_adj_rows(StageParams P, L line, const float2 *sgrad, float2 *Tg, int q0, int qn)
{
    constexpr int G = adj_row_groups<LPC>();
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNx
    const int xs = xslots<false>(n);
    float2 *buf0 = smem, *buf1 = smem + LPC * xs, *tw = smem + 2 * LPC * xs;
    constexpr int WPL = L::TPL / 32;  // warps per line (0: less than one)
    float4 *red = reinterpret_cast<float4 *>(tw + (tw_slots(n) + 1) / 2 * 2);  // [LPC][WPL] partial boundary sums
    copy_twiddles<L>(tw, P.tab.twx, n);
    const int l = threadIdx.x / L::TPL, j = threadIdx.x % L::TPL;
    // lines of whole warps sync on named barrier 1 + l
    const int bar = (L::TPL % 32 == 0 && LPC < 15) ? 1 + l : 0;
    const int ny = P.ny, nx = P.nx, nz = P.nz, padxl = P.padxl;
    const long long rows = (long long)qn * ny, row0 = (long long)blockIdx.x * LPC * G;
    const int GV = (int)min((long long)G, (rows - row0 + LPC - 1) / LPC);  // groups holding a row
    const bool tl = P.tilted != 0;
    const bool pf = P.order >= 2;
    // this thread's cotangents of row rid.  Slab gradient of (a, y, p, xx):
    // [a][y][z][x] from the y-axis resampling transpose, the forward slab
    // layout [a][z][x][ypitch] from the tilted one
    auto load_row = [&](long long rid, float2 (&v)[L::SLOTS]) {
        const bool valid = rid < rows;
        const int qq = q0 + (int)((valid ? rid : 0) / ny), y = (int)((valid ? rid : 0) % ny);
        const int a = qq / nz, p = qq % nz;
        const float2 *src = tl ? sgrad + ((size_t)a * nz + p) * nx * P.ypitch + y
                               : sgrad + (((size_t)a * ny + y) * nz + p) * nx;
        const size_t xstep = tl ? (size_t)P.ypitch : 1;
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int xx = j + r * L::TPL - padxl;
            v[r] = (valid && j + r * L::TPL < n && xx >= 0 && xx < nx) ? src[xx * xstep] : make_float2(0.f, 0.f);
        }
    };
    float2 v[L::SLOTS], vn[L::SLOTS];
    load_row(row0 + l, v);
    __syncthreads();
    int flip = 0;
#pragma unroll 1
    for (int g = 0; g < GV; ++g) {
        const long long rid = row0 + g * LPC + l;
        if (g + 1 < GV)
            load_row(rid + LPC, vn);
        if (pf) {
            float2 gA = make_float2(0.f, 0.f), gB = make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int xx = j + r * L::TPL - padxl;
                if (xx >= 0 && xx < ZPOW_N && xx < nx) {
                    const float zz = P.tab.zpow[xx];
                    gA = make_float2(fmaf(zz, v[r].x, gA.x), fmaf(zz, v[r].y, gA.y));
                }
                if (xx >= 0 && xx < nx && nx - 1 - xx < ZPOW_N) {
                    const float zz = P.tab.zpow[nx - 1 - xx];
                    gB = make_float2(fmaf(zz, v[r].x, gB.x), fmaf(zz, v[r].y, gB.y));
                }
            }
            float4 sum = make_float4(gA.x, gA.y, gB.x, gB.y);
#pragma unroll
            for (int d = 1; d < (L::TPL < 32 ? L::TPL : 32); d <<= 1) {
                sum.x += __shfl_xor_sync(0xffffffffu, sum.x, d);
                sum.y += __shfl_xor_sync(0xffffffffu, sum.y, d);
                sum.z += __shfl_xor_sync(0xffffffffu, sum.z, d);
                sum.w += __shfl_xor_sync(0xffffffffu, sum.w, d);
            }
            if constexpr (WPL > 1) {
                if ((j & 31) == 0)
                    red[l * WPL + j / 32] = sum;
                if (bar > 0)
                    line_sync(bar, L::TPL);
                else
                    __syncthreads();
                sum = red[l * WPL];
#pragma unroll
                for (int w = 1; w < WPL; ++w) {
                    const float4 t = red[l * WPL + w];
                    sum = make_float4(sum.x + t.x, sum.y + t.y, sum.z + t.z, sum.w + t.w);
                }
            }
            const float2 A = make_float2(sum.x, sum.y), B = make_float2(sum.z, sum.w);
            // d0 = u[e0] - u[e1] and d1 = u[e3] - u[e2] enter as
            // A_coef = ca d0 + cb d1, B_coef = ca d1 + cb d0
            const float2 d0g = make_float2(P.bx_ca * A.x + P.bx_cb * B.x, P.bx_ca * A.y + P.bx_cb * B.y);
            const float2 d1g = make_float2(P.bx_cb * A.x + P.bx_ca * B.x, P.bx_cb * A.y + P.bx_ca * B.y);
            const int e0 = (padxl - 1 + n) % n, e1 = (padxl + 1) % n;
            const int e2 = (padxl + nx - 2 + n) % n, e3 = (padxl + nx) % n;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int x = j + r * L::TPL;
                if (x == e0) v[r] = v[r] + d0g;
                if (x == e1) v[r] = v[r] - d0g;
                if (x == e3) v[r] = v[r] + d1g;
                if (x == e2) v[r] = v[r] - d1g;
            }
        }
        // (the transform's barriers also end the reads of the partial sums)
        line.template run<-1>(v, j, buf0 + l * xs, buf1 + l * xs, 1, tw, flip, bar);
        if (rid < rows) {
            float2 *dst = Tg + (size_t)rid * n;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int x = j + r * L::TPL;
                if (x < n && column_active(P, x))
                    dst[x] = v[r];
            }
        }
        if (g + 1 < GV) {
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r)
                v[r] = vn[r];
        }
    }
}

// Columns: forward FFT along y of the zero-padded cotangent column of every
// plane, accumulated against the conjugate propagator into Qg[slot][ky][kx].
template <class L, int KX, bool PAIR>
__global__ void __launch_bounds__(KX * L::TPL, KX * L::TPL <= 256 ? 3 : 1) k_adj_columns(StageParams P, L line, const float2 *Tg, float2 *Qg,
                                                             int q0, int qn, int ppc)
{
    if (!group_active<KX>(P, blockIdx.x * KX))
        return;
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNy
    const int xs = xslots<true>(n);
    float2 *buf0 = smem, *buf1 = smem + KX * xs, *tw = smem + 2 * KX * xs;
    float2 *stp = tw + tw_slots(n);  // [n][KX]
    float2 *red = stp + n * KX;      // [KX][2] y-prefilter boundary sums
    // [SLOTS][threads], each thread its own: sum over the boundary planes of
    // one end of pole^m Z_p
    float2 *bsum = red + 2 * KX + threadIdx.x;
    copy_twiddles<L>(tw, P.tab.twy, n);
    const int c = threadIdx.x % KX, j = threadIdx.x / KX;
    const int kx = blockIdx.x * KX + c;
    const bool colok = kx < P.lNx;
    // k_adj_rows writes the cotangent rows Tg only in the active columns;
    // a zero-band column of an active group is read as zero, never from
    // the unwritten workspace
    const bool colact = colok && column_active(P, kx);
    const int lNx = P.lNx, nz = P.nz, ny = P.ny, padyl = P.padyl;
    // tilted path: the forward's y-prefilter boundary terms (from the four
    // samples around the crop's ends) are transposed before the FFT
    const bool yfix = P.order >= 2 && P.tilted;
    const int qb = q0 + blockIdx.y * ppc;
    const int qe = min(q0 + qn, qb + ppc);
    const bool pf = P.order >= 2;
    __syncthreads();
    float2 E[L::SLOTS], Q[L::SLOTS];
    float2 R[PAIR ? L::SLOTS : 1];  // the opposite view's sum, without its constant factor
    const float copp = 2.f * P.zshift - 1.f;
    int flip = 0;
    int cur_a = -1;
    auto flush = [&](int a) {
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            if (colok && ky < n) {
                float2 *d = Qg + ((size_t)(PAIR ? 2 * a : a) * n + ky) * lNx + kx;
                atomicAdd(&d->x, Q[r].x);
                atomicAdd(&d->y, Q[r].y);
                if (PAIR) {
                    d += (size_t)n * lNx;
                    const float2 o = cmul_conj(R[r], expi_phase(P.tab.wsplit[(size_t)ky * lNx + kx], copp));
                    atomicAdd(&d->x, o.x);
                    atomicAdd(&d->y, o.y);
                }
            }
        }
    };
    // Boundary planes.  Where the two ends do not overlap, the terms
    // zl conj(alpha) Z_p + zh conj(beta) Z_p are collected as the sum over the
    // planes of one end (kind 1: zl, 2: zh) and multiplied by the table when
    // the end's planes are over: a fused multiply-add per element and plane
    // instead of table reads and, with opposite views, a sine and cosine
    // (48 of 128 planes: 90 views of 128^2 1.95 -> 1.47 ms).
    const bool split = pf && nz >= 2 * ZPOW_N;
    int kind = 0;  // of the planes in bsum, 0: none
    auto fold = [&]() {
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            if (colok && ky < n) {
                const size_t k = (size_t)ky * lNx + kx;
                const float2 t = bsum[r * KX * L::TPL];
                const float2 al = P.tab.alpha[k], be = P.tab.beta[k];
                Q[r] = Q[r] + cmul_conj(t, kind == 1 ? al : be);
                if (PAIR)  // the opposite view's, alpha and beta exchanged
                    R[r] = cfma(cmul_conj(t, kind == 1 ? be : al), expi_phase(P.tab.wsplit[k], copp), R[r]);
            }
        }
        kind = 0;
    };
    int a = qb / nz, p = qb % nz;
    // (one more turn than planes: sums are folded and flushed in one place)
    for (int q = qb;; ++q, ++p) {
        if (p == nz) {
            p = 0;
            ++a;
        }
        float zl = (pf && p < ZPOW_N) ? P.tab.zpow[p] : 0.f;
        float zh = (pf && nz - 1 - p < ZPOW_N) ? P.tab.zpow[nz - 1 - p] : 0.f;
        const int now = !split ? 0 : (zl != 0.f ? 1 : (zh != 0.f ? 2 : 0));
        if (kind && (now != kind || a != cur_a || q == qe))
            fold();
        if (cur_a >= 0 && (a != cur_a || q == qe))
            flush(cur_a);
        if (q >= qe)
            break;
        if (a != cur_a) {
            const float zp = (float)p - 0.5f * (float)nz + P.zshift;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int ky = j + r * L::TPL;
                Q[r] = make_float2(0.f, 0.f);
                if (PAIR)
                    R[r] = make_float2(0.f, 0.f);
                if (colok && ky < n) {
                    const size_t k = (size_t)ky * lNx + kx;
                    E[r] = expi_phase(P.tab.wsplit[k], zp);
                    stp[ky * KX + c] = P.tab.step[k];
                } else {
                    E[r] = make_float2(0.f, 0.f);
                }
            }
            cur_a = a;
        }
        float2 v[L::SLOTS];
        const float2 *src = Tg + (size_t)(q - q0) * ny * lNx + kx;
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int yy = j + r * L::TPL - padyl;
            v[r] = (colact && yy >= 0 && yy < ny) ? src[(size_t)yy * lNx] : make_float2(0.f, 0.f);
        }
        if (yfix) {
            // out[yy] = u[padyl + yy] + A z^yy + B z^(ny-1-yy), with A, B from
            // d0 = u[e0] - u[e1], d1 = u[e3] - u[e2]: collect the cotangent's
            // weighted sums gA, gB over the column, then scatter
            // (ca gA + cb gB) and (cb gA + ca gB) onto the four samples
            float2 gA = make_float2(0.f, 0.f), gB = make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int yy = j + r * L::TPL - padyl;
                if (yy >= 0 && yy < ny) {
                    if (yy < ZPOW_N) {
                        const float zz = P.tab.zpow[yy];
                        gA = make_float2(fmaf(zz, v[r].x, gA.x), fmaf(zz, v[r].y, gA.y));
                    }
                    if (ny - 1 - yy < ZPOW_N) {
                        const float zz = P.tab.zpow[ny - 1 - yy];
                        gB = make_float2(fmaf(zz, v[r].x, gB.x), fmaf(zz, v[r].y, gB.y));
                    }
                }
            }
            __syncthreads();  // the previous plane's reads of red are done
            if (j == 0) {
                red[c * 2] = make_float2(0.f, 0.f);
                red[c * 2 + 1] = make_float2(0.f, 0.f);
            }
            __syncthreads();
            if (gA.x != 0.f || gA.y != 0.f) {
                atomicAdd(&red[c * 2].x, gA.x);
                atomicAdd(&red[c * 2].y, gA.y);
            }
            if (gB.x != 0.f || gB.y != 0.f) {
                atomicAdd(&red[c * 2 + 1].x, gB.x);
                atomicAdd(&red[c * 2 + 1].y, gB.y);
            }
            __syncthreads();
            const float2 A = red[c * 2], B = red[c * 2 + 1];
            const float2 d0g = make_float2(P.by_ca * A.x + P.by_cb * B.x, P.by_ca * A.y + P.by_cb * B.y);
            const float2 d1g = make_float2(P.by_cb * A.x + P.by_ca * B.x, P.by_cb * A.y + P.by_ca * B.y);
            const int e0 = (padyl - 1 + n) % n, e1 = (padyl + 1) % n;
            const int e2 = (padyl + ny - 2 + n) % n, e3 = (padyl + ny) % n;
#pragma unroll
            for (int r = 0; r < L::SLOTS; ++r) {
                const int yq = j + r * L::TPL;
                if (yq == e0) v[r] = v[r] + d0g;
                if (yq == e1) v[r] = v[r] - d0g;
                if (yq == e3) v[r] = v[r] + d1g;
                if (yq == e2) v[r] = v[r] - d1g;
            }
        }
        line.template run<-1, true>(v, j, buf0 + c, buf1 + c, KX, tw, flip);
        if (split) {
            if (now) {
                const float z = zl + zh;  // (one of them is zero)
#pragma unroll
                for (int r = 0; r < L::SLOTS; ++r) {
                    float2 *b = bsum + r * KX * L::TPL;
                    *b = kind ? sfma2(z, v[r], *b) : cscale(v[r], z);
                }
                kind = now;
            }
            zl = zh = 0.f;
        }
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            // conj(P_p) Z = conj(E) Z + zl conj(alpha) Z + zh conj(beta) Z
            const float2 e = E[r];
            float2 cz = make_float2(fmaf(e.x, v[r].x, e.y * v[r].y), fmaf(e.x, v[r].y, -e.y * v[r].x));
            if ((zl != 0.f || zh != 0.f) && colok && ky < n) {
                const size_t k = (size_t)ky * lNx + kx;
                float2 b = make_float2(0.f, 0.f);
                if (zl != 0.f) {
                    const float2 al = P.tab.alpha[k];
                    b = make_float2(zl * al.x, zl * al.y);
                }
                if (zh != 0.f) {
                    const float2 be = P.tab.beta[k];
                    b = make_float2(fmaf(zh, be.x, b.x), fmaf(zh, be.y, b.y));
                }
                cz.x = fmaf(b.x, v[r].x, fmaf(b.y, v[r].y, cz.x));
                cz.y = fmaf(b.x, v[r].y, fmaf(-b.y, v[r].x, cz.y));
                if (PAIR) {
                    // the opposite view's terms, alpha and beta exchanged
                    const float2 al = P.tab.alpha[k], be = P.tab.beta[k];
                    b = make_float2(fmaf(zh, al.x, zl * be.x), fmaf(zh, al.y, zl * be.y));
                    b = cmul_conj(b, expi_phase(P.tab.wsplit[k], copp));
                    R[r].x = fmaf(b.x, v[r].x, fmaf(b.y, v[r].y, R[r].x));
                    R[r].y = fmaf(b.x, v[r].y, fmaf(-b.y, v[r].x, R[r].y));
                }
            }
            Q[r] = Q[r] + cz;
            if (PAIR)
                R[r] = cfma(e, v[r], R[r]);
            if (ky < n)
                E[r] = cmul(E[r], stp[ky * KX + c]);
        }
    }
}

// Spectrum: gain gradient dg += Re(conj(G X) Q) (X recomputed from the row
// spectra), then W = IFFT_y(conj(G g) Q) for every padded row.
template <class L, int KX>
__global__ void __launch_bounds__(KX * L::TPL) k_adj_spectrum(StageParams P, L line, const float2 *rowspec,
                                                              const float2 *Qg, float *dgain, float2 *dagain,
                                                              float2 *W)
{
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNy
    const int c = threadIdx.x % KX, j = threadIdx.x / KX;
    const int kx = blockIdx.x * KX + c;
    const bool colok = kx < P.lNx;
    const int lNx = P.lNx;
    const int sl = blockIdx.y;  // spectrum slot
    int a = sl;
    bool mirrored = false;
    if (P.units) {
        const int2 u = P.units[sl >> 1];
        mirrored = sl & 1;
        a = mirrored ? u.y : u.x;
        if (a < 0)
            return;  // no opposite view (uniform over the CTA)
    }
    const int kg = (mirrored && kx) ? lNx - kx : kx;  // the gains' column
    if (!group_active<KX>(P, blockIdx.x * KX)) {
        // all-zero columns: nothing reads W there, and the angle gains'
        // gradient is zero (the other gradients are cleared by the caller)
        if (dagain && colok) {
            for (int ky = j; ky < n; ky += L::TPL)
                dagain[((size_t)a * n + ky) * lNx + kg] = make_float2(0.f, 0.f);
        }
        return;
    }
    const int xs = xslots<true>(n);
    float2 *buf0 = smem, *buf1 = smem + KX * xs, *tw = smem + 2 * KX * xs;
    copy_twiddles<L>(tw, P.tab.twy, n);
    __syncthreads();
    int flip = 0;
    float2 X[L::SLOTS];
    const bool need_x = dgain || dagain;
    if (need_x) {
#pragma unroll
        for (int r = 0; r < L::SLOTS; ++r) {
            const int ky = j + r * L::TPL;
            X[r] = (colok && ky < n) ? rowspec[((size_t)sl * n + ky) * lNx + kx] : make_float2(0.f, 0.f);
        }
        line.template run<-1, true>(X, j, buf0 + c, buf1 + c, KX, tw, flip);
    }
    float2 v[L::SLOTS];
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int ky = j + r * L::TPL;
        v[r] = make_float2(0.f, 0.f);
        if (colok && ky < n) {
            const size_t k = (size_t)ky * lNx + kx;
            const float2 q = Qg[((size_t)sl * n + ky) * lNx + kx];
            const float2 G = P.tab.G[k];
            const size_t gk0 = (size_t)ky * lNx + kg;
            const float gk = P.gain ? P.gain[gk0] : 1.f;
            const size_t ak = (size_t)a * n * lNx + gk0;
            const float2 ga = P.again ? P.again[ak] : make_float2(1.f, 0.f);
            if (dgain) {
                // d/dg of G g ga X: Re(conj(G ga X) q)
                const float2 gx = cmul(cmul(G, ga), X[r]);
                atomicAdd(dgain + gk0, gx.x * q.x + gx.y * q.y);
            }
            if (dagain) {
                // d/d(ga) of G g ga X: conj(G g X) q
                const float2 gx = cscale(cmul(G, X[r]), gk);
                dagain[ak] = make_float2(gx.x * q.x + gx.y * q.y, gx.x * q.y - gx.y * q.x);
            }
            // conj(G g ga) q
            const float2 h = cscale(cmul(G, ga), gk);
            v[r] = make_float2(h.x * q.x + h.y * q.y, h.x * q.y - h.y * q.x);
        }
    }
    line.template run<1, true>(v, j, buf0 + c, buf1 + c, KX, tw, flip);
    if (!colok)
        return;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int ky = j + r * L::TPL;
        if (ky < n)
            W[((size_t)sl * n + ky) * lNx + kx] = v[r];
    }
}

// Transpose of the padding along one axis: padded position X contributes to
// source position pad_source with weight `c` (1 for data and edge padding, the
// ramp fraction for linear_ramp).
__device__ __forceinline__ int pad_source(int X, int n, int pad_l, int pad_r, int mode, float &c)
{
    const int i = X - pad_l;
    c = 1.f;
    if (i >= 0 && i < n)
        return i;
    if (mode == 2)
        c = i < 0 ? (float)X / (float)pad_l : (float)(pad_r - 1 - (i - n)) / (float)pad_r;
    return i < 0 ? 0 : n - 1;
}

// Rows: full backward FFT along x of W -> the cotangent of the padded plane,
// with the x padding transposed (and an opposite view's mirroring undone):
// Pg[slot][padded y][x].  (The padding's whole transpose in k_adj_pad left
// the 65 x 65 corner sums of a 128^2 view to single threads: 0.36 ms for 90
// views; 0.02 ms there and 0.03 ms more here with the x sums formed here.)
template <class L, int LPC>
__global__ void __launch_bounds__(LPC * L::TPL) k_adj_rows_full(StageParams P, L line, const float2 *W, float2 *Pg,
                                                                int nslots)
{
    extern __shared__ float2 smem[];
    const int n = line.size();  // lNx
    const int xs = xslots<false>(n);
    float2 *buf0 = smem, *buf1 = smem + LPC * xs, *tw = smem + 2 * LPC * xs;
    float2 *red = tw + tw_slots(n);  // [LPC][2] sums at the first and last column
    copy_twiddles<L>(tw, P.tab.twx, n);
    const int l = threadIdx.x / L::TPL, j = threadIdx.x % L::TPL;
    const long long lid = (long long)blockIdx.x * LPC + l;
    const bool valid = lid < (long long)nslots * P.lNy;
    const float2 *src = W + (size_t)(valid ? lid : 0) * n;
    float2 v[L::SLOTS];
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        const int x = j + r * L::TPL;
        v[r] = (valid && x < n && column_active(P, x)) ? src[x] : make_float2(0.f, 0.f);
    }
    if (threadIdx.x < 2 * LPC)
        red[threadIdx.x] = make_float2(0.f, 0.f);
    __syncthreads();
    int flip = 0;
    line.template run<1>(v, j, buf0 + l * xs, buf1 + l * xs, 1, tw, flip);
    const int nx = P.nx, padxr = P.lNx - P.nx - P.padxl;
    const bool mirrored = P.units && ((valid ? lid : 0) / P.lNy & 1);
    float2 first = make_float2(0.f, 0.f), last = first;
#pragma unroll
    for (int r = 0; r < L::SLOTS; ++r) {
        int X = j + r * L::TPL;
        if (X >= n)
            continue;
        if (mirrored) {
            X = 2 * P.padxl + nx - 1 - X;
            X += X < 0 ? n : 0;
            X -= X >= n ? n : 0;
        }
        float c;
        const int x = pad_source(X, nx, P.padxl, padxr, P.pad_mode, c);
        if (x == 0)
            first = sfma2(c, v[r], first);
        else if (x == nx - 1)
            last = sfma2(c, v[r], last);
        else if (valid)
            Pg[(size_t)lid * nx + x] = v[r];
    }
    if (first.x != 0.f || first.y != 0.f) {
        atomicAdd(&red[2 * l].x, first.x);
        atomicAdd(&red[2 * l].y, first.y);
    }
    if (last.x != 0.f || last.y != 0.f) {
        atomicAdd(&red[2 * l + 1].x, last.x);
        atomicAdd(&red[2 * l + 1].y, last.y);
    }
    __syncthreads();
    if (valid && j < 2)
        Pg[(size_t)lid * nx + (j ? nx - 1 : 0)] = red[2 * l + j];
}

// The y padding's transpose and the angle weight.
__global__ void k_adj_pad(StageParams P, const float2 *Pg, const double *weights, int nslots, float2 *dsino)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int sl = blockIdx.z;  // spectrum slot
    if (x >= P.nx || sl >= nslots)
        return;
    int a = sl;
    if (P.units) {
        const int2 u = P.units[sl >> 1];
        a = (sl & 1) ? u.y : u.x;
        if (a < 0)
            return;
    }
    const int padyr = P.lNy - P.ny - P.padyl;
    const float2 *col = Pg + (size_t)sl * P.lNy * P.nx + x;
    float2 acc = col[(size_t)(y + P.padyl) * P.nx];
    if (P.pad_mode != 0) {
        if (y == 0) {
#pragma unroll 8
            for (int Y = 0; Y < P.padyl; ++Y)
                acc = sfma2(P.pad_mode == 1 ? 1.f : (float)Y / (float)P.padyl, col[(size_t)Y * P.nx], acc);
        }
        if (y == P.ny - 1) {
#pragma unroll 8
            for (int q = 0; q < padyr; ++q)
                acc = sfma2(P.pad_mode == 1 ? 1.f : (float)(padyr - 1 - q) / (float)padyr,
                            col[(size_t)(P.padyl + P.ny + q) * P.nx], acc);
        }
    }
    const float w = weights ? (float)weights[a] : 1.f;
    dsino[((size_t)a * P.ny + y) * P.nx + x] = make_float2(w * acc.x, w * acc.y);
}

// ---------------------------------------------------------------------------
constexpr int kAdjPlanesPerBlock = 16;

template <class L>
static size_t smem_adj_rows(int n)
{
    // (the last terms: partial sums, 2 float2 per line in k_adj_rows_full, one
    // 16-byte aligned float4 per warp of a line in k_adj_rows)
    constexpr int WPL = L::TPL > 32 ? L::TPL / 32 : 1;
    return (size_t)(2 * Cfg<L>::LPC * xslots<false>(n) + tw_slots(n) + 1 + 2 * Cfg<L>::LPC * WPL) * sizeof(float2);
}
template <class L>
static size_t smem_adj_cols(int n)
{
    constexpr int KX = Cfg<L>::KX;
    return (size_t)(2 * KX * xslots<true>(n) + KX * n + tw_slots(n) + 2 * KX + L::SLOTS * KX * L::TPL) *
           sizeof(float2);
}
template <class L>
static size_t smem_adj_spectrum(int n)
{
    return (size_t)(2 * Cfg<L>::KX * xslots<true>(n) + tw_slots(n)) * sizeof(float2);
}

template <class L>
static cudaError_t set_adj_attrs(int n)
{
    if (std::is_same<L, GenericLine>::value)
        n = GenericLine::TPL * GenericLine::SLOTS;
    cudaError_t e;
    e = cudaFuncSetAttribute(k_adj_rows<L, Cfg<L>::LPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_adj_rows<L>(n));
    if (e != cudaSuccess)
        return e;
    e = cudaFuncSetAttribute(k_adj_rows_full<L, Cfg<L>::LPC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_adj_rows<L>(n));
    if (e != cudaSuccess)
        return e;
    e = cudaFuncSetAttribute(k_adj_columns<L, Cfg<L>::KX, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_adj_cols<L>(n));
    if (e != cudaSuccess)
        return e;
    e = cudaFuncSetAttribute(k_adj_columns<L, Cfg<L>::KX, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_adj_cols<L>(n));
    if (e != cudaSuccess)
        return e;
    return cudaFuncSetAttribute(k_adj_spectrum<L, Cfg<L>::KX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_adj_spectrum<L>(n));
}

cudaError_t configure_adjoint_kernels(const StageParams &P)
{
    cudaError_t e = with_line(P.lNx, [&](auto line) { return set_adj_attrs<decltype(line)>(line.n); });
    if (e != cudaSuccess)
        return e;
    return with_line(P.lNy, [&](auto line) { return set_adj_attrs<decltype(line)>(line.n); });
}

cudaError_t launch_adj_rows(const StageParams &P, const float2 *sgrad, float2 *Tg, int q0, int qn, cudaStream_t s)
{
    return with_line(P.lNx, [&](auto line) {
        using L = decltype(line);
        constexpr int LPC = Cfg<L>::LPC;
        constexpr int rpc = LPC * adj_row_groups<LPC>();
        const long long lines = (long long)qn * P.ny;
        k_adj_rows<L, LPC><<<(unsigned)((lines + rpc - 1) / rpc), LPC * L::TPL, smem_adj_rows<L>(line.n), s>>>(
            P, line, sgrad, Tg, q0, qn);
        return cudaGetLastError();
    });
}

cudaError_t launch_adj_columns(const StageParams &P, const float2 *Tg, float2 *Qg, int q0, int qn, cudaStream_t s)
{
    return with_line(P.lNy, [&](auto line) {
        using L = decltype(line);
        constexpr int KX = Cfg<L>::KX;
        dim3 grid((P.lNx + KX - 1) / KX, (qn + kAdjPlanesPerBlock - 1) / kAdjPlanesPerBlock);
        if (P.units)
            k_adj_columns<L, KX, true>
                <<<grid, KX * L::TPL, smem_adj_cols<L>(line.n), s>>>(P, line, Tg, Qg, q0, qn, kAdjPlanesPerBlock);
        else
            k_adj_columns<L, KX, false>
                <<<grid, KX * L::TPL, smem_adj_cols<L>(line.n), s>>>(P, line, Tg, Qg, q0, qn, kAdjPlanesPerBlock);
        return cudaGetLastError();
    });
}

cudaError_t launch_adj_spectrum(const StageParams &P, const float2 *rowspec, const float2 *Qg, float *dgain,
                                float2 *dagain, float2 *W, int nslots, cudaStream_t s)
{
    return with_line(P.lNy, [&](auto line) {
        using L = decltype(line);
        constexpr int KX = Cfg<L>::KX;
        dim3 grid((P.lNx + KX - 1) / KX, nslots);
        k_adj_spectrum<L, KX><<<grid, KX * L::TPL, smem_adj_spectrum<L>(line.n), s>>>(P, line, rowspec, Qg, dgain,
                                                                                 dagain, W);
        return cudaGetLastError();
    });
}

cudaError_t launch_adj_rows_full(const StageParams &P, const float2 *W, float2 *Pg, int nslots, cudaStream_t s)
{
    return with_line(P.lNx, [&](auto line) {
        using L = decltype(line);
        constexpr int LPC = Cfg<L>::LPC;
        const long long lines = (long long)nslots * P.lNy;
        k_adj_rows_full<L, LPC><<<(unsigned)((lines + LPC - 1) / LPC), LPC * L::TPL, smem_adj_rows<L>(line.n),
                                  s>>>(P, line, W, Pg, nslots);
        return cudaGetLastError();
    });
}

cudaError_t launch_adj_pad(const StageParams &P, const float2 *Pg, const double *weights, int nslots, float2 *dsino,
                           cudaStream_t s)
{
    dim3 grid((P.nx + 127) / 128, P.ny, nslots);
    k_adj_pad<<<grid, 128, 0, s>>>(P, Pg, weights, nslots, dsino);
    return cudaGetLastError();
}

}  // namespace odt
