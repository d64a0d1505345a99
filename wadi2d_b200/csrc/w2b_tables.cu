// The sub-grid table builder on the GPU: every static array of the step from the bed's pixels.
//
// Restates wadi2d/tables/core.py (cell tables :16-41, face tables :44-79, local hydraulic radius :82-179 and
// :324-371, centre beds :267-279) and wadi2d/tables/builder.py (the per-tile windows :199-238, inverts, closed faces
// and natural crests :290-308) in FP64 with the reference's summation order: every running sum is taken by one
// thread in the reference's sequence, so the only differences from the CPU build are the last-ulp rounding of CUDA's
// double cbrt and pow against glibc's, which the float32 tables almost never see, and of the local radius's sums, which
// are taken over its tent alone (local_term).
//
// Pixels are read from the whole bed with clipped indices, which is what the reference's per-tile windows of an
// ArrayBed hold (wadi2d/tables/builder.py:47-50): a window that reaches past the bed repeats its edge pixel.
#include <cmath>
#include <cstdio>

#include "w2b_common.cuh"

namespace w2b {

struct TableArgs {
    const double* z;
    int64_t zh, zw;
    int32_t roff, coff;
    const double* npix;  // per-pixel Manning n aligned with z (NaN: the cell's own), or null
    const double* nman;  // (ny, nx)
    const double *xcrest, *xlen, *xc, *ycrest, *ylen, *yc;  // (ny, nx), or null: no face edited
    const uint8_t *xwall, *ywall, *mask;                    // (ny, nx); walls may be null
    const int32_t* tiles;
    int32_t ntiles, ny, nx, k, rows, local, margin, nmax;
    double pixel, e_lo, e_hi, beta, tol;
    // outputs, tile layout (ntiles, 32, 32[, rows[, 2]]) float32
    float *hc, *dtab, *efx, *efy, *ftabx, *ftaby, *zcx, *zcy;
    float *flx, *frx, *glx, *grx, *cwx, *fly, *fry, *gly, *gry, *cwy;
    // outputs, dense (ny, nx) float64
    double *zmin, *rel, *zfx, *zfy;
    // workspace for face lines beyond shared memory: 9 * (nmax + 1) doubles per thread the caller counts
    double* ws;
    int64_t ws_threads;
};

__device__ __forceinline__ double zpix(const TableArgs& A, int64_t r, int64_t c) {
    r += A.roff;
    c += A.coff;
    r = r < 0 ? 0 : (r >= A.zh ? A.zh - 1 : r);
    c = c < 0 ? 0 : (c >= A.zw ? A.zw - 1 : c);
    return A.z[r * A.zw + c];
}

__device__ __forceinline__ double npix_at(const TableArgs& A, int64_t r, int64_t c) {
    r += A.roff;
    c += A.coff;
    r = r < 0 ? 0 : (r >= A.zh ? A.zh - 1 : r);
    c = c < 0 ? 0 : (c >= A.zw ? A.zw - 1 : c);
    return A.npix[r * A.zw + c];
}

__device__ __forceinline__ double lined(double pixel_n, double cell_n) {
    return isnan(pixel_n) ? 1.0 : cell_n / pixel_n;
}

// ------------------------------------------------------------------ cell tables (one thread per cell)

template <int K2MAX>
__global__ void __launch_bounds__(128) cell_tables_kernel(TableArgs A) {
    const int64_t ncell = (int64_t)(A.ntiles - 1) * TILE2;
    const int k = A.k, n = k * k, rows = A.rows, last = rows - 1;
    double p[K2MAX];
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += (int64_t)gridDim.x * blockDim.x) {
        const int t = (int)(c / TILE2) + 1;
        const int local = (int)(c % TILE2);
        const int64_t j = (int64_t)A.tiles[2 * t] * TILE + local / TILE;
        const int64_t i = (int64_t)A.tiles[2 * t + 1] * TILE + local % TILE;
        const int64_t r0 = j * k, c0 = i * k;
        // centre beds before the sort (wadi2d/tables/core.py:267-279)
        double cx, cy;
        {
            double col_a = INFINITY, col_b = INFINITY, row_a = INFINITY, row_b = INFINITY;
            const int ma = (k % 2) ? k / 2 : k / 2 - 1, mb = k / 2;
            for (int a = 0; a < k; ++a) {
                const double za = zpix(A, r0 + a, c0 + ma), zb = zpix(A, r0 + a, c0 + mb);
                col_a = za < col_a ? za : col_a;
                col_b = zb < col_b ? zb : col_b;
                const double ya = zpix(A, r0 + ma, c0 + a), yb = zpix(A, r0 + mb, c0 + a);
                row_a = ya < row_a ? ya : row_a;
                row_b = yb < row_b ? yb : row_b;
            }
            cx = (k % 2) ? col_b : 0.5 * (col_a + col_b);
            cy = (k % 2) ? row_b : 0.5 * (row_a + row_b);
        }
        for (int a = 0; a < k; ++a)
            for (int b = 0; b < k; ++b) p[a * k + b] = zpix(A, r0 + a, c0 + b);
        // ascending sort: insertion for small cells, heapsort beyond
        if (n <= 64) {
            for (int q = 1; q < n; ++q) {
                const double v = p[q];
                int s = q - 1;
                while (s >= 0 && p[s] > v) {
                    p[s + 1] = p[s];
                    --s;
                }
                p[s + 1] = v;
            }
        } else {
            for (int s = n / 2 - 1; s >= 0; --s) {
                int root = s;
                for (;;) {
                    int child = 2 * root + 1;
                    if (child >= n) break;
                    if (child + 1 < n && p[child] < p[child + 1]) ++child;
                    if (p[root] >= p[child]) break;
                    const double tmp = p[root];
                    p[root] = p[child];
                    p[child] = tmp;
                    root = child;
                }
            }
            for (int end = n - 1; end > 0; --end) {
                const double tmp = p[0];
                p[0] = p[end];
                p[end] = tmp;
                int root = 0;
                for (;;) {
                    int child = 2 * root + 1;
                    if (child >= end) break;
                    if (child + 1 < end && p[child] < p[child + 1]) ++child;
                    if (p[root] >= p[child]) break;
                    const double t2 = p[root];
                    p[root] = p[child];
                    p[child] = t2;
                    root = child;
                }
            }
        }
        // _cell_table, wadi2d/tables/core.py:16-41
        const double zmin = p[0];
        double sum = 0.0;
        for (int q = 0; q < n; ++q) {
            p[q] = p[q] - zmin;
            sum += p[q];
        }
        const double relmean = sum / (double)n;
        const double hc = p[n - 1] - relmean;
        float* tab = A.dtab + ((size_t)t * TILE2 + local) * rows;
        if (hc <= 1e-9) {
            for (int r = 0; r < rows; ++r) tab[r] = 0.0f;
            A.hc[(size_t)t * TILE2 + local] = 0.0f;
        } else {
            int m = 0;
            double cum = p[0];                 // sum of rel[0..m]
            double hb_m = (p[0] - cum) / (double)n;  // hbar_at[m]
            for (int r = 0; r < rows; ++r) {
                const double x = (double)r / (double)last;
                const double hb = hc * (x * x);
                while (m + 1 < n) {
                    const double cum1 = cum + p[m + 1];
                    const double hb1 = (p[m + 1] * (double)(m + 2) - cum1) / (double)n;
                    if (!(hb1 <= hb)) break;
                    m += 1;
                    cum = cum1;
                    hb_m = hb1;
                }
                const double v = p[m] + (hb - hb_m) * (double)n / (double)(m + 1);
                tab[r] = (float)(r == last ? p[n - 1] : v);
            }
            A.hc[(size_t)t * TILE2 + local] = (float)hc;
        }
        A.zmin[j * A.nx + i] = zmin;
        A.rel[j * A.nx + i] = relmean;
        // wadi2d/tables/builder.py:237, :248: centre beds over zmin, clamped at zero, NaN to zero
        double zx = cx - zmin, zy = cy - zmin;
        zx = isfinite(zx) ? (zx >= 0.0 ? zx : 0.0) : 0.0;
        zy = isfinite(zy) ? (zy >= 0.0 ? zy : 0.0) : 0.0;
        A.zcx[(size_t)t * TILE2 + local] = (float)zx;
        A.zcy[(size_t)t * TILE2 + local] = (float)zy;
    }
}

// ------------------------------------------------------------------ face tables

constexpr int KMAX = 32;
constexpr int ROWS_MAX = 64;
constexpr int FACE_THREADS = 256;
constexpr int64_t FACE_SMEM_BYTES = 200 * 1024;  // the shared memory a CTA of the face-table kernel may take
constexpr int64_t FACE_TERM_BYTES = 24 * 1024;   // of it for the pixels' conveyance terms (at least one face's)

// The higher of the two pixels meeting along a face's line (wadi2d/tables/core.py:249-264): position p along the
// line, from the first pixel of the face's cell; (r0, c0) is the cell's first pixel.
__device__ __forceinline__ double edge_pixel(const TableArgs& A, int axis, int64_t r0, int64_t c0, int64_t p) {
    const double far = axis == 0 ? zpix(A, r0 + p, c0 - 1) : zpix(A, r0 - 1, c0 + p);
    const double near = axis == 0 ? zpix(A, r0 + p, c0) : zpix(A, r0, c0 + p);
    return far >= near ? far : near;
}

// The lining weight of pixel q of a face, from the pixel that edge_pixel took.
__device__ __forceinline__ double edge_weight(const TableArgs& A, int axis, int64_t r0, int64_t c0, int q, double nm) {
    if (!A.npix) return 1.0;
    const int64_t nr = axis == 0 ? r0 + q : r0, nc = axis == 0 ? c0 : c0 + q;
    const int64_t fr = axis == 0 ? r0 + q : r0 - 1, fc = axis == 0 ? c0 - 1 : c0 + q;
    return lined(zpix(A, fr, fc) > zpix(A, nr, nc) ? npix_at(A, fr, fc) : npix_at(A, nr, nc), nm);
}

// A pixel of a face's line: its bed, and half the length of the bed from the pixel before it.
struct __align__(16) LinePixel {
    double z, half_seg;
};

// One pixel's conveyance term weight d cbrt(R)^2 at one level (_local_radius_conveyance, wadi2d/tables/core.py:
// 82-179): L is the face's conveyance line (n pixels). The local radius R weighs depth and wetted perimeter by a tent of
// half-width w = beta d / pixel (tent: beta / pixel) pixels around pixel i, inside its wet stretch. The reference takes the tent's sums as
// differences of running sums from the line's start; here they run over the tent alone, with the distance from pixel i as
// the argument, which needs no difference (so it rounds less) and sweeps 2 w pixels instead of i + w: w goes with the
// level, so most table rows' tents are far shorter than the line. A dry pixel before i starts the sums again; the first dry
// pixel after i ends them. Almost every pixel swept lies between wet ones: that case is the loops' first branch, and takes
// one 16-byte load.
__device__ __forceinline__ double local_term(const LinePixel* __restrict__ L, int n, int i, double level, double pixel,
                                             double tent, double weight) {
    const double di = level - L[i].z;
    if (!(di > 0.0)) return 0.0;
    double w = tent * di;
    if (w < 1e-9) w = 1e-9;
    int lo = (int)ceil((double)i - w), hi = (int)floor((double)i + w);
    lo = lo > 0 ? lo : 0;
    hi = hi < n - 1 ? hi : n - 1;
    const double half = 0.5 * pixel;
    // the perimeter a wet pixel has from a segment to a dry one `rise` higher
    auto partial = [&](double depth, double rise, double half_seg) {
        if (!(rise > 0.0)) return half;
        const double f = depth / rise;
        return (f <= 1.0 ? f : 1.0) * (2.0 * half_seg);
    };
    double s0 = 0.0, s1 = 0.0, p0 = 0.0, p1 = 0.0;  // sums of depth and perimeter, and of u times them
    double u = (double)(lo - i);                    // minus the distance of pixel t from pixel i
    double da = level - L[lo].z;  // depth of pixel t (dry: not over 0), and cr: the perimeter it has from its west
    double cr = 0.0;              // segment or the line's end
    if (da > 0.0) {
        if (lo == 0)
            cr = n == 1 ? half + half : half;
        else
            cr = level - L[lo - 1].z > 0.0 ? L[lo].half_seg : partial(da, L[lo - 1].z - L[lo].z, L[lo].half_seg);
    }
    auto add = [&](double per) {
        s0 += da;
        s1 = fma(u, da, s1);
        p0 += per;
        p1 = fma(u, per, p1);
    };
    for (int t = lo; t < i; ++t) {
        const LinePixel next = L[t + 1];
        const double db = level - next.z;
        if (da > 0.0 && db > 0.0) {
            add(cr + next.half_seg);
            cr = next.half_seg;
        } else if (da > 0.0) {  // the next pixel, dry, starts the sums again
            cr = 0.0;
        } else {
            s0 = s1 = p0 = p1 = 0.0;
            cr = db > 0.0 ? partial(db, L[t].z - next.z, next.half_seg) : 0.0;
        }
        da = db;
        u += 1.0;
    }
    if (i == n - 1 && i > 0) cr = half + cr;
    for (int t = i; t <= hi && da > 0.0; ++t) {
        double db = 0.0, per = cr;
        if (t + 1 < n) {
            const LinePixel next = L[t + 1];
            db = level - next.z;
            if (db > 0.0) {
                per += next.half_seg;
                cr = t + 2 == n ? half + next.half_seg : next.half_seg;
            } else {
                per += partial(da, next.z - L[t].z, next.half_seg);
            }
        }
        add(per);
        da = db;
        u -= 1.0;
    }
    const double a_sum = fma(s0, w, s1), p_sum = fma(p0, w, p1);  // both w times the tent's sum: one division in all
    const double radius = p_sum > 0.0 ? pixel * a_sum / p_sum : di;
    const double cb = cbrt(radius);
    return weight * di * (cb * cb);
}

// The same term where the line holds an infinite pixel: the reference's own running sums from the line's start. What is not
// finite in them (a perimeter against an infinite wall, a depth over an infinite hole) stays in every sum behind it, and the
// radius is then the depth; sums over the tent alone would forget it. No line of a real bed comes here: its cost, a sweep
// from the line's start a term, does not matter.
__device__ double running_term(const LinePixel* __restrict__ L, int n, int i, double level, double pixel,
                                            double beta, double weight) {
    auto depth = [&](int t) {
        const double d = level - L[t].z;
        return d > 0.0 ? d : 0.0;
    };
    const double di = depth(i);
    if (!(di > 0.0)) return 0.0;
    double w = beta * di / pixel;
    if (w < 1e-9) w = 1e-9;
    int first = i, last = i;  // the wet stretch around pixel i
    while (first > 0 && depth(first - 1) > 0.0) --first;
    while (last < n - 1 && depth(last + 1) > 0.0) ++last;
    int lo = (int)ceil((double)i - w), hi = (int)floor((double)i + w);
    lo = first > lo ? first : lo;
    hi = last < hi ? last : hi;
    // the perimeter that a wet pixel has from the segment to its neighbour of depth `other`, `rise` higher
    auto share = [&](double d, double other, double rise, double half_seg) {
        if (other > 0.0) return half_seg;
        if (!(rise > 0.0)) return 0.5 * pixel;
        const double f = d / rise;
        return (f <= 1.0 ? f : 1.0) * (2.0 * half_seg);
    };
    double s0 = 0.0, s1 = 0.0, p0 = 0.0, p1 = 0.0;        // sums over the pixels before t
    double ls0 = 0.0, ls1 = 0.0, lp0 = 0.0, lp1 = 0.0;    // before pixel lo
    double is0 = 0.0, is1 = 0.0, ip0 = 0.0, ip1 = 0.0;    // up to pixel i
    for (int t = 0; t <= hi; ++t) {
        if (t == lo) ls0 = s0, ls1 = s1, lp0 = p0, lp1 = p1;
        const double d = depth(t);
        double per = 0.0;
        if (d > 0.0) {
            if (t == 0) per += 0.5 * pixel;
            if (t == n - 1) per += 0.5 * pixel;
            if (t > 0) per += share(d, depth(t - 1), L[t - 1].z - L[t].z, L[t].half_seg);
            if (t < n - 1) per += share(d, depth(t + 1), L[t + 1].z - L[t].z, L[t + 1].half_seg);
        }
        s0 += d;
        s1 += (double)t * d;
        p0 += per;
        p1 += (double)t * per;
        if (t == i) is0 = s0, is1 = s1, ip0 = p0, ip1 = p1;
    }
    const double fi = (double)i;
    double a_sum = (1.0 - fi / w) * (is0 - ls0) + (is1 - ls1) / w;
    a_sum += (1.0 + fi / w) * (s0 - is0) - (s1 - is1) / w;
    double p_sum = (1.0 - fi / w) * (ip0 - lp0) + (ip1 - lp1) / w;
    p_sum += (1.0 + fi / w) * (p0 - ip0) - (p1 - ip1) / w;
    const double radius = p_sum > 0.0 ? pixel * a_sum / p_sum : di;
    const double cb = cbrt(radius);
    return weight * di * (cb * cb);
}

// Whether the bed holds an infinite pixel, in a place of its own only until close_faces_kernel writes it (the first cell's
// entry; zero before). A pass over the pixels that the faces' lines can reach: 25 us for 16 M of them.
__device__ __forceinline__ float* infinite_word(const TableArgs& A) { return A.flx + TILE2; }
__global__ void __launch_bounds__(256) infinite_kernel(TableArgs A) {
    auto row = [&](int64_t r) { return r < 0 ? 0 : (r >= A.zh ? A.zh - 1 : r); };
    auto col = [&](int64_t c) { return c < 0 ? 0 : (c >= A.zw ? A.zw - 1 : c); };
    const int64_t r0 = row((int64_t)A.roff - A.margin - 1), r1 = row((int64_t)A.roff + (int64_t)A.ny * A.k + A.margin);
    const int64_t c0 = col((int64_t)A.coff - A.margin - 1), c1 = col((int64_t)A.coff + (int64_t)A.nx * A.k + A.margin);
    bool found = false;
    for (int64_t r = r0 + blockIdx.x; r <= r1; r += gridDim.x) {
        const double* z = A.z + r * A.zw;
#pragma unroll 8
        for (int64_t c = c0 + threadIdx.x; c <= c1; c += blockDim.x) found |= isinf(z[c]);
    }
    if (found) *infinite_word(A) = 1.0f;
}

// The face tables (_face_table, wadi2d/tables/core.py:44-79, and the local radius's conveyance), a group of GF faces
// in a row along their own line at a time (GF divides 32: a column of a tile's west faces, a row of its north faces).
// The faces of a group share one line of GF k + 2 margin pixels, read once; then every (face, row, pixel) is a thread's
// own sweep along it (local_term), and every (face, row) a thread that adds its pixels' terms in order. Instruction issue and
// a thread's own chain bound it together (the sweeps, a division, a cbrt and four conversions a term: issue active 66 %, 56
// % at 10 x 10 pixels, FP64 28 and 37 %, 36 % of the warps a SM could hold, most of their waiting on the result before): 2.1
// M faces of 24- to 44-pixel lines (1024 x 1024 cells, 4 x 4 pixels) take 4.3 ms, 98 k faces of up to 298 (10 x 10 pixels
// of 1 m) 1.2 ms. A thread a face with its nine
// line arrays in shared memory, as this was first written, left 63 and 9 threads a SM and took 67 and 99 ms; sweeps from
// the line's start 8.5 and 2.9; the tent's sweeps with four divisions a term, the rows' levels and the indices divided out
// for each term, 5.2 and 1.26. A thread four or five pixels at once (one sweep for all, 200 registers, 8 warps a SM) was
// slower. Three CTAs of 256 threads a SM (80 registers): four (64, with spills) 5.3 and 1.39 against 5.2 and 1.26; six of
// 128 threads the same.
// LINE_SMEM: the group's line in shared memory, else (a line too long for it) in the caller's workspace, GF = 1.
// INFINITE: once more the groups whose line holds an infinite pixel, by running_term, if infinite_kernel has found any (both
// forms in one kernel, or a look for infinities in the other one, cost it 3 to 6 % of a build).
struct FaceShape {
    int gf, fc;      // faces a group; of them, whose terms are held at a time
    int line;        // pixels of a group's line
};
template <bool LINE_SMEM, bool INFINITE>
__global__ void __launch_bounds__(FACE_THREADS, 3) face_tables_kernel(TableArgs A, FaceShape F) {
    extern __shared__ __align__(16) double sws[];
    __shared__ double s_zf[TILE], s_top[TILE], s_scale[TILE], s_len[TILE], s_crest[TILE], s_nm[TILE];
    __shared__ double s_xx[ROWS_MAX];  // a row's level over the invert, of the face's full depth
    __shared__ int s_e[TILE];  // pixels the conveyance line reaches past the face's ends, -1: the strips' sum
    if (INFINITE && *infinite_word(A) == 0.0f) return;
    const int k = A.k, rows = A.rows, last = rows - 1, GF = F.gf, tid = threadIdx.x;
    double* terms = sws;
    // (the terms are an even count of doubles apart from the line's start: its pixels are 16 bytes)
    LinePixel* line = reinterpret_cast<LinePixel*>(LINE_SMEM ? sws + (((size_t)F.fc * rows * k + 1) & ~(size_t)1)
                                                             : (double*)(((uintptr_t)A.ws + 15) & ~(uintptr_t)15) +
                                                                   (size_t)blockIdx.x * 2 * F.line);
    for (int r = tid; r < rows; r += FACE_THREADS) {
        const double xr = (double)r / (double)last;
        s_xx[r] = xr * xr;
    }
    const double tent = A.beta / A.pixel;
    const int per = TILE / GF;
    const int64_t groups = (int64_t)(A.ntiles - 1) * 2 * TILE * per;
    for (int64_t g = blockIdx.x; g < groups; g += gridDim.x) {
        const int sub = (int)(g % per), c = (int)(g / per % TILE), axis = (int)(g / (per * TILE) & 1);
        const int t = (int)(g / (per * TILE * 2)) + 1;
        // the group's first face, and the step from one to the next
        const int jj0 = axis == 0 ? sub * GF : c, ii0 = axis == 0 ? c : sub * GF;
        const int64_t j0 = (int64_t)A.tiles[2 * t] * TILE + jj0, i0 = (int64_t)A.tiles[2 * t + 1] * TILE + ii0;
        const int dj = axis == 0, di = axis != 0;
        for (int s = tid; s < F.line; s += FACE_THREADS) line[s].z = edge_pixel(A, axis, j0 * k, i0 * k, s - A.margin);
        __syncthreads();
        if (INFINITE) {
            bool found = false;
            for (int s = tid; s < F.line; s += FACE_THREADS) found |= isinf(line[s].z);
            if (!__syncthreads_or(found)) continue;
        }
        if (A.local)
            for (int s = tid + 1; s < F.line; s += FACE_THREADS) {
                const double rise = line[s].z - line[s - 1].z;
                line[s].half_seg = 0.5 * sqrt(A.pixel * A.pixel + rise * rise);
            }
        const double* crests = axis == 0 ? A.xcrest : A.ycrest;
        for (int f = tid >> 5; f < GF; f += FACE_THREADS / 32) {
            const int lane = tid & 31;
            const int64_t cell = (j0 + f * dj) * A.nx + i0 + f * di;
            const double crest = crests ? crests[cell] : NAN;
            const bool natural = isnan(crest);
            double hi = -INFINITY;
            if (A.local && natural) {
                for (int s = lane; s < A.nmax; s += 32) {
                    const double v = line[f * k + s].z;
                    hi = v > hi ? v : hi;
                }
                for (int o = 16; o > 0; o >>= 1) {
                    const double v = __shfl_xor_sync(0xffffffffu, hi, o);
                    hi = v > hi ? v : hi;
                }
            }
            if (lane == 0) {
                const LinePixel* prof = line + f * k + A.margin;
                auto at = [&](int q) { return natural || prof[q].z >= crest ? prof[q].z : crest; };
                double zf = at(0);
                for (int q = 1; q < k; ++q) zf = at(q) < zf ? at(q) : zf;
                double relmax = at(0) - zf;
                for (int q = 1; q < k; ++q) {
                    const double v = at(q) - zf;
                    relmax = v > relmax ? v : relmax;
                }
                const double cut = relmax <= A.e_hi ? relmax : A.e_hi;
                double top = cut >= A.e_lo ? cut : A.e_lo;
                int e = -1;
                if (A.local && natural) {
                    // _raise_top and window_top, wadi2d/tables/core.py:354-371
                    const double relw = hi - zf;
                    const double cap = relw <= A.e_hi ? relw : A.e_hi;
                    const double wtop = top >= cap ? top : cap;
                    if (wtop > top) top = cut >= wtop ? cut : wtop;
                    e = (int)ceil(A.beta * top / A.pixel);
                    e = e > A.margin ? A.margin : e;
                }
                const double* lengths = axis == 0 ? A.xlen : A.ylen;
                const double nm = A.nman[cell];
                s_nm[f] = nm;
                s_scale[f] = A.pixel * (1.0 / nm);
                s_len[f] = lengths ? lengths[cell] : 1.0;
                s_crest[f] = crest;
                s_zf[f] = zf;
                s_top[f] = top;
                s_e[f] = e;
                const size_t o = (size_t)t * TILE2 + (jj0 + f * dj) * TILE + ii0 + f * di;
                (axis == 0 ? A.efx : A.efy)[o] = (float)top;
                (axis == 0 ? A.zfx : A.zfy)[cell] = zf;
            }
        }
        __syncthreads();
        for (int f0 = 0; f0 < GF; f0 += F.fc) {
            const int nf = GF - f0 < F.fc ? GF - f0 : F.fc;
            // term x is pixel q of face f at row r, q fastest; stepped without a division
            const int kf = k * nf, dr = FACE_THREADS / kf, rest = FACE_THREADS % kf, df = rest / k, dq = rest % k;
            int r = tid / kf, fl = tid % kf / k, q = tid % k;
            for (int x = tid; x < kf * rows && A.local; x += FACE_THREADS) {
                const int f = f0 + fl, e = s_e[f];
                if (e >= 0) {
                    const double level = s_zf[f] + s_top[f] * s_xx[r];
                    const int at = f * k + A.margin - e;
                    const int64_t j = j0 + f * dj, i = i0 + f * di;
                    const double weight = A.npix ? edge_weight(A, axis, j * k, i * k, q, s_nm[f]) : 1.0;
                    if (INFINITE)
                        terms[x] = running_term(line + at, k + 2 * e, e + q, level, A.pixel, A.beta, weight);
                    else
                        terms[x] = local_term(line + at, k + 2 * e, e + q, level, A.pixel, tent, weight);
                }
                q += dq;
                if (q >= k) q -= k, ++fl;
                fl += df;
                if (fl >= nf) fl -= nf, ++r;
                r += dr;
            }
            __syncthreads();
            for (int x = tid; x < nf * rows; x += FACE_THREADS) {
                const int r = x % rows, fl = x / rows, f = f0 + fl;
                const int64_t j = j0 + f * dj, i = i0 + f * di;
                const double crest = s_crest[f], length = s_len[f];
                const LinePixel* prof = line + f * k + A.margin;
                const double zf = s_zf[f], e = s_top[f] * s_xx[r];
                const bool strips = s_e[f] < 0;
                double area = 0.0, conv = 0.0;
                for (int q = 0; q < k; ++q) {
                    const double v = prof[q].z >= crest || isnan(crest) ? prof[q].z : crest;
                    const double dep = e - (v - zf);
                    if (dep > 0.0) {
                        area += dep;
                        if (strips) {
                            const double cb = cbrt(dep);
                            conv += edge_weight(A, axis, j * k, i * k, q, s_nm[f]) * dep * (cb * cb);
                        }
                    }
                    if (!strips) conv += terms[(r * nf + fl) * k + q];
                }
                const size_t o = (size_t)t * TILE2 + (jj0 + f * dj) * TILE + ii0 + f * di;
                float* out = (axis == 0 ? A.ftabx : A.ftaby) + (o * rows + r) * 2;
                out[0] = (float)(A.pixel * area * length);
                out[1] = (float)pow(s_scale[f] * conv * length, 0.6);
            }
            __syncthreads();  // the terms, and at the end the line and the faces' numbers, are read by every thread
        }
    }
}

// ------------------------------------------------------------------ inverts, closed faces, crests (per face)

// _faces, wadi2d/tables/builder.py:290-308; the neighbour is (j, i-1) for x faces and (j-1, i) for y faces, with
// np.roll's wrap at the grid edge.
__global__ void close_faces_kernel(TableArgs A) {
    const int64_t nface = (int64_t)(A.ntiles - 1) * TILE2 * 2;
    for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < nface; f += (int64_t)gridDim.x * blockDim.x) {
        const int axis = (int)(f & 1);
        const int64_t c = f >> 1;
        const int t = (int)(c / TILE2) + 1;
        const int local = (int)(c % TILE2);
        const int64_t j = (int64_t)A.tiles[2 * t] * TILE + local / TILE;
        const int64_t i = (int64_t)A.tiles[2 * t + 1] * TILE + local % TILE;
        const int64_t g = j * A.nx + i;
        const int64_t gn = axis == 0 ? j * A.nx + (i == 0 ? A.nx - 1 : i - 1) : (j == 0 ? A.ny - 1 : j - 1) * A.nx + i;
        const double zf = axis == 0 ? A.zfx[g] : A.zfy[g];
        const uint8_t* wall = axis == 0 ? A.xwall : A.ywall;
        const bool open = A.mask[g] && A.mask[gn] && !(wall && wall[g]);
        const double zmin = A.zmin[g], zmin_n = A.zmin[gn];
        const double zbar = zmin + A.rel[g], zbar_n = zmin_n + A.rel[gn];
        const double fl = open ? zf - zmin_n : 1.0e9;
        const double fr = open ? zf - zmin : 1.0e9;
        const double gl = open ? zf - zbar_n : 0.0;
        const double gr = open ? zf - zbar : 0.0;
        const bool natural = open && (gl > A.tol) && (gr > A.tol);
        const double* coeff = axis == 0 ? A.xc : A.yc;
        const double given = coeff ? coeff[g] : 0.0;
        double cw = given != 0.0 ? given : (natural ? 1.7046 : 0.0);
        cw = open ? cw : 0.0;
        const size_t o = (size_t)t * TILE2 + local;
        (axis == 0 ? A.flx : A.fly)[o] = (float)fl;
        (axis == 0 ? A.frx : A.fry)[o] = (float)fr;
        (axis == 0 ? A.glx : A.gly)[o] = (float)gl;
        (axis == 0 ? A.grx : A.gry)[o] = (float)gr;
        (axis == 0 ? A.cwx : A.cwy)[o] = (float)cw;
    }
}

}  // namespace w2b

using namespace w2b;

extern "C" {

int64_t w2b_table_workspace_doubles(int32_t nmax, int64_t threads) { return 9 * (int64_t)(nmax + 1) * threads; }

}  // extern "C"

// The build itself; out->ws may be null where no face line needs it.
static int32_t build(const W2BTableIn* in, const W2BTableOut* out, void* stream) {
    if (!in || !out || !in->z || !in->nman || !in->mask || !in->tiles || in->k < 1 || in->k > KMAX || in->rows < 4 ||
        in->rows > ROWS_MAX || in->ntiles < 1 || in->ny % TILE || in->nx % TILE || in->zh < 1 || in->zw < 1)
        return W2B_EINVAL;
    if (in->local && (in->margin < 0 || in->margin > W2B_TABLE_MARGIN_MAX)) return W2B_EINVAL;
    TableArgs A;
    A.z = in->z;
    A.zh = in->zh;
    A.zw = in->zw;
    A.roff = in->row_offset;
    A.coff = in->col_offset;
    A.npix = in->npix;
    A.nman = in->nman;
    A.xcrest = in->xcrest;
    A.xlen = in->xlen;
    A.xc = in->xc;
    A.ycrest = in->ycrest;
    A.ylen = in->ylen;
    A.yc = in->yc;
    A.xwall = in->xwall;
    A.ywall = in->ywall;
    A.mask = in->mask;
    A.tiles = in->tiles;
    A.ntiles = in->ntiles;
    A.ny = in->ny;
    A.nx = in->nx;
    A.k = in->k;
    A.rows = in->rows;
    A.local = in->local;
    A.margin = in->local ? in->margin : 0;
    A.nmax = in->k + 2 * A.margin;
    A.pixel = in->pixel;
    A.e_lo = in->face_depth_min;
    A.e_hi = in->face_depth_max;
    A.beta = in->beta;
    A.tol = in->crest_tolerance;
    A.hc = out->hc;
    A.dtab = out->dtab;
    A.efx = out->efx;
    A.efy = out->efy;
    A.ftabx = out->ftabx;
    A.ftaby = out->ftaby;
    A.zcx = out->zcx;
    A.zcy = out->zcy;
    A.flx = out->flx;
    A.frx = out->frx;
    A.glx = out->glx;
    A.grx = out->grx;
    A.cwx = out->cwx;
    A.fly = out->fly;
    A.fry = out->fry;
    A.gly = out->gly;
    A.gry = out->gry;
    A.cwy = out->cwy;
    A.zmin = out->zmin;
    A.rel = out->rel;
    A.zfx = out->zfx;
    A.zfy = out->zfy;
    A.ws = out->ws;
    A.ws_threads = out->ws_threads;
    cudaStream_t s = (cudaStream_t)stream;
    const int n = in->k * in->k;
    const int cblocks = 148 * 8;
    if (n <= 64)
        cell_tables_kernel<64><<<cblocks, 128, 0, s>>>(A);
    else if (n <= 256)
        cell_tables_kernel<256><<<cblocks, 128, 0, s>>>(A);
    else
        cell_tables_kernel<1024><<<cblocks, 128, 0, s>>>(A);
    // the face kernel's groups: as many faces in a row as their line and at least one face's terms fit shared memory;
    // a single face's line beyond that (about 11,000 pixels) lies in the caller's workspace, which holds its two arrays
    // for every CTA (each thread's share of the workspace is nine arrays of a line)
    FaceShape F;
    F.gf = TILE;
    const int64_t face_terms = (int64_t)in->rows * in->k * (int64_t)sizeof(double);
    int64_t term_faces = FACE_TERM_BYTES / face_terms;
    term_faces = term_faces < 1 ? 1 : (term_faces > TILE ? TILE : term_faces);
    auto line_bytes = [&](int gf) { return 2 * ((int64_t)gf * in->k + 2 * A.margin) * (int64_t)sizeof(double); };
    while (F.gf > 1 && line_bytes(F.gf) + term_faces * face_terms + 8 > FACE_SMEM_BYTES) F.gf /= 2;
    F.fc = (int)(term_faces < F.gf ? term_faces : F.gf);
    F.line = (int)(F.gf * in->k + 2 * A.margin);
    const bool line_smem = line_bytes(F.gf) + F.fc * face_terms + 8 <= FACE_SMEM_BYTES;
    const size_t bytes = (size_t)(F.fc * face_terms + 8 + (line_smem ? line_bytes(F.gf) : 0));
    int dev = 0, sms = 148, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto kernel = line_smem ? face_tables_kernel<true, false> : face_tables_kernel<false, false>;
    auto infinite = line_smem ? face_tables_kernel<true, true> : face_tables_kernel<false, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
        cudaFuncSetAttribute(infinite, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, FACE_THREADS, bytes) != cudaSuccess) {
        fprintf(stderr, "libwadi_b200: w2b_build_tables: face tables: %s\n", cudaGetErrorString(cudaGetLastError()));
        return W2B_ECUDA;
    }
    const int64_t groups = (int64_t)(in->ntiles - 1) * 2 * TILE * (TILE / F.gf);
    int64_t fblocks = (int64_t)sms * (occ > 0 ? occ : 1);
    if (!line_smem) {
        const int64_t held = (out->ws_threads * 9 * (int64_t)(A.nmax + 1) - 1) / (2 * (int64_t)F.line);
        fblocks = fblocks < held ? fblocks : held;
    }
    if (groups > 0) {
        const unsigned grid = (unsigned)(fblocks < groups ? fblocks : groups);
        kernel<<<grid, FACE_THREADS, bytes, s>>>(A, F);
        if (A.local) {
            if (cudaMemsetAsync(A.flx + TILE2, 0, sizeof(float), s) != cudaSuccess) return W2B_ECUDA;
            infinite_kernel<<<sms * 8, 256, 0, s>>>(A);
            infinite<<<grid, FACE_THREADS, bytes, s>>>(A, F);
        }
    }
    close_faces_kernel<<<148 * 8, 256, 0, s>>>(A);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "libwadi_b200: w2b_build_tables: %s\n", cudaGetErrorString(e));
        return W2B_ECUDA;
    }
    return W2B_OK;
}

extern "C" int32_t w2b_build_tables(const W2BTableIn* in, const W2BTableOut* out, void* stream) {
    if (!in || !out) return W2B_EINVAL;
    if (in->local && (!out->ws || out->ws_threads < 1 || out->ws_threads % 128)) return W2B_EINVAL;
    return build(in, out, stream);
}

// ------------------------------------------------------------------ the table build without allocation

// The longest face line (k + 2 margin pixels) w2b_build_tables_noalloc takes. Such a line and a face's terms fit a
// CTA's shared memory at every k and number of rows, so the build needs no scratch at all.
constexpr int64_t NOALLOC_LINE_MAX = 3639;
static_assert(2 * NOALLOC_LINE_MAX * 8 + (int64_t)KMAX * ROWS_MAX * 8 <= FACE_SMEM_BYTES, "a line in shared memory");

extern "C" int32_t w2b_build_tables_noalloc(const W2BTableIn* in, const W2BTableOut* out, void* stream) {
    if (!in || !out) return W2B_EINVAL;
    if (in->local && (in->margin < 0 || in->margin > W2B_TABLE_MARGIN_MAX)) return W2B_EINVAL;
    if (in->local && in->k + 2 * (int64_t)in->margin > NOALLOC_LINE_MAX) {
        fprintf(stderr, "libwadi_b200: w2b_build_tables_noalloc: face lines of %lld pixels: at most %lld\n",
                (long long)(in->k + 2 * (int64_t)in->margin), (long long)NOALLOC_LINE_MAX);
        return W2B_EINVAL;
    }
    W2BTableOut o = *out;
    o.ws = nullptr;
    o.ws_threads = 0;
    return build(in, &o, stream);
}
