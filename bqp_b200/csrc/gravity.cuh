// Spherical-harmonic gravity by the normalised column recursion.
//
// The reference evaluates the field with the unnormalised Cunningham /
// Montenbruck-Gill V/W recursion and then a separate summation over (n, m)
// terms that reads V/W at orders m-1, m, m+1 of row n+1
// (satpy_core/src/gravity.rs:291-377 and 2075-2223).  Here the same
// acceleration is computed with 4-pi normalised V/W (no overflow to degree
// 128+, and usable in FP32), and the summation is folded into the recursion:
// every term that reads cell (l, j) of V/W is gathered, on the host, into six
// per-cell weights (Ax, Bx, Ay, By, Az, Bz) so that
//
//     a_x += Ax V(l,j) + Bx W(l,j),   a_y += Ay V + By W,   a_z += Az V + Bz W
//
// The weights already carry GM/R^2, so the result is in km/s^2.
//
// FP64 form.  Inside a column V and W are the same real recursion in l times
// the column's (x' + i y')^j, x' = x R/r^2 and so on:
//
//     V(l,j) + i W(l,j) = (R/r) (x' + i y')^j s(l,j) q(l,j),
//     q(j,j) = 1,  q(j+1,j) = z',  q(l,j) = A(l,j) z' q(l-1,j) - (R/r)^2 q(l-2,j)
//
// where the constants s (which the host folds into the weights) make both the
// first cell and the recursion's second coefficient one.  So a column needs
// one recursion and six real sums, S_Ax = sum Ax s q and so on, and only at
// its end the products with the real and imaginary part of (x' + i y')^j:
// 9 FP64 operations a cell (3 + 6), against 12 when V and W are both carried
// and both multiplied by their weights in every cell.  The kernels are bound
// by the FP64 pipe and the table reads beside it: at 70x70, 1,000,003
// positions take 1,828 us (12.9e12 FP64 instructions/s in the cells; the pipe
// alone would take 1,390 us), 2,399 us with 12 operations a cell; 65,536 rows
// 130 us.
#pragma once
#include "physics.cuh"

namespace bqp {

constexpr int kCellDoubles = 8;  // a cell of the split-precision form's tables

BQP_HD int gravity_cells(int order) { return (order + 2) * (order + 3) / 2; }

// Index of the first cell of column j (columns hold rows j..order+1).
BQP_HD int gravity_col_offset(int order, int j) {
    const int rows0 = order + 2;  // cells in column 0
    return j * rows0 - j * (j - 1) / 2;
}

// FP64 table, columns ascending.  A column of L = order + 2 - j cells:
//   rows j and j+1 (row j alone for L = 1): {Ax Bx Ay By Az Bz} each
//   if L is odd and > 2, one cell {A 0 Ax Bx Ay By Az Bz}
//   pairs of cells {A A' Ax Bx Ay By Az Bz Ax' Bx' Ay' By' Az' Bz'}
// Every piece is a multiple of 16 bytes, so each is read by 16-byte loads
// (the same address in every lane): 7 for a pair, 56 bytes a cell.
// Offset of column j (j = order + 2: the table's size), in doubles: a column
// of L cells takes 7 L - 2 (no A in the first two rows) and one more where L
// is odd (the padded single cell; for L = 1 the row with 6).
BQP_HD int gravity_tab_offset(int order, int j) {
    const int odd = ((order & 1) ? j + 1 : j) >> 1;  // columns before j whose L is odd
    return 7 * gravity_col_offset(order, j) - 2 * j + odd;
}
constexpr size_t kGravityTabPad = 16;  // doubles readable past the table's end
inline size_t gravity_tab_doubles(int order) { return (size_t)gravity_tab_offset(order, order + 2); }

// (x + i y)^e for NT numbers, e >= 0 the same in every lane.
template <int NT>
BQP_HD void gravity_powers(const double* x, const double* y, int e, double* re, double* im) {
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        re[q] = 1.0;
        im[q] = 0.0;
    }
    int bit = 1;
    while (2 * bit <= e) bit *= 2;
    if (e > 0) {
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            re[q] = x[q];
            im[q] = y[q];
        }
    }
#pragma unroll 1
    for (bit >>= 1; bit > 0; bit >>= 1) {
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const double t = fma(re[q], re[q], -im[q] * im[q]);
            im[q] = 2.0 * re[q] * im[q];
            re[q] = t;
        }
        if (e & bit) {
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double t = fma(re[q], x[q], -im[q] * y[q]);
                im[q] = fma(re[q], y[q], im[q] * x[q]);
                re[q] = t;
            }
        }
    }
}

// Two interior cells {A A' Ax Bx Ay By Az Bz Ax' ...} of a column.
template <int NT>
BQP_HD void gravity_pair(const double2* cb, const double* zc, const double* c2, double* q0, double* q1,
                         double (*s)[6]) {
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        q0[q] = fma(cb[0].x * zc[q], q1[q], -c2[q] * q0[q]);
        s[q][0] = fma(cb[1].x, q0[q], s[q][0]);
        s[q][1] = fma(cb[1].y, q0[q], s[q][1]);
        s[q][2] = fma(cb[2].x, q0[q], s[q][2]);
        s[q][3] = fma(cb[2].y, q0[q], s[q][3]);
        s[q][4] = fma(cb[3].x, q0[q], s[q][4]);
        s[q][5] = fma(cb[3].y, q0[q], s[q][5]);
        q1[q] = fma(cb[0].y * zc[q], q0[q], -c2[q] * q1[q]);
        s[q][0] = fma(cb[4].x, q1[q], s[q][0]);
        s[q][1] = fma(cb[4].y, q1[q], s[q][1]);
        s[q][2] = fma(cb[5].x, q1[q], s[q][2]);
        s[q][3] = fma(cb[5].y, q1[q], s[q][3]);
        s[q][4] = fma(cb[6].x, q1[q], s[q][4]);
        s[q][5] = fma(cb[6].y, q1[q], s[q][5]);
    }
}

// The columns are dealt to `shares` shares in blocks of `shares` columns, back
// and forth: share w takes column k shares + w of an even block k and
// k shares + (shares - 1 - w) of an odd one.  A column is one cell shorter
// than the one before it, so the shares get the same number of cells to
// within half a block (328.5 +- 3.5 of 2,628 at 70x70 in 8 shares; contiguous
// runs of columns were up to 10 % apart), and shares next to one another own
// a contiguous run of columns in every block.
BQP_HD int gravity_share_column(int shares, int k, int w) {
    return k * shares + ((k & 1) ? shares - 1 - w : w);
}

// Partial field of share w for NT positions a thread.  `tab` holds the runs of
// columns of the shares wa .. wa + own - 1, block after block (own = shares:
// the whole table).
//
// Every table read feeds NT independent recursions: a 16-byte broadcast load
// moves its bytes into every lane's registers (64 bytes a cycle and
// scheduler), and while it does the FP64 pipe of that scheduler loses about
// 2.4 instructions.  Measured on registers alone the column runs at 17.7e12
// FP64 instructions/s; with its 3.5 loads a cell 14.4e12 at NT = 4, 12.9e12
// at 2 and 10.7e12 at 1.
template <int NT>
BQP_HD void gravity_part(const double* __restrict__ tab, int order, int shares, int wa, int own, int w,
                         const double* px, const double* py, const double* pz, double (*acc)[3]) {
    double c[NT], zc[NT], c2[NT], zr[NT], zi[NT], ar[NT], ai[NT], br[NT], bi[NT];
    const int ga = 2 * (shares - 1 - w) + 1, gb = 2 * w + 1;  // steps after an even and after an odd block
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        const double r2 = fma(px[q], px[q], fma(py[q], py[q], pz[q] * pz[q]));
        const double s = kReGravity / r2;  // R/r^2
        const double xc = px[q] * s, yc = py[q] * s;
        zc[q] = pz[q] * s;
        c2[q] = s * kReGravity;  // (R/r)^2
        c[q] = sqrt(c2[q]);
        acc[q][0] = acc[q][1] = acc[q][2] = 0.0;
        ar[q] = xc;  // the powers below start from these
        ai[q] = yc;
    }
    gravity_powers<NT>(ar, ai, w, zr, zi);
    {
        // the steps' powers: x^(2 w + 1) = (x^w)^2 x, and the same of shares - 1 - w
        double tr[NT], ti[NT];
        gravity_powers<NT>(ar, ai, shares - 1 - w, tr, ti);
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const double xr = ar[q], xi = ai[q];
            double r = fma(zr[q], zr[q], -zi[q] * zi[q]), i = 2.0 * zr[q] * zi[q];
            br[q] = fma(r, xr, -i * xi);
            bi[q] = fma(r, xi, i * xr);
            r = fma(tr[q], tr[q], -ti[q] * ti[q]);
            i = 2.0 * tr[q] * ti[q];
            ar[q] = fma(r, xr, -i * xi);
            ai[q] = fma(r, xi, i * xr);
        }
    }
    const int last = order + 1, ncol = order + 2;
    int step = ga, other = gb;
    int run = wa;  // first column of this block's run
    const double* at = tab;
    for (int k = 0, j = w; j < ncol; ++k) {
        const int run_off = gravity_tab_offset(order, run);
        const double2* cell = reinterpret_cast<const double2*>(at + (gravity_tab_offset(order, j) - run_off));
        double s[NT][6], q0[NT], q1[NT];
        {
            const double2 wx = cell[0], wy = cell[1], wz = cell[2];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                s[q][0] = wx.x;
                s[q][1] = wx.y;
                s[q][2] = wy.x;
                s[q][3] = wy.y;
                s[q][4] = wz.x;
                s[q][5] = wz.y;
                q0[q] = 1.0;
                q1[q] = zc[q];
            }
            cell += 3;
        }
        int n = last - j;  // rows below the first
        if (n > 0) {
            const double2 wx = cell[0], wy = cell[1], wz = cell[2];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                s[q][0] = fma(wx.x, q1[q], s[q][0]);
                s[q][1] = fma(wx.y, q1[q], s[q][1]);
                s[q][2] = fma(wy.x, q1[q], s[q][2]);
                s[q][3] = fma(wy.y, q1[q], s[q][3]);
                s[q][4] = fma(wz.x, q1[q], s[q][4]);
                s[q][5] = fma(wz.y, q1[q], s[q][5]);
            }
            cell += 3;
            --n;
        }
        if (n & 1) {
            const double2 a = cell[0], wx = cell[1], wy = cell[2], wz = cell[3];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double t = fma(a.x * zc[q], q1[q], -c2[q] * q0[q]);
                q0[q] = q1[q];
                q1[q] = t;
                s[q][0] = fma(wx.x, t, s[q][0]);
                s[q][1] = fma(wx.y, t, s[q][1]);
                s[q][2] = fma(wy.x, t, s[q][2]);
                s[q][3] = fma(wy.y, t, s[q][3]);
                s[q][4] = fma(wz.x, t, s[q][4]);
                s[q][5] = fma(wz.y, t, s[q][5]);
            }
            cell += 4;
        }
        // one pair in use, the next in flight; the load after the last pair
        // reads up to 112 bytes past the column (kGravityTabPad), unused
        double2 ca[7], cb[7];
#pragma unroll
        for (int i = 0; i < 7; ++i) ca[i] = cell[i];
        int p = n >> 1;
#pragma unroll 1
        for (; p >= 2; p -= 2) {
#pragma unroll
            for (int i = 0; i < 7; ++i) cb[i] = cell[7 + i];
            gravity_pair<NT>(ca, zc, c2, q0, q1, s);
            cell += 14;
#pragma unroll
            for (int i = 0; i < 7; ++i) ca[i] = cell[i];
            gravity_pair<NT>(cb, zc, c2, q0, q1, s);
        }
        if (p) gravity_pair<NT>(ca, zc, c2, q0, q1, s);
#pragma unroll
        for (int q = 0; q < NT; ++q) {
#pragma unroll
            for (int i = 0; i < 3; ++i) acc[q][i] = fma(s[q][2 * i], zr[q], fma(s[q][2 * i + 1], zi[q], acc[q][i]));
            const double t = fma(zr[q], ar[q], -zi[q] * ai[q]);
            zi[q] = fma(zr[q], ai[q], zi[q] * ar[q]);
            zr[q] = t;
            const double sr = ar[q], si = ai[q];  // the other step next
            ar[q] = br[q];
            ai[q] = bi[q];
            br[q] = sr;
            bi[q] = si;
        }
        j += step;
        const int t = step;
        step = other;
        other = t;
        const int run_end = run + own < ncol ? run + own : ncol;
        at += gravity_tab_offset(order, run_end) - run_off;
        run = gravity_share_column(shares, k + 1, (k & 1) ? wa : wa + own - 1);
    }
#pragma unroll
    for (int q = 0; q < NT; ++q) {
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[q][i] *= c[q];
    }
}

// Acceleration (km/s^2, Earth-fixed) of the field encoded in `tab` at an
// Earth-fixed position (km).  `tab` may point to shared or global memory.
BQP_HD void gravity_field(const double* __restrict__ tab, int order, double px, double py,
                          double pz, double* acc) {
    double a[1][3];
    gravity_part<1>(tab, order, 1, 0, 1, 0, &px, &py, &pz, a);
    acc[0] = a[0][0];
    acc[1] = a[0][1];
    acc[2] = a[0][2];
}

// First column of part p when the columns are cut into `parts` runs of about
// equal cell count (p = parts gives order + 2, one past the last column).
BQP_HD int gravity_part_column(int order, int p, int parts) {
    const int ncol = order + 2;
    if (p <= 0) return 0;
    if (p >= parts) return ncol;
    const long long target = (long long)gravity_cells(order) * p / parts;
    int j = 0;
    long long cells = 0;
    while (j < ncol && cells + (ncol - j) <= target) cells += ncol - j++;
    return j;
}

// ---------------------------------------------------------------------------
// The FP64 field with V and W both carried down every column and both
// multiplied by their weights in every cell (12 operations a cell), over the
// columns [j0, j1) of a table of cells {a, b, Ax, Bx, Ay, By, Az, Bz}.  Only
// sigma-point rows take it (PropArgs::ordered), for the order in which it
// adds.
template <int NT>
BQP_HD void gravity_columns(const double* __restrict__ tab, int order, int j0, int j1, const double* px,
                            const double* py, const double* pz, double (*acc)[3]) {
    double xc[NT], yc[NT], zc[NT], c2re[NT], vd[NT], wd[NT], ax[NT], ay[NT], az[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        const double r2 = fma(px[q], px[q], fma(py[q], py[q], pz[q] * pz[q]));
        const double c2 = kReGravity / r2;
        xc[q] = px[q] * c2;
        yc[q] = py[q] * c2;
        zc[q] = pz[q] * c2;
        c2re[q] = c2 * kReGravity;
        vd[q] = sqrt(c2re[q]);
        wd[q] = 0.0;
        ax[q] = ay[q] = az[q] = 0.0;
    }
    const int last = order + 1;
    const double2* tab2 = reinterpret_cast<const double2*>(tab);
    for (int j = 1; j < j0; ++j) {
        const double a = tab2[(size_t)gravity_col_offset(order, j) * 4].x;
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const double nv = a * fma(xc[q], vd[q], -yc[q] * wd[q]);
            const double nw = a * fma(xc[q], wd[q], yc[q] * vd[q]);
            vd[q] = nv;
            wd[q] = nw;
        }
    }
    const double2* cell = tab2 + (size_t)gravity_col_offset(order, j0) * 4;
    for (int j = j0; j < j1; ++j) {
        {
            const double2 ab = cell[0], wx = cell[1], wy = cell[2], wz = cell[3];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                if (j > 0) {
                    const double nv = ab.x * fma(xc[q], vd[q], -yc[q] * wd[q]);
                    const double nw = ab.x * fma(xc[q], wd[q], yc[q] * vd[q]);
                    vd[q] = nv;
                    wd[q] = nw;
                }
                ax[q] = fma(wx.x, vd[q], fma(wx.y, wd[q], ax[q]));
                ay[q] = fma(wy.x, vd[q], fma(wy.y, wd[q], ay[q]));
                az[q] = fma(wz.x, vd[q], fma(wz.y, wd[q], az[q]));
            }
            cell += 4;
        }
        if (j == last) break;
        double v0[NT], w0[NT], v1[NT], w1[NT];
        {
            const double2 ab = cell[0], wx = cell[1], wy = cell[2], wz = cell[3];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double a = ab.x * zc[q];
                v0[q] = vd[q];
                w0[q] = wd[q];
                v1[q] = a * vd[q];
                w1[q] = a * wd[q];
                ax[q] = fma(wx.x, v1[q], fma(wx.y, w1[q], ax[q]));
                ay[q] = fma(wy.x, v1[q], fma(wy.y, w1[q], ay[q]));
                az[q] = fma(wz.x, v1[q], fma(wz.y, w1[q], az[q]));
            }
            cell += 4;
        }
        // interior rows j+2..last, two per iteration (the row registers
        // rotate without moves); the next pair is in flight meanwhile
        const int pairs = (last - j - 1) >> 1;
        double2 nx[8];
        if (pairs > 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) nx[i] = cell[i];
        }
#pragma unroll 2
        for (int p = 0; p < pairs; ++p) {
            double2 cb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) cb[i] = nx[i];
            if (p + 1 < pairs) {
#pragma unroll
                for (int i = 0; i < 8; ++i) nx[i] = cell[8 + i];
            }
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double ta = cb[0].x * zc[q], tb = cb[0].y * c2re[q];
                v0[q] = fma(ta, v1[q], -tb * v0[q]);
                w0[q] = fma(ta, w1[q], -tb * w0[q]);
                ax[q] = fma(cb[1].x, v0[q], fma(cb[1].y, w0[q], ax[q]));
                ay[q] = fma(cb[2].x, v0[q], fma(cb[2].y, w0[q], ay[q]));
                az[q] = fma(cb[3].x, v0[q], fma(cb[3].y, w0[q], az[q]));
                const double ta2 = cb[4].x * zc[q], tb2 = cb[4].y * c2re[q];
                v1[q] = fma(ta2, v0[q], -tb2 * v1[q]);
                w1[q] = fma(ta2, w0[q], -tb2 * w1[q]);
                ax[q] = fma(cb[5].x, v1[q], fma(cb[5].y, w1[q], ax[q]));
                ay[q] = fma(cb[6].x, v1[q], fma(cb[6].y, w1[q], ay[q]));
                az[q] = fma(cb[7].x, v1[q], fma(cb[7].y, w1[q], az[q]));
            }
            cell += 8;
        }
        if ((last - j - 1) & 1) {
            const double2 ab = cell[0], wx = cell[1], wy = cell[2], wz = cell[3];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double ta = ab.x * zc[q], tb = ab.y * c2re[q];
                const double v2 = fma(ta, v1[q], -tb * v0[q]);
                const double w2 = fma(ta, w1[q], -tb * w0[q]);
                ax[q] = fma(wx.x, v2, fma(wx.y, w2, ax[q]));
                ay[q] = fma(wy.x, v2, fma(wy.y, w2, ay[q]));
                az[q] = fma(wz.x, v2, fma(wz.y, w2, az[q]));
            }
            cell += 4;
        }
    }
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        acc[q][0] = ax[q];
        acc[q][1] = ay[q];
        acc[q][2] = az[q];
    }
}

// ---------------------------------------------------------------------------
// Split-precision form.  Cell (l, j) carries only degree n = l - 1, so rows
// l <= ls hold degrees n <= ls - 1 (the central-field corrections J2...,
// kept in FP64) and every other cell the higher degrees, evaluated in FP32:
// Cells are {a, b, Ax, Bx, Ay, By, Az, Bz}, V and W both carried:
//   diagonal cell (j, j):     a = sqrt((2j+1)/(2j)) (j >= 2), sqrt(3) (j = 1)
//   sub-diagonal (j+1, j):    a = sqrt(2j+3)
//   interior (l >= j+2):      a = sqrt((2l-1)(2l+1)/((l-j)(l+j)))
//                             b = sqrt((2l+1)(l+j-1)(l-j-1)/((2l-3)(l+j)(l-j)))
//   lo: FP64 cells of columns 0..ls, rows j..ls (column-major)
//   hi: FP32 cells {a, b, Ax, Bx | Ay, By, Az, Bz} of columns 0..ls, rows
//       ls+1..order+1, then columns ls+1..order+1, rows j..order+1
// The V/W values of the last FP64 rows seed the FP32 rows below them; the
// two parts are accumulated separately and added in FP64.  Needs
// 1 <= ls <= order.
BQP_HD int split_lo_offset(int ls, int j) { return j * (ls + 1) - j * (j - 1) / 2; }
BQP_HD int split_lo_cells(int ls) { return (ls + 1) * (ls + 2) / 2; }
BQP_HD int split_hi_offset(int order, int ls, int j) {
    const int h = order + 1 - ls;  // FP32 rows under an FP64 column
    if (j <= ls + 1) return j * h;
    const int k = j - (ls + 1);
    return (ls + 1) * h + k * h - k * (k - 1) / 2;
}
BQP_HD int split_hi_cells(int order, int ls) { return split_hi_offset(order, ls, order + 2); }

template <int NT>
BQP_HD void gravity_columns_split(const double* __restrict__ lo, const float* __restrict__ hi, int order, int ls,
                                  int j0, int j1, const double* px, const double* py, const double* pz,
                                  double (*acc)[3]) {
    double xc[NT], yc[NT], zc[NT], c2re[NT], vd[NT], wd[NT], ax[NT], ay[NT], az[NT];
    float xf[NT], yf[NT], zf[NT], cf[NT], vdf[NT], wdf[NT], fx[NT], fy[NT], fz[NT];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        const double r2 = fma(px[q], px[q], fma(py[q], py[q], pz[q] * pz[q]));
        const double c2 = kReGravity / r2;
        xc[q] = px[q] * c2;
        yc[q] = py[q] * c2;
        zc[q] = pz[q] * c2;
        c2re[q] = c2 * kReGravity;
        vd[q] = sqrt(c2re[q]);
        wd[q] = 0.0;
        ax[q] = ay[q] = az[q] = 0.0;
        xf[q] = (float)xc[q];
        yf[q] = (float)yc[q];
        zf[q] = (float)zc[q];
        cf[q] = (float)c2re[q];
        vdf[q] = wdf[q] = 0.0f;
        fx[q] = fy[q] = fz[q] = 0.0f;
    }
    const int last = order + 1;
    const double2* lo2 = reinterpret_cast<const double2*>(lo);
    const float4* hi4 = reinterpret_cast<const float4*>(hi);
    // diagonal V(j,j), W(j,j) from column j-1's
    auto advance_diag = [&](int j) {
        if (j <= ls) {
            const double a = lo2[(size_t)split_lo_offset(ls, j) * 4].x;
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double nv = a * fma(xc[q], vd[q], -yc[q] * wd[q]);
                const double nw = a * fma(xc[q], wd[q], yc[q] * vd[q]);
                vd[q] = nv;
                wd[q] = nw;
            }
        } else {
            const float a = hi4[(size_t)split_hi_offset(order, ls, j) * 2].x;
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                if (j == ls + 1) {
                    vdf[q] = (float)vd[q];
                    wdf[q] = (float)wd[q];
                }
                const float nv = a * fmaf(xf[q], vdf[q], -yf[q] * wdf[q]);
                const float nw = a * fmaf(xf[q], wdf[q], yf[q] * vdf[q]);
                vdf[q] = nv;
                wdf[q] = nw;
            }
        }
    };
    // FP32 interior rows: n cells from hc, recursion seeded by rows l-2, l-1
    auto fp32_interior = [&](const float4* hc, int n, float* v0, float* w0, float* v1, float* w1) {
        const int pairs = n >> 1;
        float4 nx[4];
        if (pairs > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) nx[i] = hc[i];
        }
#pragma unroll 2
        for (int p = 0; p < pairs; ++p) {
            float4 cb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) cb[i] = nx[i];
            if (p + 1 < pairs) {
#pragma unroll
                for (int i = 0; i < 4; ++i) nx[i] = hc[4 + i];
            }
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const float ta = cb[0].x * zf[q], tb = cb[0].y * cf[q];
                v0[q] = fmaf(ta, v1[q], -tb * v0[q]);
                w0[q] = fmaf(ta, w1[q], -tb * w0[q]);
                fx[q] = fmaf(cb[0].z, v0[q], fmaf(cb[0].w, w0[q], fx[q]));
                fy[q] = fmaf(cb[1].x, v0[q], fmaf(cb[1].y, w0[q], fy[q]));
                fz[q] = fmaf(cb[1].z, v0[q], fmaf(cb[1].w, w0[q], fz[q]));
                const float ta2 = cb[2].x * zf[q], tb2 = cb[2].y * cf[q];
                v1[q] = fmaf(ta2, v0[q], -tb2 * v1[q]);
                w1[q] = fmaf(ta2, w0[q], -tb2 * w1[q]);
                fx[q] = fmaf(cb[2].z, v1[q], fmaf(cb[2].w, w1[q], fx[q]));
                fy[q] = fmaf(cb[3].x, v1[q], fmaf(cb[3].y, w1[q], fy[q]));
                fz[q] = fmaf(cb[3].z, v1[q], fmaf(cb[3].w, w1[q], fz[q]));
            }
            hc += 4;
        }
        if (n & 1) {
            const float4 c0 = hc[0], c1 = hc[1];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const float ta = c0.x * zf[q], tb = c0.y * cf[q];
                const float v2 = fmaf(ta, v1[q], -tb * v0[q]);
                const float w2 = fmaf(ta, w1[q], -tb * w0[q]);
                fx[q] = fmaf(c0.z, v2, fmaf(c0.w, w2, fx[q]));
                fy[q] = fmaf(c1.x, v2, fmaf(c1.y, w2, fy[q]));
                fz[q] = fmaf(c1.z, v2, fmaf(c1.w, w2, fz[q]));
            }
        }
    };
    for (int j = 1; j < j0; ++j) advance_diag(j);
    for (int j = j0; j < j1; ++j) {
        if (j > 0) advance_diag(j);
        float v0f[NT], w0f[NT], v1f[NT], w1f[NT];
        if (j <= ls) {
            // FP64 rows j..ls
            const double2* cell = lo2 + (size_t)split_lo_offset(ls, j) * 4;
            double v0[NT], w0[NT], v1[NT], w1[NT];
            {
                const double2 wxx = cell[1], wyy = cell[2], wzz = cell[3];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    ax[q] = fma(wxx.x, vd[q], fma(wxx.y, wd[q], ax[q]));
                    ay[q] = fma(wyy.x, vd[q], fma(wyy.y, wd[q], ay[q]));
                    az[q] = fma(wzz.x, vd[q], fma(wzz.y, wd[q], az[q]));
                    v0[q] = 0.0;
                    w0[q] = 0.0;
                    v1[q] = vd[q];
                    w1[q] = wd[q];
                }
                cell += 4;
            }
            for (int l = j + 1; l <= ls; ++l) {
                const double2 ab = cell[0], wxx = cell[1], wyy = cell[2], wzz = cell[3];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const double ta = ab.x * zc[q];
                    const double v2 = l == j + 1 ? ta * v1[q] : fma(ta, v1[q], -(ab.y * c2re[q]) * v0[q]);
                    const double w2 = l == j + 1 ? ta * w1[q] : fma(ta, w1[q], -(ab.y * c2re[q]) * w0[q]);
                    ax[q] = fma(wxx.x, v2, fma(wxx.y, w2, ax[q]));
                    ay[q] = fma(wyy.x, v2, fma(wyy.y, w2, ay[q]));
                    az[q] = fma(wzz.x, v2, fma(wzz.y, w2, az[q]));
                    v0[q] = v1[q];
                    w0[q] = w1[q];
                    v1[q] = v2;
                    w1[q] = w2;
                }
                cell += 4;
            }
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                v0f[q] = (float)v0[q];
                w0f[q] = (float)w0[q];
                v1f[q] = (float)v1[q];
                w1f[q] = (float)w1[q];
            }
            // FP32 rows ls+1..last
            const float4* hc = hi4 + (size_t)split_hi_offset(order, ls, j) * 2;
            int n = last - ls;
            if (j == ls) {  // row ls+1 is this column's sub-diagonal
                const float4 c0 = hc[0], c1 = hc[1];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const float a = c0.x * zf[q];
                    v0f[q] = v1f[q];
                    w0f[q] = w1f[q];
                    v1f[q] = a * v0f[q];
                    w1f[q] = a * w0f[q];
                    fx[q] = fmaf(c0.z, v1f[q], fmaf(c0.w, w1f[q], fx[q]));
                    fy[q] = fmaf(c1.x, v1f[q], fmaf(c1.y, w1f[q], fy[q]));
                    fz[q] = fmaf(c1.z, v1f[q], fmaf(c1.w, w1f[q], fz[q]));
                }
                hc += 2;
                --n;
            }
            fp32_interior(hc, n, v0f, w0f, v1f, w1f);
        } else {
            // all FP32: diagonal, sub-diagonal, interior
            const float4* hc = hi4 + (size_t)split_hi_offset(order, ls, j) * 2;
            {
                const float4 c0 = hc[0], c1 = hc[1];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    fx[q] = fmaf(c0.z, vdf[q], fmaf(c0.w, wdf[q], fx[q]));
                    fy[q] = fmaf(c1.x, vdf[q], fmaf(c1.y, wdf[q], fy[q]));
                    fz[q] = fmaf(c1.z, vdf[q], fmaf(c1.w, wdf[q], fz[q]));
                }
                hc += 2;
            }
            if (j == last) continue;
            {
                const float4 c0 = hc[0], c1 = hc[1];
#pragma unroll
                for (int q = 0; q < NT; ++q) {
                    const float a = c0.x * zf[q];
                    v0f[q] = vdf[q];
                    w0f[q] = wdf[q];
                    v1f[q] = a * vdf[q];
                    w1f[q] = a * wdf[q];
                    fx[q] = fmaf(c0.z, v1f[q], fmaf(c0.w, w1f[q], fx[q]));
                    fy[q] = fmaf(c1.x, v1f[q], fmaf(c1.y, w1f[q], fy[q]));
                    fz[q] = fmaf(c1.z, v1f[q], fmaf(c1.w, w1f[q], fz[q]));
                }
                hc += 2;
            }
            fp32_interior(hc, last - j - 1, v0f, w0f, v1f, w1f);
        }
    }
#pragma unroll
    for (int q = 0; q < NT; ++q) {
        acc[q][0] = ax[q] + (double)fx[q];
        acc[q][1] = ay[q] + (double)fy[q];
        acc[q][2] = az[q] + (double)fz[q];
    }
}

}  // namespace bqp
