// rad.cu -- volume radiation transfer on the device: the volume part of
// RAD_EMIS (combustion/Code/Rad_emis.f90:120-377).
//
//   k_rad_mark    wall markers: IBCELL 1 -> 101..311 where a neighbour is open
//                 (Rad_emis.f90:144-178), on a cell map of its own
//   k_rad_akl     RAD0 with ID_RAD=10 (Rad0.f90:112-166): AKL = EMF(AKL0, OPL)
//                 of the hot open cells, band-emission totals, and QREF's
//                 per-area band emission QEL0 of every emitter
//   k_rad_qe      QE of every emitter (QREF's six face powers and band sum)
//   k_rad_trace   the QRNF emitter loop (Qrn.f90:58-154) with the x-, y- or
//                 z-flux of QREF (Qre.f90:31-515) and QRTX/QRTY/QRTZ
//                 (Qrtx.f90:15-209, Qrty.f90:9-224, Qrtz.f90:15-234): one
//                 launch per direction, the three on three streams at once
//   k_rad_reduce  QAL summed over the CTAs, QA = sum over bands (QRN1,
//                 Qrn.f90:250-259), and the open cells' share of it
//
// A CTA of direction d traces that direction for one emitter at a time (cells
// in the reference's loop order, a grid-stride over the emitters); emitters
// and directions are independent, so many are in flight at once, each
// direction's CTAs sized by its own slab.  Within one emitter and direction
// the reference is sequential; the CTA keeps its order where it matters:
//   * everything the reference derives from angles -- which rows and columns of
//     a slab are visited, which parts of one cell's beam fall on which cells of
//     the next face (FIJ, a division each) -- depends on coordinates alone, so
//     it is tabulated (k_rad_table, once per handle where the tables fit) with
//     the reference's expressions and early exits; a slab reads two records;
//   * the slab arrays QTX1, QTX2, Q2M (bands fastest) and their flags live in
//     shared memory (global scratch when they do not fit);
//   * the spread across the first transverse axis (part 1 of QRTX/Y/Z) touches
//     only its own row of the slab arrays, and the spread across the second
//     (part 2) only its own column, except for the wall-corner split, which also
//     adds into the neighbouring column toward the emitter (for the emitter's
//     own column, the column its loop variable last held).  Bands are
//     independent throughout: one lane per row (column) and band, a row's bands
//     in one warp, the reference's order inside each;
//   * splits into other columns are listed per column during part 2 and added
//     after it in the reference's column order, a lane per band (associated
//     differently from the reference by a few roundings).  A target outside the
//     slab is reported as unsupported;
//   * absorption into the slab's cells is per cell.
// What bounds it: the length of the chains between a slab's barriers (a row's or
// column's walk, one shared-memory read-modify-write after the other) and the
// FP64 pipe (64 cycles a warp instruction on a sub-partition, whatever the
// active lanes; that pipe is 33 to 48% busy in a trace, a warp waits at barriers
// and in chains).  With two CTAs on an SM and ten bands a slab of 14x12x10 cells
// takes about 14 us of its CTA.  So: a lane per
// band (a tenth of the chain of a thread that loops over the bands), no division
// and no angle on the chain, the first and last columns in the same phase as the
// others, the next slab's codes loaded behind part 1, a cell's QAL and AKL
// loaded for all bands at once.  Whole transfer, 10 bands, with the exchange
// between the walls: 106.7 ms with angles and divisions per emitter and a thread
// per row, 55.8 with the tables and a lane per band, 44.8 with one phase for all
// columns, 40.5 with the loads ahead, 38.2 with QA's total for the open cells;
// 32x16x12 cells and 4 bands 131 -> 101 ms.  A first transfer, which fills the
// tables (twice where a walk is longer than four cells, as in the tank): 51 ms
// against 118.
// QAL is accumulated per CTA in its own copy (fixed emitter order) and the
// copies are summed in a fixed order (x-direction CTAs, then y, then z), so
// the result is deterministic; it differs from the reference's single running
// sum only by the association of the additions.
//
// Angles come from rad_atand, the same operations as the oracle's ATAND; this
// translation unit is compiled with --fmad=false so that no multiply-add is
// fused where the reference rounds twice: angle ties break the same way, and the
// rest of a beam, a difference that can cancel, is the reference's.
#include <algorithm>

#include "rad_split.h"
#include "state.cuh"

namespace gfm {
namespace {

constexpr double kSmall16 = 1.0e-16;

// A double's IEEE bit pattern as a signed 64-bit integer.  Two non-negative
// doubles, or any double and a positive one, compare the same way as these
// integers (no NaN occurs here), so the frequent comparisons of angles and of
// powers against SMALL16 run on the integer pipe, GB300's FP64 pipe being
// narrow; the results are those of the floating-point comparisons.
__device__ __forceinline__ long long rb(double x) { return __double_as_longlong(x); }
constexpr double kTgMn = 300.0;     // TG_MN (Rad0.f90:42)
constexpr int kRadThreads = 256;

// atan(x) in degrees: reduction to [0,1] by atan(x) = pi/2 - atan(1/x), to
// [0, tan(pi/12)] by atan(a) = pi/6 + atan((a*sqrt(3)-1)/(a+sqrt(3)))
// (Abramowitz & Stegun 4.4.34), Maclaurin series to t^29 (A&S 4.4.42) by
// Horner's rule in t^2 with fused multiply-adds.
__device__ double rad_atand(double x) {
    const double PI = 3.14159265358979323846;
    const double SQRT3 = 1.73205080756887729353;
    const double TAN_PI_12 = 0.26794919243112270647;
    double a = fabs(x);
    const bool inv = a > 1.0;
    if (inv) a = 1.0 / a;
    const bool sh = a > TAN_PI_12;
    if (sh) a = (a * SQRT3 - 1.0) / (a + SQRT3);
    const double z = a * a;
    double p = 1.0 / 29.0;
#pragma unroll
    for (int n = 13; n >= 0; --n) p = fma(p, z, ((n & 1) ? -1.0 : 1.0) / (double)(2 * n + 1));
    double r = a * p;
    if (sh) r = PI / 6.0 + r;
    if (inv) r = PI / 2.0 - r;
    const double d = r * (180.0 / PI);
    return x < 0.0 ? -d : d;
}

__global__ void k_rad_mark(RadArgs a) {
    const int n = a.MZ * a.NZ * a.LZ;
    GFM_FOR(c, n) {
        const int I = 2 * (c % a.MZ + 1), J = 2 * ((c / a.MZ) % a.NZ + 1), K = 2 * (c / (a.MZ * a.NZ) + 1);
        auto ibc = [&](int i, int j, int k) { return (int)a.g.ib[pidx(a.g, i, j, k)]; };
        int v = ibc(I, J, K);
        if (v == 1) {
            const int KM2 = max(K - 2, 2), KP2 = min(K + 2, a.LP);
            const int JM2 = max(J - 2, 2), JP2 = min(J + 2, a.NP);
            const int IM2 = max(I - 2, 2), IP2 = min(I + 2, a.MP);
            if (ibc(I, J, KM2) <= 0) v = 301;
            else if (ibc(I, J, KP2) <= 0) v = 311;
            else if (ibc(I, JM2, K) <= 0) v = 201;
            else if (ibc(I, JP2, K) <= 0) v = 211;
            else if (ibc(IM2, J, K) <= 0) v = 101;
            else if (ibc(IP2, J, K) <= 0) v = 111;
        }
        a.ibr[c] = (int16_t)v;
    }
}

__device__ void rad_debx(const RadArgs& a, double t, double* deb) {   // DEBX, Rad_fun.f90:83-101
    double eb0 = 0.0;
    for (int l = 1; l <= a.NWL - 1; ++l) {
        const double x1 = a.deb0[l - 1] / t;
        const double eb1 = rif3(x1);
        deb[l - 1] = eb1 - eb0;
        if (deb[l - 1] <= 1.0e-3) deb[l - 1] = 0.0; else eb0 = eb1;
    }
    deb[a.NWL - 1] = 1.0 - eb0;
}

// RAD0 (ID_RAD=10): AKL = EMF(AKLG + AKLS) from the band model (gas.cu), or
// from the gray bands (AKLG = AKL0, AKLS = 0).  Also the cell
// temperature in kelvin (T*T0), the one the transfer reads, and for every
// emitter (open, T > TG_MN) QREF's emission per unit area of each band,
// QEL0 = DEB*AKL*SGN*T^4 (Qre.f90:80-86), with the same DEB.  Block partials
// of the two band-emission totals are summed on the host in block order.
template <typename R>
__global__ void __launch_bounds__(256) k_rad_akl(RadArgs a, const R* __restrict__ T) {
    __shared__ double sh[2][256];
    const int n = a.MZ * a.NZ * a.LZ;
    double sg_tot = 0.0, ss_tot = 0.0;
    GFM_FOR(c, n) {
        const int I = 2 * (c % a.MZ + 1), J = 2 * ((c / a.MZ) % a.NZ + 1), K = 2 * (c / (a.MZ * a.NZ) + 1);
        const double t = (double)T[pidx(a.g, I, J, K)] * a.t0;
        a.tcell[c] = t;
        for (int l = 0; l < a.NWL; ++l) { a.aklt[(long long)c * a.NWL + l] = 0.0; a.qel0[c + (long long)l * n] = 0.0; }
        if (!(a.ibr[c] <= 0 && t >= kTgMn)) continue;
        const double dx = a.g.DX[I], dr = a.g.DR[J], dz = a.g.DZ[K];
        double vol = dx * dr * a.g.RS[J] * dz;                        // VOL_C at a cell centre (VOL_C0)
        if (a.g.HALF && a.ibr[c] <= -1) vol = vol * a.g.BVF[-a.ibr[c] - 1];
        const double sa = ((dx * dr) + (dr * dz) + (dx * dz)) * 2.0;
        if (sa <= kSmall16) continue;
        const double opl = 6.0 * vol / sa;
        if (opl <= 1.0e-10) continue;
        double deb[kRadMaxBands];
        rad_debx(a, t, deb);
        const double t2 = t * t;
        const double area_sgn_t4 = sa * a.sgn * (t2 * t2);
        double sg = 0.0, ss = 0.0;
        const bool emitter = t > kTgMn;
        const double g0 = a.sgn * (t2 * t2);
        for (int l = 0; l < a.NWL; ++l) {
            const long long cl = c + (long long)l * n;
            const double ag = a.gas_aklg ? a.gas_aklg[cl] : a.akl0[l];
            const double as = a.gas_aklg ? a.gas_akls[cl] : 0.0;
            const double akl = emf(a.gas_aklg ? ag + as : a.akl0[l], opl);
            a.aklt[(long long)c * a.NWL + l] = akl;
            if (emitter) a.qel0[cl] = deb[l] * akl * g0;
            sg = sg + deb[l] * emf(ag, opl);
            ss = ss + deb[l] * emf(as, opl);
        }
        sg_tot += area_sgn_t4 * sg;
        ss_tot += area_sgn_t4 * ss;
    }
    sh[0][threadIdx.x] = sg_tot;
    sh[1][threadIdx.x] = ss_tot;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) { sh[0][threadIdx.x] += sh[0][threadIdx.x + s]; sh[1][threadIdx.x] += sh[1][threadIdx.x + s]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) { a.akl_part[2 * blockIdx.x] = sh[0][0]; a.akl_part[2 * blockIdx.x + 1] = sh[1][0]; }
}

// One march direction of QREF: d = slab axis, u = first transverse axis (the
// part-1 spread, the part-2 columns), v = second (the part-1 rows, the part-2
// spread).  x-flux: u = y, v = z (QRTX); y-flux: u = x, v = z (QRTY); z-flux:
// u = x, v = y (QRTZ).  Slab arrays are indexed e = (v/2-1)*DA + (u/2-1).
__host__ __device__ __forceinline__ int rad_u(int d) { return d == 0 ? 1 : 0; }
__host__ __device__ __forceinline__ int rad_v(int d) { return d == 2 ? 1 : 2; }

// ---------------------------------------------------------------------------
// The angle tables.  Record of (direction d, transverse axis, emitter's slab
// d0, slab, emitter's position p0 on the axis): for every source position p1 in
// two lists -- the outward walk to smaller positions (slot p1/2-1) and to larger
// ones (the same, the emitter's own position in slot N) -- K codes, then one
// byte per position: is the row (column) visited (SANG1, SANG2 and the loops of
// QRTX/QRTY/QRTZ).  Code k of a walk is about the cell k steps outward:
//   kStop (first code): the walk ends here (A11 >= the emitter's cone);
//   kSkip (first code): no beam from this cell (A12 - A11 <= 1e-10);
//   kNone: the beam does not reach this cell's far face yet;
//   kRest: the rest of the beam falls on it;
//   else FIJ = (A22 - A21)/(A12 - A11), the part of the beam that does.
// One warp per (d0, side, p0) walks the slabs outward as the reference does,
// its lanes on the faces (angles) and on the source positions (codes).
// ---------------------------------------------------------------------------
constexpr double kStop = 4.0, kSkip = 3.0, kRest = 2.0, kNone = -1.0;
__host__ __device__ __forceinline__ long long rad_rec(int n, int K) { return (long long)(n + 1) * K + (n + 7) / 8; }

struct RadTab {
    const double *cd, *cp;       // coordinates of the slab axis and the transverse axis (1-based)
    int Dd, P, first;            // first: the axis is u (part 1; its columns end at P), else v
    int lo;                      // the first of the emitter's slabs held (blocks: cnt of them)
    int K;                       // codes kept per walk; the most any walk has goes to kmax
    double* out;
    int* kmax;
};
__global__ void __launch_bounds__(32) k_rad_table(RadTab t) {
    extern __shared__ __align__(16) unsigned char rad_smem[];
    double* a1 = reinterpret_cast<double*>(rad_smem);   // angles of the faces 1 .. P+1: the current slab's near faces,
    double* a2 = a1 + t.P + 2;                          // its far faces,
    double* cand = a2 + t.P + 2;                        // and the latter before the early exit
    const int nd = t.Dd / 2, n = t.P / 2, lane = threadIdx.x, id = blockIdx.x;
    const int p0 = 2 * (id % n) + 2, s = (id / n) % 2 ? 1 : -1, d0 = 2 * (id / (2 * n) + t.lo) + 2;
    // SANG1 for an open cell
    const double b0 = fabs(t.cd[d0 + s] - t.cd[d0]);
    const double lim = b0 < kSmall16 ? 90.0 : rad_atand(fabs(t.cp[p0 + s] - t.cp[p0]) / b0);
    for (int p = 1 + lane; p <= t.P + 1; p += 32) { a1[p] = p == p0 ? 0.0 : lim; a2[p] = a1[p]; }
    const int last = t.first ? t.P : t.P - 2;
    int kmax = 1;
    for (int slab = d0 + 2 * s; s > 0 ? slab <= t.Dd : slab >= 2; slab += 2 * s) {
        const int far = min(slab + s, t.Dd);
        const double b = fabs(t.cd[far] - t.cd[d0]);
        for (int pp = 1 + 2 * lane; pp <= t.P; pp += 64)
            cand[pp] = b < kSmall16 ? 90.0 : rad_atand(fabs(t.cp[pp] - t.cp[p0]) / b);
        __syncwarp();
        // SANG2: outward with its early exit
        if (lane < 2) {
            const int M = lane ? 1 : -1;
            for (int pp = p0 + M; M > 0 ? pp <= t.P : pp >= 2; pp += 2 * M) {
                if (rb(cand[pp]) >= rb(lim)) break;
                a2[pp] = cand[pp];
            }
        }
        __syncwarp();
        double* rec = t.out + (((long long)(d0 / 2 - 1 - t.lo) * nd + (slab / 2 - 1)) * n + (p0 / 2 - 1)) * rad_rec(n, t.K);
        // the first position after the emitter that ends the loop over them;
        // before it, each position by itself
        int exit = last + 2;
        for (int q = p0 + 2; q <= last; q += 2)
            if (rb(a2[q - 1]) >= rb(lim)) { exit = q; break; }
        unsigned char* vis = reinterpret_cast<unsigned char*>(rec + (long long)(n + 1) * t.K);
        for (int p = 2 + 2 * lane; p <= t.P; p += 64) vis[p / 2 - 1] = p < p0 ? rb(a2[p + 1]) < rb(lim) : p < exit;
        // slot i: source position 2(i+1) outward, the emitter's own to larger positions in slot n
        for (int i = lane; i <= n; i += 32) {
            const int p1 = i < n ? 2 * i + 2 : p0, M = i == n || p1 > p0 ? 2 : -2, end = M < 0 ? 2 : t.P;
            if (M > 0 ? p1 > end - M : p1 < end - M) continue;   // not a source
            double* c = rec + (long long)i * t.K;
            const double A11 = p1 == p0 ? 0.0 : a1[p1 - M / 2];
            if (rb(A11) >= rb(lim)) { c[0] = kStop; continue; }
            const double A12 = a1[p1 + M / 2], dang = A12 - A11;
            if (dang <= 1.0e-10) { c[0] = kSkip; continue; }
            double A21 = A11;
            int k = 0;
            for (int p2 = p1; M > 0 ? p2 <= end : p2 >= end; p2 += M, ++k) {
                const int pm = p2 + M / 2;
                double code;
                if (!t.first && (pm > t.P || pm < 2)) code = kRest;   // part 2: nothing beyond the last cell
                else {
                    const double A22 = a2[pm];
                    if (t.first ? A22 <= A21 : (A22 - A21) <= 1.0e-10) code = kNone;
                    else if (A22 < A12) { code = (A22 - A21) / dang; A21 = A22; }
                    else code = kRest;
                }
                if (k < t.K) c[k] = code;
                if (code == kRest) { ++k; break; }
            }
            kmax = max(kmax, k);
        }
        __syncwarp();
        for (int p = 1 + lane; p <= t.P; p += 32) a1[p] = a2[p];
        __syncwarp();
    }
    atomicMax(t.kmax, kmax);
}

struct Dir {
    int d, Dd, Du, Dv, DA, DB, A;
    int d0, u0, v0;
    int sd, su, sv;              // cell-index strides of the three axes
    int direct1, direct2;        // IBCELL codes deposited whole in part 2 (and 4)
    int lo;                      // the first of the emitter's slabs in the tables
    int Ku, Kv;
};

struct Slab {   // scratch of one CTA
    double *q1, *q2, *qm;        // QTX1, QTX2, Q2M: [e*NWL + l]
    unsigned char *f1, *f2, *fm; // IQT1, IQT2, IQTM
    double* edge;                // splits of the first and the last column: [(side*DB + row)*NWL + l]
    const int16_t* ib;           // IBCELL (with wall markers) of the current slab's cells: [e]
    const double *cu, *cv;       // the slab's angle records
};

// Corner-split additions of the interior columns into other columns, gathered
// during part 2 of one slab (those of the first and last column, which a box
// has in every slab, go to buffers of their own, added where the cells absorb):
// up to split_room of a column (rad_split.h; of the first and the last only when the
// emitter's own) in the CTA's global scratch, in the column's own order; and, in
// shared memory, the two values that decide the emitter column's target.
struct SplitList {
    int* any;                    // a column listed a split in this slab
    int* maxbelow;               // largest column below the emitter that split (0: none)
    unsigned long long* last1;   // (row << 32) | (u2 + 8) of the slab's last part-1 spread
    int* cnt;                    // [column]: entries used (zero between slabs), in shared memory
    int* meta;                   // [entry][2] from split_first of the column: target row, target column (-1: emitter's)
    double* q;                   // [entry][band] (0 where the band's power is negligible)
    int nw;
};

__device__ __forceinline__ bool rad_corner(int d, int ibc1) {
    return d == 0 ? ibc1 > 100 : (d == 1 ? ibc1 >= 100 : ibc1 > 1);
}

// Band l of the row of cells bb (part 1).  All lanes of the warp walk together
// (the walk depends on the columns' angles only); `on`: the lane's row is
// visited.  One lane of a row (l == 0) writes the flags it shares.
__device__ void part1_row(const Dir& D, const Slab& S, int bb, int l, int nw, bool on, const SplitList& SL) {
    const int n = D.Du / 2;
    const int row = (bb - 1) * D.DA - 1;   // cell u/2 of the row at row + u/2
    int last_u2 = 0;
    for (int UPM = -2; UPM <= 2; UPM += 4) {
        const int uend = UPM < 0 ? 2 : D.Du;
        for (int u1 = D.u0; UPM > 0 ? u1 <= uend - UPM : u1 >= uend - UPM; u1 += UPM) {
            const bool own = u1 == D.u0;
            const double* c = S.cu + (long long)(own && UPM > 0 ? n : u1 / 2 - 1) * D.Ku;
            const long long c0 = rb(c[0]);
            if (c0 == rb(kStop)) break;
            if (c0 == rb(kSkip)) continue;
            const int e = row + u1 / 2;
            const bool act = on && !S.f1[e];
            __syncwarp();
            if (!act) continue;
            double* q = S.q1 + e * nw + l;
            double Q11 = *q;
            if (own) Q11 = Q11 * 0.5;
            if (!own || UPM > 0) {
                *q = 0.0;
                if (l == 0) S.f1[e] = 1;
            }
            double Q12 = Q11;
            const bool some = rb(Q11) >= rb(kSmall16);
            int u2 = u1;
            for (int k = 0; UPM > 0 ? u2 <= uend : u2 >= uend; u2 += UPM, ++k) {
                const int e2 = row + u2 / 2;
                if (S.ib[e2] < 1) {
                    const double F = c[k];
                    if (rb(F) < 0) continue;   // kNone
                    if (rb(F) < rb(kRest)) {
                        if (some) {
                            const double Q21 = Q11 * F;
                            S.qm[e2 * nw + l] = S.qm[e2 * nw + l] + Q21;
                            Q12 = Q12 - Q21;
                        }
                        S.fm[e2] = 0;
                        continue;
                    }
                }
                S.qm[e2 * nw + l] = S.qm[e2 * nw + l] + Q12;
                S.fm[e2] = 0;
                break;
            }
            last_u2 = u2 + 8;   // the loop variable as the loop leaves it
        }
    }
    // rows run in parallel: the reference's last spread is the highest row's
    if (last_u2 && l == 0) atomicMax(SL.last1, ((unsigned long long)(2 * bb) << 32) | (unsigned)last_u2);
}

// Band l of the column of cells aa (part 2), as part1_row; `on`: the lane's column is visited.
__device__ void part2_col(const Dir& D, const Slab& S, int aa, int l, int nw, bool on, int* err, const SplitList& SL) {
    const int n = D.Dv / 2, u1 = 2 * aa;
    int listed = 0;
    for (int KM = -2; KM <= 2; KM += 4) {
        const int vend = KM < 0 ? 2 : D.Dv;
        for (int v1 = D.v0; KM > 0 ? v1 <= vend - KM : v1 >= vend - KM; v1 += KM) {
            const bool own = v1 == D.v0;
            const double* c = S.cv + (long long)(own && KM > 0 ? n : v1 / 2 - 1) * D.Kv;
            const long long c0 = rb(c[0]);
            if (c0 == rb(kStop)) break;
            if (c0 == rb(kSkip)) continue;
            const int e = (v1 / 2 - 1) * D.DA + (aa - 1);
            const bool act = on && !S.fm[e];
            __syncwarp();
            if (!act) continue;
            double* q = S.qm + e * nw + l;
            double Q11 = *q;
            if (own) Q11 = Q11 * 0.5;
            if (!own || KM > 0) {
                *q = 0.0;
                if (l == 0) S.fm[e] = 1;
            }
            const int ibc1 = S.ib[e];
            if (ibc1 == D.direct1 || ibc1 == D.direct2 || ibc1 == 4) {
                S.q2[e * nw + l] = S.q2[e * nw + l] + Q11;
                S.f2[e] = 0;
                continue;
            }
            double Q12 = Q11;
            const bool some = rb(Q11) >= rb(kSmall16);
            int e2 = e;
            int k = 0;
            for (int v2 = v1; KM > 0 ? v2 <= vend : v2 >= vend; v2 += KM, ++k, e2 += KM / 2 * D.DA) {
                const int ibc2 = S.ib[e2];
                if (!(ibc1 <= 0 && ibc2 >= 1)) {
                    if (rad_corner(D.d, ibc1) && ibc2 == 1) {
                        // half into the neighbouring column toward the emitter
                        // (the emitter's own column: resolved when the list is
                        // applied), half into this column's previous row
                        const int ut = u1 < D.u0 ? u1 + 2 : (u1 > D.u0 ? u1 - 2 : -1);
                        const int e2m = e2 - KM / 2 * D.DA;
                        double Q21 = 0.0;
                        if (rb(Q12) >= rb(kSmall16)) {
                            Q21 = Q12 * 0.5;
                            S.q2[e2m * nw + l] = S.q2[e2m * nw + l] + Q21;
                        }
                        const long long ent = split_first(D.DA, D.Dv, aa) + listed;
                        if (ut >= 2 && (aa == 1 || aa == D.DA)) {
                            // first and last column: only they write their buffer
                            const int r = (aa == 1 ? 0 : D.DB) + v2 / 2 - 1;
                            S.edge[r * nw + l] = S.edge[r * nw + l] + Q21;
                            S.f2[e2 + (ut - u1) / 2] = 0;
                        } else if (listed < split_room(D.DA, D.Dv, aa)) {
                            SL.q[ent * nw + l] = Q21;
                            ++listed;
                            if (l == 0) { SL.meta[2 * ent] = v2; SL.meta[2 * ent + 1] = ut; }
                        } else {
                            atomicOr(err, 1);   // more splits in one column than the list holds
                        }
                        if (l == 0 && u1 < D.u0) atomicMax(SL.maxbelow, u1);
                        S.f2[e2m] = 0;
                        break;
                    }
                    const double F = c[k];
                    if (rb(F) < 0) continue;   // kNone
                    if (rb(F) < rb(kRest)) {
                        if (some) {
                            const double Q21 = Q11 * F;
                            S.q2[e2 * nw + l] = S.q2[e2 * nw + l] + Q21;
                            Q12 = Q12 - Q21;
                        }
                        S.f2[e2] = 0;
                        continue;
                    }
                }
                S.q2[e2 * nw + l] = S.q2[e2 * nw + l] + Q12;
                S.f2[e2] = 0;
                break;
            }
        }
    }
    if (listed && l == 0) {
        SL.cnt[aa - 1] = listed;
        *SL.any = 1;
    }
}

// The listed splits in the reference's column order (and, within a column, its
// order), a lane per band of one warp; the emitter column's target is two past
// the last column below the emitter that split, else where the slab's last
// part-1 spread ended.
__device__ void rad_apply_splits(const Dir& D, const Slab& S, int l, const SplitList& SL, int* err) {
    int tgt_emitter = -1;
    if (*SL.maxbelow >= 2) tgt_emitter = *SL.maxbelow + 2;
    else if (*SL.last1 != 0ull) tgt_emitter = (int)(unsigned)(*SL.last1 & 0xffffffffull) - 8;
    for (int c = 1; c <= D.DA; ++c) {   // source columns 2, 4, .. in the reference's order
        const int m = SL.cnt[c - 1];
        __syncwarp();
        if (l == 0) SL.cnt[c - 1] = 0;
        for (int k = 0; k < m; ++k) {
            const long long ent = split_first(D.DA, D.Dv, c) + k;
            const int row = SL.meta[2 * ent];
            const int col = SL.meta[2 * ent + 1] >= 0 ? SL.meta[2 * ent + 1] : tgt_emitter;
            if (col < 2 || col > D.Du || (col & 1) || row < 2 || row > D.Dv) { if (l == 0) atomicOr(err, 1); continue; }
            const int et = (row / 2 - 1) * D.DA + (col / 2 - 1);
            if (l < SL.nw) S.q2[et * SL.nw + l] = S.q2[et * SL.nw + l] + SL.q[ent * SL.nw + l];
            if (l == 0) S.f2[et] = 0;
        }
    }
}

// Per-thread sums of the deposits by destination.  What open cells absorb on the
// way is not summed here (a quarter of the absorption's work on the FP64 pipe) but
// by k_rad_reduce, as QA over the open cells; `open` takes out what was deposited
// whole in an open cell, at the end of the box, and counts as the wall's.
struct RadAcc {
    double melt, exit, inlet, wall, open;
};

// The next slab's two angle records and IBCELL codes: loaded into registers
// before part 1, stored to the other buffers after part 2 (what does not fit the
// registers is copied then).
struct RadFetch {
    static constexpr int NR = 2, NI = 3;
    const double *tu, *tv;
    const int16_t* ibr;
    double u[NR], v[NR];
    int16_t ib[NI];
    __device__ __forceinline__ int cell(const Dir& D, int e) const { return (e % D.DA) * D.su + (e / D.DA) * D.sv; }
    __device__ __forceinline__ void load(const RadArgs& a, const Dir& D, int slab) {
        const int nd = D.Dd / 2, tid = threadIdx.x, nth = blockDim.x;
        const int ru = (int)rad_rec(D.DA, D.Ku), rv = (int)rad_rec(D.DB, D.Kv);
        const long long at = (long long)(D.d0 / 2 - 1 - D.lo) * nd + (slab / 2 - 1);
        tu = a.tab_u[D.d] + (at * D.DA + (D.u0 / 2 - 1)) * ru;
        tv = a.tab_v[D.d] + (at * D.DB + (D.v0 / 2 - 1)) * rv;
        ibr = a.ibr + (slab / 2 - 1) * D.sd;
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            if (tid + i * nth < ru) u[i] = tu[tid + i * nth];
            if (tid + i * nth < rv) v[i] = tv[tid + i * nth];
        }
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (tid + i * nth < D.A) ib[i] = ibr[cell(D, tid + i * nth)];
    }
    __device__ __forceinline__ void store(const Dir& D, double* cu, double* cv, int16_t* dst) const {
        const int tid = threadIdx.x, nth = blockDim.x;
        const int ru = (int)rad_rec(D.DA, D.Ku), rv = (int)rad_rec(D.DB, D.Kv);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            if (tid + i * nth < ru) cu[tid + i * nth] = u[i];
            if (tid + i * nth < rv) cv[tid + i * nth] = v[i];
        }
        for (int i = tid + NR * nth; i < ru; i += nth) cu[i] = tu[i];
        for (int i = tid + NR * nth; i < rv; i += nth) cv[i] = tv[i];
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (tid + i * nth < D.A) dst[tid + i * nth] = ib[i];
        for (int e = tid + NI * nth; e < D.A; e += nth) dst[e] = ibr[cell(D, e)];
    }
};

template <int NW>
__device__ void rad_direction(const RadArgs& a, const Dir& D, Slab& S, double* const rec[2], int16_t* const ibuf[2],
                              double* qalp, const double* qel1, RadAcc& acc, int* err, const SplitList& SL) {
    const int NWL = NW > 0 ? NW : a.NWL;
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
    // a lane per row (column) and band: `per` rows a warp, all bands of a row in it
    const int per = 32 / NWL, sub = lane / NWL, l = lane - sub * NWL;
    const long long ru = rad_rec(D.DA, D.Ku);
    // ALLOCATE and initialise the slab arrays of this direction
    for (int i = tid; i < D.A * NWL; i += nth) { S.q1[i] = 0.0; S.q2[i] = 0.0; S.qm[i] = 0.0; }
    for (int i = tid; i < D.A; i += nth) { S.f1[i] = 1; S.f2[i] = 1; S.fm[i] = 1; }
    for (int i = tid; i < 2 * D.DB * NWL; i += nth) S.edge[i] = 0.0;
    __syncthreads();
    const int e0 = (D.v0 / 2 - 1) * D.DA + (D.u0 / 2 - 1);
    for (int s = -1; s <= 1; s += 2) {
        const int dend = s < 0 ? 2 : D.Dd;
        int slab = D.d0 + 2 * s, buf = 0;
        if (tid < NWL) S.q1[e0 * NWL + tid] = qel1[tid];
        if (tid == 0) { S.f1[e0] = 0; *SL.any = 0; *SL.maxbelow = 0; *SL.last1 = 0ull; }
        RadFetch fetch;
        if (s > 0 ? slab <= dend : slab >= dend) {
            fetch.load(a, D, slab);
            fetch.store(D, rec[0], rec[0] + ru, ibuf[0]);
        }
        __syncthreads();
        for (; s > 0 ? slab <= dend : slab >= dend; slab += 2 * s, buf ^= 1) {
            S.cu = rec[buf];
            S.cv = rec[buf] + ru;
            S.ib = ibuf[buf];
            const unsigned char* vis_u = reinterpret_cast<const unsigned char*>(S.cu + (long long)(D.DA + 1) * D.Ku);
            const unsigned char* vis_v = reinterpret_cast<const unsigned char*>(S.cv + (long long)(D.DB + 1) * D.Kv);
            const bool more = s > 0 ? slab + 2 * s <= dend : slab + 2 * s >= dend;
            if (more) fetch.load(a, D, slab + 2 * s);
            // part 1: rows 4 .. Dv-2
            for (int r = warp * per; r < D.DB - 2; r += (nth / 32) * per) {
                const int bb = r + sub + 2;
                part1_row(D, S, bb, l, NWL, sub < per && bb < D.DB && vis_v[bb - 1], SL);
            }
            __syncthreads();
            // part 2: all columns
            for (int r = warp * per; r < D.DA; r += (nth / 32) * per) {
                const int aa = r + sub + 1;
                part2_col(D, S, aa, l, NWL, sub < per && aa <= D.DA && vis_u[aa - 1], err, SL);
            }
            __syncthreads();
            if (*SL.any) {
                if (warp == 0) rad_apply_splits(D, S, lane, SL, err);
                __syncthreads();
            }
            // the next slab's codes, fetched before part 1
            if (more) fetch.store(D, rec[buf ^ 1], rec[buf ^ 1] + ru, ibuf[buf ^ 1]);
            // absorption in the slab's cells; a cell's QAL is loaded for all bands at once
            const bool end = slab == dend;
            for (int e = tid; e < D.A; e += nth) {
                if (S.f2[e]) continue;
                const int ua = e % D.DA + 1, vb = e / D.DA + 1;
                const int c = (slab / 2 - 1) * D.sd + (ua - 1) * D.su + (vb - 1) * D.sv;
                const int ib = S.ib[e];
                const bool whole = ib >= 1 || end;
                double* qa = qalp + (long long)c * NWL;
                const double* ak = a.aklt + (long long)c * NWL;
                double* q2 = S.q2 + e * NWL;
                constexpr int NB = NW > 0 ? NW : 1;
                for (int b0 = 0; b0 < NWL; b0 += NB) {
                    double q[NB], o[NB], k[NB];
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        o[b] = qa[b0 + b];
                        if (!whole) k[b] = ak[b0 + b];
                        q[b] = q2[b0 + b];
                    }
                    // the edge columns' splits, the lower column's first
                    for (int side = 0; side < 2; ++side)
                        if (ua == (side ? D.DA - 1 : 2)) {
                            double* ed = S.edge + ((side ? D.DB : 0) + vb - 1) * NWL + b0;
#pragma unroll
                            for (int b = 0; b < NB; ++b)
                                if (rb(ed[b]) != 0) {
                                    q[b] = q[b] + ed[b];
                                    ed[b] = 0.0;
                                    q2[b0 + b] = q[b];
                                }
                        }
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        if (rb(q[b]) < rb(kSmall16)) continue;
                        if (whole) {
                            qa[b0 + b] = o[b] + q[b];
                            if (ib == 4) acc.melt += q[b];
                            else if (ib == 3) acc.exit += q[b];
                            else if (ib == 2) acc.inlet += q[b];
                            else acc.wall += q[b];
                            if (ib < 1) acc.open -= q[b];
                        } else {
                            qa[b0 + b] = fma(q[b], k[b], o[b]);
                            S.q1[e * NWL + b0 + b] = fma(-q[b], k[b], q[b]);
                            S.f1[e] = 0;
                        }
                        q2[b0 + b] = 0.0;
                        S.f2[e] = 1;
                    }
                }
            }
            if (tid == 0) { *SL.any = 0; *SL.maxbelow = 0; *SL.last1 = 0ull; }
            __syncthreads();
        }
    }
}

// One march direction d of QREF for every emitter of the grid-stride: the
// three directions are independent apart from the order of their QAL
// additions, so they run as three launches at once, each with the shared
// memory of its own slab.
template <int NW>
__global__ void __launch_bounds__(kRadThreads) k_rad_trace(RadArgs a, int d, int lo, int hi) {
    extern __shared__ __align__(16) unsigned char rad_smem[];
    __shared__ double s_qel1[kRadMaxBands];
    __shared__ double s_red[kRadThreads];
    __shared__ int s_any, s_maxbelow;
    __shared__ unsigned long long s_last1;
    const int NWL = NW > 0 ? NW : a.NWL;
    const int n = a.MZ * a.NZ * a.LZ;
    const int tid = threadIdx.x;
    Dir D;
    D.d = d;
    const int u = rad_u(d), v = rad_v(d);
    const int dims[3] = {a.MP, a.NP, a.LP};
    D.Dd = dims[d]; D.Du = dims[u]; D.Dv = dims[v];
    D.DA = D.Du / 2; D.DB = D.Dv / 2; D.A = D.DA * D.DB;
    const int strides[3] = {1, a.MZ, a.MZ * a.NZ};
    D.sd = strides[d]; D.su = strides[u]; D.sv = strides[v];
    D.direct1 = 100 * (d + 1) + 1; D.direct2 = 100 * (d + 1) + 11;
    D.Ku = a.tab_ku[d]; D.Kv = a.tab_kv[d];
    D.lo = lo;
    // layout: the slab's records and IBCELL codes, two buffers each, the edge
    // columns' splits, the lists' counts; then the slab arrays (each part in
    // shared memory, or in global scratch where it does not fit)
    unsigned char* const fixed = a.fixed_in_smem[d] ? rad_smem : a.xscratch[d] + (long long)blockIdx.x * a.fixed[d];
    const long long rr = rad_rec(D.DA, D.Ku) + rad_rec(D.DB, D.Kv);
    double* const rec[2] = {reinterpret_cast<double*>(fixed), reinterpret_cast<double*>(fixed) + rr};
    int16_t* const ib0 = reinterpret_cast<int16_t*>(rec[1] + rr);
    const int ibn = (D.A + 3) / 4 * 4;
    int16_t* const ibuf[2] = {ib0, ib0 + ibn};
    Slab S;
    S.edge = reinterpret_cast<double*>(ib0 + 2 * ibn);
    int* const cnt = reinterpret_cast<int*>(S.edge + 2 * D.DB * NWL);
    double* arr = reinterpret_cast<double*>(cnt + (D.DA + 1) / 2 * 2);
    S.q1 = a.slab_in_smem[d] ? arr : a.scratch[d] + (long long)blockIdx.x * 3 * D.A * NWL;
    S.q2 = S.q1 + (long long)D.A * NWL;
    S.qm = S.q2 + (long long)D.A * NWL;
    unsigned char* flags = a.slab_in_smem[d] ? reinterpret_cast<unsigned char*>(S.qm + (long long)D.A * NWL)
                                             : a.fscratch[d] + (long long)blockIdx.x * 3 * D.A;
    S.f1 = flags;
    S.f2 = flags + D.A;
    S.fm = flags + 2 * D.A;
    const long long lists = (long long)blockIdx.x * split_first(D.DA, D.Dv, D.DA + 1);
    const SplitList SL{&s_any, &s_maxbelow, &s_last1, cnt, a.split_meta[d] + 2 * lists, a.split_q[d] + lists * a.NWL, a.NWL};
    for (int e = tid; e < D.DA; e += blockDim.x) SL.cnt[e] = 0;
    const long long part = a.part_base[d] + blockIdx.x;
    double* qalp = a.qal_part + part * n * NWL;
    if (lo == 0)
        for (long long i = tid; i < (long long)n * NWL; i += blockDim.x) qalp[i] = 0.0;
    const double* dface[3] = {a.g.DX, a.g.DR, a.g.DZ};
    RadAcc acc{0.0, 0.0, 0.0, 0.0, 0.0};
    __syncthreads();

    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        // emitters in the reference's loop order: I outer, K inner
        const int KD2 = c % a.LZ + 1, JD2 = (c / a.LZ) % a.NZ + 1, ID2 = c / (a.LZ * a.NZ) + 1;
        const int cc = (ID2 - 1) + a.MZ * ((JD2 - 1) + a.NZ * (KD2 - 1));
        if (a.ibr[cc] >= 1 || a.tcell[cc] <= kTgMn) continue;
        const int pos[3] = {2 * ID2, 2 * JD2, 2 * KD2};
        if (pos[d] / 2 <= lo || pos[d] / 2 > hi) continue;
        D.d0 = pos[d]; D.u0 = pos[u]; D.v0 = pos[v];
        if (tid < NWL)   // power through one face of the emitter (QEL1, Qre.f90:118/241/384)
            s_qel1[tid] = a.qel0[cc + (long long)tid * n] * dface[u][D.u0] * dface[v][D.v0];
        __syncthreads();
        rad_direction<NW>(a, D, S, rec, ibuf, qalp, s_qel1, acc, a.err, SL);
        __syncthreads();
    }
    // block totals in a fixed order
    double vals[5] = {acc.melt, acc.exit, acc.inlet, acc.wall, acc.open};
    for (int k = 0; k < 5; ++k) {
        s_red[tid] = vals[k];
        __syncthreads();
        for (int st = blockDim.x / 2; st > 0; st >>= 1) {
            if (tid < st) s_red[tid] += s_red[tid + st];
            __syncthreads();
        }
        if (tid == 0) a.tot_part[8 * part + k] = lo == 0 ? s_red[0] : a.tot_part[8 * part + k] + s_red[0];
        __syncthreads();
    }
}

// QE of every emitter (QREF's QEL accumulation, Qre.f90:121/244/387, and the
// band sum, Qre.f90:503-507): the six faces' powers in the order x-, x+, y-,
// y+, z-, z+; block totals of the emission and of the emitter count.
__global__ void __launch_bounds__(256) k_rad_qe(RadArgs a) {
    __shared__ double sh[2][256];
    const int n = a.MZ * a.NZ * a.LZ;
    double qs = 0.0, cnt = 0.0;
    GFM_FOR(c, n) {
        a.qe[c] = 0.0;
        if (a.ibr[c] >= 1 || a.tcell[c] <= kTgMn) continue;
        const int I = 2 * (c % a.MZ + 1), J = 2 * ((c / a.MZ) % a.NZ + 1), K = 2 * (c / (a.MZ * a.NZ) + 1);
        double qe = 0.0;
        for (int l = 0; l < a.NWL; ++l) {
            const double q0 = a.qel0[c + (long long)l * n];
            const double fx = q0 * a.g.DR[J] * a.g.DZ[K], fy = q0 * a.g.DX[I] * a.g.DZ[K], fz = q0 * a.g.DX[I] * a.g.DR[J];
            double q = 0.0;
            q = q + fx; q = q + fx; q = q + fy; q = q + fy; q = q + fz; q = q + fz;
            qe = l == 0 ? q : qe + q;
        }
        a.qe[c] = qe;
        qs += qe;
        cnt += 1.0;
    }
    sh[0][threadIdx.x] = qs;
    sh[1][threadIdx.x] = cnt;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) { sh[0][threadIdx.x] += sh[0][threadIdx.x + s]; sh[1][threadIdx.x] += sh[1][threadIdx.x + s]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) { a.qe_part[2 * blockIdx.x] = sh[0][0]; a.qe_part[2 * blockIdx.x + 1] = sh[1][0]; }
}

// QAL = sum of the CTA copies in CTA order; QA = sum over bands (QRN1)
__global__ void __launch_bounds__(256) k_rad_reduce(RadArgs a) {
    __shared__ double sh[32];
    const int nparts = a.part_base[3];
    double open = 0.0;
    const int n = a.MZ * a.NZ * a.LZ;
    GFM_FOR(c, n) {
        double g0 = 0.0;
        for (int l = 0; l < a.NWL; ++l) {
            double s = 0.0;
            for (int b = 0; b < nparts; ++b) s += a.qal_part[((long long)b * n + c) * a.NWL + l];
            g0 = g0 + s;
        }
        a.qa[c] = g0;
        if (a.ibr[c] < 1) open += g0;
    }
    open = block_sum(open, sh);
    if (threadIdx.x == 0) a.open_part[blockIdx.x] = open;
}

// two buffers of the slab's records and IBCELL codes, the edge columns' splits, the lists' counts
size_t rad_smem_fixed(const RadArgs& a, int d, int A) {
    const int dims[3] = {a.MP, a.NP, a.LP};
    const int DA = dims[rad_u(d)] / 2, DB = dims[rad_v(d)] / 2;
    return 2 * (sizeof(double) * (size_t)(rad_rec(DA, a.tab_ku[d]) + rad_rec(DB, a.tab_kv[d])) +
                sizeof(int16_t) * (((size_t)A + 3) / 4 * 4)) +
           sizeof(double) * 2 * (size_t)DB * a.NWL + sizeof(int) * (size_t)((DA + 1) / 2 * 2);
}
size_t rad_smem_slab(const RadArgs& a, int A) { return (size_t)3 * A * a.NWL * sizeof(double) + (size_t)3 * A; }
int rad_slab_cells(const RadArgs& a, int d) {
    return d == 0 ? (a.NP / 2) * (a.LP / 2) : (d == 1 ? (a.MP / 2) * (a.LP / 2) : (a.MP / 2) * (a.NP / 2));
}
template <int NW>
int rad_plan_nw(RadArgs& a, int sms) {
    // dynamic shared memory available to one CTA: the device's opt-in
    // maximum less the kernel's static shared memory
    int dev = 0, optin = 0;
    cudaFuncAttributes fa{};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, k_rad_trace<NW>) != cudaSuccess)
        return GFM_E_CUDA;
    const size_t limit = (size_t)optin - fa.sharedSizeBytes;
    if (cudaFuncSetAttribute(k_rad_trace<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess)
        return GFM_E_CUDA;
    int base = 0;
    for (int d = 0; d < 3; ++d) {
        const int A = rad_slab_cells(a, d);
        a.fixed[d] = rad_smem_fixed(a, d, A);
        const size_t with = a.fixed[d] + rad_smem_slab(a, A);
        a.slab_in_smem[d] = with <= limit && !a.slab_global;
        a.fixed_in_smem[d] = a.fixed[d] <= limit && a.slab_global < 2;
        a.smem[d] = a.slab_in_smem[d] ? with : (a.fixed_in_smem[d] ? a.fixed[d] : 0);
        int occ = 0;
        // warps enough for a lane per column (row) and band, two sizes
        const int dims[3] = {a.MP, a.NP, a.LP}, lines = std::max(dims[rad_u(d)], dims[rad_v(d)]) / 2;
        a.threads[d] = lines <= 4 * (32 / a.NWL) ? 128 : kRadThreads;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_rad_trace<NW>, a.threads[d], a.smem[d]) != cudaSuccess)
            return GFM_E_CUDA;
        occ = occ < 1 ? 1 : (occ > 4 ? 4 : occ);
        a.grid[d] = sms * occ;
        a.part_base[d] = base;
        base += a.grid[d];
    }
    a.part_base[3] = base;
    return GFM_OK;
}

RadTab rad_tab(const RadArgs& a, int d, bool first, int lo) {
    const int dims[3] = {a.MP, a.NP, a.LP}, ax = first ? rad_u(d) : rad_v(d);
    const double* crd[3] = {a.g.X, a.g.Rr, a.g.Z};
    return RadTab{crd[d], crd[ax], dims[d], dims[ax], first, lo, (first ? a.tab_ku : a.tab_kv)[d],
                  (first ? a.tab_u : a.tab_v)[d], a.tab_kmax + 2 * d + !first};
}
// both tables of direction d for the emitter's slabs lo .. lo + tab_n[d] - 1
void rad_table_launch(const RadArgs& a, int d, int lo, cudaStream_t st) {
    for (int q = 0; q < 2; ++q) {
        const RadTab t = rad_tab(a, d, q == 0, lo);
        k_rad_table<<<std::min(a.tab_n[d], t.Dd / 2 - lo) * 2 * (t.P / 2), 32, 3 * (t.P + 2) * sizeof(double), st>>>(t);
    }
}

// Tables that hold all of a direction's emitters stay as they are; else they
// are filled again for each part of the emitters.
template <int NW>
void rad_trace_launch(const RadArgs& a, cudaStream_t const* st) {
    const int dims[3] = {a.MP, a.NP, a.LP};
    for (int d = 0; d < 3; ++d)
        for (int lo = 0; lo < dims[d] / 2; lo += a.tab_n[d]) {
            if (a.tab_n[d] < dims[d] / 2) rad_table_launch(a, d, lo, st[d]);
            k_rad_trace<NW><<<a.grid[d], a.threads[d], a.smem[d], st[d]>>>(a, d, lo, lo + a.tab_n[d]);
        }
}

}  // namespace

// The angle tables of all three directions, for as many of the emitter's slabs as
// `bytes` a direction allow (one at least, and one with slab_global = 2); called
// before rad_plan.  A grid whose tables fit (of a cube some 74 cells a side in
// kRadTabBytes) fills them once per handle, a larger one for each part of the
// emitters in every transfer (40x30x24 cells, in halves where memory is short: 613 ->
// 629 ms a transfer).
int rad_tables(RadArgs& a, cudaStream_t st, const RadMemory& m, long long bytes) {
    const int dims[3] = {a.MP, a.NP, a.LP};
    double* km = nullptr;
    for (int d = 0; d < 3; ++d) a.tab_n[d] = 0;
    if (int rc = m.alloc(m.ctx, &km, 3)) return rc;
    a.tab_kmax = reinterpret_cast<int*>(km);
    const int most = 3 * (std::max({a.MP, a.NP, a.LP}) + 2) * (int)sizeof(double);
    if (cudaMemsetAsync(a.tab_kmax, 0, 6 * sizeof(int), st) != cudaSuccess ||
        (most > 48 * 1024 && cudaFuncSetAttribute(k_rad_table, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess))
        return GFM_E_CUDA;
    // One direction after the other, with room for walks of 4 cells; where a walk is
    // longer (in the first direction of a plain box already), once more in the place
    // of the first.
    for (int d = 0; d < 3; ++d) {
        const int nd = dims[d] / 2, nu = dims[rad_u(d)] / 2, nv = dims[rad_v(d)] / 2;
        int need[6] = {};
        need[2 * d] = need[2 * d + 1] = 4;
        for (int pass = 0; pass < 2; ++pass) {
            if (pass) {
                if (need[2 * d] <= a.tab_ku[d] && need[2 * d + 1] <= a.tab_kv[d]) break;
                m.release(m.ctx, 2);
            }
            a.tab_ku[d] = std::max(need[2 * d], 4);
            a.tab_kv[d] = std::max(need[2 * d + 1], 4);
            const long long u = (long long)nd * nu * rad_rec(nu, a.tab_ku[d]), v = (long long)nd * nv * rad_rec(nv, a.tab_kv[d]);
            a.tab_bytes[d] = 8 * (u + v);
            a.tab_n[d] = a.slab_global > 1 ? 1 : (int)std::max(1LL, std::min((long long)nd, bytes / a.tab_bytes[d]));
            if (int rc = m.alloc(m.ctx, &a.tab_u[d], u * a.tab_n[d])) return rc;
            if (int rc = m.alloc(m.ctx, &a.tab_v[d], v * a.tab_n[d])) return rc;
            if (cudaStreamSynchronize(nullptr) != cudaSuccess) return GFM_E_CUDA;   // `alloc` clears on the default stream
            for (int lo = 0; lo < nd; lo += a.tab_n[d]) rad_table_launch(a, d, lo, st);
            if (cudaMemcpyAsync(need, a.tab_kmax, sizeof need, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess)
                return GFM_E_CUDA;
        }
    }
    return GFM_OK;
}

int rad_plan(RadArgs& a, int sms) {
    switch (a.NWL) {
        case 4: return rad_plan_nw<4>(a, sms);
        case 10: return rad_plan_nw<10>(a, sms);
        default: return rad_plan_nw<0>(a, sms);
    }
}

// st[0] is the caller's stream; the x-, y- and z-directions run on st[0..2],
// forked after the per-cell kernels (ev[0]) and joined before the sums
// (ev[1], ev[2]).
template <typename R>
int launch_rad_transfer(RadArgs a, R* T, long long nT, cudaStream_t const* st, cudaEvent_t const* ev) {
    const int n = a.MZ * a.NZ * a.LZ;
    const int gb = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
    k_rad_mark<<<gb, 256, 0, st[0]>>>(a);
    k_rad_akl<R><<<a.akl_blocks, 256, 0, st[0]>>>(a, T);
    k_rad_qe<<<a.akl_blocks, 256, 0, st[0]>>>(a);
    if (cudaEventRecord(ev[0], st[0]) != cudaSuccess || cudaStreamWaitEvent(st[1], ev[0], 0) != cudaSuccess ||
        cudaStreamWaitEvent(st[2], ev[0], 0) != cudaSuccess)
        return GFM_E_CUDA;
    switch (a.NWL) {
        case 4: rad_trace_launch<4>(a, st); break;
        case 10: rad_trace_launch<10>(a, st); break;
        default: rad_trace_launch<0>(a, st); break;
    }
    if (cudaEventRecord(ev[1], st[1]) != cudaSuccess || cudaEventRecord(ev[2], st[2]) != cudaSuccess ||
        cudaStreamWaitEvent(st[0], ev[1], 0) != cudaSuccess || cudaStreamWaitEvent(st[0], ev[2], 0) != cudaSuccess)
        return GFM_E_CUDA;
    k_rad_reduce<<<a.akl_blocks, 256, 0, st[0]>>>(a);
    launch_t_roundtrip<R>(T, nT, a.t0, st[0]);
    return cudaGetLastError() == cudaSuccess ? GFM_OK : GFM_E_CUDA;
}
template int launch_rad_transfer<double>(RadArgs, double*, long long, cudaStream_t const*, cudaEvent_t const*);
template int launch_rad_transfer<float>(RadArgs, float*, long long, cudaStream_t const*, cudaEvent_t const*);

}  // namespace gfm
