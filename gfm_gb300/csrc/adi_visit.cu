// adi_visit.cu -- the line solver ADLBL3 with one CTA per plane visit: ADLZ
// (Adlbl3.f90:103-141) of one x-plane, both passes L = 1, 2 with their
// averages, in shared memory and registers.  Two orders use it: red-black in
// FP64 (GFM_ADI_REDBLACK, k_pv_visit: the planes of a colour at once; FP32 has
// adi_plane.cu) and the reference's march in both precisions (GFM_ADI_MARCH,
// k_pv_march: one CTA per system walks the planes).
//
// Per ADLBL3 call (Adlbl3.f90:10-97) the system is rewritten once into
// plane-major arrays of nJ x nK points with a one-point border, point (jj, kk)
// of plane p at p*PB + (jj+1)*PS + kk+1, PS = (nK+2)|1 (odd, so that the
// z-lines' shared-memory accesses hit different banks), PB a multiple of 4:
//
//   XP  the unknown, planes -1 .. npl of the class (I = IB + 2p);
//   Q4 = (AS31, AS32, AS21, AS22), BS, AS11, AS12, AP (used while factoring),
//       and of both line directions AL and PT and what the right-hand sides take
//       (halved, see below): IA = 1/ALP in FP64, in the march also the rest of
//       1/ALP (adl_over), and ALP in FP32.
//
// Lines are factored from both ends.  The rows above the middle of a line keep
// the reference's elimination, ALP = AP - PT(prev) AS_sub, AL = AS_sub/ALP,
// PT = AS_next/ALP (ADLZY, ADLYZ, Adlbl3.f90:147-221); the rows below it run
// the same elimination from the other end with AS_sub and AS_next exchanged;
// the two rows that meet are a 2 x 2 system, DINV = 1/(1 - PT PT') kept per
// line (MID).  Solving a line then takes two chains of n/2 steps side by side
// instead of one of n.  A line with an open row whose diagonal does not dominate
// (adl_dominant) or whose pivot vanishes (|ALP| <= 1e-20, a row the reference
// copies), or with a singular middle, is factored from one end as the reference
// does (its split is n): its pivots and the rows it copies are the reference's.
// Rows copied unchanged (those, and blocked cells) store IA = -0.0, a value no
// other row stores, and AL = PT = 0.  The matrices do not change during the call,
// so all this is done once.
//
// A visit has three kinds of phases with a barrier after each:
//   point  every thread owns up to PPT points and keeps their coefficients in
//          registers for both passes: the right-hand sides
//          (BS + AS12 XT(I+2) + AS11 XT(I-2) + in-plane neighbours)/ALP of the
//          y-line and of the z-line, halved, go to VY and VZ in shared memory
//          (the halves make the average of the two results a plain sum; a
//          product by 1/2 is exact);
//   chain  two lanes per line, one from each end, y-lines and z-lines on warps
//          of their own: Q = AL Q(prev) + V, the middle, X = PT X(next) + Q,
//          in place;
//   sum    XT = VY + VZ by the points' owners; after pass L=2 straight to XP.
//
// Why this split.  A row costs one multiply-add per recurrence step and its
// loads; everything else of a row (right-hand sides, index arithmetic, record
// loads) is point-parallel over all the CTA's threads, and the records are
// fetched once per visit, before the dependency wait where they are known to
// be complete, with all of a thread's loads in flight.  The form before this
// one cut lines into 8-row segments joined by scans and loaded the records
// row by row in four passes of about 100 warp instructions per row; it was
// bound by instruction issue in FP32 and spent twice the FP64 operations (the
// segment products and corrections) on GB300's narrow FP64 pipe, where a warp
// instruction takes 64 cycles of its sub-partition whatever its active lanes.
// ms an iteration, before -> with this form: TC21 FP64 march 32.1 -> 8.5,
// red-black 2.55 -> 1.68; 48x24x16 FP64 red-black 2.75 -> 1.85; 192x96x64 FP64
// red-black 30.0 -> 25.7 (line solver 15.4 -> 11.3).  us a visit of the march,
// before -> with it: FP64 41 -> 9.1 at 22x16 points, 270 -> 55 at 96x64; FP32
// 18 -> 3.6 and 201 -> 21.  (Products by the reciprocals in place of the quotients
// took 8.8 and 49 us in FP64, 2.9 and 20 in FP32; their errors were 4 to 6% above
// the reference's.)
#include <algorithm>
#include <type_traits>

#include "state.cuh"

namespace gfm {

namespace {

template <typename R>
struct __align__(2 * sizeof(R)) Pair { R x, y; };

template <typename R>
struct PvBatch {
    Sys<R> sys[8];
    R* xp[8];
    Quad<R>* q4[8];
    R *bs[8], *a11[8], *a12[8], *bx[8], *ap[8];
    R *ia[8][2], *al[8][2], *pt[8][2], *lo[8][2];   // per line direction (0 y, 1 z); lo: what IA misses, the FP64 march's
    // (DINV, split) of line l of plane p at p*(nK + nJ) + l, the y-lines (by K)
    // before the z-lines (by J)
    Pair<R>* mid[8];
    int nsys;
};

struct PlaneDims {
    int npl, nJ, nK, PS, PB, pts;
};
template <typename R>
__host__ __device__ __forceinline__ PlaneDims dims_of(const Sys<R>& s) {
    PlaneDims d;
    d.npl = (s.ie - s.ib) / 2 + 1;
    d.nJ = (s.je - s.jb) / 2 + 1;
    d.nK = (s.ke - s.kb) / 2 + 1;
    d.PS = (d.nK + 2) | 1;
    d.PB = ((d.nJ + 2) * d.PS + 3) & ~3;
    d.pts = d.nJ * d.nK;
    return d;
}
__host__ __device__ __forceinline__ int point(const PlaneDims& d, int jj, int kk) { return (jj + 1) * d.PS + kk + 1; }
__host__ __device__ __forceinline__ int xp_index(const PlaneDims& d, int p, int jj, int kk) {
    return (p + 1) * d.PB + point(d, jj, kk);
}
// ---------------------------------------------------------------------------
// XT <-> XP, through a 32 x 32 tile in shared memory: plane index fastest on
// the class side, K fastest on the plane side.  Block (32, 8); bx over
// (plane tiles) x (K tiles), jr = J row of XP (border included), e = system.
// ---------------------------------------------------------------------------
template <typename R, bool IN>
__device__ __forceinline__ void pv_copy_planes(const GeoT<R>& g, const PvBatch<R>& b, int bx, int jr, int e, R (*tile)[33]) {
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    // IN copies the border too (planes -1..npl, rows -1..nJ, -1..nK); OUT the interior
    const int o = IN ? 1 : 0;
    const int np = d.npl + 2 * o, nj = d.nJ + 2 * o, nk = d.nK + 2 * o;
    if (jr >= nj) return;
    const int ntp = (np + 31) / 32;
    const int p0 = (bx % ntp) * 32, k0 = (bx / ntp) * 32;
    if (k0 >= nk) return;
    const int J = s.jb + 2 * (jr - o);
    R* __restrict__ xp = b.xp[e];
    const int tx = threadIdx.x, ty = threadIdx.y;
    if (IN) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int kr = k0 + ty + 8 * r, pr = p0 + tx;
            if (kr < nk && pr < np)
                tile[ty + 8 * r][tx] = s.xt[pidx(g, s.ib + 2 * (pr - o), J, s.kb + 2 * (kr - o))];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int pr = p0 + ty + 8 * r, kr = k0 + tx;
            if (kr < nk && pr < np) xp[xp_index(d, pr - o, jr - o, kr - o)] = tile[tx][ty + 8 * r];
        }
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int pr = p0 + ty + 8 * r, kr = k0 + tx;
            if (kr < nk && pr < np) tile[tx][ty + 8 * r] = xp[xp_index(d, pr, jr, kr)];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int kr = k0 + ty + 8 * r, pr = p0 + tx;
            if (kr < nk && pr < np) s.xt[pidx(g, s.ib + 2 * pr, J, s.kb + 2 * kr)] = tile[ty + 8 * r][tx];
        }
    }
}
template <typename R>
__global__ void k_pv_copy_out(GeoT<R> g, PvBatch<R> b) {
    __shared__ R tile[32][33];
    pdl_wait();
    pdl_trigger();
    pv_copy_planes<R, false>(g, b, blockIdx.x, blockIdx.y, blockIdx.z, tile);
}

// AP of a blocked cell in the plane-major copy: a NaN of its own bits
template <typename R>
__device__ __forceinline__ R blocked_mark();
template <>
__device__ __forceinline__ float blocked_mark<float>() { return __uint_as_float(0x7fc0b10cu); }
template <>
__device__ __forceinline__ double blocked_mark<double>() { return __longlong_as_double(0x7ff8b10cb10cb10cll); }
__device__ __forceinline__ bool is_blocked(float ap) { return __float_as_uint(ap) == 0x7fc0b10cu; }
__device__ __forceinline__ bool is_blocked(double ap) { return __double_as_longlong(ap) == 0x7ff8b10cb10cb10cll; }

// ---------------------------------------------------------------------------
// The point records, once per call, through a 32-plane x 16-point tile in
// shared memory: read with the plane index fastest (contiguous in the class
// arrays), written with K fastest.  Block (32, 8); nf blocks of a row over (plane
// tiles) x (K tiles), rows J, z = system; after `rows` rows of them nc blocks of a
// row of the planes, XT -> XP.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(256) k_pv_fill(GeoT<R> g, PvBatch<R> b, int nf, int rows, int nc) {
    __shared__ R tile[8][16][33];
    pdl_wait();
    pdl_trigger();
    const int e = blockIdx.z;
    if ((int)blockIdx.x >= nf * rows) {
        const int id = (int)blockIdx.x - nf * rows;
        pv_copy_planes<R, true>(g, b, id % nc, id / nc, e, tile[0]);   // 32 x 33 of the 128 rows
        return;
    }
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    const int row = (int)blockIdx.x / nf, bx = (int)blockIdx.x - row * nf;
    if (row >= d.nJ) return;
    const int ntp = (d.npl + 31) / 32;
    const int p0 = (bx % ntp) * 32, l0 = (bx / ntp) * 16;
    if (l0 >= d.nK) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const R* const src[7] = {s.as[4], s.as[5], s.as[2], s.as[3], s.bs, s.as[0], s.as[1]};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int ll = ty + 8 * r, p = p0 + tx, l = l0 + ll;
        if (p < d.npl && l < d.nK) {
            const int o = (int)pidx(g, s.ib + 2 * p, s.jb + 2 * row, s.kb + 2 * l);
#pragma unroll
            for (int f = 0; f < 7; ++f) tile[f][ll][tx] = src[f][o];
            tile[7][ll][tx] = g.ib[o] >= 1 ? blocked_mark<R>() : s.ap[o];
        }
    }
    __syncthreads();
    const int tid = ty * 32 + tx;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int idx = tid + 256 * r;
        const int ll = idx & 15, pl = idx >> 4;
        const int p = p0 + pl, l = l0 + ll;
        if (p < d.npl && l < d.nK) {
            const int q = p * d.PB + point(d, row, l);
            b.q4[e][q] = Quad<R>{tile[0][ll][pl], tile[1][ll][pl], tile[2][ll][pl], tile[3][ll][pl]};
            b.bs[e][q] = tile[4][ll][pl];
            b.a11[e][q] = tile[5][ll][pl];
            b.a12[e][q] = tile[6][ll][pl];
            b.ap[e][q] = tile[7][ll][pl];
        }
    }
}

// ---------------------------------------------------------------------------
// The factors of every line, once per call, one CTA per plane: two lanes per
// line, one from each end, 32 lines to a pair of warps.  The y-lines read their
// rows from the plane-major arrays (lanes along K, contiguous) with the rows of
// the next batch in flight; the z-lines, whose lanes are PS apart, work on a
// copy in shared memory, where each row's factors replace its coefficients, and
// leave contiguously.  The chain of a row is one division (PT; 1/ALP and AL are
// off it); a plane's two directions run side by side.
// ---------------------------------------------------------------------------
constexpr int kFactThreads = 384;
template <typename R, bool MARCH>
__global__ void __launch_bounds__(kFactThreads) k_pv_factor(PvBatch<R> b) {
    extern __shared__ __align__(16) unsigned char pv_smem[];
    constexpr int C = 4;
    const int e = blockIdx.y, p = blockIdx.x;
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    pdl_wait();
    pdl_trigger();
    if (p >= d.npl) return;
    const int PS = d.PS, PB = d.PB, nK = d.nK, nJ = d.nJ;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long rb = (long long)p * PB;
    const R* __restrict__ ap = b.ap[e] + rb;
    const Pair<R>* __restrict__ c2 = reinterpret_cast<const Pair<R>*>(b.q4[e] + rb);   // [2o] (AS31, AS32), [2o+1] (AS21, AS22)
    R* sap = reinterpret_cast<R*>(pv_smem);   // AP, AS31, AS32; then IA, AL, PT of the z-lines
    R* end_pt = sap + 3 * PB;                  // PT of each half-line's last row: [half][line]
    int* end_bad = reinterpret_cast<int*>(end_pt + 2 * (nJ + nK));
    for (int o = tid; o < PB; o += kFactThreads) {
        const Pair<R> c = c2[2 * o];
        sap[o] = ap[o];
        sap[o + PB] = c.x;
        sap[o + 2 * PB] = c.y;
    }
    __syncthreads();
    const R h = s.kb >= s.ke ? R(1) : R(0.5), h1 = s.kb >= s.ke ? R(1) : R(2);
    // what the right-hand sides take
    auto by = [&](R alp, R ia) { return sizeof(R) == 8 ? ia * h : (adl_copy(ia) ? ia : alp * h1); };
    constexpr bool LO = MARCH && sizeof(R) == 8;
    const int gy = (nK + 31) >> 5, gz = (nJ + 31) >> 5;
#pragma unroll 1
    for (int w = warp; w < 2 * (gy + gz); w += kFactThreads / 32) {
        const int grp = w >> 1, zl = grp >= gy, back = w & 1;
        const int l = (zl ? grp - gy : grp) * 32 + lane, n = zl ? nK : nJ;
        if (l >= (zl ? nJ : nK)) continue;
        const int cnt = back ? n / 2 : n - n / 2, vs = zl ? 1 : PS, st = back ? -vs : vs;
        int o = (zl ? point(d, l, -1) : point(d, -1, l)) + (back ? n : 1) * vs;
        R ptp = R(0);
        bool bad = false;
        if (zl) {
            for (int r = 0; r < cnt; ++r, o += st) {
                const R a = sap[o], lo = sap[o + PB], hi = sap[o + 2 * PB];
                R alp, ia, al, pt;
                bad |= !adl_pivot(a, back ? hi : lo, back ? lo : hi, ptp, is_blocked(a), alp, ia, al, pt);
                if (LO) b.lo[e][1][rb + o] = h * adl_low(alp, ia);
                sap[o] = by(alp, ia);
                sap[o + PB] = al;
                sap[o + 2 * PB] = pt;
            }
        } else {
            R a[C];
            Pair<R> c[C];
#pragma unroll
            for (int q = 0; q < C; ++q)
                if (q < cnt) { a[q] = ap[o + q * st]; c[q] = c2[2 * (o + q * st) + 1]; }
            for (int r = 0; r < cnt; r += C, o += C * st) {
                R an[C];
                Pair<R> cn[C];
#pragma unroll
                for (int q = 0; q < C; ++q)
                    if (r + C + q < cnt) { an[q] = ap[o + (C + q) * st]; cn[q] = c2[2 * (o + (C + q) * st) + 1]; }
#pragma unroll
                for (int q = 0; q < C; ++q)
                    if (r + q < cnt) {
                        R alp, ia, al, pt;
                        bad |= !adl_pivot(a[q], back ? c[q].y : c[q].x, back ? c[q].x : c[q].y, ptp, is_blocked(a[q]), alp, ia, al, pt);
                        const long long g = rb + o + q * st;
                        if (LO) b.lo[e][0][g] = h * adl_low(alp, ia);
                        b.ia[e][0][g] = by(alp, ia);
                        b.al[e][0][g] = al;
                        b.pt[e][0][g] = pt;
                    }
#pragma unroll
                for (int q = 0; q < C; ++q) { a[q] = an[q]; c[q] = cn[q]; }
            }
        }
        end_pt[2 * (zl ? nK + l : l) + back] = ptp;
        end_bad[2 * (zl ? nK + l : l) + back] = bad;
    }
    __syncthreads();
    for (int o = tid; o < PB; o += kFactThreads) {
        b.ia[e][1][rb + o] = sap[o];
        b.al[e][1][rb + o] = sap[o + PB];
        b.pt[e][1][rb + o] = sap[o + 2 * PB];
    }
    __syncthreads();
    for (int l = tid; l < nK + nJ; l += kFactThreads) {
        const int zl = l >= nK, n = zl ? nK : nJ, vs = zl ? 1 : PS;
        const R den = fma(-end_pt[2 * l + 1], end_pt[2 * l], R(1));   // of the chains' PT
        Pair<R> m{R(1) / den, R(n - n / 2)};
        if (end_bad[2 * l] || end_bad[2 * l + 1] || !(fabs(den) > R(1.0e-20))) {
            // from one end, as the reference
            int o = zl ? point(d, l - nK, 0) : point(d, 0, l);
            R ptp = R(0);
            for (int r = 0; r < n; ++r, o += vs) {
                const Pair<R> c = c2[2 * o + (zl ? 0 : 1)];
                R alp, ia, al, pt;
                adl_pivot(ap[o], c.x, c.y, ptp, is_blocked(ap[o]), alp, ia, al, pt);
                if (LO) b.lo[e][zl][rb + o] = h * adl_low(alp, ia);
                b.ia[e][zl][rb + o] = by(alp, ia);
                b.al[e][zl][rb + o] = al;
                b.pt[e][zl][rb + o] = pt;
            }
            m = Pair<R>{R(1), R(n)};
        }
        b.mid[e][(long long)p * (nK + nJ) + l] = m;
    }
}
template <typename R>
size_t pv_factor_smem(const PlaneDims& d) {
    return (size_t)(3 * d.PB + 2 * (d.nJ + d.nK)) * sizeof(R) + (size_t)2 * (d.nJ + d.nK) * sizeof(int);
}

// ---------------------------------------------------------------------------
// One plane visit
// ---------------------------------------------------------------------------
// Barrier of two warps.  Not the aligned form (bar.sync): it follows loops whose trip
// counts differ by lane, and where the compiler reconverges the warp is its own choice.
__device__ __forceinline__ void pair_sync(int id) { asm volatile("barrier.sync %0, 64;" ::"r"(id) : "memory"); }

// The recurrences of half a line in place, by one lane: rows o, o + st, .. (cnt
// of them, from an end of the line to its middle), QT before the first row
// `bnd`.  Another warp takes the other halves of the same lines; the two meet
// at the named barrier `bar`, with QT of their last rows at v[mine] and
// v[theirs] (border points of the line, free in VY and VZ) and PT of the other
// half's last row at pt[o + cnt*st].  (Both halves in one warp would need no
// barrier, but their rows fall on the same banks: 52 against 30 cycles a step
// with two such warps on a sub-partition, measured.)  The loads of B rows are
// issued together ahead of the chain; PRE: AL and PT of the next B rows before
// the chain of the current ones (records in global memory).  `one`: the line
// is factored from one end, and `far` is the XT after its last row.
template <typename R, bool PRE, int B>
__device__ __forceinline__ void pv_chain(R* v, const R* al, const R* pt, int o, int st, int cnt, R bnd, R dinv,
                                          bool live, int mine, int theirs, int bar, bool one, R far) {
    R q = bnd;
    int r = 0;
    R a[B];
    if (PRE) {
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (c < cnt) a[c] = al[o + c * st];
    }
#pragma unroll 1
    for (; r + B <= cnt; r += B, o += B * st) {
        R u[B], an[B];
#pragma unroll
        for (int c = 0; c < B; ++c) {
            u[c] = v[o + c * st];
            if (!PRE) a[c] = al[o + c * st];
            else if (r + B + c < cnt) an[c] = al[o + (B + c) * st];
        }
#pragma unroll
        for (int c = 0; c < B; ++c) {
            q = fma(a[c], q, u[c]);
            v[o + c * st] = q;
        }
        if (PRE) {
#pragma unroll
            for (int c = 0; c < B; ++c) a[c] = an[c];
        }
    }
    {
        R u[B];
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (r + c < cnt) {
                u[c] = v[o + c * st];
                if (!PRE) a[c] = al[o + c * st];
            }
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (r + c < cnt) {
                q = fma(a[c], q, u[c]);
                v[o + c * st] = q;
            }
    }
    o += (cnt - r - 1) * st;   // the last row of this half
    // the middle: the other half's last row is the start of this half's back
    // substitution, X = (PT' Q + Q') DINV
    if (live) v[mine] = q;
    pair_sync(bar);
    R x = far;
    if (!one) x = fma(pt[o + st], q, v[theirs]) * dinv;
    r = cnt;
    if (PRE) {
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (c < cnt) a[c] = pt[o - c * st];
    }
#pragma unroll 1
    for (; r >= B; r -= B, o -= B * st) {
        R u[B], an[B];
#pragma unroll
        for (int c = 0; c < B; ++c) {
            u[c] = v[o - c * st];
            if (!PRE) a[c] = pt[o - c * st];
            else if (r - B - c > 0) an[c] = pt[o - (B + c) * st];
        }
#pragma unroll
        for (int c = 0; c < B; ++c) {
            x = fma(a[c], x, u[c]);
            v[o - c * st] = x;
        }
        if (PRE) {
#pragma unroll
            for (int c = 0; c < B; ++c) a[c] = an[c];
        }
    }
    R u[B];
#pragma unroll
    for (int c = 0; c < B; ++c)
        if (r - c > 0) {
            u[c] = v[o - c * st];
            if (!PRE) a[c] = pt[o - c * st];
        }
#pragma unroll
    for (int c = 0; c < B; ++c)
        if (r - c > 0) {
            x = fma(a[c], x, u[c]);
            v[o - c * st] = x;
        }
}

// x/2 (or x): in FP64 on the integer pipe, a step of the exponent, where that is exact
__device__ __forceinline__ float scaled(float x, bool whole) { return whole ? x : 0.5f * x; }
__device__ __forceinline__ double scaled(double x, bool whole) {
    if (whole) return x;
    const int hi = __double2hiint(x), ex = hi & 0x7ff00000;
    if (ex > 0x00100000 && ex < 0x7ff00000) return __hiloint2double(hi - 0x00100000, __double2loint(x));
    return 0.5 * x;
}

// The compiler gathers the loads of all of a thread's points first; past four
// points that costs more registers than there are (spills, which with this much
// shared memory miss the L1).
__device__ __forceinline__ void keep_order() { asm volatile("" ::: "memory"); }

// Plane p of system e.  PPT > 0: each thread holds up to PPT points' records
// in registers and the chains' records are staged in shared memory, its arrays
// CAP elements apart (a constant, so a chain's loads share one address
// register); PPT == 0: any plane whose XT, VY and VZ fit, the records read
// again in each pass.  wait_first: the records are not known to be complete
// before the dependency wait.
// MARCH: right-hand sides are quotients by ALP, rounded once, as the reference's
// are; in red-black they are products by IA, as in the segmented passes.
template <typename R, bool MARCH, int NT, int PPT, int CAP>
__device__ __forceinline__ void pv_visit(const PvBatch<R>& b, int e, const PlaneDims& d, int p, bool one_row, R* sm,
                                          bool pdl, bool wait_first) {
    constexpr bool REG = PPT > 0;
    constexpr int NP = REG ? PPT : 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int PS = d.PS, PB = d.PB, nK = d.nK, nJ = d.nJ;
    R* xs = sm;
    const int SP = REG ? CAP : PB;   // spacing: XT, VY, VZ; REG: ALY, ALZ, PTY, PTZ, BX too
    R* vy = xs + SP;
    R* rec = xs + 3 * SP;
    R* bxs = xs + 7 * SP;
    const long long rb = (long long)p * PB;
    const Quad<R>* __restrict__ q4 = b.q4[e] + rb;
    const R* __restrict__ iay_g = b.ia[e][0] + rb;
    const R* __restrict__ iaz_g = b.ia[e][1] + rb;
    // (the march reads nothing before its wait)
    auto early = [](const auto* q) {
        if constexpr (MARCH) return *q;
        else return load_l2(q);
    };
    constexpr bool LO = MARCH && sizeof(R) == 8;
    const R* __restrict__ loy_g = b.lo[e][0] + (LO ? rb : 0);
    const R* __restrict__ loz_g = b.lo[e][1] + (LO ? rb : 0);
    R* __restrict__ xp = b.xp[e] + rb + PB;
    const R h = one_row ? R(1) : R(0.5);
    // points t = tid, tid + NT, ..: (jj, kk) advance by (dj, dk)
    const int dj = NT / nK, dk = NT - dj * nK;
    const int np = (d.pts - tid + NT - 1) / NT;   // points of this thread
    int kk = tid % nK;
    int o = point(d, tid / nK, kk);
    auto step = [&](int& oo, int& k) {
        oo += dj * PS + dk;
        k += dk;
        if (k >= nK) { k -= nK; oo += PS - nK; }
    };
    if (pdl && wait_first) { pdl_wait(); pdl_trigger(); }
    unsigned offs[(NP + 1) / 2];   // the points' offsets, two to a register
    auto off = [&](int i) { return (int)((i & 1) ? offs[i / 2] >> 16 : offs[i / 2] & 0xffffu); };
    Quad<R> A[NP];
    R iy[NP], iz[NP], ly[LO ? NP : 1], lz[LO ? NP : 1];
    constexpr int NE = NP <= 4 ? NP : 1;   // with few points the x-neighbours' records come early too
    R eb[NE], e1[NE], e2[NE];
    if (REG) {
        int oo = o, k = kk;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            if (i & 1) offs[i / 2] |= (unsigned)oo << 16;
            else offs[i / 2] = (unsigned)oo;
            if (i < np) {
                A[i] = early(q4 + oo);
                iy[i] = early(iay_g + oo);
                iz[i] = early(iaz_g + oo);
                if (LO) { ly[i % (LO ? NP : 1)] = early(loy_g + oo); lz[i % (LO ? NP : 1)] = early(loz_g + oo); }
                if (NP <= 4) {
                    eb[i % NE] = early(b.bs[e] + rb + oo);
                    e1[i % NE] = early(b.a11[e] + rb + oo);
                    e2[i % NE] = early(b.a12[e] + rb + oo);
                }
            }
            step(oo, k);
        }
        const Pair<R>* __restrict__ mid = b.mid[e] + (long long)p * (nK + nJ);
        // DINV and the split of a line in the AL and PT arrays' border point before it
        for (int l = tid; l < nK + nJ; l += NT) {
            const int zl = l >= nK;
            R* q = rec + zl * SP + (zl ? point(d, l - nK, -1) : point(d, -1, l));
            const Pair<R> m = early(mid + l);
            q[0] = m.x;
            q[2 * SP] = m.y;
        }
        // the chains' AL and PT
        const R* __restrict__ aly = b.al[e][0] + rb;
        const R* __restrict__ alz = b.al[e][1] + rb;
        const R* __restrict__ pty = b.pt[e][0] + rb;
        const R* __restrict__ ptz = b.pt[e][1] + rb;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            if (i < np) {
                const int oi = off(i);
                R* q = rec + oi;
                q[0] = early(aly + oi);
                q[SP] = early(alz + oi);
                q[2 * SP] = early(pty + oi);
                q[3 * SP] = early(ptz + oi);
            }
            if (i % 4 == 3) keep_order();
        }
    }
    if (pdl && !wait_first) {
        if (tid == 0 && NP > 4) {
            l2_prefetch(b.bs[e] + rb, PB * sizeof(R));
            l2_prefetch(b.a11[e] + rb, PB * sizeof(R));
            l2_prefetch(b.a12[e] + rb, PB * sizeof(R));
        }
        pdl_wait();
        pdl_trigger();
    }
    // XT with its border, and BX = BS + AS12 XT(I+2) + AS11 XT(I-2), fixed for the visit
    {
        const R* __restrict__ bs = b.bs[e] + rb;
        const R* __restrict__ a11 = b.a11[e] + rb;
        const R* __restrict__ a12 = b.a12[e] + rb;
        auto bxof = [&](int q) { return fma(a11[q], xp[q - PB], fma(a12[q], xp[q + PB], bs[q])); };
        if (NP <= 4 && REG) {
            // the neighbours' and the plane's loads all in flight together
            R xm[NE], xq[NE];
#pragma unroll
            for (int i = 0; i < NE; ++i)
                if (i < np) {
                    xm[i] = xp[off(i) - PB];
                    xq[i] = xp[off(i) + PB];
                }
            constexpr int NX = 6;
            static_assert(NP > 4 || CAP <= NX * NT, "the plane's loads");
            R xo[NX];
#pragma unroll
            for (int i = 0; i < NX; ++i)
                if (tid + i * NT < PB) xo[i] = xp[tid + i * NT];
#pragma unroll
            for (int i = 0; i < NX; ++i)
                if (tid + i * NT < PB) xs[tid + i * NT] = xo[i];
#pragma unroll
            for (int i = 0; i < NE; ++i)
                if (i < np) bxs[off(i)] = fma(e1[i], xm[i], fma(e2[i], xq[i], eb[i]));
        } else {
            for (int t = tid; t < PB; t += NT) xs[t] = xp[t];
        }
        if (REG) {
            if (NP > 4) {
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    if (i < np) bxs[off(i)] = bxof(off(i));
                    if (i % 4 == 3) keep_order();
                }
            }
        } else {
            R* bxg = b.bx[e] + rb;
            int oo = o, k = kk;
#pragma unroll 4
            for (int i = 0; i < np; ++i) {
                bxg[oo] = bxof(oo);
                step(oo, k);
            }
        }
    }
    __syncthreads();
    const int gy = (nK + 31) >> 5, gz = one_row ? 0 : (nJ + 31) >> 5;   // 32 lines to a pair of warps
#pragma unroll 1
    for (int L = 1; L <= 2; ++L) {
        // (keeps the points' addresses from being hoisted out of the loop into
        // registers of their own)
        if (REG) {
#pragma unroll
            for (int i = 0; i < (NP + 1) / 2; ++i) asm volatile("" : "+r"(offs[i]));
        }
        // right-hand sides of both directions
        auto over = [](R v, R ia, R low) { return MARCH ? adl_over(v, ia, ia, low) : ia * v; };   // (FP32: ALP in IA's place)
        auto rhs = [&](int q, const Quad<R>& a, R ia_y, R ia_z, R lo_y, R lo_z, R bx) {
            R y = over(fma(a.x, xs[q - 1], fma(a.y, xs[q + 1], bx)), ia_y, lo_y);
            R z = over(fma(a.z, xs[q - PS], fma(a.w, xs[q + PS], bx)), ia_z, lo_z);
            const bool cy = adl_copy(ia_y), cz = adl_copy(ia_z);
            if (cy || cz) {
                const R hx = scaled(xs[q], one_row);
                if (cy) y = hx;
                if (cz) z = hx;
            }
            vy[q] = y;
            vy[q + SP] = z;
        };
        if (REG) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if (i < np) rhs(off(i), A[i], iy[i], iz[i], LO ? ly[i % (LO ? NP : 1)] : R(0), LO ? lz[i % (LO ? NP : 1)] : R(0), bxs[off(i)]);
                if (i % 4 == 3) keep_order();
            }
        } else {
            const R* bxg = b.bx[e] + rb;
            int oo = o, k = kk;
#pragma unroll(LO ? 2 : 4)
            for (int i = 0; i < np; ++i) {
                rhs(oo, q4[oo], iay_g[oo], iaz_g[oo], LO ? loy_g[oo] : R(0), LO ? loz_g[oo] : R(0), bxg[oo]);
                step(oo, k);
            }
        }
        __syncthreads();
        // the lines, 32 to a pair of warps: the y-lines' pairs, then the
        // z-lines'; the even warp from the lines' first ends, the odd one from the last
#pragma unroll 1
        for (int w = warp; w < 2 * (gy + gz); w += NT / 32) {
            const int grp = w >> 1, zl = grp >= gy;
            const bool back = w & 1;
            const int l0 = (zl ? grp - gy : grp) * 32 + lane, nl = zl ? nJ : nK;
            const bool live = l0 < nl;
            const int l = live ? l0 : nl - 1;   // (a lane past the last line takes no steps and stores nothing)
            const int n = zl ? nK : nJ, vs = zl ? 1 : PS;
            const int ob = zl ? point(d, l, -1) : point(d, -1, l);   // the border point before the line
            R* const v = vy + zl * SP + ob;
            const R* const al = REG ? v + 2 * SP : b.al[e][zl] + rb + ob;
            const R* const pt = REG ? v + 4 * SP : b.pt[e][zl] + rb + ob;
            const Pair<R> mid = REG ? Pair<R>{al[0], pt[0]} : b.mid[e][(long long)p * (nK + nJ) + (zl ? nK + l : l)];
            const int m = (int)mid.y;
            const R far = h * xs[ob + (n + 1) * vs];
            pv_chain<R, !REG, (PPT <= 4 ? 8 : 4)>(v, al, pt, (back ? n : 1) * vs, back ? -vs : vs, !live ? 0 : back ? n - m : m,
                                                  back ? far : h * xs[ob], mid.x, live, back ? (n + 1) * vs : 0,
                                                  back ? 0 : (n + 1) * vs, 1 + (warp >> 1), m == n, far);
        }
        __syncthreads();
        // XT = (XT2 + XT3)/2; a plane with one z-row (KB >= KE) takes the
        // y-line pass alone and is done after it (Adlbl3.f90:124-130)
        const bool last = L == 2 || one_row;
        auto put = [&](int q) {
            const R x = one_row ? vy[q] : vy[q] + vy[q + SP];
            if (last) xp[q] = x;
            else xs[q] = x;
        };
        if (REG) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if (i < np) put(off(i));
                if (i % 4 == 3) keep_order();
            }
        } else {
            int oo = o, k = kk;
#pragma unroll 4
            for (int i = 0; i < np; ++i) {
                put(oo);
                step(oo, k);
            }
        }
        if (last) return;
        __syncthreads();
    }
}

// One colour visit: every plane p = colour, colour + 2, .. of the call's
// planes (I = IB + 2p), one CTA each.  The records were written two launches
// ago or earlier except for the call's first visit (`first`), so the others read
// them before their pdl_wait (device.cuh).
// `ahead` > 0: the batch's records do not stay in L2 from one visit to the
// next, and the block asks L2 for those of the block `ahead` places on (the one
// that follows on its SM), into the next colour's visit past the last block, so
// that the DRAM reads run during the chains, which leave the memory idle.
template <typename R, int NT, int PPT, int CAP>
__global__ void __launch_bounds__(NT, 1) k_pv_visit(PvBatch<R> b, int colour, int sweep, int first, int ahead) {
    extern __shared__ __align__(16) unsigned char pv_smem[];
    const int e = blockIdx.y;
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    if (ahead && !first && threadIdx.x == 0) {
        int t = (int)(blockIdx.y * gridDim.x + blockIdx.x) + ahead;
        const int all = (int)(gridDim.x * gridDim.y), nc = t >= all ? 1 - colour : colour;
        if (t >= all) t -= all;
        const int e2 = t / (int)gridDim.x, p2 = nc + 2 * (t - e2 * (int)gridDim.x);
        if (e2 < b.nsys && sweep < b.sys[e2].nim) {
            const PlaneDims d2 = dims_of(b.sys[e2]);
            if (p2 < d2.npl) {
                const long long rb = (long long)p2 * d2.PB;
                const size_t bytes = d2.PB * sizeof(R);
                l2_prefetch(b.q4[e2] + rb, 4 * bytes);
                l2_prefetch(b.bs[e2] + rb, bytes);
                l2_prefetch(b.a11[e2] + rb, bytes);
                l2_prefetch(b.a12[e2] + rb, bytes);
                for (int zl = 0; zl < 2; ++zl) {
                    l2_prefetch(b.ia[e2][zl] + rb, bytes);
                    l2_prefetch(b.al[e2][zl] + rb, bytes);
                    l2_prefetch(b.pt[e2][zl] + rb, bytes);
                }
            }
        }
    }
    if (sweep >= s.nim || (int)blockIdx.x >= (d.npl - colour + 1) / 2) {
        pdl_wait();   // nothing to do, but this launch must not end before the one it follows
        return;
    }
    pv_visit<R, false, NT, PPT, CAP>(b, e, d, colour + 2 * (int)blockIdx.x, s.kb >= s.ke, reinterpret_cast<R*>(pv_smem), true, first != 0);
}

// The reference's plane order: planes IB..IE, then IE..IB, NIM times, one CTA
// per system (each plane reads the one before it, so the walk is sequential).
template <typename R, int NT, int PPT, int CAP>
__global__ void __launch_bounds__(NT, 1) k_pv_march(PvBatch<R> b) {
    extern __shared__ __align__(16) unsigned char pv_smem[];
    const int e = blockIdx.x;
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    R* sm = reinterpret_cast<R*>(pv_smem);
    pdl_wait();
    pdl_trigger();
    for (int v = 0; v < 2 * s.nim * d.npl; ++v) {
        const int r = v % (2 * d.npl);
        const int p = r < d.npl ? r : 2 * d.npl - 1 - r;
        pv_visit<R, true, NT, PPT, CAP>(b, e, d, p, s.kb >= s.ke, sm, false, false);
        __syncthreads();   // the plane's XT is in XP, and the scratch is free
    }
}

constexpr size_t kPvMaxSmem = 227 * 1024;
constexpr size_t kPvL2Bytes = 100u << 20;   // of the 129 MB of L2
constexpr int kPvSlots = 152;               // CTAs in flight: one per SM for planes whose records exceed L2

// The forms of a visit's CTA: threads, points a thread in registers (0: read
// in each pass), shared-memory elements per array.  A batch takes the first
// form that holds its largest plane.  CAP leaves a plane of that many points
// room for its border at ordinary aspect ratios; 7264 x 8 arrays of floats are
// the 227 KB of a CTA.  Points in registers against records read in each pass, us a
// visit of the march in FP32: 44x44 points 6.5 and 10.2, 60x60 11.1 and 16.1, 80x75
// 21.9 and 23.9.  FP64 has one form for the planes of more than 1024 points in both
// orders: 512 threads leave a thread 128 registers, of the 190 (red-black) and 250
// (march) that four points take (44x44 points: 23.2 and 23.7 us reading, 18.1 and
// 26.1 with the points in registers).
template <int NT_, int PPT_, int CAP_>
struct PvForm {
    static constexpr int NT = NT_, PPT = PPT_, CAP = CAP_;
};
// f(form) of every form of the precision in turn until one returns true
template <typename R, typename F>
bool pv_forms(F&& f) {
    if (f(PvForm<128, 4, 704>{}) || f(PvForm<256, 4, 1344>{})) return true;
    if constexpr (sizeof(R) == 8) return f(PvForm<512, 0, 0>{});
    else return f(PvForm<512, 4, 2560>{}) || f(PvForm<512, 8, 4864>{}) || f(PvForm<512, 12, 7264>{}) || f(PvForm<512, 0, 0>{});
}
// whether every plane of the batch fits a form, and its shared memory
template <typename R, typename Form>
bool pv_fits(const Sys<R>* sys, int nsys, size_t& smem) {
    int pts = 0, pb = 0;
    for (int e = 0; e < nsys; ++e) {
        const PlaneDims d = dims_of(sys[e]);
        pts = std::max(pts, d.pts);
        pb = std::max(pb, d.PB);
        if (pv_factor_smem<R>(d) > kPvMaxSmem) return false;
    }
    smem = (size_t)(Form::PPT ? 8 * Form::CAP : 3 * pb) * sizeof(R);
    return smem <= kPvMaxSmem && (Form::PPT == 0 || (pts <= Form::NT * Form::PPT && pb <= Form::CAP));
}

// batch arrays and the call's set-up launches
template <typename R, bool MARCH>
int pv_setup(const GeoT<R>& g, const Sys<R>* sys, const AdiScratch<R>* scr, int nsys, bool pdl, cudaStream_t st,
              PvBatch<R>& b, int& max_np, int& nim, dim3& out_grid) {
    b.nsys = nsys;
    max_np = nim = 0;
    int max_nj = 0, max_nk = 0;
    size_t fsmem = 0;
    const long long NH = 2LL * g.CBH;   // elements of one scratch array, more than (npl + 2) PB
    for (int e = 0; e < nsys; ++e) {
        const PlaneDims d = dims_of(sys[e]);
        b.sys[e] = sys[e];
        b.xp[e] = scr[e].xs;
        b.q4[e] = scr[e].ya;
        R* f[12];
        for (int q = 0; q < 4; ++q) {
            f[q] = reinterpret_cast<R*>(scr[e].yb) + q * NH;
            f[4 + q] = reinterpret_cast<R*>(scr[e].za) + q * NH;
            f[8 + q] = reinterpret_cast<R*>(scr[e].zb) + q * NH;
        }
        b.bs[e] = f[0]; b.a11[e] = f[1]; b.a12[e] = f[2]; b.bx[e] = f[3];
        for (int zl = 0; zl < 2; ++zl) { b.ia[e][zl] = f[4 + 3 * zl]; b.al[e][zl] = f[5 + 3 * zl]; b.pt[e][zl] = f[6 + 3 * zl]; }
        b.ap[e] = f[10];
        b.mid[e] = reinterpret_cast<Pair<R>*>(f[11]);   // npl (nK + nJ) pairs
        b.lo[e][0] = scr[e].x2;
        b.lo[e][1] = scr[e].x3;
        max_np = std::max(max_np, d.npl);
        max_nj = std::max(max_nj, d.nJ);
        max_nk = std::max(max_nk, d.nK);
        nim = std::max(nim, sys[e].nim);
        fsmem = std::max(fsmem, pv_factor_smem<R>(d));
    }
    const unsigned ptiles = (unsigned)((max_np + 31) / 32);
    const unsigned tiles_in = (unsigned)(((max_np + 2 + 31) / 32) * ((max_nk + 2 + 31) / 32));
    out_grid = dim3(ptiles * ((max_nk + 31) / 32), max_nj, nsys);
    const int nf = (int)(ptiles * ((max_nk + 15) / 16));
    launch_k(pdl, k_pv_fill<R>, dim3((unsigned)(nf * max_nj) + tiles_in * (max_nj + 2), 1, nsys), dim3(32, 8), 0, st, g, b, nf, max_nj,
             (int)tiles_in);
    launch_k(pdl, k_pv_factor<R, MARCH>, dim3((unsigned)max_np, nsys), dim3(kFactThreads), fsmem, st, b);
    return 2;
}

}  // namespace

int launch_pv(const GeoT<double>& g, const Sys<double>* sys, const AdiScratch<double>* scr, int nsys, cudaStream_t st,
              int rb_flags) {
    using R = double;
    int n = 0;
    pv_forms<R>([&](auto form) {
        using F = decltype(form);
        size_t smem = 0;
        if (!pv_fits<R, F>(sys, nsys, smem)) return false;
        const bool pdl = (rb_flags & kRbPdl) != 0;
        PvBatch<R> b;
        int max_np, nim;
        dim3 go;
        n = pv_setup<R, false>(g, sys, scr, nsys, pdl, st, b, max_np, nim, go);
        const dim3 gv((unsigned)((max_np + 1) / 2), nsys);
        size_t bytes = 0;   // the batch's records and its unknown
        for (int e = 0; e < nsys; ++e) {
            const PlaneDims d = dims_of(sys[e]);
            bytes += (size_t)(F::PPT ? 14 : 15) * d.npl * d.PB * sizeof(R);
        }
        const int ahead = bytes > kPvL2Bytes ? kPvSlots : 0;
        int first = 1;
        for (int ns = 0; ns < nim; ++ns)
            for (int half = 0; half < 2; ++half)
                for (int colour = 0; colour < 2; ++colour, ++n, first = 0)
                    launch_k(pdl, k_pv_visit<R, F::NT, F::PPT, F::CAP>, gv, dim3(F::NT), smem, st, b, colour, ns, first, ahead);
        launch_k(pdl, k_pv_copy_out<R>, go, dim3(32, 8), 0, st, g, b);
        ++n;
        return true;
    });
    return n;
}

// ADLBL3 in the reference's plane order; 0 where a plane does not fit
template <typename R>
int launch_pv_march(const GeoT<R>& g, const Sys<R>* sys, const AdiScratch<R>* scr, int nsys, cudaStream_t st, int rb_flags) {
    int n = 0;
    pv_forms<R>([&](auto form) {
        using F = decltype(form);
        size_t smem = 0;
        if (!pv_fits<R, F>(sys, nsys, smem)) return false;
        const bool pdl = (rb_flags & kRbPdl) != 0;
        PvBatch<R> b;
        int max_np, nim;
        dim3 go;
        n = pv_setup<R, true>(g, sys, scr, nsys, pdl, st, b, max_np, nim, go) + 2;
        launch_k(pdl, k_pv_march<R, F::NT, F::PPT, F::CAP>, dim3((unsigned)nsys), dim3(F::NT), smem, st, b);
        launch_k(pdl, k_pv_copy_out<R>, go, dim3(32, 8), 0, st, g, b);
        return true;
    });
    return n;
}

namespace {
template <typename R>
bool pv_raise() {
    bool ok = cudaFuncSetAttribute(k_pv_factor<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPvMaxSmem) == cudaSuccess;
    if constexpr (sizeof(R) == 8)
        ok = ok && cudaFuncSetAttribute(k_pv_factor<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPvMaxSmem) == cudaSuccess;
    pv_forms<R>([&](auto form) {
        using F = decltype(form);
        ok = ok && cudaFuncSetAttribute(k_pv_march<R, F::NT, F::PPT, F::CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kPvMaxSmem) == cudaSuccess;
        if constexpr (sizeof(R) == 8)
            ok = ok && cudaFuncSetAttribute(k_pv_visit<R, F::NT, F::PPT, F::CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kPvMaxSmem) == cudaSuccess;
        return false;
    });
    return ok;
}
}  // namespace
int prepare_pv() { return pv_raise<float>() && pv_raise<double>() ? GFM_OK : GFM_E_CUDA; }

template int launch_pv_march<float>(const GeoT<float>&, const Sys<float>*, const AdiScratch<float>*, int, cudaStream_t, int);
template int launch_pv_march<double>(const GeoT<double>&, const Sys<double>*, const AdiScratch<double>*, int, cudaStream_t, int);

}  // namespace gfm
