// adi_plane.cu -- the red-black line solver (GFM_ADI_REDBLACK) of the mixed path
// (FP32) with one CTA per plane visit: ADLZ (Adlbl3.f90:103-141) of one x-plane, both passes
// L = 1, 2 with their averages, in shared memory.
//
// Per ADLBL3 call (Adlbl3.f90:10-97) the system is rewritten once into
// plane-major arrays:
//
//   XP  the unknown with a one-point border on every side, plane p of the
//       class (I = IB + 2p, p = -1 .. npl) holding (nJ+2) x (nK+2) points,
//       K fastest: element (p, jj, kk) at ((p+1)(nJ+2) + jj+1)(nK+2) + kk+1;
//   YC, YX, YP  the rows of the y-lines (I, *, K), K fastest within the plane
//       ((p nJ + jj) nK + kk): YC = (AS21, AS31, AS32, BS), YX = (AS11, AS12)
//       and YP = (1/ALP, PT) with the Thomas pivots of the line,
//       ALP = AP - PT(prev) AS21, PT = AS22/ALP (ADLZY, Adlbl3.f90:147-181);
//   ZC, ZP  the rows of the z-lines (I, J, *), J fastest ((p nK + kk) nJ + jj):
//       ZC = (AS31, AS21, AS22, -), ZP = (1/ALP, PT) with ALP = AP - PT(prev)
//       AS31, PT = AS32/ALP (ADLYZ, Adlbl3.f90:187-221).
//
// The matrices do not change during the call, so the pivots are the values
// every visit of the reference would form.  A row the reference copies
// unchanged (|ALP| <= 1e-20 or a blocked cell) stores 1/ALP = 0 and PT = -0.0,
// a value no other row stores.  One launch (k_rbp_setup) forms them: the
// coefficients by a tiled transpose, the pivots by one thread per line walking
// its rows with the loads of the next rows in flight while the chain runs over
// the current ones.
//
// A visit (k_rbp_visit) has its plane of XP in shared memory, runs the
// y-lines of pass L=1 (which also form the x-neighbour part of the right-hand
// side, BX = BS + AS12 XT(I+2) + AS11 XT(I-2), fixed for the visit since the
// other colour does not move), the z-lines of pass L=1 averaging into the
// y-line results, then pass L=2 the same way from that average, and writes the
// plane back.  The lines of a pass are cut into segments: lanes of a warp take
// 32 neighbouring lines (so a warp's loads of one row are contiguous in the
// record layout of that direction), warps take segments of at most M rows, and
// the affine recurrences of the forward elimination and the back substitution
// are joined across segments by a scan of the segment maps in shared memory.
//
// What bounds it: bringing the records (24 bytes a point and pass, four passes)
// to the SM, at 96x64-point planes 650 KB a visit, and at small planes the
// latency of the chain of passes.  So the records and the plane come by bulk
// copies into shared memory while something else runs: of a small plane both
// directions' records, read once a visit and already while the visit before is
// finishing; of a large one a pass's records into the place of the pass before
// (as its threads have them in registers), behind its scans and its back
// substitution.  When every thread loaded its own records where it used them,
// loads were 30 of the 44 thousand cycles of a visit of a 96x64 plane (SM clock).  Line
// solver of an iteration in FP32, ms: TC21 tank 0.74 -> 0.56, 96x48x32 cells 1.31
// -> 0.89, 192x96x64 cells 3.60 -> 2.99; the results are the same bit for bit.
// Tried and left out: the next CTA's records prefetched to L2 (0.1 ms slower at
// 192x96x64: the copies in use wait behind them), two half-size chunks a pass
// (0.5 ms slower there), per-thread asynchronous copies (their issue takes 2
// thousand cycles a pass).
#include <algorithm>
#include <type_traits>

#include "state.cuh"

namespace gfm {

namespace {

template <typename R>
struct __align__(2 * sizeof(R)) Pair { R x, y; };

template <typename R>
struct RbpBatch {
    Sys<R> sys[8];
    R* xp[8];
    Quad<R>* yc[8];
    Pair<R>* yx[8];
    Pair<R>* yp[8];
    Quad<R>* zc[8];
    Pair<R>* zp[8];
    int nsys;
};

struct PlaneDims {
    int npl, nJ, nK;
};
template <typename R>
__host__ __device__ __forceinline__ PlaneDims dims_of(const Sys<R>& s) {
    return PlaneDims{(s.ie - s.ib) / 2 + 1, (s.je - s.jb) / 2 + 1, (s.ke - s.kb) / 2 + 1};
}
// row pitch (odd: rows and columns of a plane in shared memory meet different
// banks) and size of a bordered plane of XP (a multiple of 16 bytes, for bulk copies)
__host__ __device__ __forceinline__ int rbp_pitch(const PlaneDims& d) { return (d.nK + 2) | 1; }
__host__ __device__ __forceinline__ int rbp_plane(const PlaneDims& d) { return ((d.nJ + 2) * rbp_pitch(d) + 3) / 4 * 4; }
__host__ __device__ __forceinline__ int xp_index(const PlaneDims& d, int p, int jj, int kk) {
    return (p + 1) * rbp_plane(d) + (jj + 1) * rbp_pitch(d) + kk + 1;
}
// the copy-row marker PT = -0.0
__device__ __forceinline__ bool rbp_copy(float pt) { return __float_as_uint(pt) == 0x80000000u; }

// ---------------------------------------------------------------------------
// XT <-> XP, through a 32 x 32 tile in shared memory: plane index fastest on
// the class side, K fastest on the plane side.  Block (32, 8); bx over
// (plane tiles) x (K tiles), jr = J row of XP (border included), e = system.
// ---------------------------------------------------------------------------
template <typename R, bool IN>
__device__ __forceinline__ void rbp_copy_planes(const GeoT<R>& g, const RbpBatch<R>& b, int bx, int jr, int e, R (*tile)[33]) {
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
__global__ void k_rbp_copy_out(GeoT<R> g, RbpBatch<R> b) {
    __shared__ R tile[32][33];
    pdl_wait();
    pdl_trigger();
    rbp_copy_planes<R, false>(g, b, blockIdx.x, blockIdx.y, blockIdx.z, tile);
}

// ---------------------------------------------------------------------------
// The coefficients of the records (YC, YX of the y-lines; ZC of the z-lines),
// once per call, through a 32-plane x 16-line tile in shared memory: read with
// the plane index fastest (contiguous in the class arrays), written with the
// line index fastest (contiguous in the records).  Block (32, 8); bx over
// (plane tiles) x (line tiles), row = J of a y-line record, K of a z-line
// record, e = system.
// ---------------------------------------------------------------------------
template <typename R, bool ZL>
__device__ __forceinline__ void rbp_fill(const GeoT<R>& g, const RbpBatch<R>& b, int bx, int row, int e, R (*tile)[16][33]) {
    constexpr int NF = ZL ? 3 : 6;
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    const int nlines = ZL ? d.nJ : d.nK, nrows = ZL ? d.nK : d.nJ;
    if (row >= nrows) return;
    const int ntp = (d.npl + 31) / 32;
    const int p0 = (bx % ntp) * 32, l0 = (bx / ntp) * 16;
    if (l0 >= nlines) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    // y-line record: AS21, AS31, AS32, BS, AS11, AS12; z-line record: AS31, AS21, AS22
    const R* src[NF];
    if (ZL) {
        src[0] = s.as[4]; src[1] = s.as[2]; src[2] = s.as[3];
    } else {
        src[0] = s.as[2]; src[1] = s.as[4]; src[2] = s.as[5];
        src[3 % NF] = s.bs; src[4 % NF] = s.as[0]; src[5 % NF] = s.as[1];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int ll = ty + 8 * r, p = p0 + tx, l = l0 + ll;
        if (p < d.npl && l < nlines) {
            const int I = s.ib + 2 * p;
            const int o = (int)(ZL ? pidx(g, I, s.jb + 2 * l, s.kb + 2 * row) : pidx(g, I, s.jb + 2 * row, s.kb + 2 * l));
#pragma unroll
            for (int f = 0; f < NF; ++f) tile[f][ll][tx] = src[f][o];
        }
    }
    __syncthreads();
    const int tid = ty * 32 + tx;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int idx = tid + 256 * r;
        const int ll = idx & 15, pl = idx >> 4;
        const int p = p0 + pl, l = l0 + ll;
        if (p < d.npl && l < nlines) {
            if (ZL) {
                b.zc[e][(p * d.nK + row) * d.nJ + l] = Quad<R>{tile[0][ll][pl], tile[1][ll][pl], tile[2][ll][pl], R(0)};
            } else {
                const int q = (p * d.nJ + row) * d.nK + l;
                b.yc[e][q] = Quad<R>{tile[0][ll][pl], tile[1][ll][pl], tile[2][ll][pl], tile[3 % NF][ll][pl]};
                b.yx[e][q] = Pair<R>{tile[4 % NF][ll][pl], tile[5 % NF][ll][pl]};
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Pivots of every line, once per call: a thread walks one line (plane p, a
// fixed cross index) row by row through the pivot chain of ADLZY/ADLYZ.
// Lanes take 32 neighbouring planes, so each row's loads are contiguous in
// the class arrays; the rows are taken kPivRows at a time, the loads of the
// next batch issued before the chain runs over the current one.  A batch's
// pivots leave through a tile in shared memory with the line index fastest,
// contiguous in the records.  Block (32, 8): 32 planes x 8 lines; bx over
// (plane tiles) x (line tiles), e = system.  ZL: z-lines (rows along K, lines
// indexed by J), else y-lines (rows along J, lines indexed by K).
// ---------------------------------------------------------------------------
constexpr int kPivRows = 4;
template <typename R, bool ZL>
__device__ __forceinline__ void rbp_pivots(const GeoT<R>& g, const RbpBatch<R>& b, int bx, int e, Pair<R> (*tile)[8][33]) {
    constexpr int C = kPivRows;
    const Sys<R>& s = b.sys[e];
    const PlaneDims d = dims_of(s);
    const int nlines = ZL ? d.nJ : d.nK, nrows = ZL ? d.nK : d.nJ;
    const int ntp = (d.npl + 31) / 32;
    const int p0 = (bx % ntp) * 32, l0 = (bx / ntp) * 8;
    if (l0 >= nlines) return;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int p = p0 + tx, l = l0 + ty;
    const bool act = p < d.npl && l < nlines;
    // y-line (I,*,K): sub AS21 = as[2], next AS22 = as[3]; z-line (I,J,*): sub AS31 = as[4], next AS32 = as[5]
    const R* __restrict__ a_sub = s.as[ZL ? 4 : 2];
    const R* __restrict__ a_next = s.as[ZL ? 5 : 3];
    const R* __restrict__ a_p = s.ap;
    const int8_t* __restrict__ ibc = g.ib;
    const int I = s.ib + 2 * p;
    const int ostep = ZL ? (int)(pidx(g, 0, 0, 2) - pidx(g, 0, 0, 0)) : (int)(pidx(g, 0, 2, 0) - pidx(g, 0, 0, 0));
    const int o0 = act ? (int)(ZL ? pidx(g, I, s.jb + 2 * l, s.kb) : pidx(g, I, s.jb, s.kb + 2 * l)) : 0;
    const int tid = ty * 32 + tx;
    R cap[C], csub[C], cnxt[C];
    bool cblk[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        if (act && c < nrows) {
            const int o = o0 + c * ostep;
            cap[c] = a_p[o]; csub[c] = a_sub[o]; cnxt[c] = a_next[o]; cblk[c] = ibc[o] >= 1;
        }
    }
    R pt_prev = R(0);
    for (int r0 = 0; r0 < nrows; r0 += C) {
        R nap[C], nsub[C], nnxt[C];
        bool nblk[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int r = r0 + C + c;
            if (act && r < nrows) {
                const int o = o0 + r * ostep;
                nap[c] = a_p[o]; nsub[c] = a_sub[o]; nnxt[c] = a_next[o]; nblk[c] = ibc[o] >= 1;
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (act && r0 + c < nrows) {
                const R alp = cap[c] - pt_prev * csub[c];
                R ia, pt;
                if (fabs(alp) <= R(1.0e-20) || cblk[c]) {
                    ia = R(0);
                    pt = -R(0);
                    pt_prev = R(0);
                } else {
                    ia = R(1) / alp;
                    pt = cnxt[c] / alp + R(0);   // +0.0: no -0.0 here
                    pt_prev = pt;
                }
                tile[c][ty][tx] = Pair<R>{ia, pt};
            }
        }
        __syncthreads();
        // C rows x 8 lines x 32 planes, the line index fastest
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const int idx = tid + 256 * i;
            const int ll = idx & 7, pl = (idx >> 3) & 31, c = idx >> 8;
            const int pw = p0 + pl, lw = l0 + ll, rw = r0 + c;
            if (pw < d.npl && lw < nlines && rw < nrows) {
                if (ZL) b.zp[e][(pw * d.nK + rw) * d.nJ + lw] = tile[c][ll][pl];
                else b.yp[e][(pw * d.nJ + rw) * d.nK + lw] = tile[c][ll][pl];
            }
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < C; ++c) {
            cap[c] = nap[c]; csub[c] = nsub[c]; cnxt[c] = nnxt[c]; cblk[c] = nblk[c];
        }
    }
}

// The three in one launch, system e = blockIdx.y: blocks of grid x for the
// pivots (first, for their chains are the longest), the records, the planes.
// They read the call's arrays and write places of their own; the records and the
// planes move under the chains, which take half the registers with 4 rows a batch
// in place of 8, so that four blocks share an SM.  Line solver of an iteration,
// three launches -> one: TC21 tank 0.555 -> 0.534 ms, 96x48x32 cells 0.890 ->
// 0.868, 192x96x64 2.99 -> 2.96 (8 rows and two blocks an SM: 3.15).
struct RbpSetup {
    int pivots_y, pivots;    // blocks of the y-lines' pivots, of both
    int fill_y, fill, rows;  // of a row of the y-lines' records, of both directions', rows
    int copy;                // of a row of the planes
};
template <typename R>
__global__ void __launch_bounds__(256, 4) k_rbp_setup(GeoT<R> g, RbpBatch<R> b, RbpSetup n) {
    __shared__ union {
        R copy[32][33];
        R fill[6][16][33];
        Pair<R> pivots[kPivRows][8][33];
    } tile;
    pdl_wait();
    pdl_trigger();
    const int e = blockIdx.y;
    int id = blockIdx.x;
    if (id < n.pivots) {
        if (id < n.pivots_y) rbp_pivots<R, false>(g, b, id, e, tile.pivots);
        else rbp_pivots<R, true>(g, b, id - n.pivots_y, e, tile.pivots);
        return;
    }
    id -= n.pivots;
    if (id < n.fill * n.rows) {
        const int bx = id % n.fill, row = id / n.fill;
        if (bx < n.fill_y) rbp_fill<R, false>(g, b, bx, row, e, tile.fill);
        else rbp_fill<R, true>(g, b, bx - n.fill_y, row, e, tile.fill);
        return;
    }
    id -= n.fill * n.rows;
    rbp_copy_planes<R, true>(g, b, id % n.copy, id / n.copy, e, tile.copy);
}

// ---------------------------------------------------------------------------
// A thread's part of a pass over the y-lines (ZL false) or the z-lines (ZL
// true): the warps take 32 neighbouring lines each (G groups) and S segments of
// at most m rows; the thread has rows e0 .. e0+cnt-1 of `line`.
template <int NT, bool ZL>
struct RbpPart {
    int nlines, n, G, S, m, grp, seg, line, e0, cnt;
    bool active;
    __device__ __forceinline__ explicit RbpPart(const PlaneDims& d) {
        nlines = ZL ? d.nJ : d.nK;
        n = ZL ? d.nK : d.nJ;
        G = (nlines + 31) >> 5;
        S = (NT / 32) / G;
        S = S < 1 ? 1 : (S > n ? n : S);
        m = (n + S - 1) / S;
        const int warp = threadIdx.x >> 5;
        grp = warp % G;
        seg = warp / G;
        line = grp * 32 + (threadIdx.x & 31);
        active = seg < S && line < nlines;
        e0 = seg * m;
        cnt = active ? n - e0 : 0;
        cnt = cnt < 0 ? 0 : (cnt > m ? m : cnt);
    }
};

// What a visit needs of a system, together in the kernel's arguments (each cache
// line of them is a miss when a CTA starts).
template <typename R>
struct RbpSys {
    R* xp;
    Quad<R>* yc;
    Pair<R> *yx, *yp;
    Quad<R>* zc;
    Pair<R>* zp;
    PlaneDims d;
    int nim, one_row;
};
template <typename R>
struct RbpVisit {
    RbpSys<R> sys[8];
    double* lost;
    int wait[2];
};

// The records of a pass in shared memory: of each segment its first `rows` rows
// (the others are read from global memory), one bulk copy a segment and array.
// The (1/ALP, PT) of a segment begin 0 or 8 bytes into their place, where their
// 16-byte unit begins.
struct RbpStage {
    unsigned char* mem;
    uint32_t bar;     // mbarrier
    int rows;
    __host__ __device__ static int slot_c(int rows, int nlines) { return rows * nlines * 16; }
    __host__ __device__ static int slot_w(int rows, int nlines) { return (rows * nlines * 8 + 15) / 16 * 16 + 16; }
};
// A thread's waits of a visit: whether one for records ran out, and the copies of
// records begun on the first mbarrier (threads of the warp that begins them).
struct RbpWait {
    bool lost;
    int begun;
};
// by one warp; the mbarrier's phase ends when the copies have arrived
template <int NT, bool ZL, typename R>
__device__ __forceinline__ void rbp_fetch(const RbpSys<R>& b, int p, const RbpPart<NT, ZL>& pt, const RbpStage& st) {
    const int k = threadIdx.x & 31, rows = st.rows < pt.m ? st.rows : pt.m;
    const int e0 = k * pt.m;
    int r = k < pt.S ? pt.n - e0 : 0;
    r = r < 0 ? 0 : (r > rows ? rows : r);
    const size_t q = (size_t)(p * pt.n + e0) * pt.nlines;
    const uint32_t bc = (uint32_t)(r * pt.nlines) * 16;
    const unsigned long long w0 = (unsigned long long)((ZL ? b.zp : b.yp) + q);
    const uint32_t bw = r ? (uint32_t)(((w0 + r * pt.nlines * 8 + 15) & ~15ull) - (w0 & ~15ull)) : 0;
    const uint32_t total = __reduce_add_sync(0xffffffffu, bc + bw);
    if (k == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(st.bar), "r"(total) : "memory");
    __syncwarp();
    if (r) {
        const uint32_t dc = smem_u32(st.mem) + k * RbpStage::slot_c(rows, pt.nlines);
        const uint32_t dw = smem_u32(st.mem) + pt.S * RbpStage::slot_c(rows, pt.nlines) + k * RbpStage::slot_w(rows, pt.nlines);
        bulk_load(dc, (ZL ? b.zc : b.yc) + q, bc, st.bar);
        bulk_load(dw, (const void*)(w0 & ~15ull), bw, st.bar);
    }
}

// The pass.  src: the plane as before the pass (bordered, row pitch PS
// over K, J rows); dst: the y-line results (ZL false) or their average with the
// z-line results (ZL true), written into dst's interior.  FIRST: pass L=1 of a
// y-line forms BX from the record, its (AS11, AS12) X and the neighbouring
// planes' xm, xq, and keeps it in bxs; otherwise BX is read from bxs.  `parity`:
// of the phase of st.bar that its records end; `next`: the records of the next
// pass, over the other lines (nx), are fetched into the same place once this pass
// has used them.  A thread whose wait for records runs out (w.lost, for the rest of
// the visit) notes it in v.lost, which the host reports as an error, and from then on
// leaves the staged records alone; nothing more is fetched.
// ---------------------------------------------------------------------------
template <int NT, int M, bool ZL, bool FIRST, typename R>
__device__ __forceinline__ void rbp_pass(const RbpVisit<R>& v, RbpWait& w, const RbpSys<R>& b, int p, int PS, const RbpPart<NT, ZL>& pt,
                                         const RbpPart<NT, !ZL>& nx, const R* __restrict__ src, R* __restrict__ dst,
                                         R* __restrict__ bxs, R* __restrict__ sA, R* __restrict__ sB, const RbpStage& st,
                                         int parity, bool next, const Pair<R> (&X)[M], const R (&xm)[M], const R (&xq)[M]) {
    const int n = pt.n, G = pt.G, S = pt.S, grp = pt.grp, seg = pt.seg, line = pt.line, e0 = pt.e0, cnt = pt.cnt;
    const int lane = threadIdx.x & 31;
    const bool active = pt.active;
    const int q0 = (p * n + e0) * pt.nlines + line;
    int rows = st.rows < pt.m ? st.rows : pt.m;
    const Quad<R>* sc = reinterpret_cast<const Quad<R>*>(st.mem + seg * RbpStage::slot_c(rows, pt.nlines)) + line;
    const Pair<R>* sw = reinterpret_cast<const Pair<R>*>(st.mem + S * RbpStage::slot_c(rows, pt.nlines) +
                                                         seg * RbpStage::slot_w(rows, pt.nlines)) +
                        (((p * n + e0) * pt.nlines) & 1) + line;
    // shared-memory offsets: (jj, kk) of the bordered plane at (jj+1)*PS + kk+1,
    // of bxs at jj*PS + kk; a row step and the two across-line neighbours
    const int rstep = ZL ? 1 : PS, across = ZL ? PS : 1;
    const int c0 = ZL ? (line + 1) * PS + 1 : PS + line + 1;   // row 0 of the line
    const int bx0 = ZL ? line * PS : line;
    const int bstep = ZL ? 1 : PS;
    R xlo = R(0), xhi = R(0);
    if (active) {
        xlo = src[c0 - rstep];
        xhi = src[c0 + n * rstep];
    }
    R rr[M], al[M], pv[M];
    if (w.lost || !mbar_wait(st.bar, parity, v.wait[1])) {
        w.lost = true;
        *v.lost = 1.0;
        rows = 0;
    }
    // KL rows at a time, their loads before their arithmetic (at 768 threads and 8
    // rows the registers hold one; 2 or 4 spill: 3.08 and 3.26 ms for 2.99 above)
    constexpr int KL = NT > 256 && M > 4 ? 1 : 4;
    auto load = [&](auto staged) {
#pragma unroll
        for (int i0 = 0; i0 < M; i0 += KL) {
            Quad<R> A[KL];   // A = (AS_sub, AS_across-, AS_across+, -), W = (1/ALP, PT)
            Pair<R> W[KL];
            R bx[KL], sp[KL], sm[KL];
#pragma unroll
            for (int u = 0; u < KL; ++u) {
                const int i = i0 + u;
                if (i < cnt) {
                    if (decltype(staged)::value || i < rows) {
                        A[u] = sc[i * pt.nlines];
                        W[u] = sw[i * pt.nlines];
                    } else {
                        A[u] = (ZL ? b.zc : b.yc)[q0 + i * pt.nlines];
                        W[u] = (ZL ? b.zp : b.yp)[q0 + i * pt.nlines];
                    }
                    if (!FIRST) bx[u] = bxs[bx0 + (e0 + i) * bstep];
                    sp[u] = src[c0 + (e0 + i) * rstep + across];
                    sm[u] = src[c0 + (e0 + i) * rstep - across];
                }
            }
#pragma unroll
            for (int u = 0; u < KL; ++u) {
                const int i = i0 + u;
                if (i < cnt) {
                    if (FIRST) {
                        bx[u] = (A[u].w + X[i].y * xq[i]) + X[i].x * xm[i];   // BS + AS12 XT(I+2) + AS11 XT(I-2)
                        bxs[bx0 + (e0 + i) * bstep] = bx[u];
                    }
                    // y: + AS32 XT(K+2) + AS31 XT(K-2); z: + AS22 XT(J+2) + AS21 XT(J-2)
                    const R x = W[u].x * ((bx[u] + A[u].z * sp[u]) + A[u].y * sm[u]);
                    rr[i] = rbp_copy(W[u].y) ? src[c0 + (e0 + i) * rstep] : x;
                    al[i] = A[u].x * W[u].x;   // AS_sub/ALP; 0 on a copied row
                    pv[i] = W[u].y;
                }
            }
        }
    };
    if (rows >= cnt) load(std::true_type{});
    else load(std::false_type{});
    // forward elimination of the segment from a zero start: q = r + a q(prev)
    R q[M], P[M];
    R qc = R(0), Pc = R(1);
#pragma unroll
    for (int i = 0; i < M; ++i) {
        if (i < cnt) {
            qc = rr[i] + al[i] * qc;
            Pc = al[i] * Pc;
            q[i] = qc;
            P[i] = Pc;
        }
    }
    sA[threadIdx.x] = cnt > 0 ? Pc : R(1);
    sB[threadIdx.x] = cnt > 0 ? qc : R(0);
    __syncthreads();
    if (next && threadIdx.x < 32 && !__any_sync(0xffffffffu, w.lost)) {   // every thread has read its records
        async_fence();
        rbp_fetch(b, p, nx, st);
        ++w.begun;
    }
    // carry into the segment: the maps of the segments before it, in order
    // (their loads taken four at a time ahead of the chain)
    R qin = xlo;
    for (int k0 = 0; k0 < seg; k0 += 4) {
        R a4[4], b4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u;
            if (k < seg) { a4[u] = sA[(k * G + grp) * 32 + lane]; b4[u] = sB[(k * G + grp) * 32 + lane]; }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + u < seg) qin = a4[u] * qin + b4[u];
    }
#pragma unroll
    for (int i = 0; i < M; ++i)
        if (i < cnt) q[i] = q[i] + P[i] * qin;
    __syncthreads();
    // back substitution of the segment from a zero end: x = q + PT x(next)
    R xc = R(0), Rc = R(1);
#pragma unroll
    for (int i = M - 1; i >= 0; --i) {
        if (i < cnt) {
            xc = pv[i] * xc + q[i];
            Rc = pv[i] * Rc;
            q[i] = xc;
            P[i] = Rc;
        }
    }
    sA[threadIdx.x] = cnt > 0 ? Rc : R(1);
    sB[threadIdx.x] = cnt > 0 ? xc : R(0);
    __syncthreads();
    R xin = xhi;
    for (int k0 = S - 1; k0 > seg; k0 -= 4) {
        R a4[4], b4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 - u;
            if (k > seg) { a4[u] = sA[(k * G + grp) * 32 + lane]; b4[u] = sB[(k * G + grp) * 32 + lane]; }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 - u > seg) xin = a4[u] * xin + b4[u];
    }
#pragma unroll
    for (int i = 0; i < M; ++i) {
        if (i < cnt) {
            const int c = c0 + (e0 + i) * rstep;
            const R x = q[i] + P[i] * xin;
            dst[c] = ZL ? (dst[c] + x) / R(2) : x;   // (XT2 + XT3)/2
        }
    }
    __syncthreads();
}

// shared memory of the planes (two with border, BX) and of the segment maps
inline size_t rbp_smem_bytes(const PlaneDims& d, int nt) {
    return (size_t)(2 * rbp_plane(d) + d.nJ * rbp_pitch(d) + 2 * nt) * sizeof(float);
}
// Rows of a segment staged, the places in shared memory of the z-lines' records
// (0: that of the y-lines', one after the other) and of the planes, the visit's
// half of its sweep.
struct RbpLaunch {
    int rows, zoff, poff, half;
};

// One colour visit: every plane p = colour, colour + 2, .. of the call's
// planes (I = IB + 2p), one CTA each.
template <typename R, int NT, int M>
__global__ void __launch_bounds__(NT, NT > 256 ? 1 : 2) k_rbp_visit(RbpVisit<R> v, int colour, int sweep, RbpLaunch rl) {
    extern __shared__ __align__(16) unsigned char rbp_smem[];
    const RbpSys<R> b = v.sys[blockIdx.y];
    const PlaneDims d = b.d;
    const int npc = (d.npl - colour + 1) / 2;
    if (sweep >= b.nim || (int)blockIdx.x >= npc) {
        pdl_wait();   // nothing to do, but this launch must not end before the one it follows
        return;
    }
    const int p = colour + 2 * (int)blockIdx.x;
    __shared__ __align__(8) unsigned long long bars[3];
    const uint32_t bar = smem_u32(bars);
    const bool both = rl.zoff != 0;
    const RbpStage sty{rbp_smem, bar, rl.rows}, stz{rbp_smem + rl.zoff, both ? bar + 8 : bar, rl.rows};
    const RbpPart<NT, false> py(d);
    const RbpPart<NT, true> pz(d);
    if (threadIdx.x == 0) {
        for (int q = 0; q < 3; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        async_fence();
    }
    __syncwarp();
    // What the visit reads of the records.  They are fixed during the call, so
    // this runs while the kernel before, a visit of the same call, is finishing
    // (device.cuh, at pdl_wait).  Only the first visit waits first.
    Pair<R> X[M];
    auto records = [&] {
        if (threadIdx.x < 32) {
            rbp_fetch(b, p, py, sty);
            if (both) rbp_fetch(b, p, pz, stz);
        }
#pragma unroll
        for (int i = 0; i < M; ++i)
            if (i < py.cnt) X[i] = load_l2(b.yx + (p * d.nJ + py.e0 + i) * d.nK + py.line);
    };
    const bool fresh = sweep == 0 && colour == 0 && rl.half == 0;
    if (!fresh) records();
    pdl_wait();
    pdl_trigger();
    if (fresh) records();
    // the plane with its border, twice: the border of both holds the line ends
    const int PS = rbp_pitch(d), PB = rbp_plane(d);
    R* xa = reinterpret_cast<R*>(rbp_smem + rl.poff);
    R* xb = xa + PB;
    R* bxs = xb + PB;
    R* sA = bxs + d.nJ * PS;
    R* sB = sA + NT;
    R* __restrict__ own = b.xp + (size_t)(p + 1) * PB;
    if (threadIdx.x == 0) {
        async_fence();
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar + 16), "r"((uint32_t)PB * 8) : "memory");
        bulk_load(smem_u32(xa), own, PB * 4, bar + 16);
        bulk_load(smem_u32(xb), own, PB * 4, bar + 16);
    }
    // the neighbouring planes at the thread's rows of pass L=1
    R xm[M], xq[M];
#pragma unroll
    for (int i = 0; i < M; ++i)
        if (i < py.cnt) {
            const int q = (py.e0 + i + 1) * PS + py.line + 1;
            xm[i] = own[q - PB];
            xq[i] = own[q + PB];
        }
    __syncthreads();   // the mbarriers are set up
    RbpWait w{false, 1};
    // no copy is in flight when the CTA ends
    auto drain = [&] {
        if (threadIdx.x != 0) return;
        bool in = mbar_wait(bar, (w.begun - 1) & 1, kAdiPolls);
        if (both) in = mbar_wait(bar + 8, 0, kAdiPolls) && in;
        in = mbar_wait(bar + 16, 0, kAdiPolls) && in;
        if (!in) *v.lost = 1.0;
    };
    if (__syncthreads_or(!mbar_wait(bar + 16, 0, v.wait[0]))) {   // the plane did not come: it stays as it is
        if (threadIdx.x == 0) *v.lost = 1.0;
        drain();
        return;
    }
    // a plane with one z-row (KB >= KE) keeps the y-line pass alone (Adlbl3.f90:124-130)
    const bool one_row = b.one_row;
    const bool next = !both && !one_row;
    // pass L=1: y-lines into xb, then the z-lines averaged into it
    rbp_pass<NT, M, false, true>(v, w, b, p, PS, py, pz, xa, xb, bxs, sA, sB, sty, 0, next, X, xm, xq);
    if (!one_row) {
        rbp_pass<NT, M, true, false>(v, w, b, p, PS, pz, py, xa, xb, bxs, sA, sB, stz, !both, next, X, xm, xq);
        // pass L=2 from the average: y-lines into xa, then the z-lines averaged into it
        rbp_pass<NT, M, false, false>(v, w, b, p, PS, py, pz, xb, xa, bxs, sA, sB, sty, 0, next, X, xm, xq);
        rbp_pass<NT, M, true, false>(v, w, b, p, PS, pz, py, xb, xa, bxs, sA, sB, stz, !both, false, X, xm, xq);
    }
    const R* out = one_row ? xb : xa;
    for (int jj = threadIdx.x >> 5; jj < d.nJ; jj += NT / 32)
        for (int kk = threadIdx.x & 31; kk < d.nK; kk += 32) own[(jj + 1) * PS + kk + 1] = out[(jj + 1) * PS + kk + 1];
    drain();
}

constexpr int kRbpM = 8;            // rows of a segment held in registers
constexpr int kRbpThreads = 768;    // threads of a visit CTA (80 registers a thread, one CTA per SM)
constexpr int kRbpSmall = 256;      // threads of a visit CTA for planes whose passes fit 8 warps
constexpr size_t kRbpMaxSmem = 227 * 1024 - 64;   // less the kernel's mbarriers

// rows of a segment when the CTA's warps share nlines lines of n rows (the
// formula of RbpPart); the pass fits when that is M at most
inline int rbp_rows(int nlines, int n, int nt) {
    const int G = (nlines + 31) / 32;
    int S = (nt / 32) / G;
    S = S < 1 ? 1 : (S > n ? n : S);
    return (n + S - 1) / S;
}
// shared memory of the staged records of a pass
inline size_t rbp_stage_bytes(int nlines, int n, int nt, int rows) {
    const int m = rbp_rows(nlines, n, nt), r = std::min(rows, m);
    int S = (nt / 32) / ((nlines + 31) / 32);
    S = S < 1 ? 1 : (S > n ? n : S);
    return (size_t)S * (RbpStage::slot_c(r, nlines) + RbpStage::slot_w(r, nlines));
}
inline bool rbp_pass_fits(int nlines, int n, int nt = kRbpThreads) { return rbp_rows(nlines, n, nt) <= kRbpM; }

}  // namespace

int launch_rbp(const GeoT<float>& g, const Sys<float>* sys, const AdiScratch<float>* scr, int nsys, cudaStream_t st,
               int rb_flags) {
    using R = float;
    const bool pdl = (rb_flags & kRbPdl) != 0;
    RbpBatch<R> b;
    b.nsys = nsys;
    size_t smem = 0;
    int max_np = 0, max_nj = 0, max_nk = 0, nim = 0;
    // planes small enough for 8 warps run on CTAs of that size: a few
    // hundred points a plane leave most of a larger CTA idle at its barriers
    bool small = true;
    for (int e = 0; e < nsys; ++e) {
        const PlaneDims d = dims_of(sys[e]);
        if (!rbp_pass_fits(d.nK, d.nJ) || !rbp_pass_fits(d.nJ, d.nK)) return 0;
        small = small && rbp_pass_fits(d.nK, d.nJ, kRbpSmall) && rbp_pass_fits(d.nJ, d.nK, kRbpSmall);
        smem = std::max(smem, rbp_smem_bytes(d, kRbpThreads));
        b.sys[e] = sys[e];
        // the records in the scratch of the segmented form (2*CBH elements each)
        const long long NH = 2LL * g.CBH;
        b.xp[e] = scr[e].xs;
        b.yc[e] = scr[e].ya;
        b.yx[e] = reinterpret_cast<Pair<R>*>(scr[e].yb);
        b.yp[e] = reinterpret_cast<Pair<R>*>(scr[e].yb) + NH;
        b.zc[e] = scr[e].za;
        b.zp[e] = reinterpret_cast<Pair<R>*>(scr[e].zb);
        max_np = std::max(max_np, d.npl);
        max_nj = std::max(max_nj, d.nJ);
        max_nk = std::max(max_nk, d.nK);
        nim = std::max(nim, sys[e].nim);
    }
    if (smem > kRbpMaxSmem) return 0;
    // records through shared memory: of both directions where they fit (each
    // read once a visit), else of one at a time, else as many rows of them as fit
    const int nt = small ? kRbpSmall : kRbpThreads;
    RbpLaunch rl{};
    smem = 0;
    for (int e = 0; e < nsys; ++e) smem = std::max(smem, rbp_smem_bytes(dims_of(sys[e]), nt));
    for (rl.rows = kRbpM; rl.rows >= 0; --rl.rows) {
        size_t y = 0, z = 0;
        for (int e = 0; e < nsys; ++e) {
            const PlaneDims d = dims_of(sys[e]);
            y = std::max(y, rbp_stage_bytes(d.nK, d.nJ, nt, rl.rows));
            z = std::max(z, rbp_stage_bytes(d.nJ, d.nK, nt, rl.rows));
        }
        const bool both = rl.rows == kRbpM && smem + y + z <= kRbpMaxSmem;
        rl.zoff = both ? (int)y : 0;
        rl.poff = (int)(both ? y + z : std::max(y, z));
        if (smem + rl.poff <= kRbpMaxSmem) break;
    }
    if (rl.rows < 0) return 0;
    smem += rl.poff;
    const unsigned tiles_in = (unsigned)(((max_np + 2 + 31) / 32) * ((max_nk + 2 + 31) / 32));
    const unsigned tiles_out = (unsigned)(((max_np + 31) / 32) * ((max_nk + 31) / 32));
    const unsigned ptiles = (unsigned)((max_np + 31) / 32);
    RbpSetup n;
    n.pivots_y = (int)(ptiles * ((max_nk + 7) / 8));
    n.pivots = n.pivots_y + (int)(ptiles * ((max_nj + 7) / 8));
    n.fill_y = (int)(ptiles * ((max_nk + 15) / 16));
    n.fill = n.fill_y + (int)(ptiles * ((max_nj + 15) / 16));
    n.rows = std::max(max_nj, max_nk);
    n.copy = (int)tiles_in;
    launch_k(pdl, k_rbp_setup<R>, dim3((unsigned)(n.pivots + n.fill * n.rows + n.copy * (max_nj + 2)), nsys), dim3(32, 8), 0, st, g, b, n);
    RbpVisit<R> v{};
    v.lost = scr[0].lost;
    for (int q = 0; q < 2; ++q) v.wait[q] = scr[0].wait[q];
    int m = 1;
    for (int e = 0; e < nsys; ++e) {
        const PlaneDims d = dims_of(sys[e]);
        v.sys[e] = RbpSys<R>{b.xp[e], b.yc[e], b.yx[e], b.yp[e], b.zc[e], b.zp[e], d, sys[e].nim, sys[e].kb >= sys[e].ke};
        m = std::max(m, std::max(rbp_rows(d.nK, d.nJ, nt), rbp_rows(d.nJ, d.nK, nt)));
    }
    auto* visit = small ? (m > 4 ? k_rbp_visit<R, kRbpSmall, kRbpM> : k_rbp_visit<R, kRbpSmall, 4>)
                        : (m > 4 ? k_rbp_visit<R, kRbpThreads, kRbpM> : k_rbp_visit<R, kRbpThreads, 4>);
    for (int ns = 0; ns < nim; ++ns)
        for (rl.half = 0; rl.half < 2; ++rl.half)
            for (int colour = 0; colour < 2; ++colour)
                launch_k(pdl, visit, dim3((unsigned)((max_np + 1) / 2), nsys), dim3(nt), smem, st, v, colour, ns, rl);
    launch_k(pdl, k_rbp_copy_out<R>, dim3(tiles_out, max_nj, nsys), dim3(32, 8), 0, st, g, b);
    return 2 + 4 * nim;
}

int prepare_rbp() {
    for (const void* k : {(const void*)k_rbp_visit<float, kRbpThreads, kRbpM>, (const void*)k_rbp_visit<float, kRbpThreads, 4>,
                          (const void*)k_rbp_visit<float, kRbpSmall, kRbpM>, (const void*)k_rbp_visit<float, kRbpSmall, 4>})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRbpMaxSmem) != cudaSuccess) return GFM_E_CUDA;
    return GFM_OK;
}

}  // namespace gfm
