// mgpu_tstep.cu -- SUBROUTINE TSTEP (multall-open-18.3.f:5470-5932) with
// SMOOTH_VAR (15352-15594) and SMOOTH_RESID (14833-14917) on the GPU.
//
// One call updates one conserved variable D with its SCREE history DIFF in
// four kernels, each but update with one CTA per J-plane (a J-plane of the
// largest configuration, 73 x 57 points, is 16 KB: it lives in shared memory);
// update's CTAs march along J over tiles of K:
//   cells    tip-gap TFLUX balance, mixing-plane flux extrapolation into
//            SOURCE, the flux sum DELTA -> STORE and DIFF, the pitchwise
//            redistribution of STORE on the mixing-plane cells, and this
//            plane's partial sums for the three multigrid levels
//   prolong  block sums assembled from the plane partials (level-1 blocks
//            span <= JR planes, level-2 <= JRBB, superblocks a row part);
//            STORE*STEP + corrections*RSTEP; per-plane sum of |STORE|
//   update   per-row mean |STORE| and the negative feedback of the cell
//            changes (1501-1525), the second mixing-plane average (1850), then
//            every node gathers its <= 8 cell changes in the order the
//            reference's scatter loop adds them (1100) -- no atomics, result
//            written to TMP
//   smooth   streamwise smoothing of plane J from TMP planes J-2..J+2, then
//            pitchwise, spanwise, corners, exit smoothing, periodic,
//            tip-gap and mixing-plane averaging in shared memory -> D
// With REDUCE_ORDER=1 the level sums and the row mean are instead formed by
// single threads in the reference's sequential REAL*4 order (parity checks);
// with REDUCE_ORDER=2 (the plain FP32 path) they are the default path's
// trees with FP32 adds.
#include <type_traits>

#include "mgpu_internal.cuh"

namespace mgpu {

static inline unsigned grid_for(size_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

// Threads per J-plane CTA: 128, 192, 256 (the default) or 512, chosen per
// problem and pass by mgpu_autotune (Dev::ts_bs); each size keeps 1024
// threads of 64 registers resident per SM (960 for 192: five CTAs).  us a step
// with both passes at 128, 192, 256 and 512: 9 x 50 x 7 72.2, 71.0, 72.6, 72.7;
// 37 x 98 x 33 104, 97.0, 94.7, 92.4; 37 x 194 x 33 116, 111, 111, 136; 49 x 162 x 41
// 148, 140, 137, 165; 65 x 242 x 49 244, 230, 229, 264; 73 x 752 x 57 674, 661, 659,
// 734; 96 x 120 x 40 218, 188, 175, 182.  A pass by itself can want another size:
// the momenta of 65 x 242 x 49 97.1 us at 192 and 99.3 at 256 (723 CTAs on 608
// slots), a grid of fewer CTAs than SMs 512.
constexpr int TS_U = 3;          // cells per thread whose loads are issued together
constexpr int SV_U = 3;          // points per thread whose streamwise loads are issued together
constexpr int SM_SEG = 4;        // points per thread of one pitchwise or spanwise smoothing segment
constexpr int SM_PAD = 2;        // floats before the plane buffers (a segment reads one before its line)
constexpr int PR_U = 3;          // the same in prolong: five CTAs an SM at 48 registers (two cells and six CTAs:
                                 // 38.9 us a launch against 37.6 on the 73 x 752 x 57 compressor, 16.5
                                 // against 15.8 at 65 x 242 x 49)
constexpr int TS_UG = 4;         // cells per thread whose loads the pair update issues together
constexpr int UG_SEG = 3;        // nodes per thread of one K column in the pair update's gather

// CTA sum of one double-float per thread (thread 0 receives it)
template <int BS>
__device__ inline df block_sum(int order, df v, df *sh) {
    for (int o = 16; o > 0; o >>= 1) v = dacc(order, v, df_shfl_down(v, o));
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    df r = df_of(0.0f);
    if (w == 0) {
        r = l < BS / 32 ? sh[l] : df_of(0.0f);
        for (int o = BS > 256 ? 8 : BS > 128 ? 4 : 2; o > 0; o >>= 1) r = dacc(order, r, df_shfl_down(r, o));
    }
    __syncthreads();
    return r;
}

// Pitchwise sum of a mixing-plane line in I order, REAL*4 as the reference
// forms it (REDUCE_ORDER 1, and the plain FP32 path, 2).
__device__ inline float mp_line_sum(const float *row, int n) {
    float s = 0.0f;
    for (int i = 0; i < n; ++i) s = s + row[i];
    return s;
}

// The default precision split's form of the same sum: accumulated in
// double-float and rounded once.  Eight lanes a row, so a warp forms four
// rows' sums at a time: each lane adds every eighth term, then three shuffle
// steps; the row's eight lanes get the total.  Every lane of the warp calls
// it (a row that is not wanted with n = 0).  A whole warp a row spent two
// thirds of its instructions in five-step trees over two terms a lane, and
// the CTAs of the mixing planes were the longest of their launch.
//
// U terms a lane are read together before they are added, so that terms in
// global memory cost one latency.  An added term has no low part: of the
// double-float addition, the steps that add it are left out (same result).
constexpr int ROW_LANES = 8;
__device__ __forceinline__ df df_add_f(df a, float x) {
    const float s = a.hi + x;
    const float bv = s - a.hi;
    float e = (a.hi - (s - bv)) + (x - bv);
    e = e + a.lo;
    const float s2 = s + e;
    return df{s2, e - (s2 - s)};
}
template <int LANES = ROW_LANES, int U = 4, class F>
__device__ __forceinline__ float row_sum64(int n, F term) {
    df s = df_of(0.0f);
#pragma unroll 1
    for (int i0 = (int)threadIdx.x % LANES; i0 < n; i0 += LANES * U) {
        float v[U];
#pragma unroll
        for (int q = 0; q < U; ++q) v[q] = i0 + LANES * q < n ? term(i0 + LANES * q) : 0.0f;
#pragma unroll
        for (int q = 0; q < U; ++q) s = df_add_f(s, v[q]);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s = df_add(s, df_shfl_xor(s, o));
    return df_val(s);
}
// Calls row(r, l, on) for the rows r of [0, nrow) with the lanes l of each;
// on is false for the lanes past the last row, which take part in the warp's
// shuffles only.
template <int LANES = ROW_LANES, class F>
__device__ __forceinline__ void for_rows(int nrow, F row) {
    const int step = (int)blockDim.x / LANES, warp0 = (int)(threadIdx.x & ~31u) / LANES;
    int r = (int)threadIdx.x / LANES;
#pragma unroll 1
    for (int r0 = warp0; r0 < nrow; r0 += step, r += step) row(r, (int)threadIdx.x % LANES, r < nrow);
}

// ---------------------------------------------------------------------
// cells: 5503-5510 (tip gap), 5516-5555 (MP extrapolation), 1000 (flux
// sum), 1750 (MP redistribution) and the multigrid partial sums
// ---------------------------------------------------------------------
template <int BS>
__global__ void __launch_bounds__(BS, 1024 / BS) k_ts_cells(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    extern __shared__ float sm[];
    const VarSet &V = d.var[v0 + blockIdx.y];
    float *__restrict__ DIFF = V.DIFF;
    __shared__ df shd[BS / 32];
    const int j = blockIdx.x + 2;
    const int IM = d.IM, IMM1 = d.IMM1, KMM1 = d.KMM1;
    const int nc = IMM1 * KMM1;
    float *st = sm;              // STORE of this plane, [k-1][i-1]
    float *lsum = sm + nc;       // per-K line sums
    // at a mixing plane: the flow's direction on each line, the pitchwise weights
    float *fdir = lsum + KMM1 + d.NIB1 * d.NKB1, *fp = fdir + KMM1;
    const PlaneInfo &pl = d.PLANE[j - 1];
    const int role = pl.role, jmx = pl.jmx, kts = pl.kts, kte = pl.kte;
    const float RATPITCH = pl.ratpitch;
    const bool lowx = d.FEXTRAP < 0.001f;
    // the cells of this thread's first level-1 block, for the partial sums below
    const int n1 = d.NIB1 * d.NKB1, n2 = d.NIB2 * d.NKB2;
    const int4 blk1 = d.MG1X[min((int)threadIdx.x, n1 - 1)], blk2 = d.MG2X[min((int)threadIdx.x, n2 - 1)];
    if (role) {
        auto flow = [&](int k) { return -A3(d.FLOWX, d.IMID, jmx, k); };
        for (int k = threadIdx.x + 1; k <= KMM1; k += BS) fdir[k - 1] = flow(k);
        for (int i = threadIdx.x + 1; i <= IMM1; i += BS) fp[i - 1] = A1(d.FP, i);
        // each I-line's XFLUX is added where it is extrapolated: read
        // straight from memory, four lanes a row so that a round takes 64
        // rows, the terms of a row in one latency
        if (role != 2 && !lowx) {
            const float *xj = V.XF + IM * (role == 1 ? j - 2 : j - 1);
            const int kx = IM * d.JM;
            if (d.REDUCE_ORDER == 0) {
                for_rows<4>(KMM1, [&](int r, int l, bool on) {
                    // after the plane (role 3) only against the flow, which is rare
                    if (role == 3 && !__any_sync(0xffffffffu, on && !(flow(r + 1) > 0.0f))) return;
                    const float *row = xj + kx * r;
                    const float s = row_sum64<4, 16>(on ? IMM1 : 0, [&](int i) { return row[i]; });
                    if (on && l == 0) lsum[r] = s;
                });
            } else {
                // stage the XFLUX plane in shared memory (coalesced), then
                // add each I-line in the reference's order
                Walk2 wx(IMM1, threadIdx.x, BS);
                for (int c = threadIdx.x; c < nc; c += BS, wx.next()) st[c] = xj[(wx.i - 1) + kx * (wx.k - 1)];
                __syncthreads();
                for (int k = threadIdx.x + 1; k <= KMM1; k += BS)
                    if ((role == 1) == (fdir[k - 1] > 0.0f)) lsum[k - 1] = mp_line_sum(st + (k - 1) * IMM1, IMM1);
            }
        }
        __syncthreads();
    }
    const float F1 = d.F1, F2 = d.F2, F3 = d.F3;
    const float *__restrict__ XF = V.XF;
    const float *__restrict__ RF = V.RF;
    const float *__restrict__ TF = V.TF;
    const float *__restrict__ SR = V.SR;
    // each thread first loads the operands of its TS_U cells, then computes:
    // the loads of all cells are in flight together.  Offsets are 32-bit
    // (a node array holds fewer than 2^31 points: commit limits IM, KM and JM)
    const int ks = IM * d.JM, pj = IM * (j - 1);
    Walk2 w(IMM1, threadIdx.x, BS);
    for (int c0 = threadIdx.x; c0 < nc; c0 += TS_U * BS) {
        float xf[TS_U], xm[TS_U], rf[TS_U], rk[TS_U], ta[TS_U], tb1[TS_U], sr[TS_U], df[TS_U];
        int ci[TS_U], ck[TS_U];
#pragma unroll
        for (int u = 0; u < TS_U; ++u) {
            ci[u] = w.i;
            ck[u] = w.k;
            w.next();
            if (c0 + u * BS < nc) {
                const int n = pj + (ci[u] - 1) + ks * (ck[u] - 1);
                xf[u] = XF[n];
                xm[u] = XF[n - IM];
                rf[u] = RF[n];
                rk[u] = RF[n + ks];
                ta[u] = TF[n];
                tb1[u] = TF[n + 1];
                sr[u] = SR[n];
                df[u] = DIFF[n];
            }
        }
#pragma unroll
        for (int u = 0; u < TS_U; ++u) {
            const int c = c0 + u * BS;
            if (c >= nc) break;
            const int i = ci[u], k = ck[u];
            const int n = pj + (i - 1) + ks * (k - 1);
            float t0 = ta[u], t1 = tb1[u];
            if (kts > 0 && k >= kts && k <= kte - 1) {
                if (i == 1 || i + 1 == IM) {
                    float tb = 0.5f * (A3(TF, 1, j, k) + A3(TF, IM, j, k));
                    if (i == 1) t0 = tb;
                    if (i + 1 == IM) t1 = tb;
                }
            }
            float src = sr[u];
            if (role && !lowx) {
                const float FLOWDIRN = fdir[k - 1];
                if (role == 1 && FLOWDIRN > 0.0f) src = src - (xm[u] - lsum[k - 1] * fp[i - 1]) * d.FEXTRAP;
                if (role == 2) src = 0.0f;
                if (role == 3 && !(FLOWDIRN > 0.0f)) src = src + (xf[u] - lsum[k - 1] * fp[i - 1]) * d.FEXTRAP;
            }
            float DELTA = xf[u] - xm[u] * RATPITCH + rf[u] - rk[u] + t0 - t1 - src;
            st[c] = F1 * DELTA + F2 * df[u];
            DIFF[n] = DELTA + F3 * df[u];
        }
    }
    __syncthreads();
    if (role == 1 || role == 3) {
        auto averaged = [&](int k) {
            const float FLOWDIRN = fdir[k - 1];
            return role == 3 ? (FLOWDIRN > 0.0f || lowx) : (FLOWDIRN < 0.0f || lowx);
        };
        if (d.REDUCE_ORDER != 0) {
            for (int k = threadIdx.x + 1; k <= KMM1; k += BS) {
                if (!averaged(k)) continue;
                float *row = st + (k - 1) * IMM1;
                const float s = mp_line_sum(row, IMM1);
                for (int i = 0; i < IMM1; ++i) row[i] = s * fp[i];
            }
        } else {
            for_rows(KMM1, [&](int r, int l, bool on) {
                on = on && averaged(r + 1);
                if (!__any_sync(0xffffffffu, on)) return;
                float *row = st + r * IMM1;
                const int n = on ? IMM1 : 0;
                const float s = row_sum64(n, [&](int i) { return row[i]; });
                for (int i = l; i < n; i += ROW_LANES) row[i] = s * fp[i];
            });
        }
        __syncthreads();
    }
    // plane sum: a thread's dozen cells in FP32, the threads' partials in
    // double-float
    float psf = 0.0f;
    {
        float *__restrict__ STj = V.ST + pj;
        Walk2 wp(IMM1, threadIdx.x, BS);
        for (int c = threadIdx.x; c < nc; c += BS, wp.next()) {
            float v = st[c];
            STj[(wp.i - 1) + ks * (wp.k - 1)] = v;
            psf += v;
        }
    }
    // (each warp's part here; the last warp adds the parts below, beside the
    // block sums)
    const int ro = d.REDUCE_ORDER, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    {
        df v = df_of(psf);
        for (int o = 16; o > 0; o >>= 1) v = dacc(ro, v, df_shfl_down(v, o));
        if (lane == 0) shd[wp] = v;
    }
    auto plane_sum = [&]() {
        if (wp != BS / 32 - 1) return;
        df r = lane < BS / 32 ? shd[lane] : df_of(0.0f);
        for (int o = BS > 256 ? 8 : BS > 128 ? 4 : 2; o > 0; o >>= 1) r = dacc(ro, r, df_shfl_down(r, o));
        if (lane == 0) V.psum[j - 1] = r;
    };
    // level-1 and level-2 partial sums of this plane
    auto block_cells = [&](int4 x) {
        float s = 0.0f;
        for (int k = x.z; k <= x.w; ++k)
            for (int i = x.x; i <= x.y; ++i) s = s + st[(k - 1) * IMM1 + (i - 1)];
        return s;
    };
    float *__restrict__ P1 = V.P1 + (size_t)(j - 1) * n1;
    float *__restrict__ P2 = V.P2 + (size_t)(j - 1) * n2;
    if (d.mg_nested) {
        // every level-2 block is a union of level-1 blocks: the level-1
        // partials first (in shared memory), then each level-2 partial as the
        // sum of its level-1 partials (a 9-term chain for 3 x 3 blocks of
        // 3 x 3 cells, where the direct sum is an 81-term chain)
        float *p1 = lsum + KMM1;
        for (int u = threadIdx.x; u < n1; u += BS) {
            const float s = block_cells(u < BS ? blk1 : d.MG1X[u]);
            p1[u] = s;
            P1[u] = s;
        }
        __syncthreads();
        plane_sum();
        for (int u = threadIdx.x; u < n2; u += BS) {
            const int4 x = u < BS ? blk2 : d.MG2X[u];
            float s = 0.0f;
            for (int kb1 = x.z; kb1 <= x.w; ++kb1)
                for (int ib1 = x.x; ib1 <= x.y; ++ib1) s = s + p1[(kb1 - 1) * d.NIB1 + (ib1 - 1)];
            P2[u] = s;
        }
        return;
    }
    for (int u = threadIdx.x; u < n1; u += BS) P1[u] = block_cells(u < BS ? blk1 : d.MG1X[u]);
    for (int u = threadIdx.x; u < n2; u += BS) P2[u] = block_cells(u < BS ? blk2 : d.MG2X[u]);
    __syncthreads();
    plane_sum();
}

// ---------------------------------------------------------------------
// reference-order level sums (REDUCE_ORDER=1): one thread per block walks
// its cells in the (K,J,I) loop order of 700; superblocks likewise
// ---------------------------------------------------------------------
__global__ void k_ts_restrict_seq(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    const VarSet &V = d.var[v0 + blockIdx.y];
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int n1 = d.NIB1 * (d.NJB1 + 1) * d.NKB1;
    int n2 = d.NIB2 * (d.NJB2 + 1) * d.NKB2;
    if (t >= n1 + n2 + d.NSBLK) return;
    if (t >= n1 + n2) {
        int sb = t - n1 - n2 + 1;
        int a = A1(d.SB_START, sb), b = A1(d.SB_END, sb);
        float s = 0.0f;
        for (int k = 1; k <= d.KMM1; ++k)
            for (int j = a; j <= b; ++j)
                for (int i = 1; i <= d.IMM1; ++i) s = s + A3(V.ST, i, j, k);
        A1(V.SBSUM, sb) = s;
        return;
    }
    const bool lv1 = t < n1;
    int u = lv1 ? t : t - n1;
    int nib = lv1 ? d.NIB1 : d.NIB2, njb = lv1 ? d.NJB1 : d.NJB2;
    int ib = u % nib + 1;
    int jb = (u / nib) % (njb + 1) + 1;
    int kb = u / (nib * (njb + 1)) + 1;
    float s = 0.0f;
    if (jb <= njb) {
        int j0 = lv1 ? A1(d.JB1_START, jb) : A1(d.JB2_START, jb), j1 = lv1 ? A1(d.JB1_END, jb) : A1(d.JB2_END, jb);
        int i0 = lv1 ? A1(d.IB1_S, ib) : A1(d.IB2_S, ib), i1 = lv1 ? A1(d.IB1_E, ib) : A1(d.IB2_E, ib);
        int k0 = lv1 ? A1(d.KB1_S, kb) : A1(d.KB2_S, kb), k1 = lv1 ? A1(d.KB1_E, kb) : A1(d.KB2_E, kb);
        for (int k = k0; k <= k1; ++k)
            for (int j = j0; j <= j1; ++j)
                for (int i = i0; i <= i1; ++i) s = s + A3(V.ST, i, j, k);
    }
    (lv1 ? V.B1CHG : V.B2CHG)[u] = s;
}

// Sum over the J planes a..e of one block's per-plane partial sums, added in
// J order in REAL*4; the loads of three planes (a level-1 block, a third of a
// level-2 block) are issued before their adds.
__device__ __forceinline__ float plane_partials_sum(const float *__restrict__ P, int n, int t, int a, int e) {
    float s = 0.0f;
    int jj = a;
    for (; jj + 2 <= e; jj += 3) {
        const float x0 = P[(size_t)(jj - 1) * n + t], x1 = P[(size_t)jj * n + t], x2 = P[(size_t)(jj + 1) * n + t];
        s = s + x0;
        s = s + x1;
        s = s + x2;
    }
    for (; jj <= e; ++jj) s = s + P[(size_t)(jj - 1) * n + t];
    return s;
}

// ---------------------------------------------------------------------
// prolong: 1500, with the block sums assembled from the plane partials.
// A block's correction, sum x block step, is one value for all of its cells,
// so it is formed once per block, and where every level-2 block is a union of
// level-1 blocks the three levels are added up once per level-1 block too; a
// cell takes its block's number from a table (CB1, CB2) and one value from
// shared memory.  Each value is the same product and sum as cell by cell,
// where gathering four block indices and two block steps for each cell made
// 120 instructions and six dependent loads of it.
// ---------------------------------------------------------------------
template <int BS>
__global__ void __launch_bounds__(BS, 1280 / BS) k_ts_prolong(const __grid_constant__ Dev d, int v0, int want_abs) {
    pdl_wait();
    extern __shared__ float sm[];
    const VarSet &V = d.var[v0 + blockIdx.y];
    __shared__ df shd[BS / 32];
    __shared__ float s_sb;
    const int j = blockIdx.x + 2;
    const int IMM1 = d.IMM1, KMM1 = d.KMM1;
    const int n1 = d.NIB1 * d.NKB1, n2 = d.NIB2 * d.NKB2;
    float *b1 = sm, *b2 = sm + n1;
    const PlaneInfo &pl = d.PLANE[j - 1];
    const int j1 = pl.jb1, j2 = pl.jb2, jsb = pl.jsb;
    const int nc = IMM1 * KMM1;
    const int m1 = d.NIB1 * (d.NJB1 + 1), m2 = d.NIB2 * (d.NJB2 + 1);
    const bool nested = d.mg_nested != 0;
    float *__restrict__ ST = V.ST;
    const float *__restrict__ STEP = d.STEP;
    const float *__restrict__ RSTEP = d.RSTEP;
    // operands of this thread's first PR_U cells, loaded before the block
    // sums so their latency overlaps the assembly below
    float pst[PR_U], pstp[PR_U], prs[PR_U];
    int pb1[PR_U], pb2[PR_U];
    unsigned pn[PR_U];
    WalkB w(IMM1, d.IM * d.JM, d.IM * (j - 1), threadIdx.x, BS);
    auto load = [&](int c0) {
#pragma unroll
        for (int u = 0; u < PR_U; ++u) {
            const int c = c0 + u * BS;
            pn[u] = w.b;
            if (c < nc) {
                pst[u] = *at(ST, w.b);
                pstp[u] = *at(STEP, w.b);
                prs[u] = *at(RSTEP, w.b);
                pb1[u] = *at(d.CB1, 2u * (unsigned)c);
                pb2[u] = nested ? 0 : *at(d.CB2, 2u * (unsigned)c);
            }
            w.next();
        }
    };
    load(threadIdx.x);
    if (d.REDUCE_ORDER == 1) {
        for (int t = threadIdx.x; t < n1; t += BS) {
            const int o = t % d.NIB1 + d.NIB1 * (j1 - 1) + m1 * (t / d.NIB1);
            b1[t] = V.B1CHG[o] * d.STEP1[o];
        }
        for (int t = threadIdx.x; t < n2; t += BS) {
            const int o = t % d.NIB2 + d.NIB2 * (j2 - 1) + m2 * (t / d.NIB2);
            b2[t] = V.B2CHG[o] * d.STEP2[o];
        }
        if (threadIdx.x == 0) s_sb = A1(V.SBSUM, jsb);
    } else {
        // the J planes of this plane's level-1 and level-2 blocks (empty past
        // the last block); each sum adds the planes' partials in J order
        const int a1 = pl.a1, e1 = pl.e1, a2 = pl.a2, e2 = pl.e2;
        for (int t = threadIdx.x; t < n1; t += BS) {
            const float st1 = d.STEP1[t % d.NIB1 + d.NIB1 * (j1 - 1) + m1 * (t / d.NIB1)];
            b1[t] = plane_partials_sum(V.P1, n1, t, a1, e1) * st1;
        }
        for (int t = threadIdx.x; t < n2; t += BS) {
            const float st2 = d.STEP2[t % d.NIB2 + d.NIB2 * (j2 - 1) + m2 * (t / d.NIB2)];
            b2[t] = plane_partials_sum(V.P2, n2, t, a2, e2) * st2;
        }
        if (threadIdx.x < 32) {
            const int ro = d.REDUCE_ORDER;
            df s = df_of(0.0f);
            for (int jj = pl.sa + (int)threadIdx.x; jj <= pl.se; jj += 32) s = dacc(ro, s, V.psum[jj - 1]);
            for (int o = 16; o > 0; o >>= 1) s = dacc(ro, s, df_shfl_down(s, o));
            if (threadIdx.x == 0) s_sb = df_val(s);
        }
    }
    if (d.IR <= 1 && d.JR <= 1 && d.KR <= 1) {
        // no multigrid: TSTEP skips the restriction (5613) and the block
        // changes keep the zeros they start from (5490-5498)
        for (int t = threadIdx.x; t < n1; t += BS) b1[t] = 0.0f;
        for (int t = threadIdx.x; t < n2; t += BS) b2[t] = 0.0f;
        if (threadIdx.x == 0) s_sb = 0.0f;
    }
    __syncthreads();
    const float SB = s_sb * pl.stepsbk;
    if (nested) {
        for (int t = threadIdx.x; t < n1; t += BS) b1[t] = b1[t] + b2[d.MG12[t]] + SB;
        __syncthreads();
    }
    float sabs = 0.0f;            // FP32 per thread, double-float across threads (as in k_ts_cells)
    // PR_U cells at a time: their loads are issued together, before the stores
    // of the group (a store of ST keeps later loads behind it)
    for (int c0 = threadIdx.x; c0 < nc; c0 += PR_U * BS) {
        if (c0 != (int)threadIdx.x) load(c0);
#pragma unroll
        for (int u = 0; u < PR_U; ++u) {
            if (c0 + u * BS >= nc) break;
            const float corr = nested ? b1[pb1[u]] : b1[pb1[u]] + b2[pb2[u]] + SB;
            const float DELTA = pst[u] * pstp[u] + corr * prs[u];
            *at(ST, pn[u]) = DELTA;
            sabs += fabsf(DELTA);
        }
    }
    if (want_abs) {
        const df t = block_sum<BS>(d.REDUCE_ORDER, df_of(sabs), shd);
        if (threadIdx.x == 0) V.pabs[j - 1] = t;
    }
}

// per-J-plane sum of |STORE| (after residual smoothing)
template <int BS>
__global__ void __launch_bounds__(BS, 1024 / BS) k_ts_plane_abs(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    __shared__ df shd[BS / 32];
    const VarSet &V = d.var[v0 + blockIdx.y];
    int j = blockIdx.x + 2;
    int nc = d.IMM1 * d.KMM1;
    float sf = 0.0f;
    for (int c = threadIdx.x; c < nc; c += BS) {
        int i = c % d.IMM1 + 1, k = c / d.IMM1 + 1;
        sf += fabsf(A3(V.ST, i, j, k));
    }
    const df s = block_sum<BS>(d.REDUCE_ORDER, df_of(sf), shd);
    if (threadIdx.x == 0) V.pabs[j - 1] = s;
}

// AVG_CHG / AVG_BLK with the reference's sequential REAL*4 sum (1501-1515)
__global__ void k_ts_avgblk_seq(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    __shared__ float chg[64];
    const VarSet &V = d.var[v0 + blockIdx.y];
    if (!d.ctl->damp_on) return;
    int NROWS = d.NROWS;
    for (int nr = threadIdx.x + 1; nr <= NROWS; nr += blockDim.x) {
        int JST = A1(d.JSTART, nr) + 1, JEN = A1(d.JMIX, nr) - 1;
        int NSUM = d.IMM1 * d.KMM1 * (JEN - JST + 1);
        float SUMCHG = 0.0f;
        for (int k = 1; k <= d.KMM1; ++k)
            for (int j = JST; j <= JEN; ++j)
                for (int i = 1; i <= d.IMM1; ++i) SUMCHG = SUMCHG + fabsf(A3(V.ST, i, j, k));
        chg[nr - 1] = SUMCHG / (float)NSUM;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float *B = V.AVG_BLK;
        if (NROWS == 1) B[0] = chg[0];
        if (NROWS == 2) {
            B[1] = 0.5f * (chg[0] + chg[1]);
            B[0] = B[1];
        }
        if (NROWS > 2) {
            for (int nr = 2; nr <= NROWS - 1; ++nr) B[nr - 1] = 0.25f * (chg[nr - 2] + chg[nr]) + 0.5f * chg[nr - 1];
            B[NROWS - 1] = 0.5f * (chg[NROWS - 2] + chg[NROWS - 1]);
            B[0] = 0.5f * (chg[0] + chg[1]);
        }
    }
}

// ---------------------------------------------------------------------
// the row's mean |STORE| after the mixing with its neighbour rows (1501-1515)
// ---------------------------------------------------------------------
__device__ inline float row_mean(const float *chg, int nr, int NROWS) {
    if (NROWS == 1) return chg[0];
    if (NROWS == 2 || nr == 1) return 0.5f * (chg[0] + chg[1]);
    if (nr == NROWS) return 0.5f * (chg[NROWS - 2] + chg[NROWS - 1]);
    return 0.25f * (chg[nr - 2] + chg[nr]) + 0.5f * chg[nr - 1];
}

// ---------------------------------------------------------------------
// update: negative feedback, second MP average, corner gather -> TMP.
//
// A CTA owns R successive node planes and a tile of K rows, all of I: one
// thread a column of UP_S nodes along K at one I, marching up J.  It damps the
// cell changes of one plane ahead into shared memory (two plane tiles, one
// barrier a plane); the corner weights, which do not depend on J, stay in
// registers, and so do the cells beside the thread's column, which serve the
// two node planes beside their plane.  So a cell is damped
// (1 + 1/R)(1 + 1/rows) times, where a CTA per plane pair damped it 1.5 times
// and read each weight and cell again for every plane, at 230 instructions a
// node.  The next plane's cells are in flight during the current one's gather.
// Cells outside the grid are zeros in shared memory.
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(UP_T, 3) k_ts_update(const __grid_constant__ Dev d, int v0, int rows, int ntile, int R) {
    pdl_wait();
    extern __shared__ float sm[];
    const VarSet &V = d.var[v0 + blockIdx.y];
    const float *__restrict__ D = V.D;
    const float *__restrict__ ST = V.ST;
    float *__restrict__ TM = V.TM;
    __shared__ float s_blk[UP_R + 1], s_fd[UP_R + 1], s_fu[UP_R + 1], s_chg[64];
    __shared__ int s_role[UP_R + 1], s_jmx[UP_R + 1];
    const int IM = d.IM, JM = d.JM, IMM1 = d.IMM1, KM = d.KM, KMM1 = d.KMM1;
    const int tile = blockIdx.x % ntile, ja = (int)(blockIdx.x / ntile) * R + 1;
    const int jb = min(ja + R - 1, JM), k0 = 1 + tile * rows;
    const int tid = threadIdx.x, seg = tid / IM, il = tid - seg * IM;     // I = il + 1
    const int PW = IM + 1, buf = (rows + 1) * PW;     // cell (i, k) at i + PW * (k - k0 + 1), i = 0 .. IM
    const bool act = seg * UP_S < rows;
    const int damp_on = d.ctl->damp_on;
    const float DAMP = d.ctl->DAMP;
    for (int t = tid; t < 2 * buf; t += blockDim.x) sm[t] = 0.0f;
    const int ks = IM * JM, kb = k0 + seg * UP_S;       // this thread's nodes: K = kb .. kb + UP_S - 1
    const int nn = il + IM * (ja - 1) + ks * (kb - 1);  // node (il + 1, ja, kb)
    int kn = act ? min(UP_S, min(k0 + rows, KM + 1) - kb) : 0;
    if (kn < 0) kn = 0;
    const bool ci = act && il < IMM1;                    // this thread has cells
    const bool c0 = ci && seg == 0 && k0 >= 2;           // and the row below the tile
    float wtr[UP_S], wtl[UP_S], wbr[UP_S], wbl[UP_S];
#pragma unroll
    for (int q = 0; q < UP_S; ++q) {
        const int k = kb + q, o = il + IM * (k - 1);
        const bool on = q < kn, hL = il >= 1, hR = il < IMM1, hD = k >= 2, hU = k <= KMM1;
        wtr[q] = on && hL && hD ? d.FTR[o - 1 - IM] : 0.0f;
        wtl[q] = on && hR && hD ? d.FTL[o - IM] : 0.0f;
        wbr[q] = on && hL && hU ? d.FBR[o - 1] : 0.0f;
        wbl[q] = on && hR && hU ? d.FBL[o] : 0.0f;
    }
    // cell changes of plane jc into this thread's registers
    float st[UP_S + 1], dv[UP_S];
    auto load_cells = [&](int jc) {
        const int n = nn + IM * (jc - ja);
        const bool pl = jc >= 2 && jc <= JM;
#pragma unroll
        for (int q = 0; q < UP_S; ++q)
            if (pl && ci && q < kn && kb + q <= KMM1) st[q] = ST[n + ks * q];
        if (pl && c0) st[UP_S] = ST[n - ks];
    };
    auto load_nodes = [&](int j) {
#pragma unroll
        for (int q = 0; q < UP_S; ++q)
            if (q < kn) dv[q] = D[nn + IM * (j - ja) + ks * q];
    };
    // the flow's direction on row r of the tile, in a plane at a mixing plane
    auto flow = [&](int p, int r) {
        const int k = k0 - 1 + r;
        const bool mp = s_role[p] == 1 || s_role[p] == 3;
        return mp && r <= rows && k >= 1 && k <= KMM1 ? -A3(d.FLOWX, d.IMID, s_jmx[p], k) : 0.0f;
    };
    // damped cells of plane jc = ja + p into its tile; fdir: the direction on
    // this thread's first row
    auto damp_cells = [&](int p, float fdir) {
        const int jc = ja + p;
        float *c = sm + (p & 1) * buf + il + 1;
        const bool pl = jc >= 2 && jc <= JM;
        const float blk = s_blk[p];
        const int role = s_role[p], nrow = rows + 1;
        const bool mp = role == 1 || role == 3;
        auto damped = [&](float v) {
            if (!damp_on) return v;
            const float FDAMP = fabsf(v) / blk;
            return v / (1.0f + FDAMP / DAMP);
        };
#pragma unroll
        for (int q = 0; q < UP_S; ++q)
            if (ci && q < kn && kb + q <= KMM1) c[PW * (seg * UP_S + q + 1)] = pl ? damped(st[q]) : 0.0f;
        if (c0) c[0] = pl ? damped(st[UP_S]) : 0.0f;
        __syncthreads();
        if (!mp) return;
        // second pitchwise average on the mixing-plane cells (1850)
        const bool lowx = d.FEXTRAP < 0.001f;
        float *row0 = sm + (p & 1) * buf + 1;
        auto averaged = [&](int r, float FLOWDIRN) {
            const int k = k0 - 1 + r;
            return k >= 1 && k <= KMM1 &&
                   (role == 3 ? (FLOWDIRN > 0.0f || lowx) : (FLOWDIRN < 0.0f || lowx));
        };
        if (d.REDUCE_ORDER != 0) {
            for (int r = tid; r < nrow; r += (int)blockDim.x) {
                if (!averaged(r, flow(p, r))) continue;
                float *row = row0 + r * PW;
                const float m = mp_line_sum(row, IMM1) / (float)IMM1;
                for (int i = 0; i < IMM1; ++i) row[i] = m;
            }
        } else {
            for_rows(nrow, [&](int r, int l, bool on) {
                on = on && averaged(r, r == tid / ROW_LANES ? fdir : flow(p, r));
                if (!__any_sync(0xffffffffu, on)) return;
                float *row = row0 + r * PW;
                const int n = on ? IMM1 : 0;
                const float m = row_sum64(n, [&](int i) { return row[i]; }) / (float)IMM1;
                for (int i = l; i < n; i += ROW_LANES) row[i] = m;
            });
        }
        __syncthreads();
    };
    // the cells beside this thread's nodes, column I-1 and I, from the row
    // below its first node to the row above its last
    float ca[UP_S + 1][2], cb[UP_S + 1][2];
    auto read_cells = [&](int p, float (*o)[2]) {
        const float *c = sm + (p & 1) * buf + il + PW * (seg * UP_S);
#pragma unroll
        for (int q = 0; q <= UP_S; ++q) {
            o[q][0] = c[PW * q];
            o[q][1] = c[PW * q + 1];
        }
    };
    load_cells(ja);
    // the row means of |STORE| (1501-1515) that this CTA's cell planes take,
    // from the planes' sums: a warp a row and its neighbour rows
    if (damp_on && d.REDUCE_ORDER != 1) {
        const int w = tid >> 5, l = tid & 31, nw = (int)blockDim.x >> 5, ro = d.REDUCE_ORDER;
        const int r0 = max(d.PLANE[ja - 1].nrow - 1, 1), r1 = min(d.PLANE[min(jb + 1, JM) - 1].nrow + 1, d.NROWS);
        for (int nr = r0 + w; nr <= r1; nr += nw) {
            const int JST = A1(d.JSTART, nr) + 1, JEN = A1(d.JMIX, nr) - 1;
            df s = df_of(0.0f);
            for (int jj = JST + l; jj <= JEN; jj += 32) s = dacc(ro, s, V.pabs[jj - 1]);
            for (int o = 16; o > 0; o >>= 1) s = dacc(ro, s, df_shfl_down(s, o));
            if (l == 0) s_chg[nr - 1] = df_val(s) / (float)(IMM1 * KMM1 * (JEN - JST + 1));
        }
    }
    __syncthreads();                       // the zeroed tiles and the rows' sums
    // per cell plane jc = ja + q: the row mean, the mixing-plane role and the
    // streamwise weights it has in the node planes before and after it
    for (int q = tid; q <= jb - ja + 1; q += blockDim.x) {
        const int jc = ja + q;
        const PlaneInfo &pl = d.PLANE[min(jc, JM) - 1];
        if (jc >= 2 && jc <= JM) {
            s_blk[q] = !damp_on ? 1.0f : d.REDUCE_ORDER == 1 ? V.AVG_BLK[pl.nrow - 1]
                                                             : row_mean(s_chg, pl.nrow, d.NROWS);
            s_fu[q] = pl.facup;
            s_role[q] = pl.role;
        } else {
            s_blk[q] = 1.0f;
            s_fu[q] = 0.0f;
            s_role[q] = 0;
        }
        s_fd[q] = jc <= JM ? pl.facdwn : 0.0f;
        s_jmx[q] = pl.jmx;
    }
    __syncthreads();
    damp_cells(0, flow(0, tid / ROW_LANES));
    load_cells(ja + 1);
    float fdir = flow(1, tid / ROW_LANES);
    load_nodes(ja);
    if (act) read_cells(0, ca);
    // not unrolled: two planes an iteration save the register moves but run
    // out of the instruction cache (62.5 us a launch against 59.7 on the
    // 73 x 752 x 57 compressor, 23.9 against 23.6 at 65 x 242 x 49)
#pragma unroll 1
    for (int j = ja; j <= jb; ++j) {
        const int p = j - ja;
        damp_cells(p + 1, fdir);
        if (j < jb) {
            load_cells(j + 2);
            fdir = flow(p + 2, tid / ROW_LANES);
        }
        if (!act) continue;
        read_cells(p + 1, cb);
        const float fd = s_fd[p], fu = s_fu[p + 1];
        float *tm = TM + nn + IM * p;
        if (fd == 1.0f && fu == 1.0f) {            // all planes but the first and the last two
#pragma unroll
            for (int q = 0; q < UP_S; ++q) {
                float v = dv[q];
                v = v + ca[q][0] * wtr[q];
                v = v + ca[q][1] * wtl[q];
                v = v + cb[q][0] * wtr[q];
                v = v + cb[q][1] * wtl[q];
                v = v + ca[q + 1][0] * wbr[q];
                v = v + ca[q + 1][1] * wbl[q];
                v = v + cb[q + 1][0] * wbr[q];
                v = v + cb[q + 1][1] * wbl[q];
                if (q < kn) tm[ks * q] = v;
            }
        } else {
#pragma unroll
            for (int q = 0; q < UP_S; ++q) {
                float v = dv[q];
                v = v + ca[q][0] * wtr[q] * fd;
                v = v + ca[q][1] * wtl[q] * fd;
                v = v + cb[q][0] * wtr[q] * fu;
                v = v + cb[q][1] * wtl[q] * fu;
                v = v + ca[q + 1][0] * wbr[q] * fd;
                v = v + ca[q + 1][1] * wbl[q] * fd;
                v = v + cb[q + 1][0] * wbr[q] * fu;
                v = v + cb[q + 1][1] * wbl[q] * fu;
                if (q < kn) tm[ks * q] = v;
            }
        }
        if (j < jb) load_nodes(j + 1);
#pragma unroll
        for (int q = 0; q <= UP_S; ++q) {
            ca[q][0] = cb[q][0];
            ca[q][1] = cb[q][1];
        }
    }
}

// ---------------------------------------------------------------------
// update over a pair of node planes: the same result as k_ts_update for
// node planes j0 and j0+1, from one CTA of PBS threads, for planes so small
// that a CTA's threads cover the three cell planes at once: on 9 x 7 points
// 10.4 us a launch against 14.3 for k_ts_update, whose march damps one plane
// after the other; on 37 x 33 points k_ts_update is the faster one.  The CTA
// damps the cell planes j0, j0+1, j0+2 once each, and each thread gathers the
// same (i, k) on both node planes.  Every value is formed by the same
// expressions in the same order as in k_ts_update.
// ---------------------------------------------------------------------
template <int PBS>
__global__ void __launch_bounds__(PBS, 1024 / PBS) k_ts_update_pair(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    extern __shared__ float sm[];
    const VarSet &V = d.var[v0 + blockIdx.y];
    const float *__restrict__ D = V.D;
    float *__restrict__ TM = V.TM;
    __shared__ float s_blk[64];
    __shared__ float chg[64];
    const int j0 = 2 * blockIdx.x + 1;
    const int IM = d.IM, JM = d.JM, IMM1 = d.IMM1, KM = d.KM, KMM1 = d.KMM1;
    const int nc = IMM1 * KMM1;
    const bool two = j0 + 1 <= JM;              // the second node plane exists
    const DevCtl *ctl = d.ctl;
    const int damp_on = ctl->damp_on;
    const float DAMP = ctl->DAMP;
    const int ks = IM * JM;
    // this thread's first cell of each cell plane, and what the planes are,
    // before the row means below: the loads' latency overlaps theirs
    float pre[3];
    int prow[3], role[3], jmx[3];
    {
        const int k = (int)threadIdx.x / IMM1, n = (int)threadIdx.x - k * IMM1 + ks * k;
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const int jc = j0 + h;
            const bool in = jc >= 2 && jc <= JM;
            const PlaneInfo &pl = d.PLANE[min(jc, JM) - 1];
            prow[h] = pl.nrow;
            role[h] = in ? pl.role : 0;
            jmx[h] = pl.jmx;
            pre[h] = in && (int)threadIdx.x < nc ? V.ST[n + IM * (jc - 1)] : 0.0f;
        }
    }
    if (damp_on) {
        if (d.REDUCE_ORDER == 1) {
            for (int r = threadIdx.x; r < d.NROWS; r += PBS) s_blk[r] = V.AVG_BLK[r];
        } else {
            const int ro = d.REDUCE_ORDER;
            int w = threadIdx.x >> 5, l = threadIdx.x & 31;
            for (int nr = w + 1; nr <= d.NROWS; nr += PBS / 32) {
                int JST = A1(d.JSTART, nr) + 1, JEN = A1(d.JMIX, nr) - 1;
                df s = df_of(0.0f);
                for (int jj = JST + l; jj <= JEN; jj += 32) s = dacc(ro, s, V.pabs[jj - 1]);
                for (int o = 16; o > 0; o >>= 1) s = dacc(ro, s, df_shfl_down(s, o));
                if (l == 0) chg[nr - 1] = df_val(s) / (float)(IMM1 * KMM1 * (JEN - JST + 1));
            }
            __syncthreads();
            for (int r = threadIdx.x; r < d.NROWS; r += PBS) s_blk[r] = row_mean(chg, r + 1, d.NROWS);
        }
        __syncthreads();
    }
    // damped cell changes of the cell planes j0, j0+1, j0+2 (those in 2..JM),
    // and the flow's direction on this thread's first row of a mixing plane
    float fdir[3];
#pragma unroll
    for (int h = 0; h < 3; ++h) {
        const int jc = j0 + h;
        const int k = (int)threadIdx.x / ROW_LANES + 1;
        fdir[h] = (role[h] == 1 || role[h] == 3) && k <= KMM1 ? -A3(d.FLOWX, d.IMID, jmx[h], k) : 0.0f;
        if (jc < 2 || jc > JM) continue;
        float *c = sm + h * nc;
        const float blk = damp_on ? s_blk[prow[h] - 1] : 1.0f;
        auto damped = [&](float v) {
            if (!damp_on) return v;
            const float FDAMP = fabsf(v) / blk;
            return v / (1.0f + FDAMP / DAMP);
        };
        if ((int)threadIdx.x < nc) c[threadIdx.x] = damped(pre[h]);
        if (nc <= PBS) continue;
        const float *__restrict__ stp = V.ST + IM * (jc - 1);
        Walk2 w(IMM1, threadIdx.x + PBS, PBS);
        for (int t0 = threadIdx.x + PBS; t0 < nc; t0 += TS_UG * PBS) {
            float sv[TS_UG];
#pragma unroll
            for (int u = 0; u < TS_UG; ++u) {
                if (t0 + u * PBS < nc) sv[u] = stp[(w.i - 1) + ks * (w.k - 1)];
                w.next();
            }
#pragma unroll
            for (int u = 0; u < TS_UG; ++u) {
                const int t = t0 + u * PBS;
                if (t >= nc) break;
                c[t] = damped(sv[u]);
            }
        }
    }
    __syncthreads();
    // second pitchwise average on the mixing-plane cells (1850)
    const bool lowx = d.FEXTRAP < 0.001f;
    bool any = false;
#pragma unroll 1
    for (int h = 0; h < 3; ++h) {
        const int rl = h == 0 ? role[0] : h == 1 ? role[1] : role[2], jm = h == 0 ? jmx[0] : h == 1 ? jmx[1] : jmx[2];
        if (rl != 1 && rl != 3) continue;
        any = true;
        float *c = sm + h * nc;
        const float f0 = h == 0 ? fdir[0] : h == 1 ? fdir[1] : fdir[2];
        auto averaged = [&](int k) {
            const float FLOWDIRN =
                k == (int)threadIdx.x / ROW_LANES + 1 ? f0 : -A3(d.FLOWX, d.IMID, jm, k);
            return rl == 3 ? (FLOWDIRN > 0.0f || lowx) : (FLOWDIRN < 0.0f || lowx);
        };
        if (d.REDUCE_ORDER != 0) {
            for (int k = threadIdx.x + 1; k <= KMM1; k += PBS) {
                if (!averaged(k)) continue;
                float *row = c + (k - 1) * IMM1;
                const float s = mp_line_sum(row, IMM1) / (float)IMM1;
                for (int i = 0; i < IMM1; ++i) row[i] = s;
            }
        } else {
            for_rows(KMM1, [&](int r, int l, bool on) {
                on = on && averaged(r + 1);
                if (!__any_sync(0xffffffffu, on)) return;
                float *row = c + r * IMM1;
                const int n = on ? IMM1 : 0;
                const float s = row_sum64(n, [&](int i) { return row[i]; }) / (float)IMM1;
                for (int i = l; i < n; i += ROW_LANES) row[i] = s;
            });
        }
    }
    if (any) __syncthreads();
    // gather (1100) on both node planes
    const float *c0 = sm, *c1 = sm + nc, *c2 = sm + 2 * nc;
    const float fdn0 = A1(d.FACDWN, j0), fup0 = two ? A1(d.FACUP, j0 + 1) : 0.0f;
    const float fdn1 = two ? A1(d.FACDWN, j0 + 1) : 0.0f;
    const float fup1 = j0 + 2 <= JM ? A1(d.FACUP, j0 + 2) : 0.0f;
    const bool hA0 = j0 >= 2, hB0 = two;         // cell planes of node plane j0
    const bool hB1 = j0 + 2 <= JM;               // node plane j0 + 1 always has its cell plane j0 + 1
    const float *__restrict__ FBL = d.FBL;
    const float *__restrict__ FBR = d.FBR;
    const float *__restrict__ FTL = d.FTL;
    const float *__restrict__ FTR = d.FTR;
    const int nb0 = IM * (j0 - 1);
    // one node of a node plane from its <= 8 cells (kc, h, ic), cA the cell
    // plane before it and cB the one after, added in the reference's order
    // (kc outer, then the plane, then ic); a cell outside the grid is
    // skipped.  One thread per column of UG_SEG nodes along K at one I, the
    // lanes on successive I: walking up the column, the cells above a node
    // are the cells below the next one, so each cell value is read from
    // shared memory once per column and the boundary nodes take the same
    // predicated path as the inner ones
    const bool pv0 = hA0, pv1 = two, pv2 = hB1;  // cell planes j0, j0 + 1, j0 + 2 present
    const int nsk = (KM + UG_SEG - 1) / UG_SEG;
    Walk2 w(IM, threadIdx.x, PBS);
    for (int t = threadIdx.x; t < IM * nsk; t += PBS, w.next()) {
        const int i = w.i, k0 = 1 + UG_SEG * (w.k - 1);
        const int len = min(UG_SEG, KM - k0 + 1);
        const bool hL = i >= 2, hR = i <= IMM1;
        // the global operands of the column's nodes, loaded together
        float dv0[UG_SEG], dv1[UG_SEG], wtr[UG_SEG], wtl[UG_SEG], wbr[UG_SEG], wbl[UG_SEG];
#pragma unroll
        for (int q = 0; q < UG_SEG; ++q) {
            if (q >= len) break;
            const int k = k0 + q;
            const int n = nb0 + (i - 1) + ks * (k - 1);
            const bool hD = k >= 2, hU = k <= KMM1;
            dv0[q] = D[n];
            dv1[q] = two ? D[n + IM] : 0.0f;
            wtr[q] = (hL && hD) ? FTR[(i - 2) + IM * (k - 2)] : 0.0f;
            wtl[q] = (hR && hD) ? FTL[(i - 1) + IM * (k - 2)] : 0.0f;
            wbr[q] = (hL && hU) ? FBR[(i - 2) + IM * (k - 1)] : 0.0f;
            wbl[q] = (hR && hU) ? FBL[(i - 1) + IM * (k - 1)] : 0.0f;
        }
        // cells (i-1, r) and (i, r) of the three cell planes, r = the cell
        // row below the node (dn) and above it (up)
        float dn0l = 0.0f, dn0r = 0.0f, dn1l = 0.0f, dn1r = 0.0f, dn2l = 0.0f, dn2r = 0.0f;
        const int cl = i - 2;                       // cell (i-1, r) at cl + IMM1*(r-1)
        if (k0 >= 2) {
            const int o = cl + IMM1 * (k0 - 2);
            if (pv0 && hL) dn0l = c0[o];
            if (pv0 && hR) dn0r = c0[o + 1];
            if (pv1 && hL) dn1l = c1[o];
            if (pv1 && hR) dn1r = c1[o + 1];
            if (pv2 && hL) dn2l = c2[o];
            if (pv2 && hR) dn2r = c2[o + 1];
        }
#pragma unroll
        for (int q = 0; q < UG_SEG; ++q) {
            if (q >= len) break;
            const int k = k0 + q;
            const bool hD = k >= 2, hU = k <= KMM1;
            float up0l = 0.0f, up0r = 0.0f, up1l = 0.0f, up1r = 0.0f, up2l = 0.0f, up2r = 0.0f;
            if (hU) {
                const int o = cl + IMM1 * (k - 1);
                if (pv0 && hL) up0l = c0[o];
                if (pv0 && hR) up0r = c0[o + 1];
                if (pv1 && hL) up1l = c1[o];
                if (pv1 && hR) up1r = c1[o + 1];
                if (pv2 && hL) up2l = c2[o];
                if (pv2 && hR) up2r = c2[o + 1];
            }
            const int n = nb0 + (i - 1) + ks * (k - 1);
            // node plane j0: cell planes j0 and j0 + 1
            float v = dv0[q];
            if (hD) {
                if (hA0 && hL) v = v + dn0l * wtr[q] * fdn0;
                if (hA0 && hR) v = v + dn0r * wtl[q] * fdn0;
                if (hB0 && hL) v = v + dn1l * wtr[q] * fup0;
                if (hB0 && hR) v = v + dn1r * wtl[q] * fup0;
            }
            if (hU) {
                if (hA0 && hL) v = v + up0l * wbr[q] * fdn0;
                if (hA0 && hR) v = v + up0r * wbl[q] * fdn0;
                if (hB0 && hL) v = v + up1l * wbr[q] * fup0;
                if (hB0 && hR) v = v + up1r * wbl[q] * fup0;
            }
            TM[n] = v;
            if (two) {
                // node plane j0 + 1: cell planes j0 + 1 and j0 + 2
                float v1 = dv1[q];
                if (hD) {
                    if (hL) v1 = v1 + dn1l * wtr[q] * fdn1;
                    if (hR) v1 = v1 + dn1r * wtl[q] * fdn1;
                    if (hB1 && hL) v1 = v1 + dn2l * wtr[q] * fup1;
                    if (hB1 && hR) v1 = v1 + dn2r * wtl[q] * fup1;
                }
                if (hU) {
                    if (hL) v1 = v1 + up1l * wbr[q] * fdn1;
                    if (hR) v1 = v1 + up1r * wbl[q] * fdn1;
                    if (hB1 && hL) v1 = v1 + up2l * wbr[q] * fup1;
                    if (hB1 && hR) v1 = v1 + up2r * wbl[q] * fup1;
                }
                TM[n + IM] = v1;
            }
            dn0l = up0l; dn0r = up0r; dn1l = up1l; dn1r = up1r; dn2l = up2l; dn2r = up2r;
        }
    }
}

// How update is cut: segments of UP_S rows per CTA (its threads are IM a
// segment, at most UP_T), the number of K tiles and the planes per CTA.  The
// segments minimise the lanes and rows that a cut leaves idle or damps twice.
// The planes minimise the launch's length, waves of CTAs times a march of R
// planes and about one and a half more for its start: the smallest grids take
// one plane a CTA (one load, one barrier, one store), a grid that fills the
// GPU as many as make whole waves.
struct UpdateCut {
    int rows, ntile, R, threads;
    size_t smem;
};
static UpdateCut update_cut(const Dev &d, int sm_count, int nv) {
    UpdateCut c{};
    double best = 1e30;
    for (int ns = 1; ns * d.IM <= UP_T && (ns == 1 || (ns - 1) * UP_S < d.KM || ns * UP_S <= d.TS_ROWS); ++ns) {
        if (d.TS_ROWS && ns * UP_S != d.TS_ROWS) continue;
        const int rows = ns * UP_S, nt = (d.KM + rows - 1) / rows, th = (ns * d.IM + 31) / 32 * 32;
        const double cost = (double)nt * (rows + 1) * th / (ns * d.IM);
        if (cost < best) {
            best = cost;
            c.rows = rows;
            c.ntile = nt;
            c.threads = th;
        }
    }
    const long long slots = (long long)sm_count * (65536 / (72 * c.threads));
    best = 1e30;
    for (int R = 1; R <= UP_R; ++R) {
        if (d.TS_PLANES && R != d.TS_PLANES) continue;
        const long long ctas = (long long)((d.JM + R - 1) / R) * c.ntile * nv;
        const double cost = (double)((ctas + slots - 1) / slots) * (R + 1.5);
        if (cost < best) {
            best = cost;
            c.R = R;
        }
    }
    c.smem = (size_t)2 * (c.rows + 1) * (d.IM + 1) * sizeof(float);
    return c;
}

// Two FP32 values in one instruction (PTX .f32x2), each rounded as the scalar
// operation is.  A product is a*b + nz with nz = -0, which is a*b to the bit: a
// mul.f32x2 whose result only an add.f32x2 takes comes out as one fused
// operation, with one rounding less than the reference has, and so does a
// product with a -0 that the assembler can see.
#define MGPU_BITS(v) reinterpret_cast<unsigned long long &>(v)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(MGPU_BITS(a)), "l"(MGPU_BITS(b)));
    return reinterpret_cast<float2 &>(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(MGPU_BITS(a)), "l"(MGPU_BITS(b)));
    return reinterpret_cast<float2 &>(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b, float2 nz) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(MGPU_BITS(a)), "l"(MGPU_BITS(b)), "l"(MGPU_BITS(nz)));
    return reinterpret_cast<float2 &>(r);
}

// ---------------------------------------------------------------------
// smooth: SMOOTH_VAR (3900-9000, 8502) + periodic (8000), tip gap (510),
// mixing-plane average (100): TMP -> D, one CTA per J-plane
// ---------------------------------------------------------------------
template <int BS>
__global__ void __launch_bounds__(BS, 1024 / BS) k_ts_smooth(const __grid_constant__ Dev d, int v0) {
    pdl_wait();
    extern __shared__ float sm[];
    const VarSet &V = d.var[v0 + blockIdx.y];
    const float *__restrict__ S = V.TM;
    float *__restrict__ D = V.D;
    const int IM = d.IM, KM = d.KM, IMM1 = d.IMM1, KMM1 = d.KMM1;
    const int np = IM * KM;
    // the plane buffers hold (i, k) at (i-1) + IMP*(k-1); the odd row pitch
    // keeps the pitchwise pass, whose lanes step from one K line to the
    // next, free of bank conflicts
    const int IMP = IM | 1;
    float *a = sm + SM_PAD, *b = a + IMP * KM;
    // FD, FU, FKD, FKU, each twice: the operand of two lanes of arithmetic
    float2 *cFD = reinterpret_cast<float2 *>(sm + SM_PAD + 2 * IMP * KM), *cFU = cFD + IM, *cFKD = cFU + IM, *cFKU = cFKD + KM;
    const int j = blockIdx.x + 1;
    const PlaneInfo &pl = d.PLANE[j - 1];
    const DevCtl *c = d.ctl;
    const bool stream = !(c->SFX < 0.0001f), mix = pl.mix != 0;
    // the pitchwise weight that this thread puts into shared memory for a
    // mixing plane's average, ahead of its use
    const float fpw = mix && (int)threadIdx.x < IMM1 ? d.FP[threadIdx.x] : 0.0f;
    for (int t = threadIdx.x; t < IM; t += BS) {
        const float fd = d.FD[t], fu = d.FU[t];
        cFD[t] = make_float2(fd, fd);
        cFU[t] = make_float2(fu, fu);
    }
    for (int t = threadIdx.x; t < KM; t += BS) {
        const float fd = d.FKD[t], fu = d.FKU[t];
        cFKD[t] = make_float2(fd, fd);
        cFKU[t] = make_float2(fu, fu);
    }
    const int ks = IM * d.JM;                        // K stride of a node array
    const float *__restrict__ Sj = S + IM * (j - 1);  // plane j: (i, k) at i-1 + ks*(k-1)
    {
        const int sc = stream ? pl.sc : 0, lc = stream ? pl.lc : 0;
        const int J1 = pl.J1, J2 = pl.J2;
        const float SFX = c->SFX, SFX1 = c->SFX1, SFXB = c->SFXB, SFXB1 = c->SFXB1, SFXBH = c->SFXBH;
        const float SFXHM1 = c->SFXHM1, SFX14 = c->SFX14, F4 = d.FAC_4TH;
        // the J planes each case reads, as node offsets from plane j
        int nq = 0;
        ptrdiff_t off[4] = {0, 0, 0, 0};
        auto add = [&](int jj) { off[nq++] = (ptrdiff_t)IM * (jj - j); };
        if (sc == 1) { add(j + 1); add(j - 1); add(j - 2); add(j + 2); }
        if (sc == 2) { add(J1 + 3); add(J1 + 1); }
        if (sc == 3) { add(J1 + 2); add(J1 + 3); add(J1 + 4); }
        if (sc == 4) { add(J2 - 1); add(J2 - 3); }
        if (sc == 5) { add(J2 - 2); add(J2 - 3); add(J2 - 4); }
        Walk2 w(IM, threadIdx.x, BS);
        for (int t0 = threadIdx.x; t0 < np; t0 += SV_U * BS) {
            float d0[SV_U], x[SV_U][4];
            int pi[SV_U], pk[SV_U];
#pragma unroll
            for (int u = 0; u < SV_U; ++u) {
                pi[u] = w.i;
                pk[u] = w.k;
                w.next();
                if (t0 + u * BS < np) {
                    const float *p = Sj + (pi[u] - 1) + ks * (pk[u] - 1);
                    d0[u] = p[0];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (q < nq) x[u][q] = p[off[q]];
                }
            }
#pragma unroll
            for (int u = 0; u < SV_U; ++u) {
                const int t = t0 + u * BS;
                if (t >= np) break;
                const int i = pi[u], k = pk[u];
                const float dd = d0[u];
                float v = dd;
                switch (sc) {
                case 1: {
                    float AVERG = 0.5f * (x[u][0] + x[u][1]);
                    float CURV = AVERG - 0.5f * dd - 0.25f * (x[u][2] + x[u][3]);
                    v = SFX1 * dd + SFX * (AVERG + F4 * CURV);
                    break;
                }
                case 2: case 4: v = SFXB1 * dd + SFXBH * (x[u][0] + x[u][1]); break;
                case 3: case 5: v = SFXB1 * dd + SFXB * (1.25f * x[u][0] + 0.5f * x[u][1] - 0.75f * x[u][2]); break;
                default: break;
                }
                if (lc && (i == 1 || i == IM)) {
                    const float *pkk = Sj + ks * (k - 1);
                    if (lc == 1) v = SFXHM1 * dd + SFX14 * (pkk[1] + pkk[IMM1 - 1]);
                    else if (i == 1) v = SFXHM1 * dd + SFX14 * (pkk[IM + 0] + pkk[IM - 1]);
                    else v = SFXHM1 * dd + SFX14 * (pkk[IM + IM - 1] + pkk[0]);
                }
                a[(i - 1) + IMP * (k - 1)] = v;
            }
        }
    }
    __syncthreads();
#define P(buf, i, k) buf[((i) - 1) + IMP * ((k) - 1)]
    const bool periodic_j = pl.periodic != 0;
    if (j >= 2 && !(c->SFT < 0.0001f)) {
        const float SFT = c->SFT, SFT1 = c->SFT1, F4 = d.FAC_4TH;
        const float2 SFT2 = make_float2(SFT, SFT), SFT12 = make_float2(SFT1, SFT1), F42 = make_float2(F4, F4);
        // Two lines a thread, in the two halves of f32x2 operations: the pass
        // is bound by its instructions on a large grid (218 a node with one
        // line a thread), and the weights, the tests for a line's ends and the
        // arithmetic are shared.  59.9 -> 57.3 us a launch on the 73 x 752 x 57
        // compressor, 11.0 -> 10.5 on the 33 x 97 x 37 row, the same at
        // 65 x 242 x 49 (segments of 6 points 61.1, of 8 points 72.5: spills).
        // one segment of SM_SEG points of two lines: x(q) gives points
        // first - 2 + q of both, FD and FU the weights of point first - 1 + q,
        // e the curvature at a line's two ends; out(q, v) takes the new points
        // -0, as the launch's (one-dimensional) block hides it
        const float nz1 = __uint_as_float(0x80000000u + (blockDim.y - 1u));
        const float2 nz = make_float2(nz1, nz1);
        auto mul = [&](float2 u, float2 v) { return mul2(u, v, nz); };
        auto segment = [&](auto x_of, const float2 *FD, const float2 *FU, float2 e, bool begins, int last, auto out) {
            float2 x[SM_SEG + 4], g[SM_SEG + 2];
#pragma unroll
            for (int q = 0; q < SM_SEG + 4; ++q) x[q] = x_of(q);
#pragma unroll
            for (int q = 0; q < SM_SEG + 2; ++q)
                g[q] = sub2(x[q + 1], add2(mul(FD[q], x[q + 2]), mul(FU[q], x[q])));
            if (begins) g[0] = e;
            if (last <= SM_SEG + 1)
#pragma unroll
                for (int q = 2; q < SM_SEG + 2; ++q)
                    if (q == last) g[q] = e;
#pragma unroll
            for (int q = 0; q < SM_SEG; ++q) {
                const float2 fd = FD[q + 1], fu = FU[q + 1];
                const float2 AVG = add2(mul(fd, x[q + 3]), mul(fu, x[q + 1]));
                const float2 SC = add2(mul(fu, g[q]), mul(fd, g[q + 2]));
                out(q, add2(mul(SFT12, x[q + 2]), mul(SFT2, add2(AVG, mul(F42, SC)))));
            }
        };
        // the points I = 2..IMM1 first, in segments of SM_SEG points of two K
        // lines half the plane apart per thread, the lanes on successive K
        // lines (an odd last line is done twice, with one result): each
        // point's curvature is formed once and the segment's values stay in
        // registers.  The curvature at I = 1 and IM, which the points I = 2
        // and IMM1 take, is one value per line (the reference's CURVE there
        // is the I = 1 value, or 0 off the periodic planes).  What a segment
        // reads past its line's end lies in the plane buffers and is not used
        const int KH = (KM + 1) / 2, nsi = (IM - 2 + SM_SEG - 1) / SM_SEG;
        Walk2 w(KH, threadIdx.x, BS);
        for (int t = threadIdx.x; t < nsi * KH; t += BS, w.next()) {
            const int k = w.i, k2 = min(k + KH, KM), i0 = 2 + SM_SEG * (w.k - 1);
            const int len = min(SM_SEG, IMM1 - i0 + 1);
            const float *a1 = a + IMP * (k - 1), *a2 = a + IMP * (k2 - 1);
            float2 cper = make_float2(0.0f, 0.0f);
            if (periodic_j)
                cper = make_float2(a1[0] - 0.5f * (a1[1] + a1[IMM1 - 1]), a2[0] - 0.5f * (a2[1] + a2[IMM1 - 1]));
            float *b1 = b + IMP * (k - 1) + i0 - 1, *b2 = b + IMP * (k2 - 1) + i0 - 1;
            const float *p1 = a1 + i0 - 3, *p2 = a2 + i0 - 3;
            segment([&](int q) { return make_float2(p1[q], p2[q]); }, cFD + i0 - 2, cFU + i0 - 2, cper, i0 == 2,
                    IM - (i0 - 1), [&](int q, float2 v) {
                        if (q < len) {
                            b1[q] = v.x;
                            b2[q] = v.y;
                        }
                    });
        }
        // then the points I = 1 and IM of every line
        for (int t = threadIdx.x; t < 2 * KM; t += BS) {
            const int i = (t & 1) ? IM : 1, k = (t >> 1) + 1;
            const float *ak = a + IMP * (k - 1) - 1;
            float AVG, SC;
            if (periodic_j) {
                AVG = 0.5f * (ak[2] + ak[IMM1]);
                const float c2 = ak[2] - (cFD[1].x * ak[3] + cFU[1].x * ak[1]);
                const float cm1 = ak[IMM1] - (cFD[IMM1 - 1].x * ak[IM] + cFU[IMM1 - 1].x * ak[d.IMM2]);
                SC = 0.5f * (c2 + cm1);
            } else {
                if (i == 1) AVG = ak[2] + cFU[0].x * (ak[2] - ak[3]);
                else AVG = ak[IMM1] + cFU[IM - 1].x * (ak[IMM1] - ak[d.IMM2]);
                SC = 0.0f;
            }
            P(b, i, k) = SFT1 * ak[i] + SFT * (AVG + F4 * SC);
        }
        __syncthreads();
        // spanwise: the points K = 2..KMM1 in segments of two I lines half the
        // plane apart, the lanes on successive I lines; the curvature at K = 1
        // and KM is zero
        const int IH = (IM + 1) / 2, nsk = (KM - 2 + SM_SEG - 1) / SM_SEG;
        w = Walk2(IH, threadIdx.x, BS);
        for (int t = threadIdx.x; t < nsk * IH; t += BS, w.next()) {
            const int i = w.i, i2 = min(i + IH, IM), k0 = 2 + SM_SEG * (w.k - 1);
            const int len = min(SM_SEG, KMM1 - k0 + 1);
            const float *p1 = b + (i - 1) + IMP * (k0 - 3), *p2 = p1 + (i2 - i);
            float *a1 = a + (i - 1) + IMP * (k0 - 1), *a2 = a1 + (i2 - i);
            segment(
                [&](int q) {
                    const bool in = q < 4 || k0 - 2 + q <= KM;
                    return make_float2(in ? p1[IMP * q] : 0.0f, in ? p2[IMP * q] : 0.0f);
                },
                cFKD + k0 - 2, cFKU + k0 - 2, make_float2(0.0f, 0.0f), k0 == 2, KM - (k0 - 1), [&](int q, float2 v) {
                    if (q < len) {
                        a1[IMP * q] = v.x;
                        a2[IMP * q] = v.y;
                    }
                });
        }
        // then the points K = 1 and KM of every line
        for (int t = threadIdx.x; t < 2 * IM; t += BS) {
            const int i = (t >> 1) + 1, k = (t & 1) ? KM : 1, k1 = (t & 1) ? KMM1 : 2, k2 = (t & 1) ? d.KMM2 : 3;
            const float y1 = k1 >= 1 ? P(b, i, k1) : 0.0f, y2 = k2 >= 1 && k2 <= KM ? P(b, i, k2) : 0.0f;
            const float AVG = y1 + 0.5f * cFKU[k - 1].x * (y1 - y2), SC = 0.0f;
            P(a, i, k) = SFT1 * P(b, i, k) + SFT * (AVG + F4 * SC);
        }
        __syncthreads();
        float cv = 0.0f;
        if (threadIdx.x < 4) {
            const float SFTH = c->SFTH;
            if (threadIdx.x == 0) cv = SFT1 * P(a, 1, 1) + SFTH * (P(a, 2, 1) + P(a, 1, 2));
            else if (threadIdx.x == 1) cv = SFT1 * P(a, IM, 1) + SFTH * (P(a, IMM1, 1) + P(a, IM, 2));
            else if (threadIdx.x == 2) cv = SFT1 * P(a, 1, KM) + SFTH * (P(a, 1, KMM1) + P(a, 2, KM));
            else cv = SFT1 * P(a, IM, KM) + SFTH * (P(a, IMM1, KM) + P(a, IM, KMM1));
        }
        __syncthreads();
        if (threadIdx.x == 0) P(a, 1, 1) = cv;
        else if (threadIdx.x == 1) P(a, IM, 1) = cv;
        else if (threadIdx.x == 2) P(a, 1, KM) = cv;
        else if (threadIdx.x == 3) P(a, IM, KM) = cv;
        __syncthreads();
    }
    if (!(d.SFEXIT < 0.0001f) && j >= d.JM + 1 - d.NSFEXIT) {
        const float SE = d.SFEXIT, SE1 = 1.0f - SE, SEH = 0.5f * SE;
        for (int k = threadIdx.x + 1; k <= KM; k += BS) {
            for (int i = 2; i <= IMM1; ++i) P(a, i, k) = SE1 * P(a, i, k) + SEH * (P(a, i + 1, k) + P(a, i - 1, k));
            P(a, 1, k) = P(a, 1, k) + SE * (2.0f * P(a, 2, k) - P(a, 3, k) - P(a, 1, k));
            P(a, IM, k) = P(a, IM, k) + SE * (2.0f * P(a, IMM1, k) - P(a, d.IMM2, k) - P(a, IM, k));
        }
        __syncthreads();
        for (int i = threadIdx.x + 1; i <= IM; i += BS) {
            for (int k = 2; k <= KMM1; ++k) P(a, i, k) = SE1 * P(a, i, k) + SEH * (P(a, i, k - 1) + P(a, i, k + 1));
            P(a, i, 1) = P(a, i, 1) + SE * (2.0f * P(a, i, 2) - P(a, i, 3) - P(a, i, 1));
            P(a, i, KM) = P(a, i, KM) + SE * (2.0f * P(a, i, KMM1) - P(a, i, d.KMM2) - P(a, i, KM));
        }
        __syncthreads();
    }
    for (int k = threadIdx.x + 1; k <= KM; k += BS) {
        if (periodic_j) {
            float v = 0.5f * (P(a, 1, k) + P(a, IM, k));
            P(a, 1, k) = v;
            P(a, IM, k) = v;
        }
        if (k >= pl.tip1 && k <= pl.tip2) {
            float v = 0.5f * (P(a, 1, k) + P(a, IM, k));
            P(a, 1, k) = v;
            P(a, IM, k) = v;
        }
    }
    float *fp = reinterpret_cast<float *>(cFU);       // the smoothing is done with it
    if (mix)
        for (int i = threadIdx.x; i < IMM1; i += BS) fp[i] = i < BS ? fpw : d.FP[i];
    __syncthreads();
    float *Dj = D + IM * (j - 1);
    if (mix) {
        if (d.REDUCE_ORDER != 0) {
            for (int k = threadIdx.x + 1; k <= KM; k += BS) {
                float s = 0.0f;
                for (int i = 1; i <= IMM1; ++i) s = s + fp[i - 1] * (P(a, i, k) + P(a, i + 1, k));
                b[k - 1] = 0.5f * s;
            }
        } else {
            for_rows(KM, [&](int r, int l, bool on) {
                const float *row = a + IMP * r;
                const float s = row_sum64(on ? IMM1 : 0, [&](int i) { return fp[i] * (row[i] + row[i + 1]); });
                if (on && l == 0) b[r] = 0.5f * s;
            });
        }
        __syncthreads();
        Walk2 w(IM, threadIdx.x, BS);
        for (int t = threadIdx.x; t < np; t += BS, w.next()) Dj[(w.i - 1) + ks * (w.k - 1)] = b[w.k - 1];
        return;
    }
#undef P
    Walk2 w(IM, threadIdx.x, BS);
    for (int t = threadIdx.x; t < np; t += BS, w.next()) Dj[(w.i - 1) + ks * (w.k - 1)] = a[(w.i - 1) + IMP * (w.k - 1)];
}

// ---------------------------------------------------------------------
// SMOOTH_RESID (14833-14917): one Jacobi pass along J, I or K of the cell
// changes inside each row, src -> dst (cells outside every row are copied)
// ---------------------------------------------------------------------
__global__ void k_resid_pass(const __grid_constant__ Dev d, int v0, int dir, float smfac, int st_to_tm) {
    pdl_wait();
    const VarSet &V = d.var[v0 + blockIdx.y];
    const float *__restrict__ src = st_to_tm ? V.ST : V.TM;
    float *__restrict__ dst = st_to_tm ? V.TM : V.ST;
    size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t N = (size_t)d.IM * d.JM * d.KM;
    if (n >= N) return;
    int i, j, k;
    node_ijk(d, n, i, j, k);
    if (i >= d.IM || j < 2 || k >= d.KM) return;
    float SFAC1 = 1.0f - smfac, SFACH = 0.5f * smfac;
    int nr = A1(d.NROW, j);
    int J1P1 = A1(d.JSTART, nr) + 1, J1P2 = J1P1 + 1, J2 = A1(d.JMIX, nr), J2M1 = J2 - 1;
    float v = src[n];
    if (j < J1P1 || j > J2) {
        dst[n] = v;
        return;
    }
#define S(ii, jj, kk) A3(src, ii, jj, kk)
    if (dir == 0) {
        if (j >= J1P2 && j <= J2M1) v = SFAC1 * v + SFACH * (S(i, j + 1, k) + S(i, j - 1, k));
        if (j == J1P1) v = S(i, J1P1, k) + SFACH * (S(i, J1P2, k) - S(i, J1P1, k));
        if (j == J2) v = S(i, J2, k) + SFACH * (S(i, J2M1, k) - S(i, J2, k));
    } else if (dir == 1) {
        int IMM1 = d.IMM1, IMM2 = d.IMM2;
        if (i >= 2 && i <= IMM2) v = SFAC1 * v + SFACH * (S(i + 1, j, k) + S(i - 1, j, k));
        if (i == 1) v = S(1, j, k) + SFACH * (S(2, j, k) - S(1, j, k));
        if (i == IMM1) v = S(IMM1, j, k) + SFACH * (S(IMM2, j, k) - S(IMM1, j, k));
    } else {
        int KMM1 = d.KMM1, KMM2 = d.KMM2;
        if (k >= 2 && k <= KMM2) v = SFAC1 * v + SFACH * (S(i, j, k + 1) + S(i, j, k - 1));
        if (k == 1) v = S(i, j, 1) + SFACH * (S(i, j, 2) - S(i, j, 1));
        if (k == KMM1) v = S(i, j, KMM1) + SFACH * (S(i, j, KMM2) - S(i, j, KMM1));
    }
#undef S
    dst[n] = v;
}

// STORE = TMP after the three SMOOTH_RESID passes
__global__ void k_copy_tm_st(const __grid_constant__ Dev d, int v0, size_t n) {
    pdl_wait();
    const VarSet &V = d.var[v0 + blockIdx.y];
    size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) V.ST[t] = V.TM[t];
}

// k_ts_update_pair where a 512-thread CTA covers a plane's points (TS_PAIR = 0:
// never).  us a step with the march and with the pair, on 98 planes: 63 points
// 77.5 and 73.5, 130 75.6 and 73.5, 289 76.7 and 73.9, 400 77.6 and 77.0, 506 78.0
// and 77.5, 672 78.8 and 82.1, 1221 91.1 and 93.9; on 50 and 194 planes the line
// lies there too.  On 322 planes, more pairs than one wave, the march is the
// faster one at every size (63 points 96.3 and 98.7, 506 109 and 113).
static bool pair_update(const Dev &d) { return d.TS_PAIR && d.IM * d.KM <= 512; }

static size_t cells_smem(const Dev &d) {
    return ((size_t)d.IMM1 * d.KMM1 + 2 * d.KMM1 + d.IMM1 + (size_t)d.NIB1 * d.NKB1) * sizeof(float);
}
static size_t prolong_smem(const Dev &d) { return ((size_t)d.NIB1 * d.NKB1 + (size_t)d.NIB2 * d.NKB2) * sizeof(float); }
static size_t update_pair_smem(const Dev &d) { return (size_t)3 * d.IMM1 * d.KMM1 * sizeof(float); }
static size_t smooth_smem(const Dev &d) {
    return ((size_t)2 * (d.IM | 1) * d.KM + 4 * (d.IM + d.KM) + SM_PAD + 4 * SM_SEG) * sizeof(float);
}

template <int BS>
static cudaError_t configure_bs(const Dev &d) {
    struct {
        const void *f;
        size_t bytes;
    } k[] = {{(const void *)k_ts_cells<BS>, cells_smem(d)},
             {(const void *)k_ts_prolong<BS>, prolong_smem(d)},
             {(const void *)k_ts_update_pair<2 * BS>, update_pair_smem(d)},
             {(const void *)k_ts_smooth<BS>, smooth_smem(d)}};
    // the limit is on what a plane takes: the smoothing weights' second copies
    // and the paddings (2.6 KB at IM = KM = 160) come on top.  The three planes
    // of the pair update bound every problem (IMM1 KMM1 <= 17066), though the
    // kernel itself runs on small planes only
    const size_t extra = (2 * (size_t)(d.IM + d.KM) + SM_PAD + 4 * SM_SEG) * sizeof(float);
    for (auto &x : k) {
        if (x.bytes - (x.f == (const void *)k_ts_smooth<BS> ? extra : 0) > 200 * 1024) return cudaErrorInvalidValue;
        cudaError_t e = raise_smem(x.f, x.bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t configure_kernels(const Dev &d) {
    cudaError_t e = configure_bs<128>(d);
    if (e == cudaSuccess) e = configure_bs<256>(d);
    if (e == cudaSuccess) e = configure_bs<192>(d);
    if (e == cudaSuccess) e = configure_bs<512>(d);
    if (e == cudaSuccess) e = configure_loss_kernels(d);
    return e != cudaSuccess ? e : configure_flux_kernels(d);
}

// TSTEP up to the negative feedback's row means: flux sum, SCREE and the
// mixing-plane redistribution (cells), the multigrid block sums and the
// time step (prolong), SMOOTH_RESID of STORE, and |STORE| per plane (or,
// with REDUCE_ORDER=1, the row means in the reference's order)
template <int BS>
static void launch_tstep_front(const Dev &d, Launch L, int v0, int nv) {
    size_t N = (size_t)d.IM * d.JM * d.KM;
    unsigned gN = grid_for(N, 256);
    const bool seq = d.REDUCE_ORDER == 1;
    const unsigned jp = (unsigned)(d.JM - 1), vy = (unsigned)nv;
    launchk(L, k_ts_cells<BS>, dim3(jp, vy), dim3(BS), cells_smem(d), d, v0);
    mark(L, "k_ts_cells");
    if (seq) {
        int nb = d.NIB1 * (d.NJB1 + 1) * d.NKB1 + d.NIB2 * (d.NJB2 + 1) * d.NKB2 + d.NSBLK;
        launchk(L, k_ts_restrict_seq, dim3(grid_for(nb, 64), vy), dim3(64), 0, d, v0);
        mark(L, "k_ts_restrict_seq");
    }
    launchk(L, k_ts_prolong<BS>, dim3(jp, vy), dim3(BS), prolong_smem(d), d, v0, (d.NRSMTH == 0 && !seq) ? 1 : 0);
    mark(L, "k_ts_prolong");
    if (d.NRSMTH > 0) {
        for (int it = 0; it < d.NRSMTH; ++it) {
            launchk(L, k_resid_pass, dim3(gN, vy), dim3(256), 0, d, v0, 0, d.RSMTH, 1);
            mark(L, "k_resid_pass");
            launchk(L, k_resid_pass, dim3(gN, vy), dim3(256), 0, d, v0, 1, d.RSMTH, 0);
            mark(L, "k_resid_pass");
            launchk(L, k_resid_pass, dim3(gN, vy), dim3(256), 0, d, v0, 2, d.RSMTH, 1);
            mark(L, "k_resid_pass");
            launchk(L, k_copy_tm_st, dim3(gN, vy), dim3(256), 0, d, v0, N);
            mark(L, "k_copy_tm_st");
        }
        if (!seq) {
            launchk(L, k_ts_plane_abs<BS>, dim3(jp, vy), dim3(BS), 0, d, v0);
            mark(L, "k_ts_plane_abs");
        }
    }
    if (seq) {
        launchk(L, k_ts_avgblk_seq, dim3(1, vy), dim3(32), 0, d, v0);
        mark(L, "k_ts_avgblk_seq");
    }
}

template <int BS>
static void launch_tstep_bs(const Dev &d, Launch L, int v0, int nv) {
    launch_tstep_front<BS>(d, L, v0, nv);
    const unsigned ja = (unsigned)d.JM, vy = (unsigned)nv;
    if (pair_update(d)) {
        launchk(L, k_ts_update_pair<2 * BS>, dim3((ja + 1) / 2, vy), dim3(2 * BS), update_pair_smem(d), d, v0);
        mark(L, "k_ts_update_pair");
    } else {
        const UpdateCut u = update_cut(d, L.sm_count, nv);
        launchk(L, k_ts_update, dim3((ja + u.R - 1) / u.R * u.ntile, vy), dim3(u.threads), u.smem, d, v0, u.rows, u.ntile,
                u.R);
        mark(L, "k_ts_update");
    }
    launchk(L, k_ts_smooth<BS>, dim3(ja, vy), dim3(BS), smooth_smem(d), d, v0);
    mark(L, "k_ts_smooth");
}

void launch_tstep_cells_prolong(const Dev &d, Launch L, int v0, int nv) {
    const int bs = d.ts_bs[0];
    if (bs == 128) launch_tstep_front<128>(d, L, v0, nv);
    else if (bs == 192) launch_tstep_front<192>(d, L, v0, nv);
    else if (bs == 512) launch_tstep_front<512>(d, L, v0, nv);
    else launch_tstep_front<256>(d, L, v0, nv);
}

void launch_tstep(const Dev &d, Launch L, int v0, int nv) {
    const int bs = d.ts_bs[nv >= 3 ? 1 : 0];
    if (bs == 128) launch_tstep_bs<128>(d, L, v0, nv);
    else if (bs == 192) launch_tstep_bs<192>(d, L, v0, nv);
    else if (bs == 512) launch_tstep_bs<512>(d, L, v0, nv);
    else launch_tstep_bs<256>(d, L, v0, nv);
}

}  // namespace mgpu
