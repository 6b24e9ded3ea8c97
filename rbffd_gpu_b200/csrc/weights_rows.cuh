// Row-per-thread elimination of the batched weight solves (included by
// weights.cu, inside its namespace): one system per CTA of NW warps, thread t
// holding rows t + 32 NW r (r < RPT) of the current 8-column panel in
// registers, the rest of the augmented matrix [A | B] column-major in shared
// memory (element (i, j) at a[j * lda + i], so a warp's rows of one column are
// consecutive).  Per panel of 8 columns:
//   8 steps: each warp finds its first maximum |a_ik| (a warp-wide integer
//     maximum over the values' high words, the low words and dgetf2's smaller
//     row position where those tie) and publishes the row's panel values and
//     the value's reciprocal; one CTA barrier; every thread picks the winner,
//     forms its multiplier and updates its own panel row;
//   the panel rows of U over the trailing columns, one column per thread (the
//     unit lower triangle solved in step order), stored over the panel's own
//     columns, which nobody needs any more (8 doubles per trailing column);
//   every remaining row takes the 8 delayed updates of each trailing column on
//     the FP64 tensor cores: a warp's rows as 8-row tiles, two m8n8k4 products
//     per 8 x 8 tile.  That instruction accumulates its four products as a
//     chain of fused multiply-adds in ascending k (checked bit for bit by the
//     tests against the eliminations that spell the chain out).
// Rows are not exchanged; each keeps its dgetf2 position for the tie rule.
// When a row becomes the pivot, the row in the last slot is given its slot, so
// that after a panel the rows left over are stored (by the trailing update)
// into consecutive slots, and warps without rows skip the work.  Pivots,
// multipliers and the order of every element's fused updates are dgetf2's, so
// the result is team_eliminate's bit for bit.
//
// What bounds it: the chain of dependent instructions through a step (about
// 930 cycles at m = 116: the maximum, the published row, the barrier, the
// multiplier, the update), two systems of 114 KB per SM.  Cycles per m = 116
// system (three operators): assembly 34k, panels 108k, U rows 14k, trailing
// updates 54k, back substitution 41k.  432 ns per system on a full device
// against 801 ns with the whole row updated in every step by team_eliminate,
// which passes over the trailing matrix 116 times instead of 15.
#pragma once

constexpr int PANEL = 8;
constexpr int TRI = PANEL * (PANEL + 1) / 2;  // packed upper triangle of a panel

// Slots per column: at least the rows, and 8 columns must hold a panel's U
// rows over the columns after it plus its triangle (8 (m + K - 8) + 36 doubles);
// odd, so one slot of consecutive columns falls in different banks.
__host__ __device__ inline int rows_lda(int m, int K) { return (m > m + K - 3 ? m : m + K - 3) | 1; }

// Doubles of shared memory besides the matrix: the assembly's coordinates and
// frame, later the elimination's scratch (the same space).
__host__ __device__ inline int rows_scratch(int m, int K, int n_pad, int nw)
{
    const int elim = PANEL * K + TRI + 2 * nw * (4 + PANEL) + PANEL * PANEL + PANEL / 2 + (m + 1) / 2 + m + 4;
    const int asmb = 3 * n_pad + 8;
    return elim > asmb ? elim : asmb;
}

__host__ __device__ inline size_t rows_smem_bytes(int m, int K, int n_pad, int nw)
{
    return ((size_t)rows_lda(m, K) * (m + K) + 2 + rows_scratch(m, K, n_pad, nw)) * sizeof(double);
}

// Offset of U(k0 + s, k0 + t), s <= t, in a panel's packed triangle.
__device__ __forceinline__ int tri_off(int s, int t) { return s * PANEL - s * (s - 1) / 2 + (t - s); }

// Place of U(k0 + s, .) among the 8 doubles of the trailing column that is
// number jj after the panel: pairs of columns alternate their halves, so the
// tensor-core operand (4 steps of 8 columns) reads all 32 banks twice.
__device__ __forceinline__ int u_place(int s, int jj) { return s ^ ((jj & 2) << 1); }

// a / b, correctly rounded, from y = 1 / b correctly rounded: a quotient within
// one unit in the last place corrected once by its exact residual is the
// rounded quotient (Markstein, IBM J. Res. Dev. 34(1), 1990, theorem 8.5 for
// fused multiply-add); the first correction brings a * y within that unit.
// Where b or a is far from 1 (underflowing residuals, infinities, NaN, zero b)
// the division itself.
__device__ __forceinline__ double div_by_reciprocal(double a, double b, double y)
{
    const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu, hb = (unsigned)__double2hiint(b) & 0x7fffffffu;
    constexpr unsigned LO = (1023u - 400u) << 20, SPAN = 800u << 20;  // 2^-400 .. 2^400
    const double q0 = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-q0, b, a), y, q0);
    const double q2 = __fma_rn(__fma_rn(-q1, b, a), y, q1);
    const bool in = hb - LO < SPAN && (ha - LO < SPAN || a == 0.0);
    if (!in) return a / b;
    return a == 0.0 ? q0 : q2;
}

// c += a b over four steps: lane l holds a(l / 4, l % 4), b(l % 4, l / 4) and c(l / 4, 2 (l % 4) + {0, 1}).
__device__ __forceinline__ void dmma_8x8x4(double& c0, double& c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

template <int NW>
__device__ __forceinline__ void rows_sync()
{
    if (NW == 1)
        __syncwarp();
    else
        __syncthreads();
}

// A warp's published pivot candidate.
struct RowsCand {
    unsigned hi, lo;  // |value|
    int place;        // dgetf2 position | slot the row will be stored in << 16
    int slot;         // slot it is read from
    double y, pad;    // 1 / value
};

// The elimination's views of the scratch space.
template <int NW>
struct RowsScratch {
    double* tail;    // the last panel's U over the right-hand sides [K][8], then its triangle
    RowsCand* cand;  // [2][NW]
    double* rows;    // [2][NW][8] the candidates' panel rows
    double* dg;      // [8][8] the panel's pivot rows: multipliers below the diagonal, U on and above
    int* pslot;      // [8] slots of the panel's pivot rows
    double* y;       // [m] 1 / u_kk
    int* pos;        // [m] dgetf2 position of each slot's row
    __device__ RowsScratch(double* s, int m, int K)
    {
        const int t = (PANEL * K + TRI + 1) & ~1;  // 16-byte alignment of what follows
        tail = s;
        cand = reinterpret_cast<RowsCand*>(s + t);
        rows = s + t + 8 * NW;
        dg = rows + 2 * NW * PANEL;
        pslot = (int*)(dg + PANEL * PANEL);
        y = dg + PANEL * PANEL + PANEL / 2;
        pos = (int*)(y + m);
    }
};

// 0, or k + 1 when the pivot column of step k is exactly zero (or NaN).
template <int NW, int RPT>
__device__ int rows_eliminate(double* a, double* scratch, int m, int K, int lda)
{
    constexpr int TH = 32 * NW;
    constexpr unsigned FULL = 0xffffffffu;
    const RowsScratch<NW> S(scratch, m, K);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int ld = m + K;
    int par = 0;
    for (int k0 = 0; k0 < m; k0 += PANEL) {
        const int na = m - k0, pw = min(PANEL, na), kend = k0 + pw;  // rows left: slots 0 .. na - 1
        const int nwa = min(NW, (na + 31) >> 5);                     // warps that hold any
        double v[RPT][PANEL];
        int pos[RPT], dst[RPT];  // dgetf2 position; slot after this panel, -1 - s once pivot of step s
        bool act[RPT];
#pragma unroll
        for (int r = 0; r < RPT; r++) {
            const int slot = tid + TH * r;
            act[r] = slot < na;
            dst[r] = slot;
            pos[r] = k0 == 0 ? slot : (act[r] ? S.pos[slot] : 0);
#pragma unroll
            for (int c = 0; c < PANEL; c++) v[r][c] = act[r] && c < pw ? a[(k0 + c) * lda + slot] : 0.0;
        }
#pragma unroll
        for (int s = 0; s < PANEL; s++) {
            if (s >= pw) break;
            const int k = k0 + s;
            RowsCand* const cand = S.cand + par * NW;
            double* const rows = S.rows + par * NW * PANEL;
            par ^= 1;
            if (w < nwa) {
                // this thread's, then the warp's first maximum of column k (NaN never a candidate)
                unsigned hi = 0, lo = 0;
                int br = -1, bp = 0;
                double bv = 1.0;
#pragma unroll
                for (int r = 0; r < RPT; r++) {
                    const unsigned h = (unsigned)__double2hiint(v[r][s]) & 0x7fffffffu;
                    const unsigned l = (unsigned)__double2loint(v[r][s]);
                    if (act[r] && v[r][s] == v[r][s] &&
                        (br < 0 || h > hi || (h == hi && (l > lo || (l == lo && pos[r] < bp))))) {
                        hi = h;
                        lo = l;
                        br = r;
                        bp = pos[r];
                        bv = v[r][s];
                    }
                }
                const double y = __drcp_rn(bv == 0.0 ? 1.0 : bv);
                const unsigned mh = __reduce_max_sync(FULL, hi);
                bool best = br >= 0 && hi == mh;
                const unsigned same = __ballot_sync(FULL, best);
                if (same & (same - 1)) {  // high words tie (or are all zero): the low words, then the positions
                    const unsigned ml = __reduce_max_sync(FULL, best ? lo : 0u);
                    best = best && lo == ml;
                    const unsigned mp = __reduce_min_sync(FULL, best ? (unsigned)bp : FULL);
                    best = best && (unsigned)bp == mp;
                } else if (same == 0 && lane == 0) {
                    cand[w].hi = cand[w].lo = 0;  // every active value of the warp is NaN
                    cand[w].place = 0xffff;
                }
                if (best) {
                    int place = 0, slot = tid;
#pragma unroll
                    for (int r = 0; r < RPT; r++)
                        if (r == br) {
                            place = pos[r] | dst[r] << 16;
                            slot = tid + TH * r;
                        }
                    *reinterpret_cast<uint4*>(&cand[w]) = make_uint4(hi, lo, (unsigned)place, (unsigned)slot);
                    cand[w].y = y;
                    double2* const d2 = reinterpret_cast<double2*>(rows + w * PANEL);
#pragma unroll
                    for (int c = s & ~1; c < PANEL; c += 2) {
                        double x0 = v[0][c], x1 = v[0][c + 1];
#pragma unroll
                        for (int r = 1; r < RPT; r++)
                            if (r == br) {
                                x0 = v[r][c];
                                x1 = v[r][c + 1];
                            }
                        d2[c / 2] = make_double2(x0, x1);
                    }
                }
            }
            rows_sync<NW>();
            // the pivot: first maximum over the warps, all candidates loaded at once
            uint4 g = *reinterpret_cast<const uint4*>(&cand[0]);
            int gw = 0;
            if (NW > 1) {
                uint4 h[NW];
#pragma unroll
                for (int q = 1; q < NW; q++) h[q] = *reinterpret_cast<const uint4*>(&cand[q]);
#pragma unroll
                for (int q = 1; q < NW; q++) {
                    const unsigned long long hk = (unsigned long long)h[q].x << 32 | h[q].y,
                                             gk = (unsigned long long)g.x << 32 | g.y;
                    if (q < nwa && (hk > gk || (hk == gk && (h[q].z & 0xffffu) < (g.z & 0xffffu)))) {
                        g = h[q];
                        gw = q;
                    }
                }
            }
            if ((g.x | g.y) == 0) return k + 1;
            if (w < nwa) {
                const int gpos = (int)(g.z & 0xffffu), gdst = (int)(g.z >> 16), gslot = (int)g.w;
                const int last = na - 1 - s;  // the last slot in use before this step
                const double y = cand[gw].y;
                double u[PANEL];
#pragma unroll
                for (int c = s & ~1; c < PANEL; c += 2) {
                    const double2 t = reinterpret_cast<const double2*>(rows + gw * PANEL)[c / 2];
                    u[c] = t.x;
                    u[c + 1] = t.y;
                }
#pragma unroll
                for (int r = 0; r < RPT; r++) {
                    if (tid + TH * r == gslot) {
                        act[r] = false;
                        dst[r] = -1 - s;
                        S.y[k] = y;
                    }
                    const double l = div_by_reciprocal(act[r] ? v[r][s] : 0.0, u[s], y);
                    if (act[r]) {
                        v[r][s] = l;
#pragma unroll
                        for (int c = s + 1; c < PANEL; c++) v[r][c] = __fma_rn(-l, u[c], v[r][c]);
                        if (pos[r] == k) pos[r] = gpos;  // dgetf2's exchange moves the row at position k to the pivot's
                        if (dst[r] == last) dst[r] = gdst;
                    }
                }
            }
        }
        // the pivot rows' panel values and slots
#pragma unroll
        for (int r = 0; r < RPT; r++)
            if (dst[r] < 0) {
                const int s = -1 - dst[r];
                S.pslot[s] = tid + TH * r;
#pragma unroll
                for (int c = 0; c < PANEL; c += 2)
                    reinterpret_cast<double2*>(S.dg + s * PANEL)[c / 2] = make_double2(v[r][c], v[r][c + 1]);
            }
        rows_sync<NW>();
        // U's rows k0 .. kend-1 beyond the panel, one column per thread
        const bool last = kend == m;
        double* const ub = last ? S.tail : a + k0 * lda;
        for (int j = kend + tid; j < ld; j += TH) {
            double x[PANEL];
            const int4 p0 = reinterpret_cast<const int4*>(S.pslot)[0], p1 = reinterpret_cast<const int4*>(S.pslot)[1];
            const int ps[PANEL] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int s = 0; s < PANEL; s++) x[s] = s < pw ? a[j * lda + ps[s]] : 0.0;
#pragma unroll
            for (int s = 1; s < PANEL; s++)
                if (s < pw)
#pragma unroll
                    for (int t = 0; t < s; t += 2) {
                        const double2 l = reinterpret_cast<const double2*>(S.dg + s * PANEL)[t / 2];
                        x[s] = __fma_rn(-l.x, x[t], x[s]);
                        if (t + 1 < s) x[s] = __fma_rn(-l.y, x[t + 1], x[s]);
                    }
            double2* const d2 = reinterpret_cast<double2*>(ub + (j - kend) * PANEL);
#pragma unroll
            for (int s = 0; s < PANEL; s += 2) d2[u_place(s, j - kend) / 2] = make_double2(x[s], x[s + 1]);
        }
        double* const tri = ub + (ld - kend) * PANEL;
        for (int e = tid; e < pw * PANEL; e += TH) {
            const int s = e / PANEL, t = e % PANEL;
            if (t >= s && t < pw) tri[tri_off(s, t)] = S.dg[e];
        }
        if (last) break;
        rows_sync<NW>();
        // the delayed updates of the remaining rows: each warp its own rows, as 8-row tiles
        if (w < nwa) {
            const int lr = lane >> 2, lc = lane & 3;
#pragma unroll
            for (int r = 0; r < RPT; r++) {
                const int row0 = TH * r + 32 * w;
                if (row0 >= na) break;
                if (act[r]) S.pos[dst[r]] = pos[r];
                double fa[4][2];  // -l of tile t's rows, steps 0-3 and 4-7
                int td[4];        // the tile's rows' slots after the update
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int src = 8 * t + lr;
                    td[t] = __shfl_sync(FULL, act[r] ? dst[r] : -1, src);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        double x = 0.0;
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const double z = __shfl_sync(FULL, v[r][4 * h + c], src);
                            if (c == lc) x = z;
                        }
                        fa[t][h] = -x;
                    }
                }
                const int nt = min(4, (na - row0 + 7) >> 3);
                for (int j = kend; j < ld; j += 8) {
                    const int jb = min(j + lr, ld - 1) - kend;  // past the last column: never stored
                    const double b0 = ub[jb * PANEL + u_place(lc, jb)], b1 = ub[jb * PANEL + u_place(lc + 4, jb)];
                    const int c0 = j + 2 * lc;
                    double* const p = a + c0 * lda;
                    const bool in0 = c0 < ld, in1 = c0 + 1 < ld;
                    double x[4][2];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const int i = row0 + 8 * t + lr;
                        x[t][0] = in0 && td[t] >= 0 ? p[i] : 0.0;
                        x[t][1] = in1 && td[t] >= 0 ? p[lda + i] : 0.0;
                    }
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (t < nt) {
                            dmma_8x8x4(x[t][0], x[t][1], fa[t][0], b0);
                            dmma_8x8x4(x[t][0], x[t][1], fa[t][1], b1);
                        }
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        if (in0 && td[t] >= 0) p[td[t]] = x[t][0];
                        if (in1 && td[t] >= 0) p[lda + td[t]] = x[t][1];
                    }
                }
            }
        }
        rows_sync<NW>();
    }
    rows_sync<NW>();
    return 0;
}

// Back substitution on the panel storage rows_eliminate leaves: KB right-hand
// sides per warp, lane l holding rows l + 32 q (q < BS).  Panel by panel from
// the last: every lane solves the panel's triangle (x_k = b_k / u_kk, then the
// rows above it in the panel), the rows of earlier panels then take the
// panel's updates b_i <- fma(-x_k, u_ik, b_i), k descending --
// back_substitute_bs's arithmetic.  out(c, i, x) receives the solution.
template <int NW, int BS, int KB, typename OutF>
__device__ void rows_back_substitute_t(const double* a, double* scratch, int m, int K, int lda, OutF out)
{
    const RowsScratch<NW> S(scratch, m, K);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ld = m + K;
    for (int c0 = w * KB; c0 < K; c0 += NW * KB) {
        const double* un[BS];  // row i's panel storage: U(i, k) at un[q][8 k + u_place(i % 8, k)]
        double b[KB][BS];
#pragma unroll
        for (int q = 0; q < BS; q++) {
            const int i = min(lane + 32 * q, m - 1), k0 = i & ~(PANEL - 1), ke = min(k0 + PANEL, m);
            un[q] = (ke == m ? S.tail : a + k0 * lda) - PANEL * ke;
#pragma unroll
            for (int c = 0; c < KB; c++) {
                const int j = m + min(c0 + c, K - 1);
                b[c][q] = un[q][PANEL * j + u_place(i & (PANEL - 1), j - ke)];
            }
        }
        for (int k0 = (m - 1) & ~(PANEL - 1); k0 >= 0; k0 -= PANEL) {
            const int ke = min(k0 + PANEL, m), pw = ke - k0, qk = k0 >> 5, l0 = k0 & 31;
            const double* tri = (ke == m ? S.tail : a + k0 * lda) + (ld - ke) * PANEL;
            double x[KB][PANEL];
#pragma unroll
            for (int c = 0; c < KB; c++) {
                double bq = b[c][0];
#pragma unroll
                for (int q = 1; q < BS; q++)
                    if (q == qk) bq = b[c][q];
#pragma unroll
                for (int s = 0; s < PANEL; s++) x[c][s] = __shfl_sync(0xffffffffu, bq, l0 + s);
            }
#pragma unroll
            for (int s = PANEL - 1; s >= 0; s--)
                if (s < pw) {
                    const double d = tri[tri_off(s, s)], y = S.y[k0 + s];
#pragma unroll
                    for (int c = 0; c < KB; c++) x[c][s] = div_by_reciprocal(x[c][s], d, y);
#pragma unroll
                    for (int t = 0; t < s; t++) {
                        const double u = tri[tri_off(t, s)];
#pragma unroll
                        for (int c = 0; c < KB; c++) x[c][t] = __fma_rn(-x[c][s], u, x[c][t]);
                    }
                }
#pragma unroll
            for (int q = 0; q < BS; q++)
                if (lane + 32 * q < k0) {
                    const double* u = un[q] + PANEL * k0;
                    const int s0 = lane & (PANEL - 1);
#pragma unroll
                    for (int s = PANEL - 1; s >= 0; s--)
                        if (s < pw) {
                            const double z = u[PANEL * s + u_place(s0, s)];  // panels before the last end at a multiple of 8
#pragma unroll
                            for (int c = 0; c < KB; c++) b[c][q] = __fma_rn(-x[c][s], z, b[c][q]);
                        }
                }
            const int s1 = lane - l0;
            if (s1 >= 0 && s1 < pw)
#pragma unroll
                for (int c = 0; c < KB; c++) {
                    double xv = x[c][0];
#pragma unroll
                    for (int s = 1; s < PANEL; s++)
                        if (s == s1) xv = x[c][s];
                    if (c0 + c < K) out(c0 + c, k0 + s1, xv);
                }
        }
    }
}

// KB right-hand sides at once per warp: as many as leave no warp with a second
// round, up to 3; a warp with more takes further rounds (8 operators on one warp: three).
template <int NW, int BS, typename OutF>
__device__ void rows_back_substitute(const double* a, double* scratch, int m, int K, int lda, OutF out)
{
    const int per = (K + NW - 1) / NW;
    if (per <= 1)
        rows_back_substitute_t<NW, BS, 1>(a, scratch, m, K, lda, out);
    else if (per == 2)
        rows_back_substitute_t<NW, BS, 2>(a, scratch, m, K, lda, out);
    else
        rows_back_substitute_t<NW, BS, 3>(a, scratch, m, K, lda, out);
}

// The systems of one size class, one per CTA at a time; CTAs take the next
// system from the class's counter.
template <int NW, int RPT, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_weights_rows(WParams P)
{
    extern __shared__ __align__(16) double smem_rows[];
    __shared__ int s_unit[2];
    const WClass C = P.cls[0];
    const int m = C.m, lda = C.lda, K = P.K;
    double* const a = smem_rows;
    double* const scratch = a + (((size_t)lda * (m + K) + 1) & ~(size_t)1);
    const Team T{(int)threadIdx.x, 32 * NW, 0};
    for (int it = 0;; it++) {
        if (threadIdx.x == 0) s_unit[it & 1] = atomicAdd(P.work, 1);
        __syncthreads();  // also: the previous system's shared memory is no longer read
        const int u = s_unit[it & 1];
        if (u >= P.nunits) break;
        const int r = P.rows[C.rows_off + u];
        int n;
        team_assemble<true>(T, P, r, a, scratch, scratch + 3 * P.n_pad, n, lda);
        const int st = rows_eliminate<NW, RPT>(a, scratch, m, K, lda);
        if (st != 0) {
            if (threadIdx.x == 0) atomicMin(P.status, r + 1);
            for (int e = threadIdx.x; e < K * P.n4; e += 32 * NW) {
                const int c = e / P.n4, j = e - c * P.n4;
                P.w[c][sell_elem(r, j, P.n4 >> 2)] = j < n ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
            }
            continue;
        }
        const int nc = P.n4 >> 2;
        rows_back_substitute<NW, NW * RPT>(a, scratch, m, K, lda, [&](int c, int j, double x) {
            // weights[type][r][j] = W(j, col) * scale (rbffd.cpp:300-306), row r of the sliced ELL
            if (j < n) P.w[c][sell_elem(r, j, nc)] = P.opbit[c] == RBFFD_HV ? x * P.hv_scale : x * 1.0;
        });
        for (int e = threadIdx.x; e < K * (P.n4 - n); e += 32 * NW) {  // padding slots
            const int c = e / (P.n4 - n), j = n + e - c * (P.n4 - n);
            P.w[c][sell_elem(r, j, nc)] = 0.0;
        }
    }
}
