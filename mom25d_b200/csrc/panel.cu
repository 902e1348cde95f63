// panel.cu - the LU's panel factorisation (GEPP of up to 64 columns, LAPACK's pivots) as one thread-block cluster.
//
// A panel is a chain of columns: what bounds it is the latency of one column's pivot search and exchange, not bytes or
// flops. How it is split:
//   - the panel's rows are split over the cluster's CTAs (up to 16), RPT rows a thread, and the columns are taken in
//     groups of GRP whose entries stay in the owner thread's registers: inside a group a column needs the pivot search,
//     the GRP entries of two rows exchanged, and nothing from memory;
//   - the exchange is by st.async into distributed shared memory, completion counted in bytes on the receiver's
//     mbarriers: every CTA sends its candidate's entry to every CTA; the winner's CTA then sends its row to all, the
//     diagonal row's CTA that row to the winner's. While the candidates travel, the rows that may be sent are made ready
//     and the other warps finish the column before; while the row travels, one warp forms the pivot's reciprocal. (Every
//     16-byte message costs the receiver an update of its mbarrier: sending every candidate's row along with it, one
//     trip a column instead of two, took 1.05 to 1.2 times as long.) What the warp of a CTA's candidate has to do in a
//     column is what a column takes, so the reciprocal (in f64 390 cycles) and the bookkeeping of the interchanges are
//     other warps' work (LUs 2 to 4% shorter at n = 2,000 to 6,000);
//   - the searches are integer redux over the bit patterns of |re| + |im| (non-negative: ordered as integers);
//   - at a group's end the group's interchanges are applied to the panel's other columns as one permutation and its
//     GRP rows of U are solved (a warp a column), then every thread updates its rows of the columns to the right: those
//     columns stay in global memory (L2), so the kernel holds no tiles in shared memory and fits beside the CTAs of a
//     trailing update on the same SM.
// The entries of a row in the registers rotate by one a column (the current column is entry 0, finished L entries come
// in at the end), so one loop body serves every column of a group.
// Every entry takes its terms a -= l u one at a time in column order, as an unblocked elimination does.
//
// 64 columns inside an LU: complex64 n = 4,977: 118 us, complex128 n = 2,921: 146 us; the panel kernel with its rows in
// shared memory (k_panel_smem) took 206 and 292 us there in a cluster of 16 and 258 to 303 us on 32 cooperative CTAs.
#include <algorithm>

#include "common.cuh"

namespace {
constexpr int PNONE = 0x7fffffff;          // no candidate
constexpr int PCL_MAX = 16;                // CTAs of a cluster (above 8: non-portable)
constexpr int PNB = 64;                    // columns of a panel at most

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t a, unsigned rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void send16(uint32_t dst, uint4 v, uint32_t bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void expect_bytes(uint32_t bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// waits for the phase of the barrier; bounded: false after about 2^20 tries or once a block reported a time-out
__device__ __forceinline__ bool wait_phase(uint32_t bar, unsigned parity, const int *err)
{
    for (long it = 1;; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((it & 255) == 0 && (it > (1L << 20) || *(volatile const int *)err == M25_DEV_TIMEOUT)) return false;
    }
}

// The largest value and its row over the warp (the smallest row on ties), in every lane; values are >= 0 where the
// row is not PNONE, so their bit patterns order as integers do.
__device__ __forceinline__ void warp_best(float &v, int &row)
{
    const unsigned k = row == PNONE ? 0u : __float_as_uint(v);
    const unsigned m = __reduce_max_sync(0xffffffffu, k);
    row = (int)__reduce_min_sync(0xffffffffu, k == m ? (unsigned)row : (unsigned)PNONE);
    v = __uint_as_float(m);
}
__device__ __forceinline__ void warp_best(double &v, int &row)
{
    const unsigned long long k = row == PNONE ? 0ull : (unsigned long long)__double_as_longlong(v);
    const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    row = (int)__reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)row : (unsigned)PNONE);
    v = __longlong_as_double((long long)(((unsigned long long)mh << 32) | ml));
}

__device__ __forceinline__ uint4 head_of(float v, int row) { return make_uint4(__float_as_uint(v), 0u, (unsigned)row, 0u); }
__device__ __forceinline__ uint4 head_of(double v, int row)
{
    const unsigned long long k = (unsigned long long)__double_as_longlong(v);
    return make_uint4((unsigned)k, (unsigned)(k >> 32), (unsigned)row, 0u);
}
__device__ __forceinline__ void of_head(uint4 h, float &v, int &row) { v = __uint_as_float(h.x); row = (int)h.z; }
__device__ __forceinline__ void of_head(uint4 h, double &v, int &row)
{
    v = __longlong_as_double((long long)(((unsigned long long)h.y << 32) | h.x));
    row = (int)h.z;
}

template <typename R> __device__ __forceinline__ cpx<R> ldc_l2(const R *p, size_t i)
{
    typedef typename vec2_of<R>::type V;
    const V v = __ldcg(reinterpret_cast<const V *>(p) + i);
    return mk<R>(v.x, v.y);
}

// the 16-byte piece `piece` of a row whose entry e is lane e's x (a warp's lanes together)
__device__ __forceinline__ uint4 piece_of(cpx<float> x, int piece)
{
    uint4 v;
    v.x = __float_as_uint(__shfl_sync(0xffffffffu, x.x, 2 * piece));
    v.y = __float_as_uint(__shfl_sync(0xffffffffu, x.y, 2 * piece));
    v.z = __float_as_uint(__shfl_sync(0xffffffffu, x.x, 2 * piece + 1));
    v.w = __float_as_uint(__shfl_sync(0xffffffffu, x.y, 2 * piece + 1));
    return v;
}
__device__ __forceinline__ uint4 piece_of(cpx<double> x, int)        // (an entry is a piece)
{
    uint4 v;
    memcpy(&v, &x, 16);
    return v;
}

template <typename R, int GRP> struct PanelShared {
    typedef cpx<R> C;
    typedef cpx_row<R, GRP> Entries;
    static constexpr int RB = Entries::PIECES;                        // 16-byte pieces of a row's GRP entries
    uint4 head[2][PCL_MAX];                  // each CTA's candidate's entry (NaN: none), by column parity
    struct Row { Entries row; uint4 p; } win[2];                      // the pivot row and its index
    uint4 rcp[2];                            // 1 / pivot
    int pos[32], src[32];                    // the group's interchanges (plan), for the other columns
    Entries diag[2];                         // the diagonal row, in the CTA of the pivot row
    struct Stage { Entries row; C l, next; } stage[2];                // a row on its way out: candidate, diagonal row
    C prow[GRP][GRP];                        // the group's pivot rows (rotated as they were sent)
    Entries u[PNB];                          // the group's rows of U on the columns to the right
    uint4 cand[2][16];                       // the warps' candidates, by column parity
    int fail[2];                             // a wait of this CTA gave up in the column before (by column parity)
    unsigned long long bar[4];               // of the candidates, then of the rows, by column parity
};

template <typename R, int GRP, int RPT, int T>
__global__ void __launch_bounds__(T, 1) k_panel_cluster(R *A, long lda, int n, int k0, int jb, int *ipiv, int *err)
{
    typedef cpx<R> C;
    typedef PanelShared<R, GRP> PS;
    constexpr int RB = PS::RB;
    __shared__ __align__(16) PS s;
    const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int nw = T / 32;
    const int cs = (n - k0 + G - 1) / G, r0 = k0 + b * cs, nr = max(0, min(n, r0 + cs) - r0);
    const int rend = r0 + nr;
    const uint32_t bar0 = smem_addr(&s.bar[0]);
    typename PS::Entries a[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int row = r0 + tid + T * r;
#pragma unroll
        for (int c = 0; c < GRP; ++c)
            a[r][c] = (row < rend && c < jb) ? ldc_l2<R>(A, (size_t)(k0 + c) * lda + row) : mk<R>(0, 0);
    }
    if (tid == 0) {
        s.fail[0] = s.fail[1] = 0;
        for (int q = 0; q < 4; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (G > 1) { cluster_arrive(); cluster_wait(); }
    bool dead = false;                                     // (block-uniform) after a failure: barriers only, to the end
    for (int g0 = 0; g0 < jb; g0 += GRP) {
        const int gw = min(GRP, jb - g0), gr = k0 + g0;    // the group's columns and its first row / column
        // the group's interchanges as a permutation, in the last warp's lanes: row pos ends with what row src held. Lanes
        // 0 .. GRP - 1: the group's own rows; lane GRP + j: the row below that column j's interchange touched first
        int pos = lane < gw ? gr + lane : -1, src = pos, plast = -1;
        R best = (R)-1;
        int bi = PNONE;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            const int row = r0 + tid + T * r;
            const R v = abs1(a[r][0]);
            if (row >= gr && row < rend && v > best) { best = v; bi = row; }
        }
        auto plan = [&](int jj) {                           // column jj's interchange with row plast
            if (plast == gr + jj) return;
            const unsigned m = __ballot_sync(0xffffffffu, pos == plast);
            const int from = m ? __ffs(m) - 1 : GRP + jj;
            if (!m && lane == from) { pos = plast; src = plast; }
            const int sj = __shfl_sync(0xffffffffu, src, jj), sf = __shfl_sync(0xffffffffu, src, from);
            if (lane == jj) src = sf;
            if (lane == from) src = sj;
        };
        // Column jj's step on a row is split in two. At once: its multiplier l, its entry of the next column (whose
        // search is the critical path). In the next column, while messages are on their way: the rest of the row. A
        // row that may be sent before that has its rest done on the way out, an entry a lane.
        C l[RPT], next[RPT];
        auto rest = [&](int jj) {
            const int col = gr + jj;
            const typename PS::Entries &urow = s.win[(g0 + jj) & 1].row;
#pragma unroll
            for (int c = 2; c < GRP; ++c) {
                const C u = urow[c];
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const C v = a[r][c];
                    C w = v;
                    cfms<R>(w, l[r], u);
                    // (finished L entries and rows stay: selected, not multiplied by 0)
                    const bool t = r0 + tid + T * r > col && c < GRP - jj;
                    a[r][c - 1] = mk<R>(t ? w.x : v.x, t ? w.y : v.y);
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) { a[r][0] = next[r]; a[r][GRP - 1] = l[r]; }
        };
        // row `row` (of a thread of this warp) as 16-byte pieces in the lanes, its rest done; its entry 0 in z
        auto prepare = [&](int jj, int row, typename PS::Stage &st, C &z) -> uint4 {
#pragma unroll
            for (int r = 0; r < RPT; ++r)
                if (r0 + tid + T * r == row) {
#pragma unroll
                    for (int q = 0; q < RB; ++q) st.row.piece(q) = a[r].piece(q);
                    st.l = l[r];
                    st.next = next[r];
                }
            __syncwarp();
            const int e = lane & (GRP - 1);
            C x;
            if (jj == 0) {
                x = st.row[e];
            } else {
                x = e == GRP - 1 ? st.l : st.row[e + 1];
                C w = x;
                cfms<R>(w, st.l, s.win[(g0 + jj - 1) & 1].row[(e + 1) & (GRP - 1)]);
                if (e + 1 < GRP - (jj - 1)) x = w;
                if (e == 0) x = st.next;
            }
            z = mk<R>(__shfl_sync(0xffffffffu, x.x, 0), __shfl_sync(0xffffffffu, x.y, 0));
            return piece_of(x, lane & (RB - 1));
        };
        for (int jj = 0; jj < gw && !dead; ++jj) {
            const int j = g0 + jj, col = k0 + j, par = j & 1, phase = (j >> 1) & 1;
            const uint32_t hbar = bar0 + 8 * par, rbar = hbar + 16;
            if (G > 1 && tid == 0) expect_bytes(hbar, (unsigned)G * 16u);
            // the block's candidate
            warp_best(best, bi);
            if (lane == 0) s.cand[par][wid] = head_of(best, bi);
            __syncthreads();
            const int failed = *(volatile int *)&s.fail[par];
            const uint4 ch = s.cand[par][lane & (nw - 1)];
            if (failed) { dead = true; break; }
            of_head(ch, best, bi);
            warp_best(best, bi);
            // its entry out to every CTA; its thread's warp, and the warp of the diagonal row's thread, get the rows
            // ready
            const int cw = bi == PNONE ? 0 : ((bi - r0) & (T - 1)) >> 5;
            const int dw = col >= r0 && col < rend ? ((col - r0) & (T - 1)) >> 5 : -1;
            uint4 cp = make_uint4(0u, 0u, 0u, 0u), dp = cp;
            const bool busy = wid == cw || wid == dw;
            auto recip = [&](C z) -> uint4 {
                C rc = mk<R>(0, 0);
                if (!(z.x == 0 && z.y == 0)) rc = cdiv<R>(mk<R>(1, 0), z);
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                memcpy(&v, &rc, sizeof(C));
                return v;
            };
            if (wid == cw) {
                if (G > 1) {
                    C z = mk<R>(0, 0);
#pragma unroll
                    for (int r = 0; r < RPT; ++r)
                        if (r0 + tid + T * r == bi) z = jj == 0 ? a[r][0] : next[r];
                    const int from = bi == PNONE ? 0 : (bi - r0) & 31;
                    z = mk<R>(__shfl_sync(0xffffffffu, z.x, from), __shfl_sync(0xffffffffu, z.y, from));
                    if (bi == PNONE) z.x = (R)NAN;
                    uint4 h = make_uint4(0u, 0u, 0u, 0u);
                    memcpy(&h, &z, sizeof(C));
                    if (lane < G) send16(peer_addr(smem_addr(&s.head[par][b]), lane), h, peer_addr(hbar, lane));
                }
                C z;
                cp = prepare(jj, bi, s.stage[0], z);
                if (G == 1 && lane == 0) s.rcp[par] = recip(z);
            }
            if (wid == dw) {
                C z;
                dp = prepare(jj, col, s.stage[1], z);
            }
            if (jj > 0) {
                if (wid == nw - 1) plan(jj - 1);
                if (!busy) rest(jj - 1);
            }
            // the winner: the largest entry, of the first CTA on ties (the CTAs' rows are in order)
            bool ok = true;
            int wq = 0;
            C piv = mk<R>(0, 0);
            if (G > 1) {
                ok = wait_phase(hbar, phase, err);
                if (lane < G) {
                    const uint4 h = s.head[par][lane];
                    memcpy(&piv, &h, sizeof(C));
                }
                R v = abs1(piv);
                const bool is = lane < G && v == v;
                int row = is ? lane : PNONE;
                warp_best(v, row);
                wq = row;
            } else if (bi == PNONE) {
                wq = PNONE;
            }
            if (!ok) dev_error(err, M25_DEV_TIMEOUT);
            else if (wq == PNONE) {                          // no candidate (NaN in the whole column): every CTA alike
                if (tid == 0) dev_error(err, M25_DEV_INDEX);
                ok = false;
            }
            // its row to every CTA, the diagonal row to its CTA; in each CTA a warp without a row forms 1 / pivot
            typename PS::Row &win = s.win[par];
            const int piece = lane & (RB - 1);
            if (ok) {
                const bool own = wq == b, swap = !own || bi != col;
                if (G > 1 && tid == 0) expect_bytes(rbar, (RB + 2 + (own && swap ? RB : 0)) * 16u);
                if (own && wid == cw) {
                    const uint4 pi = make_uint4((unsigned)bi, 0u, 0u, 0u);
                    if (G > 1) {
                        const uint32_t d = smem_addr(&win.row[0]) + 16 * piece;
#pragma unroll
                        for (int i = 0; i < PCL_MAX * RB / 32; ++i) {
                            const int q = lane / RB + 32 / RB * i;
                            if (q < G) send16(peer_addr(d, q), cp, peer_addr(rbar, q));
                        }
                        if (lane < G) send16(peer_addr(smem_addr(&win.p), lane), pi, peer_addr(rbar, lane));
                    } else {
                        if (lane < RB) win.row.piece(lane) = cp;
                        if (lane == 0) win.p = pi;
                    }
                }
                if (wid == dw && swap && lane < RB) {
                    if (G > 1) send16(peer_addr(smem_addr(&s.diag[par][0]) + 16 * lane, wq), dp, peer_addr(rbar, wq));
                    else s.diag[par].piece(lane) = dp;
                }
                const int helper = cw != 0 && dw != 0 ? 0 : cw != 1 && dw != 1 ? 1 : 2;
                if (G > 1 && wid == helper) {
                    const C z = mk<R>(__shfl_sync(0xffffffffu, piv.x, wq), __shfl_sync(0xffffffffu, piv.y, wq));
                    const uint4 v = recip(z);
                    if (lane == 0) send16(peer_addr(smem_addr(&s.rcp[par]), b), v, peer_addr(rbar, b));
                }
            }
            __syncwarp();
            if (jj > 0 && busy) rest(jj - 1);
            if (G > 1) {
                if (ok && !wait_phase(rbar, phase, err)) { ok = false; dev_error(err, M25_DEV_TIMEOUT); }
            } else {
                __syncthreads();
            }
            if (!ok) *(volatile int *)&s.fail[par ^ 1] = 1;  // (read after the next column's or the group's barrier)
            const int p = (int)win.p.x;
            plast = p;
            if (ok && b == 0 && tid == 0) ipiv[col] = p;
            C rc;
            {
                const uint4 w = s.rcp[par];
                memcpy(&rc, &w, sizeof(C));
            }
            const C u0 = win.row[0], u1 = win.row[1];
            // the interchange, column j scaled, the next column's entries; the next candidates
            best = (R)-1; bi = PNONE;
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int row = r0 + tid + T * r;
                if (row == col || row == p) {
                    const typename PS::Entries &from = row == col ? win.row : s.diag[par];
#pragma unroll
                    for (int q = 0; q < RB; ++q) a[r].piece(q) = from.piece(q);
                }
                const C a0 = a[r][0], v = a[r][1], t = a0 * rc;
                const bool act = row > col;
                l[r] = mk<R>(act ? t.x : a0.x, act ? t.y : a0.y);
                C w = v;
                cfms<R>(w, t, u1);
                const bool upd = act && jj < GRP - 1;
                next[r] = mk<R>(upd ? w.x : v.x, upd ? w.y : v.y);
                if (act && row < rend) {
                    const R x = abs1(w);
                    if (x > best) { best = x; bi = row; }
                }
            }
            if (wid == nw - 1) {
                if (lane < GRP) s.prow[jj][lane] = win.row[lane];
                if (b == 0 && lane == 0 && u0.x == 0 && u0.y == 0 && ok) dev_error(err, M25_DEV_ZEROPIV);
            }
        }
        if (wid == nw - 1 && !dead) {
            plan(gw - 1);
            s.pos[lane] = pos;
            s.src[lane] = src;
        }
        __syncthreads();
        dead = dead || *(volatile int *)&s.fail[(g0 + gw) & 1];
        if (G > 1 && g0 > 0) cluster_wait();               // the previous group's updates, by all CTAs
        if (!dead) {
            rest(gw - 1);
            pos = s.pos[lane];
            src = s.src[lane];
            for (int jj = gw; jj < GRP; ++jj)               // (a short last group: the rotation completed)
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    const C t = a[r][0];
#pragma unroll
                    for (int c = 1; c < GRP; ++c) a[r][c - 1] = a[r][c];
                    a[r][GRP - 1] = t;
                }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int row = r0 + tid + T * r;
                if (row >= gr && row < rend)
#pragma unroll
                    for (int c = 0; c < GRP; ++c)
                        if (c < gw) stc<R>(A, (size_t)(gr + c) * lda + row, a[r][c]);
            }
            __syncwarp();
            // the panel's other columns, one a warp: the permutation, and on those to the right the group's rows of U
            for (int x = b + G * wid; x < jb - gw; x += G * nw) {
                const bool right = x >= g0;
                const int c = k0 + (right ? x + gw : x);
                const bool need = pos >= 0 && ((right && lane < GRP) || src != pos);
                C v = mk<R>(0, 0);
                if (need) v = ldc_l2<R>(A, (size_t)c * lda + src);
                if (right) {
#pragma unroll
                    for (int i = 0; i < GRP - 1; ++i) {
                        C xi;
                        xi.x = __shfl_sync(0xffffffffu, v.x, i);
                        xi.y = __shfl_sync(0xffffffffu, v.y, i);
                        if (lane > i && lane < GRP)
                            cfms<R>(v, s.prow[lane][GRP - lane + i], xi);
                    }
                }
                __syncwarp();
                if (need) stc<R>(A, (size_t)c * lda + pos, v);
                __syncwarp();
            }
        }
        if (g0 + GRP >= jb) break;
        if (G > 1) { __syncwarp(); cluster_arrive(); cluster_wait(); }
        else __syncthreads();
        const int nt = jb - g0 - GRP, ng = min(GRP, nt);   // columns to the right, the next group's
        if (!dead) {
            // the group's rows of U to shared memory, with a thread's first entries on their way; FB columns past the
            // next group's in flight while the ones before are updated
            constexpr int FB = RPT == 1 ? 8 : 4;
            C nx[GRP], f[FB];
            auto fetch = [&](C (&v)[FB], const R *col0, bool act, int c0) {
#pragma unroll
                for (int q = 0; q < FB; ++q)
                    v[q] = act && c0 + q < nt ? ldc_l2<R>(col0, (size_t)(c0 + q) * lda) : mk<R>(0, 0);
            };
            auto first = [&](int r) {
                const int row = r0 + tid + T * r;
                const bool act = row >= gr + GRP && row < rend;
                const R *col0 = A + 2 * ((size_t)(gr + GRP) * lda + row);
#pragma unroll
                for (int c = 0; c < GRP; ++c) nx[c] = act && c < ng ? ldc_l2<R>(col0, (size_t)c * lda) : mk<R>(0, 0);
                fetch(f, col0, act, GRP);
            };
            first(0);
            for (int e = tid; e < GRP * nt; e += T) {
                const int c = e / GRP, i = e % GRP;
                s.u[c][i] = ldc_l2<R>(A, (size_t)(gr + GRP + c) * lda + gr + i);
            }
            __syncthreads();
            auto upd = [&](C &v, const typename PS::Entries &l, int c) {
#pragma unroll
                for (int q = 0; q < RB; ++q) {
                    const uint4 w = s.u[c].piece(q);
                    const C *uc = reinterpret_cast<const C *>(&w);
#pragma unroll
                    for (int h = 0; h < 16 / (int)sizeof(C); ++h) cfms<R>(v, l[q * (16 / (int)sizeof(C)) + h], uc[h]);
                }
            };
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int row = r0 + tid + T * r;
                const bool act = row >= gr + GRP && row < rend;
                if (r > 0) first(r);
                if (act) {
                    R *col0 = A + 2 * ((size_t)(gr + GRP) * lda + row);
#pragma unroll
                    for (int c = 0; c < GRP; ++c) upd(nx[c], a[r], c);      // (past the panel: unused)
                    for (int c = GRP; c < nt; c += FB) {
                        C f2[FB];
                        fetch(f2, col0, act, c + FB);
#pragma unroll
                        for (int q = 0; q < FB; ++q)
                            if (c + q < nt) {
                                upd(f[q], a[r], c + q);
                                stc<R>(col0, (size_t)(c + q) * lda, f[q]);
                            }
#pragma unroll
                        for (int q = 0; q < FB; ++q) f[q] = f2[q];
                    }
#pragma unroll
                    for (int c = 0; c < GRP; ++c) a[r][c] = nx[c];
                }
            }
        }
        __syncwarp();
        if (G > 1) cluster_arrive();
    }
    __syncwarp();
    if (G > 1) { cluster_arrive(); cluster_wait(); }       // no CTA leaves while another may still send to it
}

template <typename R, int GRP, int RPT, int T>
int panel_launch(R *A, long lda, int n, int k0, int jb, int *ipiv, int *err, int G, cudaStream_t s)
{
    const void *f = (const void *)k_panel_cluster<R, GRP, RPT, T>;
    if (G > 8) M25_CHECK(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)G; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    lc.gridDim = dim3(G); lc.blockDim = dim3(T); lc.stream = s; lc.attrs = at; lc.numAttrs = 1;
    void *args[] = {&A, &lda, &n, &k0, &jb, &ipiv, &err};
    M25_CHECK(cudaLaunchKernelExC(&lc, f, args));
    m25_note_launch();
    return M25_OK;
}

// the largest cluster of up to 16 CTAs the kernel can have on the current device (0: clusters unavailable)
template <typename R, int GRP, int RPT, int T> int cluster_max()
{
    const void *f = (const void *)k_panel_cluster<R, GRP, RPT, T>;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t qc = {};
    cudaLaunchAttribute qa[1];
    qa[0].id = cudaLaunchAttributeClusterDimension;
    qa[0].val.clusterDim.x = PCL_MAX; qa[0].val.clusterDim.y = 1; qa[0].val.clusterDim.z = 1;
    qc.gridDim = dim3(PCL_MAX); qc.blockDim = dim3(T); qc.attrs = qa; qc.numAttrs = 1;
    int mc = 0;
    if (cudaOccupancyMaxPotentialClusterSize(&mc, f, &qc) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return std::min(PCL_MAX, mc);
}
}  // namespace

// The largest cluster the panel kernel can have on the current device (0: none).
int m25_panel_cluster_max(int single)
{
    return single ? std::min(cluster_max<float, 16, 1, 512>(), cluster_max<float, 8, 4, 512>()) : cluster_max<double, 8, 2, 512>();
}

// Rows the cluster panel takes with cl CTAs of 512 threads: 4 (complex64) or 2 (complex128) rows a thread.
int m25_panel_cluster_rows(int single, int cl) { return cl * 512 * (single ? 4 : 2); }

// Factors the panel of columns k0 .. k0 + jb (jb <= 64), rows k0 .. n, on a cluster of at most cl CTAs.
//
// CTAs: one for every 128 rows, up to the cluster's limit (with 64 or 256 rows a CTA the LU of n = 1,000 takes 2-3%
// longer in complex64, 1-6% in complex128). Per CTA: one row a thread and 16 columns a group up to 256 rows (groups of 8
// there: 2-6% longer LUs, twice the group ends; two rows a thread of 128: 2.83 / 3.31 ms against 2.82 / 3.18 at n =
// 1,000, 17.5 / 23.2 against 16.7 / 22.1 at 4,977, complex64 / complex128), then fewer columns a group and more rows a
// thread. The kernels of 512 threads (above 256 rows a CTA in complex64, 512 in complex128) are held to 128 registers and
// spill: 156 bytes a thread stored in <float, 16, 1>, 436 in <float, 8, 4>, 752 in <double, 8, 2>; above 512 rows,
// complex64, 16 columns and two rows a thread of 512 take 43.7 ms against 43.1 at n = 9,601. (LU times of the tree that
// the choices were made on; the panel's later changes shortened both sides of each.)
int m25_panel_cluster(void *A, long lda, int n, int k0, int jb, int *ipiv, int single, int cl, int *err, cudaStream_t s)
{
    const int rows = n - k0;
    M25_REQUIRE(cl >= 1 && cl <= PCL_MAX && jb >= 1 && jb <= PNB && rows >= jb && rows <= m25_panel_cluster_rows(single, cl),
                "panel: too many rows for the cluster");
    const int G = std::min(cl, std::max(1, (rows + 127) / 128)), per = (rows + G - 1) / G;
    if (single) {
        float *F = (float *)A;
        if (per <= 256) return panel_launch<float, 16, 1, 256>(F, lda, n, k0, jb, ipiv, err, G, s);
        if (per <= 512) return panel_launch<float, 16, 1, 512>(F, lda, n, k0, jb, ipiv, err, G, s);
        if (per <= 1024) return panel_launch<float, 8, 4, 256>(F, lda, n, k0, jb, ipiv, err, G, s);
        return panel_launch<float, 8, 4, 512>(F, lda, n, k0, jb, ipiv, err, G, s);
    }
    double *F = (double *)A;
    if (per <= 256) return panel_launch<double, 16, 1, 256>(F, lda, n, k0, jb, ipiv, err, G, s);
    if (per <= 512) return panel_launch<double, 8, 2, 256>(F, lda, n, k0, jb, ipiv, err, G, s);
    return panel_launch<double, 8, 2, 512>(F, lda, n, k0, jb, ipiv, err, G, s);
}
