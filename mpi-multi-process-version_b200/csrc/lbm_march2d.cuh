// The fast build's 2D march of T = 2 or 4 time levels per pass over the populations.
//
// Included by lbm_kernels.cu inside namespace lbm::LBM_NS, after
// lbm_node2d.cuh and lbm_march.cuh (barriers, TMA copies, programmatic launch).
//
// One time level per pass reads and writes the whole state from HBM, and the
// stencil's shared-memory reads and index arithmetic (not the floating-point
// work) fill the issue slots.  Here
//   * a CTA has T groups of NT threads, one group per time level.  Group 0
//     takes rows of the state from a TMA ring and produces rows of the next
//     level into a three-row ring in shared memory; group s reads the ring of
//     group s - 1; the last group writes to global memory.  HBM traffic per
//     lattice update falls to 1/T, and the groups work on different rows at the
//     same time, so one block barrier per row paces all of them;
//   * interpolation runs along x first, on each row as it arrives, and the two
//     values the y-sum needs later (the row itself and the sum's first two
//     terms) stay in registers: a row is read once per level (31 shared-memory
//     reads a node instead of 62, 48 multiply-adds instead of 84);
//   * one tensor copy fetches all 14 population planes of a row (one more the
//     carried force).
// Measured, FP64, us a step, one level per pass (k_march2d: 62 reads a node, one
// copy per plane) against this one: 513^2 13.5 -> 9.9, 700x900 27.5 ->
// 18.5, 1024^2 48.0 -> 28.1, 2048^2 178 -> 105 (1.46 times what one pass per step
// could reach); FP32: 512^2 9.2 -> 7.7, 1023x771 23.7 -> 17.0, 2048^2 106 ->
// 78; a batch of 32 cavities FP64 404 -> 206.  What bounds it now: 470 instructions
// per 32 updates at 2048^2 (185 FP64; 519 and 202 in a batch at four levels, halo
// included) issue 54 to 56 % of the time at 12 to 15 warps per SM, in FP32 65 to
// 71 %; HBM is at 55 % there and at 34 % in the batch.  Two columns per thread needed
// 254 registers and was no faster; 16 warps in blocks of two 64-column levels with
// a three-slot input ring neither.
// Level s of rows [ja, jb) x columns [x0, x0 + w) needs T - s more nodes on
// each side; those are computed twice (by the neighbouring segment too): 2 of
// 126 columns and 2 rows per segment at T = 2.
//
// Schedule.  Let it count a segment's iterations and q = it - 3 s (s = 0 ..
// T-1).  Away from the bottom wall group s takes node row n = nb_s + q, its
// first two rows only to fill the registers.  A segment that starts at the
// bottom wall stalls one iteration after every third row for the first T-1-s
// such triples, since row 0 needs rows 1 and 2 of the level below at once:
//   q < 4 (T-1-s): n = 3 (q / 4) + q % 4, idle when q % 4 == 3; else n = q - (T-1-s).
// Either way, when group s reads rows n and n + 1, group s - 1 finished them in
// an earlier iteration and writes row n + 2 in this one, so three ring rows do.

template <int ST, int COLS_, int T_>
struct M2 {
    using S = typename Tr<ST>::S;
    static constexpr int ES = sizeof(S);
    static constexpr int COLS = COLS_, T = T_;  // threads of a group: one per column
    static constexpr int HX = 16 / ES;         // elements per 16 bytes: TMA boxes start on such a boundary
    static constexpr int WB = COLS + 2 * HX;   // elements per plane and row
    static constexpr int NS = 4;               // input ring slots: the node's row, the row above, two in flight
    static constexpr int PLANES = 14 * WB * ES;
    static constexpr int FO = (PLANES + 127) / 128 * 128;   // the force row
    static constexpr int ROW = (FO + WB * ES + 127) / 128 * 128;
    static constexpr int WR = 16;              // rows of y-weights kept, 64 bytes each
    static constexpr int E0 = NS * ROW;
    static constexpr int W0 = E0 + (T - 1) * 3 * ROW;
    static constexpr int B0 = W0 + WR * 64;
    static constexpr int K0 = B0 + 64 + kGeoStage;          // a batch's staged geometry, then its Relax
    static constexpr int SMEM = K0 + 128 + 128;
    static constexpr int TX = PLANES + WB * ES + 48;        // bytes of a row's copies
    static_assert((WB * ES) % 16 == 0 && WB <= 256 && (T == 2 || T == 4), "2D march layout");
};

// A segment: columns [x0, x0 + w) of cavity cav, rows [ja, jb).
struct Seg2 {
    int cav, x0, w, ja, jb;
};
__device__ __forceinline__ Seg2 seg2_of(const int4 q)
{
    // .x = cavity | width << 24 (width <= 128)
    return {q.x & 0xffffff, q.y, int((uint32_t)q.x >> 24), q.z, q.w};
}

template <int ST, class M, bool kStage, class CavFn>
__device__ __forceinline__ void march2d_levels(const int4 *__restrict__ segs, int sbeg, int send, CavFn cavity, int *err)
{
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    constexpr int NT = M::COLS, T = M::T, WB = M::WB, HX = M::HX, NS = M::NS;
    constexpr bool DEV = Tr<ST>::kShift, DEVT = Tr<ST>::kDevT;
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = sm_raw + ((128u - (saddr(sm_raw) & 127u)) & 127u);
    uint64_t *bar = (uint64_t *)(sm + M::B0);
    // thread 0's copy state (2 words), then the failure words of even and odd iterations
    volatile int *iss = (volatile int *)(sm + M::B0 + 40);
    Geo *sgeo = (Geo *)(sm + M::B0 + 64);
    Relax<C> *srelax = (Relax<C> *)(sm + M::K0);

    const int tid = threadIdx.x;
    const int s = tid / NT;  // the group's time level (warp-uniform)
    const int t = tid % NT;
    if (tid == 0) {
        for (int k = 0; k < NS; ++k) mbar_init(&bar[k], 1);
        fence_barrier_init();
        iss[2] = iss[3] = 0;
    }
    dep_launch();
    __syncthreads();

    uint32_t seq = 0;  // copies issued before this segment: slot and phase follow from it
    bool waited = false, aborted = false;

    for (int si = sbeg; si < send && !aborted; ++si) {
        const Seg2 sg = seg2_of(segs[si]);
        const Geo *Gp;
        const CUtensorMap *maps, *fmap;
        S *dst;
        C *Fout;
        const Bufs *Bp;
        cavity(sg.cav, Gp, maps, fmap, dst, Fout, Bp);
        if (kStage) {
            Gp = stage_geo(Gp, sgeo);
            if (tid == 0) *srelax = relax_of<C>(*Gp);
            __syncthreads();
        }
        const RunCtl *ctl = Bp->ctl;
        if (!waited) {
            dep_wait();  // from here on: what earlier kernels wrote
            waited = true;
        }
        if (!ctl->active) continue;  // a cavity whose run has stopped
        const Geo &G = *Gp;
        const int nx = G.nx, ny = G.ny;
        const int64_t P = G.plane;

        // columns: thread t of every group stands on column xs + t
        const int xs = max(sg.x0 - (T - 1), 0);
        const int bx0 = (xs - 1 + HX) / HX * HX - HX;   // the box's first column, 16-byte aligned, <= xs - 1
        const int c = xs + t;
        const bool active = c >= max(sg.x0 - (T - 1 - s), 0) && c < min(sg.x0 + sg.w + (T - 1 - s), nx);
        const int cc = active ? c - bx0 : HX;           // its index in a ring row, and its window's
        const int cw = active ? win_lo(c, nx) - bx0 : HX;
        C xp[3], xm[3], Tcn = C(0.0), sT = C(0.0);
        {
            const int ce = min(c, nx - 1);
            window_weights<C>(G.wgt[0] + (int64_t)ce * 6, ce, nx, xp, xm);
            if (DEVT) Tcn = C(tc_value(G, ce));
        }
        if (DEVT) sT = C(0.125 * G.dt * tc_gradient(G));
        // one cavity: constant-bank operands; a batch reads them where they are used
        const Relax<C> K1 = kStage ? Relax<C>{} : relax_of<C>(G);

        // rows
        const bool bottom = sg.ja < T;
        const int r0 = max(sg.ja - (T - 1 - s), 0), r1 = min(sg.jb - 1 + (T - 1 - s), ny - 1);
        const int nb = sg.ja - T + s - 1;               // away from the wall: the node of q = 0
        const int row_first = bottom ? 0 : sg.ja - T;   // input rows
        const int row_last = min(sg.jb + T - 1, ny - 1);
        const int its = (bottom ? sg.jb : sg.jb - sg.ja + 2) + 3 * (T - 1);
        // thread 0 copies input rows up to `hi`; its state (next row, copy number of row 0) is in shared memory
        auto issue_to = [&](int hi) {
            int r = iss[0];
            const uint32_t k0 = (uint32_t)iss[1];
            for (; r <= hi; ++r) {
                const int slot = (k0 + (uint32_t)r) % NS;
                unsigned char *base = sm + slot * M::ROW;
                uint64_t *b = &bar[slot];
                mbar_arrive_tx(b, M::TX);
                tma_load3(base, maps, b, bx0, r, 0);
                tma_load2(base + M::FO, fmap, b, bx0, r);
                bulk_load(sm + M::W0 + (r % M::WR) * 64, G.wgt[1] + (int64_t)r * 6, 48, b);
            }
            iss[0] = r;
        };
        if (tid == 0) {
            iss[0] = row_first;
            iss[1] = (int)(seq - (uint32_t)row_first);
            issue_to(min(row_first + NS - 1, row_last));
        }

        // per plane 2 4 | 5 6 7 8 | 11 13: the newest row's x-interpolated value and the y-sum's first two
        // terms; which sign of the y-weights it takes (2 5 6 11 come from below: +)
        constexpr bool up[8] = {true, false, true, true, false, false, true, false};
        C hx[8], hp[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) hx[k] = hp[k] = C(0.0);

        for (int it = 0; it < its; ++it) {
            const int q = it - 3 * s;
            int n = -2;   // this iteration's node row
            bool work = q >= 0;
            if (bottom) {
                const int stalls = T - 1 - s;
                if (q < 4 * stalls) {
                    n = 3 * (q >> 2) + (q & 3);
                    work = work && (q & 3) != 3;
                } else {
                    n = q - stalls;
                }
            } else {
                n = nb + q;
            }
            work = work && n <= r1;
            // the input ring: rows below group 0's node row are free
            if (s == 0) {
                int n0 = work ? n : r1 + 1;
                if (bottom && !work && q < 4 * (T - 1)) n0 = 3 * (q >> 2) + 3;  // a stall: the next row's node
                if (tid == 0) issue_to(min(n0 - 1 + NS, row_last));
            }
            bool ok = true;
            if (work) {
                const bool lo = n == 0 && bottom, hi = n == ny - 1;
                // ring rows of node row n + k
                auto rowp = [&](int r) -> const unsigned char * {
                    if (s == 0) return sm + ((seq + uint32_t(r - row_first)) % NS) * M::ROW;
                    return sm + M::E0 + ((s - 1) * 3 + r % 3) * M::ROW;
                };
                if (s == 0) {
                    auto wait = [&](int r) {
                        const uint32_t k = seq + uint32_t(r - row_first);
                        ok = ok && mbar_wait_lim(&bar[k % NS], (k / NS) & 1u);
                    };
                    if (lo) {
                        wait(0);
                        wait(1);
                        wait(2);
                    } else if (!hi) {
                        wait(n + 1);
                    }
                }
                if (ok && active) {
                    // x-interpolated values of a row for the planes whose stencil reaches along y
                    auto XR = [&](int r, C (&o)[8]) {
                        const S *b = (const S *)rowp(r);
                        const S *w = b + cw, *m = b + cc;
                        o[0] = m[2 * WB];
                        o[1] = m[4 * WB];
                        o[2] = lin3(xp, C(w[5 * WB]), C(w[5 * WB + 1]), C(w[5 * WB + 2]));
                        o[3] = lin3(xm, C(w[6 * WB]), C(w[6 * WB + 1]), C(w[6 * WB + 2]));
                        o[4] = lin3(xm, C(w[7 * WB]), C(w[7 * WB + 1]), C(w[7 * WB + 2]));
                        o[5] = lin3(xp, C(w[8 * WB]), C(w[8 * WB + 1]), C(w[8 * WB + 2]));
                        o[6] = m[11 * WB];
                        o[7] = m[13 * WB];
                    };
                    C y[8];
                    if (lo || hi) {
                        // a wall row: its one-sided window, read in one go
                        const int b = lo ? 0 : ny - 3;
                        C wp[3], wm[3], v0[8], v1[8], v2[8];
                        window_weights<C>((const double *)(sm + M::W0 + (n % M::WR) * 64), n, ny, wp, wm);
                        XR(b, v0);
                        XR(b + 1, v1);
                        XR(b + 2, v2);
#pragma unroll
                        for (int k = 0; k < 8; ++k) y[k] = lin3(up[k] ? wp : wm, v0[k], v1[k], v2[k]);
                        if (lo) {
                            const double *w1 = (const double *)(sm + M::W0 + (1 % M::WR) * 64);
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                hx[k] = v1[k];
                                hp[k] = lin2(C(w1[up[k] ? 0 : 3]), C(w1[up[k] ? 1 : 4]), v0[k], v1[k]);
                            }
                        }
                    } else {
                        C v[8];
                        XR(n + 1, v);
                        const double *wn = (const double *)(sm + M::W0 + ((n & (M::WR - 1))) * 64);
                        const double *wq = (const double *)(sm + M::W0 + (((n + 1) & (M::WR - 1))) * 64);
                        const C p2 = C(wn[2]), m2 = C(wn[5]);
                        const C p0 = C(wq[0]), p1 = C(wq[1]), m0 = C(wq[3]), m1 = C(wq[4]);
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            y[k] = fma_(up[k] ? p2 : m2, v[k], hp[k]);
                            hp[k] = lin2(up[k] ? p0 : m0, up[k] ? p1 : m1, hx[k], v[k]);
                            hx[k] = v[k];
                        }
                    }
                    if (n >= r0) {
                        const S *b = (const S *)rowp(n);
                        const S *w = b + cw, *m = b + cc;
                        C f[9], g[5];
                        f[0] = m[0];
                        f[1] = lin3(xp, C(w[WB]), C(w[WB + 1]), C(w[WB + 2]));
                        f[2] = y[0];
                        f[3] = lin3(xm, C(w[3 * WB]), C(w[3 * WB + 1]), C(w[3 * WB + 2]));
                        f[4] = y[1];
                        f[5] = y[2];
                        f[6] = y[3];
                        f[7] = y[4];
                        f[8] = y[5];
                        g[0] = m[9 * WB];
                        g[1] = lin3(xp, C(w[10 * WB]), C(w[10 * WB + 1]), C(w[10 * WB + 2]));
                        g[2] = y[6];
                        g[3] = lin3(xm, C(w[12 * WB]), C(w[12 * WB + 1]), C(w[12 * WB + 2]));
                        g[4] = y[7];
                        if (DEVT) {  // deviation from the conduction profile along x
                            g[1] = sub_(g[1], sT);
                            g[3] = add_(g[3], sT);
                        }
                        walls2d<C, DEVT>(c, n, nx, ny, C(G.Thot), C(G.Tcold), Tcn,
                                         [&](int pl) -> C { return C(m[pl * WB]); }, f, g);
                        const C F0 = ((const C *)((const unsigned char *)b + M::FO))[cc];
                        const Relax<C> K = kStage ? *srelax : K1;
                        C fp[9], gp[5], Fy, rho, u, v, Tm;
                        node2d<C, DEV, DEVT>(f, g, F0, K, Tcn, fp, gp, Fy, rho, u, v, Tm);
                        if (s == T - 1) {
                            const int64_t id = (int64_t)n * G.pitch + c;
                            Fout[id] = Fy;
                            S *o = dst + id;
#pragma unroll
                            for (int pl = 0; pl < 9; ++pl) o[pl * P] = S(fp[pl]);
#pragma unroll
                            for (int pl = 0; pl < 5; ++pl) o[(9 + pl) * P] = S(gp[pl]);
                        } else {
                            unsigned char *e = sm + M::E0 + (s * 3 + n % 3) * M::ROW;
                            S *o = (S *)e + cc;
#pragma unroll
                            for (int pl = 0; pl < 9; ++pl) o[pl * WB] = S(fp[pl]);
#pragma unroll
                            for (int pl = 0; pl < 5; ++pl) o[(9 + pl) * WB] = S(gp[pl]);
                            ((C *)(e + M::FO))[cc] = Fy;
                        }
                    }
                }
            }
            // a wait that ran out in iteration it is noted in word it & 1 and acted on, by every thread alike,
            // at the end of the next one (the test stays off the row's critical path)
            if (!ok) {
                iss[2 + (it & 1)] = 1;
                if (tid == 0) {  // and no copy into a slot whose last one this thread has not seen land; their number stays
                    iss[1] = iss[1] + iss[0] - (1 << 30);
                    iss[0] = 1 << 30;
                }
            }
            const int failed = iss[2 + ((it + 1) & 1)];
            __syncthreads();
            if (failed) {
                aborted = true;
                break;
            }
        }
        seq += uint32_t(min(sg.jb + T - 1, ny - 1) - (sg.ja < T ? 0 : sg.ja - T) + 1);
    }
    if (tid == 0 && (iss[2] | iss[3])) {
        atomicExch(err, 1);
        // let copies still in flight land before the CTA's shared memory is released
        const uint32_t n = (uint32_t)iss[1] + (uint32_t)iss[0];
        for (uint32_t k = n > NS ? n - NS : 0; k < n; ++k) mbar_wait(&bar[k % NS], (k / NS) & 1u);
    }
}

// blocks per SM: what shared memory leaves room for at the registers a thread needs
template <class M, int ST>
constexpr int m2_blocks()
{
    constexpr int regs = ST == kF64 ? 128 : 96;
    constexpr int by_smem = (228 * 1024) / (M::SMEM + 1024);
    constexpr int by_reg = 65536 / (regs * M::COLS * M::T);
    constexpr int n = by_smem < by_reg ? by_smem : by_reg;
    return n < 1 ? 1 : n;
}

// one cavity
template <int ST, int COLS, int T>
__global__ void __launch_bounds__(COLS * T, (m2_blocks<M2<ST, COLS, T>, ST>()))
k_march2d_levels(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap fmap,
          const __grid_constant__ Geo G, typename Tr<ST>::S *__restrict__ dst, typename Tr<ST>::C *__restrict__ Fout,
          const __grid_constant__ Bufs B, const int4 *__restrict__ segs,
          const int *__restrict__ seg_off, int *err)
{
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    auto cavity = [&](int, const Geo *&Gp, const CUtensorMap *&m, const CUtensorMap *&fm, S *&d, C *&Fo,
                      const Bufs *&Bp) {
        Gp = &G;
        m = &map;
        fm = &fmap;
        d = dst;
        Fo = Fout;
        Bp = &B;
    };
    march2d_levels<ST, M2<ST, COLS, T>, false>(segs, seg_off[blockIdx.x], seg_off[blockIdx.x + 1], cavity,
                                               err);
}

// many cavities; `cur` is the ping-pong buffer holding the populations read
template <int ST, int COLS, int T>
__global__ void __launch_bounds__(COLS * T, (m2_blocks<M2<ST, COLS, T>, ST>()))
k_march2d_levels_batch(const BatchDev D, int cur, int *err)
{
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    auto cavity = [&](int c, const Geo *&Gp, const CUtensorMap *&m, const CUtensorMap *&fm, S *&d, C *&Fo,
                      const Bufs *&Bp) {
        const TmapSet *ts = &D.maps[(int64_t)c * 2 + cur];
        Gp = &D.geo[c];
        m = &ts->m[0];
        fm = &ts->fmap;
        Bp = &D.bufs[c];
        d = (S *)D.bufs[c].pop[1 - cur];
        Fo = (C *)D.bufs[c].F[1 - cur];
    };
    march2d_levels<ST, M2<ST, COLS, T>, true>(D.segs, D.seg_off[blockIdx.x], D.seg_off[blockIdx.x + 1], cavity,
                                              err);
}
