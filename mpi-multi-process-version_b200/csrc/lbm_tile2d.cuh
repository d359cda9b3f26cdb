// Small 2D domains of the fast build: T time steps of a tile in shared memory.
//
// Included by lbm_kernels.cu inside namespace lbm::LBM_NS, after
// lbm_node2d.cuh and lbm_march.cuh.
//
// A domain of a few ten thousand nodes fills no GPU: a step through the march
// or the direct-load kernel is a launch (2 us) plus one pass of latency, and
// most SMs idle.  Here each CTA owns a core of cx x cy nodes, loads it with T
// more nodes on every inner side, and advances the whole patch T levels in
// shared memory, the region shrinking by a node per level; the extra nodes are
// computed by the neighbouring tiles too, on SMs that would idle.  One launch,
// one load and one store serve T steps.
//
// The patch holds its 14 populations and the force node by node (15 elements):
// every population and every x-neighbour is an immediate offset from a row's
// pointer, and 15 is odd, so lanes on consecutive nodes hit different banks.
// Two patches alternate between levels.
//
// Measured, us a step, before -> after: FP64 48x40 3.59 -> 1.46, 128^2 4.11 -> 2.11,
// 192^2 4.61 -> 3.04, 256^2 4.87 -> 4.43; FP32 128^2 3.85 -> 1.70, 256^2 4.61 -> 3.35.
// Bound by latency: at most 16 warps per SM, a level's nodes at about 10 cycles an
// instruction; the launch, load and store are 3.3 us of the 8.4 us that four
// steps of 128^2 take.

template <int ST>
__global__ void __launch_bounds__(512)
k_tile2d(const __grid_constant__ Geo G, const typename Tr<ST>::S *__restrict__ src,
         const typename Tr<ST>::C *__restrict__ Fin, typename Tr<ST>::S *__restrict__ dst,
         typename Tr<ST>::C *__restrict__ Fout, const RunCtl *ctl, const TilePlan pl)
{
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    constexpr bool DEV = Tr<ST>::kShift, DEVT = Tr<ST>::kDevT;
    constexpr int NV = 15;  // 14 populations and the force
    constexpr int NW = kTileWeights;
    extern __shared__ unsigned char sm_raw[];
    C *A = (C *)sm_raw, *Bp = A + pl.en * NV;
    C *wx = Bp + pl.en * NV;             // window weights of the patch's columns, then of its rows: 3 (+), 3 (-)
    const int tid = threadIdx.x, nthr = blockDim.x, T = pl.T;
    const int nx = G.nx, ny = G.ny;
    const int ta = blockIdx.x % pl.ntx, tb = blockIdx.x / pl.ntx;
    const int X0 = tile_cut(ta, pl.ntx, nx, 8), X1 = tile_cut(ta + 1, pl.ntx, nx, 8);
    const int Y0 = tile_cut(tb, pl.nty, ny, 1), Y1 = tile_cut(tb + 1, pl.nty, ny, 1);
    const int ex0 = max(X0 - T, 0), ex1 = min(X1 + T, nx), ey0 = max(Y0 - T, 0), ey1 = min(Y1 + T, ny);
    const int ew = ex1 - ex0, eh = ey1 - ey0;
    C *wy = wx + ew * NW;
    dep_launch();
    for (int k = tid; k < ew + eh; k += nthr) {
        const int ax = k < ew ? 0 : 1, i = ax ? ey0 + k - ew : ex0 + k;
        C wp[3], wm[3];
        window_weights<C>(G.wgt[ax] + (int64_t)i * 6, i, ax ? ny : nx, wp, wm);
        C *o = wx + k * NW;
        o[0] = wp[0]; o[1] = wp[1]; o[2] = wp[2];
        o[3] = wm[0]; o[4] = wm[1]; o[5] = wm[2];
    }
    dep_wait();  // from here on: what earlier kernels wrote
    if (!ctl->active) return;
    const int64_t P = G.plane;
    const int64_t pitch = G.pitch;
    {
        const float inv = 1.0f / float(ew);
        for (int k = tid; k < ew * eh; k += nthr) {
            const int y = int((float(k) + 0.5f) * inv), x = k - y * ew;
            const int64_t id = (int64_t)(ey0 + y) * pitch + ex0 + x;
            C v[NV];
#pragma unroll
            for (int q = 0; q < 14; ++q) v[q] = C(__ldcg(src + q * P + id));
            v[14] = __ldcg(Fin + id);
            C *o = A + k * NV;
#pragma unroll
            for (int q = 0; q < NV; ++q) o[q] = v[q];
        }
    }
    const Relax<C> K = relax_of<C>(G);
    const C sT = DEVT ? C(0.125 * G.dt * tc_gradient(G)) : C(0.0);
    __syncthreads();

    for (int l = 1; l <= T; ++l) {
        const int g = T - l;
        const int rx0 = max(X0 - g, 0), rx1 = min(X1 + g, nx), ry0 = max(Y0 - g, 0), ry1 = min(Y1 + g, ny);
        const int w = rx1 - rx0, h = ry1 - ry0;
        const float inv = 1.0f / float(w);
        for (int k = tid; k < w * h; k += nthr) {
            const int y = int((float(k) + 0.5f) * inv), i = rx0 + k - y * w, j = ry0 + y;
            const int xl = win_lo(i, nx), yl = win_lo(j, ny);
            const C *w0 = wx + (i - ex0) * NW, *w1 = wy + (j - ey0) * NW;
            const C xp[3] = {w0[0], w0[1], w0[2]}, xm[3] = {w0[3], w0[4], w0[5]};
            const C yp[3] = {w1[0], w1[1], w1[2]}, ym[3] = {w1[3], w1[4], w1[5]};
            // the window's rows; dx, dy: the node inside the window
            const C *p0 = A + ((yl - ey0) * ew + (xl - ex0)) * NV, *p1 = p0 + ew * NV, *p2 = p1 + ew * NV;
            const int dx = (i - xl) * NV;
            const C *pj = j - yl == 0 ? p0 : (j - yl == 1 ? p1 : p2), *pc = pj + dx;
            auto X = [&](const C *r, int q, const C (&ww)[3]) { return lin3(ww, r[q], r[NV + q], r[2 * NV + q]); };
            auto Y = [&](int q, const C (&ww)[3]) { return lin3(ww, p0[dx + q], p1[dx + q], p2[dx + q]); };
            auto XY = [&](int q, const C (&wa)[3], const C (&wb)[3]) {
                return lin3(wb, X(p0, q, wa), X(p1, q, wa), X(p2, q, wa));
            };
            C f[9], gg[5];
            f[0] = pc[0];
            f[1] = X(pj, 1, xp);
            f[2] = Y(2, yp);
            f[3] = X(pj, 3, xm);
            f[4] = Y(4, ym);
            f[5] = XY(5, xp, yp);
            f[6] = XY(6, xm, yp);
            f[7] = XY(7, xm, ym);
            f[8] = XY(8, xp, ym);
            gg[0] = pc[9];
            gg[1] = X(pj, 10, xp);
            gg[2] = Y(11, yp);
            gg[3] = X(pj, 12, xm);
            gg[4] = Y(13, ym);
            C Tc = C(0.0);
            if (DEVT) {
                Tc = C(tc_value(G, i));
                gg[1] = sub_(gg[1], sT);
                gg[3] = add_(gg[3], sT);
            }
            walls2d<C, DEVT>(i, j, nx, ny, C(G.Thot), C(G.Tcold), Tc, [&](int q) -> C { return pc[q]; }, f, gg);
            C fp[9], gp[5], Fy, rho, u, v, Tm;
            node2d<C, DEV, DEVT>(f, gg, pc[14], K, Tc, fp, gp, Fy, rho, u, v, Tm);
            if (l < T) {
                C *o = Bp + ((j - ey0) * ew + (i - ex0)) * NV;
#pragma unroll
                for (int q = 0; q < 9; ++q) o[q] = fp[q];
#pragma unroll
                for (int q = 0; q < 5; ++q) o[9 + q] = gp[q];
                o[14] = Fy;
            } else {
                const int64_t id = (int64_t)j * pitch + i;
                Fout[id] = Fy;
#pragma unroll
                for (int q = 0; q < 9; ++q) dst[q * P + id] = tostore<S, C>(fp[q]);
#pragma unroll
                for (int q = 0; q < 5; ++q) dst[(9 + q) * P + id] = tostore<S, C>(gp[q]);
            }
        }
        __syncthreads();
        C *t = A;
        A = Bp;
        Bp = t;
    }
}
