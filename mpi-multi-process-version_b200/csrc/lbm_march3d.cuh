// 3D march of the fast build: in-plane interpolation of each z-slice as it
// arrives, z-interpolation in registers, and a direction that alternates.
//
// Included by lbm_march.cuh inside namespace lbm::LBM_NS.
//
// A block owns a tile of 32 x TY nodes and walks along z.  The twelve planes
// whose stencil reaches along z (5 6, 11-18, 24 25) are interpolated in x or y
// once, when a slice arrives; a thread keeps the values of the last two slices
// in registers.  Reading all three slices for every output instead (as the
// direct-load kernel does) takes 84 loads from shared memory where this takes
// 28, 152 against 96 in all: 63.5 M warp instructions a launch at 128^3 instead of 70.0 M.  Two planes a
// TMA copy halve the copies, which one thread issues (FP64 128^3: 16 copies a
// slice instead of 30; single planes cost 3 % in FP32, 9 % at 61 x 50 x 47).
//
// What bounds it: at sizes past L2 a long run sits at the board's power limit
// (1000 W, the clock down to 1.6 GHz), so work saved is time saved even where
// memory bandwidth would hide it; in L2 the latency of a slice, 2.4 us with two
// blocks an SM.  Measured, us a step, all three slices read -> this: runs of seconds
// at 128^3 FP64 175 -> 167, FP32 102 -> 90; bursts of 100 steps 128^3 FP64 157 -> 156,
// FP32 92 -> 85, 61 x 50 x 47 FP64 16.3 -> 14.7, 131 x 118 x 125 FP64 215 -> 191, FP32
// 108 -> 101.  On how many blocks: march3d_blocks.
//
// Steps that read buffer 1 walk downwards (`rev`): the slices the last step
// wrote last, partly still in L2, are read first (1 to 2 % in long runs at 128^3;
// to have the copies evict first, so that more of the written data stays, loses
// the neighbours' halo rows: 163 -> 191 us).  Deeper rings are no faster (four z
// slots 166 against 168 us, three plane slots 179).
//
// The walk is written in mirrored slice numbers: step m of a downward walk is
// slice nz-1-m.  Every output is w1 v1 + (w0 v0 + w2 v2) over its window, an
// order of operations that is the same from both sides, so a node's bits depend
// neither on the direction nor on where a segment starts.  The end slices' own
// windows (0-2, nz-3 .. nz-1) take one more slice, from shared memory, where it
// is resident at that step.

template <int ST, int TY_ = 8>
struct L3 {
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    static constexpr int ES = sizeof(S);
    static constexpr int TX = 32, TY = TY_, NT = TX * TY;
    static constexpr int HX = 16 / ES;
    static constexpr int ZS = 3, NS = 2;  // ring slots: slices k .. k + 2, and k, k + 1
    // box classes: 0 tile only, 1 +-HX columns, 2 +-1 rows, 3 both; a copy takes
    // two consecutive planes (planes 0 and 19 one)
    __host__ __device__ static constexpr int bx(int c) { return TX + ((c & 1) ? 2 * HX : 0); }
    __host__ __device__ static constexpr int by(int c) { return TY + ((c & 2) ? 2 : 0); }
    __host__ __device__ static constexpr int bytes(int c) { return bx(c) * by(c) * ES; }
    static_assert((2 * bytes(0)) % 128 == 0 && bytes(0) % 128 == 0 && (2 * bytes(1)) % 128 == 0 &&
                      (2 * bytes(2)) % 128 == 0 && (2 * bytes(3)) % 128 == 0, "TMA destinations are 128-byte aligned");
    // z slot: planes 5 6 | 11 12 | 13 14 | 15 16 | 17 18 | 24 25
    __host__ __device__ static constexpr int zcl(int p) { return p == 0 || p == 5 ? 0 : (p < 3 ? 1 : 2); }
    __host__ __device__ static constexpr int zpl(int p) { return p == 0 ? 5 : (p == 5 ? 24 : 9 + 2 * p); }
    __host__ __device__ static constexpr int zpo(int p)
    {
        int o = 0;
        for (int a = 0; a < p; ++a) o += 2 * bytes(zcl(a));
        return o;
    }
    // plane zi (0-11 in the order above)
    __host__ __device__ static constexpr int zc(int zi) { return zcl(zi / 2); }
    __host__ __device__ static constexpr int zoff(int zi) { return zpo(zi / 2) + (zi & 1) * bytes(zc(zi)); }
    __host__ __device__ static constexpr int zslot() { return zpo(6); }
    __host__ __device__ static constexpr int ztx() { return zpo(6); }
    // n slot: planes 0 19 (single) | 1 2 | 20 21 | 3 4 | 22 23 | 7 8 | 9 10, then the carried-force
    // tile and the slice's six z-weights
    __host__ __device__ static constexpr int npc(int p) { return p < 2 ? 1 : (p < 4 ? 2 : 3); }  // pairs 0-5
    __host__ __device__ static constexpr int npl(int p)
    {
        return p == 0 ? 1 : (p == 1 ? 20 : (p == 2 ? 3 : (p == 3 ? 22 : (p == 4 ? 7 : 9))));
    }
    __host__ __device__ static constexpr int npo(int p)
    {
        int o = 2 * bytes(0);
        for (int a = 0; a < p; ++a) o += 2 * bytes(npc(a));
        return o;
    }
    // class and offset of in-plane plane q
    __host__ __device__ static constexpr int npair(int q)
    {
        return q < 3 ? 0 : (q < 5 ? 2 : (q < 9 ? 4 : (q < 11 ? 5 : (q < 22 ? 1 : 3))));
    }
    __host__ __device__ static constexpr int qc(int q) { return q == 0 || q == 19 ? 0 : npc(npair(q)); }
    __host__ __device__ static constexpr int qoff(int q)
    {
        return q == 0 ? 0 : (q == 19 ? bytes(0) : npo(npair(q)) + (q - npl(npair(q))) * bytes(qc(q)));
    }
    __host__ __device__ static constexpr int fbytes() { return TX * TY * (int)sizeof(C); }
    __host__ __device__ static constexpr int fo() { return npo(6); }
    __host__ __device__ static constexpr int wo() { return fo() + (fbytes() + 127) / 128 * 128; }
    __host__ __device__ static constexpr int nslot() { return wo() + 128; }
    __host__ __device__ static constexpr int ntx() { return npo(6) + fbytes() + 48; }
    // ring slots, the barriers and the abort flag, the staged Geo, slack for 128-byte alignment
    static constexpr int nbar = ZS + NS;
    __host__ __device__ static constexpr int bo() { return ZS * zslot() + NS * nslot(); }
    __host__ __device__ static constexpr int smem() { return bo() + 64 + kGeoStage + 128; }
    static_assert(nbar * 8 + 4 <= 64, "barriers and flag");
};

// A block runs segments segs[sbeg .. send), each (tile, first slice, end slice,
// cavity); tiles are numbered x-fastest within a cavity.  `cavity(c, G, maps,
// dst, Fout, B)` yields cavity c's geometry, the TMA descriptors of the buffer
// read this step, the outputs and the buffers.  rev: walk downwards, through the
// segments in reverse.
template <int ST, int TY_, bool kStage, class CavFn>
__device__ __forceinline__ void march3d_run(const int4 *__restrict__ segs, int sbeg, int send, CavFn cavity,
                                            int write_macro, int rev, int *err)
{
    using S = typename Tr<ST>::S;
    using C = typename Tr<ST>::C;
    using L = L3<ST, TY_>;
    constexpr int TX = L::TX, TY = L::TY, HX = L::HX, ZS = L::ZS, NS = L::NS;
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = sm_raw + ((128u - (saddr(sm_raw) & 127u)) & 127u);
    unsigned char *smn = sm + ZS * L::zslot();
    uint64_t *zbar = (uint64_t *)(sm + L::bo());
    uint64_t *nbar = zbar + ZS;
    volatile int &s_abort = *(volatile int *)(nbar + NS);
    Geo *sgeo = (Geo *)(sm + L::bo() + 64);

    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    if (tid == 0) {
        for (int s = 0; s < ZS; ++s) mbar_init(&zbar[s], 1);
        for (int s = 0; s < NS; ++s) mbar_init(&nbar[s], 1);
        fence_barrier_init();
        s_abort = 0;
    }
    dep_launch();
    __syncthreads();

    uint32_t znext = 0, nnext = 0;  // per-slot parity of the next copy
    int i0 = 0, j0 = 0;
    const Geo *Gp = nullptr;       // the current segment's cavity
    const TmapSet *Mp = nullptr;

    auto slice = [&](int s) -> int { return rev ? Gp->nz - 1 - s : s; };
    auto issue_z = [&](int s) {
        const int slot = s % ZS;
        if (tid == 0) {
            uint64_t *bar = &zbar[slot];
            const int z = slice(s);
            mbar_arrive_tx(bar, L::ztx());
            unsigned char *base = sm + slot * L::zslot();
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const int c = L::zcl(p);
                tma_load4(base + L::zpo(p), &Mp->m[c], bar, i0 - ((c & 1) ? HX : 0), j0 - ((c & 2) ? 1 : 0), z,
                          L::zpl(p));
            }
        }
        znext ^= 1u << slot;
    };
    auto issue_n = [&](int s) {
        const int slot = s % NS;
        if (tid == 0) {
            uint64_t *bar = &nbar[slot];
            const int z = slice(s);
            mbar_arrive_tx(bar, L::ntx());
            unsigned char *base = smn + slot * L::nslot();
            tma_load4(base + L::qoff(0), &Mp->one, bar, i0, j0, z, 0);
            tma_load4(base + L::qoff(19), &Mp->one, bar, i0, j0, z, 19);
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const int c = L::npc(p);
                tma_load4(base + L::npo(p), &Mp->m[c], bar, i0 - ((c & 1) ? HX : 0), j0 - ((c & 2) ? 1 : 0), z,
                          L::npl(p));
            }
            tma_load3(base + L::fo(), &Mp->fmap, bar, i0, j0, z);
            bulk_load(base + L::wo(), Gp->wgt[2] + (int64_t)z * 6, 48, bar);
        }
        nnext ^= 1u << slot;
    };
    const long long wlim = g_wait_limit;
    auto wait_z = [&](int s) -> bool { return mbar_wait(&zbar[s % ZS], ((znext >> (s % ZS)) & 1u) ^ 1u, wlim); };
    auto wait_n = [&](int s) -> bool { return mbar_wait(&nbar[s % NS], ((nnext >> (s % NS)) & 1u) ^ 1u, wlim); };

    bool aborted = false, waited = false;

    for (int si = sbeg; si < send && !aborted; ++si) {
        const int4 sg = segs[rev ? sbeg + send - 1 - si : si];
        S *dst;
        C *Fout;
        const Bufs *Bp;
        cavity(sg.w, Gp, Mp, dst, Fout, Bp);
        if (kStage) Gp = stage_geo(Gp, sgeo);
        const RunCtl *ctl = Bp->ctl;
        if (!waited) {
            dep_wait();  // from here on: what earlier kernels wrote
            waited = true;
        }
        if (!ctl->active) continue;  // a cavity whose run has stopped
        const Geo &G = *Gp;
        const Bufs &B = *Bp;
        const int nz = G.nz;
        const int ntx = (G.nx + TX - 1) / TX;
        const int64_t P = G.plane;
        const int t = sg.x, ka = rev ? nz - sg.z : sg.y, kb = rev ? nz - sg.y : sg.z;  // mirrored from here on
        i0 = (t % ntx) * TX;
        j0 = (t / ntx) * TY;
        // the segment's z-slices: the first step's needs, then one slice per step
        const int pre_lo = need_lo(ka, nz), pre_hi = need_hi(ka, nz);
        const int seg_hi = max(need_hi(kb - 1, nz), pre_hi);
        int zissued = min(seg_hi, max(pre_hi, ka + ZS - 2)), nissued = min(kb - 1, ka + NS - 2);
        for (int s = pre_lo; s <= zissued; ++s) issue_z(s);
        for (int s = ka; s <= nissued; ++s) issue_n(s);

        const int i = i0 + tx, j = j0 + ty;
        const bool active = i < G.nx && j < G.ny;
        C xp[3], xm[3], yp[3], ym[3];
        int xa = 0, xb = 0, ya = 0, yb = 0;
        C Tcn = C(0.0), sTc = C(0.0);  // conduction profile at the node's y and its streaming shift
        if (active) {
            load_w(G.wgt[0], i, xp, xm);
            load_w(G.wgt[1], j, yp, ym);
            if (Tr<ST>::kDevT) {
                Tcn = C(tc_value(G, j));
                sTc = C((1.0 / 12.0) * G.dt * tc_gradient(G));
            }
            xa = off_a(i, G.nx); xb = off_b(i, G.nx);
            ya = off_a(j, G.ny); yb = off_b(j, G.ny);
        } else {
#pragma unroll
            for (int e = 0; e < 3; ++e) xp[e] = xm[e] = yp[e] = ym[e] = C(0.0);
        }
        // element index of the thread's node in a box of class c
        auto ix = [&](int c) -> int { return (ty + ((c & 2) ? 1 : 0)) * L::bx(c) + tx + ((c & 1) ? HX : 0); };
        const int r2a = ya * L::bx(2), r2b = yb * L::bx(2);
        // plane zi of the slice in slot base b, interpolated in x or y
        auto V = [&](const unsigned char *b, int zi) -> C {
            const int c = L::zc(zi);
            const S *q = (const S *)(b + L::zoff(zi)) + ix(c);
            if (c == 0) return tocomp(q[0]);
            if (c == 1) {
                const C(&w)[3] = (zi & 1) ? xm : xp;  // 11 13: +x, 12 14: -x
                return ip3(w, tocomp(q[xa]), tocomp(q[0]), tocomp(q[xb]));
            }
            const C(&w)[3] = (zi & 1) ? ym : yp;      // 15 17: +y, 16 18: -y
            return ip3(w, tocomp(q[r2a]), tocomp(q[0]), tocomp(q[r2b]));
        };
        // the planes that move towards +z: 5, 11 12, 15 16, 24
        auto up = [](int zi) { return zi == 0 || zi == 2 || zi == 3 || zi == 6 || zi == 7 || zi == 10; };
        C va[12], vb[12];  // the planes' values in slices k - 1 and k
        auto read = [&](C(&v)[12], int s) {
            const unsigned char *b = sm + (s % ZS) * L::zslot();
#pragma unroll
            for (int zi = 0; zi < 12; ++zi) v[zi] = V(b, zi);
        };
#pragma unroll
        for (int zi = 0; zi < 12; ++zi) va[zi] = vb[zi] = C(0.0);
        bool ok = true;
        for (int s = pre_lo; s <= ka; ++s) ok = ok && wait_z(s);
        if (ok) {
            if (ka > 0) read(va, ka - 1);
            read(vb, ka);
        }
        __syncthreads();  // slice ka - 1 is read: its slot may be refilled

        for (int m = ka; m < kb; ++m) {
            const int k = slice(m);
            // refill the slots of the slices read last step: z-slice m - 1, plane slice m - 1 (not after a wait above
            // that gave up: a slot takes no copy before its last one was seen to land)
            if (ok && zissued < min(seg_hi, m + ZS - 1)) issue_z(++zissued);
            if (ok && nissued < min(kb - 1, m + NS - 1)) issue_n(++nissued);

            const int64_t id = (int64_t)k * G.slab + (int64_t)j * G.pitch + i;
            const bool end = m == 0 || m == nz - 1;
            for (int s = end ? need_lo(m, nz) : m + 1; s <= need_hi(m, nz); ++s) ok = ok && wait_z(s);
            ok = ok && wait_n(m);
            if (!ok) {
                atomicExch(err, 1);
                s_abort = 1;
            }
            if (active && ok) {
                const unsigned char *nb = smn + (m % NS) * L::nslot(), *zb = sm + (m % ZS) * L::zslot();
                C vc[12], o[12];  // the values in slice k + 1; the outputs
                if (m < nz - 1) read(vc, m + 1);
                {
                    const double *w = (const double *)(nb + L::wo());
                    if (!end) {
                        const int wl = rev ? 2 : 0;  // the weight of the slice behind
                        const C zp[3] = {C(w[wl]), C(w[1]), C(w[2 - wl])};
                        const C zm[3] = {C(w[3 + wl]), C(w[4]), C(w[5 - wl])};
#pragma unroll
                        for (int zi = 0; zi < 12; ++zi) o[zi] = sym3(up(zi) ? zp : zm, va[zi], vb[zi], vc[zi]);
                    } else {
                        // the wall supplies one half of the planes, this window the others
                        C wp[3], wm[3];
                        window_weights(w, k, nz, wp, wm);
                        const unsigned char *xb = sm + ((m == 0 ? 2 : nz - 3) % ZS) * L::zslot();
#pragma unroll
                        for (int zi = 0; zi < 12; ++zi) {
                            const C mid = m == 0 ? vc[zi] : va[zi];
                            o[zi] = C(0.0);
                            if (k == 0 && !up(zi)) o[zi] = sym3(wm, vb[zi], mid, V(xb, zi));
                            if (k != 0 && up(zi)) o[zi] = sym3(wp, V(xb, zi), mid, vb[zi]);
                        }
                    }
                }
                const C Fz0 = ((const C *)(nb + L::fo()))[ty * TX + tx];
                auto N = [&](int q, int off) -> C { return tocomp(((const S *)(nb + L::qoff(q)))[ix(L::qc(q)) + off]); };
                auto XI = [&](int q, const C(&w)[3]) -> C { return ip3(w, N(q, xa), N(q, 0), N(q, xb)); };
                auto YI = [&](int q, const C(&w)[3]) -> C { return ip3(w, N(q, r2a), N(q, 0), N(q, r2b)); };
                const int r3a = ya * L::bx(3), r3b = yb * L::bx(3);
                // xoy (3M:807-824): y-interpolation on three x-columns, then x
                auto XY = [&](int q, const C(&wx)[3], const C(&wy)[3]) -> C {
                    auto Y = [&](int dx) -> C { return ip3(wy, N(q, dx + r3a), N(q, dx), N(q, dx + r3b)); };
                    return ip3(wx, Y(xa), Y(0), Y(xb));
                };
                C f[19], gg[7];
                f[0] = N(0, 0);
                f[1] = XI(1, xp);
                f[2] = XI(2, xm);
                f[3] = YI(3, yp);
                f[4] = YI(4, ym);
                f[7] = XY(7, xp, yp);
                f[8] = XY(8, xm, yp);
                f[9] = XY(9, xp, ym);
                f[10] = XY(10, xm, ym);
                gg[0] = N(19, 0);
                gg[1] = XI(20, xp);
                gg[2] = XI(21, xm);
                gg[3] = YI(22, yp);
                gg[4] = YI(23, ym);
                // z-reaching planes (3M:767-804): x or y first, then z
                f[5] = o[0]; f[6] = o[1];
#pragma unroll
                for (int zi = 2; zi < 10; ++zi) f[9 + zi] = o[zi];
                gg[5] = o[10]; gg[6] = o[11];
                // deviation from the conduction profile along y (the heated axis)
                if (Tr<ST>::kDevT) {
                    gg[3] -= sTc;
                    gg[4] += sTc;
                }

                // walls: bounceback_u / bounceback_T (3B:1053-1197), centre values of slice k
                auto CN = [&](int q) -> C { return N(q, 0); };
                auto CZ = [&](int q) -> C {
                    const int zi = q < 7 ? q - 5 : (q < 19 ? q - 9 : q - 14);
                    return tocomp(((const S *)(zb + L::zoff(zi)))[ix(L::zc(zi))]);
                };
                const C two_wT = C(2.0) * (C(1.0) / C(12.0));
                if (j == 0) {
                    f[3] = CN(4); f[7] = CN(10); f[8] = CN(9); f[15] = CZ(18); f[17] = CZ(16);
                    gg[3] = -CN(23) + two_wT * (Tr<ST>::kDevT ? C(G.Thot) - Tcn : C(G.Thot));
                }
                if (j == G.ny - 1) {
                    f[4] = CN(3); f[9] = CN(8); f[10] = CN(7); f[16] = CZ(17); f[18] = CZ(15);
                    gg[4] = -CN(22) + two_wT * (Tr<ST>::kDevT ? C(G.Tcold) - Tcn : C(G.Tcold));
                }
                if (i == 0) {
                    f[1] = CN(2); f[9] = CN(8); f[7] = CN(10); f[13] = CZ(12); f[11] = CZ(14);
                    gg[1] = CN(21);
                }
                if (i == G.nx - 1) {
                    f[2] = CN(1); f[8] = CN(9); f[10] = CN(7); f[12] = CZ(13); f[14] = CZ(11);
                    gg[2] = CN(20);
                }
                if (k == 0) {
                    f[5] = CZ(6); f[11] = CZ(14); f[12] = CZ(13); f[15] = CZ(18); f[16] = CZ(17);
                    gg[5] = CZ(25);
                }
                if (k == nz - 1) {
                    f[6] = CZ(5); f[13] = CZ(12); f[14] = CZ(11); f[17] = CZ(16); f[18] = CZ(15);
                    gg[6] = CZ(24);
                }

                // macro_u / macro_t (3M:988-1025) and the collision
                C rho, u, v, w, T, fp[19], gp[7], Fz;
                node3d<C, Tr<ST>::kShift, Tr<ST>::kDevT>(f, gg, Fz0, G, fp, gp, Fz, rho, u, v, w, T, Tcn);
                if (write_macro) {
                    const int64_t mid = ((int64_t)k * G.ny + j) * G.nx + i;
                    B.rho[mid] = double(rho); B.u[mid] = double(u); B.v[mid] = double(v);
                    B.w[mid] = double(w); B.T[mid] = double(T);
                }
                Fout[id] = Fz;
#pragma unroll
                for (int q = 0; q < 19; ++q) dst[q * P + id] = tostore<S, C>(fp[q]);
#pragma unroll
                for (int q = 0; q < 7; ++q) dst[(19 + q) * P + id] = tostore<S, C>(gp[q]);
#pragma unroll
                for (int zi = 0; zi < 12; ++zi) {
                    va[zi] = vb[zi];
                    vb[zi] = vc[zi];
                }
            }
            __syncthreads();
            if (s_abort) {
                aborted = true;
                break;
            }
        }
    }
    if (aborted && tid == 0) {
        // let copies still in flight land before the CTA's shared memory is released
        for (int s = 0; s < ZS; ++s) mbar_wait(&zbar[s], ((znext >> s) & 1u) ^ 1u);
        for (int s = 0; s < NS; ++s) mbar_wait(&nbar[s], ((nnext >> s) & 1u) ^ 1u);
    }
}
