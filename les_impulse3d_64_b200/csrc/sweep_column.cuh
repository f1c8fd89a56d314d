// sweep_column.cuh - the packed FP32 momentum sweep as a walk up columns of cells: every edge evaluated once, two layers
// of a column at a time.
//
// A CTA owns TX x TY columns of cells and 2 H layers of them, and walks layers z and z + H together, one in each half of
// the FP32x2 instructions (F2, sweep_pair.cuh); a thread owns one column of the tile or of the ring of columns around it
// that its edges reach (RX x RY = (TX + 3) x (TY + 3) columns).  At layer z a thread
//   - evaluates the z-edge of its column at layer z and the y- and x-edges on z-face z + 2, each in the narrow and the
//     wide form (backend.cu:141-215): one vorticity, and its product with the interpolated velocity for either family of
//     faces that takes the edge;
//   - hands the products that faces of other columns take (a z-edge's to the u-faces along y and the v-faces along x, an
//     x-edge's to the w-faces along y, a y-edge's to the w-faces along x) and K = u.m over in shared memory, one pair
//     per column, and keeps those that faces of its own column take (a y-edge's for its u-faces, an x-edge's for its
//     v-faces) for the layers above and below in registers;
//   - completes its three lower faces: the sum of the products, -grad K, the viscous flux Laplacian with its wall and lid
//     fluxes, and the RK combination (backend.cu:232-330).
// Layers of the velocity and the impulse are staged once each into shared-memory rings of pairs (cp.async, two layers
// ahead, every thread its own column and one element of the rim); a column's values at the layers around z roll through
// registers.  Stage 0's gauge-reset blend (backend.cu:880-881) is applied by each thread to its own element of a layer
// when it lands.  Values staged outside the box are clamped copies (along y, z) or zeros (along x); every term that
// reaches them has weight zero (layout.h).
//
// What bounds the tile sweep is the L1 data pipe and instruction issue (1,220 thread instructions per cell, 72% of the
// pipe): each face evaluates its wide edges itself, and a tile stages 3.4 velocities per cell and component.  The walk
// issues 626 per cell and reads a staged pair once per edge.  16 x 16 columns are the most that leave a thread its 160
// registers (12 warps; 32 x 8 have 1.50 columns per useful one, these 1.41), and a pair holds layers of two half chunks
// because the pair's halves then share every x and y table value.  Tables stay in shared memory, in both halves: as
// register pairs they spilled (128^3, one sweep 130 us, so 117).  The branches on the order, on walls and on the layers
// before the chunk are compile-time and a layer's stores come after its loads, so the loads overlap (117 us, so 99).
// Measured against the tile sweep, us per sweep: 256^3 567 and 810, 164 x 164 x 93 122 and 156, 128^3 92 and 110, 96^3
// 45 and 51, 64 x 64 x 128 33 and 36, seven 64^3 100 and 109.  What bounds it now is the latency of shared-memory reads
// with three warps on a scheduler (issue 50%, data pipe 51%).
//
// The expressions and the order of every sum are sweep_pair.cuh's, so the results are its results bit for bit (a sign
// that it applies to a product is applied here to the factor or to the sum, which rounds the same).
#pragma once
#include "sweep_pair.cuh"

#include <type_traits>

namespace cavity {

// a column's table values (layout.h); kCL3 scaled by -1/8, kCInvWm and kCInvSp1 at the indices before and after
enum ColTab : int { kCOk1 = 0, kCL1, kCL3, kCInvSp, kCInvNd3, kCEv1Lo, kCEv1Hi, kCEv3Lo, kCEv3Hi, kCC3, kCInvW, kCInvWm,
                    kCInvSp1, kColTabs };

template <int TX_, int TY_> struct ColumnGeom {
    static constexpr int TX = TX_, TY = TY_;
    static constexpr int RX = TX + 3, RY = TY + 3;                 // columns (x0 - 1 ..) x (y0 - 1 ..)
    static constexpr int COLS = RX * RY, NT = (COLS + 31) / 32 * 32;
    // Row pitch of a layer of `w` columns: RX mod 16, so that the 64-bit reads of a half warp that runs over the end of a
    // row of threads fall on 16 different bank pairs.
    static constexpr int pitch(int w) { return w + (RX - w % 16 + 32) % 16; }
    // layers: u on x [x0-1, x0+TX+1] x y [y0-3, y0+TY+2]; v on x [x0-3, x0+TX+2] x y [y0-1, y0+TY+1];
    // w on x [x0-3, x0+TX+2] x y [y0-3, y0+TY+2]; impulse on the threads' columns
    static constexpr int UC = RX, UW = pitch(UC), UH = TY + 6, NU = UW * UH;
    static constexpr int VC = TX + 6, VW = pitch(VC), VH = RY, NV = VW * VH;
    static constexpr int WC = TX + 6, WW = pitch(WC), WH = TY + 6, NW = WW * WH;
    static constexpr int MC = RX, MW = pitch(MC), MH = RY, NM = MW * MH;
    static constexpr int SU = 5, SW = 2, SM = 4;                   // ring depths (u and v; w; each impulse component)
    static constexpr int NX = 9;                                   // exchanged pairs per column (two sets)
    static constexpr int RIM = 3 * UC + 3 * VH + (WC * WH - COLS); // elements of a layer outside the threads' columns
    static_assert(RIM <= NT, "one rim element per thread");
    static constexpr int ELEMS = SU * (NU + NV) + SW * NW + 3 * SM * NM + 2 * NX * COLS;
    static constexpr int HMAX = 64;                                // most layers of half a chunk (its z tables are staged)
    static constexpr size_t smem_bytes() { return sizeof(float2) * (size_t)(ELEMS + kNumTabs * (HMAX + 5) + kColTabs * (COLS + RY)); }
};

__device__ __forceinline__ F2 lds2(const float2* p) { return {*p}; }

template <class G, bool O4, bool EDGE> __device__ __forceinline__ void sweep_column_walk(const MomentumArgs<float>& a, const Blk& blk) {
    constexpr int TX = G::TX, TY = G::TY, RX = G::RX, RY = G::RY, COLS = G::COLS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* const SUb = reinterpret_cast<float2*>(smem_raw);
    float2* const SVb = SUb + G::SU * G::NU;
    float2* const SWb = SVb + G::SU * G::NV;
    float2* const SMb = SWb + G::SW * G::NW;                       // mx, my, mz: SM layers each
    float2* const EXb = SMb + 3 * G::SM * G::NM;
    float2* const TZ = EXb + 2 * G::NX * COLS;
    const Params& p = a.p;
    const Geo<float>& g = a.g;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const int H = (nz + 2 * (int)blk.nz - 1) / (2 * (int)blk.nz);
    const int x0 = blk.x * TX, y0 = blk.y * TY, z0 = blk.z * 2 * H, zend = min(nz, z0 + H);
    if (z0 >= nz) return;
    const int t = min((int)threadIdx.x, COLS - 1);          // the last warp's spare lanes repeat the last column
    const int ix = t % RX, iy = t / RX;
    const int x = x0 - 1 + ix, y = y0 - 1 + iy;
    const bool blend = a.stage == 0, rk = a.stage > 0;
    const bool out = (int)threadIdx.x < COLS && ix >= 1 && ix <= TX && iy >= 1 && iy <= TY && x < nx && y < ny;

    // z tables of the chunk: entry i of table k holds indices z0 - 2 + i and z0 + H - 2 + i
    const int zs = H + 5;
    for (int e = threadIdx.x; e < kNumTabs * zs; e += G::NT) {
        const int k = e / zs, i = e % zs;
        const float* src = g.tab[Z] + k * g.stride[Z] + kTabOffset;
        cp_async_elem<4>(&TZ[e].x, src + clampi(z0 - 2 + i, -2, nz + 2));
        cp_async_elem<4>(&TZ[e].y, src + clampi(z0 + H - 2 + i, -2, nz + 2));
    }
    // x and y tables, each value in both halves, the x tables an entry per column (read without bank conflicts)
    float2* const XT = TZ + kNumTabs * (G::HMAX + 5);
    float2* const YT = XT + kColTabs * COLS;
    {
        constexpr int tabs[kColTabs] = {kOk1, kL1, kL3, kInvSp, kInvNd3, kEv1Lo, kEv1Hi, kEv3Lo, kEv3Hi, kC3, kInvW, kInvW, kInvSp};
        auto entry = [&](int axis, int k, int i, int n) {
            float v = tab(g, axis, tabs[k], clampi(i + (k == kCInvSp1) - (k == kCInvWm), -2, n + 2));
            
            if (k == kCL3) v *= -0.125f;
            return make_float2(v, v);
        };
#pragma unroll
        for (int k = 0; k < kColTabs; k++) {
            XT[k * COLS + t] = entry(X, k, x, nx);
            if (threadIdx.x < RY) YT[k * RY + threadIdx.x] = entry(Y, k, y0 - 1 + (int)threadIdx.x, ny);
        }
    }
    const float2* const tx = XT + t;
    const float2* const ty = YT + iy;
    auto cx = [&](int k) { return lds2(tx + k * COLS); };
    auto cy = [&](int k) { return lds2(ty + k * RY); };

    // ---- staging: this thread's own column of every array, and one rim element of u, v or w
    const int su = (nx + 1) * ny, sv = nx * (ny + 1), sw = nx * ny;          // layer strides
    const int cxu = clampi(x, 0, nx), cxc = clampi(x, 0, nx - 1), cyv = clampi(y, 0, ny), cyc = clampi(y, 0, ny - 1);
    const int gu = cxu + (nx + 1) * cyc, gv = cxc + nx * cyv, gw = cxc + nx * cyc;
    const int ou = (iy + 2) * G::UW + ix, ov = iy * G::VW + ix + 2, ow = (iy + 2) * G::WW + ix + 2, om = iy * G::MW + ix;
    const bool real = (int)threadIdx.x < COLS;
    const bool inu = real && x >= 0 && x <= nx, inc = real && x >= 0 && x < nx;      // on an x-face / in a cell of the box
    int rim = -1, rg = 0, rs = 0, rx = 0;                                    // array (0 u, 1 v, 2 w), offsets, x
    if (t < 3 * G::UC) {                                                     // u: rows 0, 1 and UH - 1
        const int r = t / G::UC, i = t % G::UC, row = r == 2 ? G::UH - 1 : r;
        rim = 0;
        rs = row * G::UW + i;
        rx = x0 - 1 + i;
        rg = rx + (nx + 1) * clampi(y0 - 3 + row, 0, ny - 1);
    } else if (t < 3 * G::UC + 3 * G::VH) {                                  // v: columns 0, 1 and VC - 1
        const int e = t - 3 * G::UC, c = e / G::VH, row = e % G::VH, i = c == 2 ? G::VC - 1 : c;
        rim = 1;
        rs = row * G::VW + i;
        rx = x0 - 3 + i;
        rg = rx + nx * clampi(y0 - 1 + row, 0, ny);
    } else if (t < G::RIM) {                                                 // w: its rows 0, 1, WH - 1, then columns
        const int e = t - 3 * G::UC - 3 * G::VH;
        int row, i;
        if (e < 3 * G::WC) {
            row = e / G::WC;
            i = e % G::WC;
            if (row == 2) row = G::WH - 1;
        } else {
            const int f = e - 3 * G::WC, c = f / RY;
            row = 2 + f % RY;
            i = c == 2 ? G::WC - 1 : c;
        }
        rim = 2;
        rs = row * G::WW + i;
        rx = x0 - 3 + i;
        rg = rx + nx * clampi(y0 - 3 + row, 0, ny - 1);
    }
    // Columns outside the box along x stay zero: lanes that all copied the same clamped element would take turns (164 x
    // 164 x 93, whose last tile has 4 of 16 columns: that tile's CTAs 350 thousand cycles, the others 225; 185 us per
    // sweep, so 122).
    const float2 none = make_float2(0.f, 0.f);
    if (real && !inu) {
        for (int s = 0; s < G::SU; s++) SUb[s * G::NU + ou] = none;
        for (int s = 0; s < G::SM; s++) SMb[s * G::NM + om] = none;
    }
    if (real && !inc) {
        for (int s = 0; s < G::SU; s++) SVb[s * G::NV + ov] = none;
        for (int s = 0; s < G::SW; s++) SWb[s * G::NW + ow] = none;
        for (int s = G::SM; s < 3 * G::SM; s++) SMb[s * G::NM + om] = none;
    }
    if (rx < 0 || rx >= nx + (rim == 0)) {
        float2* const ring = rim == 0 ? SUb : rim == 1 ? SVb : SWb;
        const int slots = rim < 0 ? 0 : rim == 2 ? G::SW : G::SU, layer = rim == 0 ? G::NU : rim == 1 ? G::NV : G::NW;
        for (int s = 0; s < slots; s++) ring[s * layer + rs] = none;
        rim = -1;
    }
    auto pair_in = [&](float2* dst, const float* base, int lo, int hi) {
        cp_async_elem<4>(&dst->x, base + lo);
        cp_async_elem<4>(&dst->y, base + hi);
    };
    auto lay = [&](int z) { return clampi(z, 0, nz - 1); };                  // layer of a cell-centred z index
    auto fac = [&](int z) { return clampi(z, 0, nz); };                      // z-face
    // layers zu of u and v, zw of w, zm of the impulse (and H above), into ring slots
    auto stage = [&](int zu, int slu, int zw, int slw, int zm, int slm) {
        const int lu0 = lay(zu), lu1 = lay(zu + H), lw0 = fac(zw), lw1 = fac(zw + H);
        const int lm0 = lay(zm), lm1 = lay(zm + H), lz0 = fac(zm), lz1 = fac(zm + H);
        if (inu) {
            pair_in(SUb + slu * G::NU + ou, a.u[X] + gu, lu0 * su, lu1 * su);
            pair_in(SMb + slm * G::NM + om, a.m[X] + gu, lm0 * su, lm1 * su);
        }
        if (inc) {
            pair_in(SVb + slu * G::NV + ov, a.u[Y] + gv, lu0 * sv, lu1 * sv);
            pair_in(SWb + slw * G::NW + ow, a.u[Z] + gw, lw0 * sw, lw1 * sw);
            pair_in(SMb + (G::SM + slm) * G::NM + om, a.m[Y] + gv, lm0 * sv, lm1 * sv);
            pair_in(SMb + (2 * G::SM + slm) * G::NM + om, a.m[Z] + gw, lz0 * sw, lz1 * sw);
        }
        if (rim == 0) pair_in(SUb + slu * G::NU + rs, a.u[X] + rg, lu0 * su, lu1 * su);
        else if (rim == 1) pair_in(SVb + slu * G::NV + rs, a.u[Y] + rg, lu0 * sv, lu1 * sv);
        else if (rim == 2) pair_in(SWb + slw * G::NW + rs, a.u[Z] + rg, lw0 * sw, lw1 * sw);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    pdl_wait();
    // The walk begins three layers below the chunk: the wide y- and x-edges on z-face z0 - 1 are evaluated there.
    const int zb = z0 - 3;
    // columns' values below the first layer whose slots the walk reads: u, v at zb .. zb + 2, w at zb + 1
    F2 ur[4], vr[4], wr[3], mx[3], my[3], mz[3];
    {
#pragma unroll
        for (int i = 0; i < 3; i++) {
            ur[i + 1] = f2(__ldg(a.u[X] + gu + lay(zb + i) * su), __ldg(a.u[X] + gu + lay(zb + i + H) * su));
            vr[i + 1] = f2(__ldg(a.u[Y] + gv + lay(zb + i) * sv), __ldg(a.u[Y] + gv + lay(zb + i + H) * sv));
        }
        wr[2] = f2(__ldg(a.u[Z] + gw + fac(zb + 1) * sw), __ldg(a.u[Z] + gw + fac(zb + 1 + H) * sw));
        wr[1] = wr[2];
        mx[2] = my[2] = mz[2] = mx[1] = my[1] = mz[1] = f2(0.f);
    }
    const int failed = a.c->error;
    const StageConst sc = stage_const(a.stage, a.c);
    const float dt = (float)a.c->dt;
    if (failed) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        return;
    }
    const float lidv = (float)lid_speed(p, sc.tau);
    const float rka = (float)sc.a0, rkb = (float)sc.b, nu = a.nu, omr = a.one_minus_r, gr = a.r;
    const F2 zero = f2(0.f), half = f2(0.5f), mhalf = f2(-0.5f), one = f2(1.f), mone = f2(-1.f), unit = f2(a.one);
    auto sum = [&](F2 p0, F2 p1) { return fma2(p0, unit, p1); };

    F2 nU[2] = {zero, zero}, nV[2] = {zero, zero};            // narrow y- / x-edge products on z-faces z, z + 1
    F2 wU[3] = {zero, zero, zero}, wV[3] = {zero, zero, zero};    // wide ones on z-faces z - 1, z, z + 1
    F2 accW[2] = {zero, zero}, kbelow = zero;                // sums of the w-faces z, z + 1; K of layer z - 1
    int slu = 0, slw = 0, slm = 0, sle = 0;                  // slots of layers z + 3 (u, v), z + 2 (w), z + 1 (m); exchange set
    auto wrap = [](int s, int n) { return s >= n ? s - n : s; };
    // u and v of layer z0 - 1, which K there takes from the columns at x + 1 and y + 1, in the slot before layer z0's
    if (inu) pair_in(SUb + (G::SU - 1) * G::NU + ou, a.u[X] + gu, lay(zb + 2) * su, lay(zb + 2 + H) * su);
    if (inc) pair_in(SVb + (G::SU - 1) * G::NV + ov, a.u[Y] + gv, lay(zb + 2) * sv, lay(zb + 2 + H) * sv);
    stage(zb + 3, 0, zb + 2, 0, zb + 1, 0);
    stage(zb + 4, 1, zb + 3, 1, zb + 2, 1);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    F2 b0 = zero, b1 = zero, b2 = zero;                       // RK base of the faces at layer z

    auto layer = [&](int z, auto live_c) {
        constexpr bool live = decltype(live_c)::value;
        const bool up = z + H < nz;                           // the upper layer is inside the box
        if (live && rk && out) {
            b0 = f2(__ldg(a.m0[X] + gu + z * su), up ? __ldg(a.m0[X] + gu + (z + H) * su) : 0.f);
            b1 = f2(__ldg(a.m0[Y] + gv + z * sv), up ? __ldg(a.m0[Y] + gv + (z + H) * sv) : 0.f);
            b2 = f2(__ldg(a.m0[Z] + gw + z * sw), up ? __ldg(a.m0[Z] + gw + (z + H) * sw) : 0.f);
        }
        const int slz = wrap(slu + 2, G::SU);                               // slot of layer z (three layers earlier)
        const float2* pu = SUb + slz * G::NU + ou;
        const float2* pv = SVb + slz * G::NV + ov;
        const float2* pw = SWb + slw * G::NW + ow;
        const float2* pmx = SMb + wrap(slm + G::SM - 1, G::SM) * G::NM + om;    // the impulse's layer z
        const float2* pmy = pmx + G::SM * G::NM;
        const float2* pmz = pmy + G::SM * G::NM;
        float2* const q = SMb + slm * G::NM + om;                           // and this column's layer z + 1
        const float2* tz = TZ + (z - z0 + 2);                               // table k at index z + i: tz[k * zs + i]
        float2* const ex = EXb + sle * (G::NX * COLS) + t;
#pragma unroll
        for (int i = 0; i < 3; i++) { ur[i] = ur[i + 1]; vr[i] = vr[i + 1]; }
        ur[3] = lds2(SUb + slu * G::NU + ou);                               // layer z + 3
        vr[3] = lds2(SVb + slu * G::NV + ov);
        wr[0] = wr[1];
        wr[1] = wr[2];
        wr[2] = lds2(pw);                                                   // z-face z + 2
        mx[0] = mx[1]; my[0] = my[1]; mz[0] = mz[1];
        mx[1] = mx[2]; my[1] = my[2]; mz[1] = mz[2];
        mx[2] = lds2(q);
        my[2] = lds2(q + G::SM * G::NM);
        mz[2] = lds2(q + 2 * G::SM * G::NM);
        // ---- y- and x-edges on z-face f = z + 2 (u, v at layers f - 2 .. f + 1: ur[0 .. 3], vr[0 .. 3])
        constexpr int f = 2;
        F2 uYn, vXn, wYn, wXn, uYw = zero, vXw = zero, wYw = zero, wXw = zero;
        {
            const F2 okz = lds2(tz + kOk1 * zs + f), lz = lds2(tz + kL1 * zs + f), i1z = lds2(tz + kInvSp * zs + f),
                     e1lz = lds2(tz + kEv1Lo * zs + f), e1hz = lds2(tz + kEv1Hi * zs + f);
            const F2 wh = wr[2];
            {
                const F2 wl = lds2(pw - 1);
                F2 wt = okz * cx(kCOk1);
                if (O4) wt = wt * fma2(lz * cx(kCL1), f2(0.125f), one);
                const F2 wo = wt * fma2(ur[2] - ur[1], i1z, (wl - wh) * cx(kCInvSp));
                uYn = wo * fma2(cx(kCEv1Lo), wl, cx(kCEv1Hi) * wh);
                wYn = wo * fma2(e1lz, ur[1], e1hz * ur[2]);
            }
            {
                const F2 wl = lds2(pw - G::WW);
                F2 wt = cy(kCOk1) * okz;
                if (O4) wt = wt * fma2(lz * cy(kCL1), f2(0.125f), one);
                const F2 wo = wt * fma2(wh - wl, cy(kCInvSp), (vr[1] - vr[2]) * i1z);
                vXn = wo * fma2(cy(kCEv1Lo), wl, cy(kCEv1Hi) * wh);
                wXn = wo * fma2(e1lz, vr[1], e1hz * vr[2]);
            }
        }
        if (O4) {
            const F2 l3z = lds2(tz + kL3 * zs + f), i3z = lds2(tz + kInvNd3 * zs + f), e3lz = lds2(tz + kEv3Lo * zs + f),
                     e3hz = lds2(tz + kEv3Hi * zs + f);
            {
                const F2 wl = lds2(pw - 2), wh3 = lds2(pw + 1);
                const F2 wo = (l3z * cx(kCL3)) * fma2(ur[3] - ur[0], i3z, (wl - wh3) * cx(kCInvNd3));
                uYw = wo * fma2(cx(kCEv3Lo), wl, cx(kCEv3Hi) * wh3);
                wYw = wo * fma2(e3lz, ur[0], e3hz * ur[3]);
            }
            {
                const F2 wl = lds2(pw - 2 * G::WW), wh3 = lds2(pw + G::WW);
                const F2 wo = (l3z * cy(kCL3)) * fma2(wh3 - wl, cy(kCInvNd3), (vr[0] - vr[3]) * i3z);
                vXw = wo * fma2(cy(kCEv3Lo), wl, cy(kCEv3Hi) * wh3);
                wXw = wo * fma2(e3lz, vr[0], e3hz * vr[3]);
            }
        }
        // ---- z-edge at layer z, and K
        F2 uZn = zero, vZn = zero, uZw = zero, vZw = zero;
        if (live) {
            const F2 vl = lds2(pv - 1), vh = vr[0], ul = lds2(pu - G::UW), uh = ur[0];
            F2 wt = cx(kCOk1) * cy(kCOk1);
            if (O4) wt = wt * fma2(cx(kCL1) * cy(kCL1), f2(0.125f), one);
            const F2 wo = wt * fma2(vh - vl, cx(kCInvSp), (ul - uh) * cy(kCInvSp));
            uZn = wo * fma2(cx(kCEv1Lo), vl, cx(kCEv1Hi) * vh);
            vZn = wo * fma2(cy(kCEv1Lo), ul, cy(kCEv1Hi) * uh);
            if (O4) {
                const F2 vl3 = lds2(pv - 2), vh3 = lds2(pv + 1), ul3 = lds2(pu - 2 * G::UW), uh3 = lds2(pu + G::UW);
                const F2 wo3 = (cx(kCL3) * cy(kCL3) * f2(-8.f)) * fma2(vh3 - vl3, cx(kCInvNd3), (ul3 - uh3) * cy(kCInvNd3));
                uZw = wo3 * fma2(cx(kCEv3Lo), vl3, cx(kCEv3Hi) * vh3);
                vZw = wo3 * fma2(cy(kCEv3Lo), ul3, cy(kCEv3Hi) * uh3);
            }
        }
        if (blend) {
            mx[2] = fma2(f2(gr), mx[2], f2(omr) * ur[1]);
            my[2] = fma2(f2(gr), my[2], f2(omr) * vr[1]);
            mz[2] = fma2(f2(gr), mz[2], f2(omr) * wr[1]);
        }
        // (the last columns and rows of the ring read past their layers here: no face takes their K)
        const F2 kc = half * (fma2(ur[0], mx[1], lds2(pu + 1) * lds2(pmx + 1)) +
                              fma2(vr[0], my[1], lds2(pv + G::VW) * lds2(pmy + G::MW)) + fma2(wr[0], mz[1], wr[1] * mz[2]));
        // stores last: a load after one would wait for it
        if (blend) {
            *q = mx[2].v;
            q[G::SM * G::NM] = my[2].v;
            q[2 * G::SM * G::NM] = mz[2].v;
        }
        ex[4 * COLS] = wYn.v;
        ex[6 * COLS] = wXn.v;
        ex[8 * COLS] = kc.v;
        if (O4) {
            ex[5 * COLS] = wYw.v;
            ex[7 * COLS] = wXw.v;
        }
        if (live) {
            ex[0] = uZn.v;
            ex[2 * COLS] = vZn.v;
            if (O4) {
                ex[1 * COLS] = uZw.v;
                ex[3 * COLS] = vZw.v;
            }
        }
        // the copies for layer z + 1's edges, issued one layer ago, have landed; then the next ones
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        const int nslu = wrap(slu + 1, G::SU), nslw = slw ^ 1, nslm = wrap(slm + 1, G::SM);
        if (z + 2 < zend) stage(z + 5, wrap(slu + 2, G::SU), z + 4, slw, z + 3, wrap(slm + 2, G::SM));
        if (out) {
            // w-face z + 2 takes the x-edges along y and the y-edges along x on its z-face
            F2 lw = fma2(mhalf, sum(lds2(ex + 6 * COLS + RX), wXn), half * sum(lds2(ex + 4 * COLS + 1), wYn));
            if (O4) {
                const F2 c3z = lds2(tz + kC3 * zs + 2);
                lw = fma2(mone * c3z, lds2(ex + 7 * COLS + 2 * RX) + lds2(ex + 7 * COLS - RX), lw);
                lw = fma2(c3z, lds2(ex + 5 * COLS + 2) + lds2(ex + 5 * COLS - 1), lw);
            }
            if constexpr (live) {
                const int gz = z * su + gu, gvz = z * sv + gv, gwz = z * sw + gw;
                const int hu = H * su, hv = H * sv, hw = H * sw;
                const F2 wz0 = lds2(tz + kInvW * zs), wzm = lds2(tz + kInvW * zs - 1), sz0 = lds2(tz + kInvSp * zs),
                         sz1 = lds2(tz + kInvSp * zs + 1);
                const bool zf = z == 0, zl0 = z == nz - 1, zl1 = z + H == nz - 1, zwall = zf || zl0 || zl1;
                const bool yf = y == 0, yl = y == ny - 1, xf = x == 0, xl = x == nx - 1;
                auto put = [&](float* o, int i, int h, F2 v) {
                    st_out(o + i, v.v.x);
                    if (up) st_out(o + i + h, v.v.y);
                };
                // viscous flux of a face along an axis across it, x or y, with the wall fluxes
                auto across = [&](F2 hi_, F2 cc, F2 lo_, F2 s1, F2 s0, F2 iw, bool first, bool last, F2 wall, F2 top, F2 lap) {
                    F2 hi = (hi_ - cc) * s1, lo = (cc - lo_) * s0;
                    if (EDGE) {
                        const F2 wh = (top - wall) * s1, wl = wall * s0;
                        hi = sel2(last, last, wh, hi);
                        lo = sel2(first, first, wl, lo);
                    }
                    return fma2(hi - lo, iw, lap);
                };
                // and along z
                auto across_z = [&](const F2* m, F2 wall, F2 lap) {
                    F2 hi = (m[2] - m[1]) * sz1, lo = (m[1] - m[0]) * sz0;
                    if (zwall) {                                             // the whole CTA
                        const F2 wh = wall * sz1;
                        hi = f2(zl0 ? -wh.v.x : hi.v.x, zl1 ? -wh.v.y : hi.v.y);
                        if (zf) lo = f2((wall * sz0).v.x, lo.v.y);
                    }
                    return fma2(hi - lo, wz0, lap);
                };
                auto rk_value = [&](F2 cc, F2 lap, F2 L, F2 base) {
                    F2 val = fma2(f2(dt), fma2(f2(nu), lap, L), cc);
                    if (rk) val = fma2(f2(rka), base, f2(rkb) * val);
                    return val;
                };
                // ---------------- u-face x
                {
                    if (blend) put(a.m0_out[X], gz, hu, mx[1]);
                    F2 val;
                    {
                        F2 L = fma2(mhalf, nU[1] + nU[0], half * sum(lds2(ex + RX), uZn));
                        if (O4) {
                            L = fma2(cx(kCC3), lds2(ex + COLS + 2 * RX) + lds2(ex + COLS - RX), L);
                            L = fma2(mone * cx(kCC3), sum(wU[0], uYw), L);
                        }
                        L = fma2(lds2(ex + 8 * COLS - 1) - kc, cx(kCInvSp), L);
                        const F2 cc = mx[1], wall = ur[0];
                        F2 lap = fma2(lds2(pmx + 1) - cc, cx(kCInvW), (lds2(pmx - 1) - cc) * cx(kCInvWm)) * cx(kCInvSp);
                        F2 top = zero;
                        if (EDGE && yl) top = f2(lidv) * f2(__ldg(g.lid_u + x + (nx + 1) * z), up ? __ldg(g.lid_u + x + (nx + 1) * (z + H)) : 0.f);
                        lap = across(lds2(pmx + G::MW), cc, lds2(pmx - G::MW), cy(kCInvSp1), cy(kCInvSp), cy(kCInvW), yf, yl, wall, top, lap);
                        lap = across_z(mx, wall, lap);
                        val = rk_value(cc, lap, L, b0);
                        if (EDGE) val = sel2(xf, xf, zero, val);
                    }
                    put(a.out[X], gz, hu, val);
                    if (EDGE && xl) {
                        if (blend) put(a.m0_out[X], gz + 1, hu, lds2(pmx + 1));
                        put(a.out[X], gz + 1, hu, zero);
                    }
                }
                // ---------------- v-face y
                {
                    if (blend) put(a.m0_out[Y], gvz, hv, my[1]);
                    F2 val;
                    {
                        F2 L = fma2(mhalf, sum(lds2(ex + 2 * COLS + 1), vZn), half * (nV[1] + nV[0]));
                        if (O4) {
                            L = fma2(mone * cy(kCC3), lds2(ex + 3 * COLS + 2) + lds2(ex + 3 * COLS - 1), L);
                            L = fma2(cy(kCC3), sum(wV[0], vXw), L);
                        }
                        L = fma2(lds2(ex + 8 * COLS - RX) - kc, cy(kCInvSp), L);
                        const F2 cc = my[1], wall = vr[0];
                        F2 lap = across(lds2(pmy + 1), cc, lds2(pmy - 1), cx(kCInvSp1), cx(kCInvSp), cx(kCInvW), xf, xl, wall, zero, zero);
                        lap = fma2((lds2(pmy + G::MW) - cc) * cy(kCInvW) - (cc - lds2(pmy - G::MW)) * cy(kCInvWm), cy(kCInvSp), lap);
                        lap = across_z(my, wall, lap);
                        val = rk_value(cc, lap, L, b1);
                        if (EDGE) val = sel2(yf, yf, zero, val);
                    }
                    put(a.out[Y], gvz, hv, val);
                    if (EDGE && yl) {
                        if (blend) put(a.m0_out[Y], gvz + nx, hv, lds2(pmy + G::MW));
                        put(a.out[Y], gvz + nx, hv, zero);
                    }
                }
                // ---------------- w-face z
                {
                    if (blend) put(a.m0_out[Z], gwz, hw, mz[1]);
                    const F2 L = fma2(kbelow - kc, sz0, accW[0]);
                    const F2 cc = mz[1], wall = wr[0];
                    F2 lap = across(lds2(pmz + 1), cc, lds2(pmz - 1), cx(kCInvSp1), cx(kCInvSp), cx(kCInvW), xf, xl, wall, zero, zero);
                    lap = across(lds2(pmz + G::MW), cc, lds2(pmz - G::MW), cy(kCInvSp1), cy(kCInvSp), cy(kCInvW), yf, yl, wall, zero, lap);
                    lap = fma2((mz[2] - cc) * wz0 - (cc - mz[0]) * wzm, sz0, lap);
                    const F2 val = rk_value(cc, lap, L, b2);
                    put(a.out[Z], gwz, hw, f2(zf ? 0.f : val.v.x, val.v.y));
                    if (zl0 || zl1) {                                        // the top wall's faces
                        const float mtop = zl0 ? mz[2].v.x : mz[2].v.y;
                        const int i = nz * sw + gw;
                        if (blend) st_out(a.m0_out[Z] + i, mtop);
                        st_out(a.out[Z] + i, 0.f);
                    }
                }
            }
            nU[0] = nU[1];
            nU[1] = uYn;
            nV[0] = nV[1];
            nV[1] = vXn;
            wU[0] = wU[1];
            wU[1] = wU[2];
            wU[2] = uYw;
            wV[0] = wV[1];
            wV[1] = wV[2];
            wV[2] = vXw;
            accW[0] = accW[1];
            accW[1] = lw;
            kbelow = kc;
        }
        slu = nslu;
        slw = nslw;
        slm = nslm;
        sle ^= 1;
    };
    const int zwarm = min(z0, zend);
#pragma unroll 1
    for (int z = zb; z < zwarm; z++) layer(z, std::false_type{});
#pragma unroll 1
    for (int z = z0; z < zend; z++) layer(z, std::true_type{});
    pdl_launch_dependents();
}

template <class G> __device__ __forceinline__ void sweep_column_body(const MomentumArgs<float>& a, const Blk& blk) {
    const Params& p = a.p;
    const int x0 = blk.x * G::TX, y0 = blk.y * G::TY;
    const bool edge = x0 == 0 || y0 == 0 || x0 + G::TX >= p.nx || y0 + G::TY >= p.ny;     // holds faces next to a wall
    if (p.o4) {
        if (edge) sweep_column_walk<G, true, true>(a, blk);
        else sweep_column_walk<G, true, false>(a, blk);
    } else {
        sweep_column_walk<G, false, true>(a, blk);
    }
}

template <int TX, int TY>
__global__ void __launch_bounds__(ColumnGeom<TX, TY>::NT, 1) sweep_column_kernel(MomentumArgs<float> a) {
    sweep_column_body<ColumnGeom<TX, TY>>(a, real_blk());
}
// a batch of cavities: grid x runs over the work list (BatchItem)
template <int TX, int TY>
__global__ void __launch_bounds__(ColumnGeom<TX, TY>::NT, 1) sweep_column_batched(const MomentumArgs<float>* args,
                                                                                 const BatchItem* items, const int* live) {
    __shared__ MomentumArgs<float> a;
    int cav;
    const Blk k = item_blk(items, live, cav);
    if (cav < 0) return;
    load_args(a, args + cav);
    sweep_column_body<ColumnGeom<TX, TY>>(a, k);
}

}  // namespace cavity
