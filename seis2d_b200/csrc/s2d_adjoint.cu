// Adjoint FD step and gradient finalisation of libseis2d (sm_100a).
//
// The forward step (cpumodelling.cpp:115-156) written with its derivatives
//   a = Gx vx, c = Gz vz                      (D-, cpu_modelling_kernels.cpp:201-258)
//   px' = Dax px + Kx kappa a (+ source),  pz' = Daz pz + Kz kappa c
//   p' = px' + pz',  g = Hx p', h = Hz p'    (D+, :260-316)
//   vx' = Dbx vx + Lx bx g,  vz' = Dbz vz + Lz bz h
// is linear in the state.  One adjoint step maps the adjoint state after step
// kt, (mpx', mpz', mvx', mvz'), to the one before it:
//   mg = Lx bx mvx',  mh = Lz bz mvz'
//   q  = Hx^T mg + Hz^T mh (+ the adjoint source at the receivers)
//   mPX = mpx' + q,  mPZ = mpz' + q
//   mpx = Dax mPX,  mpz = Daz mPZ
//   mvx = Dbx mvx' + Gx^T (Kx kappa mPX),  mvz = Dbz mvz' + Gz^T (Kz kappa mPZ)
// and accumulates the imaging terms
//   dJ/dkappa += Kx a mPX + Kz c mPZ,  dJ/dbx += Lx g mvx',  dJ/dbz += Lz h mvz'
// with a, c, g, h of step kt saved by the forward (S2D_STEP_PRODUCTS); the
// last two go straight into dJ/db through the buoyancy averages.  All shots of
// a gradient call share one model, so they share one accumulator pair
// (dJ/dkappa, dJ/db): the terms are added with vector atomics (red.global
// .add.v4.f32), which keeps the pair in L2 instead of reading and writing a
// pair per shot from DRAM every step.  The order in which the shots' terms
// of one step arrive is not fixed, so gradients of several shots are
// reproducible to rounding, not bit for bit; one shot's are bit-exact.
//
// The transposes are the gather forms of the reference's operators, edge rows
// included: with (c0(j), c1(j)) the coefficient pair of forward row j,
//   (G^T m)[i] = c0(i) m[i] - c0(i+1) m[i+1] + c1(i-1) m[i-1] - c1(i+2) m[i+2]
//   (H^T m)[i] = c0(i-1) m[i-1] - c0(i) m[i] + c1(i-2) m[i-2] - c1(i+1) m[i+1]
// The kernel streams like the forward: a warp owns a 128-row strip, q and the
// pressure adjoint at column L-1, the velocity adjoint at column L-3.
#include <cuda_runtime.h>

#include "s2d_device.cuh"
#include "s2d_pack.cuh"

namespace s2d {

namespace {

// Kinds of tasks: interior (literal row and column coefficients, every cell
// carrying one pressure); interior columns, other rows; anything.
enum { kAdjIn = 0, kAdjRows = 1, kAdjAny = 2 };

// t0 a + t1 b + t2 c + t3 d, second product rounded, then fused in the order of
// t0, t2, t3 (the transposes' four taps; t1 and t3 hold the negated
// coefficients).
__device__ __forceinline__ V4 taps4(const V4 &t0, const V4 &a, const V4 &t1, const V4 &b, const V4 &t2, const V4 &c,
                                    const V4 &t3, const V4 &d) {
    return fma4(t3, d, fma4(t2, c, fma4(t0, a, t1 * b)));
}
struct Taps {
    V4 t0, t1, t2, t3;
};
// The taps of a lane's rows.  Even rows round and fuse as taps4, odd rows round
// the first product and fuse the second (the sums that this kernel's results
// have always had, kept bit for bit); a packed pair does both when the odd
// halves of the first two coefficients, and of their operands, change places.
__device__ __forceinline__ Taps row_taps(const V4 &t0, const V4 &t1, const V4 &t2, const V4 &t3) {
    return Taps{v4(pk(lo(t0.a), hi(t1.a)), pk(lo(t0.b), hi(t1.b))), v4(pk(lo(t1.a), hi(t0.a)), pk(lo(t1.b), hi(t0.b))), t2,
                t3};
}
// (H^T m) along z of the lane's rows: taps m[z-1], m[z], m[z-2], m[z+1].
__device__ __forceinline__ V4 hzt(const Taps &t, const V4 &m) {
    const float x = lo(m.a), y = hi(m.a), z = lo(m.b), w = hi(m.b);
    const float up_z = __shfl_up_sync(kFull, z, 1), up_w = __shfl_up_sync(kFull, w, 1);
    const float dn_x = __shfl_down_sync(kFull, x, 1);
    return taps4(t.t0, v4(pk(up_w, y), pk(y, w)), t.t1, v4(dup(x), dup(z)), t.t2, v4(pk(up_z, up_w), m.a), t.t3,
                 v4(pk(y, z), pk(w, dn_x)));
}
// (G^T m): taps m[z], m[z+1], m[z-1], m[z+2].
__device__ __forceinline__ V4 gzt(const Taps &t, const V4 &m) {
    const float x = lo(m.a), y = hi(m.a), z = lo(m.b), w = hi(m.b);
    const float up_w = __shfl_up_sync(kFull, w, 1);
    const float dn_x = __shfl_down_sync(kFull, x, 1), dn_y = __shfl_down_sync(kFull, y, 1);
    return taps4(t.t0, v4(pk(x, z), pk(z, dn_x)), t.t1, v4(dup(y), dup(w)), t.t2, v4(pk(up_w, x), pk(y, z)), t.t3,
                 v4(m.b, pk(dn_x, dn_y)));
}

// The adjoint source (transpose of the receiver sampling,
// cpumodelling.cpp:356-360) of a task whose columns come in order.  The
// receivers of column Q, and the first one's sample, are read ahead: the first
// one's row and trace two columns, its sample one.
struct AdjSource {
    int j, je, jn, z, z1, id1;
    float v;
    __device__ __forceinline__ void entry(const ShotDev &S, int e, int &zz, int &id) {
        e = min(e, S.nrec - 1);
        zz = __ldg(S.rec_z + e);
        id = __ldg(S.rec_id + e);
    }
    __device__ __forceinline__ float sample(const ShotDev &S, int id, int slot) {
        return __ldg(S.seis + (size_t)id * S.real_nt + slot);
    }
    __device__ __forceinline__ void start(const ShotDev &S, int Q, int slot) {
        j = __ldg(S.rec_ptr + Q);
        je = __ldg(S.rec_ptr + min(Q + 1, S.nnx));
        jn = __ldg(S.rec_ptr + min(Q + 2, S.nnx));
        int id;
        entry(S, j, z, id);
        v = sample(S, id, slot);
        entry(S, je, z1, id1);
    }
    __device__ __forceinline__ void add(V4 &q, int d, float r) {
        if (d == 0) q.a = pk(lo(q.a) + r, hi(q.a));
        else if (d == 1) q.a = pk(lo(q.a), hi(q.a) + r);
        else if (d == 2) q.b = pk(lo(q.b) + r, hi(q.b));
        else if (d == 3) q.b = pk(lo(q.b), hi(q.b) + r);
    }
    // Adds column Q's samples to the lane's rows z0 .. z0+3 of q.
    __device__ __forceinline__ void column(const ShotDev &S, int Q, int z0, int slot, V4 &q) {
        if (j < je) {
            add(q, z - z0, v);
            for (int e = j + 1; e < je; ++e) {
                int zz, id;
                entry(S, e, zz, id);
                if (zz - z0 >= 0 && zz - z0 < 4) add(q, zz - z0, sample(S, id, slot));
            }
        }
        j = je;
        je = jn;
        jn = __ldg(S.rec_ptr + min(Q + 3, S.nnx));
        z = z1;
        v = sample(S, id1, slot);
        entry(S, je, z1, id1);
    }
};

// One (shot, strip, segment) task of the adjoint step.  The warp streams
// along x: iteration L brings mvx' and bx at L (the x-gather of H^T needs Lx bx
// mvx' at Q-2 .. Q+1); the pressure adjoint, the z-velocity adjoint and the
// imaging terms are formed at Q = L-1, the x-velocity adjoint at W = L-3 (its
// G^T x-gather needs Kx kappa mPX at W-1 .. W+2).
//
// Cells where both pressure dampings are 1 run the forward with p alone
// (p' = p + kappa (Kx a + Kz c)); their adjoint carries one pressure field
// (mpx, mpz unused) and the forward saved Kx a + Kz c in the first product
// slot.
//
// Imaging per step: dJ/dkappa += Kx a mPX + Kz c mPZ at Q.  The buoyancy
// terms tbx = Lx g mvx', tbz = Lz h mvz' enter dJ/db through the averages
// bx = (b[x] + b[x+1]) / 2, bz = (b[z] + b[z+1]) / 2 (cpu_modelling_kernels.cpp:89-119):
// dJ/db(Q, z) += (tbx(Q) + tbx(Q-1)) / 2 + (tbz(z) + tbz(z-1)) / 2.
// tbx at the last column and tbz at the last row vanish (the forward D+
// rows there are zero), so the reference's last-row / last-column
// replication adds nothing.  tbx(Q-1) comes from the previous column
// (computed at Q = xa-1 too), tbz(z-1) from the lane above.
//
// The inputs come as per-lane asynchronous copies (16 bytes, the lane's four
// rows) into a per-warp ring, AdjDepth - 1 iterations ahead; the windows are
// registers, rotating through the names of a loop unrolled by four (interior
// tasks) or moved (the others, whose code then stays short).
//
// What bounds it: the latency of one column's chain (ring reads, three rounds
// of shuffles), with two warps on each scheduler.  1201x401, 8 shots: 69.6
// us/step (75.5 when every iteration brought all its pieces), before with the
// windows in shared memory 104 us/step.  Three blocks per SM (168 registers,
// spilling) took 97 us/step; the row coefficients in shared memory instead of
// registers 79 (the shared-memory pipe).  2301x1101, 4 shots, 147 us/step with
// all pieces: 56% of the DRAM rate, 24% of the issue slots.  Rim and interior
// tasks are cut apart (kSplitAdj in the host code): without their tasks the
// interior alone took 40 us/step of the first case.
constexpr int kAdjSlots = 11;  // mvx', bx; mpx, mvz, bz, kappa, three products; mpz, the fourth product
template <int KIND>
struct AdjDepth {
    static constexpr int value = KIND == kAdjIn ? 4 : 3;
};
constexpr int kAdjRing = 36;    // 4 iterations of 9 pieces, or 3 of 11
constexpr int kAdjWarpBytes = kAdjRing * S2D_STRIP_ROWS * 4;
static_assert(kAdjRing >= 3 * kAdjSlots, "ring of the rim tasks");

struct AdjWin {
    V4 mvx, mg, mk;  // mvx', Lx bx mvx', Kx kappa mPX of one column
};
// Column coefficients of one iteration (kAdjAny): Lx at L; Dax, Kx, Lx at Q;
// Dbx at W; read one iteration ahead.
struct AdjXc {
    float lxl, dbw;
    float4 q;
    __device__ __forceinline__ void read(const float4 *xcoef, int nnx, int L) {
        auto at = [&](int x) { return xcoef + (min(max(x, -S2D_GX), nnx + S2D_GX - 1) + S2D_GX); };
        lxl = __ldg(&at(L)->w);
        q = __ldg(at(L - 1));
        dbw = __ldg(&at(L - 3)->z);
    }
};

struct AdjTask {
    const ShotDev *S;
    V4 *ring;
    int xa, xb, z0, kt, src_q, sdz, slot;
    bool owner, inj, row0;
    V4 one, kx, kz;
    Taps xt, zt;   // literal taps along x and z
    V4 daz, kzr, dbz, lzr;  // row coefficients and taps of the lane's rows (tasks that are not interior)
    Taps hz, gz;
    AdjSource src;
    V4 tbp;        // tbx at Q-1
};

__device__ __forceinline__ void red4(float *p, const V4 &v) {
    red_add4(p, make_float4(lo(v.a), hi(v.a), lo(v.b), hi(v.b)));
}

// Iteration L: w0 holds the oldest column of the windows and receives the
// newest (mvx', mg at L; mk at L-1); w1 .. w3 the three before, w3 the latest.
template <int KIND>
__device__ __forceinline__ void adj_column(AdjTask &k, const AdjXc &xc, const V4 *in, int L, float *mpxo, float *mpzo,
                                           float *mvxo, float *mvzo, float *gk, float *gb, AdjWin &w0,
                                           const AdjWin &w1, const AdjWin &w2, const AdjWin &w3) {
    const ShotDev &S = *k.S;
    const V4 mvx = in[0];
    const V4 mg = ((KIND == kAdjAny ? dup4(xc.lxl) : k.kx) * in[32]) * mvx;
    const int Q = L - 1;
    const bool upd = k.owner && Q >= k.xa && Q < k.xb;  // this lane writes column Q
    const V4 mvz = in[96], kk = in[160];
    const V4 kz = KIND == kAdjIn ? k.kz : k.kzr, lz = KIND == kAdjIn ? k.kz : k.lzr;
    V4 dax = k.one, kx = k.kx, lx = k.kx;
    Taps hx = k.xt, gx = k.xt;
    if (KIND == kAdjAny) {
        dax = dup4(xc.q.x);
        kx = dup4(xc.q.y);
        lx = dup4(xc.q.w);
        float c0, c1;
        dp_coef(Q - 1, S.nnx, c0, c1);
        hx.t0 = dup4(c0);
        dp_coef(Q, S.nnx, c0, c1);
        hx.t1 = dup4(-c0);
        dp_coef(Q - 2, S.nnx, c0, c1);
        hx.t2 = dup4(c1);
        dp_coef(Q + 1, S.nnx, c0, c1);
        hx.t3 = dup4(-c1);
        const int W = L - 3;
        dm_coef(W, S.nnx, c0, c1);
        gx.t0 = dup4(c0);
        dm_coef(W + 1, S.nnx, c0, c1);
        gx.t1 = dup4(-c0);
        dm_coef(W - 1, S.nnx, c0, c1);
        gx.t2 = dup4(c1);
        dm_coef(W + 2, S.nnx, c0, c1);
        gx.t3 = dup4(-c1);
    }
    const Taps &hz = KIND == kAdjIn ? k.zt : k.hz, &gz = KIND == kAdjIn ? k.zt : k.gz;
    // ---- pressure adjoint at Q ----
    V4 q = hzt(hz, (lz * in[128]) * mvz) + taps4(hx.t0, w2.mg, hx.t1, w3.mg, hx.t2, w1.mg, hx.t3, mg);
    if (k.inj && Q >= 0 && Q < S.nnx && Q >= k.xa - 1) k.src.column(S, Q, k.z0, k.slot, q);
    const V4 mPX = in[64] + q;
    V4 mPZ = mPX, daz = k.one;
    bool m0 = true, m1 = true, m2 = true, m3 = true;
    V4 tk = in[192] * mPX;  // one pressure: the first product is Kx a + Kz c
    if (KIND != kAdjIn) {
        daz = k.daz;
        const bool colm = KIND == kAdjRows || xc.q.x == 1.0f;
        m0 = colm && lo(daz.a) == 1.0f;
        m1 = colm && hi(daz.a) == 1.0f;
        m2 = colm && lo(daz.b) == 1.0f;
        m3 = colm && hi(daz.b) == 1.0f;
        const V4 z = in[288] + q;
        mPZ = v4(pk(m0 ? lo(mPX.a) : lo(z.a), m1 ? hi(mPX.a) : hi(z.a)),
                 pk(m2 ? lo(mPX.b) : lo(z.b), m3 ? hi(mPX.b) : hi(z.b)));
        const V4 ts = fma4(kx * in[192], mPX, (kz * in[320]) * mPZ);
        tk = v4(pk(m0 ? lo(tk.a) : lo(ts.a), m1 ? hi(tk.a) : hi(ts.a)),
                pk(m2 ? lo(tk.b) : lo(ts.b), m3 ? hi(tk.b) : hi(ts.b)));
    }
    if (upd) {
        *reinterpret_cast<V4 *>(mpxo) = KIND == kAdjAny ? dax * mPX : mPX;
        if (KIND != kAdjIn) {
            const V4 o = daz * mPZ;
            *reinterpret_cast<V4 *>(mpzo) = v4(pk(m0 ? 0.0f : lo(o.a), m1 ? 0.0f : hi(o.a)),
                                               pk(m2 ? 0.0f : lo(o.b), m3 ? 0.0f : hi(o.b)));
        }
        red4(gk, tk);
        if (Q == k.src_q && k.sdz >= 0 && k.sdz < 4)
            S.srcadj[k.kt] = k.sdz == 0 ? lo(mPX.a) : k.sdz == 1 ? hi(mPX.a) : k.sdz == 2 ? lo(mPX.b) : hi(mPX.b);
    }
    const V4 mk = (kx * kk) * mPX;
    // ---- z-velocity adjoint at Q ----
    const V4 g = gzt(gz, (kz * kk) * mPZ);
    if (upd) *reinterpret_cast<V4 *>(mvzo) = fma4(KIND == kAdjIn ? k.one : k.dbz, mvz, g);
    // ---- buoyancy imaging at Q (xa-1 feeds column xa; 0 outside the grid) ----
    {
        const V4 tbx = (lx * in[224]) * w3.mvx, tbz = (lz * in[256]) * mvz;
        float up = __shfl_up_sync(kFull, hi(tbz.b), 1);
        if (KIND != kAdjIn && !k.row0) up = 0.0f;
        const V4 zs = v4(pk(up, lo(tbz.a)), pk(hi(tbz.a), lo(tbz.b)));
        const V4 half = dup4(0.5f);
        if (upd) red4(gb, half * ((tbx + (KIND != kAdjAny || Q >= 1 ? k.tbp : zero4())) + (tbz + zs)));
        k.tbp = tbx;
    }
    // ---- x-velocity adjoint at W = L - 3 ----
    if (k.owner && L - 3 >= k.xa && L - 3 < k.xb) {
        const V4 o = taps4(gx.t0, w2.mk, gx.t1, w3.mk, gx.t2, w1.mk, gx.t3, mk);
        *reinterpret_cast<V4 *>(mvxo) = fma4(KIND == kAdjAny ? dup4(xc.dbw) : k.one, w1.mvx, o);
    }
    w0.mvx = mvx;
    w0.mg = mg;
    w0.mk = mk;
}

template <int KIND>
__device__ __forceinline__ void adjoint_task(const StepArgs &a, const ShotDev &S, int strip, int xa, int seg_len,
                                             int kt, int lane, V4 *smem) {
    constexpr int D = AdjDepth<KIND>::value, NS = KIND == kAdjIn ? 9 : kAdjSlots;
    const int nnx = S.nnx;
    const ptrdiff_t ld = S.ld;
    const int c = strip * S2D_STRIP_OUT - 4;
    Lane<true> ln;
    lane_setup(ln, S, c, lane, kt);
    AdjTask k;
    k.S = &S;
    k.ring = smem + lane;
    k.xa = xa;
    k.xb = min(nnx, xa + seg_len);
    k.z0 = ln.z0;
    k.kt = kt;
    k.src_q = S.src_x;
    k.sdz = ln.sdz;
    k.owner = ln.owner;
    k.row0 = ln.z0 >= 1;
    k.slot = (kt + 1) / a.dt_factor - 1;
    // receiver adjoint source on recording steps, in strips whose rows hold receivers
    k.inj = !(a.flags & S2D_STEP_NO_RECORD) && S.nrec > 0 && ((kt + 1) % a.dt_factor) == 0 && k.slot < S.real_nt &&
            c + S2D_STRIP_ROWS > S.rec_zlo && c <= S.rec_zhi;
    if (k.inj) k.src.start(S, max(xa - 1, 0), k.slot);
    k.one = dup4(a.one);
    k.kx = dup4(S.kx_in);
    k.kz = dup4(S.kz_in);
    k.xt = Taps{dup4(kA0), dup4(-kA0), dup4(kA1), dup4(-kA1)};
    k.zt = row_taps(k.xt.t0, k.xt.t1, k.xt.t2, k.xt.t3);
    k.tbp = zero4();
    if (KIND != kAdjIn) {
        float r[12][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int z = ln.z0 + i, n = S.nnz;
            const float4 q = __ldg(ln.zc + i);
            r[0][i] = q.x;
            r[1][i] = q.y;
            r[2][i] = q.z;
            r[3][i] = q.w;
            float u;
            dp_coef(z - 1, n, r[4][i], u);
            dp_coef(z, n, r[5][i], u);
            dp_coef(z - 2, n, u, r[6][i]);
            dp_coef(z + 1, n, u, r[7][i]);
            dm_coef(z, n, r[8][i], u);
            dm_coef(z + 1, n, r[9][i], u);
            dm_coef(z - 1, n, u, r[10][i]);
            dm_coef(z + 2, n, u, r[11][i]);
        }
        auto tab = [&](int i, float f) { return v4(pk(f * r[i][0], f * r[i][1]), pk(f * r[i][2], f * r[i][3])); };
        k.daz = tab(0, 1.0f);
        k.kzr = tab(1, 1.0f);
        k.dbz = tab(2, 1.0f);
        k.lzr = tab(3, 1.0f);
        k.hz = row_taps(tab(4, 1.0f), tab(5, -1.0f), tab(6, 1.0f), tab(7, -1.0f));
        k.gz = row_taps(tab(8, 1.0f), tab(9, -1.0f), tab(10, 1.0f), tab(11, -1.0f));
    }
    const int pin = (kt + 1) & 1, pout = kt & 1;
    // a ghost lane reads the column's first ghost rows (zeros) and writes nothing
    const size_t off = (size_t)(ln.zl + S2D_GZ) + (size_t)S2D_GX * ld;
    const ptrdiff_t fs = S.fstride;
    const size_t F = (size_t)(nnx + 2 * S2D_GX) * ld;
    const int L0 = xa - 3, Lend = k.xb + 2;
    const int n4 = (Lend - xa + 4) / 4;  // groups of four iterations from L = xa on (the last may pass Lend)
    const int Llast = KIND == kAdjIn ? xa + 4 * n4 - 1 : Lend;
    // state, materials and products at the next iteration's column Q
    const float *ns = S.st[pin][0] + off + (ptrdiff_t)(L0 - 1) * ld;
    const float *nm = S.kappa + off + (ptrdiff_t)(L0 - 1) * ld;
    const float *np = S.prod + (size_t)(kt - a.prod_kt0) * 4 * F + off + (ptrdiff_t)(L0 - 1) * ld;
    auto issue = [&](int L, int slot) {
        V4 *st = k.ring + slot * (NS * 32);
        // Only what the iteration uses (what it computes from the rest of its
        // slot is not written): the windows' inputs first, the products and mpz
        // of the task's own columns and the one before them.  Of a segment's
        // 6 columns besides its own, three bring 2 pieces and two 6 instead of 9.
        if (L <= Lend) {
            cp_async16(st, ns + ld + 2 * fs, true);
            cp_async16(st + 32, nm + ld + fs, true);
            if (L >= xa) {
                cp_async16(st + 64, ns, true);
                cp_async16(st + 96, ns + 3 * fs, true);
                cp_async16(st + 128, nm + 2 * fs, true);
                cp_async16(st + 160, nm, true);
                if (L >= 1 && L <= k.xb) {
                    cp_async16(st + 192, np, true);
                    cp_async16(st + 224, np + 2 * F, true);
                    cp_async16(st + 256, np + 3 * F, true);
                    if (KIND != kAdjIn) {
                        cp_async16(st + 288, ns + fs, true);
                        cp_async16(st + 320, np + F, true);
                    }
                }
            }
        }
        ns += ld;
        nm += ld;
        np += ld;
    };
#pragma unroll
    for (int i = 0; i < D - 1; ++i) {
        issue(L0 + i, i);
        cp_async_commit();
    }
    auto next = [&](int L, int i) {  // bring iteration L + D - 1, wait for iteration L (in slot i)
        if (L + D - 1 <= Llast) issue(L + D - 1, KIND == kAdjIn ? (i + D - 1) % D : i == 0 ? D - 1 : i - 1);
        cp_async_commit();
        cp_async_wait<D - 1>();
        return k.ring + i * (NS * 32);
    };
    AdjWin wa, wb, wc, wd;
    wa.mvx = wa.mg = wa.mk = zero4();
    wb = wc = wd = wa;
    // iterations xa-3 .. xa-1 fill the windows of mvx' and Lx bx mvx'
    auto fill = [&](AdjWin &w, int i) {
        const V4 *in = next(L0 + i, i);
        const float lx = KIND == kAdjAny ? __ldg(S.xcoef + (L0 + i + S2D_GX)).w : S.kx_in;
        w.mvx = in[0];
        w.mg = (dup4(lx) * in[32]) * w.mvx;
    };
    fill(wb, 0);
    fill(wc, 1);
    fill(wd, 2);
    float *mpxo = S.st[pout][0] + off + (ptrdiff_t)(xa - 1) * ld, *mpzo = mpxo + fs, *mvzo = mpxo + 3 * fs;
    float *mvxo = S.st[pout][0] + off + (ptrdiff_t)(xa - 3) * ld + 2 * fs;
    float *gk = S.grad[0] + off + (ptrdiff_t)(xa - 1) * ld, *gb = S.grad[1] + off + (ptrdiff_t)(xa - 1) * ld;
    AdjXc xc{};
    int L = xa;
    if (KIND == kAdjIn) {
        for (int g = 0; g < n4; ++g) {
#define S2D_ADJ_COLUMN(J, I, A, B, C_, D_)                                                                        \
    adj_column<KIND>(k, xc, next(L + J, I), L + J, mpxo + J * ld, mpzo, mvxo + J * ld, mvzo + J * ld, gk + J * ld, \
                     gb + J * ld, A, B, C_, D_)
            S2D_ADJ_COLUMN(0, 3, wa, wb, wc, wd);
            S2D_ADJ_COLUMN(1, 0, wb, wc, wd, wa);
            S2D_ADJ_COLUMN(2, 1, wc, wd, wa, wb);
            S2D_ADJ_COLUMN(3, 2, wd, wa, wb, wc);
#undef S2D_ADJ_COLUMN
            L += 4;
            mpxo += 4 * ld;
            mvxo += 4 * ld;
            mvzo += 4 * ld;
            gk += 4 * ld;
            gb += 4 * ld;
        }
    } else {
        if (KIND == kAdjAny) xc.read(S.xcoef, nnx, L);
        int slot = 3 % D;
#pragma unroll 1
        for (; L <= Lend; ++L) {
            AdjXc xn{};
            if (KIND == kAdjAny) xn.read(S.xcoef, nnx, L + 1);
            adj_column<KIND>(k, xc, next(L, slot), L, mpxo, mpzo, mvxo, mvzo, gk, gb, wa, wb, wc, wd);
            slot = slot + 1 == D ? 0 : slot + 1;
            const AdjWin t = wa;
            wa = wb;
            wb = wc;
            wc = wd;
            wd = t;
            xc = xn;
            mpxo += ld;
            mpzo += ld;
            mvxo += ld;
            mvzo += ld;
            gk += ld;
            gb += ld;
        }
    }
    cp_async_wait<0>();
}

__global__ void __launch_bounds__(128, 2) adjoint_kernel(const StepArgs *__restrict__ A, int kt_off) {
    extern __shared__ __align__(128) unsigned char smem[];
    V4 *const mem = reinterpret_cast<V4 *>(smem + (size_t)(threadIdx.x >> 5) * kAdjWarpBytes);
    const StepArgs a = *A;
    const int lane = threadIdx.x & 31;
    const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nwarp = (int)((gridDim.x * blockDim.x) >> 5);
    const int kt = a.kt_base - kt_off;
    if (kt < 0 || kt >= a.fd_nt) return;
    // the task's shot record in this warp's shared-memory slot
    __shared__ ShotDev shot_rec[4];
    ShotDev &S = shot_rec[(threadIdx.x >> 5) & 3];
    TaskQueue queue(a.queue, nwarp, lane);
    for (int t = gwarp; t < a.total_tasks; t = queue.take()) {
        queue.draw();
        int strip, xa, seg_len;
        const ShotDev &G = task_of_split(a, t, strip, xa, seg_len);
        if (!task_in_bounds(a, G, strip, xa, seg_len, kt, true, 2)) continue;
        warp_copy_shot(S, G, lane);
        const int c = strip * S2D_STRIP_OUT - 4;
        const int xb = min(S.nnx, xa + seg_len);
        // the z-transposes read the coefficient pairs of rows c-2 .. c+129,
        // the x-gathers those of columns xa-3 .. xb+2
        const bool zf = rows_fast(S, c - kAdjRowMargin, c + S2D_STRIP_ROWS - 1 + kAdjRowMargin);
        const bool xf = xa - kAdjColLo >= S.xfast_lo && xb + kAdjColHi < S.xfast_hi;
        if (zf && xf) adjoint_task<kAdjIn>(a, S, strip, xa, seg_len, kt, lane, mem);
        else if (xf) adjoint_task<kAdjRows>(a, S, strip, xa, seg_len, kt, lane, mem);
        else adjoint_task<kAdjAny>(a, S, strip, xa, seg_len, kt, lane, mem);
    }
    queue.leave();
}

// ---- gradient finalisation ----

__device__ __forceinline__ size_t pad_id(int x, int z, int ld) {
    return (size_t)(x + S2D_GX) * ld + (z + S2D_GZ);
}

// Source term of dJ/dkappa (the amplitude fd_dt w kappa_src / (dx dz) depends
// on kappa at the source cell), added in shot order.
__global__ void add_source_terms(float *const *gk, const int *cells, const double *vals, int nshots) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (int s = 0; s < nshots; ++s) gk[s][cells[s]] = (float)((double)gk[s][cells[s]] + vals[s]);
}

__global__ void sum_shots(float *const *gk, float *const *gb, int nshots, int nnx, int nnz, int ld, float *tk,
                          float *tb) {
    const int z = blockIdx.x * blockDim.x + threadIdx.x, x = blockIdx.y;
    if (z >= nnz || x >= nnx) return;
    const size_t id = pad_id(x, z, ld);
    double a = 0, b = 0;
    for (int s = 0; s < nshots; ++s) {
        a += gk[s][id];
        b += gb[s][id];
    }
    tk[id] = (float)a;
    tb[id] = (float)b;
}

// kappa = vp^2 rho and b = 1/rho (the buoyancy averages are folded into dJ/db
// by the adjoint step).  Rows z < kfix hold kappa at 0 (free surface): their
// dJ/dkappa does not depend on vp or rho.
__global__ void chain_rule(const float *tk, const float *tb, const float *vp, const float *rho, int nx, int nz,
                           int nb, int ld, int kfix, float *gvp, float *grho) {
    const int nnx = nx + 2 * nb, nnz = nz + 2 * nb;
    const int z = blockIdx.x * blockDim.x + threadIdx.x, x = blockIdx.y;
    if (z >= nnz || x >= nnx) return;
    const size_t id = pad_id(x, z, ld);
    const double gb = tb[id];
    const double gk = z < kfix ? 0.0 : (double)tk[id];
    const int mx = min(max(x - nb, 0), nx - 1), mz = min(max(z - nb, 0), nz - 1);
    const double v = vp[(size_t)mx * nz + mz], r = rho[(size_t)mx * nz + mz];
    gvp[id] = (float)(2.0 * v * r * gk);
    grho[id] = (float)(v * v * gk + (r > 0 ? -gb / (r * r) : 0.0));
}

// Fold the sponge onto the model cells it replicates (transpose of
// cpumodelling.cpp:39-60).
__global__ void fold_sponge(const float *gvp, const float *grho, int nx, int nz, int nb, int ld, float *out_vp,
                            float *out_rho) {
    const int iz = blockIdx.x * blockDim.x + threadIdx.x, ix = blockIdx.y;
    if (iz >= nz || ix >= nx) return;
    const int nnx = nx + 2 * nb, nnz = nz + 2 * nb;
    const int x0 = ix == 0 ? 0 : ix + nb, x1 = ix == nx - 1 ? nnx - 1 : ix + nb;
    const int z0 = iz == 0 ? 0 : iz + nb, z1 = iz == nz - 1 ? nnz - 1 : iz + nb;
    double a = 0, b = 0;
    for (int x = x0; x <= x1; ++x)
        for (int z = z0; z <= z1; ++z) {
            const size_t id = pad_id(x, z, ld);
            a += gvp[id];
            b += grho[id];
        }
    out_vp[(size_t)ix * nz + iz] = (float)a;
    out_rho[(size_t)ix * nz + iz] = (float)b;
}

__global__ void residual_kernel(const float *seis, const float *obs, float *res, size_t n, double *sumsq) {
    __shared__ double part[256];
#ifdef S2D_DEVICE_CHECKS
    if (blockDim.x != 256) return;
#endif
    double acc = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float r = seis[i] - obs[i];
        res[i] = r;
        acc += (double)r * r;
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(sumsq, part[0]);
}

// ---------------------------------------------------------------- 8th order
//
// Adjoint step of the 8th-order scheme: the algebra of the header above with
// the 8-tap operators, in two cell-parallel passes (one thread per padded
// cell, blockIdx.z = shot; the gathers read their neighbours from memory):
//   pass 1: q = Hx^T(Lx bx mvx') + Hz^T(Lz bz mvz') (+ the adjoint source),
//           mPX, mPZ, the new mpx, mpz, dJ/dkappa, and Kx kappa mPX,
//           Kz kappa mPZ into the shot's two scratch fields;
//   pass 2: mvx = Dbx mvx' + Gx^T(Kx kappa mPX), mvz likewise, and dJ/db.
// Gather forms of the transposes, with c(j) the coefficients of forward row j
// (dm8 / dp8, zero outside the grid):
//   (G^T m)[i] = sum_k c_k(i-k) m[i-k] - c_k(i+1+k) m[i+1+k]
//   (H^T m)[i] = sum_k c_k(i-1-k) m[i-1-k] - c_k(i+k) m[i+k]
// (for the 4th-order pairs these are the gathers of adjoint_task).  The taps
// reach 4 cells, inside the 8 ghost columns and rows, whose scratch stays 0.

__device__ __forceinline__ size_t cell8(int x, int z, int ld) {
    return (size_t)(x + S2D_GX) * (size_t)ld + (size_t)(z + S2D_GZ);
}

__global__ void __launch_bounds__(128) adjoint8_pressure(const StepArgs *__restrict__ A, int kt_off) {
    const StepArgs a = *A;
    const int kt = a.kt_base - kt_off;
    if (kt < 0 || kt >= a.fd_nt) return;
    const ShotDev &S = a.shots[blockIdx.z];
    const int z = blockIdx.x * blockDim.x + threadIdx.x, x = blockIdx.y;
    if (z >= S.nnz || x >= S.nnx) return;
    const int ld = S.ld, nnx = S.nnx, nnz = S.nnz;
    const int pin = (kt + 1) & 1, pout = kt & 1;
    const size_t id = cell8(x, z, ld);
    const size_t F = (size_t)(nnx + 2 * S2D_GX) * (size_t)ld;
    const float *__restrict__ mvx = S.st[pin][2];
    const float *__restrict__ mvz = S.st[pin][3];
    float q = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j0 = x - 1 - k, j1 = x + k;
        const size_t i0 = cell8(j0, z, ld), i1 = cell8(j1, z, ld);
        q += comp(dp8(j0, nnx), k) * ((__ldg(S.xcoef + (j0 + S2D_GX)).w * __ldg(S.bx + i0)) * __ldg(mvx + i0));
        q -= comp(dp8(j1, nnx), k) * ((__ldg(S.xcoef + (j1 + S2D_GX)).w * __ldg(S.bx + i1)) * __ldg(mvx + i1));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j0 = z - 1 - k, j1 = z + k;
        const size_t i0 = cell8(x, j0, ld), i1 = cell8(x, j1, ld);
        q += comp(dp8(j0, nnz), k) * ((__ldg(S.zcoef + (j0 + S2D_GZ)).w * __ldg(S.bz + i0)) * __ldg(mvz + i0));
        q -= comp(dp8(j1, nnz), k) * ((__ldg(S.zcoef + (j1 + S2D_GZ)).w * __ldg(S.bz + i1)) * __ldg(mvz + i1));
    }
    // transpose of the receiver sampling (cpumodelling.cpp:356-360)
    const int slot = (kt + 1) / a.dt_factor - 1;
    if (!(a.flags & S2D_STEP_NO_RECORD) && ((kt + 1) % a.dt_factor) == 0 && slot < S.real_nt) {
        const int j1 = __ldg(S.rec_ptr + x + 1);
        for (int j = __ldg(S.rec_ptr + x); j < j1; ++j)
            if (__ldg(S.rec_z + j) == z) q += __ldg(S.seis + (size_t)__ldg(S.rec_id + j) * S.real_nt + slot);
    }
    const float4 xq = __ldg(S.xcoef + (x + S2D_GX));  // Dax, Kx, Dbx, Lx
    const float4 r = __ldg(S.zcoef + (z + S2D_GZ));   // Daz, Kz, Dbz, Lz
    const bool merged = xq.x == 1.0f && r.x == 1.0f;   // the forward carried p alone here
    const float mPX = S.st[pin][0][id] + q;
    const float mPZ = merged ? mPX : S.st[pin][1][id] + q;
    S.st[pout][0][id] = xq.x * mPX;
    S.st[pout][1][id] = merged ? 0.0f : r.x * mPZ;
    const float *__restrict__ pr = S.prod + (size_t)(kt - a.prod_kt0) * 4 * F;
    const float pa = __ldg(pr + id);
    atomicAdd(S.grad[0] + id, merged ? pa * mPX : (xq.y * pa) * mPX + (r.y * __ldg(pr + F + id)) * mPZ);
    const float k = __ldg(S.kappa + id);
    S.scr[id] = (xq.y * k) * mPX;
    S.scr[F + id] = (r.y * k) * mPZ;
    if (x == S.src_x && z == S.src_z) S.srcadj[kt] = mPX;
}

__global__ void __launch_bounds__(128) adjoint8_velocity(const StepArgs *__restrict__ A, int kt_off) {
    const StepArgs a = *A;
    const int kt = a.kt_base - kt_off;
    if (kt < 0 || kt >= a.fd_nt) return;
    const ShotDev &S = a.shots[blockIdx.z];
    const int z = blockIdx.x * blockDim.x + threadIdx.x, x = blockIdx.y;
    if (z >= S.nnz || x >= S.nnx) return;
    const int ld = S.ld, nnx = S.nnx, nnz = S.nnz;
    const int pin = (kt + 1) & 1, pout = kt & 1;
    const size_t id = cell8(x, z, ld);
    const size_t F = (size_t)(nnx + 2 * S2D_GX) * (size_t)ld;
    const float *__restrict__ sa = S.scr;
    const float *__restrict__ sb = S.scr + F;
    float gx = 0.0f, gz = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        gx += comp(dm8(x - k, nnx), k) * __ldg(sa + cell8(x - k, z, ld));
        gx -= comp(dm8(x + 1 + k, nnx), k) * __ldg(sa + cell8(x + 1 + k, z, ld));
        gz += comp(dm8(z - k, nnz), k) * __ldg(sb + cell8(x, z - k, ld));
        gz -= comp(dm8(z + 1 + k, nnz), k) * __ldg(sb + cell8(x, z + 1 + k, ld));
    }
    const float4 xq = __ldg(S.xcoef + (x + S2D_GX));
    const float4 r = __ldg(S.zcoef + (z + S2D_GZ));
    const float *__restrict__ mvx = S.st[pin][2];
    const float *__restrict__ mvz = S.st[pin][3];
    const float vx_in = __ldg(mvx + id), vz_in = __ldg(mvz + id);
    S.st[pout][2][id] = xq.z * vx_in + gx;
    S.st[pout][3][id] = r.z * vz_in + gz;
    // buoyancy imaging: tbx = Lx g mvx', tbz = Lz h mvz' through the averages
    // bx = (b[x] + b[x+1]) / 2, bz = (b[z] + b[z+1]) / 2
    const float *__restrict__ pr = S.prod + (size_t)(kt - a.prod_kt0) * 4 * F;
    const float tbx = (xq.w * __ldg(pr + 2 * F + id)) * vx_in;
    const float tbz = (r.w * __ldg(pr + 3 * F + id)) * vz_in;
    const float tbxm = x >= 1 ? (__ldg(S.xcoef + (x - 1 + S2D_GX)).w * __ldg(pr + 2 * F + id - ld)) * __ldg(mvx + id - ld)
                              : 0.0f;
    const float tbzm = z >= 1 ? (__ldg(S.zcoef + (z - 1 + S2D_GZ)).w * __ldg(pr + 3 * F + id - 1)) * __ldg(mvz + id - 1)
                              : 0.0f;
    atomicAdd(S.grad[1] + id, 0.5f * ((tbx + tbxm) + (tbz + tbzm)));
}

// ---------------------------------------------------------------- 8th order, streaming
//
// The adjoint step of the 8th-order scheme as one streaming pass (the
// algebra of adjoint8_pressure / adjoint8_velocity, the same products in the
// same order per cell): a warp owns a 128-row strip read from 112k - 8 and
// writes its middle 112 rows (lanes 2..29, the 8th-order forward's layout),
// streaming along x.  Iteration L brings mvx' and bx at L; at Q = L-3 it forms
// the pressure adjoint (x-gather of Lx bx mvx' over Q-4 .. Q+3, z-gather of Lz
// bz mvz' over the rows z-4 .. z+3 by shuffles from the neighbouring lanes),
// the z-velocity adjoint (z-gather of Kz kappa mPZ) and the imaging terms; at W
// = L-7 the x-velocity adjoint (x-gather of Kx kappa mPX over W-3 .. W+4).
//
// Copies, windows, tasks and queue as the 4th-order step's: the inputs come D -
// 1 iterations ahead by per-lane asynchronous copies, the windows (mvx', Lx bx
// mvx', Kx kappa mPX of 8 columns each) are registers, named by position in a
// loop unrolled by four and moved once per four columns (interior tasks), or
// moved every column (the others).  The 20 row coefficients of tasks that are
// not interior wait in shared memory.
//
// What bounds it: as the 4th-order step, the latency of one column's chain with
// two warps on each scheduler (255 registers, no spill).  us per step, before
// (windows in shared memory, loads where they were used, every strip one
// length) and after: 1201x401, 4 shots 103 -> 48, 8 shots 179 -> 89; 601x301, 4
// shots 51 -> 27; 2301x1101, 4 shots 340 -> 142 (2.8 TB/s of state, materials
// and products).

// Kinds of tasks: interior; interior columns and taps, any damping; interior
// columns, any row; anything.
enum { kAdj8In = 0, kAdj8Rows = 1, kAdj8Edge = 2, kAdj8Any = 3 };
template <int KIND>
struct Adj8Depth {
    static constexpr int value = KIND == kAdj8In ? 4 : 3;
};
constexpr int kAdj8Tab = 20;  // Daz, Kz, Dbz, Lz; taps of H^T and G^T along z, 4 + 4 each
constexpr int kAdj8Ring = 3 * kAdjSlots + kAdj8Tab;
constexpr int kAdj8WarpBytes = kAdj8Ring * S2D_STRIP_ROWS * 4;
static_assert(kAdj8Ring >= 4 * 9, "ring of the interior tasks");

// acc + sum_k p_k m[i-k] + n_k m[i+1+k] of packed rows, each product fused in
// the order k = 0 (p, n), 1 (p, n) ...; without acc the first one is rounded.
template <bool ACC, class P, class N>
__device__ __forceinline__ f2 gather8(f2 acc, P p, N n, const f2 *a, const f2 *b) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        acc = !ACC && k == 0 ? mul2(p(k), a[k]) : fma2(p(k), a[k], acc);
        acc = fma2(n(k), b[k], acc);
    }
    return acc;
}

// Column coefficients of one iteration (kAdj8Any): Lx at L; Dax, Kx, Lx at Q;
// Dbx at W; read one iteration ahead.
struct Adj8Xc {
    float lxl, dbw;
    float4 q;
    __device__ __forceinline__ void read(const float4 *xcoef, int nnx, int L) {
        auto at = [&](int x) { return xcoef + (min(max(x, -S2D_GX), nnx + S2D_GX - 1) + S2D_GX); };
        lxl = __ldg(&at(L)->w);
        q = __ldg(at(L - 3));
        dbw = __ldg(&at(L - 7)->z);
    }
};

struct Adj8Task {
    const ShotDev *S;
    V4 *ring, *tab;
    int xa, xb, z0, kt, src_q, sdz, slot;
    bool owner, inj, row0;
    V4 one, kx, kz;
    f2 cp[4], cn[4];  // literal taps and their negatives
    AdjSource src;
    V4 tbp;           // tbx at Q-1
};

// Iteration L: w[0..7] mvx' and g[0..7] Lx bx mvx' at L-7 .. L (the last set
// here), m[0..7] Kx kappa mPX at L-10 .. L-3 (the last set here).
template <int KIND>
__device__ __forceinline__ void adj8_column(Adj8Task &k, const Adj8Xc &xc, const V4 *in, int L, float *po, float *vo,
                                            float *gk, float *gb, ptrdiff_t fs, V4 *w, V4 *g, V4 *m) {
    const ShotDev &S = *k.S;
    const int Q = L - 3, W = L - 7, nnx = S.nnx;
    w[7] = in[0];
    g[7] = ((KIND == kAdj8Any ? dup4(xc.lxl) : k.kx) * in[32]) * w[7];
    const bool upd = k.owner && Q >= k.xa && Q < k.xb;  // this lane writes column Q
    const V4 mvz = in[96], kk = in[160];
    const V4 kz = KIND == kAdj8In ? k.kz : k.tab[32], lz = KIND == kAdj8In ? k.kz : k.tab[96];
    const V4 kx = KIND == kAdj8Any ? dup4(xc.q.y) : k.kx, lx = KIND == kAdj8Any ? dup4(xc.q.w) : k.kx;
    f2 hp[4], hn[4], vp[4], vn[4];  // taps of the x-gathers at Q and W
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        hp[i] = vp[i] = k.cp[i];
        hn[i] = vn[i] = k.cn[i];
    }
    if (KIND == kAdj8Any && (Q < 11 || Q > nnx - 8)) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            hp[i] = dup(comp(dp8(Q - 1 - i, nnx), i));
            hn[i] = dup(-comp(dp8(Q + i, nnx), i));
            vp[i] = dup(comp(dm8(W - i, nnx), i));
            vn[i] = dup(-comp(dm8(W + 1 + i, nnx), i));
        }
    }
    // ---- pressure adjoint at Q ----
    V4 q;
    {
        const f2 a0[4] = {g[3].a, g[2].a, g[1].a, g[0].a}, b0[4] = {g[4].a, g[5].a, g[6].a, g[7].a};
        const f2 a1[4] = {g[3].b, g[2].b, g[1].b, g[0].b}, b1[4] = {g[4].b, g[5].b, g[6].b, g[7].b};
        auto p = [&](int i) { return hp[i]; };
        auto n = [&](int i) { return hn[i]; };
        q = v4(gather8<false>(0ull, p, n, a0, b0), gather8<false>(0ull, p, n, a1, b1));
    }
    {
        // rows z0-4 .. z0+6 of Lz bz mvz'
        const V4 h = (lz * in[128]) * mvz;
        const float x = lo(h.a), y = hi(h.a), z = lo(h.b), v = hi(h.b);
        const float u0 = __shfl_up_sync(kFull, x, 1), u1 = __shfl_up_sync(kFull, y, 1);
        const float u2 = __shfl_up_sync(kFull, z, 1), u3 = __shfl_up_sync(kFull, v, 1);
        const float d0 = __shfl_down_sync(kFull, x, 1), d1 = __shfl_down_sync(kFull, y, 1);
        const float d2 = __shfl_down_sync(kFull, z, 1);
        const f2 u3x = pk(u3, x), yz = pk(y, z), vd0 = pk(v, d0), u23 = pk(u2, u3);
        const f2 a0[4] = {u3x, u23, pk(u1, u2), pk(u0, u1)}, b0[4] = {h.a, yz, h.b, vd0};
        const f2 a1[4] = {yz, h.a, u3x, u23}, b1[4] = {h.b, vd0, pk(d0, d1), pk(d1, d2)};
        constexpr bool TAB = KIND >= kAdj8Edge;
        q.a = gather8<true>(q.a, [&](int i) { return TAB ? k.tab[(4 + i) * 32].a : k.cp[i]; },
                            [&](int i) { return TAB ? k.tab[(8 + i) * 32].a : k.cn[i]; }, a0, b0);
        q.b = gather8<true>(q.b, [&](int i) { return TAB ? k.tab[(4 + i) * 32].b : k.cp[i]; },
                            [&](int i) { return TAB ? k.tab[(8 + i) * 32].b : k.cn[i]; }, a1, b1);
    }
    if (k.inj && Q >= 0 && Q < nnx) k.src.column(S, Q, k.z0, k.slot, q);
    const V4 mPX = in[64] + q;
    V4 mPZ = mPX, daz = k.one;
    const V4 dax = KIND == kAdj8Any ? dup4(xc.q.x) : k.one;
    bool m0 = true, m1 = true, m2 = true, m3 = true;
    V4 tk = in[192] * mPX;  // one pressure: the first product is Kx a + Kz c
    if (KIND != kAdj8In) {
        daz = k.tab[0];
        const bool colm = KIND != kAdj8Any || xc.q.x == 1.0f;
        m0 = colm && lo(daz.a) == 1.0f;
        m1 = colm && hi(daz.a) == 1.0f;
        m2 = colm && lo(daz.b) == 1.0f;
        m3 = colm && hi(daz.b) == 1.0f;
        const V4 z = in[288] + q;
        mPZ = v4(pk(m0 ? lo(mPX.a) : lo(z.a), m1 ? hi(mPX.a) : hi(z.a)),
                 pk(m2 ? lo(mPX.b) : lo(z.b), m3 ? hi(mPX.b) : hi(z.b)));
        const V4 ts = fma4(kx * in[192], mPX, (kz * in[320]) * mPZ);
        tk = v4(pk(m0 ? lo(tk.a) : lo(ts.a), m1 ? hi(tk.a) : hi(ts.a)),
                pk(m2 ? lo(tk.b) : lo(ts.b), m3 ? hi(tk.b) : hi(ts.b)));
    }
    if (upd) {
        *reinterpret_cast<V4 *>(po) = KIND == kAdj8Any ? dax * mPX : mPX;
        if (KIND != kAdj8In) {
            const V4 o = daz * mPZ;
            *reinterpret_cast<V4 *>(po + fs) = v4(pk(m0 ? 0.0f : lo(o.a), m1 ? 0.0f : hi(o.a)),
                                                  pk(m2 ? 0.0f : lo(o.b), m3 ? 0.0f : hi(o.b)));
        }
        red4(gk, tk);
        if (Q == k.src_q && k.sdz >= 0 && k.sdz < 4)
            S.srcadj[k.kt] = k.sdz == 0 ? lo(mPX.a) : k.sdz == 1 ? hi(mPX.a) : k.sdz == 2 ? lo(mPX.b) : hi(mPX.b);
    }
    m[7] = (kx * kk) * mPX;
    // ---- z-velocity adjoint at Q: rows z0-3 .. z0+7 of Kz kappa mPZ ----
    {
        const V4 s = (kz * kk) * mPZ;
        const float x = lo(s.a), y = hi(s.a), z = lo(s.b), v = hi(s.b);
        const float u1 = __shfl_up_sync(kFull, y, 1), u2 = __shfl_up_sync(kFull, z, 1);
        const float u3 = __shfl_up_sync(kFull, v, 1);
        const float d0 = __shfl_down_sync(kFull, x, 1), d1 = __shfl_down_sync(kFull, y, 1);
        const float d2 = __shfl_down_sync(kFull, z, 1), d3 = __shfl_down_sync(kFull, v, 1);
        const f2 u3x = pk(u3, x), yz = pk(y, z), vd0 = pk(v, d0), d12 = pk(d1, d2);
        const f2 a0[4] = {s.a, u3x, pk(u2, u3), pk(u1, u2)}, b0[4] = {yz, s.b, vd0, pk(d0, d1)};
        const f2 a1[4] = {s.b, yz, s.a, u3x}, b1[4] = {vd0, pk(d0, d1), d12, pk(d2, d3)};
        constexpr bool TAB = KIND >= kAdj8Edge;
        const f2 ga = gather8<false>(0ull, [&](int i) { return TAB ? k.tab[(12 + i) * 32].a : k.cp[i]; },
                                     [&](int i) { return TAB ? k.tab[(16 + i) * 32].a : k.cn[i]; }, a0, b0);
        const f2 gc = gather8<false>(0ull, [&](int i) { return TAB ? k.tab[(12 + i) * 32].b : k.cp[i]; },
                                     [&](int i) { return TAB ? k.tab[(16 + i) * 32].b : k.cn[i]; }, a1, b1);
        if (upd) *reinterpret_cast<V4 *>(po + 3 * fs) = fma4(KIND == kAdj8In ? k.one : k.tab[64], mvz, v4(ga, gc));
    }
    // ---- buoyancy imaging at Q (xa-1 feeds column xa; 0 outside the grid) ----
    {
        const V4 tbx = (lx * in[224]) * w[4], tbz = (lz * in[256]) * mvz;
        float up = __shfl_up_sync(kFull, hi(tbz.b), 1);
        if (KIND != kAdj8In && !k.row0) up = 0.0f;
        const V4 zs = v4(pk(up, lo(tbz.a)), pk(hi(tbz.a), lo(tbz.b)));
        if (upd) red4(gb, dup4(0.5f) * ((tbx + (KIND != kAdj8Any || Q >= 1 ? k.tbp : zero4())) + (tbz + zs)));
        k.tbp = tbx;
    }
    // ---- x-velocity adjoint at W ----
    if (k.owner && W >= k.xa && W < k.xb) {
        const f2 a0[4] = {m[3].a, m[2].a, m[1].a, m[0].a}, b0[4] = {m[4].a, m[5].a, m[6].a, m[7].a};
        const f2 a1[4] = {m[3].b, m[2].b, m[1].b, m[0].b}, b1[4] = {m[4].b, m[5].b, m[6].b, m[7].b};
        auto p = [&](int i) { return vp[i]; };
        auto n = [&](int i) { return vn[i]; };
        const V4 o = v4(gather8<false>(0ull, p, n, a0, b0), gather8<false>(0ull, p, n, a1, b1));
        *reinterpret_cast<V4 *>(vo) = fma4(KIND == kAdj8Any ? dup4(xc.dbw) : k.one, w[0], o);
    }
}

template <int KIND>
__device__ __forceinline__ void adjoint8s_task(const StepArgs &a, const ShotDev &S, int strip, int xa, int seg_len,
                                               int kt, int lane, V4 *smem) {
    constexpr int D = Adj8Depth<KIND>::value, NS = KIND == kAdj8In ? 9 : kAdjSlots, U = KIND == kAdj8In ? 4 : 1;
    const int nnx = S.nnx;
    const ptrdiff_t ld = S.ld;
    const int c = strip * S2D_TS_OUT - 8;
    Lane<true> ln;
    lane_setup(ln, S, c, lane, kt);
    Adj8Task k;
    k.S = &S;
    k.ring = smem + lane;
    k.tab = k.ring + 3 * kAdjSlots * 32;
    k.xa = xa;
    k.xb = min(nnx, xa + seg_len);
    k.z0 = ln.z0;
    k.kt = kt;
    k.src_q = S.src_x;
    k.sdz = ln.sdz;
    k.owner = lane >= 2 && lane <= 29 && ln.z0 >= 0 && ln.z0 < S.nnz;
    k.row0 = ln.z0 >= 1;
    k.slot = (kt + 1) / a.dt_factor - 1;
    // receiver adjoint source on recording steps, in strips whose rows hold receivers
    k.inj = !(a.flags & S2D_STEP_NO_RECORD) && S.nrec > 0 && ((kt + 1) % a.dt_factor) == 0 && k.slot < S.real_nt &&
            c + S2D_STRIP_ROWS > S.rec_zlo && c <= S.rec_zhi;
    if (k.inj) k.src.start(S, max(xa - 3, 0), k.slot);
    k.one = dup4(a.one);
    k.kx = dup4(S.kx_in);
    k.kz = dup4(S.kz_in);
    const float4 lit = make_float4(kC81, kC82, kC83, kC84);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        k.cp[i] = dup(comp(lit, i));
        k.cn[i] = dup(-comp(lit, i));
    }
    k.tbp = zero4();
    if (KIND != kAdj8In) {
        float r[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 f = __ldg(ln.zc + i);
            r[0][i] = f.x, r[1][i] = f.y, r[2][i] = f.z, r[3][i] = f.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) k.tab[i * 32] = v4(pk(r[i][0], r[i][1]), pk(r[i][2], r[i][3]));
    }
    if (KIND >= kAdj8Edge) {
        const int n = S.nnz;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float t[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int z = ln.z0 + i;
                t[0][i] = comp(dp8(z - 1 - j, n), j);
                t[1][i] = -comp(dp8(z + j, n), j);
                t[2][i] = comp(dm8(z - j, n), j);
                t[3][i] = -comp(dm8(z + 1 + j, n), j);
            }
#pragma unroll
            for (int f = 0; f < 4; ++f)
                k.tab[(4 + 4 * f + j) * 32] = v4(pk(t[f][0], t[f][1]), pk(t[f][2], t[f][3]));
        }
    }
    const int pin = (kt + 1) & 1, pout = kt & 1;
    // a ghost lane reads the column's first ghost rows (zeros) and writes nothing
    const size_t off = (size_t)(ln.zl + S2D_GZ) + (size_t)S2D_GX * ld;
    const ptrdiff_t fs = S.fstride;
    const size_t F = (size_t)(nnx + 2 * S2D_GX) * ld;
    const int L0 = xa - 7, Lend = k.xb + 6;
    const int n4 = (Lend - xa + U) / U;  // groups of U iterations from L = xa on (the last may pass Lend)
    const int Llast = xa + U * n4 - 1;
    // state, materials and products at the next iteration's column Q
    const float *ns = S.st[pin][0] + off + (ptrdiff_t)(L0 - 3) * ld;
    const float *nm = S.kappa + off + (ptrdiff_t)(L0 - 3) * ld;
    const float *np = S.prod + (size_t)(kt - a.prod_kt0) * 4 * F + off + (ptrdiff_t)(L0 - 3) * ld;
    const ptrdiff_t ovx = 3 * ld + 2 * fs, obx = 3 * ld + fs;
    auto issue = [&](int L, int slot) {
        V4 *st = k.ring + slot * (NS * 32);
        cp_async16(st, ns + ovx, true);
        cp_async16(st + 32, nm + obx, true);
        if (L >= xa) {
            cp_async16(st + 64, ns, true);
            cp_async16(st + 96, ns + 3 * fs, true);
            cp_async16(st + 128, nm + 2 * fs, true);
            cp_async16(st + 160, nm, true);
            if (KIND != kAdj8In) cp_async16(st + 288, ns + fs, true);
            if (L - 3 >= max(xa - 1, 0) && L - 3 < k.xb) {  // the columns whose imaging terms are formed
                cp_async16(st + 192, np, true);
                cp_async16(st + 224, np + 2 * F, true);
                cp_async16(st + 256, np + 3 * F, true);
                if (KIND != kAdj8In) cp_async16(st + 320, np + F, true);
            }
        }
        ns += ld;
        nm += ld;
        np += ld;
    };
#pragma unroll
    for (int i = 0; i < D - 1; ++i) {
        issue(L0 + i, i);
        cp_async_commit();
    }
    auto next = [&](int L, int sl) {  // bring iteration L + D - 1, wait for iteration L (in slot sl)
        if (L + D - 1 <= Llast) issue(L + D - 1, KIND == kAdj8In ? (sl + D - 1) % D : sl == 0 ? D - 1 : sl - 1);
        cp_async_commit();
        cp_async_wait<D - 1>();
        return k.ring + sl * (NS * 32);
    };
    V4 w[7 + U], g[7 + U], m[7 + U];
    // iterations xa-7 .. xa-1 fill the windows of mvx' and Lx bx mvx'
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        const V4 *in = next(L0 + i, i % D);
        const float lx = KIND == kAdj8Any ? __ldg(S.xcoef + (L0 + i + S2D_GX)).w : S.kx_in;
        w[i] = in[0];
        g[i] = (dup4(lx) * in[32]) * w[i];
        m[i] = zero4();
    }
    float *po = S.st[pout][0] + off + (ptrdiff_t)(xa - 3) * ld;
    float *vo = S.st[pout][0] + off + (ptrdiff_t)(xa - 7) * ld + 2 * fs;
    float *gk = S.grad[0] + off + (ptrdiff_t)(xa - 3) * ld, *gb = S.grad[1] + off + (ptrdiff_t)(xa - 3) * ld;
    Adj8Xc xc{};
    if (KIND == kAdj8Any) xc.read(S.xcoef, nnx, xa);
    int L = xa, sl = 7 % D;
#pragma unroll 1
    for (int n = 0; n < n4; ++n) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            Adj8Xc xn{};
            if (KIND == kAdj8Any) xn.read(S.xcoef, nnx, L + 1);
            adj8_column<KIND>(k, xc, next(L, U == 4 ? (7 + j) % D : sl), L, po, vo, gk, gb, fs, w + j, g + j, m + j);
            xc = xn;
            ++L;
            if (U == 1) sl = sl + 1 == D ? 0 : sl + 1;
            po += ld;
            vo += ld;
            gk += ld;
            gb += ld;
        }
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            w[i] = w[i + U];
            g[i] = g[i + U];
            m[i] = m[i + U];
        }
    }
    cp_async_wait<0>();
}

// Debug self-check (S2D_DEVICE_CHECKS) of the task's reach.
__device__ __forceinline__ bool adj8_in_bounds(const StepArgs &a, const ShotDev &S, int strip, int xa, int seg_len,
                                               int kt) {
#ifdef S2D_DEVICE_CHECKS
    const long ld = S.ld;
    const int xb = min(S.nnx, xa + seg_len);
    const long c = (long)strip * S2D_TS_OUT - 8;
    const size_t F = (size_t)(S.nnx + 2 * S2D_GX) * ld;
    if (xa - 7 < -S2D_GX || xb + 6 >= S.nnx + S2D_GX || c + S2D_GZ < 0 || c + 127 + S2D_GZ >= ld || F > S.nfield ||
        kt < a.prod_kt0 || (size_t)(kt - a.prod_kt0 + 1) * 4 * F > S.nprod) {
        if (a.err) atomicCAS(a.err, 0, (4 << 8) | 1);
        return false;
    }
#endif
    return true;
}

__global__ void __launch_bounds__(128, 2) adjoint8s_kernel(const StepArgs *__restrict__ A, int kt_off) {
    extern __shared__ __align__(128) unsigned char smem[];
    V4 *const mem = reinterpret_cast<V4 *>(smem + (size_t)(threadIdx.x >> 5) * kAdj8WarpBytes);
    const StepArgs a = *A;
    const int lane = threadIdx.x & 31;
    const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nwarp = (int)((gridDim.x * blockDim.x) >> 5);
    const int kt = a.kt_base - kt_off;
    if (kt < 0 || kt >= a.fd_nt) return;
    __shared__ ShotDev shot_rec[4];  // the task's shot record, one slot per warp
    ShotDev &S = shot_rec[(threadIdx.x >> 5) & 3];
    TaskQueue queue(a.queue, nwarp, lane);
    for (int t = gwarp; t < a.total_tasks; t = queue.take()) {
        queue.draw();
        int strip, xa, seg_len;
        const ShotDev &G = task_of_split(a, t, strip, xa, seg_len);
        if (!adj8_in_bounds(a, G, strip, xa, seg_len, kt)) continue;
        warp_copy_shot(S, G, lane);
        const int c = strip * S2D_TS_OUT - 8;
        const int xb = min(S.nnx, xa + seg_len);
        // Lanes 1..30 form mPZ from rows c .. c+127 of Lz bz mvz' with the taps
        // of forward D+ rows c .. c+126, lanes 2..29 mvz with those of D- rows
        // c+5 .. c+123.
        const bool taps = c >= 4 && c + S2D_STRIP_ROWS - 1 <= S.nnz - 5;
        const bool zf = taps && rows_fast(S, c, c + S2D_STRIP_ROWS - 1);
        // columns xa-7 .. xb+6 take part
        const bool xf = xa - kAdj8ColLo >= max(S.xfast_lo, 4) && xb + kAdj8ColHi < min(S.xfast_hi, S.nnx - 4);
        if (zf && xf) adjoint8s_task<kAdj8In>(a, S, strip, xa, seg_len, kt, lane, mem);
        else if (taps && xf) adjoint8s_task<kAdj8Rows>(a, S, strip, xa, seg_len, kt, lane, mem);
        else if (xf) adjoint8s_task<kAdj8Edge>(a, S, strip, xa, seg_len, kt, lane, mem);
        else adjoint8s_task<kAdj8Any>(a, S, strip, xa, seg_len, kt, lane, mem);
    }
    queue.leave();
}

}  // namespace

int launch_adjoint8s(const StepArgs *args_dev, int kt_off, int grid, void *stream) {
    adjoint8s_kernel<<<grid, 128, 4 * kAdj8WarpBytes, (cudaStream_t)stream>>>(args_dev, kt_off);
    return (int)cudaGetLastError();
}

// Also raises the kernel's dynamic shared-memory limit; called before the
// launches.
int adjoint8s_occupancy(int *blocks_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(adjoint8s_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         4 * kAdj8WarpBytes);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, adjoint8s_kernel, 128,
                                                             4 * kAdj8WarpBytes);
}

int launch_adjoint8(const StepArgs *args_dev, int kt_off, int nnx, int nnz, int nshots, void *stream) {
    const dim3 blk(128), grd((nnz + 127) / 128, nnx, nshots);
    adjoint8_pressure<<<grd, blk, 0, (cudaStream_t)stream>>>(args_dev, kt_off);
    adjoint8_velocity<<<grd, blk, 0, (cudaStream_t)stream>>>(args_dev, kt_off);
    return (int)cudaGetLastError();
}

int launch_adjoint(const StepArgs *args_dev, int kt_off, int grid, void *stream) {
    adjoint_kernel<<<grid, 128, 4 * kAdjWarpBytes, (cudaStream_t)stream>>>(args_dev, kt_off);
    return (int)cudaGetLastError();
}

// Also raises the kernel's dynamic shared-memory limit; called before the
// adjoint's launches.
int adjoint_kernel_occupancy(int *blocks_per_sm) {
    cudaError_t e = cudaFuncSetAttribute(adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kAdjWarpBytes);
    if (e != cudaSuccess) return (int)e;
    return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, adjoint_kernel, 128, 4 * kAdjWarpBytes);
}

int launch_gradient_finalize(float *const *gk, float *const *gb, int nshots, int nacc, const int *src_cells,
                             const double *src_vals, const float *vp, const float *rho, int nx, int nz, int nb,
                             int ld, int kappa_fixed_rows, float *tmp2, float *gvp_pad, float *grho_pad,
                             float *grad_vp, float *grad_rho, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    const int nnx = nx + 2 * nb, nnz = nz + 2 * nb;
    const size_t F = (size_t)(nnx + 2 * S2D_GX) * ld;
    add_source_terms<<<1, 1, 0, st>>>(gk, src_cells, src_vals, nshots);
    dim3 blk(256), grd((nnz + 255) / 256, nnx);
    sum_shots<<<grd, blk, 0, st>>>(gk, gb, nacc, nnx, nnz, ld, tmp2, tmp2 + F);
    chain_rule<<<grd, blk, 0, st>>>(tmp2, tmp2 + F, vp, rho, nx, nz, nb, ld, kappa_fixed_rows, gvp_pad, grho_pad);
    dim3 grd2((nz + 255) / 256, nx);
    fold_sponge<<<grd2, blk, 0, st>>>(gvp_pad, grho_pad, nx, nz, nb, ld, grad_vp, grad_rho);
    return (int)cudaGetLastError();
}

int launch_residual(const float *seis, const float *obs, float *res, size_t n, double *sumsq, void *stream) {
    int grid = (int)std::min<size_t>(4096, (n + 255) / 256);
    if (grid < 1) grid = 1;
    residual_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(seis, obs, res, n, sumsq);
    return (int)cudaGetLastError();
}

}  // namespace s2d
