// On-chip time loop of libseis2d for sm_100a: the FD steps of
// src/src_cpu/cpumodelling.cpp:115-156 (as s2d_kernels.cu has them, the same
// bits) for grids whose whole state fits the chip's registers and shared
// memory.  One cooperative launch advances up to a whole run of steps.
//
// A block (one per SM) owns a tile of one shot: a 120-row strip and NC - 6
// columns.  Lane l of a warp holds rows 4l .. 4l+3 of C columns; px, vx, vz of
// those cells live in registers for the whole launch, pz (cells in the sponge
// only), kappa and the folded Lx bx, Lz bz in shared memory.  A step is two
// phases (pressure, velocity); z-neighbours come by shuffles, the columns at a
// warp's edges through shared memory, with one block barrier per phase.
//
// Halo: the tile carries 3 columns more on each side and lanes 0 and 31 as
// halo rows.  Pressure there is updated redundantly, so the blocks exchange
// velocities alone, once per step.  A block publishes the rows and columns its
// neighbours need as 16-byte pieces {three values, step tag} (relaxed, 128-bit
// single-copy atomic), and a neighbour polls the pieces until they carry the
// step's tag.  The pieces validate themselves: no flag, no fence, one trip
// through L2 per step.  A frame has two buffers (step parity): a block
// overwrites step s's pieces at step s+2, after it has read every neighbour's
// step s+1, which that neighbour published after reading step s.
//
// Every poll is bounded (spin_limit); a block that gives up records
// S2D_DEV_ERR_WAIT and leaves, and its neighbours follow when they see the
// error word.  All blocks of a launch are co-resident (cooperative launch), but
// work of other streams may let some of them start later than others: the
// blocks count themselves in when they start and no neighbour is waited for
// before all have (a wait of its own, kStartLimit).
//
// What bounds it: latency.  Counters of 100 steps of 1080 x 1080 (8 warps with 10
// columns on 135 SMs): 29 % of the issue slots and 20 % of the FMA pipe's cycles
// in use, 7.1 cycles from one instruction of a warp to its next:
// 1.6 in fixed latencies, 1.3 in the poll for the neighbours' pieces and other
// loads, 1.0 in shared memory, 0.4 each at the barriers, in branches and for the
// FMA pipe; L2 at 6 %, DRAM at 1 %.  More warps per tile, two blocks per SM (both
// wait at the same time), pz in shared memory and smaller frames measured no
// better.  us per FD step, with one launch of the two-step kernel per two steps
// in brackets: 265 x 165 cells 2.2 (7.6), 1080 x 1080 5.3 (11.1), one 1301 x 501
// shot 3.5 (10.6).  With the gradient's products (16 bytes per cell and step,
// stored past the caches' reuse): 8 shots of 1301 x 501 39 us per step (65 with
// one launch of the per-step kernel for all eight), 4 of 701 x 401 9.3 (18).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "s2d_device.cuh"
#include "s2d_pack.cuh"

namespace s2d {

namespace {

struct Piece {
    float v[3];
    unsigned tag;
};
__device__ __forceinline__ Piece ld_piece(const uint4 *p) {
    unsigned __int128 q;
    f2 a, b;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(q) : "l"(p) : "memory");
    asm("mov.b128 {%0, %1}, %2;" : "=l"(a), "=l"(b) : "q"(q));
    Piece r;
    r.v[0] = lo(a);
    r.v[1] = hi(a);
    r.v[2] = lo(b);
    r.tag = (unsigned)(b >> 32);
    return r;
}
__device__ __forceinline__ void st_piece(uint4 *p, float x, float y, float z, unsigned tag) {
    unsigned __int128 q;
    asm("mov.b128 %0, {%1, %2};" : "=q"(q) : "l"(pk(x, y)), "l"(pk(z, __uint_as_float(tag))));
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(q) : "memory");
}

// A block's frame: nine column items by lane (vx of the last three own columns
// and vz of the last, for the right neighbour; vx of the first three and vz of
// the first two, for the left one) as two pieces each (rows 0 .. 2; row 3),
// then the row pieces of every warp (row_piece).
constexpr int kColItems = 9, kColLeft = 4, kColPieces = 2 * kColItems;

// Row pieces of a warp with C columns, as float offsets into its row buffer
// [side][C][vx, vz][4] (side 0: the strip's last four rows, for the strip
// below; side 1: its first four, for the strip above): vz.yzw of side 0, vz.xyz
// and vx.xy of side 1 per column, and vx.w of side 0 of three columns at once.
__host__ __device__ constexpr int row_pieces(int c) { return 3 * c + (c + 2) / 3; }
__device__ __forceinline__ int row_piece(int q, int c, int &stride, int &side) {
    stride = 1;
    side = q >= c && q < 3 * c;
    if (q < c) return q * 8 + 5;
    if (q < 2 * c) return q * 8 + 4;
    if (q < 3 * c) return (q - c) * 8;
    stride = 8;
    return (q - 3 * c) * 24 + 3;
}

// Shared memory of a block of NW warps with C columns each, in V4 (16 B).
template <int NW, int C>
struct ResSmem {
    static constexpr int NC = NW * C;
    static constexpr int NR = row_pieces(C);
    static constexpr int mat = 0;                             // [3][NC][32]: kappa, Lx bx, Lz bz
    static constexpr int vxe = mat + 3 * NC * 32;             // [NW + 2][3][32]: vx at the warps' edges
    static constexpr int pe = vxe + (NW + 2) * 96;            // [NW + 2][3][32]: p at the warps' edges
    static constexpr int ct = pe + (NW + 2) * 96;             // [NC][4]
    static constexpr int rt = ct + NC * 4;                    // [8][32]
    static constexpr int rowo = rt + 8 * 32;                  // [NW][2][C][2]: rows to publish
    static constexpr int rowi = rowo + NW * 4 * C + 8;        // the same: halo rows received (+8: a piece may overhang)
    static constexpr int colh = rowi + NW * 4 * C + 8;        // [kColItems][32]: halo columns received
    static constexpr int rid = colh + kColItems * 32;         // [NC] int
    static constexpr int total = rid + (NC + 3) / 4;
    static constexpr size_t bytes = (size_t)total * 16;
    static constexpr int pieces = kColPieces * 32 + NW * NR;  // of one block's frame
};

constexpr unsigned kNoPiece = 0xffffffffu;

// Bytes before the frames, for the count of started blocks: whole lines, so that
// a warp's 512 bytes of pieces stay four of them (with 16 bytes, five: 5.3
// against 5.5 us per step of 1080 x 1080).
constexpr size_t kFramesHead = 512;
// Polls (1 us or more each) for all blocks of a launch to start.  Whatever else
// runs on the GPU delays them by its own length; 2^24 are some 20 s.
constexpr int kStartLimit = 1 << 24;
__device__ __forceinline__ unsigned ld_count(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool all_started(const ResArgs &a) {
    for (int t = 0; ld_count(a.started) < gridDim.x; ++t) {
        if (t >= kStartLimit) {
            atomicOr(a.err, S2D_DEV_ERR_WAIT);
            return false;
        }
        if ((t & 255) == 255 && *reinterpret_cast<volatile int *>(a.err) != 0) return false;
        __nanosleep(500);
    }
    return true;
}

// What the columns of a warp are: all in the shot's fast columns (dampings 1,
// literal operator pairs); all damped, with literal pairs; anything.
enum { kIn = 0, kDamped = 1, kAny = 2 };

// TILE: the kind of tile, bit 0 every row of the strip in the shot's fast rows
// (undamped, literal operator pairs), bit 1 every column of the tile in its
// fast columns; kAnyTile: decided at run time (zf_rt), for the widest tiles,
// whose registers leave the compiler no room for the specialised copies
// (10 columns per warp: 5.0 us per step against 6.8), and for products from 5
// columns on (7 columns, 8 shots of 1301 x 501: 39 us per step against 43).
constexpr int kAnyTile = 4;
// PROD: every step also leaves its products (S2D_STEP_PRODUCTS, the slots that
// the adjoint step reads) of the tile's own cells.
template <int NW, int C, int TILE, bool PROD>
__device__ __forceinline__ void resident_tile(const ResArgs &a, const ResShot &rs, const ShotDev &S, int cx, int cz,
                                              bool zf_rt, V4 *sm, int *s_rec, int *s_fail) {
    constexpr bool XI = TILE != kAnyTile && (TILE & 2);
    const bool zf = TILE == kAnyTile ? zf_rt : (TILE & 1) != 0;
    using L = ResSmem<NW, C>;
    constexpr int NC = L::NC, NT = NW * 32, WD = NC - 6;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int xt = cx * WD - 3;                   // column of local column 0; own columns are local 3 .. NC-4
    const int zc = cz * S2D_STRIP_OUT - 4;        // first row of lane 0
    const int z0 = zc + 4 * lane;
    const int lc0 = w * C;                        // local column of this warp's first
    const ptrdiff_t ld = S.ld;
    const int fs = S.fstride;
    V4 *const pe = sm + L::pe + (w + 1) * 96 + lane;
    V4 *const vxe = sm + L::vxe + (w + 1) * 96 + lane;
    const V4 *const mat = sm + L::mat + lc0 * 32 + lane;
    const V4 *const ct = sm + L::ct + lc0 * 4;
    const V4 *const rt = sm + L::rt + lane;
    const V4 *const colh = sm + L::colh + lane;
    float *const smf = reinterpret_cast<float *>(sm);
    int *const rid = reinterpret_cast<int *>(sm + L::rid);

    // ---- load the tile ----
    V4 px[C], pz[C], vx[C], vz[C];
    {
        const float *const st = S.st[0][0] + (size_t)a.par0 * 4 * fs + (z0 + S2D_GZ) + (ptrdiff_t)S2D_GX * ld;
        const float *const kp = S.kappa + (z0 + S2D_GZ) + (ptrdiff_t)S2D_GX * ld;
        V4 *const m = sm + L::mat + lc0 * 32 + lane;
        V4 lz;
        {
            const float4 *zp = S.zcoef + (z0 + S2D_GZ);
            lz = v4(pk(__ldg(zp).w, __ldg(zp + 1).w), pk(__ldg(zp + 2).w, __ldg(zp + 3).w));
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const int x = xt + lc0 + j;
            V4 k = zero4(), bx = zero4(), bz = zero4();
            px[j] = pz[j] = vx[j] = vz[j] = zero4();
            if (x < S.nnx) {  // x >= -3: the ghost columns before the grid hold zeros
                const ptrdiff_t o = (ptrdiff_t)x * ld;
                px[j] = v4(__ldcg(reinterpret_cast<const float4 *>(st + o)));
                pz[j] = v4(__ldcg(reinterpret_cast<const float4 *>(st + o + fs)));
                vx[j] = v4(__ldcg(reinterpret_cast<const float4 *>(st + o + 2 * (ptrdiff_t)fs)));
                vz[j] = v4(__ldcg(reinterpret_cast<const float4 *>(st + o + 3 * (ptrdiff_t)fs)));
                k = v4(ld4(kp + o));
                // the folded products of the velocity update, rounded as upd() rounds them
                bx = dup4(__ldg(S.xcoef + (x + S2D_GX)).w) * v4(ld4(kp + o + fs));
                bz = lz * v4(ld4(kp + o + 2 * (ptrdiff_t)fs));
            }
            m[j * 32] = k;
            m[(NC + j) * 32] = bx;
            m[(2 * NC + j) * 32] = bz;
        }
    }
    // everything after the materials starts at zero: the halo rows and
    // columns outside the grid are never received and stay so
    for (int i = L::vxe + threadIdx.x; i < L::total; i += NT) sm[i] = zero4();
    __syncthreads();
    if (w == 0) {
        float r[8][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 q = __ldg(S.zcoef + (z0 + i + S2D_GZ));
            r[0][i] = q.x;
            r[1][i] = q.y;
            r[4][i] = q.z;
            dm_coef(z0 + i, S.nnz, r[2][i], r[3][i]);
            dp_coef(z0 + i, S.nnz, r[5][i], r[6][i]);
            // bits of pz that rows keep (none of undamped ones: the cell carries p in px alone).  A mask, not a
            // factor 0: an overflowed derivative times 0 would leave NaN there
            r[7][i] = q.x == 1.0f ? 0.0f : __int_as_float(-1);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) sm[L::rt + k * 32 + lane] = v4(pk(r[k][0], r[k][1]), pk(r[k][2], r[k][3]));
    }
    // column coefficients, doubled for the packed operations:
    // (Dax, Kx), (Dbx, D+ c0), (D- pair), (D+ c1)
    for (int lc = threadIdx.x; lc < NC; lc += NT) {
        const int x = xt + lc;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        float m0 = 0.f, m1 = 0.f, p0 = 0.f, p1 = 0.f;
        if (x < S.nnx) {
            q = __ldg(S.xcoef + (x + S2D_GX));
            dm_coef(x, S.nnx, m0, m1);
            dp_coef(x, S.nnx, p0, p1);
        }
        V4 *c = sm + L::ct + lc * 4;
        c[0] = v4(dup(q.x), dup(q.y));
        c[1] = v4(dup(q.z), dup(p0));
        c[2] = v4(dup(m0), dup(m1));
        c[3] = v4(dup(p1), 0ull);
    }
    int cls = kIn;
    if (!XI) {
        const int x0 = xt + lc0, x1 = x0 + C;  // the warp's columns
        const int x = x0 + lane;
        const bool und = lane < C && x < S.nnx && __ldg(S.xcoef + (x + S2D_GX)).x == 1.0f;
        const bool none = __ballot_sync(kFull, und) == 0;
        cls = x0 >= S.xfast_lo && x1 <= S.xfast_hi ? kIn : none && x0 >= 2 && x1 <= S.nnx - 2 ? kDamped : kAny;
    }
    // Receivers of the tile's own cells.  All on one row and at most one per
    // column (a surface line): their trace indices by column; else the lists
    // are read as they stand.
    const bool rec = !(a.flags & S2D_STEP_NO_RECORD) && S.rec_zhi >= zc + 4 && S.rec_zlo < zc + 4 + S2D_STRIP_OUT;
    if (rec) {
        for (int c = threadIdx.x; c < NC; c += NT) {
            const int x = xt + c;
            int id = -1;
            if (c >= 3 && c < NC - 3 && x < S.nnx) {
                const int j0 = __ldg(S.rec_ptr + x), n = __ldg(S.rec_ptr + x + 1) - j0;
                if (n > 0) atomicOr(s_rec, n > 1 || S.rec_zlo != S.rec_zhi ? 3 : 1);
                if (n > 0) id = __ldg(S.rec_id + j0);
            }
            rid[c] = id;
        }
    }
    const int rl = (S.rec_zlo - zc) >> 2, ri = (S.rec_zlo - zc) & 3;
    // source cell (halo copies of it included): this lane's column and row
    int sj = -1, si = 0;
    {
        const int c = S.src_x - xt - lc0, r = S.src_z - z0;
        if (c >= 0 && c < C && r >= 0 && r < 4) {
            sj = c;
            si = r;
        }
    }
    const bool src_warp = __any_sync(kFull, sj >= 0);

    // ---- frames ----
    const int cta = rs.cta0 + cx * rs.ncz + cz;
    uint4 *const fr = reinterpret_cast<uint4 *>(a.frames);
    const size_t plane = (size_t)gridDim.x * L::pieces;
    uint4 *const mine = fr + (size_t)cta * L::pieces;
    const bool has_l = cx > 0, has_r = cx + 1 < rs.ncx, has_u = cz > 0, has_d = cz + 1 < rs.ncz;
    const bool edge_lane = lane == 1 || lane == 30;
    V4 *const row_out = sm + L::rowo + w * 4 * C + (lane == 1 ? 2 * C : 0);
    // Outgoing row pieces of the warp: float offset (kNoPiece: none) and stride
    constexpr int NO = (L::NR + 31) / 32;
    unsigned ro[NO];
    int rs_[NO];
#pragma unroll
    for (int i = 0; i < NO; ++i) {
        const int q = lane + 32 * i;
        int side;
        const int o = row_piece(q, C, rs_[i], side);
        ro[i] = q < L::NR && (side ? has_u : has_d) ? (unsigned)((L::rowo + w * 4 * C) * 4 + o) : kNoPiece;
    }
    // Incoming pieces, spread over all threads: the row pieces of every warp
    // (side 0 from the strip above, side 1 from the strip below), then the
    // column pieces by lane, lanes 0 and 31 from the diagonal blocks.
    constexpr int kRow = NW * L::NR, kCol = kColPieces * 32, NI = (kRow + kCol + NT - 1) / NT;
    unsigned at[NI];
    unsigned to[NI];  // float offset, stride << 16
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int q = threadIdx.x + i * NT;
        at[i] = kNoPiece;
        to[i] = 0;
        int stride;
        if (q < kRow) {
            int side;
            const int o = row_piece(q % L::NR, C, stride, side);
            if (side ? has_d : has_u) at[i] = (unsigned)((cta + (side ? 1 : -1)) * L::pieces + kColPieces * 32 + q);
            to[i] = (unsigned)((L::rowi + q / L::NR * 4 * C) * 4 + o + (stride << 16));
        } else if (q < kRow + kCol) {
            const int p = (q - kRow) / 32, ln = (q - kRow) % 32, item = p / 2, half = p % 2;
            const int dx = item < kColLeft ? -1 : 1, dz = ln == 0 ? -1 : ln == 31 ? 1 : 0;
            const int from = ln == 0 ? 30 : ln == 31 ? 1 : ln;
            if ((dx < 0 ? has_l : has_r) && cz + dz >= 0 && cz + dz < rs.ncz)
                at[i] = (unsigned)((cta + dx * rs.ncz + dz) * L::pieces + p * 32 + from);
            stride = half ? 0 : 1;
            to[i] = (unsigned)((L::colh + item * 32 + ln) * 4 + 3 * half + (stride << 16));
        }
    }
    const bool top = lane == 0 && has_u, bot = lane == 31 && has_d;
    const V4 *const row_in = sm + L::rowi + w * 4 * C + (lane == 31 ? 2 * C : 0);

    // vx of the warp's edge columns for its neighbours: columns 0, C-2, C-1
    vxe[0] = vx[0];
    vxe[32] = vx[C - 2];
    vxe[64] = vx[C - 1];
    __syncthreads();
    const int n_rec = *s_rec;
    const int nstep = a.nsteps;
    float amp = src_warp ? __ldg(S.amp + a.kt0) : 0.0f;
    const V4 A0 = dup4(kA0), A1 = dup4(kA1);
    // 1 in a register the compiler knows nothing of: a fused multiply-add by a
    // literal 1 is rewritten into one that fuses the product of its addend too
    const V4 one = dup4(a.one);
    const V4 kx_in = dup4(S.kx_in), kz_in = dup4(S.kz_in);
    // steps until the next recorded one, and its sample
    int slot = (a.kt0 + 1 + a.dt_factor - 1) / a.dt_factor - 1;
    int wait = (slot + 1) * a.dt_factor - 1 - a.kt0;
    const bool merged = zf && (XI || cls == kIn);  // every cell of the warp carries p in px alone
    // products: the lane's rows of the warp's own columns (bit j of own)
    const size_t F = (size_t)(S.nnx + 2 * S2D_GX) * ld;
    float *prod = nullptr;
    unsigned own = 0;
    if (PROD) {
        prod = S.prod + (size_t)(a.kt0 - a.prod_kt0) * 4 * F + (z0 + S2D_GZ) + (ptrdiff_t)(xt + lc0 + S2D_GX) * ld;
        if (lane >= 1 && lane <= 30 && z0 < S.nnz) {
#pragma unroll
            for (int j = 0; j < C; ++j)
                if (lc0 + j >= 3 && lc0 + j < NC - 3 && xt + lc0 + j < S.nnx) own |= 1u << j;
        }
    }
    auto keep = [&](int slot, int j, const V4 &v) {
        if (own >> j & 1) __stcs(reinterpret_cast<float4 *>(prod + slot * F + (ptrdiff_t)j * ld),
                                 make_float4(lo(v.a), hi(v.a), lo(v.b), hi(v.b)));
    };

    for (int s = 0; s < nstep; ++s) {
        V4 q0 = vxe[-64], q1 = vxe[-32], qr = vxe[96];
        if (s > 0) {
            // the neighbours' velocities after the previous step: the halo rows
            // (only the values next to the strip are received and needed) ...
            if (top || bot) {
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    vx[j] = row_in[j * 2];
                    vz[j] = row_in[j * 2 + 1];
                }
                if (w > 0) {
                    q0 = row_in[(C - 2) * 2 - 4 * C];
                    q1 = row_in[(C - 1) * 2 - 4 * C];
                }
                if (w + 1 < NW) qr = row_in[4 * C];
            }
            // ... then the halo columns: lanes 0 and 31 take the diagonal blocks'
            if (has_l) {
                if (w == 0) {
                    vx[0] = colh[0];
                    vx[1] = colh[32];
                    vx[2] = colh[64];
                    vz[2] = colh[96];
                }
                if (C == 3 && w == 1) q0 = colh[32];
                if (C <= 4 && w == 1) (C == 3 ? q1 : q0) = colh[64];
            }
            if (has_r) {
                if (w == NW - 1) {
                    vx[C - 3] = colh[4 * 32];
                    vx[C - 2] = colh[5 * 32];
                    vx[C - 1] = colh[6 * 32];
                    vz[C - 3] = colh[7 * 32];
                    vz[C - 2] = colh[8 * 32];
                }
                if (C == 3 && w == NW - 2) qr = colh[4 * 32];
            }
        }
        const bool rec_step = wait == 0 && n_rec != 0 && slot < S.real_nt;
        const float amp_next = src_warp && s + 1 < nstep ? __ldg(S.amp + a.kt0 + s + 1) : 0.0f;
        // ---- pressure: column j needs vx at j-2 .. j+1 ----
        // (no branch inside the unrolled loop: the columns overlap)
        auto pressure = [&](auto cls_, auto zf_) {
            constexpr int CLS = decltype(cls_)::value;
            constexpr bool ZF = decltype(zf_)::value;
            const V4 kz = ZF ? kz_in : rt[1 * 32], daz = ZF ? one : rt[0];
            const V4 m0 = ZF ? A0 : rt[2 * 32], m1 = ZF ? A1 : rt[3 * 32];
            const V4 keep_pz = ZF ? one : rt[7 * 32];
            const bool r0 = lo(daz.a) == 1.0f, r1 = hi(daz.a) == 1.0f, r2 = lo(daz.b) == 1.0f, r3 = hi(daz.b) == 1.0f;
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const V4 q2 = vx[j], q3 = j + 1 < C ? vx[j + 1 < C ? j + 1 : 0] : qr;
                V4 dax = one, kx = kx_in, cm0 = A0, cm1 = A1;
                if (CLS != kIn) {
                    const V4 c = ct[j * 4];
                    dax = v4(c.a, c.a);
                    kx = v4(c.b, c.b);
                }
                if (CLS == kAny) {
                    const V4 c = ct[j * 4 + 2];
                    cm0 = v4(c.a, c.a);
                    cm1 = v4(c.b, c.b);
                }
                const V4 k = mat[j * 32];
                const V4 dx = dif4(cm0, q2 - q1, cm1, q3 - q0);
                const V4 dz = dminus_z(m0, m1, vz[j]);
                // a cell whose column and row are undamped carries p alone
                const V4 t = dif4(kx, dx, kz, dz);
                const V4 pm = fma4(k, t, px[j]);
                if (CLS == kIn && ZF) {
                    px[j] = pm;
                    if (PROD) keep(0, j, t);
                } else {
                    const V4 ps = fma4(dax, px[j], (kx * k) * dx);
                    const V4 pn = fma4(daz, pz[j], (kz * k) * dz);
                    if (CLS == kDamped) {
                        px[j] = ps;
                        pz[j] = pn;
                        if (PROD) {
                            keep(0, j, dx);
                            keep(1, j, dz);
                        }
                    } else {
                        const bool und = CLS == kIn || lo(dax.a) == 1.0f;
                        const bool u0 = und && r0, u1 = und && r1, u2 = und && r2, u3 = und && r3;
                        px[j] = v4(pk(u0 ? lo(pm.a) : lo(ps.a), u1 ? hi(pm.a) : hi(ps.a)),
                                   pk(u2 ? lo(pm.b) : lo(ps.b), u3 ? hi(pm.b) : hi(ps.b)));
                        pz[j] = CLS == kIn ? v4(pn.a & keep_pz.a, pn.b & keep_pz.b)
                                           : v4(pk(u0 ? 0.0f : lo(pn.a), u1 ? 0.0f : hi(pn.a)),
                                                pk(u2 ? 0.0f : lo(pn.b), u3 ? 0.0f : hi(pn.b)));
                        if (PROD) {
                            keep(0, j, v4(pk(u0 ? lo(t.a) : lo(dx.a), u1 ? hi(t.a) : hi(dx.a)),
                                          pk(u2 ? lo(t.b) : lo(dx.b), u3 ? hi(t.b) : hi(dx.b))));
                            keep(1, j, v4(pk(u0 ? 0.0f : lo(dz.a), u1 ? 0.0f : hi(dz.a)),
                                          pk(u2 ? 0.0f : lo(dz.b), u3 ? 0.0f : hi(dz.b))));
                        }
                    }
                }
                q0 = q1;
                q1 = q2;
            }
        };
        if (XI || cls == kIn) {
            if (zf) pressure(std::integral_constant<int, kIn>(), std::true_type());
            else pressure(std::integral_constant<int, kIn>(), std::false_type());
        } else if (cls == kDamped) {
            pressure(std::integral_constant<int, kDamped>(), std::false_type());
        } else {
            pressure(std::integral_constant<int, kAny>(), std::false_type());
        }
        if (src_warp) {
#pragma unroll
            for (int j = 0; j < C; ++j)
                if (j == sj) {
                    if (si == 0) px[j].a = pk(lo(px[j].a) + amp, hi(px[j].a));
                    else if (si == 1) px[j].a = pk(lo(px[j].a), hi(px[j].a) + amp);
                    else if (si == 2) px[j].b = pk(lo(px[j].b) + amp, hi(px[j].b));
                    else px[j].b = pk(lo(px[j].b), hi(px[j].b) + amp);
                }
            amp = amp_next;
        }
        // p of the edge columns for the neighbour warps
        if (merged) {
            pe[0] = px[0];
            pe[32] = px[1];
            pe[64] = px[C - 1];
        } else {
            pe[0] = px[0] + pz[0];
            pe[32] = px[1] + pz[1];
            pe[64] = px[C - 1] + pz[C - 1];
        }
        __syncthreads();
        // ---- velocity: column j needs p at j-1 .. j+2 ----
        const unsigned tag = (unsigned)(s + 1);
        uint4 *const out = mine + (s & 1 ? plane : 0);
        const bool publish = s + 1 < nstep && !(s == a.fault_step && cta == 0);
        auto velocity = [&](auto cls_, auto zf_) {
            constexpr int CLS = decltype(cls_)::value;
            constexpr bool ZF = decltype(zf_)::value;
            const V4 dbz = ZF ? one : rt[4 * 32];
            const V4 p0 = ZF ? A0 : rt[5 * 32], p1 = ZF ? A1 : rt[6 * 32];
            auto p_of = [&](int j) { return CLS == kIn && ZF ? px[j] : px[j] + pz[j]; };
            V4 g0 = pe[-32], g1 = p_of(0), g2 = p_of(1);
            const V4 gr0 = pe[96], gr1 = pe[128];
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const V4 g3 = j + 2 < C ? p_of(j + 2 < C ? j + 2 : 0) : j + 2 == C ? gr0 : gr1;
                V4 dbx = one, cp0 = A0, cp1 = A1;
                if (CLS != kIn) {
                    const V4 c = ct[j * 4 + 1];
                    dbx = v4(c.a, c.a);
                    if (CLS == kAny) {
                        cp0 = v4(c.b, c.b);
                        const f2 c1 = ct[j * 4 + 3].a;
                        cp1 = v4(c1, c1);
                    }
                }
                const V4 bx = mat[(NC + j) * 32], bz = mat[(2 * NC + j) * 32];
                const V4 ex = dif4(cp0, g2 - g1, cp1, g3 - g0);
                const V4 ez = dplus_z(p0, p1, g1);
                if (PROD) {
                    keep(2, j, ex);
                    keep(3, j, ez);
                }
                vx[j] = fma4(dbx, vx[j], bx * ex);
                vz[j] = fma4(dbz, vz[j], bz * ez);
                g0 = g1;
                g1 = g2;
                g2 = g3;
            }
        };
        if (XI || cls == kIn) {
            if (zf) velocity(std::integral_constant<int, kIn>(), std::true_type());
            else velocity(std::integral_constant<int, kIn>(), std::false_type());
        } else if (cls == kDamped) {
            velocity(std::integral_constant<int, kDamped>(), std::false_type());
        } else {
            velocity(std::integral_constant<int, kAny>(), std::false_type());
        }
        // ---- publish the frame ----
        if (edge_lane) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
                row_out[j * 2] = vx[j];
                row_out[j * 2 + 1] = vz[j];
            }
        }
        vxe[0] = vx[0];
        vxe[32] = vx[C - 2];
        vxe[64] = vx[C - 1];
        if (publish) {
            auto col = [&](int item, const V4 &v) {
                uint4 *o = out + item * 64 + lane;
                st_piece(o, lo(v.a), hi(v.a), lo(v.b), tag);
                st_piece(o + 32, hi(v.b), hi(v.b), hi(v.b), tag);
            };
#pragma unroll
            for (int j = 0; j < C; ++j) {
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    if ((3 + r) % C == j && w == (3 + r) / C && has_l) {
                        col(4 + r, vx[j]);
                        if (r < 2) col(7 + r, vz[j]);
                    }
                    if ((NC - 6 + r) % C == j && w == (NC - 6 + r) / C && has_r) {
                        col(r, vx[j]);
                        if (r == 2) col(3, vz[j]);
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NO; ++i)
                if (ro[i] != kNoPiece) {
                    const float *v = smf + ro[i];
                    st_piece(out + kColPieces * 32 + w * L::NR + lane + 32 * i, v[0], v[rs_[i]], v[2 * rs_[i]], tag);
                }
        }
        // ---- receivers (cpumodelling.cpp:356-360) ----
        if (rec_step) {
            auto p_of = [&](int j) { return merged ? px[j] : px[j] + pz[j]; };
            if (n_rec == 1) {
                if (lane == rl) {
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        const int id = rid[lc0 + j];
                        const V4 p = p_of(j);
                        if (id >= 0)
                            S.seis[(size_t)id * S.real_nt + slot] =
                                ri == 0 ? lo(p.a) : ri == 1 ? hi(p.a) : ri == 2 ? lo(p.b) : hi(p.b);
                    }
                }
            } else if (lane >= 1 && lane <= 30) {
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    const int lc = lc0 + j, x = xt + lc;
                    if (lc < 3 || lc >= NC - 3 || x >= S.nnx) continue;
                    const V4 p = p_of(j);
                    const int e1 = __ldg(S.rec_ptr + x + 1);
                    for (int e = __ldg(S.rec_ptr + x); e < e1; ++e) {
                        const int r = __ldg(S.rec_z + e) - z0;
                        if (r >= 0 && r < 4)
                            S.seis[(size_t)__ldg(S.rec_id + e) * S.real_nt + slot] =
                                r == 0 ? lo(p.a) : r == 1 ? hi(p.a) : r == 2 ? lo(p.b) : hi(p.b);
                    }
                }
            }
        }
        if (PROD) prod += 4 * F;
        if (wait == 0) {
            wait = a.dt_factor;
            ++slot;
        }
        --wait;
        if (s + 1 == nstep) break;
        // ---- receive the neighbours' velocities of this step ----
        {
            const uint4 *const base = fr + (s & 1 ? plane : 0);
            Piece v[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i)
                if (at[i] != kNoPiece) v[i] = ld_piece(base + at[i]);
            bool ok = false;
            for (int t = 0; !ok; ++t) {
                ok = true;
#pragma unroll
                for (int i = 0; i < NI; ++i) ok = ok && (at[i] == kNoPiece || v[i].tag == tag);
                if (ok) break;
                if (t >= a.spin_limit) {
                    atomicOr(a.err, S2D_DEV_ERR_WAIT);
                    break;
                }
                if ((t & 255) == 255 && *reinterpret_cast<volatile int *>(a.err) != 0) break;
#pragma unroll
                for (int i = 0; i < NI; ++i)
                    if (at[i] != kNoPiece && v[i].tag != tag) v[i] = ld_piece(base + at[i]);
            }
            if (!ok) *s_fail = 1;
#pragma unroll
            for (int i = 0; i < NI; ++i)
                if (at[i] != kNoPiece) {
                    const unsigned stride = to[i] >> 16;
                    float *d = smf + (to[i] & 0xffff);
                    d[0] = v[i].v[0];
                    d[stride] = v[i].v[1];
                    d[2 * stride] = v[i].v[2];
                }
        }
        __syncthreads();
        if (*s_fail) return;
    }

    // ---- write the state of step kt0 + nsteps ----
    {
        float *const st =
            S.st[0][0] + (size_t)a.par1 * 4 * fs + (z0 + S2D_GZ) + (ptrdiff_t)S2D_GX * ld;
        if (lane >= 1 && lane <= 30 && z0 < S.nnz) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const int lc = lc0 + j, x = xt + lc;
                if (lc >= 3 && lc < NC - 3 && x < S.nnx) {
                    float *o = st + (ptrdiff_t)x * ld;
                    *reinterpret_cast<V4 *>(o) = px[j];
                    *reinterpret_cast<V4 *>(o + fs) = pz[j];
                    *reinterpret_cast<V4 *>(o + 2 * (ptrdiff_t)fs) = vx[j];
                    *reinterpret_cast<V4 *>(o + 3 * (ptrdiff_t)fs) = vz[j];
                }
            }
        }
    }
}

template <int NW, int C, bool PROD>
__global__ void __launch_bounds__(NW * 32, 1) resident_kernel(const ResArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_rec, s_fail;
    __shared__ ShotDev S;
    // the block's shot and tile
    int g = 0;
    while (g + 1 < a.nrs && __ldg(&a.rs[g + 1].cta0) <= (int)blockIdx.x) ++g;
    const ResShot rs = a.rs[g];
    if (threadIdx.x == 0) {
        atomicAdd(a.started, 1u);
        s_rec = 0;
        s_fail = !all_started(a);
    }
    if (threadIdx.x < sizeof(ShotDev) / 8)
        reinterpret_cast<unsigned long long *>(&S)[threadIdx.x] =
            reinterpret_cast<const unsigned long long *>(a.shots + rs.shot)[threadIdx.x];
    __syncthreads();
    if (s_fail) return;
    const int b = (int)blockIdx.x - rs.cta0;
    const int cz = b % rs.ncz, cx = b / rs.ncz;
    const int zc = cz * S2D_STRIP_OUT - 4;
    const int xt = cx * (NW * C - 6) - 3;
    V4 *const sm = reinterpret_cast<V4 *>(smem);
    const bool zf = rows_fast(S, zc, zc + S2D_STRIP_ROWS - 1);
    const bool xi = xt >= S.xfast_lo && xt + NW * C <= S.xfast_hi;
    if constexpr (C >= 8 || (PROD && C >= 5)) {
        resident_tile<NW, C, kAnyTile, PROD>(a, rs, S, cx, cz, zf, sm, &s_rec, &s_fail);
    } else {
        if (zf && xi) resident_tile<NW, C, 3, PROD>(a, rs, S, cx, cz, zf, sm, &s_rec, &s_fail);
        else if (zf) resident_tile<NW, C, 1, PROD>(a, rs, S, cx, cz, zf, sm, &s_rec, &s_fail);
        else if (xi) resident_tile<NW, C, 2, PROD>(a, rs, S, cx, cz, zf, sm, &s_rec, &s_fail);
        else resident_tile<NW, C, 0, PROD>(a, rs, S, cx, cz, zf, sm, &s_rec, &s_fail);
    }
}

template <int NW, int C, bool PROD>
int launch_c(const ResArgs &a, int grid, cudaStream_t st) {
    static_assert(ResSmem<NW, C>::bytes <= 226 * 1024, "shared memory of a block");
    const void *k = (const void *)resident_kernel<NW, C, PROD>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ResSmem<NW, C>::bytes);
    if (e != cudaSuccess) return (int)e;
    ResArgs v = a;
    v.one = 1.0f;
    v.started = reinterpret_cast<unsigned *>(v.frames);
    v.frames += kFramesHead / sizeof(*v.frames);
    void *args[] = {&v};
    return (int)cudaLaunchCooperativeKernel(k, dim3(grid), dim3(NW * 32), args, ResSmem<NW, C>::bytes, st);
}

}  // namespace

// Block shapes (warps, columns per warp) and the measured time of one step of
// such a tile, us (exchange included, all SMs busy).
#define S2D_RES_SHAPES(X)                                                                                        \
    X(4, 3, 2.3) X(4, 4, 2.4) X(8, 3, 2.35) X(8, 4, 2.55) X(8, 5, 2.95) X(8, 6, 3.3) X(8, 7, 3.55) X(8, 8, 4.35) \
    X(8, 9, 4.8) X(8, 10, 5.4)

size_t resident_frame_bytes(int nw, int c, int ctas) {
    return kFramesHead + (size_t)2 * ctas * (kColPieces * 32 + nw * row_pieces(c)) * 16;
}

int launch_resident(int nw, int c, const ResArgs &a, int grid, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
#define X(W, N, US) \
    if (nw == W && c == N) return a.flags & S2D_STEP_PRODUCTS ? launch_c<W, N, true>(a, grid, st) : launch_c<W, N, false>(a, grid, st);
    S2D_RES_SHAPES(X)
#undef X
    return (int)cudaErrorInvalidValue;
}

int resident_shapes(int i, int *nw, int *c, double *us) {
    static const struct {
        int nw, c;
        double us;
    } s[] = {
#define X(W, N, US) {W, N, US},
        S2D_RES_SHAPES(X)
#undef X
    };
    if (i < 0 || i >= (int)(sizeof(s) / sizeof(s[0]))) return 0;
    *nw = s[i].nw;
    *c = s[i].c;
    *us = s[i].us;
    return 1;
}

bool resident_plan(int sm_count, int nnx, int nnz, int nshots, bool plain, int shape, ResPlan *out) {
    ResPlan best;
    const int ncz = num_strips(nnz);
    int nw, c;
    double us;
    for (int i = 0; resident_shapes(i, &nw, &c, &us); ++i) {
        if (shape && shape != nw * 100 + c) continue;
        const int own = nw * c - 6, ncx = (nnx + own - 1) / own;
        const int conc = (int)std::min<long>(plain ? 1 : nshots, sm_count / ((long)ncx * ncz));
        if (conc < 1) continue;
        const double t = us * ((nshots + conc - 1) / conc);
        if (!best.conc || t < best.step_us) best = ResPlan{conc, ncx, ncz, nw, c, t};
    }
    *out = best;
    return best.conc > 0;
}

}  // namespace s2d
