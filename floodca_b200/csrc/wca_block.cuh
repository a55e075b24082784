// The FP32 step on column pairs, one CTA per row range.
//
// The same arithmetic as sweep_segment (FloodCA src/kernels/physics.h and
// src/common/model.c:321-605), organised as passes of BLK_ROWS rows by a CTA
// of BLK_ROWS warps. In a pass warp w holds row i = first + w of a strip of
// 64 columns (two adjacent columns per lane, one packed f32x2 pair) and runs
//
//     A  the faces of row i (x) and between rows i-1 and i (y, diagonals)
//     C  outflow and limiter of row i-1
//     D  depth update of row i-2, hmax, tmax
//     E  the next step's stable velocity of row i-3, when the pass has a
//        candidate for it
//
// with a CTA barrier after A, C and D. What a phase leaves for other rows
// (face discharges X, Y, E, W, limiter S, new level L) goes through shared
// memory; the rows of z, h, n and hmax come by TMA, one tile a field and pass,
// BLK_STAGES - 1 passes ahead.
//
// What bounds it, and why this split. A sweep in which each warp carries its
// rows from A to E in registers needs every phase's state at once: 128
// registers, 16 warps per SM, 709 warp instructions per 64-column row. With a
// barrier between the phases each phase's registers die with it (64
// registers, 32 warps per SM), the row ring is a fixed address distance
// instead of register moves, and rows are shared by the CTA, so a range costs
// six rows of halo per CTA instead of per warp. About 420 warp instructions
// per row at 63 % of the issue slots. Measured on a B200, microseconds a
// step, warm grids, one warp per row range (before) and this: 4096^2 350 and
// 215, 2048^2 112 and 65, 1024^2 51.5 and 22.9, 256^2 20.1 and 10.5, 1003 x
// 1498 with K = 8 104 and 49, 733 x 1101 with SEA and WALL cells 54 and 26.
// Bound by issue slots and the barriers (HBM is at 24 %). Tried and slower: 3
// CTAs of 80 registers without spills 2 %, CTAs of four warps 4 % (20 to 35 % on
// small grids), the next pass's A before the barrier after D 10 %.
//
// Grids with SEA or WALL cells (GEN) carry the mask in the device copies of z
// and n (k_encode_mask): n is NaN on every cell that is not LAND, z is PAD_Z
// on WALL (a face to it carries nothing, as to the padding) and -PAD_Z on SEA.
// A row whose cells are all LAND runs the same code as on an all-LAND grid
// after a vote on its n; the others take a branch that puts in the sea level
// and keeps the cells that are not LAND as they are.
#pragma once

#include <cstddef>
#include <type_traits>

#include "wca_f2.cuh"
#include "wca_tma.cuh"

namespace fcab {

constexpr int BLK_ROWS = 8;                 // rows per pass = warps per CTA
constexpr int BLK_THREADS = 32 * BLK_ROWS;
constexpr int BLK_STAGES = 3;               // tile stages: the pass at work and those ahead
constexpr uint32_t BLK_ROW_B = 256;         // bytes of a strip row
// Cells up to which the step's last CTA does a missed seed's velocity pass
// alone: it reads the depths and evaluates the cells deep enough to matter, a
// few as a rule, but all wet ones after a sharp fall of the maximum: 10 ns a
// cell (3809 x 132 masked with a point inflow, two such passes in 169 steps:
// 15.5 ms a run with a limit of 2^20 cells, 5.6 with the pass launched). One
// step in a hundred needs it; a kernel that could launch the pass costs 1.3 us
// more to launch every step and cannot overlap its start with the step before,
// and a graph of such kernels takes 3.5 ms more to build and free. What the
// grids between pay for that worst case: 300 steps of 733 x 1101 9.9 ms with
// this limit, 9.1 with 2^20; a call of fca_cuda_run of 400 steps at 1024^2
// 17.0 ms (20.5 with a graph built for it) against 16.0.
constexpr long long BLK_SOLO = 1ll << 16;

// Shared memory, in bytes from a 128-byte boundary. Tile stage: rows
// first-2 .. first+7 of z, h, n and rows first-2 .. first+5 of hmax, so that a
// warp's rows i, i-1, i-2 sit at fixed distances from one address. Rings: two
// buffers per phase value, each of BLK_ROWS + 2 slots; warp w leaves its row
// in slot w + 2 and finds the two rows above in slots w + 1 and w. The last
// two warps write their rows to slots 0 and 1 of the other buffer as well,
// where the next pass looks for them.
constexpr uint32_t BLK_TILE_B = (BLK_ROWS + 2) * BLK_ROW_B;
constexpr uint32_t BLK_Z = 0, BLK_H = BLK_TILE_B, BLK_N = 2 * BLK_TILE_B, BLK_M = 3 * BLK_TILE_B;
constexpr uint32_t BLK_STAGE_B = 3 * BLK_TILE_B + BLK_ROWS * BLK_ROW_B;
constexpr uint32_t BLK_RINGS = BLK_STAGES * BLK_STAGE_B;
constexpr uint32_t BLK_X = 0, BLK_Y = BLK_TILE_B, BLK_S = 2 * BLK_TILE_B, BLK_L = 3 * BLK_TILE_B;
constexpr uint32_t BLK_E = 4 * BLK_TILE_B, BLK_W = 5 * BLK_TILE_B;      // K = 8
template <int K>
__host__ __device__ constexpr uint32_t blk_buf()
{
    return (K == 8 ? 6 : 4) * BLK_TILE_B;
}
template <int K>
__host__ __device__ constexpr uint32_t blk_tail()
{
    return BLK_RINGS + 2 * blk_buf<K>();
}

// Packed per-step constants. Products with a negated constant replace the
// negations of the Newton and Markstein corrections.
struct BlkK {
    f2 dx, nrdx, dd, nrdd, w, A, nA, invA, gK, dt, rain;
    f2 rden, nden;                      // RN(1/(2K dt)), -(2K dt)
    float tau_l, tau_h;
};

// The CTA's current unit, written by its first thread. Here rather than in
// registers: thirty values that every pass carried cost 48 to 104 B of spills.
struct BlkUnit {
    int H, passes;              // rows; passes
    int lo, hi;                 // rows r0 + rel with rel < lo or rel >= hi are special
    int r0, c_first, edges;     // open edges: bit 0 north, 1 south, 2 west, 3 east
    int tx, ty, h_cur;          // column of the tiles; row of the next tiles to load
    unsigned pass;              // passes of the CTA so far: stages and barrier parities
    float hcut;                 // depth below which no cell raises the velocity maximum
};

// After the rings: what every thread of the CTA reads (so that no phase holds
// it in registers) and the CTA's rare sums.
template <typename AccT>
struct BlkTail {
    unsigned long long bar[BLK_STAGES];
    BlkK c;
    StepVals<float> sv;
    BlkUnit un;
    TimePre pre;
    AccT a_clamp, a_bnd, a_rain, a_sea; // clamped volume, open-edge outflow, rain, outflow to SEA
    long long rain_cells;       // LAND output cells (uniform rain)
    double bnd[BLK_ROWS][2];    // outflow of the warps' west and east edge cells
    float qo[2][32];            // open discharge of west and east edge cells, by row
    unsigned cap;               // faces whose volume cap bound
    unsigned vmax;              // bits of the CTA's largest next-step velocity
    int bad;
    int unit[2];                // next unit of the CTA, by unit parity
    int nblk, units;            // units per strip and in all
};
template <int K>
__host__ __device__ constexpr int blk_smem_bytes()
{
    return 128 + (int)blk_tail<K>() + (int)sizeof(BlkTail<double>);
}

__device__ __forceinline__ f2 ld2(const float *p)
{
    const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
    return mk2(v.x, v.y);
}
__device__ __forceinline__ f2 ld2_rw(const float *p)
{
    const float2 v = *reinterpret_cast<const float2 *>(p);
    return mk2(v.x, v.y);
}
__device__ __forceinline__ void st2(float *p, f2 v)
{
    *reinterpret_cast<float2 *>(p) = make_float2(lo2(v), hi2(v));
}
// Shared memory by 32-bit shared address.
__device__ __forceinline__ f2 sld(uint32_t a)
{
    f2 v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v.u) : "r"(a));
    return v;
}
__device__ __forceinline__ float slf(uint32_t a)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ int sli(uint32_t a)
{
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sst(uint32_t a, f2 v)
{
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v.u) : "memory");
}
// Sign changes and magnitudes by halves: packed instructions take the sign
// change as an operand modifier.
__device__ __forceinline__ f2 ng2(f2 a) { return mk2(-lo2(a), -hi2(a)); }
__device__ __forceinline__ f2 ab2(f2 a) { return mk2(fabsf(lo2(a)), fabsf(hi2(a))); }
// magnitude of a with the sign of s, one three-input logic operation a half
__device__ __forceinline__ float csign(float a, float s)
{
    float r;
    asm("lop3.b32 %0, %1, %2, 0x7fffffff, 0xe4;" : "=f"(r) : "f"(a), "f"(s));
    return r;
}
// -(u*u) per half, rounded (scalar products: never contracted into a sum)
__device__ __forceinline__ f2 nsq2(f2 u)
{
    return mk2(__fmul_rn(-lo2(u), lo2(u)), __fmul_rn(-hi2(u), hi2(u)));
}
// RN(a / c) given rc = RN(1/c), nc = -c (Markstein, as div2_mk)
__device__ __forceinline__ f2 div2_c(f2 a, f2 rc, f2 nc)
{
    const f2 q = mul2(a, rc);
    return fma2(fma2(q, nc, a), rc, q);
}

// RN(sqrt(g*hf)) per half of the exact product g*hf (as the reference's
// (real)sqrt((double)g*(double)hf), physics.h:107-108): from p = RN(g*hf),
// its error pe = g*hf - p (exact, one fused multiply-add) and s = RN(sqrt(p)),
// the root of p + pe is s + (p - s^2 + pe)/(2s) to far better than 2^-20 ulp;
// that sum is rounded to y with its error e (Fast2Sum). `unsure` per half:
// |e| within 2^-11 of half an ulp of y (tested as fma(e, 1 + 2^-11, y) != y),
// which also covers the reference's double rounding (its root is rounded to
// double first, which can only matter within 2^-29 ulp of a midpoint). The
// exact value is never a float midpoint: a midpoint has 25 significant bits,
// its square at least 49, and g*hf at most 48.
__device__ __forceinline__ f2 vcrit2(f2 g, f2 hf, bool &unsure0, bool &unsure1)
{
    const f2 p = mul2(g, hf);
    const f2 pe = fma2(g, hf, neg2(p));
    const f2 y0 = rsqrt_2(p);
    const f2 s0 = mul2(p, y0);
    const f2 h = mul2(bc2(0.5f), y0);
    const f2 s = fma2(fma2(neg2(s0), s0, p), h, s0);       // RN(sqrt(p))
    const f2 r = add2(fma2(neg2(s), s, p), pe);              // g*hf - s^2
    const f2 corr = mul2_sep(r, h);
    const f2 y = add2(s, corr);
    const f2 e = add2(sub2(s, y), corr);
    const f2 chk = fma2(e, bc2(1.00048828125f), y);
    float y0f, y1f, k0, k1;
    sp2(y, y0f, y1f);
    sp2(chk, k0, k1);
    unsure0 = k0 != y0f;
    unsure1 = k1 != y1f;
    return y;
}

// The exact next-step velocity of the flagged halves (physics.h:193-217),
// folded into the running maximum vm.
template <int K, int MATH>
__device__ __noinline__ float pair_velocity(float vm, bool x0, bool x1, f2 mo, f2 md, f2 hv, f2 nv,
                                            const StepK<float> *kp)
{
    const StepK<float> k = *kp;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        if (j == 0 ? x0 : x1) {
            float Smax = Mth<float, MATH>::div(get2(mo, j), k.dx);
            if constexpr (K == 8) {
                const float Sd = Mth<float, MATH>::div(get2(md, j), k.d_diag);
                Smax = Sd > Smax ? Sd : Smax;
            }
            const float v = cell_velocity<float, MATH>(get2(hv, j), get2(nv, j), Smax, k);
            vm = v > vm ? v : vm;
        }
    }
    return vm;
}

// hf^(2/3) = RN(cbrt(hf*hf)) per half, without the exactness fix-up: the
// cube root u of hf by one Newton step on a log2/exp2 estimate u0
// (u = u0 - (u0^3 - hf)/(3 u0^2), the residual taken exactly by fused
// multiply-adds), then u^2 as the float pair s_hi + t, t = s_lo - 2 u0 corr,
// rounded to y with its rounding error e (Fast2Sum). The value y + e is
// within about 2^-40 relative of cbrt(hf^2) for hf in [2^-20, 2^20].
// `unsure` is raised when that is not enough to decide the rounding of either
// half: |e| within 2^-11 of half an ulp of y (tested as fma(e, 1 + 2^-11, y)
// != y, which also covers the halved gap below a power of two), or hf outside
// [2^-20, 2^20]; the caller then evaluates the pair exactly (cbrt_sq_rn).
__device__ __forceinline__ f2 cbrt_sq2n(f2 hf, bool &unsure)
{
    const f2 l = lg2_2(hf);
    const f2 u0 = ex2_2(mul2(l, bc2(0.333333343f)));
    const f2 p = nsq2(u0);                                  // -s_hi
    const f2 s_lo = fma2(u0, u0, p);
    const f2 nr = fma2(ng2(s_lo), u0, fma2(p, u0, hf));     // hf - u0^3
    const f2 c2 = mul2(nr, rcp_2(mul2(bc2(1.5f), p)));      // 2 (u0 - u)
    const f2 t = fma2(ng2(u0), c2, s_lo);
    const f2 y = sub2(t, p);
    const f2 e = sub2(t, add2(p, y));
    const f2 chk = fma2(e, bc2(1.00048828125f), y);
    unsure = unsure || lo2(chk) != lo2(y) || hi2(chk) != hi2(y) || !(fabsf(lo2(l)) <= 20.0f) ||
             !(fabsf(hi2(l)) <= 20.0f);
    return y;
}

static __device__ __noinline__ float blk_cbrt(float hf) { return cbrt_sq_rn(hf); }
static __device__ __noinline__ float blk_vcr(float g, float hf) { return sqrt_prod_rn(g, hf); }

// One face pair between evaluation and use. A half that carries no flow
// (|dL| < tau_l or hf < tau_h) continues with dL = 0 and hf = 1: it raises no
// flag, and its volume cap is zero, so its discharge is.
struct BlkFace {
    f2 dL, hf, cb, v, rs;
};

// Faces a -> b between cells of levels La, Lb, elevations za, zb and Manning n
// of sum ns, centre distance d (nrd = -RN(1/d)) (FloodCA
// src/kernels/physics.h:51-125), every operation rounded as the reference's,
// in three steps so that the faces of a row run as one block of independent
// work. blk_face_v: everything up to the factors of the Manning velocity
// v * cb * rs = (1/nf) * hf^(2/3) * sqrt(S); `unsure`: a cube root of the lane
// must be settled by the exact scalar function.
template <int MATH>
__device__ __forceinline__ BlkFace blk_face_v(f2 La, f2 Lb, f2 za, f2 zb, f2 ns, f2 d, f2 nrd,
                                              float tau_l, float tau_h, bool &unsure)
{
    BlkFace f;
    const f2 dL = sub2(La, Lb);
    const f2 hf = sub2(max2(La, Lb), max2(za, zb));
    const bool live0 = fabsf(lo2(dL)) >= tau_l && lo2(hf) >= tau_h;
    const bool live1 = fabsf(hi2(dL)) >= tau_l && hi2(hf) >= tau_h;
    f.dL = sel2(live0, live1, dL, bc2(0.0f));
    f.hf = sel2(live0, live1, hf, bc2(1.0f));
    const f2 nf = max2(mul2(bc2(0.5f), ns), bc2(1e-12f));
    if constexpr (MATH == MATH_EXACT) {
        f.v = rcp_2(nf);
        f.v = fma2(fma2(ng2(nf), f.v, bc2(1.0f)), f.v, f.v);
        const f2 q = mul2(ab2(f.dL), nrd);                      // -RN(|dL| rd)
        const f2 nS = fma2(fma2(q, d, ab2(f.dL)), nrd, q);      // -RN(|dL|/d)
        const f2 y = rsqrt_2(ng2(nS));
        const f2 s = mul2(nS, y);
        f.rs = fma2(ng2(fma2(s, s, nS)), mul2(bc2(0.5f), y), ng2(s));
        f.cb = cbrt_sq2n(f.hf, unsure);
    } else {
        const f2 S = mul2(ab2(f.dL), ng2(nrd));
        f.rs = mul2(S, rsqrt_2(S));
        f.cb = ex2_2(mul2(lg2_2(f.hf), bc2(0.666666687f)));
        f.v = rcp_2(nf);
    }
    return f;
}

// v = (1/nf) cb sqrt(S); `crit`: a half may reach the critical velocity
// sqrt(g hf) (a dead half's v is NaN and raises nothing)
__device__ __forceinline__ void blk_face_m(BlkFace &f, f2 gK, bool &crit)
{
    f.v = mul2(mul2(f.v, f.cb), f.rs);
    const f2 v2 = mul2(f.v, f.v);
    // exact: v^2 < g hf (1 - 1e-6) leaves v surely below the critical velocity
    const f2 pm = mul2(gK, f.hf);
    crit = crit || lo2(v2) >= lo2(pm) || hi2(v2) >= hi2(pm);
}

// v = min(v, RN(sqrt(g hf))) on the halves that may exceed it
template <int MATH>
__device__ __forceinline__ void blk_face_crit(BlkFace &f, f2 gK, float g)
{
    const f2 v2 = mul2(f.v, f.v);
    const f2 pm = mul2(gK, f.hf);
    const bool cr0 = lo2(v2) >= lo2(pm), cr1 = hi2(v2) >= hi2(pm);
    f2 vcr;
    if constexpr (MATH == MATH_EXACT) {
        bool u0, u1;
        vcr = vcrit2(bc2(g), f.hf, u0, u1);
        if (cr0 && u0)
            vcr = mk2(blk_vcr(g, lo2(f.hf)), hi2(vcr));
        if (cr1 && u1)
            vcr = mk2(lo2(vcr), blk_vcr(g, hi2(f.hf)));
    } else {
        const f2 p = mul2(bc2(g), f.hf);
        vcr = mul2(p, rsqrt_2(p));
    }
    f.v = sel2(cr0, cr1, min2(f.v, vcr), f.v);
}

// sign(dL) min(v hf w, RN(RN(|dL| A)/(2K dt))); caps: plus the number of
// halves whose volume cap binds
template <int MATH>
__device__ __forceinline__ f2 blk_face_q(const BlkFace &f, f2 w, f2 A, f2 rden, f2 nden,
                                         unsigned &caps, bool &c0, bool &c1)
{
    const f2 Qm = mul2(mul2(f.v, f.hf), w);
    const f2 num = mul2(ab2(f.dL), A);
    f2 Qc;
    if constexpr (MATH == MATH_EXACT)
        Qc = div2_c(num, rden, nden);
    else
        Qc = mul2(num, rden);
    c0 = lo2(Qc) < lo2(Qm);
    c1 = hi2(Qc) < hi2(Qm);
    if (c0)
        caps += 1u;
    if (c1)
        caps += 1u;
    const f2 Q = min2(Qm, Qc);
    return mk2(csign(lo2(Q), lo2(f.dL)), csign(hi2(Q), hi2(f.dL)));
}

// Discharges of two cells (z, h, n) across an open edge, to the virtual
// neighbour z - S_bnd*dx, h = 0, same n, clipped at zero (FloodCA
// src/common/model.c:166-177); cap: bit per half whose volume cap binds.
// kc, sv: shared addresses of the step's constants. Evaluated on the pair like
// any other face: the scalar formula took half of a 61 x 93 grid's step.
struct OpenPair {
    f2 q;
    unsigned cap;
};
static __device__ __noinline__ OpenPair open_pair(f2 z, f2 h, f2 n, uint32_t kc, uint32_t sv)
{
    const f2 L = add2(z, h);
    const float S = slf(sv + (uint32_t)offsetof(StepVals<float>, k.S_bnd));
    const float dxs = slf(sv + (uint32_t)offsetof(StepVals<float>, k.dx));
    const float g = slf(sv + (uint32_t)offsetof(StepVals<float>, k.g));
    const f2 lv = sub2(z, bc2(__fmul_rn(S, dxs)));
    bool unsure = false, crit = false;
    BlkFace f = blk_face_v<MATH_EXACT>(L, lv, z, lv, add2(n, n), bc2(dxs),
                                       sld(kc + (uint32_t)offsetof(BlkK, nrdx)),
                                       slf(kc + (uint32_t)offsetof(BlkK, tau_l)),
                                       slf(kc + (uint32_t)offsetof(BlkK, tau_h)), unsure);
    if (unsure)
        f.cb = mk2(blk_cbrt(lo2(f.hf)), blk_cbrt(hi2(f.hf)));
    const f2 gK = bc2(g * 0.999999f);
    blk_face_m(f, gK, crit);
    if (crit)
        blk_face_crit<MATH_EXACT>(f, gK, g);
    unsigned caps = 0u;
    OpenPair o;
    bool c0, c1;
    o.q = blk_face_q<MATH_EXACT>(f, sld(kc + (uint32_t)offsetof(BlkK, w)),
                                 sld(kc + (uint32_t)offsetof(BlkK, A)),
                                 sld(kc + (uint32_t)offsetof(BlkK, rden)),
                                 sld(kc + (uint32_t)offsetof(BlkK, nden)), caps, c0, c1);
    o.cap = (c0 ? 1u : 0u) | (c1 ? 2u : 0u);
    o.q = max2(o.q, bc2(0.0f));
    return o;
}

// Open sides of the cells (r, c) and (r, c+1); edges as in BlockSweep::run.
__device__ __forceinline__ void open_sides(int r, int c, int nr, int nc, int r_lo, int r_hi,
                                           int edges, int &k0, int &k1)
{
    const int rows = (r == 0 && (edges & 1)) + (r == nr - 1 && (edges & 2));
    const bool rin = r >= r_lo && r < r_hi;
    k0 = rin && c >= 0 && c < nc ? rows + (c == 0 && (edges & 4)) + (c == nc - 1 && (edges & 8))
                                 : 0;
    k1 = rin && c + 1 >= 0 && c + 1 < nc
             ? rows + (c + 1 == 0 && (edges & 4)) + (c + 1 == nc - 1 && (edges & 8))
             : 0;
}

// Cells that are not LAND (n NaN; a LAND cell may have any finite elevation,
// a raster's -3.4e38 too): elevation and level of SEA cells (z = -PAD_Z) are
// the sea level, the level of WALL cells their elevation PAD_Z.
__device__ __forceinline__ void sea_levels(f2 &z, f2 &L, f2 n, float zs)
{
    const bool o0 = lo2(n) != lo2(n), o1 = hi2(n) != hi2(n);
    z = sel2(o0 && lo2(z) < -1e29f, o1 && hi2(z) < -1e29f, bc2(zs), z);
    L = sel2(o0, o1, z, L);
}
// Sum of two cells' Manning n for their mean; a cell that is not LAND (NaN)
// takes the other's.
__device__ __forceinline__ f2 nsum2(f2 a, f2 b)
{
    const f2 x = sel2(lo2(a) != lo2(a), hi2(a) != hi2(a), b, a);
    return add2(x, sel2(lo2(b) != lo2(b), hi2(b) != hi2(b), x, b));
}

// Q s of the upwind cell (s_down for Q < 0): one of the products is zero.
__device__ __forceinline__ f2 upwind2(f2 Q, f2 s_up, f2 s_down)
{
    const f2 z0 = bc2(0.0f);
    return fma2(min2(Q, z0), s_down, mul2(max2(Q, z0), s_up));
}

// GEN: grids with SEA or WALL cells (with the rain as a field).
template <typename AccT, int K, int MATH, bool RAINF, bool GEN>
struct BlockSweep {
    static_assert(RAINF || !GEN, "masked grids carry the rain as a field");
    using SS = StepSums<float, AccT>;
    using Tail = BlkTail<AccT>;
    static constexpr int NF = K == 8 ? 4 : 2;
    static constexpr uint32_t TAIL = blk_tail<K>();
    static constexpr uint32_t KC = TAIL + (uint32_t)offsetof(Tail, c);
    static constexpr uint32_t SV = TAIL + (uint32_t)offsetof(Tail, sv);
    static constexpr uint32_t UN = TAIL + (uint32_t)offsetof(Tail, un);
#define FCAB_KC(m) sld(sb + KC + (uint32_t)offsetof(BlkK, m))
#define FCAB_SV(m) slf(sb + SV + (uint32_t)offsetof(StepVals<float>, m))
#define FCAB_UN(m) sli(sb + UN + (uint32_t)offsetof(BlkUnit, m))

    // The CTA's memory: shared address (128-byte aligned), and its tail, whose
    // generic address is made where it is used (rare paths).
    struct Cta {
        uint32_t sb;
        __device__ __forceinline__ Tail *tail() const
        {
            uint64_t p;
            asm volatile("{\n\t.reg .u64 t;\n\tcvt.u64.u32 t, %1;\n\t"
                         "cvta.shared.u64 %0, t;\n\t}"
                         : "=l"(p)
                         : "r"(sb + TAIL));
            return reinterpret_cast<Tail *>(p);
        }
    };

    // What a unit reads of a row above its first one, from rings that no
    // phase has written yet, only reaches rows that are dropped: the rings
    // need no clearing.
    static __device__ __forceinline__ void attach(Cta &T, char *sm) { T.sb = smem_addr(sm); }
    // one thread, once per CTA
    static __device__ __forceinline__ void init_barriers(Cta &T)
    {
        for (int q = 0; q < BLK_STAGES; q++)
            mbar_init2(T.sb + TAIL + 8u * q);
        T.tail()->bad = 0;
        T.tail()->un.pass = 0u;
        fence_proxy_async_smem();
    }

    // Once per step (one thread; a barrier follows): constants and sums.
    static __device__ __forceinline__ void begin(Cta &T, const GridD<float> &g,
                                                 const RunK<float> &rk, const Ctl *ctl)
    {
        Tail &t = *T.tail();
        const StepVals<float> sv = step_vals<float, K>(g, rk, ctl);
        const StepK<float> &k = sv.k;
        t.sv = sv;
        t.a_clamp = t.a_bnd = t.a_rain = t.a_sea = 0;
        t.vmax = t.cap = 0u;
        for (int q = 0; q < 2 * BLK_ROWS; q++)
            t.bnd[q >> 1][q & 1] = 0.0;
        t.rain_cells = 0;
        BlkK &c = t.c;
        c.dx = bc2(k.dx);
        c.nrdx = bc2(-k.rdx);
        c.dd = bc2(k.d_diag);
        c.nrdd = bc2(-k.rdd);
        c.w = bc2(k.w);
        c.A = bc2(k.A);
        c.nA = bc2(-k.A);
        c.invA = bc2(k.inv_A);
        c.gK = bc2(k.g * (MATH == MATH_EXACT ? 0.999999f : 1.0f));
        c.dt = bc2(sv.dt);
        c.rain = bc2(sv.rainv);
        c.rden = bc2(k.rden);
        c.nden = bc2(-k.den);
        c.tau_l = k.tau_l;
        c.tau_h = k.tau_h;
    }

    // one thread: the tiles of a pass (from row y0, two above the pass's
    // first) into its stage. The barrier of a stage takes two arrivals, one
    // with the fields that never change (z, n) and one with those that the
    // step before wrote (h, hmax).
    static __device__ __forceinline__ void issue_fixed(uint32_t sb, const CUtensorMap *tm, int tx,
                                                       int y0, unsigned pass)
    {
        const unsigned st = pass % BLK_STAGES;
        const uint32_t bar = sb + TAIL + 8u * st, dst = sb + st * BLK_STAGE_B;
        mbar_arrive_tx(bar, 2 * BLK_TILE_B);
        tma_load_tile(dst + BLK_Z, tm, bar, tx, y0);
        tma_load_tile(dst + BLK_N, tm + 1, bar, tx, y0);
    }
    static __device__ __forceinline__ void issue_state(uint32_t sb, const CUtensorMap *tm,
                                                       const CUtensorMap *th, int tx, int y0,
                                                       unsigned pass)
    {
        const unsigned st = pass % BLK_STAGES;
        const uint32_t bar = sb + TAIL + 8u * st, dst = sb + st * BLK_STAGE_B;
        mbar_arrive_tx(bar, BLK_STAGE_B - 2 * BLK_TILE_B);
        tma_load_tile(dst + BLK_H, th, bar, tx, y0);
        tma_load_tile(dst + BLK_M, tm + 4, bar, tx, y0);
    }
    static __device__ __forceinline__ void issue(uint32_t sb, const CUtensorMap *tm,
                                                 const CUtensorMap *th, int tx, int y0,
                                                 unsigned pass)
    {
        fence_proxy_async_smem();
        issue_fixed(sb, tm, tx, y0, pass);
        issue_state(sb, tm, th, tx, y0, pass);
    }
    // one thread: a unit's descriptor
    static __device__ __forceinline__ void open_unit(const Cta &T, const GridD<float> &g,
                                                     const RunK<float> &rk, int strip, int r0,
                                                     int r1)
    {
        using Gm = Geom<2>;
        BlkUnit &u = T.tail()->un;
        const int c = strip * Gm::OW - Gm::HL;
        u.H = r1 - r0;
        u.passes = (r1 - r0 + 6 + BLK_ROWS - 1) / BLK_ROWS;
        // special rows: r < 1 or r >= nr - 2; in strips with a column outside
        // the grid, column 0 or nc-1, or the inflow cell, all of them
        const bool all = c <= 0 || c + Gm::SW > g.nc - 1 ||
                         (rk.inflow_c >= c && rk.inflow_c < c + Gm::SW);
        u.lo = all ? 0x7fffffff : 1 - r0;
        u.hi = g.nr - 2 - r0;
        u.r0 = r0;
        u.c_first = c;
        u.edges = !rk.open ? 0
                           : (rk.edge_n ? 1 : 0) | (rk.edge_s ? 2 : 0) |
                                 (rk.edge_w && c <= 0 ? 4 : 0) |
                                 (rk.edge_e && c + Gm::SW > g.nc - 1 ? 8 : 0);
        u.tx = c + PADC;            // a multiple of 4 floats
        u.ty = r0 - 5 + PADR;
    }
    // one thread, after open_unit: the tiles of its first passes, the fixed
    // fields, then (h_cur known) the state
    static __device__ __forceinline__ void first_fixed(const Cta &T, const GridD<float> &g)
    {
        const BlkUnit &u = T.tail()->un;
        fence_proxy_async_smem();
        for (int b = 0; b < min(u.passes, BLK_STAGES - 1); b++)
            issue_fixed(T.sb, g.tmap, u.tx, u.ty + b * BLK_ROWS, u.pass + b);
    }
    static __device__ __forceinline__ void first_state(const Cta &T, const GridD<float> &g,
                                                       int h_cur)
    {
        BlkUnit &u = T.tail()->un;
        for (int b = 0; b < min(u.passes, BLK_STAGES - 1); b++)
            issue_state(T.sb, g.tmap, g.tmap + (h_cur ? 3 : 2), u.tx, u.ty + b * BLK_ROWS,
                        u.pass + b);
        u.h_cur = h_cur;
        u.ty += (BLK_STAGES - 1) * BLK_ROWS;
    }
    // one thread, instead of first_state: the fixed tiles land and are dropped
    static __device__ __forceinline__ void first_drop(const Cta &T)
    {
        const BlkUnit &u = T.tail()->un;
        for (int b = 0; b < min(u.passes, BLK_STAGES - 1); b++) {
            mbar_arrive(T.sb + TAIL + 8u * ((u.pass + b) % BLK_STAGES));
            arrived(T, u.pass + b);
        }
    }
    // one thread: waits for the tiles of a pass
    static __device__ __forceinline__ void arrived(const Cta &T, unsigned pass)
    {
        if (!mbar_wait_bounded(T.sb + TAIL + 8u * (pass % BLK_STAGES), (pass / BLK_STAGES) & 1u))
            T.tail()->bad = 1;
    }
    // a row of a phase value: into slot w + 2, and for the last two warps
    // into the other buffer's slot w - 6 (`over`: the distance to it)
    static __device__ __forceinline__ void keep(uint32_t at, f2 v, bool last2, uint32_t over)
    {
        sst(at + 2 * BLK_ROW_B, v);
        if (last2)
            sst(at + over, v);
    }

    // whether all cells of a row have an open edge
    static __device__ __forceinline__ bool open_row(int edges, int r, int nr)
    {
        return (r == 0 && (edges & 1)) || (r == nr - 1 && (edges & 2));
    }
    // The open west (first BLK_ROWS lanes) and east (next) edge cells of the
    // pass's rows, a row per lane: their discharges into Tail::qo by row (modulo 32).
    // One evaluation a pass instead of two per row of an edge strip: with both
    // open, a 2048^2 step took 109 us that way and takes 67 this way (66 closed).
    static __device__ __forceinline__ void open_ends(Tail &tl, uint32_t sb, uint32_t tiles,
                                                     int first, int nr, int nc, int lane)
    {
        const int edges = tl.un.edges, r0 = tl.un.r0, r1 = r0 + tl.un.H;
        const int side = lane / BLK_ROWS & 1, slot = lane % BLK_ROWS, row = r0 + first + slot;
        const int c = (side ? nc - 1 : 0) - tl.un.c_first;
        float z = 0.0f, h = 0.0f, n = 1.0f;
        const bool on = lane < 2 * BLK_ROWS && (edges & (4 << side));
        if (on) {
            const uint32_t a = tiles + (slot + 2) * BLK_ROW_B + 4u * (uint32_t)c;
            z = slf(a + BLK_Z);
            h = slf(a + BLK_H);
            n = slf(a + BLK_N);
        }
        const OpenPair o = open_pair(bc2(z), bc2(h), bc2(n), sb + KC, sb + SV);
        if (on) {
            const bool land = !GEN || n == n;
            tl.qo[side][row & 31] = land ? lo2(o.q) : 0.0f;
            // counted by the strip that writes the column; rows with open
            // cells all along count theirs in phase C
            if (land && (o.cap & 1u) && c < Geom<2>::HL + Geom<2>::OW && row >= r0 && row < r1 &&
                !open_row(edges, row, nr))
                atomicAdd(&tl.cap, 1u);
        }
    }

    // What cells (r, c) and (r, c+1) lose across the open west and east edges,
    // scaled by s, summed over their open sides.
    static __device__ __forceinline__ f2 end_flow(const Tail &tl, int r, int c, int nr, int nc,
                                                  int r_lo, int r_hi, int edges, f2 s)
    {
        int k0, k1;
        open_sides(r, c, nr, nc, r_lo, r_hi, edges & 12, k0, k1);
        const float e = tl.qo[1][r & 31];
        const float q = c == 0 && (edges & 4) ? tl.qo[0][r & 31] : e;   // column 0 is a low half
        return mk2(open_sum<float>(__fmul_rn(q, lo2(s)), k0),
                   open_sum<float>(__fmul_rn(e, hi2(s)), k1));
    }

    // The velocity below which no cell can raise the step's maximum: the CTA's
    // largest so far, or the seed; and the depth below which no cell reaches it
    // (g h <= thr^2 (1 - 1e-6)).
    static __device__ __forceinline__ float threshold(const Tail &t)
    {
        const float vm = __uint_as_float(*(const volatile unsigned *)&t.vmax);
        return vm > t.sv.vseed ? vm : t.sv.vseed;
    }
    static __device__ __forceinline__ float height_cut(const Tail &t, float thr)
    {
        return fmaxf(thr * thr * 0.999998f * __frcp_rn(t.sv.k.g), t.sv.k.tau_h);
    }

    // The CTA's sums and velocity maximum to the control block.
    static __device__ __forceinline__ void publish(Cta &T, const SS &ss, Ctl *ctl, int lane,
                                                   int slot)
    {
        using Gm = Geom<2>;
        Tail &t = *T.tail();
        // halo lanes evaluate faces that other strips own
        const bool out = lane * 2 >= Gm::HL && lane * 2 < Gm::HL + Gm::OW;
        const unsigned cap = __reduce_add_sync(0xffffffffu, out ? ss.capn : 0u);
        if (lane == 0 && cap)
            atomicAdd(&t.cap, cap);
        if constexpr (sizeof(AccT) == 4) {
            const AccT r = warp_sum(ss.a_rain);
            if (lane == 0)
                atomicAdd(&t.a_rain, r);
        } else if constexpr (RAINF) {
            const double r = warp_sum(ss.rain_sum);
            if (lane == 0)
                atomicAdd(&t.a_rain, (double)t.sv.A * r);
        }
        __syncthreads();
        // the sums are read by the host only: warp 1 adds them, so that warp
        // 0's fence does not wait for them
        if (threadIdx.x == 32) {
            AccT rain = t.a_rain;
            if constexpr (sizeof(AccT) == 8 && !RAINF)
                rain = (double)t.rain_cells * ((double)t.sv.A * (double)t.sv.rainv);
            AccT *const acc = sizeof(AccT) == 8 ? (AccT *)&ctl->accd[0][slot]
                                                : (AccT *)&ctl->accf[0][slot];
            if (rain != 0)
                atomicAdd(acc, rain);
            if (t.a_clamp != 0)
                atomicAdd(acc + NSLOT, t.a_clamp);
            if (GEN && t.a_sea != 0)
                atomicAdd(acc + 2 * NSLOT, t.a_sea);
            AccT bnd = t.a_bnd;
            for (int q = 0; q < 2 * BLK_ROWS; q++)
                bnd += (AccT)t.bnd[q >> 1][q & 1];
            if (bnd != 0)
                atomicAdd(acc + 3 * NSLOT, bnd);
            if (t.cap)
                atomicAdd(&ctl->cap[slot], (unsigned long long)t.cap);
        }
        if (threadIdx.x == 0) {
            if (t.sv.want_v && t.vmax)
                atomicMax(&ctl->vmax_bits, (unsigned long long)t.vmax);
            if (t.bad)
                ctl->err = CTL_LOST_TILE;
        }
    }

    // The unit at T.tail()->un, by the whole CTA; its first tiles are on their
    // way. wp: the warp's index, as a warp-uniform value.
    static __device__ __forceinline__ void run(const Cta &T, const GridD<float> &g,
                                               const RunK<float> &rk, int wp, int lane, SS &ss)
    {
        using Gm = Geom<2>;
        const uint32_t sb = T.sb;
        const f2 z0 = bc2(0.0f);
        const bool out_lane = lane * 2 >= Gm::HL && lane * 2 < Gm::HL + Gm::OW;
        const int pitch = (int)g.pitch;
        if (wp == 0 && lane == 0) {
            Tail &tl = *T.tail();
            tl.un.hcut = height_cut(tl, threshold(tl));
            arrived(T, tl.un.pass);
        }
        __syncthreads();

        const bool last2 = wp >= BLK_ROWS - 2;
        const uint32_t sl = sb + lane * 8 + wp * BLK_ROW_B;
        uint32_t rb = sl + BLK_RINGS;                               // this pass's rings
        uint32_t tb = sl + (unsigned)FCAB_UN(pass) % BLK_STAGES * BLK_STAGE_B; // and tiles
        int rel = wp - 5;                   // row i-2 relative to r0
        int off2 = (FCAB_UN(r0) + rel + PADR) * pitch + FCAB_UN(c_first) + lane * 2 + PADC;
        bool prev_cand = false;

        for (int left = FCAB_UN(passes); left > 0; left--) {
            if (wp == 0 && lane == 0 && left > BLK_STAGES - 1) {
                // the stage's rows were last read in the pass before, before its last barrier
                BlkUnit &u = T.tail()->un;
                issue(sb, g.tmap, g.tmap + (u.h_cur ? 3 : 2), u.tx, u.ty,
                      u.pass + BLK_STAGES - 1);
                u.ty += BLK_ROWS;
            }
            // to the other buffer, less the slots of the last two warps
            const uint32_t over = (rb == sl + BLK_RINGS ? blk_buf<K>() : 0u - blk_buf<K>()) -
                                  (BLK_ROWS - 2) * BLK_ROW_B;
            const int H = FCAB_UN(H);
            const bool own2 = (unsigned)rel < (unsigned)H;          // row i-2 is written
            // rows i-1, i-2 on or outside the grid's first and last rows, or a
            // special strip: they run the copy of C and D with the branches
            const bool spec = rel < FCAB_UN(lo) || rel >= FCAB_UN(hi);

            // ---- A: x faces of row i; y (and diagonal) faces of rows i-1, i
            f2 Y1, E1 = z0, W1 = z0;
            {
                f2 z = sld(tb + BLK_Z + 2 * BLK_ROW_B);
                const f2 n = sld(tb + BLK_N + 2 * BLK_ROW_B);
                f2 L = add2(z, sld(tb + BLK_H + 2 * BLK_ROW_B));
                f2 zp = sld(tb + BLK_Z + BLK_ROW_B);
                const f2 npv = sld(tb + BLK_N + BLK_ROW_B);
                f2 Lp = add2(zp, sld(tb + BLK_H + BLK_ROW_B));
                bool odd = false;           // a cell of the two rows is not LAND
                if constexpr (GEN) {
                    odd = lo2(n) != lo2(n) || hi2(n) != hi2(n) || lo2(npv) != lo2(npv) ||
                          hi2(npv) != hi2(npv);
                    odd = __any_sync(0xffffffffu, odd);
                    if (odd) {
                        const float zs = FCAB_SV(k.z_sea);
                        sea_levels(z, L, n, zs);
                        sea_levels(zp, Lp, npv, zs);
                    }
                }
                const f2 zr = right2(z), Lr = right2(L), nrr = right2(n);
                const f2 dx = FCAB_KC(dx), nrdx = FCAB_KC(nrdx);
                const float tau_l = slf(sb + KC + (uint32_t)offsetof(BlkK, tau_l));
                const float tau_h = slf(sb + KC + (uint32_t)offsetof(BlkK, tau_h));
                BlkFace f[NF];
                bool unsure = false, crit = false;
                f2 nx = add2(n, nrr), ny = add2(npv, n);
                if (GEN && odd) {
                    nx = nsum2(n, nrr);
                    ny = nsum2(npv, n);
                }
                f[0] = blk_face_v<MATH>(L, Lr, z, zr, nx, dx, nrdx, tau_l, tau_h, unsure);
                f[1] = blk_face_v<MATH>(Lp, L, zp, z, ny, dx, nrdx, tau_l, tau_h, unsure);
                if constexpr (K == 8) {
                    const f2 zpr = right2(zp), Lpr = right2(Lp), npr = right2(npv);
                    const f2 dd = FCAB_KC(dd), nrdd = FCAB_KC(nrdd);
                    f2 ne = add2(npv, nrr), nw = add2(npr, n);
                    if (GEN && odd) {
                        ne = nsum2(npv, nrr);
                        nw = nsum2(npr, n);
                    }
                    f[2] = blk_face_v<MATH>(Lp, Lr, zp, zr, ne, dd, nrdd, tau_l, tau_h, unsure);
                    f[3] = blk_face_v<MATH>(Lpr, L, zpr, z, nw, dd, nrdd, tau_l, tau_h, unsure);
                }
                if constexpr (MATH == MATH_EXACT) {
                    if (__any_sync(0xffffffffu, unsure)) {
                        if (unsure) {
#pragma unroll
                            for (int q = 0; q < NF; q++)
                                f[q].cb = mk2(blk_cbrt(lo2(f[q].hf)), blk_cbrt(hi2(f[q].hf)));
                        }
                    }
                }
                const f2 gK = FCAB_KC(gK);
#pragma unroll
                for (int q = 0; q < NF; q++)
                    blk_face_m(f[q], gK, crit);
                if (__any_sync(0xffffffffu, crit)) {
                    const float gr = FCAB_SV(k.g);
#pragma unroll
                    for (int q = 0; q < NF; q++)
                        blk_face_crit<MATH>(f[q], gK, gr);
                }
                // volume caps are counted by the cell that holds the face: x
                // faces by row i, the others by row i-1
                unsigned cx = 0u, cy = 0u;
                bool c0, c1;
                const f2 w = FCAB_KC(w), A = FCAB_KC(A), rden = FCAB_KC(rden), nden = FCAB_KC(nden);
                const f2 X = blk_face_q<MATH>(f[0], w, A, rden, nden, cx, c0, c1);
                Y1 = blk_face_q<MATH>(f[1], w, A, rden, nden, cy, c0, c1);
                keep(rb + BLK_X, X, last2, over);
                keep(rb + BLK_Y, Y1, last2, over);
                if constexpr (K == 8) {
                    E1 = blk_face_q<MATH>(f[2], w, A, rden, nden, cy, c0, c1);
                    W1 = blk_face_q<MATH>(f[3], w, A, rden, nden, cy, c0, c1);
                    keep(rb + BLK_E, E1, last2, over);
                    keep(rb + BLK_W, W1, last2, over);
                }
                if (wp == BLK_ROWS - 1 && (FCAB_UN(edges) & 12))
                    open_ends(*T.tail(), sb, tb - lane * 8 - wp * BLK_ROW_B, rel + 2 - wp, g.nr,
                              g.nc, lane);
                if ((unsigned)(rel + 2) < (unsigned)H)
                    ss.capn += cx;
                if ((unsigned)(rel + 1) < (unsigned)H)
                    ss.capn += cy;
            }
            __syncthreads();

            // ---- C: outflow volume and limiter of row i-1 (model.c:180-238,
            //      489-502), in the reference order +x, -x, +y, -y, d1+, d1-,
            //      d2+, d2-, open slots
            f2 Y2, S1 = bc2(1.0f), E2 = z0, W2 = z0;
            auto phase_c = [&](auto special_tag) {
                constexpr bool special = decltype(special_tag)::value;
                const int r = special ? FCAB_UN(r0) + rel : 0;
                const int edges = special ? FCAB_UN(edges) : 0;
                const int cbase = special ? FCAB_UN(c_first) + lane * 2 : 0;
                const int nr = g.nr, nc = g.nc;
                const f2 X1 = sld(rb + BLK_X + BLK_ROW_B);
                Y2 = sld(rb + BLK_Y + BLK_ROW_B);
                f2 out = sub2(max2(X1, z0), min2(left2(X1), z0));
                out = add2(out, max2(Y1, z0));
                out = sub2(out, min2(Y2, z0));
                if constexpr (K == 8) {
                    E2 = sld(rb + BLK_E + BLK_ROW_B);
                    W2 = sld(rb + BLK_W + BLK_ROW_B);
                    out = add2(out, max2(E1, z0));
                    out = sub2(out, min2(left2(E2), z0));
                    out = add2(out, max2(left2(W1), z0));
                    out = sub2(out, min2(W2, z0));
                }
                const f2 hp = sld(tb + BLK_H + BLK_ROW_B);
                if (special && open_row(edges, r + 1, nr)) {
                    const OpenPair o = open_pair(sld(tb + BLK_Z + BLK_ROW_B), hp,
                                                 sld(tb + BLK_N + BLK_ROW_B), sb + KC, sb + SV);
                    int k0, k1;
                    open_sides(r + 1, cbase, nr, nc, g.r_lo, g.r_hi, edges, k0, k1);
                    if constexpr (GEN) {        // LAND cells only
                        const f2 n = sld(tb + BLK_ROW_B + BLK_N);
                        k0 = lo2(n) == lo2(n) ? k0 : 0;
                        k1 = hi2(n) == hi2(n) ? k1 : 0;
                    }
                    if ((unsigned)(rel + 1) < (unsigned)H)
                        ss.capn += (o.cap & 1u ? k0 : 0) + (o.cap & 2u ? k1 : 0);
                    out = add2(out, mk2(open_sum<float>(lo2(o.q), k0),
                                        open_sum<float>(hi2(o.q), k1)));
                } else if (special && (edges & 12)) {
                    out = add2(out, end_flow(*T.tail(), r + 1, cbase, nr, nc, g.r_lo, g.r_hi, edges,
                                             bc2(1.0f)));
                }
                const f2 ov = mul2(out, FCAB_KC(dt));
                const f2 hold = mul2(hp, FCAB_KC(A));
                const f2 hz = max2(hold, z0);
                const bool l0 = lo2(ov) > lo2(hz), l1 = hi2(ov) > hi2(hz);
                if (__any_sync(0xffffffffu, l0 || l1)) {
                    const f2 o = sel2(l0, l1, ov, bc2(1.0f));
                    f2 q;
                    if constexpr (MATH == MATH_EXACT)
                        q = div2_mk(hold, o, rcp2_nr(o));
                    else
                        q = mul2(hold, rcp_2(o));
                    S1 = sel2(l0, l1, q, S1);
                }
                keep(rb + BLK_S, S1, last2, over);
            };
            if (spec)
                phase_c(std::true_type{});
            else
                phase_c(std::false_type{});
            __syncthreads();

            // ---- D: net inflow of row i-2 from the upwind-scaled
            //      discharges, depth update, clamp, inflow, hmax and tmax
            //      (model.c:511-597)
            bool cand = false;
            auto phase_d = [&](auto special_tag) {
                constexpr bool special = decltype(special_tag)::value;
                const int r = special ? FCAB_UN(r0) + rel : 0;
                const int edges = special ? FCAB_UN(edges) : 0;
                const int nr = g.nr, nc = g.nc;
                auto column = [&]() { return FCAB_UN(c_first) + lane * 2; };
                const f2 S2 = sld(rb + BLK_S + BLK_ROW_B), S3 = sld(rb + BLK_S);
                // the limiter binds in few rows (it is 1 in the others, and the
                // discharges their own products with it): measured 1 to 3 % of a step
                f2 sr = S2, Qr = sld(rb + BLK_X), Ql, Qd = Y2, Qu = sld(rb + BLK_Y);
                const bool lim = fminf(fminf(lo2(S1), lo2(S2)), lo2(S3)) < 1.0f ||
                                 fminf(fminf(hi2(S1), hi2(S2)), hi2(S3)) < 1.0f;
                if (K == 8 || __any_sync(0xffffffffu, lim)) {
                    sr = right2(S2);
                    Qr = upwind2(Qr, S2, sr);
                    Qd = upwind2(Y2, S2, S1);
                    Qu = upwind2(Qu, S3, S2);
                }
                Ql = left2(Qr);
                f2 net = sub2(Ql, Qr);
                net = sub2(net, Qd);
                net = add2(net, Qu);
                f2 Qrd = z0, Qlu = z0, Qld = z0, Qru = z0;
                if constexpr (K == 8) {
                    Qrd = upwind2(E2, S2, right2(S1));
                    Qlu = left2(upwind2(sld(rb + BLK_E), S3, sr));
                    Qld = left2(upwind2(W2, sr, S1));
                    Qru = upwind2(sld(rb + BLK_W), right2(S3), S2);
                    net = sub2(net, Qrd);
                    net = add2(net, Qlu);
                    net = sub2(net, Qld);
                    net = add2(net, Qru);
                }
                bool l0 = true, l1 = true, odd = false;     // LAND cells; a row with others
                if constexpr (GEN) {
                    const f2 n = sld(tb + BLK_N);
                    l0 = lo2(n) == lo2(n);
                    l1 = hi2(n) == hi2(n);
                    odd = __any_sync(0xffffffffu, !l0 || !l1);
                    if (odd) {
                        // what SEA cells receive has left the domain (model.c:241-319,
                        // there counted by the LAND cell of the face)
                        const f2 z = sld(tb + BLK_Z);
                        const int cbase = column();
                        const bool own = own2 && out_lane;
                        const bool sea0 = own && !l0 && lo2(z) < -1e29f && cbase >= 0 &&
                                          cbase < nc;
                        const bool sea1 = own && !l1 && hi2(z) < -1e29f && cbase + 1 >= 0 &&
                                          cbase + 1 < nc;
                        AccT sea = 0;
                        const float dt = FCAB_SV(dt);
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            if (j == 0 ? sea0 : sea1) {
                                sea += acc_mul<AccT, float>(dt, -get2(Qr, j)) +
                                       acc_mul<AccT, float>(dt, get2(Ql, j)) +
                                       acc_mul<AccT, float>(dt, -get2(Qd, j)) +
                                       acc_mul<AccT, float>(dt, get2(Qu, j));
                                if constexpr (K == 8)
                                    sea += acc_mul<AccT, float>(dt, -get2(Qrd, j)) +
                                           acc_mul<AccT, float>(dt, get2(Qlu, j)) +
                                           acc_mul<AccT, float>(dt, -get2(Qld, j)) +
                                           acc_mul<AccT, float>(dt, get2(Qru, j));
                            }
                        }
                        if (__any_sync(0xffffffffu, sea != 0)) {
                            sea = warp_sum(sea);
                            if (lane == 0)
                                atomicAdd(&T.tail()->a_sea, sea);
                        }
                    }
                }
                const f2 h = sld(tb + BLK_H);
                if (special && open_row(edges, r, nr)) {
                    // open-edge outflow scaled by the cell's own limiter
                    // (model.c:553-559), summed over its open slots
                    const OpenPair o = open_pair(sld(tb + BLK_Z), h, sld(tb + BLK_N), sb + KC,
                                                 sb + SV);
                    int k0, k1;
                    const int cbase = column();
                    open_sides(r, cbase, nr, nc, g.r_lo, g.r_hi, edges, k0, k1);
                    if constexpr (GEN) {        // LAND cells only
                        const f2 n = sld(tb + BLK_N);
                        k0 = lo2(n) == lo2(n) ? k0 : 0;
                        k1 = hi2(n) == hi2(n) ? k1 : 0;
                    }
                    const f2 qs = mul2_sep(o.q, S2);
                    const float q0 = open_sum<float>(lo2(qs), k0);
                    const float q1 = open_sum<float>(hi2(qs), k1);
                    net = sub2(net, mk2(q0, q1));
                    const float dt = FCAB_SV(dt);
                    AccT bnd = 0;
                    if (own2 && out_lane)
                        bnd = acc_mul<AccT, float>(dt, q0) + acc_mul<AccT, float>(dt, q1);
                    bnd = warp_sum(bnd);
                    if (lane == 0 && bnd != 0)
                        atomicAdd(&T.tail()->a_bnd, bnd);
                } else if (special && (edges & 12)) {
                    const int cbase = column();
                    const f2 qs = end_flow(*T.tail(), r, cbase, nr, nc, g.r_lo, g.r_hi, edges, S2);
                    net = sub2(net, qs);
                    // at most one lane each holds column 0 and column nc-1
                    if (own2 && out_lane && (lo2(qs) != 0.0f || hi2(qs) != 0.0f)) {
                        const float dt = FCAB_SV(dt);
                        T.tail()->bnd[wp][cbase == 0 ? 0 : 1] +=
                            (double)(acc_mul<AccT, float>(dt, lo2(qs)) +
                                     acc_mul<AccT, float>(dt, hi2(qs)));
                    }
                }
                f2 rain;
                if constexpr (RAINF) {
                    // rows r0-1 and r1 too: stage E reads their new levels
                    rain = (unsigned)(rel + 1) <= (unsigned)(H + 1) ? ld2(g.cr + off2) : z0;
                    rain = mul2_sep(rain, bc2(FCAB_SV(F)));
                } else {
                    rain = FCAB_KC(rain);
                }
                f2 dq;
                if constexpr (MATH == MATH_EXACT)
                    dq = div2_c(net, FCAB_KC(invA), FCAB_KC(nA));
                else
                    dq = mul2(net, FCAB_KC(invA));
                f2 hu = add2(h, add2(mul2_sep(FCAB_KC(dt), dq), rain));
                if (GEN && odd)
                    hu = sel2(l0, l1, hu, z0);
                if (__any_sync(0xffffffffu, lo2(hu) < 0.0f || hi2(hu) < 0.0f)) {
                    float a0 = lo2(hu), a1 = hi2(hu);
                    const bool own = own2 && out_lane;
                    const int cbase = column();
                    const float A = FCAB_SV(A);
                    if (a0 < 0.0f) {
                        if (own && l0 && cbase >= 0 && cbase < nc)
                            atomicAdd(&T.tail()->a_clamp, acc_mul<AccT, float>(-a0, A));
                        a0 = 0.0f;
                    }
                    if (a1 < 0.0f) {
                        if (own && l1 && cbase + 1 >= 0 && cbase + 1 < nc)
                            atomicAdd(&T.tail()->a_clamp, acc_mul<AccT, float>(-a1, A));
                        a1 = 0.0f;
                    }
                    hu = mk2(a0, a1);
                }
                const f2 z = sld(tb + BLK_Z);
                f2 Ln = add2(z, hu);
                if (special) {
                    const bool rin = r >= g.r_lo && r < g.r_hi;
                    const int cbase = column();
                    const bool in0 = rin && cbase >= 0 && cbase < nc;
                    const bool in1 = rin && cbase + 1 >= 0 && cbase + 1 < nc;
                    if (r == rk.inflow_r) {
                        const int d = rk.inflow_c - cbase;
                        const float dh = FCAB_SV(inflow_dh);
                        if (d == 0)
                            hu = mk2(lo2(hu) + dh, hi2(hu));
                        else if (d == 1)
                            hu = mk2(lo2(hu), hi2(hu) + dh);
                        Ln = add2(z, hu);
                    }
                    // cells outside the grid: no level for stage E, no rain,
                    // and they keep their padding depth of zero
                    Ln = sel2(in0, in1, Ln, bc2(__int_as_float(0x7fc00000)));
                    hu = sel2(in0, in1, hu, h);
                    rain = sel2(in0, in1, rain, z0);
                }
                if (GEN && odd) {
                    const float zs = FCAB_SV(k.z_sea), nan = __int_as_float(0x7fc00000);
                    Ln = sel2(l0, l1, Ln, mk2(lo2(z) < -1e29f ? zs : nan,
                                              hi2(z) < -1e29f ? zs : nan));
                    hu = sel2(l0, l1, hu, h);
                }
                keep(rb + BLK_L, Ln, last2, over);
                if (own2 && out_lane) {
                    if constexpr (sizeof(AccT) == 4) {
                        const float A = FCAB_SV(A);
                        ss.a_rain += A * lo2(rain) + A * hi2(rain);
                    } else if constexpr (RAINF) {
                        ss.rain_sum += (double)lo2(rain) + (double)hi2(rain);
                    }
                    // a cell that could raise the velocity maximum
                    const float hcut = __int_as_float(FCAB_UN(hcut));
                    cand = (l0 && lo2(hu) >= hcut) || (l1 && hi2(hu) >= hcut);
                    const f2 hm = sld(tb + BLK_M);                  // hmax of row i-2
                    const uint64_t ho = sld(sb + SV + (uint32_t)offsetof(StepVals<float>, hout)).u;
                    st2(reinterpret_cast<float *>(ho) + off2, hu);
                    f2 hx = max2(hu, hm);
                    if (GEN && odd)
                        hx = sel2(l0, l1, hx, hm);
                    st2(g.hmax + off2, hx);
                    float *const tmx = g.tmax + off2;
                    const float tv = FCAB_SV(tmax_val);
                    if (l0 && lo2(hu) > lo2(hm))
                        tmx[0] = tv;
                    if (l1 && hi2(hu) > hi2(hm))
                        tmx[1] = tv;
                }
            };
            if (spec)
                phase_d(std::true_type{});
            else
                phase_d(std::false_type{});
            if (wp == 0 && lane == 0) {
                BlkUnit &u = T.tail()->un;
                u.pass += 1;
                if (left > 1)
                    arrived(T, u.pass);
            }
            const bool any_cand = __syncthreads_or(cand) != 0;

            // ---- E: next step's stable velocity of row i-3 from the new
            //      levels of rows i-4..i-2 (physics.h:158-217). A candidate
            //      of this pass sits in rows i-3 of this pass or, for the
            //      last warp's row, of the next one.
            if (any_cand || prev_cand) {
                Tail &tl = *T.tail();
                const float thr = threshold(tl), hcut = height_cut(tl, thr);
                const int r = tl.un.r0 + rel, cbase = tl.un.c_first + lane * 2;
                if (tl.sv.want_v && (unsigned)(rel - 1) < (unsigned)H)
                    velocity_row(tl, g, sld(rb + BLK_L + BLK_ROW_B),
                                 sld(rb + BLK_L + 2 * BLK_ROW_B), sld(rb + BLK_L), r - 1, cbase,
                                 tl.un.edges, out_lane && cbase >= 0 && cbase < g.nc,
                                 out_lane && cbase + 1 >= 0 && cbase + 1 < g.nc, off2 - pitch,
                                 thr, hcut);
                if (wp == 0 && lane == 0)
                    tl.un.hcut = hcut;      // read in D, after two barriers
            }
            prev_cand = any_cand;

            rb = 2 * (sl + BLK_RINGS) + blk_buf<K>() - rb;
            tb = tb == sl + (BLK_STAGES - 1) * BLK_STAGE_B ? sl : tb + BLK_STAGE_B;
            rel += BLK_ROWS;
            off2 += BLK_ROWS * pitch;
        }
        // uniform rain on LAND output cells
        if constexpr (sizeof(AccT) == 8 && !RAINF) {
            if (wp == 0 && lane == 0) {
                Tail &tl = *T.tail();
                const int c0 = tl.un.c_first + Gm::HL;
                tl.rain_cells += (long long)tl.un.H * (min(g.nc, c0 + Gm::OW) - c0);
            }
        }
    }

    // Stage E of one row: candidates are the output cells whose new depth
    // reaches hcut; a multiply-only bound v^6 <= h^4 S^3 / n^6 against thr^6
    // goes first, the exact velocity only where it could exceed thr.
    static __device__ __forceinline__ void velocity_row(Tail &tl, const GridD<float> &g, f2 la,
                                                        f2 lb, f2 lt, int r, int cbase, int edges,
                                                        bool in0, bool in1, int off, float thr,
                                                        float hcut)
    {
        const StepVals<float> &sv = tl.sv;
        const f2 z0 = bc2(0.0f);
        f2 mo = max2(abs2(sub2(la, right2(la))), abs2(sub2(la, left2(la))));
        mo = max2(mo, max2(abs2(sub2(la, lb)), abs2(sub2(la, lt))));
        mo = max2(mo, z0);
        f2 md = z0;
        if constexpr (K == 8) {
            md = max2(abs2(sub2(la, right2(lb))), abs2(sub2(la, left2(lb))));
            md = max2(md, max2(abs2(sub2(la, right2(lt))), abs2(sub2(la, left2(lt)))));
            md = max2(md, z0);
        }
        // a candidate's new depth was stored by this CTA before the last barrier
        const f2 hv = in0 || in1 ? ld2_rw(sv.hout + off) : z0;
        bool e0 = in0 && lo2(hv) >= hcut, e1 = in1 && hi2(hv) >= hcut;
        if (!(e0 || e1))
            return;
        const f2 nv = ld2(g.n + off);
        if constexpr (GEN) {
            e0 = e0 && lo2(nv) == lo2(nv);
            e1 = e1 && hi2(nv) == hi2(nv);
        }
        if ((edges & 12) || open_row(edges, r, g.nr)) {
            // the open virtual neighbour z - S_bnd*dx, h = 0 (physics.h:183-189)
            const bool erow = (r == 0 && (edges & 1)) || (r == g.nr - 1 && (edges & 2));
            const f2 zz = ld2(g.z + off);
            const f2 dv = abs2(sub2(la, sub2(zz, bc2(sv.k.S_bnd * sv.k.dx))));
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int cc = cbase + j;
                if (erow || (cc == 0 && (edges & 4)) || (cc == g.nc - 1 && (edges & 8)))
                    put2(mo, j, fmaxf(get2(mo, j), get2(dv, j)));
            }
        }
        const f2 n2 = mul2(nv, nv);
        f2 S = mul2(mo, bc2(sv.k.rdx));
        if constexpr (K == 8)
            S = max2(S, mul2(md, bc2(sv.k.rdd)));
        const f2 h2 = mul2(hv, hv);
        const f2 lhs = mul2(mul2(h2, h2), mul2(mul2(S, S), S));
        const float t2 = thr * thr;
        // 0 when thr < 1e-6: every velocity is at least 1e-6 (physics.h:214-216)
        const float T6 = thr >= 1e-6f ? t2 * t2 * t2 * 0.9998f : 0.0f;
        const f2 rhs = mul2(mul2(mul2(n2, n2), n2), bc2(T6));
        const bool x0 = e0 && (lo2(lhs) >= lo2(rhs) || lo2(lhs) < 1e-30f);
        const bool x1 = e1 && (hi2(lhs) >= hi2(rhs) || hi2(lhs) < 1e-30f);
        if (x0 || x1) {
            const float vm = pair_velocity<K, MATH>(0.0f, x0, x1, mo, md, hv, nv, &sv.k);
            atomicMax(&tl.vmax, __float_as_uint(vm));
        }
    }
#undef FCAB_KC
#undef FCAB_SV
#undef FCAB_UN
};

}  // namespace fcab
