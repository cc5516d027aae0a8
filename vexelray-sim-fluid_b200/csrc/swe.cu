// swe.cu -- the shallow-water step (ShallowWater.java) on TMA-staged shared-memory halo tiles,
// and the vf_swe_* C-ABI: PatchSimulation (vexelray-sim-fluid-gui/.../gui/PatchSimulation.java).
// Reference paths: vexelray-sim-fluid-core/src/main/java/dev/vexelray/sim/fluid/stencil/.
//
// Built with --fmad=false and IEEE division and square root: every operation rounds as the reference's strict f32 (Java)
// arithmetic does, so a step's output is bit-identical to the reference's CPU semantics (and to the oracle), and so are
// the tick counts it derives.
//
// A second arithmetic, the fast mode (vf_swe_set_exact(h, 0)), keeps the flux form but rounds differently: fused
// multiply-adds (written out as fmaf, since the file forbids contraction), one approximate reciprocal of a cell's depth
// shared by its two velocities, one approximate reciprocal of each face's wave span shared by its three fluxes, and an
// approximate square root for the wave speed. It is within a stated tolerance of the reference rather than equal to it,
// and the water still moves only between neighbours. The tick count from the previous step's speed stays IEEE.
//
// One kernel, k_swe_strip, runs both: a CTA's tile and its halo land in shared memory by TMA, and every lane walks two
// columns up the tile in registers, each face's flux computed once (the reference computes it twice, once from each side,
// with identical inputs and so identical bits).
//
// What bounds a step is its instructions, not the 24 bytes a cell: some 160 a cell exact and 120 fast, at 15 warps an SM,
// which leave the schedulers 58 and 61% busy with fixed latencies and (exact) instruction fetches between. Exact they hold three
// quotients a face and two a cell, and a square root, each correctly rounded. They cost little here because they are shared and branch-free: the quotients over one
// denominator take one reciprocal, refined once, and a multiply and two fused operations each (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), two faces at a time in paired
// fp32; the square root is a reciprocal root and three fused operations by the same paper. For operands inside the ranges
// tested below this is the IEEE result to the bit: on this GPU the quotient was checked against exact residuals for all
// 2^46 pairs of significands and the root for all 2^24, with no mismatch, and scaling by powers of two changes no step.
// Operands outside the ranges (wave fronts' vanishing tails, overflow) take the IEEE operations.
// The staged form that this replaces (primitives and fluxes in shared memory between block barriers, a division at a
// time) took 0.301 ms a step at 4096^2 and 10.6 us on a 201 x 117 patch; this takes 0.143 ms and 5.0 us. The fast mode, one
// column a lane, took 0.123 ms at 4096^2 and takes 0.103, 60% of the measured copy rate.
#include <cuda.h>

#include <cmath>
#include <vector>

#include "profiler.cuh"
#include "snapshot.cuh"
#include "sort.cuh"

using namespace vf;

namespace {

struct SweArgs {
    const float* in[3];
    float* out[3];
    const float* params;                        // [g, courant, dx, dy, dry] (ShallowWater.java:120)
    const int* speed_in;
    int* speed_out;
    int* speed_clear;
    const int* budget_in;
    int* budget_out;
    int* clamped;
    uint32_t* status;
    int nx, ny;
    int edge[4];                                // west, east, south, north: VF_EDGE_*
    int use_tma;
    float nzero;                                // -0: the addend of a product that must not be fused into a sum (mulz2)
};

struct Face {
    float mass, normal, tangent;
};

__device__ __forceinline__ float velocity(float h, float q, float dry) { return h > dry ? q / h : 0.0f; }

__device__ __forceinline__ bool poll_barrier(uint32_t addr, int phase, int limit) {
    for (int it = 0; it < limit; it++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Bounded wait on an mbarrier phase. On giving up it sets the status bit, then waits once more,
// again bounded, so copies still in flight land before the CTA leaves; returns false.
__device__ __forceinline__ bool wait_barrier(unsigned long long* bar, int phase, uint32_t* status) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(bar);
    if (poll_barrier(addr, phase, 1 << 22)) return true;
    set_status(status, ST_TIMEOUT);
    poll_barrier(addr, phase, 1 << 22);
    return false;
}

// ------------------------------------------------------------------ paired and shared arithmetic

__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ float2 min2(float2 a, float2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ float2 max2(float2 a, float2 b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }

// a * b rounded on its own: a fused operation whose addend, -0, comes from memory (nz = -0 twice). A paired product written
// as one is fused into a sum that reads it, even where nvcc is told to contract nothing, and the reference rounds it first.
__device__ __forceinline__ float2 mulz2(float2 a, float2 b, float2 nz) { return __ffma2_rn(a, b, nz); }
// a - b: one fused operation, the same rounding and the same zeros.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.0f, -1.0f), a); }

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The larger, or NaN where either is (fmaxf gives the other one).
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The negated reciprocals of b, refined (the correctly rounded ones, for b in range).
__device__ __forceinline__ float2 neg_recip2(float2 b) {
    const float2 y = f2(rcp_approx(-b.x), rcp_approx(-b.y));
    return __ffma2_rn(y, __ffma2_rn(b, y, f2(1.0f, 1.0f)), y);
}

// -(a / b) correctly rounded, y = neg_recip2(b): the quotient and one exact residual's correction. With the signs this way
// a zero numerator gives the zero that the division gives.
__device__ __forceinline__ float2 neg_quot2(float2 a, float2 b, float2 y) {
    const float2 q = __fmul2_rn(a, y);
    return __ffma2_rn(__ffma2_rn(b, q, a), y, q);
}

// Where that holds: a numerator zero or at least 2^-100 (its residual is then exact and its quotient normal), quotients and
// reciprocals far from overflow. `low` of a zero is past every other's, so one minimum tests both.
__device__ __forceinline__ unsigned low_of(float a) { return 2u * __float_as_uint(a) - 1u; }
constexpr unsigned LOW_MIN = 2u * (27u << 23) - 1u;      // low_of(2^-100)
constexpr float A_MAX = 0x1p64f, B_MIN = 0x1p-24f, B_MAX = 0x1p22f;
constexpr float A_MAX_DRY = 0x1p26f, B_MIN_DRY = 0x1p-100f;   // a face between dry cells: span 1e-30

// The fast mode's square root (approximate, zero at zero); below the normal range, whose root is 2^-63, `least`.
__device__ __forceinline__ float sqrt_fast(float x, float least = 0.0f) { return x >= 0x1p-126f ? x * rsqrt_approx(x) : least; }

// The IEEE operations, out of line: few cells need them.
__device__ __noinline__ float div_ieee(float a, float b) { return a / b; }
__device__ __noinline__ float sqrt_ieee(float a) { return sqrtf(a); }

// -(a / b) for a numerator below those bounds: scaled up by 2^64, which is exact, and the quotient q scaled back, which
// rounds it again where the result is subnormal. That second rounding is wrong only where q lies halfway between two
// subnormals and the true quotient on the side it was not rounded to; the residual tells. (A wave's front runs ahead of it
// through every power of two down to the smallest, a cell or so each, so these are common in water that starts at rest.)
__device__ __forceinline__ float2 neg_quot2_small(float2 a, float2 b, float2 y) {
    const float2 up = f2(0x1p64f, 0x1p64f), down = f2(0x1p-64f, 0x1p-64f);
    const float2 as = __fmul2_rn(a, up), q = neg_quot2(as, b, y);
    const float2 left = __ffma2_rn(b, q, as);            // -(a/b) is q - left/b
    const float2 r = __fmul2_rn(q, down), d = sub2(q, __fmul2_rn(r, up));
    const float2 other = __fmul2_rn(__fadd2_rn(q, d), down);
    constexpr float HALF = 0x1p-86f;                     // half the subnormals' spacing, scaled
    auto pick = [&](float d1, float left1, float r1, float other1) {   // d1 and left1 of opposite signs
        const bool past = left1 != 0.0f && (__float_as_int(left1) ^ __float_as_int(d1)) < 0;
        return fabsf(d1) == HALF && past ? other1 : r1;
    };
    return f2(pick(d.x, left.x, r.x, other.x), pick(d.y, left.y, r.y, other.y));
}
constexpr float A_MAX_SMALL = 0x1p40f;

// ------------------------------------------------------------------ cells and faces

// Cells of ordinary depth and speed, which is nearly all of them in nearly all scenes: wet, a depth in [2^-20, 2^20], speeds
// under 2^20, g within reason. Between such cells a face needs no tests but one. With c >= 2^-16 and span = hi - lo >= 2c:
//   normal: its numerator is A + B, A = hi fL - lo fR >= span/2 g h^2/2 >= 2^-68; where B cancels it, B is as large as A
//     and both are multiples of 2^-92, so the numerator is zero or far above 2^-100;
//   mass: a numerator under 2^-100 may give a quotient an ulp off, which under a depth of 2^-20 or more is lost: beside a
//     second face of 2^-44 or more its difference is already rounded away, and below that the depth keeps its value;
//   tangent: tested.
// Everything stays under 2^84. A warp takes the short way when all its cells of the two rows are ordinary.
struct Ordinary {
    unsigned base, range;   // float bits: the least ordinary depth, and the span of bits to 2^20
    bool g;
};

__device__ __forceinline__ Ordinary ordinary_depths(float g, float dry) {
    const float least = fmaxf(0x1p-20f, dry > 0.0f ? __uint_as_float(__float_as_uint(dry) + 1u) : 0.0f);
    Ordinary o;
    o.base = __float_as_uint(least);
    o.g = least <= 0x1p20f && g >= 0x1p-12f && g <= 0x1p20f;
    o.range = o.g ? __float_as_uint(0x1p20f) - o.base : 0u;
    return o;
}

// Two neighbouring cells of a row: depths and momenta, velocities and (negated) wave speeds, and their own terms of the
// fluxes across their sides: along x fx = hu u + g h^2 / 2 and tx = hu v, along y fy = hv v + g h^2 / 2 and ty = hv u.
struct Cells {
    float2 h, qx, qy, u, v, nc, fx, fy, tx, ty;
};

// One velocity outside neg_quot2's ranges, or of a dry cell.
__device__ __forceinline__ float velocity_any(float h, float q, float small, float dry) {
    if (!(h > dry)) return 0.0f;
    return h >= B_MIN && h <= B_MAX && fabsf(q) < A_MAX_SMALL ? -small : div_ieee(q, h);
}

// `fine` comes back false where a cell is not ordinary.
template <bool EXACT>
__device__ __forceinline__ Cells cells_of(float2 h, float2 qx, float2 qy, float g, const Ordinary& ord, float dry, float2 nz,
                                          bool& fine) {
    Cells q;
    q.h = h;
    q.qx = qx;
    q.qy = qy;
    const float2 mone = f2(-1.0f, -1.0f), hg = f2(0.5f * g, 0.5f * g);
    const float2 p = mulz2(hg, __fmul2_rn(h, h), nz);
    fine = max(__float_as_uint(h.x) - ord.base, __float_as_uint(h.y) - ord.base) <= ord.range;
    if (EXACT) {
        const float2 y = neg_recip2(h);
        const float2 nx = __fmul2_rn(h, f2(-g, -g));
        const float2 z = f2(rsqrt_approx(-nx.x), rsqrt_approx(-nx.y)), ns = __fmul2_rn(nx, z);
        q.u = __fmul2_rn(neg_quot2(qx, h, y), mone);
        q.v = __fmul2_rn(neg_quot2(qy, h, y), mone);
        q.nc = __ffma2_rn(__ffma2_rn(ns, ns, nx), __fmul2_rn(z, f2(0.5f, 0.5f)), ns);
        const unsigned low = min(min(low_of(qx.x), low_of(qx.y)), min(low_of(qy.x), low_of(qy.y)));
        // a quotient that overflows, or an infinite momentum's, comes out of neg_quot2 as NaN: not fine either
        fine = fine && ord.g &&
               max_nan(max_nan(fabsf(q.u.x), fabsf(q.u.y)), max_nan(fabsf(q.v.x), fabsf(q.v.y))) < 0x1p20f;
        if (!(fine && low >= LOW_MIN)) {
            const float2 su = neg_quot2_small(qx, h, y), sv = neg_quot2_small(qy, h, y);
            q.u = f2(velocity_any(h.x, qx.x, su.x, dry), velocity_any(h.y, qx.y, su.y, dry));
            q.v = f2(velocity_any(h.x, qy.x, sv.x, dry), velocity_any(h.y, qy.y, sv.y, dry));
            if (!fine) q.nc = f2(nx.x == 0.0f ? nx.x : -sqrt_ieee(-nx.x), nx.y == 0.0f ? nx.y : -sqrt_ieee(-nx.y));
        }
        q.fx = __fadd2_rn(mulz2(qx, q.u, nz), p);
        q.fy = __fadd2_rn(mulz2(qy, q.v, nz), p);
    } else {
        const float2 inv = f2(h.x > dry ? rcp_approx(h.x) : 0.0f, h.y > dry ? rcp_approx(h.y) : 0.0f);
        q.u = __fmul2_rn(qx, inv);
        q.v = __fmul2_rn(qy, inv);
        q.nc = f2(-sqrt_fast(g * h.x), -sqrt_fast(g * h.y));
        q.fx = __ffma2_rn(qx, q.u, p);
        q.fy = __ffma2_rn(qy, q.v, p);
    }
    q.tx = mulz2(qx, q.v, nz);
    q.ty = mulz2(qy, q.u, nz);
    return q;
}

// One side of two faces: depth, normal and tangential momentum, normal velocity, negated wave speed, and the cell's own
// terms of the normal's and the tangent's flux.
struct Side {
    float2 h, qn, qt, un, nc, fn, ft;
};

__device__ __forceinline__ Side side_y(const Cells& q) { return Side{q.h, q.qy, q.qx, q.v, q.nc, q.fy, q.ty}; }
__device__ __forceinline__ Side side_x(const Cells& q) { return Side{q.h, q.qx, q.qy, q.u, q.nc, q.fx, q.tx}; }

// The west sides of a lane's two cells' west faces: the left lane's second cell, and its own first.
__device__ __forceinline__ Side west_x(const Side& a) {
    const unsigned all = 0xffffffffu;
    return Side{f2(__shfl_up_sync(all, a.h.y, 1), a.h.x),   f2(__shfl_up_sync(all, a.qn.y, 1), a.qn.x),
                f2(__shfl_up_sync(all, a.qt.y, 1), a.qt.x), f2(__shfl_up_sync(all, a.un.y, 1), a.un.x),
                f2(__shfl_up_sync(all, a.nc.y, 1), a.nc.x), f2(__shfl_up_sync(all, a.fn.y, 1), a.fn.x),
                f2(__shfl_up_sync(all, a.ft.y, 1), a.ft.x)};
}

// The ghosts of two cells across a side (ShallowWater.neighbour, ShallowWater.java:316-326): a wall negates the normal
// momentum (and so the normal velocity and the tangent's flux), an open side copies the cell.
__device__ __forceinline__ Side ghost(Side q, bool wall) {
    if (wall) {
        const float2 mone = f2(-1.0f, -1.0f);
        q.qn = __fmul2_rn(q.qn, mone);
        q.un = __fmul2_rn(q.un, mone);
        q.ft = __fmul2_rn(q.ft, mone);
    }
    return q;
}

__device__ __forceinline__ void set_x(Side& q, const Side& a, bool second, bool from_second) {
    auto put = [&](float2& d, const float2& v) { (second ? d.y : d.x) = from_second ? v.y : v.x; };
    put(q.h, a.h);
    put(q.qn, a.qn);
    put(q.qt, a.qt);
    put(q.un, a.un);
    put(q.nc, a.nc);
    put(q.fn, a.fn);
    put(q.ft, a.ft);
}

// ShallowWater.hll (ShallowWater.java:336-378) with combine (381-384), NEGATED, for two faces at once.
struct Faces {
    float2 mass, normal, tangent;
};

// ORDINARY: both sides' cells are ordinary.
template <bool EXACT, bool ORDINARY>
__device__ __forceinline__ Faces neg_hll2(float dry, float2 nz, const Side& L, const Side& R) {
    const float2 lm = __fadd2_rn(L.un, L.nc), lp = sub2(L.un, L.nc), rm = __fadd2_rn(R.un, R.nc), rp = sub2(R.un, R.nc);
    float2 sL = min2(lm, rm), sR = max2(lp, rp);
    if (!ORDINARY) {   // a dry side's wave speeds
        const float2 l2 = __ffma2_rn(f2(-2.0f, -2.0f), L.nc, L.un), r2 = __ffma2_rn(f2(2.0f, 2.0f), R.nc, R.un);
        if (!(R.h.x > dry)) { sL.x = lm.x; sR.x = l2.x; }
        if (!(R.h.y > dry)) { sL.y = lm.y; sR.y = l2.y; }
        if (!(L.h.x > dry)) { sL.x = r2.x; sR.x = rp.x; }
        if (!(L.h.y > dry)) { sL.y = r2.y; sR.y = rp.y; }
    }
    const float2 lo = min2(sL, f2(0.0f, 0.0f)), hi = max2(sR, f2(0.0f, 0.0f));
    float2 span = sub2(hi, lo);
    if (!ORDINARY) span = max2(span, f2(1e-30f, 1e-30f));
    const float2 lohi = mulz2(lo, hi, nz);
    Faces f;
    if (EXACT) {
        // ((hi FL - lo FR) + lo hi (UR - UL)) / span
        auto combine = [&](float2 fl, float2 fr, float2 ul, float2 ur) {
            return __fadd2_rn(sub2(mulz2(hi, fl, nz), mulz2(lo, fr, nz)), mulz2(lohi, sub2(ur, ul), nz));
        };
        const float2 m = combine(L.qn, R.qn, L.h, R.h), n = combine(L.fn, R.fn, L.qn, R.qn), t = combine(L.ft, R.ft, L.qt, R.qt);
        const float2 y = neg_recip2(span);
        f.mass = neg_quot2(m, span, y);
        f.normal = neg_quot2(n, span, y);
        f.tangent = neg_quot2(t, span, y);
        const unsigned low_t = min(low_of(t.x), low_of(t.y));
        if (ORDINARY) {
            if (low_t < LOW_MIN) f.tangent = neg_quot2_small(t, span, y);
        } else {
            const unsigned low = min(min(min(low_of(m.x), low_of(m.y)), min(low_of(n.x), low_of(n.y))), low_t);
            const float most = fmaxf(fmaxf(fmaxf(fabsf(m.x), fabsf(m.y)), fmaxf(fabsf(n.x), fabsf(n.y))),
                                     fmaxf(fabsf(t.x), fabsf(t.y)));
            const float least = fminf(span.x, span.y), widest = fmaxf(span.x, span.y);
            if (!(low >= LOW_MIN && most < A_MAX && least >= B_MIN && widest <= B_MAX)) {
                if (least >= B_MIN && widest <= B_MAX && most < A_MAX_SMALL) {
                    f.mass = neg_quot2_small(m, span, y);
                    f.normal = neg_quot2_small(n, span, y);
                    f.tangent = neg_quot2_small(t, span, y);
                } else if (!(low >= LOW_MIN && most < A_MAX_DRY && least >= B_MIN_DRY && widest <= B_MAX)) {
                    f.mass = f2(-div_ieee(m.x, span.x), -div_ieee(m.y, span.y));
                    f.normal = f2(-div_ieee(n.x, span.x), -div_ieee(n.y, span.y));
                    f.tangent = f2(-div_ieee(t.x, span.x), -div_ieee(t.y, span.y));
                }
            }
        }
    } else {
        const float2 inv = f2(rcp_approx(-span.x), rcp_approx(-span.y));
        auto combine = [&](float2 fl, float2 fr, float2 ul, float2 ur) {
            return __fmul2_rn(__ffma2_rn(lohi, sub2(ur, ul), sub2(__fmul2_rn(hi, fl), __fmul2_rn(lo, fr))), inv);
        };
        f.mass = combine(L.qn, R.qn, L.h, R.h);
        f.normal = combine(L.fn, R.fn, L.qn, R.qn);
        f.tangent = combine(L.ft, R.ft, L.qt, R.qt);
    }
    return f;
}

// ------------------------------------------------------------------ the step

// One CTA of four warps per tile of 248 columns x ROWS rows. The tile and a halo (256 columns from four left of the tile's
// even origin, ROWS + 2 rows) land in shared memory by three 2D TMA loads (4-byte asynchronous copies where the row pitch is
// not TMA's); then every lane walks two neighbouring columns up the tile in registers, the pair in the two halves of paired
// fp32 throughout: lane L of warp w holds columns s + 2L and s + 2L + 1, s = X0 + 62 w - 2, of which the warp updates
// s + 1 .. s + 62. A cell's west face is computed from its left neighbour's state (the lane's own other cell, or a
// shuffle), its east face is the right neighbour's west face, its south face was computed one row below and its north face
// is computed from the next row: every face once (twice where two warps meet, from the same inputs), the state read from
// shared memory once. One column a lane, pairing its x-face with its y-face, needed registers moved into pairs and twice
// the shuffles: 0.168 ms a step at 4096^2 where this took 0.147 at the time.
constexpr int STRIP_WARPS = 4;
constexpr int WARP_COLS = 62;                          // columns a warp updates
constexpr int STRIP_COLS = WARP_COLS * STRIP_WARPS;    // a multiple of 4: the box's x stays aligned
constexpr int STRIP_BW = 256;                          // box width: columns X0-4 .. X0+251, X0 = 248 * tile

template <int ROWS>
struct StripShared {
    float box[3][(ROWS + 2) * STRIP_BW];
    unsigned long long bar;
    int red[STRIP_WARPS];
    int clamps;
};

// One CTA's walk. INTERIOR: the tile and its halo lie inside the domain. EXACT: every operation as the reference's strict
// f32 rounds it; otherwise the fast mode's arithmetic. `best` starts at a speed already reached (the same in every lane
// of a warp), and a row's speeds are formed exactly only where an approximate one, a part in 2^16 up, exceeds it: the
// maximum is the same, and after the first tiles of a step few rows need it. (The approximate root of a subnormal is taken as
// the largest of them. The approximate reciprocal of a depth past 2^126 is zero, but a step's flux squares its depths, so the
// momenta of such a cell are then none, and those are formed exactly.)
template <int ROWS, bool INTERIOR, bool EXACT>
__device__ __forceinline__ void strip_walk(const SweArgs& a, StripShared<ROWS>& S, int X0, int y0, float g, float dry, float rx,
                                           float ry, int budget, int ticks, int& best, int& clamps) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned all = 0xffffffffu;
    const int nx = a.nx, ny = a.ny;
    const float2 nz = f2(a.nzero, a.nzero), rx2 = f2(rx, rx), ry2 = f2(ry, ry), mry2 = f2(-ry, -ry), mrx2 = f2(-rx, -rx);
    const int ca = X0 + WARP_COLS * warp + 2 * lane - 2, cb = ca + 1;   // this lane's columns; ca is even
    const bool own_a = lane > 0 && (INTERIOR || (ca >= 0 && ca < nx)), own_b = lane < 31 && (INTERIOR || (cb >= 0 && cb < nx));
    // With an even pitch a lane's two cells are stored as one 8-byte access; the warp's first and last lane own one each.
    const bool even = (nx & 1) == 0, pair = own_a && own_b, only = own_a != own_b;
    float* out[3];
#pragma unroll
    for (int f = 0; f < 3; f++) out[f] = a.out[f] + ((int64_t)y0 * nx + ca + (even && only && own_b ? 1 : 0));
    const bool wall_w = a.edge[0] == VF_EDGE_WALL, wall_e = a.edge[1] == VF_EDGE_WALL;
    const bool wall_s = a.edge[2] == VF_EDGE_WALL, wall_n = a.edge[3] == VF_EDGE_WALL;
    const Ordinary ord = ordinary_depths(g, dry);
    const float* at = &S.box[0][WARP_COLS * warp + 2 * lane + 2];
    auto load = [&](int r, bool& fine) {
        const float* b = at + r * STRIP_BW;
        constexpr int F = (ROWS + 2) * STRIP_BW;
        float2 h = *reinterpret_cast<const float2*>(b);
        if (!INTERIOR) {   // cells outside the domain (staged as zeros) reach no face that is used: an ordinary depth
            const bool row = y0 - 1 + r >= 0 && y0 - 1 + r < ny;
            h = f2(row && ca >= 0 && ca < nx ? h.x : 1.0f, row && cb >= 0 && cb < nx ? h.y : 1.0f);
        }
        return cells_of<EXACT>(h, *reinterpret_cast<const float2*>(b + F), *reinterpret_cast<const float2*>(b + 2 * F), g, ord,
                               dry, nz, fine);
    };
    const int last = INTERIOR ? ROWS + 1 : min(ROWS + 1, ny - y0 + 1);   // the row above the tile's, or the domain's, last
    bool fine;
    Cells prev = load(0, fine);
    bool fine_prev = __all_sync(all, fine);   // the warp's cells of the row are all ordinary
    const float2 zero = f2(0.0f, 0.0f);
    Faces gs = {zero, zero, zero}, dw = {zero, zero, zero};   // south faces; west minus east faces (all negated fluxes)
    // two rows an iteration, so that no register moves from this row's to the last one's; but the exact body is long, and
    // in short tiles the instruction cache's misses cost more (learned steps at 1024^2: 599 us a pass, 627 with two)
    constexpr int ROWS_AT_ONCE = EXACT && ROWS < 8 ? 1 : 2;
#pragma unroll ROWS_AT_ONCE
    for (int r = 1; r <= last; r++) {
        const int y = y0 - 1 + r;   // this box row's row of the domain
        const Cells cur = load(r, fine);
        const bool fine_cur = __all_sync(all, fine);
        Side bot = side_y(prev), top = side_y(cur), right = side_x(cur), left = west_x(right);
        if (!INTERIOR) {
            if (y == 0) bot = ghost(top, wall_s);
            if (y == ny) top = ghost(bot, wall_n);
            if (ca == 0) set_x(left, ghost(right, wall_w), false, false);      // nx even or odd: column 0 is a first cell
            if (ca == nx) set_x(right, ghost(left, wall_e), false, false);
            if (cb == nx) set_x(right, ghost(left, wall_e), true, true);
        }
        Faces gn, fw;   // between rows y-1 and y, and row y's west faces
        if (fine_prev && fine_cur) {
            gn = neg_hll2<EXACT, true>(dry, nz, bot, top);
            fw = neg_hll2<EXACT, true>(dry, nz, left, right);
        } else {
            gn = neg_hll2<EXACT, false>(dry, nz, bot, top);
            fw = neg_hll2<EXACT, false>(dry, nz, left, right);
        }
        if (r >= 2) {
            // the update of row y-1 (ShallowWater.java:206-235) from its four faces, their negated fluxes' differences
            // taken the other way round
            float2 h, hu, hv;
            if (EXACT) {
                auto update = [&](float2 q, float2 x, float2 s, float2 n) {
                    return sub2(sub2(q, mulz2(rx2, x, nz)), mulz2(ry2, sub2(s, n), nz));
                };
                h = update(prev.h, dw.mass, gs.mass, gn.mass);
                hu = update(prev.qx, dw.normal, gs.tangent, gn.tangent);
                hv = update(prev.qy, dw.tangent, gs.normal, gn.normal);
            } else {
                h = __ffma2_rn(mry2, sub2(gs.mass, gn.mass), __ffma2_rn(mrx2, dw.mass, prev.h));
                hu = __ffma2_rn(mry2, sub2(gs.tangent, gn.tangent), __ffma2_rn(mrx2, dw.normal, prev.qx));
                hv = __ffma2_rn(mry2, sub2(gs.normal, gn.normal), __ffma2_rn(mrx2, dw.tangent, prev.qy));
            }
            const float2 nh = max2(h, zero);
            const float2 now[3] = {nh, hu, hv};
            if (even) {
                if (pair) {
#pragma unroll
                    for (int f = 0; f < 3; f++) *reinterpret_cast<float2*>(out[f]) = now[f];
                }
                if (only) {
#pragma unroll
                    for (int f = 0; f < 3; f++) *out[f] = own_a ? now[f].x : now[f].y;
                }
            } else {
#pragma unroll
                for (int f = 0; f < 3; f++) {
                    if (own_a) out[f][0] = now[f].x;
                    if (own_b) out[f][1] = now[f].y;
                }
            }
#pragma unroll
            for (int f = 0; f < 3; f++) out[f] += nx;
            if (own_a && h.x < 0.0f) clamps++;
            if (own_b && h.y < 0.0f) clamps++;
            if (!INTERIOR && own_a && ca == 0 && y == 1) {
                *a.speed_clear = 0;
                *a.budget_out = budget - ticks;
            }
            // the fastest wave: max(|u|, |v|) + sqrt(g h); the larger quotient is the larger numerator's
            const float2 most = f2(fmaxf(fabsf(hu.x), fabsf(hv.x)), fmaxf(fabsf(hu.y), fabsf(hv.y)));
            const float2 inv = f2(nh.x > dry ? rcp_approx(nh.x) : 0.0f, nh.y > dry ? rcp_approx(nh.y) : 0.0f);
            const float2 x = __fmul2_rn(nh, f2(g, g));
            constexpr float LEAST = EXACT ? 0x1p-63f : 0.0f;
            const float2 speed = __ffma2_rn(most, inv, f2(sqrt_fast(x.x, LEAST), sqrt_fast(x.y, LEAST)));
            if (EXACT) {
                const float reached = __int_as_float(best);
                const bool over = (own_a && !(speed.x * (1.0f + 0x1p-16f) <= reached)) ||
                                  (own_b && !(speed.y * (1.0f + 0x1p-16f) <= reached));
                if (__any_sync(all, over)) {
                    if (own_a)
                        best = max(best, __float_as_int((nh.x > dry ? div_ieee(most.x, nh.x) : 0.0f) + sqrt_ieee(x.x)));
                    if (own_b)
                        best = max(best, __float_as_int((nh.y > dry ? div_ieee(most.y, nh.y) : 0.0f) + sqrt_ieee(x.y)));
                    best = __reduce_max_sync(all, best);
                }
            } else {
                if (own_a) best = max(best, __float_as_int(speed.x));
                if (own_b) best = max(best, __float_as_int(speed.y));
            }
        }
        gs = gn;
        // this row's west minus east faces for its update at the next row: an east face is the west face of the lane's
        // other cell, or of the right lane's first
        dw.mass = sub2(fw.mass, f2(fw.mass.y, __shfl_down_sync(all, fw.mass.x, 1)));
        dw.normal = sub2(fw.normal, f2(fw.normal.y, __shfl_down_sync(all, fw.normal.x, 1)));
        dw.tangent = sub2(fw.tangent, f2(fw.tangent.y, __shfl_down_sync(all, fw.tangent.x, 1)));
        prev = cur;
        fine_prev = fine_cur;
    }
}

// One step. Launched as a programmatic dependent of the previous step: its CTAs may become resident during that step's
// last wave, set up their barrier, and wait (griddepcontrol.wait: until the previous grid has completed and its stores are
// visible) before reading anything the previous step wrote.
template <int ROWS, bool EXACT>
__global__ void __launch_bounds__(STRIP_WARPS * 32) k_swe_strip(SweArgs a, const __grid_constant__ CUtensorMap tm_h,
                                                                    const __grid_constant__ CUtensorMap tm_hu,
                                                                    const __grid_constant__ CUtensorMap tm_hv) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(128) unsigned char strip_raw[];
    const uint32_t mis = (uint32_t)__cvta_generic_to_shared(strip_raw) & 127u;
    StripShared<ROWS>& S = *reinterpret_cast<StripShared<ROWS>*>(strip_raw + ((128u - mis) & 127u));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        S.clamps = 0;
        if (a.use_tma) {
            const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&S.bar);
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int X0 = blockIdx.x * STRIP_COLS, y0 = blockIdx.y * ROWS;
    const int nx = a.nx, ny = a.ny;
    // 1. the tile and its halo on their way
    if (a.use_tma) {
        if (tid == 0) {
            const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&S.bar);
            const uint32_t bytes = 3u * (ROWS + 2) * STRIP_BW * 4u;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            const CUtensorMap* maps[3] = {&tm_h, &tm_hu, &tm_hv};
            const int bx = X0 - 4, by = y0 - 1;   // bx is a multiple of 4: 16-byte aligned
            for (int f = 0; f < 3; f++) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&S.box[f][0]);
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
                    "[%4];" ::"r"(dst),
                    "l"(maps[f]), "r"(bx), "r"(by), "r"(bar)
                    : "memory");
            }
        }
    } else {
        // two columns a thread, every row in flight together; nothing is read outside the domain
        for (int ly = 0; ly < ROWS + 2; ly++) {
            const int gy = y0 - 1 + ly;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int lx = tid + q * STRIP_WARPS * 32, gx = X0 - 4 + lx;
                const bool in = gx >= 0 && gx < nx && gy >= 0 && gy < ny;
                const int64_t k = in ? (int64_t)gy * nx + gx : 0;
#pragma unroll
                for (int f = 0; f < 3; f++)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(&S.box[f][ly * STRIP_BW + lx])),
                                 "l"(a.in[f] + k), "r"(in ? 4 : 0)
                                 : "memory");
            }
        }
    }
    // ShallowWater.java:184-192: the step from the fastest wave, in whole ticks, within the budget
    const float g = a.params[0], courant = a.params[1], dx = a.params[2], dy = a.params[3], dry = a.params[4];
    const float fastest = __int_as_float(__ldcg(a.speed_in));
    const float allowed = fminf((courant * fminf(dx, dy)) / fmaxf(fastest, 1e-30f), 2000.0f);
    int ticks = (int)(allowed * 1000000.0f);
    const int budget = __ldcg(a.budget_in);
    if (budget < ticks) ticks = budget;
    const float dt = (float)ticks * (float)(1.0 / 1000000.0);
    const float rx = dt / dx;
    const float ry = dt / dy;
    int best = __ldcg(a.speed_out), clamps = 0;   // what other tiles have reached already (it only grows within a step)
    bool loaded = true;
    if (a.use_tma) loaded = wait_barrier(&S.bar, 0, a.status);
    else asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    if (!__syncthreads_and(loaded)) return;   // a TMA that never landed: the status says so, nothing is written

    // 2. the column walk: tiles that touch no side of the domain skip every ghost and bounds test
    best = __shfl_sync(0xffffffffu, best, 0);   // one value a warp
    // (the columns held, X0-2 .. X0+247, and the one right of the last updated)
    const bool interior = X0 >= 2 && X0 + STRIP_COLS <= nx && y0 >= 1 && y0 + ROWS + 1 <= ny;
    if (interior)
        strip_walk<ROWS, true, EXACT>(a, S, X0, y0, g, dry, rx, ry, budget, ticks, best, clamps);
    else if (__any_sync(0xffffffffu, X0 + WARP_COLS * warp - 1 < nx))   // a warp of the last tile may update no column
        strip_walk<ROWS, false, EXACT>(a, S, X0, y0, g, dry, rx, ry, budget, ticks, best, clamps);
    // 3. the CTA's fastest wave and clamp count, one atomic each
    best = __reduce_max_sync(0xffffffffu, best);
    clamps = __reduce_add_sync(0xffffffffu, clamps);
    if (lane == 0) {
        S.red[warp] = best;
        if (clamps) atomicAdd(&S.clamps, clamps);
    }
    __syncthreads();
    if (tid == 0) {
        int m = 0;
        for (int w = 0; w < STRIP_WARPS; w++) m = max(m, S.red[w]);
        // only a filter: the buffer only grows within a step (ShallowWater.java:227-235)
        if (m > *(volatile int*)a.speed_out) atomicMax(a.speed_out, m);
        if (S.clamps) atomicAdd(a.clamped, S.clamps);
    }
}

// ------------------------------------------------------------------ diagnostics (Diagnostics.of)

struct DiagPart {
    double volume, min_depth, max_depth, max_speed, max_froude, max_wave;
    int non_finite, negative, wet;
};

// The next step's wave speed from a state the host or another kernel changed: bits of the largest
// max(|u|, |v|) + sqrt(g h), the same per-cell expression the step's update computes (ShallowWater.java:236-241). Eight
// cells a thread in flight, and as in the step's walk the exact quotient and root only where an approximate speed exceeds the
// thread's largest so far, a part in 2^15 down (or is none: a depth that is negative, vanishing or not a number, or so large
// that its approximate reciprocal is zero). 11 -> 5 us for 1024^2 cells.
// Up to two blocks an SM take one cell a thread: 6.3 us a measurement of 64^2 or 201 x 117 cells, 8.5 with eight cells a thread,
// of which seven may be the last cell again; at 500^2 cells 11.5 and 8.6.
constexpr int SPEED_CELLS = 8;
template <int CELLS>
__global__ void __launch_bounds__(256) k_swe_speed(const float* __restrict__ h, const float* __restrict__ hu,
                                                   const float* __restrict__ hv, int64_t n, const float* params, int* speed) {
    const float g = params[0], dry = params[4];
    int best = 0;
    float reached = -1.0f;   // approximate speeds up to this are no larger than the best
    const int64_t all = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += CELLS * all) {
        float d[CELLS], qu[CELLS], qv[CELLS];
#pragma unroll
        for (int k = 0; k < CELLS; k++) {
            const int64_t i = min(i0 + k * all, n - 1);
            d[k] = h[i];
            qu[k] = hu[i];
            qv[k] = hv[i];
        }
#pragma unroll
        for (int k = 0; k < CELLS; k++) {
            const float x = g * d[k], most = fmaxf(fabsf(qu[k]), fabsf(qv[k]));   // the larger quotient's numerator
            const float near = (d[k] > dry ? most * rcp_approx(d[k]) : 0.0f) + sqrt_fast(x);
            if (!(x >= 0x1p-126f && d[k] <= 0x1p126f && near <= reached)) {
                const float u = velocity(d[k], qu[k], dry), w = velocity(d[k], qv[k], dry);
                best = max(best, __float_as_int(fmaxf(fabsf(u), fabsf(w)) + sqrtf(x)));
                reached = __int_as_float(best) * (1.0f - 0x1p-15f);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(speed, best);
}

// Coarse cell (i, j) of the box [x0, x0 + cnx) x [y0, y0 + cny) = the mean of fine cells (2i..2i+1, 2j..2j+1)
// counted from the fine patch's cell (fx0, fy0).
// One device word from a kernel argument: the budget written in stream order, without a host wait.
__global__ void k_swe_set_word(int* p, int v) { *p = v; }

__global__ void k_swe_restrict(const float* const* fine, int fnx, int fx0, int fy0, float* const* coarse, int ccnx,
                               int x0, int y0, int cnx, int cny) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (int64_t)cnx * cny) return;
    const int i = (int)(k % cnx), j = (int)(k / cnx);
    const int64_t f = (int64_t)(fy0 + 2 * j) * fnx + fx0 + 2 * i;
    const int64_t c = (int64_t)(y0 + j) * ccnx + x0 + i;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const float* a = fine[q];
        coarse[q][c] = 0.25f * ((a[f] + a[f + 1]) + (a[f + fnx] + a[f + fnx + 1]));
    }
}

// Fine patch cell (fi, fj) = coarse cell (x0 + fi/2, y0 + fj/2), the coarse index clamped into its grid.
__global__ void k_swe_prolong(const float* const* coarse, int ccnx, int ccny, int x0, int y0, float* const* fine, int fnx,
                              int fny) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (int64_t)fnx * fny) return;
    const int fi = (int)(k % fnx), fj = (int)(k / fnx);
    const int ci = min(max(x0 + fi / 2, 0), ccnx - 1), cj = min(max(y0 + fj / 2, 0), ccny - 1);
    const int64_t c = (int64_t)cj * ccnx + ci;
#pragma unroll
    for (int q = 0; q < 3; q++) fine[q][k] = coarse[q][c];
}

// Per tile of t x t cells: the largest relative depth jump to the east or north neighbour,
// (|h(i+1,j) - h(i,j)| + |h(i,j+1) - h(i,j)|) / max(h(i,j), dry), as float bits (atomicMax).
__global__ void k_swe_jump(const float* h, int nx, int ny, int t, int tiles_x, float dry, int* out) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (int64_t)nx * ny) return;
    const int i = (int)(k % nx), j = (int)(k / nx);
    const float d = h[k];
    const float ex = i < nx - 1 ? fabsf(h[k + 1] - d) : 0.0f;
    const float ny_ = j < ny - 1 ? fabsf(h[k + nx] - d) : 0.0f;
    const float jump = (ex + ny_) / fmaxf(d, dry);
    atomicMax(&out[(j / t) * tiles_x + i / t], __float_as_int(jump));
}

__global__ void __launch_bounds__(256) k_swe_diag(const float* h, const float* hu, const float* hv, int64_t n,
                                                  double g, double dry, DiagPart* parts) {
    DiagPart p{0.0, INFINITY, 0.0, 0.0, 0.0, 0.0, 0, 0, 0};
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const float hk = h[k], uk = hu[k], vk = hv[k];
        if (!isfinite(hk) || !isfinite(uk) || !isfinite(vk)) {
            p.non_finite++;
            continue;
        }
        if (hk < 0) p.negative++;
        p.volume += hk;
        p.max_depth = fmax(p.max_depth, (double)hk);
        if ((double)hk <= dry) continue;
        p.wet++;
        p.min_depth = fmin(p.min_depth, (double)hk);
        const double u = (double)uk / hk, v = (double)vk / hk;
        const double c = sqrt(g * hk);
        const double speed = sqrt(u * u + v * v);
        p.max_speed = fmax(p.max_speed, speed);
        if (hk >= 1e-3) p.max_froude = fmax(p.max_froude, speed / c);
        p.max_wave = fmax(p.max_wave, fmax(fabs(u), fabs(v)) + c);
    }
    __shared__ DiagPart sp[256];
    sp[threadIdx.x] = p;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            DiagPart& a = sp[threadIdx.x];
            const DiagPart& b = sp[threadIdx.x + s];
            a.volume += b.volume;
            a.min_depth = fmin(a.min_depth, b.min_depth);
            a.max_depth = fmax(a.max_depth, b.max_depth);
            a.max_speed = fmax(a.max_speed, b.max_speed);
            a.max_froude = fmax(a.max_froude, b.max_froude);
            a.max_wave = fmax(a.max_wave, b.max_wave);
            a.non_finite += b.non_finite;
            a.negative += b.negative;
            a.wet += b.wet;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) parts[blockIdx.x] = sp[0];
}


// A 2D tensor map over one nx x ny f32 field with an hx x hy box; false if TMA cannot take it
// (row pitch not a multiple of 16 bytes, or an unaligned base).
bool make_map(CUtensorMap* m, const float* base, int nx, int ny, int hx, int hy) {
    EncodeTiled enc = tensor_map_encoder();
    if (!enc) return false;
    if (((uintptr_t)base & 15) || ((int64_t)nx * 4) % 16 != 0) return false;
    cuuint64_t dims[2] = {(cuuint64_t)nx, (cuuint64_t)ny};
    cuuint64_t strides[1] = {(cuuint64_t)nx * 4};
    cuuint32_t box[2] = {(cuuint32_t)hx, (cuuint32_t)hy};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace

// ------------------------------------------------------------------ the handle

struct vf_swe {
    int nx, ny;
    int edges[4];
    int64_t cells;
    cudaStream_t stream = nullptr;
    DeviceBuffer state[2];    // 3 fields each
    DeviceBuffer small;       // speed[3], budget[2], clamped, params[5] (as ints/floats)
    DeviceBuffer status, diag;
    int32_t* host_words = nullptr;   // pinned: the budget and the status word read back together
    CUtensorMap maps[4][2][3];   // [rows 16, 8, 4, 2][state][field]
    bool tma = false;
    int tile_w = 64;             // vf_swe_set_tile_width: 64 picks the tiles' rows by the grid's size, 32 takes 4, 0 takes 16
    bool pdl = true;             // steps launched as programmatic dependents of the previous step
    bool exact = true;           // false: the fast mode's arithmetic (vf_swe_set_exact)
    // PatchSimulation.java:52-56
    int64_t clock_now = 0;
    int32_t clock_outstanding = 0;
    int64_t dispatched = 0;
    int64_t total_steps = 0;
    int64_t last_step = 0;
    float host_params[5];
    Profiler prof;
};

namespace {

int* small_i(vf_swe* h) { return h->small.as<int>(); }
int* speed_slot(vf_swe* h, int k) { return small_i(h) + k; }          // 0..2
int* budget_slot(vf_swe* h, int k) { return small_i(h) + 3 + k; }     // 3..4
int* clamped_ptr(vf_swe* h) { return small_i(h) + 5; }                // 5
float* params_ptr(vf_swe* h) { return h->small.as<float>() + 8; }     // 8..12

float* field(vf_swe* h, int s, int f) { return h->state[s].as<float>() + (int64_t)f * h->cells; }

int32_t swe_params_check(const int32_t* params, int32_t n, float out[5]) {
    VF_REQUIRE(params && n == 5, VF_EINVAL, "ShallowWater.params has 5 words, got %d", n);
    for (int k = 0; k < 5; k++) out[k] = bits_to_float(params[k]);
    // ShallowWater.paramsAllowingInstability refuses a Courant number that is not positive (262-264);
    // above 1/2 is the caller's choice (params vs paramsAllowingInstability).
    VF_REQUIRE(out[1] > 0, VF_EINVAL, "a Courant number must be positive, got %g", out[1]);
    return VF_OK;
}

// The tiles' rows: 16, 8, 4 or 2. A tile computes ROWS + 1 rows of faces and reads ROWS + 2 of cells, so tall tiles do
// least; but a CTA is four warps, and a grid that gives every SM few of them is over sooner in short ones. The first height
// that gives each SM this many tiles, by arithmetic (exact, fast), measured in us a step: exact 2048^2 51 with 8 rows, 55
// with 16 and 4; 1024^2 22 with 4, 27 with 8; 512^2 12 with 2, 13 with 4; 201 x 117 5.3 with 2, 7.0 with 4; fast 2048^2 35
// with 16, 37 with 8; 300 x 4000 20.5 with 16, 21.2 with 8; 1024^2 15.8 with 8, 16.8 with 4; 512^2 8.7 with 4, 9.6 with 2
// (the fast ones since 32, 18.6, 14.6 and 7.9: two rows an iteration, which spares a row's registers their move, and fewer
// stores).
constexpr int STRIP_ROWS[4] = {16, 8, 4, 2};
constexpr int TILES_PER_SM[2][3] = {{8, 8, 3}, {3, 3, 1}};
int tile_rows_index(int nx, int ny, bool exact) {
    const int64_t strips = nx / STRIP_COLS + 1;
    for (int k = 0; k < 3; k++)
        if (strips * div_up(ny, STRIP_ROWS[k]) >= (int64_t)TILES_PER_SM[exact ? 0 : 1][k] * sm_count()) return k;
    return 3;
}

size_t strip_smem(int rows) {
    return 128 + (rows == 16  ? sizeof(StripShared<16>)
                  : rows == 8 ? sizeof(StripShared<8>)
                  : rows == 4 ? sizeof(StripShared<4>)
                              : sizeof(StripShared<2>));
}

const void* strip_kernel(int k, bool exact) {
    switch (k) {
        case 0: return exact ? (const void*)k_swe_strip<16, true> : (const void*)k_swe_strip<16, false>;
        case 1: return exact ? (const void*)k_swe_strip<8, true> : (const void*)k_swe_strip<8, false>;
        case 2: return exact ? (const void*)k_swe_strip<4, true> : (const void*)k_swe_strip<4, false>;
        default: return exact ? (const void*)k_swe_strip<2, true> : (const void*)k_swe_strip<2, false>;
    }
}

// One dispatch: step k of the rotation (PatchSimulation.dispatch, PatchSimulation.java:197-205).
int32_t dispatch(vf_swe* h) {
    const int64_t k = h->dispatched;
    const int si = (int)(k % 2), so = (int)((k + 1) % 2);
    SweArgs a;
    for (int f = 0; f < 3; f++) {
        a.in[f] = field(h, si, f);
        a.out[f] = field(h, so, f);
    }
    a.params = params_ptr(h);
    a.speed_in = speed_slot(h, (int)(k % 3));
    a.speed_out = speed_slot(h, (int)((k + 1) % 3));
    a.speed_clear = speed_slot(h, (int)((k + 2) % 3));
    a.budget_in = budget_slot(h, si);
    a.budget_out = budget_slot(h, so);
    a.clamped = clamped_ptr(h);
    a.status = h->status.as<uint32_t>();
    a.nx = h->nx;
    a.ny = h->ny;
    for (int e = 0; e < 4; e++) a.edge[e] = h->edges[e];
    a.use_tma = h->tma ? 1 : 0;
    a.nzero = -0.0f;
    int k3 = h->tile_w == 64 ? tile_rows_index(h->nx, h->ny, h->exact) : h->tile_w == 32 ? 2 : 0;
    while (k3 > 0 && div_up(h->ny, STRIP_ROWS[k3]) > 65535) k3--;   // the most a launch has in y
    const int rows = STRIP_ROWS[k3];
    CUtensorMap* m = h->maps[k3][si];
    void* args[] = {&a, &m[0], &m[1], &m[2]};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(div_up(h->nx + 1, STRIP_COLS), div_up(h->ny, rows));   // tile t updates columns 248t - 1 .. 248t + 246
    cfg.blockDim = dim3(STRIP_WARPS * 32);
    cfg.dynamicSmemBytes = strip_smem(rows);
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = h->pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const void* fn = strip_kernel(k3, h->exact);
    h->prof.begin(h->exact ? "k_swe_strip" : "k_swe_strip_fast", h->stream);
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    h->prof.end(h->stream);
    VF_TRY_CUDA(e);
    h->dispatched++;
    return VF_OK;
}

// The budget left in slot and the device status word, in one host wait.
int32_t read_budget(vf_swe* h, int slot, int32_t* out, uint32_t* status) {
    VF_TRY_CUDA(cudaMemcpyAsync(h->host_words, budget_slot(h, slot), 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaMemcpyAsync(h->host_words + 1, h->status.ptr, 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    *out = h->host_words[0];
    if (status) *status = (uint32_t)h->host_words[1];
    return VF_OK;
}

// Stream-ordered: the steps dispatched after it read the new budget; no host wait.
int32_t write_budget(vf_swe* h, int slot, int32_t v) {
    VF_LAUNCH(h->prof, "k_swe_set_word", h->stream, k_swe_set_word, 1, 1, 0, budget_slot(h, slot), v);
    return VF_OK;
}

// A nonzero device status (read back with the budget): cleared, and reported as the error it is.
int32_t status_error(vf_swe* h, uint32_t st) {
    if (!st) return VF_OK;
    VF_TRY_CUDA(cudaMemsetAsync(h->status.ptr, 0, 4, h->stream));
    set_error("a kernel flagged device status 0x%x", st);
    return (st & ST_TIMEOUT) ? VF_ETIMEOUT : VF_EDEVICE;
}

int32_t status_swe(vf_swe* h) {
    VF_TRY_CUDA(cudaMemcpyAsync(h->host_words + 1, h->status.ptr, 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return status_error(h, (uint32_t)h->host_words[1]);
}

// ShallowWater.fastestWave (ShallowWater.java:287-295), on the host.
int32_t fastest_wave_bits(const float* h, const float* hu, const float* hv, int64_t n, double g, double dry) {
    float fastest = 0.0f;
    for (int64_t k = 0; k < n; k++) {
        float u = (double)h[k] > dry ? hu[k] / h[k] : 0.0f;
        float w = (double)h[k] > dry ? hv[k] / h[k] : 0.0f;
        float c = (float)std::sqrt(g * (double)h[k]);
        float s = std::fmax(std::fabs(u), std::fabs(w)) + c;
        if (std::isnan(s) || std::isnan(fastest)) fastest = NAN;
        else fastest = fastest > s ? fastest : s;
    }
    int32_t b;
    memcpy(&b, &fastest, 4);
    return b;
}

}  // namespace

extern "C" {

int32_t vf_swe_create(int32_t nx, int32_t ny, const int32_t edges[4], vf_swe** out) {
    VF_REQUIRE(out && edges, VF_EINVAL, "null argument");
    *out = nullptr;
    VF_REQUIRE(nx >= 1 && ny >= 1, VF_EINVAL, "a patch needs at least one cell each way, got %d x %d", nx, ny);
    for (int e = 0; e < 4; e++)
        VF_REQUIRE(edges[e] == VF_EDGE_WALL || edges[e] == VF_EDGE_OPEN, VF_EINVAL, "every side of a patch needs an edge");
    int32_t rc = require_device();
    if (rc) return rc;
    vf_swe* h = new vf_swe();
    h->nx = nx;
    h->ny = ny;
    for (int e = 0; e < 4; e++) h->edges[e] = edges[e];
    h->cells = (int64_t)nx * ny;
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete h;
        set_error("cudaStreamCreate failed");
        return VF_ECUDA;
    }
    if ((rc = h->state[0].alloc((size_t)3 * h->cells * 4)) || (rc = h->state[1].alloc((size_t)3 * h->cells * 4)) ||
        (rc = h->small.alloc(64)) || (rc = h->status.alloc(16)) || (rc = h->diag.alloc(sizeof(DiagPart) * 1184))) {
        vf_swe_destroy(h);
        return rc;
    }
    if (cudaMallocHost(&h->host_words, 16) != cudaSuccess) {
        h->host_words = nullptr;
        vf_swe_destroy(h);
        set_error("cudaMallocHost(16) failed");
        return VF_ENOMEM;
    }
    for (DeviceBuffer* b : {&h->state[0], &h->state[1], &h->small, &h->status}) cudaMemsetAsync(b->ptr, 0, b->bytes, h->stream);
    for (int k = 0; k < 8; k++)
        if (cudaFuncSetAttribute(strip_kernel(k / 2, k % 2), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)strip_smem(STRIP_ROWS[k / 2])) != cudaSuccess) {
            vf_swe_destroy(h);
            set_error("cannot give the shallow-water kernel %zu bytes of shared memory", strip_smem(STRIP_ROWS[k / 2]));
            return VF_ECUDA;
        }
    bool tma = true;
    for (int k = 0; k < 4; k++)
        for (int q = 0; q < 2; q++)
            for (int f = 0; f < 3; f++)
                tma = tma && make_map(&h->maps[k][q][f], field(h, q, f), nx, ny, STRIP_BW, STRIP_ROWS[k] + 2);
    h->tma = tma;
    if (!tma) memset(h->maps, 0, sizeof h->maps);
    h->tile_w = 64;
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) {
        vf_swe_destroy(h);
        set_error("clearing buffers failed");
        return VF_ECUDA;
    }
    *out = h;
    return VF_OK;
}

int32_t vf_swe_load(vf_swe* h, const float* hcell, const float* hu, const float* hv, const int32_t* params,
                    int32_t nparams) {
    VF_REQUIRE(h && hcell && hu && hv, VF_EINVAL, "null argument");
    float p[5];
    int32_t rc = swe_params_check(params, nparams, p);
    if (rc) return rc;
    memcpy(h->host_params, p, sizeof p);
    h->dispatched = 0;
    h->total_steps = 0;
    h->last_step = 0;
    h->clock_now = 0;
    h->clock_outstanding = 0;
    const float* src[3] = {hcell, hu, hv};
    for (int f = 0; f < 3; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(field(h, 0, f), src[f], (size_t)h->cells * 4, cudaMemcpyHostToDevice, h->stream));
    int32_t small[16] = {0};
    small[0] = fastest_wave_bits(hcell, hu, hv, h->cells, (double)p[0], (double)p[4]);   // PatchSimulation.java:100-102
    memcpy(small + 8, p, sizeof p);
    VF_TRY_CUDA(cudaMemcpyAsync(h->small.ptr, small, sizeof small, cudaMemcpyHostToDevice, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

int32_t vf_swe_params(vf_swe* h, const int32_t* params, int32_t nparams) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    float p[5];
    int32_t rc = swe_params_check(params, nparams, p);
    if (rc) return rc;
    memcpy(h->host_params, p, sizeof p);
    VF_TRY_CUDA(cudaMemcpyAsync(params_ptr(h), p, sizeof p, cudaMemcpyHostToDevice, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

// PatchSimulation.advance (PatchSimulation.java:120-145). The clock is the host's i64 tick count:
// grant gives up to 2^31-1 ticks to the device as its budget; settle moves the clock by what was spent.
int32_t vf_swe_advance(vf_swe* h, int64_t ticks, int32_t max_steps, int32_t* steps_out, int64_t* spent,
                       int64_t* behind) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(ticks >= 0 && max_steps >= 0, VF_EINVAL, "ticks and maxSteps must be >= 0");
    const int64_t before = h->clock_now;
    const int64_t want = (before + ticks) - h->clock_now;
    const int32_t granted = (int32_t)(want < 0 ? 0 : want > 2147483647LL ? 2147483647LL : want);
    h->clock_outstanding = granted;
    int32_t rc = write_budget(h, (int)(h->dispatched % 2), granted);
    if (rc) return rc;
    int32_t left = granted;
    int32_t steps = 0;
    bool read = false;
    uint32_t st = 0;
    while (left > 0 && steps < max_steps) {
        const int32_t batch =
            h->last_step > 0 ? (int32_t)std::min<int64_t>(max_steps - steps, ((int64_t)left + h->last_step - 1) / h->last_step)
                             : 1;
        for (int s = 0; s < batch; s++)
            if ((rc = dispatch(h))) return rc;
        steps += batch;
        int32_t now = 0;
        if ((rc = read_budget(h, (int)(h->dispatched % 2), &now, &st))) return rc;
        read = true;
        if (now > 0 && now < left) h->last_step = (left - now) / batch;
        left = now;
    }
    h->clock_now += h->clock_outstanding - left;   // settle
    h->clock_outstanding = 0;
    h->total_steps += steps;
    if (steps_out) *steps_out = steps;
    if (spent) *spent = h->clock_now - before;
    if (behind) *behind = left;
    return read ? status_error(h, st) : status_swe(h);
}

int32_t vf_swe_read(vf_swe* h, float* hcell, float* hu, float* hv) {
    VF_REQUIRE(h && hcell && hu && hv, VF_EINVAL, "null argument");
    const int s = (int)(h->dispatched % 2);
    float* dst[3] = {hcell, hu, hv};
    for (int f = 0; f < 3; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(dst[f], field(h, s, f), (size_t)h->cells * 4, cudaMemcpyDeviceToHost, h->stream));
    return status_swe(h);
}

int32_t vf_swe_fastest_wave(vf_swe* h, double* out) {
    VF_REQUIRE(h && out, VF_EINVAL, "null argument");
    int32_t b = 0;
    VF_TRY_CUDA(cudaMemcpyAsync(&b, speed_slot(h, (int)(h->dispatched % 3)), 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    *out = (double)bits_to_float(b);
    return VF_OK;
}

int32_t vf_swe_clamped(vf_swe* h, int32_t* out) {
    VF_REQUIRE(h && out, VF_EINVAL, "null argument");
    VF_TRY_CUDA(cudaMemcpyAsync(out, clamped_ptr(h), 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

int64_t vf_swe_now(const vf_swe* h) { return h ? h->clock_now : 0; }

int64_t vf_swe_steps(const vf_swe* h) { return h ? h->total_steps : 0; }

int32_t vf_swe_dispatch(vf_swe* h, int32_t n) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(n >= 0, VF_EINVAL, "n must be >= 0");
    for (int k = 0; k < n; k++) {
        int32_t rc = dispatch(h);
        if (rc) return rc;
    }
    return VF_OK;
}

int64_t vf_swe_dispatched(const vf_swe* h) { return h ? h->dispatched : 0; }

// The snapshot's body: the 16-word device block (speed words in their rotation, budget words, clamp count, params),
// the host clock, dispatch count, step total and last step's ticks, then h, hu, hv of the current state.
int32_t vf_swe_snapshot(vf_swe* h, void* buf, int64_t cap, int64_t* size) {
    VF_REQUIRE(h && size, VF_EINVAL, "null argument");
    const size_t fields = (size_t)3 * h->cells * 4;
    const uint64_t payload = 64 + 4 * 8 + fields;
    *size = (int64_t)(sizeof(SnapHeader) + payload);
    if (!buf) return VF_OK;
    VF_REQUIRE(cap >= *size, VF_EINVAL, "a snapshot of this patch takes %lld bytes, the buffer has %lld",
               (long long)*size, (long long)cap);
    VF_REQUIRE(h->clock_outstanding == 0, VF_ESTATE, "a grant is outstanding");
    char* body = static_cast<char*>(buf) + sizeof(SnapHeader);
    VF_TRY_CUDA(cudaMemcpyAsync(body, h->small.ptr, 64, cudaMemcpyDeviceToHost, h->stream));
    const int64_t clock[4] = {h->clock_now, h->dispatched, h->total_steps, h->last_step};
    memcpy(body + 64, clock, sizeof clock);
    const int s = (int)(h->dispatched % 2);
    for (int f = 0; f < 3; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(body + 96 + (size_t)f * h->cells * 4, field(h, s, f), (size_t)h->cells * 4,
                                    cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    int32_t rc = status_swe(h);
    if (rc) return rc;
    const int32_t edges = h->edges[0] | h->edges[1] << 8 | h->edges[2] << 16 | h->edges[3] << 24;
    SnapHeader hd = snap_header(SNAP_SWE, h->nx, h->ny, 1, edges, h->cells, h->total_steps, payload);
    hd.checksum = fnv1a(body, payload);
    memcpy(buf, &hd, sizeof hd);
    return VF_OK;
}

int32_t vf_swe_restore(vf_swe* h, const void* buf, int64_t size) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    const int32_t edges = h->edges[0] | h->edges[1] << 8 | h->edges[2] << 16 | h->edges[3] << 24;
    SnapHeader want = snap_header(SNAP_SWE, h->nx, h->ny, 1, edges, h->cells, 0, 64 + 4 * 8 + (size_t)3 * h->cells * 4);
    SnapHeader got;
    int32_t rc = snap_check(buf, size, want, &got);
    if (rc) return rc;
    const char* body = static_cast<const char*>(buf) + sizeof(SnapHeader);
    int32_t small[16];
    memcpy(small, body, sizeof small);
    float p[5];
    if ((rc = swe_params_check(small + 8, 5, p))) return rc;
    int64_t clock[4];
    memcpy(clock, body + 64, sizeof clock);
    VF_REQUIRE(clock[1] >= 0 && clock[2] >= 0 && clock[3] >= 0, VF_EINVAL, "a snapshot with negative counts");
    const int s = (int)(clock[1] % 2);
    for (int f = 0; f < 3; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(field(h, s, f), body + 96 + (size_t)f * h->cells * 4, (size_t)h->cells * 4,
                                    cudaMemcpyHostToDevice, h->stream));
    VF_TRY_CUDA(cudaMemcpyAsync(h->small.ptr, small, sizeof small, cudaMemcpyHostToDevice, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    memcpy(h->host_params, p, sizeof p);
    h->clock_now = clock[0];
    h->dispatched = clock[1];
    h->total_steps = clock[2];
    h->last_step = clock[3];
    h->clock_outstanding = 0;
    return VF_OK;
}

int32_t vf_swe_set_tile_width(vf_swe* h, int32_t width) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    VF_REQUIRE(width == 0 || width == 32 || width == 64, VF_EINVAL,
               "64 (tiles' height by the grid's size), 32 (4 rows) or 0 (16 rows), got %d", width);
    h->tile_w = width;
    return VF_OK;
}

int32_t vf_swe_tile_width(const vf_swe* h) { return h ? h->tile_w : 0; }

int32_t vf_swe_set_exact(vf_swe* h, int32_t on) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    h->exact = on != 0;
    return VF_OK;
}

int32_t vf_swe_exact(const vf_swe* h) { return h && h->exact ? 1 : 0; }

int32_t vf_swe_set_overlap(vf_swe* h, int32_t on) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    h->pdl = on != 0;
    return VF_OK;
}

int32_t vf_swe_write_budget(vf_swe* h, int32_t slot, int32_t ticks) {
    VF_REQUIRE(h && (slot == 0 || slot == 1), VF_EINVAL, "budget slot is 0 or 1");
    return write_budget(h, slot, ticks);
}

int32_t vf_swe_read_budget(vf_swe* h, int32_t slot, int32_t* ticks) {
    VF_REQUIRE(h && ticks && (slot == 0 || slot == 1), VF_EINVAL, "budget slot is 0 or 1");
    uint32_t st = 0;
    int32_t rc = read_budget(h, slot, ticks, &st);
    return rc ? rc : status_error(h, st);
}

int32_t vf_swe_diagnostics(vf_swe* h, double g, double dry, double dt, double dx, double dy, double out[9]) {
    VF_REQUIRE(h && out, VF_EINVAL, "null argument");
    const int s = (int)(h->dispatched % 2);
    const int blocks = 1184;
    k_swe_diag<<<blocks, 256, 0, h->stream>>>(field(h, s, 0), field(h, s, 1), field(h, s, 2), h->cells,
                                              g, dry,
                                              h->diag.as<DiagPart>());
    VF_CHECK_LAUNCH();
    std::vector<DiagPart> parts(blocks);
    VF_TRY_CUDA(cudaMemcpyAsync(parts.data(), h->diag.ptr, sizeof(DiagPart) * blocks, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    DiagPart t{0.0, INFINITY, 0.0, 0.0, 0.0, 0.0, 0, 0, 0};
    for (const DiagPart& p : parts) {
        t.volume += p.volume;
        t.min_depth = std::fmin(t.min_depth, p.min_depth);
        t.max_depth = std::fmax(t.max_depth, p.max_depth);
        t.max_speed = std::fmax(t.max_speed, p.max_speed);
        t.max_froude = std::fmax(t.max_froude, p.max_froude);
        t.max_wave = std::fmax(t.max_wave, p.max_wave);
        t.non_finite += p.non_finite;
        t.negative += p.negative;
        t.wet += p.wet;
    }
    out[0] = t.volume * dx * dy;
    out[1] = t.wet == 0 ? 0 : t.min_depth;
    out[2] = t.max_depth;
    out[3] = t.max_speed;
    out[4] = t.max_froude;
    out[5] = t.max_wave * dt / std::fmin(dx, dy);
    out[6] = t.non_finite;
    out[7] = t.negative;
    out[8] = t.wet;
    return VF_OK;
}

void* vf_swe_stream(vf_swe* h) { return h ? (void*)h->stream : nullptr; }

int32_t vf_swe_profile(vf_swe* h, int32_t enable) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    h->prof.reset();
    h->prof.on = enable != 0;
    return VF_OK;
}

int32_t vf_swe_profile_read(vf_swe* h, int32_t index, char* name, size_t cap, double* total_ms, int64_t* launches) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    return h->prof.read(index, name, cap, total_ms, launches);
}

int64_t vf_swe_launches(const vf_swe* h) { return h ? h->prof.launches : 0; }

int32_t vf_swe_on_gpu(const vf_swe* h) { return h ? 1 : 0; }

void vf_swe_destroy(vf_swe* h) {
    if (!h) return;
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (DeviceBuffer* b : {&h->state[0], &h->state[1], &h->small, &h->status, &h->diag}) b->release();
    if (h->host_words) cudaFreeHost(h->host_words);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}


// ------------------------------------------------------------------ the state on the device

int32_t vf_swe_state(vf_swe* h, float** hcell, float** hu, float** hv) {
    VF_REQUIRE(h && hcell && hu && hv, VF_EINVAL, "null argument");
    const int s = (int)(h->dispatched % 2);
    *hcell = field(h, s, 0);
    *hu = field(h, s, 1);
    *hv = field(h, s, 2);
    return VF_OK;
}

int32_t vf_swe_measure_speed(vf_swe* h) {
    VF_REQUIRE(h, VF_EINVAL, "null handle");
    const int s = (int)(h->dispatched % 2);
    int* slot = speed_slot(h, (int)(h->dispatched % 3));
    VF_TRY_CUDA(cudaMemsetAsync(slot, 0, 4, h->stream));
    const int most = sm_count() * 8, ones = div_up(h->cells, 256);
    if (ones <= 2 * sm_count())
        VF_LAUNCH(h->prof, "k_swe_speed", h->stream, k_swe_speed<1>, ones, 256, 0, field(h, s, 0), field(h, s, 1), field(h, s, 2),
                  h->cells, params_ptr(h), slot);
    else
        VF_LAUNCH(h->prof, "k_swe_speed", h->stream, k_swe_speed<SPEED_CELLS>, std::min(div_up(h->cells, 256 * SPEED_CELLS), most),
                  256, 0, field(h, s, 0), field(h, s, 1), field(h, s, 2), h->cells, params_ptr(h), slot);
    return VF_OK;   // the next dispatch, on the same stream, reads the word
}

namespace {

// The three current fields of a handle as a device array of pointers (a small upload on the handle's stream).
struct FieldPtrs {
    DeviceBuffer buf;
    int32_t make(vf_swe* h) {
        const int s = (int)(h->dispatched % 2);
        float* p[3] = {field(h, s, 0), field(h, s, 1), field(h, s, 2)};
        int32_t rc = buf.alloc(sizeof p);
        if (rc) return rc;
        VF_TRY_CUDA(cudaMemcpyAsync(buf.ptr, p, sizeof p, cudaMemcpyHostToDevice, h->stream));
        return VF_OK;
    }
};

}  // namespace

int32_t vf_swe_restrict(vf_swe* fine, vf_swe* coarse) {
    VF_REQUIRE(fine && coarse, VF_EINVAL, "null handle");
    VF_REQUIRE(fine->nx == 2 * coarse->nx && fine->ny == 2 * coarse->ny, VF_EINVAL,
               "a %d x %d grid restricts to %d x %d, not %d x %d", fine->nx, fine->ny, fine->nx / 2, fine->ny / 2,
               coarse->nx, coarse->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(fine->stream));
    FieldPtrs f, c;
    int32_t rc;
    if ((rc = f.make(fine)) || (rc = c.make(coarse))) return rc;
    VF_TRY_CUDA(cudaStreamSynchronize(fine->stream));
    VF_LAUNCH(coarse->prof, "k_swe_restrict", coarse->stream, k_swe_restrict, div_up(coarse->cells, 256), 256, 0,
              f.buf.as<const float*>(), fine->nx, 0, 0, c.buf.as<float*>(), coarse->nx, 0, 0, coarse->nx, coarse->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(coarse->stream));
    return vf_swe_measure_speed(coarse);
}

int32_t vf_swe_prolong(vf_swe* coarse, int32_t x0, int32_t y0, vf_swe* fine) {
    VF_REQUIRE(fine && coarse, VF_EINVAL, "null handle");
    VF_REQUIRE(fine->nx % 2 == 0 && fine->ny % 2 == 0, VF_EINVAL, "a patch of even size, got %d x %d", fine->nx, fine->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(coarse->stream));
    FieldPtrs f, c;
    int32_t rc;
    if ((rc = f.make(fine)) || (rc = c.make(coarse))) return rc;
    VF_TRY_CUDA(cudaStreamSynchronize(coarse->stream));
    VF_LAUNCH(fine->prof, "k_swe_prolong", fine->stream, k_swe_prolong, div_up(fine->cells, 256), 256, 0,
              c.buf.as<const float*>(), coarse->nx, coarse->ny, x0, y0, f.buf.as<float*>(), fine->nx, fine->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(fine->stream));
    return vf_swe_measure_speed(fine);
}

int32_t vf_swe_restrict_patch(vf_swe* fine, int32_t fx0, int32_t fy0, vf_swe* coarse, int32_t x0, int32_t y0,
                              int32_t nx, int32_t ny) {
    VF_REQUIRE(fine && coarse, VF_EINVAL, "null handle");
    VF_REQUIRE(nx >= 1 && ny >= 1 && fx0 >= 0 && fy0 >= 0 && fx0 + 2 * nx <= fine->nx && fy0 + 2 * ny <= fine->ny,
               VF_EINVAL, "%d x %d coarse cells from fine cell (%d, %d) leave the %d x %d patch", nx, ny, fx0, fy0,
               fine->nx, fine->ny);
    VF_REQUIRE(x0 >= 0 && y0 >= 0 && x0 + nx <= coarse->nx && y0 + ny <= coarse->ny, VF_EINVAL,
               "coarse cells [%d, %d) x [%d, %d) leave the %d x %d grid", x0, x0 + nx, y0, y0 + ny, coarse->nx, coarse->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(fine->stream));
    FieldPtrs f, c;
    int32_t rc;
    if ((rc = f.make(fine)) || (rc = c.make(coarse))) return rc;
    VF_TRY_CUDA(cudaStreamSynchronize(fine->stream));
    VF_LAUNCH(coarse->prof, "k_swe_restrict", coarse->stream, k_swe_restrict, div_up((int64_t)nx * ny, 256), 256, 0,
              f.buf.as<const float*>(), fine->nx, fx0, fy0, c.buf.as<float*>(), coarse->nx, x0, y0, nx, ny);
    VF_TRY_CUDA(cudaStreamSynchronize(coarse->stream));
    return VF_OK;
}

int32_t vf_swe_copy_state(vf_swe* dst, vf_swe* src) {
    VF_REQUIRE(dst && src, VF_EINVAL, "null handle");
    VF_REQUIRE(dst->nx == src->nx && dst->ny == src->ny, VF_EINVAL, "grids differ: %d x %d and %d x %d", dst->nx,
               dst->ny, src->nx, src->ny);
    VF_TRY_CUDA(cudaStreamSynchronize(src->stream));
    const int sd = (int)(dst->dispatched % 2), ss = (int)(src->dispatched % 2);
    for (int f = 0; f < 3; f++)
        VF_TRY_CUDA(cudaMemcpyAsync(field(dst, sd, f), field(src, ss, f), (size_t)src->cells * 4, cudaMemcpyDeviceToDevice,
                                    dst->stream));
    return vf_swe_measure_speed(dst);
}

int32_t vf_swe_jump_indicator(vf_swe* h, int32_t tile, float* out, int32_t ntiles) {
    VF_REQUIRE(h && out && tile >= 1, VF_EINVAL, "null argument or tile < 1");
    const int tx = (h->nx + tile - 1) / tile, ty = (h->ny + tile - 1) / tile;
    VF_REQUIRE(ntiles == tx * ty, VF_EINVAL, "%d tiles of %d cells cover the grid, got %d", tx * ty, tile, ntiles);
    DeviceBuffer d;
    int32_t rc = d.alloc((size_t)ntiles * 4);
    if (rc) return rc;
    VF_TRY_CUDA(cudaMemsetAsync(d.ptr, 0, (size_t)ntiles * 4, h->stream));
    const int s = (int)(h->dispatched % 2);
    VF_LAUNCH(h->prof, "k_swe_jump", h->stream, k_swe_jump, div_up(h->cells, 256), 256, 0, field(h, s, 0), h->nx, h->ny,
              tile, tx, h->host_params[4], d.as<int>());
    VF_TRY_CUDA(cudaMemcpyAsync(out, d.ptr, (size_t)ntiles * 4, cudaMemcpyDeviceToHost, h->stream));
    VF_TRY_CUDA(cudaStreamSynchronize(h->stream));
    return VF_OK;
}

}  // extern "C"
