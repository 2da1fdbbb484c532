// sl_tile_exact.cuh -- the exact form's pairs of one 32 x 32 block tile
// (ColliderSingleCore.cpp:104-253 for each pair, in the reference's
// orientation A > B), shared by the single-system pair kernel (sl_step.cu)
// and the batched exact solver's pair-tile pass (sl_batch.cu).  Must be
// compiled with --fmad=false (the exact arithmetic contract).
//
// Two passes per tile.  The sweep walks the A block and evaluates every pair
// by the branch-free integer path (sl_pair_fast.cuh).  Pairs in contact, and
// pairs whose rounding that path leaves open (about 4%), are marked; after
// the sweep their (A, B) are packed into a list and evaluated 32 at a time by
// the general path, one pair per lane.  A contact costs ~10,000 cycles of
// dependent FP64 divisions and square roots: inside the sweep each row with
// one held the whole warp for that long, which set the time of small systems
// (N=96: 117 us for six tiles).
//
// What bounds it (N=5000, GB300, ncu): with every add and product on the FP64
// pipe that pipe was the limit; now no unit is -- FP64 62% of its nominal
// cycles (14 operations of a warp's 32 pairs), ALU 54%, the integer
// multiplier (fmaheavy) 58%, issue 53%, at 16 warps per SM.  Pair kernel per
// step: 0.775 ms with quotients rounded by exact remainders, 0.632 ms with
// the unpacked path's divisions alone, 0.478 ms with its products too.
#pragma once
#include "sl_device.cuh"
#include "sl_fp64_exact.cuh"
#include "sl_pair_exact.cuh"
#include "sl_pair_fast.cuh"
#include "sl_vdw_energy.cuh"

namespace sl {

// Per-warp staging of the A block (lane l holds sphere X*32+l).
struct ABlock {
    double x[kBlock], y[kBlock], z[kBlock], R[kBlock], twoR[kBlock], fourR[kBlock], cR3[kBlock], m[kBlock];
    unsigned long long rm[kBlock];
};

// Per-warp shared staging of sphere B's terms (lane = B) for four
// consecutive partners: [component][lane][4 + 1 padding] doubles, so that a
// lane's 8-byte accesses at a 40-byte stride fall in distinct banks per
// half-warp.
constexpr int kBStageRow = 5;
constexpr int kBStagePlane = kBlock * kBStageRow;
constexpr int kBStageDoubles = 3 * kBStagePlane;

// A tile may be taken in strips of 8 of its 32 rows.
constexpr int kStripRows = 8, kStrips = kBlock / kStripRows;

// One warp's shared memory.  The list of marked pairs (at most 32 x 32
// entries of 16 bits) takes the B staging's place after the sweep.
struct TileScratch {
    ABlock ab;
    double bstage[kBStageDoubles];
    uint32_t rowc[kBlock], colc[kBlock];  // contact bits found by the general path
};
static_assert(sizeof(double) * kBStageDoubles >= kBlock * kBlock * sizeof(uint16_t), "list fits in the staging");

// Where a tile's potentials (write steps) are added up: nowhere; with the
// forces; or the contacts' with the forces and the others' in work items of
// their own (strip_potentials).
enum PeMode { kNoPe = 0, kPeInline = 1, kPeApart = 2 };

// One pair by the general path: rounds every quotient and root by its exact
// remainder (sl_fp64_exact.cuh), with the hardware operations behind it, for
// any operands; contact or not.
template <int PE>
__device__ __forceinline__ bool general_pair(const System& s, const ABlock& ab, int X, int a, int B, double& pe)
{
    const size_t plane = (size_t)s.npad * s.npad;
    const int A = X * kBlock + a;
    const double Ra = ab.R[a], Rb = s.R[B], twoRb = s.twoR[B], mb = s.m[B];
    const double sumRaRb = Ra + Rb;                                                   // :104
    const double rx = s.pos.c[0][B] - ab.x[a], ry = s.pos.c[1][B] - ab.y[a], rz = s.pos.c[2][B] - ab.z[a];  // :105
    const double d2 = rx * rx + ry * ry + rz * rz;
    int p;
    unsigned long long F;
    const unsigned long long Yr = rsqrt_fix(d2, p, F);            // ~1/sqrt(d2), integer pipe
    const double dist = sqrt_fix(d2, F, Yr, p);                   // :107, RN(sqrt)
    const double overlap = sumRaRb - dist;                        // :110
    // the comparisons of the step are made on the bit patterns (integer
    // pipe): for doubles of one sign the integer order is the FP order; NaN
    // is excluded explicitly
    const long long ob = __double_as_longlong(overlap);
    const bool contact = ob > 0 && ob <= 0x7ff0000000000000ll;    // overlap > 0
    double fx, fy, fz;
    if (contact) {
        const ContactIn in = gather_contact(s, A, B);
        const ContactOut o = contact_pair_exact<PE != kNoPe>(in, s.mat, rx, ry, rz, dist, overlap, Ra, Rb, ab.twoR[a],
                                                       twoRb, ab.fourR[a], ab.cR3[a]);
        fx = o.fx; fy = o.fy; fz = o.fz;
        const double im_a = s.inv_moi[A], mo_a = s.moi[A];
        const double im_b = s.inv_moi[B], mo_b = s.moi[B];
        double* ta = s.torqbuf + (size_t)A * s.npad + B;   // :187
        double* tb = s.torqbuf + (size_t)B * s.npad + A;   // :188
        ta[0] = div_by_recip(o.tax, mo_a, im_a);
        ta[plane] = div_by_recip(o.tay, mo_a, im_a);
        ta[2 * plane] = div_by_recip(o.taz, mo_a, im_a);
        tb[0] = div_by_recip(o.tbx, mo_b, im_b);
        tb[plane] = div_by_recip(o.tby, mo_b, im_b);
        tb[2 * plane] = div_by_recip(o.tbz, mo_b, im_b);
        if (PE != kNoPe) pe += o.pe;
    } else {
        long long hb = ob & 0x7fffffffffffffffll;                  // :211-215 |overlap|
        const long long h_min_bits = __double_as_longlong(s.mat.h_min);
        if (hb < h_min_bits) hb = h_min_bits;                      // h < h_min (NaN stays NaN)
        const double h = __longlong_as_double(hb);
        const double coef = vdw_coef_fix(h, Ra, Rb, ab.twoR[a], twoRb, ab.fourR[a], ab.cR3[a]);
        fx = coef * div_by_rsqrt(rx, dist, Yr, p);                    // :221-227
        fy = coef * div_by_rsqrt(ry, dist, Yr, p);
        fz = coef * div_by_rsqrt(rz, dist, Yr, p);
        if (PE == kPeInline) pe += vdw_energy_far_df(s.mat.Ha, h, Ra, Rb, ab.twoR[a]);  // :239
    }
    // :249-250 -- acc[A] += F/m[A]; acc[B] -= F/m[B] (stored negated)
    const double ma = ab.m[a];
    const unsigned long long rma = ab.rm[a], rmb = s.rm[B];
    double* pa = s.pairbuf + (size_t)A * s.npad + B;
    double* pb = s.pairbuf + (size_t)B * s.npad + A;
    __stcs(pa, div_by_fixed<false>(fx, ma, rma));
    __stcs(pa + plane, div_by_fixed<false>(fy, ma, rma));
    __stcs(pa + 2 * plane, div_by_fixed<false>(fz, ma, rma));
    __stcs(pb, div_by_fixed<false, true>(fx, mb, rmb));
    __stcs(pb + plane, div_by_fixed<false, true>(fy, mb, rmb));
    __stcs(pb + 2 * plane, div_by_fixed<false, true>(fz, mb, rmb));
    return contact;
}

// Packs the pairs of a tile given by the lanes' masks (lane's bit a = pair
// (32X + a, 32Y + lane)) into the list, entry a << 5 | lane; their number.
__device__ __forceinline__ int pack_list(TileScratch& ws, uint32_t marked)
{
    const int lane = threadIdx.x & 31;
    uint16_t* list = reinterpret_cast<uint16_t*>(ws.bstage);
    const int cnt = __popc(marked);
    int at = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31);
    at -= cnt;
    __syncwarp();  // the staging's last reads are done
    for (uint32_t w = marked; w; w &= w - 1) list[at++] = (uint16_t)(((__ffs(w) - 1) << 5) | lane);
    __syncwarp();
    return total;
}

// The marked pairs of a tile, packed and evaluated one per lane; ws.rowc and
// ws.colc get the contacts.  Out of line: the sweep's registers are dead here.
template <int PE>
__device__ __noinline__ double general_pairs(const System& s, TileScratch& ws, int X, int Y, uint32_t marked)
{
    const int lane = threadIdx.x & 31;
    double pe = 0;
    const uint16_t* list = reinterpret_cast<const uint16_t*>(ws.bstage);
    ws.rowc[lane] = 0;
    ws.colc[lane] = 0;
    const int total = pack_list(ws, marked);
    for (int e = lane; e < total; e += 32) {
        const int a = list[e] >> 5, b = list[e] & 31;
        if (general_pair<PE>(s, ws.ab, X, a, Y * kBlock + b, pe)) {
            atomicOr(&ws.rowc[a], 1u << b);
            atomicOr(&ws.colc[b], 1u << a);
        }
    }
    __syncwarp();
    return pe;
}

// The van der Waals potential of a write step's near pairs (settled by the
// sweep, but too close for vdw_energy_series), packed and evaluated one per
// lane as well: the closed form is ~3000 cycles of dependent FP64 divisions
// and a logarithm, and a row of a dense cluster nearly always has one.
// N=201 (112 strips of 8 rows, one warp each), pair kernel of a write step:
// 63.5 -> 57.3 us.
static __device__ __noinline__ double near_potentials(const System& s, TileScratch& ws, int X, int Y, uint32_t near)
{
    const ABlock& ab = ws.ab;
    double pe = 0;
    const uint16_t* list = reinterpret_cast<const uint16_t*>(ws.bstage);
    const int total = pack_list(ws, near);
    for (int e = threadIdx.x & 31; e < total; e += 32) {
        const int a = list[e] >> 5, B = Y * kBlock + (list[e] & 31);
        const double Ra = ab.R[a], Rb = s.R[B];
        const double rx = s.pos.c[0][B] - ab.x[a], ry = s.pos.c[1][B] - ab.y[a], rz = s.pos.c[2][B] - ab.z[a];
        const double h = fabs((Ra + Rb) - sqrt(rx * rx + ry * ry + rz * rz));
        pe += vdw_energy(s.mat.Ha, h < s.mat.h_min ? s.mat.h_min : h, Ra, Rb, ab.twoR[a]);  // :239
    }
    __syncwarp();
    return pe;
}

// The potentials of the pairs out of contact in rows a0 .. a1 - 1 of a tile,
// ws.ab loaded (kPeApart).
__device__ __forceinline__ double strip_potentials(const System& s, TileScratch& ws, int X, int Y, int lane, int a0,
                                                   int a1)
{
    const ABlock& ab = ws.ab;
    const int B = Y * kBlock + lane;
    const double bx = s.pos.c[0][B], by = s.pos.c[1][B], bz = s.pos.c[2][B], Rb = s.R[B];
    double pe = 0;
    uint32_t near = 0;
#pragma unroll 2
    for (int a = a0; a < a1; ++a) {
        const double Ra = ab.R[a];
        const double rx = bx - ab.x[a], ry = by - ab.y[a], rz = bz - ab.z[a];
        const double overlap = (Ra + Rb) - sqrt(rx * rx + ry * ry + rz * rz);
        if (B < s.n && (X != Y || lane < a) && !(overlap > 0)) {
            double h = fabs(overlap);
            if (h < s.mat.h_min) h = s.mat.h_min;
            const VdwArg v = vdw_arg(h, Ra, Rb, ab.twoR[a]);
            if (v.far()) pe += vdw_energy_series(s.mat.Ha, v);
            else near |= 1u << a;
        }
    }
    if (__any_sync(0xffffffffu, near != 0u)) pe += near_potentials(s, ws, X, Y, near);
    return pe;
}

// The tile (X, Y) for lane = sphere B = 32Y + lane, partners A = 32X + a for
// a in [a0, a1) (a0 a multiple of 4): terms to pairbuf and torqbuf, contact
// bits to rowbits (row A = 32X + lane) and colbits (row B), PE (write steps)
// to pe.  ws.ab must hold the A block.
//
// Off the diagonal, sphere B's terms -- which go to B's own row of pairbuf, a
// different row per lane -- are gathered four at a time in ws.bstage and
// written as whole 32-byte sectors (two 16-byte stores per component) instead
// of one 8-byte store per term from 32 rows at once; partners past the last
// sphere are written as +0.0, the value those entries hold anyway.  The
// diagonal tile stores every term as it is computed, because its B-side and
// A-side terms share rows.
//
// UNI: all 64 spheres have one radius and one mass (monodisperse clusters).
// The radius products are formed once, and sphere B's term is the negation
// of sphere A's (RN(-x) = -RN(x)).  Every remaining operation is the general
// form's, in its order.
//
// ROWS rows at a time (1, 2 or 4): their chains side by side, where a warp has
// its SM sub-partition to itself.  Rows past a1 are computed from the block's
// padding and dropped.
template <int PE, bool UNI, int ROWS, bool ZEROS>
__device__ __forceinline__ void sweep_pairs(const System& s, TileScratch& ws, int X, int Y, int lane, int a0, int a1,
                                            double bx, double by, double bz, const pf::Sphere& sb,
                                            const pf::Uniform& un, bool bvalid, double& pe, uint32_t& marked,
                                            uint32_t& near)
{
    const ABlock& ab = ws.ab;
    const size_t plane = (size_t)s.npad * s.npad;
    const int B = Y * kBlock + lane;
    const long long h_min_bits = __double_as_longlong(s.mat.h_min);
    const bool staged = X != Y;
    double* my_stage = ws.bstage + lane * kBStageRow;
    double* rowA = s.pairbuf + (size_t)(X * kBlock) * s.npad + B;  // + a*npad: term for A
    double* rowB = s.pairbuf + (size_t)B * s.npad + X * kBlock;    // + a: term for B
    for (int r0 = a0; r0 < a1; r0 += ROWS) {
        pf::Pair prs[ROWS];
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            const int a = r0 + k;
            pf::Sphere sa;
            if (UNI) {
                sa = sb;
            } else {
                sa.R = ab.R[a];
                sa.sR = pf::unpack(sa.R);
                sa.cR3 = ab.cR3[a];
                sa.rm = ab.rm[a];
                sa.em = pf::unpack(ab.m[a]).e;
            }
            prs[k] = pf::pair_terms<UNI, ZEROS>(bx - ab.x[a], by - ab.y[a], bz - ab.z[a], sa, sb, un, h_min_bits);
        }
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            const int a = r0 + k;
            const pf::Pair& pr = prs[k];
            const bool valid = bvalid && (X != Y || lane < a) && (ROWS == 1 || a < a1);
            // contact (overlap > 0), or a result this path does not settle: the
            // general path writes these entries after the sweep
            const bool mark = valid && (__double_as_longlong(pr.overlap) > 0 || !pr.fl.sure());
            if (mark) marked |= 1u << a;
            if (PE == kPeInline) {
                if (valid && !mark) {  // :239
                    const double Ra = UNI ? sb.R : ab.R[a];
                    const VdwArg v = vdw_arg(pr.h, Ra, sb.R, 2 * Ra);
                    if (v.far()) pe += vdw_energy_series(s.mat.Ha, v);
                    else near |= 1u << a;
                }
            }
            if (valid) {
                double* pa = rowA + (size_t)a * s.npad;
                __stcs(pa, pr.ta[0]);
                __stcs(pa + plane, pr.ta[1]);
                __stcs(pa + 2 * plane, pr.ta[2]);
                if (staged) {
                    double* st = my_stage + (a & 3);
                    st[0] = pr.tb[0];
                    st[kBStagePlane] = pr.tb[1];
                    st[2 * kBStagePlane] = pr.tb[2];
                } else {
                    double* pb = rowB + a;
                    __stcs(pb, pr.tb[0]);
                    __stcs(pb + plane, pr.tb[1]);
                    __stcs(pb + 2 * plane, pr.tb[2]);
                }
            }
        }
        static_assert(kStripRows % ROWS == 0 && ROWS <= 4, "rows r0 .. share a sector of row B");
        const int last = min(r0 + ROWS, a1) - 1;
        if (staged && bvalid && ((last & 3) == 3 || last == a1 - 1)) {
            // row B, partners q0 .. q0+3: a 32-byte aligned sector (npad and
            // 32X are multiples of 4, the buffer is 256-byte aligned)
            const int q0 = last & ~3;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double* st = my_stage + c * kBStagePlane;
                const double v0 = st[0];
                const double v1 = q0 + 1 < a1 ? st[1] : 0.0;
                const double v2 = q0 + 2 < a1 ? st[2] : 0.0;
                const double v3 = q0 + 3 < a1 ? st[3] : 0.0;
                double2* dst = reinterpret_cast<double2*>(rowB + c * plane + q0);
                __stcs(dst, make_double2(v0, v1));
                __stcs(dst + 1, make_double2(v2, v3));
            }
        }
    }
}

// Sphere i as a pair's B
__device__ __forceinline__ pf::Sphere column_sphere(const System& s, int i)
{
    const double R = s.R[i];
    return {R, pf::unpack(R), s.cR3[i], s.rm[i], pf::unpack(s.m[i]).e};
}

// The constants of a tile of one radius and one mass
__device__ __forceinline__ pf::Uniform tile_uniform(const ABlock& ab)
{
    const double R = ab.R[0];
    return {R + R, ab.fourR[0] * R, pf::unpack(ab.cR3[0] * R * R * R)};
}

// The sweep in the ZEROS form, out of line, so that the plain one's code stays as
// it is.  Systems that need it throughout (us per step, the general path for
// every such pair / here): in a plane N=1000 228 / 118, N=5000 2832 / 984; no
// cohesion N=1000 278 / 125, N=5000 3888 / 1036; a cubic lattice N=5000 1426 / 943.
struct Swept {
    double pe;
    uint32_t marked, near;
};

template <int PE, bool UNI>
__device__ __noinline__ Swept sweep_zeros(const System& s, TileScratch& ws, int X, int Y, int a0, int a1)
{
    const int lane = threadIdx.x & 31, B = Y * kBlock + lane, iB = min(B, s.n - 1);
    const pf::Uniform un = UNI ? tile_uniform(ws.ab) : pf::Uniform{0.0, 0.0, {0, 0}};
    Swept o{0.0, 0, 0};
    sweep_pairs<PE, UNI, 1, true>(s, ws, X, Y, lane, a0, a1, s.pos.c[0][iB], s.pos.c[1][iB], s.pos.c[2][iB],
                                  column_sphere(s, iB), un, B < s.n, o.pe, o.marked, o.near);
    return o;
}

// Loads sphere i into lane's place of the A block.
__device__ __forceinline__ void load_a(const System& s, ABlock& ab, int lane, int i)
{
    ab.x[lane] = s.pos.c[0][i]; ab.y[lane] = s.pos.c[1][i]; ab.z[lane] = s.pos.c[2][i];
    ab.R[lane] = s.R[i]; ab.twoR[lane] = s.twoR[i]; ab.fourR[lane] = s.fourR[i];
    ab.cR3[lane] = s.cR3[i]; ab.m[lane] = s.m[i]; ab.rm[lane] = s.rm[i];
}

// Partners a0 .. a1 - 1 of the tile (X, Y), the A block loaded: the sweep, or
// where a constant leaves the integer path's range (masses or strengths far
// from 1) the general path for every pair, then the marked pairs.
template <int PE, int ROWS = 1>
__device__ __forceinline__ void tile_pairs(const System& s, TileScratch& ws, int X, int Y, int lane, int a0, int a1,
                                           int iB, bool bvalid, double& pe, uint32_t& rowbits, uint32_t& colbits)
{
    const ABlock& ab = ws.ab;
    const double bx = s.pos.c[0][iB], by = s.pos.c[1][iB], bz = s.pos.c[2][iB];
    const double Rb = s.R[iB], mb = s.m[iB];
    const pf::Sphere sb = column_sphere(s, iB);
    const bool areal = X * kBlock + lane < s.n;  // padding takes no part in a pair
    const pf::Sphere sa{ab.R[lane], pf::unpack(ab.R[lane]), ab.cR3[lane], 0, pf::unpack(ab.m[lane]).e};
    // fit: the constants are in the integer path's range.  special: the tile takes
    // the ZEROS form of the sweep -- without cohesion or with repulsion, or where the
    // last row meets a zero displacement component (spheres in a plane or on a grid).
    // Either form is right for any row: a pair that the plain one does not settle
    // takes the general path.  One row stands for the tile because a vote in every
    // row cost the other systems up to 9% (N=5000, host step 705 -> 769 us), and one
    // vote covers both questions (two, and the force's sign in the plain form: 709;
    // this 705).
    const bool cohesive = s.mat.Ha > 0;
    const int last = max(a1 - 1, 0);
    const bool fit = (!areal || (pf::in_range(sa) && (pf::is_zero(s.mat.Ha) || pf::in_range_cR3(sa.cR3)))) &&
                     (!bvalid || pf::in_range(sb));
    const bool special = !cohesive || (bvalid && (X != Y || lane < last) &&
                                       (pf::equal(bx, ab.x[last]) || pf::equal(by, ab.y[last]) ||
                                        pf::equal(bz, ab.z[last])));
    const bool plain = __all_sync(0xffffffffu, fit && !special);
    // equality on the bit patterns (R, m > 0)
    const auto same = [](double x, double y) { return __double_as_longlong(x) == __double_as_longlong(y); };
    const double R0 = ab.R[0], m0 = ab.m[0];
    const bool uni = __all_sync(0xffffffffu, (!areal || (same(sa.R, R0) && same(ab.m[lane], m0))) &&
                                                 (!bvalid || (same(Rb, R0) && same(mb, m0))));
    uint32_t marked = 0, near = 0;
    if (!plain && !__all_sync(0xffffffffu, fit)) {
        const uint32_t all = (a1 >= 32 ? ~0u : (1u << a1) - 1u) & ~((1u << a0) - 1u);
        marked = bvalid ? (X != Y ? all : all & ~((2u << lane) - 1u)) : 0u;
    } else if (!plain) {
        const Swept o = uni ? sweep_zeros<PE, true>(s, ws, X, Y, a0, a1) : sweep_zeros<PE, false>(s, ws, X, Y, a0, a1);
        pe += o.pe;
        marked = o.marked;
        near = o.near;
    } else if (uni) {
        const pf::Uniform un = tile_uniform(ab);
        sweep_pairs<PE, true, ROWS, false>(s, ws, X, Y, lane, a0, a1, bx, by, bz, sb, un, bvalid, pe, marked, near);
    } else {
        const pf::Uniform un{0.0, 0.0, {0, 0}};
        sweep_pairs<PE, false, ROWS, false>(s, ws, X, Y, lane, a0, a1, bx, by, bz, sb, un, bvalid, pe, marked, near);
    }
    if (PE == kPeInline && __any_sync(0xffffffffu, near != 0u)) pe += near_potentials(s, ws, X, Y, near);
    rowbits = colbits = 0;
    if (__any_sync(0xffffffffu, marked != 0u)) {
        pe += general_pairs<PE>(s, ws, X, Y, marked);
        rowbits = ws.rowc[lane];
        colbits = ws.colc[lane];
        __syncwarp();
    }
}

// Contact words of an item of tile (X, Y): row A = 32X + lane gets block Y's
// bits, row B block X's; on the diagonal both describe row 32X + lane.
// strip < 0: the whole tile.  Strip w holds rows 8w .. 8w + 7: those rows'
// words, and byte w of every column's word, so that the strips' stores are
// disjoint.  On the diagonal, row i of strip w has its bytes below w from
// rowbits, byte w from both, and those above from the later strips' columns.
__device__ __forceinline__ void store_contacts(const System& s, int X, int Y, int lane, int strip, uint32_t rowbits,
                                               uint32_t colbits)
{
    static_assert(kStripRows == 8, "a strip's column bits are one byte");
    uint32_t* wa = s.cmask + (size_t)(X * kBlock + lane) * s.nb + Y;
    uint32_t* wb = s.cmask + (size_t)(Y * kBlock + lane) * s.nb + X;
    if (strip < 0) {
        if (X == Y) {
            *wa = rowbits | colbits;
        } else {
            *wa = rowbits;
            *wb = colbits;
        }
        return;
    }
    uint8_t* ba = reinterpret_cast<uint8_t*>(wa);
    const int mine = lane / kStripRows;
    if (X != Y) {
        if (mine == strip) *wa = rowbits;
        reinterpret_cast<uint8_t*>(wb)[strip] = (uint8_t)(colbits >> (8 * strip));
    } else if (mine == strip) {
        for (int k = 0; k <= strip; ++k) ba[k] = (uint8_t)((rowbits | colbits) >> (8 * k));
    } else if (mine < strip) {
        ba[strip] = (uint8_t)(colbits >> (8 * strip));
    }
}

// The first tile of T that is taken in strips.  A strip costs its share of a
// tile and ~12% more (its own blocks, and a quarter of the marked pairs in a warp
// of their own), and pays where the warps are not all busy to the end.  Of 16
// warps per SM, with T tiles (us per step, GB300, no strips against these):
//   - T up to half of them: all tiles.  The step is a warp's latency, 32 rows of
//     ~1500 cycles.  N=96 65.5 -> 30.9, N=300 69.8 -> 34.8, N=1000 111 -> 85,
//     N=1400 128 -> 115.
//   - more: as many as half the warps, the last ones, which shortens the tail:
//     N=1733 162 -> 152, N=3000 311 -> 305, N=5000 692.6 -> 688.5.
//   - a last round that is nearly full without them: none.  N=2200 (99% full):
//     199, 205 with them.
// 16 is a tuned value: large plain steps have 20 warps per SM resident, and
// counting those is no better (16 / 20: N=2400 269 / 272, N=3000 358 / 361, N=3500
// 443 / 446, N=4000 551 / 547, N=5000 795 / 785, N=7000 the same).
__host__ __device__ inline long long strip_from(long long tiles, int num_sms)
{
    const long long warps = 16LL * num_sms;
    if (2 * tiles <= warps) return 0;
    return 10 * (tiles % warps) > 9 * warps ? tiles : tiles - warps / 2;
}

}  // namespace sl
