// sl_tile_mixed.cuh -- the double-float mixed form's pairs of one 32 x 32
// tile with the close pairs listed, shared by the one-column pair kernel of
// small systems and write steps (sl_step_mixed.cu) and the batched solver's
// pair-tile pass (sl_batch_mixed.cu).
//
// One warp; lane b holds column sphere b, the rows are in shared memory, and
// at step k of the sweep lane b takes the pair (row (b + k) mod 32, column b).
// Nearly all pairs are far apart and take a short FP32 path.  The others --
// closer than far_sq, contacts among them -- are found before the sweep,
// packed into a list and evaluated one per lane, and the sweep only fetches
// their forces: evaluated inside the sweep, every step with a close lane held
// the warp for that lane's path (close ~150 instructions, a contact several
// microseconds), and its code, twice unrolled, did not fit the instruction
// cache.  The order in which forces are added is the sweep's either way.
//
// Finding them costs a distance test per pair; a tile whose
// blocks' bounding boxes are further apart than the threshold skips it, which
// is half of the tiles of the batch's Z-ordered spheres.
#pragma once
#include "sl_device.cuh"
#include "sl_df.cuh"
#include "sl_f32x2.cuh"
#include "sl_pair_mixed.cuh"

#include <type_traits>

// What bounds it (GB300, ncu): at 20 warps per SM the shared-memory pipe at 75%,
// beside issue at 70%; with an instance per CTA (16 warps) latency, issue 46%.
// So the sweep takes two steps at a time in packed FP32
// arithmetic, and in tiles of one radius reads 24 bytes of a row instead of
// 32.  512 collisions of up to 2400 spheres, whole instances at 512 threads:
// 1.16 ms per step with the close path in the sweep, 1.03 listed.
namespace sl {
namespace mt {

using f2::F32x2;
using f2::add2;
using f2::fma2;
using f2::mul2;
using f2::pair2;
using f2::split2;

// Rows in shared memory, kRow floats each (16-byte loads of 32 different rows
// fall in distinct banks).  Two steps of the sweep are taken at once, so row r
// holds its own values beside row r + 1's (mod 32):
//   [0..3]   -hi x of r, r + 1, -hi y of r, r + 1   (scaled positions)
//   [4..7]   -hi z, scaled radius
//   [8..11]  -lo x, -lo y
//   [12..15] -lo z, c_vdw R^3
//   [16..19] row r's other values, the users'
constexpr int kRow = 20;

struct Row {
    float x, y, z, R, xl, yl, zl, c;
};

// Lane's row, and its neighbour's beside it, as whole 16-byte stores
__device__ __forceinline__ void put_row(float* rows, int lane, const Row& v, const float4& other)
{
    const int nxt = (lane + 1) & 31;
    const auto next = [nxt](float f) { return __shfl_sync(0xffffffffu, f, nxt); };
    float4* w = reinterpret_cast<float4*>(rows + lane * kRow);
    w[0] = make_float4(-v.x, -next(v.x), -v.y, -next(v.y));
    w[1] = make_float4(-v.z, -next(v.z), v.R, next(v.R));
    w[2] = make_float4(-v.xl, -next(v.xl), -v.yl, -next(v.yl));
    w[3] = make_float4(-v.zl, -next(v.zl), v.c, next(v.c));
    w[4] = other;
}

// 16 bytes, or only the first 8 of them: shared-memory bandwidth is what the
// sweep takes most of
__device__ __forceinline__ void load_half(float4& q, const float* w, bool half)
{
    if (half) {
        const float2 h = *reinterpret_cast<const float2*>(w);
        q = make_float4(h.x, h.y, 0.0f, 0.0f);
    } else {
        q = *reinterpret_cast<const float4*>(w);
    }
}

__device__ __forceinline__ Row get_row(const float* rows, int r)
{
    const float* w = rows + r * kRow;
    return {-w[0], -w[2], -w[4], w[6], -w[8], -w[10], -w[12], w[14]};
}

// List entries: all close pairs of four steps at least
constexpr int kCap = 128;

// VALUES floats per entry: the force on the row sphere, then the user's
template <int VALUES>
struct List {
    float v[kCap][VALUES];
    uint16_t pair[kCap];  // row << 5 | column
};

// A lane's column sphere
struct Col {
    float x, y, z, xl, yl, zl, R, R3;
    bool valid;
};

// The pair's displacement, |r|^2 and far force: vdW without a square root, for
// |r| >= 1.25 (Ra + Rb) or more, h = |r| - Ra - Rb above the clamp h_min:
// Ra^3 Rb^3 (h + Ra + Rb) / (S^2 T^2) along r/|r| (ColliderSingleCore.cpp:
// 205-226) with h + Ra + Rb = |r|, S = |r|^2 - (Ra + Rb)^2, T = |r|^2 - (Ra -
// Rb)^2.
struct Far {
    float rx, ry, rz, d2, sum2, fr;  // fr: |F| / |r|
};

__device__ __forceinline__ Far far_pair(const Row& q, const Col& c)
{
    Far f;
    f.rx = (c.x - q.x) + (c.xl - q.xl);
    f.ry = (c.y - q.y) + (c.yl - q.yl);
    f.rz = (c.z - q.z) + (c.zl - q.zl);
    f.d2 = fmaf(f.rx, f.rx, fmaf(f.ry, f.ry, f.rz * f.rz));
    const float sumR = q.R + c.R, difR = q.R - c.R;
    f.sum2 = sumR * sumR;
    const float P = (f.d2 - f.sum2) * fmaf(-difR, difR, f.d2);
    f.fr = (q.c * c.R3) * rcp_approx(P * P);
    return f;
}

// Order-preserving map of float bits to int, and back
__device__ __forceinline__ int ord(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float unord(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
__device__ __forceinline__ float warp_min(float f) { return unord(__reduce_min_sync(0xffffffffu, ord(f))); }
__device__ __forceinline__ float warp_max(float f) { return unord(__reduce_max_sync(0xffffffffu, ord(f))); }

// Steps k at which the lane's pair is close, with the lo parts as in the sweep:
// the search of tiles so far from the origin that the hi parts alone would take
// many more pairs for close.  Out of line: the usual search's code stays as it is.
static __device__ __noinline__ uint32_t near_far_from_origin(const float* rows, const Col col, float far_sq)
{
    const int lane = threadIdx.x & 31;
    const F32x2 cx = pair2(col.x, col.x), cy = pair2(col.y, col.y), cz = pair2(col.z, col.z);
    const F32x2 cxl = pair2(col.xl, col.xl), cyl = pair2(col.yl, col.yl), czl = pair2(col.zl, col.zl);
    uint32_t near = 0;
#pragma unroll 2
    for (int k = 0; k < 32; k += 2) {
        const float* w = rows + ((lane + k) & 31) * kRow;
        const float4 q0 = *reinterpret_cast<const float4*>(w);
        const float4 q1 = *reinterpret_cast<const float4*>(w + 4);
        const float4 q2 = *reinterpret_cast<const float4*>(w + 8);
        const float2 q3 = *reinterpret_cast<const float2*>(w + 12);
        const F32x2 rx = add2(add2(cx, pair2(q0.x, q0.y)), add2(cxl, pair2(q2.x, q2.y)));
        const F32x2 ry = add2(add2(cy, pair2(q0.z, q0.w)), add2(cyl, pair2(q2.z, q2.w)));
        const F32x2 rz = add2(add2(cz, pair2(q1.x, q1.y)), add2(czl, pair2(q3.x, q3.y)));
        const float2 d2 = split2(fma2(rx, rx, fma2(ry, ry, mul2(rz, rz))));
        const float s0 = q1.z + col.R, s1 = q1.w + col.R;
        if (!(d2.x > far_sq * (s0 * s0))) near |= 1u << k;
        if (!(d2.y > far_sq * (s1 * s1))) near |= 2u << k;
    }
    return near;
}

// The pairs of one tile.  rows: 32 kRow floats; valid row r: r < nA; diag: row
// and column blocks are one (pairs with lane < r).  close(q, row, col, pe,
// pe_far) evaluates list entry q -- whatever its distance -- into list.v[q]:
// the force on the row sphere, then the user's values; taken(q, row) is called
// in the sweep's order, by the column's lane, when entry q's force is added.  a:
// the row sums, lane l's of row l; b: the lane's column sums.
template <bool WRITE, int VALUES, class Close, class Taken>
__device__ __forceinline__ void tile(const float* rows, List<VALUES>& list, const Col& col, int nA, bool diag,
                                     float far_sq, Close&& close, Taken&& taken, float (&a)[3], float (&b)[3],
                                     double& pe, df::Sum& pe_far)
{
    const int lane = threadIdx.x & 31;
    const int nxt = (lane + 1) & 31;
    const Row mine = get_row(rows, lane);
    const bool rvalid = lane < nA;
    const float R0 = rows[6];
    const bool uni = __all_sync(0xffffffffu, (!rvalid || mine.R == R0) && (!col.valid || col.R == R0));
    const float u_sum2 = (R0 + R0) * (R0 + R0), u_crr = rows[14] * (R0 * R0 * R0);

    // Close pairs, by the hi parts alone: a component of r is then off by at
    // most 2^-23 of the largest coordinate and 2^-24 of itself, |r| by four
    // times that; a pair within the margin is listed too.  Where the coordinates
    // make that a twentieth of the reach the lo parts are added (us per step at 0 /
    // 1e6 / 1e7 radii from the origin, N=1000: hi parts alone 20.5 / 24.7 / 36.6,
    // here 20.5 / 20.6 / 20.8).
    uint32_t near = 0;
    bool any = diag, fine;
    float margin;
    {
        const float inf = __int_as_float(0x7f800000);
        const float lo[3] = {warp_min(rvalid ? mine.x : inf), warp_min(rvalid ? mine.y : inf),
                             warp_min(rvalid ? mine.z : inf)};
        const float hi[3] = {warp_max(rvalid ? mine.x : -inf), warp_max(rvalid ? mine.y : -inf),
                             warp_max(rvalid ? mine.z : -inf)};
        const float Rmax = warp_max(fmaxf(rvalid ? mine.R : 0.0f, col.valid ? col.R : 0.0f));
        const float cx = fmaxf(fmaxf(fabsf(col.x), fabsf(col.y)), fabsf(col.z));
        float X = warp_max(col.valid ? cx : 0.0f);
#pragma unroll
        for (int c = 0; c < 3; ++c) X = fmaxf(X, fmaxf(fabsf(lo[c]), fabsf(hi[c])));
        const float reach = sqrtf(far_sq) * 2.0f * Rmax * 1.0001f;
        const float delta = X * 4.8e-7f + reach * 4.8e-7f;  // 2^-21: four times 2^-23
        margin = (2.0f * reach + delta) * delta * 1.0001f;
        fine = X * 4.8e-7f > 0.05f * reach;
        // the column spheres against the rows' box
        const float gx = fmaxf(fmaxf(lo[0] - col.x, col.x - hi[0]), 0.0f);
        const float gy = fmaxf(fmaxf(lo[1] - col.y, col.y - hi[1]), 0.0f);
        const float gz = fmaxf(fmaxf(lo[2] - col.z, col.z - hi[2]), 0.0f);
        const float g2 = fmaf(gx, gx, fmaf(gy, gy, gz * gz));
        any = __any_sync(0xffffffffu, diag || (col.valid && !(g2 > (reach + delta) * (reach + delta))));
    }
    if (any && fine)
        near = near_far_from_origin(rows, col, far_sq);
    else if (any) {
        const float u_thr = fmaf(far_sq, u_sum2, margin);
        // (unrolled eight times: 512 collisions 26.1 ms, twice 25.8; 64 of them in lockstep 5.18, 5.07)
        const F32x2 cx = pair2(col.x, col.x), cy = pair2(col.y, col.y), cz = pair2(col.z, col.z);
#pragma unroll 2
        for (int k = 0; k < 32; k += 2) {
            const float* w = rows + ((lane + k) & 31) * kRow;
            const float4 q0 = *reinterpret_cast<const float4*>(w);
            float4 q1;
            load_half(q1, w + 4, uni);
            const F32x2 dx = add2(cx, pair2(q0.x, q0.y)), dy = add2(cy, pair2(q0.z, q0.w)),
                        dz = add2(cz, pair2(q1.x, q1.y));
            const float2 d2 = split2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))));
            float t0 = u_thr, t1 = u_thr;
            if (!uni) {
                const float s0 = q1.z + col.R, s1 = q1.w + col.R;
                t0 = fmaf(far_sq, s0 * s0, margin);
                t1 = fmaf(far_sq, s1 * s1, margin);
            }
            if (!(d2.x > t0)) near |= 1u << k;
            if (!(d2.y > t1)) near |= 2u << k;
        }
    }
    if (any) {
        // valid pairs only: rows r < nA, on the diagonal r > lane
        uint32_t ok = nA >= 32 ? 0xffffffffu : (1u << max(nA, 0)) - 1u;
        if (diag) ok &= ~((2u << lane) - 1u);
        ok = __funnelshift_r(ok, ok, lane);  // bit k: row (lane + k) mod 32
        near = col.valid ? near & ok : 0u;
    }

#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = b[c] = 0.0f;
    const int total = __reduce_add_sync(0xffffffffu, __popc(near));
    const int seg = total <= kCap ? 32 : 4;  // steps whose close pairs fit the list

    // two steps at a time in packed arithmetic, their forces added in turn
    auto sweep = [&](auto uni_tag, auto full_tag, int k0, int at) {
        constexpr bool UNI = decltype(uni_tag)::value, FULL = decltype(full_tag)::value;
        const F32x2 cx = pair2(col.x, col.x), cy = pair2(col.y, col.y), cz = pair2(col.z, col.z);
        const F32x2 cxl = pair2(col.xl, col.xl), cyl = pair2(col.yl, col.yl), czl = pair2(col.zl, col.zl);
        const F32x2 cR = pair2(col.R, col.R), ncR = pair2(-col.R, -col.R), cR3 = pair2(col.R3, col.R3);
        const F32x2 minus1 = pair2(-1.0f, -1.0f);
        const F32x2 usum2 = pair2(-u_sum2, -u_sum2), ucrr = pair2(u_crr, u_crr);
#pragma unroll 2
        for (int k = k0; k < k0 + seg; k += 2) {
            const float* w = rows + ((lane + k) & 31) * kRow;
            const float4 q0 = *reinterpret_cast<const float4*>(w);
            const float4 q2 = *reinterpret_cast<const float4*>(w + 8);
            float4 q1, q3;
            load_half(q1, w + 4, UNI);
            load_half(q3, w + 12, UNI);
            const F32x2 rx = add2(add2(cx, pair2(q0.x, q0.y)), add2(cxl, pair2(q2.x, q2.y)));
            const F32x2 ry = add2(add2(cy, pair2(q0.z, q0.w)), add2(cyl, pair2(q2.z, q2.w)));
            const F32x2 rz = add2(add2(cz, pair2(q1.x, q1.y)), add2(czl, pair2(q3.x, q3.y)));
            const F32x2 d2 = fma2(rx, rx, fma2(ry, ry, mul2(rz, rz)));
            F32x2 S, T = d2, crr = ucrr;  // UNI: T = |r|^2
            if (UNI) {
                S = add2(d2, usum2);
            } else {
                const F32x2 R = pair2(q1.z, q1.w);
                const F32x2 sumR = add2(R, cR), difR = add2(R, ncR);
                // the square rounded by itself, as in the other kernels: a packed product
                // is fused into a packed sum
                const float2 s = split2(sumR);
                S = add2(d2, pair2(-__fmul_rn(s.x, s.x), -__fmul_rn(s.y, s.y)));
                T = fma2(mul2(difR, minus1), difR, d2);
                crr = mul2(pair2(q3.z, q3.w), cR3);
            }
            const F32x2 P = mul2(S, T);
            const float2 PP = split2(mul2(P, P));
            const F32x2 fr = mul2(crr, pair2(rcp_approx(PP.x), rcp_approx(PP.y)));
            const float2 fx2 = split2(mul2(fr, rx)), fy2 = split2(mul2(fr, ry)), fz2 = split2(mul2(fr, rz));
            const float2 d22 = split2(d2);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int r = (lane + k + j) & 31;
                const bool valid = FULL || (col.valid && r < nA && (!diag || lane < r));
                float fx = j ? fx2.y : fx2.x, fy = j ? fy2.y : fy2.x, fz = j ? fz2.y : fz2.x;
                const bool listed = (near >> (k + j)) & 1u;
                if (listed) {
                    fx = list.v[at][0];
                    fy = list.v[at][1];
                    fz = list.v[at][2];
                    taken(at, r);
                    ++at;
                }
                if (WRITE && valid && !listed) pe_far.add(vdw_bracket(j ? d22.y : d22.x, UNI ? col.R : j ? q1.w : q1.z, col.R));
                if (!FULL && !valid) fx = fy = fz = 0.0f;
                a[0] += fx; a[1] += fy; a[2] += fz;
                b[0] += fx; b[1] += fy; b[2] += fz;
                a[0] = __shfl_sync(0xffffffffu, a[0], nxt);
                a[1] = __shfl_sync(0xffffffffu, a[1], nxt);
                a[2] = __shfl_sync(0xffffffffu, a[2], nxt);
            }
        }
    };
    const bool full = __all_sync(0xffffffffu, col.valid && nA >= 32 && !diag);
    for (int k0 = 0; k0 < 32; k0 += seg) {
        int at = 0;
        if (total) {
            const uint32_t mask = seg == 32 ? near : near & (0xfu << k0);
            const int cnt = __popc(mask);
            at = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, at, o);
                if (lane >= o) at += v;
            }
            const int n = __shfl_sync(0xffffffffu, at, 31);
            at -= cnt;
            __syncwarp();  // the last segment's entries have been taken
            int e = at;
            for (uint32_t w = mask; w; w &= w - 1)
                list.pair[e++] = (uint16_t)((((lane + __ffs(w) - 1) & 31) << 5) | lane);
            __syncwarp();
            for (int q = lane; q < n; q += 32) close(q, list.pair[q] >> 5, list.pair[q] & 31, pe, pe_far);
            __syncwarp();
        }
        if (uni) {
            if (full)
                sweep(std::true_type{}, std::true_type{}, k0, at);
            else
                sweep(std::true_type{}, std::false_type{}, k0, at);
        } else {
            if (full)
                sweep(std::false_type{}, std::true_type{}, k0, at);
            else
                sweep(std::false_type{}, std::false_type{}, k0, at);
        }
    }
}

}  // namespace mt
}  // namespace sl
