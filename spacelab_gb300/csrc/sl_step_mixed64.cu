// sl_step_mixed64.cu -- the mixed-precision form of the step with FP64
// geometry and accumulation (SL_MODE_MIXED).
//
// What stays FP64, and where in the reference each piece sits:
//   * positions and the whole integration: drift_kernel (pass 1, shared with
//     the exact form) and pass 3 in mixed64_finish_kernel
//     (ColliderSingleCore.cpp:82-97, 263-267);
//   * the pair subtraction r = pos[B] - pos[A] (:105): the FP64 positions are
//     held as three FP32 parts (written by the drift), whose differences
//     give r rounded once to FP32 (parts::sub3, sl_parts.cuh);
//   * for pairs closer than far_sq (1.25 radii sums or more), r itself,
//     |r|^2, the squared gap g = (R_A + R_B)^2 - |r|^2, |r| and the overlap
//     R_A + R_B - |r| = g / (R_A + R_B + |r|) (:106-110) in FP64, which set the
//     contact test, the elastic force and the clamped vdW gap; and the
//     previous-step distance test that chooses kin or kout (:119-126);
//   * per-sphere force and torque accumulation: a pair's force goes into both
//     spheres' sums over the tile's 32 partners, which carry every rounding
//     error on (df::Sum3, more than FP64's 53 bits) and end as one FP64
//     partial; the partials, and contact torques, are summed in FP64
//     (:249-250, 187-188);
//   * the write-step energies: close pairs' potential in FP64, far pairs'
//     vdW bracket by the cancellation-free series (vdw_bracket, FP32) added
//     the same way, and the FP64 totals.
// FP32 does the force and torque arithmetic on the relative displacement
// r and the FP64 overlap: the vdW coefficient, elastic, gravity, sliding and
// rolling friction and the torques, in lengths scaled by 2^-len_shift.
//
// What bounds it (ncu, N=9000): the FP32 pipe at 75%, beside issue at 71%; nearly
// half of its work are the six error-free sums, the two spheres' of a component
// added in packed arithmetic.  On the FP64 pipe the subtraction
// and the sums were 9 adds a pair at 19 SM-cycles each (one narrow unit per SM),
// 171 cycles for a warp's 32 pairs, at 0.96 of that unit's rate; now it is some
// 60.  N=20000 polydisperse, 20 steps: 74.2 -> 23.1 ms with the subtraction to
// 2^-47 of the coordinates (sums one by one, unrolled twice 23.8; 3 and 5 CTAs per
// SM 25.2 and 23.9), 24.2 with it rounded once (x and y packed 24.5).
//
// Accumulation order: one warp evaluates a 32 x 32 tile in a diagonal sweep
// (lane b holds column sphere B's sum; row r's sum travels one lane down per
// step to meet its next term), so each sphere's terms from a partner block
// are added in a fixed order into one FP64 partial.
// mixed64_finish_kernel adds a sphere's partials over the partner blocks in
// ascending order.  Every order is fixed, so runs repeat bit for bit.
#include "sl_device.cuh"
#include "sl_df.cuh"
#include "sl_kernels.h"
#include "sl_pair_mixed.cuh"
#include "sl_parts.cuh"

#include <type_traits>

namespace sl {

namespace {

// Row spheres of a tile in shared memory, kRow64 floats each, so that a warp's
// 16-byte loads of 32 different rows fall in distinct banks: scaled position
// parts x, y, z and the scaled radius, the second parts and c_vdw R^3, the
// third parts.
constexpr int kRow64 = 12;
constexpr int kM64Warps = 4;
constexpr int kM64CtasPerSm = 4;  // resident CTAs per SM (the launch bounds' minimum)

// a + b + c as FP64
__device__ __forceinline__ double total(const df::Sum3& s)
{
    return f2d_bits(s.a) + (f2d_bits(s.b) + f2d_bits(s.c));
}

// One warp per lower-triangular 32 x 32 block tile (X, Y), X >= Y: column
// lane b is sphere B = 32Y + b, row r is sphere A = 32X + r (A > B).  The
// force computed for a pair is the force on A; B receives its negative.
// Writes the FP64 partials part64[c][Y][A] (forces on sphere A from block
// Y) and part64[c][X][B], or on the diagonal one partial part64[c][X][i];
// contact bits to cmask[K][i]; contact torques (FP64) to torqbuf [A][B] and
// [B][A]; on write steps the tile's potential energy to pe_tile[t].
template <bool WRITE>
__global__ void __launch_bounds__(32 * kM64Warps, kM64CtasPerSm) mixed64_pair_kernel(const __grid_constant__ System s)
{
    __shared__ __align__(16) float rows_all[kM64Warps][kBlock * kRow64];
    pdl_next();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    float* rows = rows_all[wib];
    const long long nwarps = (long long)gridDim.x * kM64Warps;
    const size_t plane = (size_t)s.npad * s.npad;  // torque planes
    const size_t pplane = (size_t)s.nb * s.npad;   // partial planes
    const int sh = s.len_shift;
    const float L = ldexpf(1.0f, sh);
    const float hmin_s = (float)s.mat.h_min / L;
    const float c_vdw = (float)(s.mat.Ha / 6 * 64) / L;  // dyn per unit vdw_shape
    const int nxt = (lane + 1) & (kBlock - 1);

    // A first round of tiles in warp order; then whichever warp is free
    // takes the next tile from a counter that the drift kernel zeroes.  A
    // tile's results do not depend on the warp that computes it.
    long long t = (long long)blockIdx.x * kM64Warps + wib;
    while (t < s.ntiles) {
        int X, Y;
        tile_coords(t, X, Y);
        {
            const int i = X * kBlock + lane;  // < npad
            float* row = rows + lane * kRow64;
            const float Ri = s.f_R[i];
            *reinterpret_cast<float4*>(row) = make_float4(s.f_pos[0][i], s.f_pos[1][i], s.f_pos[2][i], Ri);
            *reinterpret_cast<float4*>(row + 4) =
                make_float4(s.f_pos[3][i], s.f_pos[4][i], s.f_pos[5][i], c_vdw * (Ri * Ri * Ri));
            *reinterpret_cast<float4*>(row + 8) = make_float4(s.f_pos[6][i], s.f_pos[7][i], s.f_pos[8][i], 0.0f);
        }
        __syncwarp();
        const int B = Y * kBlock + lane;
        const bool bvalid = B < s.n;
        const float bx1 = s.f_pos[0][B], by1 = s.f_pos[1][B], bz1 = s.f_pos[2][B];
        const float bx2 = s.f_pos[3][B], by2 = s.f_pos[4][B], bz2 = s.f_pos[5][B];
        const float bx3 = s.f_pos[6][B], by3 = s.f_pos[7][B], bz3 = s.f_pos[8][B];
        const float Rbs = s.f_R[B];
        const float Rb3 = Rbs * Rbs * Rbs;
        const int nA = s.n - X * kBlock;  // rows r < nA are spheres
        double pe = 0.0;       // close pairs' potential (FP64)
        df::Sum3 pe_far{};     // far pairs' vdW brackets, times -Ha/6 at the end
        uint32_t colbits = 0;
        // low halves: the running sum of row (lane + k) mod 32 at step k; high
        // halves: sphere B's sum
        df::Sum3x2 sum[3] = {};
        // FULL: a tile off the diagonal whose rows and columns are all spheres
        auto sweep = [&](auto full_tag) {
            constexpr bool FULL = decltype(full_tag)::value;
#pragma unroll 4
            for (int k = 0; k < kBlock; ++k) {
                const int r = (lane + k) & (kBlock - 1);
                const bool valid = FULL || (bvalid && r < nA && (X != Y || lane < r));
                const float4 q1 = *reinterpret_cast<const float4*>(rows + r * kRow64);
                const float4 q2 = *reinterpret_cast<const float4*>(rows + r * kRow64 + 4);
                const float4 q3 = *reinterpret_cast<const float4*>(rows + r * kRow64 + 8);
                const float Ras = q1.w;
                // the pair subtraction (:105), rounded to FP32
                const float rx = parts::sub3(bx1, bx2, bx3, q1.x, q2.x, q3.x);
                const float ry = parts::sub3(by1, by2, by3, q1.y, q2.y, q3.y);
                const float rz = parts::sub3(bz1, bz2, bz3, q1.z, q2.z, q3.z);
                const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
                const float sumR = Ras + Rbs, difR = Ras - Rbs;
                const float sum2 = sumR * sumR;
                // far pair out of contact, h above the clamp h_min: the vdW
                // force (:205-226) Ra^3 Rb^3 (h + Ra + Rb) / (S^2 T^2) along
                // r / |r| with h + Ra + Rb = |r|, S = |r|^2 - (Ra + Rb)^2 and
                // T = |r|^2 - (Ra - Rb)^2, without a square root
                const float S = d2 - sum2;
                const float T = fmaf(-difR, difR, d2);
                const float P = S * T;
                const float fr = (q2.w * Rb3) * rcp_approx(P * P);  // |F| / |r|
                float fx = fr * rx, fy = fr * ry, fz = fr * rz;
                const bool closep = d2 < s.far_sq * sum2;
                if (valid && closep) {
                    const int A = X * kBlock + r;
                    // FP64 r, |r|^2, squared gap, |r| and overlap (:105-110)
                    const double rx64 = s.pos.c[0][B] - s.pos.c[0][A];
                    const double ry64 = s.pos.c[1][B] - s.pos.c[1][A];
                    const double rz64 = s.pos.c[2][B] - s.pos.c[2][A];
                    const double d2_64 = fma(rx64, rx64, fma(ry64, ry64, rz64 * rz64));
                    const double Ra64 = s.R[A], Rb64 = s.R[B];
                    const double sum64 = Ra64 + Rb64;
                    const double gap2 = fma(sum64, sum64, -d2_64);
                    const double dist64 = sqrt(d2_64);
                    const double ovl64 = gap2 / (sum64 + dist64);
                    const float dist_s = d2f_bits(dist64, sh);
                    const float ovl_s = d2f_bits(ovl64, sh);
                    const float inv_d = 1.0f / dist_s;
                    const float nx = rx * inv_d, ny = ry * inv_d, nz = rz * inv_d;
                    if (gap2 > 0.0) {  // contact (:119)
                        colbits |= 1u << r;
                        const ContactIn in = gather_contact(s, A, B);
                        const ContactF o = contact_mixed(in, s.mat, sh, d2_64, nx, ny, nz, dist_s * L, ovl_s * L,
                                                         Ras, Rbs);
                        fx = o.fx; fy = o.fy; fz = o.fz;
                        double* ta = s.torqbuf + (size_t)A * s.npad + B;
                        double* tb = s.torqbuf + (size_t)B * s.npad + A;
                        ta[0] = f2d_bits(o.tax); ta[plane] = f2d_bits(o.tay); ta[2 * plane] = f2d_bits(o.taz);
                        tb[0] = f2d_bits(o.tbx); tb[plane] = f2d_bits(o.tby); tb[2 * plane] = f2d_bits(o.tbz);
                        if (WRITE) pe += pair_pe_fp64(s.mat, Ra64, Rb64, gap2, d2_64, true, o.k);
                    } else {
                        const float hn = fmaxf(-ovl_s, hmin_s);  // :211-215
                        const float f = c_vdw * vdw_shape(hn, Ras, Rbs);
                        fx = f * nx; fy = f * ny; fz = f * nz;
                        if (WRITE) pe += pair_pe_fp64(s.mat, Ra64, Rb64, gap2, d2_64, false, 0.0);
                    }
                } else if (WRITE && valid) {
                    pe_far.add(vdw_bracket(d2, Ras, Rbs));
                }
                if (!FULL && !valid) fx = fy = fz = 0.0f;
                // both spheres' sums (:249-250)
                const float f[3] = {fx, fy, fz};
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    sum[c].add(f2::pair2(f[c], f[c]));
                    const auto pass = [nxt](f2::F32x2& v) {  // the row's part moves on
                        const float2 h = f2::split2(v);
                        v = f2::pair2(__shfl_sync(0xffffffffu, h.x, nxt), h.y);
                    };
                    pass(sum[c].a);
                    pass(sum[c].b);
                    pass(sum[c].c);
                }
            }
        };
        if (X != Y && (X + 1) * kBlock <= s.n)
            sweep(std::true_type{});
        else
            sweep(std::false_type{});
        // lane l now holds row l's sum; its contact bits are the transpose of
        // the lanes' column bits
        uint32_t rowbits = 0;
        if (__any_sync(0xffffffffu, colbits != 0u)) {
            for (int r = 0; r < kBlock; ++r) {
                const uint32_t wd = __ballot_sync(0xffffffffu, (colbits >> r) & 1u);
                if (lane == r) rowbits = wd;
            }
        }
        const int iA = X * kBlock + lane;
        double* Pt = s.part64;
        double rsum[3], csum[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 a = f2::split2(sum[c].a), b = f2::split2(sum[c].b), d = f2::split2(sum[c].c);
            rsum[c] = total({a.x, b.x, d.x});
            csum[c] = total({a.y, b.y, d.y});
        }
        if (X == Y) {  // sphere iA == B: partners j < i as A (row), j > i as B (column)
            const size_t o = (size_t)X * s.npad + iA;
#pragma unroll
            for (int c = 0; c < 3; ++c) Pt[o + c * pplane] = rsum[c] - csum[c];
            s.cmask[o] = rowbits | colbits;
            if (rowbits | colbits) s.contact_flag[iA] = 1;
        } else {
            const size_t oa = (size_t)Y * s.npad + iA, ob = (size_t)X * s.npad + B;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                Pt[oa + c * pplane] = rsum[c];
                Pt[ob + c * pplane] = -csum[c];
            }
            s.cmask[oa] = rowbits;
            s.cmask[ob] = colbits;
            if (rowbits) s.contact_flag[iA] = 1;  // every writer stores 1
            if (colbits) s.contact_flag[B] = 1;
        }
        if (WRITE) {
            pe += -s.mat.Ha / 6 * total(pe_far);
            for (int off = 16; off > 0; off >>= 1) pe += __shfl_xor_sync(0xffffffffu, pe, off);
            if (lane == 0) s.pe_tile[t] = pe;
        }
        __syncwarp();
        int next = 0;
        if (lane == 0) next = atomicAdd(s.tile_counter, 1);
        t = nwarps + __shfl_sync(0xffffffffu, next, 0);
    }
}

constexpr int kFin64Slices = 8;

// Per-sphere totals, then pass 3.  Block = 32 spheres (lanes) x
// kFin64Slices warps; warp w adds partner blocks [nb w / S, nb (w+1) / S)
// of its lane's sphere in ascending order: the FP64 force partials
// part64[c][K][i] (coalesced along i) and the FP64 torques of contact
// partners (bits of cmask[K][i], ascending).  Warp c < 3 then adds
// component c's slices in order and integrates it in FP64: acc = F / m,
// aacc = torque / moi (the reference divides each pair's term, :249-250,
// 187-188; here the sums are divided once), then
// ColliderSingleCore.cpp:263-267.
__global__ void __launch_bounds__(32 * kFin64Slices) mixed64_finish_kernel(const __grid_constant__ System s)
{
    __shared__ double fs[kFin64Slices][6][kBlock];  // (slice, force x y z, torque x y z, sphere)
    pdl_next();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const int i = blockIdx.x * kBlock + lane;  // < npad
    const int K0 = (int)((long long)s.nb * w / kFin64Slices);
    const int K1 = (int)((long long)s.nb * (w + 1) / kFin64Slices);
    const size_t pplane = (size_t)s.nb * s.npad;
    const size_t plane = (size_t)s.npad * s.npad;
    const double* p = s.part64 + i;
    const uint32_t* mk = s.cmask + i;
    const bool any_contact = i < s.n && s.contact_flag[i] != 0;
    const double* tb = s.torqbuf + (size_t)i * s.npad;
    double f[3] = {0.0, 0.0, 0.0};
    double tq[3] = {0.0, 0.0, 0.0};
    auto torques = [&](uint32_t wd, int K) {
        while (wd) {
            const int j = K * kBlock + __ffs(wd) - 1;
            wd &= wd - 1;
#pragma unroll
            for (int c = 0; c < 3; ++c) tq[c] += tb[j + c * plane];
        }
    };
    constexpr int U = 8;  // loads in flight per array
    // the last batch's entries past K1 are read as zeros: one at a time they
    // cost a round trip each, which was most of the kernel for nb < 64
    auto batch = [&](int K, auto whole_tag) {
        constexpr bool WHOLE = decltype(whole_tag)::value;
        double v[3][U];
        uint32_t m[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t o = (size_t)(K + u) * s.npad;
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c][u] = WHOLE || K + u < K1 ? __ldcs(p + o + c * pplane) : 0.0;
            m[u] = any_contact && (WHOLE || K + u < K1) ? __ldcs(mk + o) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] += v[c][u];
            torques(m[u], K + u);
        }
    };
    int K = K0;
    for (; K + U <= K1; K += U) batch(K, std::true_type{});
    if (K < K1) batch(K, std::false_type{});
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        fs[w][c][lane] = f[c];
        fs[w][3 + c][lane] = tq[c];
    }
    __syncthreads();
    if (w >= 3 || i >= s.n) return;
    const int c = w;
    double F = 0.0, Q = 0.0;
#pragma unroll
    for (int ww = 0; ww < kFin64Slices; ++ww) {
        F += fs[ww][c][lane];
        Q += fs[ww][3 + c][lane];
    }
    const double acc = F / s.m[i];
    const double aacc = Q / s.moi[i];
    const double dt = s.sc->dt;
    const double v = s.velh.c[c][i] + (.5 * acc) * dt;   // :265
    const double wv = s.wh.c[c][i] + (.5 * aacc) * dt;  // :266
    s.acc.c[c][i] = acc;
    s.aacc.c[c][i] = aacc;
    s.vel.c[c][i] = v;
    s.w.c[c][i] = wv;
    if (!isfinite(v) || !isfinite(wv) || !isfinite(s.pos.c[c][i])) atomicOr(s.status, 1u);
}

}  // namespace

void launch_step_mixed64(const System& s, bool write, int num_sms, cudaStream_t st, StepTimers* tm)
{
    launch_drift(s, st);
    if (tm) cudaEventRecord(tm->ev[0], st);
    const long long want = (s.ntiles + kM64Warps - 1) / kM64Warps;
    const long long cap = (long long)num_sms * kM64CtasPerSm;  // one wave of persistent warps
    const int pb = (int)(want < cap ? want : cap);
    // a dependent launch up to one CTA per SM (us per step, dependent / plain: N=64
    // 28.8 / 29.7, N=500 27.5 / 28.2, N=1000 30.0 / 30.2, N=1080 31.0 / 30.4, N=1200 31.2 /
    // 32.1, N=1500 32.3 / 31.8, N=2000 35.4 / 35.2): a larger grid, placed while the
    // drift still runs, is spread unevenly over the SMs
    launch_pdl(pb <= num_sms, write ? mixed64_pair_kernel<true> : mixed64_pair_kernel<false>, pb, 32 * kM64Warps, 0, st, s);
    if (tm) cudaEventRecord(tm->ev[1], st);
    // plainly: placed beside the pair kernel's last blocks, the finish blocks share
    // SMs (us per step, dependent / plain: N=64 36 / 28, N=1000 31.0 / 29.1, N=2500
    // 76.5 / 71.0)
    mixed64_finish_kernel<<<s.nb, 32 * kFin64Slices, 0, st>>>(s);
    if (tm) cudaEventRecord(tm->ev[2], st);
    if (write) launch_energy(s, st);
}

}  // namespace sl
