// sl_batch_mixed.cu -- batched solver in the mixed-precision form: the same
// persistent work-queue launch as sl_batch.cu, with the pair math of the
// mixed form: far pairs entirely in FP32 (no square root), close pairs with
// double-float (sl_df.cuh) displacement, |r|^2 and squared gap from the
// double-float positions the drift writes; FP32 forces and torques; FP64
// kin/kout test and write-step potential energy of close pairs from the
// FP64 positions (far pairs: the FP32 series of vdw_bracket).  The
// non-contact pair path issues no FP64 instruction.  Two pair passes over
// each instance's Z-ordered slots (sl_batch.h): the pair-tile pass (shape
// tile 0, every pair once, per-CTA partial sums) and the per-sphere loop
// (j-tiles of 32/64/128, every pair from both sides, FP32 sums per j-tile
// joined in compensated per-sphere totals).
#include "sl_batch.h"
#include "sl_batch_common.cuh"
#include "sl_df.cuh"
#include "sl_pair_mixed.cuh"
#include "sl_tile_mixed.cuh"

#include <type_traits>

namespace sl {

namespace {

using batch::drift;
using batch::kick;

template <int TILE>
struct JTileM {
    float4 q0[TILE];  // scaled position hi x, y, z and scaled radius R
    float4 q1[TILE];  // scaled position lo x, y, z and R^3
    float Rlo[TILE];  // the radius's double-float lo part
    int idx[TILE];    // the sphere's index in the instance (its slot's perm entry)
};

// |pos[gB] - pos[gA]|^2 in FP64, the previous-step formula of contact_mixed
__device__ __forceinline__ double fp64_d2(const Batch& b, int gA, int gB)
{
    const double rx = b.pos.c[0][gB] - b.pos.c[0][gA];
    const double ry = b.pos.c[1][gB] - b.pos.c[1][gA];
    const double rz = b.pos.c[2][gB] - b.pos.c[2][gA];
    return fma(rx, rx, fma(ry, ry, rz * rz));
}

// Thread i walks partners j through shared-memory j-tiles and adds the
// force on i, F_ij, into a plain FP32 sum per tile, which joins i's
// compensated total; acc[i] = total / m[i].  A far pair
// (|r| >= 1.25 (R_i + R_j) or more, far_sq) takes the FP32 path of the all-pairs mixed
// kernel: vdW along
// r = pos[j] - pos[i] without a square root, (c R_i^3 R_j^3) r / (S T)^2 with
// S = |r|^2 - (R_i + R_j)^2 and T = |r|^2 - (R_i - R_j)^2; a near pair the
// double-float geometry and, in contact, contact_mixed in the pair's own
// (A, B) orientation (ColliderSingleCore.cpp:104-253).
template <int TILE, bool WRITE>
__device__ double pair_pass_mixed(const Batch& b, int off, int n, const Material& M, double kin, double kout,
                                  JTileM<TILE>& jt)
{
    const int sh = b.len_shift;
    const float L = ldexpf(1.0f, sh);
    const float hmin_s = (float)M.h_min / L;
    const float c_vdw = (float)(M.Ha / 6 * 64) / L;
    double pe = 0;
    df::Sum pe_far{0.0f, 0.0f};  // far pairs' vdW brackets (write steps, i = A)
    for (int ibase = 0; ibase < n; ibase += blockDim.x) {
        const bool active = ibase + threadIdx.x < n;
        const int si = off + (active ? ibase + threadIdx.x : 0);  // slot: Z-order, a warp's spheres are close
        const int gi = b.perm[si];
        const int i = gi - off;
        const float pih[3] = {b.f_pos[0][si], b.f_pos[1][si], b.f_pos[2][si]};
        const float pil[3] = {b.f_pos[3][si], b.f_pos[4][si], b.f_pos[5][si]};
        const float Ri = b.f_R[si], Rilo = b.f_Rlo[si];
        const float cR3i = c_vdw * (Ri * Ri * Ri);
        const float imoii = b.f_inv_moi[si];
        df::Sum ax{0.0f, 0.0f}, ay{0.0f, 0.0f}, az{0.0f, 0.0f};
        double tx = 0, ty = 0, tz = 0;
        for (int jbase = 0; jbase < n; jbase += TILE) {
            for (int t = threadIdx.x; t < TILE; t += blockDim.x) {
                const int j = jbase + t;
                if (j < n) {
                    const int g = off + j;  // slot
                    const float r = b.f_R[g];
                    jt.q0[t] = make_float4(b.f_pos[0][g], b.f_pos[1][g], b.f_pos[2][g], r);
                    jt.q1[t] = make_float4(b.f_pos[3][g], b.f_pos[4][g], b.f_pos[5][g], r * r * r);
                    jt.Rlo[t] = b.f_Rlo[g];
                    jt.idx[t] = b.perm[g] - off;
                }
            }
            __syncthreads();
            if (active) {
                // close pair in slot jbase + t: double-float geometry, contact or
                // clamped vdW in the pair's (A, B) orientation; the force on i
                auto close_pair = [&](int t, float& fx, float& fy, float& fz) {
                    const int j = jt.idx[t];
                    const bool iA = i > j;
                    const float4 q0 = jt.q0[t], q1 = jt.q1[t];
                    const float Rj = q0.w;
                    // r = pos[B] - pos[A] in double-float; the sign flips with the orientation
                    const df::F2 pj[3] = {{q0.x, q1.x}, {q0.y, q1.y}, {q0.z, q1.z}};
                    df::F2 r3[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const df::F2 pi{pih[c], pil[c]};
                        r3[c] = iA ? df::sub(pj[c], pi) : df::sub(pi, pj[c]);
                    }
                    const df::F2 dd2 = df::add(df::add(df::sqr(r3[0]), df::sqr(r3[1])), df::sqr(r3[2]));
                    const df::F2 sum = df::add({Ri, Rilo}, {Rj, jt.Rlo[t]});
                    const df::F2 gap2 = df::sub(df::sqr(sum), dd2);
                    const float Ras = iA ? Ri : Rj, Rbs = iA ? Rj : Ri;
                    const float d2s = dd2.hi;
                    const float inv_d = rsqrtf(d2s);
                    const float dist_s = d2s * inv_d;
                    const float ovl_s = __fdividef(gap2.hi, Ras + Rbs + dist_s);
                    const float nx = r3[0].hi * inv_d, ny = r3[1].hi * inv_d, nz = r3[2].hi * inv_d;
                    float Fx, Fy, Fz;  // force on A
                    const int gA = off + (iA ? i : j), gB = off + (iA ? j : i);
                    if (gap2.hi > 0.0f || (gap2.hi == 0.0f && gap2.lo > 0.0f)) {
                        ContactIn in;
                        for (int c = 0; c < 3; ++c) {
                            in.prevA[c] = b.prev.c[c][gA]; in.prevB[c] = b.prev.c[c][gB];
                            in.wA[c] = b.w.c[c][gA]; in.wB[c] = b.w.c[c][gB];
                            in.vA[c] = b.vel.c[c][gA]; in.vB[c] = b.vel.c[c][gB];
                        }
                        in.mA = b.m[gA]; in.mB = b.m[gB]; in.kin = kin; in.kout = kout;
                        // kin/kout: |r|^2 against the previous step's, both FP64 by one formula
                        const double d2_64 = fp64_d2(b, gA, gB);
                        const ContactF o = contact_mixed(in, M, sh, d2_64, nx, ny, nz, dist_s * L, ovl_s * L, Ras, Rbs);
                        Fx = o.fx; Fy = o.fy; Fz = o.fz;
                        const float qx = iA ? o.tax : o.tbx, qy = iA ? o.tay : o.tby, qz = iA ? o.taz : o.tbz;
                        tx += f2d_bits(qx * imoii); ty += f2d_bits(qy * imoii); tz += f2d_bits(qz * imoii);
                        if (WRITE && iA) {
                            const double sum64 = b.R[gA] + b.R[gB];
                            pe += pair_pe_fp64(M, b.R[gA], b.R[gB], fma(sum64, sum64, -d2_64), d2_64, true, o.k);
                        }
                    } else {
                        const float h = fmaxf(-ovl_s, hmin_s);
                        const float f = c_vdw * vdw_shape(h, Ras, Rbs);
                        Fx = f * nx; Fy = f * ny; Fz = f * nz;
                        if (WRITE && iA) {
                            const double d2_64 = fp64_d2(b, gA, gB), sum64 = b.R[gA] + b.R[gB];
                            pe += pair_pe_fp64(M, b.R[gA], b.R[gB], fma(sum64, sum64, -d2_64), d2_64, false, 0.0);
                        }
                    }
                    // acc[A] += F/m[A]; acc[B] -= F/m[B]
                    fx = iA ? Fx : -Fx; fy = iA ? Fy : -Fy; fz = iA ? Fz : -Fz;
                };
                // far pair (or not a pair): its force on i, 0 where it is not
                // far; returns whether it is close
                auto far_pair = [&](int t, float& fx, float& fy, float& fz) {
                    const int j = jt.idx[t];
                    const bool valid = j != i;
                    const float4 q0 = jt.q0[t], q1 = jt.q1[t];
                    const float Rj = q0.w;
                    const float rx = (q0.x - pih[0]) + (q1.x - pil[0]);
                    const float ry = (q0.y - pih[1]) + (q1.y - pil[1]);
                    const float rz = (q0.z - pih[2]) + (q1.z - pil[2]);
                    const float d2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
                    const float sumR = Ri + Rj, difR = Ri - Rj;
                    const float sum2 = sumR * sumR;
                    const float S = d2 - sum2;
                    const float T = fmaf(-difR, difR, d2);
                    const float P = S * T;
                    const float fr = (cR3i * q1.w) * rcp_approx(P * P);
                    const bool close = d2 < b.far_sq * sum2;
                    const bool use = valid && !close;
                    fx = use ? fr * rx : 0.0f;
                    fy = use ? fr * ry : 0.0f;
                    fz = use ? fr * rz : 0.0f;
                    if (WRITE && use && i > j) pe_far.add(vdw_bracket(d2, Ri, Rj));
                    return valid && close;
                };
                const int jend = min(TILE, n - jbase);
                float sx = 0, sy = 0, sz = 0;  // this tile's forces on i
                int t = 0;
                // four partners at a time, so that their far-pair arithmetic
                // interleaves; the close ones after, in one branch
                for (; t + 4 <= jend; t += 4) {
                    uint32_t closem = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float fx, fy, fz;
                        closem |= (uint32_t)far_pair(t + u, fx, fy, fz) << u;
                        sx += fx; sy += fy; sz += fz;
                    }
                    if (closem) {
#pragma unroll 1
                        for (int u = 0; u < 4; ++u)
                            if ((closem >> u) & 1u) {
                                float fx, fy, fz;
                                close_pair(t + u, fx, fy, fz);
                                sx += fx; sy += fy; sz += fz;
                            }
                    }
                }
                for (; t < jend; ++t) {
                    float fx, fy, fz;
                    if (far_pair(t, fx, fy, fz)) close_pair(t, fx, fy, fz);
                    sx += fx; sy += fy; sz += fz;
                }
                ax.add(sx); ay.add(sy); az.add(sz);
            }
            __syncthreads();
        }
        if (active) {
            const double imi = f2d_bits(b.f_inv_m[si]);
            b.acc.c[0][gi] = (f2d_bits(ax.s) + f2d_bits(ax.c)) * imi;
            b.acc.c[1][gi] = (f2d_bits(ay.s) + f2d_bits(ay.c)) * imi;
            b.acc.c[2][gi] = (f2d_bits(az.s) + f2d_bits(az.c)) * imi;
            b.aacc.c[0][gi] = tx; b.aacc.c[1][gi] = ty; b.aacc.c[2][gi] = tz;
        }
    }
    if (WRITE) pe += -M.Ha / 6 * (f2d_bits(pe_far.s) + f2d_bits(pe_far.c));
    return pe;
}

template <int TILE>
__global__ void __launch_bounds__(256) batch_mixed_kernel(const __grid_constant__ Batch b, int first_step, int nsteps,
                                                          int skip, int do_init)
{
    __shared__ JTileM<TILE> jt;
    __shared__ double sh[8][32];
    __shared__ int s_next;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_next = atomicAdd(b.counter, 1);
        __syncthreads();
        const int k = s_next;
        if (k >= b.ninst) return;
        const int inst = b.order[k];
        const int off = b.off[inst], n = b.cnt[inst];
        Material M = b.mat;
        M.u_s = b.u_s[inst];
        const double dt = b.dt[inst], kin = b.kin[inst], kout = b.kout[inst];
        double* recs = b.energy + (size_t)inst * b.nrec * 8;
        if (do_init) {
            drift(b, off, n, 0.0);
            __syncthreads();
            const double pe = pair_pass_mixed<TILE, true>(b, off, n, M, kin, kout, jt);
            __syncthreads();
            kick(b, inst, off, n, 0.0, true, pe, recs, sh);
            __syncthreads();
        }
        for (int q = 0; q < nsteps; ++q) {
            const int step = first_step + q;
            const bool write = skip > 0 && step % skip == 0;
            drift(b, off, n, dt);
            __syncthreads();
            double pe = 0;
            if (write)
                pe = pair_pass_mixed<TILE, true>(b, off, n, M, kin, kout, jt);
            else
                pair_pass_mixed<TILE, false>(b, off, n, M, kin, kout, jt);
            __syncthreads();
            const int r = write ? step / skip : 0;
            kick(b, inst, off, n, dt, write, pe, recs + (size_t)(r < b.nrec ? r : b.nrec - 1) * 8, sh);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Pair-tile pass: every unordered pair once.  The CTA's warps take the
// instance's lower-triangular 32 x 32 slot-block tiles in turn and sweep
// each diagonally as the all-pairs mixed kernel does (sl_step_mixed.cu): at
// step k lane b takes (row (b + k) mod 32, column b), its column sum stays in
// a register and each row sum moves one lane down per step.  A tile writes one
// FP32 partial per sphere and component -- forces and torques -- to the CTA's
// scratch part[6][nb][np] (slot-indexed), and the CTA then adds each sphere's
// partials over the partner blocks in ascending order in compensated sums.
// Torques exist only in contact: a row sphere's arrive by shared-memory adds
// (one lane per row in a step, the steps in program order, so the order is
// fixed), a column sphere's in a register.
constexpr int kTileWarps = 16;  // up to 512 threads: a large instance can have a whole SM
constexpr uint16_t kTouching = 0x8000;  // mark of a list entry in contact

// One warp's shared memory: rows [16] the radius's lo part, [17]
// 1/m, [18] 1/moi, [19] the index in the instance; row torques; listed pairs with both
// spheres' torques.
struct TileSmem {
    float rows[kBlock * mt::kRow];
    float rowtq[3 * kBlock];
    mt::List<9> list;
};

// The batch's constants in scaled lengths, formed once per kernel: the FP64
// division is worth a fifth of a tile.
struct MixedConst {
    float L, hmin_s, c_vdw;
};

__device__ __forceinline__ MixedConst mixed_const(const Batch& b)
{
    const float L = ldexpf(1.0f, b.len_shift);
    return {L, (float)b.mat.h_min / L, (float)(b.mat.Ha / 6 * 64) / L};
}

// One tile (X, Y) of the instance with spheres off .. off + n - 1, by one
// warp (sl_tile_mixed.cuh); partials to part (rows of part_np floats, pplane
// per component).  tmask given, a sphere's torque partials are written only
// where they are not zero, and its bit K of tmask (words of 32 partner blocks,
// part_np apart) says so: contacts are few, and the torques are half of the
// partials' traffic.
template <bool WRITE>
__device__ __forceinline__ void tile_mixed(const Batch& b, int off, int n, const Material& M, double kin, double kout,
                                           const MixedConst& mc, int X, int Y, TileSmem& sm, float* part, int part_np,
                                           size_t pplane, uint32_t* tmask, double& pe, df::Sum& pe_far)
{
    const int lane = threadIdx.x & 31;
    const int sh = b.len_shift;
    const float L = mc.L, hmin_s = mc.hmin_s, c_vdw = mc.c_vdw;
    float* rows = sm.rows;
    float* rowtq = sm.rowtq;
    {
        const int sA = off + min(X * kBlock + lane, n - 1);  // slot (padding rows repeat the last)
        const float Ri = b.f_R[sA];
        mt::put_row(rows, lane, {b.f_pos[0][sA], b.f_pos[1][sA], b.f_pos[2][sA], Ri, b.f_pos[3][sA],
                                 b.f_pos[4][sA], b.f_pos[5][sA], c_vdw * (Ri * Ri * Ri)},
                    make_float4(b.f_Rlo[sA], b.f_inv_m[sA], b.f_inv_moi[sA], __int_as_float(b.perm[sA] - off)));
        rowtq[lane] = 0.0f; rowtq[kBlock + lane] = 0.0f; rowtq[2 * kBlock + lane] = 0.0f;
    }
    __syncwarp();
    const int sB = Y * kBlock + lane;  // slot in the instance
    auto load_column = [&](int slot) {
        const int g = off + min(slot, n - 1);
        mt::Col c;
        c.x = b.f_pos[0][g]; c.y = b.f_pos[1][g]; c.z = b.f_pos[2][g];
        c.xl = b.f_pos[3][g]; c.yl = b.f_pos[4][g]; c.zl = b.f_pos[5][g];
        c.R = b.f_R[g];
        c.R3 = c.R * c.R * c.R;
        c.valid = slot < n;
        return c;
    };
    const mt::Col col = load_column(sB);
    const float inv_mb = b.f_inv_m[off + min(sB, n - 1)], inv_moib = b.f_inv_moi[off + min(sB, n - 1)];
    const int nA = n - X * kBlock;
    float ctx = 0, cty = 0, ctz = 0;     // the column sphere's torque sum
    // listed pair (row r, column slot 32Y + cb): double-float geometry, then
    // the contact branch in the reference's orientation (A = the larger
    // index in the instance) or the clamped vdW; the force on the row
    // sphere, and in contact both spheres' torques
    auto close = [&](int q, int r, int cb, double& pe_, df::Sum& far_) {
        const mt::Col c = load_column(Y * kBlock + cb);
        const int gs = off + min(Y * kBlock + cb, n - 1);
        const mt::Row row = mt::get_row(rows, r);
        float* out = sm.list.v[q];
        const float Ras = row.R, Rbs = c.R;
        const mt::Far f = mt::far_pair(row, c);
        if (!(f.d2 < b.far_sq * f.sum2)) {
            out[0] = f.fr * f.rx; out[1] = f.fr * f.ry; out[2] = f.fr * f.rz;
            if (WRITE) far_.add(vdw_bracket(f.d2, Ras, Rbs));
            return;
        }
        const int iA = __float_as_int(rows[r * mt::kRow + 19]), iB = b.perm[gs] - off;
        const df::F2 drx = df::sub({c.x, c.xl}, {row.x, row.xl});
        const df::F2 dry = df::sub({c.y, c.yl}, {row.y, row.yl});
        const df::F2 drz = df::sub({c.z, c.zl}, {row.z, row.zl});
        const df::F2 dd2 = df::add(df::add(df::sqr(drx), df::sqr(dry)), df::sqr(drz));
        const df::F2 sum = df::add({Ras, rows[r * mt::kRow + 16]}, {Rbs, b.f_Rlo[gs]});
        const df::F2 gap2 = df::sub(df::sqr(sum), dd2);
        const float d2s = dd2.hi;
        const float inv_dn = rsqrtf(d2s);
        const float dist_s = d2s * inv_dn;
        const float ovl_s = __fdividef(gap2.hi, Ras + Rbs + dist_s);
        const float nx = drx.hi * inv_dn, ny = dry.hi * inv_dn, nz = drz.hi * inv_dn;  // row -> column
        const bool rowA = iA > iB;
        const int gA = off + (rowA ? iA : iB), gB = off + (rowA ? iB : iA);
        if (gap2.hi > 0.0f || (gap2.hi == 0.0f && gap2.lo > 0.0f)) {
            ContactIn in;
            for (int k = 0; k < 3; ++k) {
                in.prevA[k] = b.prev.c[k][gA]; in.prevB[k] = b.prev.c[k][gB];
                in.wA[k] = b.w.c[k][gA]; in.wB[k] = b.w.c[k][gB];
                in.vA[k] = b.vel.c[k][gA]; in.vB[k] = b.vel.c[k][gB];
            }
            in.mA = b.m[gA]; in.mB = b.m[gB]; in.kin = kin; in.kout = kout;
            // kin/kout: |r|^2 against the previous step's, both FP64 by one formula
            const double d2_64 = fp64_d2(b, gA, gB);
            const float sg = rowA ? 1.0f : -1.0f;  // unit vector A -> B
            const ContactF o = contact_mixed(in, M, sh, d2_64, sg * nx, sg * ny, sg * nz, dist_s * L, ovl_s * L,
                                             rowA ? Ras : Rbs, rowA ? Rbs : Ras);
            out[0] = sg * o.fx; out[1] = sg * o.fy; out[2] = sg * o.fz;  // o.f acts on A; B takes -o.f
            const float imoia = rows[r * mt::kRow + 18];
            out[3] = (rowA ? o.tax : o.tbx) * imoia;
            out[4] = (rowA ? o.tay : o.tby) * imoia;
            out[5] = (rowA ? o.taz : o.tbz) * imoia;
            out[6] = rowA ? o.tbx : o.tax;
            out[7] = rowA ? o.tby : o.tay;
            out[8] = rowA ? o.tbz : o.taz;
            sm.list.pair[q] |= kTouching;
            if (WRITE) {
                const double sum64 = b.R[gA] + b.R[gB];
                pe_ += pair_pe_fp64(M, b.R[gA], b.R[gB], fma(sum64, sum64, -d2_64), d2_64, true, o.k);
            }
            return;
        }
        const float hn = fmaxf(-ovl_s, hmin_s);
        const float fv = c_vdw * vdw_shape(hn, Ras, Rbs);
        out[0] = fv * nx; out[1] = fv * ny; out[2] = fv * nz;
        if (WRITE) {
            const double d2_64 = fp64_d2(b, gA, gB), sum64 = b.R[gA] + b.R[gB];
            pe_ += pair_pe_fp64(M, b.R[gA], b.R[gB], fma(sum64, sum64, -d2_64), d2_64, false, 0.0);
        }
    };
    // a contact's torques, in the sweep's order: one lane per row in a step
    auto taken = [&](int q, int r) {
        if (!(sm.list.pair[q] & kTouching)) return;
        const float* v = sm.list.v[q];
        atomicAdd(&rowtq[r], v[3]);
        atomicAdd(&rowtq[kBlock + r], v[4]);
        atomicAdd(&rowtq[2 * kBlock + r], v[5]);
        ctx = fmaf(v[6], inv_moib, ctx);
        cty = fmaf(v[7], inv_moib, cty);
        ctz = fmaf(v[8], inv_moib, ctz);
    };
    float av[3], bv[3];
    mt::tile<WRITE>(rows, sm.list, col, nA, X == Y, b.far_sq, close, taken, av, bv, pe, pe_far);
    const float ax = av[0], ay = av[1], az = av[2], bsx = bv[0], bsy = bv[1], bsz = bv[2];
    __syncwarp();  // the row torques' shared-memory adds
    // lane l holds row l's force sum (rows and columns beyond n hold 0)
    const int sAl = X * kBlock + lane;
    const float ima = rows[lane * mt::kRow + 17];
    const float rtx = rowtq[lane], rty = rowtq[kBlock + lane], rtz = rowtq[2 * kBlock + lane];
    // sphere at slot p: torques from block K
    auto put_torque = [&](int K, int p, float tx, float ty, float tz) {
        if (tmask) {
            if (tx == 0.0f && ty == 0.0f && tz == 0.0f) return;
            if (p < n) atomicOr(tmask + (size_t)(K >> 5) * part_np + p, 1u << (K & 31));
        }
        float* o = part + (size_t)K * part_np + p + 3 * pplane;
        __stcs(o, tx); __stcs(o + pplane, ty); __stcs(o + 2 * pplane, tz);
    };
    if (X == Y) {  // the same sphere: partners before it in slot order (row), after it (column)
        const size_t o = (size_t)X * part_np + sAl;
        __stcs(part + o, fmaf(ima, ax, -inv_mb * bsx));
        __stcs(part + o + pplane, fmaf(ima, ay, -inv_mb * bsy));
        __stcs(part + o + 2 * pplane, fmaf(ima, az, -inv_mb * bsz));
        put_torque(X, sAl, rtx + ctx, rty + cty, rtz + ctz);
    } else {
        const size_t oa = (size_t)Y * part_np + sAl, ob = (size_t)X * part_np + sB;
        __stcs(part + oa, ima * ax); __stcs(part + oa + pplane, ima * ay); __stcs(part + oa + 2 * pplane, ima * az);
        __stcs(part + ob, -inv_mb * bsx);
        __stcs(part + ob + pplane, -inv_mb * bsy);
        __stcs(part + ob + 2 * pplane, -inv_mb * bsz);
        put_torque(Y, sAl, rtx, rty, rtz);
        put_torque(X, sB, ctx, cty, ctz);
    }
    __syncwarp();
}

template <bool WRITE>
__device__ double tile_pass_mixed(const Batch& b, int off, int n, const Material& M, double kin, double kout,
                                  TileSmem* smem)
{
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nbk = (n + kBlock - 1) / kBlock;
    const long long ntiles = (long long)nbk * (nbk + 1) / 2;
    float* part = b.part + (size_t)blockIdx.x * b.part_cta;
    const size_t pplane = (size_t)b.part_nb * b.part_np;
    const MixedConst mc = mixed_const(b);
    double pe = 0;
    df::Sum pe_far{0.0f, 0.0f};  // far pairs' vdW brackets (write steps)
    for (long long t = warp; t < ntiles; t += nwarps) {
        int X, Y;
        tile_coords(t, X, Y);
        tile_mixed<WRITE>(b, off, n, M, kin, kout, mc, X, Y, smem[warp], part, b.part_np, pplane, nullptr, pe, pe_far);
    }
    if (WRITE) pe += -M.Ha / 6 * (f2d_bits(pe_far.s) + f2d_bits(pe_far.c));
    return pe;
}

// The CTA's per-sphere totals from the tile partials (partner blocks in
// ascending order, compensated sums), to acc and aacc in the caller's order.
__device__ __forceinline__ void tile_totals(const Batch& b, int off, int n)
{
    const int nbk = (n + kBlock - 1) / kBlock;
    const float* part = b.part + (size_t)blockIdx.x * b.part_cta;
    const size_t pplane = (size_t)b.part_nb * b.part_np;
    for (int p = threadIdx.x; p < n; p += blockDim.x) {
        df::Sum tot[6] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
        for (int K = 0; K < nbk; ++K) {
            const float* e = part + (size_t)K * b.part_np + p;
#pragma unroll
            for (int q = 0; q < 6; ++q) tot[q].add(e[q * pplane]);
        }
        const int g = b.perm[off + p];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            b.acc.c[c][g] = f2d_bits(tot[c].s) + f2d_bits(tot[c].c);
            b.aacc.c[c][g] = f2d_bits(tot[3 + c].s) + f2d_bits(tot[3 + c].c);
        }
    }
}

__global__ void __launch_bounds__(32 * kTileWarps) batch_mixed_tiles_kernel(const __grid_constant__ Batch b,
                                                                           int first_step, int nsteps, int skip,
                                                                           int do_init)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    TileSmem* ts = reinterpret_cast<TileSmem*>(tile_raw);
    __shared__ double sh[8][32];
    __shared__ int s_next;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_next = atomicAdd(b.counter, 1);
        __syncthreads();
        const int k = s_next;
        if (k >= b.ninst) return;
        const int inst = b.order[k];
        const int off = b.off[inst], n = b.cnt[inst];
        Material M = b.mat;
        M.u_s = b.u_s[inst];
        const double dt = b.dt[inst], kin = b.kin[inst], kout = b.kout[inst];
        double* recs = b.energy + (size_t)inst * b.nrec * 8;
        if (do_init) {
            drift(b, off, n, 0.0);
            __syncthreads();
            const double pe = tile_pass_mixed<true>(b, off, n, M, kin, kout, ts);
            __syncthreads();
            tile_totals(b, off, n);
            __syncthreads();
            kick(b, inst, off, n, 0.0, true, pe, recs, sh);
            __syncthreads();
        }
        for (int q = 0; q < nsteps; ++q) {
            const int step = first_step + q;
            const bool write = skip > 0 && step % skip == 0;
            drift(b, off, n, dt);
            __syncthreads();
            double pe = 0;
            if (write)
                pe = tile_pass_mixed<true>(b, off, n, M, kin, kout, ts);
            else
                tile_pass_mixed<false>(b, off, n, M, kin, kout, ts);
            __syncthreads();
            tile_totals(b, off, n);
            __syncthreads();
            const int r = write ? step / skip : 0;
            kick(b, inst, off, n, dt, write, pe, recs + (size_t)(r < b.nrec ? r : b.nrec - 1) * 8, sh);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Lockstep form of the pair-tile pass (see sl_batch.cu): all instances take a
// step together, so that the largest ones do not set the time.  The tiles are
// the same function of the same operands, and a sphere's partials are added in
// the same order, so the results are the form's above.
//   pairs   tiles of all instances from a queue
//   rows    one warp per 32-slot block, lane = sphere: totals, pass 3, on write
//           steps the energy terms, and the next step's pass 1
// Energy records are summed per instance under the next pairs phase.
constexpr int kGridWarpsM = 20;

// isfinite on the integer pipe
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// Pass 1 of slot p's sphere g (batch::drift's operations)
__device__ __forceinline__ void drift_sphere(const Batch& b, int slot, int g, double dt)
{
    const double scale = ldexp(1.0, b.len_shift);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double vh = b.vel.c[c][g] + (.5 * b.acc.c[c][g]) * dt;   // :84
        const double whc = b.w.c[c][g] + (.5 * b.aacc.c[c][g]) * dt;   // :87
        const double p = b.pos.c[c][g];
        const double pn = p + vh * dt;                                 // :90
        b.velh.c[c][g] = vh;
        b.wh.c[c][g] = whc;
        b.prev.c[c][g] = p;
        b.pos.c[c][g] = pn;
        const float hi = d2f_bits(pn, b.len_shift);
        b.f_pos[c][slot] = hi;
        b.f_pos[3 + c][slot] = d2f_bits(pn - f2d_bits(hi) * scale, b.len_shift);
    }
}

template <bool WRITE>
__device__ void grid_pairs_mixed(const Batch& b, TileSmem& sm, int* queue, double* pe_out)
{
    const int lane = threadIdx.x & 31;
    const long long nw = (long long)gridDim.x * kGridWarpsM;
    const MixedConst mc = mixed_const(b);
    // the next tile is taken, and its header read, ahead of this one's work
    const auto take = [&](int4& head) {
        int k = 0;
        if (lane == 0) k = atomicAdd(queue, 1);
        const long long u = nw + __shfl_sync(0xffffffffu, k, 0);
        if (u < b.gtiles) head = __ldg(b.gtile + u);
        return u;
    };
    long long u = (long long)blockIdx.x * kGridWarpsM + (threadIdx.x >> 5);
    if (u >= b.gtiles) return;
    int4 tile = __ldg(b.gtile + u);
    while (u < b.gtiles) {
        int4 ahead = tile;
        const long long next = take(ahead);
        const int inst = tile.x, off = tile.y, n = tile.z, X = tile.w >> 16, Y = tile.w & 0xffff;
        Material M = b.mat;
        M.u_s = b.u_s[inst];
        const int nb = (n + kBlock - 1) / kBlock;
        double pe = 0;
        df::Sum pe_far{0.0f, 0.0f};
        tile_mixed<WRITE>(b, off, n, M, b.kin[inst], b.kout[inst], mc, X, Y, sm, b.gpart + b.gpair_off[inst],
                          nb * kBlock, (size_t)nb * nb * kBlock, b.xmask + b.gmask_off[inst], pe, pe_far);
        if (WRITE) {
            pe += -M.Ha / 6 * (f2d_bits(pe_far.s) + f2d_bits(pe_far.c));
            for (int o = 16; o > 0; o >>= 1) pe += __shfl_xor_sync(0xffffffffu, pe, o);
            if (lane == 0) pe_out[u] = pe;
        }
        u = next;
        tile = ahead;
    }
}

__device__ void grid_rows_mixed(const Batch& b, bool init, bool write, bool more)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kGridWarpsM + (threadIdx.x >> 5), nw = gridDim.x * kGridWarpsM;
    for (int item = gw; item < b.gblocks; item += nw) {
        const int inst = b.gblk_inst[item], p = b.gblk[item] * kBlock + lane;
        const int off = b.off[inst], n = b.cnt[inst];
        const int nb = (n + kBlock - 1) / kBlock;
        const bool live = p < n;
        double e[7] = {0, 0, 0, 0, 0, 0, 0};
        if (live) {
            const size_t pplane = (size_t)nb * nb * kBlock;
            const float* part = b.gpart + b.gpair_off[inst] + p;
            df::Sum tot[6] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
            constexpr int U = 8;  // partner blocks in flight; those past the last read as zeros
            for (int K = 0; K < nb; K += U) {
                float v[U][3];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        v[u][q] = K + u < nb ? __ldcs(part + (size_t)(K + u) * nb * kBlock + q * pplane) : 0.0f;
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int q = 0; q < 3; ++q) tot[q].add(v[u][q]);
            }
            uint32_t* tm = b.xmask + b.gmask_off[inst] + p;
            for (int W = 0; W < (nb + 31) / 32; ++W) {
                uint32_t bits = tm[(size_t)W * nb * kBlock];
                if (!bits) continue;
                tm[(size_t)W * nb * kBlock] = 0;  // for the next step
                for (; bits; bits &= bits - 1) {
                    const float* e = part + (size_t)(32 * W + __ffs(bits) - 1) * nb * kBlock + 3 * pplane;
#pragma unroll
                    for (int q = 0; q < 3; ++q) tot[3 + q].add(e[q * pplane]);
                }
            }
            const int g = b.perm[off + p];
            const double dt = init ? 0.0 : b.dt[inst];
            double v[3], w[3];
            bool bad = false;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double acc = f2d_bits(tot[c].s) + f2d_bits(tot[c].c);
                const double aacc = f2d_bits(tot[3 + c].s) + f2d_bits(tot[3 + c].c);
                b.acc.c[c][g] = acc;
                b.aacc.c[c][g] = aacc;
                v[c] = b.velh.c[c][g] + (.5 * acc) * dt;    // :265
                w[c] = b.wh.c[c][g] + (.5 * aacc) * dt;     // :266
                b.vel.c[c][g] = v[c];
                b.w.c[c][g] = w[c];
                bad |= !finite_bits(v[c]) || !finite_bits(w[c]) || !finite_bits(b.pos.c[c][g]);
            }
            if (bad) atomicOr(&b.status[inst], 1u);
            if (write) {
                const double m = b.m[g], moi = b.moi[g];
                const double px = b.pos.c[0][g], py = b.pos.c[1][g], pz = b.pos.c[2][g];
                e[0] = .5 * m * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) +
                       .5 * moi * (w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
                e[1] = m * v[0]; e[2] = m * v[1]; e[3] = m * v[2];
                e[4] = m * (py * v[2] - pz * v[1]) + moi * w[0];
                e[5] = m * (pz * v[0] - px * v[2]) + moi * w[1];
                e[6] = m * (px * v[1] - py * v[0]) + moi * w[2];
            }
            if (more) drift_sphere(b, off + p, g, b.dt[inst]);
        }
        if (write) {
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                for (int o = 16; o > 0; o >>= 1) e[k] += __shfl_xor_sync(0xffffffffu, e[k], o);
                if (lane == 0) b.gke[(size_t)item * 8 + k] = e[k];
            }
        }
    }
}

// The energy records of a write step: an instance's tiles and row blocks are
// contiguous in the lists
__device__ void grid_energy_mixed(const Batch& b, const double* pe, int rec, double (*sh)[32])
{
    for (int k = blockIdx.x; k < b.ninst; k += gridDim.x) {
        const int inst = b.order[k];
        const int nb = (b.cnt[inst] + kBlock - 1) / kBlock;
        const long long b0 = b.gblk_off[k];
        double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (long long u = b.gtile_off[k] + threadIdx.x; u < b.gtile_off[k + 1]; u += blockDim.x) e[0] += pe[u];
        for (int i = threadIdx.x; i < nb; i += blockDim.x)
#pragma unroll
            for (int j = 0; j < 7; ++j) e[1 + j] += b.gke[(size_t)(b0 + i) * 8 + j];
        batch::cta_sum8(e, sh);
        if (threadIdx.x == 0)
            for (int j = 0; j < 8; ++j) b.energy[((size_t)inst * b.nrec + rec) * 8 + j] = e[j];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(32 * kGridWarpsM, 1) batch_mixed_grid_kernel(const __grid_constant__ Batch b,
                                                                               int first_step, int nsteps, int skip,
                                                                               int do_init)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ double sh[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    TileSmem& sm = reinterpret_cast<TileSmem*>(tile_raw)[warp];
    unsigned long long phase = 0;
    const int q0 = do_init ? -1 : 0;
    if (q0 >= nsteps) return;
    for (int item = blockIdx.x * kGridWarpsM + warp; item < b.gblocks; item += gridDim.x * kGridWarpsM) {
        const int inst = b.gblk_inst[item], p = b.gblk[item] * kBlock + lane;
        if (p < b.cnt[inst])
            drift_sphere(b, b.off[inst] + p, b.perm[b.off[inst] + p], do_init ? 0.0 : b.dt[inst]);
    }
    if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
    int rec = -1;  // the record whose parts the last rows phase left
    for (int q = q0; q < nsteps; ++q) {
        const int step = first_step + q, par = q & 1;
        const bool init = q < 0, write = init || (skip > 0 && step % skip == 0), more = q + 1 < nsteps;
        if (rec >= 0) grid_energy_mixed(b, b.gpe + (par ^ 1) * b.gtiles, rec, sh);
        if (write)
            grid_pairs_mixed<true>(b, sm, b.gqueue + par, b.gpe + par * b.gtiles);
        else
            grid_pairs_mixed<false>(b, sm, b.gqueue + par, b.gpe + par * b.gtiles);
        if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) b.gqueue[par ^ 1] = 0;  // the next step's queue
        grid_rows_mixed(b, init, write, more);
        rec = !write ? -1 : init ? 0 : min(step / skip, b.nrec - 1);
        if (!more && rec < 0) break;
        if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
        if (!more) grid_energy_mixed(b, b.gpe + par * b.gtiles, rec, sh);
    }
}

}  // namespace

// Dynamic shared memory of the pair-tile kernels; the attribute belongs to
// the current device's context, and setting it is a host-side table update.
template <typename K>
static size_t tile_smem(K kernel, int warps)
{
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, warps * (int)sizeof(TileSmem));
    return (size_t)warps * sizeof(TileSmem);
}

cudaError_t launch_batch_mixed_grid(const Batch& b, int num_sms, int first_step, int nsteps, int skip, int do_init,
                                    cudaStream_t st)
{
    return launch_cooperative(batch_mixed_grid_kernel, num_sms, 32 * kGridWarpsM,
                              tile_smem(batch_mixed_grid_kernel, kGridWarpsM), st, b, first_step, nsteps, skip,
                              do_init);
}

bool batch_mixed_grid_fits()
{
    int nb = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_mixed_grid_kernel, 32 * kGridWarpsM,
                                                         tile_smem(batch_mixed_grid_kernel, kGridWarpsM)) ==
               cudaSuccess && nb >= 1;
}

void launch_batch_mixed(const Batch& b, int tile, int threads, int blocks, int first_step, int nsteps, int skip,
                        int do_init, cudaStream_t st)
{
    switch (tile) {
        case 0:
            batch_mixed_tiles_kernel<<<blocks, threads, tile_smem(batch_mixed_tiles_kernel, threads / 32), st>>>(
                b, first_step, nsteps, skip, do_init);
            break;
        case 32: batch_mixed_kernel<32><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
        case 64: batch_mixed_kernel<64><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
        default: batch_mixed_kernel<128><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
    }
}

int batch_mixed_max_blocks_per_sm(int tile, int threads)
{
    int nb = 0;
    switch (tile) {
        case 0:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_mixed_tiles_kernel, threads,
                                                          tile_smem(batch_mixed_tiles_kernel, threads / 32));
            break;
        case 32: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_mixed_kernel<32>, threads, 0); break;
        case 64: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_mixed_kernel<64>, threads, 0); break;
        default: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_mixed_kernel<128>, threads, 0); break;
    }
    return nb;
}

}  // namespace sl
