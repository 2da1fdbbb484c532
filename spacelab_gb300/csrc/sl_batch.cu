// sl_batch.cu -- batched exact FP64 solver: thousands of independent
// systems (projectile-target collisions of uneven sphere counts) advanced by
// ONE persistent launch.
//
// The pair-tile pass runs in lockstep where that balances better (in the exact
// form always): a cooperative launch of one CTA per SM in which all instances
// take a step together, their tiles and rows being one queue each and the
// phases separated by a grid barrier (bounded; runs_in_lockstep in
// sl_batch_capi.cu).  Otherwise each CTA takes whole instances from an atomic
// work queue (largest first) and runs all of an instance's steps before taking
// the next one; the only synchronisation is then __syncthreads inside the CTA.
// The state is the same bit for bit.  The energy records hold the same terms
// summed in another order, which in lockstep depends on where the batch's strips
// begin, and so on the other instances (1e-10 of the largest total).
//
// Within an instance a step is the reference's three passes
// (ColliderSingleCore.cpp:82-97, 100-256, 263-287):
//   drift    one thread per sphere (strided);
//   pairs    either the pair-tile pass (shape tile 0: every pair once into
//            the CTA's pair-term buffers by the single system's tile routine,
//            then ordered row sums), or the per-sphere loop: thread i walks
//            partners j ascending through j-tiles staged in shared memory and
//            adds each term to its running sum in the order the reference
//            adds them to acc[i].  Either way the result is bit-identical to
//            the reference step, pair terms being computed in the
//            reference's (A = max, B = min) orientation;
//   kick     pass 3, plus the write-step energy totals reduced in a fixed
//            tree inside the CTA.
// The pass, its j-tile size and the threads per instance (block size) are
// chosen by the host autotuner (sl_batch_capi.cu).
#include "sl_batch.h"
#include "sl_batch_common.cuh"
#include "sl_fp64_exact.cuh"
#include "sl_pair_exact.cuh"
#include "sl_tile_exact.cuh"
#include "sl_vdw_energy.cuh"

namespace sl {

namespace {

using batch::cta_sum8;
using batch::drift;
using batch::kick;

template <int TILE>
struct JTile {
    double x[TILE], y[TILE], z[TILE], R[TILE], twoR[TILE], fourR[TILE], cR3[TILE];
};

// Pass 2 for one instance; returns this thread's share of the PE (pairs
// are counted once, by the thread of sphere A).
template <int TILE, bool WRITE>
__device__ double pair_pass(const Batch& b, int off, int n, const Material& M, double kin, double kout,
                            JTile<TILE>& jt)
{
    double pe = 0;
    for (int ibase = 0; ibase < n; ibase += blockDim.x) {
        const int i = ibase + threadIdx.x;
        const bool active = i < n;
        const int gi = off + (active ? i : 0);
        const double xi = b.pos.c[0][gi], yi = b.pos.c[1][gi], zi = b.pos.c[2][gi];
        const double Ri = b.R[gi], twoRi = b.twoR[gi], fourRi = b.fourR[gi], cR3i = b.cR3[gi];
        const double mi = b.m[gi], moii = b.moi[gi], imoii = b.inv_moi[gi];
        const unsigned long long rmi = b.rm[gi];
        double ax = 0, ay = 0, az = 0, tx = 0, ty = 0, tz = 0;
        for (int jbase = 0; jbase < n; jbase += TILE) {
            for (int t = threadIdx.x; t < TILE; t += blockDim.x) {
                const int j = jbase + t;
                if (j < n) {
                    const int g = off + j;
                    jt.x[t] = b.pos.c[0][g]; jt.y[t] = b.pos.c[1][g]; jt.z[t] = b.pos.c[2][g];
                    jt.R[t] = b.R[g]; jt.twoR[t] = b.twoR[g]; jt.fourR[t] = b.fourR[g]; jt.cR3[t] = b.cR3[g];
                }
            }
            __syncthreads();
            if (active) {
                const int jend = min(TILE, n - jbase);
                for (int t = 0; t < jend; ++t) {
                    const int j = jbase + t;
                    if (j == i) continue;
                    const bool iA = i > j;  // the reference's orientation: A = max, B = min
                    const double Ax = iA ? xi : jt.x[t], Ay = iA ? yi : jt.y[t], Az = iA ? zi : jt.z[t];
                    const double Bx = iA ? jt.x[t] : xi, By = iA ? jt.y[t] : yi, Bz = iA ? jt.z[t] : zi;
                    const double RA = iA ? Ri : jt.R[t], RB = iA ? jt.R[t] : Ri;
                    const double twoRA = iA ? twoRi : jt.twoR[t], twoRB = iA ? jt.twoR[t] : twoRi;
                    const double fourRA = iA ? fourRi : jt.fourR[t], cR3A = iA ? cR3i : jt.cR3[t];
                    const double sumRaRb = RA + RB;                                  // :104
                    const double rx = Bx - Ax, ry = By - Ay, rz = Bz - Az;           // :105
                    const double d2 = rx * rx + ry * ry + rz * rz;
                    int p;
                    unsigned long long F;
                    const unsigned long long Y = rsqrt_fix(d2, p, F);
                    const double dist = sqrt_fix(d2, F, Y, p);                       // :107
                    const double overlap = sumRaRb - dist;                           // :110
                    double fx, fy, fz;
                    if (overlap > 0) {
                        const int gA = off + (iA ? i : j), gB = off + (iA ? j : i);
                        ContactIn in;
                        for (int c = 0; c < 3; ++c) {
                            in.prevA[c] = b.prev.c[c][gA]; in.prevB[c] = b.prev.c[c][gB];
                            in.wA[c] = b.w.c[c][gA]; in.wB[c] = b.w.c[c][gB];
                            in.vA[c] = b.vel.c[c][gA]; in.vB[c] = b.vel.c[c][gB];
                        }
                        in.mA = b.m[gA]; in.mB = b.m[gB]; in.kin = kin; in.kout = kout;
                        const ContactOut o = contact_pair_exact<WRITE>(in, M, rx, ry, rz, dist, overlap, RA, RB,
                                                                       twoRA, twoRB, fourRA, cR3A);
                        fx = o.fx; fy = o.fy; fz = o.fz;
                        const double qx = iA ? o.tax : o.tbx, qy = iA ? o.tay : o.tby, qz = iA ? o.taz : o.tbz;
                        tx += div_by_recip(qx, moii, imoii);                         // :187-188
                        ty += div_by_recip(qy, moii, imoii);
                        tz += div_by_recip(qz, moii, imoii);
                        if (WRITE && iA) pe += o.pe;
                    } else {
                        double h = fabs(overlap);                                    // :211-215
                        if (h < M.h_min) h = M.h_min;
                        const double coef = vdw_coef_fix(h, RA, RB, twoRA, twoRB, fourRA, cR3A);
                        fx = coef * div_by_rsqrt(rx, dist, Y, p);
                        fy = coef * div_by_rsqrt(ry, dist, Y, p);
                        fz = coef * div_by_rsqrt(rz, dist, Y, p);
                        if (WRITE && iA) pe += vdw_energy_far_df(M.Ha, h, RA, RB, twoRA);
                    }
                    const double qx = div_by_fixed<false>(fx, mi, rmi);              // :249-250
                    const double qy = div_by_fixed<false>(fy, mi, rmi);
                    const double qz = div_by_fixed<false>(fz, mi, rmi);
                    if (iA) { ax += qx; ay += qy; az += qz; }
                    else { ax -= qx; ay -= qy; az -= qz; }
                }
            }
            __syncthreads();
        }
        if (active) {
            b.acc.c[0][gi] = ax; b.acc.c[1][gi] = ay; b.acc.c[2][gi] = az;
            b.aacc.c[0][gi] = tx; b.aacc.c[1][gi] = ty; b.aacc.c[2][gi] = tz;
        }
    }
    return pe;
}

template <int TILE>
__global__ void __launch_bounds__(256) batch_exact_kernel(const __grid_constant__ Batch b, int first_step, int nsteps,
                                                          int skip, int do_init)
{
    __shared__ JTile<TILE> jt;
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
        if (do_init) {  // initial forces: a step with dt = 0 (init_conditions)
            drift(b, off, n, 0.0);
            __syncthreads();
            const double pe = pair_pass<TILE, true>(b, off, n, M, kin, kout, jt);
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
                pe = pair_pass<TILE, true>(b, off, n, M, kin, kout, jt);
            else
                pair_pass<TILE, false>(b, off, n, M, kin, kout, jt);
            __syncthreads();
            const int r = write ? step / skip : 0;
            kick(b, inst, off, n, dt, write, pe, recs + (size_t)(r < b.nrec ? r : b.nrec - 1) * 8, sh);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Pair-tile pass (shape tile 0): every pair once, as the single-system step
// does it.  The CTA's warps take the instance's 32 x 32 block tiles and run
// the single system's tile routine (tile_pairs, sl_tile_exact.cuh) on a
// System view of the instance whose pair-term, torque and contact buffers are
// the CTA's scratch; then thread (c, i) adds row i of the pair terms in
// ascending partner order and its contact torques likewise -- the
// reference's order, so the result stays bit-identical -- and the half-kick
// follows.  This evaluates each pair once where the per-sphere loop does it
// twice, at the price of the row sums' dependent FP64 adds.
__device__ void make_view(System& v, const Batch& b, int inst, int off, int n, int npad, double* pair, double* torq,
                          uint32_t* mask)
{
    v = System{};
    v.n = n;
    v.nb = (n + kBlock - 1) / kBlock;
    v.npad = npad;  // the buffers' row stride
    v.ntiles = (long long)v.nb * (v.nb + 1) / 2;
    v.nitems = v.ntiles;
    const Vec3Soa* src[8] = {&b.pos, &b.prev, &b.vel, &b.velh, &b.w, &b.wh, &b.acc, &b.aacc};
    Vec3Soa* dst[8] = {&v.pos, &v.prev, &v.vel, &v.velh, &v.w, &v.wh, &v.acc, &v.aacc};
    for (int k = 0; k < 8; ++k)
        for (int c = 0; c < 3; ++c) dst[k]->c[c] = src[k]->c[c] + off;
    v.R = b.R + off; v.m = b.m + off; v.moi = b.moi + off;
    v.twoR = b.twoR + off; v.fourR = b.fourR + off; v.cR3 = b.cR3 + off;
    v.rm = b.rm + off; v.inv_moi = b.inv_moi + off;
    v.pairbuf = pair;
    v.torqbuf = torq;
    v.cmask = mask;
    v.sc = b.isc + inst;
    v.mat = b.mat;
    v.mat.u_s = b.u_s[inst];
}

template <bool WRITE>
__device__ double exact_tile_pass(const System& s, TileScratch* scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    TileScratch& ws = scratch[warp];
    const int n = s.n;
    double pe = 0;
    for (long long t = warp; t < s.ntiles; t += nwarps) {
        int X, Y;
        tile_coords(t, X, Y);
        load_a(s, ws.ab, lane, min(X * kBlock + lane, n - 1));  // padding rows repeat the last sphere (never paired)
        __syncwarp();
        const int B = Y * kBlock + lane;
        uint32_t rowbits, colbits;
        tile_pairs<WRITE ? kPeInline : kNoPe>(s, ws, X, Y, lane, 0, min(kBlock, n - X * kBlock), min(B, n - 1), B < n, pe, rowbits,
                          colbits);
        store_contacts(s, X, Y, lane, -1, rowbits, colbits);
        __syncwarp();
    }
    return pe;
}

// Thread (c, i): acc_c[i] and aacc_c[i] in the reference's order
// (ColliderSingleCore.cpp:100-103, 249-250): partners j < i, then j > i.
__device__ void exact_row_sums(const System& s)
{
    const int n = s.n;
    const size_t plane = (size_t)s.npad * s.npad;
    for (int t = threadIdx.x; t < 3 * n; t += blockDim.x) {
        const int c = t / n, i = t - c * n;
        const double* row = s.pairbuf + c * plane + (size_t)i * s.npad;
        double acc = 0;
        for (int j = 0; j < i; ++j) acc += row[j];
        for (int j = i + 1; j < n; ++j) acc += row[j];
        const double* trow = s.torqbuf + c * plane + (size_t)i * s.npad;
        const uint32_t* mrow = s.cmask + (size_t)i * s.nb;
        double aacc = 0;
        for (int Y = 0; Y < s.nb; ++Y) {
            uint32_t wd = mrow[Y];
            while (wd) {
                const int j = Y * kBlock + __ffs(wd) - 1;
                wd &= wd - 1;
                aacc += trow[j];
            }
        }
        s.acc.c[c][i] = acc;
        s.aacc.c[c][i] = aacc;
    }
}

constexpr int kExactTileWarps = 8;

__global__ void __launch_bounds__(32 * kExactTileWarps) batch_exact_tiles_kernel(const __grid_constant__ Batch b,
                                                                                int first_step, int nsteps, int skip,
                                                                                int do_init)
{
    extern __shared__ __align__(16) unsigned char tile_raw[];
    TileScratch* scratch = reinterpret_cast<TileScratch*>(tile_raw);  // one per warp
    __shared__ System sv;
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
        const double dt = b.dt[inst];
        double* recs = b.energy + (size_t)inst * b.nrec * 8;
        if (threadIdx.x == 0) make_view(sv, b, inst, off, n, b.x_np, b.xpair + (size_t)blockIdx.x * b.xpair_cta,
                                        b.xtorq + (size_t)blockIdx.x * b.xpair_cta,
                                        b.xmask + (size_t)blockIdx.x * b.xmask_cta);
        __syncthreads();
        if (do_init) {
            drift(b, off, n, 0.0);
            __syncthreads();
            const double pe = exact_tile_pass<true>(sv, scratch);
            __syncthreads();
            exact_row_sums(sv);
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
                pe = exact_tile_pass<true>(sv, scratch);
            else
                exact_tile_pass<false>(sv, scratch);
            __syncthreads();
            exact_row_sums(sv);
            __syncthreads();
            const int r = write ? step / skip : 0;
            kick(b, inst, off, n, dt, write, pe, recs + (size_t)(r < b.nrec ? r : b.nrec - 1) * 8, sh);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// Lockstep form of the pair-tile pass: all instances take a step together, one
// phase over the items of all of them, then the next, with a barrier over the
// grid between (a cooperative launch, one CTA per SM).  In the form above an
// instance's step is one CTA's latency -- its tiles taken by a few warps, then
// its rows' dependent adds -- and the batch waits for its largest instances;
// here every warp has work until a phase's last items, and only the phases'
// order is kept.  It needs pair-term buffers for every instance (48 npad^2
// bytes each), so it is taken where they fit the budget (sl_batch_capi.cu).
//
//   pairs   items (tiles, or strips of 8 rows as strip_from says) from a queue
//   rows    one warp per (component, 32-row block): the ordered sums and pass
//           3, and on plain steps the next step's pass 1 of the same rows
//   energy  write steps: one CTA per instance, then pass 1 of the next step
constexpr int kGridWarps = 16;

struct GridWarp {
    TileScratch scratch;
    System view;
    int inst;
};

// Row i's ordered sum of the pair terms: every entry is added, the row's own
// column and the padding too, which are never written and hold +0.0.  16
// bytes a load, 8 loads ahead of the adds.
__device__ __forceinline__ double ordered_row(const double* row, int n)
{
    constexpr int kBatch = 8;
    const double2* p = reinterpret_cast<const double2*>(row);
    const int nq = (n + 1) / 2;
    double2 cur[kBatch], nxt[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) cur[k] = k < nq ? __ldcs(p + k) : make_double2(0.0, 0.0);
    double sum = 0.0;
    for (int q = 0; q < nq; q += kBatch) {
#pragma unroll
        for (int k = 0; k < kBatch; ++k)
            nxt[k] = q + kBatch + k < nq ? __ldcs(p + q + kBatch + k) : make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            sum += cur[k].x;
            sum += cur[k].y;
            cur[k] = nxt[k];
        }
    }
    return sum;
}

// Pass 1 of one component of one sphere (:84-90)
__device__ __forceinline__ void drift_one(const System& s, int c, int i, double v, double w, double acc, double aacc,
                                          double dt)
{
    const double vh = v + (.5 * acc) * dt;
    const double whc = w + (.5 * aacc) * dt;
    const double p = s.pos.c[c][i];
    s.velh.c[c][i] = vh;
    s.wh.c[c][i] = whc;
    s.prev.c[c][i] = p;
    s.pos.c[c][i] = p + vh * dt;
}

// Pass 1 of every sphere
__device__ void grid_drift(const Batch& b, bool init)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kGridWarps + (threadIdx.x >> 5), nw = gridDim.x * kGridWarps;
    for (int item = gw; item < 3 * b.gblocks; item += nw) {
        const int blk = item / 3, c = item - 3 * blk;
        const int inst = b.gblk_inst[blk], i = b.gblk[blk] * kBlock + lane;
        const System& s = b.views[inst];
        if (i < s.n)
            drift_one(s, c, i, s.vel.c[c][i], s.w.c[c][i], s.acc.c[c][i], s.aacc.c[c][i], init ? 0.0 : b.dt[inst]);
    }
}

template <bool WRITE>
__device__ void grid_pairs(const Batch& b, GridWarp& gw, int num_sms, int* queue, double* pe_out)
{
    const int lane = threadIdx.x & 31;
    const long long split = strip_from(b.gtiles, num_sms);
    const long long items = split + kStrips * (b.gtiles - split);
    const long long nw = (long long)gridDim.x * kGridWarps;
    for (long long q = (long long)blockIdx.x * kGridWarps + (threadIdx.x >> 5); q < items;) {
        const bool whole = q < split;
        const long long u = whole ? q : split + (q - split) / kStrips;
        const int strip = whole ? -1 : (int)((q - split) % kStrips);
        const int4 tile = __ldg(b.gtile + u);
        const int inst = tile.x, X = tile.w >> 16, Y = tile.w & 0xffff;
        if (inst != gw.inst) {  // the instance's view, by the whole warp
            __syncwarp();
            const uint32_t* src = reinterpret_cast<const uint32_t*>(b.views + inst);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&gw.view);
            for (int w = lane; w < (int)(sizeof(System) / 4); w += 32) dst[w] = src[w];
            if (lane == 0) gw.inst = inst;
            __syncwarp();
        }
        const System& s = gw.view;
        load_a(s, gw.scratch.ab, lane, min(X * kBlock + lane, s.n - 1));
        __syncwarp();
        const int B = Y * kBlock + lane;
        const int a_end = min(kBlock, s.n - X * kBlock);
        const int a0 = whole ? 0 : strip * kStripRows, a1 = whole ? a_end : min(a_end, a0 + kStripRows);
        double pe = 0;
        uint32_t rowbits, colbits;
        tile_pairs<WRITE ? kPeInline : kNoPe>(s, gw.scratch, X, Y, lane, a0, a1, min(B, s.n - 1), B < s.n, pe, rowbits, colbits);
        store_contacts(s, X, Y, lane, strip, rowbits, colbits);
        if (WRITE) {
            for (int o = 16; o > 0; o >>= 1) pe += __shfl_xor_sync(0xffffffffu, pe, o);
            if (lane == 0) pe_out[q] = pe;
        }
        __syncwarp();
        int next = 0;
        if (lane == 0) next = atomicAdd(queue, 1);
        q = nw + __shfl_sync(0xffffffffu, next, 0);
    }
}

// Ordered sums and pass 3; drift_next: the following step's pass 1 too
__device__ void grid_rows(const Batch& b, bool init, bool drift_next)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kGridWarps + (threadIdx.x >> 5), nw = gridDim.x * kGridWarps;
    for (int item = gw; item < 3 * b.gblocks; item += nw) {
        const int blk = item / 3, c = item - 3 * blk;
        const int inst = b.gblk_inst[blk], i = b.gblk[blk] * kBlock + lane;
        const System& s = b.views[inst];
        if (i >= s.n) continue;  // no warp-wide operation below
        const size_t plane = (size_t)s.npad * s.npad;
        const double acc = ordered_row(s.pairbuf + c * plane + (size_t)i * s.npad, s.n);
        const double* trow = s.torqbuf + c * plane + (size_t)i * s.npad;
        const uint32_t* mrow = s.cmask + (size_t)i * s.nb;
        double aacc = 0;
        for (int Y = 0; Y < s.nb; ++Y) {
            uint32_t wd = mrow[Y];
            while (wd) {
                const int j = Y * kBlock + __ffs(wd) - 1;
                wd &= wd - 1;
                aacc += trow[j];
            }
        }
        s.acc.c[c][i] = acc;
        s.aacc.c[c][i] = aacc;
        const double dt = init ? 0.0 : b.dt[inst];
        const double v = s.velh.c[c][i] + (.5 * acc) * dt;    // :265
        const double wv = s.wh.c[c][i] + (.5 * aacc) * dt;    // :266
        s.vel.c[c][i] = v;
        s.w.c[c][i] = wv;
        if (!isfinite(v) || !isfinite(wv) || !isfinite(s.pos.c[c][i])) atomicOr(&b.status[inst], 1u);
        if (drift_next) drift_one(s, c, i, v, wv, acc, aacc, b.dt[inst]);
    }
}

// The energy records of a write step, one CTA per instance
__device__ void grid_energy(const Batch& b, int num_sms, const double* pe, int rec, double (*sh)[32])
{
    const long long split = strip_from(b.gtiles, num_sms);
    const auto first_item = [split](long long u) { return u <= split ? u : split + (u - split) * kStrips; };
    for (int k = blockIdx.x; k < b.ninst; k += gridDim.x) {
        const int inst = b.order[k];
        const System& s = b.views[inst];
        double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (long long q = first_item(b.gtile_off[k]) + threadIdx.x; q < first_item(b.gtile_off[k + 1]); q += blockDim.x)
            e[0] += pe[q];
        for (int i = threadIdx.x; i < s.n; i += blockDim.x) {
            const double m = s.m[i], moi = s.moi[i];
            const double vx = s.vel.c[0][i], vy = s.vel.c[1][i], vz = s.vel.c[2][i];
            const double wx = s.w.c[0][i], wy = s.w.c[1][i], wz = s.w.c[2][i];
            const double px = s.pos.c[0][i], py = s.pos.c[1][i], pz = s.pos.c[2][i];
            e[1] += .5 * m * (vx * vx + vy * vy + vz * vz) + .5 * moi * (wx * wx + wy * wy + wz * wz);
            e[2] += m * vx; e[3] += m * vy; e[4] += m * vz;
            e[5] += m * (py * vz - pz * vy) + moi * wx;
            e[6] += m * (pz * vx - px * vz) + moi * wy;
            e[7] += m * (px * vy - py * vx) + moi * wz;
        }
        cta_sum8(e, sh);
        if (threadIdx.x == 0)
            for (int j = 0; j < 8; ++j) b.energy[((size_t)inst * b.nrec + rec) * 8 + j] = e[j];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(32 * kGridWarps, 1) batch_exact_grid_kernel(const __grid_constant__ Batch b,
                                                                              int num_sms, int first_step, int nsteps,
                                                                              int skip, int do_init)
{
    extern __shared__ __align__(16) unsigned char grid_raw[];
    GridWarp& gw = reinterpret_cast<GridWarp*>(grid_raw)[threadIdx.x >> 5];
    __shared__ double sh[8][32];
    if ((threadIdx.x & 31) == 0) gw.inst = -1;
    __syncwarp();
    const long long items = strip_from(b.gtiles, num_sms) + kStrips * (b.gtiles - strip_from(b.gtiles, num_sms));
    unsigned long long phase = 0;
    const int q0 = do_init ? -1 : 0;
    if (q0 >= nsteps) return;
    grid_drift(b, do_init != 0);
    if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
    for (int q = q0; q < nsteps; ++q) {
        const int step = first_step + q, par = q & 1;
        const bool init = q < 0, write = init || (skip > 0 && step % skip == 0), more = q + 1 < nsteps;
        double* pe = b.gpe + par * items;
        if (write)
            grid_pairs<true>(b, gw, num_sms, b.gqueue + par, pe);
        else
            grid_pairs<false>(b, gw, num_sms, b.gqueue + par, pe);
        if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) b.gqueue[par ^ 1] = 0;  // the next step's queue
        grid_rows(b, init, more && !write);
        if (!more && !write) break;
        if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
        if (write) {
            const int r = init ? 0 : min(step / skip, b.nrec - 1);
            grid_energy(b, num_sms, pe, r, sh);
            if (!more) break;
            if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
            grid_drift(b, false);
            if (!batch::grid_sync(b.gsync, phase, b.give_up)) return;
        }
    }
}

__global__ void batch_views_kernel(const __grid_constant__ Batch b)
{
    const int inst = blockIdx.x * blockDim.x + threadIdx.x;
    if (inst >= b.ninst) return;
    const int n = b.cnt[inst];
    System v;
    make_view(v, b, inst, b.off[inst], n, (n + kBlock - 1) / kBlock * kBlock, b.xpair + b.gpair_off[inst],
              b.xtorq + b.gpair_off[inst], b.xmask + b.gmask_off[inst]);
    b.views[inst] = v;
}

__global__ void batch_derive_kernel(const __grid_constant__ Batch b)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b.total) return;
    const double R = b.R[i], m = b.m[i], moi = b.moi[i];
    b.twoR[i] = 2 * R;
    b.fourR[i] = 4 * R;
    b.cR3[i] = b.mat.Ha / 6 * 64 * R * R * R;
    b.rm[i] = recip_of(m);
    b.inv_moi[i] = 1.0 / moi;
    if (b.f_R) {  // mixed form: slot i holds sphere perm[i]
        const int g = b.perm[i];
        const double Rg = b.R[g];
        const float rh = d2f_bits(Rg, b.len_shift);
        b.f_R[i] = rh;
        b.f_Rlo[i] = d2f_bits(Rg - f2d_bits(rh) * ldexp(1.0, b.len_shift), b.len_shift);
        b.f_inv_m[i] = d2f_bits(1.0 / b.m[g], 0);
        b.f_inv_moi[i] = d2f_bits(1.0 / b.moi[g], 0);
    }
}

}  // namespace

void launch_batch_derive(const Batch& b, cudaStream_t st)
{
    batch_derive_kernel<<<(b.total + 255) / 256, 256, 0, st>>>(b);
    if (b.views) batch_views_kernel<<<(b.ninst + 63) / 64, 64, 0, st>>>(b);
}

static size_t exact_grid_smem()
{
    cudaFuncSetAttribute(batch_exact_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kGridWarps * (int)sizeof(GridWarp));
    return kGridWarps * sizeof(GridWarp);
}

cudaError_t launch_batch_exact_grid(const Batch& b, int num_sms, int first_step, int nsteps, int skip, int do_init,
                                    cudaStream_t st)
{
    return launch_cooperative(batch_exact_grid_kernel, num_sms, 32 * kGridWarps, exact_grid_smem(), st, b, num_sms,
                              first_step, nsteps, skip, do_init);
}

bool batch_grid_fits(bool mixed)
{
    if (mixed) return batch_mixed_grid_fits();
    int nb = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_exact_grid_kernel, 32 * kGridWarps,
                                                         exact_grid_smem()) == cudaSuccess && nb >= 1;
}

long long batch_grid_items(long long tiles, int num_sms, bool mixed)
{
    const long long split = mixed ? tiles : strip_from(tiles, num_sms);
    return split + kStrips * (tiles - split);
}

// Dynamic shared memory of the pair-tile pass (above the 48 KB that need no
// opt-in at eight warps); the attribute belongs to the current device's
// context, and setting it is a host-side table update.
static size_t exact_tiles_smem(int threads)
{
    cudaFuncSetAttribute(batch_exact_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kExactTileWarps * (int)sizeof(TileScratch));
    return (size_t)(threads / 32) * sizeof(TileScratch);
}

void launch_batch_exact(const Batch& b, int tile, int threads, int blocks, int first_step, int nsteps, int skip,
                        int do_init, cudaStream_t st)
{
    switch (tile) {
        case 0:
            batch_exact_tiles_kernel<<<blocks, threads, exact_tiles_smem(threads), st>>>(b, first_step, nsteps, skip,
                                                                                        do_init);
            break;
        case 32: batch_exact_kernel<32><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
        case 64: batch_exact_kernel<64><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
        default: batch_exact_kernel<128><<<blocks, threads, 0, st>>>(b, first_step, nsteps, skip, do_init); break;
    }
}

int batch_max_blocks_per_sm(int tile, int threads, bool mixed)
{
    if (mixed) return batch_mixed_max_blocks_per_sm(tile, threads);
    int nb = 0;
    switch (tile) {
        case 0:
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_exact_tiles_kernel, threads,
                                                          exact_tiles_smem(threads));
            break;
        case 32: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_exact_kernel<32>, threads, 0); break;
        case 64: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_exact_kernel<64>, threads, 0); break;
        default: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_exact_kernel<128>, threads, 0); break;
    }
    return nb;
}

}  // namespace sl
