// tma_pair.cu -- the smoothing passes of large levels with FP32 records, on grids
// without periodic axes: red and black half-steps from zero down, black and
// red up, planes staged by the Tensor Memory Accelerator.
//
// With 16-byte records a pass is bound by their HBM and L2 traffic and by the
// shared memory of their planes, and a third half-step (tma_fused.cu) costs more
// than it saves: 43 and 46 us a pass against 28 and 27 on 128^3, for 16 CG
// iterations instead of 20 (jet 196x310x18: 14.3 ms a projection against 12.3).
//
//   down, from zero:  e_r = r/d;  e_b = (r + sum beta e_r)/d;  the residual of
//                     the red cells is restricted (a black cell's is zero)
//   up:               e_b = (r + sum beta e_r)/d;  e_r = (r + sum beta e_b)/d
//
//  * One thread with no other task issues, per plane, one
//    cp.async.bulk.tensor copy of each input: the smoother records (a 4-D box
//    over the split rows: half-row columns, even/odd half, y, z) and the level
//    vectors (3-D boxes of RH rows from x0-4, so the first coordinate is
//    16-byte aligned).  The copies of a plane complete on one mbarrier; two
//    mbarriers alternate between planes.  Cells outside the grid arrive as
//    zeros, the closed wall.
//  * 224 threads take at most one task in every stage (216 red/prolongation
//    quads, 180 black quads, 128 tile quads).  The 16 interior quads of a
//    staged row go to one half-warp, so its shared-memory accesses are
//    contiguous; the halo quads of all rows follow.
//  * Records and corrections sit in five-slot rings (planes zA-3 .. zA+1), so
//    a step needs two barriers: warps that finish the tile stage of plane zA-2
//    go on to the next plane's red stage while others are still busy.
//
// Every wait on an mbarrier is bounded: when it runs out the block stops
// issuing copies, marks the solve as stalled and converged (the host reports a
// timeout), and finishes its loop without waiting again.
#include <algorithm>

#include "kernels.h"
#include "fused_common.cuh"
#include "tma_common.cuh"

namespace mhdproj {

namespace {
using namespace staged;
using namespace fused;
using namespace tma;

struct PGeo {
    static constexpr int FTY = 8;                      // tile rows
    static constexpr int RH = FTY + 4;                 // staged rows y0-2 .. y0+FTY+1
    static constexpr int NRED = RH * NQ;               // red / prolongation quads
    static constexpr int NBR = FTY + 2;                // black rows y0-1 .. y0+FTY
    static constexpr int NBLK = NBR * NQ;              // black quads
    static constexpr int NOWN = QX * FTY;              // tile quads
    static constexpr int NT = (NRED + 32) / 32 * 32;   // threads: one red task each, and a spare issuing thread
    static constexpr int NS = 5;                       // ring slots of records and corrections: zA-3 .. zA+1
    static_assert(NBLK <= NT && NOWN <= NT && NRED < NT, "one task per thread");
};
constexpr int VW = RW;  // staged rows of a level vector: x0-4 .. x0+67
constexpr int CVW = 44, CVH = PGeo::RH / 2;  // staged coarse rows: x0/2-8 .. x0/2+35, y0/2-1 .. y0/2+4

// Shared memory of the pre-smoothing pass: records and corrections of planes
// zA-3 .. zA+1 (five slots), the copied residual and q of planes zA, zA+1.
template <bool UPDATE>
struct PairPreSm {
    using G = PGeo;
    alignas(128) float4 c[G::NS][G::RH][RW];
    alignas(128) float rv[2][G::RH][VW];
    alignas(128) float qv[UPDATE ? 2 : 1][UPDATE ? G::RH : 1][VW];
    alignas(16) float er[G::NS][G::RH][RW];
    float2 ypart[G::FTY][QX];
    unsigned long long bar[2];
    int abort_;
};
// Shared memory of the post-smoothing pass: records and smoothed corrections
// of planes zA-3 .. zA+1, the copied pre-smoothed correction and right-hand
// side of planes zA, zA+1, and (COPY) the coarse planes of two pairs of planes.
template <bool COPY>
struct PairPostSm {
    using G = PGeo;
    alignas(128) float ec[COPY ? 2 : 1][COPY ? (CVH * CVW + 31) / 32 * 32 : 32];
    alignas(128) float4 c[G::NS][G::RH][RW];
    alignas(128) float ev[2][G::RH][VW];
    alignas(128) float rv[2][G::RH][VW];
    alignas(16) float ep[G::NS][G::RH][RW];
    unsigned long long bar[2];
    int abort_;
};
}  // namespace

// ------------------------------------------------------ pre-smoothing pass
// rin and q arrive through tm_r
// and tm_q, the records through tm_rec.  A step handles the red stage of
// plane zA, the black stage of zA-1 and the tile stage of zA-2 with two
// barriers: the five-slot rings let the next step's copies and red stage
// start while other warps still finish the tile stage.
template <bool UPDATE, bool FINE>
__global__ void __launch_bounds__(PGeo::NT, 2)
    k_pre_pair(const __grid_constant__ CUtensorMap tm_rec, const __grid_constant__ CUtensorMap tm_r,
              const __grid_constant__ CUtensorMap tm_q, Grid3 g, Grid3 gc, float* __restrict__ r_out,
              float* __restrict__ e, float* __restrict__ rc, Scalars* sc, double* partials, int nblocks) {
    if (sc->converged) return;
    using G = PGeo;
    using SM = PairPreSm<UPDATE>;
    constexpr int FTY = G::FTY, NT = G::NT, RH = G::RH, NS = G::NS, SL = RH * RW;
    constexpr unsigned BYTES =
        RH * RW * sizeof(float4) + RH * VW * sizeof(float) + (UPDATE ? RH * VW * 4 : 0);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SM& S = aligned_smem<SM>(smem_raw);
    __shared__ double sh[NT / 32];
    const int t = threadIdx.x;
    constexpr int ISSUER = NT - 1;  // no task in any stage
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float alpha = UPDATE ? sc->alpha_f : 0.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * FTY;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const int zs = z0 - 2, nsteps = z1 - z0 + 4;  // planes zs .. z1+1
    const long long sxy = (long long)g.nx * g.ny;
    int last_issued = 0;
    auto issue = [&](int k, int off) {  // the copies of plane zs + k
        const int zz = zs + k;
        unsigned long long* b = &S.bar[k & 1];
        fence_proxy_async();
        mbar_expect_tx(b, BYTES);
        tma_4d(&S.c[0][0][0] + off, &tm_rec, 2 * x0 - 8, 0, y0 - 2, zz, b);
        tma_3d(&S.rv[k & 1][0][0], &tm_r, x0 - XO, y0 - 2, zz, b);
        if (UPDATE) tma_3d(&S.qv[k & 1][0][0], &tm_q, x0 - XO, y0 - 2, zz, b);
        last_issued = k;
    };
    if (t == ISSUER) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        S.abort_ = 0;
        fence_barrier_init();
    }
    __syncthreads();
    if (t == ISSUER) issue(0, 0);

    // red task
    int r_row, r_q;
    const bool has_red = stage_task(t, RH, 0, &r_row, &r_q);
    const int r_o = r_row * RW + 2 * r_q;             // split offset of the quad's even half
    const int r_v = r_row * VW + 4 * r_q;  // its cells in a copied vector row
    const int r_qv = r_row * VW + 4 * r_q;
    const int r_gx = x0 - XO + 4 * r_q, r_gy = y0 - 2 + r_row;
    const int r_par = r_gy & 1;
    const int r_own = (has_red && r_row >= 2 && r_row < FTY + 2 && r_q >= 1 && r_q <= QX && r_gx < g.nx && r_gy < g.ny)
                          ? r_gx + g.nx * r_gy
                          : -1;
    // black task
    int b_row, b_q;
    const bool has_blk = stage_task(t, G::NBR, 1, &b_row, &b_q);
    const int b_o = b_row * RW + 2 * b_q;
    const int b_par = (y0 - 2 + b_row) & 1;
    // tile task: the own quad
    const bool has_own = t < G::NOWN;
    const int tx = t % QX, ty = t / QX;
    const int ox = x0 + 4 * tx, oy = y0 + ty;
    const bool own_inside = has_own && ox < g.nx && oy < g.ny;
    const int oo = (ty + 2) * RW + 2 * (tx + 1);
    const long long og = ox + (long long)g.nx * oy;

    const float4* c0 = &S.c[0][0][0];
    float* e0 = &S.er[0][0][0];
    float rr_thread = 0.f;
    float2 part = make_float2(0.f, 0.f);
    int rc_z = -1;
    auto flush_rc = [&]() {
        if (rc_z >= 0 && own_inside && !(ty & 1)) {
            const float2 a = S.ypart[ty][tx], b = S.ypart[ty + 1][tx];
            st2<float>(rc + (ox >> 1) + (long long)gc.nx * ((oy >> 1) + (long long)gc.ny * rc_z),
                     make_float2(0.25f * (a.x + b.x), 0.25f * (a.y + b.y)));
        }
        rc_z = -1;
    };
    // element offsets of the ring slots of planes zA, zA-1, zA-2, zA-3
    int o0 = 0, o1 = (NS - 1) * SL, o2 = (NS - 2) * SL, o3 = (NS - 3) * SL;
    auto step = [&](auto ph, int k) {
        constexpr int P = decltype(ph)::value;  // k & 3; zs is even, so plane zA has parity P & 1
        const int zA = zs + k;
        const bool aborted = *reinterpret_cast<volatile int*>(&S.abort_) != 0;
        if (t == ISSUER && k + 1 < nsteps && !aborted) issue(k + 1, o0 == (NS - 1) * SL ? 0 : o0 + SL);
        if (!aborted && !mbar_wait(&S.bar[P & 1], P >> 1)) {
            S.abort_ = 1;
            sc->stalled = 1;
            sc->converged = 1;
        }
        // ---- red stage: plane zA over the 2-halo rows
        if (has_red) {
            const float4* C = c0 + o0;
            float* ER = e0 + o0;
            float4 rn = cvt4r<float>(*reinterpret_cast<const float4*>(&S.rv[P & 1][0][0] + r_v));
            if (UPDATE) {
                const float4 qq = *reinterpret_cast<const float4*>(&S.qv[P & 1][0][0] + r_qv);
                rn = make_float4(fmaf(-alpha, qq.x, rn.x), fmaf(-alpha, qq.y, rn.y), fmaf(-alpha, qq.z, rn.z),
                                 fmaf(-alpha, qq.w, rn.w));
            }
            const int p = r_par ^ (P & 1);
            float4 d0, d1;
            rec2<0>(C + r_o + p * HW, &d0, &d1);
            const float2 rr = p ? make_float2(rn.y, rn.w) : make_float2(rn.x, rn.z);  // red cells
            const float2 rb = p ? make_float2(rn.x, rn.z) : make_float2(rn.y, rn.w);  // black cells
            const float2 ev = divide2(make_float2(sigma * rr.x, sigma * rr.y), make_float2(d0.w, d1.w));
            *reinterpret_cast<float2*>(ER + r_o + p * HW) = ev;
            *reinterpret_cast<float2*>(ER + r_o + (1 - p) * HW) = make_float2(sigma * rb.x, sigma * rb.y);
            if (UPDATE && r_own >= 0 && zA >= z0 && zA < z1) {
                *reinterpret_cast<float4*>(r_out + sxy * zA + r_own) = rn;
                rr_thread = fmaf(rn.x, rn.x, fmaf(rn.y, rn.y, fmaf(rn.z, rn.z, fmaf(rn.w, rn.w, rr_thread))));
            }
        }
        __syncthreads();
        flush_rc();
        // ---- black stage: plane zA-1 over the 1-halo rows, in place
        if (has_blk && zA - 1 >= z0 - 1) {
            const float4* C = c0 + o1;
            const float4* CN = c0 + o0;
            float* E = e0 + o1;
            const float* EM = e0 + o2;
            const float* EP = e0 + o0;
            const int h = b_par ^ (P & 1);  // black half of the row at plane zA-1
            const int o = b_o + h * HW;
            float2 d;
            const float2 s = gs_sum2<0>(C, CN, E, EM, EP, o, h, *reinterpret_cast<const float2*>(E + o), &d);
            *reinterpret_cast<float2*>(E + o) = divide2(s, d);
        }
        __syncthreads();
        // ---- correction out and restriction: plane zA-2 over the tile
        const int zC = zA - 2;
        if (has_own && zC >= z0 && zC < z1) {
            const float4* C = c0 + o2;
            const float4* CN = c0 + o1;
            const float* E = e0 + o2;
            const float* EM = e0 + o3;
            const float* EP = e0 + o1;
            const int p = (oy & 1) ^ (P & 1);  // red half of the own quad
            float2 d;
            const float2 s = gs_sum2<0>(C, CN, E, EM, EP, oo + p * HW, p, make_float2(0.f, 0.f), &d);
            part.x += s.x;
            part.y += s.y;
            if (own_inside) {
                const float2 ev = *reinterpret_cast<const float2*>(E + oo);
                const float2 od = *reinterpret_cast<const float2*>(E + oo + HW);
                st4<float>(e + (og + sxy * zC), make_float4(ev.x, od.x, ev.y, od.y));
            }
            if ((zC & 1) || zC + 1 == z1) {
                // the row pair sum is formed after the next step's first barrier
                S.ypart[ty][tx] = part;
                rc_z = zC >> 1;
                part = make_float2(0.f, 0.f);
            }
        }
    };
    auto advance = [&]() {
        o3 = o2;
        o2 = o1;
        o1 = o0;
        o0 = o0 == (NS - 1) * SL ? 0 : o0 + SL;
    };
    for (int k = 0;;) {
        step(Phase<0>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<1>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<2>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<3>{}, k);
        advance();
        if (++k >= nsteps) break;
    }
    __syncthreads();
    flush_rc();
    if (t == ISSUER && S.abort_) (void)mbar_wait(&S.bar[last_issued & 1], (last_issued >> 1) & 1);
    if (UPDATE) finish_residual_norm(rr_thread, sc, partials, nblocks, sh);
}

// ----------------------------------------------------- post-smoothing pass
// e and r arrive through tm_e and tm_r, the records through tm_rec, the coarse
// correction through tm_c (COPY) or by a load per quad, where coarse rows are
// no whole 16 bytes (x extents that 8 does not divide).  256^3: 141 us a pass with
// the copies, 152 with the loads.  Step structure as in k_pre_pair.
template <bool FINE, bool COPY>
__global__ void __launch_bounds__(PGeo::NT, 2)
    k_post_pair(const __grid_constant__ CUtensorMap tm_rec, const __grid_constant__ CUtensorMap tm_e,
               const __grid_constant__ CUtensorMap tm_r, const __grid_constant__ CUtensorMap tm_c, Grid3 g, Grid3 gc,
               const float* __restrict__ ec, float* __restrict__ out, const float* __restrict__ accum, float w, Scalars* sc, double* partials,
               int nblocks, long long n_active) {
    if (sc->converged) return;
    using G = PGeo;
    using SM = PairPostSm<COPY>;
    constexpr int FTY = G::FTY, NT = G::NT, RH = G::RH, NS = G::NS, SL = RH * RW;
    constexpr unsigned BYTES = RH * RW * sizeof(float4) + 2 * RH * VW * sizeof(float);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SM& S = aligned_smem<SM>(smem_raw);
    __shared__ double sh[NT / 32];
    const int t = threadIdx.x;
    constexpr int ISSUER = NT - 1;
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float is = FINE ? sc->inv_sigma : 1.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * FTY;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const int zs = z0 - 2, nsteps = z1 - z0 + 4;
    const long long sxy = (long long)g.nx * g.ny;
    int last_issued = 0;
    auto issue = [&](int k, int off) {  // the copies of plane zs + k
        const int zz = zs + k;
        unsigned long long* b = &S.bar[k & 1];
        fence_proxy_async();
        mbar_expect_tx(b, BYTES + (COPY && !(k & 1) ? CVH * CVW * (unsigned)sizeof(float) : 0u));
        tma_4d(&S.c[0][0][0] + off, &tm_rec, 2 * x0 - 8, 0, y0 - 2, zz, b);
        tma_3d(&S.ev[k & 1][0][0], &tm_e, x0 - XO, y0 - 2, zz, b);
        tma_3d(&S.rv[k & 1][0][0], &tm_r, x0 - XO, y0 - 2, zz, b);
        // zs is even: an even step starts a coarse plane
        if (COPY && !(k & 1)) tma_3d(&S.ec[(k >> 1) & 1][0], &tm_c, (x0 >> 1) - 8, (y0 >> 1) - 1, zz >> 1, b);
        last_issued = k;
    };
    if (t == ISSUER) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        S.abort_ = 0;
        fence_barrier_init();
    }
    __syncthreads();
    if (t == ISSUER) issue(0, 0);

    int r_row, r_q;
    const bool has_red = stage_task(t, RH, 0, &r_row, &r_q);
    const int r_o = r_row * RW + 2 * r_q;
    const int r_v = r_row * VW + 4 * r_q;
    const int r_gx = x0 - XO + 4 * r_q, r_gy = y0 - 2 + r_row;
    const int r_par = r_gy & 1;
    const bool r_inside = has_red && r_gx >= 0 && r_gx < g.nx && r_gy >= 0 && r_gy < g.ny;
    // the quad's two coarse parents: their place in the copied plane, or loaded two
    // steps before the pair of planes that shares them (168 us one step ahead and
    // on every plane)
    const int r_ce = (r_row >> 1) * CVW + 6 + 2 * r_q;
    const long long r_c = r_inside ? (r_gx >> 1) + (long long)gc.nx * (r_gy >> 1) : 0, csxy = (long long)gc.nx * gc.ny;
    float2 ccur = make_float2(0.f, 0.f), cnext = ccur;
    auto parents = [&](int zz) {  // of planes zz and zz + 1, zz even
        cnext = ldg_pair<float>(ec + r_c + csxy * (zz >> 1), r_inside && zz >= 0 && zz < g.nz);
    };
    if (!COPY) parents(zs);
    int b_row, b_q;
    const bool has_blk = stage_task(t, G::NBR, 1, &b_row, &b_q);
    const int b_o = b_row * RW + 2 * b_q;
    const int b_par = (y0 - 2 + b_row) & 1;
    const bool has_own = t < G::NOWN;
    const int tx = t % QX, ty = t / QX;
    const int ox = x0 + 4 * tx, oy = y0 + ty;
    const bool own_inside = has_own && ox < g.nx && oy < g.ny;
    const int oo = (ty + 2) * RW + 2 * (tx + 1);
    const int ov = (ty + 2) * VW + 4 * (tx + 1);
    const long long og = ox + (long long)g.nx * oy;
    const float4* c0 = &S.c[0][0][0];
    float* e0 = &S.ep[0][0][0];
    Acc acc;
    float4 rq_own[4];  // own quad's right-hand side of planes zA-3 .. zA (slot zA & 3)

    int o0 = 0, o1 = (NS - 1) * SL, o2 = (NS - 2) * SL, o3 = (NS - 3) * SL;
    auto step = [&](auto ph, int k) {
        constexpr int P = decltype(ph)::value;
        const int zA = zs + k;
        const bool aborted = *reinterpret_cast<volatile int*>(&S.abort_) != 0;
        if (t == ISSUER && k + 1 < nsteps && !aborted) issue(k + 1, o0 == (NS - 1) * SL ? 0 : o0 + SL);
        if (!aborted && !mbar_wait(&S.bar[P & 1], P >> 1)) {
            S.abort_ = 1;
            sc->stalled = 1;
            sc->converged = 1;
        }
        if (has_own) rq_own[P] = *reinterpret_cast<const float4*>(&S.rv[P & 1][0][0] + ov);
        // ---- prolongation: plane zA over the 2-halo rows
        if (has_red) {
            float* EP = e0 + o0;
            float4 ev = make_float4(0.f, 0.f, 0.f, 0.f), rq = ev;
            float2 cv = make_float2(0.f, 0.f);
            if (!COPY && !(P & 1)) {
                ccur = cnext;
                parents(zA + 2);
            }
            if (r_inside && zA >= 0 && zA < g.nz) {
                cv = COPY ? *reinterpret_cast<const float2*>(&S.ec[P >> 1][0] + r_ce) : ccur;
                ev = cvt4r<float>(*reinterpret_cast<const float4*>(&S.ev[P & 1][0][0] + r_v));
                rq = cvt4r<float>(*reinterpret_cast<const float4*>(&S.rv[P & 1][0][0] + r_v));
            }
            const int p = r_par ^ (P & 1);
            const float2 er = p ? make_float2(ev.y, ev.w) : make_float2(ev.x, ev.z);
            const float2 rb = p ? make_float2(rq.x, rq.z) : make_float2(rq.y, rq.w);
            *reinterpret_cast<float2*>(EP + r_o + p * HW) = make_float2(fmaf(w, cv.x, er.x), fmaf(w, cv.y, er.y));
            *reinterpret_cast<float2*>(EP + r_o + (1 - p) * HW) = make_float2(sigma * rb.x, sigma * rb.y);
        }
        __syncthreads();
        // ---- black half-step: plane zA-1 over the 1-halo rows, in place
        if (has_blk && zA - 1 >= z0 - 1) {
            const float4* C = c0 + o1;
            const float4* CN = c0 + o0;
            float* E = e0 + o1;
            const float* EM = e0 + o2;
            const float* EP = e0 + o0;
            const int h = b_par ^ (P & 1);
            const int o = b_o + h * HW;
            float2 d;
            const float2 s = gs_sum2<0>(C, CN, E, EM, EP, o, h, *reinterpret_cast<const float2*>(E + o), &d);
            *reinterpret_cast<float2*>(E + o) = divide2(s, d);
        }
        __syncthreads();
        // ---- red half-step: plane zA-2 over the tile, out = z
        const int zC = zA - 2;
        if (has_own && zC >= z0 && zC < z1) {
            const float4* C = c0 + o2;
            const float4* CN = c0 + o1;
            const float* E = e0 + o2;
            const float* EM = e0 + o3;
            const float* EP = e0 + o1;
            const int p = (oy & 1) ^ (P & 1);
            const float4 rv = cvt4r<float>(rq_own[(P + 2) & 3]);
            const float2 rr = p ? make_float2(rv.y, rv.w) : make_float2(rv.x, rv.z);
            float2 d;
            const float2 s = gs_sum2<0>(C, CN, E, EM, EP, oo + p * HW, p, make_float2(sigma * rr.x, sigma * rr.y), &d);
            const float2 zr = divide2(s, d);
            const float2 zb = *reinterpret_cast<const float2*>(E + oo + (1 - p) * HW);
            float4 zv = p ? make_float4(zb.x, zr.x, zb.y, zr.y) : make_float4(zr.x, zb.x, zr.y, zb.y);
            if (own_inside) {
                if (accum) {  // out = accum + z (second W-cycle visit)
                    const float4 a = cvt4r<float>(*reinterpret_cast<const float4*>(accum + og + sxy * zC));
                    zv = make_float4(a.x + zv.x, a.y + zv.y, a.z + zv.z, a.w + zv.w);
                }
                st4<float>(out + og + sxy * zC, zv);
                if (FINE) {
                    acc.add_prod(rv.x, zv.x * is);
                    acc.add_prod(rv.y, zv.y * is);
                    acc.add_prod(rv.z, zv.z * is);
                    acc.add_prod(rv.w, zv.w * is);
                }
            }
        }
    };
    auto advance = [&]() {
        o3 = o2;
        o2 = o1;
        o1 = o0;
        o0 = o0 == (NS - 1) * SL ? 0 : o0 + SL;
    };
    for (int k = 0;;) {
        step(Phase<0>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<1>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<2>{}, k);
        advance();
        if (++k >= nsteps) break;
        step(Phase<3>{}, k);
        advance();
        if (++k >= nsteps) break;
    }
    __syncthreads();
    if (t == ISSUER && S.abort_) (void)mbar_wait(&S.bar[last_issued & 1], (last_issued >> 1) & 1);
    if (FINE) finish_rz(acc.total(), sc, partials, nblocks, n_active, sh);
}

namespace {
// ------------------------------------------------------------------ host
int p_sms = 0, p_occ[2][2] = {};  // [fine 0, coarse 1][pre, post]

// 3-D map of a level vector (x-fastest cells), box of width x rows x 1.
bool vec_map(CUtensorMap* m, const void* base, const Grid3& g, int rows, int width = VW) {
    const cuuint64_t dims[3] = {(cuuint64_t)g.nx, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
    const cuuint64_t strides[2] = {(cuuint64_t)g.nx * 4, (cuuint64_t)g.nx * g.ny * 4};
    const cuuint32_t box[3] = {(cuuint32_t)width, (cuuint32_t)rows, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                    const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// 4-D map of the split-row smoother records: (4 values x nx/2 records of a
// half row, even/odd half, y, z), box 144 values x 2 halves x rows x 1.
bool rec_map(CUtensorMap* m, const void* base, const Grid3& g, int rows) {
    const cuuint64_t half = (cuuint64_t)2 * g.nx;  // values per half row
    const cuuint64_t dims[4] = {half, 2, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
    const cuuint64_t strides[3] = {half * 4, 2 * half * 4, 2 * half * 4 * g.ny};
    const cuuint32_t box[4] = {(cuuint32_t)(2 * RW), 2, (cuuint32_t)rows, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                    const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

Launch pair_launch(const Grid3& g, int occ) {
    return run_launch(g, dim3(PGeo::NT, 1, 1), PGeo::FTY, (p_sms > 0 ? p_sms : 152) * (occ > 0 ? occ : 1), 4);
}

template <bool UPDATE, bool FINE>
void pre_pair(const Grid3& g, const Grid3& gc, const void* sm, const void* rin, const float* q, float* r_out, void* e,
              void* rc, Scalars* sc, double* partials, cudaStream_t s) {
    CUtensorMap tm_rec, tm_r, tm_q;  // the maps' shapes were tried at pair_level_init
    (void)rec_map(&tm_rec, sm, g, PGeo::RH);
    (void)vec_map(&tm_r, rin, g, PGeo::RH);
    (void)vec_map(&tm_q, UPDATE ? (const void*)q : rin, g, PGeo::RH);
    const Launch P = pair_launch(g, p_occ[FINE ? 0 : 1][0]);
    k_pre_pair<UPDATE, FINE><<<P.grid, P.block, sizeof(PairPreSm<UPDATE>) + 128, s>>>(
        tm_rec, tm_r, tm_q, P.g, gc, r_out, (float*)e, (float*)rc, sc, partials, P.nblocks);
}
template <bool FINE, bool COPY>
void post_pair(const CUtensorMap& tm_c, const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec,
               const void* r, void* out, const void* accum, float w, Scalars* sc, double* partials, long long n_active,
               cudaStream_t s) {
    CUtensorMap tm_rec, tm_e, tm_r;
    (void)rec_map(&tm_rec, sm, g, PGeo::RH);
    (void)vec_map(&tm_e, e, g, PGeo::RH);
    (void)vec_map(&tm_r, r, g, PGeo::RH);
    const Launch P = pair_launch(g, p_occ[FINE ? 0 : 1][1]);
    k_post_pair<FINE, COPY><<<P.grid, P.block, sizeof(PairPostSm<COPY>) + 128, s>>>(
        tm_rec, tm_e, tm_r, tm_c, P.g, gc, (const float*)ec, (float*)out, (const float*)accum, w, sc, partials,
        P.nblocks, n_active);
}
cudaError_t prep(const void* fn, size_t bytes, int* occ) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && occ) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, fn, PGeo::NT, bytes);
    return e;
}
}  // namespace

cudaError_t pair_prepare_attributes() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = prep((const void*)k_pre_pair<true, true>, sizeof(PairPreSm<true>) + 128, &p_occ[0][0]);
    if (e == cudaSuccess) e = prep((const void*)k_pre_pair<false, true>, sizeof(PairPreSm<false>) + 128, nullptr);
    if (e == cudaSuccess) e = prep((const void*)k_post_pair<true, true>, sizeof(PairPostSm<true>) + 128, &p_occ[0][1]);
    if (e == cudaSuccess) e = prep((const void*)k_post_pair<true, false>, sizeof(PairPostSm<false>) + 128, nullptr);
    if (e == cudaSuccess) e = prep((const void*)k_pre_pair<false, false>, sizeof(PairPreSm<false>) + 128, &p_occ[1][0]);
    if (e == cudaSuccess) e = prep((const void*)k_post_pair<false, true>, sizeof(PairPostSm<true>) + 128, &p_occ[1][1]);
    if (e == cudaSuccess) e = prep((const void*)k_post_pair<false, false>, sizeof(PairPostSm<false>) + 128, nullptr);
    return e;
}
// A level of FP32 records whose rows the copies can read: no periodic axis, nx
// a multiple of 4 (16-byte rows).
bool pair_level_init(const Grid3& g, const void* sm, const void* r) {
    CUtensorMap tm;
    return tma_level_ok(g) && rec_map(&tm, sm, g, PGeo::RH) && vec_map(&tm, r, g, PGeo::RH);
}
void pair_pre(bool fine, bool update, const Grid3& g, const Grid3& gc, const void* sm, const void* rin, const float* q,
              float* r_out, void* e, void* rc, Scalars* sc, double* partials, cudaStream_t s) {
    if (fine && update) pre_pair<true, true>(g, gc, sm, rin, q, r_out, e, rc, sc, partials, s);
    else if (fine) pre_pair<false, true>(g, gc, sm, rin, q, r_out, e, rc, sc, partials, s);
    else pre_pair<false, false>(g, gc, sm, rin, q, r_out, e, rc, sc, partials, s);
}
void pair_post(bool fine, const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec, const void* r,
               void* out, const void* accum, float w, Scalars* sc, double* partials, long long n_active, cudaStream_t s) {
    CUtensorMap tm_c = {};  // read where coarse rows are whole 16 bytes
    const bool copy = gc.nx % 4 == 0 && vec_map(&tm_c, ec, gc, CVH, CVW);
#define POST(FINE, COPY) post_pair<FINE, COPY>(tm_c, g, gc, sm, e, ec, r, out, accum, w, sc, partials, n_active, s)
    if (copy) fine ? POST(true, true) : POST(false, true);
    else fine ? POST(true, false) : POST(false, false);
#undef POST
}

}  // namespace mhdproj
