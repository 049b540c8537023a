// tma_fused.cu -- the multigrid smoothing passes of large levels with FP16 or
// BF16 records, on grids without periodic axes: one pass down (residual update,
// three half-steps from zero, restriction) and one pass up (prolongation, three
// half-steps, the CG dot product), the smoother records staged by the Tensor
// Memory Accelerator.
//
// Smoother.  A pass runs red, black, red half-steps of Gauss-Seidel, the
// black one over-relaxed by SOR_BLACK:
//   down, from zero:  e_r = r/d;  e_b = w (r + sum beta e_r)/d;
//                     e_r += (sum beta e_b)/d
//   up:               e_r = (r + sum beta e_b)/d;
//                     e_b += w ((r + sum beta e_r)/d - e_b);
//                     e_r = (r + sum beta e_b)/d
// The up pass is the down pass reversed, so the cycle is symmetric.  Against
// one red and one black half-step per pass the third one cuts the CG
// iterations (jet 256^3: 23 -> 15, column 512x256x256: 13 -> 7, at 1e-6 and smaller
// errors) while the HBM traffic of a pass stays the same.  After
// the down pass the residual is zero on red cells, so the restriction sums
// black residuals only; the up pass overwrites the red values first, so only
// the black half of the down pass's correction is kept in HBM (compact rows of
// nx/2 values).
//
// Work split.  A block marches a 64 x FTY (x, y) tile along z.  A thread owns
// one octet, eight consecutive cells of a row: the tile's octets and those of
// the halo that some stage needs, ring by ring.  In an octet the cells of one
// colour are the four cells of one x parity.  In step k a thread runs the
// first half-step on plane k, the second on plane k-1, the third on plane k-2
// and the output stage on plane k-3:
//  * z neighbours are the thread's own values of the planes before and after,
//    in registers;
//  * x and y neighbours were written to shared memory by the previous step
//    (two half-planes per stage, alternating), so a step has one barrier, and
//    its stores come last so that the loads of the later stages overlap the
//    arithmetic of the earlier ones;
//  * the four cells a stage works on sit at the same x parity h in all of a
//    step's planes, so the record half that a stage reads as its own holds
//    the z-high mobilities of the next stage: they pass on in registers;
//  * the steps of the two parities are straight-line code, one copy for the
//    warps with the tile's octets and one for the halo's.
// What bounds it: the latency of a step (about 2700 cycles down and 3100 up, the
// stages' shared memory loads and dependent sums, twelve warps per SM, issue
// slots busy 0.39 and 0.36 of the time) and the L2 traffic of the halo (1.5 reads
// per cell).  jet 256^3, FP16 records: 106 us down, 121 us up (403 and 333 MB of
// HBM traffic).  Passes of two half-steps on quads with every neighbour from
// shared memory took 101 and 98 us; three half-steps in that form would take
// half as long again.  16 tile rows and two blocks per SM: 142 and 154 us (halo
// 1.7, registers capped at 128); values of earlier planes from shared memory
// instead of registers: 152 and 192 us.
//
// Records in HBM: per grid row four half rows of `pitch` entries: (beta_x,
// beta_y) of the even-x cells, of the odd-x cells, (beta_z, diagonal) of the
// even-x cells, of the odd-x cells; an entry is two FP16/BF16 values.  Rows are
// padded to 16 bytes.  One cp.async.bulk.tensor box of 40 entries x 4 half
// rows x RH rows brings a plane (entries x0/2-4 .. x0/2+35: the first
// coordinate is 16-byte aligned); cells outside the grid arrive as zeros, the closed wall.
//
// Every wait on an mbarrier is bounded: when it runs out the block stops
// issuing copies, marks the solve as stalled and converged (the host reports
// a timeout), and finishes its loop without waiting again.  Periodic grids
// (a copy box cannot wrap around) take the passes of fused_kernels.cu.
#include <algorithm>
#include <cstdlib>

#include "kernels.h"
#include "fused_common.cuh"
#include "tma_common.cuh"

namespace mhdproj {

namespace {
using namespace staged;
using namespace fused;
using namespace tma;

constexpr int HH = 40;         // staged entries of a half row: x0/2-4 .. x0/2+35
constexpr int NO = 10;         // octets of a staged row: x0-8 .. x0+71
constexpr int QO = PX / 8;     // own octets of a row
constexpr int RS = 4 * HH;     // entries of a staged record row

struct OGeo {
    static constexpr int FTY = 32;                     // tile rows
    static constexpr int RH = FTY + 6;                 // staged rows y0-3 .. y0+FTY+2
    static constexpr int C0 = QO * FTY / 2;            // own octets of one row parity
    static constexpr int WP = C0 / 32 + 2;             // warps per row parity: own octets, then the halo's
    static constexpr int NT = 64 * WP;                 // threads; the last one only issues copies
    static constexpr int NS = 5;                       // record ring: planes k+1 .. k-3
    static_assert(C0 % 32 == 0, "own octets fill warps");
};
// Record entries: two values.
using Entry = unsigned;
// Four entries of a half row as loaded.
template <int CK> struct Rec4 { uint4 v; };
template <int CK>
__device__ __forceinline__ Rec4<CK> ld_rec(const Entry* p) {
    return Rec4<CK>{*reinterpret_cast<const uint4*>(p)};
}
template <int CK>
__device__ __forceinline__ float half_lo(unsigned u) {
    if constexpr (CK == 1) return __low2float(*reinterpret_cast<const __half2*>(&u));
    else return __uint_as_float(u << 16);
}
template <int CK>
__device__ __forceinline__ float half_hi(unsigned u) {
    if constexpr (CK == 1) return __high2float(*reinterpret_cast<const __half2*>(&u));
    else return __uint_as_float(u & 0xffff0000u);
}
// The first / second values of the four entries.
template <int CK>
__device__ __forceinline__ void rec_lo(const Rec4<CK>& r, float (&o)[4]) {
    o[0] = half_lo<CK>(r.v.x); o[1] = half_lo<CK>(r.v.y); o[2] = half_lo<CK>(r.v.z); o[3] = half_lo<CK>(r.v.w);
}
template <int CK>
__device__ __forceinline__ void rec_hi(const Rec4<CK>& r, float (&o)[4]) {
    o[0] = half_hi<CK>(r.v.x); o[1] = half_hi<CK>(r.v.y); o[2] = half_hi<CK>(r.v.z); o[3] = half_hi<CK>(r.v.w);
}

struct PassSm {
    using ET = Entry;
    using G = OGeo;
    alignas(128) ET c[G::NS][G::RH][RS];
    // the three stages' half-planes, each for the next step (slot: step & 1)
    alignas(16) float ex[3][2][G::RH][HH];
    float4 ypart[2][G::FTY / 2][QO];  // restriction sums of the odd rows (slot: rc_slot)
    unsigned long long bar[2];
    int abort_;
};

// A thread's octet: staged row, octet in the row, halo ring (0: own, 4: none).
// The rows of a warp have one parity, so the colour of a half row is the same
// for all its lanes, and the warps of the two parities alternate, so that the
// warps with own octets (the most stages) spread over the four schedulers.
// The rings follow the seven-point stencil: a ring's corners belong to the
// next one.  Record rows start at the same bank, so the halo's octets are
// dealt out over groups of eight lanes (the lanes that load together): the
// side octets of two rows, then octets of the rows beyond the tile.
__device__ __forceinline__ int octet_index(int t) { return (t >> 6) * 32 + (t & 31); }
template <class G>
struct Octet {
    int row, oc, ring;
    __device__ __forceinline__ explicit Octet(int t) {
        constexpr int RPG = G::FTY >= 16 ? G::FTY / 16 : 1;  // rows whose sides one group holds
        const int par = (t >> 5) & 1, u = octet_index(t);
        int ty = par;
        oc = 1;
        ring = 4;
        if (u < G::C0) {
            ty = 2 * (u / QO) + par;
            oc = 1 + u % QO;
            ring = 0;
        } else {
            const int e = u - G::C0, grp = e >> 3, j = e & 7;
            if (j < 2 * RPG) {
                const int rr = grp * RPG + (j >> 1);
                if (rr < G::FTY / 2) {
                    ty = 2 * rr + par;
                    oc = (j & 1) ? NO - 1 : 0;
                    ring = 1;
                }
            } else {
                // rows beyond the tile, eight octets each: -1 / FTY (ring 1), -2 / FTY+1
                // (ring 2), -3 / FTY+2 (ring 3); corners of the first (ring 2) and of
                // the second (ring 3)
                const int m = grp * (8 - 2 * RPG) + (j - 2 * RPG);
                int out = 0;
                if (m < 3 * QO) {
                    out = ring = 1 + m / QO;
                    oc = 1 + m % QO;
                } else if (m < 3 * QO + 4) {
                    const int c = m - 3 * QO;
                    out = 1 + (c >> 1);
                    ring = out + 1;
                    oc = (c & 1) ? NO - 1 : 0;
                }
                if (out) {
                    const bool low = ((out & 1) != 0) == (par != 0);
                    ty = low ? -out : G::FTY - 1 + out;
                }
            }
        }
        row = ty + 3;
    }
};

// 1/d for a positive diagonal, 0 for a cell without one.
__device__ __forceinline__ float rcp_or_zero(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return d > 1e-37f ? r : 0.0f;
}
__device__ __forceinline__ void put4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void copy4(float (&a)[4], const float (&b)[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) a[j] = b[j];
}

__device__ __forceinline__ void get4(float (&v)[4], const float* p) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
}
// beta_x of one entry.
template <int CK>
__device__ __forceinline__ float entry_lo(const Entry* p) {
    return half_lo<CK>(*p);
}
// Sums of beta times the other colour over the six neighbours of an octet's
// four cells of x parity H, added to acc; d: their diagonals; bz: in, the
// z-high mobilities (of plane + 1), out, their own z-low ones (the z-high
// ones of the stage one plane below).  C: the octet's first entry in its
// record plane; X: the other colour's half-plane at the octet; o, zm, zp: the
// octet's values of the other colour in this plane, the one below and the
// one above.  At the ends of a staged row the outermost cell takes a value of
// another row: nothing reads that cell.
template <int CK, int H>
__device__ __forceinline__ void gs_octet(const Entry* C, const float* X, const float (&o)[4],
                                         const float (&zm)[4], const float (&zp)[4], float (&bz)[4], float (&acc)[4],
                                         float (&d)[4]) {
    const Rec4<CK> A = ld_rec<CK>(C + H * HH), Q = ld_rec<CK>(C + (1 - H) * HH);
    const Rec4<CK> Y = ld_rec<CK>(C + RS + H * HH), B = ld_rec<CK>(C + (2 + H) * HH);
    float m[4], p[4];
    get4(m, X - HH);
    get4(p, X + HH);
    const float s = X[H ? 4 : -1];
    const float a4 = H ? entry_lo<CK>(C + 4) : 0.f;
    float bxl[4], byl[4], byh[4], t[4], bzl[4];
    rec_lo<CK>(A, bxl);
    rec_hi<CK>(A, byl);
    rec_hi<CK>(Y, byh);
    rec_lo<CK>(B, bzl);
    rec_hi<CK>(B, d);
    rec_lo<CK>(Q, t);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float left = H ? o[j] : (j ? o[j - 1] : s), right = H ? (j < 3 ? o[j + 1] : s) : o[j];
        const float bxh = H ? (j < 3 ? t[j + 1] : a4) : t[j];
        float a = acc[j];
        a = fmaf(bxl[j], left, a);
        a = fmaf(bxh, right, a);
        a = fmaf(byl[j], m[j], a);
        a = fmaf(byh[j], p[j], a);
        a = fmaf(bzl[j], zm[j], a);
        a = fmaf(bz[j], zp[j], a);
        acc[j] = a;
        bz[j] = bzl[j];
    }
}
__device__ __forceinline__ void block_bar() { asm volatile("bar.sync 0;\n" ::: "memory"); }

// The plane ring of records: issue, wait and slot bookkeeping shared by the
// two passes.
struct RecordRing {
    using G = OGeo;
    using SM = PassSm;
    static constexpr int ISSUER = G::NT - 1;
    static constexpr unsigned BYTES = G::RH * RS * sizeof(Entry);
    SM& S;
    const CUtensorMap* tm;
    int x0, y0, zs, last = 0;
    static constexpr int SLOT = G::RH * RS;
    // ring offsets of planes k .. k-3 and of the next copy's slot
    int s0 = 0, s1 = (G::NS - 1) * SLOT, s2 = (G::NS - 2) * SLOT, s3 = (G::NS - 3) * SLOT, ahead = SLOT;
    __device__ __forceinline__ RecordRing(SM& S_, const CUtensorMap* tm_, int x0_, int y0_, int zs_)
        : S(S_), tm(tm_), x0(x0_), y0(y0_), zs(zs_) {
        if (threadIdx.x == ISSUER) {
            mbar_init(&S.bar[0], 1);
            mbar_init(&S.bar[1], 1);
            S.abort_ = 0;
            fence_barrier_init();
        }
        __syncthreads();
        if (threadIdx.x == ISSUER) issue(0, 0);
    }
    __device__ __forceinline__ void issue(int k, int off) {  // the copy of plane zs + k (ring offset off)
        unsigned long long* b = &S.bar[k & 1];
        fence_proxy_async();
        mbar_expect_tx(b, BYTES);
        tma_4d(&S.c[0][0][0] + off, tm, (x0 >> 1) - 4, 0, y0 - 3, zs + k, b);
        last = k;
    }
    // step k: rotate the slots, issue plane k+1 into the slot of plane k-4, wait
    // for plane k
    __device__ __forceinline__ void step(int k, int nsteps, Scalars* sc) {
        if (k) {
            const int t = s3;
            s3 = s2;
            s2 = s1;
            s1 = s0;
            s0 = ahead;
            ahead = t;
        }
        const bool aborted = *reinterpret_cast<volatile int*>(&S.abort_) != 0;
        if (threadIdx.x == ISSUER && k + 1 < nsteps && !aborted) issue(k + 1, ahead);
        if (!aborted && !mbar_wait(&S.bar[k & 1], (k >> 1) & 1)) {
            S.abort_ = 1;
            sc->stalled = 1;
            sc->converged = 1;
        }
    }
    // after a timed-out wait the copies in flight land before the block exits
    __device__ __forceinline__ void drain() {
        if (threadIdx.x == ISSUER && S.abort_)
            for (int j = max(0, last - 1); j <= last; j++) (void)mbar_wait(&S.bar[j & 1], (j >> 1) & 1);
    }
};

// Restriction sums of a run of planes z0 .. z1-1: in step k, whose output stage
// works on plane zC = z0 + k - 6, a coarse plane's sums are complete after its odd
// plane or the run's last one.  The odd rows' threads leave theirs in shared
// memory late in that step and the even rows' take them at the start of the next
// one.  With an odd number of planes the last two steps of a run each complete a
// coarse plane, so a step may leave one while it takes another: two slots, by the
// coarse plane's parity.
constexpr bool rc_complete(int k, int zC, int z1) { return k >= 6 && ((zC & 1) || zC + 1 == z1); }
__host__ __device__ constexpr int rc_slot(int zc) { return zc & 1; }
// No step of a run takes from the slot that it leaves sums in (one barrier
// separates two steps, none the ends of one).
constexpr bool rc_exchange_ordered() {
    for (int n = 1; n <= 9; n++) {  // planes of a run from z0 = 0
        int pending = -1;
        for (int k = 0; k < n + 6; k++) {
            const int taken = pending;
            pending = rc_complete(k, k - 6, n) ? rc_slot((k - 6) >> 1) : -1;
            if (pending >= 0 && pending == taken) return false;
        }
    }
    return true;
}
static_assert(rc_exchange_ordered(), "a slot of restriction sums is overwritten in the step that reads it");

// ---------------------------------------------------------------- down pass
// rin (VT) -> the black half of the correction (compact rows) and the coarse
// residual rc.  UPDATE (finest level inside CG): r_out = rin - alpha q is
// formed first, written for the tile's cells, and ||r_out||^2 decides
// convergence.  FINE: the right-hand side is sigma * r.
template <int CK, class VT, class VTc, bool UPDATE, bool FINE>
__global__ void __launch_bounds__(OGeo::NT, 1)
    k_pre_tma(const __grid_constant__ CUtensorMap tm_rec, Grid3 g, Grid3 gc, const VT* __restrict__ rin,
              const float* __restrict__ q, float* __restrict__ r_out, VT* __restrict__ ek, VTc* __restrict__ rc,
              Scalars* sc, double* partials, int nblocks) {
    if (sc->converged) return;
    using ET = Entry;
    using G = OGeo;
    using SM = PassSm;
    using R4 = typename Raw4<VT>::T;
    constexpr int NT = G::NT;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SM& S = aligned_smem<SM>(smem_raw);
    __shared__ double sh[NT / 32];
    const int t = threadIdx.x;
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float alpha = UPDATE ? sc->alpha_f : 0.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * G::FTY;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const int zs = z0 - 3, nsteps = z1 - z0 + 6;  // planes zs .. z1+2
    const Octet<G> T(t);
    const int gx = x0 - 8 + 8 * T.oc, gy = y0 - 3 + T.row;
    const bool in_y = T.ring < 4 && gy >= 0 && gy < g.ny;
    // of the side octets only the quad next to the tile is read
    const bool in_a = in_y && T.oc != 0 && gx < g.nx, in_b = in_y && T.oc != NO - 1 && gx + 4 >= 0 && gx + 4 < g.nx;
    const bool own_warp = octet_index(t) < G::C0;
    const int sxy = g.nx * g.ny, go = gx + g.nx * gy;
    // rows 0 and RH-1 run no stage that reads their outer rows; lanes off a
    // stage read in range and are not stored
    const int rs = min(max(T.row, 1), G::RH - 2);
    const ET* const c_own = &S.c[0][rs][4 * T.oc];
    const ET* const c_r0 = &S.c[0][T.row][4 * T.oc];
    float* const x_own = &S.ex[0][0][rs][4 * T.oc];
    float* const x_put = &S.ex[0][0][T.row][4 * T.oc];
    constexpr int XP = G::RH * HH, ST = 2 * XP;  // one half-plane, one stage
    R4 rv[2];
    float4 qv[2];
    auto load = [&](int zz) {  // the octet's residual (and q) of plane zz
        const bool okz = zz >= 0 && zz < g.nz;  // (planes beyond the last one are loaded and not used)
        const long long o = (long long)sxy * zz + go;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const bool ok = okz && (u ? in_b : in_a);
            rv[u] = ldg_quad<VT>(rin + o + 4 * u, ok);
            if (UPDATE) qv[u] = ldg_quad<float>(q + o + 4 * u, ok);
        }
    };
    load(zs);
    RecordRing ring(S, &tm_rec, x0, y0, zs);
    float rr_thread = 0.f;
    // restriction sums of the coarse planes of planes k-3 and k-1; the finished
    // ones of the even rows until the odd rows' arrive
    float pa[4] = {}, pb[4] = {}, ph[4] = {};
    int rc_z = -1;  // coarse plane of ph
    auto flush_rc = [&]() {
        if (rc_z >= 0 && own_warp && !(gy & 1)) {
            const float4 o = S.ypart[rc_slot(rc_z)][(T.row - 3) >> 1][T.oc - 1];
            VTc* cp = rc + ((gx >> 1) + (long long)gc.nx * ((gy >> 1) + (long long)gc.ny * rc_z));
            if (in_a) st2<VTc>(cp, make_float2(0.25f * (ph[0] + o.x), 0.25f * (ph[1] + o.y)));
            if (in_b) st2<VTc>(cp + 2, make_float2(0.25f * (ph[2] + o.z), 0.25f * (ph[3] + o.w)));
        }
        rc_z = -1;
    };
    // the octet's values by step parity: first-stage reds (index H: plane k-2,
    // 1-H: k-1), blacks (H: k-2, 1-H: k-3), third-stage reds (H: k-4, 1-H: k-3);
    // black right-hand side of plane k-1
    float r_[2][4] = {}, b_[2][4] = {}, f_[2][4] = {}, g1[4] = {};
    auto step = [&](auto hc, auto role, int k) {
        constexpr int H = decltype(hc)::value;  // red half of plane k, black half of plane k-1, ...
        constexpr int ROLE = decltype(role)::value;
        const int zA = zs + k;
        const int cur = (k & 1) * XP, prv = XP - cur;
        ring.step(k, nsteps, sc);
        if (ROLE == 0) flush_rc();
        // ---- first red half-step, plane k
        float r0[4], g0[4], bz[4];
        {
            float4 ra = cvt4r<VT>(rv[0]), rb = cvt4r<VT>(rv[1]);
            if (UPDATE) {
                ra = make_float4(fmaf(-alpha, qv[0].x, ra.x), fmaf(-alpha, qv[0].y, ra.y), fmaf(-alpha, qv[0].z, ra.z),
                                 fmaf(-alpha, qv[0].w, ra.w));
                rb = make_float4(fmaf(-alpha, qv[1].x, rb.x), fmaf(-alpha, qv[1].y, rb.y), fmaf(-alpha, qv[1].z, rb.z),
                                 fmaf(-alpha, qv[1].w, rb.w));
                if (ROLE == 0 && zA >= z0 && zA < z1) {
                    float* rp = r_out + ((long long)sxy * zA + go);
                    if (in_a) *reinterpret_cast<float4*>(rp) = ra;
                    if (in_b) *reinterpret_cast<float4*>(rp + 4) = rb;
                    rr_thread = fmaf(ra.x, ra.x, fmaf(ra.y, ra.y, fmaf(ra.z, ra.z, fmaf(ra.w, ra.w, rr_thread))));
                    rr_thread = fmaf(rb.x, rb.x, fmaf(rb.y, rb.y, fmaf(rb.z, rb.z, fmaf(rb.w, rb.w, rr_thread))));
                }
            }
            load(zA + 1);
            const Rec4<CK> B = ld_rec<CK>(c_r0 + ring.s0 + (2 + H) * HH);
            float d[4];
            rec_lo<CK>(B, bz);
            rec_hi<CK>(B, d);
            const float re[4] = {ra.x, ra.z, rb.x, rb.z}, rd[4] = {ra.y, ra.w, rb.y, rb.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                r0[j] = (H ? rd[j] : re[j]) * (sigma * rcp_or_zero(d[j]));
                g0[j] = sigma * (H ? re[j] : rd[j]);
            }
        }
        // ---- black half-step, plane k-1
        float b1[4], f2[4], acc[4], d[4];
        copy4(acc, g1);
        gs_octet<CK, H>(c_own + ring.s1, x_own + prv, r_[1 - H], r_[H], r0, bz, acc, d);
#pragma unroll
        for (int j = 0; j < 4; j++) b1[j] = acc[j] * (SOR_BLACK * rcp_or_zero(d[j]));
        if (ROLE == 0 && k >= 4) {  // right-hand side minus d e of the black residual
#pragma unroll
            for (int j = 0; j < 4; j++) pb[j] += fmaf(-d[j], b1[j], g1[j]);
        }
        copy4(g1, g0);
        // ---- second red half-step, plane k-2
        if constexpr (ROLE <= 1) {
#pragma unroll
            for (int j = 0; j < 4; j++) acc[j] = 0.f;
            gs_octet<CK, H>(c_own + ring.s2, x_own + ST + prv, b_[H], b_[1 - H], b1, bz, acc, d);
#pragma unroll
            for (int j = 0; j < 4; j++) f2[j] = fmaf(acc[j], rcp_or_zero(d[j]), r_[H][j]);
            // ---- correction out, black residual and restriction, plane k-3
            if constexpr (ROLE == 0) {
                const int zC = zA - 3;
#pragma unroll
                for (int j = 0; j < 4; j++) acc[j] = 0.f;
                gs_octet<CK, H>(c_own + ring.s3, x_own + 2 * ST + prv, f_[1 - H], f_[H], f2, bz, acc, d);
                if (k >= 6) {
                    VT* ep = ek + ((long long)(sxy >> 1) * zC + ((g.nx >> 1) * gy + (gx >> 1)));
                    if (in_a) st2<VT>(ep, make_float2(b_[1 - H][0], b_[1 - H][1]));
                    if (in_b) st2<VT>(ep + 2, make_float2(b_[1 - H][2], b_[1 - H][3]));
#pragma unroll
                    for (int j = 0; j < 4; j++) pa[j] += acc[j];
                }
                const bool complete = rc_complete(k, zC, z1);
                if (complete) {
                    if (gy & 1) put4(&S.ypart[rc_slot(zC >> 1)][(T.row - 3) >> 1][T.oc - 1].x, pa);
                    copy4(ph, pa);
                    rc_z = zC >> 1;
                }
                if (complete || k == 5) {  // at k = 5 planes z0 and z0+1 become the first pair
                    copy4(pa, pb);
#pragma unroll
                    for (int j = 0; j < 4; j++) pb[j] = 0.f;
                }
                copy4(f_[H], f2);
            }
            copy4(b_[1 - H], b1);
            if (ROLE == 0 || T.ring <= 1) put4(x_put + 2 * ST + cur, f2);
        }
        if (ROLE == 0 || T.ring < 4) put4(x_put + cur, r0);
        if (ROLE == 0 || T.ring <= 2) put4(x_put + ST + cur, b1);
        copy4(r_[H], r0);
    };
    // Straight-line steps in pairs of the two parities; a role's warps run the
    // stages their octets take part in (0: all, 1: without the output stage,
    // 2: the first two).  The first steps of a run work on planes that are not
    // there yet: nothing valid reads their results.
    auto run = [&](auto role) {
        int k = 0;
        if ((gy + zs) & 1) {
            step(Phase<1>{}, role, 0);
            block_bar();
            k = 1;
        }
        for (;;) {
            step(Phase<0>{}, role, k);
            if (++k >= nsteps) break;
            block_bar();
            step(Phase<1>{}, role, k);
            if (++k >= nsteps) break;
            block_bar();
        }
    };
    if (own_warp) run(Phase<0>{});
    else run(Phase<1>{});
    __syncthreads();
    flush_rc();
    ring.drain();
    if (UPDATE) finish_residual_norm(rr_thread, sc, partials, nblocks, sh);
}

// ------------------------------------------------------------------ up pass
// The black correction ek of the down pass plus w P ec, three half-steps, out
// (VT).  DOT (finest level): r . out / sigma gives rz and beta; the next
// V-cycle's sigma is then taken from ||r||^2.
template <int CK, class VT, class VTc, bool DOT, bool FINE>
__global__ void __launch_bounds__(OGeo::NT, 1)
    k_post_tma(const __grid_constant__ CUtensorMap tm_rec, Grid3 g, Grid3 gc, const VT* __restrict__ ek,
               const VTc* __restrict__ ec, const VT* __restrict__ rin, VT* __restrict__ out,
               const VT* __restrict__ accum, float w, Scalars* sc, double* partials, int nblocks,
               long long n_active) {
    if (sc->converged) return;
    using ET = Entry;
    using G = OGeo;
    using SM = PassSm;
    using R4 = typename Raw4<VT>::T;
    using P2 = typename Raw2<VT>::T;
    using C2 = typename Raw2<VTc>::T;
    constexpr int NT = G::NT;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SM& S = aligned_smem<SM>(smem_raw);
    __shared__ double sh[NT / 32];
    const int t = threadIdx.x;
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float is = FINE ? sc->inv_sigma : 1.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * G::FTY;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const int zs = z0 - 3, nsteps = z1 - z0 + 6;
    const Octet<G> T(t);
    const int gx = x0 - 8 + 8 * T.oc, gy = y0 - 3 + T.row;
    const bool in_y = T.ring < 4 && gy >= 0 && gy < g.ny;
    // of the side octets only the quad next to the tile is read
    const bool in_a = in_y && T.oc != 0 && gx < g.nx, in_b = in_y && T.oc != NO - 1 && gx + 4 >= 0 && gx + 4 < g.nx;
    const bool own_warp = octet_index(t) < G::C0;
    const int sxy = g.nx * g.ny, go = gx + g.nx * gy;
    const int ko = (gx >> 1) + (g.nx >> 1) * gy, co = (gx >> 1) + gc.nx * (gy >> 1), csxy = gc.nx * gc.ny;
    const int rs = min(max(T.row, 1), G::RH - 2);
    const ET* const c_own = &S.c[0][rs][4 * T.oc];
    float* const x_own = &S.ex[0][0][rs][4 * T.oc];
    float* const x_put = &S.ex[0][0][T.row][4 * T.oc];
    constexpr int XP = G::RH * HH, ST = 2 * XP;
    R4 rv[2];
    P2 kv[2];
    C2 cv[2];
    auto load = [&](int zz) {  // right-hand side, black correction and coarse parents of plane zz
        const bool okz = zz >= 0 && zz < g.nz;
        const VT* rp = rin + ((long long)sxy * zz + go);
        const VT* kp = ek + ((long long)(sxy >> 1) * zz + ko);
        const VTc* cp = ec + ((long long)csxy * (zz >> 1) + co);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const bool ok = okz && (u ? in_b : in_a);
            rv[u] = ldg_quad<VT>(rp + 4 * u, ok);
            kv[u] = ldg_pair<VT>(kp + 2 * u, ok);
            cv[u] = ldg_pair<VTc>(cp + 2 * u, ok);
        }
    };
    load(zs);
    RecordRing ring(S, &tm_rec, x0, y0, zs);
    Acc acc_rz;
    // the octet's values by step parity: prolonged blacks (index 1-H: plane k-1,
    // H: k-2), first reds (H: k-2, 1-H: k-3), changes of the blacks (1-H: k-3,
    // H: k-4); right-hand sides: reds of plane k-1, blacks (1-H: k-1, H: k-2);
    // smoothed blacks of plane k-3
    float p_[2][4] = {}, r_[2][4] = {}, b_[2][4] = {}, gr1[4] = {}, gb_[2][4] = {}, zb[4] = {};
    auto step = [&](auto hc, auto role, int k) {
        constexpr int H = decltype(hc)::value;  // red half of plane k; the stages' cells sit at half 1 - H
        constexpr int ROLE = decltype(role)::value;
        const int zA = zs + k;
        const int cur = (k & 1) * XP, prv = XP - cur;
        ring.step(k, nsteps, sc);
        // the right-hand side of plane k-3, for r . z
        R4 rz[2];
        const long long oC = (long long)sxy * (zA - 3) + go;
        if (DOT && ROLE == 0) {
            rz[0] = ldg_quad<VT>(rin + oC, k >= 6 && in_a);
            rz[1] = ldg_quad<VT>(rin + oC + 4, k >= 6 && in_b);
        }
        // ---- prolongation onto the black cells, plane k
        float p0[4], gr0[4], gb0[4], bz[4];
        {
            const float4 ra = cvt4r<VT>(rv[0]), rb = cvt4r<VT>(rv[1]);
            const float2 ka = cvt2(kv[0]), kb = cvt2(kv[1]), ca = cvt2(cv[0]), cb = cvt2(cv[1]);
            load(zA + 1);
            p0[0] = fmaf(w, ca.x, ka.x);
            p0[1] = fmaf(w, ca.y, ka.y);
            p0[2] = fmaf(w, cb.x, kb.x);
            p0[3] = fmaf(w, cb.y, kb.y);
            const float re[4] = {ra.x, ra.z, rb.x, rb.z}, rd[4] = {ra.y, ra.w, rb.y, rb.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                gr0[j] = sigma * (H ? rd[j] : re[j]);
                gb0[j] = sigma * (H ? re[j] : rd[j]);
            }
        }
        // ---- first red half-step, plane k-1
        float r1[4], b2[4], acc[4], d[4];
        rec_lo<CK>(ld_rec<CK>(c_own + ring.s0 + (3 - H) * HH), bz);  // z-high mobilities: plane k, the same half
        copy4(acc, gr1);
        gs_octet<CK, 1 - H>(c_own + ring.s1, x_own + prv, p_[1 - H], p_[H], p0, bz, acc, d);
#pragma unroll
        for (int j = 0; j < 4; j++) r1[j] = acc[j] * rcp_or_zero(d[j]);
        copy4(gr1, gr0);
        if constexpr (ROLE <= 1) {
            // ---- black half-step, plane k-2: its change of the prolonged value
            float zn[4];
            copy4(acc, gb_[H]);
            gs_octet<CK, 1 - H>(c_own + ring.s2, x_own + ST + prv, r_[H], r_[1 - H], r1, bz, acc, d);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float ri = rcp_or_zero(d[j]);
                b2[j] = ri > 0.f ? SOR_BLACK * fmaf(acc[j], ri, -p_[H][j]) : -p_[H][j];
                zn[j] = p_[H][j] + b2[j];
            }
            if constexpr (ROLE == 0) {
                // ---- second red half-step, plane k-3, out = z: the red values move
                // by the sum over the black changes
#pragma unroll
                for (int j = 0; j < 4; j++) acc[j] = 0.f;
                gs_octet<CK, 1 - H>(c_own + ring.s3, x_own + 2 * ST + prv, b_[1 - H], b_[H], b2, bz, acc, d);
                if (k >= 6) {
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const float za = fmaf(acc[2 * u], rcp_or_zero(d[2 * u]), r_[1 - H][2 * u]);
                        const float zc = fmaf(acc[2 * u + 1], rcp_or_zero(d[2 * u + 1]), r_[1 - H][2 * u + 1]);
                        // red cells at half 1 - H, black cells at half H
                        float4 z4 = H ? make_float4(za, zb[2 * u], zc, zb[2 * u + 1])
                                      : make_float4(zb[2 * u], za, zb[2 * u + 1], zc);
                        if (!(u ? in_b : in_a)) continue;
                        if (!DOT && accum) {  // out = accum + z (second W-cycle visit)
                            const float4 a = cvt4r<VT>(*reinterpret_cast<const R4*>(accum + oC + 4 * u));
                            z4 = make_float4(a.x + z4.x, a.y + z4.y, a.z + z4.z, a.w + z4.w);
                        }
                        st4<VT>(out + oC + 4 * u, z4);
                        if (DOT) {
                            const float4 r4 = cvt4r<VT>(rz[u]);
                            acc_rz.add_prod(r4.x, z4.x * is);
                            acc_rz.add_prod(r4.y, z4.y * is);
                            acc_rz.add_prod(r4.z, z4.z * is);
                            acc_rz.add_prod(r4.w, z4.w * is);
                        }
                    }
                }
                copy4(zb, zn);
                copy4(b_[H], b2);
            }
            copy4(r_[1 - H], r1);
            copy4(gb_[H], gb0);
            if (ROLE == 0 || T.ring <= 1) put4(x_put + 2 * ST + cur, b2);
        }
        if (ROLE == 0 || T.ring < 4) put4(x_put + cur, p0);
        if (ROLE == 0 || T.ring <= 2) put4(x_put + ST + cur, r1);
        copy4(p_[H], p0);
    };
    // see k_pre_tma
    auto run = [&](auto role) {
        int k = 0;
        if ((gy + zs) & 1) {
            step(Phase<1>{}, role, 0);
            block_bar();
            k = 1;
        }
        for (;;) {
            step(Phase<0>{}, role, k);
            if (++k >= nsteps) break;
            block_bar();
            step(Phase<1>{}, role, k);
            if (++k >= nsteps) break;
            block_bar();
        }
    };
    if (own_warp) run(Phase<0>{});
    else run(Phase<1>{});
    __syncthreads();
    ring.drain();
    if (DOT) finish_rz(acc_rz.total(), sc, partials, nblocks, n_active, sh);
}

// ------------------------------------------------- records and residuals
// Entries of a half row: nx/2, rounded up to 16 bytes.
__host__ __device__ inline int rec_pitch(int nx) { return (nx / 2 + 3) / 4 * 4; }
template <int CK>
__device__ __forceinline__ float2 entry2(const Entry& e) {
    return make_float2(half_lo<CK>(e), half_hi<CK>(e));
}
// (beta_x, beta_y) and (beta_z, diagonal) per cell from the level's
// coefficient records (beta_x, beta_y, beta_z, reaction); the diagonal is the
// FP32 sum of the record-precision values, rounded up to the record
// precision (the operator stays diagonally dominant).  The betas are exact
// in the record precision already.
template <int CK>
__global__ void __launch_bounds__(TILE_THREADS) k_tma_records(Grid3 g, const void* __restrict__ coef_v,
                                                              void* __restrict__ sm_v) {
    using CT = typename CoefStore<CK>::T;
    using ET = Entry;
    const CT* coef = reinterpret_cast<const CT*>(coef_v);
    ET* sm = reinterpret_cast<ET*>(sm_v);
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= g.nx || y >= g.ny) return;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const int pitch = rec_pitch(g.nx), h = x & 1;
    for (int z = z0; z < z1; z++) {
        const long long i = x + sy * y + sz * z;
        const float4 c = unpack<CK>(coef[i]);
        const float bxh = x + 1 < g.nx ? unpack<CK>(coef[i + 1]).x : 0.f;
        const float byh = y + 1 < g.ny ? unpack<CK>(coef[i + sy]).y : 0.f;
        const float bzh = z + 1 < g.nz ? unpack<CK>(coef[i + sz]).z : 0.f;
        const float d = ((c.x + bxh) + (c.y + byh)) + ((c.z + bzh) + c.w);
        ET* row = sm + (((long long)z * g.ny + y) * 4 + h) * pitch + (x >> 1);
        const uint2 u = coef[i];
        unsigned short dh;
        if constexpr (CK == 1) {
            const __half v = __float2half_ru(d);
            dh = *reinterpret_cast<const unsigned short*>(&v);
        } else {
            const __nv_bfloat16 v = __float2bfloat16_ru(d);
            dh = *reinterpret_cast<const unsigned short*>(&v);
        }
        row[0] = u.x;
        row[2 * pitch] = (u.y & 0x0000ffffu) | ((unsigned)dh << 16);
    }
}
// r2 = r - A e with the records' betas and diagonal: the right-hand side of a
// W-cycle level's second visit.
template <int CK, class VT>
__global__ void __launch_bounds__(TILE_THREADS) k_tma_residual(Grid3 g, const void* __restrict__ sm_v,
                                                               const VT* __restrict__ r, const VT* __restrict__ e,
                                                               VT* __restrict__ r2, const Scalars* sc) {
    if (sc->converged) return;
    using ET = Entry;
    const ET* sm = reinterpret_cast<const ET*>(sm_v);
    const int x = blockIdx.x * TX + threadIdx.x, y = blockIdx.y * TY + threadIdx.y;
    if (x >= g.nx || y >= g.ny) return;
    const int z0 = blockIdx.z * g.zper, z1 = min(g.nz, z0 + g.zper);
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const int pitch = rec_pitch(g.nx), h = x & 1;
    const long long rsy = 4ll * pitch, rsz = rsy * g.ny;
    for (int z = z0; z < z1; z++) {
        const long long i = x + sy * y + sz * z;
        const ET* row = sm + rsz * z + rsy * y + (x >> 1);
        const float2 a = entry2<CK>(row[h * pitch]), b = entry2<CK>(row[(2 + h) * pitch]);
        const float bxh = x + 1 < g.nx ? entry2<CK>(row[(1 - h) * pitch + h]).x : 0.f;
        const float byh = y + 1 < g.ny ? entry2<CK>(row[rsy + h * pitch]).y : 0.f;
        const float bzh = z + 1 < g.nz ? entry2<CK>(row[rsz + (2 + h) * pitch]).x : 0.f;
        float nsum = 0.f;
        nsum = fmaf(a.x, x > 0 ? to_f(e[i - 1]) : 0.f, nsum);
        nsum = fmaf(bxh, x + 1 < g.nx ? to_f(e[i + 1]) : 0.f, nsum);
        nsum = fmaf(a.y, y > 0 ? to_f(e[i - sy]) : 0.f, nsum);
        nsum = fmaf(byh, y + 1 < g.ny ? to_f(e[i + sy]) : 0.f, nsum);
        nsum = fmaf(b.x, z > 0 ? to_f(e[i - sz]) : 0.f, nsum);
        nsum = fmaf(bzh, z + 1 < g.nz ? to_f(e[i + sz]) : 0.f, nsum);
        r2[i] = from_f<VT>(to_f(r[i]) - (b.y * to_f(e[i]) - nsum));
    }
}

// ------------------------------------------------------------------ host
bool g_tma_enabled = false;
int g_sms = 0;
int g_occ[3][2][2] = {};  // [records precision][coarse level][down / up]: resident blocks per SM

// 4-D map of the records: (entries of a half row, four half rows, y, z), box
// HH x 4 x rows x 1; entries beyond nx/2 are out of bounds (zero).
bool rec_map(CUtensorMap* m, const void* base, const Grid3& g, int rows) {
    const cuuint64_t es = 4;
    const cuuint64_t half = (cuuint64_t)rec_pitch(g.nx) * es;
    const cuuint64_t dims[4] = {(cuuint64_t)(g.nx / 2), 4, (cuuint64_t)g.ny, (cuuint64_t)g.nz};
    const cuuint64_t strides[3] = {half, 4 * half, 4 * half * g.ny};
    const cuuint32_t box[4] = {(cuuint32_t)HH, 4, (cuuint32_t)rows, 1};
    const cuuint32_t unit[4] = {1, 1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4,
                    const_cast<void*>(base), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

Launch tma_launch(const Grid3& g, int occ) {
    return run_launch(g, dim3(OGeo::NT, 1, 1), OGeo::FTY, (g_sms > 0 ? g_sms : 152) * (occ > 0 ? occ : 1), 6);
}

template <int CK, class VT, class VTc, bool UPDATE, bool FINE>
void pre_tma(const Grid3& g, const Grid3& gc, const void* sm, const void* rin, const float* q, float* r_out, void* e,
             void* rc, Scalars* sc, double* partials, cudaStream_t s) {
    CUtensorMap tm_rec;
    (void)rec_map(&tm_rec, sm, g, OGeo::RH);  // the same encode succeeded at tma_level_init
    const Launch P = tma_launch(g, g_occ[CK][FINE ? 0 : 1][0]);
    k_pre_tma<CK, VT, VTc, UPDATE, FINE><<<P.grid, P.block, sizeof(PassSm) + 128, s>>>(
        tm_rec, P.g, gc, (const VT*)rin, q, r_out, (VT*)e, (VTc*)rc, sc, partials, P.nblocks);
}
template <int CK, class VT, class VTc, bool DOT, bool FINE>
void post_tma(const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec, const void* r, void* out,
              const void* accum, float w, Scalars* sc, double* partials, long long n_active, cudaStream_t s) {
    CUtensorMap tm_rec;
    (void)rec_map(&tm_rec, sm, g, OGeo::RH);  // the same encode succeeded at tma_level_init
    const Launch P = tma_launch(g, g_occ[CK][FINE ? 0 : 1][1]);
    k_post_tma<CK, VT, VTc, DOT, FINE><<<P.grid, P.block, sizeof(PassSm) + 128, s>>>(
        tm_rec, P.g, gc, (const VT*)e, (const VTc*)ec, (const VT*)r, (VT*)out, (const VT*)accum, w, sc, partials,
        P.nblocks, n_active);
}

template <class F>
cudaError_t prep(F* fn, size_t bytes, int threads, int* occ) {
    cudaError_t e = cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && occ) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, (const void*)fn, threads, bytes);
    return e;
}
template <int CK, class VT, class VTc>
cudaError_t prep_level(bool fine) {
    using G = OGeo;
    cudaError_t e = cudaSuccess;
    const size_t bytes = sizeof(PassSm) + 128;
    if (fine) {
        if (e == cudaSuccess) e = prep(k_pre_tma<CK, VT, VTc, true, true>, bytes, G::NT, &g_occ[CK][0][0]);
        if (e == cudaSuccess) e = prep(k_pre_tma<CK, VT, VTc, false, true>, bytes, G::NT, nullptr);
        if (e == cudaSuccess) e = prep(k_post_tma<CK, VT, VTc, true, true>, bytes, G::NT, &g_occ[CK][0][1]);
    } else {
        if (e == cudaSuccess) e = prep(k_pre_tma<CK, VT, VTc, false, false>, bytes, G::NT, &g_occ[CK][1][0]);
        if (e == cudaSuccess) e = prep(k_post_tma<CK, VT, VTc, false, false>, bytes, G::NT, &g_occ[CK][1][1]);
    }
    return e;
}
}  // namespace

PFN_cuTensorMapEncodeTiled_v12000 tma::encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        (void)cudaGetLastError();
        return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
    }();
    return fn;
}

cudaError_t tma_prepare_attributes() {
    const char* ev = getenv("MHDPROJ_TMA");
    g_tma_enabled = !(ev && ev[0] == '0') && encoder() != nullptr;
    if (!g_tma_enabled) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = prep_level<1, float, __half>(true);
    if (e == cudaSuccess) e = prep_level<2, float, __nv_bfloat16>(true);
    if (e == cudaSuccess) e = prep_level<1, __half, __half>(false);
    if (e == cudaSuccess) e = prep_level<2, __nv_bfloat16, __nv_bfloat16>(false);
    return e;
}

bool tma_level_ok(const Grid3& g) { return g_tma_enabled && g.periodic == 0 && g.nx % 4 == 0; }
bool tma_level_init(const Grid3& g, const void* sm) {
    CUtensorMap tm;
    return tma_level_ok(g) && rec_map(&tm, sm, g, OGeo::RH);
}
size_t tma_record_bytes(const Grid3& g) { return (size_t)g.ny * g.nz * 4 * rec_pitch(g.nx) * sizeof(Entry); }
void tma_records(int ck, const Launch& L, const void* coef, void* sm, cudaStream_t s) {
    if (ck == 1) k_tma_records<1><<<L.grid, L.block, 0, s>>>(L.g, coef, sm);
    else k_tma_records<2><<<L.grid, L.block, 0, s>>>(L.g, coef, sm);
}
void tma_level_residual(int ck, const Launch& L, const void* sm, const void* r, const void* e, void* r2,
                        const Scalars* sc, cudaStream_t s) {
    if (ck == 1)
        k_tma_residual<1, __half><<<L.grid, L.block, 0, s>>>(L.g, sm, (const __half*)r, (const __half*)e, (__half*)r2, sc);
    else
        k_tma_residual<2, __nv_bfloat16><<<L.grid, L.block, 0, s>>>(L.g, sm, (const __nv_bfloat16*)r,
                                                                    (const __nv_bfloat16*)e, (__nv_bfloat16*)r2, sc);
}

#define MHDPROJ_TMA_PRE(CK, VT, VTc, UPD, FINE) \
    pre_tma<CK, VT, VTc, UPD, FINE>(g, gc, sm, rin, q, r_out, e, rc, sc, partials, s)
void tma_pre(int ck, bool fine, bool update, const Grid3& g, const Grid3& gc, const void* sm, const void* rin,
             const float* q, float* r_out, void* e, void* rc, Scalars* sc, double* partials, cudaStream_t s) {
    if (fine && update) {
        if (ck == 1) MHDPROJ_TMA_PRE(1, float, __half, true, true);
        else MHDPROJ_TMA_PRE(2, float, __nv_bfloat16, true, true);
    } else if (fine) {
        if (ck == 1) MHDPROJ_TMA_PRE(1, float, __half, false, true);
        else MHDPROJ_TMA_PRE(2, float, __nv_bfloat16, false, true);
    } else {
        if (ck == 1) MHDPROJ_TMA_PRE(1, __half, __half, false, false);
        else MHDPROJ_TMA_PRE(2, __nv_bfloat16, __nv_bfloat16, false, false);
    }
}
#undef MHDPROJ_TMA_PRE
#define MHDPROJ_TMA_POST(CK, VT, VTc, DOT, FINE) \
    post_tma<CK, VT, VTc, DOT, FINE>(g, gc, sm, e, ec, r, out, accum, w, sc, partials, n_active, s)
void tma_post(int ck, bool fine, const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec,
              const void* r, void* out, const void* accum, float w, Scalars* sc, double* partials, long long n_active,
              cudaStream_t s) {
    if (fine) {
        if (ck == 1) MHDPROJ_TMA_POST(1, float, __half, true, true);
        else MHDPROJ_TMA_POST(2, float, __nv_bfloat16, true, true);
    } else {
        if (ck == 1) MHDPROJ_TMA_POST(1, __half, __half, false, false);
        else MHDPROJ_TMA_POST(2, __nv_bfloat16, __nv_bfloat16, false, false);
    }
}
#undef MHDPROJ_TMA_POST

}  // namespace mhdproj
