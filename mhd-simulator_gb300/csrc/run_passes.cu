// run_passes.cu -- the smoothing passes of small levels: the passes of
// fused_kernels.cu (red, black, red half-steps), each stage over every plane
// of a block's run at once.
//
// On a level of up to about 64^3 cells a pass that marches along z is a chain
// of plane steps, each of four dependent stages, and that chain's latency sets
// its time, not bandwidth: 9 steps of 2 barriers for a run of two planes.
// Here a block takes a 64 x 8 (x, y) tile and a run of two planes, keeps the
// run and three halo planes on each side in shared memory, and goes through
// the stages once: first stage over eight planes, second over six, third over
// four, output over the run's two; four barriers in all.  Halo cells are
// recomputed, four times the work per cell of a long run, which an idle chip
// has room for.  Sixteen warps, two groups that take alternate planes.  All
// loads are issued when the block starts.  FP16 48x40x56: 10.3 and 11.5 us a
// pass on the finest level with the launch, 16 and 18 marching; the former
// passes of two half-steps took 10.5 and 11.8.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "fused_common.cuh"

namespace mhdproj {

namespace {
using namespace staged;
using namespace fused;

constexpr int WTY = 8;                 // tile rows
constexpr int WRH = WTY + 6;           // staged rows y0-3 .. y0+WTY+2
constexpr int WNP = 8;                 // planes: a run of two with its halo
constexpr int WGT = 256, WGROUPS = 2;  // threads of a group, groups
constexpr int WNT = WGT * WGROUPS;
constexpr int WSL = WRH * RW;          // cells of a staged plane
static_assert(WRH * NQ <= WGT, "one first-stage quad per thread and plane");

template <int CK>
struct RunSm {
    using CT = typename CoefStore<CK>::T;
    CT c[WNP][WRH][RW];
    float e[WNP][WRH][RW];
    float gb[WNP][WRH][HW];  // the black cells' right-hand side sigma r
    float2 zpart[2][WTY][QX];
};

// All planes' records, zero outside the grid.
template <int CK>
__device__ __forceinline__ void stage_records(RunSm<CK>& S, const typename CoefStore<CK>::T* sm, const Grid3& g, int x0,
                                              int y0, int zs) {
    using CT = typename CoefStore<CK>::T;
    constexpr int RPC = CK == 0 ? 1 : 2, PER = HW / RPC, NC = WRH * 2 * PER;  // 16-byte copies of a plane
    const long long sxy = (long long)g.nx * g.ny;
    for (int k = threadIdx.x; k < NC; k += WNT) {
        const int row = k / (2 * PER), rem = k - row * 2 * PER;
        const int h = rem / PER, ci = rem - h * PER;
        bool okx, oky;
        const int sx = axis_wrap(x0 - XO + 2 * RPC * ci, g.nx, g.periodic & 1, &okx);
        const int sy = axis_wrap(y0 - 3 + row, g.ny, g.periodic & 2, &oky);
        const bool okxy = okx && oky;
        const long long o = okxy ? (long long)g.nx * sy + h * (g.nx >> 1) + (sx >> 1) : 0;
        CT* dst = &S.c[0][0][0] + row * RW + h * HW + RPC * ci;
#pragma unroll
        for (int p = 0; p < WNP; p++) {
            bool okz;
            const int sz = axis_wrap(zs + p, g.nz, (g.periodic & 4) != 0, &okz);
            const bool ok = okxy && okz;
            cp_async16(dst + p * WSL, sm + (ok ? o + sxy * sz : 0), ok);
        }
    }
    cp_commit();
}
}  // namespace

// As k_presmooth_restrict (fused_kernels.cu).
template <int CK, class VT, class VTc, bool UPDATE, bool FINE>
__global__ void __launch_bounds__(WNT, CK == 0 ? 1 : 2)
    k_pre_run(Grid3 g, Grid3 gc, const void* __restrict__ sm_v, const VT* __restrict__ rin,
              const float* __restrict__ q, float* __restrict__ r_out, VT* __restrict__ e, VTc* __restrict__ rc,
              Scalars* sc, double* partials, int nblocks) {
    if (sc->converged) return;
    using CT = typename CoefStore<CK>::T;
    using R4 = typename Raw4<VT>::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& S = *reinterpret_cast<RunSm<CK>*>(smem_raw);
    __shared__ double sh[WNT / 32];
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float alpha = UPDATE ? sc->alpha_f : 0.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * WTY, z0 = blockIdx.z * 2, zs = z0 - 3;
    const int t = threadIdx.x % WGT, grp = threadIdx.x / WGT;
    const long long sxy = (long long)g.nx * g.ny;
    float rr_thread = 0.f;
    stage_records<CK>(S, reinterpret_cast<const CT*>(sm_v), g, x0, y0, zs);
    // ---- first red half-step: planes 0 .. 7 over the 3-halo rows
    {
        int row, qd;
        const bool has = stage_task(t, WRH, 0, &row, &qd);
        const int gx = x0 - XO + 4 * qd, gy = y0 - 3 + row;
        bool okx, oky;
        const int sx = axis_wrap(gx, g.nx, g.periodic & 1, &okx);
        const int sy = axis_wrap(gy, g.ny, g.periodic & 2, &oky);
        const bool okxy = has && okx && oky;
        const long long o2 = okxy ? sx + (long long)g.nx * sy : 0;
        R4 rv[WNP / WGROUPS];
        float4 qv[WNP / WGROUPS];
#pragma unroll
        for (int j = 0; j < WNP / WGROUPS; j++) {
            bool okz;
            const int sz = axis_wrap(zs + WGROUPS * j + grp, g.nz, (g.periodic & 4) != 0, &okz);
            const bool ok = okxy && okz;
            rv[j] = ldg_quad<VT>(rin + o2 + (ok ? sxy * sz : 0), ok);
            if (UPDATE) qv[j] = ok ? __ldg(reinterpret_cast<const float4*>(q + o2 + sxy * sz)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        cp_wait<0>();
        __syncthreads();
        if (has) {
            const int o = row * RW + 2 * qd;
            const bool tile = row >= 3 && row < WTY + 3 && qd >= 1 && qd <= QX && gx < g.nx && gy < g.ny;
#pragma unroll
            for (int j = 0; j < WNP / WGROUPS; j++) {
                const int k = WGROUPS * j + grp, z = zs + k;
                float4 rn = cvt4r<VT>(rv[j]);
                if (UPDATE)
                    rn = make_float4(fmaf(-alpha, qv[j].x, rn.x), fmaf(-alpha, qv[j].y, rn.y),
                                     fmaf(-alpha, qv[j].z, rn.z), fmaf(-alpha, qv[j].w, rn.w));
                const int p = red_half(gy, z);
                const CT* C = &S.c[k][0][0];
                float* E = &S.e[k][0][0];
                float4 d0, d1;
                rec2<CK>(C + o + p * HW, &d0, &d1);
                const float2 rr = p ? make_float2(rn.y, rn.w) : make_float2(rn.x, rn.z);
                const float2 rb = p ? make_float2(rn.x, rn.z) : make_float2(rn.y, rn.w);
                *reinterpret_cast<float2*>(E + o + p * HW) =
                    divide2(make_float2(sigma * rr.x, sigma * rr.y), make_float2(d0.w, d1.w));
                *reinterpret_cast<float2*>(&S.gb[k][row][2 * qd]) = make_float2(sigma * rb.x, sigma * rb.y);
                if (UPDATE && tile && k >= 3 && k < 5 && z < g.nz) {
                    *reinterpret_cast<float4*>(r_out + gx + (long long)g.nx * gy + sxy * z) = rn;
                    rr_thread = fmaf(rn.x, rn.x, fmaf(rn.y, rn.y, fmaf(rn.z, rn.z, fmaf(rn.w, rn.w, rr_thread))));
                }
            }
        }
    }
    __syncthreads();
    // ---- black half-step: planes 1 .. 6 over the 2-halo rows
    {
        int row, qd;
        if (stage_task(t, WRH - 2, 1, &row, &qd)) {
#pragma unroll
            for (int j = 0; j < 6 / WGROUPS; j++) {
                const int k = 1 + WGROUPS * j + grp;
                const int h = 1 - red_half(y0 - 3 + row, zs + k), o = row * RW + 2 * qd + h * HW;
                float* E = &S.e[k][0][0];
                float2 d;
                const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o, h,
                                             *reinterpret_cast<const float2*>(&S.gb[k][row][2 * qd]), &d);
                const float2 v = divide2(s, d);
                *reinterpret_cast<float2*>(E + o) = make_float2(SOR_BLACK * v.x, SOR_BLACK * v.y);
            }
        }
    }
    __syncthreads();
    // ---- second red half-step: planes 2 .. 5 over the 1-halo rows
    {
        int row, qd;
        if (stage_task(t, WRH - 4, 2, &row, &qd)) {
#pragma unroll
            for (int j = 0; j < 4 / WGROUPS; j++) {
                const int k = 2 + WGROUPS * j + grp;
                const int h = red_half(y0 - 3 + row, zs + k), o = row * RW + 2 * qd + h * HW;
                float* E = &S.e[k][0][0];
                float2 d;
                const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o, h,
                                             make_float2(0.f, 0.f), &d);
                const float2 dv = divide2(s, d), ev = *reinterpret_cast<const float2*>(E + o);
                *reinterpret_cast<float2*>(E + o) = make_float2(ev.x + dv.x, ev.y + dv.y);
            }
        }
    }
    __syncthreads();
    // ---- correction out and restriction: planes 3, 4 over the tile
    const int tx = t % QX, ty = t / QX;
    const int ox = x0 + 4 * tx, oy = y0 + ty;
    const bool inside = ty < WTY && ox < g.nx && oy < g.ny;
    if (ty < WTY) {
        const int k = 3 + grp, z = zs + k;
        const int h = 1 - red_half(oy, z), o = (ty + 3) * RW + 2 * (tx + 1) + h * HW;
        const float* E = &S.e[k][0][0];
        const float2 bv = *reinterpret_cast<const float2*>(E + o);
        float2 d;
        const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o, h,
                                     *reinterpret_cast<const float2*>(&S.gb[k][ty + 3][2 * (tx + 1)]), &d);
        S.zpart[grp][ty][tx] = z < g.nz ? make_float2(fmaf(-d.x, bv.x, s.x), fmaf(-d.y, bv.y, s.y)) : make_float2(0.f, 0.f);
        if (inside && z < g.nz) st2<VT>(e + ((ox + (long long)g.nx * oy + sxy * z) >> 1), bv);
    }
    __syncthreads();
    if (grp == 0 && inside && !(ty & 1)) {
        const float2 a = S.zpart[0][ty][tx], b = S.zpart[1][ty][tx], c = S.zpart[0][ty + 1][tx], f = S.zpart[1][ty + 1][tx];
        st2<VTc>(rc + (ox >> 1) + (long long)gc.nx * ((oy >> 1) + (long long)gc.ny * (z0 >> 1)),
                 make_float2(0.25f * ((a.x + b.x) + (c.x + f.x)), 0.25f * ((a.y + b.y) + (c.y + f.y))));
    }
    if (UPDATE) finish_residual_norm(rr_thread, sc, partials, nblocks, sh);
}

// As k_prolong_postsmooth (fused_kernels.cu).
template <int CK, class VT, class VTc, bool DOT, bool FINE>
__global__ void __launch_bounds__(WNT, CK == 0 ? 1 : 2)
    k_post_run(Grid3 g, Grid3 gc, const void* __restrict__ sm_v, const VT* __restrict__ e, const VTc* __restrict__ ec,
               const VT* __restrict__ r, VT* __restrict__ out, const VT* __restrict__ accum, float w, Scalars* sc,
               double* partials, int nblocks, long long n_active) {
    if (sc->converged) return;
    using CT = typename CoefStore<CK>::T;
    using R4 = typename Raw4<VT>::T;
    using V2 = typename Raw2<VT>::T;
    using C2 = typename Raw2<VTc>::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& S = *reinterpret_cast<RunSm<CK>*>(smem_raw);
    __shared__ double sh[WNT / 32];
    const float sigma = FINE ? sc->sigma : 1.0f;
    const float is = FINE ? sc->inv_sigma : 1.0f;
    const int x0 = blockIdx.x * PX, y0 = blockIdx.y * WTY, z0 = blockIdx.z * 2, zs = z0 - 3;
    const int t = threadIdx.x % WGT, grp = threadIdx.x / WGT;
    const long long sxy = (long long)g.nx * g.ny, csxy = (long long)gc.nx * gc.ny;
    const int tx = t % QX, ty = t / QX;
    const int ox = x0 + 4 * tx, oy = y0 + ty, oz = z0 + grp;  // the thread's quad of the output stage
    const bool inside = ty < WTY && ox < g.nx && oy < g.ny && oz < g.nz;
    const long long og = ox + (long long)g.nx * oy + sxy * oz;
    stage_records<CK>(S, reinterpret_cast<const CT*>(sm_v), g, x0, y0, zs);
    const R4 rov = ldg_quad<VT>(r + (inside ? og : 0), inside);
    // ---- prolongation: planes 0 .. 7 over the 3-halo rows
    {
        int row, qd;
        if (stage_task(t, WRH, 0, &row, &qd)) {
            const int gx = x0 - XO + 4 * qd, gy = y0 - 3 + row;
            bool okx, oky;
            const int sx = axis_wrap(gx, g.nx, g.periodic & 1, &okx);
            const int sy = axis_wrap(gy, g.ny, g.periodic & 2, &oky);
            const bool okxy = okx && oky;
            const long long o2 = okxy ? sx + (long long)g.nx * sy : 0;
            const long long c2 = okxy ? (sx >> 1) + (long long)gc.nx * (sy >> 1) : 0;
            R4 rv[WNP / WGROUPS];
            V2 ev[WNP / WGROUPS];
            C2 cv[WNP / WGROUPS];
#pragma unroll
            for (int j = 0; j < WNP / WGROUPS; j++) {
                bool okz;
                const int sz = axis_wrap(zs + WGROUPS * j + grp, g.nz, (g.periodic & 4) != 0, &okz);
                const bool ok = okxy && okz;
                const long long pl = ok ? sxy * sz : 0;
                rv[j] = ldg_quad<VT>(r + o2 + pl, ok);
                ev[j] = ldg_pair<VT>(e + ((o2 + pl) >> 1), ok);
                cv[j] = ldg_pair<VTc>(ec + c2 + (ok ? csxy * (sz >> 1) : 0), ok);
            }
            const int o = row * RW + 2 * qd;
#pragma unroll
            for (int j = 0; j < WNP / WGROUPS; j++) {
                const int k = WGROUPS * j + grp, p = red_half(gy, zs + k);
                float* E = &S.e[k][0][0];
                const float4 rq = cvt4r<VT>(rv[j]);
                const float2 b = cvt2(ev[j]), c = cvt2(cv[j]);
                const float2 rr = p ? make_float2(rq.y, rq.w) : make_float2(rq.x, rq.z);
                const float2 rb = p ? make_float2(rq.x, rq.z) : make_float2(rq.y, rq.w);
                *reinterpret_cast<float2*>(E + o + p * HW) = make_float2(sigma * rr.x, sigma * rr.y);
                *reinterpret_cast<float2*>(E + o + (1 - p) * HW) = make_float2(fmaf(w, c.x, b.x), fmaf(w, c.y, b.y));
                *reinterpret_cast<float2*>(&S.gb[k][row][2 * qd]) = make_float2(sigma * rb.x, sigma * rb.y);
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
    // ---- first red half-step: planes 1 .. 6 over the 2-halo rows, in place
    {
        int row, qd;
        if (stage_task(t, WRH - 2, 1, &row, &qd)) {
#pragma unroll
            for (int j = 0; j < 6 / WGROUPS; j++) {
                const int k = 1 + WGROUPS * j + grp;
                const int h = red_half(y0 - 3 + row, zs + k), o = row * RW + 2 * qd + h * HW;
                float* E = &S.e[k][0][0];
                float2 d;
                const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o, h,
                                             *reinterpret_cast<const float2*>(E + o), &d);
                *reinterpret_cast<float2*>(E + o) = divide2(s, d);
            }
        }
    }
    __syncthreads();
    // ---- black half-step: planes 2 .. 5 over the 1-halo rows
    {
        int row, qd;
        if (stage_task(t, WRH - 4, 2, &row, &qd)) {
#pragma unroll
            for (int j = 0; j < 4 / WGROUPS; j++) {
                const int k = 2 + WGROUPS * j + grp;
                const int h = 1 - red_half(y0 - 3 + row, zs + k), o = row * RW + 2 * qd + h * HW;
                float* E = &S.e[k][0][0];
                float2 d;
                const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o, h,
                                             *reinterpret_cast<const float2*>(&S.gb[k][row][2 * qd]), &d);
                const float2 v = divide2(s, d), pv = *reinterpret_cast<const float2*>(E + o);
                *reinterpret_cast<float2*>(E + o) = make_float2(d.x > 0.f ? fmaf(SOR_BLACK, v.x - pv.x, pv.x) : 0.f,
                                                                d.y > 0.f ? fmaf(SOR_BLACK, v.y - pv.y, pv.y) : 0.f);
            }
        }
    }
    __syncthreads();
    // ---- second red half-step: planes 3, 4 over the tile, out = z
    Acc acc;
    if (inside) {
        const int k = 3 + grp, p = red_half(oy, oz), o = (ty + 3) * RW + 2 * (tx + 1);
        const float* E = &S.e[k][0][0];
        const float4 rv = cvt4r<VT>(rov);
        const float2 rr = p ? make_float2(rv.y, rv.w) : make_float2(rv.x, rv.z);
        float2 d;
        const float2 s = gs_sum2<CK>(&S.c[k][0][0], &S.c[k + 1][0][0], E, E - WSL, E + WSL, o + p * HW, p,
                                     make_float2(sigma * rr.x, sigma * rr.y), &d);
        const float2 zr = divide2(s, d);
        const float2 zb = *reinterpret_cast<const float2*>(E + o + (1 - p) * HW);
        float4 zv = p ? make_float4(zb.x, zr.x, zb.y, zr.y) : make_float4(zr.x, zb.x, zr.y, zb.y);
        if (accum) {  // out = accum + z (second W-cycle visit)
            const float4 a = cvt4r<VT>(*reinterpret_cast<const R4*>(accum + og));
            zv = make_float4(a.x + zv.x, a.y + zv.y, a.z + zv.z, a.w + zv.w);
        }
        st4<VT>(out + og, zv);
        if (DOT) {
            acc.add_prod(rv.x, zv.x * is);
            acc.add_prod(rv.y, zv.y * is);
            acc.add_prod(rv.z, zv.z * is);
            acc.add_prod(rv.w, zv.w * is);
        }
    }
    if (DOT) finish_rz(acc.total(), sc, partials, nblocks, n_active, sh);
}

// ------------------------------------------------------------------ host
namespace {
int r_sms = 0;
dim3 run_grid(const Grid3& g) {
    return dim3((g.nx + PX - 1) / PX, (g.ny + WTY - 1) / WTY, (g.nz + 1) / 2);
}
template <int CK, class VT, class VTc>
cudaError_t prep_run(bool fine) {
    const int bytes = (int)sizeof(RunSm<CK>);
    auto set = [&](const void* fn) { return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
    cudaError_t e = cudaSuccess;
    if (fine) {
        e = set((const void*)k_pre_run<CK, VT, VTc, true, true>);
        if (e == cudaSuccess) e = set((const void*)k_pre_run<CK, VT, VTc, false, true>);
        if (e == cudaSuccess) e = set((const void*)k_post_run<CK, VT, VTc, true, true>);
    } else {
        e = set((const void*)k_pre_run<CK, VT, VTc, false, false>);
        if (e == cudaSuccess) e = set((const void*)k_post_run<CK, VT, VTc, false, false>);
    }
    return e;
}
template <int CK, class VT, class VTc, bool UPDATE, bool FINE>
void pre_run(const Grid3& g, const Grid3& gc, const void* sm, const void* rin, const float* q, float* r_out, void* e,
             void* rc, Scalars* sc, double* partials, cudaStream_t s) {
    const dim3 grid = run_grid(g);
    k_pre_run<CK, VT, VTc, UPDATE, FINE><<<grid, WNT, sizeof(RunSm<CK>), s>>>(
        g, gc, sm, (const VT*)rin, q, r_out, (VT*)e, (VTc*)rc, sc, partials, (int)(grid.x * grid.y * grid.z));
}
template <int CK, class VT, class VTc, bool FINE>
void post_run(const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec, const void* r, void* out,
              const void* accum, float w, Scalars* sc, double* partials, long long n_active, cudaStream_t s) {
    const dim3 grid = run_grid(g);
    k_post_run<CK, VT, VTc, FINE, FINE><<<grid, WNT, sizeof(RunSm<CK>), s>>>(
        g, gc, sm, (const VT*)e, (const VTc*)ec, (const VT*)r, (VT*)out, (const VT*)accum, w, sc, partials,
        (int)(grid.x * grid.y * grid.z), n_active);
}
}  // namespace

cudaError_t run_prepare_attributes() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&r_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = prep_run<0, float, float>(true);
    if (e == cudaSuccess) e = prep_run<1, float, __half>(true);
    if (e == cudaSuccess) e = prep_run<2, float, __nv_bfloat16>(true);
    if (e == cudaSuccess) e = prep_run<0, float, float>(false);
    if (e == cudaSuccess) e = prep_run<1, __half, __half>(false);
    if (e == cudaSuccess) e = prep_run<2, __nv_bfloat16, __nv_bfloat16>(false);
    return e;
}

// One wave of resident blocks.  64^3 FP16 (256 blocks): 13.6 and 14.2 us a pass
// on the finest level, 15.8 and 17.4 marching (tma_fused.cu); a second wave
// loses (FP32 176x40x24, 180 blocks at one per SM: 21.1 and 21.3 us against
// 19.3 and 20.8).
bool run_level_ok(int ck, const Grid3& g) {
    const dim3 b = run_grid(g);
    const long long blocks = (long long)b.x * b.y * b.z, cap = (r_sms > 0 ? r_sms : 152) * (ck == 0 ? 1 : 2);
    return blocks <= MAX_REDUCE_BLOCKS && blocks <= cap;
}

void run_pre(int ck, bool fine, bool update, const Grid3& g, const Grid3& gc, const void* sm, const void* rin,
             const float* q, float* r_out, void* e, void* rc, Scalars* sc, double* partials, cudaStream_t s) {
#define PRE(CK, VT, VTc, UPD, FINE) pre_run<CK, VT, VTc, UPD, FINE>(g, gc, sm, rin, q, r_out, e, rc, sc, partials, s)
    if (fine && update) {
        if (ck == 1) PRE(1, float, __half, true, true);
        else if (ck == 2) PRE(2, float, __nv_bfloat16, true, true);
        else PRE(0, float, float, true, true);
    } else if (fine) {
        if (ck == 1) PRE(1, float, __half, false, true);
        else if (ck == 2) PRE(2, float, __nv_bfloat16, false, true);
        else PRE(0, float, float, false, true);
    } else {
        if (ck == 1) PRE(1, __half, __half, false, false);
        else if (ck == 2) PRE(2, __nv_bfloat16, __nv_bfloat16, false, false);
        else PRE(0, float, float, false, false);
    }
#undef PRE
}
void run_post(int ck, bool fine, const Grid3& g, const Grid3& gc, const void* sm, const void* e, const void* ec,
              const void* r, void* out, const void* accum, float w, Scalars* sc, double* partials, long long n_active,
              cudaStream_t s) {
#define POST(CK, VT, VTc, FINE) \
    post_run<CK, VT, VTc, FINE>(g, gc, sm, e, ec, r, out, accum, w, sc, partials, n_active, s)
    if (fine) {
        if (ck == 1) POST(1, float, __half, true);
        else if (ck == 2) POST(2, float, __nv_bfloat16, true);
        else POST(0, float, float, true);
    } else {
        if (ck == 1) POST(1, __half, __half, false);
        else if (ck == 2) POST(2, __nv_bfloat16, __nv_bfloat16, false);
        else POST(0, float, float, false);
    }
#undef POST
}

}  // namespace mhdproj
