// Kernels of the explicit Godunov step (FP64 state and arithmetic).
//
// One step = [viscous: grad1 cell pass, grad1 node pass] -> fused cell
// kernel -> node kernel.  The fused cell kernel does, per cell,
// calcOneStageMUSCLcpuFast (calcOneStageMUSCLcpuFast.jl:3-107) followed by
// updateVariablesSA (evaluate2d.jl:52-110) and writes its tile's reduction
// record; the first blocks of the node kernel fold a case's records and
// finalize its statistics and next time step (no device-wide barrier, no
// spin: a case of one tile group is folded by one block, in a larger one a
// counter elects the last warp).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "gd2d_internal.h"
#include "face_exact.cuh"
#include "physics.cuh"

// Register budget of the node-side passes, as resident 256-thread blocks per SM.
#ifndef GD2D_NODE_MINB
#define GD2D_NODE_MINB 4
#endif

namespace gd2d {

// Programmatic dependent launch (launch_dependent): every step kernel lets
// the next one be scheduled as soon as all its blocks run, and waits for
// the previous one before it reads or writes any state.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads and stores of data a step touches once (per-cell and per-face mesh
// arrays, the conservative state): marked evict-first, so that the caches
// keep the gathered node and neighbour data instead.
template <class T>
__device__ __forceinline__ T ld_once(const T *p) {
    return __ldcs(p);
}
__device__ __forceinline__ double4 ld_once(const double4 *p) {
    const double2 a = __ldcs(reinterpret_cast<const double2 *>(p)), b = __ldcs(reinterpret_cast<const double2 *>(p) + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st_once(double4 *p, const double4 &v) {
    __stcs(reinterpret_cast<double2 *>(p), make_double2(v.x, v.y));
    __stcs(reinterpret_cast<double2 *>(p) + 1, make_double2(v.z, v.w));
}

__device__ __forceinline__ int nbr_k(const int4 &v, int k) {
    return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

// ------------------------------------------------------- block reductions

struct Part {
    double res[4], tot[4], ek, vmax, rmin, rhomin, rhomax, bad;
    __device__ void init() {
        for (int v = 0; v < 4; ++v) { res[v] = 0.0; tot[v] = 0.0; }
        ek = 0.0; vmax = 0.0; rmin = INFINITY; rhomin = INFINITY; rhomax = -INFINITY; bad = 0.0;
    }
    __device__ void combine(const Part &o) {
        for (int v = 0; v < 4; ++v) { res[v] += o.res[v]; tot[v] += o.tot[v]; }
        ek += o.ek;
        vmax = fmax(vmax, o.vmax);
        rmin = fmin(rmin, o.rmin);
        rhomin = fmin(rhomin, o.rhomin);
        rhomax = fmax(rhomax, o.rhomax);
        bad = fmax(bad, o.bad);
    }
    __device__ void load_cg(const double *p) {
        for (int v = 0; v < 4; ++v) { res[v] = __ldcg(p + P_RES0 + v); tot[v] = __ldcg(p + P_TOT0 + v); }
        ek = __ldcg(p + P_EK); vmax = __ldcg(p + P_VMAX); rmin = __ldcg(p + P_RMIN);
        rhomin = __ldcg(p + P_RHOMIN); rhomax = __ldcg(p + P_RHOMAX); bad = __ldcg(p + P_BAD);
    }
};

// Fields of a Part in record order; 0-8 are sums, then max, min, min, max, max.
constexpr int kPartFields = 14;
__device__ __forceinline__ double part_op(int f, double a, double b) {
    if (f < 9) return a + b;
    return (f == 10 || f == 11) ? fmin(a, b) : fmax(a, b);
}

// Field f of a Part (record order).
__device__ __forceinline__ double part_get(const Part &p, int f) {
    switch (f) {
    case 0: case 1: case 2: case 3: return p.res[f];
    case 4: case 5: case 6: case 7: return p.tot[f - 4];
    case 8: return p.ek;
    case 9: return p.vmax;
    case 10: return p.rmin;
    case 11: return p.rhomin;
    case 12: return p.rhomax;
    default: return p.bad;
    }
}
__device__ __forceinline__ void part_set(Part &p, int f, double x) {
    switch (f) {
    case 0: case 1: case 2: case 3: p.res[f] = x; break;
    case 4: case 5: case 6: case 7: p.tot[f - 4] = x; break;
    case 8: p.ek = x; break;
    case 9: p.vmax = x; break;
    case 10: p.rmin = x; break;
    case 11: p.rhomin = x; break;
    case 12: p.rhomax = x; break;
    default: p.bad = x; break;
    }
}

// Records [b, e) (kPartials doubles apart) reduced by one warp in a fixed
// order: lane l folds records b + l, b + l + 32, ..., then a fixed shuffle
// tree per field.  The result is valid in lane 0.
__device__ __forceinline__ Part warp_reduce_records(const double *recs, int64_t b, int64_t e) {
    const int lane = threadIdx.x & 31;
    Part acc;
    acc.init();
    for (int64_t q = b + lane; q < e; q += 32) {
        Part o;
        o.load_cg(recs + q * kPartials);
        acc.combine(o);
    }
#pragma unroll
    for (int f = 0; f < kPartFields; ++f) {
        double x = part_get(acc, f);
        for (int off = 16; off > 0; off >>= 1) x = part_op(f, x, __shfl_down_sync(0xffffffffu, x, off));
        part_set(acc, f, x);
    }
    return acc;
}

// Per-case finalization, by one thread, from the case's reduction and its
// state `in` before the step: publish the step statistics and advance time (flowTime += dt, testInviscidFluxesGPUx32.jl:401)
// and the next dt: the fixed solControls.dt the reference steps with, or
// opt-in, the tau it reports (testInviscidFluxesGPUx32.jl:299,324) or the
// local-CFL extension.
static __device__ __forceinline__ void finalize_case(const DevMesh &m, const DevState &s, int c, const CaseState &in,
                                                     const Part &acc, bool is_init) {
    const DevCase &P = m.cases[c];
    CaseState out = in;
    const double vnew = acc.vmax, rnew = acc.rmin;
    if (!is_init) {
        DevStats st;
        st.dt = in.dt;
        st.flow_time = in.t;
        st.velmax = in.velmax;
        st.tau = P.CFL * P.maxEdge / jl_max(in.velmax, 1.0e-6);
        for (int v = 0; v < 4; ++v) { st.residual[v] = acc.res[v]; st.totals[v] = acc.tot[v]; }
        st.rho_min = acc.rhomin;
        st.rho_max = acc.rhomax;
        st.kinetic_energy = acc.ek;
        st.step = in.step + 1;
        st.nonfinite = acc.bad > 0.0 ? 1 : 0;
        st.reserved0 = 0;
        const int64_t row = (in.step % s.ring_len) * m.ncases + c;
        s.ring[row] = st;
        s.ring_host[row] = st;  // over PCIe: the host reads it after the stream's sync
        out.t = in.t + in.dt;
        out.step = in.step + 1;
        if (acc.bad > 0.0) out.nonfinite = 1;
    }
    double dtn;
    if (P.dt_mode == DT_REFERENCE_TAU) dtn = P.CFL * P.maxEdge / jl_max(vnew, 1.0e-6);
    else if (P.dt_mode == DT_LOCAL_CFL) dtn = P.CFL * rnew;
    else dtn = P.dt_fixed;
    out.dt = dtn;
    out.velmax = vnew;
    out.rmin = rnew;
    out.tiles_done = 0u;
    s.cstate[c] = out;
}

// Field f of tile q's reduction record.  Two layouts, measured per
// precision on the 2.09M-cell viscous cylinder: FIELD_MAJOR (one row of
// ntiles doubles per field), which makes the FP64 cell kernel 10 us faster
// than records of kPartials doubles and the mixed one 6 us slower, so the
// FP64 kernels use it and the mixed kernels do not.  The layout is a
// template parameter: strides read at run time cost the mixed cell kernel
// spills and 4 us.
template <bool FIELD_MAJOR>
__device__ __forceinline__ double *part_at(const DevMesh &m, const DevState &s, int64_t q, int f) {
    return FIELD_MAJOR ? s.part + (int64_t)f * m.ntiles + q : s.part + q * kPartials + f;
}

// Largest key of a warp: doubles mapped to unsigned 64-bit keys in their
// order, the high words' maximum first, then the low words' among its owners
// (two instructions of the warp's reduction unit in place of five levels of
// 64-bit shuffles and compares).  `sign` -1 maps the reverse order, for a
// minimum.  NaN takes the key 0, so that it is passed over as fmax and fmin
// do; a warp of nothing but NaN gives `none`.
template <int SIGN>
__device__ __forceinline__ double warp_extreme(double x, double none) {
    const int h = hi_word(x);
    const unsigned flip = (unsigned)(h >> 31) | 0x80000000u;  // all bits of a negative number, the sign of others
    unsigned kh = (unsigned)h ^ flip, kl = lo_word(x) ^ (unsigned)(h >> 31);
    if (SIGN < 0) { kh = ~kh; kl = ~kl; }
    if (x != x) kh = kl = 0u;
    const unsigned mh = __reduce_max_sync(0xffffffffu, kh);
    const unsigned ml = __reduce_max_sync(0xffffffffu, kh == mh ? kl : 0u);
    if (mh == 0u && ml == 0u) return none;
    unsigned rh = mh, rl = ml;
    if (SIGN < 0) { rh = ~rh; rl = ~rl; }
    const unsigned back = (rh >> 31) ? 0x80000000u : 0xffffffffu;
    return __hiloint2double((int)(rh ^ back), (int)(rl ^ ((rh >> 31) ? 0u : 0xffffffffu)));
}

// One warp's share of the tile's reduction record: its 32 cells' values
// folded in a fixed order into 14 doubles of shared memory.  The eight sums
// of four-component fields are halved between lane pairs at distances 16, 8
// and 4 (each lane passes on the half it does not keep) and folded over the
// last four lanes, so that eight full sums take nine exchanges instead of
// forty.
__device__ __forceinline__ void warp_record(const Part &p, double *out) {
    const int lane = threadIdx.x & 31;
    double v[8] = {p.res[0], p.res[1], p.res[2], p.res[3], p.tot[0], p.tot[1], p.tot[2], p.tot[3]};
#pragma unroll
    for (int half = 4, off = 16; half > 0; half >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    double x = v[0], ek = p.ek;
    x = x + __shfl_xor_sync(0xffffffffu, x, 2);
    x = x + __shfl_xor_sync(0xffffffffu, x, 1);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ek = ek + __shfl_xor_sync(0xffffffffu, ek, off);
    // lane 4 q of the warp holds the sum of field q (its three kept halves)
    const double vmax = warp_extreme<1>(p.vmax, 0.0), rmin = warp_extreme<-1>(p.rmin, INFINITY);
    const double rhomin = warp_extreme<-1>(p.rhomin, INFINITY), rhomax = warp_extreme<1>(p.rhomax, -INFINITY);
    const double bad = __any_sync(0xffffffffu, p.bad > 0.0) ? 1.0 : 0.0;
    if ((lane & 3) == 0) out[lane >> 2] = x;
    if (lane == 1) {
        out[P_EK] = ek; out[P_VMAX] = vmax; out[P_RMIN] = rmin;
        out[P_RHOMIN] = rhomin; out[P_RHOMAX] = rhomax; out[P_BAD] = bad;
    }
}
// The tile's record from its warps' shares (kPartials doubles each), field f
// by the caller's thread.
template <bool FIELD_MAJOR>
__device__ __forceinline__ void fold_warps(const DevMesh &m, const DevState &s, int64_t tile, int f,
                                           const double *shares, int nwarps) {
    double x = shares[f];
    for (int w = 1; w < nwarps; ++w) x = part_op(f, x, shares[w * kPartials + f]);
    *part_at<FIELD_MAJOR>(m, s, tile, f) = x;
}

// The tile's reduction record: every warp's share in shared memory (`shares`
// holds kPartials doubles a warp), folded by the first threads.  With
// ALIASED, `shares` overlays buffers the block used for the tile, so a
// barrier retires them first.  Nothing more happens at the tile's end: the
// next node pass folds the records (fold_block), so no tile waits for a
// fence or an atomic.  The last barrier retires `shares`.
template <bool FIELD_MAJOR, bool ALIASED>
__device__ __forceinline__ void tile_record(const DevMesh &m, const DevState &s, int64_t tile, const Part &p,
                                            double *shares) {
    if (ALIASED) __syncthreads();
    warp_record(p, shares + (threadIdx.x >> 5) * kPartials);
    __syncthreads();
    if (threadIdx.x < kPartFields) fold_warps<FIELD_MAJOR>(m, s, tile, threadIdx.x, shares, blockDim.x >> 5);
    __syncthreads();
}

// Identity of field f of a Part (record order), as Part::init sets it.
__device__ __forceinline__ double part_ident(int f) {
    if (f == 10 || f == 11) return INFINITY;
    return f == 12 ? -INFINITY : 0.0;
}

// Blocks of a node pass that fold one tile group: one warp per (group,
// field) pair, so a group takes kPartFields / warps-per-block blocks.
__host__ __device__ __forceinline__ int fold_blocks_per_group(int block) {
    const int nw = block / 32;
    return (kPartFields + nw - 1) / nw;
}

// The step's two-level reduction, done by the first blocks of the node pass
// that follows the cell kernel (the cell kernel's tile records are visible
// there: pdl_wait has returned).  A warp folds one field of one tile group
// (up to kGroupTiles tiles of one case): lane l takes records l, l + 32, ...,
// l + kGroupTiles - 32 of the group in turn, then a fixed shuffle tree over
// the lanes.  No thread waits on another's atomic and no order depends on
// which warp finishes last or on the node pass's block size, so the results
// are deterministic.
//
// What is known before the wait: the block's group and case.
struct FoldTask {
    int c, n;        // case; tiles of the group
    int64_t gid, t0; // group; its first tile
    int groups;      // groups of the case
};
__device__ __forceinline__ FoldTask fold_task(const DevMesh &m, int64_t g0) {
    FoldTask k;
    k.gid = g0 + blockIdx.x / fold_blocks_per_group(blockDim.x);
    k.c = m.group_case[k.gid];
    const DevCase &P = m.cases[k.c];
    k.t0 = P.tile_begin + (k.gid - P.group_begin) * kGroupTiles;
    k.n = (int)((k.t0 + kGroupTiles < P.tile_end) ? kGroupTiles : P.tile_end - k.t0);
    k.groups = (int)(P.group_end - P.group_begin);
    return k;
}
template <bool FIELD_MAJOR>
__device__ __forceinline__ double fold_group(const DevMesh &m, const DevState &s, const FoldTask &k, int f) {
    constexpr int kPerLane = kGroupTiles / 32;
    const int lane = threadIdx.x & 31;
    const double id = part_ident(f);
    double v[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j)
        v[j] = (lane + 32 * j < k.n) ? __ldcg(part_at<FIELD_MAJOR>(m, s, k.t0 + lane + 32 * j, f)) : id;
    double x = v[0];
#pragma unroll
    for (int j = 1; j < kPerLane; ++j) x = part_op(f, x, v[j]);
    for (int off = 16; off > 0; off >>= 1) x = part_op(f, x, __shfl_down_sync(0xffffffffu, x, off));
    return x;
}

// Block b < nred of a node pass.  A case of one group (up to 65,536 cells) is
// folded and finalized by one block of four or more warps through shared
// memory (two warps would take seven fields in turn).  Otherwise a warp
// takes one (group, field) pair, writes it to the group's record and counts
// it done for the case; the warp that completes the case's last pair reduces
// the case's group records and finalizes the case.  On a small mesh the fold
// is the step's critical path: eight dependent trips to memory through the
// records, fences and the counter made the step 2.4 us longer than without
// (7,900-cell Taylor-Green box 20.2 us a step, by one block 16.3).
template <bool FIELD_MAJOR>
__device__ __forceinline__ void fold_block(const DevMesh &m, const DevState &s, const FoldTask &k, bool is_init) {
    __shared__ double s_fold[kPartials];
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, part = blockIdx.x % fold_blocks_per_group(blockDim.x);
    const int lane = threadIdx.x & 31;
    if (k.groups == 1 && nw >= 4) {
        if (part != 0) return;
        CaseState in = {};
        if (threadIdx.x == 0) in = s.cstate[k.c];
        for (int f = warp; f < kPartFields; f += nw) {
            const double x = fold_group<FIELD_MAJOR>(m, s, k, f);
            if (lane == 0) s_fold[f] = x;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            Part acc;
            acc.init();
            Part o;
#pragma unroll
            for (int f = 0; f < kPartFields; ++f) part_set(o, f, s_fold[f]);
            acc.combine(o);
            finalize_case(m, s, k.c, in, acc, is_init);
        }
        return;
    }
    const int f = part * nw + warp;
    if (f >= kPartFields) return;
    const double x = fold_group<FIELD_MAJOR>(m, s, k, f);
    int last = 0;
    if (lane == 0) {
        s.gpart[k.gid * kPartials + f] = x;  // field f is record slot f
        __threadfence();
        const unsigned int need = (unsigned int)(k.groups * kPartFields);
        last = (atomicAdd(&s.cstate[k.c].tiles_done, 1u) == need - 1u) ? 1 : 0;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (last) {
        __threadfence();
        const int64_t g = m.cases[k.c].group_begin;
        const Part acc = warp_reduce_records(s.gpart, g, g + k.groups);
        if (lane == 0) finalize_case(m, s, k.c, s.cstate[k.c], acc, is_init);
    }
}

// --------------------------------------------------------- MUSCL + flux

// computeInterfaceSlope, computeslope2d.jl:3-136, for face k of cell g as it
// stands in physics.cuh, all operands read from memory: the faces whose
// operands face_flux_exact does not cover.  nbk: neighbour cell or
// -(bc slot+1).
template <int FLUX, bool QUAD>
__device__ __forceinline__ void face_flux_plain(const DevMesh &m, const DevCase &P, const double4 *__restrict__ pin,
                                                const double4 *__restrict__ nodeP, int64_t g, int k, int nbk, int dnk,
                                                int upk, int dn2k, int up2k, bool is_quad, const double *t,
                                                double *f) {
    const int64_t og = (int64_t)k * m.Nc + g;
    const double side = m.len[og], nx = m.nx[og], ny = m.ny[og];
    const double4 own = pin[g];
    const double uL[4] = {own.x, own.y, own.z, own.w};
    double hx_own = m.hx[g], hxR = hx_own;
    double uR[4], uUp[4], uDn[4];
    if (nbk >= 0) {
        if (QUAD && is_quad) {
            double4 a = nodeP[upk], a2 = nodeP[up2k], b = nodeP[dnk], b2 = nodeP[dn2k];
            uUp[0] = 0.5 * (a.x + a2.x); uUp[1] = 0.5 * (a.y + a2.y);
            uUp[2] = 0.5 * (a.z + a2.z); uUp[3] = 0.5 * (a.w + a2.w);
            uDn[0] = 0.5 * (b.x + b2.x); uDn[1] = 0.5 * (b.y + b2.y);
            uDn[2] = 0.5 * (b.z + b2.z); uDn[3] = 0.5 * (b.w + b2.w);
        } else {
            double4 a = nodeP[upk], b = nodeP[dnk];
            uUp[0] = a.x; uUp[1] = a.y; uUp[2] = a.z; uUp[3] = a.w;
            uDn[0] = b.x; uDn[1] = b.y; uDn[2] = b.z; uDn[3] = b.w;
        }
        const double4 r = pin[nbk];
        uR[0] = r.x; uR[1] = r.y; uR[2] = r.z; uR[3] = r.w;
        hxR = m.hx[nbk];
    } else {
        bc_ghost<double>(P, m, -nbk - 1, g, k, uL, nx, ny, *t, uR);
        for (int v = 0; v < 4; ++v) { uDn[v] = uL[v]; uUp[v] = uR[v]; }
    }
    double UpL[4], UpR[4];
    if (P.limiter == LIM_VENKAT) {
        // eps^2 = (K*HX)^3 times the face's (uL^2 + uR^2)/2 of each variable
        double KL = P.venkat_K * hx_own, KR = P.venkat_K * hxR;
        double e2L = KL * KL * KL, e2R = KR * KR * KR;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const double sc = 0.5 * (uL[v] * uL[v] + uR[v] * uR[v]);
            UpL[v] = uL[v] + 0.5 * lim_venkat(uL[v] - uDn[v], uR[v] - uL[v], e2L * sc);
            UpR[v] = uR[v] + 0.5 * lim_venkat(uR[v] - uUp[v], uL[v] - uR[v], e2R * sc);
        }
    } else {
        const int lk = P.limiter;
        const double ksi = P.ksi;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            UpL[v] = uL[v] + 0.5 * limiter(lk, uL[v] - uDn[v], uR[v] - uL[v], ksi);
            UpR[v] = uR[v] - 0.5 * limiter(lk, uR[v] - uL[v], uUp[v] - uR[v], ksi);
        }
    }
    face_flux_fn<FLUX, double>(UpR, UpL, nx, ny, side, P.gamma, P.face.g2, f);
}

// Half of a cell's (K HX)^3, the Venkatakrishnan limiter's scale.
__device__ __forceinline__ double venkat_half(const FaceCase &P, double hx) {
    const double K = P.venkat_K * hx;
    return 0.5 * (K * K * K);
}

// The same face from operands in registers: the cell's primitives uL, the
// neighbour's r, the up and down node values a and b (quads: averaged), the
// face geometry, and with the Venkatakrishnan limiter the two cells' eh =
// venkat_half.  Straight-line arithmetic (face_exact.cuh); the rare face with
// an operand out of its range is done over from memory by face_flux_plain
// (its pointer is made opaque to the compiler, which would otherwise hold
// every operand in registers across the fast path).
template <int FLUX, bool QUAD>
__device__ __forceinline__ void face_flux_at(const DevMesh &m, const DevCase &P, const FaceCase &K,
                                             const double4 *__restrict__ pin, const double4 *__restrict__ nodeP,
                                             int64_t g, int k, int nbk, int dnk, int upk, int dn2k, int up2k,
                                             bool is_quad, const double *uL, const double4 &r, const double4 &a,
                                             const double4 &b, double eh_own, double ehR, double side, double nx,
                                             double ny, const double *t, double *f) {
    double uR[4], uUp[4], uDn[4];
    if (nbk >= 0) {
        uUp[0] = a.x; uUp[1] = a.y; uUp[2] = a.z; uUp[3] = a.w;
        uDn[0] = b.x; uDn[1] = b.y; uDn[2] = b.z; uDn[3] = b.w;
        uR[0] = r.x; uR[1] = r.y; uR[2] = r.z; uR[3] = r.w;
    } else {
        bc_ghost<double>(P, m, -nbk - 1, g, k, uL, nx, ny, *t, uR);
        for (int v = 0; v < 4; ++v) { uDn[v] = uL[v]; uUp[v] = uR[v]; }
        ehR = eh_own;
    }
    if (__builtin_expect(!face_flux_exact<FLUX>(K, uL, uDn, uR, uUp, eh_own, ehR, nx, ny, side, f), 0)) {
        const double4 *pin2 = pin, *nodeP2 = nodeP;
        asm volatile("" : "+l"(pin2), "+l"(nodeP2));
        face_flux_plain<FLUX, QUAD>(m, P, pin2, nodeP2, g, k, nbk, dnk, upk, dn2k, up2k, is_quad, t, f);
    }
}

// Up and down node values of a face (quads: of its two nodes each, averaged).
template <bool QUAD>
__device__ __forceinline__ void face_nodes(const double4 *__restrict__ nodeP, int dnk, int upk, int dn2k, int up2k,
                                           bool is_quad, double4 &a, double4 &b) {
    a = nodeP[upk];
    b = nodeP[dnk];
    if (QUAD && is_quad) {
        const double4 a2 = nodeP[up2k], b2 = nodeP[dn2k];
        a = make_double4(0.5 * (a.x + a2.x), 0.5 * (a.y + a2.y), 0.5 * (a.z + a2.z), 0.5 * (a.w + a2.w));
        b = make_double4(0.5 * (b.x + b2.x), 0.5 * (b.y + b2.y), 0.5 * (b.z + b2.z), 0.5 * (b.w + b2.w));
    }
}

// Face k of cell g, fetching its operands from the per-cell arrays.
template <int FLUX, bool QUAD>
__device__ __forceinline__ void face_flux(const DevMesh &m, const DevCase &P, const double4 *__restrict__ pin,
                                          const double4 *__restrict__ nodeP, int64_t g, int k, int nbk,
                                          int dnk, int upk, int dn2k, int up2k, bool is_quad, const double *uL,
                                          double eh_own, const double *t, double *f) {
    const int64_t o = (int64_t)k * m.Nc + g;
    const double side = m.len[o], nx = m.nx[o], ny = m.ny[o];
    double4 r = make_double4(0.0, 0.0, 0.0, 0.0), a = r, b = r;
    double ehR = eh_own;
    if (nbk >= 0) {
        face_nodes<QUAD>(nodeP, dnk, upk, dn2k, up2k, is_quad, a, b);
        r = pin[nbk];
        if (P.limiter == LIM_VENKAT) ehR = venkat_half(P.face, m.hx[nbk]);
    }
    face_flux_at<FLUX, QUAD>(m, P, P.face, pin, nodeP, g, k, nbk, dnk, upk, dn2k, up2k, is_quad, uL, r, a, b, eh_own,
                             ehR, side, nx, ny, t, f);
}

// The fluxes of a cell's faces summed in face order
// (calcOneStageMUSCLcpuFast.jl:66-85).  A rolled loop: one face's quotients
// already overlap, and unrolled the face's code would not stay in the
// instruction cache.
template <int FLUX, bool QUAD>
__device__ __forceinline__ void cell_fluxes(const DevMesh &m, const DevCase &P, const double4 *__restrict__ pin,
                                            const double4 *__restrict__ nodeP, int64_t g, const int4 &nb, bool is_quad,
                                            const double *uL, double eh_own, const double *t, double *F) {
    const int4 dn = m.dn[g], up = m.up[g];
    int4 dn2 = make_int4(0, 0, 0, 0), up2 = make_int4(0, 0, 0, 0);
    if (QUAD && is_quad) { dn2 = m.dn2[g]; up2 = m.up2[g]; }
    const int nf = (QUAD && is_quad) ? 4 : 3;
#pragma unroll 1
    for (int k = 0; k < nf; ++k) {
        double f[4];
        face_flux<FLUX, QUAD>(m, P, pin, nodeP, g, k, nbr_k(nb, k), nbr_k(dn, k), nbr_k(up, k), nbr_k(dn2, k),
                              nbr_k(up2, k), is_quad, uL, eh_own, t, f);
#pragma unroll
        for (int v = 0; v < 4; ++v) F[v] = k == 0 ? f[v] : F[v] + f[v];
    }
}

// A cell's nodes in edge order, where the mesh has them.
__device__ __forceinline__ int4 cell_nodes(const DevMesh &m, int64_t g) {
    return m.cn ? ld_once(m.cn + g) : make_int4(0, 0, 0, 0);
}

// Artificial viscosity of a cell of density rho and size HX whose velocity
// divergence is divU (calcArtViscosity.jl:46-75); a: the sensor's threshold.
__device__ __forceinline__ double art_viscosity(double rho, double HX, double divU, double a) {
    if (-divU > a) {
        const double tmp = divU * divU - a * a;
        if (tmp > 0.0) return 0.5 * rho * HX / sqrt(2.0) * HX / sqrt(2.0) * sqrt(tmp) * 1.0e-5;
    }
    return 0.0;
}

// The transport model of diff_source with straight-line quotients
// (face_exact.cuh); false, and nothing written, where an operand is out of
// their range or the model is the reference's (whose air conductivity takes
// a power).
__device__ __forceinline__ bool diff_model_exact(const DevCase &P, const double4 &me, const double *sx,
                                                 const double *sy, double du, double dv, double area, double rarea,
                                                 bool art, double HX, double *diff) {
    if (P.visc_model == VISC_REFERENCE || !P.face.exact_rows) return false;
    Numerators n(sx[0]);
    n.add(sy[0]);
    Below<700> big(sx[0]);
    big.add(sy[0]);
    double lap[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        lap[v] = div_by(sx[v], area, rarea) + div_by(sy[v], area, rarea);
        if (v > 0) {
            n.add(sx[v]);
            n.add(sy[v]);
            big.add(sx[v]);
            big.add(sy[v]);
        }
    }
    InRange<-150, 200> r(me.w);
    Divisors<-150, 200> d(me.x);
    const double yrho = rcp_rn(me.x);
    double mu = P.mu_ref;
    if (P.visc_model == VISC_SUTHERLAND) {
        const double T = div_by(div_by(me.w, me.x, yrho), P.R, P.rR);
        const double w = 1.0 + div_rn(116.0, T);
        d.add(T);
        d.add(w);
        mu = P.mu_ref * div_by(div_rn(1.4792e-6 * sqrt_rn(T), w), P.suth_ref, P.rsuth);
    }
    double divU = 0.0, a = 0.0;
    if (art) {
        // (a divergence too small to be rounded right is far above -a)
        divU = div_by(du, area, rarea) + div_by(dv, area, rarea);
        big.add(du);
        big.add(dv);
        const double aS2 = div_by(P.gamma * me.w, me.x, yrho);
        r.add(aS2);
        const double root2 = sqrt(2.0);
        a = div_by(div_rn(0.05 * sqrt_rn(aS2), HX), root2, 1.0 / root2);
    }
    if (!n.ok() || !r.ok() || !d.ok() || !big.ok()) return false;
    const double mue = mu + (art ? art_viscosity(me.x, HX, divU, a) : 0.0);
    diff[1] = mue * lap[0];
    diff[2] = mue * lap[1];
    diff[3] = mue * lap[2];
    return true;
}

// Second Green-Gauss pass and transport model: the diffusion source of
// calcDiffTerm (calcDiffTerm.jl:88-113; gradients per calcGradients.jl:36-139,
// artificial viscosity per calcArtViscosity.jl:46-75).  cn: the cell's nodes
// in edge order (DevMesh::cn), loaded by the caller ahead of its use.
template <bool QUAD, class Geo>
__device__ __forceinline__ void diff_source(const DevMesh &m, const DevState &s, const DevCase &P, int64_t g,
                                            bool is_quad, const double4 &me, const int4 &cn, const Geo &geo,
                                            double area, double rarea, double HX, double *diff) {
    const int nf = (QUAD && is_quad) ? 4 : 3;
    double sx[3] = {0.0, 0.0, 0.0}, sy[3] = {0.0, 0.0, 0.0};
    double du = 0.0, dv = 0.0;
    const bool art = (P.visc_model != VISC_REFERENCE) && P.art_visc;
    // one edge's terms from its two nodes' gradients and velocities
    auto edge = [&](int k, const NodeGrad &A, const NodeGrad &B, const double2 &na, const double2 &nb) {
        double nx, ny, side;
        geo(k, nx, ny, side);
        double fx, fy;
        fx = 0.5 * (A.ru.x + B.ru.x) * -ny * side; fy = 0.5 * (A.ru.y + B.ru.y) * -nx * side;
        sx[0] = (k == 0) ? fx : sx[0] + fx; sy[0] = (k == 0) ? fy : sy[0] + fy;
        fx = 0.5 * (A.rv.x + B.rv.x) * -ny * side; fy = 0.5 * (A.rv.y + B.rv.y) * -nx * side;
        sx[1] = (k == 0) ? fx : sx[1] + fx; sy[1] = (k == 0) ? fy : sy[1] + fy;
        fx = 0.5 * (A.re.x + B.re.x) * -ny * side; fy = 0.5 * (A.re.y + B.re.y) * -nx * side;
        sx[2] = (k == 0) ? fx : sx[2] + fx; sy[2] = (k == 0) ? fy : sy[2] + fy;
        if (art) {
            const double fu = 0.5 * (na.x + nb.x) * -nx * side;
            const double fv = 0.5 * (na.y + nb.y) * -ny * side;
            du = (k == 0) ? fu : du + fu;
            dv = (k == 0) ? fv : dv + fv;
        }
    };
    auto velocity = [&](int n) {
        return art ? make_double2(s.nodeP[n].y, s.nodeP[n].z) : make_double2(0.0, 0.0);
    };
    if (m.cn) {
        // every node once: a cell's edges are a closed walk over its nodes
        const NodeGrad A = s.nodeG[cn.x], B = s.nodeG[cn.y], C = s.nodeG[cn.z];
        const double2 na = velocity(cn.x), nb = velocity(cn.y), nc = velocity(cn.z);
        edge(0, A, B, na, nb);
        edge(1, B, C, nb, nc);
        if (nf == 3) {
            edge(2, C, A, nc, na);
        } else {
            const NodeGrad D = s.nodeG[cn.w];
            const double2 nd = velocity(cn.w);
            edge(2, C, D, nc, nd);
            edge(3, D, A, nd, na);
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < nf; ++k) {
            const int2 e = ld_once(m.c2n + (int64_t)k * m.Nc + g);
            edge(k, s.nodeG[e.x], s.nodeG[e.y], velocity(e.x), velocity(e.y));
        }
    }
    diff[0] = 0.0;
    if (__builtin_expect(diff_model_exact(P, me, sx, sy, du, dv, area, rarea, art, HX, diff), 1)) return;
    double lap[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) lap[v] = sx[v] / area + sy[v] / area;
    const double T = me.w / me.x / P.R;
    if (P.visc_model == VISC_REFERENCE) {
        const double mu = P.mu_ref;
        diff[1] = mu * lap[0];
        diff[2] = mu * lap[1];
        diff[3] = mu * air_conductivity(T) * lap[2];
    } else {
        const double mu = (P.visc_model == VISC_SUTHERLAND) ? P.mu_ref * (sutherland(T) / P.suth_ref) : P.mu_ref;
        double mart = 0.0;
        if (art) {
            const double divU = du / area + dv / area;
            const double aS = sqrt(P.gamma * me.w / me.x);
            mart = art_viscosity(me.x, HX, divU, 0.05 * aS / HX / sqrt(2.0));
        }
        // laplacians of u, v and phi = |u|^2/2 + (gamma/Pr) e
        const double mue = mu + (P.art_visc ? mart : 0.0);
        diff[1] = mue * lap[0];
        diff[2] = mue * lap[1];
        diff[3] = mue * lap[2];
    }
}

// The same for cell g with everything read from the per-cell arrays.
template <bool QUAD>
__device__ __forceinline__ void diff_source_at(const DevMesh &m, const DevState &s, const DevCase &P, int64_t g,
                                               bool is_quad, const double4 &me, double *diff) {
    auto geo = [&](int k, double &nx, double &ny, double &side) {
        const int64_t o = (int64_t)k * m.Nc + g;
        side = m.len[o];
        nx = m.nx[o];
        ny = m.ny[o];
    };
    diff_source<QUAD>(m, s, P, g, is_quad, me, cell_nodes(m, g), geo, ld_once(m.area + g), ld_once(m.rarea + g),
                      ld_once(m.hx + g), diff);
}

// Euler update (calcOneStageMUSCLcpuFast.jl:94-99), the densityConstrained
// clamp (evaluate2d.jl:63-77), updateVariablesSA (evaluate2d.jl:87-104) and
// the cell's contribution to the step's reductions.
// The per-cell arrays the update reads, loaded by the caller (the tile
// kernel issues these loads before its flux barrier).
struct CellIn {
    double4 U;  // conservative state before the step
    double rarea, area, charlen;
};
__device__ __forceinline__ CellIn load_cell_in(const DevMesh &m, const DevState &s, int64_t g) {
    CellIn r;
    r.U = ld_once(s.U + g);
    r.rarea = ld_once(m.rarea + g);
    r.area = ld_once(m.area + g);
    r.charlen = ld_once(m.charlen + g);
    return r;
}

__device__ __forceinline__ void cell_update(const DevMesh &m, const DevState &s, const DevCase &P, int64_t g,
                                            const double4 &me, const double *F, const double *diff, double dt,
                                            const CellIn &in, double4 *__restrict__ pout, Part &part) {
    const double4 U = in.U;
    const double rarea = in.rarea;
    const double Uo[4] = {U.x, U.y, U.z, U.w};
    double Un[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) Un[v] = (Uo[v] - F[v] * P.beta * dt * rarea + P.beta * dt * diff[v]);
    if (P.density_constrained == 1) {
        if (Un[0] >= P.rho_max) Un[0] = P.rho_max;
        if (Un[0] <= P.rho_min) Un[0] = P.rho_min;
    }
    st_once(s.U + g, make_double4(Un[0], Un[1], Un[2], Un[3]));
    const double gam = P.gamma;
    const double rho = Un[0];
    CellPrims q;
    if (__builtin_expect(!(prims_exact(Un, gam, in.charlen, q) && P.face.exact_rows), 0)) {
        q.ux = Un[1] / Un[0];
        q.uy = Un[2] / Un[0];
        q.p = (gam - 1.0) * (Un[3] - 0.5 * (Un[1] * Un[1] + Un[2] * Un[2]) / Un[0]);
        const double a = sqrt(gam * q.p / rho);
        q.vmax = sqrt(q.ux * q.ux + q.uy * q.uy) + a;
        q.rmin = in.charlen / q.vmax;
    }
    const double ux = q.ux, uy = q.uy, p = q.p;
    pout[g] = make_double4(rho, ux, uy, p);
    const double area = in.area;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const double d = Un[v] - Uo[v];
        part.res[v] = d * d;
        part.tot[v] = Un[v] * area;
    }
    part.ek = 0.5 * rho * (ux * ux + uy * uy) * area;
    part.vmax = q.vmax;
    part.rmin = q.rmin;
    part.rhomin = me.x;
    part.rhomax = me.x;
    const bool ok = isfinite(Un[0]) && isfinite(Un[1]) && isfinite(Un[2]) && isfinite(Un[3]) && (rho > 0.0) &&
                    (p > 0.0);
    part.bad = ok ? 0.0 : 1.0;
}

// ---------------------------------------------------- fused cell kernel

template <int FLUX, bool VISC, bool QUAD, int MINB>
__global__ void __launch_bounds__(256, MINB) k_cell_step(const DevMesh m, const DevState s) {
    __shared__ double s_red[8 * kPartials];
    pdl_trigger();
    pdl_wait();
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    double4 *__restrict__ pout = s.prim + (int64_t)(par ^ 1) * m.Nc;
    const double4 *__restrict__ nodeP = s.nodeP;
    for (int64_t tile = blockIdx.x; tile < m.ntiles; tile += gridDim.x) {
        const int c = m.tile_case[tile];
        const DevCase &P = m.cases[c];
        const double dt = s.cstate[c].dt;
        const int64_t g = tile * blockDim.x + threadIdx.x;
        Part part;
        part.init();
        const int4 nb = m.nbr[g];
        if (nb.x != kAbsent) {
            const bool is_quad = QUAD && (nb.w != kAbsent);
            const double4 me = pin[g];
            const double uL[4] = {me.x, me.y, me.z, me.w};
            const double eh_own = (P.limiter == LIM_VENKAT) ? venkat_half(P.face, m.hx[g]) : 0.0;
            double F[4];
            cell_fluxes<FLUX, QUAD>(m, P, pin, nodeP, g, nb, is_quad, uL, eh_own, &s.cstate[c].t, F);
            double diff[4] = {0.0, 0.0, 0.0, 0.0};
            if (VISC) diff_source_at<QUAD>(m, s, P, g, is_quad, me, diff);
            cell_update(m, s, P, g, me, F, diff, dt, load_cell_in(m, s, g), pout, part);
        }
        tile_record<true, false>(m, s, tile, part, s_red);
    }
}

// The fused cell kernel over tile-local face lists (GD2D_LOOP_TILE_FACES).
// Phase 1 stages the tile's primitives (and the limiter's scale) in shared
// memory; phase 2 runs the tile's face list, one face per thread: a face
// between two cells of the tile is computed once, from its lower-indexed
// cell, and its flux stored negated into the other cell's slot -- exact
// because the listed pairs are only those whose face state and flux are
// antisymmetric bit for bit under exchange of the two cells (checked on the
// host: AUSM+ with the Minmod or Venkatakrishnan limiter or none, negated
// normals, exchanged down/up nodes); every other face slot is computed from
// its own cell as in k_cell_step.  Phase 3 sums each cell's slots in face
// order (calcOneStageMUSCLcpuFast.jl:66-85) and finishes the cell as
// k_cell_step.
//
// What bounds it (2.09M-cell viscous cylinder, 276 us; 365 before the
// divisions went into straight-line rows): issue and latency together.  Half
// the issue slots and 40% of the FP64 pipe are used; with all arithmetic
// taken out 184 us remain, with the face loop taken out 191, so a tile's
// gathers and its arithmetic overlap only across the three blocks of an SM.
template <int FLUX, bool VISC, bool QUAD, int MINB>
__global__ void __launch_bounds__(256, MINB) k_cell_step_tf(const DevMesh m, const DevState s) {
    constexpr int NS = QUAD ? 4 : 3;
    // the tile's primitives, then its flux slots, which the step reduction
    // reuses once they have been consumed
    __shared__ double4 s_mem[(1 + NS) * 256];
    __shared__ double s_eh[256];  // venkat_half of the tile's cells
    __shared__ FaceCase s_face;
    double4 *const s_prim = s_mem;
    double4 (*const s_flux)[256] = reinterpret_cast<double4 (*)[256]>(s_mem + 256);
    const int B = blockDim.x, tid = threadIdx.x;
    pdl_trigger();
    for (int64_t tile = blockIdx.x; tile < m.ntiles; tile += gridDim.x) {
        const int64_t base = tile * B;
        const int64_t g = base + tid;
        // the mesh does not depend on the kernel before this one: what a
        // tile reads of it first is asked for before the wait
        const int fb = (int)m.tf_off[tile] + tid, fe = (int)m.tf_off[tile + 1];
        int4 next = make_int4(0, 0, 0, 0), cn = next;
        if (fb < fe) next = ld_once(m.tf_rec + fb);
        if (VISC) cn = cell_nodes(m, g);
        const double eh = m.eh[g];
        const int c = m.tile_case[tile];
        const DevCase &P = m.cases[c];
        double faceconst = 0.0;
        if (tid < (int)(sizeof(FaceCase) / 8)) faceconst = reinterpret_cast<const double *>(&P.face)[tid];
        if (tile == blockIdx.x) pdl_wait();
        const int par = *s.parity;
        const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
        double4 *__restrict__ pout = s.prim + (int64_t)(par ^ 1) * m.Nc;
        s_prim[tid] = pin[g];
        s_eh[tid] = eh;
        if (tid < (int)(sizeof(FaceCase) / 8)) reinterpret_cast<double *>(&s_face)[tid] = faceconst;
        __syncthreads();
        for (int f = fb; f < fe; f += B) {
            const int4 rec = next;
            if (f + B < fe) next = ld_once(m.tf_rec + f + B);
            const TileFace tf = unpack_tile_face(rec.y);
            const double4 a4 = s_prim[tf.la];
            const double uL[4] = {a4.x, a4.y, a4.z, a4.w};
            const double eh_own = s_eh[tf.la];
            double4 r = make_double4(0.0, 0.0, 0.0, 0.0), up = r, down = r;
            double ehR = eh_own;
            int2 q2 = make_int2(0, 0);
            if (QUAD && tf.quad) q2 = m.tf_q[f];
            if (rec.x >= 0) {
                face_nodes<QUAD>(s.nodeP, rec.z, rec.w, q2.x, q2.y, QUAD && tf.quad, up, down);
                const unsigned lr = (unsigned)rec.x - (unsigned)base;  // (cell indices fit 31 bits)
                if (lr < (unsigned)B) {
                    r = s_prim[lr];
                    ehR = s_eh[lr];
                } else {
                    r = pin[rec.x];
                    ehR = m.eh[rec.x];
                }
            }
            // (32-bit plane offsets: 4 planes of the cells that fit the device's
            // memory stay under 2^32 elements)
            const unsigned og = (unsigned)tf.ka * (unsigned)m.Nc + (unsigned)base + (unsigned)tf.la;
            double fv[4];
            face_flux_at<FLUX, QUAD>(m, P, s_face, pin, s.nodeP, base + tf.la, tf.ka, rec.x, rec.z, rec.w, q2.x, q2.y,
                                     QUAD && tf.quad, uL, r, up, down, eh_own, ehR, m.len[og], m.nx[og], m.ny[og],
                                     &s.cstate[c].t, fv);
            s_flux[tf.ka][tf.la] = make_double4(fv[0], fv[1], fv[2], fv[3]);
            if (tf.lbp) s_flux[tf.kb][tf.lbp - 1] = make_double4(-fv[0], -fv[1], -fv[2], -fv[3]);
        }
        // the cell's viscous source needs no flux: evaluated before the
        // barrier, it fills the time a thread with fewer faces would wait
        const double4 me = s_prim[tid];
        const double dt = s.cstate[c].dt;
        // triangles: the viscous source is evaluated for padding cells too
        // (node 0 in their edge slots, zero area; the result is unused), and
        // a padding cell is told by its zero inverse area; quads read the
        // neighbour record, which also tells triangles from quads
        bool live = true, is_quad = false;
        if (QUAD) {
            const int4 nb = ld_once(m.nbr + g);
            live = nb.x != kAbsent;
            is_quad = nb.w != kAbsent;
        }
        double diff[4] = {0.0, 0.0, 0.0, 0.0};
        if (VISC && live) {
            auto geo = [&](int k, double &nx, double &ny, double &side) {
                const unsigned o = (unsigned)k * (unsigned)m.Nc + (unsigned)g;
                side = m.len[o];
                nx = m.nx[o];
                ny = m.ny[o];
            };
            diff_source<QUAD>(m, s, P, g, is_quad, me, cn, geo, m.area[g], m.rarea[g], ld_once(m.hx + g), diff);
        }
        // the update's own loads go out before the barrier (padded arrays:
        // in bounds for padding cells, whose values are not used)
        const CellIn cin = load_cell_in(m, s, g);
        if (!QUAD) live = cin.rarea != 0.0;
        __syncthreads();
        Part part;
        part.init();
        if (live) {
            const double4 a0 = s_flux[0][tid], a1 = s_flux[1][tid], a2 = s_flux[2][tid];
            double F[4] = {a0.x + a1.x, a0.y + a1.y, a0.z + a1.z, a0.w + a1.w};
            F[0] = F[0] + a2.x; F[1] = F[1] + a2.y; F[2] = F[2] + a2.z; F[3] = F[3] + a2.w;
            if (QUAD && is_quad) {
                const double4 a3 = s_flux[NS - 1][tid];
                F[0] = F[0] + a3.x; F[1] = F[1] + a3.y; F[2] = F[2] + a3.z; F[3] = F[3] + a3.w;
            }
            cell_update(m, s, P, g, me, F, diff, dt, cin, pout, part);
        }
        // (every thread has read the primitives: the reduction's shares go
        // there, clear of the flux slots still being read)
        tile_record<true, false>(m, s, tile, part, reinterpret_cast<double *>(s_prim));
    }
}

// ------------------------------------------------------------ node kernel

// cells2nodesSolutionReconstructionWithStencils (utilsFVM2dp.jl:299-365):
// weighted primitive averages; with VISC also calcPhiInCellCluster's
// unweighted means of rho u, rho v, E (calcGradients.jl:3-18) for the next
// step's viscous term.  The last block flips the step parity.  The first
// `nred` blocks instead fold the cell kernel's tile groups g0, g0 + 1, ...
// (fold_block): they start first and their latency hides behind the node
// gathers; nothing here reads what they write.
// The node-side kernels are bound by the latency of their gathers; their
// register budget is capped for 4 resident blocks per SM (more warps in
// flight; measured faster than the unconstrained 76-register build).
template <bool VISC, bool UNIT>
__global__ void __launch_bounds__(256, GD2D_NODE_MINB) k_node_avg(const DevMesh m, const DevState s, int flip, int zero_prims,
                                                  int64_t n0, int64_t n1, int64_t g0, int nred, int is_init) {
    pdl_trigger();
    if ((int)blockIdx.x < nred) {
        const FoldTask task = fold_task(m, g0);
        pdl_wait();
        fold_block<true>(m, s, task, is_init != 0);
        return;
    }
    pdl_wait();
    // FP64 node passes take their blocks from the last to the first: what the
    // cell pass before wrote last is still in L2 (with grad1_nodes: 2.09M-cell
    // viscous cylinder 406.5 -> 403.8 us a step, 523,000 cells 113.7 -> 112.9;
    // meshes that L2 holds, and the mixed passes with half the bytes, gain
    // nothing and the latter keep the ascending order)
    const int64_t bid = (int64_t)(gridDim.x - 1 - blockIdx.x), nblk = (int64_t)gridDim.x - nred;
    const int par = *s.parity;
    const double4 *__restrict__ src = s.prim + (int64_t)(flip ? (par ^ 1) : par) * m.Nc;
    const int W = m.cluster_w;
    for (int64_t J = n0 + bid * blockDim.x + threadIdx.x; J < n1; J += nblk * blockDim.x) {
        bool prim_form = false;
        double gop = 0.0, gm1 = 0.0;
        if (VISC) {
            const DevCase &P = m.cases[ld_once(m.node_case + J)];
            prim_form = P.visc_model != VISC_REFERENCE;
            gop = P.gamma_over_Pr;
            gm1 = P.face.gm1;
        }
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, det = 0.0;
        double c0 = 0.0, c1 = 0.0, c2 = 0.0;
        int cnt = 0;
        // phi = |u|^2/2 + (gamma/Pr) p / ((gamma-1) rho)
        auto phi_plain = [&](const double4 &p) {
            return 0.5 * (p.y * p.y + p.z * p.z) + gop * (p.w / (gm1 * p.x));
        };
        Divisors<-150, 200> dr(1.0);
        InRange<-150, 200> pr(1.0);
        auto add = [&](int c, const double4 &p, double w) {
            if (UNIT) {
                a0 = a0 + p.x; a1 = a1 + p.y; a2 = a2 + p.z; a3 = a3 + p.w;
            } else {
                a0 = a0 + p.x * w; a1 = a1 + p.y * w; a2 = a2 + p.z * w; a3 = a3 + p.w * w;
                det = det + w;
            }
            if (VISC) {
                if (prim_form) {
                    // (unit weights: the velocities' means are the primitives')
                    if (!UNIT) { c0 = c0 + p.y; c1 = c1 + p.z; }
                    const double d = gm1 * p.x;
                    dr.add(d);
                    pr.add(p.w);
                    c2 = c2 + (0.5 * (p.y * p.y + p.z * p.z) + gop * div_rn(p.w, d));
                } else {
                    const double4 u = s.U[c];
                    c0 = c0 + u.y; c1 = c1 + u.z; c2 = c2 + u.w;
                }
            }
            ++cnt;
        };
        // all cluster indices first, then the gathers in an unrolled
        // sequence the compiler can overlap (sums keep the reference order)
        int ci[kMaxCluster];
#pragma unroll
        for (int j = 0; j < kMaxCluster; ++j) ci[j] = (j < W) ? ld_once(m.cl + (int64_t)j * m.Nn + J) : -1;
#pragma unroll
        for (int j = 0; j < kMaxCluster; ++j)
            if (ci[j] >= 0) add(ci[j], src[ci[j]], UNIT ? 1.0 : ld_once(m.wt + (int64_t)j * m.Nn + J));
        for (int j = kMaxCluster; j < W; ++j) {
            const int c = ld_once(m.cl + (int64_t)j * m.Nn + J);
            if (c >= 0) add(c, src[c], UNIT ? 1.0 : ld_once(m.wt + (int64_t)j * m.Nn + J));
        }
        if (VISC && prim_form && __builtin_expect(!(dr.ok() && pr.ok()), 0)) {
            c2 = 0.0;
            for (int j = 0; j < W; ++j) {
                const int c = m.cl[(int64_t)j * m.Nn + J];
                if (c >= 0) c2 = c2 + phi_plain(src[c]);
            }
        }
        if (UNIT) det = (double)cnt;
        // quotients over the count share its reciprocal (unit weights; sums
        // too small for that, and other weights, take the plain `/`)
        const double dc = (double)cnt, y = rcp_rn(dc);
        Numerators tiny(a0);
        tiny.add(a1); tiny.add(a2); tiny.add(a3);
        if (VISC) { tiny.add(c0); tiny.add(c1); tiny.add(c2); }
        const double huge = fmax(fmax(fabs(a0), fabs(a1)), fmax(fabs(a2), fabs(a3)));
        const bool finite = huge < 1e200 && (!VISC || (fabs(c0) < 1e200 && fabs(c1) < 1e200 && fabs(c2) < 1e200)) &&
                            !(a0 != a0 || a1 != a1 || a2 != a2 || a3 != a3);
        const bool exact = cnt != 0 && finite && tiny.ok();
        if (UNIT && exact) {
            a0 = div_by(a0, dc, y); a1 = div_by(a1, dc, y); a2 = div_by(a2, dc, y); a3 = div_by(a3, dc, y);
        } else if (det != 0.0) {
            a0 = a0 / det; a1 = a1 / det; a2 = a2 / det; a3 = a3 / det;
        }
        s.nodeP[J] = zero_prims ? make_double4(0.0, 0.0, 0.0, 0.0) : make_double4(a0, a1, a2, a3);
        if (VISC) {
            if (exact) {
                c0 = div_by(c0, dc, y); c1 = div_by(c1, dc, y); c2 = div_by(c2, dc, y);
            } else if (cnt != 0) {
                c0 = c0 / dc; c1 = c1 / dc; c2 = c2 / dc;
            }
            if (UNIT && prim_form) { c0 = a1; c1 = a2; }
            s.nodeC[J] = make_double4(c0, c1, c2, 0.0);
        }
    }
    if (flip) {
        // Every warp of the block has read the parity once the barrier is
        // passed; the block that completes the count flips it.  Nothing in
        // this kernel reads what the others wrote, so no fence: stream order
        // makes the flip and the node values visible to the next kernel.
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(s.node_done, 1u) == (unsigned int)nblk - 1u) {
            *s.node_done = 0u;
            *s.parity = par ^ 1;
        }
    }
}

// ------------------------------------------------------ viscous passes

// First Green-Gauss gradient of rho u, rho v, E from the unweighted node
// means (calcScalarFieldGreenGaussNodesBasedGradient, calcGradients.jl:36-139:
// gradX pairs with -ny, gradY with -nx).
template <bool QUAD>
__global__ void __launch_bounds__(256, GD2D_NODE_MINB) k_grad1_cells(const DevMesh m, const DevState s) {
    constexpr int NF = QUAD ? 4 : 3;
    pdl_trigger();
    const bool exact = m.exact_rows != 0;
    pdl_wait();
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < m.Nc; g += (int64_t)gridDim.x * blockDim.x) {
        // Every per-cell load is issued before any of them is tested, so a
        // cell costs two trips to memory (its own arrays, then the node
        // gathers).  Padding cells (zero area, node 0 in their edge slots)
        // are dropped at the store; a triangle's fourth edge has zero length.
        const double area = ld_once(m.area + g);
        double side[NF], nx[NF], ny[NF];
        int2 e[NF];
        const int4 cn = cell_nodes(m, g);
#pragma unroll
        for (int k = 0; k < NF; ++k) {
            const int64_t o = (int64_t)k * m.Nc + g;
            side[k] = ld_once(m.len + o);
            nx[k] = ld_once(m.nx + o);
            ny[k] = ld_once(m.ny + o);
            if (!m.cn) e[k] = ld_once(m.c2n + o);
        }
        const int nf = (QUAD && side[NF - 1] != 0.0) ? 4 : 3;
        double sx[3] = {0.0, 0.0, 0.0}, sy[3] = {0.0, 0.0, 0.0};
        auto edge = [&](int k, const double4 &A, const double4 &B) {
            double fx, fy;
            fx = 0.5 * (A.x + B.x) * -ny[k] * side[k]; fy = 0.5 * (A.x + B.x) * -nx[k] * side[k];
            sx[0] = (k == 0) ? fx : sx[0] + fx; sy[0] = (k == 0) ? fy : sy[0] + fy;
            fx = 0.5 * (A.y + B.y) * -ny[k] * side[k]; fy = 0.5 * (A.y + B.y) * -nx[k] * side[k];
            sx[1] = (k == 0) ? fx : sx[1] + fx; sy[1] = (k == 0) ? fy : sy[1] + fy;
            fx = 0.5 * (A.z + B.z) * -ny[k] * side[k]; fy = 0.5 * (A.z + B.z) * -nx[k] * side[k];
            sx[2] = (k == 0) ? fx : sx[2] + fx; sy[2] = (k == 0) ? fy : sy[2] + fy;
        };
        if (m.cn) {
            const double4 A = s.nodeC[cn.x], B = s.nodeC[cn.y], C = s.nodeC[cn.z];
            edge(0, A, B);
            edge(1, B, C);
            if (nf == 3) {
                edge(2, C, A);
            } else {
                const double4 D = s.nodeC[cn.w];
                edge(2, C, D);
                edge(NF - 1, D, A);
            }
        } else {
#pragma unroll
            for (int k = 0; k < NF; ++k)
                if (k < nf) edge(k, s.nodeC[e[k].x], s.nodeC[e[k].y]);
        }
        if (area == 0.0) continue;
        // six quotients over one area (face_exact.cuh's range: the area's is
        // the case's, a sum too small or too large to be divided right takes
        // the plain `/`)
        const double y = rcp_rn(area);
        double qx[3], qy[3];
        Numerators n(sx[0]);
        Below<700> big(sx[0]);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            qx[v] = div_by(sx[v], area, y);
            qy[v] = div_by(sy[v], area, y);
            if (v > 0) {
                n.add(sx[v]);
                big.add(sx[v]);
            }
            n.add(sy[v]);
            big.add(sy[v]);
        }
        if (__builtin_expect(!(exact && n.ok() && big.ok()), 0)) {
#pragma unroll
            for (int v = 0; v < 3; ++v) { qx[v] = sx[v] / area; qy[v] = sy[v] / area; }
        }
        NodeGrad r;
        r.ru = make_double2(qx[0], qy[0]);
        r.rv = make_double2(qx[1], qy[1]);
        r.re = make_double2(qx[2], qy[2]);
        s.g1[g] = r;
    }
}

// Unweighted node means of the first gradients (calcPhiInCellCluster on the
// gradient fields, calcGradients.jl:3-18), bound by the latency of their
// gathers.  NV = 3: one thread a node takes its three variables in turn.
// NV = 1: three neighbouring threads a node take one variable each, 16 (mixed:
// 8) bytes of a gather's 48 (24), which puts three times the threads to work
// on a mesh that does not fill the device but reads the cluster lists three
// times.  T2: double2 or float2.
template <int NV, class T2>
__device__ __forceinline__ void grad1_nodes(const DevMesh &m, const T2 *__restrict__ g1, T2 *__restrict__ out) {
    const int W = m.cluster_w;
    // FP64: from the last block to the first (see k_node_avg)
    const unsigned bid = sizeof(T2) == 16 ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
    for (int64_t i = (int64_t)bid * blockDim.x + threadIdx.x; i < (3 / NV) * m.Nn;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t J = NV == 3 ? i : (int64_t)((unsigned)i / 3u), v0 = NV == 3 ? 0 : i - 3 * J;
        T2 x[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v].x = x[v].y = 0;
        int cnt = 0;
        auto add = [&](int64_t c) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const T2 q = g1[3 * c + v0 + v];
                x[v].x = x[v].x + q.x;
                x[v].y = x[v].y + q.y;
            }
            ++cnt;
        };
        int ci[kMaxCluster];
#pragma unroll
        for (int j = 0; j < kMaxCluster; ++j) ci[j] = (j < W) ? ld_once(m.cl + (int64_t)j * m.Nn + J) : -1;
#pragma unroll
        for (int j = 0; j < kMaxCluster; ++j)
            if (ci[j] >= 0) add(ci[j]);
        for (int j = kMaxCluster; j < W; ++j) {
            const int c = ld_once(m.cl + (int64_t)j * m.Nn + J);
            if (c >= 0) add(c);
        }
        using T = decltype(x[0].x);
        const T dc = cnt != 0 ? cnt : 1;  // (the sums of no cells are zero)
        const T r = T(1) / dc;            // FP32 multiplies by the reciprocal
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            x[v].x = sizeof(T) == 4 ? x[v].x * r : x[v].x / dc;
            x[v].y = sizeof(T) == 4 ? x[v].y * r : x[v].y / dc;
            out[3 * J + v0 + v] = x[v];
        }
    }
}
template <int NV>
__global__ void __launch_bounds__(256, GD2D_NODE_MINB) k_grad1_nodes(const DevMesh m, const DevState s) {
    pdl_trigger();
    pdl_wait();
    grad1_nodes<NV>(m, reinterpret_cast<const double2 *>(s.g1), reinterpret_cast<double2 *>(s.nodeG));
}

// ------------------------------------------------------------ state init

// phs2dcns2dcellsSA (utilsFVM2dp.jl:4-17) on the current primitives and the
// reductions that give the first step's dt (createFields2d's VMAX).
static __global__ void __launch_bounds__(256) k_init_state(const DevMesh m, const DevState s, int64_t t0, int64_t t1) {
    __shared__ double s_red[8 * kPartials];
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    for (int64_t tile = t0 + blockIdx.x; tile < t1; tile += gridDim.x) {
        const int c = m.tile_case[tile];
        const DevCase &P = m.cases[c];
        const int64_t g = tile * blockDim.x + threadIdx.x;
        Part part;
        part.init();
        const int4 nb = m.nbr[g];
        if (nb.x != kAbsent) {
            const double4 q = pin[g];
            const double G = P.gamma;
            const double r = q.x, u = q.y, v = q.z, pp = q.w;
            s.U[g] = make_double4(r, r * u, r * v, pp / (G - 1.0) + 0.5 * r * (u * u + v * v));
            const double a = sqrt(G * pp / r);
            const double vmax = sqrt(u * u + v * v) + a;
            part.vmax = vmax;
            part.rmin = m.charlen[g] / vmax;
        }
        tile_record<true, false>(m, s, tile, part, s_red);
    }
}

// ------------------------------------------------------- face-loop variants

// One thread per face: the flux seen from cell a (face slot ka), added to a
// and subtracted from the neighbour b (FACE_COLOURED: into Facc, faces of
// one launch never share a cell) or stored in the slots (a, ka) and (b, kb)
// (FACE_SLOTS).  face = (a, neighbour code of slot ka, ka | kb << 8, -).
template <int FLUX, bool QUAD, bool SLOTS>
__global__ void __launch_bounds__(256) k_face_flux(const DevMesh m, const DevState s, const int4 *__restrict__ faces,
                                                   int64_t f0, int64_t f1, int tile_cells,
                                                   double4 *__restrict__ Facc, double4 *__restrict__ Fslot) {
    const int64_t f = f0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= f1) return;
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    const int4 fc = faces[f];
    const int64_t a = fc.x;
    const int nbk = fc.y, ka = fc.z & 255, kb = fc.z >> 8;
    const int c = m.tile_case[a / tile_cells];
    const DevCase &P = m.cases[c];
    const int4 nb = m.nbr[a];
    const bool is_quad = QUAD && (nb.w != kAbsent);
    const double4 me = pin[a];
    const double uL[4] = {me.x, me.y, me.z, me.w};
    const double eh_own = (P.limiter == LIM_VENKAT) ? venkat_half(P.face, m.hx[a]) : 0.0;
    const int4 dn = m.dn[a], up = m.up[a];
    int4 dn2 = make_int4(0, 0, 0, 0), up2 = make_int4(0, 0, 0, 0);
    if (QUAD && is_quad) { dn2 = m.dn2[a]; up2 = m.up2[a]; }
    double fv[4];
    face_flux<FLUX, QUAD>(m, P, pin, s.nodeP, a, ka, nbk, nbr_k(dn, ka), nbr_k(up, ka), nbr_k(dn2, ka),
                          nbr_k(up2, ka), is_quad, uL, eh_own, &s.cstate[c].t, fv);
    if (SLOTS) {
        Fslot[(int64_t)ka * m.Nc + a] = make_double4(fv[0], fv[1], fv[2], fv[3]);
        if (nbk >= 0) Fslot[(int64_t)kb * m.Nc + nbk] = make_double4(-fv[0], -fv[1], -fv[2], -fv[3]);
    } else {
        double4 x = Facc[a];
        Facc[a] = make_double4(x.x + fv[0], x.y + fv[1], x.z + fv[2], x.w + fv[3]);
        if (nbk >= 0) {
            double4 y = Facc[nbk];
            Facc[nbk] = make_double4(y.x - fv[0], y.y - fv[1], y.z - fv[2], y.w - fv[3]);
        }
    }
}

// Euler update and updateVariablesSA after a face loop: the cell kernel's
// second half, with the face-flux sum read back (FACE_SLOTS: summed in face
// order k = 1..nf as calcOneStageMUSCLcpuFast.jl:66-85; FACE_COLOURED: the
// accumulator, reset to zero for the next step).
template <bool VISC, bool QUAD, bool SLOTS, int MINB>
__global__ void __launch_bounds__(256, MINB) k_face_update(const DevMesh m, const DevState s,
                                                          double4 *__restrict__ Facc,
                                                          const double4 *__restrict__ Fslot) {
    __shared__ double s_red[8 * kPartials];
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    double4 *__restrict__ pout = s.prim + (int64_t)(par ^ 1) * m.Nc;
    for (int64_t tile = blockIdx.x; tile < m.ntiles; tile += gridDim.x) {
        const int c = m.tile_case[tile];
        const DevCase &P = m.cases[c];
        const double dt = s.cstate[c].dt;
        const int64_t g = tile * blockDim.x + threadIdx.x;
        Part part;
        part.init();
        const int4 nb = m.nbr[g];
        if (nb.x != kAbsent) {
            const bool is_quad = QUAD && (nb.w != kAbsent);
            const double4 me = pin[g];
            double F[4];
            if (SLOTS) {
                double4 a0 = Fslot[g], a1 = Fslot[m.Nc + g], a2 = Fslot[2 * m.Nc + g];
                F[0] = a0.x + a1.x + a2.x; F[1] = a0.y + a1.y + a2.y;
                F[2] = a0.z + a1.z + a2.z; F[3] = a0.w + a1.w + a2.w;
                if (QUAD && is_quad) {
                    double4 a3 = Fslot[3 * m.Nc + g];
                    F[0] = F[0] + a3.x; F[1] = F[1] + a3.y; F[2] = F[2] + a3.z; F[3] = F[3] + a3.w;
                }
            } else {
                double4 a0 = Facc[g];
                F[0] = a0.x; F[1] = a0.y; F[2] = a0.z; F[3] = a0.w;
                Facc[g] = make_double4(0.0, 0.0, 0.0, 0.0);
            }
            double diff[4] = {0.0, 0.0, 0.0, 0.0};
            if (VISC) diff_source_at<QUAD>(m, s, P, g, is_quad, me, diff);
            cell_update(m, s, P, g, me, F, diff, dt, load_cell_in(m, s, g), pout, part);
        }
        tile_record<true, false>(m, s, tile, part, s_red);
    }
}

// ------------------------------------ the reference's functions one at a time

// calcOneStageMUSCLcpuFast alone (calcOneStageMUSCLcpuFast.jl:3-107): FLUXES
// and Unew from the current primitives, node primitives, Uold and Diff
// (diff may be NULL: zero), with the caller's beta, dt and flowTime.  One
// tile of blockDim cells per block, as the fused kernel.
template <int FLUX, bool QUAD>
__global__ void __launch_bounds__(256) k_stage_only(const DevMesh m, const DevState s, double beta, double dt,
                                                    double t, const double4 *__restrict__ diffs,
                                                    double4 *__restrict__ unew, double4 *__restrict__ fluxes) {
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    const int64_t tile = blockIdx.x;
    const int c = m.tile_case[tile];
    const DevCase &P = m.cases[c];
    const int64_t g = tile * blockDim.x + threadIdx.x;
    const int4 nb = m.nbr[g];
    if (nb.x == kAbsent) return;
    const bool is_quad = QUAD && (nb.w != kAbsent);
    const double4 me = pin[g];
    const double uL[4] = {me.x, me.y, me.z, me.w};
    const double eh_own = (P.limiter == LIM_VENKAT) ? venkat_half(P.face, m.hx[g]) : 0.0;
    double F[4];
    cell_fluxes<FLUX, QUAD>(m, P, pin, s.nodeP, g, nb, is_quad, uL, eh_own, &t, F);
    double diff[4] = {0.0, 0.0, 0.0, 0.0};
    if (diffs) {
        const double4 d = diffs[g];
        diff[0] = d.x; diff[1] = d.y; diff[2] = d.z; diff[3] = d.w;
    }
    const double rarea = m.rarea[g];
    const double4 U = s.U[g];
    const double Uo[4] = {U.x, U.y, U.z, U.w};
    double Un[4];
    for (int v = 0; v < 4; ++v) Un[v] = (Uo[v] - F[v] * beta * dt * rarea + beta * dt * diff[v]);
    unew[g] = make_double4(Un[0], Un[1], Un[2], Un[3]);
    fluxes[g] = make_double4(F[0], F[1], F[2], F[3]);
}

// updateVariablesSA alone (evaluate2d.jl:52-110): primitives of Unew in
// place, Delta = Unew - Uold, Uold <- Unew (density clamp as configured).
static __global__ void __launch_bounds__(256) k_update_only(const DevMesh m, const DevState s, double4 *__restrict__ unew,
                                                     double4 *__restrict__ delta) {
    const int par = *s.parity;
    double4 *__restrict__ prim = s.prim + (int64_t)par * m.Nc;
    const int64_t tile = blockIdx.x;
    const DevCase &P = m.cases[m.tile_case[tile]];
    const int64_t g = tile * blockDim.x + threadIdx.x;
    if (m.nbr[g].x == kAbsent) return;
    double4 un = unew[g];
    if (P.density_constrained == 1) {
        if (un.x >= P.rho_max) un.x = P.rho_max;
        if (un.x <= P.rho_min) un.x = P.rho_min;
        unew[g] = un;
    }
    const double G = P.gamma;
    const double rho = un.x, ux = un.y / un.x, uy = un.z / un.x;
    const double p = (G - 1.0) * (un.w - 0.5 * (un.y * un.y + un.z * un.z) / un.x);
    prim[g] = make_double4(rho, ux, uy, p);
    const double4 uo = s.U[g];
    delta[g] = make_double4(un.x - uo.x, un.y - uo.y, un.z - uo.z, un.w - uo.w);
    s.U[g] = un;
}

// calcDiffTerm alone (calcDiffTerm.jl:31-121): the diffusion source from
// the first-gradient node means (the grad1 passes must have run).
template <bool QUAD>
__global__ void __launch_bounds__(256) k_diff_only(const DevMesh m, const DevState s, double4 *__restrict__ diffs) {
    const int par = *s.parity;
    const double4 *__restrict__ pin = s.prim + (int64_t)par * m.Nc;
    const int64_t tile = blockIdx.x;
    const DevCase &P = m.cases[m.tile_case[tile]];
    const int64_t g = tile * blockDim.x + threadIdx.x;
    const int4 nb = m.nbr[g];
    if (nb.x == kAbsent) return;
    double diff[4];
    diff_source_at<QUAD>(m, s, P, g, QUAD && nb.w != kAbsent, pin[g], diff);
    diffs[g] = make_double4(diff[0], diff[1], diff[2], diff[3]);
}

}  // namespace gd2d
