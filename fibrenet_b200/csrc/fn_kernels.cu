/*
 * fn_kernels.cu -- sm_100a kernels of the FibreNet step loop.
 *
 * One time step is one launch of k_step: every thread owns one bead and
 *   1. rebuilds the base force the reference writes in AdvancePosition
 *      (damping * v + gravity + wall penalty, kernel.cl:231-261),
 *   2. gathers its incident springs (kernel.cl:366-441), angles
 *      (kernel.cl:268-363) and contacts (kernel.cl:792-1011) in a fixed order
 *      instead of the reference's FP64 atomics,
 *   3. applies AdvanceVelocity (kernel.cl:444-464), and
 *   4. applies the next step's AdvancePosition (kernel.cl:195-265), writing the
 *      drifted position into the other half of a ping-pong pair so neighbours
 *      still read this step's positions.
 * A standalone k_drift opens each fn_step call.  The contact list is rebuilt
 * between steps (k_cells -> scan -> k_scatter -> k_cell_sort -> k_lists),
 * giving the same pair set as FillGrid + BuildContactList (kernel.cl:487-789)
 * with deterministic order.
 *
 * All force arithmetic is FP64 with the reference's operation order; the
 * library is built with -fmad=false so nothing is contracted into FMAs, and
 * the roots, reciprocals and quotients of fn_rounded.cuh round as the operators
 * do, which keeps results bit-identical to the host mirror checker.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>

#include "fn_detmath.h"
#include "fn_device.cuh"
#include "fn_kernels.h"
#include "fn_launch.cuh"
#include "fn_rounded.cuh"
#include "fn_types.h"

namespace fn {

__device__ __forceinline__ int spring_pts(double ax, double ay, double az, double bx, double by,
                                          double bz, float4 par, int type, double& fx, double& fy,
                                          double& fz, int& broke);

/* Spring s (kernel.cl:371-437): returns 1 when a force acts, f = force on p1
   (p2 takes f * -1.0); broke = 1 when this evaluation breaks an HR_FL
   spring (kernel.cl:391-397). */
__device__ __forceinline__ int spring_eval(const StepArgs& A, int s, double& fx, double& fy,
                                           double& fz, int& broke) {
    broke = 0;
    const int type = A.sp_type[s];
    if (!(type == 0 || type == 1)) return 0;
    if (A.sp_status[s] != 1) return 0;
    const int2 e = A.sp_ends[s];
    const double4 a = A.img_in[e.x];
    const double4 b = A.img_in[e.y];
    return spring_pts(a.x, a.y, a.z, b.x, b.y, b.z, A.sp_par[s], type, fx, fy, fz, broke);
}

/* The spring force of kernel.cl:377-424 from the image positions of p1 (a)
   and p2 (b); shared by the incidence and chain kernels. */
__device__ __forceinline__ int spring_pts(double ax, double ay, double az, double bx, double by,
                                          double bz, float4 par, int type, double& fx, double& fy,
                                          double& fz, int& broke) {
    broke = 0;
    double dx = ax - bx, dy = ay - by, dz = az - bz;
    double l, il;
    root_and_inverse(dx * dx + dy * dy + dz * dz, l, il);
    double factor = (double)par.x - l;
    dx *= il;
    dy *= il;
    dz *= il;
    if (type == 1) {
        double stress = -(double)par.z * factor * il;
        if (fabs(stress) > (double)par.w) {
            broke = 1;
            return 0;
        }
    }
    factor *= (double)par.y;
    fx = dx * factor;
    fy = dy * factor;
    fz = dz * factor;
    return 1;
}

__device__ __forceinline__ int spring_alive_after(const StepArgs& A, int s) {
    if (A.sp_status[s] != 1) return 0;
    double fx, fy, fz;
    int broke;
    spring_eval(A, s, fx, fy, fz, broke);
    return !broke;
}

/* fn_acos with the root of its half-angle reduction from fn_rounded.cuh. */
__device__ __forceinline__ double acos_rounded(double x) {
    const double ax = fabs(x);
    if (!(ax > 0.5)) return 1.5707963267948966 - fn_asin_poly(x); /* NaN stays NaN */
    const double h = (1.0 - ax) * 0.5;
    double s;
    if (fn_fast_range(h))
        s = root_from(h, rsqrt_seeded(h));
    else
        s = sqrt(h);
    const double a = 2.0 * fn_asin_poly(s);
    return x > 0.0 ? a : 3.141592653589793 - a;
}

/* Angle force (kernel.cl:291-348) from the arms ba = b1 - b2 and cb = b2 - b3,
   their lengths and the inverses of those (correctly rounded): pa acts on b1,
   pc on b3.  Swapping the arms swaps pa and pc bit for bit. */
__device__ __forceinline__ void angle_arms(double bax, double bay, double baz, double cbx, double cby, double cbz,
                                           double l_ba, double il_ba, double l_bc, double il_bc, float2 par,
                                           double& pax, double& pay, double& paz, double& pcx, double& pcy,
                                           double& pcz) {
    const double bcx = -cbx, bcy = -cby, bcz = -cbz;
    const double dot = bax * bcx + bay * bcy + baz * bcz;
    const double ll = l_ba * l_bc;
    const bool fast = fn_fast_range(ll);
    /* |dot| <= ll up to rounding: finite, and where it is too small for the
       quotient's residual the arc cosine does not see it */
    double dotp = fast ? quotient(dot, ll, recip_near(ll, il_ba * il_bc)) : dot / ll;
    if (dotp < -1.0) dotp = -0.999999;
    if (dotp > 1.0) dotp = 0.999999;
    const double angle = acos_rounded(dotp);
    const double magnitude = -2.0 * (double)par.y * (angle - (double)par.x);
    const bool fast_ends = fast && fn_quotient_range(magnitude);
    const double fa = fast_ends ? quotient(magnitude, l_ba, il_ba) : magnitude / l_ba;
    const double fc = fast_ends ? quotient(magnitude, l_bc, il_bc) : magnitude / l_bc;
    const double tx = bay * bcz - baz * bcy;
    const double ty = baz * bcx - bax * bcz;
    const double tz = bax * bcy - bay * bcx;
    double ln, il;
    pax = (bay * tz - baz * ty);
    pay = (baz * tx - bax * tz);
    paz = (bax * ty - bay * tx);
    root_and_inverse(pax * pax + pay * pay + paz * paz, ln, il);
    il *= fa;
    pax *= il;
    pay *= il;
    paz *= il;
    pcx = (cby * tz - cbz * ty);
    pcy = (cbz * tx - cbx * tz);
    pcz = (cbx * ty - cby * tx);
    root_and_inverse(pcx * pcx + pcy * pcy + pcz * pcz, ln, il);
    il *= fc;
    pcx *= il;
    pcy *= il;
    pcz *= il;
}

/* The same from the image positions of b1 (t1), b2 (t2), b3 (t3). */
__device__ __forceinline__ void angle_pts(double t1x, double t1y, double t1z, double t2x,
                                          double t2y, double t2z, double t3x, double t3y,
                                          double t3z, float2 par, double& pax, double& pay,
                                          double& paz, double& pcx, double& pcy, double& pcz) {
    const double bax = t1x - t2x, bay = t1y - t2y, baz = t1z - t2z;
    const double cbx = t2x - t3x, cby = t2y - t3y, cbz = t2z - t3z;
    double la, ila, lc, ilc;
    root_and_inverse(bax * bax + bay * bay + baz * baz, la, ila);
    root_and_inverse(cbx * cbx + cby * cby + cbz * cbz, lc, ilc);
    angle_arms(bax, bay, baz, cbx, cby, cbz, la, ila, lc, ilc, par, pax, pay, paz, pcx, pcy, pcz);
}

__device__ __forceinline__ void angle_eval(const StepArgs& A, int4 b, float2 par, double& pax,
                                           double& pay, double& paz, double& pcx, double& pcy,
                                           double& pcz) {
    const double4 t2 = A.img_in[b.y];
    const double4 t1 = A.img_in[b.x];
    const double4 t3 = A.img_in[b.z];
    angle_pts(t1.x, t1.y, t1.z, t2.x, t2.y, t2.z, t3.x, t3.y, t3.z, par, pax, pay, paz, pcx, pcy,
              pcz);
}

/* One contact-list entry (kernel.cl:835-999) under the pair law P: force on
   bead i.  Roots, reciprocals and quotients of the distance share one seed
   (fn_rounded.cuh); distances outside its range take the operators.  Also the
   separation (rx, ry, rz), the distance r and its inverse of an acting pair. */
__device__ __forceinline__ int contact_law(const FnNet& N, const FnPair& law, double4 pi, double4 pj, double& Rx,
                                           double& Ry, double& Rz, double& rx, double& ry, double& rz, double& r,
                                           double& ir) {
    const FnPair* P = &law;
    rx = pi.x - pj.x;
    ry = pi.y - pj.y;
    rz = pi.z - pj.z;
    double length = rx * rx + ry * ry + rz * rz;
    length = min_image(N, rx, ry, rz, length, N.force_mi);
    const int kind = P->kind;
    if (kind == 1) {
        if (!(length < N.cutoff_sq)) return 0;
        const double r2 = length;
        double fpr;
        if (r2 >= P->lj_r2_min) {
            const double y = rsqrt_seeded(r2);
            r = root_from(r2, y);
            if (!(r < P->c[2])) return 0;
            ir = recip_from(r, y);
            const double ir2 = recip_near(r2, y * y);
            const double fr2 = quotient(P->lj_s2, r2, ir2);
            const double fr6 = fr2 * fr2 * fr2;
            fpr = quotient(P->lj_e48 * fr6 * (fr6 - 0.5), r2, ir2);
        } else {
            r = sqrt(r2);
            if (!(r < P->c[2])) return 0;
            const double fr2 = P->lj_s2 / r2;
            const double fr6 = fr2 * fr2 * fr2;
            fpr = P->lj_e48 * fr6 * (fr6 - 0.5) / r2;
            ir = (r != 0.0) ? 1.0 / r : 0.0;
        }
        fpr -= P->c[3];
        Rx = fpr * (rx * ir);
        Ry = fpr * (ry * ir);
        Rz = fpr * (rz * ir);
        return 1;
    }
    double mag;
    if (kind == 2) {
        root_and_inverse(length, r, ir);
        mag = ((double)w_radius(pi.w) + (double)w_radius(pj.w)) - r;
        if (!(mag > 0.0)) return 0;
        mag *= P->c[0];
    } else if (kind == 4) {
        /* extension, no counterpart in the reference: penalty spring K (c1)
           on the overlap plus a soft harmonic repulsion k (c2) below rc (c3) */
        root_and_inverse(length, r, ir);
        const double penetration = ((double)w_radius(pi.w) + (double)w_radius(pj.w)) - r;
        mag = 0.0;
        int acts = 0;
        if (penetration > 0.0) {
            mag += penetration * P->c[0];
            acts = 1;
        }
        if (r < P->c[2]) {
            mag += (P->c[2] - r) * P->c[1];
            acts = 1;
        }
        if (!acts) return 0;
    } else if (kind == 3) {
        if (!(length < P->c[3])) return 0;
        root_and_inverse(length, r, ir);
        mag = (P->c[1] - r);
        mag *= P->c[0]; /* both arms of kernel.cl:970-973 multiply by K */
        mag += (P->c[5] - r) * P->c[4];
    } else {
        return 0;
    }
    Rx = mag * (rx * ir);
    Ry = mag * (ry * ir);
    Rz = mag * (rz * ir);
    return 1;
}

__device__ __forceinline__ int contact_force(const FnNet& N, const FnPair& law, double4 pi, double4 pj, double& Rx,
                                             double& Ry, double& Rz) {
    double rx, ry, rz, r, ir;
    return contact_law(N, law, pi, pj, Rx, Ry, Rz, rx, ry, rz, r, ir);
}

/* The same with the law looked up by the beads' types. */
__device__ __forceinline__ int contact_eval(const FnNet& N, const FnPair* __restrict__ pairs,
                                            double4 pi, double4 pj, double& Rx, double& Ry,
                                            double& Rz) {
    return contact_force(N, pairs[N.pair_base + getadress(w_type(pi.w), w_type(pj.w), N.types_num)], pi, pj, Rx, Ry,
                         Rz);
}

/* AdvancePosition (kernel.cl:200-250) on registers: returns the drifted
   position/image, the predicted velocity. */
__device__ __forceinline__ void drift(const FnNet& N, double minv, float fx, float fy, float fz,
                                      float vox, float voy, float voz, double4& p, double4& im,
                                      float4& v) {
    const double lambda_dt = N.lambda_dt * minv;
    const double half_dt2 = N.half_dt2 * minv;
    v.x = (float)((double)fx * lambda_dt + (double)vox);
    v.y = (float)((double)fy * lambda_dt + (double)voy);
    v.z = (float)((double)fz * lambda_dt + (double)voz);
    v.w = 0.0f;
    double ix = (double)vox, iy = (double)voy, iz = (double)voz;
    ix *= N.dt;
    iy *= N.dt;
    iz *= N.dt;
    ix = (double)fx * half_dt2 + ix;
    iy = (double)fy * half_dt2 + iy;
    iz = (double)fz * half_dt2 + iz;
    p.x += ix;
    p.y += iy;
    p.z += iz;
    im.x += ix;
    im.y += iy;
    im.z += iz;
    /* snap wrap, kernel.cl:241-250 */
    if (N.periodic & 4)
        if (p.z < 0.0) p.z = N.box[2];
    if (N.periodic & 2)
        if (p.y < 0.0) p.y = N.box[1];
    if (N.periodic & 1)
        if (p.x < 0.0) p.x = N.box[0];
    if (N.periodic & 4)
        if (p.z > N.box[2]) p.z = 0.0;
    if (N.periodic & 2)
        if (p.y > N.box[1]) p.y = 0.0;
    if (N.periodic & 1)
        if (p.x > N.box[0]) p.x = 0.0;
}

/* Base force of AdvancePosition: damping * v + gravity, then the wall
   penalty at the drifted position (kernel.cl:231-261). */
template <bool DAMP>
__device__ __forceinline__ void base_force(const StepArgs& A, const FnNet& N, int i, double4 p,
                                           double& Fx, double& Fy, double& Fz) {
    if (DAMP) {
        const float4 v = A.vel[i];
        Fx = N.damping * (double)v.x;
        Fy = N.damping * (double)v.y;
        Fz = N.damping * (double)v.z;
    } else {
        Fx = 0.0;
        Fy = 0.0;
        Fz = 0.0;
    }
    Fx += N.g[0];
    Fy += N.g[1];
    Fz += N.g[2];
    if (N.walls) {
        if ((N.walls & 4) && p.z < 0.0) Fz += p.z * N.wall_k * -1.0;
        if ((N.walls & 2) && p.y < 0.0) Fy += p.y * N.wall_k * -1.0;
        if ((N.walls & 1) && p.x < 0.0) Fx += p.x * N.wall_k * -1.0;
        if ((N.walls & 4) && p.z > N.box[2]) Fz += (p.z - N.box[2]) * N.wall_k * -1.0;
        if ((N.walls & 2) && p.y > N.box[1]) Fy += (p.y - N.box[1]) * N.wall_k * -1.0;
        if ((N.walls & 1) && p.x > N.box[0]) Fx += (p.x - N.box[0]) * N.wall_k * -1.0;
    }
}

/* Flags of the step kernels: what a step does after the kick, and the terms
   that the chain kernel's forces-only form evaluates. */
enum { FN_STEP_SPRINGS = 1, FN_STEP_ANGLES = 2, FN_STEP_CONTACTS = 4, FN_STEP_DRIFT = 8, FN_STEP_STORE_V = 16 };

/* What the kick reads of bead i: its image position, force and velocity_old. */
struct KickState {
    double4 im;
    float4 fo, vo;
};

__device__ __forceinline__ KickState kick_state(const StepArgs& A, int i) {
    return KickState{A.img_in[i], A.force[i], A.vold[i]};
}

/* AdvanceVelocity and the next AdvancePosition for bead i with its complete
   force (Fx, Fy, Fz), then the stores. */
template <bool DAMP>
__device__ __forceinline__ void kick_drift(const StepArgs& A, const FnNet& N, int i, double4 p, double Fx, double Fy,
                                           double Fz, KickState k, bool do_drift, bool store_v) {
    double4 im = k.im;
    const float4 fo = k.fo, vo = k.vo;
    const float fx = (float)Fx, fy = (float)Fy, fz = (float)Fz;
    if (!(isfinite(fx) && isfinite(fy) && isfinite(fz)))
        atomicAdd(A.counters + FN_CNT_NONFINITE, 1ull);

    /* AdvanceVelocity, kernel.cl:451-462 */
    const double minv = im.w;
    const double half_dt = N.half_dt * minv;
    double tx = (double)fx, ty = (double)fy, tz = (double)fz;
    tx += (double)fo.x;
    ty += (double)fo.y;
    tz += (double)fo.z;
    const float vox = (float)(tx * half_dt + (double)vo.x);
    const float voy = (float)(ty * half_dt + (double)vo.y);
    const float voz = (float)(tz * half_dt + (double)vo.z);
    A.force[i] = make_float4(fx, fy, fz, 0.0f);
    A.vold[i] = make_float4(vox, voy, voz, 0.0f);

    if (do_drift) {
        float4 v;
        drift(N, minv, fx, fy, fz, vox, voy, voz, p, im, v);
        A.pos_out[i] = p;
        A.img_out[i] = im;
        if (store_v) A.vel[i] = v;
    }
}

/* Contacts, AdvanceVelocity and the next step's AdvancePosition for bead i,
   given its base + bonded force (Fx, Fy, Fz) in FP64.  The next list index is
   loaded one item ahead. */
template <bool DAMP, bool UNIFORM>
__device__ __forceinline__ void finish_bead(const StepArgs& A, const FnNet& N, int i, double4 p, double Fx, double Fy,
                                            double Fz, int flags) {
    int n = A.list_count[i];
    if (n > A.list_cap) n = A.list_cap;
    const int* row = A.list + i;
    int jn = *row;
    for (int k = 0; k < n; ++k) {
        const int j = jn;
        if (k + 1 < A.list_cap) row += A.list_stride;
        jn = *row;
        double Rx, Ry, Rz;
        if (UNIFORM ? contact_force(N, A.pair0, p, A.pos_in[j], Rx, Ry, Rz)
                    : contact_eval(N, A.pairs, p, A.pos_in[j], Rx, Ry, Rz)) {
            Fx += Rx;
            Fy += Ry;
            Fz += Rz;
        }
    }
    /* late: the next step's blocks take shared memory and slots from this one's
       (60k beads: 19.1 us per step, 20.2 with this at the kernel's start) */
    let_next_start();
    /* loaded before the finiteness test: behind its branch these loads, and
       with them every load of the kernel that reaches DRAM, take twice as
       long (1M-bead tensile step 204 us against 108, the same sectors, hits
       and DRAM bytes; networks that fit L2 see no difference) */
    const KickState state = kick_state(A, i);
    kick_drift<DAMP>(A, N, i, p, Fx, Fy, Fz, state, (flags & FN_STEP_DRIFT) != 0, DAMP || (flags & FN_STEP_STORE_V));
}

template <bool DAMP>
__global__ void __launch_bounds__(512) k_step(const __grid_constant__ StepArgs A, int flags) {
    await_previous();
    const FnTile t = A.tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    if (i >= t.end) return;
    const FnNet& N = A.nets[t.net];

    const double4 p = A.pos_in[i];
    double Fx, Fy, Fz;
    base_force<DAMP>(A, N, i, p, Fx, Fy, Fz);

    /* springs */
    const int se = A.sp_off[i + 1];
    for (int e = A.sp_off[i]; e < se; ++e) {
        const int ent = A.sp_ent[e];
        const int s = ent >> 1;
        double fx, fy, fz;
        int broke;
        if (spring_eval(A, s, fx, fy, fz, broke)) {
            if ((ent & 1) == 0) {
                Fx += fx;
                Fy += fy;
                Fz += fz;
            } else {
                Fx += fx * -1.0;
                Fy += fy * -1.0;
                Fz += fz * -1.0;
            }
        }
        if (broke && (ent & 1) == 0) A.sp_status[s] = 0;
    }

    /* angles */
    const int ae = A.an_off[i + 1];
    for (int e = A.an_off[i]; e < ae; ++e) {
        const int ent = A.an_ent[e];
        const int a = ent >> 2;
        const int role = ent & 3;
        if (A.an_status[a] != 1) continue;
        const int4 b = A.an_b[a];
        if (b.w == 1) {
            const int2 ss = A.an_s[a];
            if (!spring_alive_after(A, ss.x) || !spring_alive_after(A, ss.y)) {
                if (role == 1) A.an_status[a] = 0;
                continue;
            }
        }
        double pax, pay, paz, pcx, pcy, pcz;
        angle_eval(A, b, A.an_par[a], pax, pay, paz, pcx, pcy, pcz);
        if (role == 0) {
            Fx += pax;
            Fy += pay;
            Fz += paz;
        } else if (role == 2) {
            Fx += pcx;
            Fy += pcy;
            Fz += pcz;
        } else {
            Fx += -pax - pcx;
            Fy += -pay - pcy;
            Fz += -paz - pcz;
        }
    }

    finish_bead<DAMP, false>(A, N, i, p, Fx, Fy, Fz, flags);
}

/* The same step with the bonded terms evaluated once per tile: the block
   first evaluates every spring, then every angle incident to its beads into
   shared memory (flag bits: 1 force acts, 2 broke this step, 4 alive at step
   start), then each thread gathers its bead's terms from the shared slots in
   the same order as k_step, so the result is bit-identical to k_step. */
template <bool DAMP, bool UNIFORM>
__global__ void __launch_bounds__(512) k_step_tiled(const __grid_constant__ StepArgs A, int flags) {
    await_previous();
    extern __shared__ double smem[];
    const int t = blockIdx.x;
    const FnTile tile = A.tiles[t];
    double* sp_f = smem;
    double* an_f = sp_f + 3 * A.max_tile_sp;
    unsigned char* sp_flag = reinterpret_cast<unsigned char*>(an_f + 6 * A.max_tile_an);
    unsigned char* an_flag = sp_flag + A.max_tile_sp;

    const int sp0 = A.tile_sp_off[t], nsp = A.tile_sp_off[t + 1] - sp0;
    for (int q = threadIdx.x; q < nsp; q += blockDim.x) {
        const int s = A.tile_sp[sp0 + q];
        double fx = 0.0, fy = 0.0, fz = 0.0;
        int broke;
        const int alive0 = A.sp_status[s] == 1;
        const int acts = spring_eval(A, s, fx, fy, fz, broke);
        sp_f[3 * q] = fx;
        sp_f[3 * q + 1] = fy;
        sp_f[3 * q + 2] = fz;
        sp_flag[q] = (unsigned char)(acts | (broke << 1) | (alive0 << 2));
        if (broke) A.sp_status[s] = 0;
    }
    __syncthreads();
    const int an0 = A.tile_an_off[t], nan = A.tile_an_off[t + 1] - an0;
    for (int q = threadIdx.x; q < nan; q += blockDim.x) {
        const int a = A.tile_an[an0 + q];
        int alive = A.an_status[a] == 1;
        const int4 b = A.an_b[a];
        if (alive && b.w == 1) {
            const int2 ss = A.tile_an_sslot[an0 + q];
            const unsigned f1 = sp_flag[ss.x], f2 = sp_flag[ss.y];
            const int ok1 = (f1 & 4) && !(f1 & 2);
            const int ok2 = (f2 & 4) && !(f2 & 2);
            if (!ok1 || !ok2) {
                alive = 0;
                A.an_status[a] = 0;
            }
        }
        an_flag[q] = (unsigned char)alive;
        if (alive) {
            double* o = an_f + 6 * q;
            angle_eval(A, b, A.an_par[a], o[0], o[1], o[2], o[3], o[4], o[5]);
        }
    }
    __syncthreads();

    const int i = tile.begin + (int)threadIdx.x;
    if (i >= tile.end) return;
    const FnNet& N = UNIFORM ? A.net0 : A.nets[tile.net];
    const double4 p = A.pos_in[i];
    double Fx, Fy, Fz;
    base_force<DAMP>(A, N, i, p, Fx, Fy, Fz);
    const int se = A.sp_off[i + 1];
    for (int e = A.sp_off[i]; e < se; ++e) {
        const int ent = A.sp_slot[e];
        const int q = ent >> 1;
        if (sp_flag[q] & 1) {
            const double* f = sp_f + 3 * q;
            if ((ent & 1) == 0) {
                Fx += f[0];
                Fy += f[1];
                Fz += f[2];
            } else {
                Fx += f[0] * -1.0;
                Fy += f[1] * -1.0;
                Fz += f[2] * -1.0;
            }
        }
    }
    const int ae = A.an_off[i + 1];
    for (int e = A.an_off[i]; e < ae; ++e) {
        const int ent = A.an_slot[e];
        const int q = ent >> 2;
        const int role = ent & 3;
        if (!an_flag[q]) continue;
        const double* o = an_f + 6 * q;
        if (role == 0) {
            Fx += o[0];
            Fy += o[1];
            Fz += o[2];
        } else if (role == 2) {
            Fx += o[3];
            Fy += o[4];
            Fz += o[5];
        } else {
            Fx += -o[0] - o[3];
            Fy += -o[1] - o[4];
            Fz += -o[2] - o[5];
        }
    }
    finish_bead<DAMP, UNIFORM>(A, N, i, p, Fx, Fy, Fz, flags);
}

/* Exclusive prefix sum of v over the block (any size up to 1024); total
   receives the block sum.  warp_sums needs 33 ints. */
__device__ __forceinline__ int block_scan_any(int v, int* warp_sums, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < nwarps ? warp_sums[lane] : 0;
        int sacc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, sacc, o);
            if (lane >= o) sacc += y;
        }
        warp_sums[lane] = sacc - w;
        if (lane == 31) warp_sums[32] = sacc;
    }
    __syncthreads();
    total = warp_sums[32];
    const int r = x - v + warp_sums[warp];
    __syncthreads();
    return r;
}

/* A network's constants into shared memory, by the block's first threads. */
__device__ __forceinline__ void copy_net(const FnNet* __restrict__ from, FnNet* to) {
    static_assert(sizeof(FnNet) % 8 == 0 && sizeof(FnNet) / 8 <= 64, "one word per thread");
    if (threadIdx.x < sizeof(FnNet) / 8)
        reinterpret_cast<long long*>(to)[threadIdx.x] = reinterpret_cast<const long long*>(from)[threadIdx.x];
}

/* The spring from a bead to the next one, (x, y, z) apart (kernel.cl:377-424):
   their distance l and its inverse, the force on the bead, and the bead's
   status after the step. */
__device__ __forceinline__ void chain_spring(unsigned fl, unsigned st0, float4 par, bool wanted, double x, double y,
                                             double z, double& l, double& il, double& gx, double& gy, double& gz,
                                             unsigned& st) {
    root_and_inverse(x * x + y * y + z * z, l, il);
    if ((fl & FN_CH_SPRING) && (st0 & 1) && !(fl & FN_CH_SP_INERT)) {
        double factor = (double)par.x - l;
        if ((fl & FN_CH_SP_FL) && fabs(-(double)par.z * factor * il) > (double)par.w) {
            st &= ~1u; /* breaks: no force from this step on (kernel.cl:391-397) */
        } else if (wanted) {
            factor *= (double)par.y;
            gx = x * il * factor;
            gy = y * il * factor;
            gz = z * il * factor;
        }
    }
}

/* A bead's bonded terms in ascending bond order: previous spring, next spring
   (f: its slot of the springs' forces), angles centred on the previous bead,
   on itself (cx, cy, cz) and on the next one (o: its slot of the angles'). */
__device__ __forceinline__ void chain_gather(const double* f, const double* o, double cx, double cy, double cz,
                                             double& Fx, double& Fy, double& Fz) {
    Fx -= f[-3];
    Fy -= f[-2];
    Fz -= f[-1];
    Fx += f[0];
    Fy += f[1];
    Fz += f[2];
    Fx += o[-3];
    Fy += o[-2];
    Fz += o[-1];
    Fx += cx;
    Fy += cy;
    Fz += cz;
    Fx += o[6];
    Fy += o[7];
    Fz += o[8];
}

/* Step kernel for networks in chain form (every spring joins consecutive
   beads j, j+1 and every angle is centred on its middle bead, as fibres
   are).  Thread t of a block works for bead j = tile begin - 2 + t (the tile
   and a two-bead halo on each side): the block puts the image positions in
   shared memory, then each thread evaluates the spring (j, j+1) and the
   angle centred on j (springs first: an HR_FL angle dies with either of its
   springs in the same step, kernel.cl:274-286), and the tile's threads add
   their bead's terms in ascending bond order -- previous spring, next
   spring, angles centred on j-1, j, j+1 -- which is the order of the
   incidence path, so both produce identical bits.  A spring listed from its
   upper bead and an angle listed from its far arm give the same bits as the
   forward ones (every operation is symmetric under the swap), so the
   records' direction is not read.  An angle takes its arms' lengths and
   their inverses from the springs' threads.  FORCES_ONLY evaluates the
   selected terms alone (no base force, no kick or drift, no status change).
   CONSTS says what comes from the kernel parameters, as constant operands,
   instead of being loaded for every contact: the network's constants and its
   one pair law (1M-bead tensile step 108 us against 120 with them loaded), the
   law alone (several networks that share it), or nothing; a network's
   constants then lie in shared memory.
   Bound by instruction issue and the latency of dependent loads and FP64
   chains, not by DRAM (229 MB per 1M-bead step).  Sharing the roots' seeds
   and the arms' lengths took it from 71.7M to 56.5M warp instructions: 130 to
   108 us on the 1M-bead tensile network, 600 to 526 us on the 4M-bead mat, 24
   to 20 us at 111k beads (one wave of blocks).  At most 256 threads per block
   and 4 such blocks per SM, i.e. 64 registers: both resident warps and the
   registers that keep the next list index in flight hide the loads' latency. */
template <bool DAMP, bool FORCES_ONLY, int CONSTS>
__global__ void __launch_bounds__(kChainMaxBlock, 4) k_step_chain(const __grid_constant__ StepArgs A, int flags) {
    extern __shared__ __align__(32) unsigned char smem_raw[];
    const FnTile tile = A.tiles[blockIdx.x];
    const int tid = threadIdx.x, n = tile.end - tile.begin;
    const int i = tile.begin - 2 + tid; /* this thread's bead */
    const ChainSmem L = chain_smem_layout(blockDim.x);
    double* s_img = reinterpret_cast<double*>(smem_raw + L.img);
    double2* s_len = reinterpret_cast<double2*>(smem_raw + L.len);
    double* s_spf = reinterpret_cast<double*>(smem_raw + L.spf);
    double* s_ang = reinterpret_cast<double*>(smem_raw + L.ang);
    unsigned char* s_ok = smem_raw + L.ok;
    __shared__ FnNet s_net;
    if (CONSTS != FN_CONST_ALL) copy_net(A.nets + tile.net, &s_net);
    const FnNet& N = CONSTS == FN_CONST_ALL ? A.net0 : s_net; /* past the first barrier */

    /* tiles and flags are written by no kernel of the step sequence; loading the
       bonds' records here too gains 2 % on 480 beads and costs 1.5 % on the
       large networks (registers) */
    const bool mine = tid < n + 4 && i >= 0 && i < A.nb;
    unsigned fl = 0, st0 = 0;
    if (mine) fl = A.ch_flags[i];
    await_previous();
    double x = 0.0, y = 0.0, z = 0.0;
    if (mine) {
        const double4 q = A.img_in[i];
        x = q.x;
        y = q.y;
        z = q.z;
        st0 = A.ch_status[i];
    }
    s_img[3 * tid] = x;
    s_img[3 * tid + 1] = y;
    s_img[3 * tid + 2] = z;
    __syncthreads();

    /* spring (i, i+1): force on bead i (kernel.cl:377-424) */
    double l = 0.0, il = 0.0;
    double gx = 0.0, gy = 0.0, gz = 0.0;
    unsigned st = st0; /* statuses after this step */
    if (tid < n + 3) {
        x -= s_img[3 * tid + 3];
        y -= s_img[3 * tid + 4];
        z -= s_img[3 * tid + 5];
        chain_spring(fl, st0, (fl & FN_CH_SPRING) ? A.ch_sp[i] : make_float4(0.f, 0.f, 0.f, 0.f),
                     !FORCES_ONLY || (flags & FN_STEP_SPRINGS), x, y, z, l, il, gx, gy, gz, st);
        s_len[tid] = make_double2(l, il);
        s_spf[3 * tid] = gx;
        s_spf[3 * tid + 1] = gy;
        s_spf[3 * tid + 2] = gz;
        s_ok[tid] = (unsigned char)((fl & FN_CH_SPRING) && (st & 1));
    }
    __syncthreads();

    /* angle centred on bead i */
    double cx = 0.0, cy = 0.0, cz = 0.0; /* its force on bead i */
    if (tid >= 1 && tid < n + 3) {
        double pax = 0.0, pay = 0.0, paz = 0.0, pcx = 0.0, pcy = 0.0, pcz = 0.0;
        if ((fl & FN_CH_ANGLE) && (st0 & 2)) {
            if ((fl & FN_CH_AN_FL) && !(s_ok[tid - 1] && s_ok[tid])) {
                st &= ~2u; /* kernel.cl:278-284 */
            } else if (!FORCES_ONLY || (flags & FN_STEP_ANGLES)) {
                const double* q = s_img + 3 * tid;
                const double2 lp = s_len[tid - 1];
                angle_arms(q[-3] - q[0], q[-2] - q[1], q[-1] - q[2], x, y, z, lp.x, lp.y, l, il, A.ch_an[i], pax, pay,
                           paz, pcx, pcy, pcz);
                cx = -pax - pcx;
                cy = -pay - pcy;
                cz = -paz - pcz;
            }
        }
        double* o = s_ang + 6 * tid;
        o[0] = pax;
        o[1] = pay;
        o[2] = paz;
        o[3] = pcx;
        o[4] = pcy;
        o[5] = pcz;
    }
    __syncthreads();

    const bool active = tid >= 2 && tid < n + 2;
    /* a block that stages this bead as halo may see the old status or the
       new one: a bond that dies in this step acts in neither case */
    if (!FORCES_ONLY && active && st != st0) A.ch_status[i] = (unsigned char)st;
    double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    int nc = 0;
    if (active) {
        p = A.pos_in[i];
        if (!FORCES_ONLY) base_force<DAMP>(A, N, i, p, Fx, Fy, Fz);
        chain_gather(s_spf + 3 * tid, s_ang + 6 * tid, cx, cy, cz, Fx, Fy, Fz);
        if (!FORCES_ONLY || (flags & FN_STEP_CONTACTS)) {
            nc = A.list_count[i];
            if (nc > A.list_cap) nc = A.list_cap;
        }
    }

    /* contacts, load-balanced inside each warp: after a direct phase over the
       leading items of every list, the remaining items are taken 32 at a
       time, lane l evaluating item (window base + l); a 32-byte map tells each
       lane whose item it holds, results go to shared memory and every bead
       then adds its own items in list order (the order of a sequential loop
       over its list, so the sums are identical).  Only warp barriers are
       involved. */
    {
        const int lane = tid & 31, wid = tid >> 5;
        const int i0 = tile.begin - 2 + (tid & ~31); /* bead of the warp's lane 0 */
        unsigned char* s_map = smem_raw + L.wmap + 32 * (size_t)wid;
        double* s_R = reinterpret_cast<double*>(smem_raw + L.wres) + 3 * 32 * (size_t)wid;
        unsigned char* s_Rf = smem_raw + L.wresf + 32 * (size_t)wid;
        double4* s_pos = reinterpret_cast<double4*>(smem_raw + L.pos) + (tid & ~31);
        if (active) s_pos[lane] = p;
        auto contact = [&](double4 a, double4 b, double& Rx, double& Ry, double& Rz) {
            return CONSTS != FN_CONST_NONE ? contact_force(N, A.pair0, a, b, Rx, Ry, Rz) : contact_eval(N, A.pairs, a, b, Rx, Ry, Rz);
        };
        /* direct phase: every lane first evaluates the leading KD items of its
           own list, one list row per iteration (coalesced loads, no window
           bookkeeping); the longer lists' tails then go through the windows.
           KD is picked per warp among mean - 1 .. mean + 2 (mean rounded
           down) to minimise 2 x KD + 3 x windows, a window costing about 1.5
           direct iterations. */
        int kd;
        {
            const int m = __reduce_add_sync(0xffffffffu, nc) >> 5;
            kd = m;
            int best = 2 * m + 3 * ((__reduce_add_sync(0xffffffffu, max(nc - m, 0)) + 31) >> 5);
            for (int k = max(m - 1, 0); k <= m + 2; ++k) {
                if (k == m) continue;
                const int c = 2 * k + 3 * ((__reduce_add_sync(0xffffffffu, max(nc - k, 0)) + 31) >> 5);
                if (c < best) {
                    best = c;
                    kd = k;
                }
            }
        }
        const int nd = min(nc, kd);
        const int nr = nc - nd; /* items left for the windows */
        int off = nr;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, off, o);
            if (lane >= o) off += y;
        }
        const int total = __shfl_sync(0xffffffffu, off, 31);
        off -= nr; /* exclusive */
        /* owner lane and list index of the first window's items, loaded
           before the direct phase so their latency overlaps it */
        int b_first = 0, j_first = 0;
        if (total > 0) {
            const int lim = min(32, total);
            for (int w = off; w < min(off + nr, lim); ++w) s_map[w] = (unsigned char)lane;
            __syncwarp();
            b_first = lane < lim ? s_map[lane] : 0;
            const int ob = __shfl_sync(0xffffffffu, off - nd, b_first);
            if (lane < lim) j_first = A.list[(size_t)(lane - ob) * A.list_stride + (i0 + b_first)];
        }
        /* the next list index is loaded one item ahead, by every lane and
           without a condition (a bead's own column, rows up to the list's
           last): a conditional load is merged with the old value at once,
           which waits for it */
        const int* row = A.list + (active ? i : tile.begin);
        int jn = *row;
        for (int k = 0; k < kd; ++k) {
            const int j = jn;
            if (k + 1 < A.list_cap) row += A.list_stride;
            jn = *row;
            if (k < nd) {
                double Rx = 0.0, Ry = 0.0, Rz = 0.0;
                if (contact(p, A.pos_in[j], Rx, Ry, Rz)) {
                    Fx += Rx;
                    Fy += Ry;
                    Fz += Rz;
                }
            }
        }
        for (int base = 0; base < total; base += 32) {
            const int lim = min(base + 32, total);
            const int w = base + lane;
            int b = b_first, j = j_first;
            if (base > 0) {
                for (int q = max(off, base); q < min(off + nr, lim); ++q) s_map[q - base] = (unsigned char)lane;
                __syncwarp();
                b = w < lim ? s_map[lane] : 0;
                const int ob = __shfl_sync(0xffffffffu, off - nd, b); /* list row = w - ob */
                if (w < lim) j = A.list[(size_t)(w - ob) * A.list_stride + (i0 + b)];
            }
            if (w < lim) {
                double Rx = 0.0, Ry = 0.0, Rz = 0.0;
                const int acts = contact(s_pos[b], A.pos_in[j], Rx, Ry, Rz);
                s_R[3 * lane] = Rx;
                s_R[3 * lane + 1] = Ry;
                s_R[3 * lane + 2] = Rz;
                s_Rf[lane] = (unsigned char)acts;
            }
            __syncwarp();
            for (int q = max(off, base); q < min(off + nr, lim); ++q) {
                if (s_Rf[q - base]) {
                    Fx += s_R[3 * (q - base)];
                    Fy += s_R[3 * (q - base) + 1];
                    Fz += s_R[3 * (q - base) + 2];
                }
            }
            __syncwarp();
        }
    }
    if (!active) return;
    if (FORCES_ONLY) {
        A.force[i] = make_float4((float)Fx, (float)Fy, (float)Fz, 0.0f);
        return;
    }
    let_next_start();
    const KickState state = kick_state(A, i); /* before the finiteness test, as in finish_bead */
    kick_drift<DAMP>(A, N, i, p, Fx, Fy, Fz, state, (flags & FN_STEP_DRIFT) != 0, DAMP || (flags & FN_STEP_STORE_V));
}

/* The chain step for small contexts, five warps per 28 beads at most: one warp
   evaluates the bonds (thread t for bead begin - 2 + t, as in k_step_chain)
   while four others evaluate the contacts, four lanes per bead and
   kWideItems contacts at a time into shared memory; then the first warp adds
   them to its beads' forces in list order and moves the beads.  The terms and
   their order are k_step_chain's, so the bits are.
   A bead's step is then a few dependent loads and one or two contacts deep
   instead of as many as its warp's longest list, and the bonds' chain of roots
   and the arc cosine runs beside it: small networks wait for those chains (10k
   beads 9.6 -> 4.3 us per step). */
constexpr int kWideBeads = 28, kWideItems = 16, kWideThreads = 160;

/* A barrier of the block's five warps, reached from the code of either role;
   true when `p` is on any thread. */
__device__ __forceinline__ bool wide_barrier_or(bool p) {
    int any;
    asm volatile(
        "{\n .reg .pred a, b;\n setp.ne.s32 a, %1, 0;\n barrier.cta.red.or.pred b, 1, %2, a;\n selp.s32 %0, 1, 0, b;\n}"
        : "=r"(any)
        : "r"((int)p), "n"(kWideThreads)
        : "memory");
    return any != 0;
}
__device__ __forceinline__ void wide_barrier() {
    asm volatile("barrier.cta.sync 2, %0;" ::"n"(kWideThreads) : "memory");
}

template <bool DAMP, int CONSTS>
__global__ void __launch_bounds__(kWideThreads, 6) k_step_wide(const __grid_constant__ StepArgs A, int flags, int parts,
                                                               int width) {
    __shared__ double s_img[3 * 32], s_spf[3 * 33], s_ang[6 * 33];
    __shared__ double2 s_len[32];
    __shared__ double s_R[kWideBeads * (3 * kWideItems + 1)];
    __shared__ unsigned char s_Rf[kWideBeads * kWideItems], s_ok[32];
    const FnTile tile = A.tiles[blockIdx.x / parts];
    const int begin = tile.begin + (blockIdx.x % parts) * width;
    const int n = min(tile.end - begin, width); /* may be <= 0: nothing to do */
    const int tid = threadIdx.x;
    __shared__ FnNet s_net;
    if (CONSTS != FN_CONST_ALL) {
        copy_net(A.nets + tile.net, &s_net);
        __syncthreads();
    }
    const FnNet& N = CONSTS == FN_CONST_ALL ? A.net0 : s_net;
    await_previous();
    if (tid >= 32) {
        const int b = (tid - 32) >> 2, g = tid & 3;
        const int i = begin + b;
        int nc = 0;
        double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
        if (b < n) {
            nc = min(A.list_count[i], A.list_cap);
            p = A.pos_in[i];
        }
        double* R = s_R + b * (3 * kWideItems + 1);
        unsigned char* Rf = s_Rf + b * kWideItems;
        for (int k0 = 0;; k0 += kWideItems) {
            const int k1 = min(nc, k0 + kWideItems);
            /* two items at a time, their loads together */
            for (int k = k0 + g; k < k1; k += 8) {
                const int* row = A.list + (size_t)k * A.list_stride + i;
                const bool two = k + 4 < k1;
                const int j0 = row[0];
                const int j1 = two ? row[4 * (size_t)A.list_stride] : j0;
                const double4 q0 = A.pos_in[j0], q1 = A.pos_in[j1];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h == 1 && !two) break;
                    const double4 q = h == 0 ? q0 : q1;
                    double Rx = 0.0, Ry = 0.0, Rz = 0.0;
                    const int acts = CONSTS != FN_CONST_NONE ? contact_force(N, A.pair0, p, q, Rx, Ry, Rz)
                                             : contact_eval(N, A.pairs, p, q, Rx, Ry, Rz);
                    const int at = k - k0 + 4 * h;
                    R[3 * at] = Rx;
                    R[3 * at + 1] = Ry;
                    R[3 * at + 2] = Rz;
                    Rf[at] = (unsigned char)acts;
                }
            }
            if (!wide_barrier_or(nc > k0 + kWideItems)) break;
            wide_barrier(); /* added: the next items may overwrite them */
        }
        return;
    }

    const int i = begin - 2 + tid; /* this thread's bead */
    const bool active = tid >= 2 && tid < n + 2;
    unsigned fl = 0, st0 = 0;
    double x = 0.0, y = 0.0, z = 0.0;
    float4 sp = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 an = make_float2(0.f, 0.f);
    KickState state{};
    double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
    int nc = 0;
    if (tid < n + 4 && i >= 0 && i < A.nb) {
        state.im = A.img_in[i];
        x = state.im.x;
        y = state.im.y;
        z = state.im.z;
        fl = A.ch_flags[i];
        st0 = A.ch_status[i];
        sp = A.ch_sp[i];
        an = A.ch_an[i];
        if (active) {
            nc = min(A.list_count[i], A.list_cap);
            p = A.pos_in[i];
        }
    }
    s_img[3 * tid] = x;
    s_img[3 * tid + 1] = y;
    s_img[3 * tid + 2] = z;
    __syncwarp();
    double l = 0.0, il = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    unsigned st = st0;
    if (tid < n + 3) {
        x -= s_img[3 * tid + 3];
        y -= s_img[3 * tid + 4];
        z -= s_img[3 * tid + 5];
        chain_spring(fl, st0, sp, true, x, y, z, l, il, gx, gy, gz, st);
        s_len[tid] = make_double2(l, il);
    }
    s_spf[3 * tid] = gx;
    s_spf[3 * tid + 1] = gy;
    s_spf[3 * tid + 2] = gz;
    s_ok[tid] = (unsigned char)((fl & FN_CH_SPRING) && (st & 1));
    __syncwarp();
    double cx = 0.0, cy = 0.0, cz = 0.0;
    {
        double pax = 0.0, pay = 0.0, paz = 0.0, pcx = 0.0, pcy = 0.0, pcz = 0.0;
        if (tid >= 1 && tid < n + 3 && (fl & FN_CH_ANGLE) && (st0 & 2)) {
            if ((fl & FN_CH_AN_FL) && !(s_ok[tid - 1] && s_ok[tid])) {
                st &= ~2u; /* kernel.cl:278-284 */
            } else {
                const double* q = s_img + 3 * tid;
                const double2 lp = s_len[tid - 1];
                angle_arms(q[-3] - q[0], q[-2] - q[1], q[-1] - q[2], x, y, z, lp.x, lp.y, l, il, an, pax, pay, paz,
                           pcx, pcy, pcz);
                cx = -pax - pcx;
                cy = -pay - pcy;
                cz = -paz - pcz;
            }
        }
        double* o = s_ang + 6 * tid;
        o[0] = pax;
        o[1] = pay;
        o[2] = paz;
        o[3] = pcx;
        o[4] = pcy;
        o[5] = pcz;
    }
    __syncwarp();
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    if (active) {
        state.fo = A.force[i];
        state.vo = A.vold[i];
        base_force<DAMP>(A, N, i, p, Fx, Fy, Fz);
        chain_gather(s_spf + 3 * tid, s_ang + 6 * tid, cx, cy, cz, Fx, Fy, Fz);
    }
    const double* R = s_R + (tid - 2) * (3 * kWideItems + 1);
    const unsigned char* Rf = s_Rf + (tid - 2) * kWideItems;
    for (int k0 = 0;; k0 += kWideItems) {
        const bool more = wide_barrier_or(false);
        const int m = min(nc - k0, kWideItems);
        for (int k = 0; k < m; ++k)
            if (Rf[k]) {
                Fx += R[3 * k];
                Fy += R[3 * k + 1];
                Fz += R[3 * k + 2];
            }
        if (!more) break;
        wide_barrier();
    }
    let_next_start();
    if (!active) return;
    if (st != st0) A.ch_status[i] = (unsigned char)st;
    kick_drift<DAMP>(A, N, i, p, Fx, Fy, Fz, state, (flags & FN_STEP_DRIFT) != 0, DAMP || (flags & FN_STEP_STORE_V));
}

/* ------------------------------------------------------------------------ */
/* Staged chain step kernel                                                  */

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

/* mbarrier + bulk-copy (TMA, non-tensor) primitives for one CTA */
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
/* Waits for phase `parity` of the barrier for at most ~2 s of SM clock;
   false when the wait ran out. */
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > 4000000000LL) return false;
    return true;
}
/* bytes (a multiple of 16) from global src to shared dst, both 16-byte
   aligned, completing on the barrier */
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
/* 16 bytes global -> shared through L2 (LDGSTS) */
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_all;" ::: "memory");
}

/* Issues the partner-position copies of contact items [c0, c0 + nch) of the
   tile: item q's partner j (tile-compacted list) -> pj slot q - c0.  The
   entries are loaded first, all at once, so their latency is paid once. */
__device__ __forceinline__ void gather_partners(const StepArgs& A, const int* __restrict__ ent, int c0,
                                                int nch, unsigned char* s_pj) {
    int j[kStagedMaxItemsPerThread];
#pragma unroll
    for (int k = 0; k < kStagedMaxItemsPerThread; ++k) {
        const int q = (int)threadIdx.x + k * (int)blockDim.x;
        j[k] = q < nch ? ent[c0 + q] : -1;
    }
#pragma unroll
    for (int k = 0; k < kStagedMaxItemsPerThread; ++k) {
        const int q = (int)threadIdx.x + k * (int)blockDim.x;
        if ((unsigned)j[k] < (unsigned)A.nb) {
            const double4* src = A.pos_in + j[k];
            const uint32_t dst = smem_addr(s_pj + 32 * (size_t)q);
            cp_async16(dst, src);
            cp_async16(dst + 16, reinterpret_cast<const char*>(src) + 16);
        }
    }
}

/* The chain step (same arithmetic and summation order as k_step_chain, so
   the same bits) with the tile's data staged in shared memory before any of
   it is used, instead of a chain of dependent loads:
     - one thread issues bulk copies (cp.async.bulk, completing on an
       mbarrier) of the image positions (with a two-bead halo each side),
       positions, forces, velocities_old and spring records of the tile;
     - meanwhile every thread loads the tile's contact entries (a contiguous
       run of the tile-compacted list) and copies each partner's position
       into shared memory (cp.async), and the byte-sized flags, statuses,
       angle records and list lengths with plain loads;
     - then springs and angles are evaluated once per tile, every contact
       item is evaluated by some thread of the block (items spread evenly over
       the threads, results kept per item), and each thread sums its bead's
       terms in the fixed order: base, previous and next spring, angles
       centred on j-1, j, j+1, contacts in list order.
   Tiles with more contact items than `chunk` take them in rounds. */
template <bool DAMP, bool DRIFT, bool STORE_V>
__global__ void __launch_bounds__(kChainMaxBlock) k_step_staged(const StepArgs A) {
    await_previous();
    extern __shared__ __align__(128) unsigned char sm[];
    const StagedSmem L = staged_smem_layout(blockDim.x, A.chunk);
    const FnTile tile = A.tiles[blockIdx.x];
    const int items = A.tile_items[blockIdx.x];
    const int b0 = tile.begin, n = tile.end - tile.begin;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int* __restrict__ ent = A.csr + (size_t)blockIdx.x * (size_t)A.csr_region;
    const uint32_t bar = smem_addr(sm + L.bar);
    const int j0 = max(b0 - 2, 0), j1 = min(b0 + n + 2, A.nb), js1 = min(b0 + n + 1, A.nb);
    double* s_spf = reinterpret_cast<double*>(sm + L.spf);
    double* s_ang = reinterpret_cast<double*>(sm + L.ang);
    const double4* s_img = reinterpret_cast<const double4*>(sm + L.img);
    const double4* s_pos = reinterpret_cast<const double4*>(sm + L.pos);
    const float4* s_frc = reinterpret_cast<const float4*>(sm + L.frc);
    const float4* s_vold = reinterpret_cast<const float4*>(sm + L.vold);
    const float4* s_chsp = reinterpret_cast<const float4*>(sm + L.chsp);
    float2* s_chan = reinterpret_cast<float2*>(sm + L.chan);
    unsigned char* s_pj = sm + L.pj;
    int* s_off = reinterpret_cast<int*>(sm + L.off);
    int* s_ws = reinterpret_cast<int*>(sm + L.ws);
    unsigned char* s_owner = sm + L.owner;
    unsigned char* s_flag = sm + L.flag;
    unsigned char* s_stat = sm + L.stat;
    unsigned char* s_tsp = sm + L.tsp;
    unsigned char* s_tan = sm + L.tan;

    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0) {
        const uint32_t bytes = 32u * (uint32_t)(j1 - j0) + 32u * (uint32_t)n + 32u * (uint32_t)n +
                               16u * (uint32_t)(js1 - j0);
        mbar_expect_tx(bar, bytes);
        bulk_g2s(smem_addr(sm + L.img) + 32u * (uint32_t)(j0 - (b0 - 2)), A.img_in + j0, 32u * (j1 - j0), bar);
        bulk_g2s(smem_addr(sm + L.pos), A.pos_in + b0, 32u * n, bar);
        bulk_g2s(smem_addr(sm + L.frc), A.force + b0, 16u * n, bar);
        bulk_g2s(smem_addr(sm + L.vold), A.vold + b0, 16u * n, bar);
        bulk_g2s(smem_addr(sm + L.chsp) + 16u * (uint32_t)(j0 - (b0 - 2)), A.ch_sp + j0, 16u * (js1 - j0), bar);
    }
    /* the first round's contact partners, while the bulk copies run */
    const int nch0 = min(items, A.chunk);
    gather_partners(A, ent, 0, nch0, s_pj);
    /* byte-sized and 8-byte arrays, list length */
    const bool active = tid < n;
    const int i = b0 + tid;
    int nc = 0;
    if (active) {
        nc = A.list_count[i];
        if (nc > A.list_cap) nc = A.list_cap;
    }
    for (int u = tid; u < n + 4; u += nt) {
        const int j = b0 - 2 + u;
        unsigned char fl = 0, st = 0;
        if (j >= 0 && j < A.nb) {
            fl = A.ch_flags[j];
            st = A.ch_status[j];
        }
        s_flag[u] = fl;
        s_stat[u] = st;
        if (u < n + 2) {
            const int ja = b0 - 1 + u;
            s_chan[u] = (ja >= 0 && ja < A.nb) ? A.ch_an[ja] : make_float2(0.f, 0.f);
        }
    }
    /* each bead's first contact item and the item -> bead map of round 0 */
    int total;
    const int off = block_scan_any(nc, s_ws, total);
    if (tid < n) s_off[tid] = off;
    for (int q = off; q < min(off + nc, nch0); ++q) s_owner[q] = (unsigned char)tid;

    cp_async_wait_all();
    bool ok = mbar_wait_bounded(bar, 0);
    ok = __syncthreads_and(ok);
    if (!ok) {
        /* the staged data never arrived: skip the tile, counted for fn_sync */
        if (tid == 0) {
            atomicAdd(A.counters + FN_CNT_STALL, 1ull);
            mbar_wait_bounded(bar, 0);
        }
        __syncthreads();
        return;
    }

    /* springs: lower bead b0 - 2 + u, u < n + 3 */
    for (int u = tid; u < n + 3; u += nt) {
        const unsigned fl = s_flag[u];
        unsigned char tf = 0;
        if (fl & FN_CH_SPRING) {
            const int alive0 = s_stat[u] & 1;
            tf = (unsigned char)(alive0 << 2);
            if (alive0 && !(fl & FN_CH_SP_INERT)) {
                const double4 a = s_img[(fl & FN_CH_SP_REV) ? u + 1 : u];
                const double4 b = s_img[(fl & FN_CH_SP_REV) ? u : u + 1];
                double fx = 0.0, fy = 0.0, fz = 0.0;
                int broke;
                const int acts = spring_pts(a.x, a.y, a.z, b.x, b.y, b.z, s_chsp[u], (fl & FN_CH_SP_FL) ? 1 : 0,
                                            fx, fy, fz, broke);
                s_spf[3 * u] = fx;
                s_spf[3 * u + 1] = fy;
                s_spf[3 * u + 2] = fz;
                tf |= (unsigned char)(acts | (broke << 1));
            }
        }
        s_tsp[u] = tf;
    }
    __syncthreads();
    /* angles: centre b0 - 1 + u, u < n + 2 */
    for (int u = tid; u < n + 2; u += nt) {
        const unsigned fl = s_flag[u + 1];
        int alive = (fl & FN_CH_ANGLE) && (s_stat[u + 1] & 2);
        if (alive && (fl & FN_CH_AN_FL)) {
            const unsigned f1 = s_tsp[u], f2 = s_tsp[u + 1];
            if (!((f1 & 4) && !(f1 & 2)) || !((f2 & 4) && !(f2 & 2))) alive = 0;
        }
        s_tan[u] = (unsigned char)alive;
        if (alive) {
            const double4 t1 = s_img[(fl & FN_CH_AN_REV) ? u + 2 : u];
            const double4 t2 = s_img[u + 1];
            const double4 t3 = s_img[(fl & FN_CH_AN_REV) ? u : u + 2];
            double* o = s_ang + 6 * u;
            angle_pts(t1.x, t1.y, t1.z, t2.x, t2.y, t2.z, t3.x, t3.y, t3.z, s_chan[u], o[0], o[1], o[2], o[3],
                      o[4], o[5]);
        }
    }
    __syncthreads();

    const FnNet& N = A.nets[tile.net];
    double4 p = make_double4(0.0, 0.0, 0.0, 0.0);
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    if (active) {
        p = s_pos[tid];
        base_force<DAMP>(A, N, i, p, Fx, Fy, Fz);
        const unsigned fp = s_flag[tid + 1];
        if ((fp & FN_CH_SPRING) && (s_tsp[tid + 1] & 1)) {
            const double* f = s_spf + 3 * (tid + 1);
            if (fp & FN_CH_SP_REV) {
                Fx += f[0];
                Fy += f[1];
                Fz += f[2];
            } else {
                Fx += f[0] * -1.0;
                Fy += f[1] * -1.0;
                Fz += f[2] * -1.0;
            }
        }
        const unsigned fn = s_flag[tid + 2];
        if ((fn & FN_CH_SPRING) && (s_tsp[tid + 2] & 1)) {
            const double* f = s_spf + 3 * (tid + 2);
            if (fn & FN_CH_SP_REV) {
                Fx += f[0] * -1.0;
                Fy += f[1] * -1.0;
                Fz += f[2] * -1.0;
            } else {
                Fx += f[0];
                Fy += f[1];
                Fz += f[2];
            }
        }
        if (s_tan[tid]) {
            const double* o = s_ang + 6 * tid;
            const int k = (s_flag[tid + 1] & FN_CH_AN_REV) ? 0 : 3;
            Fx += o[k];
            Fy += o[k + 1];
            Fz += o[k + 2];
        }
        if (s_tan[tid + 1]) {
            const double* o = s_ang + 6 * (tid + 1);
            Fx += -o[0] - o[3];
            Fy += -o[1] - o[4];
            Fz += -o[2] - o[5];
        }
        if (s_tan[tid + 2]) {
            const double* o = s_ang + 6 * (tid + 2);
            const int k = (s_flag[tid + 3] & FN_CH_AN_REV) ? 3 : 0;
            Fx += o[k];
            Fy += o[k + 1];
            Fz += o[k + 2];
        }
    }

    /* contacts, in rounds of at most `chunk` items */
    for (int c0 = 0; c0 < items; c0 += A.chunk) {
        const int nch = min(items - c0, A.chunk);
        if (c0 > 0) {
            __syncthreads(); /* the previous round's results are summed */
            gather_partners(A, ent, c0, nch, s_pj);
            for (int q = max(off, c0); q < min(off + nc, c0 + nch); ++q) s_owner[q - c0] = (unsigned char)tid;
            cp_async_wait_all();
            __syncthreads();
        }
        for (int q = tid; q < nch; q += nt) {
            const int t = min((int)s_owner[q], n - 1);
            double4* slot = reinterpret_cast<double4*>(s_pj + 32 * (size_t)q);
            const double4 pj = *slot;
            double Rx = 0.0, Ry = 0.0, Rz = 0.0;
            const int acts = contact_eval(N, A.pairs, s_pos[t], pj, Rx, Ry, Rz);
            *slot = make_double4(Rx, Ry, Rz, acts ? 1.0 : 0.0);
        }
        __syncthreads();
        if (active) {
            for (int q = max(off, c0); q < min(off + nc, c0 + nch); ++q) {
                const double4 r = *reinterpret_cast<const double4*>(s_pj + 32 * (size_t)(q - c0));
                if (r.w != 0.0) {
                    Fx += r.x;
                    Fy += r.y;
                    Fz += r.z;
                }
            }
        }
    }
    if (!active) return;

    /* statuses after this step (kernel.cl:396-397, 278-284) */
    const unsigned st0 = s_stat[tid + 2];
    unsigned st = st0;
    if ((s_tsp[tid + 2] & 2)) st &= ~1u;
    if ((st0 & 2) && (s_flag[tid + 2] & FN_CH_ANGLE) && !s_tan[tid + 1]) st &= ~2u;
    if (st != st0) A.ch_status[i] = (unsigned char)st;

    /* AdvanceVelocity (kernel.cl:451-462) and the next AdvancePosition */
    const float fx = (float)Fx, fy = (float)Fy, fz = (float)Fz;
    if (!(isfinite(fx) && isfinite(fy) && isfinite(fz))) atomicAdd(A.counters + FN_CNT_NONFINITE, 1ull);
    double4 im = s_img[tid + 2];
    const double minv = im.w;
    const double half_dt = N.half_dt * minv;
    const float4 fo = s_frc[tid];
    const float4 vo = s_vold[tid];
    double tx = (double)fx, ty = (double)fy, tz = (double)fz;
    tx += (double)fo.x;
    ty += (double)fo.y;
    tz += (double)fo.z;
    const float vox = (float)(tx * half_dt + (double)vo.x);
    const float voy = (float)(ty * half_dt + (double)vo.y);
    const float voz = (float)(tz * half_dt + (double)vo.z);
    A.force[i] = make_float4(fx, fy, fz, 0.0f);
    A.vold[i] = make_float4(vox, voy, voz, 0.0f);
    if (DRIFT) {
        float4 v;
        drift(N, minv, fx, fy, fz, vox, voy, voz, p, im, v);
        A.pos_out[i] = p;
        A.img_out[i] = im;
        if (DAMP || STORE_V) A.vel[i] = v;
    }
}

template <bool STORE_V>
__global__ void __launch_bounds__(512) k_drift(const StepArgs A) {
    await_previous();
    let_next_start();
    const FnTile t = A.tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    if (i >= t.end) return;
    const FnNet& N = A.nets[t.net];
    double4 p = A.pos_in[i];
    double4 im = A.img_in[i];
    const float4 f = A.force[i];
    const float4 vo = A.vold[i];
    float4 v;
    drift(N, im.w, f.x, f.y, f.z, vo.x, vo.y, vo.z, p, im, v);
    A.pos_out[i] = p;
    A.img_out[i] = im;
    if (STORE_V) A.vel[i] = v;
}

/* Forces alone (no base, no kick, no drift), selected terms; for the
   one-step force parity checks.  Writes force and the bond statuses. */
__global__ void k_forces_only(const StepArgs A, int terms) {
    const FnTile t = A.tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    if (i >= t.end) return;
    const FnNet& N = A.nets[t.net];
    const double4 p = A.pos_in[i];
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    if (terms & 1) {
        for (int e = A.sp_off[i]; e < A.sp_off[i + 1]; ++e) {
            const int ent = A.sp_ent[e];
            double fx, fy, fz;
            int broke;
            if (spring_eval(A, ent >> 1, fx, fy, fz, broke)) {
                const double sg = (ent & 1) ? -1.0 : 1.0;
                Fx += fx * sg;
                Fy += fy * sg;
                Fz += fz * sg;
            }
        }
    }
    if (terms & 2) {
        for (int e = A.an_off[i]; e < A.an_off[i + 1]; ++e) {
            const int ent = A.an_ent[e];
            const int a = ent >> 2, role = ent & 3;
            if (A.an_status[a] != 1) continue;
            const int4 b = A.an_b[a];
            if (b.w == 1) {
                const int2 ss = A.an_s[a];
                if (!spring_alive_after(A, ss.x) || !spring_alive_after(A, ss.y)) continue;
            }
            double pax, pay, paz, pcx, pcy, pcz;
            angle_eval(A, b, A.an_par[a], pax, pay, paz, pcx, pcy, pcz);
            if (role == 0) {
                Fx += pax; Fy += pay; Fz += paz;
            } else if (role == 2) {
                Fx += pcx; Fy += pcy; Fz += pcz;
            } else {
                Fx += -pax - pcx; Fy += -pay - pcy; Fz += -paz - pcz;
            }
        }
    }
    if (terms & 4) {
        int n = A.list_count[i];
        if (n > A.list_cap) n = A.list_cap;
        for (int k = 0; k < n; ++k) {
            const int j = A.list[(size_t)k * A.list_stride + i];
            double Rx, Ry, Rz;
            if (contact_eval(N, A.pairs, p, A.pos_in[j], Rx, Ry, Rz)) {
                Fx += Rx; Fy += Ry; Fz += Rz;
            }
        }
    }
    A.force[i] = make_float4((float)Fx, (float)Fy, (float)Fz, 0.0f);
}

/* ResetBeadEnergy, kernel.cl:468-483. */
__global__ void k_reset_energy(float4* force, float4* vel, float4* vold, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    force[i] = z;
    vel[i] = z;
    vold[i] = z;
}

/* ------------------------------------------------------------------------ */
/* Contact-list rebuild                                                      */

/* Displacement-triggered mode: every rebuild kernel returns at once unless
   the device gate says a rebuild is due (a null gate always rebuilds). */
#define FN_GATED(g)                   \
    if ((g) != nullptr && *(g) == 0) \
    return

__global__ void k_fill_int(int* p, long long n, int v, const int* gate) {
    await_previous();
    let_next_start();
    FN_GATED(gate);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        p[i] = v;
}

/* FillGrid's cell computation (kernel.cl:492-501) + per-cell counting. */
__global__ void k_cells(const RebuildArgs R) {
    await_previous();
    let_next_start();
    FN_GATED(R.gate);
    const FnTile t = R.tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    if (i >= t.end) return;
    const FnNet& N = R.nets[t.net];
    const double4 p = R.pos[i];
    const double qx = floor(p.x / N.step[0]);
    const double qy = floor(p.y / N.step[1]);
    const double qz = floor(p.z / N.step[2]);
    int cell = -1;
    if (qx >= 0.0 && qx < (double)N.nx && qy >= 0.0 && qy < (double)N.ny && qz >= 0.0 &&
        qz < (double)N.nz) {
        cell = N.cell_base + (int)qx + (int)qy * N.nx + (int)qz * N.nxy;
        atomicAdd(R.cell_count + cell, 1);
    }
    R.cell_of[i] = cell;
    R.list_count[i] = 0; /* k_lists counts only the beads it lists */
    if (R.ref) R.ref[i] = R.img[i];
}

/* FillGrid's slot of each bead in its cell: the bead as the list build's first
   test reads it, 16 bytes with its position rounded to FP32 and its index. */
__global__ void k_scatter(const __grid_constant__ RebuildArgs R, int nb) {
    await_previous();
    let_next_start();
    FN_GATED(R.gate);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nb) return;
    const int c = R.cell_of[i];
    if (c < 0) return;
    const double4 p = R.pos[i];
    const int slot = atomicAdd(R.cell_fill + c, 1);
    R.cell_raw[R.cell_start[c] + slot] = make_float4((float)p.x, (float)p.y, (float)p.z, __int_as_float(i));
}

/* The first n <= W beads of a cell by index: Batcher's network for W = 4 or 8
   on (index, slot) keys in registers, absent slots last. */
template <int W>
__device__ __forceinline__ void cell_sort_small(const float4* raw, int n, int* b, float4* e) {
    constexpr int N4 = 5, N8 = 19;
    constexpr int net[N8][2] = {{0, 1}, {2, 3}, {0, 2}, {1, 3}, {1, 2}, {4, 5}, {6, 7}, {4, 6}, {5, 7}, {5, 6},
                                {0, 4}, {1, 5}, {2, 6}, {3, 7}, {2, 4}, {3, 5}, {1, 2}, {3, 4}, {5, 6}};
    unsigned long long v[W];
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] = k < n ? ((unsigned long long)__float_as_uint(raw[k].w) << 3) | k : ~0ull;
#pragma unroll
    for (int q = 0; q < (W == 4 ? N4 : N8); ++q) {
        const unsigned long long lo = min(v[net[q][0]], v[net[q][1]]);
        const unsigned long long hi = max(v[net[q][0]], v[net[q][1]]);
        v[net[q][0]] = lo;
        v[net[q][1]] = hi;
    }
#pragma unroll
    for (int k = 0; k < W; ++k)
        if (k < n) {
            b[k] = (int)(v[k] >> 3);
            e[k] = raw[v[k] & 7];
        }
}

/* One cell of n > 0 beads. */
__device__ __forceinline__ void cell_sort_one(const RebuildArgs& R, int c, int n) {
    const int start = R.cell_start[c];
    const float4* raw = R.cell_raw + start;
    int* b = R.cell_beads + start;
    float4* e = R.cell_pos + start;
    if (n == 1) {
        const float4 v = raw[0];
        b[0] = __float_as_int(v.w);
        e[0] = v;
        return;
    }
    if (n <= 4 && n <= R.cell_cap) {
        cell_sort_small<4>(raw, n, b, e);
        return;
    }
    if (n <= 8 && n <= R.cell_cap) {
        cell_sort_small<8>(raw, n, b, e);
        return;
    }
    /* selection of the first min(n, cap) positions: ascending order there,
       O(cap * n) even for an overfull cell */
    for (int k = 0; k < n; ++k) e[k] = raw[k];
    const int keep = n < R.cell_cap ? n : R.cell_cap;
    for (int k = 0; k < keep; ++k) {
        int best = k;
        for (int m = k + 1; m < n; ++m)
            if (__float_as_int(e[m].w) < __float_as_int(e[best].w)) best = m;
        const float4 v = e[best];
        e[best] = e[k];
        e[k] = v;
    }
    for (int k = 0; k < n; ++k) b[k] = __float_as_int(e[k].w);
    if (n > R.cell_cap) {
        for (int k = R.cell_cap; k < n; ++k) R.cell_of[b[k]] = -1;
        atomicAdd(R.counters + FN_CNT_CELL_OVERFLOW, (unsigned long long)(n - R.cell_cap));
    }
}

/* Orders each cell's beads by index (the order a one-thread FillGrid sweep
   would store them in) and drops the ones beyond the cell capacity, like the
   `old < GRID_TAIL_SIZE` test of kernel.cl:503.  One thread per cell: cells
   hold about one bead, and a warp's cells are one run of both arrays (counting
   each bead's rank with the bead's own thread reads its cell at random: 188 us
   against 52 on the 4M-bead mat). */
__global__ void k_cell_sort(const __grid_constant__ RebuildArgs R, int ncells) {
    await_previous();
    let_next_start();
    FN_GATED(R.gate);
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    const int n = R.cell_count[c];
    if (n > 0) cell_sort_one(R, c, n);
}

/* The same for grids of mostly empty cells: one thread per bead in the grid, of
   which the one at its cell's first place sorts the cell. */
__global__ void k_cell_sort_sparse(const __grid_constant__ RebuildArgs R, int nb, long long ncells) {
    await_previous();
    let_next_start();
    FN_GATED(R.gate);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb || t >= R.cell_start[ncells]) return;
    const int c = R.cell_of[__float_as_int(R.cell_raw[t].w)];
    /* -1: dropped by its overfull cell's first thread just now */
    if (c >= 0 && R.cell_start[c] == t) cell_sort_one(R, c, R.cell_count[c]);
}

/* BuildContactList's test (kernel.cl:574-586, 630-659) once the (minimum-
   image) squared distance is known: exclusion of bonded neighbours, then the
   listing radius of the pair kind (the cut-off, widened by the Verlet skin in
   displacement-triggered mode; radius + skin radius for hs pairs). */
__device__ __forceinline__ bool list_accept(const FnNet& N, int kind, double length, double4 pi, int4 bi, double4 pj,
                                            int4 bj) {
    if (bi.x == bj.x && abs(bi.y - bj.y) <= 1) return false;
    if (kind == 1 || kind == 3) return length < N.list_cut_sq;
    if (kind == 2 || kind == 4) {
        if (kind == 4 && length < N.list_cut_sq) return true;
        const double si = (double)__int_as_float(bi.w), sj = (double)__int_as_float(bj.w);
        const double ri = (double)w_radius(pi.w), rj = (double)w_radius(pj.w);
        const double min_skin = (si > sj) ? sj : si;
        const double max_radius = (ri > rj) ? ri : rj;
        const double lim = max_radius + min_skin;
        return length < lim * lim;
    }
    return false;
}

__device__ __forceinline__ bool list_accept(const FnNet& N, const FnPair* __restrict__ pairs,
                                            double length, double4 pi, int4 bi, double4 pj,
                                            int4 bj) {
    return list_accept(N, pairs[N.pair_base + getadress(bi.z, bj.z, N.types_num)].kind, length, pi, bi, pj, bj);
}

/* BuildContactList's test of the pair i, j in FP64. */
template <bool UNIFORM>
__device__ __forceinline__ bool list_pair(const RebuildArgs& R, const FnNet& N, double4 pi, int4 bi, double4 pj,
                                          int4 bj) {
    double rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
    double length = rx * rx + ry * ry + rz * rz;
    if (N.list_mi) length = min_image(N, rx, ry, rz, length, N.list_mi);
    if (!(length < N.list_r2_max)) return false;
    return UNIFORM ? list_accept(N, R.pair0.kind, length, pi, bi, pj, bj)
                   : list_accept(N, R.pairs, length, pi, bi, pj, bj);
}

/* The second test of a near candidate (its index, the sign set when the first
   test left its distance open): the exclusion of bonded neighbours, where the
   distance is open the test in FP64, and where its row is long enough to hold
   an overfull cell (crowded), that its cell has kept it. */
template <bool UNIFORM>
__device__ __forceinline__ bool list_second(const RebuildArgs& R, const FnNet& N, int i, int4 bi, int w, bool crowded,
                                            int& j) {
    j = w & 0x7fffffff;
    const int4 bj = R.binfo[j];
    if (crowded && R.cell_of[j] < 0) return false;
    if (bi.x == bj.x && abs(bi.y - bj.y) <= 1) return false;
    return w >= 0 || list_pair<UNIFORM>(R, N, R.pos[i], bi, R.pos[j], bj);
}

/* Network owning bead i (networks hold consecutive bead ranges). */
__device__ __forceinline__ int net_of_bead(const FnNet* __restrict__ nets, int n_nets, int i) {
    int lo = 0, hi = n_nets - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (nets[mid].bead_begin <= i)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

/* Candidates j of one run of consecutive beads in cell order. */
__device__ __forceinline__ void scan_run(const RebuildArgs& R, const FnNet& N, int i, double4 pi,
                                         int4 bi, const int* ids, int m, int* __restrict__ out,
                                         int& n) {
    for (int k = 0; k < m; ++k) {
        const int j = ids[k];
        if (j == i) continue;
        const double4 pj = R.pos[j];
        double rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
        double length = rx * rx + ry * ry + rz * rz;
        if (N.list_mi) length = min_image(N, rx, ry, rz, length, N.list_mi);
        if (!(length < N.list_r2_max)) continue; /* listed by no pair kind */
        if (list_accept(N, R.pairs, length, pi, bi, pj, R.binfo[j])) {
            if (n < R.list_cap) out[(size_t)n * R.list_stride] = j;
            ++n;
        }
    }
}

/* The place of global cell c in its network's grid. */
__device__ __forceinline__ void cell_coords(const FnNet& N, int c, int& cx, int& cy, int& cz) {
    const int lc = max(c - N.cell_base, 0);
    cz = (int)(__umulhi((unsigned)lc, N.div_nxy) >> N.shift_nxy);
    const int r = lc - cz * N.nxy;
    cy = (int)(__umulhi((unsigned)r, N.div_nx) >> N.shift_nx);
    cx = r - cy * N.nx;
}

__device__ __forceinline__ void list_one_bead(const RebuildArgs& R, const FnNet& N, int i, int c);

/* The longest run of three cells that the builds below take as one run of the
   sorted array: at twice the beads that three full cells keep, testing the
   dropped ones costs about as much as it saves to test in FP32. */
__device__ __forceinline__ int longest_run(int cell_cap) { return 6 * min(cell_cap, 1 << 28); }

/* Per axis the smaller of |d| and its distance from the box side (`side`,
   infinite where the axis is not periodic): no image of the pair is nearer. */
__device__ __forceinline__ float fold_axis(float d, float side) { return fminf(fabsf(d), fabsf(side - fabsf(d))); }
__device__ __forceinline__ float fold_side(const FnNet& N, int a) {
    return N.periodic >> a & 1 ? (float)N.box[a] : __int_as_float(0x7f800000);
}

/* A row's candidates: number k < end is entry (k < split ? a : b) + k; shift says
   how the bead moves for them, two bits per axis (1 down by the box, 2 up),
   bits 0-1 for the first part in x, 2-3 for the second, 4-5 y, 6-7 z. */
struct ListRow {
    int a, b, split, end;
};

/* The near candidates a group keeps between the tests. */
constexpr int kListNear = 32;

/* Full per-bead lists over the 27-cell neighbourhood (dz, dy, dx ascending,
   beads ascending within a cell): the symmetric closure of the reference's
   half-shell pair set, in a fixed order.  G lanes of a warp work on one bead;
   the groups walk the beads in cell order, so neighbouring groups share their
   candidates' cache lines.
     1. The nine (dz, dy) rows: three cells of a row are one run of the sorted
        bead array (two where the row wraps in x); the lanes load the rows'
        cell starts together and a scan over the group numbers the candidates.
     2. First test: the candidates, G at a time, from their FP32 positions
        (16 bytes with the index); the near ones are kept in order by a ballot
        over the group.
     3. Second test: the near ones, G at a time, in FP64 with the pair law's
        radius and the exclusion of bonded neighbours; the accepted ones are
        written in order by a ballot over the group.
   A row with more beads than one cell may keep can hold an overfull cell; its
   dropped beads, the last of their cell, fail the second test (whole rebuild,
   100k beads at 22 per cell: 377 us, 788 when such rows took the FP64 test
   candidate by candidate).  Beads next to a cell far over its capacity
   (longest_run) are listed cell by cell, the kept beads G at a time, in FP64.
   A bead's loads are then a handful of dependent rounds instead of one per
   candidate, which is what small networks wait for. */
template <int G, bool UNIFORM>
__global__ void __launch_bounds__(128, 10) k_lists_group(const __grid_constant__ RebuildArgs R, long long ncells) {
    await_previous();
    FN_GATED(R.gate);
    constexpr int PER = 128 / G, J = (9 + G - 1) / G;
    __shared__ ListRow s_row[9 * PER];
    __shared__ unsigned char s_shift[9 * PER];
    __shared__ int s_near[kListNear * PER];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, gl = threadIdx.x % G, grp = threadIdx.x / G;
    const int t = blockIdx.x * PER + grp;
    int i = -1, c = 0;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < R.cell_start[ncells]) { /* beads placed in the grid */
        o = R.cell_pos[t];
        i = __float_as_int(o.w);
        c = R.cell_of[i];
        if (c < 0) i = -1; /* beyond its cell's capacity: listed nowhere */
    }
    const FnNet& N = UNIFORM ? R.net0 : R.nets[i >= 0 ? net_of_bead(R.nets, R.n_nets, i) : 0];
    const float r2 = N.list_out_r2;
    const bool fold = N.list_fold;
    int widest = 0; /* beads of the fullest run */
    ListRow* rows = s_row + 9 * grp;
    unsigned char* shifts = s_shift + 9 * grp;
    int* near = s_near + kListNear * grp;
    int total = 0;
    bool moved = false; /* some row lies beyond a periodic side */
    {
        int cx, cy, cz;
        cell_coords(N, c, cx, cy, cz);
        const int xa = max(cx - 1, 0), xb = min(cx + 2, N.nx);
        const bool wl = cx == 0 && (N.periodic & 1), wr = cx + 1 == N.nx && (N.periodic & 1);
#pragma unroll
        for (int q = 0; q < J; ++q) {
            const int k = q * G + gl;
            int a0 = 0, na = 0, b0 = 0, nb = 0, shift = 0;
            if (k < 9 && i >= 0) {
                int z = cz + k / 3 - 1, y = cy + k % 3 - 1;
                bool ok = true;
                /* a cell below the grid lies at the far side: the bead moves up */
                if (z < 0 || z >= N.nz) {
                    ok = N.periodic & 4;
                    shift |= z < 0 ? 128 : 64;
                    z = z < 0 ? N.nz - 1 : 0;
                }
                if (y < 0 || y >= N.ny) {
                    ok = ok && (N.periodic & 2);
                    shift |= y < 0 ? 32 : 16;
                    y = y < 0 ? N.ny - 1 : 0;
                }
                if (ok) {
                    const int* row = R.cell_start + (N.cell_base + y * N.nx + z * N.nxy);
                    a0 = row[xa];
                    na = row[xb] - a0;
                    if (wl) { /* the cell beyond the side comes first */
                        b0 = a0;
                        nb = na;
                        a0 = row[N.nx - 1];
                        na = row[N.nx] - a0;
                        shift |= 2;
                    } else if (wr) {
                        b0 = row[0];
                        nb = row[1] - b0;
                        shift |= 4;
                    }
                    widest = max(widest, max(na, nb));
                }
            }
            /* number the candidates: inclusive scan over the group's lanes */
            int e = na + nb;
#pragma unroll
            for (int d = 1; d < G; d <<= 1) {
                const int v = __shfl_up_sync(full, e, d, G);
                if (gl >= d) e += v;
            }
            const int first = total + e - na - nb;
            if (k < 9) {
                rows[k] = ListRow{a0 - first, b0 - first - na, first + na, first + na + nb};
                shifts[k] = (unsigned char)shift;
            }
            moved |= shift != 0;
            total += __shfl_sync(full, e, G - 1, G);
        }
    }
    const unsigned gmask = G == 32 ? full : (((1u << G) - 1u) << (lane & ~(G - 1)));
    const unsigned below = (1u << lane) - 1u;
    const bool plain = (__ballot_sync(full, widest > longest_run(R.cell_cap)) & gmask) != 0;
    const bool crowded = __any_sync(full, widest > R.cell_cap);
    moved = __any_sync(full, moved || fold);
    if (plain || i < 0) total = 0;
    __syncwarp();
    int4 bi = make_int4(0, 0, 0, 0);
    if (total > 0 || plain) bi = R.binfo[i];
    const float in_r2 = N.list_in_r2;
    int* __restrict__ out = R.list + (i >= 0 ? i : 0);
    int n = 0, m = 0;
    /* writes the accepted candidates of the group's lanes, in order */
    auto add = [&](bool acc, int j) {
        const unsigned mine = __ballot_sync(full, acc) & gmask;
        if (acc) {
            const int at = n + __popc(mine & below);
            if (at < R.list_cap) out[(size_t)at * R.list_stride] = j;
        }
        n += __popc(mine);
    };
    /* second test of the m near candidates */
    auto flush = [&]() {
        __syncwarp();
        const int most = __reduce_max_sync(full, m);
        for (int k0 = 0; k0 < most; k0 += G) {
            const int k = k0 + gl;
            bool acc = false;
            int j = -1;
            if (k < m) acc = list_second<UNIFORM>(R, N, i, bi, near[k], crowded, j);
            add(acc, j);
        }
        m = 0;
        __syncwarp();
    };
    const int most = __reduce_max_sync(full, total);
    ListRow u = rows[0];
    int r = 0;
    for (int k0 = 0; k0 < most; k0 += G) {
        const int k = k0 + gl;
        bool hit = false;
        int j = -1;
        if (k < total) {
            while (k >= u.end) u = rows[++r];
            const float4 e = R.cell_pos[(k < u.split ? u.a : u.b) + k];
            j = __float_as_int(e.w);
            float dx = o.x - e.x, dy = o.y - e.y, dz = o.z - e.z;
            if (moved) {
                if (fold) {
                    dx = fold_axis(dx, fold_side(N, 0));
                    dy = fold_axis(dy, fold_side(N, 1));
                    dz = fold_axis(dz, fold_side(N, 2));
                } else {
                    const int sh = shifts[r], sx = k < u.split ? sh : sh >> 2;
                    const float bx = (float)N.box[0], by = (float)N.box[1], bz = (float)N.box[2];
                    dx += sx & 1 ? -bx : sx & 2 ? bx : 0.0f;
                    dy += sh & 16 ? -by : sh & 32 ? by : 0.0f;
                    dz += sh & 64 ? -bz : sh & 128 ? bz : 0.0f;
                }
            }
            const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
            hit = !(d2 > r2) && j != i;
            if (!(d2 <= in_r2)) j |= (int)0x80000000;
        }
        const unsigned mine = __ballot_sync(full, hit) & gmask;
        if (hit) near[m + __popc(mine & below)] = j;
        m += __popc(mine);
        if (__any_sync(full, m > kListNear - G)) flush();
    }
    flush();
    if (__any_sync(full, plain)) {
        double4 pi = make_double4(0.0, 0.0, 0.0, 0.0);
        if (plain) pi = R.pos[i];
        int cx, cy, cz;
        cell_coords(N, c, cx, cy, cz);
        for (int d = 0; d < 27; ++d) {
            int z = cz + d / 9 - 1, y = cy + d / 3 % 3 - 1, x = cx + d % 3 - 1;
            bool ok = plain;
            if (z < 0 || z >= N.nz) {
                ok = ok && (N.periodic & 4);
                z = z < 0 ? N.nz - 1 : 0;
            }
            if (y < 0 || y >= N.ny) {
                ok = ok && (N.periodic & 2);
                y = y < 0 ? N.ny - 1 : 0;
            }
            if (x < 0 || x >= N.nx) {
                ok = ok && (N.periodic & 1);
                x = x < 0 ? N.nx - 1 : 0;
            }
            int s = 0, kept = 0;
            if (ok) {
                const int* at = R.cell_start + (N.cell_base + x + y * N.nx + z * N.nxy);
                s = at[0];
                kept = min(at[1] - s, R.cell_cap);
            }
            const int rounds = __reduce_max_sync(full, kept);
            for (int k0 = 0; k0 < rounds; k0 += G) {
                const int k = k0 + gl;
                bool acc = false;
                int j = -1;
                if (k < kept) {
                    j = R.cell_beads[s + k];
                    acc = list_pair<UNIFORM>(R, N, pi, bi, R.pos[j], R.binfo[j]);
                }
                add(acc, j);
            }
        }
    }
    if (gl == 0 && i >= 0) {
        if (n > R.list_cap)
            atomicAdd(R.counters + FN_CNT_LIST_OVERFLOW, (unsigned long long)(n - R.list_cap));
        R.list_count[i] = n;
    }
}

/* Near candidates a thread of k_lists keeps between its two tests. */
constexpr int kListKeep = 24;

/* The same lists with one thread per bead, for networks large enough to hide
   one thread's loads: fewer instructions per bead (no scan, no ballots).
   Bound by instruction issue (about 3,300 per warp, 60 % of the slots) and
   load latency.  The FP32 test from 16 bytes per candidate, with FP64 only
   where it cannot decide, took the rebuild of the 1M-bead tensile network
   from 313 to 211 us and that of the 4M-bead mat from 1,340 to 943 us (202
   and 904 since its launches are chained and its scan reads wider). */
template <bool UNIFORM, bool FOLD>
__global__ void __launch_bounds__(128, 8) k_lists(const __grid_constant__ RebuildArgs R, long long ncells) {
    await_previous();
    FN_GATED(R.gate);
    __shared__ int s_first[9 * 128];
    __shared__ unsigned short s_len[9 * 128];
    __shared__ int s_near[kListKeep * 128];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= R.cell_start[ncells]) return; /* beads placed in the grid */
    const float4 o = R.cell_pos[t];
    const int i = __float_as_int(o.w);
    const int c = R.cell_of[i];
    if (c < 0) return; /* beyond its cell's capacity: listed nowhere */
    const FnNet& N = UNIFORM ? R.net0 : R.nets[net_of_bead(R.nets, R.n_nets, i)];
    const float out_r2 = N.list_out_r2, in_r2 = N.list_in_r2;
    int* first = s_first + threadIdx.x;
    unsigned short* len = s_len + threadIdx.x;
    int* near = s_near + threadIdx.x;
    int cx, cy, cz;
    cell_coords(N, c, cx, cy, cz);
    const int longest = min(longest_run(R.cell_cap), 65535); /* s_len */
    /* the nine rows (dz, dy ascending): the row's cells in place are one run
       of the sorted arrays; all cell starts are loaded together */
    const int xa = max(cx - 1, 0), xb = min(cx + 2, N.nx);
    const int zlo = cz > 0 ? -N.nxy : N.periodic & 4 ? (N.nz - 1) * N.nxy : INT_MIN;
    const int zhi = cz + 1 < N.nz ? N.nxy : N.periodic & 4 ? -cz * N.nxy : INT_MIN;
    const int ylo = cy > 0 ? -N.nx : N.periodic & 2 ? (N.ny - 1) * N.nx : INT_MIN;
    const int yhi = cy + 1 < N.ny ? N.nx : N.periodic & 2 ? -cy * N.nx : INT_MIN;
    int widest = 0;
    const int* own = R.cell_start + (c - cx);
    {
        int s0[9], s1[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int dz = k < 3 ? zlo : k < 6 ? 0 : zhi, dy = k % 3 == 0 ? ylo : k % 3 == 1 ? 0 : yhi;
            const bool ok = dz != INT_MIN && dy != INT_MIN;
            const int* row = own + (ok ? dz + dy : 0);
            s0[k] = row[xa];
            s1[k] = ok ? row[xb] : s0[k];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            widest = max(widest, s1[k] - s0[k]);
            first[128 * k] = s0[k];
            len[128 * k] = (unsigned short)(s1[k] - s0[k]);
        }
    }
    /* beyond a periodic side in x, one more cell of each row, before or after
       the others */
    const bool wl = cx == 0 && (N.periodic & 1), wr = cx + 1 == N.nx && (N.periodic & 1);
    const bool moved = wl || wr || (cz == 0 || cz + 1 == N.nz) || (cy == 0 || cy + 1 == N.ny);
    const bool fold = FOLD && N.list_fold; /* then the bead stays where it is */
    const int4 bi = R.binfo[i];
    int* __restrict__ out = R.list + i;
    int n = 0, m = 0;
    /* second test of the near candidates */
    auto test = [&](bool crowded) {
        for (int k = 0; k < m; ++k) {
            int j;
            if (list_second<UNIFORM>(R, N, i, bi, near[128 * k], crowded, j)) { /* i itself is excluded, as a bonded neighbour */
                if (n < R.list_cap) out[(size_t)n * R.list_stride] = j;
                ++n;
            }
        }
        m = 0;
    };
    auto flush = [&]() {
        if (widest > R.cell_cap)
            test(true);
        else
            test(false);
    };
    /* first test of a candidate (dx, dy, dz) away */
    auto keep = [&](float4 v, float dx, float dy, float dz) {
        const float d2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
        if (!(d2 > out_r2)) near[128 * m++] = __float_as_int(v.w) | (d2 <= in_r2 ? 0 : (int)0x80000000);
    };
    for (int k = 0; k < 9 && widest <= longest; ++k) {
        float ox = o.x, oy = o.y, oz = o.z;
        int q = first[128 * k], left = len[128 * k];
        int q2 = 0, left2 = 0;
        if (moved) {
            /* cells below the grid lie at the far side: the bead moves up */
            const int dz = k < 3 ? zlo : k < 6 ? 0 : zhi, dy = k % 3 == 0 ? ylo : k % 3 == 1 ? 0 : yhi;
            if (!fold) {
                if (k < 3 && cz == 0) oz += (float)N.box[2];
                if (k >= 6 && cz + 1 == N.nz) oz -= (float)N.box[2];
                if (k % 3 == 0 && cy == 0) oy += (float)N.box[1];
                if (k % 3 == 2 && cy + 1 == N.ny) oy -= (float)N.box[1];
            }
            if ((wl || wr) && dz != INT_MIN && dy != INT_MIN) {
                const int* w = own + dz + dy + (wl ? N.nx - 1 : 0);
                q2 = w[0];
                left2 = w[1] - q2;
                widest = max(widest, left2);
                if (wl) { /* first */
                    int v = q;
                    q = q2;
                    q2 = v;
                    v = left;
                    left = left2;
                    left2 = v;
                    if (!fold) ox += (float)N.box[0];
                }
            }
        }
        for (int part = 0; part < 2; ++part) {
            while (left > 0) {
                if (m + left > kListKeep) flush();
                const int stop = q + min(left, kListKeep);
                left -= stop - q;
                if (fold) {
                    const float fx = fold_side(N, 0), fy = fold_side(N, 1), fz = fold_side(N, 2);
#pragma unroll 2
                    for (; q < stop; ++q) {
                        const float4 v = R.cell_pos[q];
                        keep(v, fold_axis(ox - v.x, fx), fold_axis(oy - v.y, fy), fold_axis(oz - v.z, fz));
                    }
                    continue;
                }
#pragma unroll 2
                for (; q < stop; ++q) {
                    const float4 v = R.cell_pos[q];
                    keep(v, ox - v.x, oy - v.y, oz - v.z);
                }
            }
            if (left2 == 0) break;
            q = q2;
            left = left2;
            left2 = 0;
            ox = wl || fold ? o.x : o.x - (float)N.box[0];
        }
    }
    if (widest > longest) {
        list_one_bead(R, N, i, c); /* candidate by candidate in FP64 */
        return;
    }
    flush();
    if (n > R.list_cap)
        atomicAdd(R.counters + FN_CNT_LIST_OVERFLOW, (unsigned long long)(n - R.list_cap));
    R.list_count[i] = n;
}

/* Bead i's full list, reading its candidates from global memory (k_lists,
   and bricks with more candidates than their shared memory holds). */
__device__ __forceinline__ void list_one_bead(const RebuildArgs& R, const FnNet& N, int i, int c) {
    const double4 pi = R.pos[i];
    const int4 bi = R.binfo[i];
    const int lc = c - N.cell_base;
    const int cz = lc / N.nxy;
    const int cy = (lc - cz * N.nxy) / N.nx;
    const int cx = lc - cz * N.nxy - cy * N.nx;
    int* __restrict__ out = R.list + i;
    int n = 0;
    for (int dz = -1; dz <= 1; ++dz) {
        int z = cz + dz;
        if (z < 0 || z >= N.nz) {
            if (!(N.periodic & 4)) continue;
            z = z < 0 ? N.nz - 1 : 0;
        }
        for (int dy = -1; dy <= 1; ++dy) {
            int y = cy + dy;
            if (y < 0 || y >= N.ny) {
                if (!(N.periodic & 2)) continue;
                y = y < 0 ? N.ny - 1 : 0;
            }
            const int row = N.cell_base + y * N.nx + z * N.nxy;
            if (cx >= 1 && cx + 1 < N.nx) {
                const int c0 = row + cx - 1;
                const int s0 = R.cell_start[c0];
                const int s3 = R.cell_start[c0 + 3];
                if (s3 - s0 <= R.cell_cap ||
                    (R.cell_count[c0] <= R.cell_cap && R.cell_count[c0 + 1] <= R.cell_cap &&
                     R.cell_count[c0 + 2] <= R.cell_cap)) {
                    scan_run(R, N, i, pi, bi, R.cell_beads + s0, s3 - s0, out, n);
                    continue;
                }
            }
            for (int dx = -1; dx <= 1; ++dx) {
                int x = cx + dx;
                if (x < 0 || x >= N.nx) {
                    if (!(N.periodic & 1)) continue;
                    x = x < 0 ? N.nx - 1 : 0;
                }
                const int nc = row + x;
                int m = R.cell_count[nc];
                if (m > R.cell_cap) m = R.cell_cap;
                scan_run(R, N, i, pi, bi, R.cell_beads + R.cell_start[nc], m, out, n);
            }
        }
    }
    if (n > R.list_cap)
        atomicAdd(R.counters + FN_CNT_LIST_OVERFLOW, (unsigned long long)(n - R.list_cap));
    R.list_count[i] = n;
}

/* BuildContactList by bricks of cells (the same lists as k_lists, entry for
   entry): one block per brick of kBrickX x kBrickY x kBrickZ cells of one
   network.  The block stages, once, every listable bead of the brick's cells
   and of the cells around them (ids, positions and bead info, in cell order:
   halo rows z-major, then y, then x, beads ascending within a cell, the first
   cell_cap of a full cell), in three wide rounds of loads -- cell counts and
   starts, bead ids, then positions and bead info by cp.async -- instead of a
   chain of dependent loads per candidate.  Each bead of the brick then scans
   its 27 cells from shared memory in k_lists' order (dz, dy, dx ascending),
   so the lists are k_lists' lists.  A brick whose halo holds more than
   kBrickCands beads lists its beads from global memory (list_one_bead). */
constexpr int kBrickHalo = (kBrickX + 2) * (kBrickY + 2) * (kBrickZ + 2);
constexpr int kBrickCells = kBrickX * kBrickY * kBrickZ;
constexpr int kBrickThreads = 128;

/* last index h of a[0..n] with a[h] <= q (a non-decreasing, a[0] <= q) */
__device__ __forceinline__ int last_le(const int* a, int n, int q) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a[mid] <= q)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

/* exclusive scan of v[0..n) into out[0..n] (out[n] the total) by one block */
__device__ __forceinline__ void block_scan_array(const int* v, int n, int* out, int* ws) {
    const int per = (n + (int)blockDim.x - 1) / (int)blockDim.x;
    const int b = threadIdx.x * per, e = min(b + per, n);
    int sum = 0;
    for (int k = b; k < e; ++k) sum += v[k];
    int total;
    int acc = block_scan_any(sum, ws, total);
    for (int k = b; k < e; ++k) {
        out[k] = acc;
        acc += v[k];
    }
    if (threadIdx.x == 0) out[n] = total;
    __syncthreads();
}

__global__ void __launch_bounds__(kBrickThreads) k_lists_brick(const RebuildArgs R, const int4* __restrict__ bricks) {
    await_previous();
    FN_GATED(R.gate);
    __shared__ int s_cnt[kBrickHalo], s_start[kBrickHalo], s_coff[kBrickHalo + 1];
    __shared__ int s_icnt[kBrickCells], s_ioff[kBrickCells + 1];
    __shared__ int s_ws[33];
    __shared__ int s_id[kBrickCands];
    __shared__ double4 s_pos[kBrickCands];
    __shared__ int4 s_bin[kBrickCands];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int4 B = bricks[blockIdx.x]; /* network, first cell x, y, z */
    const FnNet& N = R.nets[B.x];
    const int ex = min(kBrickX, N.nx - B.y), ey = min(kBrickY, N.ny - B.z), ez = min(kBrickZ, N.nz - B.w);
    const int HX = ex + 2, HY = ey + 2, H = HX * HY * (ez + 2), NIC = ex * ey * ez;
    /* round 1: count (first cell_cap of a full cell) and start of every halo
       cell; a cell off a non-periodic side holds nothing */
    for (int hc = tid; hc < H; hc += nt) {
        const int hx = hc % HX, hy = (hc / HX) % HY, hz = hc / (HX * HY);
        int gx = B.y - 1 + hx, gy = B.z - 1 + hy, gz = B.w - 1 + hz;
        bool ok = true;
        if (gx < 0 || gx >= N.nx) {
            if (N.periodic & 1)
                gx = gx < 0 ? N.nx - 1 : 0;
            else
                ok = false;
        }
        if (gy < 0 || gy >= N.ny) {
            if (N.periodic & 2)
                gy = gy < 0 ? N.ny - 1 : 0;
            else
                ok = false;
        }
        if (gz < 0 || gz >= N.nz) {
            if (N.periodic & 4)
                gz = gz < 0 ? N.nz - 1 : 0;
            else
                ok = false;
        }
        int cnt = 0, st = 0;
        if (ok) {
            const int cell = N.cell_base + gx + gy * N.nx + gz * N.nxy;
            cnt = min(R.cell_count[cell], R.cell_cap);
            st = R.cell_start[cell];
        }
        s_cnt[hc] = cnt;
        s_start[hc] = st;
    }
    __syncthreads();
    for (int ic = tid; ic < NIC; ic += nt) {
        const int ix = ic % ex, iy = (ic / ex) % ey, iz = ic / (ex * ey);
        s_icnt[ic] = s_cnt[((iz + 1) * HY + (iy + 1)) * HX + (ix + 1)];
    }
    __syncthreads();
    block_scan_array(s_cnt, H, s_coff, s_ws);
    block_scan_array(s_icnt, NIC, s_ioff, s_ws);
    const int C = s_coff[H], NI = s_ioff[NIC];
    if (C > kBrickCands) {
        /* too many to stage: each bead from global memory */
        for (int u = tid; u < NI; u += nt) {
            const int ic = last_le(s_ioff, NIC, u);
            const int ix = ic % ex, iy = (ic / ex) % ey, iz = ic / (ex * ey);
            const int hc = ((iz + 1) * HY + (iy + 1)) * HX + (ix + 1);
            const int i = R.cell_beads[s_start[hc] + (u - s_ioff[ic])];
            list_one_bead(R, N, i, R.cell_of[i]);
        }
        return;
    }
    /* round 2: bead ids; round 3: their positions and bead info */
    constexpr int kPer = (kBrickCands + kBrickThreads - 1) / kBrickThreads;
    int ids[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int q = tid + k * nt;
        ids[k] = -1;
        if (q < C) {
            const int hc = last_le(s_coff, H, q);
            ids[k] = R.cell_beads[s_start[hc] + (q - s_coff[hc])];
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int q = tid + k * nt;
        if (q < C && ids[k] >= 0) {
            s_id[q] = ids[k];
            const uint32_t dp = smem_addr(s_pos + q), db = smem_addr(s_bin + q);
            cp_async16(dp, R.pos + ids[k]);
            cp_async16(dp + 16, reinterpret_cast<const char*>(R.pos + ids[k]) + 16);
            cp_async16(db, R.binfo + ids[k]);
        }
    }
    cp_async_wait_all();
    __syncthreads();
    for (int u = tid; u < NI; u += nt) {
        const int ic = last_le(s_ioff, NIC, u);
        const int ix = ic % ex, iy = (ic / ex) % ey, iz = ic / (ex * ey);
        const int q = s_coff[((iz + 1) * HY + (iy + 1)) * HX + (ix + 1)] + (u - s_ioff[ic]);
        const int i = s_id[q];
        const double4 pi = s_pos[q];
        const int4 bi = s_bin[q];
        int* __restrict__ out = R.list + i;
        int n = 0;
        for (int dz = 0; dz < 3; ++dz)
            for (int dy = 0; dy < 3; ++dy) {
                const int row = ((iz + dz) * HY + (iy + dy)) * HX + ix; /* halo cell of dx = -1 */
                const int q1 = s_coff[row + 3];
                for (int qq = s_coff[row]; qq < q1; ++qq) {
                    const int j = s_id[qq];
                    if (j == i) continue;
                    const double4 pj = s_pos[qq];
                    double rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
                    double length = rx * rx + ry * ry + rz * rz;
                    if (N.list_mi) length = min_image(N, rx, ry, rz, length, N.list_mi);
                    if (!(length < N.list_r2_max)) continue; /* listed by no pair kind */
                    if (list_accept(N, R.pairs, length, pi, bi, pj, s_bin[qq])) {
                        if (n < R.list_cap) out[(size_t)n * R.list_stride] = j;
                        ++n;
                    }
                }
            }
        if (n > R.list_cap)
            atomicAdd(R.counters + FN_CNT_LIST_OVERFLOW, (unsigned long long)(n - R.list_cap));
        R.list_count[i] = n;
    }
}

/* Tile-compacted copy of the contact list for the staged step kernel: tile
   t's entries, bead after bead and in list order within a bead, from
   csr + t * region (region >= beads per tile x list capacity), and their
   number in tile_items[t].  One block of at least the tile's bead count. */
__global__ void k_list_tiles(const RebuildArgs R) {
    await_previous();
    let_next_start();
    FN_GATED(R.gate);
    __shared__ int ws[33];
    const FnTile t = R.tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    int c = 0;
    if (i < t.end) {
        c = R.list_count[i];
        if (c > R.list_cap) c = R.list_cap;
    }
    int total;
    const int off = block_scan_any(c, ws, total);
    int* out = R.csr + (size_t)blockIdx.x * (size_t)R.csr_region + off;
    for (int k = 0; k < c; ++k) out[k] = R.list[(size_t)k * R.list_stride + i];
    if (threadIdx.x == 0) R.tile_items[blockIdx.x] = total;
}

/* ------------------------------------------------------------------------ */
/* Exclusive scan of int counts (1024 threads x ITEMS items per block).
   The direct last pass adds up the sums of all blocks before its own: with 2
   items per thread that work and the 4-byte loads took 260 us on the 32M
   cells of 64 batched networks, with 8 and 16-byte loads 130 (the 4M-bead
   mat's whole rebuild 930 -> 904 us); below 2M cells the smaller tile keeps
   more SMs busy (10k beads, 100k cells: 27 us against 29).                   */

constexpr int SCAN_THREADS = 1024;
constexpr long long SCAN_SMALL = 2 << 20; /* cells from which on a thread takes 8 */

static inline int scan_items(long long n) { return n >= SCAN_SMALL ? 8 : 2; }

template <int SCAN_ITEMS>
__device__ __forceinline__ void scan_load(const int* in, long long base, long long n, int* v) {
    if (SCAN_ITEMS % 4 == 0 && base + SCAN_ITEMS <= n && ((uintptr_t)in & 15) == 0) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k += 4) {
            const int4 q = *reinterpret_cast<const int4*>(in + base + k);
            v[k] = q.x;
            v[k + 1] = q.y;
            v[k + 2] = q.z;
            v[k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) v[k] = base + k < n ? in[base + k] : 0;
    }
}

template <int SCAN_ITEMS>
__device__ __forceinline__ void scan_store(int* out, long long base, long long n, const int* v) {
    if (SCAN_ITEMS % 4 == 0 && base + SCAN_ITEMS <= n && ((uintptr_t)out & 15) == 0) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k += 4)
            *reinterpret_cast<int4*>(out + base + k) = make_int4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k)
            if (base + k < n) out[base + k] = v[k];
    }
}

/* Writes the exclusive sums of v, starting from ex; clears zero alongside. */
template <int SCAN_ITEMS>
__device__ __forceinline__ void scan_finish(int* out, int* zero, long long base, long long n, int* v, int ex) {
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int c = v[k];
        v[k] = ex;
        ex += c;
    }
    scan_store<SCAN_ITEMS>(out, base, n, v);
    if (zero) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) v[k] = 0;
        scan_store<SCAN_ITEMS>(zero, base, n, v);
    }
}

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sums[lane];
        int s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s - w;
        if (lane == 31) warp_sums[32] = s;
    }
    __syncthreads();
    total = warp_sums[32];
    const int r = x - v + warp_sums[warp];
    __syncthreads();
    return r;
}

template <int SCAN_ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_partials(const int* in, long long n,
                                                                 int* block_sums, const int* gate) {
    await_previous();
    let_next_start();
    FN_GATED(gate);
    __shared__ int ws[33];
    const long long base = (long long)blockIdx.x * (SCAN_THREADS * SCAN_ITEMS) + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS], s = 0;
    scan_load<SCAN_ITEMS>(in, base, n, v);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) s += v[k];
    int total;
    block_exclusive_scan(s, ws, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

/* One block scans the block sums in chunks, carrying the running total. */
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(int* block_sums, int nblocks, int* grand_total) {
    __shared__ int ws[33];
    int carry = 0;
    for (int base = 0; base < nblocks; base += SCAN_THREADS) {
        const int idx = base + (int)threadIdx.x;
        const int v = idx < nblocks ? block_sums[idx] : 0;
        int total;
        const int ex = block_exclusive_scan(v, ws, total);
        if (idx < nblocks) block_sums[idx] = ex + carry;
        carry += total;
    }
    if (threadIdx.x == 0) *grand_total = carry;
}

/* Exclusive scan, last pass: each block's offset added, written to out. */
template <int SCAN_ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(const int* in, long long n,
                                                              const int* block_sums, int* out) {
    __shared__ int ws[33];
    const long long base = (long long)blockIdx.x * (SCAN_THREADS * SCAN_ITEMS) + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
    scan_load<SCAN_ITEMS>(in, base, n, v);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) s += v[k];
    int total;
    const int ex = block_exclusive_scan(s, ws, total) + block_sums[blockIdx.x];
    scan_finish<SCAN_ITEMS>(out, nullptr, base, n, v, ex);
}

/* Exclusive scan, last pass, without a pass of its own over the block sums:
   each block adds up the raw sums of the blocks before it (a few thousand at
   most, read from L2), the last block writes the grand total; zero (if
   given) is cleared alongside. */
template <int SCAN_ITEMS>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply_direct(const int* in, long long n,
                                                                     const int* block_sums, int nblocks,
                                                                     int* out, int* grand_total,
                                                                     const int* gate, int* zero) {
    await_previous();
    let_next_start();
    FN_GATED(gate);
    __shared__ int ws[33];
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += SCAN_THREADS) before += block_sums[b];
    int offset;
    block_exclusive_scan(before, ws, offset); /* offset: the block sums' total */
    const long long base = (long long)blockIdx.x * (SCAN_THREADS * SCAN_ITEMS) + (long long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
    scan_load<SCAN_ITEMS>(in, base, n, v);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) s += v[k];
    int total;
    const int ex = block_exclusive_scan(s, ws, total) + offset;
    scan_finish<SCAN_ITEMS>(out, zero, base, n, v, ex);
    if (blockIdx.x == nblocks - 1 && threadIdx.x == 0) *grand_total = offset + total;
}

/* ------------------------------------------------------------------------ */
/* Observables: deterministic two-pass FP64 reduction per network.           */

__global__ void k_observe_partial(const ObserveArgs O) {
    await_previous();
    let_next_start();
    __shared__ double sx[256], sy[256], sz[256];
    __shared__ long long sb[256], sa[256];
    const int tid = threadIdx.x;
    double x = 0.0, y = 0.0, z = 0.0;
    long long nb = 0, na = 0;
    for (int i = O.bead_begin + blockIdx.x * blockDim.x + tid; i < O.bead_end;
         i += gridDim.x * blockDim.x) {
        if (w_type(O.pos[i].w) == O.reaction_type) {
            const float4 f = O.force[i];
            x += (double)f.x;
            y += (double)f.y;
            z += (double)f.z;
        }
    }
    if (O.ch_flags) {
        for (int i = O.bead_begin + blockIdx.x * blockDim.x + tid; i < O.bead_end;
             i += gridDim.x * blockDim.x) {
            const unsigned f = O.ch_flags[i], st = O.ch_status[i];
            nb += (f & FN_CH_SPRING) && !(st & 1);
            na += (f & FN_CH_ANGLE) && !(st & 2);
        }
    } else {
        for (int s = O.spring_begin + blockIdx.x * blockDim.x + tid; s < O.spring_end;
             s += gridDim.x * blockDim.x)
            nb += O.sp_status[s] == 0;
        for (int a = O.angle_begin + blockIdx.x * blockDim.x + tid; a < O.angle_end;
             a += gridDim.x * blockDim.x)
            na += O.an_status[a] == 0;
    }
    sx[tid] = x;
    sy[tid] = y;
    sz[tid] = z;
    sb[tid] = nb;
    sa[tid] = na;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (tid < o) {
            sx[tid] += sx[tid + o];
            sy[tid] += sy[tid + o];
            sz[tid] += sz[tid + o];
            sb[tid] += sb[tid + o];
            sa[tid] += sa[tid + o];
        }
        __syncthreads();
    }
    if (tid == 0) {
        double* o = O.partial + 5 * (size_t)blockIdx.x;
        o[0] = sx[0];
        o[1] = sy[0];
        o[2] = sz[0];
        o[3] = (double)sb[0];
        o[4] = (double)sa[0];
    }
}

/* The sum over the blocks' partial sums of quantity `warp` of NQ, one warp per
   quantity: lane l adds blocks l, l + 32, ... and the lanes are added by
   halves, a fixed order.  (One thread adding up to 1,024 x 5 doubles one
   after the other took 197 us, 13x the partial sums themselves.) */
template <int NQ>
__device__ __forceinline__ void add_partials(const double* partial, int nblocks, double* out) {
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    if (k >= NQ) return;
    double a = 0.0;
#pragma unroll 8
    for (int b = lane; b < nblocks; b += 32) a += partial[NQ * (size_t)b + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) out[k] = a;
}

__global__ void k_observe_final(const double* partial, int nblocks, double* out) {
    await_previous();
    let_next_start();
    add_partials<5>(partial, nblocks, out);
}

/* ------------------------------------------------------------------------ */
/* launch wrappers                                                           */

static int step_flags(bool do_drift, bool store_v) {
    return FN_STEP_SPRINGS | FN_STEP_ANGLES | FN_STEP_CONTACTS | (do_drift ? FN_STEP_DRIFT : 0) |
           (store_v ? FN_STEP_STORE_V : 0);
}

cudaError_t launch_step(const StepArgs& A, int ntiles, int block, bool damp, bool do_drift,
                        bool store_v, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    if (damp)
        launch_next(k_step<true>, ntiles, block, 0, s, A, step_flags(do_drift, store_v));
    else
        launch_next(k_step<false>, ntiles, block, 0, s, A, step_flags(do_drift, store_v));
    return cudaGetLastError();
}

template <bool DAMP, bool UNI>
static cudaError_t set_tiled_smem(size_t bytes) {
    return cudaFuncSetAttribute(k_step_tiled<DAMP, UNI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

/* The dynamic shared-memory limit is an attribute of the kernel on a
   device, shared by every context of the process: it is only ever raised
   (a context with smaller tiles must not lower it under another's launch). */
static bool raise_limit(size_t* table, size_t& bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
    if (bytes <= table[dev]) return false;
    table[dev] = bytes;
    return true;
}

cudaError_t prepare_step_tiled(size_t bytes) {
    static size_t done[64] = {};
    if (!raise_limit(done, bytes)) return cudaSuccess;
    cudaError_t e;
    if ((e = set_tiled_smem<true, true>(bytes))) return e;
    if ((e = set_tiled_smem<true, false>(bytes))) return e;
    if ((e = set_tiled_smem<false, true>(bytes))) return e;
    return set_tiled_smem<false, false>(bytes);
}

cudaError_t launch_step_tiled(const StepArgs& A, int ntiles, int block, bool damp, bool do_drift,
                              bool store_v, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    const size_t sm = step_tiled_smem(A.max_tile_sp, A.max_tile_an);
    const int flags = step_flags(do_drift, store_v);
    const bool all = A.uniform == FN_CONST_ALL;
    if (damp && all)
        launch_next(k_step_tiled<true, true>, ntiles, block, sm, s, A, flags);
    else if (damp)
        launch_next(k_step_tiled<true, false>, ntiles, block, sm, s, A, flags);
    else if (all)
        launch_next(k_step_tiled<false, true>, ntiles, block, sm, s, A, flags);
    else
        launch_next(k_step_tiled<false, false>, ntiles, block, sm, s, A, flags);
    return cudaGetLastError();
}

template <bool DAMP, bool FO, int CONSTS>
static cudaError_t set_chain_smem(size_t bytes) {
    return cudaFuncSetAttribute(k_step_chain<DAMP, FO, CONSTS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)bytes);
}

cudaError_t prepare_step_chain(size_t bytes) {
    static size_t done[64] = {};
    if (!raise_limit(done, bytes)) return cudaSuccess;
    cudaError_t e;
    if ((e = set_chain_smem<true, false, FN_CONST_NONE>(bytes))) return e;
    if ((e = set_chain_smem<true, false, FN_CONST_LAW>(bytes))) return e;
    if ((e = set_chain_smem<true, false, FN_CONST_ALL>(bytes))) return e;
    if ((e = set_chain_smem<false, false, FN_CONST_NONE>(bytes))) return e;
    if ((e = set_chain_smem<false, false, FN_CONST_LAW>(bytes))) return e;
    if ((e = set_chain_smem<false, false, FN_CONST_ALL>(bytes))) return e;
    return set_chain_smem<false, true, FN_CONST_NONE>(bytes);
}

cudaError_t launch_step_chain(const StepArgs& A, int ntiles, int block, bool damp, bool do_drift,
                              bool store_v, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    const size_t sm = step_chain_smem(block);
    const int flags = step_flags(do_drift, store_v);
    if (A.wide) {
        const int parts = (block - 4 + kWideBeads - 1) / kWideBeads, width = (block - 4 + parts - 1) / parts;
        auto go = [&](auto kernel) { launch_next(kernel, ntiles * parts, kWideThreads, 0, s, A, flags, parts, width); };
        if (A.uniform == FN_CONST_ALL)
            damp ? go(k_step_wide<true, FN_CONST_ALL>) : go(k_step_wide<false, FN_CONST_ALL>);
        else if (A.uniform == FN_CONST_LAW)
            damp ? go(k_step_wide<true, FN_CONST_LAW>) : go(k_step_wide<false, FN_CONST_LAW>);
        else
            damp ? go(k_step_wide<true, FN_CONST_NONE>) : go(k_step_wide<false, FN_CONST_NONE>);
        return cudaGetLastError();
    }
    auto go = [&](auto kernel) { launch_next(kernel, ntiles, block, sm, s, A, flags); };
    if (A.uniform == FN_CONST_ALL)
        damp ? go(k_step_chain<true, false, FN_CONST_ALL>) : go(k_step_chain<false, false, FN_CONST_ALL>);
    else if (A.uniform == FN_CONST_LAW)
        damp ? go(k_step_chain<true, false, FN_CONST_LAW>) : go(k_step_chain<false, false, FN_CONST_LAW>);
    else
        damp ? go(k_step_chain<true, false, FN_CONST_NONE>) : go(k_step_chain<false, false, FN_CONST_NONE>);
    return cudaGetLastError();
}

template <bool DAMP, bool DRIFT, bool STORE_V>
static cudaError_t set_staged_smem(size_t bytes) {
    return cudaFuncSetAttribute(k_step_staged<DAMP, DRIFT, STORE_V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)bytes);
}

cudaError_t prepare_step_staged(size_t bytes) {
    static size_t done[64] = {};
    if (!raise_limit(done, bytes)) return cudaSuccess;
    cudaError_t e;
    if ((e = set_staged_smem<true, true, true>(bytes))) return e;
    if ((e = set_staged_smem<true, false, false>(bytes))) return e;
    if ((e = set_staged_smem<false, true, true>(bytes))) return e;
    if ((e = set_staged_smem<false, true, false>(bytes))) return e;
    return set_staged_smem<false, false, false>(bytes);
}

cudaError_t launch_step_staged(const StepArgs& A, int ntiles, int block, bool damp, bool do_drift,
                               bool store_v, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    const size_t sm = step_staged_smem(block, A.chunk);
    if (damp) {
        if (do_drift)
            launch_next(k_step_staged<true, true, true>, ntiles, block, sm, s, A);
        else
            launch_next(k_step_staged<true, false, false>, ntiles, block, sm, s, A);
    } else {
        if (do_drift) {
            if (store_v)
                launch_next(k_step_staged<false, true, true>, ntiles, block, sm, s, A);
            else
                launch_next(k_step_staged<false, true, false>, ntiles, block, sm, s, A);
        } else {
            launch_next(k_step_staged<false, false, false>, ntiles, block, sm, s, A);
        }
    }
    return cudaGetLastError();
}


cudaError_t launch_forces_chain(const StepArgs& A, int ntiles, int block, int terms, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    launch_next(k_step_chain<false, true, FN_CONST_NONE>, ntiles, block, step_chain_smem(block), s, A, terms);
    return cudaGetLastError();
}

cudaError_t launch_drift(const StepArgs& A, int ntiles, int block, bool store_v, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    if (store_v)
        launch_next(k_drift<true>, ntiles, block, 0, s, A);
    else
        launch_next(k_drift<false>, ntiles, block, 0, s, A);
    return cudaGetLastError();
}

cudaError_t launch_forces_only(const StepArgs& A, int ntiles, int block, int terms,
                               cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    k_forces_only<<<ntiles, block, 0, s>>>(A, terms);
    return cudaGetLastError();
}

cudaError_t launch_reset_energy(float4* force, float4* vel, float4* vold, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_reset_energy<<<(n + 255) / 256, 256, 0, s>>>(force, vel, vold, n);
    return cudaGetLastError();
}

long long scan_block_count(long long n) {
    const long long tile = (long long)SCAN_THREADS * scan_items(n);
    return (n + tile - 1) / tile;
}

template <int ITEMS>
static void launch_scan(const int* in, long long n, int* out, int* block_sums, cudaStream_t s) {
    const unsigned nblk = (unsigned)scan_block_count(n);
    k_scan_partials<ITEMS><<<nblk, SCAN_THREADS, 0, s>>>(in, n, block_sums, nullptr);
    k_scan_sums<<<1, SCAN_THREADS, 0, s>>>(block_sums, (int)nblk, out + n);
    k_scan_apply<ITEMS><<<nblk, SCAN_THREADS, 0, s>>>(in, n, block_sums, out);
}

cudaError_t launch_exclusive_scan(const int* in, long long n, int* out, int* block_sums, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (scan_items(n) == 8)
        launch_scan<8>(in, n, out, block_sums, s);
    else
        launch_scan<2>(in, n, out, block_sums, s);
    return cudaGetLastError();
}

/* The rebuild's scan of the cell counts, as part of the step sequence. */
template <int ITEMS>
static void launch_cell_scan(const RebuildArgs& R, long long ncells, int* block_sums, cudaStream_t s) {
    const unsigned nblk = (unsigned)scan_block_count(ncells);
    launch_next(k_scan_partials<ITEMS>, nblk, SCAN_THREADS, 0, s, R.cell_count, ncells, block_sums, R.gate);
    launch_next(k_scan_apply_direct<ITEMS>, nblk, SCAN_THREADS, 0, s, R.cell_count, ncells, block_sums, (int)nblk,
                R.cell_start, R.cell_start + ncells, R.gate, R.cell_fill);
}

/* Largest context whose bead-by-bead build takes four lanes per bead: below
   it one thread per bead leaves the SMs waiting for its loads (whole rebuild
   before its launches were chained, four lanes against one: 10k beads 38 against 42 us, 100k dense 60 against
   91, 111k tensile 68 against 66), above it the instructions of the scan and
   the ballots count (300k tensile 111 against 90, 1M 320 against 211). */
constexpr int kGroupedBeads = 200000;

/* every bead may sit in the grid; groups past the grid total do nothing */
template <int G>
static void launch_lists_group(const RebuildArgs& R, int nb, long long ncells, cudaStream_t s) {
    constexpr int PER = 128 / G;
    if (R.uniform == FN_CONST_ALL)
        launch_next(k_lists_group<G, true>, (nb + PER - 1) / PER, 128, 0, s, R, ncells);
    else
        launch_next(k_lists_group<G, false>, (nb + PER - 1) / PER, 128, 0, s, R, ncells);
}

cudaError_t launch_rebuild(const RebuildArgs& R, int ntiles, int block, int nb, long long ncells,
                           int* scan_block_sums, cudaStream_t s) {
    const unsigned fill_blocks = (unsigned)std::min<long long>(4096, (ncells + 255) / 256 + 1);
    /* cell fills are cleared by the scan's last pass and list counts by
       k_cells, so only the cell counts need a pass of their own */
    launch_next(k_fill_int, fill_blocks, 256, 0, s, R.cell_count, ncells, 0, R.gate);
    if (ntiles > 0) launch_next(k_cells, ntiles, block, 0, s, R);
    if (scan_items(ncells) == 8)
        launch_cell_scan<8>(R, ncells, scan_block_sums, s);
    else
        launch_cell_scan<2>(R, ncells, scan_block_sums, s);
    if (nb > 0) launch_next(k_scatter, (nb + 255) / 256, 256, 0, s, R, nb);
    /* 10 cells per bead (64 batched networks): 59 us against 210 */
    if (nb > 0 && ncells >= SCAN_SMALL && ncells >= 4ll * nb)
        launch_next(k_cell_sort_sparse, (nb + 255) / 256, 256, 0, s, R, nb, ncells);
    else
        launch_next(k_cell_sort, (unsigned)((ncells + 255) / 256), 256, 0, s, R, (int)ncells);
    if (R.bricks) {
        if (R.nbricks > 0) launch_next(k_lists_brick, R.nbricks, kBrickThreads, 0, s, R, R.bricks);
    } else if (nb > 0 && R.list_lanes == 8) {
        launch_lists_group<8>(R, nb, ncells, s);
    } else if (nb > 0 && nb <= kGroupedBeads) {
        launch_lists_group<4>(R, nb, ncells, s);
    } else if (nb > 0) {
        const bool all = R.uniform == FN_CONST_ALL;
        launch_next(R.fold ? (all ? k_lists<true, true> : k_lists<false, true>)
                           : (all ? k_lists<true, false> : k_lists<false, false>),
                    (nb + 127) / 128, 128, 0, s, R, ncells);
    }
    /* the staged step kernel's copy, one block per tile (tiles are at most
       block - 4 beads wide) */
    if (R.csr && ntiles > 0) launch_next(k_list_tiles, ntiles, block, 0, s, R);
    return cudaGetLastError();
}

/* Displacement mode: raises the gate when a bead has moved more than the
   threshold since the last rebuild (image positions, so wraps do not count). */
__global__ void k_disp_check(const FnTile* tiles, const double4* img, const double4* ref, double thresh2,
                             int* gate) {
    await_previous();
    let_next_start();
    const FnTile t = tiles[blockIdx.x];
    const int i = t.begin + (int)threadIdx.x;
    if (i >= t.end) return;
    const double4 a = img[i], b = ref[i];
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    if (!(dx * dx + dy * dy + dz * dz <= thresh2)) *gate = 1;
}

__global__ void k_gate_clear(int* gate, unsigned long long* counters) {
    await_previous();
    let_next_start();
    if (*gate) {
        counters[FN_CNT_REBUILDS] += 1ull;
        *gate = 0;
    }
}

cudaError_t launch_verlet_rebuild(const RebuildArgs& R, const FnTile* tiles, const double4* img,
                                  double4* ref, double thresh2, int* gate, int ntiles, int block, int nb,
                                  long long ncells, int* scan_block_sums, cudaStream_t s) {
    if (ntiles > 0) launch_next(k_disp_check, ntiles, block, 0, s, tiles, img, ref, thresh2, gate);
    RebuildArgs G = R;
    G.img = img;
    G.ref = ref;
    cudaError_t e = launch_rebuild(G, ntiles, block, nb, ncells, scan_block_sums, s);
    if (e) return e;
    launch_next(k_gate_clear, 1, 1, 0, s, gate, R.counters);
    return cudaGetLastError();
}

/* Export of one bead field in upload order as x, y, z doubles (the host
   buffer layout of fn_download): out[3 u + a] = src[inv[u]].a. */
template <class T>
__global__ void k_export_xyz(const T* __restrict__ src, const int* __restrict__ inv, int n,
                             double* __restrict__ out) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    const T v = src[inv[u]];
    out[3 * (size_t)u] = (double)v.x;
    out[3 * (size_t)u + 1] = (double)v.y;
    out[3 * (size_t)u + 2] = (double)v.z;
}

cudaError_t launch_export_xyz(const double4* src, const int* inv, int n, double* out, cudaStream_t s) {
    if (n > 0) k_export_xyz<double4><<<(n + 255) / 256, 256, 0, s>>>(src, inv, n, out);
    return cudaGetLastError();
}

cudaError_t launch_export_xyz(const float4* src, const int* inv, int n, double* out, cudaStream_t s) {
    if (n > 0) k_export_xyz<float4><<<(n + 255) / 256, 256, 0, s>>>(src, inv, n, out);
    return cudaGetLastError();
}

/* ---------------------------------------------------------------------------
   Energy and virial (an addition: the reference computes neither).  Each term
   is the potential whose negative gradient is the force the step applies:
     spring   k/2 (L - L0)^2                      (F = k (L0 - L) u)
     angle    k (theta - theta0)^2                (M = -2 k (theta - theta0))
     hs       K/2 p^2, p = r_i + r_j - r > 0
     hsr      K/2 p^2 + k/2 (rc - r)^2 for r < rc
     lj       48 eps s^12/13 (r^-13 - rc^-13) - 24 eps s^6/7 (r^-7 - rc^-7)
              + c4 (r - rc), the integral of the shifted force to rc = c3
     st       K (c2 (rc - r) - (rc^2 - r^2)/2) + K0 (c6 (rc - r) - (rc^2 - r^2)/2)
     wall     wall_k/2 d^2 for a penetration d past a wall
     gravity  -g . x (image position; g is a force per bead)
   Kinetic energy is m/2 |v|^2 of the step-end velocity (velocity_old) over
   beads of non-zero mass.  The virial is sum r_ij (x) F_ij over springs,
   angles (r_ba (x) F_a + r_bc (x) F_c) and contact pairs, each pair once. */
__device__ __forceinline__ double contact_energy(const FnNet& N, const FnPair* __restrict__ pairs,
                                                 double4 pi, double4 pj, double& Rx, double& Ry,
                                                 double& Rz, double& rx, double& ry, double& rz,
                                                 int& acts) {
    const FnPair* P = pairs + N.pair_base + getadress(w_type(pi.w), w_type(pj.w), N.types_num);
    double r, ir;
    acts = contact_law(N, *P, pi, pj, Rx, Ry, Rz, rx, ry, rz, r, ir);
    if (!acts) return 0.0;
    const double rsum = (double)w_radius(pi.w) + (double)w_radius(pj.w);
    switch (P->kind) {
    case 1: {
        const double rc = P->c[2], s2 = P->c[0] * P->c[0], eps = P->c[1];
        const double s6 = s2 * s2 * s2, s12 = s6 * s6;
        const double irc = 1.0 / rc;
        if (r == 0.0) ir = 1.0 / r; /* the force terms take 0 there; the potential is singular */
        /* r^-7 and r^-13 by products (within a few ulp of pow, far cheaper) */
        const double ir2 = ir * ir, ir6 = ir2 * ir2 * ir2, ir7 = ir6 * ir, ir13 = ir6 * ir7;
        const double irc2 = irc * irc, irc6 = irc2 * irc2 * irc2, irc7 = irc6 * irc, irc13 = irc6 * irc7;
        return 48.0 * eps * s12 / 13.0 * (ir13 - irc13) - 24.0 * eps * s6 / 7.0 * (ir7 - irc7) +
               P->c[3] * (r - rc);
    }
    case 2: {
        const double p = rsum - r;
        return 0.5 * P->c[0] * p * p;
    }
    case 3: {
        const double rc = sqrt(P->c[3]);
        const double q = 0.5 * (rc * rc - r * r);
        return P->c[0] * (P->c[1] * (rc - r) - q) + P->c[4] * (P->c[5] * (rc - r) - q);
    }
    case 4: {
        const double p = rsum - r;
        double u = p > 0.0 ? 0.5 * P->c[0] * p * p : 0.0;
        if (r < P->c[2]) u += 0.5 * P->c[1] * (P->c[2] - r) * (P->c[2] - r);
        return u;
    }
    }
    return 0.0;
}

__device__ __forceinline__ void add_outer(double* w, double ax, double ay, double az, double bx,
                                          double by, double bz) {
    w[0] += ax * bx;
    w[1] += ax * by;
    w[2] += ax * bz;
    w[3] += ay * bx;
    w[4] += ay * by;
    w[5] += ay * bz;
    w[6] += az * bx;
    w[7] += az * by;
    w[8] += az * bz;
}

/* At most 85 registers (3 blocks of 256 per SM, a few accumulators spilled):
   the per-bead contact walk waits on partner loads, which more resident warps
   hide (measured on the 1M-bead tensile network: 0.37 ms per evaluation
   against 0.45 ms at the 102 registers the compiler picks unbounded). */
__global__ void __launch_bounds__(256, 3) k_energy_partial(const EnergyArgs E) {
    await_previous();
    __shared__ double red[8][FN_EN_N];
    const FnNet& N = E.nets[E.net];
    double acc[FN_EN_N];
#pragma unroll
    for (int k = 0; k < FN_EN_N; ++k) acc[k] = 0.0;
    double* W = acc + FN_EN_VIRIAL;
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;

    for (int i = E.bead_begin + t0; i < E.bead_end; i += stride) {
        const double4 p = E.pos[i];
        const double4 im = E.img[i];
        if (im.w > 0.0) {
            const float4 v = E.vold[i];
            const double vx = v.x, vy = v.y, vz = v.z;
            acc[FN_EN_KINETIC] += 0.5 / im.w * (vx * vx + vy * vy + vz * vz);
        }
        acc[FN_EN_GRAVITY] -= N.g[0] * im.x + N.g[1] * im.y + N.g[2] * im.z;
        if (N.walls) {
            const double pc[3] = {p.x, p.y, p.z};
            for (int a = 0; a < 3; ++a) {
                if (!(N.walls & (1 << a))) continue;
                double d = 0.0;
                if (pc[a] < 0.0) d = pc[a];
                if (pc[a] > N.box[a]) d = pc[a] - N.box[a];
                acc[FN_EN_WALL] += 0.5 * N.wall_k * d * d;
            }
        }
        int n = E.list_count[i];
        if (n > E.list_cap) n = E.list_cap;
        for (int k = 0; k < n; ++k) {
            const int j = E.list[(size_t)k * E.list_stride + i];
            if (j <= i) continue;
            double Rx, Ry, Rz, rx, ry, rz;
            int acts;
            const double u = contact_energy(N, E.pairs, p, E.pos[j], Rx, Ry, Rz, rx, ry, rz, acts);
            if (acts) {
                acc[FN_EN_CONTACT] += u;
                acc[FN_EN_CONTACTS] += 1.0;
                add_outer(W, rx, ry, rz, Rx, Ry, Rz);
            }
        }
    }
    for (int s = E.spring_begin + t0; s < E.spring_end; s += stride) {
        const int type = E.sp_type[s];
        if (!(type == 0 || type == 1)) continue;
        const int2 e = E.sp_ends[s];
        const int alive = E.ch_status ? (E.ch_status[min(e.x, e.y)] & 1) : (E.sp_status[s] == 1);
        if (!alive) continue;
        const double4 a = E.img[e.x], b = E.img[e.y];
        const float4 par = E.sp_par[s];
        double fx, fy, fz;
        int broke;
        spring_pts(a.x, a.y, a.z, b.x, b.y, b.z, par, 0, fx, fy, fz, broke);
        const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
        const double L = sqrt(dx * dx + dy * dy + dz * dz) - (double)par.x;
        acc[FN_EN_SPRING] += 0.5 * (double)par.y * L * L;
        add_outer(W, dx, dy, dz, fx, fy, fz);
    }
    for (int q = E.angle_begin + t0; q < E.angle_end; q += stride) {
        const int4 b = E.an_b[q];
        const int alive = E.ch_status ? ((E.ch_status[b.y] >> 1) & 1) : (E.an_status[q] == 1);
        if (!alive) continue;
        const double4 t1 = E.img[b.x], t2 = E.img[b.y], t3 = E.img[b.z];
        const float2 par = E.an_par[q];
        double pax, pay, paz, pcx, pcy, pcz;
        angle_pts(t1.x, t1.y, t1.z, t2.x, t2.y, t2.z, t3.x, t3.y, t3.z, par, pax, pay, paz, pcx,
                  pcy, pcz);
        const double bax = t1.x - t2.x, bay = t1.y - t2.y, baz = t1.z - t2.z;
        const double bcx = t3.x - t2.x, bcy = t3.y - t2.y, bcz = t3.z - t2.z;
        double dotp = (bax * bcx + bay * bcy + baz * bcz) /
                      (sqrt(bax * bax + bay * bay + baz * baz) * sqrt(bcx * bcx + bcy * bcy + bcz * bcz));
        if (dotp < -1.0) dotp = -0.999999;
        if (dotp > 1.0) dotp = 0.999999;
        const double d = fn_acos(dotp) - (double)par.x;
        acc[FN_EN_ANGLE] += (double)par.y * d * d;
        add_outer(W, bax, bay, baz, pax, pay, paz);
        add_outer(W, bcx, bcy, bcz, pcx, pcy, pcz);
    }
    /* fixed-order block reduction: each warp by halves, then the warps in
       order (the block-wide tree, a barrier per halving and quantity, was a
       third of the kernel on a 100k-bead network) */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < FN_EN_N; ++k) {
        double a = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) red[warp][k] = a;
    }
    __syncthreads();
    if (threadIdx.x < FN_EN_N) {
        double a = 0.0;
        for (int w = 0; w < 8; ++w) a += red[w][threadIdx.x];
        E.partial[(size_t)FN_EN_N * blockIdx.x + threadIdx.x] = a;
    }
}

__global__ void k_energy_final(const double* partial, int nblocks, double* out) {
    await_previous();
    let_next_start();
    add_partials<FN_EN_N>(partial, nblocks, out);
}

cudaError_t launch_energy(const EnergyArgs& E, int nblocks, double* out, cudaStream_t s) {
    launch_next(k_energy_partial, nblocks, 256, 0, s, E);
    launch_next(k_energy_final, 1, 32 * FN_EN_N, 0, s, E.partial, nblocks, out);
    return cudaGetLastError();
}

cudaError_t launch_observe(const ObserveArgs& O, int nblocks, double* out, cudaStream_t s) {
    launch_next(k_observe_partial, nblocks, 256, 0, s, O);
    launch_next(k_observe_final, 1, 32 * 5, 0, s, O.partial, nblocks, out);
    return cudaGetLastError();
}

}  // namespace fn
