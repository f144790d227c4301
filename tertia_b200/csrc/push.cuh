// push.cu — plasma macro-particle push across one xi-layer with current /
// density deposit (reference Mesh::MoveParticlesLayerSplit,
// movepart_splitlayer.cpp:781-1544, DepositCurrentsInCellSplit :1547-1655,
// ExchangeCurrentsSplit :1685-1711; dead GPU twin cuMoveSplitParticles,
// plasma_particles.cu:72-863).
//
// Layout: particles are SoA (y, z, px, py, pz, w, cell) grouped by cell in
// ascending cell order, one thread per particle.  In the reference's live
// NGP path a particle never leaves its seeded cell (the full-step relink at
// :1507 uses the outer jtmp = j), so the grouping is permanent and the 4-8
// particles of a cell sit in consecutive lanes: their deposits are summed
// with a warp-segmented reduction over runs of equal destination cell and a
// single lane per run issues the global atomics.  The guard-ring fold of
// ExchangeCurrentsSplit is done by depositing at (j mod My, k mod Mz).
//
// The FP64 kernel (push_f64.cu, compiled with -fmad=false) follows the
// reference's expression order without contraction and reproduces the oracle
// bit for bit on identical inputs, cell indices included.  The FP32 kernel
// (push_f32.cu) uses the same physics with the divisions factored into six
// reciprocals and FMA contraction allowed: it is instruction bound, not
// memory bound, and this halves its instruction count.
#pragma once
#include <type_traits>

#include "qs_common.cuh"
#include "qs_internal.h"
#include "pdl.cuh"
#include "pushmath.cuh"
#include "trace.cuh"

namespace qs {

template <class T>
__device__ __forceinline__ T ld(const T* p) { return __ldg(p); }

template <class T>
__device__ __forceinline__ T sqrt_t(T x);
template <>
__device__ __forceinline__ float sqrt_t<float>(float x) { return __fsqrt_rn(x); }
template <>
__device__ __forceinline__ double sqrt_t<double>(double x) { return __dsqrt_rn(x); }

template <class T>
__device__ __forceinline__ T floor_t(T x);
template <>
__device__ __forceinline__ float floor_t<float>(float x) { return floorf(x); }
template <>
__device__ __forceinline__ double floor_t<double>(double x) { return floor(x); }

template <class T>
__device__ __forceinline__ T fabs_t(T x) { return x < T(0) ? -x : x; }

__device__ __forceinline__ int wrap_idx(int j, int M) {
    // shifts are small (|shift| <= a few cells): avoid the integer modulo
    while (j >= M) j -= M;
    while (j < 0) j += M;
    return j;
}


// Sub-cycled transverse move and deposit of one particle (:1389-1479 with
// DepositCurrentsInCellSplit :1547-1615 or the CIC of MoveInCell), then the
// full-step store (:1501-1512).  The first sub-step's deposit is returned in
// (key, v) for the warp-level reduction; later sub-steps deposit directly.
template <class T, int SHAPE, bool PRECISE, int NV>
__device__ __forceinline__ void move_and_deposit(const PushArgs<T>& a, int64_t i, int j, int k,
                                                 T yp, T zp, T px, T py, T pz, T djx, T djy,
                                                 T djz, T drho, T dy, T dz, int& key, T (&v)[NV]) {
    const T one = T(1);
    const int My = a.My, Mz = a.Mz;
    const size_t plane = a.plane;
    T partdx = T(0), step = one;
    if (fabs_t(dy) > one || fabs_t(dz) > one) {
        if (fabs_t(dy) > fabs_t(dz)) step = partdx = fabs_t(dy);
        else step = partdx = fabs_t(dz);
    }
    if (partdx < one) partdx = step = one;
    const T MyT = T(My), MzT = T(Mz);
    T ytmp = yp, ztmp = zp;
    int jb = j, kb = k, jj = j, kk = k;
    bool first = true;
    while (partdx > T(0)) {
        T part_step;
        if (partdx > one) {
            partdx -= one;
            part_step = one / step;
        } else {
            part_step = partdx / step;
            partdx = T(0);
        }
        if (SHAPE == QS_SHAPE_NGP && !PRECISE) {
            // reference form (:1420-1437); the added j is the outer j_jump
            ytmp += dy * part_step + T(j);
            ztmp += dz * part_step + T(k);
            while (ytmp > MyT) ytmp -= MyT;
            while (ytmp < T(0)) ytmp += MyT;
            while (ztmp > MzT) ztmp -= MzT;
            while (ztmp < T(0)) ztmp += MzT;
            jj = (int)ytmp;
            kk = (int)ztmp;
            ytmp -= T(jj);
            ztmp -= T(kk);
        } else {
            const T uy = ytmp + dy * part_step;
            const T uz = ztmp + dz * part_step;
            const T fy = floor_t<T>(uy), fz = floor_t<T>(uz);
            T ry = uy - fy, rz = uz - fz;
            int sy = (int)fy, sz = (int)fz;
            if (ry >= one) { ry = T(0); sy += 1; }
            if (rz >= one) { rz = T(0); sz += 1; }
            const int bj = (SHAPE == QS_SHAPE_NGP) ? j : jb;
            const int bk = (SHAPE == QS_SHAPE_NGP) ? k : kb;
            jj = wrap_idx(bj + sy, My);
            kk = wrap_idx(bk + sz, Mz);
            ytmp = ry;
            ztmp = rz;
            jb = jj;
            kb = kk;
        }
        const T s = part_step;
        const int fj = wrap_idx(jj, My), fk = wrap_idx(kk, Mz);
        if (SHAPE == QS_SHAPE_NGP) {
            const T d0 = djx * s, d1 = djy * s, d2 = djz * s, d3 = drho * s;
            if (first) {
                key = fj + My * fk;
                v[0] = d0; v[1] = d1; v[2] = d2; v[3] = d3;
            } else {
                const size_t n = (size_t)fj + (size_t)My * fk;
                atomicAdd(a.dep + 0 * plane + n, d0);
                atomicAdd(a.dep + 1 * plane + n, d1);
                atomicAdd(a.dep + 2 * plane + n, d2);
                atomicAdd(a.dep + 3 * plane + n, d3);
            }
        } else {
            const T ayp = ytmp, ayc = one - ayp, azp = ztmp, azc = one - azp;
            const T w00 = ayc * azc, w10 = ayp * azc, w01 = ayc * azp, w11 = ayp * azp;
            const T q[4] = {djx * s, djy * s, djz * s, drho * s};
            const T wc[4] = {w00, w10, w01, w11};
            if (first) {
                key = fj + My * fk;
#pragma unroll
                for (int cnr = 0; cnr < 4; cnr++)
#pragma unroll
                    for (int qq = 0; qq < 4; qq++) v[cnr * 4 + qq] = q[qq] * wc[cnr];
            } else {
                const int j1 = wrap_idx(fj + 1, My), k1 = wrap_idx(fk + 1, Mz);
                const size_t nn[4] = {(size_t)fj + (size_t)My * fk,
                                      (size_t)j1 + (size_t)My * fk,
                                      (size_t)fj + (size_t)My * k1,
                                      (size_t)j1 + (size_t)My * k1};
#pragma unroll
                for (int cnr = 0; cnr < 4; cnr++)
#pragma unroll
                    for (int qq = 0; qq < 4; qq++)
                        atomicAdd(a.dep + qq * plane + nn[cnr], q[qq] * wc[cnr]);
            }
        }
        first = false;
    }
    const int jf = wrap_idx(jj, My), kf = wrap_idx(kk, Mz);
    if (a.dep_cell) a.dep_cell[i] = jf + My * kf;
    if (a.full) {
        a.px[i] = px;
        a.py[i] = py;
        a.pz[i] = pz;
        a.y[i] = ytmp;
        a.z[i] = ztmp;
        if (SHAPE == QS_SHAPE_CIC) a.cell_out[i] = jf + My * kf;
    }
}

// SHAPE: QS_SHAPE_NGP / QS_SHAPE_CIC.  PRECISE: cell-relative position
// update (u = frac + d*part_step measured from the base cell) instead of the
// reference's ytmp + j form; the FP32 kernels use it to keep the in-cell
// fraction at full float precision.
//
// A few warps per SM at most sizes it runs at, so a chain bounds it: particle,
// cell, the cell's 48 field values, some twenty IEEE divisions in the
// reference's order (FAST: five), the warp's sums, the atomics.  The particle
// is read ahead of the wait for the kernel in front where the caller can tell
// that nothing before it still writes it, and the sums stop at the warp's longest
// run of one cell (five steps of 16 values against two or three).  Plain FP64
// march per layer, 128^2 69.7 -> 66.9 us, 256^2 172.4 -> 157.5, 512^2
// 842 -> 814; FP32 NGP of 5 per cell at 128^2 24.2 -> 23.0 (with both and
// blocks of 128 threads).
template <class T, int SHAPE, bool PRECISE, bool FAST>
__global__ void __launch_bounds__(128) push_kernel(PushArgs<T> a) {
    constexpr int NV = (SHAPE == QS_SHAPE_NGP) ? 4 : 16;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int My = a.My, Mz = a.Mz;
    int key = -1;          // base cell of the first sub-step deposit
    T v[NV];
#pragma unroll
    for (int c = 0; c < NV; c++) v[c] = T(0);

    if (!a.early) pdl_wait();
    const bool in = i < a.n;
    const int cell = in ? a.cell[i] : 0;
    const T yp = in ? a.y[i] : T(0), zp = in ? a.z[i] : T(0);
    T px = in ? a.px[i] : T(0), py = in ? a.py[i] : T(0), pz = in ? a.pz[i] : T(0);
    const T weight = in ? a.w[i] : T(0);
    if (a.early) pdl_wait();
    if (in) {
        const T one = T(1), two = T(2), half = T(0.5);
        int j, k;
        if (FAST) cell_jk(cell, My, a.invMy, j, k);
        else { j = cell % My; k = cell / My; }
        if (!(yp >= T(0) && yp <= one && zp >= T(0) && zp <= one)) {
            atomicOr(a.err, DEV_ERR_RANGE);
        } else {
            if constexpr (FAST) {
            // ---- FP32: the same update with the divisions factored out, and
            // 1 - Vx in its cancellation-free form (pushmath.cuh)
            const T inv_gp = one / sqrt_t<T>(one + px * px + py * py + pz * pz);
            const T Vxp = px * inv_gp, Vyp = py * inv_gp, Vzp = pz * inv_gp;
            const T q2m = a.q2m;
            const size_t plane = a.plane;
            T ex, ey, ez, bx, by, bz;
            if (SHAPE == QS_SHAPE_NGP) {
                const size_t n = (size_t)cell;
                ex = half * (ld(a.P + 0 * plane + n) + ld(a.C + 0 * plane + n));
                ey = half * (ld(a.P + 1 * plane + n) + ld(a.C + 1 * plane + n));
                ez = half * (ld(a.P + 2 * plane + n) + ld(a.C + 2 * plane + n));
                bx = half * (ld(a.P + 3 * plane + n) + ld(a.C + 3 * plane + n));
                by = half * (ld(a.P + 4 * plane + n) + ld(a.C + 4 * plane + n));
                bz = half * (ld(a.P + 5 * plane + n) + ld(a.C + 5 * plane + n));
            } else {
                const T ayc = one - yp, ayp = yp, azc = one - zp, azp = zp;
                const T acc = ayc * azc, apc = ayp * azc, acp = ayc * azp, app = ayp * azp;
                const int j1 = wrap_idx(j + 1, My), k1 = wrap_idx(k + 1, Mz);
                const size_t n00 = (size_t)j + (size_t)My * k, n10 = (size_t)j1 + (size_t)My * k,
                             n01 = (size_t)j + (size_t)My * k1, n11 = (size_t)j1 + (size_t)My * k1;
                T g[6];
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    const T* Pc = a.P + c * plane;
                    const T* Cc = a.C + c * plane;
                    T vp = acc * ld(Pc + n00) + apc * ld(Pc + n10) + acp * ld(Pc + n01) +
                           app * ld(Pc + n11);
                    T vc = acc * ld(Cc + n00) + apc * ld(Cc + n10) + acp * ld(Cc + n01) +
                           app * ld(Cc + n11);
                    g[c] = half * (vp + vc);
                }
                ex = g[0]; ey = g[1]; ez = g[2]; bx = g[3]; by = g[4]; bz = g[5];
            }
            const T omp = one_minus_vx(px, py, pz, inv_gp);   // 1 - Vx before the kick
            const T inv1 = one / omp;
            const T kE = a.sE * inv1;                 // q2m*hx/2 / (1 - Vx)
            ex *= kE;
            ey *= kE;
            ez *= kE;
            px += ex;
            py += ey;
            pz += ez;
            const T gamma_r = one / sqrt_t<T>(one + px * px + py * py + pz * pz);
            const T kB = gamma_r * kE;               // gamma_r*q2m/(1-Vx)*hx/2
            bx = (bx + a.bxe) * kB;
            by = (by + a.bye) * kB;
            bz = (bz + a.bze) * kB;
            const T co = two / (one + bx * bx + by * by + bz * bz);
            const T p3x = (py * bz - pz * by + px) * co;
            const T p3y = (pz * bx - px * bz + py) * co;
            const T p3z = (px * by - py * bx + pz) * co;
            px += ex + (p3y * bz - p3z * by);
            py += ey + (p3z * bx - p3x * bz);
            pz += ez + (p3x * by - p3y * bx);
            const T inv_g = one / sqrt_t<T>(one + px * px + py * py + pz * pz);
            const T Vxm = px * inv_g, Vym = py * inv_g, Vzm = pz * inv_g;
            const T Vy = half * (Vym + Vyp);
            const T Vz = half * (Vzm + Vzp);
            // 1 - (Vxm + Vxp)/2 = ((1 - Vxm) + (1 - Vxp))/2
            const T inv2 = one / (half * (one_minus_vx(px, py, pz, inv_g) + omp));
            const T wq = weight * inv2;
            const T djx = wq * a.djx0 * Vxm;
            const T djy = wq * a.djy0 * Vym;
            const T djz = wq * a.djz0 * Vzm;
            const T drho = wq * a.drho0;
            const T dy = Vy * a.hxhy * inv2;
            const T dz = Vz * a.hxhz * inv2;
            move_and_deposit<T, SHAPE, PRECISE, NV>(a, i, j, k, yp, zp, px, py, pz, djx, djy, djz,
                                                   drho, dy, dz, key, v);
            } else {
            T gammap = sqrt_t<T>(one + px * px + py * py + pz * pz);
            T Vx = px / gammap;
            const T Vxp = Vx, Vyp = py / gammap, Vzp = pz / gammap;
            const T q2m = a.q2m;
            const size_t plane = a.plane;
            T ex, ey, ez, bx, by, bz;
            if (SHAPE == QS_SHAPE_NGP) {
                const size_t n = (size_t)cell;
                ex = half * (ld(a.P + 0 * plane + n) + ld(a.C + 0 * plane + n));
                ey = half * (ld(a.P + 1 * plane + n) + ld(a.C + 1 * plane + n));
                ez = half * (ld(a.P + 2 * plane + n) + ld(a.C + 2 * plane + n));
                bx = half * (ld(a.P + 3 * plane + n) + ld(a.C + 3 * plane + n));
                by = half * (ld(a.P + 4 * plane + n) + ld(a.C + 4 * plane + n));
                bz = half * (ld(a.P + 5 * plane + n) + ld(a.C + 5 * plane + n));
            } else {
                const T ayc = one - yp, ayp = yp, azc = one - zp, azp = zp;
                const T acc = ayc * azc, apc = ayp * azc, acp = ayc * azp, app = ayp * azp;
                const int j1 = wrap_idx(j + 1, My), k1 = wrap_idx(k + 1, Mz);
                const size_t n00 = (size_t)j + (size_t)My * k, n10 = (size_t)j1 + (size_t)My * k,
                             n01 = (size_t)j + (size_t)My * k1, n11 = (size_t)j1 + (size_t)My * k1;
                T g[6];
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    const T* Pc = a.P + c * plane;
                    const T* Cc = a.C + c * plane;
                    T vp = acc * ld(Pc + n00) + apc * ld(Pc + n10) + acp * ld(Pc + n01) +
                           app * ld(Pc + n11);
                    T vc = acc * ld(Cc + n00) + apc * ld(Cc + n10) + acp * ld(Cc + n01) +
                           app * ld(Cc + n11);
                    g[c] = half * (vp + vc);
                }
                ex = g[0]; ey = g[1]; ez = g[2]; bx = g[3]; by = g[4]; bz = g[5];
            }
            const T hx = a.hx;
            const T sE = q2m * hx / two;
            ex *= sE;
            ey *= sE;
            ez *= sE;
            px += ex / (one - Vx);
            py += ey / (one - Vx);
            pz += ez / (one - Vx);
            T gamma = sqrt_t<T>(one + px * px + py * py + pz * pz);
            const T gamma_r = one / gamma;
            bx += a.bxe;
            by += a.bye;
            bz += a.bze;
            bx = bx * gamma_r * q2m / (one - Vx) * hx / two;
            by = by * gamma_r * q2m / (one - Vx) * hx / two;
            bz = bz * gamma_r * q2m / (one - Vx) * hx / two;
            const T co = two / (one + (bx * bx) + (by * by) + (bz * bz));
            T p3x = py * bz - pz * by + px;
            T p3y = pz * bx - px * bz + py;
            T p3z = px * by - py * bx + pz;
            p3x *= co;
            p3y *= co;
            p3z *= co;
            const T px_new = p3y * bz - p3z * by;
            const T py_new = p3z * bx - p3x * bz;
            const T pz_new = p3x * by - p3y * bx;
            px += ex / (one - Vx) + px_new;
            py += ey / (one - Vx) + py_new;
            pz += ez / (one - Vx) + pz_new;
            gamma = sqrt_t<T>(one + px * px + py * py + pz * pz);
            const T Vxm = px / gamma, Vym = py / gamma, Vzm = pz / gamma;
            Vx = half * (Vxm + Vxp);
            const T Vy = half * (Vym + Vyp);
            const T Vz = half * (Vzm + Vzp);
            T djx = weight * a.djx0 * Vxm;
            T djy = weight * a.djy0 * Vym;
            T djz = weight * a.djz0 * Vzm;
            T drho = weight * a.drho0;
            djx *= one / (one - Vx);
            djy *= one / (one - Vx);
            djz *= one / (one - Vx);
            drho *= one / (one - Vx);
            T dy = Vy * hx / a.hy;
            T dz = Vz * hx / a.hz;
            dy = dy / (one - Vx);
            dz = dz / (one - Vx);
            move_and_deposit<T, SHAPE, PRECISE, NV>(a, i, j, k, yp, zp, px, py, pz, djx, djy, djz,
                                                   drho, dy, dz, key, v);
            }
        }
    }

    pdl_trigger();
    // warp-segmented sum over runs of equal first-deposit cell
    const unsigned full = 0xffffffffu;
    const int nextKey = __shfl_down_sync(full, key, 1);
    const int prevKey = __shfl_up_sync(full, key, 1);
    const bool last = (lane == 31) || (nextKey != key);
    const unsigned lastMask = __ballot_sync(full, last);
    const int end = __ffs(lastMask & (full << lane)) - 1;
    const bool head = (lane == 0) || (prevKey != key);
    // no run is longer than maxrun: the steps beyond it would add nothing
    const int maxrun = (int)__reduce_max_sync(full, (unsigned)(end - lane + 1));
    for (int d = 1; d < maxrun; d <<= 1) {
#pragma unroll
        for (int c = 0; c < NV; c++) {
            const T o = __shfl_down_sync(full, v[c], d);
            if (lane + d <= end) v[c] += o;
        }
    }
    if (head && key >= 0) {
        const size_t plane = a.plane;
        if (SHAPE == QS_SHAPE_NGP) {
            const size_t n = (size_t)key;
#pragma unroll
            for (int qq = 0; qq < 4; qq++) atomicAdd(a.dep + qq * plane + n, v[qq]);
        } else {
            const int fj = key % My, fk = key / My;
            const int j1 = wrap_idx(fj + 1, My), k1 = wrap_idx(fk + 1, Mz);
            const size_t nn[4] = {(size_t)fj + (size_t)My * fk, (size_t)j1 + (size_t)My * fk,
                                  (size_t)fj + (size_t)My * k1, (size_t)j1 + (size_t)My * k1};
#pragma unroll
            for (int cnr = 0; cnr < 4; cnr++)
#pragma unroll
                for (int qq = 0; qq < 4; qq++)
                    atomicAdd(a.dep + qq * plane + nn[cnr], v[cnr * 4 + qq]);
        }
    }
}

// ---------------------------------------------------------------------------
// FP32 NGP push, one thread per cell, for the uniform lattice layout
// (particle p of the layer sits in cell p / PPC): in the live reference path a
// particle never leaves its seeded cell, so this layout is permanent.  The
// cell's fields are gathered once, its PPC particles are read and written as
// float4 vectors, deposits into the cell itself are summed in registers and
// flushed with 4 atomics; deposits that land in another cell go straight to
// global atomics.  Same physics as push_kernel<float, NGP, precise, fast>,
// with approximate reciprocals (a few ulp) for the divisions.
template <int PPC>
__global__ void __launch_bounds__(128) push_cell_kernel(PushArgs<float> a) {
    static_assert(PPC == 4, "float4 particle vectors");
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    const int My = a.My, Mz = a.Mz;
    if (cell >= My * Mz) return;
    pdl_wait();
    int j, k;
    cell_jk(cell, My, a.invMy, j, k);
    const size_t plane = a.plane;
    const size_t n = (size_t)cell;
    const float ex0 = 0.5f * (ld(a.P + 0 * plane + n) + ld(a.C + 0 * plane + n));
    const float ey0 = 0.5f * (ld(a.P + 1 * plane + n) + ld(a.C + 1 * plane + n));
    const float ez0 = 0.5f * (ld(a.P + 2 * plane + n) + ld(a.C + 2 * plane + n));
    const float bx0 = 0.5f * (ld(a.P + 3 * plane + n) + ld(a.C + 3 * plane + n)) + a.bxe;
    const float by0 = 0.5f * (ld(a.P + 4 * plane + n) + ld(a.C + 4 * plane + n)) + a.bye;
    const float bz0 = 0.5f * (ld(a.P + 5 * plane + n) + ld(a.C + 5 * plane + n)) + a.bze;
    const size_t base = (size_t)cell * PPC;
    float4 Y = *(const float4*)(a.y + base), Z = *(const float4*)(a.z + base);
    float4 PX = *(const float4*)(a.px + base), PY = *(const float4*)(a.py + base);
    float4 PZ = *(const float4*)(a.pz + base);
    const float4 W = *(const float4*)(a.w + base);
    float* yv = &Y.x; float* zv = &Z.x; float* pxv = &PX.x; float* pyv = &PY.x;
    float* pzv = &PZ.x; const float* wv = &W.x;
    float own0 = 0.f, own1 = 0.f, own2 = 0.f, own3 = 0.f;
#pragma unroll
    for (int q = 0; q < PPC; q++) {
        const float yp = yv[q], zp = zv[q];
        if (!(yp >= 0.f && yp <= 1.f && zp >= 0.f && zp <= 1.f)) {
            atomicOr(a.err, DEV_ERR_RANGE);
            continue;
        }
        float px = pxv[q], py = pyv[q], pz = pzv[q];
        const float inv_gp = rsqrtf(1.f + px * px + py * py + pz * pz);
        const float Vyp = py * inv_gp, Vzp = pz * inv_gp;
        const float omp = one_minus_vx(px, py, pz, inv_gp);   // 1 - Vx before the kick
        const float kE = a.sE * rcp_approx(omp);
        const float ex = ex0 * kE, ey = ey0 * kE, ez = ez0 * kE;
        px += ex; py += ey; pz += ez;
        const float kB = rsqrtf(1.f + px * px + py * py + pz * pz) * kE;
        const float bx = bx0 * kB, by = by0 * kB, bz = bz0 * kB;
        const float co = __fdividef(2.f, 1.f + bx * bx + by * by + bz * bz);
        const float p3x = (py * bz - pz * by + px) * co;
        const float p3y = (pz * bx - px * bz + py) * co;
        const float p3z = (px * by - py * bx + pz) * co;
        px += ex + (p3y * bz - p3z * by);
        py += ey + (p3z * bx - p3x * bz);
        pz += ez + (p3x * by - p3y * bx);
        const float inv_g = rsqrtf(1.f + px * px + py * py + pz * pz);
        const float Vxm = px * inv_g, Vym = py * inv_g, Vzm = pz * inv_g;
        const float Vy = 0.5f * (Vym + Vyp), Vz = 0.5f * (Vzm + Vzp);
        const float inv2 = rcp_approx(0.5f * (one_minus_vx(px, py, pz, inv_g) + omp));
        const float wq = wv[q] * inv2;
        const float djx = wq * a.djx0 * Vxm, djy = wq * a.djy0 * Vym, djz = wq * a.djz0 * Vzm;
        const float drho = wq * a.drho0;
        const float dy = Vy * a.hxhy * inv2, dz = Vz * a.hxhz * inv2;
        float partdx = 0.f, step = 1.f;
        if (fabsf(dy) > 1.f || fabsf(dz) > 1.f) step = partdx = fmaxf(fabsf(dy), fabsf(dz));
        if (partdx < 1.f) partdx = step = 1.f;
        float ytmp = yp, ztmp = zp;
        while (partdx > 0.f) {
            float ps;
            if (partdx > 1.f) { partdx -= 1.f; ps = rcp_approx(step); }
            else { ps = __fdividef(partdx, step); partdx = 0.f; }
            // cell-relative update; the base cell stays the seeded cell (the
            // reference adds the outer j_jump = j at every sub-step)
            const float uy = ytmp + dy * ps, uz = ztmp + dz * ps;
            const float fy = floorf(uy), fz = floorf(uz);
            float ry = uy - fy, rz = uz - fz;
            int sy = (int)fy, sz = (int)fz;
            if (ry >= 1.f) { ry = 0.f; sy += 1; }
            if (rz >= 1.f) { rz = 0.f; sz += 1; }
            ytmp = ry;
            ztmp = rz;
            const float d0 = djx * ps, d1 = djy * ps, d2 = djz * ps, d3 = drho * ps;
            if (sy == 0 && sz == 0) {
                own0 += d0; own1 += d1; own2 += d2; own3 += d3;
            } else {
                const int jj = wrap_idx(j + sy, My), kk = wrap_idx(k + sz, Mz);
                const size_t m = (size_t)jj + (size_t)My * kk;
                atomicAdd(a.dep + 0 * plane + m, d0);
                atomicAdd(a.dep + 1 * plane + m, d1);
                atomicAdd(a.dep + 2 * plane + m, d2);
                atomicAdd(a.dep + 3 * plane + m, d3);
            }
        }
        yv[q] = ytmp; zv[q] = ztmp; pxv[q] = px; pyv[q] = py; pzv[q] = pz;
    }
    pdl_trigger();
    atomicAdd(a.dep + 0 * plane + n, own0);
    atomicAdd(a.dep + 1 * plane + n, own1);
    atomicAdd(a.dep + 2 * plane + n, own2);
    atomicAdd(a.dep + 3 * plane + n, own3);
    if (a.full) {
        *(float4*)(a.y + base) = Y; *(float4*)(a.z + base) = Z;
        *(float4*)(a.px + base) = PX; *(float4*)(a.py + base) = PY;
        *(float4*)(a.pz + base) = PZ;
    }
}

// ---------------------------------------------------------------------------
// CIC push over particles grouped by cell (the counting sort in sort.cu
// regroups them every few full pushes), FP32, or FP64 with FMA contraction
// for the FP64 path on FFT transforms.  A block owns a tile of 32 x TY cells
// and stages the fields (P and C averaged) of the tile's cells and the cells
// around them in shared memory for the gather.  A warp owns one row of 32
// cells for the whole launch and lane l owns cell c0 + l.  The row's
// particles are processed in windows of WIN slots:
//  - phase 1, particle-parallel (lane = particle, the next one prefetched):
//    the push; the first sub-step's charges q = dq * ps, its in-cell position
//    and its cell (and the final cell) are staged in shared memory, further
//    sub-steps (|dy| or |dz| above a cell, rare) deposit by global atomics;
//  - phase 2, cell-parallel (lane = cell): each lane walks the slots of its
//    own cell inside the window (regrouped, they are [offset(c),
//    offset(c + 1))), rebuilds the 4 corner weights and adds the 4 x ND
//    corner values to registers.  A particle whose first sub-step ended in
//    another cell (it moved since the last regrouping) is added by global
//    atomics instead; on a full push followed by a regrouping the lane counts
//    the particles that stay in its cell and adds one count per cell.
// No shuffles or matches sum the deposits.  At the end each lane spreads its
// cell's corner sums (the right-hand corners through a shuffle to the next
// lane), the warps combine their rows in the block tile in two ordered phases,
// and the tile is flushed, times the species' charge factors, with one global
// atomic per touched cell and current.  The staged fields reach one cell around
// the tile, for particles that moved there since the regrouping; the few
// beyond read the fields from global memory.  ND = 3
// leaves out the density deposit, which the march does not read.  The full
// push stores the particles in place with their new cell.  Same physics
// as push_kernel<T, CIC, precise, fast> (movepart_layer_CIC.cpp:165-193,
// 449-496 weights), the divisions factored into reciprocals.
//
// What bounds it: instruction issue (a half push of 1,048,576 particles at
// 512 x 512 issues 13.6 M warp instructions, two thirds of the issue slots)
// and the dependent loads at a block's start.  Against the form with floor(),
// divided cell indices, unshared 1 + p^2 and one staged word per value
// (15.1 M instructions, 64 registers): 103.8 -> 98.3 us per layer of the warm
// 512 x 512 x 1024 march, 407 -> 398 us at 1024 x 1024, 190.7 -> 186.3 us in
// FP64.  72 registers, 7 blocks per SM; capped at 64 registers the spills cost
// more than the eighth block gives (105.0 us).  The cells around the tile, and
// 32-bit offsets: 95.3 -> 93.2 us, 256 x 256 adjoint 86.7 -> 85.6 us, 1024 x 1024
// 349 -> 346 us; the head of the box, where few particles have moved, would be
// 81.5 without those cells and is 82.2.
template <class T>
__device__ __forceinline__ int cell_offset(const PushArgs<T>& a, int c) {
    return a.loff[c] + a.bpref[c >> 10];
}

// the reciprocal forms of the grouped push: approximate in FP32, IEEE in FP64
template <class T>
struct RowMath;
template <>
struct RowMath<float> {
    static __device__ __forceinline__ float rsq(float x) { return rsq_approx(x); }
    static __device__ __forceinline__ float rcp(float x) { return rcp_approx(x); }
    static __device__ __forceinline__ float twice_rcp(float x) { return 2.f * rcp_approx(x); }
    static __device__ __forceinline__ float div(float a, float b) { return __fdividef(a, b); }
};
template <>
struct RowMath<double> {
    static __device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
    static __device__ __forceinline__ double rcp(double x) { return 1.0 / x; }
    static __device__ __forceinline__ double twice_rcp(double x) { return 2.0 / x; }
    static __device__ __forceinline__ double div(double a, double b) { return a / b; }
};

// one CIC sub-step of a particle (cell-relative move from base cell (jb, kb),
// periodic wrap, the 4 corner weights of the new position)
template <class T>
__device__ __forceinline__ void cic_substep(T dy, T dz, T ps, T& ytmp, T& ztmp, int& jb, int& kb,
                                            int My, int Mz, T (&wc)[4]) {
    const T one = T(1);
    const T uy = ytmp + dy * ps, uz = ztmp + dz * ps;
    const T fy = floor_t<T>(uy), fz = floor_t<T>(uz);
    T ry = uy - fy, rz = uz - fz;
    int sy = (int)fy, sz = (int)fz;
    if (ry >= one) { ry = T(0); sy += 1; }
    if (rz >= one) { rz = T(0); sz += 1; }
    jb = wrap1(jb + sy, My);   // |dy * ps| <= 1: the shift is at most one cell
    kb = wrap1(kb + sz, Mz);
    ytmp = ry;
    ztmp = rz;
    wc[0] = (one - ry) * (one - rz);
    wc[1] = ry * (one - rz);
    wc[2] = (one - ry) * rz;
    wc[3] = ry * rz;
}

// Element i of an array.  In FP32 by a 32-bit byte offset from its base (Off =
// unsigned): one address operand for all arrays of a particle or all planes of
// a node, 95.3 -> 93.2 us per layer of the warm 512 x 512 march.  In FP64, whose
// registers are full, the plain form (180.7 us against 183.9), and so for FP32
// arrays of 4 GB and more (WIDE, chosen by the launch), which a byte offset
// does not reach.
template <class T, bool WIDE>
using RowOff = std::conditional_t<sizeof(T) == 4 && !WIDE, unsigned, size_t>;
template <class Off, class U>
__device__ __forceinline__ U* at32(U* base, Off i) {
    if constexpr (sizeof(Off) == 4) {
        static_assert(sizeof(U) == 4);
        using B = std::conditional_t<std::is_const_v<U>, const char, char>;
        return reinterpret_cast<U*>(reinterpret_cast<B*>(base) + i * 4u);
    } else {
        return base + i;
    }
}

// (j, k) of a cell, and an index wrapped into its period: bit operations when
// the sizes are powers of two (P2), else the general forms
template <bool P2, class T>
__device__ __forceinline__ void split_cell(const PushArgs<T>& a, int cell, int& j, int& k) {
    if constexpr (P2) {
        j = cell & (a.My - 1);
        k = cell >> a.lgMy;
    } else {
        cell_jk(cell, a.My, a.invMy, j, k);
    }
}
template <bool P2>
__device__ __forceinline__ int wrap_p(int j, int M) {
    if constexpr (P2) return j & (M - 1);
    else return wrap1(j, M);
}

// One axis of a move by d, |d| <= 1, from y in [0, 1]: the in-cell position
// and the cell shift.  u = y + d lies in [-1, 2], so that floor(u) is two
// comparisons (floor and the conversion to int run at a quarter of their
// rate); a position that rounds to 1 belongs to the next cell.
template <class T>
__device__ __forceinline__ T move_axis(T y, T d, int& s) {
    const T u = y + d;
    const bool up = u >= T(1), dn = u < T(0);
    T r = up ? u - T(1) : u;
    r = dn ? u + T(1) : r;
    s = (up ? 1 : 0) - (dn ? 1 : 0);
    if (r >= T(1)) {
        r = T(0);
        s += 1;
    }
    return r;
}

// The deposits staged between the two phases of the grouped push, one slot
// per particle of a warp's window: the charges q, the in-cell position and the
// cell of the first sub-step.  In FP32 without the density two vector words,
// so that a slot costs two stores and two loads instead of six; lanes of
// phase 2 read slots about ppc apart, and one pad word per 8 slots of 16
// bytes (per 16 slots of 8 bytes) puts these on distinct banks.  The other
// variants keep one array per value, with one pad per 32 slots.
template <class T, int ND, int WIN>
struct DepositStage {
    T v[ND + 2][WIN + WIN / 32];
    int key[WIN + WIN / 32];
    __device__ __forceinline__ void put(int s, const T (&q)[ND], T ry, T rz, int k) {
        const int p = s + (s >> 5);
#pragma unroll
        for (int d = 0; d < ND; d++) v[d][p] = q[d];
        v[ND][p] = ry;
        v[ND + 1][p] = rz;
        key[p] = k;
    }
    __device__ __forceinline__ int get(int s, T (&q)[ND], T& ry, T& rz) const {
        const int p = s + (s >> 5);
#pragma unroll
        for (int d = 0; d < ND; d++) q[d] = v[d][p];
        ry = v[ND][p];
        rz = v[ND + 1][p];
        return key[p];
    }
};
template <int WIN>
struct DepositStage<float, 3, WIN> {
    float4 a[WIN + WIN / 8];
    float2 b[WIN + WIN / 16];
    __device__ __forceinline__ void put(int s, const float (&q)[3], float ry, float rz, int k) {
        a[s + (s >> 3)] = make_float4(q[0], q[1], q[2], ry);
        b[s + (s >> 4)] = make_float2(rz, __int_as_float(k));
    }
    __device__ __forceinline__ int get(int s, float (&q)[3], float& ry, float& rz) const {
        const float4 x = a[s + (s >> 3)];
        const float2 y = b[s + (s >> 4)];
        q[0] = x.x; q[1] = x.y; q[2] = x.z;
        ry = x.w;
        rz = y.x;
        return __float_as_int(y.y);
    }
};

// A particle's momentum through the gathered fields g, and its move: the
// velocity after the push, the weight over 1 - Vx (wq), the move (dy, dz) in
// cells, and its first sub-step (dy1, dz1) of at most one cell with the share
// wf of wq; partdx is what remains of a move of more than one cell, whose
// full sub-steps cover 1/step.
template <class T>
struct PushStep {
    T Vx, Vy, Vz, wq, wf, dy, dz, dy1, dz1, partdx, step;
};
template <class T>
__device__ __forceinline__ PushStep<T> push_step(const PushArgs<T>& a, const T (&g)[6], T w,
                                                 T& px, T& py, T& pz) {
    using M = RowMath<T>;
    const T one = T(1), half = T(0.5);
    PushStep<T> u;
    T inv_gp, omp;                            // 1 - Vx before the kick
    vel_terms(px, py, pz, inv_gp, omp);
    const T Vyp = py * inv_gp, Vzp = pz * inv_gp;
    const T kE = a.sE * M::rcp(omp);
    const T ex = g[0] * kE, ey = g[1] * kE, ez = g[2] * kE;
    px += ex; py += ey; pz += ez;
    const T kB = M::rsq(one + px * px + py * py + pz * pz) * kE;
    const T bx = (g[3] + a.bxe) * kB, by = (g[4] + a.bye) * kB, bz = (g[5] + a.bze) * kB;
    const T co = M::twice_rcp(one + bx * bx + by * by + bz * bz);
    const T p3x = (py * bz - pz * by + px) * co;
    const T p3y = (pz * bx - px * bz + py) * co;
    const T p3z = (px * by - py * bx + pz) * co;
    px += ex + (p3y * bz - p3z * by);
    py += ey + (p3z * bx - p3x * bz);
    pz += ez + (p3x * by - p3y * bx);
    T inv_g, omm;
    vel_terms(px, py, pz, inv_g, omm);
    u.Vx = px * inv_g;
    u.Vy = py * inv_g;
    u.Vz = pz * inv_g;
    const T inv2 = M::rcp(half * (omm + omp));
    const T hinv = half * inv2;
    u.wf = u.wq = w * inv2;
    u.dy1 = u.dy = (u.Vy + Vyp) * (a.hxhy * hinv);
    u.dz1 = u.dz = (u.Vz + Vzp) * (a.hxhz * hinv);
    const T ady = fabs_t(u.dy), adz = fabs_t(u.dz);
    const T mx = ady > adz ? ady : adz;
    u.partdx = T(0);
    u.step = one;
    if (mx > one) {
        u.step = mx;
        u.partdx = mx - one;
        const T ps = M::rcp(mx);
        u.wf = u.wq * ps;
        // the larger share may round to a little over one cell
        u.dy1 = min(max(u.dy * ps, -one), one);
        u.dz1 = min(max(u.dz * ps, -one), one);
    }
    return u;
}

template <int TY, int ND, int WIN, bool P2, class T, bool WIDE = false>
__global__ void __launch_bounds__(32 * TY) push_cic_row_kernel(PushArgs<T> a) {
    using M = RowMath<T>;
    using FP = FPair<T>;
    using P2T = typename FP::type;
    constexpr int TX = 32, W = TX + 1, H = TY + 1;
    constexpr int GW = TX + 3, GH = TY + 3;   // nodes of the tile's cells and their neighbours
    static_assert(WIN % 32 == 0, "whole warps per window");
    const T one = T(1), zero = T(0), half = T(0.5);
    __shared__ P2T Fs[3][GH][GW];        // field pairs (P, C averaged) of the tile's cells and one
                                         // cell around them
    __shared__ T Tt[ND][H][W];           // block deposit tile [current][row][col]
    __shared__ DepositStage<T, ND, WIN> S[TY];   // staged deposits of each warp's window
    __shared__ int Kl[TY][WIN + WIN / 32];       // counting push: the final cells
    const int lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
    const int My = a.My, Mz = a.Mz;
    using Off = RowOff<T, WIDE>;
    const Off plane = (Off)a.plane;
    const int tiles_x = My / TX;
    const int j0 = (blockIdx.x % tiles_x) * TX, k0 = (blockIdx.x / tiles_x) * TY;
    const int c0 = j0 + My * (k0 + wr);   // this warp's 32 cells: c0 .. c0+31
    const int mycell = c0 + lane;
    QS_TRACE_ENTRY();
    // The offsets and then the first particles are two dependent loads: they
    // go first, and the fields' loads and the block's barrier overlap them.
    // In the march nothing since the kernel before last writes them, so they
    // need not wait for the kernel in front either.
    if (!a.early) pdl_wait();
    // (offsets out of step with the arrays, which the regrouping reports, stay
    // inside them)
    const int lo = min(cell_offset(a, mycell), (int)a.n);
    const int hi = (Off)(mycell + 1) < plane ? min(cell_offset(a, mycell + 1), (int)a.n) : (int)a.n;
    for (int i = threadIdx.x; i < ND * H * W; i += 32 * TY) (&Tt[0][0][0])[i] = zero;
    const int pbeg = __shfl_sync(0xffffffffu, lo, 0);
    const int pend = __shfl_sync(0xffffffffu, hi, 31);
    // the particle of the next pass is loaded while this one is pushed
    int nx_cell = 0;
    T nx_y = zero, nx_z = zero, nx_px = zero, nx_py = zero, nx_pz = zero, nx_w = zero;
    if (pbeg + lane < pend) {
        const Off q = pbeg + lane;
        nx_cell = *at32<Off>(a.cell, q); nx_y = *at32<Off>(a.y, q); nx_z = *at32<Off>(a.z, q);
        nx_px = *at32<Off>(a.px, q); nx_py = *at32<Off>(a.py, q); nx_pz = *at32<Off>(a.pz, q);
        nx_w = *at32<Off>(a.w, q);
    }
    if (a.early) pdl_wait();
    QS_TRACE_WAITED();
    const bool one_set = a.P == a.C;     // an averaged set: (x + x) / 2 = x
    {
        int r = threadIdx.x / GW, cc = threadIdx.x - r * GW;
        for (int i = threadIdx.x; i < GH * GW; i += 32 * TY) {
            const Off m = (Off)wrap_p<P2>(j0 + cc - 1, My) + (Off)My * wrap_p<P2>(k0 + r - 1, Mz);
            if (one_set) {
#pragma unroll
                for (int q = 0; q < 3; q++)
                    Fs[q][r][cc] = FP::make(ld(at32<Off>(a.C + 2 * q * plane, m)),
                                            ld(at32<Off>(a.C + (2 * q + 1) * plane, m)));
            } else {
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const P2T pp = FP::make(ld(at32<Off>(a.P + 2 * q * plane, m)),
                                            ld(at32<Off>(a.P + (2 * q + 1) * plane, m)));
                    const P2T cp = FP::make(ld(at32<Off>(a.C + 2 * q * plane, m)),
                                            ld(at32<Off>(a.C + (2 * q + 1) * plane, m)));
                    Fs[q][r][cc] = FP::mul(half, FP::add(pp, cp));
                }
            }
            cc += (32 * TY) % GW;      // the node 32 * TY further
            r += (32 * TY) / GW;
            if (cc >= GW) { cc -= GW; r += 1; }
        }
    }
    __syncthreads();
    // the tile's own cells of the gathered fields, for the push adjoint (the
    // march, which skips the density deposit, is what the adjoint recomputes)
    if constexpr (ND == 3)
        if (a.favg)
            for (int i = threadIdx.x; i < TY * TX; i += 32 * TY) {
                const int r = i / TX, cc = i - r * TX;
                const Off m = (Off)(j0 + cc) + (Off)My * (k0 + r);
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    a.favg[2 * q * plane + m] = Fs[q][r + 1][cc + 1].x;
                    a.favg[(2 * q + 1) * plane + m] = Fs[q][r + 1][cc + 1].y;
                }
            }
    const bool count = a.full && a.cnt;
    int stay = 0;                        // particles that end the full push in mycell
    const T dj[4] = {a.djx0, a.djy0, a.djz0, a.drho0};   // the species' factor of each current
    // the cell's sums of current d (without dj) at its corners (0, 1) and (2, 3)
    P2T acc[ND][2];
#pragma unroll
    for (int d = 0; d < ND; d++) acc[d][0] = acc[d][1] = FP::make(zero, zero);
    // the 4 corners of cell (jc, kc) get q[d] * dj[d] * weight by global atomics
    auto scatter = [&](int jc, int kc, const T (&q)[ND], const T (&wc)[4]) {
        const int jc1 = wrap_p<P2>(jc + 1, My), kc1 = wrap_p<P2>(kc + 1, Mz);
        const Off nd[4] = {(Off)(jc + My * kc), (Off)(jc1 + My * kc), (Off)(jc + My * kc1),
                           (Off)(jc1 + My * kc1)};
#pragma unroll
        for (int d = 0; d < ND; d++) {
            const T x = q[d] * dj[d];
#pragma unroll
            for (int r = 0; r < 4; r++) atomicAdd(at32<Off>(a.dep + d * plane, nd[r]), x * wc[r]);
        }
    };
    for (int wbase = pbeg; wbase < pend; wbase += WIN) {
        const int wend = min(pend, wbase + WIN);
        // phase 1: lane = particle
        for (int base = wbase; base < wend; base += 32) {
            const int p = base + lane;
            const int cell = nx_cell;
            const T yp = nx_y, zp = nx_z, w = nx_w;
            T px = nx_px, py = nx_py, pz = nx_pz;
            if (p + 32 < pend) {
                const Off q = p + 32;
                nx_cell = *at32<Off>(a.cell, q); nx_y = *at32<Off>(a.y, q); nx_z = *at32<Off>(a.z, q);
                nx_px = *at32<Off>(a.px, q); nx_py = *at32<Off>(a.py, q); nx_pz = *at32<Off>(a.pz, q);
                nx_w = *at32<Off>(a.w, q);
            }
            int key = -1, last = cell;
            T qv[ND], ay = zero, az = zero;
#pragma unroll
            for (int d = 0; d < ND; d++) qv[d] = zero;
            if (p < pend) {
                if (!(yp >= zero && yp <= one && zp >= zero && zp <= one)) {
                    atomicOr(a.err, DEV_ERR_RANGE);   // no deposit; it stays in its cell
                } else {
                    int j, k;
                    split_cell<P2>(a, cell, j, k);
                    const T wg[4] = {(one - yp) * (one - zp), yp * (one - zp), (one - yp) * zp,
                                     yp * zp};
                    T g[6];
                    // the particle's node in the tile (moved since the regrouping,
                    // it may sit in a cell around the tile's own)
                    int tj = j - j0 + 1, tk = k - k0 + 1;
                    if constexpr (P2) {   // across the periodic edge too
                        tj &= My - 1;
                        tk &= Mz - 1;
                    }
                    if ((unsigned)tj < TX + 2 && (unsigned)tk < TY + 2) {
#pragma unroll
                        for (int q = 0; q < 3; q++) {
                            P2T gq = FP::mul(wg[0], Fs[q][tk][tj]);
                            gq = FP::fma(wg[1], Fs[q][tk][tj + 1], gq);
                            gq = FP::fma(wg[2], Fs[q][tk + 1][tj], gq);
                            gq = FP::fma(wg[3], Fs[q][tk + 1][tj + 1], gq);
                            g[2 * q] = gq.x;
                            g[2 * q + 1] = gq.y;
                        }
                    } else {
                        const int j1 = wrap_p<P2>(j + 1, My), k1 = wrap_p<P2>(k + 1, Mz);
                        const Off nn[4] = {(Off)(j + My * k), (Off)(j1 + My * k),
                                           (Off)(j + My * k1), (Off)(j1 + My * k1)};
#pragma unroll
                        for (int f = 0; f < 6; f++) {
                            T s = zero;
#pragma unroll
                            for (int r = 0; r < 4; r++)
                                s += wg[r] * half * (ld(at32<Off>(a.P + f * plane, nn[r])) +
                                                     ld(at32<Off>(a.C + f * plane, nn[r])));
                            g[f] = s;
                        }
                    }
                    const PushStep<T> u = push_step(a, g, w, px, py, pz);
                    const T dy = u.dy, dz = u.dz, wq = u.wq;
                    T partdx = u.partdx;
                    // first sub-step: staged for the cell-parallel sum
                    int sy, sz;
                    ay = move_axis(yp, u.dy1, sy);
                    az = move_axis(zp, u.dz1, sz);
                    int jb = wrap_p<P2>(j + sy, My), kb = wrap_p<P2>(k + sz, Mz);
                    key = jb + My * kb;
                    qv[0] = u.wf * u.Vx;
                    qv[1] = u.wf * u.Vy;
                    qv[2] = u.wf * u.Vz;
                    if constexpr (ND == 4) qv[3] = u.wf;
                    T ytmp = ay, ztmp = az;
                    // further sub-steps: direct atomics
                    while (partdx > zero) {
                        T ps;
                        if (partdx > one) { partdx -= one; ps = M::rcp(u.step); }
                        else { ps = M::div(partdx, u.step); partdx = zero; }
                        T wc[4];
                        cic_substep<T>(dy, dz, ps, ytmp, ztmp, jb, kb, My, Mz, wc);
                        T qs[ND] = {wq * ps * u.Vx, wq * ps * u.Vy, wq * ps * u.Vz};
                        if constexpr (ND == 4) qs[3] = wq * ps;
                        scatter(jb, kb, qs, wc);
                    }
                    last = jb + My * kb;
                    if (a.full) {
                        const Off q = p;
                        *at32<Off>(a.y, q) = ytmp; *at32<Off>(a.z, q) = ztmp; *at32<Off>(a.px, q) = px;
                        *at32<Off>(a.py, q) = py; *at32<Off>(a.pz, q) = pz;
                        *at32<Off>(a.cell_out, q) = last;
                    }
                }
            }
            const int s = base - wbase + lane;
            S[wr].put(s, qv, ay, az, key);
            if (count) Kl[wr][s + (s >> 5)] = last;
        }
        __syncwarp();
        // phase 2: lane = cell.  Particles that left the cell are noted and
        // added by global atomics in a loop of their own, which runs as often
        // as the lane with the most of them needs, not in every pass where
        // one lane has one.
        const int qa = max(lo, wbase), qb = min(hi, wend);
        unsigned moved = 0;
        auto add_moved = [&](int s) {
            T qv[ND], ry, rz;
            const int key = S[wr].get(s, qv, ry, rz);
            const T wc[4] = {(one - ry) * (one - rz), ry * (one - rz), (one - ry) * rz, ry * rz};
            int kj, kk;
            split_cell<P2>(a, key, kj, kk);
            scatter(kj, kk, qv, wc);
        };
        for (int q = qa; q < qb; q++) {
            const int s = q - wbase;
            T qv[ND], ry, rz;
            const int key = S[wr].get(s, qv, ry, rz);
            if (count) {
                const int last = Kl[wr][s + (s >> 5)];
                if (last == mycell) stay++;
                else atomicAdd(a.cnt + last, 1);
            }
            if (key == mycell) {
                // corner weights in pairs: (1 - rz) (1 - ry, ry) and rz (1 - ry, ry)
                const P2T wy = FP::make(one - ry, ry);
                const P2T w01 = FP::mul(one - rz, wy), w23 = FP::mul(rz, wy);
#pragma unroll
                for (int d = 0; d < ND; d++) {
                    acc[d][0] = FP::fma(qv[d], w01, acc[d][0]);
                    acc[d][1] = FP::fma(qv[d], w23, acc[d][1]);
                }
            } else if (key >= 0) {
                if (q - qa < 32) moved |= 1u << (q - qa);
                else add_moved(s);
            }
        }
        while (moved) {
            const int b = __ffs(moved) - 1;
            moved &= moved - 1;
            add_moved(qa + b - wbase);
        }
        __syncwarp();
    }
    if (stay) atomicAdd(a.cnt + mycell, stay);
    pdl_trigger();
    // spread the per-cell sums to the corners: the lane of cell (l, row) owns
    // column l of rows row and row+1; the right-hand corners go to lane l+1
    const unsigned full = 0xffffffffu;
    T row0[ND], row1[ND], edge0[ND], edge1[ND];
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const T c00 = acc[d][0].x, c10 = acc[d][0].y;
        const T c01 = acc[d][1].x, c11 = acc[d][1].y;
        const T l10 = __shfl_up_sync(full, c10, 1), l11 = __shfl_up_sync(full, c11, 1);
        row0[d] = c00 + (lane > 0 ? l10 : zero);
        row1[d] = c01 + (lane > 0 ? l11 : zero);
        edge0[d] = c10;   // used by lane 31 only: column 32
        edge1[d] = c11;
    }
#pragma unroll
    for (int d = 0; d < ND; d++) {
        Tt[d][wr][lane] += row0[d];
        if (lane == 31) Tt[d][wr][TX] += edge0[d];
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < ND; d++) {
        Tt[d][wr + 1][lane] += row1[d];
        if (lane == 31) Tt[d][wr + 1][TX] += edge1[d];
    }
    __syncthreads();
    int fr = threadIdx.x / W, fc = threadIdx.x - fr * W;
    for (int i = threadIdx.x; i < H * W; i += 32 * TY) {
        const Off m = (Off)wrap_p<P2>(j0 + fc, My) + (Off)My * wrap_p<P2>(k0 + fr, Mz);
#pragma unroll
        for (int d = 0; d < ND; d++) {
            const T x = Tt[d][fr][fc];
            if (x != zero) atomicAdd(at32<Off>(a.dep + d * plane, m), dj[d] * x);
        }
        fc += (32 * TY) % W;
        fr += (32 * TY) / W;
        if (fc >= W) { fc -= W; fr += 1; }
    }
    QS_TRACE_END(a.full ? trace::K_PUSH_FULL : trace::K_PUSH_HALF);
}

// The full push's move alone, one thread per particle, from the arrays of one
// layer's entry state to those of the next: the adjoint's recomputation, which
// needs the particles and no deposit.  The fields are one gathered set (a.C,
// the march's own), read through L1 (the particles are grouped by cell), and
// the arithmetic is push_step, the row kernel's.  In its place the row push
// with its unread deposit and a copy of the state took 11.2 + 6.3 us at 256 x
// 256 (262,144 particles); this takes 7.1 us (cold).
template <bool P2, class T>
__global__ void __launch_bounds__(128) move_cic_kernel(PushArgs<T> a) {
    using M = RowMath<T>;
    using FP = FPair<T>;
    using P2T = typename FP::type;
    const T one = T(1), zero = T(0);
    const int My = a.My, Mz = a.Mz;
    const size_t plane = a.plane;
    pdl_wait();
    const int p = blockIdx.x * 128 + threadIdx.x;
    pdl_trigger();
    if (p >= a.n) return;
    const int cell = a.cell[p];
    T y = a.y[p], z = a.z[p], px = a.px[p], py = a.py[p], pz = a.pz[p];
    int jb, kb;
    split_cell<P2>(a, cell, jb, kb);
    if (y >= zero && y <= one && z >= zero && z <= one) {   // else it stays as it is
        const int j1 = wrap_p<P2>(jb + 1, My), k1 = wrap_p<P2>(kb + 1, Mz);
        const int nn[4] = {jb + My * kb, j1 + My * kb, jb + My * k1, j1 + My * k1};
        const T wg[4] = {(one - y) * (one - z), y * (one - z), (one - y) * z, y * z};
        T g[6];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const T *f0 = a.C + 2 * q * plane, *f1 = f0 + plane;
            P2T gq = FP::mul(wg[0], FP::make(ld(f0 + nn[0]), ld(f1 + nn[0])));
#pragma unroll
            for (int r = 1; r < 4; r++)
                gq = FP::fma(wg[r], FP::make(ld(f0 + nn[r]), ld(f1 + nn[r])), gq);
            g[2 * q] = gq.x;
            g[2 * q + 1] = gq.y;
        }
        const PushStep<T> u = push_step(a, g, one, px, py, pz);
        int sy, sz;
        y = move_axis(y, u.dy1, sy);
        z = move_axis(z, u.dz1, sz);
        jb = wrap_p<P2>(jb + sy, My);
        kb = wrap_p<P2>(kb + sz, Mz);
        T partdx = u.partdx;
        while (partdx > zero) {
            T ps;
            if (partdx > one) { partdx -= one; ps = M::rcp(u.step); }
            else { ps = M::div(partdx, u.step); partdx = zero; }
            T wc[4];
            cic_substep<T>(u.dy, u.dz, ps, y, z, jb, kb, My, Mz, wc);
        }
    } else {
        atomicOr(a.err, DEV_ERR_RANGE);
    }
    a.y_out[p] = y; a.z_out[p] = z; a.px_out[p] = px; a.py_out[p] = py; a.pz_out[p] = pz;
    a.cell_out[p] = jb + My * kb;
}

template <class T>
int launch_move(const PushArgs<T>& a, cudaStream_t st) {
    const dim3 grid((unsigned)((a.n + 127) / 128));
    if (a.lgMy >= 0) launch_pdl(move_cic_kernel<true, T>, grid, dim3(128), 0, st, a);
    else launch_pdl(move_cic_kernel<false, T>, grid, dim3(128), 0, st, a);
    return 1;
}

// the grouped CIC push (both widths): 0 when the layout does not fit it
template <class T>
int launch_push_rows(const PushArgs<T>& a, cudaStream_t st) {
    constexpr int TY = 4, WIN = 128;
    if (a.move_only) return launch_move(a, st);
    if (!a.loff || a.dep_cell) return 0;   // grouped by cell with offsets (the engine checks the shape)
    const dim3 grid((a.My / 32) * (a.Mz / TY));
    const dim3 block(32 * TY);
    // FP32's 32-bit byte offsets reach arrays below 4 GB
    if constexpr (sizeof(T) == 4)
        if ((uint64_t)a.n >= (1ull << 30) || (uint64_t)a.plane >= (1ull << 30)) {
            if (a.skip_dens)
                launch_pdl(push_cic_row_kernel<TY, 3, WIN, false, T, true>, grid, block, 0, st, a);
            else
                launch_pdl(push_cic_row_kernel<TY, 4, WIN, false, T, true>, grid, block, 0, st, a);
            return 1;
        }
    if (a.skip_dens) {
        if (a.lgMy >= 0) launch_pdl(push_cic_row_kernel<TY, 3, WIN, true, T>, grid, block, 0, st, a);
        else launch_pdl(push_cic_row_kernel<TY, 3, WIN, false, T>, grid, block, 0, st, a);
    } else {
        if (a.lgMy >= 0) launch_pdl(push_cic_row_kernel<TY, 4, WIN, true, T>, grid, block, 0, st, a);
        else launch_pdl(push_cic_row_kernel<TY, 4, WIN, false, T>, grid, block, 0, st, a);
    }
    return 1;
}

int launch_push_rows_f64(const PushArgs<double>& a, cudaStream_t st);   // push_f64fma.cu

template <class T>
int launch_push(const PushArgs<T>& a, int shape, bool precise, cudaStream_t st) {
    if (a.n <= 0) return 0;
    constexpr bool F32 = sizeof(T) == 4;
    // 128 threads spread the blocks of a small grid over the SMs more evenly
    // than 256 (128^2 x 4: 512 blocks, not 256, on 148 SMs; 64 add nothing)
    const int threads = 128;
    const unsigned blocks = (unsigned)((a.n + threads - 1) / threads);
    if (shape == QS_SHAPE_NGP) {
        if constexpr (F32) {
            if (a.uniform_ppc == 4 && a.n == (int64_t)a.My * a.Mz * 4 && !a.dep_cell) {
                // blocks of one warp, to spread a small grid's cells over the
                // SMs, are no better there (march per layer at 64 x 64 20.7 us
                // against 20.5, 128 x 128 23.6 against 23.0) and worse from
                // 128 x 256 on (27.2 against 26.2)
                const int cells = a.My * a.Mz;
                launch_pdl(push_cell_kernel<4>, dim3((cells + 127) / 128), dim3(128), 0, st, a);
                return 1;
            }
            launch_pdl(push_kernel<T, QS_SHAPE_NGP, true, true>, dim3(blocks), dim3(threads), 0, st, a);
        } else {
            if (precise) launch_pdl(push_kernel<T, QS_SHAPE_NGP, true, false>, dim3(blocks), dim3(threads), 0, st, a);
            else launch_pdl(push_kernel<T, QS_SHAPE_NGP, false, false>, dim3(blocks), dim3(threads), 0, st, a);
        }
    } else {
        if constexpr (F32) {
            if (launch_push_rows<float>(a, st)) return 1;
        } else {
            if (a.loff && !a.dep_cell) return launch_push_rows_f64(a, st);
        }
        launch_pdl(push_kernel<T, QS_SHAPE_CIC, true, F32>, dim3(blocks), dim3(threads), 0, st, a);
    }
    return 1;
}

}  // namespace qs
