// Wave-step 2D level-set sweep kernel for sm_103a.
//
// The wavefront of sweep_wave.cu in two dimensions: a warp owns 32 z'-rows, one per lane, and at
// step s lane l updates x' = x0 + s - l; the z'-upwind time arrives by one shuffle, the other two
// are the lane's own values of the step before.  Rows stream through the same shared-memory ring
// (row l at (l >> 2) + 8 (l & 3): no bank conflicts), the z' face crosses warp blocks as one
// tagged word per step, read a group of four steps ahead, and blocks start at the first updated row.
//
// A field is a chain of nx + nz dependent updates a sweep.  In FP64 each of an update's
// instructions takes the pipe for 64 cycles, whatever the number of lanes, so the update is
// arranged to issue few of them (fd2UniformFar has about 60):
//   * nodes that no operator can lower leave on FP32 bounds, without an FP64 instruction;
//   * comparisons run on integer order keys, minima of slowness on the bit patterns, and the
//     slowness arrives multiplied by h (with h > 0, h min(s, ..) is min(h s, ..) bit for bit);
//   * the diagonal operator comes first; another operator is evaluated only where its FP32
//     lower bound is not above the best candidate so far.
// What bounds a field is that chain (issue slots 14 % taken, DRAM idle); many fields share its latency
// until the FP64 pipe is full.  Measured, a solve of 4 + 8 sweeps of 501 x 251 nodes in double, ms, the
// kernel before (32-row blocks, the whole operator in FP64) and this one: 1 field 26.3, 7.8 (8.8 with
// one ordering per launch); 64 fields 32.2, 9.2 (13.5).  With non-uniform spacing 2673 to 1244 us a
// refinement sweep (2034 with the exit test alone in FP32).
#include <algorithm>
#include "sweep.h"
#include "wave.cuh"

namespace eikx {
namespace wave {

constexpr int kRows2 = kWaveRows2;
constexpr int kBeyond2 = kG - 1 + kWaveRows2 - kG;   // steps a block publishes beyond its last
constexpr int kThreads2 = 32 * kWarpsPerBlock;

// Shared memory of one warp: a plane of travel times and one of slowness, four chunk slots of 33
// rows each (32: the slowness of the row below the block), planes aligned to their size.  The
// halo of one group fills spare rows.
template <class T> struct Smem2 {
    static constexpr unsigned kChunkB = kG * sizeof(T);
    static constexpr unsigned kSlotB = 64 * kChunkB;
    static constexpr unsigned kPlaneB = 4 * kSlotB;
    static constexpr unsigned kWarpB = 2 * kPlaneB;
    static constexpr unsigned kHalo = 48 * kChunkB;
};

// Out of line: the factored branch, and all Cartesian operators, from the unscaled slowness: cell
// (cx, cz) of spNeg at (cz + 1) pitch + cx + 1, edges replicated, or (FP64 on a uniform grid) the
// model's own cells with pitch nx - 1, so that a solve keeps two copies of the slowness and not four.
template <class T, bool UNIFORM, bool NEAR>
__device__ __noinline__ T node2(T h, const Spacing2<T> &g, const SourceT<T> &src, const SweepSigns sg, int ix, int iz, T t1,
                                T t2, T t3, const T *sp, int pitch, int nz) {
    const bool fx = sg.ixShift > 0, fz = sg.izShift > 0;
    const int xu = fx ? ix + 1 : ix, xo = fx ? ix : ix + 1, zu = fz ? iz + 1 : iz, zo = fz ? iz : iz + 1;
    auto S = [&](int x, int z) -> T {
        if constexpr (UNIFORM && sizeof(T) == 8) {
            x = min(max(x - 1, 0), pitch - 1);
            z = min(max(z - 1, 0), nz - 2);
        }
        return sp[static_cast<long long>(z) * pitch + x];
    };
    const T s0 = S(xu, zu), s1 = S(xo, zu), s3 = S(xu, zo);
    if constexpr (UNIFORM)
        return NEAR ? fd2UniformNear<T>(h, src, sg, ix, iz, s0, s1, s3, t1, t2, t3) : fd2UniformFar<T>(h, s0, s1, s3, t1, t2, t3);
    else
        return NEAR ? fd2NonUniformNear<T>(g, src, sg, ix, iz, s0, s1, s3, t1, t2, t3)
                    : fd2NonUniformFar<T>(g, s0, s1, s3, t1, t2, t3);
}

// SCALED: the ring's slowness is h * slowness (FP64 on a uniform grid).
template <class T, bool UNIFORM, bool BOTH>
__global__ void __launch_bounds__(kThreads2) sweep2WaveKernel(const Sweep2Args<T> a) {
    constexpr int W = sizeof(T) / 4;
    constexpr unsigned kT = sizeof(T);
    constexpr bool SCALED = UNIFORM && sizeof(T) == 8;
    using SM = Smem2<T>;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned tBase = ((smemAddr(smemRaw) + SM::kPlaneB - 1) & ~(SM::kPlaneB - 1)) + warp * SM::kWarpB;
    auto rowOf = [](int l) { return (l >> 2) + 8 * (l & 3); };
    const unsigned laneOff = rowOf(lane) * SM::kChunkB;
    constexpr unsigned toO = SM::kPlaneB;
    const unsigned toN = SM::kPlaneB + (lane ? rowOf(lane - 1) : 32) * SM::kChunkB - laneOff;
    const unsigned halo = tBase + SM::kHalo;
    const SolveState &st = a.st;
    if (blockIdx.x == 0 && threadIdx.x == 0) *st.queue[a.buf ^ 1] = 0u;
    if (ldVolatile(st.abortFlag)) return;
    if constexpr (BOTH) {   // nothing to do: leave the queue alone
        bool work = false;
        for (int f = lane; f < a.nFields; f += 32) work |= !st.converged[f] && (a.passMode == kBothSweeps || st.pairState[f] == kPairOpen);
        if (!__any_sync(kFull, work)) return;
    }
    const T huge = static_cast<T>(1.e10);
    const int Px = a.pitch, nx = a.nx, nz = a.nz, nChunks = Px / kG;
    const T *raw = a.spNeg;               // the unscaled slowness (node2)
    if constexpr (SCALED) raw = a.cells;
    const int rawPitch = SCALED ? nx - 1 : a.spPitch;
    const long long fieldWords = static_cast<long long>(a.tilesZ) * waveStepCap2(Px) * W;
    const float hF = view(a.h), dxF = view(a.sp2.dx), dzF = view(a.sp2.dz), dMinF = fminf(dxF, dzF);
    bool ok = true;

    while (ok) {
        unsigned q = 0;
        if (lane == 0) q = atomicAdd(st.queue[a.buf], 1u);
        q = __shfl_sync(kFull, q, 0);
        if (q >= static_cast<unsigned>(st.totalItems)) break;
        const int4 item = st.order[q];
        const int f = item.x, c = item.z;
        if (st.converged[f]) continue;
        // both orderings of a pair, as in sweep_wave.cu
        int passes = 1;
        if constexpr (BOTH) {
            const int state = st.pairState[f];
            if (a.passMode == kSecondSweep && state != kPairOpen) continue;
            if (a.passMode == kBothSweeps && state != kPairHeld) passes = 2;
        }
#pragma unroll 1
        for (int pass = 0; pass < (BOTH ? passes : 1); ++pass) {
            const int sweep = a.sweep + pass;
            const unsigned tag = *st.epoch + static_cast<unsigned>(a.sweepIndex + pass);
            const int fx = sweep & 1, fz = (sweep >> 1) & 1;
            const int dir = fx ? -1 : 1;
            const unsigned slotStep = fx ? 3 * SM::kSlotB : SM::kSlotB;
            SweepSigns sg;
            sg.ixShift = fx ? 1 : -1; sg.iyShift = 0; sg.izShift = fz ? 1 : -1;
            sg.signX = fx ? -1 : 1; sg.signY = 1; sg.signZ = fz ? -1 : 1;
            const T *sp = SCALED ? (fx ? a.hsNeg : a.hsPos) : (fx ? a.spNeg : a.spPos);
            const int sShift = fx ? 0 : 16 / static_cast<int>(sizeof(T));
            const SourceT<T> &src = a.srcs[f];
            const int isx = src.isx;
            int xlo, xhi, zlo, zhi;
            axisBounds(nx, fx, a.init, isx, xlo, xhi);
            axisBounds(nz, fz, a.init, src.isz, zlo, zhi);
            const int wz = fz ? nz - 1 - zhi : zlo;        // first updated row in walk order (>= 1)
            const int z0 = wz + kRows2 * c;
            if (z0 >= nz) break;
            const int xaS = fx ? xhi + 2 : xlo - 2;        // lane 0's column at step 0
            const int walkLen = fx ? xaS + 1 : Px - xaS;
            const int nSteps = (walkLen + kRows2 - 1 + kG - 1) / kG * kG;
            const int zW = z0 + lane;
            const bool valid = zW < nz;
            const int za = reflect(valid ? zW : z0, nz, fz), zBelow = reflect(z0 - 1, nz, fz);
            T *field = a.tt + static_cast<long long>(f) * a.fieldStride;
            T *row = field + static_cast<long long>(za) * Px;
            const T *below = field + static_cast<long long>(zBelow) * Px;
            auto srowAt = [&](int z) { return sp + static_cast<long long>(z + (fz ? 0 : 1)) * a.spPitch + sShift; };
            const T *srow = srowAt(za), *sBelow = srowAt(zBelow);
            const unsigned cnt = valid ? static_cast<unsigned>(xhi - xlo + 1) : 0u;
            const bool rowNear = valid && abs(src.isz - za) <= a.radius;
            const bool tileNear = __any_sync(kFull, rowNear);
            const int rx = min(a.radius, Px), nearFrom = dir * (isx - xaS) - rx - 2;   // progress of the first near column

            // the z' face [step + 1]; lanes below 4 read a group's words, or the row below from the field
            unsigned long long *face = st.mbox + (BOTH ? 2 * f + fx : f) * fieldWords + static_cast<long long>(c) * waveStepCap2(Px) * W;
            const bool pub = z0 + kRows2 < nz && lane == kRows2 - 1;
            const bool mail = lane < kG && c > 0, fromField = lane < kG && c == 0;
            const unsigned long long *next = face - static_cast<long long>(waveStepCap2(Px)) * W + static_cast<long long>(kRows2 + lane) * W;
            Words<T> zw;
            T zf = huge;
            packWords<T>(mail ? 0u : tag, huge, zw);       // no sweep's tag is 0
            auto issue = [&](int g) {
                loadIf(mail, next, zw);
                const int x = xaS + dir * (kG * g + lane);
                loadIf(fromField && x >= 0 && x < Px, below + x, zf);
            };

            int xa = xaS - dir * lane;                     // this step's column
            unsigned R[kG];
#pragma unroll
            for (int e = 0; e < kG; ++e) {
                const unsigned u = static_cast<unsigned>(xa + dir * e + 64);
                R[e] = tBase + ((u >> 2) & 3u) * SM::kSlotB + (u & 3u) * kT + laneOff;
            }
            auto slotAfter = [&](unsigned r) { return (r & ~(SM::kPlaneB - 1)) | ((r + slotStep) & (SM::kPlaneB - 1)); };
            auto copyChunk = [&](unsigned dst, const T *src16) {
#pragma unroll
                for (unsigned q16 = 0; q16 < SM::kChunkB / 16; ++q16)
                    cpAsync16(dst + 16 * q16, reinterpret_cast<const char *>(src16) + 16 * q16);
            };
            int gFill = -1;
            auto fill = [&]() {
                const int k = (xaS + dir * (kG * gFill + kG - 1 - lane)) >> 2;
                if (valid && k >= 0 && k < nChunks) {
                    const unsigned dst = tBase + (static_cast<unsigned>(k) & 3u) * SM::kSlotB + laneOff;
                    copyChunk(dst, row + k * kG);
                    copyChunk(dst + SM::kPlaneB, srow + k * kG);
                }
                const int kb = (xaS + dir * (kG * gFill + kG)) >> 2;          // the row below: a lane -1
                if (lane == 0 && kb >= 0 && kb < nChunks)
                    copyChunk(tBase + SM::kPlaneB + (static_cast<unsigned>(kb) & 3u) * SM::kSlotB + 32 * SM::kChunkB, sBelow + kb * kG);
                cpCommit();
                ++gFill;
            };
            fill();
            fill();
            issue(0);

            T o1 = huge, nP = huge, snP = huge, soP = huge;   // t1, t2; s0, s3
            float vo = 1.e10f, vnP = 1.e10f;
            unsigned long long *out = face + W;               // index step + 1
            T res = 0;
            unsigned changedNow = 0, changedLast = 0;
            int p = -lane - 2;                                // progress (updates start at 0)
            for (int g = 0;; ++g) {
                // store the chunk passed by the last group
                const int k = (xa >> 2) - dir;
                if ((changedNow | changedLast) && k >= 0 && k < nChunks) {
                    const unsigned srcA = tBase + (static_cast<unsigned>(k) & 3u) * SM::kSlotB + laneOff;
#pragma unroll
                    for (unsigned q16 = 0; q16 < SM::kChunkB / 16; ++q16)
                        *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(row + k * kG) + 16 * q16) = lds16(srcA + 16 * q16);
                }
                changedLast = changedNow;
                changedNow = 0;
                if (kG * g >= nSteps) break;
                {
                    unsigned long long it = 0;
                    while (!__all_sync(kFull, ready(zw, tag))) {
                        bool stop = false;
                        if ((++it & 31ull) == 0) {
                            stop = ldVolatile(st.abortFlag) != 0;
                            if (it > st.spinLimit) {
                                atomicExch(st.abortFlag, 1);
                                stop = true;
                            }
                        }
                        if (__any_sync(kFull, stop)) {
                            ok = false;
                            break;
                        }
                        loadIf(mail, next, zw);
                    }
                    if (!ok) break;
                }
                if (lane < kG) sts(halo + lane * kT, mail ? value<T>(zw) : zf);
                fill();
                next += kG * W;
                issue(g + 1);
                cpWait<1>();
                __syncwarp();
#pragma unroll 1
                for (int e = 0; e < kG; ++e) {
                    const unsigned r = R[0];
                    const T sO = lds(r + toO, T()), sN = lds(r + toN, T()), t0 = lds(r, T());
                    T N = __shfl_up_sync(kFull, o1, 1);
                    ldsIf(lane == 0, N, halo + e * kT);
                    const float vN = view(N);
                    // t1 = o1, t2 = nP, t3 = N; s0 = snP, s1 = sN, s3 = soP
                    const bool upd = static_cast<unsigned>(p) < cnt;
                    const float v0 = Bounds<T>::upper(view(t0)), mx = fmaxf(vo, vN), E = mx * Bounds<T>::kE;
                    float low;
                    // A 1D operator or one of a cell edge is >= t1 or >= t3; the diagonal one, its window
                    // open, is >= t2 + h s0 less the rounding (the 3D planes' bound, sweep_wave.cu), and on a
                    // non-uniform grid >= t2 + min(dx s0, dz s0) less a rounding error below 64 u
                    // max(t1, t2, t3): with d = t1 - t3 between -dx s0 and dz s0, the exact operator is concave
                    // in d and dx s0, dz s0 above t2 at the ends, and each of its terms is at most
                    // 3 max(t1, t2, t3) there.
                    if (UNIFORM && SCALED) low = vnP + __fmaf_rn(view(snP), kC20, -E);
                    else if (UNIFORM) low = vnP - E;
                    else low = vnP + __fmaf_rn(dMinF * view(snP), kC20, -fmaxf(mx, vnP) * 1.52587890625e-5f);   // 2^-16
                    bool need = upd & !(v0 <= fminf(fminf(vo, vN), low));
                    T v = t0;
                    if (tileNear) {
                        if (rowNear && upd && static_cast<unsigned>(p - nearFrom) <= 2u * rx) {
                            need = false;
                            const T tu = node2<T, UNIFORM, true>(a.h, a.sp2, src, sg, xa, za, o1, nP, N, raw, rawPitch, nz);
                            if (tu < v) v = tu;
                        }
                    }
                    if (__any_sync(kFull, need)) {
                        if constexpr (SCALED) {
                            T best = t0;
                            const float f0 = view(snP);
                            // the diagonal operator t2 + sqrt(2 (h s0)^2 - (t1 - t3)^2), where the wave runs
                            // outwards (t1, t3 >= t2) within the window |t1 - t3| <= h s0 (FP32 decides unless
                            // within its error)
                            const float df = fabsf(vo - vN), slack = mx * (1.0f / 1048576.0f);
                            bool c3 = need & !above(nP, N) & !above(nP, o1) & (low <= v0) &
                                      (df - slack <= f0 * (1.0f + 2.0f / 1048576.0f));
                            if (__any_sync(kFull, c3)) {
                                const T d = o1 - N, hh = snP * snP, det = fmaT(T(2), hh, -(d * d));   // 2 hh is exact
                                c3 = c3 & above(det, T(0));
                                if (__any_sync(kFull, c3 & !(df + slack < f0 * kC20)))
                                    c3 = c3 & !above(N, o1 + snP) & !above(o1, N + snP);
                                const T u = nP + dsqrt(c3 ? det : T(1));
                                if (c3 & above(best, u)) best = u;
                            }
                            // along x and z: t1 + h min(s0, s3), t3 + h min(s0, s1)
                            const T hx = pmin(snP, soP), hz = pmin(snP, sN);
                            const bool gx = need & (vo + __fmaf_rn(view(hx), kC20, -E) <= Bounds<T>::upper(view(best)));
                            if (__any_sync(kFull, gx)) {
                                const T u = o1 + hx;
                                if (gx & above(best, u)) best = u;
                            }
                            const bool gz = need & (vN + __fmaf_rn(view(hz), kC20, -E) <= Bounds<T>::upper(view(best)));
                            if (__any_sync(kFull, gz)) {
                                const T u = N + hz;
                                if (gz & above(best, u)) best = u;
                            }
                            // of the cell's edges: t1 + h sqrt((h s0)^2 - (t1 - t2)^2) where 0 <= t1 - t2
                            // <= h s0 / sqrt 2, t3 likewise: all operators again where FP32 cannot rule it out
                            const float ub = Bounds<T>::upper(view(best));
                            auto edge = [&](float va, bool outward) {
                                const float hi = fmaxf(va - vnP, 0.f) + fmaxf(va, vnP) * (1.0f / 1048576.0f);   // >= t_a - t2
                                const float lo = va - vnP - fmaxf(va, vnP) * (1.0f / 1048576.0f);
                                const float w = __fmaf_rn(f0 * (1.0f - 1.0f / 262144.0f), f0, -(hi * hi));   // <= (h s0)^2 - hi^2
                                float root;
                                asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(fmaxf(w, 0.f)));
                                return outward & (lo <= 0.7072f * f0) & (va + hF * root * (1.0f - 1.0f / 1024.0f) - E <= ub);
                            };
                            const bool again = need & (edge(vo, !above(nP, o1)) | edge(vN, !above(nP, N)));
                            if (__any_sync(kFull, again)) {
                                if (again) best = dmin(best, node2<T, UNIFORM, false>(a.h, a.sp2, src, sg, xa, za, o1, nP, N, raw, rawPitch, nz));
                            }
                            if (need) v = best;
                        } else if constexpr (!UNIFORM && sizeof(T) == 8) {
                            // fd2NonUniformFar, each operator only where FP32 cannot rule it out
                            const Spacing2<T> &g2 = a.sp2;
                            T best = t0;
                            const float f0 = view(snP), big = fmaxf(mx, vnP) * (1.0f / 1048576.0f);
                            constexpr float kUp = 1.0f + 1.0f / 65536.0f;
                            const bool outX = !above(nP, o1), outZ = !above(nP, N);   // t1 >= t2, t3 >= t2
                            bool c3 = need & outX & outZ & (low <= v0) & (vo - vN <= f0 * dzF * kUp + big) & (vN - vo <= f0 * dxF * kUp + big);
                            if (__any_sync(kFull, c3)) {
                                const T hx = g2.dx * snP, hz = g2.dz * snP, d = o1 - N, det = hx * hx + hz * hz - d * d;
                                c3 = c3 & above(det, T(0)) & above(N + hz, o1) & above(o1 + hx, N);
                                const T tx = o1 - N + nP, tz = N - o1 + nP, dxdz = g2.cosTheta * g2.sinTheta;
                                const T u = dxdz * (tx * g2.dz_dx + tz * g2.dx_dz + 2 * dsqrt(c3 ? det : T(1)));
                                if (c3 && !(u < 0) && u < best) best = u;
                            }
                            const bool gx = need & (vo + __fmaf_rn(dxF * fminf(f0, view(soP)), kC20, -E) <= Bounds<T>::upper(view(best)));
                            if (__any_sync(kFull, gx)) {
                                const T u = o1 + g2.dx * pmin(snP, soP);
                                if (gx & above(best, u)) best = u;
                            }
                            const bool gz = need & (vN + __fmaf_rn(dzF * fminf(f0, view(sN)), kC20, -E) <= Bounds<T>::upper(view(best)));
                            if (__any_sync(kFull, gz)) {
                                const T u = N + g2.dz * pmin(snP, sN);
                                if (gz & above(best, u)) best = u;
                            }
                            // t1 + dx / dz sqrt((dz s0)^2 - (t1 - t2)^2) where 0 <= t1 - t2 <= dz sin s0; t3 likewise
                            auto edge = [&](float va, float dF, float ratio, float sine) {
                                const float hi = fmaxf(va - vnP, 0.f) + big, lo = va - vnP - big, h = dF * f0;
                                const float w = __fmaf_rn(h * (1.0f - 1.0f / 131072.0f), h, -(hi * hi));
                                float root;
                                asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(fmaxf(w, 0.f)));
                                return (lo <= h * sine * kUp) & (va + ratio * root * (1.0f - 1.0f / 1024.0f) - E <= Bounds<T>::upper(view(best)));
                            };
                            const bool ea = need & outX & edge(vo, dzF, view(g2.dx_dz), view(g2.sinTheta));
                            if (__any_sync(kFull, ea)) {
                                const T hz = g2.dz * snP, d = o1 - nP, det = hz * hz - d * d;
                                const T u = o1 + g2.dx_dz * dsqrt(ea && det >= 0 ? det : T(1));
                                if (ea && det >= 0 && d <= g2.dz * (g2.sinTheta * snP) && u < best) best = u;
                            }
                            const bool eb = need & outZ & edge(vN, dxF, view(g2.dz_dx), view(g2.cosTheta));
                            if (__any_sync(kFull, eb)) {
                                const T hx = g2.dx * snP, d = N - nP, det = hx * hx - d * d;
                                const T u = N + g2.dz_dx * dsqrt(eb && det >= 0 ? det : T(1));
                                if (eb && det >= 0 && d <= g2.dx * (g2.cosTheta * snP) && u < best) best = u;
                            }
                            if (need) v = best;
                        } else {
                            T tu;
                            if constexpr (UNIFORM) tu = fd2UniformFar<T>(a.h, snP, sN, soP, o1, nP, N);
                            else tu = fd2NonUniformFar<T>(a.sp2, snP, sN, soP, o1, nP, N);
                            if (need && tu < v) v = tu;
                        }
                    }
                    if (above(t0, v) & upd) {
                        res = dmax(res, t0 - v);
                        changedNow = 1;
                        sts(r, v);
                    }
                    if (pub) {
                        Words<T> w;
                        packWords<T>(tag, v, w);
                        storeWords<T>(out, w);
                    }
                    out += W;
                    o1 = v; nP = N; snP = sN; soP = sO;
                    vo = view(v); vnP = vN;
                    const unsigned rn = slotAfter(r);
#pragma unroll
                    for (int i = 0; i + 1 < kG; ++i) R[i] = R[i + 1];
                    R[kG - 1] = rn;
                    xa += dir;
                    ++p;
                }
            }
            cpWait<0>();   // no copy into the ring outlives the work item
            __syncwarp();
            if (!ok) break;
            // the words beyond the last step, which the block after waits for (no update uses them)
            Words<T> w;
            packWords<T>(tag, huge, w);
            if (pub)
#pragma unroll 1
                for (int e = 0; e < kBeyond2; ++e) storeWords<T>(out + e * W, w);
            const double rMax = warpMax(static_cast<double>(res));
            if (lane == 0 && rMax > 0)
                atomicMax(st.residual + static_cast<long long>(f) * st.residualStride + a.residualSlot + pass,
                          static_cast<unsigned long long>(__double_as_longlong(rMax)));
            if (BOTH) __threadfence();   // the next pass copies the rows that this one stored
        }
    }
}

template <class T> constexpr size_t smemBytes2() {
    return static_cast<size_t>(Smem2<T>::kWarpB) * kWarpsPerBlock + Smem2<T>::kPlaneB;
}
template <class K> int occupancy2(K kernel, size_t smem) {
    int n = 0;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads2, smem);
    return n > 0 ? n : 1;
}

}  // namespace wave

template <class T, class F> auto withWaveKernel2(bool uniform, bool both, F f) {
    using namespace wave;
    if (both) return uniform ? f(sweep2WaveKernel<T, true, true>) : f(sweep2WaveKernel<T, false, true>);
    return uniform ? f(sweep2WaveKernel<T, true, false>) : f(sweep2WaveKernel<T, false, false>);
}
template <class T> int sweep2WaveBlocksPerSM(bool uniform) {
    auto f = [](auto k) { return wave::occupancy2(k, wave::smemBytes2<T>()); };
    return std::min(withWaveKernel2<T>(uniform, false, f), withWaveKernel2<T>(uniform, true, f));
}
// The caller asks sweep2WaveBlocksPerSM for the grid size first, which sets the kernel's
// shared-memory limit.
template <class T> cudaError_t launchSweep2Wave(const Sweep2Args<T> &a, bool uniform, int blocks, cudaStream_t s) {
    if (uniform && sizeof(T) == 8 && (!a.hsPos || !a.hsNeg || !a.cells)) return cudaErrorInvalidValue;
    return withWaveKernel2<T>(uniform, a.passMode != kOneSweep, [&](auto k) {
        k<<<blocks, wave::kThreads2, wave::smemBytes2<T>(), s>>>(a);
        return cudaGetLastError();
    });
}
template int sweep2WaveBlocksPerSM<float>(bool);
template int sweep2WaveBlocksPerSM<double>(bool);
template cudaError_t launchSweep2Wave<float>(const Sweep2Args<float> &, bool, int, cudaStream_t);
template cudaError_t launchSweep2Wave<double>(const Sweep2Args<double> &, bool, int, cudaStream_t);

}  // namespace eikx
