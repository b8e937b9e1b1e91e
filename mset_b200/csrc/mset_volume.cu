// mset_volume.cu -- volume kernels of the reconstruction update:
// TV / TV-FISTA proximal operator (func_lib/TV_method.m:5-28 and helpers
// :32-83, func_lib/TV_FISTA_method.m:5-38), positivity
// (Run_MSET_recon.m:183-185), max-normalisation (Run_MSET_recon.m:268-270),
// and the glue between beam-frame slab gradients and the lab-frame volume.
//
// All stencils are periodic (MATLAB circshift).  Volumes are C order
// [n3][n2][n1] = MATLAB (n1, n2, n3); MATLAB dim 1 is the fastest axis.
// HBM/L2-bound elementwise work: grid-stride loops over 148 x 8 CTAs (the
// scalar TV stencils: over rows, one CTA per row).  TV runs on one of three
// routes (tv_prox): every iteration in one cluster launch where the volume fits
// its shared memory and few slices fall to a CTA (tv_cluster_pays), one marching
// kernel per iteration where rows are whole float4 groups, else two kernels per
// iteration.
#include <algorithm>
#include <cmath>

#include "fft_core.cuh"
#include "mset_volume.cuh"

namespace mset {

namespace {
constexpr int kThreads = 256;

inline int grid_for(long total) {
    long g = (total + kThreads - 1) / kThreads;
    return (int)std::min<long>(std::max<long>(g, 1), 148L * 8);
}

__device__ __forceinline__ long wrap(long i, long n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// The TV stencils run one CTA per row (i2, i3) of the volume in a
// grid-stride loop over rows, threads over i1: the periodic neighbours' rows
// are found once per row (one 32-bit division) instead of three 64-bit
// divisions per element, which made these kernels integer-bound.
struct Rows {
    int n1, n2, n3;
    long V;
    // first element of row (i2, i3); neighbour rows with periodic wrap
    __device__ __forceinline__ long at(int i2, int i3) const { return ((long)i3 * n2 + i2) * n1; }
};

// D = TV_div(Y) - in / lambda   (the argument of TV_del in TV_method.m:21)
__global__ void k_tv_d(const float *Y, const float *in, float *D, Rows g, float inv_lam) {
    const long V = g.V;
    for (int row = blockIdx.x; row < g.n2 * g.n3; row += gridDim.x) {
        const int i2 = row % g.n2, i3 = row / g.n2;
        const long b = g.at(i2, i3), b2 = g.at(i2 == 0 ? g.n2 - 1 : i2 - 1, i3),
                   b3 = g.at(i2, i3 == 0 ? g.n3 - 1 : i3 - 1);
        for (int i1 = threadIdx.x; i1 < g.n1; i1 += blockDim.x) {
            const long r = b + i1;
            const int i1m = i1 == 0 ? g.n1 - 1 : i1 - 1;
            const float d = Y[r] + Y[V + r] + Y[2 * V + r] - Y[b + i1m] - Y[V + b2 + i1] - Y[2 * V + b3 + i1];
            D[r] = d - in[r] * inv_lam;
        }
    }
}

// P <- TV_project(src + tau TV_del(D)); FISTA: Y <- P + m (P - P_old) in FP64
__global__ void k_tv_step(float *P, float *Y, const float *D, Rows g, float tau, double m, int fista) {
    const long V = g.V;
    for (int row = blockIdx.x; row < g.n2 * g.n3; row += gridDim.x) {
        const int i2 = row % g.n2, i3 = row / g.n2;
        const long b = g.at(i2, i3), b2 = g.at(i2 == g.n2 - 1 ? 0 : i2 + 1, i3),
                   b3 = g.at(i2, i3 == g.n3 - 1 ? 0 : i3 + 1);
        for (int i1 = threadIdx.x; i1 < g.n1; i1 += blockDim.x) {
            const long r = b + i1;
            const int i1p = i1 == g.n1 - 1 ? 0 : i1 + 1;
            const float d0 = D[r];
            const float t1 = tau * (D[b + i1p] - d0);
            const float t2 = tau * (D[b2 + i1] - d0);
            const float t3 = tau * (D[b3 + i1] - d0);
            const float *src = fista ? Y : P;
            const float q1 = src[r] + t1, q2 = src[V + r] + t2, q3 = src[2 * V + r] + t3;
            const float nrm = sqrtf(fmaxf(1.0f, q1 * q1 + q2 * q2 + q3 * q3));
            const float p1 = q1 / nrm, p2 = q2 / nrm, p3 = q3 / nrm;
            if (fista) {
                const double o1 = P[r], o2 = P[V + r], o3 = P[2 * V + r];
                Y[r] = (float)(p1 + m * (p1 - o1));
                Y[V + r] = (float)(p2 + m * (p2 - o2));
                Y[2 * V + r] = (float)(p3 + m * (p3 - o3));
            }
            P[r] = p1;
            P[V + r] = p2;
            P[2 * V + r] = p3;
        }
    }
}

// out = in - lambda TV_div(P)   (TV_method.m:26)
__global__ void k_tv_out(const float *P, const float *in, float *out, Rows g, float lam) {
    const long V = g.V;
    for (int row = blockIdx.x; row < g.n2 * g.n3; row += gridDim.x) {
        const int i2 = row % g.n2, i3 = row / g.n2;
        const long b = g.at(i2, i3), b2 = g.at(i2 == 0 ? g.n2 - 1 : i2 - 1, i3),
                   b3 = g.at(i2, i3 == 0 ? g.n3 - 1 : i3 - 1);
        for (int i1 = threadIdx.x; i1 < g.n1; i1 += blockDim.x) {
            const long r = b + i1;
            const int i1m = i1 == 0 ? g.n1 - 1 : i1 - 1;
            const float dv = P[r] + P[V + r] + P[2 * V + r] - P[b + i1m] - P[V + b2 + i1] - P[2 * V + b3 + i1];
            out[r] = in[r] - lam * dv;
        }
    }
}

// err += lambda sum |TV_del(u)|   (TV_method.m:27, 71-83), FP64 accumulation
__global__ void k_tv_err(const float *u, Rows g, double lam, double *err) {
    double acc = 0.0;
    for (int row = blockIdx.x; row < g.n2 * g.n3; row += gridDim.x) {
        const int i2 = row % g.n2, i3 = row / g.n2;
        const long b = g.at(i2, i3), b2 = g.at(i2 == g.n2 - 1 ? 0 : i2 + 1, i3),
                   b3 = g.at(i2, i3 == g.n3 - 1 ? 0 : i3 + 1);
        for (int i1 = threadIdx.x; i1 < g.n1; i1 += blockDim.x) {
            const long r = b + i1;
            const int i1p = i1 == g.n1 - 1 ? 0 : i1 + 1;
            const float u0 = u[r];
            const float d1 = u[b + i1p] - u0;
            const float d2 = u[b2 + i1] - u0;
            const float d3 = u[b3 + i1] - u0;
            acc += sqrt((double)d1 * d1 + (double)d2 * d2 + (double)d3 * d3);
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(err, lam * acc);
}

// Four consecutive voxels per thread (n1 a multiple of 4): 16-byte loads and
// stores of every array, the one periodic neighbour along i1 outside the
// thread's four voxels read as a 4-byte load (an L1 hit: the neighbouring
// thread loads its line).  Fewer, wider requests keep more bytes in flight per
// SM; same arithmetic per voxel.
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }

__device__ __forceinline__ void tv_project(float q1, float q2, float q3, float &p1, float &p2, float &p3) {
    const float nrm = sqrtf(fmaxf(1.0f, q1 * q1 + q2 * q2 + q3 * q3));
    p1 = q1 / nrm;
    p2 = q2 / nrm;
    p3 = q3 / nrm;
}

// One iteration as one kernel (rows of whole float4 groups): D = div(src) -
// in / lambda is never stored.  A CTA takes ty adjacent rows of a slice, full
// length, and marches through zc slices: per slice it computes D of the next
// one (its rows and the row above them) from that slice's dual values, which
// stay in registers as the next step's source, leaves it in shared memory for
// the neighbours along i1 and i2, and finishes the current slice.  The dual
// field is read from src and written to dst, so the neighbours' old values
// survive.  Per voxel it moves 16 B of source and input (and 1 / zc + 1 / ty
// of them again), 12 of P and 24 of results, against 20 + 52 in two kernels
// with D in memory, and half the launches: 164.8 -> 110.3 us per FISTA iteration
// at 256 x 256 x 192 (6.0 TB/s of HBM), 24.8 -> 20.5 at 128^3 (L2 and the
// chain of a step), 16.3 -> 10.0 at 96^3, 12.3 -> 6.1 at 64^3.
//
// Each iteration's kernel is set up while the one before drains (programmatic
// dependent launch; the wait stands before the first access): 108.2, 18.6 (16.4
// since the chunks go by whole waves, tv_prox), 8.8 and 3.9 us there, 3.4 against
// 6.1 at 48^3; inside a captured iteration, whose launches cost less, 2.5% of it at
// 48^3 and 0.5 to 2% above.  The kernels do not signal early: CTAs of the next
// iteration then take places among the running ones, whose neighbours share slices
// in L2 (129.7 us at 256 x 256 x 192, 19.8 at 128^3).
struct Quad {
    float v[4];
};
__device__ __forceinline__ Quad quad(const float *p) {
    const float4 q = ld4(p);
    return Quad{{q.x, q.y, q.z, q.w}};
}
__device__ __forceinline__ void put(float *p, const Quad &q) { st4(p, make_float4(q.v[0], q.v[1], q.v[2], q.v[3])); }

// D of four voxels at row offset b (+ i1) with the neighbours' rows b2 (i2 - 1)
// and m3 = Y3 one slice below; the dual values come back in y
__device__ __forceinline__ Quad tv_d4(const float *Y, const float *in, long V, long b, long b2, int i1, int n1,
                                      float inv_lam, const Quad &m3, Quad y[3]) {
    const Quad m2 = quad(Y + V + b2 + i1), u = quad(in + b + i1);
#pragma unroll
    for (int c = 0; c < 3; ++c) y[c] = quad(Y + c * V + b + i1);
    const float y1m = Y[b + (i1 == 0 ? n1 - 1 : i1 - 1)];
    Quad d;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        d.v[e] = (y[0].v[e] + y[1].v[e] + y[2].v[e] - (e ? y[0].v[e ? e - 1 : 0] : y1m) - m2.v[e] - m3.v[e]) -
                 u.v[e] * inv_lam;
    return d;
}

template <bool FISTA>
__global__ void __launch_bounds__(256) k_tv_march(const float *src, float *dst, float *P, const float *in, Rows g,
                                                  int ty, int zc, float inv_lam, float tau, double m) {
    extern __shared__ __align__(16) float dsm[];
    const long V = g.V;
    const int q1 = g.n1 / 4, i1 = 4 * (threadIdx.x % q1), r = threadIdx.x / q1;
    const int tiles = (g.n2 + ty - 1) / ty;
    const int y0 = (blockIdx.x % tiles) * ty, z0 = (blockIdx.x / tiles) * zc, z1 = min(z0 + zc, g.n3);
    const int rows = min(ty, g.n2 - y0);
    const bool on = r < rows, halo = r == 0;
    // the iteration before has finished and its stores are visible
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int y = y0 + (on ? r : 0), ym = y == 0 ? g.n2 - 1 : y - 1;
    const int yh = y0 + rows == g.n2 ? 0 : y0 + rows, yhm = y0 + rows - 1;
    float *cur = dsm, *nxt = dsm + (ty + 1) * g.n1;
    Quad yc[3], d0;
    {
        const int zm = z0 == 0 ? g.n3 - 1 : z0 - 1;
        if (on) {
            d0 = tv_d4(src, in, V, g.at(y, z0), g.at(ym, z0), i1, g.n1, inv_lam, quad(src + 2 * V + g.at(y, zm) + i1), yc);
            put(cur + r * g.n1 + i1, d0);
        }
        if (halo) {
            Quad yy[3];
            put(cur + rows * g.n1 + i1, tv_d4(src, in, V, g.at(yh, z0), g.at(yhm, z0), i1, g.n1, inv_lam,
                                              quad(src + 2 * V + g.at(yh, zm) + i1), yy));
        }
    }
    __syncthreads();
    for (int z = z0; z < z1; ++z) {
        const int zp = z + 1 == g.n3 ? 0 : z + 1;
        Quad yn[3], dn, p[3];
        if (on) {
            const long o = g.at(y, z) + i1;
            if constexpr (FISTA) {
#pragma unroll
                for (int c = 0; c < 3; ++c) p[c] = quad(P + c * V + o);
            }
            dn = tv_d4(src, in, V, g.at(y, zp), g.at(ym, zp), i1, g.n1, inv_lam, yc[2], yn);
            put(nxt + r * g.n1 + i1, dn);
            const float *row = cur + r * g.n1;
            const float dp = row[i1 + 4 == g.n1 ? 0 : i1 + 4];
            const Quad du = quad(row + g.n1 + i1);
            Quad w[3];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float t1 = tau * ((e < 3 ? d0.v[e < 3 ? e + 1 : 3] : dp) - d0.v[e]);
                const float t2 = tau * (du.v[e] - d0.v[e]);
                const float t3 = tau * (dn.v[e] - d0.v[e]);
                tv_project(yc[0].v[e] + t1, yc[1].v[e] + t2, yc[2].v[e] + t3, w[0].v[e], w[1].v[e], w[2].v[e]);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if constexpr (FISTA) {
                    Quad f;
#pragma unroll
                    for (int e = 0; e < 4; ++e) f.v[e] = (float)(w[c].v[e] + m * (w[c].v[e] - (double)p[c].v[e]));
                    put(dst + c * V + o, f);
                    put(P + c * V + o, w[c]);
                } else {
                    put(dst + c * V + o, w[c]);
                }
                yc[c] = yn[c];
            }
            d0 = dn;
        }
        if (halo && z + 1 < z1) {
            Quad yy[3];
            put(nxt + rows * g.n1 + i1, tv_d4(src, in, V, g.at(yh, zp), g.at(yhm, zp), i1, g.n1, inv_lam,
                                              quad(src + 2 * V + g.at(yh, z) + i1), yy));
        }
        __syncthreads();
        float *s = cur;
        cur = nxt;
        nxt = s;
    }
}

// All iterations of a small volume in one launch: the slices are dealt out over
// a cluster, K per CTA, and the dual fields stay in shared memory.  Launches
// bound the kernels above at these sizes; here it is the arithmetic of one
// CTA's slices (square root, three divisions, FP64 momentum per voxel), so the
// cluster is the largest one (24^3: 8.1 us per iteration of two launches, 2.5 on
// 8 CTAs, 1.9 on 16) and its route ends where a CTA's share gets long
// (tv_cluster_pays).  Per iteration a CTA
// computes D of its slices and of the one above them, steps, and hands its
// bottom slice's new dual values to the CTA below and its top slice's third
// component to the CTA above (two halo buffers in turn, so one cluster barrier
// per iteration orders both the reads and the writes).  A thread of a warp of
// its own works out the next momentum factor meanwhile.
constexpr int kTvCl = 16;  // 8 where the device holds no cluster of 16

// floats of shared memory for planes of `plane` voxels, K slices per CTA
inline long tv_cluster_floats(long plane, int K, bool fista) {
    return plane * ((fista ? 6L : 3L) * K + 2L * (K + 1) + 8);
}

template <bool FISTA>
__global__ void __launch_bounds__(1024) k_tv_cluster(float *Pout, const float *in, Rows g, int K, float inv_lam,
                                                     float tau, int niter) {
    extern __shared__ __align__(16) float dsm[];
    __shared__ double s_m[2];
    const int A = g.n1 * g.n2, lanes = blockDim.x - 32, tid = threadIdx.x;
    unsigned rk;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rk));
    const int rank = (int)rk, z0 = rank * K, busy = (g.n3 + K - 1) / K;
    const int own = max(0, min(K, g.n3 - z0));
    float *Y = dsm, *Pp = Y + 3 * K * A, *U = Pp + (FISTA ? 3 * K * A : 0), *D = U + (K + 1) * A;
    float *hy = D + (K + 1) * A, *hz = hy + 6 * A;  // [2][3][A] and [2][A]
    for (int i = tid; i < (FISTA ? 6 : 3) * K * A; i += blockDim.x) Y[i] = 0.f;
    for (int i = tid; i < 8 * A; i += blockDim.x) hy[i] = 0.f;
    if (own)
        for (int i = tid; i < (own + 1) * A; i += blockDim.x) U[i] = in[(long)((z0 + i / A) % g.n3) * A + i % A];
    float *const below = peer(hy, (rank + busy - 1) % busy), *const above = peer(hz, (rank + 1) % busy);
    // this thread's first column and its neighbours; others are found as met
    int xm, ym, xp, yp;
    auto column = [&](int c) {
        const int i1 = c % g.n1;
        xm = i1 == 0 ? c + g.n1 - 1 : c - 1;
        ym = c < g.n1 ? c + A - g.n1 : c - g.n1;
        xp = i1 + 1 == g.n1 ? c - i1 : c + 1;
        yp = c + g.n1 < A ? c + g.n1 : i1;
    };
    const bool work = own && tid < lanes, one = A <= lanes;
    column(tid);
    double t = 1.0;
    auto momentum = [&](int h) {  // TV_FISTA_method.m:31, rounded as on the host
        const double t0 = t;
        t = __ddiv_rn(__dadd_rn(1.0, __dsqrt_rn(__dadd_rn(1.0, __dmul_rn(__dmul_rn(4.0, t0), t0)))), 2.0);
        s_m[h] = __ddiv_rn(t0 - 1.0, t);
    };
    const bool clock = FISTA && tid == (int)blockDim.x - 1;
    if (clock) momentum(0);
    cluster_sync();
    for (int it = 0; it < niter; ++it) {
        const int h = it & 1;
        const float *hyc = hy + 3 * h * A, *hzc = hz + h * A;
        if (work)
            for (int c = tid; c < A; c += lanes) {
                if (!one) column(c);
                float y3m = hzc[c];
                for (int k = 0; k <= own; ++k) {
                    const float *q = k < own ? Y + 3 * k * A : hyc;
                    const float y3 = q[2 * A + c];
                    const float d = q[c] + q[A + c] + y3 - q[xm] - q[A + ym] - y3m;
                    D[k * A + c] = d - U[k * A + c] * inv_lam;
                    y3m = y3;
                }
            }
        __syncthreads();
        if (work) {
            const double m = FISTA ? s_m[h] : 0.0;
            for (int c = tid; c < A; c += lanes) {
                if (!one) column(c);
                for (int k = 0; k < own; ++k) {
                    const float *dk = D + k * A;
                    float *q = Y + 3 * k * A + c;
                    const float d0 = dk[c];
                    const float t1 = tau * (dk[xp] - d0);
                    const float t2 = tau * (dk[yp] - d0);
                    const float t3 = tau * (dk[A + c] - d0);
                    float p[3], f[3];
                    tv_project(q[0] + t1, q[A] + t2, q[2 * A] + t3, p[0], p[1], p[2]);
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        f[e] = p[e];
                        if constexpr (FISTA) {
                            float *o = Pp + (3 * k + e) * A + c;
                            f[e] = (float)(p[e] + m * (p[e] - (double)*o));
                            *o = p[e];
                        }
                        q[e * A] = f[e];
                        if (k == 0) below[(3 * (h ^ 1) + e) * A + c] = f[e];
                    }
                    if (k == own - 1) above[(h ^ 1) * A + c] = f[2];
                }
            }
        } else if (clock) {
            momentum(h ^ 1);
        }
        cluster_sync();
    }
    const float *res = FISTA ? Pp : Y;
    for (int i = tid; i < 3 * own * A; i += blockDim.x)
        Pout[(i / A % 3) * g.V + (long)(z0 + i / (3 * A)) * A + i % A] = res[i];
}

__global__ void k_tv_out4(const float *P, const float *in, float *out, Rows g, float lam) {
    const long V = g.V;
    const int q1 = g.n1 / 4;
    for (int row = blockIdx.x; row < g.n2 * g.n3; row += gridDim.x) {
        const int i2 = row % g.n2, i3 = row / g.n2;
        const long b = g.at(i2, i3), b2 = g.at(i2 == 0 ? g.n2 - 1 : i2 - 1, i3),
                   b3 = g.at(i2, i3 == 0 ? g.n3 - 1 : i3 - 1);
        for (int k = threadIdx.x; k < q1; k += blockDim.x) {
            const int i1 = 4 * k;
            const long r = b + i1;
            const float4 p1 = ld4(P + r), p2 = ld4(P + V + r), p3 = ld4(P + 2 * V + r);
            const float4 m2 = ld4(P + V + b2 + i1), m3 = ld4(P + 2 * V + b3 + i1), u = ld4(in + r);
            const float p1m = P[b + (i1 == 0 ? g.n1 - 1 : i1 - 1)];
            float4 o;
            o.x = u.x - lam * (p1.x + p2.x + p3.x - p1m - m2.x - m3.x);
            o.y = u.y - lam * (p1.y + p2.y + p3.y - p1.x - m2.y - m3.y);
            o.z = u.z - lam * (p1.z + p2.z + p3.z - p1.y - m2.z - m3.z);
            o.w = u.w - lam * (p1.w + p2.w + p3.w - p1.z - m2.w - m3.w);
            st4(out + r, o);
        }
    }
}

// in = vol / max(vol) with max from *mx; the max itself by k_max
__global__ void k_max(const float *v, long n, unsigned *mx_bits) {
    float m = -INFINITY;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        m = fmaxf(m, v[i]);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    // order-preserving integer image of the float
    if ((threadIdx.x & 31) == 0) {
        unsigned b = __float_as_uint(m);
        b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
        atomicMax(mx_bits, b);
    }
}

__global__ void k_bits_to_float(const unsigned *mx_bits, float *mx) {
    unsigned b = *mx_bits;
    b = (b & 0x80000000u) ? (b & 0x7fffffffu) : ~b;
    *mx = __uint_as_float(b);
}

__global__ void k_scale(const float *v, float *out, long n, const float *div) {
    const float d = *div;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        out[i] = v[i] / d;
}

__global__ void k_mul(const float *v, float *out, long n, const float *mul) {
    const float m = *mul;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        out[i] = v[i] * m;
}

__global__ void k_positivity(float *v, long n) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        if (v[i] < 0.f) v[i] = 0.f;
}

// beam-frame volume of a tilt: V[z][y][x] (n x n window) = centred copy of
// the rotated nv^3 volume (zero elsewhere): the volume zero-padded laterally
// to the probe window (exact under the periodic multislice: V = 0 gives T = 1)
// beam-frame volume [n3][n2][n1] centred in the n x n window: V [n3][n][n]
__global__ void k_pad(const float *src, float *V, int n1, int n2, int n3, int n) {
    const long nn = (long)n * n, total = nn * n3;
    const int o1 = (n - n1) / 2, o2 = (n - n2) / 2;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int z = (int)(i / nn), y = (int)((i / n) % n), x = (int)(i % n);
        const int yy = y - o2, xx = x - o1;
        V[i] = (yy >= 0 && yy < n2 && xx >= 0 && xx < n1) ? src[((long)z * n2 + yy) * n1 + xx] : 0.f;
    }
}

// lab-frame gradient contribution of a tilt: slab gradient G[s] (n x n,
// FP64) replicated over the slab's voxels and cropped to the [n3][n2][n1] volume
__global__ void k_slab_to_volume(const double *G, float *out, int n1, int n2, int n3, int n, int b) {
    const long total = (long)n1 * n2 * n3;
    const int o1 = (n - n1) / 2, o2 = (n - n2) / 2;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int z = (int)(i / ((long)n1 * n2)), y = (int)((i / n1) % n2), x = (int)(i % n1);
        out[i] = (float)G[(long)(z / b) * n * n + (long)(y + o2) * n + (x + o1)];
    }
}

__global__ void k_accumulate(const float *g, double *acc, long n, int zero) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        acc[i] = (zero ? 0.0 : acc[i]) + (double)g[i];
}

// rec += step0 * acc
__global__ void k_update(float *rec, const double *acc, long n, float step0) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        rec[i] += step0 * (float)acc[i];
}
}  // namespace

namespace {
// rows of whole float4 groups, at most one CTA long
inline bool tv_rows4(int n1) { return n1 % 4 == 0 && n1 <= 1024; }

// Whether K slices per CTA of planes of A voxels run on the cluster kernel; march:
// the marching kernel is the other choice, else two kernels per iteration are.
// The cluster's time per iteration is a thread's chain through its columns, 0.3 to
// 0.6 us a slice by the warps there are, on top of 0.9; the march takes 2.4 to 3.0
// whatever the volume up to 40^3.  Microseconds per iteration in a captured
// graph (one B200, cluster / march; bare launches of the march cost 0.2 more):
//   FISTA  24^3 (K 2)  1.87 / 2.66   16x16x64 (K 4)  2.28 / 2.49   24x24x48 (K 3)  2.50 / 2.68
//          24x24x64 (K 4)  3.08 / 2.66   24x32x48 (K 3)  2.84 / 2.67   16x16x128 (K 8)  3.95 / 2.46
//          32^3 (K 2, two columns a thread)  4.16 / 2.70   24x24x160 (K 10)  6.42 / 3.25
//   TV     24x24x48 (K 3)  1.84 / 2.45   24x24x64 (K 4)  2.23 / 2.44   24x24x96 (K 6)  2.98 / 2.60
//          16x16x128 (K 8)  2.71 / 2.28   32^3 (K 2)  3.28 / 2.47
// Against two kernels per iteration (8.2 bare for FISTA and TV alike):
//   FISTA  30x30x60 (K 4)  4.3   34^3 (K 3, two columns)  5.6   26x26x100 (K 7)  5.3
//          9x9x200 (K 13)  5.6   6x6x500 (K 32)  13.0   5x5x4000 (K 250)  97.9 (two kernels: 18.4)
inline bool tv_cluster_pays(long A, int K, bool fista, bool march) {
    const long columns = (A + 991) / 992;  // per thread
    if (march) return columns == 1 && K <= 4 && A * K <= (fista ? 1728 : 2304);
    return columns * K <= 16;
}

// launch configuration of the cluster kernel over a volume; false: it does not
// fit one cluster's shared memory, or another route is faster
template <bool FISTA>
struct TvCluster {
    cudaLaunchAttribute at[1] = {};
    cudaLaunchConfig_t cfg = {};
    int K = 0;
    bool prepare(int n1, int n2, int n3, bool march, cudaStream_t st) {
        const long A = (long)n1 * n2;
        for (int cl : {kTvCl, 8}) {
            K = (n3 + cl - 1) / cl;
            const long bytes = tv_cluster_floats(A, K, FISTA) * (long)sizeof(float);
            if (bytes > 220 * 1024 || !tv_cluster_pays(A, K, FISTA, march)) continue;
            auto k = k_tv_cluster<FISTA>;
            if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
                (cl > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
                cudaGetLastError();  // the answer, not a later launch's error
                continue;
            }
            cfg.gridDim = dim3(cl);
            cfg.blockDim = dim3((unsigned)std::min(992L, (A + 31) / 32 * 32) + 32);
            cfg.dynamicSmemBytes = (size_t)bytes;
            cfg.stream = st;
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cl;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cl <= 8) return true;
            if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) cudaGetLastError();
            else if (n > 0) return true;
        }
        return false;
    }
};
// every iteration in one launch; -1: not on this route
template <bool FISTA>
int tv_cluster(const TvArgs &a, bool march, const Rows &rows, float inv_lam, float tau, cudaStream_t st) {
    TvCluster<FISTA> c;
    if (!c.prepare(a.n1, a.n2, a.n3, march, st)) return -1;
    return (int)cudaLaunchKernelEx(&c.cfg, k_tv_cluster<FISTA>, a.P, a.in, rows, c.K, inv_lam, tau, a.niter);
}
}  // namespace

bool tv_wants_second(int n1, int n2, int n3, bool fista) {
    TvCluster<true> c;
    return fista && tv_rows4(n1) && !c.prepare(n1, n2, n3, true, nullptr);
}

int tv_prox(const TvArgs &a, cudaStream_t st) {
    const long V = (long)a.n1 * a.n2 * a.n3;
    const Rows rows{a.n1, a.n2, a.n3, V};
    // threads over i1 (whole warps, at most 256), CTAs over rows: up to 16
    // CTAs of 128 threads per SM
    const int bt = std::min(256, (a.n1 + 31) / 32 * 32);
    const int g = (int)std::min<long>((long)a.n2 * a.n3, 148L * (2048 / bt));
    // four voxels per thread where rows split into 16-byte groups (every
    // array is 16-byte aligned and n1 a multiple of 4)
    const bool vec = a.n1 % 4 == 0;
    const int bt4 = std::min(256, std::max(1, (a.n1 / 4 + 31) / 32) * 32);
    const int g4 = (int)std::min<long>((long)a.n2 * a.n3, 148L * std::min(32, 2048 / bt4));
    const float tau = 1.0f / 12.0f;  // 3D (TV_method.m:13-16)
    const float inv_lam = (float)(1.0 / a.lambda);
    float *res = a.P;  // the dual field after the last iteration
    cudaError_t e;
    int rc = -1;
    // one kernel per iteration needs a second dual field: Y2 (FISTA), or P and Y
    // in turn
    const bool march = tv_rows4(a.n1) && (!a.fista || a.Y2);
    if (a.niter > 0)
        rc = a.fista ? tv_cluster<true>(a, march, rows, inv_lam, tau, st)
                     : tv_cluster<false>(a, march, rows, inv_lam, tau, st);
    if (rc > 0) return rc;
    if (rc < 0) {
        if ((e = cudaMemsetAsync(a.P, 0, sizeof(float) * 3 * V, st)) != cudaSuccess) return (int)e;
        if ((e = cudaMemsetAsync(a.Y, 0, sizeof(float) * 3 * V, st)) != cudaSuccess) return (int)e;
        const int q1 = std::max(1, a.n1 / 4), ty = std::max(1, std::min(128 / q1, a.n2));
        const int tiles = (a.n2 + ty - 1) / ty;
        // chunks of zc slices: every wave of resident CTAs (80 registers: 25 warps an
        // SM) takes a chunk's chain, 1.4 us a slice and 0.9 slices' time to start,
        // however full it is; what moves through memory comes on top of that
        // alike for every zc.  Within 3% of the best zc at each of 34 volumes timed,
        // 4x4x1000 to 256^3 (128^3: 16.4 us an iteration at zc = 5, one wave; 17.1 at
        // 3, two; 19.0 at 7; 19.5 at 1, five; 160x160x96: 21.0 at 6, 24.4 at 8;
        // 192x192x96: 32.7 at 8, 43.6 at 16; 256x256x64: 38.4 at 5, 42.2 at 13)
        const double wave = 148.0 * (25 / ((q1 * ty + 31) / 32));
        int zc = 1;
        double best = 0;
        for (int c = 1; c <= std::min(16, a.n3); ++c) {
            const double cost = (c + 0.9) * std::ceil(tiles * ((a.n3 + c - 1) / c) / wave);
            if (c == 1 || cost < best) {
                best = cost;
                zc = c;
            }
        }
        const int grid = tiles * ((a.n3 + zc - 1) / zc);
        const size_t sm = sizeof(float) * 2 * (size_t)(ty + 1) * a.n1;
        float *src = a.fista ? a.Y : a.P, *dst = a.fista ? a.Y2 : a.Y;
        double t = 1.0;
        for (int it = 0; it < a.niter; ++it) {
            const double t0 = t;
            t = (1.0 + std::sqrt(1.0 + 4.0 * t0 * t0)) / 2.0;  // TV_FISTA_method.m:31
            const double m = (t0 - 1.0) / t;
            if (march) {
                // set up while the iteration before drains; the first follows
                // the clearing of its fields
                cudaLaunchAttribute chain = {};
                chain.id = cudaLaunchAttributeProgrammaticStreamSerialization;
                chain.val.programmaticStreamSerializationAllowed = 1;
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(grid);
                cfg.blockDim = dim3(q1 * ty);
                cfg.dynamicSmemBytes = sm;
                cfg.stream = st;
                cfg.attrs = &chain;
                cfg.numAttrs = it > 0 ? 1 : 0;
                e = cudaLaunchKernelEx(&cfg, a.fista ? k_tv_march<true> : k_tv_march<false>, (const float *)src, dst,
                                       a.fista ? a.P : nullptr, a.in, rows, ty, zc, inv_lam, tau, m);
                if (e != cudaSuccess) return (int)e;
                std::swap(src, dst);
            } else {
                k_tv_d<<<g, bt, 0, st>>>(a.fista ? a.Y : a.P, a.in, a.D, rows, inv_lam);
                k_tv_step<<<g, bt, 0, st>>>(a.P, a.Y, a.D, rows, tau, m, a.fista);
            }
        }
        if (march && !a.fista) res = src;
    }
    if (vec) k_tv_out4<<<g4, bt4, 0, st>>>(res, a.in, a.out, rows, (float)a.lambda);
    else k_tv_out<<<g, bt, 0, st>>>(res, a.in, a.out, rows, (float)a.lambda);
    if (a.err) k_tv_err<<<g, bt, 0, st>>>(a.out, rows, a.lambda, a.err);
    return (int)cudaGetLastError();
}

int vol_max(const float *v, long n, unsigned *bits, float *mx, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(bits, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return (int)e;
    k_max<<<grid_for(n), kThreads, 0, st>>>(v, n, bits);
    k_bits_to_float<<<1, 1, 0, st>>>(bits, mx);
    return (int)cudaGetLastError();
}

int vol_scale(const float *v, float *out, long n, const float *div, cudaStream_t st) {
    k_scale<<<grid_for(n), kThreads, 0, st>>>(v, out, n, div);
    return (int)cudaGetLastError();
}

int vol_mul(const float *v, float *out, long n, const float *mul, cudaStream_t st) {
    k_mul<<<grid_for(n), kThreads, 0, st>>>(v, out, n, mul);
    return (int)cudaGetLastError();
}

int vol_positivity(float *v, long n, cudaStream_t st) {
    k_positivity<<<grid_for(n), kThreads, 0, st>>>(v, n);
    return (int)cudaGetLastError();
}

int vol_pad(const float *src, float *V, int n1, int n2, int n3, int n, cudaStream_t st) {
    k_pad<<<grid_for((long)n * n * n3), kThreads, 0, st>>>(src, V, n1, n2, n3, n);
    return (int)cudaGetLastError();
}

int vol_slab_to_volume(const double *G, float *out, int n1, int n2, int n3, int n, int b, cudaStream_t st) {
    k_slab_to_volume<<<grid_for((long)n1 * n2 * n3), kThreads, 0, st>>>(G, out, n1, n2, n3, n, b);
    return (int)cudaGetLastError();
}

int vol_accumulate(const float *g, double *acc, long n, bool zero, cudaStream_t st) {
    k_accumulate<<<grid_for(n), kThreads, 0, st>>>(g, acc, n, zero ? 1 : 0);
    return (int)cudaGetLastError();
}

int vol_update(float *rec, const double *acc, long n, float step0, cudaStream_t st) {
    k_update<<<grid_for(n), kThreads, 0, st>>>(rec, acc, n, step0);
    return (int)cudaGetLastError();
}

}  // namespace mset
