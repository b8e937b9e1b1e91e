// seq_kernel.cuh -- the sequential modes (kSeq: the reference-semantics pass,
// kStep: the per-position steps) on one field spread over a thread-block
// cluster, for sm_100a.
//
// These modes walk one probe position at a time, so all that runs at once is
// one N x N field: the time is the length of the dependent chain (per slab a
// 2D transform, the propagator, the inverse transform, forward and adjoint),
// not arithmetic or bandwidth.  The chain here is
//
//   rows:     [inverse row transform] -> real-space stage -> [row transform]
//             -> send every column's elements to the CTA that owns the column
//   columns:  [column transform] -> Fourier-space stage -> [inverse column
//             transform] -> send every row's elements to the row's owner
//
// with CTA r of the cluster owning the rows y = n1 + R1 j of N1C residues n1
// (N = R1 R2, the one-CTA shapes' factors and scrambled layouts) and RC = N /
// CL adjacent column frequencies.  A line's transform is two register passes
// (A: R2 points, B: R1 points) with one exchange through the CTA's own shared
// memory between them.
//
// The exchanges between CTAs are st.async pushes (one remote store that also
// counts its bytes on the receiver's mbarrier), so a CTA waits for its data
// only: no cluster barrier, no release fence that would drain the saved-wave
// stores.  A push moves 16 B per clock and SM when a warp's store covers whole
// 32-byte sectors of the destination (16 KB exchanged per CTA of 8: 1231
// cycles; 2000 with 16-byte pieces at a 64-byte stride; remote stores followed
// by a cluster barrier 1490; remote loads after one 3300), so the layouts
// below put the lanes of every push side by side in the receiver's buffer.
//
// What a thread needs for the next real-space stage from global memory
// (transmission, saved wave, voxels) it fetches after its push and before it
// waits, and a slab's volume update and its new transmission are written in
// those slots too: they overlap the exchanges (the transmission computed from
// the voxels where it is used put 1777 of 4192 cycles per slab and direction
// at 64^2 on the chain).  The propagator of a thread's spectrum elements
// stays in registers for the whole call, the probe spectrum in shared memory;
// positions' sums are written per warp and added up once at the end.
//
// What bounds it: the chain.  Of 6030 cycles per slab and direction at 128^2 (8
// CTAs of 16 rows, 16 KB each way per CTA) the pushes and waits take 2860, the
// slots between them 1060, the passes 2050; of 3050 at 64^2 (8 CTAs of 8 rows)
// 1080, 720 and 1190.
// The times per window and cluster size stand at MSET_SEQ_FIELDS in
// mset_dispatch.cu.
#pragma once
#include "mset_kernels_impl.cuh"
#include "seq_exchange.h"

namespace mset {

template <int N_, int R1_, int CL_>
struct SeqGeo {
    static constexpr int N = N_, R1 = R1_, R2 = N_ / R1_, CL = CL_;
    static constexpr int NN = N * N;
    static constexpr int RC = N / CL;    // rows (and columns) per CTA
    static constexpr int N1C = R1 / CL;  // residues n1 per CTA
    static constexpr int NT = RC * R1;   // one pass-A task (line, n1) per thread
    static constexpr int NB = RC * R2;   // pass-B tasks (line, k2)
    static constexpr int NW = NT / 32;
    static constexpr bool EVEN = R2 % 2 == 0;  // 16-byte pass-A accesses
    // element (n1, line, t) at (n1 / N1C) BLK + line RCP + (n1 % N1C) R2 + t.
    // RCP / 2 odd and BLK = 2 mod 16 keep the 16-byte pass-A accesses of 8
    // adjacent lines or of 8 adjacent residues on different banks (R2 odd:
    // 8-byte accesses, odd strides)
    static constexpr int RCP = EVEN ? (RC % 4 == 2 ? RC : RC + 2) : (RC % 2 ? RC : RC + 1);
    static constexpr int BLK = CL == 1 ? RC * RCP : EVEN ? (RC * RCP + 13) / 16 * 16 + 2 : RC * RCP + 1;
    static constexpr int FIELD = CL * BLK;
    // pass-B tasks of a half-warp: 8 lines x 2 k2 where that keeps 8-byte
    // accesses at a stride of 4 banks apart
    static constexpr bool SPLIT_B = RC % 16 == 0 && R2 % 2 == 0;
    static_assert(R1 * R2 == N && R1 % CL == 0 && N % CL == 0, "the cluster deals out whole residues and columns");
    static_assert(NT % 32 == 0 && NT <= 1024 && NB <= NT, "one pass-A task per thread");
    __device__ __forceinline__ static int at(int n1, int line, int t) {
        return (n1 / N1C) * BLK + line * RCP + (n1 % N1C) * R2 + t;
    }
    // dynamic shared memory: row buffer, column buffer, probe spectrum, the
    // shift factors of the position
    static constexpr int COL = (FIELD + 1) & ~1, QS = 2 * COL, E1 = QS + RC * N, E2 = E1 + N, END = E2 + N;
    static constexpr size_t kSmem = sizeof(float2) * END;
};

__device__ __forceinline__ void st_async(uint32_t addr, float2 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "r"(bar)
                 : "memory");
}
// bounded wait on an mbarrier phase that remote pushes complete
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (i > 1024) __nanosleep(64);
    }
    return false;
}

template <class G, int METHOD, int ADJ, int MODE>
struct SeqKernel {
    static constexpr int N = G::N, NN = G::NN, R1 = G::R1, R2 = G::R2, CL = G::CL, RC = G::RC, N1C = G::N1C;

    // voxel planes of a slab fetched a stage ahead of their update (registers)
    static constexpr int kPlanes = R2 <= 10 ? 2 : 1;

    const LaunchArgs &a;
    float2 *const rowbuf, *const colbuf, *const qs, *const e1, *const e2;
    uint32_t bars;          // shared address of the row mbarrier; the column one follows
    uint32_t peer_base[CL];  // shared::cluster address of every CTA's dynamic shared memory
    uint32_t peer_bars[CL];
    uint32_t row_base = 0, row_bar = 0;  // the CTA that owns the rows of the column pass-A task
    int rank;
    SeqProgress at_x;  // exchanges so far
    // pass-A tasks: row (yr, n1r) and column (xc, n1c); pass-B task (lb, kb) of
    // rows and of columns alike
    int n1r, lr, n1c, lc, lb, kb;
    bool tb;
    int y;                 // field row of the row pass-A task
    float2 twr[R2], twc[R2];  // twiddles W^(n1 k2), sign -1
    float2 P[R1];          // propagator / N^2 of the column pass-B task

    __device__ __forceinline__ SeqKernel(const LaunchArgs &args, float2 *sm, uint64_t *mb)
        : a(args), rowbuf(sm), colbuf(sm + G::COL), qs(sm + G::QS), e1(sm + G::E1), e2(sm + G::E2) {
        const int t = threadIdx.x;
        rank = 0;
        if constexpr (CL > 1) {
            unsigned r;
            asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
            rank = (int)r;
            bars = (uint32_t)__cvta_generic_to_shared(mb);
#pragma unroll
            for (int q = 0; q < CL; ++q) {
                peer_base[q] = peer_addr(sm, q);
                peer_bars[q] = peer_addr(mb, q);
            }
            if (t == 0) {
                for (int i = 0; i < 2; ++i)
                    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8u * i) : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
        }
        n1r = t % R1;
        lr = t / R1;
        lc = t % RC;
        n1c = t / RC;
        if constexpr (CL > 1) {
            row_base = peer_addr(sm, n1c / N1C);
            row_bar = peer_addr(mb, n1c / N1C);
        }
        tb = t < G::NB;
        if constexpr (G::SPLIT_B) {
            const int u = t / 16;
            lb = t % 8 + 8 * (u % (RC / 8));
            kb = (t / 8) % 2 + 2 * (u / (RC / 8));
        } else {
            lb = t % RC;
            kb = t / RC;
        }
        y = row_of(lr);
#pragma unroll
        for (int k = 0; k < R2; ++k) {
            twr[k] = a.twn[k * R1 + n1r];
            twc[k] = a.twn[k * R1 + n1c];
        }
        if (tb) {
#pragma unroll
            for (int i = 0; i < R1; ++i)
                P[i] = a.psep ? cmul(a.psep[loc_y(i)], a.psep[N + loc_x()]) : a.pscr[(size_t)loc_y(i) * N + loc_x()];
        }
        if constexpr (CL > 1) {
            __syncthreads();
            arm(0);
            arm(1);
            cluster_sync();
        }
    }

    // field row of local row l; scrambled locations and frequencies of element
    // i of this thread's column pass-B task
    __device__ __forceinline__ int row_of(int l) const { return rank * N1C + l / R2 + R1 * (l % R2); }
    __device__ __forceinline__ int loc_y(int i) const { return i + R1 * kb; }
    __device__ __forceinline__ int frq_y(int i) const { return kb + R2 * i; }
    __device__ __forceinline__ int frq_x() const { return rank * RC + lb; }
    __device__ __forceinline__ int loc_x() const { return frq_x() / R2 + R1 * (frq_x() % R2); }

    // expect the next exchange's bytes: which = 0 rows, 1 columns (thread 0,
    // once per phase, after the phase before has completed)
    __device__ __forceinline__ void arm(int which) {
        if (threadIdx.x == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8u * which),
                         "r"((unsigned)(RC * N * sizeof(float2)))
                         : "memory");
    }
    // Every thread waits for its exchange.  A buffer is written again only
    // when every CTA has received the exchange in between, which this CTA's
    // threads send after their last reads of it; and no phase can complete
    // twice unseen, since each stage's CTA barrier stands between this wait
    // and those sends.
    __device__ __forceinline__ void wait(int which) {
        if constexpr (CL == 1) {
            __syncthreads();
        } else {
            bool done = true;
            if (at_x.waits()) {
                const unsigned par = at_x.parity(which);
                done = mbar_wait_cluster(bars + 8u * which, par);
                if (!done) {
                    if (a.fault) atomicOr(a.fault, 1u);
                    mbar_wait_cluster(bars + 8u * which, par);  // let late pushes land
                }
            }
            at_x.waited(which, done);
            if (at_x.arms()) arm(which);
        }
    }
    // this CTA's element `off` of the row (which = 0) or column buffer of CTA q
    __device__ __forceinline__ void push(int which, uint32_t base, uint32_t bar, int off, float2 v) const {
        if constexpr (CL == 1) (which ? colbuf : rowbuf)[off] = v;
        else if (at_x.sends())
            st_async(base + (uint32_t)sizeof(float2) * (uint32_t)((which ? G::COL : 0) + off), v, bar + 8u * which);
    }

    static __device__ __forceinline__ void load_a(const float2 *p, float2 *v) {
        if constexpr (G::EVEN) {
#pragma unroll
            for (int k = 0; k < R2; k += 2) {
                const float4 q = *reinterpret_cast<const float4 *>(p + k);
                v[k] = make_float2(q.x, q.y);
                v[k + 1] = make_float2(q.z, q.w);
            }
        } else {
#pragma unroll
            for (int k = 0; k < R2; ++k) v[k] = p[k];
        }
    }
    static __device__ __forceinline__ void store_a(float2 *p, const float2 *v) {
        if constexpr (G::EVEN) {
#pragma unroll
            for (int k = 0; k < R2; k += 2)
                *reinterpret_cast<float4 *>(p + k) = make_float4(v[k].x, v[k].y, v[k + 1].x, v[k + 1].y);
        } else {
#pragma unroll
            for (int k = 0; k < R2; ++k) p[k] = v[k];
        }
    }
    // pass A of sign SG: scrambled -> natural (twiddle, transform) or back
    template <int SG>
    static __device__ __forceinline__ void a_in(float2 *v, const float2 *tw) {
#pragma unroll
        for (int k = 1; k < R2; ++k) v[k] = cmul(v[k], SG < 0 ? tw[k] : cconj(tw[k]));
        DFT<R2, SG>::run(v);
    }
    template <int SG>
    static __device__ __forceinline__ void a_out(float2 *v, const float2 *tw) {
        DFT<R2, SG>::run(v);
#pragma unroll
        for (int k = 1; k < R2; ++k) v[k] = cmul(v[k], SG < 0 ? tw[k] : cconj(tw[k]));
    }

    // rows: finish the inverse transform of sign IN, op on the R2 values at
    // x = n1r + R1 j of field row y, start the transform of sign OUT
    template <int IN, int OUT, class Op>
    __device__ __forceinline__ void rows(Op &&op) {
        wait(0);
        if (tb) {
            float2 v[R1];
            float2 *p = rowbuf + lb * G::RCP + kb;
#pragma unroll
            for (int i = 0; i < R1; ++i) v[i] = p[G::at(i, 0, 0)];
            DFT<R1, IN>::run(v);
#pragma unroll
            for (int i = 0; i < R1; ++i) p[G::at(i, 0, 0)] = v[i];
        }
        __syncthreads();
        {
            float2 v[R2];
            float2 *p = rowbuf + G::at(n1r, lr, 0);
            load_a(p, v);
            a_in<IN>(v, twr);
            op(v);
            a_out<OUT>(v, twr);
            store_a(p, v);
        }
        __syncthreads();
        if (tb) {
            float2 v[R1];
            const float2 *p = rowbuf + lb * G::RCP + kb;
#pragma unroll
            for (int i = 0; i < R1; ++i) v[i] = p[G::at(i, 0, 0)];
            DFT<R1, OUT>::run(v);
            // column frequency kb + R2 i: CTA i / N1C, its column (i % N1C) R2 + kb
#pragma unroll
            for (int i = 0; i < R1; ++i)
                push(1, peer_base[i / N1C], peer_bars[i / N1C], rank * G::BLK + ((i % N1C) * R2 + kb) * G::RCP + lb,
                     v[i]);
        }
    }

    // columns: finish the transform of sign IN, op on the R1 spectrum values of
    // the pass-B task, start the inverse transform of sign OUT
    template <int IN, int OUT, class Op>
    __device__ __forceinline__ void cols(Op &&op) {
        if constexpr (IN != 0) {
            wait(1);
            float2 v[R2];
            float2 *p = colbuf + G::at(n1c, lc, 0);
            load_a(p, v);
            a_out<IN>(v, twc);
            store_a(p, v);
            __syncthreads();
        }
        if (tb) {
            float2 v[R1];
            float2 *p = colbuf + lb * G::RCP + kb;
            if constexpr (IN != 0) {
#pragma unroll
                for (int i = 0; i < R1; ++i) v[i] = p[G::at(i, 0, 0)];
                DFT<R1, IN>::run(v);
            }
            op(v);
            if constexpr (OUT != 0) {
                DFT<R1, OUT>::run(v);
#pragma unroll
                for (int i = 0; i < R1; ++i) p[G::at(i, 0, 0)] = v[i];
            }
        }
        if constexpr (OUT != 0) {
            __syncthreads();
            float2 v[R2];
            load_a(colbuf + G::at(n1c, lc, 0), v);
            a_in<OUT>(v, twc);
            // row n1c + R1 j: CTA n1c / N1C, its row (n1c % N1C) R2 + j
#pragma unroll
            for (int j = 0; j < R2; ++j)
                push(0, row_base, row_bar, rank * G::BLK + ((n1c % N1C) * R2 + j) * G::RCP + lc, v[j]);
        }
    }

    // voxel range of slab s
    __device__ __forceinline__ void slab(int s, int &z0, int &z1) const {
        z0 = METHOD == kSSET ? 0 : s * a.b;
        z1 = METHOD == kSSET ? a.nz : min(z0 + a.b, a.nz);
    }
    // transmission of slab s at this thread's row pass-A elements
    __device__ __forceinline__ void load_t(const TiltDev &t, int s, float2 *T) const {
        const float2 *p = t.T + (size_t)s * NN + (size_t)y * N + n1r;
#pragma unroll
        for (int j = 0; j < R2; ++j) T[j] = p[R1 * j];
    }

    // a saved-wave element that another CTA may have written
    static __device__ __forceinline__ float2 shared_wave(const float2 *p) { return CL > 1 ? __ldcg(p) : *p; }

    // one position at scan coordinates (sx, sy); part: this warp's two
    // scan-position sums; err: this thread's error sum
    __device__ __forceinline__ void position(const TiltDev &t, int p, float sx, float sy, double *part, double &err) {
        const int ns = METHOD == kSSET ? 1 : a.ns;
        float2 *const save = a.save;
        float *const V = t.V;
        const size_t el = (size_t)y * N + n1r;  // this thread's first element of a plane
        const bool fwd = MODE != kStep || a.step_phase == 1;
        const bool adj = MODE != kStep || a.step_phase == 2;
        __syncthreads();  // the shift factors of the position before are read
        {
            const float s1 = sy - a.center, s2 = sx - a.center;  // mset.cu:121
            for (int k = threadIdx.x; k < N; k += G::NT) {
                float sn, cs;
                sincosf(2.0f * MSET_REF_PI * (s1 * shift_grid(k, N) / (float)N), &sn, &cs);
                e1[k] = make_float2(cs, sn);
                sincosf(2.0f * MSET_REF_PI * (s2 * shift_grid(k, N) / (float)N), &sn, &cs);
                e2[k] = make_float2(cs, sn);
            }
        }
        __syncthreads();
        float2 T[R2], W[R2];
        if (fwd) load_t(t, 0, T);
        const float2 ex = tb ? e2[frq_x()] : make_float2(0.f, 0.f);
        if (fwd) {
            // incident wave psi0 = F(Q fs)  (mset.cu:110-131)
            cols<0, -1>([&](float2 *v) {
#pragma unroll
                for (int i = 0; i < R1; ++i) v[i] = cmul(cmul(qs[i * G::NB + threadIdx.x], e1[frq_y(i)]), ex);
            });
            rows<-1, -1>([&](float2 *v) {
#pragma unroll
                for (int j = 0; j < R2; ++j) {
                    save[el + R1 * j] = v[j];
                    v[j] = cmul(v[j], T[j]);
                }
            });
            // psi0 is read across CTAs at the end of the position
            if constexpr (ADJ == kREF && MODE != kStep && CL > 1)
                asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            // forward slabs (mset.cu:157-183)
            if constexpr (METHOD == kMSET) {
                for (int s = 0; s < ns; ++s) {
                    const bool last = s + 1 == ns;
                    if (!last) load_t(t, s + 1, T);
                    cols<-1, +1>([&](float2 *v) {
#pragma unroll
                        for (int i = 0; i < R1; ++i) v[i] = cmul(v[i], P[i]);
                    });
                    rows<+1, -1>([&](float2 *v) {
                        float2 *o = save + (size_t)(s + 1) * NN + el;
#pragma unroll
                        for (int j = 0; j < R2; ++j) {
                            o[R1 * j] = v[j];
                            if (!last) v[j] = cmul(v[j], T[j]);
                        }
                    });
                }
            }
        }
        // what the adjoint of slab s reads: the transmission, the saved wave
        // (REF: the one saved after the slab, mset.cu:248-251; EXACT: the one
        // entering it) and the first voxel planes of the volume update
        const bool grow = MODE != kStep || a.step04;  // RVol += step0 Re(g)
        float vox[kPlanes][R2];
        auto operands = [&](int s) {
            const float2 *w = save + (size_t)((METHOD == kSSET || ADJ == kEXACT) ? s : s + 1) * NN + el;
#pragma unroll
            for (int j = 0; j < R2; ++j) W[j] = w[R1 * j];
            load_t(t, s, T);
            if (grow) {
                int z0, z1;
                slab(s, z0, z1);
#pragma unroll
                for (int k = 0; k < kPlanes; ++k)
                    if (z0 + k < z1)
#pragma unroll
                        for (int j = 0; j < R2; ++j) vox[k][j] = V[(size_t)(z0 + k) * NN + el + R1 * j];
            }
        };
        if (adj) operands(ns - 1);
        // far field, error, residual (mset.cu:186-227)
        float M[R1];
        const size_t lo = tb ? (size_t)loc_x() : 0;
        if (fwd && tb) {
            const float *amp = t.amp + (size_t)p * NN + lo;
#pragma unroll
            for (int i = 0; i < R1; ++i) M[i] = __ldg(amp + (size_t)loc_y(i) * N);
        }
        auto to_adjoint = [&](float2 r, int i) {
            return METHOD == kMSET ? cmulc(r, P[i]) : cscale(r, 1.0f / (float)NN);
        };
        if constexpr (MODE == kStep) {
            if (a.step_phase == 1) {
                // STEP02_FORWARD_4D.m:36-49: residual (scrambled), |Psi|^2 (centred)
                cols<-1, 0>([&](float2 *v) {
#pragma unroll
                    for (int i = 0; i < R1; ++i) {
                        const float a2 = v[i].x * v[i].x + v[i].y * v[i].y;
                        const float A = sqrtf(a2 + 1e-30f);
                        const float d = A - M[i];
                        err += (double)(d * d);
                        a.step_resi[(size_t)loc_y(i) * N + lo] = cscale(v[i], 1.0f - M[i] / A);
                        const int h = (N + 1) / 2;
                        int r = frq_y(i) - h, c = frq_x() - h;
                        if (r < 0) r += N;
                        if (c < 0) c += N;
                        a.step_calc[(size_t)r * N + c] = a2;
                    }
                });
                return;
            }
            // STEP03_BACK.m:10-13
            cols<0, +1>([&](float2 *v) {
#pragma unroll
                for (int i = 0; i < R1; ++i) v[i] = to_adjoint(a.step_resi[(size_t)loc_y(i) * N + lo], i);
            });
        } else {
            cols<-1, +1>([&](float2 *v) {
#pragma unroll
                for (int i = 0; i < R1; ++i) {
                    const float a2 = v[i].x * v[i].x + v[i].y * v[i].y;
                    const float A = sqrtf(a2 + 1e-30f);
                    const float d = A - M[i];
                    err += (double)(d * d);
                    v[i] = to_adjoint(cscale(v[i], 1.0f - M[i] / A), i);
                }
            });
        }
        // adjoint (mset.cu:232-271; STEP03_BACK.m:12-26)
        double pdx = 0.0, pdy = 0.0;
        float du[R2];
        auto gradient = [&](int s, float2 *v) {
#pragma unroll
            for (int j = 0; j < R2; ++j) {
                const float2 u = cmulc(cmulc(v[j], T[j]), W[j]);  // g = i conj(T) conj(psi) chi
                du[j] = a.step0 * -u.y;
                if constexpr (MODE == kStep)
                    a.step_grad[(size_t)s * NN + el + R1 * j] = make_float2(-u.y, u.x);
                v[j] = cmulc(v[j], T[j]);
            }
        };
        // RVol += step0 Re(g) on every voxel of the slab (mset.cu:273-284), by
        // the thread that reads these voxels; sum: the slab's new column sums
        float sum[R2];
        auto update = [&](int s) {
            if (!grow) return;
            int z0, z1;
            slab(s, z0, z1);
            float *q = V + el;
#pragma unroll
            for (int j = 0; j < R2; ++j) sum[j] = 0.f;
#pragma unroll
            for (int k = 0; k < kPlanes; ++k)
                if (z0 + k < z1)
#pragma unroll
                    for (int j = 0; j < R2; ++j) {
                        const float o = vox[k][j] + du[j];
                        q[(size_t)(z0 + k) * NN + R1 * j] = o;
                        sum[j] += o;
                    }
            for (int z = z0 + kPlanes; z < z1; ++z) {
                float o[R2];
#pragma unroll
                for (int j = 0; j < R2; ++j) o[j] = q[(size_t)z * NN + R1 * j];
#pragma unroll
                for (int j = 0; j < R2; ++j) {
                    o[j] += du[j];
                    q[(size_t)z * NN + R1 * j] = o[j];
                    sum[j] += o[j];
                }
            }
        };
        // the updated slab's transmission, for the next position: half of it in
        // each of the slab's two slots (a sincosf costs about 110 cycles)
        auto retransmit = [&](int s, auto half) {
            if constexpr (MODE != kStep) {
                constexpr int H = decltype(half)::value, J0 = H ? R2 / 2 : 0, J1 = H ? R2 : R2 / 2;
                float2 *o = const_cast<float2 *>(t.T) + (size_t)s * NN + el;
#pragma unroll
                for (int j = J0; j < J1; ++j) {
                    float sn, cs;
                    sincosf(a.sdz * sum[j], &sn, &cs);
                    o[R1 * j] = make_float2(cs, sn);
                }
            }
        };
        for (int s = ns - 1; s > 0; --s) {
            rows<+1, -1>([&](float2 *v) { gradient(s, v); });
            update(s);
            operands(s - 1);
            retransmit(s, IC<0>{});
            cols<-1, +1>([&](float2 *v) {
#pragma unroll
                for (int i = 0; i < R1; ++i) v[i] = cmulc(v[i], P[i]);
            });
            retransmit(s, IC<1>{});
        }
        if constexpr (ADJ == kREF && MODE != kStep) {
            if constexpr (CL > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
        rows<+1, +1>([&](float2 *v) {
            gradient(0, v);
            // scan-position direction: finite differences of conj(psi0)
            // (mset.cu:316-327; utility.cu:829-876)
            if constexpr (ADJ == kREF) {
#pragma unroll
                for (int j = 0; j < R2; ++j) {
                    const int x = n1r + R1 * j;
                    const float2 *f = save + el + R1 * j;
                    const int xm = x == 0 ? 0 : -1, xp = x == N - 1 ? 0 : 1;
                    const int ym = y == 0 ? 0 : -N, yp = y == N - 1 ? 0 : N;
                    float2 dx = csub(shared_wave(f + xp), shared_wave(f + xm));
                    float2 dy = csub(shared_wave(f + yp), shared_wave(f + ym));
                    if (xp - xm == 2) dx = cscale(dx, 0.5f);
                    if (yp - ym == 2 * N) dy = cscale(dy, 0.5f);
                    pdx += (double)(dx.x * v[j].x + dx.y * v[j].y);  // Re(conj(d) chi0)
                    pdy += (double)(dy.x * v[j].x + dy.y * v[j].y);
                }
            }
        });
        update(0);
        retransmit(0, IC<0>{});
        // probe direction d = F^{-1}(chi0) fs(-s), applied to the spectrum
        // (mset.cu:288-312); EXACT: spectral derivative of psi0 by position
        const float inv = 1.0f / (float)NN;
        cols<+1, 0>([&](float2 *v) {
            const float kx = 2.0f * MSET_REF_PI * shift_grid(frq_x(), N) / (float)N;
#pragma unroll
            for (int i = 0; i < R1; ++i) {
                const float2 fs = cmul(e1[frq_y(i)], ex);
                const float2 d = cscale(cmulc(v[i], fs), inv);
                float2 q = qs[i * G::NB + threadIdx.x];
                if constexpr (ADJ == kEXACT) {
                    const float2 qf = cmul(q, fs);
                    const float ky = 2.0f * MSET_REF_PI * shift_grid(frq_y(i), N) / (float)N;
                    const float2 Xx = make_float2(-qf.y * kx, qf.x * kx);
                    const float2 Xy = make_float2(-qf.y * ky, qf.x * ky);
                    pdx -= (double)(Xx.x * v[i].x + Xx.y * v[i].y);
                    pdy -= (double)(Xy.x * v[i].x + Xy.y * v[i].y);
                }
                q.x -= a.step1 * d.x;
                q.y -= a.step1 * d.y;
                qs[i * G::NB + threadIdx.x] = q;
            }
        });
        retransmit(0, IC<1>{});
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            pdx += __shfl_xor_sync(0xffffffffu, pdx, o);
            pdy += __shfl_xor_sync(0xffffffffu, pdy, o);
        }
        if ((threadIdx.x & 31) == 0) {
            part[0] = pdx;
            part[1] = pdy;
        }
    }

    // the probe spectrum between global memory and this CTA's column tasks
    __device__ __forceinline__ void probe(float2 *Q, bool store) {
        if (!tb) return;
#pragma unroll
        for (int i = 0; i < R1; ++i) {
            float2 *g = Q + (size_t)loc_y(i) * N + loc_x();
            float2 *l = qs + i * G::NB + threadIdx.x;
            if (store) *g = *l;
            else *l = *g;
        }
    }
};

template <class G, int METHOD, int ADJ, int MODE>
__global__ void __launch_bounds__(G::NT, 1) k_sequential(const LaunchArgs a) {
    extern __shared__ __align__(16) float2 smem[];
    __shared__ __align__(8) uint64_t mbars[2];
    const TiltDev t = a.tilts[a.seq_tilt];
    SeqKernel<G, METHOD, ADJ, MODE> k(a, smem, mbars);
    constexpr int W = G::CL * G::NW;
    const int w = k.rank * G::NW + (int)(threadIdx.x >> 5);
    const int npos = MODE == kStep ? 1 : t.npos;
    k.probe(t.Q, false);
    double err = 0.0;
    if constexpr (MODE == kStep) {
        k.position(t, a.step_k, a.step_x, a.step_y, a.seq_part + 2 * w, err);
    } else {
        for (int p = 0; p < npos; ++p)
            k.position(t, p, t.sx[p], t.sy[p], a.seq_part + (size_t)2 * W * p + 2 * w, err);
    }
    k.probe(t.Q, true);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
    double *const epart = a.seq_part + (size_t)2 * W * npos;
    if ((threadIdx.x & 31) == 0) epart[w] = err;
    // every push of the cluster has landed and every partial sum is written
    if constexpr (G::CL > 1) cluster_sync();
    else __syncthreads();
    if (k.rank != 0) return;
    const bool pos = MODE != kStep || a.step_phase == 2;
    for (int p = threadIdx.x; pos && p < npos; p += G::NT) {
        double dx = 0.0, dy = 0.0;
        for (int i = 0; i < W; ++i) {
            dx += __ldcg(a.seq_part + (size_t)2 * W * p + 2 * i);
            dy += __ldcg(a.seq_part + (size_t)2 * W * p + 2 * i + 1);
        }
        if constexpr (MODE == kStep) {
            a.step_pos[0] = a.step_x + a.step2 * (float)dx;  // STEP03_BACK.m:37-38
            a.step_pos[1] = a.step_y + a.step2 * (float)dy;
        } else {
            t.sx[p] += a.step2 * (float)dx;  // mset.cu:322
            t.sy[p] += a.step2 * (float)dy;  // mset.cu:327
        }
    }
    if (threadIdx.x == 0 && (MODE != kStep || a.step_phase == 1)) {
        double e = 0.0;
        for (int i = 0; i < W; ++i) e += __ldcg(epart + i);
        *(MODE == kStep ? a.step_err : t.err) += e;
    }
}

// launch configuration of one instance (clusters of more than 8 CTAs are opt-in)
template <class G>
struct SeqConfig {
    cudaLaunchAttribute at[1] = {};
    cudaLaunchConfig_t cfg = {};
    template <class K>
    int prepare(K *k, cudaStream_t st) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::kSmem);
        if (e == cudaSuccess && G::CL > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = G::CL;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(G::CL);
        cfg.blockDim = dim3(G::NT);
        cfg.dynamicSmemBytes = G::kSmem;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = G::CL > 1 ? 1 : 0;
        return (int)e;
    }
};

template <class G, int METHOD, int ADJ, int MODE>
int seq_launch(const LaunchArgs &a, cudaStream_t st) {
    auto k = k_sequential<G, METHOD, ADJ, MODE>;
    SeqConfig<G> c;
    const int rc = c.prepare(k, st);
    return rc ? rc : (int)cudaLaunchKernelEx(&c.cfg, k, a);
}

template <class G>
int seq_positions(int method, int adjoint, int mode, const LaunchArgs &a, cudaStream_t st) {
#define MSET_L(M, A, MO) \
    if (method == M && adjoint == A && mode == MO) return seq_launch<G, M, A, MO>(a, st);
    MSET_L(kMSET, kREF, kSeq) MSET_L(kMSET, kEXACT, kSeq) MSET_L(kSSET, kREF, kSeq) MSET_L(kSSET, kEXACT, kSeq)
    MSET_L(kMSET, kREF, kStep) MSET_L(kMSET, kEXACT, kStep) MSET_L(kSSET, kREF, kStep) MSET_L(kSSET, kEXACT, kStep)
#undef MSET_L
    return (int)cudaErrorInvalidValue;
}

// whether the device can hold one cluster (8 CTAs are always schedulable)
template <class G>
bool seq_fits() {
    if constexpr (G::CL > 8) {
        auto k = k_sequential<G, kMSET, kREF, kSeq>;
        SeqConfig<G> c;
        int n = 0;
        if (c.prepare(k, nullptr) == 0 && cudaOccupancyMaxActiveClusters(&n, k, &c.cfg) == cudaSuccess) return n > 0;
        cudaGetLastError();  // the query's error is the answer, not a later launch's
        return false;
    } else {
        return true;
    }
}

}  // namespace mset

// the sequential modes of window N_ over CL_ CTAs: table entry kSeqField<N_>
#define MSET_DEFINE_SEQ(N_, R1_, CL_)                                                                      \
    namespace mset {                                                                                       \
    using SeqField##N_ = SeqGeo<N_, R1_, CL_>;                                                             \
    extern const SeqOps kSeqField##N_ = {N_, R1_, CL_, CL_ * SeqField##N_::NW, &seq_fits<SeqField##N_>,    \
                                         &seq_positions<SeqField##N_>};                                    \
    }
