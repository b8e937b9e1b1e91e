// mset_dispatch.cu -- window-size dispatch and the size-independent
// kernels of the batched update.
#include <algorithm>
#include <cmath>
#include "mset_kernels.cuh"


namespace mset {

// Every compiled geometry.  The default shape of a batched session is the
// first entry of its window whose range (lo, hi] holds its positions per SM
// (entries with an empty range are the autotuner's alternatives); the shapes
// with the same scrambled layouts are the session's variants.  The lines, by
// measurement (one B200, microseconds per pass of P positions):
//  24, 32  one shape (192 threads at 24: 81 us at P = 148, 648 at 3000, 24
//          slabs; 64 threads took 138 and 805)
//  48      192 threads with 128 registers x 2 CTAs up to 2 positions per SM
//          (314 against 363 at P = 296, 32 slabs; ahead at each of five counts
//          from 0.25 an SM on), x 4 above (448 against 498 at 2.5 an SM, 1691
//          against 1950 at 13.5; ahead at each of eight counts)
//  64      256 threads x 2 CTAs up to 6 positions per SM, 128 x 4 above.  By how
//          their last waves fill they lead in turn between 2 and 6 (32 slabs:
//          450 against 521 at 2, 670 / 646 at 3, 854 / 806 at 4, 1021 / 1089 at 5,
//          1245 / 1194 at 6); below the first is ahead (308 / 449 at 1), above the
//          second (1372 / 1334 at 6.5, 1761 / 1576 at 8, 10248 / 9385 at 54)
//  96      384 threads x 2 CTAs (80 registers; 984 against 1105 with one CTA and
//          128 registers at 1.25 positions per SM, 32 slabs, 3613 against 4396 at
//          8; ahead at each of nine counts); one CTA up to one position per SM
//          (586 against 643 at 1, 552 against 599 at 0.25)
//  128     the three-phase shape; the two-pass one serves the sequential
//          sessions
//  256     the saved-wave rows staged by bulk copies (1.443 s against 1.474 s
//          per pass of 3 large tilts)
// At 24, 32, 64 and 128 the transmission and the saved waves are kept in the
// kernel's lane order (Geo::LANES): 172.0 -> 165.2 ns per slab of a position at
// 128, 44.1 -> 42.4 at 64; at 64 the rotated rows (Geo::ROT) gave 52.3 -> 44.1.
struct GeoEntry {
    const GeoOps *g;
    float lo, hi;
};
#define MSET_GEOS(X)                                                                                          \
    X(24, 0, INFINITY) X(32, 0, INFINITY) X(48a, 2, INFINITY) X(48, 0, 2) X(64p, 6, INFINITY) X(64, 0, 6) \
    X(96a, 1, INFINITY) X(96, 0, 1) X(128t, 0, INFINITY) X(128w, 0, 0) X(128, 0, 0) X(160, 0, INFINITY)       \
    X(160v2, 0, 0) X(256s, 0, INFINITY) X(256, 0, 0) X(256v2, 0, 0)
#define X(N_, LO_, HI_) extern const GeoOps kGeo##N_;
MSET_GEOS(X)
#undef X

static const GeoEntry kAllGeos[] = {
#define X(N_, LO_, HI_) {&kGeo##N_, LO_, HI_},
    MSET_GEOS(X)
#undef X
};

// the reference-semantics pass and the per-position steps walk one position
// at a time: one field spread over the CTAs of a cluster (seq_kernel.cuh).
// CTAs per field by measurement, microseconds per slab, forward and adjoint
// (32 slabs of one plane, one B200):
//   window   1 CTA   2       4       8       16
//   24       1.90    2.30
//   32       2.34    2.39    2.25
//   48       6.03    4.50    3.69    3.19
//   64               6.31    4.03    3.33
//   96                       8.02    5.19    4.55
//   128                              6.59    5.43
//   160                              12.3    7.71
//   256                              32.7    14.9
// Small fields lose more to the exchanges than they gain; 128 keeps the 8
// CTAs that mset_sequential_split documents.  The kernels before (one CTA per
// field up to 160, 8 CTAs with remote loads and cluster barriers at 128) took
// 8.4 us at 24 (24 slabs), 25.6 at 64 (24 slabs), 19.4 at 128 (64 slabs of two
// planes) and 87 at 160 (95 slabs); these take 1.7, 3.1, 6.3 and 7.0 there.
#define MSET_SEQ_FIELDS(X) X(24) X(32) X(48) X(64) X(96) X(128) X(160) X(256)
#define X(N_) extern const SeqOps kSeqField##N_;
MSET_SEQ_FIELDS(X)
#undef X
static const SeqOps *const kSeqFields[] = {
#define X(N_) &kSeqField##N_,
    MSET_SEQ_FIELDS(X)
#undef X
};

const SeqOps *seq_ops_for(int n) {
    for (const SeqOps *q : kSeqFields)
        if (q->n == n) return q;
    return nullptr;
}

static void fill_plan(const GeoOps *g, Plan *p) {
    p->n = g->n;
    p->r1 = g->r1;
    p->ry1 = g->ry1;
    p->nt = g->nt;
    p->cl = g->cl;
    p->staged = g->staged;
    p->max_clusters = 0;
    p->smem = g->smem;
    p->ctas_per_sm = 0;
    p->ops = g;
}

static bool same_layout(const GeoOps *a, const GeoOps *b) {
    return a->n == b->n && a->r1 == b->r1 && a->ry1 == b->ry1;
}

bool plan_for(int n, long positions, int sms, Plan *p) {
    const float per_sm = (float)positions / (float)(sms > 0 ? sms : 1);
    const GeoOps *first = nullptr;
    for (const GeoEntry &e : kAllGeos) {
        if (e.g->n != n) continue;
        if (!first) first = e.g;
        if (e.lo < per_sm && per_sm <= e.hi) {
            fill_plan(e.g, p);
            return true;
        }
    }
    if (first) fill_plan(first, p);  // no positions yet
    return first != nullptr;
}

bool plan_for_seq(int n, Plan *p) {
    for (const GeoEntry &e : kAllGeos)
        if (e.g->n == n && e.g->seq) {
            fill_plan(e.g, p);
            return true;
        }
    return false;
}

int plan_variants(int n) {
    const GeoOps *d = nullptr;
    int c = 0;
    for (const GeoEntry &e : kAllGeos) {
        if (e.g->n == n && !d) d = e.g;
        c += d && e.g->batch && same_layout(e.g, d);
    }
    return c;
}

bool plan_variant(const Plan &base, int variant, Plan *p) {
    if (variant == 0) {
        fill_plan(base.ops, p);
        return true;
    }
    for (const GeoEntry &e : kAllGeos)
        if (e.g != base.ops && e.g->batch && same_layout(e.g, base.ops) && --variant == 0) {
            fill_plan(e.g, p);
            return true;
        }
    return false;
}

int launch_positions(const Plan &pl, int method, int adjoint, int mode, const LaunchArgs &a, int grid,
                     cudaStream_t st) {
    return pl.ops->positions(method, adjoint, mode, a, grid, st);
}
int launch_prep_amp(const Plan &pl, const float *meas, float *amp, long npos, cudaStream_t st) {
    return pl.ops->prep_amp(meas, amp, npos, st);
}
int launch_prep_amp_bf16(const Plan &pl, const float *meas, unsigned short *ib, long npos, cudaStream_t st) {
    return pl.ops->prep_amp_bf16(meas, ib, npos, st);
}
int launch_prep_prop(const Plan &pl, const float *prop, float2 *pscr, cudaStream_t st) {
    return pl.ops->prep_prop(prop, pscr, st);
}
int launch_probe_to_q(const Plan &pl, const float2 *probe, float2 *q, const float2 *twn, cudaStream_t st) {
    return pl.ops->probe_q(true, probe, q, twn, st);
}
int launch_q_to_probe(const Plan &pl, const float2 *q, float2 *probe, const float2 *twn, cudaStream_t st) {
    return pl.ops->probe_q(false, q, probe, twn, st);
}

// batched update: V += step0 * G (slab-replicated), Q -= step1 * qacc,
// positions += step2 * posdir
__global__ void k_apply_volume(float *V, const double *g, int n2, int nz, int b, float step0) {
    const long total = (long)nz * n2;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int z = (int)(i / n2);
        const int l = (int)(i % n2);
        const int s = z / b;
        V[i] += step0 * (float)g[(long)s * n2 + l];
    }
}
__global__ void k_apply_probe(float2 *Q, const double *qacc, int n2, float step1) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
        float2 q = Q[i];
        q.x -= step1 * (float)qacc[2 * i];
        q.y -= step1 * (float)qacc[2 * i + 1];
        Q[i] = q;
    }
}
__global__ void k_apply_pos(float *sx, float *sy, const double *pd, int npos, float step2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npos; i += gridDim.x * blockDim.x) {
        sx[i] += step2 * (float)pd[2 * i];
        sy[i] += step2 * (float)pd[2 * i + 1];
    }
}

// transmission slabs of every tilt: T[s][y][x] = exp(i sdz sum_{z in slab s} V)
// (mset.cu:134-153), once per pass so the position kernel reads one complex
// value instead of recomputing it in the forward and the adjoint
__global__ void k_transmission(const TiltDev *tilts, int ntilts, int n2, int nz, int b, int ns, float sdz) {
    const long per = (long)ns * n2;
    const long total = per * ntilts;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int j = (int)(i / per);
        const long r = i % per;
        const int s = (int)(r / n2);
        const int l = (int)(r % n2);
        const TiltDev &t = tilts[j];
        const int z0 = s * b, z1 = min(z0 + b, nz);
        float acc = 0.f;
        for (int z = z0; z < z1; ++z) acc += __ldg(t.V + (size_t)z * n2 + l);
        float sn, cs;
        sincosf(sdz * acc, &sn, &cs);
        const_cast<float2 *>(t.T)[r] = make_float2(cs, sn);
    }
}

int launch_transmission(const TiltDev *tilts, int ntilts, int n, int nz, int b, int ns, float sdz, cudaStream_t st) {
    const long total = (long)ntilts * ns * n * n;
    const int grid = (int)std::min<long>((total + 255) / 256, 148L * 16);
    k_transmission<<<grid, 256, 0, st>>>(tilts, ntilts, n * n, nz, b, ns, sdz);
    return (int)cudaGetLastError();
}

int launch_apply_batch(int n, int nz, int b, int ns, int method, float step0, float step1, float step2,
                       const TiltDev *tilts, int ntilts, cudaStream_t st) {
    (void)ns;
    const int n2 = n * n;
    const int bb = method == kSSET ? nz : b;
    for (int j = 0; j < ntilts; ++j) {
        const TiltDev &t = tilts[j];
        k_apply_volume<<<592, 256, 0, st>>>(t.V, t.grad, n2, nz, bb, step0);
        k_apply_probe<<<64, 256, 0, st>>>(t.Q, t.qacc, n2, step1);
        k_apply_pos<<<8, 256, 0, st>>>(t.sx, t.sy, t.posdir, t.npos, step2);
    }
    return (int)cudaGetLastError();
}

int launch_apply_probe_pos(const TiltDev *tilts, int ntilts, int n, float step1, float step2, cudaStream_t st) {
    for (int j = 0; j < ntilts; ++j) {
        const TiltDev &t = tilts[j];
        k_apply_probe<<<64, 256, 0, st>>>(t.Q, t.qacc, n * n, step1);
        if (t.npos) k_apply_pos<<<8, 256, 0, st>>>(t.sx, t.sy, t.posdir, t.npos, step2);
    }
    return (int)cudaGetLastError();
}

}  // namespace mset
