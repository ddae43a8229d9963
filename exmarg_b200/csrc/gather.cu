// The table read of Eq. (C7) (exmarg/search/gather.py:32-107) on the B200.
//
// k_gather_planes (the pe_intrinsic path): one block per (lag r, template chunk, node k).  The block walks
// the 48 phase-plane pairs (p, p+1) of the node's lag slab T[k, r]; for each plane it stages, with one TMA
// copy, a window of 80-160 beta rows x 160 (16-bit tables: 176) Delta columns into shared memory (three
// slots: two planes in use, one in flight).  The descriptors of the lag are sorted by (plane pair,
// template) in groups of four taps of one template, and each warp owns a contiguous range of groups: it
// evaluates the bilinear x linear interpolation of a lane's four taps from shared memory, takes their maximum and
// adds their exponentials to the lane's running partial of that template, and merges partials across lanes with
// warp shuffles into a per-template accumulator that only it writes.
// A value is carried as (B, e) with B a stored float32 table value and e a small float32 correction up to its
// exponential, so a tap of size ~1e3 keeps ~1e-7 absolute precision; a partial is (m, S), S exp(m), with m the
// largest value.  Taps outside the window, and taps whose beta is clamped to the table, take an exact float64
// path that reads the table from global memory.
//
// What bounds it (2048 templates x 53 nodes x 87 lags x 2048 times, 1.65e10 taps): shared-memory reads (eight a
// tap, 79 % of the data pipe) and instruction issue (63 %) together; DRAM is at 0.36 of its rate.  92.7 -> 61.5 ms:
//  * four taps of one template per group: the bookkeeping of templates, the ranges and the running maximum are paid
//    once for four taps (5.4 -> 2.8 warp instructions per tap); padding the runs to whole groups adds 3.8 % taps;
//  * a row pitch of a multiple of the 32 banks, and taps ordered so that a step's lanes hit different banks
//    (k_tap_order): 3.4 -> 2.5 cycles per read;
//  * boundary points in blocks of their own, so the accumulators take 24 instead of 80 bytes a template and a block
//    takes up to 2048 templates: every plane pair costs a block a fixed ~1.7 us of waits (planes_tch);
//  * a warp's first descriptors and end templates of the next pair loaded before it waits for that pair's planes.
//  * descriptors loaded by whole chunks: no lane's loads are predicated or replaced by constants (65.3 -> 62.7).
// 20 warps at 96 registers; with two thirds of the templates a block 63.9 ms, 16 warps 65.3 (too few to cover the
// latencies), 24 warps 66.8 and 28 warps 78.8 (they spill).
//
// k_gather_simple (the gather_cpu / gather_gpu contract, any table per slot): one
// block per (row, lag), the reference's arithmetic in float64.
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

// the plane gather's dynamic shared memory; its parts are addressed by 32-bit byte offsets (fewer
// registers in the tap loop than 64-bit generic pointers)
extern __shared__ __align__(1024) unsigned char exm_gsm[];
__device__ __forceinline__ float *gsm_f(unsigned off) { return (float *)(exm_gsm + off); }

#define EXM_WAIT_CYCLES (2000000000LL)   // about one second at 1.9 GHz
#define EXM_TEST_WAIT_CYCLES (20000LL)   // the wait-expiry test's limit (no copy is ever in flight then)

struct PlaneArgs {
    const uint4 *desc;
    const int32_t *tside;
    const int *off;
    const float2 *H, *L;
    const float *Hlo, *Llo;      // residuals of ln|z| (filter precision 'fp64'), else null
    const void *T;               // node tables, element type of the kernel's TE
    const int *mlo, *mhi, *bnode, *win, *tau;
    const double *boff, *cb, *ckd;
    double *part;
    unsigned *err;
    unsigned long long *stats;   // [0] slow-path taps, [1] boundary taps (may be null)
    long long tstride, per_lag;
    int nn, ntau, nphif, nb, nd, ndp, nt, nmc, nwalk, m_base, nm_total, r0, tch, nch;
    int wb, ng, nparts;          // window rows, groups per lane and chunk, parts of the plane pairs
    float lw, wr;                // log weight of a random draw, and its exponential
    int nbn, nchb, tchb;         // boundary nodes, template chunks of each, templates of a chunk
    int bn_k[EXM_MAX_NODES], bn_lo[EXM_MAX_NODES], bn_hi[EXM_MAX_NODES];   // ... and their templates
    double rph, rdb, rdd, offd;
    long long wait_cycles;       // limit of the pipeline's barrier waits (EXM_WAIT_CYCLES)
    int stage;                   // 1: stage the planes; 0 (the wait-expiry test): no copy is issued, so the
                                 // first wait runs out and the kernel returns its timeout status
    int cki[EXM_MAX_NODES];
    float ckf[EXM_MAX_NODES];    // fraction of a node's beta shift
    float tsc[EXM_MAX_NODES];    // per node: value = tsc * stored element
};

// ------------------------------------------------------------------ TMA + mbarrier

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void tma_load_plane(const CUtensorMap *map, uint64_t *bar, void *dst, int x, int y, int z,
                                               int w, int v, unsigned bytes)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
        "[%7];" ::"r"(smem_u32(dst)),
        "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(v), "r"(smem_u32(bar))
        : "memory");
}


// bounded wait on a phase of an mbarrier; false (and the error word set) if it ran out after `limit` cycles
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, unsigned *err,
                                          long long limit = EXM_WAIT_CYCLES)
{
    const uint32_t a = smem_u32(bar);
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > limit) {
            atomicOr(err, EXM_DEVERR_TIMEOUT);
            return false;
        }
    }
}

// ------------------------------------------------------------------ log-sum-exp partials (m, S): S exp(m)

#define EXM_L2E 1.4426950408889634f
#define EXM_MNONE (-1e30f)   // the reference of an empty partial

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void ms_merge(float &m, float &S, float m2, float S2)
{
    // (m, S) += (m2, S2): the larger of the two becomes the reference, without a branch
    const float d = m2 - m;
    const float e = ex2_approx(-fabsf(d) * EXM_L2E);
    S = d > 0.f ? fmaf(S, e, S2) : fmaf(S2, e, S);
    m = fmaxf(m, m2);
}

// segmented reduction over lanes with equal id (ids non-decreasing along the lanes); afterwards the
// first lane of each run holds the run's total.  The references first (a running maximum), then the sums
// scaled to the run's reference: two shuffles and two operations a round instead of a merge.  Rounds end
// when no run reaches further.
__device__ __forceinline__ bool seg_reduce(int id, float &m, float &S)
{
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, id, 1);
    const bool head = lane == 0 || prev != id;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    // lanes from here to the end of the lane's run, and the run's first lane
    const unsigned above = heads & ~((2u << lane) - 1u);
    const int left = (above ? __ffs(above) - 1 : 32) - lane;
    const int first = 31 - __clz(heads & ((2u << lane) - 1u));
    const int longest = __reduce_max_sync(0xffffffffu, left);
    float M = m;
    for (int o = 1; o < longest; o <<= 1) {
        const float m2 = __shfl_down_sync(0xffffffffu, M, o);
        if (o < left) M = fmaxf(M, m2);
    }
    M = __shfl_sync(0xffffffffu, M, first);
    S *= ex2_approx((m - M) * EXM_L2E);
    m = M;
    for (int o = 1; o < longest; o <<= 1) {
        const float S2 = __shfl_down_sync(0xffffffffu, S, o);
        if (o < left) S += S2;
    }
    return head;
}

// two float32 operations in one instruction (planes p and p + 1 of a tap side by side)
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float a, float b)
{
    f2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b)
{
    f2_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b)
{
    f2_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c)
{
    f2_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// bilinear in (beta, Delta) on planes p and p+1 of the staged windows, linear in phase;
// value = B + E with B the stored value at (p, b0, d0).  16-bit elements are interpolated as
// stored (float32 arithmetic) and the result scaled by the node's power-of-two scale, which is
// exact.
template <typename TE>
__device__ __forceinline__ void interp_window(const TE *s0, const TE *s1, int o, float fbf, float fd, float w, float sc,
                                              float &B, float &E)
{
    constexpr int WD = TabElem<TE>::wd;
    const float t00 = TabElem<TE>::cvt(s0[o]), t01 = TabElem<TE>::cvt(s0[o + 1]);
    const float t10 = TabElem<TE>::cvt(s0[o + WD]), t11 = TabElem<TE>::cvt(s0[o + WD + 1]);
    const float u00 = TabElem<TE>::cvt(s1[o]), u01 = TabElem<TE>::cvt(s1[o + 1]);
    const float u10 = TabElem<TE>::cvt(s1[o + WD]), u11 = TabElem<TE>::cvt(s1[o + WD + 1]);
    const f2_t p00 = f2_pack(t00, u00);
    const f2_t a = f2_sub(f2_pack(t01, u01), p00), c = f2_sub(f2_pack(t10, u10), p00);
    const f2_t e = f2_sub(f2_sub(f2_pack(t11, u11), f2_pack(t10, u10)), a);
    const f2_t fd2 = f2_pack(fd, fd), fb2 = f2_pack(fbf, fbf);
    const f2_t eps = f2_fma(fd2, a, f2_mul(fb2, f2_fma(fd2, e, c)));
    float eps0, eps1;
    f2_unpack(eps, eps0, eps1);
    B = t00;
    E = fmaf(w, (u00 - t00) + (eps1 - eps0), eps0);
    if (!std::is_same<TE, float>::value) {
        B *= sc;
        E *= sc;
    }
}

// -1 where the sum f of a tap's and a node's beta fractions stays below 1, 0 where it carries into the row: by the bits,
// since with four more predicates the tap loop spills (2048 templates x 53 nodes 62.8 ms, this 61.5)
__device__ __forceinline__ int no_carry(float f) { return ((int)__float_as_uint(f) - 0x3F800000) >> 31; }

// One run of tap descriptors (sorted by template, in groups of EXM_GT taps of one template) on the
// two staged planes of pair p.  Each lane takes ng consecutive groups of a chunk; a template that
// lies inside one lane's groups is merged into its accumulator by that lane, one that spans lanes
// is combined by a segmented shuffle reduction once per chunk.
// byte offsets below are into exm_gsm
struct RunCtx {
    const uint4 *descr;
    unsigned s0, s1;            // the staged windows of planes p and p + 1 (element type TE)
    float sc;                   // the node's scale (16-bit tables)
    unsigned acc, accst;        // accumulator set of the run's templates (m at acc + 4 t; S at + accst)
    unsigned bsh, bcf;          // boundary blocks: per-template window offset (int; EXM_BSH_NONE for templates
                                // whose boundary point is not this node) and beta fraction
    int ng;                     // groups per lane and chunk
    int dm, n, k, r;            // block-local template = descriptor's + dm
    int sh;                     // window offset of a tap = its o0 + sh (+ a row when the beta fractions carry)
    unsigned lim;               // the taps the windows serve have offsets below lim
    float ckf;                  // the node's beta fraction
    float wr, lw;               // weight of a random draw (a factor up to EXM_LW_FACTOR) and its logarithm
    int beg, end;               // the warp's sorted positions (whole groups)
    int tF, tL;                 // the templates at the two ends of this warp's taps (may be shared with
    unsigned eF, eL;            // neighbouring warps): their partials go to this warp's edge slots (m, S)
    unsigned q, qn;             // this warp's queue of exact-path taps for the pair (int2 entries) and its count
    // the lane's next group of descriptors: whether it lies in [beg, end), its first position, its chunk's, its
    // index in the chunk, its address
    uint4 nx[EXM_GT];
    bool in;
    int jl, jc, gn;
    const uint4 *pn;
};

// load the lane's next group and step to the one after.  A lane whose group lies outside [beg, end) loads what is
// stored there (its chunk is a chunk of the run) and discards it by `in`; a chunk past the run's last is not read.
__device__ __forceinline__ void next_group(RunCtx &c)
{
    c.in = c.jl >= c.beg && c.jl < c.end;
    if (c.jc < c.end) {
#pragma unroll
        for (int u = 0; u < EXM_GT; ++u) c.nx[u] = __ldg(c.pn + 32 * u);
    }
    c.pn += 32 * EXM_GT;
    c.jl += EXM_GT;
    if (++c.gn == c.ng) {   // on to the next chunk
        c.gn = 0;
        c.jl += EXM_GT * 31 * c.ng;
        c.jc += EXM_GT * 32 * c.ng;
    }
}

__device__ __forceinline__ void acc_merge(const RunCtx &c, int tr, float m, float S)
{
    const bool f = tr == c.tF, l = tr == c.tL;
    const unsigned off = f ? c.eF : (l ? c.eL : c.acc + 4u * (unsigned)tr);
    const unsigned st = (f || l) ? 4u : c.accst;
    float *pm = gsm_f(off), *pS = gsm_f(off + st);
    float m1 = *pm, S1 = *pS;
    ms_merge(m1, S1, m, S);
    *pm = m1;
    *pS = S1;
}

#define EXM_SLOWQ 12   // exact-path taps a consumer warp queues per plane pair for the producer
#define EXM_BSH_NONE (1 << 29)   // bsh entry of a template whose boundary point is another node

// the exact float64 value of a tap outside the staged window (rare)
template <bool BND, typename TE>
__device__ __forceinline__ double slow_tap(const PlaneArgs &a, int il, int tm, int k, int r, int m_base, float sc)
{
    const int nt = a.nt;
    const int tau0 = ((a.tau[r] % nt) + nt) % nt;
    int i1 = tm + tau0;
    if (i1 >= nt) i1 -= nt;
    const int gi = il + m_base;
    const double offb = (BND ? a.cb[gi] : a.ckd[k]) + a.boff[gi];   // ckd: (ln s_k - beta0)/dbeta
    return exm_tap_fp64<TE>(a.L[(long long)il * nt + tm], a.H[(long long)il * nt + i1],
                            a.Llo ? a.Llo[(long long)il * nt + tm] : 0.f, a.Hlo ? a.Hlo[(long long)il * nt + i1] : 0.f,
                            offb, r,
                            (const TE *)a.T + (long long)k * a.tstride, sc, a.nphif, a.nb, a.nd, a.ndp, a.rph, a.rdb,
                            a.rdd, a.offd);
}

// a float64 value as a partial: its float32 rounding and the exponential of the rest
__device__ __forceinline__ void split_double(double v, float &m, float &S)
{
    m = (float)v;
    S = ex2_approx((float)(v - (double)m) * EXM_L2E);
}

// the taps of a group that the windows do not serve (storage index pj + 32 u): queued for the producer, which
// computes them 32 at a time instead of stalling the warp on one lane's float64 path; those a full queue
// cannot take are computed here and merged into the lane's running partial
template <bool BND, typename TE>
__device__ __forceinline__ void slow_group(const PlaneArgs &a, const RunCtx &c, int pj, int t, int sh, float ckf,
                                           float &m, float &S, unsigned &n_slow)
{
    const int lane = threadIdx.x & 31;
    int *qn = (int *)(exm_gsm + c.qn);
#pragma unroll 1
    for (int u = 0; u < EXM_GT; ++u, pj += 32) {
        bool sl = false;
        uint4 q = make_uint4(0u, 0u, 0u, EXM_DESC_PAD);
        if (t >= 0) {
            q = __ldg(c.descr + pj);
            const int o = ((int)q.w >> 13) + sh + (~no_carry(__uint_as_float(q.x) + ckf) & TabElem<TE>::wd);
            sl = (unsigned)o >= c.lim && (int)q.w >= EXM_DESC_REAL;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, sl);
        if (!bal) continue;
        const int n0 = *qn;
        const int pos = n0 + __popc(bal & ((1u << lane) - 1u));
        __syncwarp();
        if (sl) {
            ++n_slow;
            const int il = (int)(q.w & 0x1FFFu);
            if (pos < EXM_SLOWQ) {
                ((int2 *)(exm_gsm + c.q))[pos] = make_int2(pj, il | (int)((q.z >> 31) << 29));
            } else {
                double v = slow_tap<BND, TE>(a, il, a.tside[(c.r - a.r0) * a.per_lag + pj], c.k, c.r, a.m_base, c.sc);
                if (q.z >> 31) v += (double)c.lw;
                float m2, S2;
                split_double(v, m2, S2);
                ms_merge(m, S, m2, S2);
            }
        }
        if (lane == 0) *qn = min(EXM_SLOWQ, n0 + __popc(bal));
        __syncwarp();
    }
}

#define EXM_EDGE_F 6   // floats of a warp's edge slots: (m, S, template) of its first and of its last template

// the template of the descriptor at sorted position j (block-local)
__device__ __forceinline__ int desc_template(const RunCtx &c, int j)
{
    return (int)(__ldg(&c.descr[exm_desc_phys(j, c.ng)].w) & 0x1FFFu) + c.dm;
}

// this warp's share [c.beg, c.end) of the pair's run [beg, end): whole storage chunks per warp, as evenly as
// they divide (the first and last may be partial), and the loads of its first group and of its end
// templates, which are in flight while the warp waits for the pair's planes.
// The warps with work are a prefix: the edge fold merges equal templates of neighbouring lanes only, so
// an empty warp between two that share a template would let both update its accumulator at once.  When
// every warp has a chunk, the rem warps that take one more are a cyclic window that moves by rem with the
// pair, so that no warp takes the extra chunk at every pair: a warp runs at most one pair ahead, so with a
// fixed prefix the others would wait at every pair.
template <int NW>
__device__ __forceinline__ void open_share(RunCtx &c, int beg, int end, int pair)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ch = EXM_GT * 32 * c.ng;
    const int cb = beg / ch, nc = (end + ch - 1) / ch - cb;
    const int q = nc / NW, rem = nc % NW;
    const int s = q > 0 ? (pair * rem) % NW : 0, se = s + rem;
    const int before = max(0, min(warp, se) - s) + max(0, min(warp, se - NW));   // extra chunks of warps < warp
    const int c0 = cb + warp * q + before, c1 = c0 + q + ((warp - s + NW) % NW < rem ? 1 : 0);
    c.beg = max(beg, c0 * ch);
    c.end = min(end, c1 * ch);
    c.tF = c.tL = -1;
    if (c.beg < c.end) {
        const int jstart = c.beg & ~(ch - 1);
        c.gn = 0;
        c.jc = jstart;
        c.jl = jstart + EXM_GT * c.ng * lane;
        c.pn = c.descr + jstart + lane;
        next_group(c);
        c.tF = desc_template(c, c.beg);
        c.tL = desc_template(c, c.end - 1);
    }
}

// the warp's edge slots of the pair, empty: one template only takes the L slot
__device__ __forceinline__ void open_edge(RunCtx &c, unsigned eo)
{
    if (c.tF == c.tL) c.tF = -1;
    c.eF = eo;
    c.eL = eo + 12u;
    if ((threadIdx.x & 31) == 0) {
        float *e = gsm_f(eo);
        e[0] = EXM_MNONE;
        e[1] = 0.f;
        e[2] = __int_as_float(c.tF);
        e[3] = EXM_MNONE;
        e[4] = 0.f;
        e[5] = __int_as_float(c.tL);
    }
    __syncwarp();
}

// The draws' weight enters as a factor exp(lw) of their exponentials, outside the running maximum: one fused
// multiply-add a tap.  That holds while the factor and its products with the exponentials stay within float32:
// with |lw| <= EXM_LW_FACTOR what underflows (below 2^-126 of the largest unweighted value) is less than
// 2^-126 e^60 = 1.3e-12 of the sum.  LOGW, for any other weight, adds lw to the tap's value, so that the maximum
// includes it.
#define EXM_LW_FACTOR 60.0

template <bool BND, int PF, typename TE, bool LOGW>
__device__ __forceinline__ void process_run(const PlaneArgs &a, RunCtx &c, unsigned &n_slow)
{
    // the warp's positions walked in chunks of 128 ng; lane l takes the chunk's groups l ng + g, tap u of it
    // stored at (g EXM_GT + u) 32 + l
    constexpr int WD = TabElem<TE>::wd;
    const int lane = threadIdx.x & 31;
    const int ng = c.ng, ch = EXM_GT * 32 * ng, end = c.end;
    for (int j0 = c.beg & ~(ch - 1); j0 < end; j0 += ch) {
        int cT = -1, fT = -1;
        float cm = EXM_MNONE, cS = 0.f, fm = EXM_MNONE, fS = 0.f;
#pragma unroll 1
        for (int g = 0; g < ng; ++g) {
            // the group's template (-1: nothing to do) and the window shift of its taps
            int t = (int)(c.nx[0].w & 0x1FFFu) + c.dm;
            if (!c.in) t = -1;
            if (t >= c.n) {   // outside the block's templates: report and skip
                atomicOr(a.err, EXM_DEVERR_BOUNDS);
                t = -1;
            }
            int sh = c.sh;
            float ckf = c.ckf;
            if (BND) {
                sh = EXM_BSH_NONE;
                ckf = 0.f;
                if (t >= 0) {
                    sh = ((const int *)gsm_f(c.bsh))[t];
                    ckf = gsm_f(c.bcf)[t];
                }
                if (sh == EXM_BSH_NONE) t = -1;
            }
            // window offset, beta and Delta fractions, plane weight and draw weight of the four taps
            int o[EXM_GT];
            float fb[EXM_GT], fd[EXM_GT], w[EXM_GT], wt[EXM_GT];
            bool fast[EXM_GT];
            bool sl = false;
#pragma unroll
            for (int u = 0; u < EXM_GT; ++u) {
                const float f = __uint_as_float(c.nx[u].x) + ckf;   // the fractions carry into the row
                const int nc = no_carry(f);
                const int ou = ((int)c.nx[u].w >> 13) + sh + (~nc & WD);
                fast[u] = (unsigned)ou < c.lim;
                sl = sl || (!fast[u] && (int)c.nx[u].w >= EXM_DESC_REAL);
                o[u] = fast[u] ? ou : lane;
                fb[u] = f - __uint_as_float(~nc & 0x3F800000);
                fd[u] = __uint_as_float(c.nx[u].y);
                w[u] = __uint_as_float(c.nx[u].z);
                // the bit: a draw's plane weight may be zero
                wt[u] = (int)c.nx[u].z < 0 ? (LOGW ? c.lw : c.wr) : (LOGW ? 0.f : 1.f);
            }
            next_group(c);
            // close the running template where another one begins
            const bool nw = t != cT;
            const bool close = nw && cT >= 0;
            const bool toF = close && fT < 0;      // ... as the lane's first closed partial
            if (close && !toF) acc_merge(c, cT, cm, cS);
            fT = toF ? cT : fT;
            fm = toF ? cm : fm;
            fS = toF ? cS : fS;
            cT = t;
            cm = nw ? EXM_MNONE : cm;
            cS = nw ? 0.f : cS;
            float B[EXM_GT], E[EXM_GT];
            float m = cm;
#pragma unroll
            for (int u = 0; u < EXM_GT; ++u) {
                interp_window<TE>((const TE *)(exm_gsm + c.s0), (const TE *)(exm_gsm + c.s1), o[u], fb[u], fd[u],
                                  fabsf(w[u]), c.sc, B[u], E[u]);
                if (LOGW) E[u] += wt[u];
                const float v = B[u] + E[u];
                if (fast[u]) m = fmaxf(m, v);
                if (PF == 1 && u == 1) __syncwarp();   // two taps' window reads in flight, for shapes with few registers
            }
            float S = cS * ex2_approx((cm - m) * EXM_L2E);
#pragma unroll
            for (int u = 0; u < EXM_GT; ++u) {
                const float x = ex2_approx(((B[u] - m) + E[u]) * EXM_L2E);
                if (fast[u]) S = LOGW ? S + x : fmaf(x, wt[u], S);
            }
            cm = m;
            cS = S;
            if (__any_sync(0xffffffffu, sl && t >= 0))
                slow_group<BND, TE>(a, c, j0 + 32 * EXM_GT * g + lane, t, sh, ckf, cm, cS, n_slow);
        }
        // the first closed template of lane l + 1 continues lane l's last one, or is lane l + 1's alone
        const int nT = __shfl_down_sync(0xffffffffu, fT, 1);
        const float nm = __shfl_down_sync(0xffffffffu, fm, 1);
        const float nS = __shfl_down_sync(0xffffffffu, fS, 1);
        const int pT = __shfl_up_sync(0xffffffffu, cT, 1);
        if (lane < 31 && nT >= 0 && nT == cT) ms_merge(cm, cS, nm, nS);
        if (fT >= 0 && !(lane > 0 && pT == fT)) acc_merge(c, fT, fm, fS);
        __syncwarp();
        // last templates: runs across consecutive lanes
        const bool head = seg_reduce(cT >= 0 ? cT : -2 - lane, cm, cS);
        if (head && cT >= 0) acc_merge(c, cT, cm, cS);
        __syncwarp();
    }
}

// fold the warps' edge partials into the accumulators: one warp, lane w holding warp w's first (F)
// and last (L) partials; templates ascend along the warps, so this is the lane-level merge again
__device__ __forceinline__ void fold_edges(float *edge, int nw, float *am, float *aS, int n)
{
    const int lane = threadIdx.x & 31;
    float fm = EXM_MNONE, fS = 0.f, cm = EXM_MNONE, cS = 0.f;
    int fT = -1, cT = -1;
    if (lane < nw) {
        const float *e = edge + EXM_EDGE_F * lane;
        fm = e[0];
        fS = e[1];
        fT = __float_as_int(e[2]);
        cm = e[3];
        cS = e[4];
        cT = __float_as_int(e[5]);
        if (!(fT >= 0 && fT < n && fS > 0.f)) fT = -1;
        if (!(cT >= 0 && cT < n)) cT = -1;
    }
    const int nT = __shfl_down_sync(0xffffffffu, fT, 1);
    const float nm = __shfl_down_sync(0xffffffffu, fm, 1);
    const float nS = __shfl_down_sync(0xffffffffu, fS, 1);
    const int pT = __shfl_up_sync(0xffffffffu, cT, 1);
    if (lane < 31 && nT >= 0 && nT == cT) ms_merge(cm, cS, nm, nS);
    if (fT >= 0 && !(lane > 0 && pT == fT)) {
        float m = am[fT], S = aS[fT];
        ms_merge(m, S, fm, fS);
        am[fT] = m;
        aS[fT] = S;
    }
    __syncwarp();
    const bool head = seg_reduce(cT >= 0 ? cT : -2 - lane, cm, cS);
    if (head && cT >= 0 && cS > 0.f) {
        float m = am[cT], S = aS[cT];
        ms_merge(m, S, cm, cS);
        am[cT] = m;
        aS[cT] = S;
    }
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// shared memory of the plane gather after the three window slots, in bytes from the slots' end: barriers;
// the accumulators, three sets of 2 x tch floats (m, S): pairs of parity 0 / 1, edges and exact-path taps
// (producer) -- a boundary block has fewer templates, with bcf and bsh after its sets; the edge slots [pair
// parity][EXM_EDGE_F floats per consumer warp]; exact-path queues [pair mod 3][consumer warp]: counts, then
// EXM_SLOWQ int2 entries (storage index of the tap; template | random flag << 29)
#define EXM_ACC_F 6    // floats per template: three sets of (m, S)
#define EXM_ACCB_F 8   // ... of a boundary block: and bcf, bsh
#define EXM_MAX_NC 27  // most consumer warps of a launch shape
#define EXM_EDGE_B (4 * 2 * EXM_EDGE_F * EXM_MAX_NC)
#define EXM_QCNT_B (4 * 3 * 32)
#define EXM_QENT_B (8 * 3 * EXM_MAX_NC * EXM_SLOWQ)
#define EXM_GATHER_FIXED_B (64 + EXM_EDGE_B + EXM_QCNT_B + EXM_QENT_B)

// Warp NW - 1 is the producer: it stages the planes with TMA and, once every consumer warp has
// arrived on the pair's "done" barrier, folds that pair's edge partials and refills the slot of
// the plane no longer needed.  The NW - 1 consumer warps walk the pairs without a block barrier:
// a fast warp runs at most one pair ahead of the slowest (pair p + 2 needs plane p + 3, staged
// only after pair p is done everywhere).  So at most two consecutive pairs are in flight, and the
// consumers' accumulators alternate with the pair's parity (two warps in different pairs never
// share a word), while the producer folds edges into a third set of its own.
template <int NW, int PF, typename TE, bool LOGW>
__global__ void __launch_bounds__(NW * 32, 1) k_gather_planes(const __grid_constant__ CUtensorMap tmap,
                                                                const __grid_constant__ PlaneArgs a)
{
    constexpr int NC = NW - 1;   // consumer warps
    static_assert(NC <= EXM_MAX_NC, "shared memory is laid out for EXM_MAX_NC consumers");
    const int SLOT = a.wb * TabElem<TE>::wd;
    const unsigned SLOT_B = (unsigned)SLOT * (unsigned)sizeof(TE);
    unsigned char *smem = exm_gsm;
    TE *win = (TE *)smem;
    uint64_t *full = (uint64_t *)(smem + 3 * SLOT_B);   // [3] plane staged in slot s
    uint64_t *done = full + 3;                          // [2] every consumer is done with a pair (parity)
    // block -> (lag, template chunk, node, part of the plane pairs): the blocks of one (lag, chunk), which
    // read the same descriptors, run together; after a lag's regular blocks those of its boundary points
    int blk = blockIdx.x;
    const int part_i = blk % a.nparts;
    blk /= a.nparts;
    const int per_r = a.nn * a.nch + a.nbn * a.nchb;
    const int rl = blk / per_r, r = a.r0 + rl;
    blk %= per_r;
    const bool bnd = blk >= a.nn * a.nch;
    if (bnd) blk -= a.nn * a.nch;
    const int bi = bnd ? blk % a.nbn : 0;
    const int k = bnd ? a.bn_k[bi] : blk % a.nn;
    const int tch = bnd ? a.tchb : a.tch;
    const int c_idx = bnd ? blk / a.nbn : blk / a.nn;
    const int lo0 = bnd ? a.bn_lo[bi] : max(a.mlo[k], a.m_base);
    const int hi0 = bnd ? a.bn_hi[bi] : min(a.mhi[k], a.m_base + a.nmc);
    const int lo = lo0 + c_idx * tch;
    const int hi = min(hi0, lo + tch);
    if (lo >= hi) return;
    const int n = hi - lo;
    const int p_beg = part_i * EXM_NPAIR / a.nparts, np = (part_i + 1) * EXM_NPAIR / a.nparts - p_beg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned acc_o = 3 * SLOT_B + 64;
    float *acc = gsm_f(acc_o);
    const unsigned bcf_o = acc_o + 4u * EXM_ACC_F * tch, bsh_o = bcf_o + 4u * tch;   // boundary blocks
    const unsigned edge_o = acc_o + 4u * EXM_ACC_F * a.tch;
    const unsigned qcnt_o = edge_o + EXM_EDGE_B, qent_o = qcnt_o + EXM_QCNT_B;
    int *qcnt = (int *)(smem + qcnt_o);
    const int2 *qent = (const int2 *)(smem + qent_o);
    auto edge_off = [&](int par) { return edge_o + 4u * (unsigned)(par * EXM_EDGE_F * NC); };
    __shared__ unsigned bad_sh;

    if (tid == 0) bad_sh = 0;
    // the node's window: column C0, first row R0 = Rh + cki clamped to the table; a tap's window row
    // is its beta-hat row from Rh (in the descriptor), plus the carry of the beta fractions, plus sh
    const int C0 = a.win[0], R0 = a.win[1 + k], Rh = a.win[1 + EXM_MAX_NODES];
    const int sh = Rh + a.cki[k] - R0;
    for (int j = tid; j < n; j += NW * 32) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            acc[(2 * q) * tch + j] = EXM_MNONE;
            acc[(2 * q + 1) * tch + j] = 0.f;
        }
        if (bnd) {
            int bs = EXM_BSH_NONE;
            float bf = 0.f;
            if (a.bnode[lo + j] == k) {
                const double cbv = a.cb[lo + j];
                const double f = floor(cbv);
                const int rows = (int)f - a.cki[k] + sh;
                bs = EXM_BSH_FAR;   // no tap reaches the window: every one takes the exact path
                if (abs(rows) <= EXM_MAX_SHIFT) {
                    bs = rows * TabElem<TE>::wd;
                    bf = (float)(cbv - f);
                }
            }
            ((int *)gsm_f(bsh_o))[j] = bs;
            gsm_f(bcf_o)[j] = bf;
        }
    }
    if (tid == 0) {
        for (int s = 0; s < 3; ++s) mbar_init(&full[s], 1);
        for (int s = 0; s < 2; ++s) mbar_init(&done[s], NC * 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    unsigned n_slow = 0, n_bnd = 0;

    if (warp == NC) {
        // ---------------------------------------------------------------- producer
        const int32_t *tsr_all = a.tside + (long long)rl * a.per_lag;
        const int nplanes = np + 1;
        int issued = 0;
        if (a.stage) {
            if (lane == 0)
                for (int q = 0; q < 3 && q < nplanes; ++q)
                    tma_load_plane(&tmap, &full[q], win + q * SLOT, C0, R0, p_beg + q, r, k, SLOT_B);
            issued = min(3, nplanes);
        }
        bool ok = true;
        for (int p = 0; p < np; ++p) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&done[p & 1], (p >> 1) & 1, a.err, a.wait_cycles));
            if (!ok) break;
            fold_edges(gsm_f(edge_off(p & 1)), NC, acc + 4 * tch, acc + 5 * tch, n);
            __syncwarp();
            // plane p is no longer needed anywhere: its slot takes plane p + 3
            if (a.stage && p + 3 < nplanes) {
                if (lane == 0)
                    tma_load_plane(&tmap, &full[p % 3], win + (p % 3) * SLOT, C0, R0, p_beg + p + 3, r, k, SLOT_B);
                ++issued;
            }
            // the exact-path taps the consumers queued for pair p: 32 lanes compute them, lane 0 merges them
            // in warp and queue order into the producer's set (the consumers reuse these queues at pair
            // p + 3, after plane p + 4, which is staged only after this)
            {
                const int par = p % 3;
                const int cw = lane < NC ? qcnt[par * 32 + lane] : 0;
                int incl = cw;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                const int excl = incl - cw;
                for (int b0 = 0; b0 < total; b0 += 32) {
                    const int i = b0 + lane;
                    double v = 0.0;
                    int tr = 0;
                    int wi = 0;   // the warp whose entries [excl, incl) hold i (shuffles kept converged)
                    for (int l = 1; l < NC; ++l) {
                        const int el = __shfl_sync(0xffffffffu, excl, l);
                        wi += (i < total && el <= i) ? 1 : 0;
                    }
                    const int wexcl = __shfl_sync(0xffffffffu, excl, wi);
                    if (i < total) {
                        const int2 e = qent[(par * NC + wi) * EXM_SLOWQ + (i - wexcl)];
                        const int il = e.y & 0x1FFF;
                        const int tm = tsr_all[e.x];
                        v = bnd ? slow_tap<true, TE>(a, il, tm, k, r, a.m_base, a.tsc[k])
                                : slow_tap<false, TE>(a, il, tm, k, r, a.m_base, a.tsc[k]);
                        v += ((e.y >> 29) & 1) ? (double)a.lw : 0.0;
                        tr = il + a.m_base - lo;
                    }
                    const int nb2 = min(32, total - b0);
                    for (int qq = 0; qq < nb2; ++qq) {
                        const double vq = __shfl_sync(0xffffffffu, v, qq);
                        const int tq = __shfl_sync(0xffffffffu, tr, qq);
                        if (lane == 0 && tq >= 0 && tq < n) {
                            float m2, S2;
                            split_double(vq, m2, S2);
                            float *F = acc + 4 * tch;
                            float m = F[tq], S = F[tch + tq];
                            ms_merge(m, S, m2, S2);
                            F[tq] = m;
                            F[tch + tq] = S;
                        }
                    }
                }
                __syncwarp();
            }
        }
        if (!ok) {
            if (lane == 0) {
                atomicOr(&bad_sh, 1u);
                // drain: the newest copy of each slot completes after the older ones of that slot (bounded by
                // the full limit whatever the pipeline's: the block must not exit with a copy in flight)
                for (int q = max(0, issued - 3); q < issued; ++q) mbar_wait(&full[q % 3], (q / 3) & 1, a.err);
            }
        }
    } else {
        // ---------------------------------------------------------------- consumers
        const int *offr = a.off + (long long)rl * EXM_NPAIR * (a.nmc + 1);
        RunCtx rc;
        rc.descr = a.desc + (long long)rl * a.per_lag;
        rc.bsh = bsh_o;
        rc.bcf = bcf_o;
        rc.accst = 4u * tch;
        rc.ng = a.ng;
        rc.dm = a.m_base - lo;
        rc.n = n;
        // rows 0 .. up of the window are served: up + 1 must be in the window, and the table's last row
        // pair, where the reference clamps beta just below the top, is left to the exact path
        const int up = min(a.wb - 2, a.nb - 3 - R0);
        const bool near = bnd || abs(sh) <= EXM_MAX_SHIFT;
        rc.sh = near ? sh * TabElem<TE>::wd : EXM_BSH_FAR;
        rc.lim = (up >= 0 && near) ? (unsigned)((up + 1) * TabElem<TE>::wd) : 0u;
        rc.ckf = a.ckf[k];
        rc.sc = a.tsc[k];
        rc.k = k;
        rc.r = r;
        rc.lw = a.lw;
        rc.wr = a.wr;
        // the run offsets are loaded two pairs ahead, a warp's first descriptors and end templates one
        const int *offp = offr + (long long)p_beg * (a.nmc + 1) + (lo - a.m_base);
        open_share<NC>(rc, offp[0], offp[n], 0);
        int nb0 = 0, nb1 = 0;
        if (np > 1) {
            offp += a.nmc + 1;
            nb0 = offp[0];
            nb1 = offp[n];
        }
        bool ok = true;
        for (int p = 0; p < np; ++p) {
            // warp-uniform: the lanes go on to shuffles together
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[p % 3], (p / 3) & 1, a.err, a.wait_cycles));
            ok = ok && __all_sync(0xffffffffu,
                                  mbar_wait(&full[(p + 1) % 3], ((p + 1) / 3) & 1, a.err, a.wait_cycles));
            if (lane == 0) qcnt[(p % 3) * 32 + warp] = 0;
            __syncwarp();
            rc.qn = qcnt_o + 4u * ((p % 3) * 32 + warp);
            rc.q = qent_o + 8u * (((p % 3) * NC + warp) * EXM_SLOWQ);
            if (!ok) {   // no work: empty edge slots for the producer
                rc.tF = rc.tL = -1;
                rc.beg = rc.end = 0;
            }
            open_edge(rc, edge_off(p & 1) + 4u * EXM_EDGE_F * warp);
            if (rc.beg < rc.end) {
                rc.s0 = (p % 3) * SLOT_B;
                rc.s1 = ((p + 1) % 3) * SLOT_B;
                rc.acc = acc_o + 4u * (2u * (p & 1) * tch);
                if (bnd)
                    process_run<true, PF, TE, LOGW>(a, rc, n_slow);
                else
                    process_run<false, PF, TE, LOGW>(a, rc, n_slow);
            }
            __syncwarp();
            mbar_arrive(&done[p & 1]);
            if (p + 1 < np) {
                const int b0 = nb0, b1 = nb1;
                if (p + 2 < np) {
                    offp += a.nmc + 1;
                    nb0 = offp[0];
                    nb1 = offp[n];
                }
                open_share<NC>(rc, b0, b1, p + 1);
            }
        }
        if (!ok && lane == 0) atomicOr(&bad_sh, 1u);
    }
    __syncthreads();
    const bool ok = bad_sh == 0;
    const long long prow = a.ntau * a.nparts;   // partial sums per node and template
    for (int j = tid; j < n; j += NW * 32) {
        // the three sets of a template: both pair parities, and the producer's
        float m = acc[j], S = acc[tch + j];
        ms_merge(m, S, acc[2 * tch + j], acc[3 * tch + j]);
        ms_merge(m, S, acc[4 * tch + j], acc[5 * tch + j]);
        const double v = (ok && S > 0.f) ? (double)m + log((double)S) : -INFINITY;
        if (!bnd) {
            a.part[(k * prow + r * a.nparts + part_i) * a.nm_total + lo + j] = v;
        } else if (a.bnode[lo + j] == k) {
            a.part[(a.nn * prow + r * a.nparts + part_i) * a.nm_total + lo + j] = v;
            if (part_i == 0) n_bnd += (unsigned)a.nwalk;
        }
    }
    if (a.stats) {
        const unsigned sl_ = __reduce_add_sync(0xffffffffu, n_slow), bd_ = __reduce_add_sync(0xffffffffu, n_bnd);
        if (lane == 0 && (sl_ | bd_)) {
            atomicAdd(&a.stats[0], (unsigned long long)sl_);
            atomicAdd(&a.stats[1], (unsigned long long)bd_);
        }
    }
}

// ------------------------------------------------------------------ launch

// launch shapes the autotuner chooses from: warps per block including the producer, and the pairs of taps
// whose window reads a lane has in flight; the first is the default of an untuned context
struct GatherCfg {
    int nw, pf;
};
static const GatherCfg kGatherCfgs[] = {{20, 2}, {28, 1}, {16, 2}, {24, 2}, {24, 1}};
static const int kNumGatherCfgs = (int)(sizeof(kGatherCfgs) / sizeof(kGatherCfgs[0]));

template <int NW, int PF, typename TE, bool LOGW = false>
static void launch_planes(exm_ctx *ctx, const PlaneArgs &a, dim3 grid, size_t smem)
{
    exm_allow_smem(ctx, (const void *)k_gather_planes<NW, PF, TE, LOGW>, smem);
    k_gather_planes<NW, PF, TE, LOGW><<<grid, NW * 32, smem, ctx->stream>>>(ctx->tmap, a);
}

template <typename TE>
static void launch_cfg_t(exm_ctx *ctx, int cfg, const PlaneArgs &a, dim3 grid, size_t smem)
{
    if (!(std::fabs((double)a.lw) <= EXM_LW_FACTOR)) {   // weights given by the caller: one shape is enough
        launch_planes<20, 2, TE, true>(ctx, a, grid, smem);
        return;
    }
    switch (cfg) {
    case 0: launch_planes<20, 2, TE>(ctx, a, grid, smem); break;
    case 1: launch_planes<28, 1, TE>(ctx, a, grid, smem); break;
    case 2: launch_planes<16, 2, TE>(ctx, a, grid, smem); break;
    case 3: launch_planes<24, 2, TE>(ctx, a, grid, smem); break;
    default: launch_planes<24, 1, TE>(ctx, a, grid, smem); break;
    }
}

static void launch_cfg(exm_ctx *ctx, int cfg, const PlaneArgs &a, dim3 grid, size_t smem)
{
    if (ctx->dtype == EXM_DTYPE_F16)
        launch_cfg_t<__half>(ctx, cfg, a, grid, smem);
    else if (ctx->dtype == EXM_DTYPE_BF16)
        launch_cfg_t<__nv_bfloat16>(ctx, cfg, a, grid, smem);
    else
        launch_cfg_t<float>(ctx, cfg, a, grid, smem);
}

int exm_gather_num_cfgs() { return kNumGatherCfgs; }

static size_t planes_smem(int tch, int wb, int dtype)
{
    return 3 * (size_t)wb * exm_dtype_wd(dtype) * exm_dtype_bytes(dtype) + EXM_GATHER_FIXED_B + (size_t)tch * EXM_ACC_F * 4;
}

// templates a gather block may hold next to windows of wb rows (2 KB are left for the static shared memory)
static int planes_tch_max(const exm_ctx *ctx, int wb)
{
    const size_t fixed = planes_smem(0, wb, ctx->dtype) + 2048;
    const size_t room = ctx->smem_optin > fixed ? ctx->smem_optin - fixed : 0;
    return (int)std::min<size_t>(EXM_TCH, room / (EXM_ACC_F * 4) / 16 * 16);
}

// templates per gather block: pct / 150 of the most that still gives every SM eight blocks (a block's start,
// the waits at each plane pair and the staging of its windows are paid once for all its templates), between
// 256 and EXM_TCH at 150, then the same for every chunk of a node.  2048 templates x 53 nodes at 352 / 512 / 704 /
// 1024 / 2048: 75.5 / 70.9 / 68.0 / 65.4 ms, and on a later kernel 65.2 / 63.1 / 61.1 at the last three.
static int planes_tch_of(int sm_count, long long pairs, int maxn, int rc, int pct)
{
    long long tch = pairs * rc / std::max(1, 8 * sm_count);
    tch = std::min<long long>(std::max<long long>(tch, 256), EXM_TCH);
    tch = std::min<long long>(tch * pct / 150, EXM_TCH);
    tch = std::max<long long>(1, std::min<long long>(tch, maxn));
    const long long nch = std::max<long long>(1, (maxn + tch - 1) / tch);
    return (int)(((maxn + nch - 1) / nch + 15) / 16 * 16);
}

// (template, node) pairs of a pass over nmc templates from m_base, and the most of one node
static long long planes_pairs(const exm_ctx *ctx, int m_base, int nmc, int *maxn_out)
{
    long long pairs = 0;
    *maxn_out = 0;
    for (int k = 0; k < ctx->nn; ++k) {
        const int n = std::max(0, std::min(ctx->mhi[k], m_base + nmc) - std::max(ctx->mlo[k], m_base));
        pairs += n;
        *maxn_out = std::max(*maxn_out, n);
    }
    return pairs;
}

static int planes_tch(const exm_ctx *ctx, const ChunkInfo &ci, int rc, int pct, int *maxn_out)
{
    const long long pairs = planes_pairs(ctx, ci.m_base, ci.nmc, maxn_out);
    return planes_tch_of(ctx->sm_count, pairs, *maxn_out, rc, pct);
}

// The windows' height and the descriptors' chunk, which the tap build and the gather share.  Rows: the most that
// fit beside the accumulators of the templates a default block takes (at least EXM_WB_MIN, at most
// EXM_WB_MAX): every row more leaves fewer taps to the exact path.  Groups per lane: 4 (chunks of 512 taps),
// fewer when a plane pair of a block has too few taps to give every warp a chunk (gather ms at 4 / 2 / 1 groups:
// 10900 taps 10.6 / 11.2 / 12.9, 8000 7.8 / 7.8 / 8.8, 5100 7.3 / 6.7 / 7.4, 2700 0.45 / 0.34 / 0.35).
void exm_gather_plan(const exm_ctx *ctx, const ChunkInfo &ci, int rc, int *wb_out, int *ng_out)
{
    int maxn = 0;
    const int tch = std::max(16, planes_tch(ctx, ci, rc, 150, &maxn));
    const size_t fixed = EXM_GATHER_FIXED_B + 2048 + (size_t)tch * EXM_ACC_F * 4;
    const size_t row = 3 * (size_t)exm_dtype_wd(ctx->dtype) * exm_dtype_bytes(ctx->dtype);
    int wb = (int)((ctx->smem_optin - fixed) / row) / 8 * 8;
    wb = std::min(wb, std::max(EXM_WB_MIN, (ctx->nb + 7) / 8 * 8));
    *wb_out = std::max(EXM_WB_MIN, std::min(wb, EXM_WB_MAX));
    const double taps = (double)std::min(tch, std::max(maxn, 1)) * ci.nwalk / EXM_NPAIR;   // of a pair of a block
    *ng_out = taps >= 8000 ? 4 : (taps >= 2500 ? 2 : 1);
}

// Parts of the 48 plane pairs a (node, lag, template chunk) is split into, each a block of its own: one, or
// more when the launch has too few blocks to keep the SMs busy to the end.  Gather ms at 1 / 2 / 4 / 8 parts:
// 3.5 waves of blocks (24 templates, every time) 1.22 / 1.05 / 0.97 / 1.00, (150 x 6 nodes) 1.66 / 1.49 / 1.45 / 1.50; 9.5
// waves (333 x 21, two segments) 6.81 / 6.58 / 6.67 / 6.96; 15 waves (58 x 53) 1.92 / 1.93 / 2.04 / 2.28.
int exm_gather_parts_of(int sm_count, long long pairs, int maxn, int nn, int rc)
{
    const int tch = std::max(16, planes_tch_of(sm_count, pairs, maxn, rc, 150));
    const long long blocks = (long long)rc * nn * ((maxn + tch - 1) / std::max(tch, 1));
    const long long waves = blocks / std::max(1, sm_count);
    return waves >= 12 ? 1 : (waves >= 4 ? 2 : 4);
}

int exm_gather_parts(const exm_ctx *ctx, int nmc, int m_base, int rc)
{
    int maxn = 0;
    const long long pairs = planes_pairs(ctx, m_base, nmc, &maxn);
    return exm_gather_parts_of(ctx->sm_count, pairs, maxn, ctx->nn, rc);
}

void exm_run_gather_planes(exm_ctx *ctx, exm_slot &sl, const ChunkInfo &ci, int r0, int rc)
{
    exm_make_tmap(ctx, sl.wb);
    PlaneArgs a;
    memset(&a, 0, sizeof(a));
    a.desc = (const uint4 *)sl.desc.p;
    a.tside = (const int32_t *)sl.tside.p;
    a.off = (const int *)sl.cnt.p;
    a.H = (const float2 *)sl.traj.p;
    a.L = a.H + (size_t)ci.nmc * ctx->nt;
    a.Hlo = ctx->traj_fp64 ? (const float *)sl.trajlo.p : nullptr;
    a.Llo = a.Hlo ? a.Hlo + (size_t)ci.nmc * ctx->nt : nullptr;
    a.T = ctx->T.p;
    a.mlo = (const int *)ctx->d_mlo.p;
    a.mhi = (const int *)ctx->d_mhi.p;
    a.bnode = (const int *)ctx->d_bnode.p;
    a.win = (const int *)sl.win.p;
    a.tau = (const int *)ctx->d_tau.p;
    a.boff = (const double *)ctx->d_bhat_off.p;
    a.cb = (const double *)ctx->d_cb.p;
    a.ckd = (const double *)ctx->d_ckd.p;
    a.part = (double *)sl.part.p;
    a.err = (unsigned *)sl.dev_err.p;
    a.stats = (unsigned long long *)ctx->d_stats.p;
    a.tstride = (long long)ctx->tstride;
    a.per_lag = exm_desc_pitch(ci.nmc, ci.nwalk);   // storage stride of a lag's descriptors
    a.nn = ctx->nn;
    a.ntau = ctx->ntau;
    a.nphif = ctx->nphif;
    a.nb = ctx->nb;
    a.nd = ctx->nd;
    a.ndp = ctx->ndp;
    a.nt = ctx->nt;
    a.nmc = ci.nmc;
    a.nwalk = ci.nwalk;
    a.m_base = ci.m_base;
    a.nm_total = ctx->nm;
    a.r0 = r0;
    a.wb = sl.wb;
    a.ng = sl.ng;
    a.nparts = sl.nparts;
    a.lw = ci.lw;
    a.wr = (float)std::exp((double)ci.lw);
    a.rph = EXM_NPHI / 6.283185307179586;
    a.rdb = 2.0 / ctx->dbeta;
    a.rdd = 1.0 / ctx->ddelta;
    a.offd = -ctx->delta0 / ctx->ddelta;
    a.stage = ctx->test_wait_expiry ? 0 : 1;
    a.wait_cycles = ctx->test_wait_expiry ? EXM_TEST_WAIT_CYCLES : EXM_WAIT_CYCLES;
    for (int k = 0; k < ctx->nn; ++k) {
        const double f = std::floor(ctx->ck[k]);
        a.cki[k] = (int)f;
        a.ckf[k] = (float)(ctx->ck[k] - f);
        a.tsc[k] = ctx->tscale[k];
    }
    int maxn = 0;
    int tch = planes_tch(ctx, ci, rc, ctx->gather_chunk_pct, &maxn);
    if (maxn <= 0) return;
    tch = std::min(tch, planes_tch_max(ctx, sl.wb));
    a.nch = (maxn + tch - 1) / tch;
    tch = std::min(tch, ((maxn + a.nch - 1) / a.nch + 15) / 16 * 16);   // equal chunks
    a.tch = tch;
    // boundary points: the templates of each node that has some, in chunks whose extra arrays fit the same space
    int maxb = 0;
    for (int k = 0; k < ctx->nn; ++k) {
        int lo = -1, hi = -1;
        for (int i = ci.m_base; i < ci.m_base + ci.nmc; ++i)
            if (ctx->bnode[i] == k) {
                if (lo < 0) lo = i;
                hi = i + 1;
            }
        if (lo < 0) continue;
        a.bn_k[a.nbn] = k;
        a.bn_lo[a.nbn] = lo;
        a.bn_hi[a.nbn++] = hi;
        maxb = std::max(maxb, hi - lo);
    }
    a.tchb = std::max(1, tch * EXM_ACC_F / EXM_ACCB_F);
    a.nchb = (maxb + a.tchb - 1) / a.tchb;
    const size_t smem = planes_smem(tch, sl.wb, ctx->dtype);
    dim3 grid(rc * (ctx->nn * a.nch + a.nbn * a.nchb) * a.nparts);
    const int cfg = (ctx->gather_cfg >= 0 && ctx->gather_cfg < kNumGatherCfgs) ? ctx->gather_cfg : 0;
    launch_cfg(ctx, cfg, a, grid, smem);
    EXM_CUDA(cudaGetLastError());
    // algorithmic work of this launch: one node-tap per (template slot, lag, walked time)
    double slots = 0;
    for (int k = 0; k < ctx->nn; ++k) {
        const int lo = std::max(ctx->mlo[k], ci.m_base), hi = std::min(ctx->mhi[k], ci.m_base + ci.nmc);
        slots += std::max(0, hi - lo);
    }
    for (int i = ci.m_base; i < ci.m_base + ci.nmc; ++i) slots += ctx->bnode[i] >= 0;
    ctx->node_taps += slots * rc * ci.nwalk;
    ctx->tlw += (double)ci.nmc * rc * ci.nwalk;
    ctx->gather_launches += 1;
    ctx->launches += 1;
}

// ------------------------------------------------------------------ the general gather contract, float64

struct SimpleArgs {
    const float2 *H, *L;
    const float *Hlo, *Llo;
    const int32_t *sel;
    const void *T;              // node tables (element type TE of the kernel)
    const float *tsc;           // per node scale
    const int *rows, *tab, *tau;
    const double *lna;
    double *om, *os;
    long long tstride;
    int nt, nwalk, use_sel, ns, nsel, nphif, nb, nd, ndp, ntau;
    float lw;
    double beta0, dbeta, rph, rdb, rdd, offd;
};

template <typename TE>
__device__ __forceinline__ void ld_pair(const TE *row, int d0, int d1, double &x, double &y)
{
    x = (double)TabElem<TE>::ld(row + d0);
    y = (double)TabElem<TE>::ld(row + d1);
}

// One block per (row, lag).  A tap's phase planes and Delta coordinate do not depend on the slot, so kSlots slots share
// them and the tap's loads (the Delta coordinate changes only where a slot clamps beta); the running maximum and sum of
// a slot take one exponential without a branch.  The float64 arithmetic is the reference's, in its order.  Bound by
// instruction issue and the reads of four random table rows a tap together, so four blocks an SM (64 registers):
// a call of 96 rows x 6 slots x 87 lags x 2048 times 1.98 ms with every slot on its own, 1.48 with three (two 1.49,
// four 1.61, three at five blocks 1.80, at the compiler's 80 registers 1.78; aligned four-wide loads 2.4).
constexpr int kSlots = 3;

template <typename TE>
__global__ void __launch_bounds__(256, 4) k_gather_simple(SimpleArgs a)
{
    __shared__ double shm[kSlots][8], shs[kSlots][8];
    const int j = blockIdx.x, r = blockIdx.y;
    const int row = a.rows[j];
    const int nt = a.nt, nb = a.nb, nd = a.nd, ndp = a.ndp;
    const int tau0 = ((a.tau[r] % nt) + nt) % nt;
    const float2 *H = a.H + (long long)row * nt, *L = a.L + (long long)row * nt;
    const float *Hlo = a.Hlo ? a.Hlo + (long long)row * nt : nullptr, *Llo = a.Llo ? a.Llo + (long long)row * nt : nullptr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double bmax = nb - 1 - 1e-6, dmax = nd - 1 - 1e-6;
    const long long plane = (long long)nb * ndp;
    for (int n0 = 0; n0 < a.ns; n0 += kSlots) {
        const TE *Tn[kSlots];
        double sc[kSlots], offb[kSlots], m[kSlots], s[kSlots];
#pragma unroll
        for (int n = 0; n < kSlots; ++n) {
            const int at = j * a.ns + min(n0 + n, a.ns - 1);
            const int tb = a.tab[at];
            Tn[n] = (const TE *)a.T + (long long)tb * a.tstride + (long long)r * a.nphif * plane;
            sc[n] = (double)a.tsc[tb];
            offb[n] = (a.lna[at] - a.beta0) / a.dbeta;
            m[n] = -1e300;
            s[n] = 0.0;
        }
        for (int kk = threadIdx.x; kk < a.nwalk; kk += blockDim.x) {
            int t = kk, flag = 0;
            if (a.use_sel) {
                const int v = a.sel[(long long)row * a.nwalk + kk];
                t = v & 0x7FFFFFFF;
                flag = (unsigned)v >> 31;
            }
            int i1 = t + tau0;
            if (i1 >= nt) i1 -= nt;
            const float2 l = L[t], h = H[i1];
            double x3 = (double)(h.y - l.y) * a.rph;
            if (x3 < 0.0) x3 += EXM_NPHI;
            if (x3 >= EXM_NPHI) x3 -= EXM_NPHI;
            int c0 = (int)x3;
            c0 = c0 < 0 ? 0 : (c0 > EXM_NPHI - 1 ? EXM_NPHI - 1 : c0);
            const double fc = x3 - c0;
            int c1 = (c0 + 1) % EXM_NPHI;
            if (c0 > EXM_NPHI / 2) c0 = EXM_NPHI - c0;
            if (c1 > EXM_NPHI / 2) c1 = EXM_NPHI - c1;
            const double aL = (double)l.x + (double)(Llo ? Llo[t] : 0.f), aH = (double)h.x + (double)(Hlo ? Hlo[i1] : 0.f);
            double xs = (aH - aL) * a.rdd + a.offd;
            if (xs < 0.0) xs = 0.0; else if (xs > dmax) xs = dmax;
#pragma unroll
            for (int n = 0; n < kSlots; ++n) {
                if (n0 + n >= a.ns) break;
                const double xbr = aL * a.rdb + offb[n];
                double xb = xbr, xd = xs;
                if (xb < 0.0) xb = 0.0; else if (xb > bmax) xb = bmax;
                if (xb != xbr) {   // a clamped beta moves ln q_L, and Delta with it
                    const double aLc = aL + (xb - xbr) / a.rdb;
                    xd = (aH - aLc) * a.rdd + a.offd;
                    if (xd < 0.0) xd = 0.0; else if (xd > dmax) xd = dmax;
                }
                const int d0 = (int)xd;
                const double fdf = xd - d0, fd0 = 1.0 - fdf;
                const int d1 = d0 + 1 < nd ? d0 + 1 : nd - 1;
                const int b0 = (int)xb;
                const double fbf = xb - b0, fb0 = 1.0 - fbf;
                const int b1 = b0 + 1 < nb ? b0 + 1 : nb - 1;
                const long long o0 = (long long)b0 * ndp, o1 = (long long)b1 * ndp;
                double x00, x01, x10, x11, y00, y01, y10, y11;
                const TE *p0 = Tn[n] + c0 * plane, *p1 = Tn[n] + c1 * plane;
                ld_pair(p0 + o0, d0, d1, x00, x01);
                ld_pair(p0 + o1, d0, d1, x10, x11);
                ld_pair(p1 + o0, d0, d1, y00, y01);
                ld_pair(p1 + o1, d0, d1, y10, y11);
                const double v0 = fb0 * (fd0 * x00 + fdf * x01) + fbf * (fd0 * x10 + fdf * x11);
                const double v1 = fb0 * (fd0 * y00 + fdf * y01) + fbf * (fd0 * y10 + fdf * y11);
                double acc = (1.0 - fc) * v0;
                acc += fc * v1;
                acc *= sc[n];
                if (a.use_sel) acc += flag ? (double)a.lw : 0.0;
                const bool up = acc > m[n];
                const double e = exp(up ? m[n] - acc : acc - m[n]);
                s[n] = up ? s[n] * e + 1.0 : s[n] + e;
                m[n] = up ? acc : m[n];
            }
        }
#pragma unroll
        for (int n = 0; n < kSlots; ++n) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double m2 = __shfl_down_sync(0xffffffffu, m[n], o), s2 = __shfl_down_sync(0xffffffffu, s[n], o);
                if (m2 > m[n]) {
                    s[n] = s2 + s[n] * exp(m[n] - m2);
                    m[n] = m2;
                } else {
                    s[n] = s[n] + s2 * exp(m2 - m[n]);
                }
            }
            if (lane == 0) {
                shm[n][warp] = m[n];
                shs[n][warp] = s[n];
            }
        }
        __syncthreads();
        if (threadIdx.x < kSlots && n0 + (int)threadIdx.x < a.ns) {
            const int n = threadIdx.x;
            double M = shm[n][0], S = shs[n][0];
            for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
                if (shm[n][q] > M) {
                    S = shs[n][q] + S * exp(M - shm[n][q]);
                    M = shm[n][q];
                } else {
                    S = S + shs[n][q] * exp(shm[n][q] - M);
                }
            }
            const long long o = ((long long)(n0 + n) * a.ntau + r) * a.nsel + j;
            a.om[o] = M;
            a.os[o] = S;
        }
        __syncthreads();
    }
}

__global__ void k_lse_lags(const double *om, const double *os, int ns, int ntau, int nsel, int nt, double *out)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= ns * nsel) return;
    const int n = idx / nsel, j = idx - n * nsel;
    double mx = -INFINITY;
    for (int r = 0; r < ntau; ++r) mx = fmax(mx, om[((long long)n * ntau + r) * nsel + j]);
    double tot = 0.0;
    for (int r = 0; r < ntau; ++r) {
        const long long o = ((long long)n * ntau + r) * nsel + j;
        tot += os[o] * exp(om[o] - mx);
    }
    out[idx] = mx + log(tot) - log((double)nt);
}

void exm_run_gather_simple(exm_ctx *ctx, exm_slot &sl, int nsel, int ns, const int *d_rows, const int *d_tab,
                           const double *d_lna, int nwalk, int use_sel, float lw, double *d_out)
{
    SimpleArgs a;
    a.H = (const float2 *)sl.traj.p;
    a.L = a.H + (size_t)ctx->nm * ctx->nt;
    a.Hlo = ctx->traj_fp64 ? (const float *)sl.trajlo.p : nullptr;
    a.Llo = a.Hlo ? a.Hlo + (size_t)ctx->nm * ctx->nt : nullptr;
    a.sel = (const int32_t *)sl.sel.p;
    a.T = ctx->T.p;
    a.tsc = (const float *)ctx->d_tscale.p;
    a.rows = d_rows;
    a.tab = d_tab;
    a.tau = (const int *)ctx->d_tau.p;
    a.lna = d_lna;
    a.om = (double *)sl.part.p;
    a.os = a.om + (size_t)ns * ctx->ntau * nsel;
    a.tstride = (long long)ctx->tstride;
    a.nt = ctx->nt;
    a.nwalk = nwalk;
    a.use_sel = use_sel;
    a.ns = ns;
    a.nsel = nsel;
    a.nphif = ctx->nphif;
    a.nb = ctx->nb;
    a.nd = ctx->nd;
    a.ndp = ctx->ndp;
    a.ntau = ctx->ntau;
    a.lw = lw;
    a.beta0 = ctx->beta0;
    a.dbeta = ctx->dbeta;
    a.rph = EXM_NPHI / 6.283185307179586;
    a.rdb = 2.0 / ctx->dbeta;
    a.rdd = 1.0 / ctx->ddelta;
    a.offd = -ctx->delta0 / ctx->ddelta;
    dim3 grid(nsel, ctx->ntau);
    if (ctx->dtype == EXM_DTYPE_F16)
        k_gather_simple<__half><<<grid, 256, 0, ctx->stream>>>(a);
    else if (ctx->dtype == EXM_DTYPE_BF16)
        k_gather_simple<__nv_bfloat16><<<grid, 256, 0, ctx->stream>>>(a);
    else
        k_gather_simple<float><<<grid, 256, 0, ctx->stream>>>(a);
    k_lse_lags<<<(ns * nsel + 255) / 256, 256, 0, ctx->stream>>>(a.om, a.os, ns, ctx->ntau, nsel, ctx->nt, d_out);
    EXM_CUDA(cudaGetLastError());
}
