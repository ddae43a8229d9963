// Tap descriptors for the plane-staged gather.
//
// A tap is one (template, walked time, lag).  Its plane pair p, the weight of plane
// p + 1, beta-hat and the Delta coordinate do not depend on the node, so they are
// computed once per tap (in float64, as the reference computes them per node) and
// packed into 16 bytes:
//   x = fraction of beta-hat (float), y = fd (float, fraction of Delta),
//   z = w (float, weight of plane p + 1) | bit 31: the time is a random draw,
//   w = window offset (19 bits, signed) << 13 | template (13 bits),
// with the staging windows already placed (k_windows runs between the count and the
// scatter): the offset is (floor(beta-hat) - Rh) * columns + (d0 - C0), with Rh the row origin of the
// windows in beta-hat and C0 their first column; node k's window offset of the tap is then this plus a
// constant of the node plus a row when the two beta fractions carry, so the gather adds only the node's
// part.  EXM_O_FAR marks a tap outside every window (the exact path).
// For each lag the descriptors are counting-sorted by (p, template), so every node's
// gather block reads, for each plane pair it has staged, one contiguous run per warp.  Every (p, template)
// run is padded to whole groups of EXM_GT with entries that count for nothing (EXM_DESC_PAD).
// A second array holds each descriptor's time index for the exact slow path.
#include "common.cuh"
#include "kernels.cuh"

struct TapArgs {
    const float2 *H, *L;
    const float *Hlo, *Llo;   // residuals of ln|z| (filter precision 'fp64'), else null
    const int32_t *sel;
    const double *boff;   // [nmc] -ln(u)/dbeta of the chunk's templates
    const int *tau;       // [ntau]
    int *cnt;             // [rc][48][nmc + 1]
    int *cq;              // [nq][rc][48][nmc]: counts of each part of the walked times (nq > 1)
    int *hist_b;          // [EXM_HB_N]
    int *hist_d;          // [256]
    uint4 *desc;
    int32_t *tside;
    TapGeom g;
    int nmc, nwalk, use_sel, r0, rc, nq, want_hb;
    int hstep;            // the window histograms take every hstep-th walked time (a power of two)
    long long pitch;      // descriptors stored per lag (exm_desc_pitch)
    const int *win;       // window origins (k_windows): [0] column C0, [1 + EXM_MAX_NODES] beta-hat row Rh
    int wd;               // window columns
};

// The count: a block is one (template, part of its walked times), a lane one lag, walking the part's times in
// order; the template's samples at the walked times are staged kTapTile at a time.  The 32 lags of a warp read
// 32 consecutive samples of H (256 bytes) where one lag over 32 walked times reads 32 scattered sectors, and
// kTapBatch of them are in flight (2048 templates x 87 lags x 2048 times: 0.93 ms; a warp of walked times at one
// lag 4.6).
constexpr int kTapTile = 128;
constexpr int kTapBatch = 8;    // samples of H a lane of the count has in flight
constexpr int kTapWarps = 4;    // lag groups of 32 a block of the count takes at a time

struct WalkEntry {
    float x, y, lo;   // ln|z_L|, arg z_L, residual of ln|z_L|
    int t;            // the time; bit 31: a random draw
};

__device__ __forceinline__ void stage_walk(const TapArgs &a, int i, const float2 *L, const float *Llo, int k0, int k1,
                                           WalkEntry *w)
{
    __syncthreads();
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int v = a.use_sel ? a.sel[(long long)i * a.nwalk + k] : k;
        const int t = v & 0x7FFFFFFF;
        const float2 l = L[t];
        w[k - k0] = {l.x, l.y, Llo ? Llo[t] : 0.f, v};
    }
    __syncthreads();
}

// index of H's sample at lag tau0 for walked time k of the tile [k0, k1) (clamped to it)
__device__ __forceinline__ int sample_at(const WalkEntry *w, int k, int k0, int k1, int tau0, int nt)
{
    const int i1 = (w[min(k, k1 - 1) - k0].t & 0x7FFFFFFF) + tau0;
    return i1 >= nt ? i1 - nt : i1;
}

// counts per (lag, pair, template), and the histograms that place the staging windows (the beta-hat rows in the
// first pass over the lags; the Delta columns of every lag).  A lane's counters, one per plane pair, are its own
// column of shared memory: no atomics and no conflicts.
__global__ void __launch_bounds__(32 * kTapWarps) k_tap_count(TapArgs a)
{
    extern __shared__ int tc_sm[];   // [warps][EXM_NPAIR][32]
    int (*c)[EXM_NPAIR][32] = (int (*)[EXM_NPAIR][32])tc_sm;
    __shared__ WalkEntry w[kTapTile];
    __shared__ int hd[256];
    const int i = blockIdx.x, part = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ka = (int)((long long)a.nwalk * part / a.nq), kb = (int)((long long)a.nwalk * (part + 1) / a.nq);
    for (int q = threadIdx.x; q < 256; q += blockDim.x) hd[q] = 0;
    const int nt = a.g.nt;
    const float2 *H = a.H + (long long)i * nt, *L = a.L + (long long)i * nt;
    const float *Hlo = a.Hlo ? a.Hlo + (long long)i * nt : nullptr, *Llo = a.Llo ? a.Llo + (long long)i * nt : nullptr;
    const double boff = a.boff[i];
    for (int g0 = 0; g0 < a.rc; g0 += 32 * nw) {
        const int rl = g0 + 32 * warp + lane;
        const bool on = rl < a.rc;
        const int tau0 = on ? ((a.tau[a.r0 + rl] % nt) + nt) % nt : 0;
        for (int p = 0; p < EXM_NPAIR; ++p) c[warp][p][lane] = 0;
        for (int k0 = ka; k0 < kb; k0 += kTapTile) {
            const int k1 = min(kb, k0 + kTapTile);
            stage_walk(a, i, L, Llo, k0, k1, w);
            if (a.want_hb && g0 == 0)
                for (int k = k0 + threadIdx.x * a.hstep; k < k1; k += blockDim.x * a.hstep)
                    atomicAdd(&a.hist_b[exm_tap_row(w[k - k0].x, w[k - k0].lo, boff, a.g) - EXM_HB_LO], 1);
            if (on) {
                for (int kk = k0; kk < k1; kk += kTapBatch) {
                    float2 h[kTapBatch];
#pragma unroll
                    for (int m = 0; m < kTapBatch; ++m) h[m] = __ldg(H + sample_at(w, kk + m, k0, k1, tau0, nt));
#pragma unroll
                    for (int m = 0; m < kTapBatch; ++m) {
                        const int k = kk + m;
                        if (k >= k1) break;
                        const WalkEntry e = w[k - k0];
                        int p;
                        float wp;
                        exm_tap_phase(e.y, h[m].y, a.g, p, wp);
                        c[warp][p][lane] += 1;
                        if ((k & (a.hstep - 1)) == 0) {
                            int d0;
                            float fd;
                            const float hlo = Hlo ? Hlo[sample_at(w, k, k0, k1, tau0, nt)] : 0.f;
                            exm_tap_delta(e.x, e.lo, h[m].x, hlo, a.g, d0, fd);
                            atomicAdd(&hd[d0], 1);
                        }
                    }
                }
            }
        }
        if (on)
            for (int p = 0; p < EXM_NPAIR; ++p) {
                const int v = c[warp][p][lane];
                if (a.nq == 1)
                    a.cnt[((long long)rl * EXM_NPAIR + p) * (a.nmc + 1) + i] = v;
                else
                    a.cq[(((long long)part * a.rc + rl) * EXM_NPAIR + p) * a.nmc + i] = v;
            }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 256; q += blockDim.x)
        if (hd[q]) atomicAdd(&a.hist_d[q], hd[q]);
}

// exclusive scan over (pair, template) per lag of the counts in whole groups: cnt becomes the start
// offsets; column nmc of pair p is the start of pair p + 1
// (cq, nq > 1: the counts come in nq parts)
__global__ void __launch_bounds__(1024) k_tap_scan(int *cnt, int nmc, const int *cq, int nq, int rc)
{
    constexpr int E = 8;   // consecutive entries a thread
    __shared__ int sh[33];
    const int rl = blockIdx.x;
    int *c = cnt + (long long)rl * EXM_NPAIR * (nmc + 1);
    const int n = EXM_NPAIR * nmc;
    int carry = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = 0; base < n; base += blockDim.x * E) {
        int p = (base + (int)threadIdx.x * E) / nmc, i = base + (int)threadIdx.x * E - p * nmc;
        int v[E], at[E], sum = 0;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            at[k] = p * (nmc + 1) + i;
            v[k] = 0;
            if (p < EXM_NPAIR) {
                if (nq == 1) {
                    v[k] = c[at[k]];
                } else {
                    for (int q = 0; q < nq; ++q) v[k] += cq[(((long long)q * rc + rl) * EXM_NPAIR + p) * nmc + i];
                }
            }
            if (++i == nmc) {
                i = 0;
                ++p;
            }
        }
#pragma unroll
        for (int k = 0; k < E; ++k) {
            v[k] = (v[k] + EXM_GT - 1) & ~(EXM_GT - 1);
            sum += v[k];
        }
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sh[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int s = sh[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            sh[lane] = s;
        }
        __syncthreads();
        int run = carry + x - sum + (warp ? sh[warp - 1] : 0);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            if (at[k] < EXM_NPAIR * (nmc + 1)) c[at[k]] = run;
            run += v[k];
        }
        carry += sh[31];
        __syncthreads();
    }
    for (int p = threadIdx.x; p < EXM_NPAIR; p += blockDim.x)
        c[p * (nmc + 1) + nmc] = (p + 1 < EXM_NPAIR) ? c[(p + 1) * (nmc + 1)] : carry;
}

// descriptors, scattered to their (lag, pair, template) runs in order of time, and the padding entries at
// the runs' ends.  A block is one template and a range of the lags, one lag at a time: a batch is SCATTER_ROUNDS
// rounds of 256 walked times; each warp counts its taps per pair in each round, a thread per pair turns the
// counts into exclusive prefixes in (round, warp) order -- the order of time -- and every tap lands at its
// run's next position + the prefix + its rank among the equal pairs of its warp.  The walked times stay in
// shared memory for every lag (kScatterCache of them; longer walks are staged again for each lag), and the
// next batch's samples of H are loaded while this one is placed.  One lag at a time, although several would
// share the sectors of H: the stores go to 48 runs of a lag, all blocks being at about the same lag, and with two
// or four lags in flight the pages of the descriptors no longer stay translated (2048 templates x 87 lags x
// 2048 times, the whole tap build: 10.6 ms with one lag, 12.0 with two, 13.3 with four; 30 with a lag a lane).
#define SCATTER_ROUNDS 4
constexpr int kScatterCache = 2048;
constexpr int kScatterBatch = SCATTER_ROUNDS * 256;

__global__ void __launch_bounds__(256) k_tap_scatter(TapArgs a)
{
    __shared__ unsigned short wcnt[SCATTER_ROUNDS][8][EXM_NPAIR];   // counts, then prefixes within the batch
    __shared__ int base[EXM_NPAIR];
    extern __shared__ WalkEntry w[];
    const int i = blockIdx.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int ra = a.rc * blockIdx.y / gridDim.y, rb = a.rc * (blockIdx.y + 1) / gridDim.y;
    const int nt = a.g.nt;
    const float2 *H = a.H + (long long)i * nt, *L = a.L + (long long)i * nt;
    const float *Hlo = a.Hlo ? a.Hlo + (long long)i * nt : nullptr, *Llo = a.Llo ? a.Llo + (long long)i * nt : nullptr;
    const double boff = a.boff[i];
    const unsigned lt = (1u << lane) - 1u;
    const int C0 = a.win[0], Rh = a.win[1 + EXM_MAX_NODES];
    for (int rl = ra; rl < rb; ++rl) {
        const int tau0 = ((a.tau[a.r0 + rl] % nt) + nt) % nt;
        uint4 *desc = a.desc + (long long)rl * a.pitch;
        int32_t *tside = a.tside + (long long)rl * a.pitch;
        if (tid < EXM_NPAIR)   // read after the next barrier
            base[tid] = a.cnt[((long long)rl * EXM_NPAIR + tid) * (a.nmc + 1) + i];
        for (int c0 = 0; c0 < a.nwalk; c0 += kScatterCache) {
            const int c1 = min(a.nwalk, c0 + kScatterCache);
            if (rl == ra || a.nwalk > kScatterCache) stage_walk(a, i, L, Llo, c0, c1, w);
            float2 h[SCATTER_ROUNDS];
            float hlo[SCATTER_ROUNDS];
            auto load = [&](int k0) {
#pragma unroll
                for (int m = 0; m < SCATTER_ROUNDS; ++m) {
                    const int i1 = sample_at(w, k0 + m * 256 + tid, c0, c1, tau0, nt);
                    h[m] = __ldg(H + i1);
                    hlo[m] = Hlo ? __ldg(Hlo + i1) : 0.f;
                }
            };
            load(c0);
            for (int k0 = c0; k0 < c1; k0 += kScatterBatch) {
                // the batch's pairs, plane weights and Delta coordinates; then its samples make room for the next's
                int p[SCATTER_ROUNDS], rk[SCATTER_ROUNDS], d0[SCATTER_ROUNDS];
                float wp[SCATTER_ROUNDS], fd[SCATTER_ROUNDS];
#pragma unroll
                for (int m = 0; m < SCATTER_ROUNDS; ++m) {
                    const int k = k0 + m * 256 + tid;
                    p[m] = -1;
                    d0[m] = 0;
                    wp[m] = fd[m] = 0.f;
                    if (k < c1) {
                        const WalkEntry e = w[k - c0];
                        exm_tap_phase(e.y, h[m].y, a.g, p[m], wp[m]);
                        exm_tap_delta(e.x, e.lo, h[m].x, hlo[m], a.g, d0[m], fd[m]);
                    }
                }
                if (k0 + kScatterBatch < c1) load(k0 + kScatterBatch);
                for (int q = tid; q < SCATTER_ROUNDS * 8 * EXM_NPAIR / 2; q += blockDim.x)
                    ((unsigned *)&wcnt[0][0][0])[q] = 0;
                __syncthreads();
#pragma unroll
                for (int m = 0; m < SCATTER_ROUNDS; ++m) {
                    const unsigned peers = __match_any_sync(0xffffffffu, p[m]);
                    rk[m] = __popc(peers & lt);
                    if (p[m] >= 0 && rk[m] == 0) wcnt[m][warp][p[m]] = (unsigned short)__popc(peers);
                }
                __syncthreads();
                int run = 0;
                if (tid < EXM_NPAIR) {   // exclusive prefixes per pair in (round, warp) order
#pragma unroll
                    for (int m = 0; m < SCATTER_ROUNDS; ++m)
#pragma unroll
                        for (int ww = 0; ww < 8; ++ww) {
                            const int v = wcnt[m][ww][tid];
                            wcnt[m][ww][tid] = (unsigned short)run;
                            run += v;
                        }
                }
                __syncthreads();
#pragma unroll
                for (int m = 0; m < SCATTER_ROUNDS; ++m) {
                    if (p[m] < 0) continue;
                    const int pos = base[p[m]] + wcnt[m][warp][p[m]] + rk[m];
                    const WalkEntry e = w[k0 - c0 + m * 256 + tid];
                    int ib;
                    float fb;
                    exm_tap_beta(e.x, e.lo, boff, a.g, ib, fb);
                    const int rd = d0[m] - C0, rb0 = ib - Rh;
                    const bool far = (unsigned)rd > (unsigned)(a.wd - 2) || rb0 < -1024 || rb0 > 1023;
                    if (pos >= 0 && pos < a.pitch) {   // sorted order; k_tap_order rearranges each chunk afterwards
                        desc[pos] = make_uint4(__float_as_uint(fb), __float_as_uint(fd[m]),
                                               __float_as_uint(wp[m]) | ((unsigned)e.t & 0x80000000u),
                                               ((unsigned)(far ? EXM_O_FAR : rb0 * a.wd + rd) << 13) | (unsigned)i);
                        tside[pos] = e.t & 0x7FFFFFFF;
                    }
                }
                __syncthreads();
                if (tid < EXM_NPAIR) base[tid] += run;
            }
        }
        if (tid < EXM_NPAIR)
            for (long long pos = base[tid]; pos & (EXM_GT - 1); ++pos)
                if (pos < a.pitch) {
                    desc[pos] = make_uint4(0u, 0u, 0u, EXM_DESC_PAD | (unsigned)i);
                    tside[pos] = 0;
                }
    }
}

// Each chunk of descriptors (and time indices) of every lag, from sorted order to the gather's
// lane-interleaved order (exm_desc_phys), in place through shared memory: writing the interleaved order
// directly from the scatter would spread 16-byte stores over many sectors.
//
// The order of a lane's taps of one template is free, and the gather's shared loads are bound by bank
// conflicts: the window's pitch is a multiple of the 32 banks, so a tap's bank is its column's, the same at every
// node.  So each step of the chunk (one tap of every lane) takes taps of different banks where it can: every lane
// proposes a bank not yet used, the first of its candidates' from a start that differs from lane to lane and
// turns with the step; the lowest lane of a bank wins, the others propose again (kOrderRounds1 times; then
// kOrderRounds2 times for a second tap per bank, then whatever is left).  The fullest bank holds about 26 of
// a chunk's 512 taps, so 1.6 taps per step is the least any order could reach; this one reaches 2.9 (2.7 with
// eight rounds and the fullest banks first), the sorted order 3.6.  More rounds cost this kernel what they save the
// gather (rounds 1 + 2: gather 63.0 and tap build 10.2 ms, 2 + 2: 62.7 and 10.7, 4 + 3: 62.9 and 11.3).  One warp per chunk;
// the banks of a lane's taps are bytes of four registers and the candidates are bit masks.
constexpr int kOrderRounds1 = 1, kOrderRounds2 = 2;
constexpr int kOrderWarps = 4;
// a warp's shared memory: the chunk, a lane's taps padded by one against conflicts, and per bank the claim of a
// round (its number << 5 | 31 - lane of the lowest proposer).  It is as small as the chunk: the kernel waits on
// its own short chains, and small chunks leave room for more warps.
inline size_t order_warp_bytes(int ng) { return (32 * (EXM_GT * ng + 1)) * (sizeof(uint4) + sizeof(int32_t)) + 32 * sizeof(unsigned); }

__global__ void __launch_bounds__(32 * kOrderWarps) k_tap_order(uint4 *__restrict__ desc, int32_t *__restrict__ tside,
                                                                const int *__restrict__ cnt, int nmc, long long pitch,
                                                                int ng, int shift)
{
    // shift: 0 for float32 tables (a bank per column), 1 for 16-bit (two columns a bank)
    extern __shared__ unsigned char osm[];
    __shared__ int pair0[EXM_NPAIR];   // the first position of each plane pair
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rl = blockIdx.y, tpl = EXM_GT * ng, size = 32 * tpl, row_d = tpl + 1;
    uint4 *sm_d = (uint4 *)(osm + (size_t)warp * (32 * row_d * (sizeof(uint4) + sizeof(int32_t)) + 32 * sizeof(unsigned)));
    int32_t *sm_t = (int32_t *)(sm_d + 32 * row_d);
    unsigned *sm_claim = (unsigned *)(sm_t + 32 * row_d);
    if (threadIdx.x < EXM_NPAIR) pair0[threadIdx.x] = cnt[((long long)rl * EXM_NPAIR + threadIdx.x) * (nmc + 1)];
    __syncthreads();
    const int used_taps = (int)min((long long)cnt[(long long)(rl + 1) * EXM_NPAIR * (nmc + 1) - 1], pitch);
    const int n_chunks = (used_taps + size - 1) / size;
    sm_claim[lane] = 0u;
    unsigned stamp = 0u;
    for (int ch = blockIdx.x * kOrderWarps + warp; ch < n_chunks; ch += gridDim.x * kOrderWarps) {
        uint4 *d = desc + rl * pitch + (long long)ch * size;
        int32_t *t = tside + rl * pitch + (long long)ch * size;
#pragma unroll 4
        for (int q = lane; q < size; q += 32) {
            const bool in = ch * size + q < used_taps;
            const uint4 v = in ? d[q] : make_uint4(0u, 0u, 0u, EXM_DESC_PAD);
            const int at = (q / tpl) * row_d + q % tpl;
            sm_d[at] = v;
            sm_t[at] = in ? t[q] : 0;
        }
        __syncwarp();
        // this lane's taps: their banks, and per group the lane's groups of the same run
        const uint4 *row = sm_d + lane * row_d;
        unsigned bk[EXM_NG_MAX], same[EXM_NG_MAX], tm[EXM_NG_MAX];
#pragma unroll
        for (int g = 0; g < EXM_NG_MAX; ++g) {
            bk[g] = 0xFFFFFFFFu;
            tm[g] = 0xFFFFFFFFu;
            if (g < ng) {
                unsigned v = 0;
#pragma unroll
                for (int u = 0; u < EXM_GT; ++u) {
                    const unsigned w = row[g * EXM_GT + u].w;
                    const int o0 = (int)w >> 13;
                    // far and padding entries read the window at the lane's own column
                    const int bank = (o0 != EXM_O_FAR && o0 != EXM_O_PAD) ? (o0 >> shift) & 31 : lane >> shift;
                    v |= (unsigned)bank << (8 * u);
                    tm[g] = w & 0x1FFFu;
                }
                bk[g] = v;
                // a run is a template's taps of one plane pair; the entries after the last run are one of their own
                const int pos = ch * size + lane * tpl + g * EXM_GT;
                int p = 0;
                for (int st = 32; st > 0; st >>= 1)
                    if (p + st < EXM_NPAIR && pair0[p + st] <= pos) p += st;
                tm[g] = pos < used_taps ? tm[g] | ((unsigned)p << 13) : 0xFFFFFFFEu;
            }
        }
#pragma unroll
        for (int g = 0; g < EXM_NG_MAX; ++g) {
            same[g] = 0;
#pragma unroll
            for (int h = 0; h < EXM_NG_MAX; ++h)
                if (tm[h] == tm[g]) same[g] |= 0xFu << (EXM_GT * h);
        }
        unsigned rem = (1u << tpl) - 1u;   // the lane's taps not yet placed
#pragma unroll 1
        for (int g = 0; g < ng; ++g) {
            unsigned sg = same[0];
#pragma unroll
            for (int h = 1; h < EXM_NG_MAX; ++h) sg = g == h ? same[h] : sg;
            unsigned cand = rem & sg;
            unsigned banks = 0;   // the candidates' banks
#pragma unroll
            for (int s = 0; s < EXM_GT * EXM_NG_MAX; ++s)
                if ((cand >> s) & 1u) banks |= 1u << ((bk[s / EXM_GT] >> (8 * (s % EXM_GT))) & 31u);
#pragma unroll 1
            for (int u = 0; u < EXM_GT; ++u) {
                int pick = -1;
                const int off = (lane + 5 * (g * EXM_GT + u)) & 31;
#pragma unroll 1
                for (int ph = 0; ph < 2; ++ph) {
                    unsigned taken = 0;
                    const int rounds = ph ? kOrderRounds2 : kOrderRounds1;
#pragma unroll 1
                    for (int k = 0; k < rounds; ++k) {
                        const unsigned av = pick < 0 ? banks & ~taken : 0u;
                        const int r = (__ffs(__funnelshift_r(av, av, off)) - 1 + off) & 31;
                        const unsigned asked = __reduce_or_sync(0xffffffffu, av ? 1u << r : 0u);
                        if (!asked) break;
                        taken |= asked;
                        // the lowest lane that proposes the same bank
                        stamp += 32u;
                        if (av) atomicMax(&sm_claim[r], stamp | (31u - lane));
                        __syncwarp();
                        if (av && sm_claim[r] == (stamp | (31u - lane))) pick = r;
                        __syncwarp();
                    }
                }
                if (pick < 0) pick = __ffs(banks) - 1;
                // a candidate of that bank, and whether it was the bank's last
                unsigned eq = 0;
#pragma unroll
                for (int h = 0; h < EXM_NG_MAX; ++h)
                    eq |= (((__vcmpeq4(bk[h], 0x01010101u * (unsigned)pick) & 0x08040201u) * 0x01010101u) >> 24) << (EXM_GT * h);
                eq &= cand;
                const int j = __ffs(eq) - 1;
                if ((eq & (eq - 1u)) == 0u) banks &= ~(1u << pick);
                cand &= ~(1u << j);
                rem &= ~(1u << j);
                const int at = lane * row_d + j, ph = (g * EXM_GT + u) * 32 + lane;
                d[ph] = sm_d[at];
                t[ph] = sm_t[at];
            }
        }
        __syncwarp();
    }
}

// staging-window origins: column C0 (a multiple of calign elements, 16 bytes), per node the
// first beta row, and the beta-hat row origin Rh they derive from; wb rows x wd columns per window
__global__ void __launch_bounds__(1024) k_windows(const int *hist_b, const int *hist_d, const int *cki, int nn, int nb,
                                                  int nd, int ndp, int wb, int wd, int calign, int *win)
{
    // sums over windows as differences of prefix sums, in shared memory
    __shared__ unsigned pb[EXM_HB_N + 1], pd[256 + 1];
    __shared__ unsigned long long best[2];
    __shared__ unsigned ws[33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 2) best[tid] = 0;
    if (tid == 0) pb[0] = pd[0] = 0;
    for (int ph = 0; ph < 2; ++ph) {   // the beta-hat histogram, two bins a thread; then the columns
        const unsigned v0 = ph ? (tid < 256 ? (unsigned)hist_d[tid] : 0u) : (unsigned)hist_b[2 * tid];
        const unsigned v1 = ph ? 0u : (unsigned)hist_b[2 * tid + 1];
        unsigned x = v0 + v1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned s = ws[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            ws[lane] = s;
        }
        __syncthreads();
        const unsigned incl = x + (warp ? ws[warp - 1] : 0u);
        if (ph == 0) {
            pb[2 * tid + 1] = incl - v1;
            pb[2 * tid + 2] = incl;
        } else if (tid < 256) {
            pd[tid + 1] = incl;
        }
        __syncthreads();
    }
    // columns: d0 in [C0, C0 + wd - 2]
    const int cmax = max(0, ndp - wd);
    for (int c0 = tid * calign; c0 <= cmax; c0 += blockDim.x * calign) {
        const unsigned s = pd[min(c0 + wd - 2, nd - 1) + 1] - pd[c0];
        atomicMax(&best[0], ((unsigned long long)s << 12) | (4095 - c0 / calign));
    }
    // beta-hat rows: ib in [Rh, Rh + wb - 3]
    for (int rh = tid; rh < EXM_HB_N; rh += blockDim.x) {
        const unsigned s = pb[min(rh + wb - 3, EXM_HB_N - 1) + 1] - pb[rh];
        atomicMax(&best[1], ((unsigned long long)s << 12) | (4095 - rh));
    }
    __syncthreads();
    const int rh = (4095 - (int)(best[1] & 4095)) + EXM_HB_LO;
    if (tid == 0) {
        win[0] = (4095 - (int)(best[0] & 4095)) * calign;
        win[1 + EXM_MAX_NODES] = rh;
    }
    if (tid < nn) win[1 + tid] = max(0, min(rh + cki[tid], nb - wb));
}

// Parts of the walked times in the count: as many as give each SM about 16 warps of lags, of at least 64 times (more
// parts cost more than they bring: every part writes its own counts, each to a sector of its own)
int exm_tap_parts(int sm_count, int nmc, int nwalk, int rc)
{
    const long long warps = (long long)nmc * ((rc + 31) / 32);
    long long nq = 1;
    while (nq < 32 && warps * nq < 16LL * sm_count && nwalk / (2 * nq) >= 64) nq *= 2;
    return (int)nq;
}

void exm_run_taps(exm_ctx *ctx, exm_slot &sl, const ChunkInfo &ci, int r0, int rc, bool first_chunk_of_lags)
{
    const int nt = ctx->nt;
    TapArgs a;
    a.H = (const float2 *)sl.traj.p;
    a.L = a.H + (size_t)ci.nmc * nt;
    a.Hlo = ctx->traj_fp64 ? (const float *)sl.trajlo.p : nullptr;
    a.Llo = a.Hlo ? a.Hlo + (size_t)ci.nmc * nt : nullptr;
    a.sel = (const int32_t *)sl.sel.p;
    a.boff = (const double *)ctx->d_bhat_off.p + ci.m_base;
    a.tau = (const int *)ctx->d_tau.p;
    a.cnt = (int *)sl.cnt.p;
    a.hist_b = (int *)sl.hist.p;
    a.hist_d = a.hist_b + EXM_HB_N;
    a.desc = (uint4 *)sl.desc.p;
    a.tside = (int32_t *)sl.tside.p;
    a.g.rph = EXM_NPHI / 6.283185307179586;
    a.g.rdb = 2.0 / ctx->dbeta;
    a.g.rdd = 1.0 / ctx->ddelta;
    a.g.offd = -ctx->delta0 / ctx->ddelta;
    a.g.nd = ctx->nd;
    a.g.nt = nt;
    a.nmc = ci.nmc;
    a.nwalk = ci.nwalk;
    a.use_sel = ci.use_sel;
    a.r0 = r0;
    a.rc = rc;
    a.nq = exm_tap_parts(ctx->sm_count, ci.nmc, ci.nwalk, rc);
    a.cq = a.cnt + (size_t)rc * EXM_NPAIR * (ci.nmc + 1);
    a.hstep = (long long)ci.nmc * ci.nwalk > (1 << 18) ? 8 : 1;   // enough samples to place the windows
    a.want_hb = first_chunk_of_lags ? 1 : 0;
    a.pitch = exm_desc_pitch(ci.nmc, ci.nwalk);
    exm_gather_plan(ctx, ci, rc, &sl.wb, &sl.ng);
    if (first_chunk_of_lags) EXM_CUDA(cudaMemsetAsync(a.hist_b, 0, sizeof(int) * EXM_HB_N, ctx->stream));
    EXM_CUDA(cudaMemsetAsync(a.hist_d, 0, sizeof(int) * 256, ctx->stream));
    a.win = (const int *)sl.win.p;
    a.wd = exm_dtype_wd(ctx->dtype);
    const dim3 grid(ci.nmc, a.nq);
    const int warps = std::min(kTapWarps, (rc + 31) / 32);
    k_tap_count<<<grid, 32 * warps, (size_t)warps * EXM_NPAIR * 32 * sizeof(int), ctx->stream>>>(a);
    k_tap_scan<<<rc, 1024, 0, ctx->stream>>>(a.cnt, ci.nmc, a.cq, a.nq, rc);
    k_windows<<<1, 1024, 0, ctx->stream>>>(a.hist_b, a.hist_d, (const int *)ctx->d_cki.p, ctx->nn, ctx->nb, ctx->nd,
                                           ctx->ndp, sl.wb, a.wd, exm_dtype_calign(ctx->dtype), (int *)sl.win.p);
    // about twelve blocks an SM: a small bank's lags are shared out
    const int lag_parts = std::min(rc, std::max(1, (12 * ctx->sm_count + ci.nmc - 1) / ci.nmc));
    k_tap_scatter<<<dim3(ci.nmc, lag_parts), 256, std::min(kScatterCache, ci.nwalk) * sizeof(WalkEntry), ctx->stream>>>(a);
    const long long n_chunks = a.pitch / (32 * EXM_GT * sl.ng);
    const size_t osm = kOrderWarps * order_warp_bytes(sl.ng);
    exm_allow_smem(ctx, (const void *)k_tap_order, osm);
    const dim3 go((unsigned)std::min<long long>((n_chunks + kOrderWarps - 1) / kOrderWarps,
                                                std::max(1, ctx->sm_count * 40 / rc)), rc);
    k_tap_order<<<go, 32 * kOrderWarps, osm, ctx->stream>>>(a.desc, a.tside, a.cnt, ci.nmc, a.pitch, sl.ng,
                                                           ctx->dtype == EXM_DTYPE_F32 ? 0 : 1);
    EXM_CUDA(cudaGetLastError());
    ctx->launches += 5;
}
