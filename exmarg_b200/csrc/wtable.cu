// Stage 1 of the offline table build (scripts/build_tables/w_gpu.py:67-182): the GORFs at fixed distance
// at every node s_j, by quadrature over the sky pixels, the polarization angle psi and chi = cos(inclination):
//
//   Wraw_j(tau, (n, a, b)) = sum_pix dep(pix, tau) sum_q Bw_j(q) cos(m dph_q) m1_q^(a+b) m2_q^(2n-a-b),  m = a - b
//   Bw_j(q) = exp(-(s_j |R1|^2 + s_j |R2|^2)) w_q,  m_I = |R_I| / sqrt 2,  dph = arg R1 - arg R2
//   W_j = Wraw_j scale_j(n)
//
// One pixel at a time (its delay deposits on two tau bins, so within a launch every (node, tau, key) is
// written by one block and launches are ordered on the stream: no atomics):
//   k_w_prep: per quadrature point q, the responses R_I in float32 as the reference forms them (products and
//             sums rounded one by one; |R| and arg R rounded to float32 from float64), then in float64 the
//             power ladders m_I^k (k = 0 .. 2 n_max), dph and the damping Bw_j of every node;
//   k_w_cos:  cos(m dph_q) of every phase class m;
//   k_w_gemm: for a phase class m the keys form the triangle pw1 = m + 2x, pw2 = m + 2y, x + y <= n_max - m.
//             The triangle's columns of 8 x-values (x0 .. x0 + 7, y), y <= n_max - m - x0, are laid out one x-block
//             after the other, and a block takes 16 of them (128 keys, of one x-block and perhaps the next) and R RG
//             rows (nodes): a register-tiled float64 product over q, A[j][q] = Bw_j(q) and B[q][(x, y)] = m1_q^pw1
//             (m2_q^pw2 cos(m dph_q)), formed in registers from the tile's 8 or 16 + 16 ladder rows; three stages of
//             inputs arrive by asynchronous copies, one block barrier a step.
//   k_w_scale: W = Wraw * scale, rounded to float32, non-finite entries counted.
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace {

constexpr int kWRows = 64;       // most nodes
constexpr int kWX = 8;           // powers of |R1| of a tile
constexpr int kWY = 16;          // powers of |R2| of a tile
constexpr int kWCols = kWX * kWY;
constexpr int kWQ = 32;          // quadrature points per step
constexpr int kWPitch = kWQ + 2; // of a row in shared memory (doubles): 16-byte rows, two-way conflicts at most
constexpr int kWStages = 3;
constexpr int kWThreads = 128;

// quadrature points as stored: rows of a multiple of the step, zero beyond Q (such points add nothing)
inline int w_pitch(int Q) { return (Q + kWQ - 1) / kWQ * kWQ; }

__global__ void __launch_bounds__(128) k_w_prep(const float *__restrict__ resp, const float *__restrict__ c2p,
                                                const float *__restrict__ s2p, const float *__restrict__ ap,
                                                const float *__restrict__ cg, const double *__restrict__ wq, int n_psi,
                                                int n_chi, int n_nodes, const double *__restrict__ s, int nl, int Qp,
                                                double *__restrict__ lad1, double *__restrict__ lad2,
                                                double *__restrict__ dph, double *__restrict__ bw)
{
    const int Q = n_psi * n_chi;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= Qp) return;
    if (q >= Q) {
        dph[q] = 0.0;
        for (int k = 0; k < nl; ++k) lad1[(size_t)k * Qp + q] = lad2[(size_t)k * Qp + q] = 0.0;
        for (int j = 0; j < n_nodes; ++j) bw[(size_t)j * Qp + q] = 0.0;
        return;
    }
    const int ip = q / n_chi, ic = q - ip * n_chi;
    float mag[2], ang[2];
    for (int I = 0; I < 2; ++I) {
        const float fp0 = resp[2 * I], fx0 = resp[2 * I + 1];
        const float Fp = __fsub_rn(__fmul_rn(fp0, c2p[ip]), __fmul_rn(fx0, s2p[ip]));
        const float Fx = __fadd_rn(__fmul_rn(fp0, s2p[ip]), __fmul_rn(fx0, c2p[ip]));
        const double re = (double)__fmul_rn(ap[ic], Fp), im = (double)__fmul_rn(cg[ic], Fx);
        mag[I] = (float)sqrt(__dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im)));
        ang[I] = (float)atan2(im, re);
    }
    const double S1 = (double)__fmul_rn(mag[0], mag[0]), S2 = (double)__fmul_rn(mag[1], mag[1]);
    dph[q] = (double)__fsub_rn(ang[0], ang[1]);
    const double m1 = sqrt(S1 / 2.0), m2 = sqrt(S2 / 2.0);
    double a1 = 1.0, a2 = 1.0;
    lad1[q] = 1.0;
    lad2[q] = 1.0;
    for (int k = 1; k < nl; ++k) {
        a1 = __dmul_rn(a1, m1);
        a2 = __dmul_rn(a2, m2);
        lad1[(size_t)k * Qp + q] = a1;
        lad2[(size_t)k * Qp + q] = a2;
    }
    const double w = wq[ic];
    for (int j = 0; j < n_nodes; ++j)
        bw[(size_t)j * Qp + q] = __dmul_rn(exp(-__dadd_rn(__dmul_rn(s[j], S1), __dmul_rn(s[j], S2))), w);
}

// cm[m][q] = cos(m dph_q), once per pixel for all the tiles of a phase class
__global__ void __launch_bounds__(128) k_w_cos(const double *__restrict__ dph, int Qp, double *__restrict__ cm)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
    if (q < Qp) cm[(size_t)m * Qp + q] = cos(__dmul_rn((double)m, dph[q]));
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid)
{
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem), "r"(valid ? 16 : 0));
}

// RG row groups of R nodes and QG = 8 / RG groups of threads that share out the quadrature points: thread
// (tc, rg, qg) holds R nodes x 8 keys (x0 + c, y0 + tc) over the points qg, qg + QG, ... of each step, and the
// point groups' sums are added at the end.  Bound by the float64 pipe and its latency: the fewest rows that hold the
// nodes cost the fewest operations, and fewer sums a thread leave registers for three or four blocks an SM (R <= 7,
// R <= 4) instead of two.  Per pixel at order 120: 6 nodes 8.6 ms, 14 nodes 15.6, 30 nodes 32.7, 53 nodes 51.0; with
// square tiles (8 x 16, 78 % of their keys in the triangle against 90; at order 42 52 % against 68) 8.9, 17.4, 38.1, 55.9;
// groups of 8 rows whatever the nodes, on those, took 12.1, 20.4, 38.1, 67.2, and one tile of 64 rows with its products
// staged in shared memory (three barriers a step) 79.  The cosines' row between the two x-blocks keeps their lanes off
// each other's banks.  Twice the row groups of half the rows were slower (on square tiles 6 nodes 10.0, 14
// nodes 21.4) but at exactly 8 nodes (11.9 against 12.2): each thread forms the products of its keys again for fewer rows.
constexpr int w_rows(int rg, int r) { return r * rg + 2 * kWX + kWY + 1; }
constexpr int w_blocks(int r) { return r <= 4 ? 4 : r <= 7 ? 3 : 2; }
constexpr size_t w_smem(int rg, int r)
{
    const size_t st = sizeof(double) * kWStages * w_rows(rg, r) * kWPitch;
    return st > 32768 ? st : 32768;   // at the end: 32 KB of sums to add
}

template <int RG, int R>
__global__ void __launch_bounds__(kWThreads, w_blocks(R)) k_w_gemm(const int4 *__restrict__ tiles, int Qp, int n_nodes, int n_max,
                                                         const double *__restrict__ lad1, const double *__restrict__ lad2,
                                                         const double *__restrict__ cm, const double *__restrict__ bw,
                                                         int t0, double w0, double w1, int n_tau, long long n_keys,
                                                         double *__restrict__ Wraw)
{
    constexpr int QG = 8 / RG, NR = w_rows(RG, R), XC = R * RG + kWX, Y0 = XC + 1 + kWX;
    extern __shared__ __align__(16) double wsm[];   // [stage][row: nodes, x ladder, cos, x ladder of the next block, y ladder][point]
    const int4 tl = tiles[blockIdx.x];
    const int m = tl.x, x0 = tl.y, y0 = tl.z, na = tl.w;   // the tile's first na columns lie in the block x0, the others in the next
    const int L = n_max - m + 1;
    const int tid = threadIdx.x, tc = tid & 15, g = tid >> 4, rg = g % RG, qg = g / RG;
    const int nsteps = Qp / kWQ;
    auto issue = [&](int step, int buf) {
        double *st = wsm + (size_t)buf * NR * kWPitch;
        for (int i = tid; i < NR * (kWQ / 2); i += kWThreads) {
            const int row = i / (kWQ / 2), qq = 2 * (i - row * (kWQ / 2));
            const double *src = bw;
            bool ok;
            if (row < R * RG) {
                ok = row < n_nodes;
                if (ok) src = bw + (size_t)row * Qp;
            } else if (row == XC) {
                ok = true;
                src = cm + (size_t)m * Qp;
            } else if (row < Y0) {
                const int c = row - R * RG - (row > XC), x = x0 + c;
                ok = x <= L - 1 && (c < kWX || na < kWY);
                if (ok) src = lad1 + (size_t)(m + 2 * x) * Qp;
            } else {
                const int c = row - Y0, y = c < na ? y0 + c : c - na;
                ok = y <= L - 1;
                if (ok) src = lad2 + (size_t)(m + 2 * y) * Qp;
            }
            cp_async16(st + row * kWPitch + qq, src + (ok ? step * kWQ + qq : 0), ok);
        }
    };
    double acc[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[r][c] = 0.0;
#pragma unroll
    for (int k = 0; k < kWStages - 1; ++k) {
        if (k < nsteps) issue(k, k);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    for (int k = 0; k < nsteps; ++k) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kWStages - 2));
        __syncthreads();   // step k has arrived everywhere, and step k - 1's buffer is free
        if (k + kWStages - 1 < nsteps) issue(k + kWStages - 1, (k + kWStages - 1) % kWStages);
        asm volatile("cp.async.commit_group;\n" ::);
        const double *st = wsm + (size_t)(k % kWStages) * NR * kWPitch;
        const double *pa = st + rg * R * kWPitch, *px = st + (tc < na ? R * RG : XC + 1) * kWPitch;
        const double *py = st + (Y0 + tc) * kWPitch, *pc = st + XC * kWPitch;
#pragma unroll 2
        for (int qq = qg; qq < kWQ; qq += QG) {
            const double yc = __dmul_rn(py[qq], pc[qq]);
            double a[R], b[8];
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = pa[r * kWPitch + qq];
#pragma unroll
            for (int c = 0; c < 8; ++c) b[c] = __dmul_rn(px[c * kWPitch + qq], yc);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    // the point groups' sums, halving their number each time
#pragma unroll
    for (int h = QG / 2; h > 0; h /= 2) {
        __syncthreads();
        double *red = wsm + (size_t)((qg % h) * RG + rg) * R * 8 * 16 + tc;
        if (qg >= h && qg < 2 * h)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) red[(r * 8 + c) * 16] = acc[r][c];
        __syncthreads();
        if (qg < h)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[r][c] = __dadd_rn(acc[r][c], red[(r * 8 + c) * 16]);
    }
    if (qg) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int row = rg * R + r;
        if (row >= n_nodes) continue;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int x = (tc < na ? x0 : x0 + kWX) + c, y = tc < na ? y0 + tc : tc - na;
            if (x + y > L - 1) continue;
            const long long n = m + x + y, a = m + x, b = x;
            const long long key = n * (n + 1) * (n + 2) / 6 + a * (a + 1) / 2 + b;
            double *dst = Wraw + ((size_t)row * n_tau + t0) * n_keys + key;
            dst[0] = __dadd_rn(dst[0], __dmul_rn(w0, acc[r][c]));
            dst[n_keys] = __dadd_rn(dst[n_keys], __dmul_rn(w1, acc[r][c]));
        }
    }
}

__global__ void k_w_scale(const double *__restrict__ Wraw, const double *__restrict__ scale, int n_tau, long long n_keys,
                          long long n, float *__restrict__ out, unsigned long long *__restrict__ nonfinite)
{
    unsigned long long bad = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long k = i % n_keys, j = i / (n_keys * n_tau);
        const double v = __dmul_rn(Wraw[i], scale[j * n_keys + k]);
        out[i] = (float)v;
        bad += !isfinite(v);
    }
    if (bad) atomicAdd(nonfinite, bad);
}

}   // namespace

extern "C" int exm_w_build(exm_ctx *ctx, int n_nodes, const double *s_nodes, int n_max, int n_psi, int n_chi,
                           const float *c2p, const float *s2p, const float *ap, const float *cg, const double *wq,
                           int n_pix, const float *resp, const int *j0, const double *w, int n_tau, const double *scale,
                           float *W_out, long long *n_nonfinite_out, double *ms_out)
{
    if (!ctx) return EXM_ERR_ARG;
    try {
        EXM_CUDA(cudaSetDevice(ctx->dev));
        if (!(n_nodes >= 1 && n_nodes <= kWRows && n_max >= 0 && n_max <= 255 && n_psi >= 1 && n_chi >= 1 &&
              n_pix >= 1 && n_tau >= 2))
            EXM_THROW(EXM_ERR_ARG, "need 1 <= nodes <= 64, 0 <= n_max <= 255, quadrature and pixels >= 1, n_tau >= 2");
        if (!(s_nodes && c2p && s2p && ap && cg && wq && resp && j0 && w && scale && W_out))
            EXM_THROW(EXM_ERR_ARG, "null argument");
        for (int p = 0; p < n_pix; ++p)
            if (j0[p] < 0 || j0[p] > n_tau - 2) EXM_THROW(EXM_ERR_ARG, "delay bin outside the tau grid");
        const int Q = n_psi * n_chi, Qp = w_pitch(Q), nl = 2 * n_max + 1;
        const long long n_keys = (long long)(n_max + 1) * (n_max + 2) * (n_max + 3) / 6;
        std::vector<int4> tiles;
        for (int m = 0; m <= n_max; ++m) {
            const int L = n_max - m + 1;
            int x0 = 0, y0 = 0;   // the next column to be placed
            while (x0 < L) {
                const int na = std::min(kWY, L - x0 - y0);
                tiles.push_back(make_int4(m, x0, y0, na));
                if (na < kWY) x0 += kWX, y0 = kWY - na;
                else y0 += kWY;
                if (x0 + y0 >= L) x0 += kWX, y0 = 0;
            }
        }
        const size_t nW = (size_t)n_nodes * n_tau * n_keys;
        dbuf d_s, d_c2p, d_s2p, d_ap, d_cg, d_wq, d_resp, d_scale, d_W, d_out, d_tiles, d_l1, d_l2, d_dph, d_bw, d_bad;
        struct Guard {
            exm_ctx *c;
            std::vector<dbuf *> b;
            ~Guard()
            {
                for (dbuf *x : b)
                    if (x->p) exm_free(c, *x);
            }
        } guard{ctx, {&d_s, &d_c2p, &d_s2p, &d_ap, &d_cg, &d_wq, &d_resp, &d_scale, &d_W, &d_out, &d_tiles, &d_l1,
                      &d_l2, &d_dph, &d_bw, &d_bad}};
        auto up = [&](dbuf &b, const void *src, size_t bytes) {
            exm_alloc(ctx, b, bytes);
            exm_copy_in(ctx, b.p, src, bytes);
        };
        up(d_s, s_nodes, n_nodes * sizeof(double));
        up(d_c2p, c2p, n_psi * sizeof(float));
        up(d_s2p, s2p, n_psi * sizeof(float));
        up(d_ap, ap, n_chi * sizeof(float));
        up(d_cg, cg, n_chi * sizeof(float));
        up(d_wq, wq, n_chi * sizeof(double));
        up(d_resp, resp, (size_t)n_pix * 4 * sizeof(float));
        up(d_scale, scale, (size_t)n_nodes * n_keys * sizeof(double));
        up(d_tiles, tiles.data(), tiles.size() * sizeof(int4));
        exm_alloc(ctx, d_W, nW * sizeof(double));
        // the result's memory holds a pixel's cosines until the last product is done
        exm_alloc(ctx, d_out, std::max(nW * sizeof(float), (size_t)(n_max + 1) * Qp * sizeof(double)));
        exm_alloc(ctx, d_l1, (size_t)nl * Qp * sizeof(double));
        exm_alloc(ctx, d_l2, (size_t)nl * Qp * sizeof(double));
        exm_alloc(ctx, d_dph, (size_t)Qp * sizeof(double));
        exm_alloc(ctx, d_bw, (size_t)n_nodes * Qp * sizeof(double));
        exm_alloc(ctx, d_bad, sizeof(unsigned long long));
        EXM_CUDA(cudaMemsetAsync(d_W.p, 0, nW * sizeof(double), ctx->stream));
        EXM_CUDA(cudaMemsetAsync(d_bad.p, 0, sizeof(unsigned long long), ctx->stream));
        cudaEvent_t e0, e1, e2;
        EXM_CUDA(cudaEventCreate(&e0));
        EXM_CUDA(cudaEventCreate(&e1));
        EXM_CUDA(cudaEventCreate(&e2));
        EXM_CUDA(cudaEventRecord(e0, ctx->stream));
        auto gemm = [&](auto rg, auto rr, int p) {
            constexpr int RG = decltype(rg)::value, R = decltype(rr)::value;
            exm_allow_smem(ctx, (const void *)k_w_gemm<RG, R>, w_smem(RG, R));
            k_w_gemm<RG, R><<<(int)tiles.size(), kWThreads, w_smem(RG, R), ctx->stream>>>(
                (const int4 *)d_tiles.p, Qp, n_nodes, n_max, (const double *)d_l1.p, (const double *)d_l2.p,
                (const double *)d_out.p, (const double *)d_bw.p, j0[p], w[2 * p], w[2 * p + 1], n_tau, n_keys,
                (double *)d_W.p);
        };
        for (int p = 0; p < n_pix; ++p) {
            k_w_prep<<<(Qp + 127) / 128, 128, 0, ctx->stream>>>((const float *)d_resp.p + 4 * (size_t)p,
                                                                (const float *)d_c2p.p, (const float *)d_s2p.p,
                                                                (const float *)d_ap.p, (const float *)d_cg.p,
                                                                (const double *)d_wq.p, n_psi, n_chi, n_nodes,
                                                                (const double *)d_s.p, nl, Qp, (double *)d_l1.p,
                                                                (double *)d_l2.p, (double *)d_dph.p, (double *)d_bw.p);
            k_w_cos<<<dim3((Qp + 127) / 128, n_max + 1), 128, 0, ctx->stream>>>((const double *)d_dph.p, Qp,
                                                                               (double *)d_out.p);
            // the fewest rows that hold the nodes: one row group up to 8 nodes, else 5 to 8 rows in each of 2, 4 or 8
            const int rg = n_nodes <= 8 ? 1 : n_nodes <= 16 ? 2 : n_nodes <= 32 ? 4 : 8;
            auto rows = [&](auto r) {
                if (rg == 1) gemm(std::integral_constant<int, 1>(), r, p);
                if constexpr (decltype(r)::value >= 5) {
                    if (rg == 2) gemm(std::integral_constant<int, 2>(), r, p);
                    if (rg == 4) gemm(std::integral_constant<int, 4>(), r, p);
                    if (rg == 8) gemm(std::integral_constant<int, 8>(), r, p);
                }
            };
            switch ((n_nodes + rg - 1) / rg) {
                case 1: rows(std::integral_constant<int, 1>()); break;
                case 2: rows(std::integral_constant<int, 2>()); break;
                case 3: rows(std::integral_constant<int, 3>()); break;
                case 4: rows(std::integral_constant<int, 4>()); break;
                case 5: rows(std::integral_constant<int, 5>()); break;
                case 6: rows(std::integral_constant<int, 6>()); break;
                case 7: rows(std::integral_constant<int, 7>()); break;
                default: rows(std::integral_constant<int, 8>()); break;
            }
        }
        EXM_CUDA(cudaGetLastError());
        EXM_CUDA(cudaEventRecord(e1, ctx->stream));
        k_w_scale<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>((const double *)d_W.p, (const double *)d_scale.p, n_tau,
                                                              n_keys, (long long)nW, (float *)d_out.p,
                                                              (unsigned long long *)d_bad.p);
        EXM_CUDA(cudaGetLastError());
        unsigned long long bad = 0;
        exm_copy_out(ctx, W_out, d_out.p, nW * sizeof(float));
        EXM_CUDA(cudaMemcpyAsync(&bad, d_bad.p, sizeof(bad), cudaMemcpyDeviceToHost, ctx->stream));
        EXM_CUDA(cudaEventRecord(e2, ctx->stream));
        EXM_CUDA(cudaStreamSynchronize(ctx->stream));
        float k_ms = 0.f, all_ms = 0.f;
        cudaEventElapsedTime(&k_ms, e0, e1);
        cudaEventElapsedTime(&all_ms, e0, e2);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaEventDestroy(e2);
        if (n_nonfinite_out) *n_nonfinite_out = (long long)bad;
        if (ms_out) {
            ms_out[0] = k_ms;
            ms_out[1] = all_ms;
        }
        ctx->launches += 3 * n_pix + 1;
    } catch (const exm_error &e) {
        ctx->err = e.msg;
        return e.code;
    } catch (const std::bad_alloc &) {
        ctx->err = "host memory exhausted";
        return EXM_ERR_OOM;
    } catch (const std::exception &e) {
        ctx->err = e.what();
        return EXM_ERR_CUDA;
    }
    return 0;
}
