// Learned directional guide (rtpg_mlp_*): inference and training of the vMF-mixture MLP on
// the tensor cores (tcgen05), Adam, and the record buffer the tracer fills.
//
// The guide has no counterpart in RTLib; it learns the same quantity the SD-tree records per
// trace vertex (TraceVertexT::Commit, OPX7UtilsPathGuiding.h:830-866: the luminance of the
// incident radiance times |cos| over the sampling pdf, in the sampled direction) and is trained
// to minimise the weighted negative log-likelihood of those directions (the KL divergence of
// the mixture to the recorded radiance distribution).
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include "common.cuh"
#include "mlp_dev.cuh"

namespace rtpg {

// ------------------------------------------------------------------ inference
// N floats (a multiple of 4) to dst: 16-byte stores if dst is 16-byte aligned, else scalars
template <int N>
__device__ __forceinline__ void store_row(float* dst, const float* v) {
    if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
#pragma unroll
        for (int c = 0; c < N; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    } else {
#pragma unroll
        for (int c = 0; c < N; ++c) dst[c] = v[c];
    }
}

// out_raw: 48 floats per sample (the network output); out_lobes: 40 floats per sample, lobe k
// = (mu xyz, kappa, weight).  Either may be null.  Bound by the phases of the four tiles an SM holds
// (issue slots 58 % busy).  2^20 samples: 148.6 us with one thread per sample, 136.9 with two and the
// next tile's inputs fetched ahead; eight tiles per SM sharing weights, one thread per sample: 133,
// but 6 % slower at 10^5 samples.
__global__ void __launch_bounds__(kMlpThreads, 4) k_mlp_eval(MlpDev P, int64_t n, const float* __restrict__ pos,
                                                            const float* __restrict__ nrm, const float* __restrict__ wo,
                                                            float* __restrict__ out_raw, float* __restrict__ out_lobes) {
    extern __shared__ __align__(128) uint8_t sm[];
    EvalCta c = eval_begin(sm, P.wq);
    bool ok = true;
    const bool hi = threadIdx.x >= kMlpTile;
    const int64_t stride = int64_t(gridDim.x) * kMlpTile;
    int64_t i = int64_t(blockIdx.x) * kMlpTile + threadIdx.x % kMlpTile;
    float3 x = f3(0.f, 0.f, 0.f), nv = x, wv = x;
    auto fetch = [&](int64_t k) {
        if (k >= n) return;
        x = f3(pos[3 * k], pos[3 * k + 1], pos[3 * k + 2]);
        if (!hi) return;  // the upper half holds these features
        nv = f3(nrm[3 * k], nrm[3 * k + 1], nrm[3 * k + 2]);
        wv = f3(wo[3 * k], wo[3 * k + 1], wo[3 * k + 2]);
    };
    fetch(i);
    for (int64_t base = int64_t(blockIdx.x) * kMlpTile; base < n; base += stride, i += stride) {
        store_features(c.x0, i < n, x, nv, wv, P.mn, P.inv_ext);
        fetch(i + stride);  // the next tile's inputs arrive while this one is evaluated
        if (!mlp_forward_tile(P, c.d, c.sw, c.x0, c.mbar, c.phase, ok)) break;  // uniform: issue nothing more
        // half of a sample's row (192 or 160 bytes) in 16-byte stores when the array allows it; the
        // loads from tensor memory take the whole warp
        if (out_raw) {
            float q[kMlpOut / 2];
            ld_row<kMlpOut / 2>(c.d, hi ? kMlpOut / 2 : 0, q);
            if (i < n && ok) store_row<kMlpOut / 2>(out_raw + i * kMlpOut + (hi ? kMlpOut / 2 : 0), q);
        }
        if (out_lobes) {
            float o[kMlpOut];
            ld_row<kMlpOut>(c.d, 0, o);
            if (i < n && ok) {
                VmfLobe L[kMlpLobes / 2];
                mlp_head_half(o, hi, L);
                float q[20];
#pragma unroll
                for (int k = 0; k < kMlpLobes / 2; ++k) {
                    q[5 * k] = L[k].mu.x; q[5 * k + 1] = L[k].mu.y; q[5 * k + 2] = L[k].mu.z;
                    q[5 * k + 3] = L[k].kappa; q[5 * k + 4] = L[k].weight;
                }
                store_row<20>(out_lobes + i * 40 + (hi ? 20 : 0), q);
            }
        }
    }
    eval_end(c, ok, P.poll_limit, P.status);
}

// ------------------------------------------------------------------ training
// d(loss)/d(raw outputs) of one record: loss = -w log q(wi) (scaled by inv_wsum), q the mixture
// of mlp_head_half's lobes.  Each of the record's two threads forms its half of the lobes and hands their
// terms to the other through s_f (lobe-major): both add the eight terms of q in order.  The thread's
// 20 gradients go to g; returns -log q.
__device__ __forceinline__ float head_grad(const float* o, bool hi, float3 wi, float scale, float (*s_f)[kMlpTile], float* g) {
    VmfLobe L[kMlpLobes / 2];
    mlp_head_half(o, hi, L);
    const int row = threadIdx.x & (kMlpTile - 1);
    float fk[kMlpLobes / 2], q = 0.0f;
#pragma unroll
    for (int k = 0; k < kMlpLobes / 2; ++k) {
        fk[k] = vmf_pdf(L[k], wi);
        s_f[hi ? k + 4 : k][row] = __fmul_rn(L[k].weight, fk[k]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kMlpLobes; ++k) q = __fadd_rn(q, s_f[k][row]);
    q = fmaxf(q, 1e-30f);
#pragma unroll
    for (int k = 0; k < kMlpLobes / 2; ++k) {
        const float r = L[k].weight * fk[k] / q;  // responsibility
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = hi ? o[5 * (k + 4) + j] : o[5 * k + j];
        const float3 m = f3(v[0], v[1], v[2]);
        const float len = fmaxf(sqrtf(dot3(m, m)), 1e-12f);
        const float kap = L[k].kappa, mw = dot3(L[k].mu, wi);
        // d log q / d m = r kappa (wi - (mu.wi) mu) / |m|
        const float3 gm = (wi - L[k].mu * mw) * (r * kap / len);
        const float e = __expf(-2.0f * kap);
        const float dlk = 1.0f / kap - 2.0f * e / (1.0f - e) + (mw - 1.0f);
        const float gs = (v[3] > kLogKappaMin && v[3] < kLogKappaMax) ? r * kap * dlk : 0.0f;
        g[5 * k] = -scale * gm.x;
        g[5 * k + 1] = -scale * gm.y;
        g[5 * k + 2] = -scale * gm.z;
        g[5 * k + 3] = -scale * gs;
        g[5 * k + 4] = -scale * (r - L[k].weight);
    }
    return -__logf(q);
}

// Sum of the first `parts` of p, the same in every lane (fixed order).  The whole warp calls it.
__device__ __forceinline__ double warp_sum_parts(const double* p, int parts) {
    double s = 0.0;
    for (int k = threadIdx.x & 31; k < parts; k += 32) s += p[k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// One pass over n records: forward, loss gradient, backward; dW of all layers accumulate in
// TMEM across the CTA's tiles and go to the CTA's row of grad_rows (fp32, [in][out] per layer) at the
// end, its share of the loss to loss_rows; k_mlp_adam or k_mlp_add_grads sums the rows.  wsum: the
// minibatch's weight sum in wparts parts (k_wsum), in double: one unit in the last place of the float it
// becomes moves some twenty of a minibatch's output gradients to another bf16 value.  No sum depends on the order in which CTAs finish:
// Adam divides a gradient by its own size, so what the order of float atomics left in the last bits
// grew to 4e-4 of the parameters within 16 steps.
// A minibatch gives each CTA one tile, so its time is that tile's chain of phases: features, eight
// dependent MMA phases with an epilogue each, the gradient flush.  Launched as a dependent of the
// previous step's Adam it forms the first tile's features, which do not depend on the weights, while
// that still runs (records and wsum are ready before the first launch of a call).  16 steps of 16384
// records: 574 us with 128 threads per tile and a memset, a weight sum and an Adam launched one after
// the other around it, 320 us now.
__global__ void __launch_bounds__(kMlpThreads, 1) k_mlp_train(MlpDev P, int64_t n, Records R, const double* wsum, int wparts,
                                                            float* __restrict__ grad_rows, float* __restrict__ loss_rows) {
    extern __shared__ __align__(128) uint8_t sm[];
    __nv_bfloat16* ws = reinterpret_cast<__nv_bfloat16*>(sm);
    __nv_bfloat16* x0 = reinterpret_cast<__nv_bfloat16*>(sm + kSmemW);
    __nv_bfloat16* hs[3];
    for (int k = 0; k < 3; ++k) hs[k] = reinterpret_cast<__nv_bfloat16*>(sm + kSmemW + kSmemX + k * kSmemH);
    __nv_bfloat16* dy = reinterpret_cast<__nv_bfloat16*>(sm + kSmemW + kSmemX + 3 * kSmemH);
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kSmemW + kSmemX + 4 * kSmemH);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kSmemW + kSmemX + 4 * kSmemH + 8);
    __shared__ float s_f[kMlpLobes][kMlpTile];
    __shared__ float s_loss[kMlpTile / 32];
    grid_launch_dependents();
    const int t = threadIdx.x, row = t & (kMlpTile - 1);
    const bool hi = t >= kMlpTile;
    if (t < 32) tmem_alloc(tslot, kTrainCols);
    if (t == 0) mbar_init(mbar, 1);
    const uint32_t sw = smem_u32(ws), sx = smem_u32(x0), sdy = smem_u32(dy);
    const uint32_t sh[3] = {smem_u32(hs[0]), smem_u32(hs[1]), smem_u32(hs[2])};
    const float total = (float)warp_sum_parts(wsum, wparts);
    const float scale = total > 0.0f ? 1.0f / total : 0.0f;
    // record weights are Monte Carlo estimates with a heavy tail: clamp at kWeightClamp times
    // their mean so that single rare paths do not dominate a step
    const float wmax = kWeightClamp * (total / (float)n);
    uint32_t phase = 0, tmem = 0;
    bool ok = true, first = true;
    float lsum = 0.0f;
    auto commit_wait = [&] {
        if (t == 0 && !P.skip_mma) umma_commit(mbar);
        ok = mma_complete(mbar, phase, P.poll_limit);
    };
    for (int64_t base = int64_t(blockIdx.x) * kMlpTile; base < n; base += int64_t(gridDim.x) * kMlpTile) {
        const int64_t i = base + row;
        const bool live = i < n;
        float3 x = f3(0.f, 0.f, 0.f), nv = x, wv = x, wi = f3(0.f, 0.f, 1.f);
        float w = 0.0f;
        if (live) {
            x = f3(R.pos[3 * i], R.pos[3 * i + 1], R.pos[3 * i + 2]);
            nv = f3(R.nrm[3 * i], R.nrm[3 * i + 1], R.nrm[3 * i + 2]);
            wv = f3(R.wo[3 * i], R.wo[3 * i + 1], R.wo[3 * i + 2]);
            wi = f3(R.wi[3 * i], R.wi[3 * i + 1], R.wi[3 * i + 2]);
            w = fminf(fmaxf(R.w[i], 0.0f), wmax);
        }
        store_features(x0, live, x, nv, wv, P.mn, P.inv_ext);
        if (first) {
            grid_dependency_wait();  // the weights
            load_weights(ws, P.wq);
        }
        // forward, keeping H1..H3
        bool go = true;
        for (int l = 0; l < 4 && go; ++l) {
            if (!(go = mma_barrier(ok))) break;
            if (l == 0 && first) tmem = *tslot;
            if (t == 0 && !P.skip_mma) {
                if (l == 0) issue_fwd(tmem + kColD, sx, kMlpIn, kMlpIn, sw + 2 * kW0, kMlpHidden);
                else if (l < 3) issue_fwd(tmem + kColD, sh[l - 1], kMlpHidden, kMlpHidden, sw + 2 * (l == 1 ? kW1 : kW2), kMlpHidden);
                else issue_fwd(tmem + kColD, sh[2], kMlpHidden, kMlpHidden, sw + 2 * kW3, kMlpOut);
            }
            commit_wait();
            if (l < 3) epilogue_relu(tmem + kColD, hs[l]);
        }
        if (!go) break;
        // loss gradient at the outputs -> dY [128 x 64] (columns 40..63 zero)
        {
            float o[kMlpOut], g[20];
            ld_row<kMlpOut>(tmem, kColD, o);
            const float nl = head_grad(o, hi, wi, w * scale, s_f, g);
            if (w > 0.0f && !hi) lsum += w * nl;
            const int c0 = hi ? 20 : 0;
#pragma unroll
            for (int c = 0; c < 20; c += 4) {
                __nv_bfloat162 p[2] = {__floats2bfloat162_rn(g[c], g[c + 1]), __floats2bfloat162_rn(g[c + 2], g[c + 3])};
                *reinterpret_cast<uint2*>(dy + blk(row, c0 + c, kMlpHidden)) = *reinterpret_cast<const uint2*>(p);
            }
            if (hi)
#pragma unroll
                for (int c = 40; c < kMlpHidden; c += 8)
                    *reinterpret_cast<uint4*>(dy + blk(row, c, kMlpHidden)) = make_uint4(0u, 0u, 0u, 0u);
        }
        // backward: layer 3 .. 0
        for (int l = 3; l >= 0; --l) {
            if (!(go = mma_barrier(ok))) break;
            if (t == 0 && !P.skip_mma) {
                const uint32_t cw = l == 3 ? kColW3 : (l == 2 ? kColW2 : (l == 1 ? kColW1 : kColW0));
                if (l > 0) {
                    const uint32_t wl = l == 3 ? kW3 : (l == 2 ? kW2 : kW1);
                    issue_dx(tmem + kColD, sdy, l == 3 ? kMlpOut : kMlpHidden, sw + 2 * wl, kMlpHidden);
                    issue_dw(tmem + cw, sdy, sh[l - 1], kMlpHidden, kMlpHidden, !first);
                } else {
                    issue_dw(tmem + cw, sdy, sx, kMlpIn, kMlpIn, !first);
                }
            }
            commit_wait();
            if (l > 0) {
                // dH = dX masked by ReLU' of the activation it came from, back into dY
                const __nv_bfloat16* hl = hs[l - 1];
                const int c0 = hi ? 32 : 0;
                float v[32];
                ld_row<32>(tmem, kColD + c0, v);
#pragma unroll
                for (int c = 0; c < 32; c += 8) {
                    // the activation's 8 bf16 of this chunk in one 16-byte load
                    const uint4 hv = *reinterpret_cast<const uint4*>(hl + blk(row, c0 + c, kMlpHidden));
                    const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&hv);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (!(__bfloat162float(hb[k]) > 0.0f)) v[c + k] = 0.0f;
                    st_bf16x8(dy + blk(row, c0 + c, kMlpHidden), v + c);
                }
            }
        }
        if (!go) break;
        first = false;
    }
    // flush dW^T (M = 64 rows in lanes 16w .. 16w+15 of warp w's quarter, the two warps of a quarter
    // taking alternate column groups) into the CTA's row; after a wait gave up the accumulators are
    // incomplete and the row is zero
    const bool done = mma_barrier(ok);
    float* const grads = grad_rows + size_t(blockIdx.x) * kMlpParams;
    if (!done) {
        for (int i = t; i < kMlpParams; i += kMlpThreads) grads[i] = 0.0f;
    } else {
        const int warp = t >> 5, lane = t & 31;
        const int out = 16 * (warp & 3) + lane;  // output feature
        const uint32_t cols[4] = {kColW0, kColW1, kColW2, kColW3};
        const int nin[4] = {kMlpIn, kMlpHidden, kMlpHidden, kMlpHidden};
        const int nout[4] = {kMlpHidden, kMlpHidden, kMlpHidden, kMlpOut};
        const int off[4] = {kW0, kW1, kW2, kW3};
        for (int l = 0; l < 4; ++l) {
            for (int c = hi ? 16 : 0; c < nin[l]; c += 32) {
                float v[16];
                ld_row<16>(tmem, cols[l] + c, v);
                if (lane < 16 && out < nout[l])
                    for (int k = 0; k < 16; ++k) grads[off[l] + (c + k) * nout[l] + out] = v[k];
            }
        }
    }
    // loss
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if ((t & 31) == 0 && !hi) s_loss[t >> 5] = lsum * scale;
    if (!done) {
        if (t == 0) atomicOr(P.status, RTPG_STATUS_TIMEOUT);
        mma_drain(mbar, phase, P.poll_limit);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (t == 0) loss_rows[blockIdx.x] = s_loss[0] + s_loss[1] + s_loss[2] + s_loss[3];
    if (t < 32) tmem_dealloc(*tslot, kTrainCols);
}

// Sums of the nonnegative weights of gridDim.y minibatches of `batch` records (the last shorter), each
// in gridDim.x parts, kWsumParts apart.
constexpr int kWsumParts = 64, kWsumBlock = 256;
__global__ void __launch_bounds__(kWsumBlock) k_wsum(int64_t n, int64_t batch, const float* w, double* out) {
    __shared__ double s_w[kWsumBlock / 32];
    const int64_t b0 = blockIdx.y * batch, m = min(batch, n - b0);
    double s = 0.0;
    for (int64_t i = blockIdx.x * int64_t(kWsumBlock) + threadIdx.x; i < m; i += int64_t(gridDim.x) * kWsumBlock)
        s += (double)fmaxf(w[b0 + i], 0.0f);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = warp_sum_parts(s_w, kWsumBlock / 32);
        if (threadIdx.x == 0) out[blockIdx.y * kWsumParts + blockIdx.x] = s;
    }
}
static int wsum_parts(int64_t batch) { return (int)std::min<int64_t>(kWsumParts, (batch + 1023) / 1024); }

// fp32 master [in][out] -> bf16 core-matrix layout of each matrix
__device__ __forceinline__ uint32_t packed_index(int i) {
    const int l = i < kW1 ? 0 : (i < kW2 ? 1 : (i < kW3 ? 2 : 3));
    const int off = l == 0 ? kW0 : (l == 1 ? kW1 : (l == 2 ? kW2 : kW3));
    const int nout = l == 3 ? kMlpOut : kMlpHidden;
    const int r = (i - off) / nout, c = (i - off) % nout;
    return off + blk(r, c, nout);
}
__global__ void k_mlp_pack(const float* w, __nv_bfloat16* wq) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x)
        wq[packed_index(i)] = __float2bfloat16_rn(w[i]);
}
// What the CTAs of one k_mlp_train left: its gradient rows and shares of the loss.
struct GradRows {
    const float *grads, *loss;
    int count;
};
// Launches of kGradCtas CTAs of 256 threads: the first kMlpParams / 32 have a parameter per lane, whose
// rows their eight warps sum side by side, the last sums the loss.  Sums in double, in a fixed order.
// 16 steps of 16384 records (128 rows, 8.4 MB a step that stay in the L2): 319 us, 317 with float
// atomics into one accumulator (303 and 293 from a flushed L2).
constexpr int kGradCtas = kMlpParams / 32 + 1, kGradWarps = 8;
// The sum over all rows of parameter i = blockIdx.x * 32 + lane, in warp 0 (false elsewhere and in
// the CTA of the loss).  All threads call it.
__device__ __forceinline__ bool sum_rows(const GradRows& r, float* __restrict__ loss, int& i, float& sum) {
    __shared__ double s_part[kGradWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == kMlpParams / 32) {
        if (warp) return false;
        double s = 0.0;
        for (int k = lane; k < r.count; k += 32) s += (double)r.loss[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) *loss = (float)s;
        return false;
    }
    i = blockIdx.x * 32 + lane;
    double s = 0.0;
#pragma unroll 8
    for (int k = warp; k < r.count; k += kGradWarps) s += (double)r.grads[size_t(k) * kMlpParams + i];
    s_part[warp][lane] = s;
    __syncthreads();
    if (warp) return false;
    for (int k = 1; k < kGradWarps; ++k) s += s_part[k][lane];
    sum = (float)s;
    return true;
}
// gradients of one pass added to g
__global__ void __launch_bounds__(32 * kGradWarps) k_mlp_add_grads(GradRows r, float* g, float* loss) {
    int i;
    float s;
    if (sum_rows(r, loss, i, s)) g[i] += s;
}
// Adam (Kingma & Ba 2015) with bias correction; g (gradients added before) zeroed after use
__global__ void __launch_bounds__(32 * kGradWarps) k_mlp_adam(GradRows r, float* loss, float* w, float* g, float* m, float* v,
                                                              __nv_bfloat16* wq, float lr, float b1, float b2, float eps,
                                                              float c1, float c2) {
    grid_launch_dependents();
    grid_dependency_wait();
    int i;
    float s;
    if (!sum_rows(r, loss, i, s)) return;
    const float gi = g[i] + s;
    const float mi = __fmaf_rn(1.0f - b1, gi, __fmul_rn(b1, m[i]));
    const float vi = __fmaf_rn(__fmul_rn(1.0f - b2, gi), gi, __fmul_rn(b2, v[i]));
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    g[i] = 0.0f;
    wq[packed_index(i)] = __float2bfloat16_rn(wi);
}

}  // namespace rtpg

using namespace rtpg;

constexpr int64_t kMlpGroup = 256;  // minibatches whose weights are summed in one launch
// scratch of training: weight sums of a group of minibatches in parts (double), a CTA's share of the loss and
// gradient row each for a launch of k_mlp_train (float; 9.9 MB in all, in doubles)
constexpr size_t kLossRows = kMlpGroup * kWsumParts, kGradRowsAt = kLossRows + 128,
                 kTrainScratch = kGradRowsAt + size_t(kSMs) * kMlpParams / 2;
static_assert(kSMs <= 256, "loss shares");

struct rtpg_mlp {
    MlpDev dev{};
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    float* loss = nullptr;      // of the newest step, behind the gradients
    double* scratch = nullptr;  // kTrainScratch (scratch_alloc)
    int device = 0;             // of scratch
    __nv_bfloat16* wq = nullptr;
    float lr = 1e-3f, b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    uint32_t step = 0;
    float mn[3], mx[3];
    // record buffer (filled by the tracer or rtpg_mlp_add_records)
    uint32_t capacity = 0;
    float *r_pos = nullptr, *r_nrm = nullptr, *r_wo = nullptr, *r_wi = nullptr, *r_w = nullptr, *r_pdf = nullptr;
    uint32_t* r_count = nullptr;
    unsigned* status = nullptr;
    std::vector<void*> allocs;
    template <class T>
    int alloc(T** p, size_t count) {
        void* q = nullptr;
        cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(RTPG_ENOMEM, "cudaMalloc(%zu bytes) failed: %s", count * sizeof(T), cudaGetErrorString(e));
        }
        allocs.push_back(q);
        *p = static_cast<T*>(q);
        return RTPG_OK;
    }
    ~rtpg_mlp() {
        for (void* p : allocs) cudaFree(p);
        if (scratch) {
            int cur = device;
            cudaGetDevice(&cur);
            if (cur != device) cudaSetDevice(device);
            cudaDeviceSynchronize();  // memory of a pool is freed without waiting for its last use
            cudaFree(scratch);
            if (cur != device) cudaSetDevice(cur);
        }
    }
};

// Training scratch comes from a pool of its own on each device: mapping and unmapping 9.9 MB by cudaMalloc
// and cudaFree costs 0.7 ms a guide, as much as all else in creating it.  The pool keeps at most
// kScratchKept bytes that no guide uses.
constexpr uint64_t kScratchKept = 32u << 20;
static int scratch_alloc(rtpg_mlp* h) {
    static std::mutex mu;
    static std::map<int, cudaMemPool_t> pools;
    int dev = 0;
    RTPG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    cudaMemPool_t& pool = pools[dev];
    if (!pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        uint64_t kept = kScratchKept;
        RTPG_CUDA(cudaMemPoolCreate(&pool, &props));
        RTPG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept));
    }
    h->device = dev;
    const cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&h->scratch), sizeof(double) * kTrainScratch, pool, nullptr);
    if (e != cudaSuccess) {
        cudaGetLastError();
        h->scratch = nullptr;
        return fail(RTPG_ENOMEM, "rtpg_mlp_create: %zu bytes of training scratch: %s", sizeof(double) * kTrainScratch,
                    cudaGetErrorString(e));
    }
    return RTPG_OK;
}

namespace rtpg {
MlpView mlp_view(const rtpg_mlp* h) {
    return MlpView{h->dev, h->r_pos, h->r_nrm, h->r_wo, h->r_wi, h->r_w, h->r_pdf, h->r_count, h->capacity};
}
size_t mlp_eval_smem() { return kSmemEval; }
}

static uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

static bool g_mlp_attr = false;
static int mlp_set_attrs() {
    if (g_mlp_attr) return RTPG_OK;
    RTPG_CUDA(cudaFuncSetAttribute(k_mlp_eval, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemEval));
    RTPG_CUDA(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemTrain));
    g_mlp_attr = true;
    return RTPG_OK;
}

extern "C" {

int rtpg_mlp_create(const float* aabb_min, const float* aabb_max, uint32_t seed, float learning_rate,
                    uint32_t record_capacity, rtpg_mlp** out) {
    if (!aabb_min || !aabb_max || !out) return fail(RTPG_EINVAL, "rtpg_mlp_create: null argument");
    for (int k = 0; k < 3; ++k)
        if (!(aabb_max[k] > aabb_min[k])) return fail(RTPG_EINVAL, "rtpg_mlp_create: empty AABB");
    int r = mlp_set_attrs();
    if (r) return r;
    auto* h = new (std::nothrow) rtpg_mlp();
    if (!h) return fail(RTPG_ENOMEM, "rtpg_mlp_create: out of host memory");
    h->lr = learning_rate > 0.0f ? learning_rate : 1e-3f;
    h->capacity = record_capacity;
    const size_t C = std::max<uint32_t>(record_capacity, 1);
    if ((r = h->alloc(&h->w, kMlpParams)) || (r = h->alloc(&h->g, kMlpParams + 1)) || (r = h->alloc(&h->m, kMlpParams)) ||
        (r = h->alloc(&h->v, kMlpParams)) || (r = h->alloc(&h->wq, kMlpParams)) || (r = scratch_alloc(h)) ||
        (r = h->alloc(&h->r_pos, 3 * C)) || (r = h->alloc(&h->r_nrm, 3 * C)) || (r = h->alloc(&h->r_wo, 3 * C)) ||
        (r = h->alloc(&h->r_wi, 3 * C)) || (r = h->alloc(&h->r_w, C)) || (r = h->alloc(&h->r_pdf, C)) ||
        (r = h->alloc(&h->r_count, 1)) ||
        (r = h->alloc(&h->status, 1))) {
        delete h;
        return r;
    }
    h->loss = h->g + kMlpParams;
    for (int k = 0; k < 3; ++k) {
        h->mn[k] = aabb_min[k];
        h->mx[k] = aabb_max[k];
    }
    h->dev.mn = make_float3(aabb_min[0], aabb_min[1], aabb_min[2]);
    h->dev.inv_ext = make_float3(1.0f / (aabb_max[0] - aabb_min[0]), 1.0f / (aabb_max[1] - aabb_min[1]),
                                 1.0f / (aabb_max[2] - aabb_min[2]));
    h->dev.wq = h->wq;
    h->dev.status = h->status;
    h->dev.skip_mma = 0;
    h->dev.poll_limit = kMbarPollLimit;
    // He-uniform initialisation from a seeded SplitMix64 stream; output padding columns zero
    std::vector<float> w(kMlpParams, 0.0f);
    uint64_t s = 0x5DEECE66Dull ^ (uint64_t(seed) << 17);
    const int nin[4] = {kMlpIn, kMlpHidden, kMlpHidden, kMlpHidden};
    const int nout[4] = {kMlpHidden, kMlpHidden, kMlpHidden, kMlpOut};
    const int off[4] = {kW0, kW1, kW2, kW3};
    for (int l = 0; l < 4; ++l) {
        const float bound = std::sqrt(6.0f / (float)(l == 0 ? 79 : nin[l])) * (l == 3 ? 0.5f : 1.0f);
        for (int i = 0; i < nin[l]; ++i)
            for (int o = 0; o < nout[l]; ++o) {
                const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
                float val = (float)((2.0 * u - 1.0) * bound);
                if ((l == 0 && i >= 79) || (l == 3 && o >= 40)) val = 0.0f;
                w[off[l] + i * nout[l] + o] = val;
            }
    }
    cudaError_t e;
    if ((e = cudaMemcpy(h->w, w.data(), sizeof(float) * kMlpParams, cudaMemcpyHostToDevice)) ||
        (e = cudaMemset(h->g, 0, sizeof(float) * (kMlpParams + 1))) || (e = cudaMemset(h->m, 0, sizeof(float) * kMlpParams)) ||
        (e = cudaMemset(h->v, 0, sizeof(float) * kMlpParams)) || (e = cudaMemset(h->r_count, 0, 4)) ||
        (e = cudaMemset(h->status, 0, 4))) {
        delete h;
        return fail(RTPG_ECUDA, "rtpg_mlp_create: %s", cudaGetErrorString(e));
    }
    k_mlp_pack<<<64, 256>>>(h->w, h->wq);
    if ((e = cudaDeviceSynchronize())) {
        delete h;
        return fail(RTPG_ECUDA, "rtpg_mlp_create: %s", cudaGetErrorString(e));
    }
    *out = h;
    return RTPG_OK;
}

int rtpg_mlp_destroy(rtpg_mlp* h) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mlp_destroy: null handle");
    delete h;
    return RTPG_OK;
}

// Copy the fp32 parameters ([in][out] per layer, 16384 floats) out or in (in: also resets Adam).
int rtpg_mlp_params(rtpg_mlp* h, float* host_get, const float* host_set, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mlp_params: null handle");
    cudaStream_t st = as_stream(stream);
    if (host_set) {
        RTPG_CUDA(cudaMemcpyAsync(h->w, host_set, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, st));
        RTPG_CUDA(cudaMemsetAsync(h->m, 0, sizeof(float) * kMlpParams, st));
        RTPG_CUDA(cudaMemsetAsync(h->v, 0, sizeof(float) * kMlpParams, st));
        RTPG_CUDA(cudaMemsetAsync(h->g, 0, sizeof(float) * kMlpParams, st));
        k_mlp_pack<<<64, 256, 0, st>>>(h->w, h->wq);
        RTPG_LAUNCH_CHECK();
        h->step = 0;
    }
    if (host_get) {
        RTPG_CUDA(cudaMemcpyAsync(host_get, h->w, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, st));
        RTPG_CUDA(cudaStreamSynchronize(st));
    }
    return RTPG_OK;
}

// Network evaluation of n samples (device arrays, 3 floats each): raw outputs (48 per sample)
// and / or the mixture (8 lobes x mu xyz, kappa, weight).
int rtpg_mlp_eval(rtpg_mlp* h, int64_t n, const float* pos, const float* nrm, const float* wo, float* out_raw,
                  float* out_lobes, void* stream) {
    if (!h || n < 0 || (n > 0 && (!pos || !nrm || !wo))) return fail(RTPG_EINVAL, "rtpg_mlp_eval: bad arguments");
    if (n == 0) return RTPG_OK;
    const int g = (int)std::min<int64_t>((n + kMlpTile - 1) / kMlpTile, kSMs * 4);
    k_mlp_eval<<<g, kMlpThreads, kSmemEval, as_stream(stream)>>>(h->dev, n, pos, nrm, wo, out_raw, out_lobes);
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

// weight sums of up to kMlpGroup minibatches of `batch` records (n records in all)
static int mlp_group(rtpg_mlp* h, int64_t n, int64_t batch, const float* w, cudaStream_t st) {
    const int64_t nb = (n + batch - 1) / batch;
    k_wsum<<<dim3((unsigned)wsum_parts(batch), (unsigned)nb), kWsumBlock, 0, st>>>(n, batch, w, h->scratch);
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}
// gradient over the n records of minibatch k of the group, left in rows; chained: a dependent of the
// previous step's Adam, before which records and weight sums were complete
static int mlp_grad(rtpg_mlp* h, int64_t k, int64_t n, int64_t batch, const Records& R, bool chained, GradRows& rows,
                    cudaStream_t st) {
    const int g = (int)std::min<int64_t>((n + kMlpTile - 1) / kMlpTile, kSMs);
    const double* const wsum = h->scratch + k * kWsumParts;
    float *const grads = reinterpret_cast<float*>(h->scratch + kGradRowsAt), *const loss = reinterpret_cast<float*>(h->scratch + kLossRows);
    if (chained) {
        RTPG_CUDA(launch_dependent(k_mlp_train, g, kMlpThreads, kSmemTrain, st, h->dev, n, R, wsum, wsum_parts(batch), grads, loss));
    } else {
        k_mlp_train<<<g, kMlpThreads, kSmemTrain, st>>>(h->dev, n, R, wsum, wsum_parts(batch), grads, loss);
        RTPG_LAUNCH_CHECK();
    }
    rows = GradRows{grads, loss, g};
    return RTPG_OK;
}

// Gradient of the loss over n records (device arrays) ADDED to the device buffer `grads` (16384
// floats, NULL: the handle's own accumulator); returns the loss through host_loss (NULL: none).
// The loss is -sum w log q(wi) / sum w.
int rtpg_mlp_loss_grad(rtpg_mlp* h, int64_t n, const float* pos, const float* nrm, const float* wo, const float* wi,
                       const float* w, float* grads, float* host_loss, void* stream) {
    if (!h || n <= 0 || !pos || !nrm || !wo || !wi || !w) return fail(RTPG_EINVAL, "rtpg_mlp_loss_grad: bad arguments");
    cudaStream_t st = as_stream(stream);
    GradRows rows;
    int r = mlp_group(h, n, n, w, st);
    if (r || (r = mlp_grad(h, 0, n, n, Records{pos, nrm, wo, wi, w}, false, rows, st))) return r;
    k_mlp_add_grads<<<kGradCtas, 32 * kGradWarps, 0, st>>>(rows, grads ? grads : h->g, h->loss);
    RTPG_LAUNCH_CHECK();
    if (host_loss) {
        RTPG_CUDA(cudaMemcpyAsync(host_loss, h->loss, 4, cudaMemcpyDeviceToHost, st));
        RTPG_CUDA(cudaStreamSynchronize(st));
    }
    return RTPG_OK;
}

// Adam steps over the record buffer (or the given records): the records are split into
// `batch`-sized minibatches, one gradient + Adam update each, `epochs` times.
int rtpg_mlp_train(rtpg_mlp* h, int64_t n, const float* pos, const float* nrm, const float* wo, const float* wi,
                   const float* w, uint32_t batch, uint32_t epochs, float* host_last_loss, void* stream) {
    if (!h || batch == 0) return fail(RTPG_EINVAL, "rtpg_mlp_train: bad arguments");
    cudaStream_t st = as_stream(stream);
    if (!pos) {
        uint32_t c = 0;
        RTPG_CUDA(cudaMemcpyAsync(&c, h->r_count, 4, cudaMemcpyDeviceToHost, st));
        RTPG_CUDA(cudaStreamSynchronize(st));
        n = std::min<uint32_t>(c, h->capacity);
        pos = h->r_pos; nrm = h->r_nrm; wo = h->r_wo; wi = h->r_wi; w = h->r_w;
    } else if (!nrm || !wo || !wi || !w) {
        return fail(RTPG_EINVAL, "rtpg_mlp_train: record arrays missing");
    }
    for (uint32_t e = 0; e < epochs; ++e)
        for (int64_t g0 = 0; g0 < n; g0 += kMlpGroup * batch) {
            const int64_t in_group = std::min<int64_t>(kMlpGroup * batch, n - g0);
            int r = mlp_group(h, in_group, batch, w + g0, st);
            if (r) return r;
            for (int64_t b = 0; b < in_group; b += batch) {
                const int64_t at = g0 + b;
                GradRows rows;
                r = mlp_grad(h, b / batch, std::min<int64_t>(batch, in_group - b), batch,
                             Records{pos + 3 * at, nrm + 3 * at, wo + 3 * at, wi + 3 * at, w + at}, b > 0, rows, st);
                if (r) return r;
                ++h->step;
                const float c1 = 1.0f - std::pow(h->b1, (float)h->step), c2 = 1.0f - std::pow(h->b2, (float)h->step);
                RTPG_CUDA(launch_dependent(k_mlp_adam, kGradCtas, 32 * kGradWarps, 0, st, rows, h->loss, h->w, h->g, h->m, h->v, h->wq, h->lr, h->b1, h->b2,
                                           h->eps, c1, c2));
            }
        }
    if (host_last_loss) {
        RTPG_CUDA(cudaMemcpyAsync(host_last_loss, h->loss, 4, cudaMemcpyDeviceToHost, st));
        RTPG_CUDA(cudaStreamSynchronize(st));
    }
    return RTPG_OK;
}

// Record buffer: count (device, may exceed capacity: records beyond it were dropped), clear.
int rtpg_mlp_records(rtpg_mlp* h, uint32_t* host_count, int clear, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mlp_records: null handle");
    cudaStream_t st = as_stream(stream);
    if (host_count) {
        RTPG_CUDA(cudaMemcpyAsync(host_count, h->r_count, 4, cudaMemcpyDeviceToHost, st));
        RTPG_CUDA(cudaStreamSynchronize(st));
    }
    if (clear) RTPG_CUDA(cudaMemsetAsync(h->r_count, 0, 4, st));
    return RTPG_OK;
}

// Device pointers of the record arrays (pos, nrm, wo, wi: 3 floats per record; w: 1).
int rtpg_mlp_record_arrays(rtpg_mlp* h, float** pos, float** nrm, float** wo, float** wi, float** w) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mlp_record_arrays: null handle");
    if (pos) *pos = h->r_pos;
    if (nrm) *nrm = h->r_nrm;
    if (wo) *wo = h->r_wo;
    if (wi) *wi = h->r_wi;
    if (w) *w = h->r_w;
    return RTPG_OK;
}

// Test mode of the bounded tensor-core waits: with skip_mma = 1 the kernels of this guide
// issue neither MMAs nor commits, so each completion wait runs out after poll_limit polls,
// sets RTPG_STATUS_TIMEOUT and the kernel returns with nothing in flight.  skip_mma = 0 and
// poll_limit = 0 restore normal operation.
int rtpg_mlp_set_wait_test(rtpg_mlp* h, int skip_mma, uint32_t poll_limit) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mlp_set_wait_test: null handle");
    h->dev.skip_mma = skip_mma ? 1u : 0u;
    h->dev.poll_limit = poll_limit ? poll_limit : kMbarPollLimit;
    return RTPG_OK;
}

// Device pointer of the records' sampling densities (1 float per record): the woPdf with which
// the tracer sampled the record's direction, so that a record's integrand value is w * pdf.
int rtpg_mlp_record_pdfs(rtpg_mlp* h, float** wo_pdf) {
    if (!h || !wo_pdf) return fail(RTPG_EINVAL, "rtpg_mlp_record_pdfs: null argument");
    *wo_pdf = h->r_pdf;
    return RTPG_OK;
}

int rtpg_mlp_status(rtpg_mlp* h, uint32_t* host_status, int clear, void* stream) {
    if (!h || !host_status) return fail(RTPG_EINVAL, "rtpg_mlp_status: null argument");
    cudaStream_t st = as_stream(stream);
    RTPG_CUDA(cudaMemcpyAsync(host_status, h->status, 4, cudaMemcpyDeviceToHost, st));
    if (clear) RTPG_CUDA(cudaMemsetAsync(h->status, 0, 4, st));
    RTPG_CUDA(cudaStreamSynchronize(st));
    return RTPG_OK;
}

}  // extern "C"
