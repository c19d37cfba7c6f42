// conv_tc.cu — the learned proposer's 3x3 convolutions on the 5th-generation tensor
// cores: tcgen05.mma kind::tf32 (operands rounded to TF32, 10 mantissa bits, to nearest
// with ties away from zero, as they are staged in shared memory; FP32 accumulation in
// TMEM).  Activations keep the layout of learn.cu: [b][c][h][t] FP32, t = 128 angles
// (circular), h = radius (zero-padded).
//
// k_conv3_tc — forward, and data gradient with the flipped weights:
//   out[b][co][h][t] = bias[co] + sum_{ci,dh,dt} W[co][ci][dh][dt] in[b][ci][h+dh-1][t+dt-1].
//   Per output row (b, h) one product D[t][(dt, co)] = sum_{dh, ci} X_{h+dh-1}[t][ci] Wd[(dt, co)][ci]
//   (M = 128 angles, N = 3 Cout, K = 3 blocks of Cin rounded up to 8, 16 or 32), and the angle
//   offset of the kernel's three columns is applied to the product's rows afterwards:
//   out[t][co] = D[t-1][(0, co)] + D[t][(1, co)] + D[t+1][(2, co)] (lane shuffles across
//   the 128 TMEM lanes).  Two output rows a step; each input row is staged once, unshifted,
//   and serves three output rows from a ring of four.  What is elementwise around the
//   convolution happens on its registers: the average of radius pairs and the ReLU's gate
//   bits on the way out, the gradient through both on the way in (see the modes below).
// k_conv3_wgrad_tc — weight and bias gradients:
//   dW[co][ci][dh][dt] = sum_{b,h,s} dpre[b][co][h][s-dt+1] in[b][ci][h+dh-1][s].
//   Per (b, h): D[(dt, co)][(x, ci)] += sum_s Pd[(dt, co)][s] X_x[ci][s] over the input rows
//   x = h-1, h, h+1 at once (K = 128 angles), accumulated in TMEM over all rows of the
//   block; the angle offset is applied while dpre is staged.  Partial sums go to the
//   scratch, one set per block, and k_wgrad_sum adds them in a fixed order.
// k_wgrad_first — the weight gradient of one input channel, whose nine sums per output channel
//   are no contraction: FP32 FMA on the same TF32-rounded operands.
//
// Operands use the K-major 128-byte-swizzled layout (tc.cuh).  Waits are bounded (1 s); a
// timeout sets *err, every thread of the block leaves together, the outstanding MMAs are
// waited for (bounded) and TMEM is freed.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "launch.h"
#include "tc.cuh"

namespace cryoim {
namespace {

constexpr int CT_NT = 128;               // angles = product rows
constexpr unsigned long long CT_WAIT_NS = 1000000000ull;
constexpr int CT_ROW_BYTES = CT_NT * 128;  // one staged input row: 128 angles x 32 channels x 4 B

__device__ __forceinline__ float tf32r(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// instruction descriptor of kind::tf32: D = F32 (bits 4-5 = 1), A and B = TF32 (2 at bits
// 7-9 and 10-12), both K-major, N >> 3 at bits 17-22, M = 128 (M >> 4 at bits 24-28)
__host__ __device__ constexpr uint32_t idesc_tf32(int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

template <int COLS> __device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::su32(slot)), "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int COLS> __device__ __forceinline__ void tmem_free(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}
// C (4 or 8) columns each at three TMEM addresses of this warp's 32 lanes
template <int C> __device__ __forceinline__ void tmem_ld3(uint32_t t0, uint32_t t1, uint32_t t2, float (&v)[3][C]) {
    static_assert(C == 4 || C == 8, "columns");
    if constexpr (C == 8)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=f"(v[0][0]), "=f"(v[0][1]), "=f"(v[0][2]), "=f"(v[0][3]), "=f"(v[0][4]), "=f"(v[0][5]),
              "=f"(v[0][6]), "=f"(v[0][7]), "=f"(v[1][0]), "=f"(v[1][1]), "=f"(v[1][2]), "=f"(v[1][3]),
              "=f"(v[1][4]), "=f"(v[1][5]), "=f"(v[1][6]), "=f"(v[1][7]), "=f"(v[2][0]), "=f"(v[2][1]),
              "=f"(v[2][2]), "=f"(v[2][3]), "=f"(v[2][4]), "=f"(v[2][5]), "=f"(v[2][6]), "=f"(v[2][7])
            : "r"(t0), "r"(t1), "r"(t2)
            : "memory");
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%12];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%13];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%14];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=f"(v[0][0]), "=f"(v[0][1]), "=f"(v[0][2]), "=f"(v[0][3]), "=f"(v[1][0]), "=f"(v[1][1]),
              "=f"(v[1][2]), "=f"(v[1][3]), "=f"(v[2][0]), "=f"(v[2][1]), "=f"(v[2][2]), "=f"(v[2][3])
            : "r"(t0), "r"(t1), "r"(t2)
            : "memory");
}

// What a convolution does to its operands on the way.
//   CONV_PLAIN  out = conv(in) (+ bias, ReLU) and, with gate_out (Cout = 16), the gate below
//   CONV_POOL   forward: out[b][co][h/2][t] = average of the ReLU outputs of rows h, h + 1, and,
//               with gate_out, where the ReLU's output is positive
//   CONV_BACK   data gradient: the input row h is 0.5 in[b][ci][h/2][t] where gate_in has channel
//               ci of (b, h, t), else 0 (in: the gradient of the pooled rows), W is the
//               forward's (its flip is read in place), and with gate_res (Cout = 16) the
//               result is kept only where gate_res has its channel
// A gate is 4 bytes for each (b, h, t), byte g for the g-th quarter of the channels, lowest first.
enum { CONV_PLAIN, CONV_POOL, CONV_BACK };

struct ConvTcArgs {
    const float* in;    // [B][Cin][H][128]; CONV_BACK [B][Cin][H / 2][128]
    const float* W;     // [Cout][Cin][3][3]; CONV_BACK [Cin][Cout][3][3]
    const float* bias;  // [Cout] or null
    float* out;         // [B][Cout][H][128]; CONV_POOL [B][Cout][H / 2][128]
    const unsigned char *gate_in, *gate_res;
    unsigned char* gate_out;
    int B, Cin, H, relu, steps_per_cta;
    int* err;
};

// 16 warps that move data and one that issues the MMAs.  Warps w, w + 4, w + 8, w + 12 share
// TMEM lanes 32 (w & 3) .. + 31 (angle t); group w >> 2 stages a quarter of the input channels
// of its angles and writes a quarter of the output channels.
constexpr int CT_ROW_THREADS = 512, CT_THREADS = CT_ROW_THREADS + 32;

template <int COUT>
constexpr int conv_fwd_smem() {
    return 1024 + 4 * CT_ROW_BYTES + 3 * (3 * COUT * 128) + 2 * 2 * 8 * COUT * 4 + COUT * 4 + 64;
}

// Forward and data gradient, two output rows (2j, 2j + 1) a step.  Stage i of a sample is the
// input rows 2i - 1 and 2i (zeros outside the sample) in one of two pairs of ring slots; step j
// reads stages j and j + 1.  While step k is written out of TMEM, the MMAs of step k + 1 fill the
// other accumulator and the loads of step k + 2's rows are in flight, over the end of a sample
// too; one barrier a step.  The warp that issues does nothing else, so no data waits for it.
// Bound: the chain of a step in one block (at 32 channels 3.1 us for two rows, of which waiting
// for the MMAs, edges and barrier 0.6, staging 0.7, loads 0.2, epilogue 1.0, MMAs in the way of
// the staging 0.5), not bandwidth: 0.2 of it.  Two blocks an SM of 8 warps with one accumulator
// took 159, 110 and 64 us at layers 2 to 4.
// The form before it (one row a step, every warp waiting for its MMAs, guards and branches per
// channel, rows written in full and pooled by a pass of its own) took, for a batch of 256
// samples, 184, 274, 149 and 85 us at layers 1 to 4 and 102 us of pooling; this one takes 89, 142, 94
// and 53 us.  Data gradients of layers 4 to 2: 82, 141 and 191 us and 205 us for the gates and
// the pooling; now 55, 95 and 174 us.
template <int CINP, int COUT, int MODE>
__global__ void __launch_bounds__(CT_THREADS, 1) k_conv3_tc(ConvTcArgs a) {
    constexpr int N = 3 * COUT;                     // product columns (dt, co)
    constexpr int WB = N * 128;                     // one dh block of the weight operand
    constexpr int CH = COUT / 4;                    // output channels of a group
    constexpr int CN = CINP / 4 < 4 ? 4 : CINP / 4;  // staged channels of a group
    constexpr int TM = COUT == 32 ? 512 : 256;      // TMEM columns: two steps of two rows of N
    extern __shared__ unsigned char smraw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    unsigned char* sX = sm;                      // ring of 4 staged input rows
    unsigned char* sWt = sm + 4 * CT_ROW_BYTES;  // 3 dh blocks of N rows
    float* sEdge = (float*)(sWt + 3 * WB);       // [2 steps][2 rows][2][4 lane quarters][COUT]
    float* sBias = sEdge + 2 * 2 * 8 * COUT;
    uint64_t* bar = (uint64_t*)(sBias + COUT);  // MMAs of even steps, of odd steps
    uint32_t* tslot = (uint32_t*)(bar + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quarter = warp & 3, grp = warp >> 2;
    const bool mover = warp < CT_ROW_THREADS / 32;
    const int t = 32 * quarter + lane;  // the angle (product row, TMEM lane) of this thread
    const int Cin = a.Cin, H = a.H, S = (H + 1) / 2;
    const int s0 = blockIdx.x * a.steps_per_cta;
    const int cnt = min(a.B * S - s0, a.steps_per_cta);
    if (cnt <= 0) return;  // uniform over the block

    if (tid == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<TM>(tslot);
    // weights: block dh, row n = dt * COUT + co, element ci (zero beyond Cin)
    for (int i = tid; i < 3 * N * CINP; i += CT_THREADS) {
        const int dh = i / (N * CINP), rem = i - dh * N * CINP, n = rem / CINP, ci = rem % CINP;
        const int dt = n / COUT, co = n - dt * COUT;
        float v = 0.f;
        if (ci < Cin)
            v = tf32r(__ldg(a.W + (MODE == CONV_BACK ? ((ci * COUT + co) * 3 + 2 - dh) * 3 + 2 - dt
                                                     : ((co * Cin + ci) * 3 + dh) * 3 + dt)));
        *(float*)(sWt + dh * WB + tc::swz128_off4(n, ci)) = v;
    }
    if (tid < COUT) sBias[tid] = a.bias ? __ldg(a.bias + tid) : 0.f;

    // The rows a step adds: rows 2j + 1 and 2j + 2 of sample b (pre[0], pre[1]) and, with the
    // first step of a sample, row 0 (row0).  CONV_BACK: pre[0] is the pooled row j, which rows
    // 2j and 2j + 1 come from, pre[1] the pooled row j + 1; gb the gates of rows 2j, 2j + 1, 2j + 2.
    float pre[2][CN], row0[MODE == CONV_BACK ? 1 : CN];
    uint32_t gb[3] = {0u, 0u, 0u};
    const int c0 = CN * grp;
    const int nch = min(max(Cin - c0, 0), CN);  // CONV_PLAIN: staged channels that exist
    const bool stages = mover && c0 < CINP;
    auto load = [&](int b, int j, bool fresh) {
        if (!stages) return;
        if constexpr (MODE == CONV_BACK) {
            const unsigned cs = (unsigned)S * CT_NT;
            const float* src = a.in + ((long)b * Cin + c0) * cs + t;
            const int r1 = min(j + 1, S - 1);  // a row beyond the sample is gated off
#pragma unroll
            for (int c = 0; c < CN; ++c) {
                pre[0][c] = fresh ? tf32r(0.5f * __ldg(src + c * cs + j * CT_NT)) : pre[1][c];
                pre[1][c] = __ldg(src + c * cs + r1 * CT_NT);
            }
            const unsigned char* g = a.gate_in + (((long)b * H + 2 * j) * CT_NT + t) * 4 + grp;
            if (fresh) gb[0] = __ldg(g);
            gb[1] = __ldg(g + 4 * CT_NT);
            gb[2] = j + 1 < S ? __ldg(g + 8 * CT_NT) : 0;
        } else {
            const unsigned cs = (unsigned)H * CT_NT;
            const float* src = a.in + ((long)b * Cin + c0) * cs + t;
            const int r = 2 * j + 1;
            const bool k0 = r < H, k1 = r + 1 < H;
#pragma unroll
            for (int c = 0; c < CN; ++c) {
                const bool in = MODE != CONV_PLAIN || c < nch;
                if (fresh) row0[c] = in ? __ldg(src + c * cs) : 0.f;
                pre[0][c] = in && k0 ? __ldg(src + c * cs + r * CT_NT) : 0.f;
                pre[1][c] = in && k1 ? __ldg(src + c * cs + (r + 1) * CT_NT) : 0.f;
            }
        }
    };
    auto put_row = [&](int slot, const float* v, uint32_t gate) {
        unsigned char* dst = sX + slot * CT_ROW_BYTES + t * 128;
#pragma unroll
        for (int k4 = 0; k4 < CN / 4; ++k4) {
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = 4 * k4 + e;
                if constexpr (MODE == CONV_BACK)
                    x[e] = (gate >> c) & 1u ? v[c] : 0.f;
                else
                    x[e] = tf32r(v[c]);
            }
            const int c4 = CN / 4 * grp + k4;
            *(float4*)(dst + ((c4 ^ (t & 7)) << 4)) = make_float4(x[0], x[1], x[2], x[3]);
        }
    };
    const float none[CN] = {};
    // CONV_BACK: pooled row j + 1, as loaded, halved and rounded once for its two rows (pre[0] is so already)
    auto halve = [&]() {
        if constexpr (MODE == CONV_BACK) {
#pragma unroll
            for (int c = 0; c < CN; ++c) pre[1][c] = tf32r(0.5f * pre[1][c]);
        }
    };
    // lo, hi: ring pairs of the step's stages j and j + 1
    auto put = [&](int lo, int hi, bool fresh) {
        if (!stages) return;
        halve();
        if (fresh) {
            put_row(2 * lo, none, 0u);
            if constexpr (MODE == CONV_BACK)
                put_row(2 * lo + 1, pre[0], gb[0]);
            else
                put_row(2 * lo + 1, row0, 0u);
        }
        put_row(2 * hi, pre[0], gb[1]);
        put_row(2 * hi + 1, pre[1], gb[2]);
    };

    int b = s0 / S, j = s0 - b * S;  // of the step that is loaded next
    int lo = 0, hi = 1;
    bool fresh = j == 0;
    auto advance = [&]() {
        fresh = ++j == S;
        if (fresh) {
            j = 0;
            ++b;
        }
    };
    if (!fresh && stages) {
        // a block that starts inside a sample: rows 2j - 1 and 2j
        if constexpr (MODE == CONV_BACK) {
            load(b, j - 1, true);
            halve();
            put_row(2 * lo, pre[0], gb[1]);
            put_row(2 * lo + 1, pre[1], gb[2]);
        } else {
            load(b, j - 1, false);
            put_row(2 * lo, pre[0], 0u);
            put_row(2 * lo + 1, pre[1], 0u);
        }
    }
    load(b, j, fresh);
    put(lo, hi, fresh);
    int ob = b, oj = j;  // of the step that is written next
    advance();
    if (cnt > 1) load(b, j, fresh);
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    constexpr uint32_t idesc = idesc_tf32(N);
    const uint64_t dx = tc::sdesc(tc::su32(sX)), dw = tc::sdesc(tc::su32(sWt));
    auto issue = [&](int k, int lo_, int hi_) {  // the MMAs of step k, by one thread
        const uint32_t d = tmem + (k & 1) * 2 * N;
        const uint64_t xl = dx + (uint32_t)(lo_ * 2 * (CT_ROW_BYTES >> 4));
        const uint64_t xh = dx + (uint32_t)(hi_ * 2 * (CT_ROW_BYTES >> 4));
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int dh = 0; dh < 3; ++dh) {
                const int w = r + dh;  // row of the four
                const uint64_t x = w < 2 ? xl + w * (CT_ROW_BYTES >> 4) : xh + (w - 2) * (CT_ROW_BYTES >> 4);
#pragma unroll
                for (int kk = 0; kk < CINP / 8; ++kk)
                    mma_tf32(d + r * N, x + 2 * kk, dw + dh * (WB >> 4) + 2 * kk, idesc, (dh | kk) != 0);
            }
        tc::commit(bar + (k & 1));
    };
    if (tid == CT_ROW_THREADS) issue(0, lo, hi);

    bool ok = true;
    int k = 0;
    for (; k < cnt; ++k) {
        bool got = true;
        const uint32_t tl = tmem + ((uint32_t)(32 * quarter) << 16) + (k & 1) * 2 * N + CH * grp;
        float* edge = sEdge + (k & 1) * 16 * COUT + CH * grp;
        // pairs of the step after this one: its older stage is this step's newer one, or, at the
        // first step of a sample, both are new
        if (!fresh) {
            const int s = lo;
            lo = hi;
            hi = s;
        }
        if (mover) {
            got = tc::mbar_wait(bar + (k & 1), (uint32_t)(k >> 1) & 1u, a.err, false, CT_WAIT_NS);
            tc::fence_after();
            // the product rows of the angles next to another warp's
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float P[3][CH];
                tmem_ld3<CH>(tl + r * N, tl + r * N, tl + r * N + 2 * COUT, P);
                float* e = edge + r * 8 * COUT + quarter * COUT;
#pragma unroll
                for (int c = 0; c < CH; c += 4) {
                    if (lane == 31) *(float4*)(e + c) = make_float4(P[0][c], P[0][c + 1], P[0][c + 2], P[0][c + 3]);
                    if (lane == 0)
                        *(float4*)(e + 4 * COUT + c) = make_float4(P[2][c], P[2][c + 1], P[2][c + 2], P[2][c + 3]);
                }
            }
            if (k + 1 < cnt) put(lo, hi, fresh);
            tc::fence_proxy_async();
        }
        tc::fence_before();
        if (!__syncthreads_and(got)) {
            ok = false;
            break;
        }
        tc::fence_after();
        if (!mover) {
            if (lane == 0 && k + 1 < cnt) issue(k + 1, lo, hi);
            __syncwarp();
            advance();
            continue;
        }
        const int wb_ = ob, wj = oj;
        ob = b;
        oj = j;
        advance();
        if (k + 2 < cnt) load(b, j, fresh);
        float v[2][CH];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float P[3][CH], elo[CH], ehi[CH];
            const float* e0 = edge + r * 8 * COUT + ((quarter + 3) & 3) * COUT;
            const float* e1 = edge + r * 8 * COUT + (4 + ((quarter + 1) & 3)) * COUT;
#pragma unroll
            for (int c = 0; c < CH; c += 4) {
                *(float4*)(elo + c) = *(const float4*)(e0 + c);
                *(float4*)(ehi + c) = *(const float4*)(e1 + c);
            }
            tmem_ld3<CH>(tl + r * N, tl + r * N + COUT, tl + r * N + 2 * COUT, P);
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const float l = __shfl_up_sync(0xffffffffu, P[0][c], 1);
                const float h = __shfl_down_sync(0xffffffffu, P[2][c], 1);
                v[r][c] = (lane == 0 ? elo[c] : l) + P[1][c] + (lane == 31 ? ehi[c] : h);
            }
        }
        uint32_t gm[2] = {0u, 0u};
        if constexpr (MODE != CONV_BACK) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                const float bias = sBias[CH * grp + c];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    v[r][c] += bias;
                    if (MODE == CONV_POOL || a.relu) v[r][c] = fmaxf(v[r][c], 0.f);
                    gm[r] |= v[r][c] > 0.f ? 1u << c : 0u;
                }
            }
        }
        const long g0 = (((long)wb_ * H + 2 * wj) * CT_NT + t) * 4 + grp;
        if constexpr (MODE == CONV_POOL) {
            float* o = a.out + (((long)wb_ * COUT + CH * grp) * S + wj) * CT_NT + t;
#pragma unroll
            for (int c = 0; c < CH; ++c) o[(unsigned)(c * S) * CT_NT] = 0.5f * (v[0][c] + v[1][c]);
            if (a.gate_out) {
                a.gate_out[g0] = (unsigned char)gm[0];
                a.gate_out[g0 + 4 * CT_NT] = (unsigned char)gm[1];
            }
        } else {
            float* o = a.out + (((long)wb_ * COUT + CH * grp) * H + 2 * wj) * CT_NT + t;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (2 * wj + r >= H) continue;
                if (MODE == CONV_BACK && COUT == 16 && a.gate_res) {
                    const uint32_t g = __ldg(a.gate_res + g0 + r * 4 * CT_NT);
#pragma unroll
                    for (int c = 0; c < CH; ++c) v[r][c] = (g >> c) & 1u ? v[r][c] : 0.f;
                }
#pragma unroll
                for (int c = 0; c < CH; ++c) o[(unsigned)(c * H + r) * CT_NT] = v[r][c];
                if (MODE == CONV_PLAIN && COUT == 16 && a.gate_out)
                    a.gate_out[g0 + r * 4 * CT_NT] = (unsigned char)gm[r];
            }
        }
    }
    if (!ok && tid == 0)  // MMAs still in flight
        tc::mbar_wait(bar + (k & 1), (uint32_t)(k >> 1) & 1u, a.err, false, CT_WAIT_NS);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tmem_free<TM>(tmem);
    }
}

struct ConvWgTcArgs {
    const float* in;    // [B][Cin][H][128]
    const float* dpre;  // [B][Cout][H][128]; gated: the pooled rows' gradient [B][Cout][H / 2][128]
    const unsigned int* gate;  // gated: [B][H][128], a bit per output channel
    float* part;        // [gridDim.x][9 Cin Cout + Cout]: (dh, ci, dt, co), then the bias
    int B, Cin, H, rows_per_cta;
    int* err;
};

// a row is read once and 80 KB of loads are in flight on an SM beside 172 KB of shared memory:
// without a line in L1 each (at the 32-channel layers 136 -> 119 us)
__device__ __forceinline__ float4 ldg_once(const float4* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// Weight gradient.  Of the 16 warps that move data, warp w stages the channels w, w + 16 of a
// row: lane l has the angles 4l .. 4l + 3 (16 bytes), the neighbours for the angle offsets come
// by shuffle.
// A (dpre, rows (dt, co)): 4 planes of 32 angles, two buffers; plane p starts at p * PA with
// PA = 3 Cout rows of 128 B, so the MMA's rows beyond 3 Cout read the next plane (their
// products are never used).  B: 4 planes of a ring of 4 input rows (slot, ci), so that the
// window of up to three rows is one operand of N = 3 CINP columns (two where it wraps); the
// rows outside the sample are left out of the product instead of staged as zeros.  Slots
// and windows move together, so the row h whose slot is a adds to accumulator a of four, and
// in accumulator a the columns of slot s belong to dh = 1 + (s - a) mod 4.
// Row i is staged while the MMAs of row i - 1 run (they read the other A buffer and none of
// the slots written); those of row i - 2 have completed.  Rows are loaded two ahead.
// Bound: shared memory, 64 KB written and 112 KB read by the MMAs a row at 32 channels, and the
// barrier a row.  With one load and three stores of 4 bytes a channel and angle, a product per
// dh (A read three times), one buffer and 9216 atomic adds a block, the batch of 256 took 265,
// 172 and 118 us at layers 2 to 4; this one takes 166, 120 and 66 us, from the pooled rows, and
// 8 us of k_wgrad_sum.
template <int CINP, int COUT>
struct WgGeom {
    static constexpr int M = 3 * COUT, PA = M * 128, ABUF = 4 * PA + (128 - M) * 128;
    static constexpr int NB = 4 * CINP, PB = NB * 128;
    static constexpr int SMEM = 1024 + 2 * ABUF + 4 * PB + 64;
};

template <int CINP, int COUT, bool GATED>
__global__ void __launch_bounds__(CT_THREADS, 1) k_conv3_wgrad_tc(ConvWgTcArgs a) {
    using G = WgGeom<CINP, COUT>;
    constexpr int M = G::M, PA = G::PA, PB = G::PB, NB = G::NB;
    constexpr int KA = COUT / 16, KX = CINP / 16;  // channels a warp stages
    extern __shared__ unsigned char smraw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = sm;
    unsigned char* sB = sm + 2 * G::ABUF;
    uint64_t* bar = (uint64_t*)(sB + 4 * PB);  // MMAs of even rows, of odd rows, of the start
    uint32_t* tslot = (uint32_t*)(bar + 3);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool mover = warp < CT_ROW_THREADS / 32;
    const int Cin = a.Cin, H = a.H;
    const long q0 = (long)blockIdx.x * a.rows_per_cta;
    const int cnt = (int)(min((long)a.B * H, q0 + a.rows_per_cta) - q0);
    if (cnt <= 0) return;  // uniform over the block

    // a row's data: dpre row h and input row h + 1; x0: input row h for the first row of a
    // sample or of the block
    struct Row {
        float4 a[KA], x[KX];
        uint4 gate;
    };
    Row ra, rb;
    float4 x0[KX];
    auto loadX = [&](int b, int x, float4* v) {
        const float* src = a.in + (((long)b * Cin + warp) * H + x) * CT_NT + 4 * lane;
#pragma unroll
        for (int k = 0; k < KX; ++k)
            v[k] = warp + 16 * k < Cin ? ldg_once((const float4*)(src + (unsigned)(16 * k * H) * CT_NT))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto load = [&](Row& r, int b, int h) {
        const int S = GATED ? H / 2 : H;
        const float* src = a.dpre + (((long)b * COUT + warp) * S + (GATED ? h / 2 : h)) * CT_NT + 4 * lane;
#pragma unroll
        for (int k = 0; k < KA; ++k) r.a[k] = ldg_once((const float4*)(src + (unsigned)(16 * k * S) * CT_NT));
        if (GATED) r.gate = __ldg((const uint4*)(a.gate + ((long)b * H + h) * CT_NT + 4 * lane));
        if (h + 1 < H) loadX(b, h + 1, r.x);
    };
    const int pl = lane >> 3, ch = lane & 7;  // plane and 16-byte chunk of this lane's angles
    auto round4 = [](float4 v) { return make_float4(tf32r(v.x), tf32r(v.y), tf32r(v.z), tf32r(v.w)); };
    auto putX = [&](int slot, const float4* v) {
#pragma unroll
        for (int k = 0; k < KX; ++k) {
            const int r = slot * CINP + warp + 16 * k;
            *(float4*)(sB + pl * PB + r * 128 + ((ch ^ (r & 7)) << 4)) = round4(v[k]);
        }
    };
    float dbacc[KA];
#pragma unroll
    for (int k = 0; k < KA; ++k) dbacc[k] = 0.f;
    auto putA = [&](int buf, const Row& row) {
#pragma unroll
        for (int k = 0; k < KA; ++k) {
            float4 v = row.a[k];
            if constexpr (GATED) {
                const int co = warp + 16 * k;
                v.x = (row.gate.x >> co) & 1u ? 0.5f * v.x : 0.f;
                v.y = (row.gate.y >> co) & 1u ? 0.5f * v.y : 0.f;
                v.z = (row.gate.z >> co) & 1u ? 0.5f * v.z : 0.f;
                v.w = (row.gate.w >> co) & 1u ? 0.5f * v.w : 0.f;
            }
            dbacc[k] += (v.x + v.y) + (v.z + v.w);
            v = round4(v);
            const float nx = __shfl_sync(0xffffffffu, v.x, (lane + 1) & 31);
            const float pv = __shfl_sync(0xffffffffu, v.w, (lane + 31) & 31);
            unsigned char* dst = sA + buf * G::ABUF + pl * PA;
#pragma unroll
            for (int dt = 0; dt < 3; ++dt) {  // element s of row (dt, co): dpre at s - dt + 1
                const int r = dt * COUT + warp + 16 * k;
                *(float4*)(dst + r * 128 + ((ch ^ (r & 7)) << 4)) =
                    dt == 0 ? make_float4(v.y, v.z, v.w, nx) : dt == 1 ? v : make_float4(pv, v.x, v.y, v.z);
            }
        }
    };

    // b, h, fresh, off: of the row that is staged next (off: ring slot of input row x is
    // (x + off) & 3); lb, lh: of the row that is loaded next
    int b = (int)(q0 / H), h = (int)(q0 - (long)b * H), off = 0;
    bool fresh = true;
    int lb = b, lh = h;
    auto load_next = [&](Row& r) {
        load(r, lb, lh);
        if (++lh == H) {
            lh = 0;
            ++lb;
        }
    };
    if (mover) {
        if (h > 0) loadX(b, h - 1, rb.x);
        loadX(b, h, x0);
        load_next(ra);
    }
    if (tid == 0) {
        for (int k = 0; k < 3; ++k) tc::mbar_init(bar + k, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc<4 * NB>(tslot);
    // rows the MMAs read but whose products are unused, and channels beyond Cin, stay zero
    for (int i = tid; i < (2 * G::ABUF + 4 * PB) / 16; i += CT_THREADS)
        ((float4*)sm)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    const uint64_t da0 = tc::sdesc(tc::su32(sA)), db0 = tc::sdesc(tc::su32(sB));
    // the accumulators start at zero: products of the zeroed operands
    if (tid == CT_ROW_THREADS) {
        for (int k = 0; k < 4; ++k) mma_tf32(tmem + k * NB, da0, db0, idesc_tf32(NB), 0u);
        tc::commit(bar + 2);
    }
    bool got = tc::mbar_wait(bar + 2, 0u, a.err, false, CT_WAIT_NS);
    if (mover) {
        if (h > 0) putX((h - 1) & 3, rb.x);
        if (cnt > 1) load_next(rb);
    }

    int issued = 0;
    // row i from r, whose registers then take the row after the next; false: a wait ran out
    auto step = [&](int i, Row& r) {
        if (mover) {
            if (i >= 2) got = tc::mbar_wait(bar + (i & 1), ((uint32_t)(i >> 1) - 1u) & 1u, a.err, false, CT_WAIT_NS);
            putA(i & 1, r);
            if (fresh) putX((h + off) & 3, x0);
            if (h + 1 < H) putX((h + 1 + off) & 3, r.x);
            if (i + 2 < cnt) load_next(r);
            if (h + 1 == H && i + 1 < cnt) loadX(b + 1, 0, x0);
            tc::fence_proxy_async();
        }
        tc::fence_before();
        if (!__syncthreads_and(got)) return false;
        tc::fence_after();
        if (tid == CT_ROW_THREADS) {
            const int acc = (h + off) & 3;
            const int x0 = h > 0 ? h - 1 : h, nx = (h + 1 < H ? h + 1 : h) - x0 + 1;
            const int sl = (x0 + off) & 3, n1 = min(nx, 4 - sl), n2 = nx - n1;
            const uint64_t da = da0 + (uint32_t)((i & 1) * (G::ABUF >> 4));
            const uint64_t db = db0 + (uint32_t)(sl * CINP * 8);
            const uint32_t d0 = tmem + acc * NB, d1 = d0 + sl * CINP;
            const uint32_t id1 = idesc_tf32(n1 * CINP), id2 = idesc_tf32(n2 * CINP);
#pragma unroll
            for (int kk = 0; kk < 16; ++kk) {
                const int p = kk >> 2, o = (kk & 3) * 2;
                mma_tf32(d1, da + (p * (PA >> 4) + o), db + (p * (PB >> 4) + o), id1, 1u);
            }
            if (n2) {
#pragma unroll
                for (int kk = 0; kk < 16; ++kk) {
                    const int p = kk >> 2, o = (kk & 3) * 2;
                    mma_tf32(d0, da + (p * (PA >> 4) + o), db0 + (p * (PB >> 4) + o), id2, 1u);
                }
            }
            tc::commit(bar + (i & 1));
        }
        __syncwarp();
        issued = i + 1;
        fresh = ++h == H;
        if (fresh) {
            off = (off + H) & 3;
            h = 0;
            ++b;
        }
        return true;
    };
    bool ok = true;
    for (int i = 0; ok && i < cnt; i += 2) {
        ok = step(i, ra);
        if (ok && i + 1 < cnt) ok = step(i + 1, rb);
    }
    for (int k = max(issued - 2, 0); k < issued; ++k)  // the MMAs in flight
        got = tc::mbar_wait(bar + (k & 1), (uint32_t)(k >> 1) & 1u, a.err, false, CT_WAIT_NS) && got;
    tc::fence_after();
    if (__syncthreads_and(got && ok) && mover) {
        const int quarter = warp & 3, m = 32 * quarter + lane;  // product row (dt, co)
        float* part = a.part + (long)blockIdx.x * (9 * Cin * COUT + COUT);
        if (32 * quarter < M) {
            const uint32_t tl = tmem + ((uint32_t)(32 * quarter) << 16);
            for (int it = warp >> 2; it < 3 * KX; it += 4) {
                const int dh = it % 3, c0 = it / 3 * 16;
                float s[16], v[16];
                tc::tmem_ld16(tl + ((dh + 3) & 3) * CINP + c0, s);
#pragma unroll
                for (int acc = 1; acc < 4; ++acc) {
                    tc::tmem_ld16(tl + acc * NB + ((acc + dh + 3) & 3) * CINP + c0, v);
#pragma unroll
                    for (int c = 0; c < 16; ++c) s[c] += v[c];
                }
                if (m < M) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        if (c0 + c < Cin) part[(dh * Cin + c0 + c) * M + m] = s[c];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < KA; ++k) {
            float v = dbacc[k];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) part[9 * Cin * COUT + warp + 16 * k] = v;
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tmem_free<4 * NB>(tmem);
    }
}

// One input channel, weight gradient: warp w sums output channel 16 blockIdx.y + w over the
// rows of its block, lane l at the angles 4l .. 4l + 3 (16 bytes a load), WF_AHEAD rows in
// flight.  TF32-rounded operands, FP32 sums.  Bound: the read of dpre (134 MB for a batch of
// 256, 20 us).  On the tensor cores (one input channel of the 16 that N takes) it took 210 us,
// a thread an angle and four channels with one row in flight 88; this one 48 us.
constexpr int WF_AHEAD = 4;
__global__ void __launch_bounds__(CT_ROW_THREADS) k_wgrad_first(ConvWgTcArgs a, int cout) {
    const int lane = threadIdx.x & 31, co = 16 * blockIdx.y + (threadIdx.x >> 5);
    const int H = a.H;
    const long q0 = (long)blockIdx.x * a.rows_per_cta;
    const int cnt = (int)(min((long)a.B * H, q0 + a.rows_per_cta) - q0);
    float s[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) s[k] = 0.f;
    // dpre at angle t meets the input at t - 1, t, t + 1: six inputs of a row for four angles
    auto widen = [&](float4 v, float* x) {
        x[1] = tf32r(v.x);
        x[2] = tf32r(v.y);
        x[3] = tf32r(v.z);
        x[4] = tf32r(v.w);
        x[0] = __shfl_sync(0xffffffffu, x[4], (lane + 31) & 31);
        x[5] = __shfl_sync(0xffffffffu, x[1], (lane + 1) & 31);
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto input = [&](int b, int x) {
        return x >= 0 && x < H ? __ldg((const float4*)(a.in + ((long)b * H + x) * CT_NT + 4 * lane)) : zero;
    };
    auto grad = [&](int b, int h) {
        return __ldg((const float4*)(a.dpre + (((long)b * cout + co) * H + h) * CT_NT + 4 * lane));
    };
    float4 g[WF_AHEAD], y[WF_AHEAD];  // dpre row h and input row h + 1 of the rows in flight
    int b = (int)(q0 / H), h = (int)(q0 - (long)b * H), lb = b, lh = h, loaded = 0;
    auto load = [&](int k) {
        if (loaded >= cnt) return;
        g[k] = grad(lb, lh);
        y[k] = input(lb, lh + 1);
        ++loaded;
        if (++lh == H) {
            lh = 0;
            ++lb;
        }
    };
    float x[3][6];  // input rows h - 1, h, h + 1
    widen(input(b, h - 1), x[0]);
    widen(input(b, h), x[1]);
#pragma unroll
    for (int k = 0; k < WF_AHEAD; ++k) load(k);
    for (int i0 = 0; i0 < cnt; i0 += WF_AHEAD) {
#pragma unroll
        for (int k = 0; k < WF_AHEAD; ++k) {
            if (i0 + k >= cnt) break;
            const float4 v = g[k];
            widen(y[k], x[2]);
            load(k);
            s[9] += (v.x + v.y) + (v.z + v.w);
            const float d[4] = {tf32r(v.x), tf32r(v.y), tf32r(v.z), tf32r(v.w)};
#pragma unroll
            for (int dh = 0; dh < 3; ++dh)
#pragma unroll
                for (int dt = 0; dt < 3; ++dt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[3 * dh + dt] = fmaf(d[e], x[dh][e + dt], s[3 * dh + dt]);
            const bool wrap = ++h == H;
            if (wrap) {
                h = 0;
                ++b;
                widen(i0 + k + 1 < cnt ? input(b, 0) : zero, x[1]);
            }
#pragma unroll
            for (int e = 0; e < 6; ++e) {
                x[0][e] = wrap ? 0.f : x[1][e];
                x[1][e] = wrap ? x[1][e] : x[2][e];
            }
        }
    }
    float* part = a.part + (long)blockIdx.x * (10 * cout);
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        float v = s[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) part[k * cout + co] = v;  // (dh, dt, co), then the bias
    }
}

// adds the blocks' partial sums to dW [co][ci][dh][dt] and db, in the order of the blocks
__global__ void __launch_bounds__(256) k_wgrad_sum(const float* __restrict__ part, int nblk, int Cin, int Cout,
                                                  float* __restrict__ dW, float* __restrict__ db) {
    __shared__ float red[4][64];
    const int nw = 9 * Cin * Cout, n = nw + Cout, q = blockIdx.x * 64 + (threadIdx.x & 63), sl = threadIdx.x >> 6;
    float s = 0.f;
    if (q < n)
        for (int k = sl; k < nblk; k += 4) s += part[(long)k * n + q];
    red[sl][threadIdx.x & 63] = s;
    __syncthreads();
    if (sl || q >= n) return;
    s = (red[0][threadIdx.x] + red[1][threadIdx.x]) + (red[2][threadIdx.x] + red[3][threadIdx.x]);
    if (q >= nw) {
        db[q - nw] += s;
        return;
    }
    const int co = q % Cout, dt = q / Cout % 3, ci = q / (3 * Cout) % Cin, dh = q / (3 * Cout * Cin);
    dW[((co * Cin + ci) * 3 + dh) * 3 + dt] += s;
}

template <int CINP, int COUT, int MODE>
cudaError_t launch_fwd(ConvTcArgs a, cudaStream_t st) {
    constexpr int smem = conv_fwd_smem<COUT>();
    const long steps = (long)a.B * ((a.H + 1) / 2), ctas = sm_count();  // one block per SM
    if (steps > 0x7fffffffL) return cudaErrorInvalidValue;
    a.steps_per_cta = (int)((steps + ctas - 1) / ctas);
    const int grid = (int)((steps + a.steps_per_cta - 1) / a.steps_per_cta);
    const cudaError_t e = allow_smem(k_conv3_tc<CINP, COUT, MODE>, smem);
    if (e != cudaSuccess) return e;
    k_conv3_tc<CINP, COUT, MODE><<<grid, CT_THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

template <int CINP, int COUT, bool GATED>
cudaError_t launch_wgrad(const ConvWgTcArgs& a, int grid, cudaStream_t st) {
    constexpr int smem = WgGeom<CINP, COUT>::SMEM;
    const cudaError_t e = allow_smem(k_conv3_wgrad_tc<CINP, COUT, GATED>, smem);
    if (e != cudaSuccess) return e;
    k_conv3_wgrad_tc<CINP, COUT, GATED><<<grid, CT_THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t wgrad(const float* in, const float* dpre, const unsigned int* gate, int B, int Cin, int H, int Cout,
                  float* dW, float* db, float* part, int* err, cudaStream_t st) {
    const long rows = (long)B * H;
    ConvWgTcArgs a{in, dpre, gate, part, B, Cin, H, 0, err};
    a.rows_per_cta = (int)((rows + sm_count() - 1) / sm_count());  // one block per SM
    const int grid = (int)((rows + a.rows_per_cta - 1) / a.rows_per_cta);
    cudaError_t e;
    if (Cin == 1) {
        k_wgrad_first<<<dim3(grid, Cout / 16), CT_ROW_THREADS, 0, st>>>(a, Cout);
        e = cudaGetLastError();
    } else if (gate) {  // Cout = 32
        e = Cin > 16 ? launch_wgrad<32, 32, true>(a, grid, st) : launch_wgrad<16, 32, true>(a, grid, st);
    } else if (Cout == 32) {
        e = Cin > 16 ? launch_wgrad<32, 32, false>(a, grid, st) : launch_wgrad<16, 32, false>(a, grid, st);
    } else {
        e = Cin > 16 ? launch_wgrad<32, 16, false>(a, grid, st) : launch_wgrad<16, 16, false>(a, grid, st);
    }
    if (e != cudaSuccess) return e;
    k_wgrad_sum<<<(9 * Cin * Cout + Cout + 63) / 64, 256, 0, st>>>(part, grid, Cin, Cout, dW, db);
    return cudaGetLastError();
}

}  // namespace

long lp_wgrad_scratch() { return (long)sm_count() * (9 * 32 * 32 + 32); }

cudaError_t launch_lp_conv3_tc(const float* in, int B, int Cin, int H, const float* W, const float* bias, int Cout,
                               bool relu, float* out, int* err, cudaStream_t st, unsigned int* gate_out) {
    if (B < 1 || H < 1 || Cin < 1 || Cin > 32 || (Cout != 16 && Cout != 32) || !err || (gate_out && Cout != 16))
        return cudaErrorInvalidValue;
    const ConvTcArgs a{in, W, bias, out, nullptr, nullptr, (unsigned char*)gate_out, B, Cin, H, relu ? 1 : 0, 0, err};
    if (Cout == 32)
        return Cin > 16  ? launch_fwd<32, 32, CONV_PLAIN>(a, st)
               : Cin > 8 ? launch_fwd<16, 32, CONV_PLAIN>(a, st)
                         : launch_fwd<8, 32, CONV_PLAIN>(a, st);
    return Cin > 16  ? launch_fwd<32, 16, CONV_PLAIN>(a, st)
           : Cin > 8 ? launch_fwd<16, 16, CONV_PLAIN>(a, st)
                     : launch_fwd<8, 16, CONV_PLAIN>(a, st);
}

cudaError_t launch_lp_conv3_pool_tc(const float* in, int B, int Cin, int H, const float* W, const float* bias,
                                    float* pooled, unsigned int* gate, int* err, cudaStream_t st) {
    if (B < 1 || H < 2 || H % 2 || (Cin != 16 && Cin != 32) || !bias || !err) return cudaErrorInvalidValue;
    const ConvTcArgs a{in, W, bias, pooled, nullptr, nullptr, (unsigned char*)gate, B, Cin, H, 1, 0, err};
    return Cin == 32 ? launch_fwd<32, 32, CONV_POOL>(a, st) : launch_fwd<16, 32, CONV_POOL>(a, st);
}

cudaError_t launch_lp_conv3_back_tc(const float* dp, const unsigned int* gate, int B, int H, const float* W, int Cin,
                                    const unsigned int* gate_in, float* din, int* err, cudaStream_t st) {
    if (B < 1 || H < 2 || H % 2 || (Cin != 16 && Cin != 32) || (Cin == 32 && gate_in) || !gate || !err)
        return cudaErrorInvalidValue;
    const ConvTcArgs a{dp, W, nullptr, din, (const unsigned char*)gate, (const unsigned char*)gate_in, nullptr, B, 32, H, 0, 0, err};
    return Cin == 32 ? launch_fwd<32, 32, CONV_BACK>(a, st) : launch_fwd<32, 16, CONV_BACK>(a, st);
}

cudaError_t launch_lp_conv3_wgrad_tc(const float* in, const float* dpre, int B, int Cin, int H, int Cout, float* dW,
                                     float* db, float* scratch, int* err, cudaStream_t st) {
    if (B < 1 || H < 1 || !(Cin == 1 || (Cin % 8 == 0 && Cin <= 32)) || (Cout != 16 && Cout != 32) || !scratch ||
        !err)
        return cudaErrorInvalidValue;
    return wgrad(in, dpre, nullptr, B, Cin, H, Cout, dW, db, scratch, err, st);
}

cudaError_t launch_lp_conv3_wgrad_pool_tc(const float* in, const float* dp, const unsigned int* gate, int B, int Cin,
                                          int H, float* dW, float* db, float* scratch, int* err, cudaStream_t st) {
    if (B < 1 || H < 2 || H % 2 || (Cin != 16 && Cin != 32) || !gate || !scratch || !err)
        return cudaErrorInvalidValue;
    return wgrad(in, dp, gate, B, Cin, H, 32, dW, db, scratch, err, st);
}

}  // namespace cryoim
