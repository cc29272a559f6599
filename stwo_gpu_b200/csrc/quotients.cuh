// DEEP-quotient parameters shared by the quotient kernel (quotients.cu), its host
// entry points and the prover's device channel, which fills the sample-dependent
// fields on the device.
#pragma once
#include <cstdint>

#include "field.cuh"

namespace stwo {

constexpr int QUOT_MAX_COLS = 512;
constexpr int QUOT_MAX_SAMPLES = 512;
constexpr int QUOT_MAX_BATCHES = 16;

// Circle-group point tables (quotients.cu): G^i for i < 2^11, G^(2^11 i) for i < 2^11
// and G^(2^22 i) for i < 2^9, consecutive.
constexpr uint32_t CIRCLE_TAB_LO = 2048;
constexpr uint32_t CIRCLE_TAB_SIZE = 2 * CIRCLE_TAB_LO + 512;
// Device address of the tables on the current device (filled on first use).
int circle_point_table(const cpoint **out);

template <int MAXC, int MAXS>
struct QuotParamsT {
    const uint32_t *cols[MAXC];
    qm31 c2[MAXS];                        // c_j (canonical)
    uint16_t col_idx[MAXS];
    qm31 a_sum[QUOT_MAX_BATCHES], b_sum[QUOT_MAX_BATCHES], batch_coeff[QUOT_MAX_BATCHES];
    cm31 prx[QUOT_MAX_BATCHES], pry[QUOT_MAX_BATCHES], pix[QUOT_MAX_BATCHES], piy[QUOT_MAX_BATCHES];
    cm31 den_k[QUOT_MAX_BATCHES];          // Pr.x Pi.y - Pr.y Pi.x: den_b(p) = K_b - p.x Pi.y + p.y Pi.x
    uint32_t batch_end[QUOT_MAX_BATCHES];  // cumulative sample counts
    uint32_t n_batches;
    uint32_t half_init, half_step;        // half coset indices
    uint32_t log_size;                    // domain log size
    uint32_t *out[4];
    const cpoint *tab;                    // circle_point_table() of the launching device
};

// The prover's device-resident parameters: up to 1024 columns and samples.
using QuotParamsDev = QuotParamsT<1024, 1024>;

// Sample-dependent fields of batch b (samples off .. off+count-1 at point (px, py)):
// the batch coefficient rc^count and, per sample j with alpha = rc^(j+1),
// (a, b, c) = alpha * (conj(v) - v, v*c0 - a*py, c0), c0 = conj(py) - py
// (complex_conjugate_line_coeffs); a and b summed per batch, c stored per sample.
// With several batches, quot_scale_batches then folds the accumulation's Horner
// coefficients into these fields.
template <class QP>
__host__ __device__ inline void quot_fill_point(QP &p, uint32_t b, qm31 px, qm31 py) {
    p.prx[b] = px.a;
    p.pix[b] = px.b;
    p.pry[b] = py.a;
    p.piy[b] = py.b;
    p.den_k[b] = cm31_sub(cm31_mul(px.a, py.b), cm31_mul(py.a, px.b));
}

template <class QP>
__host__ __device__ inline void quot_fill_batch(QP &p, uint32_t b, qm31 rc, qm31 px, qm31 py, const qm31 *vals,
                                                uint32_t count, uint32_t off) {
    quot_fill_point(p, b, px, py);
    p.batch_coeff[b] = qm31_pow(rc, count);
    const qm31 c0 = qm31_sub(qm31_conj(py), py);
    qm31 alpha = qm31_one(), as = qm31_zero(), bs = qm31_zero();
    for (uint32_t j = 0; j < count; j++) {
        alpha = qm31_mul(alpha, rc);
        const qm31 v = vals[j];
        qm31 a = qm31_sub(qm31_conj(v), v);
        qm31 bb = qm31_sub(qm31_mul(v, c0), qm31_mul(a, py));
        a = qm31_mul(alpha, a);
        bb = qm31_mul(alpha, bb);
        const qm31 c = qm31_mul(alpha, c0);
        as = qm31_add(as, a);
        bs = qm31_add(bs, bb);
        p.c2[off + j] = c;
    }
    p.a_sum[b] = as;
    p.b_sum[b] = bs;
}

// The accumulation over batches, acc = acc * rc^|b| + num_b / den_b in batch order
// (quotients.cu:111-178), equals sum_b C_b num_b / den_b with C_b the product of the
// later batches' coefficients rc^|b'|. num_b is linear in the batch's a, b and c
// fields, so multiplying those by C_b (here, once per call) leaves the kernel a plain
// sum over batches. The last batch has C = 1; with one batch nothing changes.
template <class QP>
__host__ __device__ inline void quot_scale_batches(QP &p, uint32_t n_batches) {
    qm31 cb = qm31_one();
    for (int b = (int)n_batches - 1; b >= 0; b--) {
        if (b + 1 < (int)n_batches) {
            cb = qm31_mul(cb, p.batch_coeff[b + 1]);
            const uint32_t j0 = b == 0 ? 0u : p.batch_end[b - 1];
            for (uint32_t j = j0; j < p.batch_end[b]; j++) p.c2[j] = qm31_mul(p.c2[j], cb);
            p.a_sum[b] = qm31_mul(p.a_sum[b], cb);
            p.b_sum[b] = qm31_mul(p.b_sum[b], cb);
        }
    }
}

// Sum of one QM31 per lane over the warp; every lane gets the sum.
__device__ __forceinline__ qm31 warp_sum_qm31(qm31 v) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        v.a.a = m31_add(v.a.a, __shfl_xor_sync(0xffffffffu, v.a.a, m));
        v.a.b = m31_add(v.a.b, __shfl_xor_sync(0xffffffffu, v.a.b, m));
        v.b.a = m31_add(v.b.a, __shfl_xor_sync(0xffffffffu, v.b.a, m));
        v.b.b = m31_add(v.b.b, __shfl_xor_sync(0xffffffffu, v.b.b, m));
    }
    return v;
}

// quot_fill_batch of two single-batch groups at one point by a CTA of 256 threads: thread t
// takes samples t, t + 256, ... of both with alpha = rc^(j+1) (the first group has at most
// 256), and the a / b sums of both are reduced across the CTA together. For the prover's
// groups: no quot_scale_batches step is needed with one batch, nor the batch coefficient
// it reads. sh: 32 QM31 of shared memory.
template <class QP>
__device__ inline void quot_fill_two_block(QP &p0, const qm31 *vals0, uint32_t count0, QP &p1, const qm31 *vals1,
                                           uint32_t count1, qm31 rc, qm31 px, qm31 py, qm31 *sh) {
    constexpr uint32_t T = 256;
    const uint32_t tid = threadIdx.x;
    const qm31 c0 = qm31_sub(qm31_conj(py), py);
    qm31 alpha = qm31_pow(rc, tid + 1);
    qm31 sum[4] = {qm31_zero(), qm31_zero(), qm31_zero(), qm31_zero()};  // a and b of group 0, of group 1
    auto fill = [&](QP &p, const qm31 *vals, uint32_t j, qm31 c, qm31 &as, qm31 &bs) {
        const qm31 v = vals[j], a = qm31_sub(qm31_conj(v), v);
        as = qm31_add(as, qm31_mul(alpha, a));
        bs = qm31_add(bs, qm31_mul(alpha, qm31_sub(qm31_mul(v, c0), qm31_mul(a, py))));
        p.c2[j] = c;
    };
    if (tid < count0) fill(p0, vals0, tid, qm31_mul(alpha, c0), sum[0], sum[1]);
    if (tid < count1) fill(p1, vals1, tid, qm31_mul(alpha, c0), sum[2], sum[3]);
    if (count1 > T) {
        const qm31 step = qm31_pow(rc, T);
        for (uint32_t j = tid + T; j < count1; j += T) {
            alpha = qm31_mul(alpha, step);
            fill(p1, vals1, j, qm31_mul(alpha, c0), sum[2], sum[3]);
        }
    }
    __syncthreads();  // sh may hold earlier values
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const qm31 w = warp_sum_qm31(sum[q]);
        if ((tid & 31u) == 0) sh[8 * q + (tid >> 5)] = w;
    }
    __syncthreads();
    if (tid == 0 || tid == 32) {
        QP &p = tid ? p1 : p0;
        const qm31 *s = sh + (tid ? 16 : 0);
        qm31 as = qm31_zero(), bs = qm31_zero();
        for (int w = 0; w < 8; w++) {
            as = qm31_add(as, s[w]);
            bs = qm31_add(bs, s[8 + w]);
        }
        quot_fill_point(p, 0, px, py);
        p.a_sum[0] = as;
        p.b_sum[0] = bs;
    }
}

// The column-independent fields: domain, outputs, point tables.
template <class QP>
inline void quot_init_static(QP &p, uint32_t half_init, uint32_t half_step, uint32_t log_size, uint32_t *const *out4,
                             const cpoint *tab) {
    p.tab = tab;
    p.half_init = half_init;
    p.half_step = half_step;
    p.log_size = log_size;
    for (int c = 0; c < 4; c++) p.out[c] = out4[c];
}

// Launches the quotient kernel on parameters resident in device memory (n_samples:
// the total sample count, batch_end of the last batch); jobs parameter blocks of one
// shape at once, block k at p_dev moved by k * js bytes.
int quotients_dev_async(const QuotParamsDev *p_dev, uint32_t log_size, uint32_t n_samples, uint32_t jobs, size_t js,
                        cudaStream_t st);

}  // namespace stwo
