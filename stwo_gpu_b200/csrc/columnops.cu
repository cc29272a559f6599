// ColumnOps::bit_reverse_column and FieldOps::batch_inverse.
//
// Bit reversal (reference: one thread per swap with uncoalesced 4/16-byte
// accesses, cuda/src/bit_reverse.cu:6-33). Here, for n = 2^L with L >= 10, the index
// splits as (a | b | c) with a and c of 5 bits: bitrev(a|b|c) = (rev c | rev b | rev a).
// A CTA takes the 32x32 block of (a, c) for middle b and the block for rev(b),
// loads both with 128-byte row reads, and writes each transposed-and-reversed into
// the other, so every HBM access is a full line and in-place is safe.
//
// Batch inverse (reference: per-block product tree in shared memory,
// cuda/src/batch_inverse.cu:25-155). Here each thread inverts the product of its own 8 or
// 16 elements (a warp's accesses are whole lines) and unwinds it: no shared memory, no
// barrier, no shuffles. QM31 elements are inverted through their M31 norms.
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace stwo {
namespace {

template <int WORDS>
struct Elem { uint32_t w[WORDS]; };

template <int WORDS>
__global__ void bitrev_simple_kernel(Elem<WORDS> *a, uint32_t L) {
    const uint64_t n = 1ull << L;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t j = bit_reverse_bits((uint32_t)i, L);
        if (j > i) {
            Elem<WORDS> t = a[i];
            a[i] = a[j];
            a[j] = t;
        }
    }
}

// One CTA per (b, rev b) pair with b <= rev b; 256 threads; WORDS words per element.
template <int WORDS>
__global__ void __launch_bounds__(256) bitrev_tiled_kernel(uint32_t *a, uint32_t L, const uint32_t *pairs) {
    __shared__ uint32_t t0[32][32 * WORDS + 1];
    __shared__ uint32_t t1[32][32 * WORDS + 1];
    const uint32_t mb = L - 10;  // middle bits
    const uint32_t b0 = pairs[blockIdx.x];
    const uint32_t b1 = bit_reverse_bits(b0, mb);
    const uint32_t tid = threadIdx.x;
    // Element (a, b, c) lives at index (a << (L-5)) | (b << 5) | c.
    for (uint32_t e = tid; e < 32 * 32 * WORDS; e += 256) {
        uint32_t row = e / (32 * WORDS), col = e % (32 * WORDS);
        uint64_t base0 = (((uint64_t)row << (L - 5)) | ((uint64_t)b0 << 5)) * WORDS;
        uint64_t base1 = (((uint64_t)row << (L - 5)) | ((uint64_t)b1 << 5)) * WORDS;
        t0[row][col] = a[base0 + col];
        t1[row][col] = a[base1 + col];
    }
    __syncthreads();
    // Destination of (a, b0, c) is (rev c, rev b0 = b1, rev a): row rev c of block b1, column rev a.
    for (uint32_t e = tid; e < 32 * 32 * WORDS; e += 256) {
        uint32_t row = e / (32 * WORDS), col = e % (32 * WORDS);
        uint32_t ci = col / WORDS, w = col % WORDS;  // ci = element column within the row
        uint32_t src_row = bit_reverse_bits(ci, 5), src_c = bit_reverse_bits(row, 5);
        uint64_t base1 = (((uint64_t)row << (L - 5)) | ((uint64_t)b1 << 5)) * WORDS;
        uint64_t base0 = (((uint64_t)row << (L - 5)) | ((uint64_t)b0 << 5)) * WORDS;
        a[base1 + col] = t0[src_row][src_c * WORDS + w];
        a[base0 + col] = t1[src_row][src_c * WORDS + w];
    }
}

// ---------------------------------------------------------------- batch inverse
constexpr int BI_THREADS = 128;
constexpr int BI_M31_PER_THREAD = 16;
constexpr int BI_QM31_PER_THREAD = 8;

// Montgomery's batch inverse with a thread's own elements as the batch: prefix products in
// registers, one field inversion of the thread's product (30 squarings and 8 products,
// 2.4 an element), and the inverses unwound from the last element down. A warp's elements
// are base + i * 32 + lane, so loads and stores are whole lines; no lane needs another's
// values. (A warp-wide product with one inversion, computed by every lane all the same,
// cost the same instructions plus two shuffle scans on the critical path: 4 x 9999991
// values 100 us, against 82 us with 8 elements a thread and 72 us with 16.)
__global__ void __launch_bounds__(BI_THREADS) batch_inverse_m31_kernel(const uint32_t *__restrict__ src,
                                                                       uint32_t *__restrict__ dst, uint64_t n) {
    chain_wait();
    constexpr int E = BI_M31_PER_THREAD;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp_global = ((uint64_t)blockIdx.x * BI_THREADS + threadIdx.x) >> 5;
    const uint64_t base = warp_global * (32 * E) + lane;
    uint32_t v[E], pre[E];
    uint32_t run = 1;
#pragma unroll
    for (int i = 0; i < E; i++) {
        const uint64_t idx = base + (uint64_t)i * 32;
        v[i] = (idx < n) ? src[idx] : 1u;
        run = m31_mul(run, v[i]);
        pre[i] = run;
    }
    uint32_t r = m31_inv(run);
#pragma unroll
    for (int i = E - 1; i >= 0; i--) {
        const uint32_t inv_i = i > 0 ? m31_mul(r, pre[i - 1]) : r;
        const uint64_t idx = base + (uint64_t)i * 32;
        if (idx < n) dst[idx] = inv_i;
        r = m31_mul(r, v[i]);
    }
}

// QM31 batch inverse through norms. For z = a + b u (a, b in CM31, u^2 = R = 2 + i):
// z (a - b u) = a^2 - R b^2 = N in CM31, and N conj(N) = |N|^2 in M31, so
// z^-1 = (a - b u) conj(N) / |N|^2. A thread's Montgomery inverse then runs on the
// M31 norms of its elements instead of on QM31 values; the inverse is unique, so the
// values are the same. Bound by instruction issue next to HBM (32 bytes an element): no
// shuffle scans (as above), CM31 products as two-term dot products with one three-
// instruction reduction (m31_dot2), and 72 registers for seven CTAs of 128 threads an SM.
// Calls one after another, us: 9999991 elements 82.9 -> 67.8, 2^24 133 -> 95 (5.6 TB/s, 86%
// of the measured copy rate); under the profiler 2^24 takes 139 -> 103. The kernel alone
// on 9999991: 65.5 with 8 elements a thread, 65.6 with 6, 71.6 with 4, 68.5 with 12, and
// 67.6-69.6 in CTAs of 256 threads.
__global__ void __launch_bounds__(BI_THREADS, 7) batch_inverse_qm31_norm_kernel(const qm31 *__restrict__ src,
                                                                                qm31 *__restrict__ dst, uint64_t n) {
    chain_wait();
    constexpr int E = BI_QM31_PER_THREAD;
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp_global = ((uint64_t)blockIdx.x * BI_THREADS + threadIdx.x) >> 5;
    const uint64_t base = warp_global * (32 * E) + lane;
    qm31 v[E];
    cm31 nrm[E];
    uint32_t pre[E], mag[E];
    uint32_t run = 1;
#pragma unroll
    for (int i = 0; i < E; i++) {
        const uint64_t idx = base + (uint64_t)i * 32;
        v[i] = (idx < n) ? src[idx] : qm31_one();
        const cm31 a2 = cm31_sqr(v[i].a), b2 = cm31_sqr(v[i].b);
        const cm31 rb2 = {m31_sub(m31_add(b2.a, b2.a), b2.b), m31_add(m31_add(b2.b, b2.b), b2.a)};  // R b^2
        nrm[i] = cm31_sub(a2, rb2);
        mag[i] = m31_dot2(nrm[i].a, nrm[i].a << 1, nrm[i].b, nrm[i].b << 1);
        run = m31_mul(run, mag[i]);
        pre[i] = run;
    }
    uint32_t r = m31_inv(run);
#pragma unroll
    for (int i = E - 1; i >= 0; i--) {
        const uint32_t minv = i > 0 ? m31_mul(r, pre[i - 1]) : r;  // 1 / |N_i|^2
        const uint64_t idx = base + (uint64_t)i * 32;
        r = m31_mul(r, mag[i]);
        // 1 / N_i = c + d i with c = N.a / |N|^2, d = -N.b / |N|^2; the products
        // (x + y i)(c + d i) = (x c + y (p - d)) + (x d + y c) i reduced once each, and
        // negated for the u part by the coefficients (p - c, p - d)
        const uint32_t c = m31_mul(nrm[i].a, minv), nd = m31_mul(nrm[i].b, minv);
        const uint32_t c2 = c << 1, nd2 = nd << 1, d2 = (P - nd) << 1, nc2 = (P - c) << 1;
        const qm31 z = v[i];
        const cm31 lo = {m31_dot2(z.a.a, c2, z.a.b, nd2), m31_dot2(z.a.a, d2, z.a.b, c2)};
        const cm31 nhi = {m31_dot2(z.b.a, nc2, z.b.b, d2), m31_dot2(z.b.a, nd2, z.b.b, nc2)};
        if (idx < n) dst[idx] = {lo, nhi};
    }
}

}  // namespace

int bit_reverse_async(uint32_t *col, uint64_t n, uint32_t words, cudaStream_t st) {
    STWO_REQUIRE(is_pow2(n) && n <= (1ull << 31), STWO_ERR_INVALID_ARGUMENT, "bit reverse of %llu elements",
                 (unsigned long long)n);
    STWO_REQUIRE(words == 1 || words == 4, STWO_ERR_INVALID_ARGUMENT, "element of %u words", words);
    uint32_t L = log2_u64(n);
    if (L < 10) {
        uint32_t blocks = (uint32_t)((n + 255) / 256);
        if (words == 1) bitrev_simple_kernel<1><<<blocks, 256, 0, st>>>(reinterpret_cast<Elem<1> *>(col), L);
        else bitrev_simple_kernel<4><<<blocks, 256, 0, st>>>(reinterpret_cast<Elem<4> *>(col), L);
        STWO_LAUNCH_CHECK("bitrev_simple_kernel");
        return STWO_OK;
    }
    // Middle indices b with b <= rev(b): built on the host once per device and size, and
    // cached (the cache is shared by all threads and streams, under a lock).
    static std::mutex mu;
    static std::map<std::pair<int, uint32_t>, std::pair<uint32_t *, uint32_t>> cache;
    int dev = 0;
    STWO_CUDA_TRY(cudaGetDevice(&dev));
    uint32_t *pairs = nullptr, cnt = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find({dev, L});
        if (it == cache.end()) {
            uint32_t mb = L - 10, m = 1u << mb;
            std::vector<uint32_t> h;
            h.reserve(m);
            for (uint32_t b = 0; b < m; b++)
                if (b <= bit_reverse_bits(b, mb)) h.push_back(b);
            uint32_t *d = nullptr;
            cudaError_t e = cudaMalloc(&d, sizeof(uint32_t) * h.size());
            if (e == cudaSuccess) e = cudaMemcpy(d, h.data(), sizeof(uint32_t) * h.size(), cudaMemcpyHostToDevice);
            if (e != cudaSuccess) return set_error(STWO_ERR_CUDA, "bit reverse table: %s", cudaGetErrorString(e));
            it = cache.emplace(std::make_pair(dev, L), std::make_pair(d, (uint32_t)h.size())).first;
        }
        pairs = it->second.first;
        cnt = it->second.second;
    }
    if (words == 1) bitrev_tiled_kernel<1><<<cnt, 256, 0, st>>>(col, L, pairs);
    else bitrev_tiled_kernel<4><<<cnt, 256, 0, st>>>(col, L, pairs);
    STWO_LAUNCH_CHECK("bitrev_tiled_kernel");
    return STWO_OK;
}

int batch_inverse_m31_async(const uint32_t *src, uint32_t *dst, uint64_t n, cudaStream_t st) {
    if (n == 0) return STWO_OK;
    uint64_t blocks = (n + BI_THREADS * BI_M31_PER_THREAD - 1) / (BI_THREADS * BI_M31_PER_THREAD);
    launch_chained(batch_inverse_m31_kernel, (unsigned)blocks, BI_THREADS, 0, st, src, dst, n);
    STWO_LAUNCH_CHECK("batch_inverse_m31_kernel");
    return STWO_OK;
}

int batch_inverse_qm31_async(const uint32_t *src, uint32_t *dst, uint64_t n, cudaStream_t st) {
    if (n == 0) return STWO_OK;
    uint64_t blocks = (n + BI_THREADS * BI_QM31_PER_THREAD - 1) / (BI_THREADS * BI_QM31_PER_THREAD);
    launch_chained(batch_inverse_qm31_norm_kernel, (unsigned)blocks, BI_THREADS, 0, st,
                   reinterpret_cast<const qm31 *>(src), reinterpret_cast<qm31 *>(dst), n);
    STWO_LAUNCH_CHECK("batch_inverse_qm31_norm_kernel");
    return STWO_OK;
}

}  // namespace stwo

using namespace stwo;

extern "C" {

int stwo_bit_reverse_m31(uint32_t *column, uint64_t n, void *stream) {
    return bit_reverse_async(column, n, 1, as_stream(stream));
}
int stwo_bit_reverse_qm31(uint32_t *column, uint64_t n, void *stream) {
    return bit_reverse_async(column, n, 4, as_stream(stream));
}
int stwo_batch_inverse_m31(const uint32_t *src, uint32_t *dst, uint64_t n, void *stream) {
    return batch_inverse_m31_async(src, dst, n, as_stream(stream));
}
int stwo_batch_inverse_qm31(const uint32_t *src, uint32_t *dst, uint64_t n, void *stream) {
    return batch_inverse_qm31_async(src, dst, n, as_stream(stream));
}

void bit_reverse_base_field(uint32_t *array, size_t size) { sync_default_stream(bit_reverse_async(array, size, 1, 0)); }
void bit_reverse_secure_field(uint32_t *array, size_t size) { sync_default_stream(bit_reverse_async(array, size, 4, 0)); }
void batch_inverse_base_field(const uint32_t *from, uint32_t *dst, size_t size) {
    sync_default_stream(batch_inverse_m31_async(from, dst, size, 0));
}
void batch_inverse_secure_field(const uint32_t *from, uint32_t *dst, size_t size) {
    sync_default_stream(batch_inverse_qm31_async(from, dst, size, 0));
}

}  // extern "C"
