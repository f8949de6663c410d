// qs_state.cu — state-wide kernels: initialisation, measurement, read-back.
//
// Measurement replaces the two scalar passes of Register::try_measure
// (src/register.rs:306-339): a deterministic FP64 reduction of |a|^2 split by
// the target bit (fixed grid, warp shuffles, fixed-order block and grid
// combination), the outcome decision on the host, then one collapse sweep.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "qs_device.cuh"
#include "qs_kernels.h"

namespace qs {

static inline cudaError_t counted(cudaError_t e, uint64_t launches = 1) {
    if (e == cudaSuccess) note_launches(launches);
    return e;
}

constexpr int kT = 256;

static int grid_cap(uint64_t work, int sms, int per_thread = 1) {
    uint64_t b = (work + uint64_t(kT) * per_thread - 1) / (uint64_t(kT) * per_thread);
    uint64_t cap = uint64_t(sms) * 32;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return int(b);
}

__device__ __forceinline__ double2 to_d2(double2 v) { return v; }
__device__ __forceinline__ double2 to_d2(float2 v) { return make_double2(double(v.x), double(v.y)); }
// Reductions and the collapse read complex64 amplitudes through an integer-pipe conversion: the FP64
// pipe (~1/64 of the FP32 rate on GB300) is left to the sums and quotients themselves. Exact for
// every float (subnormals take a rare branch), so the values equal double(v).
__device__ __forceinline__ double2 to_d2_int(double2 v) { return v; }
__device__ __forceinline__ double2 to_d2_int(float2 v) { return make_double2(df_f2d(v.x), df_f2d(v.y)); }
__device__ __forceinline__ void from_d2(double2* dst, double2 v) { *dst = v; }
__device__ __forceinline__ void from_d2(float2* dst, double2 v) { *dst = make_float2(float(v.x), float(v.y)); }

// ---------------------------------------------------------------- initialisation
template <typename T>
__global__ void __launch_bounds__(kT) k_init_basis(T* __restrict__ st, uint64_t N, uint64_t index) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < N; i += stride) {
        double2 v = make_double2(i == index ? 1.0 : 0.0, 0.0);
        from_d2(&st[i], v);
    }
}

struct ProductArgs {
    int n;
    double q[64][4];  // qubit j: (re0, im0, re1, im1)
};

// Register::try_from_qubits folds kron(q_j, acc) from qubit 0 upwards
// (src/register.rs:91-96); amplitude i is q_{n-1}[b] * (... * (q_0[b] * 1)),
// each product rounded as num-complex does.
template <typename T>
__global__ void __launch_bounds__(kT) k_init_product(T* __restrict__ st, uint64_t N,
                                                     const __grid_constant__ ProductArgs a) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < N; i += stride) {
        double2 acc = make_double2(1.0, 0.0);
        for (int j = 0; j < a.n; j++) {
            const int b = int((i >> j) & 1ull);
            acc = cmul_exact(a.q[j][2 * b], a.q[j][2 * b + 1], acc);
        }
        from_d2(&st[i], acc);
    }
}

cudaError_t launch_init_basis(void* state, int n, int prec, uint64_t index, cudaStream_t s, int sms) {
    const uint64_t N = 1ull << n;
    if (prec == QS_PREC_C64)
        k_init_basis<float2><<<grid_cap(N, sms), kT, 0, s>>>((float2*)state, N, index);
    else
        k_init_basis<double2><<<grid_cap(N, sms), kT, 0, s>>>((double2*)state, N, index);
    return counted(cudaGetLastError());
}

// One doubling level of the same fold: the partial product after qubits 0..j-1 depends only on the
// low j bits of the index, so st[0, half) holding those partials becomes
// st[b * half + k] = q_j[b] * st[k] for b = 0, 1: the very products the per-amplitude loop forms at
// step j, computed once per partial instead of once per amplitude.
__global__ void __launch_bounds__(kT) k_product_level(double2* __restrict__ st, uint64_t half, double q0r, double q0i,
                                                      double q1r, double q1i) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t k = uint64_t(blockIdx.x) * kT + threadIdx.x; k < half; k += stride) {
        const double2 v = st[k];
        st[k + half] = cmul_exact(q1r, q1i, v);
        st[k] = cmul_exact(q0r, q0i, v);
    }
}

cudaError_t launch_init_product(void* state, int n, int prec, const double* qubits, cudaStream_t s, int sms) {
    ProductArgs a;
    std::memset(&a, 0, sizeof(a));
    // complex128: the first 16 qubits per amplitude, the rest by doubling levels (2^(n+1) products
    // in all instead of n * 2^n). complex64 keeps the whole product in double and rounds it once.
    const int n0 = (prec == QS_PREC_C64) ? n : std::min(n, 16);
    a.n = n0;
    for (int j = 0; j < n0; j++)
        for (int c = 0; c < 4; c++) a.q[j][c] = qubits[4 * j + c];
    const uint64_t N0 = 1ull << n0;
    if (prec == QS_PREC_C64) {
        k_init_product<float2><<<grid_cap(N0, sms), kT, 0, s>>>((float2*)state, N0, a);
        return counted(cudaGetLastError());
    }
    k_init_product<double2><<<grid_cap(N0, sms), kT, 0, s>>>((double2*)state, N0, a);
    cudaError_t e = counted(cudaGetLastError());
    for (int j = n0; j < n && e == cudaSuccess; j++) {
        const uint64_t half = 1ull << j;
        const double* q = qubits + 4 * j;
        k_product_level<<<grid_cap(half, sms), kT, 0, s>>>((double2*)state, half, q[0], q[1], q[2], q[3]);
        e = counted(cudaGetLastError());
    }
    return e;
}

// ---------------------------------------------------------------- measurement
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block sum of (a, b) in a fixed order; result valid in thread 0.
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double sa[kT / 32], sb[kT / 32];
    a = warp_sum(a);
    b = warp_sum(b);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        sa[w] = a;
        sb[w] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double ta = 0.0, tb = 0.0;
        for (int i = 0; i < kT / 32; i++) {
            ta += sa[i];
            tb += sb[i];
        }
        a = ta;
        b = tb;
    }
}

// A measurement visits the pairs (i0, i0 | tb) of its target inside the register's live subspace:
// amplitudes whose collapsed qubits (earlier measurements, no gate on them since) differ from the
// recorded outcomes are exact zeros, so they add nothing to a probability sum and a collapse leaves
// them as they are. The pair index t expands to i0 with the target bit 0 and the collapsed bits at
// their values.
static IndexMap subspace_map(int target, uint64_t zmask, uint64_t zval) {
    IndexMap m;
    std::memset(&m, 0, sizeof(m));
    const uint64_t pos = (zmask & ~(1ull << target)) | (1ull << target);
    int k = 0;
    for (int b = 0; b < 64; b++)
        if (pos >> b & 1ull) m.pos[k++] = uint8_t(b);
    m.npos = k;
    m.fixval = zval & zmask & ~(1ull << target);
    return m;
}

static uint64_t subspace_pairs(int n, int target, uint64_t zmask) {
    return 1ull << (n - 1 - __builtin_popcountll(zmask & ~(1ull << target)));
}

// Sums of squares of complex64 amplitudes, split by a bit, without the FP64 pipe (64 cycles per warp
// instruction and sub-partition on sm_103a, where conversion, square and sum of an amplitude took five). The
// square of a float is a 48-bit integer at an even power of two, so a thread adds squares as 64-bit integers
// on a scale set by the largest amplitude seen: kSqGuard bits below the unit of that amplitude's square, and
// one binade above it for larger ones to come (2^-54 of its square is the unit). At most kSqChunks chunks
// (128 squares, 2^63) go into one integer before it is added to the FP64 sum, so what is cut off is no more
// than what the FP64 additions that it replaces would round.
// 30 qubits, the first sums (2^30 amplitudes): 3.63 ms to 2.46 ms, bound by the integer pipe now.
constexpr int kSqChunk = 8;    // amplitudes of a thread per chunk, their loads in flight together
constexpr int kSqChunks = 8;   // chunks per FP64 addition
constexpr int kSqGuard = 10;
constexpr int kSqBlocks = 4;   // resident blocks per SM
constexpr uint32_t kSqTop = 0x7f800000u;           // infinities and NaN: summed in FP64
constexpr uint32_t kSqLow = uint32_t(48) << 23;    // a chunk with nothing of 2^-79 or more: in FP64 too

struct SquareSum {  // of one value of the bit: the rarer outcome keeps its own scale
    unsigned long long s = 0;
    uint32_t e = 48;  // biased exponent of the scale; zeros and subnormals shift out of any scale used
    int chunks = 0;
    double p = 0.0;

    __device__ __forceinline__ void flush() {
        // unit: 2^(2 (e - 150) - kSqGuard)
        p = fma(__ull2double_rn(s), __hiloint2double(int(uint32_t(1023 + 2 * (int(e) - 150) - kSqGuard) << 20), 0), p);
        s = 0;
        chunks = 0;
    }
    // before a chunk whose largest component has the bits `top` (sign cleared)
    __device__ __forceinline__ void open(uint32_t top) {
        const uint32_t et = (top >> 23) + 1u;
        if (et > e || chunks == kSqChunks) {
            flush();
            e = max(et, 48u);
        }
        chunks++;
    }
};

// the square of the component with the bits a (sign cleared) on the scale of exponent e
__device__ __forceinline__ unsigned long long scaled_square(uint32_t a, uint32_t e) {
    const uint32_t m = ((a & 0x007fffffu) | 0x00800000u) << (kSqGuard / 2);
    unsigned long long q;
    asm("{\n\t.reg .u64 w;\n\tmul.wide.u32 w, %1, %1;\n\tshr.u64 %0, w, %2;\n\t}"
        : "=l"(q)
        : "r"(m), "r"(2u * (e - (a >> 23))));
    return q;
}

// A chunk's largest component (bits, sign cleared) allows integers: 0, or of a normal size.
__device__ __forceinline__ bool top_fits(uint32_t top) { return top == 0u || top - kSqLow < kSqTop - kSqLow; }

__device__ __forceinline__ uint32_t abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

__global__ void __launch_bounds__(kT) k_prob_partials(const double2* __restrict__ st, uint64_t npairs, uint64_t tb,
                                                      const __grid_constant__ IndexMap map,
                                                      double* __restrict__ partials) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    double p0 = 0.0, p1 = 0.0;
    for (uint64_t t = uint64_t(blockIdx.x) * kT + threadIdx.x; t < npairs; t += stride) {
        const uint64_t i0 = expand_index(t, map);
        const double2 a = st[i0];
        const double2 b = st[i0 | tb];
        p0 = fma(a.x, a.x, p0);
        p0 = fma(a.y, a.y, p0);
        p1 = fma(b.x, b.x, p1);
        p1 = fma(b.y, b.y, p1);
    }
    block_sum2(p0, p1);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = p0;
        partials[2 * blockIdx.x + 1] = p1;
    }
}

// The same on complex64: chunks of kSqChunk / 2 pairs per thread.
__global__ void __launch_bounds__(kT, kSqBlocks)
    k_prob_partials_c64(const float2* __restrict__ st, uint64_t npairs, uint64_t tb, const __grid_constant__ IndexMap map,
                        double* __restrict__ partials) {
    constexpr int P = kSqChunk / 2;
    const uint64_t stride = uint64_t(gridDim.x) * (kT * P);
    SquareSum sum0, sum1;
    for (uint64_t t0 = uint64_t(blockIdx.x) * (kT * P) + threadIdx.x; t0 < npairs; t0 += stride) {
        float2 v[kSqChunk];
        uint32_t top0 = 0, top1 = 0;
#pragma unroll
        for (int j = 0; j < P; j++) {
            const uint64_t t = t0 + uint64_t(j) * kT;
            v[2 * j] = v[2 * j + 1] = make_float2(0.0f, 0.0f);
            if (t < npairs) {
                const uint64_t i0 = expand_index(t, map);
                v[2 * j] = st[i0];
                v[2 * j + 1] = st[i0 | tb];
            }
        }
#pragma unroll
        for (int j = 0; j < P; j++) {
            top0 = max(top0, max(abs_bits(v[2 * j].x), abs_bits(v[2 * j].y)));
            top1 = max(top1, max(abs_bits(v[2 * j + 1].x), abs_bits(v[2 * j + 1].y)));
        }
        if (top_fits(top0) && top_fits(top1)) {
            sum0.open(top0);
            sum1.open(top1);
#pragma unroll
            for (int j = 0; j < P; j++) {
                sum0.s += scaled_square(abs_bits(v[2 * j].x), sum0.e) + scaled_square(abs_bits(v[2 * j].y), sum0.e);
                sum1.s +=
                    scaled_square(abs_bits(v[2 * j + 1].x), sum1.e) + scaled_square(abs_bits(v[2 * j + 1].y), sum1.e);
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < P; j++) {
                const uint64_t t = t0 + uint64_t(j) * kT;
                if (t >= npairs) break;
                const uint64_t i0 = expand_index(t, map);
                const double2 a = to_d2_int(st[i0]), b = to_d2_int(st[i0 | tb]);
                sum0.p += fma(a.x, a.x, a.y * a.y);
                sum1.p += fma(b.x, b.x, b.y * b.y);
            }
        }
    }
    sum0.flush();
    sum1.flush();
    block_sum2(sum0.p, sum1.p);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = sum0.p;
        partials[2 * blockIdx.x + 1] = sum1.p;
    }
}

__global__ void __launch_bounds__(kT) k_prob_final(const double* __restrict__ partials, int nblocks,
                                                   double* __restrict__ out) {
    double p0 = 0.0, p1 = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += kT) {
        p0 += partials[2 * b];
        p1 += partials[2 * b + 1];
    }
    block_sum2(p0, p1);
    if (threadIdx.x == 0) {
        out[0] = p0;
        out[1] = p1;
    }
}

// The probability sums in the reference's order (src/register.rs:306-315): norm_sqr = re*re + im*im
// rounded per operation, added to prob_0 or prob_1 one amplitude after another in index order, so
// acc = RN(acc + t) for every t of a chain (the squares with target bit 0, or 1). Taken literally
// that is a chain of FP64 additions, and sm_103a needs 64 cycles for each (8.6 ms for 2^18 squares).
// The same values come from integers: while acc stays in one binade, with ulp u, acc = A u for an
// integer A and RN(acc + t) = (A + d) u, where d is t / u rounded to nearest, ties to the even A + d.
// Only a tie looks at A, and only at its parity, so a run of squares is a pair of integers (what it
// adds to an even and to an odd A), and runs compose associatively. Because the squares are not
// negative, a run is right whenever it ends at A <= 2^53, the end of the binade; the one square that
// crosses it is added in FP64, and the next run starts in the next binade.
struct SeqRun {
    long long d0, d1;  // added to an even / odd A
};

constexpr long long kSeqTop = 1ll << 53;
constexpr long long kSeqHuge = 1ll << 55;  // a run that cannot end in the binade (saturated)

__device__ __forceinline__ SeqRun seq_compose(SeqRun a, SeqRun b) {  // a, then b
    SeqRun r;
    r.d0 = a.d0 + ((a.d0 & 1) ? b.d1 : b.d0);
    r.d1 = a.d1 + ((a.d1 & 1) ? b.d0 : b.d1);
    if (r.d0 > kSeqHuge) r.d0 = kSeqHuge;
    if (r.d1 > kSeqHuge) r.d1 = kSeqHuge;
    return r;
}

// One square t >= 0 (or an infinity or NaN: huge) against a binade with exponent field e >= 1.
__device__ __forceinline__ SeqRun seq_square(double t, int e) {
    const long long bits = __double_as_longlong(t);
    const int et = int(bits >> 52) & 0x7ff;
    long long m = bits & 0xfffffffffffffll;
    if (et) m |= 1ll << 52;
    const int sh = e - (et ? et : 1);
    SeqRun r;
    if (sh < 0 || et == 0x7ff) {  // above the binade
        r.d0 = r.d1 = m ? kSeqHuge : 0;
        return r;
    }
    if (sh > 53) {  // below half an ulp
        r.d0 = r.d1 = 0;
        return r;
    }
    const long long q = m >> sh, rem = m - (q << sh), half = sh ? 1ll << (sh - 1) : 1ll;
    const long long up = q + (rem > half ? 1 : 0);
    const bool tie = rem == half && sh;
    r.d0 = up + ((tie && (q & 1)) ? 1 : 0);
    r.d1 = up + ((tie && !(q & 1)) ? 1 : 0);
    return r;
}

// acc's binade as its exponent field, 0 when the integer form does not apply (zero, subnormal,
// infinite, NaN).
__device__ __forceinline__ int seq_binade(double acc) {
    const int e = int(__double_as_longlong(acc) >> 52) & 0x7ff;
    return e == 0x7ff ? 0 : e;
}
__device__ __forceinline__ long long seq_integer(double acc) {
    return (__double_as_longlong(acc) & 0xfffffffffffffll) | (1ll << 52);
}
__device__ __forceinline__ double seq_double(long long A, int e) {  // 2^52 <= A <= 2^53
    // A = 2^53 carries into the exponent field
    return __longlong_as_double((static_cast<long long>(e - 1) << 52) + A);
}

// acc after the squares t[0, len) (shared or global memory), by one warp; every lane returns it. A
// step takes 32 x kSeqLane squares; the step that leaves the binade keeps its squares up to the
// crossing one, adds that one in FP64 and continues behind it.
constexpr int kSeqLane = 8;
__device__ double seq_warp(double acc, const double* t, int len) {
    const int lane = threadIdx.x & 31;
    int at = 0;
    while (at < len) {
        const int e = seq_binade(acc);
        const int first = at + lane * kSeqLane;
        double v[kSeqLane];
#pragma unroll
        for (int j = 0; j < kSeqLane; j++) v[j] = first + j < len ? t[first + j] : 0.0;
        if (e == 0) {
            if (!(acc < __longlong_as_double(0x7ffll << 52))) {  // infinite or NaN: only a NaN changes it
                bool nan = false;
#pragma unroll
                for (int j = 0; j < kSeqLane; j++) nan |= v[j] != v[j];
                if (__ballot_sync(0xffffffffu, nan)) acc = __longlong_as_double(0x7ff8ll << 48);
                at += 32 * kSeqLane;
                continue;
            }
            int mine = kSeqLane;  // up to the first square that is not zero, which is added in FP64
#pragma unroll
            for (int j = kSeqLane - 1; j >= 0; j--)
                if (v[j] != 0.0) mine = j;
            const unsigned any = __ballot_sync(0xffffffffu, mine < kSeqLane);
            if (!any) {
                at += 32 * kSeqLane;
                continue;
            }
            const int l = __ffs(any) - 1;
            const int idx = at + l * kSeqLane + __shfl_sync(0xffffffffu, mine, l);
            acc = __dadd_rn(acc, t[idx]);
            at = idx + 1;
            continue;
        }
        SeqRun run = seq_square(v[0], e);
#pragma unroll
        for (int j = 1; j < kSeqLane; j++) run = seq_compose(run, seq_square(v[j], e));
        SeqRun incl = run;  // the runs of lanes 0..lane
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            SeqRun p;
            p.d0 = __shfl_up_sync(0xffffffffu, incl.d0, o);
            p.d1 = __shfl_up_sync(0xffffffffu, incl.d1, o);
            if (lane >= o) incl = seq_compose(p, incl);
        }
        const long long A = seq_integer(acc);
        const long long after = A + ((A & 1) ? incl.d1 : incl.d0);
        const unsigned over = __ballot_sync(0xffffffffu, after > kSeqTop);
        if (!over) {
            acc = seq_double(__shfl_sync(0xffffffffu, after, 31), e);
            at += 32 * kSeqLane;
            continue;
        }
        const int l = __ffs(over) - 1;  // the first lane whose squares leave the binade
        long long B = __shfl_sync(0xffffffffu, after, l ? l - 1 : 0);
        if (l == 0) B = A;
        int cross = kSeqLane;
        if (lane == l) {
            cross = 0;
#pragma unroll
            for (int j = 0; j < kSeqLane; j++) {
                const SeqRun q = seq_square(v[j], e);
                const long long C = B + ((B & 1) ? q.d1 : q.d0);
                if (cross == j && C <= kSeqTop) {
                    B = C;
                    cross = j + 1;
                }
            }
        }
        cross = __shfl_sync(0xffffffffu, cross, l);
        B = __shfl_sync(0xffffffffu, B, l);
        const int idx = at + l * kSeqLane + cross;
        acc = __dadd_rn(seq_double(B, e), t[idx]);
        at = idx + 1;
    }
    return acc;
}

// One block for both chains, chunk after chunk of squares in shared memory: what registers of up to
// 13 qubits take (4096 squares: 5 us against 28 us for the additions one by one), and larger ones
// when the scratch of the three-kernel form below cannot be had.
constexpr int kSeqChunk = 2048;  // pairs per chunk
__global__ void __launch_bounds__(1024) k_prob_seq_block(const double2* __restrict__ st, uint64_t npairs, uint64_t tb,
                                                         const __grid_constant__ IndexMap map,
                                                         double* __restrict__ out) {
    __shared__ double sq[2][kSeqChunk];
    double acc = 0.0;  // warp 0: prob_0, warp 1: prob_1
    for (uint64_t base = 0; base < npairs; base += kSeqChunk) {
        const int len = int(npairs - base < uint64_t(kSeqChunk) ? npairs - base : uint64_t(kSeqChunk));
        for (int j = threadIdx.x; j < 2 * len; j += blockDim.x) {
            const int c = j >= len, k = c ? j - len : j;
            const double2 a = st[expand_index(base + uint64_t(k), map) | (c ? tb : 0ull)];
            sq[c][k] = __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
        }
        __syncthreads();
        if (threadIdx.x < 64) acc = seq_warp(acc, sq[threadIdx.x >> 5], len);
        __syncthreads();
    }
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) out[threadIdx.x >> 5] = acc;
}

// The same on the whole chip, for larger registers: (1) every square, and the sum of every group of
// kSeqGroup of them; (2) each group's run in the binade that the sums before it predict; (3) one warp
// per chain composes the groups, 32 at a time, and goes through a group square by square (seq_warp)
// only where the binade changes or was not the predicted one. A wrong prediction costs time, not
// the result. 2^18 pairs take 20 us (single SM: its FP64 pipe takes 200 us for the squares alone).
constexpr int kSeqGroup = 512;
struct SeqGroup {
    SeqRun run;
    long long e;  // the binade's exponent field, 0: none, -1: every square is zero (any acc)
};

__global__ void __launch_bounds__(kT) k_seq_squares(const double2* __restrict__ st, uint64_t npairs, uint64_t tb,
                                                    const __grid_constant__ IndexMap map, double* __restrict__ sq,
                                                    float* __restrict__ sums) {
    const uint64_t groups = npairs / kSeqGroup;  // per chain
    const uint64_t w = uint64_t(blockIdx.x) * (kT / 32) + (threadIdx.x >> 5);
    if (w >= 2 * groups) return;
    const int lane = threadIdx.x & 31;
    const bool one = w >= groups;
    const uint64_t p0 = (one ? w - groups : w) * kSeqGroup;
    float s = 0.0f;
    bool any = false;
#pragma unroll 4
    for (int j = lane; j < kSeqGroup; j += 32) {
        const double2 a = st[expand_index(p0 + uint64_t(j), map) | (one ? tb : 0ull)];
        const double v = __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
        sq[w * kSeqGroup + j] = v;
        s += float(v);
        any |= v != 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    any = __ballot_sync(0xffffffffu, any) != 0u;
    if (lane == 0) sums[w] = any ? s : -0.0f;  // -0: a group of zeros
}

__global__ void __launch_bounds__(kT) k_seq_groups(const double* __restrict__ sq, uint64_t groups,
                                                   const float* __restrict__ sums, SeqGroup* __restrict__ out) {
    const uint64_t w = uint64_t(blockIdx.x) * (kT / 32) + (threadIdx.x >> 5);
    if (w >= 2 * groups) return;
    const int lane = threadIdx.x & 31;
    if (__float_as_uint(sums[w]) == 0x80000000u) {
        if (lane == 0) out[w] = SeqGroup{{0, 0}, -1};
        return;
    }
    float s = 0.0f;  // the sum of the chain before this group
    for (uint64_t g = (w >= groups ? groups : 0) + lane; g < w; g += 32) s += sums[g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const uint32_t fe = (__float_as_uint(s) >> 23) & 0xffu;
    const int e = (fe == 0u || fe == 255u) ? 0 : int(fe) + 896;
    SeqRun run{0, 0};
    if (e) {
        constexpr int per = kSeqGroup / 32;
        const double2* t = reinterpret_cast<const double2*>(sq + w * kSeqGroup + lane * per);
#pragma unroll
        for (int j = 0; j < per / 2; j++) {
            const double2 v = t[j];
            run = seq_compose(run, seq_compose(seq_square(v.x, e), seq_square(v.y, e)));
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            SeqRun p;
            p.d0 = __shfl_down_sync(0xffffffffu, run.d0, o);
            p.d1 = __shfl_down_sync(0xffffffffu, run.d1, o);
            if (lane + o < 32) run = seq_compose(run, p);
        }
    }
    if (lane == 0) out[w] = SeqGroup{run, e};
}

__global__ void __launch_bounds__(64) k_seq_resolve(const double* __restrict__ sq, uint64_t groups,
                                                    const SeqGroup* __restrict__ runs, double* __restrict__ out) {
    const int lane = threadIdx.x & 31, chain = threadIdx.x >> 5;
    sq += uint64_t(chain) * groups * kSeqGroup;
    runs += uint64_t(chain) * groups;
    double acc = 0.0;
    uint64_t g = 0;
    while (g < groups) {
        const int e = seq_binade(acc);
        SeqGroup mine{{0, 0}, 0};
        if (g + lane < groups) mine = runs[g + lane];
        bool ok = mine.e == -1 || (e != 0 && mine.e == e);
        SeqRun incl = mine.run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            SeqRun p;
            p.d0 = __shfl_up_sync(0xffffffffu, incl.d0, o);
            p.d1 = __shfl_up_sync(0xffffffffu, incl.d1, o);
            if (lane >= o) incl = seq_compose(p, incl);
        }
        const long long A = seq_integer(acc);
        const long long after = A + ((A & 1) ? incl.d1 : incl.d0);
        ok = ok && (e == 0 || after <= kSeqTop);
        const unsigned bad = ~__ballot_sync(0xffffffffu, ok);
        const int n = bad ? __ffs(bad) - 1 : 32;  // groups taken as they are
        if (n > 0 && e != 0) acc = seq_double(__shfl_sync(0xffffffffu, after, n - 1), e);
        g += n;
        if (n < 32 && g < groups) {
            acc = seq_warp(acc, sq + g * kSeqGroup, kSeqGroup);
            g++;
        }
    }
    if (lane == 0) out[chain] = acc;
}

// The three kernels take whole groups; smaller subspaces take the one-block kernel.
constexpr uint64_t kSeqGridPairs = 4096;
static_assert(kSeqGridPairs % kSeqGroup == 0, "whole groups");
static_assert((sizeof(float) + sizeof(SeqGroup)) * 2 * ((1u << 19) / kSeqGroup) <= 2 * 4096 * sizeof(double),
              "the group tables of a 20-qubit register fit the partials");

cudaError_t launch_measure_probs(const void* state, int n, int prec, int target, double* partials,
                                 int max_partials, double* out, cudaStream_t s, int sms, uint64_t zmask,
                                 uint64_t zval, bool sequential, double* squares) {
    const IndexMap map = subspace_map(target, zmask, zval);
    const uint64_t npairs = subspace_pairs(n, target, zmask);
    const uint64_t tb = 1ull << target;
    if (sequential && prec == QS_PREC_C128) {
        const double2* st = static_cast<const double2*>(state);
        const uint64_t groups = npairs / kSeqGroup;
        const size_t table = 2 * groups * sizeof(SeqGroup);
        if (squares && npairs >= kSeqGridPairs &&
            table + 2 * groups * sizeof(float) <= 2 * size_t(max_partials) * sizeof(double)) {
            SeqGroup* runs = reinterpret_cast<SeqGroup*>(partials);
            float* sums = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(partials) + table);
            const int grid = int((2 * groups + kT / 32 - 1) / (kT / 32));
            k_seq_squares<<<grid, kT, 0, s>>>(st, npairs, tb, map, squares, sums);
            k_seq_groups<<<grid, kT, 0, s>>>(squares, groups, sums, runs);
            k_seq_resolve<<<1, 64, 0, s>>>(squares, groups, runs, out);
            return counted(cudaGetLastError(), 3);
        }
        const int threads = int(std::min<uint64_t>(1024, std::max<uint64_t>(64, 2 * npairs)));
        k_prob_seq_block<<<1, (threads + 31) / 32 * 32, 0, s>>>(st, npairs, tb, map, out);
        return counted(cudaGetLastError());
    }
    int grid = grid_cap(npairs, sms, 4);
    if (prec == QS_PREC_C64) grid = std::min(grid, kSqBlocks * sms);  // one wave
    if (grid > max_partials) grid = max_partials;
    if (prec == QS_PREC_C64)
        k_prob_partials_c64<<<grid, kT, 0, s>>>((const float2*)state, npairs, tb, map, partials);
    else
        k_prob_partials<<<grid, kT, 0, s>>>((const double2*)state, npairs, tb, map, partials);
    k_prob_final<<<1, kT, 0, s>>>(partials, grid, out);
    return counted(cudaGetLastError(), 2);
}

// How the kept amplitudes are divided by d = sqrt(total). Complex128: the correctly rounded quotient (Rust's `/`)
// on the integer pipe (quotient). Complex64: as a pair of floats, one FP64 multiply by RN(1/d), or a true division
// where RN(1/d) is not usable.
constexpr int kDivTrue = 1, kDivMul = 2, kDivPair = 3;

// d for integer quotients: with the 53-bit significands mx and md, mx / md 2^62 is the upper half of 2^11 mx times
// r = floor(2^115 / md), or up to 2 less.
struct Divisor {
    double d, rinv;
    uint32_t rh, rl;
    uint32_t low, span;  // exponent fields (<< 20) of x that give a normal quotient
    int32_t base;        // of the quotient's high word, beside x's exponent
};

static Divisor make_divisor(double d, double rinv) {
    Divisor v;
    std::memset(&v, 0, sizeof(v));
    v.d = d;
    v.rinv = rinv;
    uint64_t bits;
    std::memcpy(&bits, &d, 8);
    const int e = int(bits >> 52);  // the sign is clear, or d is a NaN
    if (!(std::isfinite(rinv) && d > 1e-300 && std::isfinite(d))) return v;  // span 0: true divisions
    const uint64_t md = (bits & 0xfffffffffffffull) | (1ull << 52);
    // 2^115 / md by long division: at most 2^63
    uint64_t q = 0, rem = 0;
    for (int i = 115; i >= 0; i--) {
        rem = (rem << 1) | (i == 115 ? 1u : 0u);
        q <<= 1;
        if (rem >= md) rem -= md, q |= 1;
    }
    v.rh = uint32_t(q >> 32);
    v.rl = uint32_t(q);
    // from 2^-959 up: quotient_rare's remainder x - q d is a multiple of ulp(q) ulp(d) >= 2^-105 x, which has to be
    // a double too (2^-1074 and more)
    const int lo = std::max(64, e - 1020), hi = std::min(2046, e + 1020);
    v.low = uint32_t(lo) << 20;
    v.span = uint32_t(std::max(0, hi - lo + 1)) << 20;
    v.base = (1021 - e) * (1 << 20);
    return v;
}

// x / d where the integers do not say: a quotient so near to the middle of two doubles that its missing part
// decides (Markstein's step: with q = RN(x rinv) within an ulp, r = x - q d exactly by FMA, RN(q + r rinv) is the
// correctly rounded quotient; P. Markstein, IBM J. Res. Dev. 34(1), 1990), and what is not normal.
__device__ __noinline__ double quotient_rare(double x, double d, double rinv, bool middle) {
    if (!middle) return x / d;
    const double q = x * rinv;
    return fma(fma(-q, d, x), rinv, q);
}

// The correctly rounded x / d: Q = mx / md 2^62 to within 2 below, rounded at bit 9 or 10. A quotient of two 53-bit
// significands is never the middle of two doubles, so only Q's lower bits just below the middle are undecided (1 in
// 512). FP64 took 3 instructions a component, at 64 cycles per warp and sub-partition: 27 qubits, every qubit
// measured, 2.85 ms in the collapses then, 1.45 ms now (their traffic: 0.95 ms).
__device__ __forceinline__ double quotient(double x, const Divisor& v) {
    const uint32_t hi = uint32_t(__double2hiint(x)), lo = uint32_t(__double2loint(x)), h = hi & 0x7fffffffu;
    if (h - v.low >= v.span) return (h | lo) == 0u && v.span ? x : quotient_rare(x, v.d, v.rinv, false);
    const uint32_t xh = __funnelshift_l(lo, hi, 11) | 0x80000000u, xl = lo << 11;
    const uint64_t t = im_madw(xl, v.rl, 0ull);
    const uint64_t u = im_madw(xh, v.rl, t >> 32);
    const uint64_t w = im_madw(xl, v.rh, u & 0xffffffffull);
    const uint64_t Q = im_madw(xh, v.rh, u >> 32) + (w >> 32);
    const uint32_t top = uint32_t(Q >> 62);  // 1: the quotient of the significands is 1 or more
    const uint64_t q = Q << (1u - top);
    if ((uint32_t(q) & 1023u) == 510u + top) return quotient_rare(x, v.d, v.rinv, true);
    const uint64_t r = (q + 512u) >> 10;  // the implicit bit (and a carry) adds to the exponent
    const uint32_t rh = uint32_t(r >> 32) + (h & 0x7ff00000u) + uint32_t(v.base) + (top << 20);
    return __hiloint2double(int(rh | (hi & 0x80000000u)), int(uint32_t(r)));
}

// The kept amplitude divided by sqrt(total) (src/register.rs:337), in the state's type.
__device__ __forceinline__ double2 collapse_value(double2 v, const Divisor& d) {
    return make_double2(quotient(v.x, d), quotient(v.y, d));
}
template <int DIV>
__device__ __forceinline__ float2 collapse_value(float2 v, double d, double rinv, double2* as_double) {
    const double2 x = to_d2_int(v);
    float2 y;
    if constexpr (DIV == kDivTrue)
        y = make_float2(float(x.x / d), float(x.y / d));
    else  // rounded to float on the integer pipe
        y = make_float2(d2f_int(x.x * rinv), d2f_int(x.y * rinv));
    *as_double = make_double2(df_f2d(y.x), df_f2d(y.y));
    return y;
}

// Complex64 collapse on the FP32 and integer pipes. 1/d = rh + rl to 48 bits, so p = x rh rounded, its
// remainder x rh - p (exact) plus x rl, and p plus that sum is x / d within 2^-46 before its one rounding
// to a float: the value of the FP64 product, but where x / d lies that near to the middle of two floats (1 in 2^21).
// That holds for 2^-100 <= |p| < inf (below, the remainder
// would not be exact) and reciprocals that the host found within 2^+-60; a chunk with any other
// component but 0 takes the FP64 form of collapse_value. src(t) and dst(t) are the kept amplitude's places,
// drop(t) clears the other one, one(t) is the next target's bit. 30 qubits, all 30 collapses: 16.5 ms with five
// FP64 instructions an amplitude, 5.0 ms now.
constexpr uint32_t kPairLow = uint32_t(127 - 100) << 23;

__device__ __forceinline__ float pair_product(float x, float rh, float rl) {
    const float p = x * rh;
    const float y = p + fmaf(x, rl, fmaf(x, rh, -p));
    return __uint_as_float((__float_as_uint(y) & 0x7fffffffu) | (__float_as_uint(p) & 0x80000000u));  // keeps -0
}

template <int DIV, bool SUMS, typename Src, typename Dst, typename Drop, typename One>
__device__ __forceinline__ void collapse_chunks(uint64_t npairs, double d, double rinv, double* __restrict__ partials,
                                                Src src, Dst dst, Drop drop, One one) {
    const uint64_t stride = uint64_t(gridDim.x) * (kT * kSqChunk);
    const float rh = float(rinv), rl = float(rinv - double(rh));
    SquareSum sum0, sum1;
    for (uint64_t t0 = uint64_t(blockIdx.x) * (kT * kSqChunk) + threadIdx.x; t0 < npairs; t0 += stride) {
        bool fast = false;
        if constexpr (DIV == kDivPair) {
            float2 y[kSqChunk];
            uint32_t top0 = 0, top1 = 0, low = ~0u;
#pragma unroll
            for (int j = 0; j < kSqChunk; j++) {
                const uint64_t t = t0 + uint64_t(j) * kT;
                y[j] = make_float2(0.0f, 0.0f);
                if (t < npairs) y[j] = *src(t);
            }
#pragma unroll
            for (int j = 0; j < kSqChunk; j++) {
                y[j].x = pair_product(y[j].x, rh, rl);
                y[j].y = pair_product(y[j].y, rh, rl);
                const uint32_t a = abs_bits(y[j].x), b = abs_bits(y[j].y);
                const bool o = SUMS && one(t0 + uint64_t(j) * kT);
                top0 = max(top0, o ? 0u : max(a, b));
                top1 = max(top1, o ? max(a, b) : 0u);
                low = min(low, min(a - 1u, b - 1u));  // zeros don't count
            }
            fast = top_fits(top0) && top_fits(top1) && low >= kPairLow;
            if (fast) {
                if (SUMS) {
                    sum0.open(top0);
                    sum1.open(top1);
                }
#pragma unroll
                for (int j = 0; j < kSqChunk; j++) {
                    const uint64_t t = t0 + uint64_t(j) * kT;
                    if (SUMS) {
                        const bool o = one(t);
                        const uint32_t e = o ? sum1.e : sum0.e;
                        const unsigned long long q = scaled_square(abs_bits(y[j].x), e) + scaled_square(abs_bits(y[j].y), e);
                        sum0.s += o ? 0ull : q;
                        sum1.s += o ? q : 0ull;
                    }
                    if (t < npairs) {
                        *dst(t) = y[j];
                        drop(t);
                    }
                }
            }
        }
        if (!fast) {
#pragma unroll 1
            for (int j = 0; j < kSqChunk; j++) {
                const uint64_t t = t0 + uint64_t(j) * kT;
                if (t >= npairs) break;
                double2 y;
                *dst(t) = collapse_value<DIV == kDivPair ? kDivMul : DIV>(*src(t), d, rinv, &y);
                drop(t);
                const double q = fma(y.x, y.x, y.y * y.y);
                const bool o = SUMS && one(t);
                sum0.p += o ? 0.0 : q;
                sum1.p += o ? q : 0.0;
            }
        }
    }
    if (SUMS) {
        sum0.flush();
        sum1.flush();
        block_sum2(sum0.p, sum1.p);
        if (threadIdx.x == 0) {
            partials[2 * blockIdx.x] = sum0.p;
            partials[2 * blockIdx.x + 1] = sum1.p;
        }
    }
}

// In place, as k_collapse.
template <int DIV, bool SUMS>
__global__ void __launch_bounds__(kT, kSqBlocks)
    k_collapse_c64(float2* st, uint64_t npairs, uint64_t tb, const __grid_constant__ IndexMap map, int outcome, double d,
                   double rinv, uint64_t next_tb, double* __restrict__ partials) {
    const uint64_t kb = outcome ? tb : 0;
    auto at = [&](uint64_t t) { return st + (expand_index(t, map) | kb); };
    collapse_chunks<DIV, SUMS>(npairs, d, rinv, partials, at, at,
                               [&](uint64_t t) { st[expand_index(t, map) | (tb ^ kb)] = make_float2(0.0f, 0.0f); },
                               [&](uint64_t t) { return ((expand_index(t, map) | kb) & next_tb) != 0; });
}

template <bool SUMS>
static void collapse_c64(void* state, uint64_t npairs, uint64_t tb, const IndexMap& map, int outcome, double d,
                         double rinv, int mode, uint64_t ntb, double* partials, int grid, cudaStream_t s) {
    auto k = mode == kDivTrue ? k_collapse_c64<kDivTrue, SUMS>
             : mode == kDivMul ? k_collapse_c64<kDivMul, SUMS>
                               : k_collapse_c64<kDivPair, SUMS>;
    k<<<grid, kT, 0, s>>>(static_cast<float2*>(state), npairs, tb, map, outcome, d, rinv, ntb, partials);
}

// Grid of a collapse: shared by the in-place and the compact form, whose sums have to agree.
static int collapse_grid(uint64_t npairs, int prec, int sms) {
    return prec == QS_PREC_C64 ? std::min(grid_cap(npairs, sms, kSqChunk), kSqBlocks * sms) : grid_cap(npairs, sms, 2);
}

// In place on complex128. With SUMS, the collapse of one measurement fused with the probability sums of the next
// one (measure_circuit, src/register.rs:371-377): the kept amplitudes, once divided, are the only non-zero
// amplitudes the next target sees, so their squares are summed by that target's bit in the same pass.
template <bool SUMS>
__global__ void __launch_bounds__(kT) k_collapse(double2* __restrict__ st, uint64_t npairs, uint64_t tb,
                                                 const __grid_constant__ IndexMap map, int outcome,
                                                 const __grid_constant__ Divisor d, uint64_t next_tb,
                                                 double* __restrict__ partials) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    double p0 = 0.0, p1 = 0.0;
    for (uint64_t t = uint64_t(blockIdx.x) * kT + threadIdx.x; t < npairs; t += stride) {
        const uint64_t i0 = expand_index(t, map);
        const uint64_t keep = outcome ? (i0 | tb) : i0, drop = outcome ? i0 : (i0 | tb);
        const double2 y = collapse_value(st[keep], d);
        st[keep] = y;
        st[drop] = make_double2(0.0, 0.0);
        if constexpr (SUMS) {
            const double q = fma(y.x, y.x, y.y * y.y);
            if (keep & next_tb)
                p1 += q;
            else
                p0 += q;
        }
    }
    if constexpr (SUMS) {
        block_sum2(p0, p1);
        if (threadIdx.x == 0) {
            partials[2 * blockIdx.x] = p0;
            partials[2 * blockIdx.x + 1] = p1;
        }
    }
}

// Complex64 multiplies by RN(1/d) unless it must divide: as a pair of floats where both fit well inside
// their range.
static int div_mode_c64(double d, double rinv) {
    if (!(std::isfinite(rinv) && d > 1e-300 && std::isfinite(d))) return kDivTrue;
    return rinv > 0x1p-60 && rinv < 0x1p60 ? kDivPair : kDivMul;
}

cudaError_t launch_collapse(void* state, int n, int prec, int target, int outcome, double d, double rinv,
                            cudaStream_t s, int sms, uint64_t zmask, uint64_t zval) {
    const IndexMap map = subspace_map(target, zmask, zval);
    const uint64_t npairs = subspace_pairs(n, target, zmask);
    const uint64_t tb = 1ull << target;
    const int grid = collapse_grid(npairs, prec, sms);
    if (prec == QS_PREC_C64)
        collapse_c64<false>(state, npairs, tb, map, outcome, d, rinv, div_mode_c64(d, rinv), 0, nullptr, grid, s);
    else
        k_collapse<false><<<grid, kT, 0, s>>>(static_cast<double2*>(state), npairs, tb, map, outcome,
                                              make_divisor(d, rinv), 0, nullptr);
    return counted(cudaGetLastError());
}

cudaError_t launch_collapse_probs(void* state, int n, int prec, int target, int outcome, double d, double rinv,
                                  int next_target, double* partials, int max_partials, double* out, cudaStream_t s,
                                  int sms, uint64_t zmask, uint64_t zval) {
    const IndexMap map = subspace_map(target, zmask, zval);
    const uint64_t npairs = subspace_pairs(n, target, zmask);
    const uint64_t tb = 1ull << target, ntb = 1ull << next_target;
    int grid = collapse_grid(npairs, prec, sms);
    if (grid > max_partials) grid = max_partials;
    if (prec == QS_PREC_C64)
        collapse_c64<true>(state, npairs, tb, map, outcome, d, rinv, div_mode_c64(d, rinv), ntb, partials, grid, s);
    else
        k_collapse<true><<<grid, kT, 0, s>>>(static_cast<double2*>(state), npairs, tb, map, outcome,
                                             make_divisor(d, rinv), ntb, partials);
    k_prob_final<<<1, kT, 0, s>>>(partials, grid, out);
    return counted(cudaGetLastError(), 2);
}

// ---------------------------------------------------------------- measurement on a compact subspace
// A measurement sequence on a dense state (qs_measure_sequence): after the first collapse the live
// amplitudes are strided through the state (the measured qubits' bits fixed), so in-place passes
// move whole 32-byte sectors for every live 16-byte amplitude. Here each pass instead reads the
// kept half of a buffer whose index runs over the free bits only and writes it, divided, densely
// into the next buffer; the sums of the next target come from the same pass. Every pass visits the
// pairs t in the order and with the grid of k_collapse (the free bits in ascending order, the
// target's bit inserted) and divides as it does, so the sums, outcomes and divided amplitudes are
// bit for bit those of the in-place passes.
template <bool SUMS>
__global__ void __launch_bounds__(kT) k_collapse_compact(const double2* __restrict__ src, double2* __restrict__ dst,
                                                         uint64_t npairs, const __grid_constant__ IndexMap map,
                                                         uint64_t keepbit, const __grid_constant__ Divisor d,
                                                         uint64_t next_bit, double* __restrict__ partials) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    double p0 = 0.0, p1 = 0.0;
    for (uint64_t t = uint64_t(blockIdx.x) * kT + threadIdx.x; t < npairs; t += stride) {
        const double2 y = collapse_value(src[expand_index(t, map) | keepbit], d);
        dst[t] = y;
        if constexpr (SUMS) {
            const double q = fma(y.x, y.x, y.y * y.y);
            if (t & next_bit)
                p1 += q;
            else
                p0 += q;
        }
    }
    if constexpr (SUMS) {
        block_sum2(p0, p1);
        if (threadIdx.x == 0) {
            partials[2 * blockIdx.x] = p0;
            partials[2 * blockIdx.x + 1] = p1;
        }
    }
}

template <int DIV, bool SUMS>
__global__ void __launch_bounds__(kT, kSqBlocks)
    k_collapse_compact_c64(const float2* __restrict__ src, float2* __restrict__ dst, uint64_t npairs,
                           const __grid_constant__ IndexMap map, uint64_t keepbit, double d, double rinv,
                           uint64_t next_bit, double* __restrict__ partials) {
    collapse_chunks<DIV, SUMS>(npairs, d, rinv, partials,
                               [&](uint64_t t) { return src + (expand_index(t, map) | keepbit); },
                               [&](uint64_t t) { return dst + t; }, [](uint64_t) {},
                               [&](uint64_t t) { return (t & next_bit) != 0; });
}

template <bool SUMS>
static void collapse_compact_c64(const void* src, void* dst, uint64_t npairs, const IndexMap& map, uint64_t keepbit,
                                 double d, double rinv, int mode, int next_pos, double* partials, int grid,
                                 cudaStream_t s) {
    auto k = mode == kDivTrue ? k_collapse_compact_c64<kDivTrue, SUMS>
             : mode == kDivMul ? k_collapse_compact_c64<kDivMul, SUMS>
                               : k_collapse_compact_c64<kDivPair, SUMS>;
    k<<<grid, kT, 0, s>>>(static_cast<const float2*>(src), static_cast<float2*>(dst), npairs, map, keepbit, d, rinv,
                          SUMS ? 1ull << next_pos : 0ull, partials);
}

cudaError_t launch_collapse_compact(const void* src, void* dst, int nfree, int prec, int pos, int outcome, double d,
                                    double rinv, int next_pos, double* partials, int max_partials, double* out,
                                    cudaStream_t s, int sms) {
    const IndexMap map = subspace_map(pos, 0, 0);
    const uint64_t npairs = 1ull << (nfree - 1);
    const uint64_t keepbit = outcome ? (1ull << pos) : 0ull;
    int grid = collapse_grid(npairs, prec, sms);
    if (next_pos >= 0 && grid > max_partials) grid = max_partials;  // the in-place pass's grid
    const uint64_t nb = next_pos >= 0 ? 1ull << next_pos : 0ull;
    if (prec == QS_PREC_C64) {
        const int mode = div_mode_c64(d, rinv);
        if (next_pos >= 0)
            collapse_compact_c64<true>(src, dst, npairs, map, keepbit, d, rinv, mode, next_pos, partials, grid, s);
        else
            collapse_compact_c64<false>(src, dst, npairs, map, keepbit, d, rinv, mode, 0, nullptr, grid, s);
    } else {
        auto k = next_pos >= 0 ? k_collapse_compact<true> : k_collapse_compact<false>;
        k<<<grid, kT, 0, s>>>(static_cast<const double2*>(src), static_cast<double2*>(dst), npairs, map, keepbit,
                              make_divisor(d, rinv), nb, partials);
    }
    if (next_pos < 0) return counted(cudaGetLastError());
    k_prob_final<<<1, kT, 0, s>>>(partials, grid, out);
    return counted(cudaGetLastError(), 2);
}

template <typename T>
__global__ void __launch_bounds__(kT) k_scatter_live(T* __restrict__ st, const T* __restrict__ src, uint64_t count,
                                                     const __grid_constant__ IndexMap map) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t t = uint64_t(blockIdx.x) * kT + threadIdx.x; t < count; t += stride) st[expand_index(t, map)] = src[t];
}

cudaError_t launch_scatter_live(void* state, const void* src, int n, int prec, uint64_t zmask, uint64_t zval,
                                cudaStream_t s, int sms) {
    IndexMap map;
    std::memset(&map, 0, sizeof(map));
    int k = 0;
    for (int b = 0; b < 64; b++)
        if (zmask >> b & 1ull) map.pos[k++] = uint8_t(b);
    map.npos = k;
    map.fixval = zval & zmask;
    const uint64_t count = 1ull << (n - k);
    const int grid = grid_cap(count, sms, 2);
    if (prec == QS_PREC_C64)
        k_scatter_live<float2><<<grid, kT, 0, s>>>((float2*)state, (const float2*)src, count, map);
    else
        k_scatter_live<double2><<<grid, kT, 0, s>>>((double2*)state, (const double2*)src, count, map);
    return counted(cudaGetLastError());
}

// ---------------------------------------------------------------- read-back
// norm_sqr = re*re + im*im, rounded as num-complex computes it.
template <typename T>
__global__ void __launch_bounds__(kT) k_norm_sqr(const T* __restrict__ st, uint64_t first, uint64_t count,
                                                 double* __restrict__ dst) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < count; i += stride) {
        const double2 a = to_d2(st[first + i]);
        dst[i] = __dadd_rn(__dmul_rn(a.x, a.x), __dmul_rn(a.y, a.y));
    }
}

cudaError_t launch_norm_sqr(const void* state, int prec, uint64_t first, uint64_t count, double* dst,
                            cudaStream_t s, int sms) {
    if (prec == QS_PREC_C64)
        k_norm_sqr<float2><<<grid_cap(count, sms), kT, 0, s>>>((const float2*)state, first, count, dst);
    else
        k_norm_sqr<double2><<<grid_cap(count, sms), kT, 0, s>>>((const double2*)state, first, count, dst);
    return counted(cudaGetLastError());
}

__global__ void __launch_bounds__(kT) k_f2_to_d2(const float2* __restrict__ st, uint64_t first, uint64_t count,
                                                 double2* __restrict__ dst) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < count; i += stride)
        dst[i] = to_d2(st[first + i]);
}
__global__ void __launch_bounds__(kT) k_d2_to_f2(float2* __restrict__ st, uint64_t first, uint64_t count,
                                                 const double2* __restrict__ src) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < count; i += stride)
        from_d2(&st[first + i], src[i]);
}

cudaError_t launch_to_c128(const void* state, int prec, uint64_t first, uint64_t count, double* dst,
                           cudaStream_t s, int sms) {
    if (prec != QS_PREC_C64) return cudaErrorInvalidValue;
    k_f2_to_d2<<<grid_cap(count, sms), kT, 0, s>>>((const float2*)state, first, count, (double2*)dst);
    return counted(cudaGetLastError());
}
cudaError_t launch_from_c128(void* state, int prec, uint64_t first, uint64_t count, const double* src,
                             cudaStream_t s, int sms) {
    if (prec != QS_PREC_C64) return cudaErrorInvalidValue;
    k_d2_to_f2<<<grid_cap(count, sms), kT, 0, s>>>((float2*)state, first, count, (const double2*)src);
    return counted(cudaGetLastError());
}

// PartialEq (src/register.rs:409-413): all(|a_i - b_i| < tol) with norm() = hypot.
template <typename TA, typename TB>
__global__ void __launch_bounds__(kT) k_count_diff(const TA* __restrict__ a, const TB* __restrict__ b, uint64_t N,
                                                   double tol, unsigned long long* count) {
    const uint64_t stride = uint64_t(gridDim.x) * kT;
    unsigned long long c = 0;
    for (uint64_t i = uint64_t(blockIdx.x) * kT + threadIdx.x; i < N; i += stride) {
        const double2 x = to_d2(a[i]), y = to_d2(b[i]);
        if (!(hypot(x.x - y.x, x.y - y.y) < tol)) c++;
    }
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

cudaError_t launch_count_diff(const void* a, const void* b, int n, int prec, double tol,
                              unsigned long long* count, cudaStream_t s, int sms) {
    const uint64_t N = 1ull << n;
    if (prec == QS_PREC_C64)
        k_count_diff<float2, float2><<<grid_cap(N, sms), kT, 0, s>>>((const float2*)a, (const float2*)b, N, tol,
                                                                     count);
    else
        k_count_diff<double2, double2><<<grid_cap(N, sms), kT, 0, s>>>((const double2*)a, (const double2*)b, N,
                                                                       tol, count);
    return counted(cudaGetLastError());
}

}  // namespace qs
