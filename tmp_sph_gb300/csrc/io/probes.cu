// probes.cu — measurements of the resident state on the GPU: pressure probes, water-height
// gauges, the surge front and FP64 global reductions (mass, energy, extreme speed and density,
// the CFL step).
//
// Reference counterpart: output_fluid_file (src/io/io.cu:154-279) copies the whole state to
// the host every output interval and scans it there for the gauge heights (the largest z of
// fluid particles within 1.5 dx of a vertical line) and reads the pressure of four fixed
// particle indices.  Here one kernel scans the state where it lives and returns a few numbers;
// a pressure probe is a Shepard-normalised kernel average over the fluid around a point
// instead of the pressure of one particle, which has no fixed position in a Lagrangian flow.
//
// One launch of at most four blocks per SM strides over all particles.  GB300 runs FP64 at 1/64 of
// FP32, so only the two sums (v^2 and z) are formed in FP64 per particle; counts are integers,
// extremes are kept as the state's own type or as order-preserving integers, and a probe's FP64
// test runs only for the particles an FP32 test with a margin lets through.  4.96M particles, six
// probes: 624 us with every test and extreme in FP64, about 95 now (mixed precision 138; the state
// is read in 24).  Converting to FP64 by integer instructions was slower (159 against 138).
// Sums are accumulated per thread, then per warp with shuffles, per block in shared memory, then
// one global atomic per block and quantity.  The order-preserving map of a double onto a 64-bit
// unsigned integer lets atomicMax/atomicMin on the integers order the doubles.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <type_traits>

#include "sph_internal.h"

namespace sph {

namespace {

constexpr int PROBE_THREADS = 256;

struct ProbeSet {
    sph_probe p[SPH_MAX_PROBES];
    // half-widths of the FP32 box that holds every particle the FP64 test of a probe can pass:
    // its radius (kh for a pressure) and room for the rounding of positions and differences
    float wx[SPH_MAX_PROBES], wy[SPH_MAX_PROBES];
    int n;
};

__device__ __forceinline__ unsigned long long ord(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__host__ __device__ inline double unord(unsigned long long u) {
    const unsigned long long b = (u >> 63) ? (u & 0x7fffffffffffffffull) : ~u;
    double d;
    memcpy(&d, &b, sizeof(d));
    return d;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_down_sync(0xffffffffu, v, o);
        v = u > v ? u : v;
    }
    return v;
}
__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
    return ~warp_max(~v);
}

// Block reduction of one value with the warp reduction `op` (identity `id`), result valid in
// thread 0.  The leading barrier lets consecutive reductions reuse s_buf.
template <class V, class Op>
__device__ __forceinline__ V block_reduce(V v, unsigned long long* s_buf, Op op, V id) {
    V* buf = reinterpret_cast<V*>(s_buf);
    v = op(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) buf[w] = v;
    __syncthreads();
    V r = id;
    if (w == 0) {
        r = lane < PROBE_THREADS / 32 ? buf[lane] : id;
        r = op(r);
    }
    return r;
}

// Largest and smallest of values that are not NaN (as fmax and fmin take them), of the state's own
// type: FP32 values by FP32 comparisons, FP64 ones by their ordered integers.  Without any, -MOST
// and MOST.
constexpr double MOST = 1.0e300;
struct Extreme32 {
    float hi = -INFINITY, lo = INFINITY;
    __device__ __forceinline__ void add(float v) {
        hi = fmaxf(hi, v);
        lo = fminf(lo, v);
    }
    __device__ __forceinline__ unsigned long long top() const {
        return ord(hi == -INFINITY ? -MOST : (double)hi);
    }
    __device__ __forceinline__ unsigned long long bottom() const {
        return ord(lo == INFINITY ? MOST : (double)lo);
    }
};
struct Extreme64 {
    unsigned long long hi = ord(-MOST), lo = ord(MOST);
    __device__ __forceinline__ void add(double v) {
        const unsigned long long u = ord(v);
        if (u >= 0x000fffffffffffffull && u <= 0xfff0000000000000ull) {  // not NaN
            hi = u > hi ? u : hi;
            lo = u < lo ? u : lo;
        }
    }
    __device__ __forceinline__ unsigned long long top() const { return hi; }
    __device__ __forceinline__ unsigned long long bottom() const { return lo; }
};

// a == b of two doubles without an FP64 instruction (b is not NaN).
__device__ __forceinline__ bool same_value(double a, double b) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(a);
    const unsigned long long v = (unsigned long long)__double_as_longlong(b);
    return u == v || ((u | v) << 1) == 0ull;
}
__device__ __forceinline__ bool same_value(float a, double b) { return a == (float)b; }

// Accumulator layout (doubles / 64-bit words), ACC_WORDS in total:
enum {
    A_MASS = 0, A_KIN, A_POT, A_FLUID, A_PARKED,  // sums (doubles; counts summed as doubles)
    A_VMAX, A_RHOMAX, A_RHOMIN, A_FRONT,          // extremes (ordered 64-bit words)
    A_PROBE,                                      // per probe: num, den (doubles), max (word)
    ACC_WORDS = A_PROBE + 3 * SPH_MAX_PROBES
};

template <class P>
__global__ void __launch_bounds__(PROBE_THREADS)
k_probes(KParamsT<typename P::T> k, ParticleSetT<typename P::T> set, ProbeSet probes,
         double* __restrict__ acc) {
    __shared__ unsigned long long s_buf[PROBE_THREADS / 32];
    __shared__ double s_num[SPH_MAX_PROBES], s_den[SPH_MAX_PROBES];
    __shared__ unsigned long long s_max[SPH_MAX_PROBES];
    for (int q = threadIdx.x; q < probes.n; q += blockDim.x) {
        s_num[q] = 0.0;
        s_den[q] = 0.0;
        s_max[q] = 0ull;
    }
    __syncthreads();
    using R = typename std::conditional<P::kMixed, double, typename P::T>::type;  // positions
    using Extreme =
        typename std::conditional<std::is_same<R, float>::value, Extreme32, Extreme64>::type;
    const double mass = (double)k.mass, g = (double)k.g;
    const double kh2 = (double)k.kh * (double)k.kh, inv_h = 1.0 / (double)k.h;
    double v2s = 0.0, zs = 0.0;
    int fluid = 0, parked = 0;
    unsigned long long v2max = 0ull;  // bits of the largest v^2
    Extreme rho, front;               // rho: of rho - rho0 in mixed precision
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < k.n;
         i += (long)gridDim.x * blockDim.x) {
        const auto a = set.rec[2 * (size_t)i];
        const auto v = set.rec[2 * (size_t)i + 1];
        if (!(v.w > 0)) continue;  // fluid only
        R x, y, z, rr;
        if constexpr (P::kMixed) {
            const dvec4 xm = set.xm[i];  // FP64 position and rho - rho0
            x = xm.x;
            y = xm.y;
            z = xm.z;
            rr = xm.w;
        } else {
            x = a.x;
            y = a.y;
            z = a.z;
            rr = v.w;
        }
        const double vx = v.x, vy = v.y, vz = v.z;
        const double v2 = fma_rn(vz, vz, fma_rn(vy, vy, mul_rn(vx, vx)));
        fluid++;
        if (same_value(x, (double)k.park_x) && same_value(y, (double)k.park_y) &&
            same_value(z, (double)k.park_z))
            parked++;
        v2s = add_rn(v2s, v2);
        zs = add_rn(zs, (double)z);
        const unsigned long long b2 = (unsigned long long)__double_as_longlong(v2);
        if (b2 <= 0x7ff0000000000000ull && b2 > v2max) v2max = b2;
        rho.add(rr);
        front.add(x);
        const float xf = (float)x, yf = (float)y;
        for (int q = 0; q < probes.n; q++) {
            const sph_probe& pb = probes.p[q];
            if (!(fabsf(xf - pb.x) <= probes.wx[q] && fabsf(yf - pb.y) <= probes.wy[q])) continue;
            if (pb.kind == SPH_PROBE_PRESSURE) {
                const double dx = (double)x - pb.x, dy = (double)y - pb.y, dz = (double)z - pb.z;
                const double r2 = dx * dx + dy * dy + dz * dz;
                if (r2 < kh2) {
                    const double s = sqrt(r2) * inv_h, t = 1.0 - 0.5 * s;
                    const double w = (double)k.adh * t * t * t * t * (2.0 * s + 1.0);
                    atomicAdd(&s_num[q], (double)a.w * w);
                    atomicAdd(&s_den[q], w);
                }
            } else if (pb.kind == SPH_PROBE_HEIGHT) {
                if (fabs((double)x - pb.x) < pb.radius && fabs((double)y - pb.y) < pb.radius &&
                    (pb.zmax <= 0.f || z < pb.zmax))
                    atomicMax(&s_max[q], ord((double)z));
            }
        }
    }
    // block reductions, one global atomic per quantity
    auto sum = [](double v) { return warp_sum(v); };
    auto top = [](unsigned long long v) { return warp_max(v); };
    auto bottom = [](unsigned long long v) { return warp_min(v); };
    auto count = [](unsigned v) { return __reduce_add_sync(0xffffffffu, v); };
    const double b_v2 = block_reduce(v2s, s_buf, sum, 0.0);
    const double b_z = block_reduce(zs, s_buf, sum, 0.0);
    const unsigned b_fluid = block_reduce((unsigned)fluid, s_buf, count, 0u);
    const unsigned b_parked = block_reduce((unsigned)parked, s_buf, count, 0u);
    const unsigned long long b_vmax = block_reduce(v2max, s_buf, top, 0ull);
    const unsigned long long b_rmax = block_reduce(rho.top(), s_buf, top, 0ull);
    const unsigned long long b_rmin = block_reduce(rho.bottom(), s_buf, bottom, ~0ull);
    const unsigned long long b_front = block_reduce(front.top(), s_buf, top, 0ull);
    __syncthreads();
    if (threadIdx.x == 0 && b_fluid > 0u) {
        unsigned long long* u = reinterpret_cast<unsigned long long*>(acc);
        const double rho0 = P::kMixed ? (double)k.rho0 : 0.0;
        atomicAdd(&acc[A_MASS], mass * (double)b_fluid);
        atomicAdd(&acc[A_KIN], 0.5 * mass * b_v2);
        atomicAdd(&acc[A_POT], -mass * g * b_z);
        atomicAdd(&acc[A_FLUID], (double)b_fluid);
        if (b_parked) atomicAdd(&acc[A_PARKED], (double)b_parked);
        atomicMax(&u[A_VMAX], ord(sqrt(__longlong_as_double((long long)b_vmax))));
        atomicMax(&u[A_RHOMAX], ord(rho0 + unord(b_rmax)));
        atomicMin(&u[A_RHOMIN], ord(rho0 + unord(b_rmin)));
        atomicMax(&u[A_FRONT], b_front);
    }
    for (int q = threadIdx.x; q < probes.n; q += blockDim.x) {
        unsigned long long* u = reinterpret_cast<unsigned long long*>(acc);
        if (s_den[q] != 0.0) {
            atomicAdd(&acc[A_PROBE + 3 * q], s_num[q]);
            atomicAdd(&acc[A_PROBE + 3 * q + 1], s_den[q]);
        }
        if (s_max[q]) atomicMax(&u[A_PROBE + 3 * q + 2], s_max[q]);
    }
}

}  // namespace

size_t probe_acc_words() { return ACC_WORDS; }

template <class P>
cudaError_t launch_probes(const KParamsT<typename P::T>& k, const ParticleSetT<typename P::T>& set,
                          const sph_probe* probes, int nprobes, double* acc, cudaStream_t s) {
    if (nprobes < 0 || nprobes > SPH_MAX_PROBES) return cudaErrorInvalidValue;
    ProbeSet ps{};
    for (int q = 0; q < nprobes; q++) {
        ps.p[q] = probes[q];
        const float r = 1.00001f * (probes[q].kind == SPH_PROBE_PRESSURE ? (float)k.kh
                                                                         : probes[q].radius);
        ps.wx[q] = r + 1.0e-5f * std::fabs(probes[q].x);
        ps.wy[q] = r + 1.0e-5f * std::fabs(probes[q].y);
    }
    ps.n = nprobes;
    cudaError_t e = cudaMemsetAsync(acc, 0, ACC_WORDS * sizeof(double), s);
    if (e == cudaSuccess)  // rho_min starts at the largest ordered word
        e = cudaMemsetAsync(acc + A_RHOMIN, 0xff, sizeof(double), s);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long blocks = ((long)k.n + PROBE_THREADS - 1) / PROBE_THREADS;
    const long cap = 4L * (sms > 0 ? sms : 1);
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    k_probes<P><<<(int)blocks, PROBE_THREADS, 0, s>>>(k, set, ps, acc);
    return cudaGetLastError();
}

void probe_results(const double* acc, const sph_probe* probes, int nprobes, double cfl, double h,
                   double cs, sph_stats* stats, double* values) {
    const unsigned long long* u = reinterpret_cast<const unsigned long long*>(acc);
    const bool any = acc[A_FLUID] > 0.0;
    if (stats) {
        stats->fluid = (long long)acc[A_FLUID];
        stats->parked = (long long)acc[A_PARKED];
        stats->mass = acc[A_MASS];
        stats->kinetic = acc[A_KIN];
        stats->potential = acc[A_POT];
        stats->max_speed = any ? unord(u[A_VMAX]) : 0.0;
        stats->rho_max = any ? unord(u[A_RHOMAX]) : 0.0;
        stats->rho_min = any ? unord(u[A_RHOMIN]) : 0.0;
        stats->front_x = any ? unord(u[A_FRONT]) : 0.0;
        stats->cfl_dt = cfl * h / (cs + stats->max_speed);
    }
    for (int q = 0; values && q < nprobes; q++) {
        const double num = acc[A_PROBE + 3 * q], den = acc[A_PROBE + 3 * q + 1];
        const unsigned long long m = u[A_PROBE + 3 * q + 2];
        if (probes[q].kind == SPH_PROBE_FRONT)
            values[q] = any ? unord(u[A_FRONT]) : 0.0;
        else if (probes[q].kind == SPH_PROBE_PRESSURE)
            values[q] = den != 0.0 ? num / den : 0.0;
        else
            values[q] = m ? unord(m) : 0.0;
    }
}

#define SPH_PROBE_INSTANTIATE(P)                                                                \
    template cudaError_t launch_probes<P>(const KParamsT<P::T>&, const ParticleSetT<P::T>&,     \
                                          const sph_probe*, int, double*, cudaStream_t);
SPH_PROBE_INSTANTIATE(PrecF32)
SPH_PROBE_INSTANTIATE(PrecF64)
SPH_PROBE_INSTANTIATE(PrecMix)
SPH_PROBE_INSTANTIATE(PrecMixC)
SPH_PROBE_INSTANTIATE(PrecMixA)
#undef SPH_PROBE_INSTANTIATE

}  // namespace sph
