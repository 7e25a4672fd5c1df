// qm_kernels.cu -- per-gate, noise, reduction and sampling kernels of libqmb200.so
// (sm_100a).  The fused multi-gate pass kernel lives in qm_fused.cu.
//
// All kernels here are streaming passes bounded by HBM bandwidth: every amplitude is
// read and written at most once per launch with 16-byte (complex128) or 8-byte
// (complex64) accesses that are contiguous across a warp whenever the gate's target
// is not among the lowest qubits.
#include <cuda_runtime.h>

#include <algorithm>

#include "qm_device.cuh"
#include "qm_internal.h"

namespace qm {

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 2;  // independent pairs per thread (memory-level parallelism)

// Enumeration of the active pairs of one gate: the item index gets zero bits inserted at
// the target and every control position (ascending), then the controls are set.  Only
// pairs whose control bits are all one are visited, so controlled gates read and write
// only the amplitudes they change (CudaStateVectorKernel.cs:41-48 visits every pair and
// filters).
struct GateLaunch {
    uint32_t count;
    int32_t npos;
    int32_t pos[32];
    uint32_t set_mask;
    uint32_t target_bit;
    uint32_t swap_bit;
    int32_t a_is_one, d_is_one;
    double a[2], b[2], c[2], d[2];
};

__device__ __forceinline__ uint32_t first_of(const GateLaunch& L, uint32_t item) {
    uint32_t x = item;
    for (int i = 0; i < L.npos; ++i) x = insert_zero(x, L.pos[i]);
    return x | L.set_mask;
}

template <typename T, int KIND>
__global__ void __launch_bounds__(kThreads) k_gate(typename Vec2<T>::type* __restrict__ s, const GateLaunch L) {
    uint32_t base = (blockIdx.x * kThreads + threadIdx.x) * kItems;
    uint32_t firsts[kItems], seconds[kItems];
    bool live[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        uint32_t item = base + u;
        live[u] = item < L.count;
        uint32_t f = first_of(L, live[u] ? item : 0);
        uint32_t g = f | L.target_bit;
        if (KIND == QM_KERNEL_SWAP) g = (f ^ L.swap_bit) | L.target_bit;
        firsts[u] = f;
        seconds[u] = g;
    }
    if (KIND == QM_KERNEL_DIAGONAL) {
        T ar = (T)L.a[0], ai = (T)L.a[1], dr = (T)L.d[0], di = (T)L.d[1];
        Cx<T> x[kItems], y[kItems];
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            if (!live[u]) continue;
            if (!L.a_is_one) x[u] = load_amp<T>(s, firsts[u]);
            if (!L.d_is_one) y[u] = load_amp<T>(s, seconds[u]);
        }
#pragma unroll
        for (int u = 0; u < kItems; ++u) {
            if (!live[u]) continue;
            if (!L.a_is_one) store_amp<T>(s, firsts[u], cmul<T>(ar, ai, x[u]));
            if (!L.d_is_one) store_amp<T>(s, seconds[u], cmul<T>(dr, di, y[u]));
        }
        return;
    }
    Cx<T> x[kItems], y[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        if (!live[u]) continue;
        x[u] = load_amp<T>(s, firsts[u]);
        y[u] = load_amp<T>(s, seconds[u]);
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
        if (!live[u]) continue;
        Cx<T> o0, o1;
        if (KIND == QM_KERNEL_EXCHANGE || KIND == QM_KERNEL_SWAP) {
            o0 = y[u];
            o1 = x[u];
        } else if (KIND == QM_KERNEL_HADAMARD) {
            T h = (T)L.a[0];
            o0 = Cx<T>{h * x[u].re + h * y[u].re, h * x[u].im + h * y[u].im};
            o1 = Cx<T>{h * x[u].re - h * y[u].re, h * x[u].im - h * y[u].im};
        } else {
            o0 = cmac2<T>((T)L.a[0], (T)L.a[1], x[u], (T)L.b[0], (T)L.b[1], y[u]);
            o1 = cmac2<T>((T)L.c[0], (T)L.c[1], x[u], (T)L.d[0], (T)L.d[1], y[u]);
        }
        store_amp<T>(s, firsts[u], o0);
        store_amp<T>(s, seconds[u], o1);
    }
}

template <typename T>
cudaError_t launch_gate_t(void* amps, int qubits, const DevGate& g, cudaStream_t st) {
    GateLaunch L;
    uint32_t positions = g.target_bit | g.control_mask | g.swap_bit;
    L.npos = 0;
    for (int b = 0; b < 32; ++b)
        if (positions & (1u << b)) L.pos[L.npos++] = b;
    if (L.npos > qubits) return cudaErrorInvalidValue;
    L.count = (uint32_t)((1ull << qubits) >> L.npos);
    L.set_mask = g.control_mask | g.swap_bit;
    L.target_bit = g.target_bit;
    L.swap_bit = g.swap_bit;
    L.a_is_one = g.a_is_one;
    L.d_is_one = g.d_is_one;
    for (int i = 0; i < 2; ++i) {
        L.a[i] = g.a[i]; L.b[i] = g.b[i]; L.c[i] = g.c[i]; L.d[i] = g.d[i];
    }
    if (L.count == 0) return cudaSuccess;
    uint32_t per_block = kThreads * kItems;
    dim3 grid((L.count + per_block - 1) / per_block);
    auto* s = reinterpret_cast<typename Vec2<T>::type*>(amps);
    switch (g.kernel) {
    case QM_KERNEL_MATRIX: k_gate<T, QM_KERNEL_MATRIX><<<grid, kThreads, 0, st>>>(s, L); break;
    case QM_KERNEL_HADAMARD: k_gate<T, QM_KERNEL_HADAMARD><<<grid, kThreads, 0, st>>>(s, L); break;
    case QM_KERNEL_EXCHANGE: k_gate<T, QM_KERNEL_EXCHANGE><<<grid, kThreads, 0, st>>>(s, L); break;
    case QM_KERNEL_DIAGONAL:
        if (g.a_is_one && g.d_is_one) return cudaSuccess;
        k_gate<T, QM_KERNEL_DIAGONAL><<<grid, kThreads, 0, st>>>(s, L);
        break;
    case QM_KERNEL_SWAP: k_gate<T, QM_KERNEL_SWAP><<<grid, kThreads, 0, st>>>(s, L); break;
    default: return cudaSuccess;  // identity
    }
    return cudaGetLastError();
}

// Up to kSmallGates gates on a state of at most kSmallQubits qubits in one launch: the state sits in
// one block's shared memory and the gates run one after another, a pair of amplitudes per thread (up
// to four).  Such a state fills a fraction of one SM, so the serial chain bounds it: 0.2 to 0.4 us a
// gate (mask and coefficient loads, amplitude loads, four dependent multiply-adds, stores, a barrier).
// The barrier is of the warp while targets are among the lowest six qubits, whose pairs keep to 64
// amplitudes per warp (and 64 more per further pair).  Device time of a brick of depth 26, against one
// launch per gate (8 qubits: 1198 to 62 us for 299 gates) and passes of 16 amplitudes per thread, two
// warps or four in all (10 qubits: 221 to 104 us for 377 gates; 11: 249 to 178).
constexpr int kSmallThreads = 256;
static_assert(1 << (kSmallQubits - 1) <= 4 * kSmallThreads, "at most four pairs per thread");

struct SmallGate {
    int32_t kernel, target;
    uint32_t control, swap;
    double c[8];
};
template <int N>
struct SmallProgram {
    int32_t qubits, count;
    SmallGate gate[N];
};

// The gates travel as a kernel parameter: the constant cache feeds their masks and coefficients, and
// shared memory only the amplitudes.  At most eight warps, with PAIRS pairs per thread, since every
// warp loads every gate.
template <typename T, int N, int PAIRS>
__global__ void __launch_bounds__(kSmallThreads) k_small(typename Vec2<T>::type* __restrict__ s,
                                                         const __grid_constant__ SmallProgram<N> P) {
    extern __shared__ __align__(16) unsigned char smem[];
    using V = typename Vec2<T>::type;
    V* state = reinterpret_cast<V*>(smem);
    const uint32_t t = threadIdx.x, nt = blockDim.x, pairs = 1u << (P.qubits - 1);
    for (uint32_t i = t; i < 2 * pairs; i += nt) state[i] = s[i];
    __syncthreads();
    bool wide = false;  // the previous gate left its warp's amplitudes
    SmallGate next = P.gate[0];
    for (int k = 0; k < P.count; ++k) {
        const SmallGate g = next;
        next = P.gate[min(k + 1, P.count - 1)];  // asked for a gate ahead: it is a constant-cache miss
        const bool spans = g.target >= 6 || g.swap >= 64u;
        if (wide || spans) __syncthreads();
        else __syncwarp();
        wide = spans;
        const uint32_t need = g.control | g.swap;
        uint32_t f[PAIRS], o[PAIRS];
        bool on[PAIRS];
        Cx<T> x[PAIRS], y[PAIRS];
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
            f[j] = insert_zero(t + kSmallThreads * j, g.target);
            on[j] = t < pairs && (f[j] & need) == need;
            // a swap trades target 0 and swap bit 1 for target 1 and swap bit 0
            o[j] = (f[j] ^ g.swap) | (1u << g.target);
            if (on[j]) {
                x[j] = load_amp<T>(state, f[j]);
                y[j] = load_amp<T>(state, o[j]);
            }
        }
        if (g.kernel == QM_KERNEL_MATRIX) {
#pragma unroll
            for (int j = 0; j < PAIRS; ++j) {
                if (!on[j]) continue;
                store_amp<T>(state, f[j], cmac2<T>((T)g.c[0], (T)g.c[1], x[j], (T)g.c[2], (T)g.c[3], y[j]));
                store_amp<T>(state, o[j], cmac2<T>((T)g.c[4], (T)g.c[5], x[j], (T)g.c[6], (T)g.c[7], y[j]));
            }
        } else if (g.kernel == QM_KERNEL_HADAMARD) {
            const T h = (T)g.c[0];
#pragma unroll
            for (int j = 0; j < PAIRS; ++j) {
                if (!on[j]) continue;
                store_amp<T>(state, f[j], Cx<T>{h * x[j].re + h * y[j].re, h * x[j].im + h * y[j].im});
                store_amp<T>(state, o[j], Cx<T>{h * x[j].re - h * y[j].re, h * x[j].im - h * y[j].im});
            }
        } else if (g.kernel == QM_KERNEL_DIAGONAL) {
            const bool a_one = g.c[0] == 1.0 && g.c[1] == 0.0, d_one = g.c[6] == 1.0 && g.c[7] == 0.0;
#pragma unroll
            for (int j = 0; j < PAIRS; ++j) {
                if (on[j] && !a_one) store_amp<T>(state, f[j], cmul<T>((T)g.c[0], (T)g.c[1], x[j]));
                if (on[j] && !d_one) store_amp<T>(state, o[j], cmul<T>((T)g.c[6], (T)g.c[7], y[j]));
            }
        } else {
#pragma unroll
            for (int j = 0; j < PAIRS; ++j) {
                if (!on[j]) continue;
                store_amp<T>(state, f[j], y[j]);
                store_amp<T>(state, o[j], x[j]);
            }
        }
    }
    __syncthreads();
    for (uint32_t i = t; i < 2 * pairs; i += nt) s[i] = state[i];
}

template <typename T, int N>
cudaError_t launch_small_n(void* amps, int qubits, const DevGate* gates, int count, cudaStream_t st) {
    SmallProgram<N> P;
    P.qubits = qubits;
    P.count = count;
    for (int k = 0; k < count; ++k) {
        const DevGate& g = gates[k];
        SmallGate& o = P.gate[k];
        o.kernel = g.kernel;
        o.target = g.target;
        o.control = g.control_mask;
        o.swap = g.swap_bit;
        for (int i = 0; i < 2; ++i) {
            o.c[i] = g.a[i];
            o.c[2 + i] = g.b[i];
            o.c[4 + i] = g.c[i];
            o.c[6 + i] = g.d[i];
        }
    }
    using V = typename Vec2<T>::type;
    const int pairs = 1 << (qubits - 1), threads = std::min(kSmallThreads, std::max(32, pairs));
    const size_t smem = sizeof(V) << qubits;
    if (pairs <= kSmallThreads) k_small<T, N, 1><<<1, threads, smem, st>>>(static_cast<V*>(amps), P);
    else if (pairs == 2 * kSmallThreads) k_small<T, N, 2><<<1, threads, smem, st>>>(static_cast<V*>(amps), P);
    else k_small<T, N, 4><<<1, threads, smem, st>>>(static_cast<V*>(amps), P);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- state utilities

template <typename T>
__global__ void k_reset(typename Vec2<T>::type* s, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) store_amp<T>(s, i, Cx<T>{i == 0 ? (T)1 : (T)0, (T)0});
}

__global__ void k_f64_to_f32(float2* dst, const double2* src, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        double2 v = src[i];
        dst[i] = make_float2((float)v.x, (float)v.y);
    }
}

__global__ void k_f32_to_f64(double2* dst, const float2* src, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) {
        float2 v = src[i];
        dst[i] = make_double2((double)v.x, (double)v.y);
    }
}

int stream_blocks(uint64_t n) {
    uint64_t b = (n + kThreads - 1) / kThreads;
    return (int)std::min<uint64_t>(b, 148ull * 16);
}

// ---------------------------------------------------------------- noise

// Amplitudes in one 16-byte access, and accesses per thread and round of the streaming reductions.
template <typename T> constexpr int kPer = 16 / (int)sizeof(typename Vec2<T>::type);
constexpr int kLoads = 4;

// Born masses of the amplitudes whose masked bits equal `pattern` and of the others: the target-zero
// and target-one masses of a damping (CpuNoiseChannelBackend.cs:88-106; mask = the target, pattern
// 0) and a marginal's selected mass with the rest of the total (StateVector.MarginalProbability,
// StateVector.Observations.cs:10-36).  Compensated FP64 per thread, deterministic block tree, one
// (sum, compensation) pair of each per block.  Bound by HBM; the state is read in index order with
// four 16-byte loads per thread in flight, whatever the masked bits are.  Three rounds of a monitored
// 26-qubit complex128 circuit (damping, marginal, measurement): 8.31 to 7.90 ms, with the branch's own
// mass and projection below.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_split_masses(const typename Vec2<T>::type* __restrict__ s, uint64_t n,
                                                           uint64_t mask, uint64_t pattern, double* out) {
    __shared__ KSum red[kThreads / 32];
    KSum sel{0, 0}, rest{0, 0};
    const uint64_t loads = n / kPer<T>;
    for (uint64_t i0 = (uint64_t)blockIdx.x * (kThreads * kLoads) + threadIdx.x; i0 < loads;
         i0 += (uint64_t)gridDim.x * (kThreads * kLoads)) {
        __align__(16) T v[kLoads][2 * kPer<T>];
#pragma unroll
        for (int j = 0; j < kLoads; ++j)
            if (i0 + j * kThreads < loads)
                *reinterpret_cast<uint4*>(v[j]) = __ldg(reinterpret_cast<const uint4*>(s) + i0 + j * kThreads);
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
            if (i0 + j * kThreads >= loads) break;
#pragma unroll
            for (int u = 0; u < kPer<T>; ++u) {
                const double re = v[j][2 * u], im = v[j][2 * u + 1];
                const bool on = (((i0 + j * kThreads) * kPer<T> + u) & mask) == pattern;
                KSum a = on ? sel : rest;
                a.add(re * re + im * im);
                sel = on ? a : sel;
                rest = on ? rest : a;
            }
        }
    }
    const KSum st = block_reduce_ksum(sel, red);
    const KSum rt = block_reduce_ksum(rest, red);
    if (threadIdx.x == 0) {
        out[4 * blockIdx.x + 0] = st.s;
        out[4 * blockIdx.x + 1] = st.c;
        out[4 * blockIdx.x + 2] = rt.s;
        out[4 * blockIdx.x + 3] = rt.c;
    }
}

// Pauli branch (CpuNoiseChannelBackend.cs:59-80): X swaps, Y swaps with phases
// (psi0' = -i psi1, psi1' = i psi0), Z negates the target-one half.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_pauli(typename Vec2<T>::type* __restrict__ s, uint32_t pairs, int target,
                                                    int pauli) {
    uint32_t bit = 1u << target;
    for (uint32_t p = blockIdx.x * kThreads + threadIdx.x; p < pairs; p += gridDim.x * kThreads) {
        uint32_t f = insert_zero(p, target);
        if (pauli == 3) {
            Cx<T> y = load_amp<T>(s, f | bit);
            store_amp<T>(s, f | bit, Cx<T>{-y.re, -y.im});
            continue;
        }
        Cx<T> x = load_amp<T>(s, f), y = load_amp<T>(s, f | bit);
        if (pauli == 1) {
            store_amp<T>(s, f, y);
            store_amp<T>(s, f | bit, x);
        } else {
            store_amp<T>(s, f, Cx<T>{y.im, -y.re});
            store_amp<T>(s, f | bit, Cx<T>{-x.im, x.re});
        }
    }
}

// Damping branch (CpuNoiseChannelBackend.cs:118-142).  Scales arrive in FP64 and are
// applied in the state's precision.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_damping(typename Vec2<T>::type* __restrict__ s, uint32_t pairs,
                                                      int target, int jump, double scale, double jump_scale,
                                                      double stay_scale) {
    uint32_t bit = 1u << target;
    for (uint32_t p = blockIdx.x * kThreads + threadIdx.x; p < pairs; p += gridDim.x * kThreads) {
        uint32_t f = insert_zero(p, target);
        Cx<T> y = load_amp<T>(s, f | bit);
        if (jump) {
            store_amp<T>(s, f, Cx<T>{(T)(jump_scale * (double)y.re), (T)(jump_scale * (double)y.im)});
            store_amp<T>(s, f | bit, Cx<T>{(T)0, (T)0});
        } else {
            Cx<T> x = load_amp<T>(s, f);
            store_amp<T>(s, f, Cx<T>{(T)((double)x.re * scale), (T)((double)x.im * scale)});
            store_amp<T>(s, f | bit, Cx<T>{(T)((double)y.re * stay_scale), (T)((double)y.im * stay_scale)});
        }
    }
}

// ---------------------------------------------------------------- observables

// One pass per distinct flip mask F.  Each pair {j, j^F} is read once; every term of the
// group (same F) gets conj(psi[j^F]) psi[j] times its Y phase and Z sign for both members
// (StateVector.Observations.cs:115-132).  With F == 0 each amplitude is its own partner.
// The Born mass rides along in the F == 0 pass as an extra column.
constexpr int kGroupMax = 8;
struct GroupLaunch {
    uint32_t flip;
    int32_t low;          // lowest set bit of flip (pair enumeration); -1 when flip == 0
    int32_t terms;        // <= kGroupMax
    int32_t with_mass;
    uint32_t sign[kGroupMax];
    int32_t phase[kGroupMax];  // y_count & 3
    int32_t column[kGroupMax]; // output column of each term
    int32_t mass_column;
    int32_t columns;           // row width of the partial table
};

template <typename T>
__global__ void __launch_bounds__(kThreads) k_pauli_group(const typename Vec2<T>::type* __restrict__ s, uint32_t items,
                                                          const GroupLaunch L, double* partials) {
    __shared__ KSum red[kThreads / 32];
    KSum acc[kGroupMax + 1];
#pragma unroll
    for (int t = 0; t <= kGroupMax; ++t) acc[t] = KSum{0, 0};
    for (uint32_t it = blockIdx.x * kThreads + threadIdx.x; it < items; it += gridDim.x * kThreads) {
        if (L.low < 0) {
            Cx<T> v = load_amp<T>(s, it);
            double p = (double)v.re * (double)v.re + (double)v.im * (double)v.im;
#pragma unroll
            for (int t = 0; t < kGroupMax; ++t) {
                if (t >= L.terms) break;
                // overlap = |psi|^2 (real); phase classes 1 and 3 take its zero imaginary part
                double c = (L.phase[t] & 1) ? 0.0 : (L.phase[t] == 2 ? -p : p);
                acc[t].add((__popc(it & L.sign[t]) & 1) ? -c : c);
            }
            if (L.with_mass) acc[kGroupMax].add(p);
        } else {
            uint32_t j = insert_zero(it, L.low);
            uint32_t k = j ^ L.flip;
            Cx<T> a = load_amp<T>(s, j), b = load_amp<T>(s, k);
            double ar = a.re, ai = a.im, br = b.re, bi = b.im;
            // conj(psi_k) psi_j; the partner's overlap is its conjugate
            double ore = br * ar + bi * ai;
            double oim = br * ai - bi * ar;
#pragma unroll
            for (int t = 0; t < kGroupMax; ++t) {
                if (t >= L.terms) break;
                double cj, ck;
                switch (L.phase[t]) {
                case 0: cj = ore; ck = ore; break;
                case 1: cj = -oim; ck = oim; break;
                case 2: cj = -ore; ck = -ore; break;
                default: cj = oim; ck = -oim; break;
                }
                if (__popc(j & L.sign[t]) & 1) cj = -cj;
                if (__popc(k & L.sign[t]) & 1) ck = -ck;
                acc[t].add(cj + ck);
            }
            if (L.with_mass) acc[kGroupMax].add(ar * ar + ai * ai + br * br + bi * bi);
        }
    }
    for (int t = 0; t < L.terms; ++t) {
        KSum r = block_reduce_ksum(acc[t], red);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * L.columns + L.column[t]] = r.value();
    }
    if (L.with_mass) {
        KSum r = block_reduce_ksum(acc[kGroupMax], red);
        if (threadIdx.x == 0) partials[(size_t)blockIdx.x * L.columns + L.mass_column] = r.value();
    }
}

// Column sums of a [rows][columns] table in fixed order: one block per column, so that the few
// hundred rows of a reduction are four or five loads per thread and not a chain of twenty.
__global__ void __launch_bounds__(128) k_finish_sums(const double* __restrict__ partials, int rows, int columns,
                                                     double* out) {
    __shared__ KSum red[4];
    KSum acc{0, 0};
    for (int r = threadIdx.x; r < rows; r += 128) acc.add(partials[(size_t)r * columns + blockIdx.x]);
    acc = block_reduce_ksum(acc, red);
    if (threadIdx.x == 0) out[blockIdx.x] = acc.value();
}

// ---------------------------------------------------------------- sampling

// Sampling reads the state once into a two-level table of Born masses: fine chunks of kFineAmps
// amplitudes, one warp each, and coarse chunks of `per_block` fine ones, one block each.  A shot
// then reads the coarse prefix, the fine masses of one coarse chunk and the amplitudes of one fine
// chunk.  The pass is bound by HBM: 1000 shots of a 27-qubit complex128 state take 0.40 ms with all
// launches, 0.33 of them the state's read at the copy rate.  512 amplitudes a fine chunk keep 16
// (complex64: 8) independent 16-byte loads per lane in flight and the table at 1/1024 of a
// complex128 state's bytes.
constexpr int kFineAmps = 512;

template <typename T>
__global__ void __launch_bounds__(kThreads) k_cdf_chunks(const typename Vec2<T>::type* __restrict__ s, uint32_t fine_amps,
                                                         uint32_t per_block, double* fine, double* sums, int64_t* last) {
    __shared__ KSum red[kThreads / 32];
    __shared__ int64_t lastw[kThreads / 32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    KSum all{0, 0};
    int64_t my_last = -1;
    for (uint32_t f = warp; f < per_block; f += kThreads / 32) {
        const uint32_t chunk = blockIdx.x * per_block + f;
        KSum acc{0, 0};
        if (fine_amps == kFineAmps) {
            constexpr int kFineLoads = kFineAmps / (32 * kPer<T>);
            const uint32_t first = chunk * (kFineAmps / kPer<T>) + lane;
            __align__(16) T v[kFineLoads][2 * kPer<T>];
#pragma unroll
            for (int j = 0; j < kFineLoads; ++j)
                *reinterpret_cast<uint4*>(v[j]) = __ldg(reinterpret_cast<const uint4*>(s) + first + 32 * j);
#pragma unroll
            for (int j = 0; j < kFineLoads; ++j)
#pragma unroll
                for (int u = 0; u < kPer<T>; ++u) {
                    const double re = v[j][2 * u], im = v[j][2 * u + 1];
                    const double p = re * re + im * im;
                    acc.add(p);
                    if (p > 0) my_last = (int64_t)(first + 32 * j) * kPer<T> + u;
                }
        } else {
            for (uint32_t i = lane; i < fine_amps; i += 32) {
                const Cx<T> v = load_amp<T>(s, chunk * fine_amps + i);
                const double p = (double)v.re * (double)v.re + (double)v.im * (double)v.im;
                acc.add(p);
                if (p > 0) my_last = chunk * fine_amps + i;
            }
        }
        all.merge(acc);
        for (int d = 16; d > 0; d >>= 1) acc.merge(shfl_down_ksum(acc, d));
        if (lane == 0) fine[chunk] = acc.value();
    }
    for (int d = 16; d > 0; d >>= 1) {
        const int64_t o = __shfl_down_sync(0xffffffffu, my_last, d);
        my_last = o > my_last ? o : my_last;
    }
    if (lane == 0) lastw[warp] = my_last;
    const KSum r = block_reduce_ksum(all, red);
    if (threadIdx.x == 0) {
        int64_t m = -1;
        for (int w = 0; w < kThreads / 32; ++w) m = lastw[w] > m ? lastw[w] : m;
        sums[blockIdx.x] = r.value();
        last[blockIdx.x] = m;
    }
}

// Exclusive prefix of the coarse masses (at most 2048 of them), the total and the last supported
// index, by one block: on the device, so that a draw needs no host round trip between its passes.
__global__ void __launch_bounds__(1024) k_cdf_prefix(const double* __restrict__ sums, const int64_t* __restrict__ last,
                                                     int blocks, double* prefix, SampleSummary* summary) {
    __shared__ double wsum[32];
    __shared__ int64_t wlast[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const double a = 2 * t < blocks ? sums[2 * t] : 0.0, b = 2 * t + 1 < blocks ? sums[2 * t + 1] : 0.0;
    int64_t m = -1;
    if (2 * t < blocks) m = last[2 * t];
    if (2 * t + 1 < blocks && last[2 * t + 1] > m) m = last[2 * t + 1];
    double inc = a + b;
    for (int d = 1; d < 32; d <<= 1) {
        const double o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
    }
    for (int d = 16; d > 0; d >>= 1) {
        const int64_t o = __shfl_xor_sync(0xffffffffu, m, d);
        m = o > m ? o : m;
    }
    if (lane == 31) wsum[warp] = inc;
    if (lane == 0) wlast[warp] = m;
    __syncthreads();
    if (warp == 0) {
        double w = wsum[lane];
        for (int d = 1; d < 32; d <<= 1) {
            const double o = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += o;
        }
        wsum[lane] = w;
        int64_t l = wlast[lane];
        for (int d = 16; d > 0; d >>= 1) {
            const int64_t o = __shfl_xor_sync(0xffffffffu, l, d);
            l = o > l ? o : l;
        }
        if (lane == 0) {
            summary->last = l;
            summary->total = wsum[31];
            prefix[0] = 0.0;
        }
    }
    __syncthreads();
    const double base = warp ? wsum[warp - 1] : 0.0;
    double excl = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) excl = 0.0;
    if (2 * t < blocks) prefix[2 * t + 1] = base + (excl + a);
    if (2 * t + 1 < blocks) prefix[2 * t + 2] = base + inc;
}

// The first position of a run of nonnegative values, 8 per lane in order, at which the running sum
// exceeds t: its index within the warp's 256 values, or -1.  `running` becomes the sum before that
// position, or the sum of all when there is none; `value` its value.
__device__ __forceinline__ int warp_crossing(const double (&v)[8], double t, double& running, double& value) {
    const int lane = threadIdx.x & 31;
    double own = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) own += v[j];
    double inc = own;
    for (int d = 1; d < 32; d <<= 1) {
        const double o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
    }
    // only lanes that hold mass: rounding of the scan must not pick an empty one
    const unsigned hit = __ballot_sync(0xffffffffu, running + inc > t && own > 0.0);
    if (!hit) {
        running += __shfl_sync(0xffffffffu, inc, 31);
        return -1;
    }
    const int l = __ffs(hit) - 1;
    const double excl = __shfl_up_sync(0xffffffffu, inc, 1);
    double cum = running + (lane ? excl : 0.0), before = cum, pv = 0.0;
    int at = -1;
    bool open = true;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        // the first value that carries the sum past t, else (rounding) the lane's last with mass
        if (open && v[j] > 0.0) {
            before = cum;
            pv = v[j];
            at = j;
            open = !(cum + v[j] > t);
        }
        cum += v[j];
    }
    running = __shfl_sync(0xffffffffu, before, l);
    value = __shfl_sync(0xffffffffu, pv, l);
    return 8 * l + __shfl_sync(0xffffffffu, at, l);
}

// One warp per shot: the strict upper-bound search of StateVectorSimulator.cs:72-88 for
// draw * total, through the coarse prefix, the fine masses of that coarse chunk and the amplitudes
// of that fine chunk, 256 values a step with 8 loads per lane in flight.  When rounding carries the
// target past a chunk the walk goes on in the next one that holds mass.  out[shot] = the index, or
// the last supported one when the target lies beyond the final cumulative mass; out[shots + shot]
// = 1 then, and when the target lies within 1e-12 of the total of the cumulative mass at either
// side of the index.  27 qubits complex128, 1000 shots: the search alone took 2.53 ms when each warp
// walked its whole coarse chunk, the call 2.90 ms; it is 0.40 ms with the two levels.
template <typename T>
__global__ void __launch_bounds__(128) k_cdf_search(const typename Vec2<T>::type* __restrict__ s, uint32_t fine_amps,
                                                    uint32_t per_block, int blocks, const double* __restrict__ fine,
                                                    const double* __restrict__ sums, const double* __restrict__ prefix,
                                                    SampleSummary* summary, const double* __restrict__ draws,
                                                    int shots, int64_t* out) {
    const int shot = (int)(blockIdx.x * 4u + (threadIdx.x >> 5));
    const uint32_t lane = threadIdx.x & 31;
    if (shot >= shots) return;
    const double total = summary->total;
    int64_t found = -1;
    int ambiguous = 0;
    if (total > 0.0 && isfinite(total)) {
        const double t = draws[shot] * total, margin = 1e-12 * total;
        int lo = 0, hi = blocks;  // the first chunk whose end lies beyond t
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid + 1] <= t) lo = mid + 1; else hi = mid;
        }
        for (int b = lo; b < blocks && found < 0; ++b) {
            if (!(sums[b] > 0.0)) continue;
            double running = prefix[b];
            for (uint32_t f0 = 0; f0 < per_block && found < 0; f0 += 256) {
                double v[8], mass = 0.0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t f = f0 + 8 * lane + j;
                    v[j] = f < per_block ? fine[b * per_block + f] : 0.0;
                }
                const int at = warp_crossing(v, t, running, mass);
                if (at < 0) continue;
                // the amplitudes of that fine chunk, and of the next ones while rounding asks for them
                for (uint32_t f = f0 + at; f < per_block && found < 0; ++f) {
                    const uint32_t first = (b * per_block + f) * fine_amps;
                    if (f > f0 + at && !(fine[b * per_block + f] > 0.0)) continue;
                    for (uint32_t i0 = 0; i0 < fine_amps && found < 0; i0 += 256) {
                        double p[8], own = 0.0;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t i = i0 + 8 * lane + j;
                            p[j] = 0.0;
                            if (i < fine_amps) {
                                const Cx<T> x = load_amp<T>(s, first + i);
                                p[j] = (double)x.re * (double)x.re + (double)x.im * (double)x.im;
                            }
                        }
                        const int k = warp_crossing(p, t, running, own);
                        if (k >= 0) {
                            found = (int64_t)first + i0 + k;
                            // the reference's CDF could still be <= t here (it would pick a later
                            // index), or could already exceed t one supported index earlier; with no
                            // mass before this index there is no earlier outcome to pick
                            ambiguous = (running + own - t <= margin) || (running > 0 && t - running <= margin);
                        }
                    }
                }
                break;
            }
        }
    }
    if (lane == 0) {
        out[shot] = found >= 0 ? found : summary->last;
        out[shots + shot] = ambiguous || found < 0;
        if (shot == 0) summary->outcome = out[shot];
    }
}

// The mass of the branch a measurement selected: only the amplitudes whose masked bits equal the
// outcome's are visited (the item index gets zeros inserted at the masked bits, ascending), so a
// measurement of c qubits reads 1/2^c of the state.
struct BranchLaunch {
    uint64_t mask;
    uint32_t items;  // 2^(qubits - masked bits)
    int32_t npos;
    int32_t pos[32];
};

template <typename T>
__global__ void __launch_bounds__(kThreads) k_branch_mass(const typename Vec2<T>::type* __restrict__ s,
                                                          const BranchLaunch L, const SampleSummary* __restrict__ summary,
                                                          double* out) {
    __shared__ KSum red[kThreads / 32];
    KSum acc{0, 0};
    const uint32_t pattern = (uint32_t)((uint64_t)summary->outcome & L.mask);
    for (uint64_t i0 = (uint64_t)blockIdx.x * (kThreads * kLoads) + threadIdx.x; i0 < L.items;
         i0 += (uint64_t)gridDim.x * (kThreads * kLoads)) {
        uint32_t x[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; ++j) x[j] = (uint32_t)i0 + j * kThreads;
        for (int k = 0; k < L.npos; ++k)
#pragma unroll
            for (int j = 0; j < kLoads; ++j) x[j] = insert_zero(x[j], L.pos[k]);
        Cx<T> v[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; ++j)
            v[j] = i0 + j * kThreads < L.items ? load_amp<T>(s, x[j] | pattern) : Cx<T>{(T)0, (T)0};
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
            const double re = v[j].re, im = v[j].im;
            acc.add(re * re + im * im);
        }
    }
    acc = block_reduce_ksum(acc, red);
    if (threadIdx.x == 0) {
        out[2 * blockIdx.x + 0] = acc.s;
        out[2 * blockIdx.x + 1] = acc.c;
    }
}

// Measure's projection (StateVector.Observations.cs:86-93): the matching branch divided by the
// square root of its mass, every other amplitude zero.  Only the branch is read; a branch or total
// without finite positive mass leaves the state as it is.  Bound by HBM: one write of the state and
// one read of the branch.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_project(typename Vec2<T>::type* s, uint64_t n, uint64_t mask,
                                                      const SampleSummary* __restrict__ summary) {
    const double mass = summary->branch[0] + summary->branch[1];
    if (!(summary->total > 0.0 && isfinite(summary->total) && mass > 0.0 && isfinite(mass))) return;
    const double norm = sqrt(mass);
    const uint64_t pattern = (uint64_t)summary->outcome & mask;
    const uint64_t loads = n / kPer<T>;
    uint4* p = reinterpret_cast<uint4*>(s);
    for (uint64_t i0 = (uint64_t)blockIdx.x * (kThreads * kLoads) + threadIdx.x; i0 < loads;
         i0 += (uint64_t)gridDim.x * (kThreads * kLoads)) {
        __align__(16) T v[kLoads][2 * kPer<T>];
        bool on[kLoads][kPer<T>];
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
            const uint64_t i = i0 + j * kThreads;
            bool any = false;
#pragma unroll
            for (int u = 0; u < kPer<T>; ++u) any |= on[j][u] = ((i * kPer<T> + u) & mask) == pattern;
            if (i < loads && any) *reinterpret_cast<uint4*>(v[j]) = p[i];
        }
#pragma unroll
        for (int j = 0; j < kLoads; ++j) {
            const uint64_t i = i0 + j * kThreads;
#pragma unroll
            for (int u = 0; u < kPer<T>; ++u) {
                v[j][2 * u] = on[j][u] ? (T)((double)v[j][2 * u] / norm) : (T)0;
                v[j][2 * u + 1] = on[j][u] ? (T)((double)v[j][2 * u + 1] / norm) : (T)0;
            }
            if (i < loads) p[i] = *reinterpret_cast<const uint4*>(v[j]);
        }
    }
}

// MeasureAll's collapse onto the drawn basis state; no write without a drawn outcome.
template <typename T>
__global__ void k_collapse(typename Vec2<T>::type* s, uint64_t n, const SampleSummary* __restrict__ summary) {
    if (!(summary->total > 0.0 && isfinite(summary->total))) return;
    const uint64_t outcome = (uint64_t)summary->outcome;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) store_amp<T>(s, i, Cx<T>{i == outcome ? (T)1 : (T)0, (T)0});
}

}  // namespace

// ---------------------------------------------------------------- launchers

cudaError_t launch_gate(void* amps, int qubits, int precision, const DevGate& g, cudaStream_t s) {
    return precision == QM_FP32 ? launch_gate_t<float>(amps, qubits, g, s) : launch_gate_t<double>(amps, qubits, g, s);
}

cudaError_t launch_small(void* amps, int qubits, int precision, const DevGate* gates, int count, cudaStream_t st) {
    if (qubits < 1 || qubits > kSmallQubits || count < 0 || count > kSmallGates) return cudaErrorInvalidValue;
    if (precision == QM_FP32)
        return count <= 48 ? launch_small_n<float, 48>(amps, qubits, gates, count, st)
                           : launch_small_n<float, kSmallGates>(amps, qubits, gates, count, st);
    return count <= 48 ? launch_small_n<double, 48>(amps, qubits, gates, count, st)
                       : launch_small_n<double, kSmallGates>(amps, qubits, gates, count, st);
}

cudaError_t launch_reset(void* amps, int qubits, int precision, cudaStream_t st) {
    uint64_t n = 1ull << qubits;
    if (precision == QM_FP32) k_reset<float><<<stream_blocks(n), kThreads, 0, st>>>((float2*)amps, n);
    else k_reset<double><<<stream_blocks(n), kThreads, 0, st>>>((double2*)amps, n);
    return cudaGetLastError();
}

cudaError_t launch_convert_from_f64(void* dst, const double* src, int64_t n, cudaStream_t st) {
    k_f64_to_f32<<<stream_blocks((uint64_t)n), kThreads, 0, st>>>((float2*)dst, (const double2*)src, (uint64_t)n);
    return cudaGetLastError();
}

cudaError_t launch_convert_to_f64(double* dst, const void* src, int64_t n, cudaStream_t st) {
    k_f32_to_f64<<<stream_blocks((uint64_t)n), kThreads, 0, st>>>((double2*)dst, (const float2*)src, (uint64_t)n);
    return cudaGetLastError();
}

static int reduce_blocks(uint64_t items) {
    uint64_t b = (items + kThreads * 8 - 1) / (kThreads * 8);
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(b, (uint64_t)kReduceBlocksMax));
}

cudaError_t launch_split_masses(const void* amps, int qubits, int precision, uint64_t mask, uint64_t pattern,
                                double* scratch, int* blocks_out, cudaStream_t st) {
    const uint64_t n = 1ull << qubits;
    const int blocks = reduce_blocks(n);
    *blocks_out = blocks;
    if (precision == QM_FP32)
        k_split_masses<float><<<blocks, kThreads, 0, st>>>((const float2*)amps, n, mask, pattern, scratch);
    else
        k_split_masses<double><<<blocks, kThreads, 0, st>>>((const double2*)amps, n, mask, pattern, scratch);
    return cudaGetLastError();
}

cudaError_t launch_pauli(void* amps, int qubits, int precision, int target, int pauli, cudaStream_t st) {
    uint32_t pairs = (uint32_t)((1ull << qubits) >> 1);
    int blocks = stream_blocks(pairs);
    if (precision == QM_FP32) k_pauli<float><<<blocks, kThreads, 0, st>>>((float2*)amps, pairs, target, pauli);
    else k_pauli<double><<<blocks, kThreads, 0, st>>>((double2*)amps, pairs, target, pauli);
    return cudaGetLastError();
}

cudaError_t launch_damping(void* amps, int qubits, int precision, int target, int jump, double scale,
                           double jump_scale, double stay_scale, cudaStream_t st) {
    uint32_t pairs = (uint32_t)((1ull << qubits) >> 1);
    int blocks = stream_blocks(pairs);
    if (precision == QM_FP32)
        k_damping<float><<<blocks, kThreads, 0, st>>>((float2*)amps, pairs, target, jump, scale, jump_scale, stay_scale);
    else
        k_damping<double><<<blocks, kThreads, 0, st>>>((double2*)amps, pairs, target, jump, scale, jump_scale, stay_scale);
    return cudaGetLastError();
}

// Groups terms by flip mask and runs one pass per group (chunks of kGroupMax terms).
// Partials table: [blocks][terms + 1]; the last column is the Born mass.
cudaError_t launch_expectation(const void* amps, int qubits, int precision, const DevPauli* terms, int count,
                               double* scratch, int* blocks_out, cudaStream_t st) {
    uint64_t n = 1ull << qubits;
    int columns = count + 1;
    int blocks = reduce_blocks(n);
    *blocks_out = blocks;
    std::vector<int> order(count);
    for (int i = 0; i < count; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return terms[x].flip < terms[y].flip; });
    bool mass_done = false;
    size_t i = 0;
    auto run = [&](GroupLaunch& L) -> cudaError_t {
        L.columns = columns;
        L.mass_column = count;
        uint32_t items = L.low < 0 ? (uint32_t)n : (uint32_t)(n >> 1);
        if (precision == QM_FP32)
            k_pauli_group<float><<<blocks, kThreads, 0, st>>>((const float2*)amps, items, L, scratch);
        else
            k_pauli_group<double><<<blocks, kThreads, 0, st>>>((const double2*)amps, items, L, scratch);
        return cudaGetLastError();
    };
    while (i < order.size()) {
        uint32_t flip = terms[order[i]].flip;
        GroupLaunch L{};
        L.flip = flip;
        L.low = flip ? __builtin_ctz(flip) : -1;
        L.terms = 0;
        while (i < order.size() && terms[order[i]].flip == flip && L.terms < kGroupMax) {
            int t = order[i++];
            L.sign[L.terms] = terms[t].sign;
            L.phase[L.terms] = terms[t].phase & 3;
            L.column[L.terms] = t;
            ++L.terms;
        }
        L.with_mass = !mass_done;
        mass_done = true;
        cudaError_t e = run(L);
        if (e != cudaSuccess) return e;
    }
    if (!mass_done) {
        GroupLaunch L{};
        L.flip = 0;
        L.low = -1;
        L.terms = 0;
        L.with_mass = 1;
        cudaError_t e = run(L);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int expectation_blocks(int qubits) { return reduce_blocks(1ull << qubits); }

cudaError_t launch_pauli_group(const void* amps, int qubits, int precision, uint32_t flip, int terms,
                               const uint32_t* sign, const int32_t* phase, const int32_t* column, int with_mass,
                               int mass_column, int columns, double* partials, cudaStream_t st) {
    if (terms < 0 || terms > kGroupMax) return cudaErrorInvalidValue;
    const uint64_t n = 1ull << qubits;
    GroupLaunch L{};
    L.flip = flip;
    L.low = flip ? __builtin_ctz(flip) : -1;
    L.terms = terms;
    L.with_mass = with_mass;
    for (int t = 0; t < terms; ++t) {
        L.sign[t] = sign[t];
        L.phase[t] = phase[t] & 3;
        L.column[t] = column[t];
    }
    L.columns = columns;
    L.mass_column = mass_column;
    const uint32_t items = L.low < 0 ? (uint32_t)n : (uint32_t)(n >> 1);
    const int blocks = reduce_blocks(n);
    if (precision == QM_FP32)
        k_pauli_group<float><<<blocks, kThreads, 0, st>>>((const float2*)amps, items, L, partials);
    else
        k_pauli_group<double><<<blocks, kThreads, 0, st>>>((const double2*)amps, items, L, partials);
    return cudaGetLastError();
}

cudaError_t launch_finish_sums(const double* partials, int rows, int columns, double* out, cudaStream_t st) {
    k_finish_sums<<<columns, 128, 0, st>>>(partials, rows, columns, out);
    return cudaGetLastError();
}

SampleShape sample_shape(int qubits) {
    SampleShape g;
    const uint64_t n = 1ull << qubits;
    g.fine_amps = (uint32_t)std::min<uint64_t>(kFineAmps, n);
    // coarse chunks: powers of two, eight fine chunks (one per warp) or more, about 8 per SM
    uint64_t c = 8ull * kFineAmps;
    while (c < n / (148 * 8)) c <<= 1;
    c = std::min(c, n);
    g.per_block = (uint32_t)(c / g.fine_amps);
    g.blocks = (int)(n / c);
    return g;
}

cudaError_t launch_sample(const void* amps, int precision, const SampleShape& g, double* fine, double* sums,
                          int64_t* last, double* prefix, SampleSummary* summary, const double* draws, int shots,
                          int64_t* out, cudaStream_t st) {
    const unsigned grid = ((unsigned)shots + 3) / 4;
    if (precision == QM_FP32) {
        k_cdf_chunks<float><<<g.blocks, kThreads, 0, st>>>((const float2*)amps, g.fine_amps, g.per_block, fine, sums, last);
        k_cdf_prefix<<<1, 1024, 0, st>>>(sums, last, g.blocks, prefix, summary);
        k_cdf_search<float><<<grid, 128, 0, st>>>((const float2*)amps, g.fine_amps, g.per_block, g.blocks, fine, sums,
                                                  prefix, summary, draws, shots, out);
    } else {
        k_cdf_chunks<double><<<g.blocks, kThreads, 0, st>>>((const double2*)amps, g.fine_amps, g.per_block, fine, sums, last);
        k_cdf_prefix<<<1, 1024, 0, st>>>(sums, last, g.blocks, prefix, summary);
        k_cdf_search<double><<<grid, 128, 0, st>>>((const double2*)amps, g.fine_amps, g.per_block, g.blocks, fine, sums,
                                                   prefix, summary, draws, shots, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_measure(void* amps, int qubits, int precision, uint64_t mask, SampleSummary* summary,
                           double* partials, cudaStream_t st) {
    const uint64_t n = 1ull << qubits;
    BranchLaunch L{};
    L.mask = mask;
    for (int b = 0; b < qubits; ++b)
        if ((mask >> b) & 1) L.pos[L.npos++] = b;
    L.items = (uint32_t)(n >> L.npos);
    const int blocks = reduce_blocks(L.items);
    const unsigned grid = (unsigned)std::max(1, stream_blocks((n + kLoads - 1) / kLoads));
    if (precision == QM_FP32) {
        k_branch_mass<float><<<blocks, kThreads, 0, st>>>((const float2*)amps, L, summary, partials);
        k_finish_sums<<<2, 128, 0, st>>>(partials, blocks, 2, summary->branch);
        k_project<float><<<grid, kThreads, 0, st>>>((float2*)amps, n, mask, summary);
    } else {
        k_branch_mass<double><<<blocks, kThreads, 0, st>>>((const double2*)amps, L, summary, partials);
        k_finish_sums<<<2, 128, 0, st>>>(partials, blocks, 2, summary->branch);
        k_project<double><<<grid, kThreads, 0, st>>>((double2*)amps, n, mask, summary);
    }
    return cudaGetLastError();
}

cudaError_t launch_collapse(void* amps, int qubits, int precision, const SampleSummary* summary, cudaStream_t st) {
    uint64_t n = 1ull << qubits;
    if (precision == QM_FP32) k_collapse<float><<<stream_blocks(n), kThreads, 0, st>>>((float2*)amps, n, summary);
    else k_collapse<double><<<stream_blocks(n), kThreads, 0, st>>>((double2*)amps, n, summary);
    return cudaGetLastError();
}

}  // namespace qm
