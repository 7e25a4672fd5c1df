// qm_dense_direct.cu -- dense fused gates on the vector and FP64 tensor pipes (sm_100a).
//
// Two kernels apply one dense 2^m x 2^m unitary to every column of the state (out(a, c) =
// sum_b U(a, b) in(b, c)); qm_dense.cu says what a fused gate is and picks the kernel.
//
// k_dense_reg, m <= 4, both precisions: one thread per column, its 2^m amplitudes in registers.
// Nothing is shared between threads, so there is no staging, no barrier and no tail, and the whole
// chip's warps keep loads in flight; the unitary is a kernel parameter, read as a constant operand
// of the multiply-adds, so the inner loop is multiply-adds only.  Algorithmic bytes: 2 S; 4 * 2^m
// multiply-adds per amplitude, so HBM bounds it up to m = 4 (30 qubits complex128, m = 4: 5.3 ms of
// HBM, 3.7 ms of FP64).  Amplitudes adjacent in memory that belong to one column (the gate holds the
// lowest qubits) move in 16- or 32-byte accesses, so sectors are used whole.  Against tiles staged by
// TMA with 4 x 4 outputs per thread (27 qubits complex128, one gate): m = 3 on qubits 8-10 0.75 to
// 0.63 ms (6.8 TB/s) and on 0-2 8.4 to 0.78 ms; m = 4 on 8-11 1.04 to 0.63 ms and on 0-3 4.7 to
// 0.79 ms; a 26-qubit brick of depth 12 in 57 such gates 53.7 to 20.0 ms, 19.0 of it HBM time.
//
// k_dense_mma, m = 5 and 6, complex128: 256 multiply-adds per amplitude at m = 6 make it a
// contraction on the FP64 pipe (30 qubits: 14.8 ms at 64 per clock and SM, HBM 5.3 ms).  With 4 x 4
// outputs per thread the operand reads from shared memory filled its return path at the rate of the
// multiply-adds.  Here the unitary is a real 2^(m+1) square matrix in the A fragments of
// mma.m8n8k4.f64, held in registers for the whole launch (16 rows per warp, 128 registers at m = 6),
// so a step of 8 products reads four 8-byte fragments.  Tiles of 4096 amplitudes come in by
// cp.async, two tiles ahead, into a ring of three buffers; every 16 bytes go to a slot XORed with
// higher index bits, so that fragments of any gate qubits spread over the banks.  Results go
// straight from the accumulators to global memory (pairs of lanes swap halves so that each writes
// 16 bytes).  27 qubits, one gate on the middle qubits: m = 5 1.66 to 1.16 ms (FP64 pipe 0.93, with two
// blocks of 2048-amplitude tiles per SM; 1.42 with one of 4096), m = 6 2.88 to 2.17 ms (FP64 1.85).
#include <cuda_runtime.h>

#include <algorithm>

#include "qm_device.cuh"
#include "qm_internal.h"

namespace qm {

namespace {

// ---------------------------------------------------------------- m <= 4

template <typename T, int M>
struct RegDense {
    uint32_t columns;           // 2^(qubits - M)
    int32_t q[M];               // the gate's qubits, ascending
    uint32_t off[1 << M];       // index bits of local value b
    T u[1 << M][1 << M][2];     // U(a, b)
};

// N adjacent amplitudes (16 or 32 bytes, or one complex64) between memory and registers.
template <typename T, int N>
__device__ __forceinline__ void load_run(const typename Vec2<T>::type* p, Cx<T> (&x)[N]) {
    if constexpr (sizeof(T) == 8 && N == 2) {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(x[0].re), "=d"(x[0].im), "=d"(x[1].re), "=d"(x[1].im) : "l"(p) : "memory");
    } else if constexpr (sizeof(T) == 4 && N == 4) {
        asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(x[0].re), "=f"(x[0].im), "=f"(x[1].re), "=f"(x[1].im), "=f"(x[2].re), "=f"(x[2].im),
                       "=f"(x[3].re), "=f"(x[3].im) : "l"(p) : "memory");
    } else if constexpr (sizeof(T) == 4 && N == 2) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        x[0] = Cx<T>{v.x, v.y};
        x[1] = Cx<T>{v.z, v.w};
    } else {
        static_assert(N == 1, "16 or 32 bytes");
        x[0] = load_amp<T>(p, 0);
    }
}

template <typename T, int N>
__device__ __forceinline__ void store_run(typename Vec2<T>::type* p, const Cx<T> (&x)[N]) {
    if constexpr (sizeof(T) == 8 && N == 2) {
        asm volatile("st.global.v4.f64 [%4], {%0, %1, %2, %3};" ::"d"(x[0].re), "d"(x[0].im), "d"(x[1].re),
                     "d"(x[1].im), "l"(p) : "memory");
    } else if constexpr (sizeof(T) == 4 && N == 4) {
        asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(x[0].re), "f"(x[0].im),
                     "f"(x[1].re), "f"(x[1].im), "f"(x[2].re), "f"(x[2].im), "f"(x[3].re), "f"(x[3].im), "l"(p)
                     : "memory");
    } else if constexpr (sizeof(T) == 4 && N == 2) {
        *reinterpret_cast<float4*>(p) = make_float4(x[0].re, x[0].im, x[1].re, x[1].im);
    } else {
        store_amp<T>(p, 0, x[0]);
    }
}

constexpr int kRegThreads = 128;

// V: how many of the lowest qubits, from qubit 0 up, are the gate's own: 2^V amplitudes of a column
// are adjacent and move together.  PAIR (complex64, gates on qubit 1 but not 0; V = 1): a thread takes
// the two columns of qubit 0, so that its accesses are the whole 32 bytes of qubits 0 and 1 and not
// half sectors.  Pairs without qubit 1 were slower than single columns (27 qubits, m = 4: 0.38
// against 0.36 ms).
template <typename T, int M, int V, bool PAIR>
__global__ void __launch_bounds__(kRegThreads) k_dense_reg(typename Vec2<T>::type* __restrict__ s,
                                                           const __grid_constant__ RegDense<T, M> P) {
    constexpr int D = 1 << M, RUN = 1 << V, COLS = PAIR ? 2 : 1;
    constexpr int G = D < 4 ? D : 4;  // outputs at a time: eight chains of multiply-adds
    const uint32_t column = (blockIdx.x * kRegThreads + threadIdx.x) * COLS;
    if (column >= P.columns) return;
    uint32_t base = column;
#pragma unroll
    for (int i = 0; i < M; ++i) base = insert_zero(base, P.q[i]);
    Cx<T> x[D / RUN][RUN * COLS];
#pragma unroll
    for (int b = 0; b < D; b += RUN) load_run<T, RUN * COLS>(s + (base | P.off[b]), x[b / RUN]);
#pragma unroll
    for (int a0 = 0; a0 < D; a0 += G) {
        Cx<T> o[G / RUN][RUN * COLS];
#pragma unroll
        for (int a = 0; a < G / RUN; ++a)
#pragma unroll
            for (int c = 0; c < RUN * COLS; ++c) o[a][c] = Cx<T>{(T)0, (T)0};
#pragma unroll
        for (int b = 0; b < D; ++b)
#pragma unroll
            for (int a = 0; a < G; ++a) {
                const T ur = P.u[a0 + a][b][0], ui = P.u[a0 + a][b][1];
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    const Cx<T> v = x[b / RUN][(b % RUN) * COLS + c];
                    Cx<T>& w = o[a / RUN][(a % RUN) * COLS + c];
                    w.re = fma(ur, v.re, w.re);
                    w.re = fma(-ui, v.im, w.re);
                    w.im = fma(ur, v.im, w.im);
                    w.im = fma(ui, v.re, w.im);
                }
            }
#pragma unroll
        for (int a = 0; a < G; a += RUN) store_run<T, RUN * COLS>(s + (base | P.off[a0 + a]), o[a / RUN]);
    }
}

template <typename T, int M, int V, bool PAIR>
cudaError_t launch_reg_v(void* amps, const RegDense<T, M>& P, cudaStream_t st) {
    const uint32_t threads = PAIR ? P.columns / 2 : P.columns;
    k_dense_reg<T, M, V, PAIR><<<(threads + kRegThreads - 1) / kRegThreads, kRegThreads, 0, st>>>(
        reinterpret_cast<typename Vec2<T>::type*>(amps), P);
    return cudaGetLastError();
}

template <typename T, int M>
cudaError_t launch_reg_m(void* amps, int qubits, const DenseOp& op, const double* matrix, cudaStream_t st) {
    constexpr int D = 1 << M;
    RegDense<T, M> P;
    P.columns = (uint32_t)((1ull << qubits) >> M);
    for (int i = 0; i < M; ++i) P.q[i] = op.q[i];
    for (int b = 0; b < D; ++b) {
        P.off[b] = 0;
        for (int i = 0; i < M; ++i)
            if ((b >> i) & 1) P.off[b] |= 1u << op.q[i];
        for (int a = 0; a < D; ++a)
            for (int k = 0; k < 2; ++k) P.u[a][b][k] = (T)matrix[2 * ((size_t)b * D + a) + k];
    }
    // adjacent amplitudes of one column, up to 32 bytes, or two adjacent columns of complex64
    int v = 0;
    const int most = std::min(M, sizeof(T) == 8 ? 1 : 2);
    while (v < most && op.q[v] == v) ++v;
    if constexpr (sizeof(T) == 4) {
        if constexpr (M >= 2)
            if (v == 2) return launch_reg_v<T, M, 2, false>(amps, P, st);
        if (op.q[0] == 1) return launch_reg_v<T, M, 1, true>(amps, P, st);  // qubit 0 exists and is free
    }
    return v >= 1 ? launch_reg_v<T, M, 1, false>(amps, P, st) : launch_reg_v<T, M, 0, false>(amps, P, st);
}

template <typename T>
cudaError_t launch_reg(void* amps, int qubits, const DenseOp& op, const double* matrix, cudaStream_t st) {
    switch (op.m) {
    case 1: return launch_reg_m<T, 1>(amps, qubits, op, matrix, st);
    case 2: return launch_reg_m<T, 2>(amps, qubits, op, matrix, st);
    case 3: return launch_reg_m<T, 3>(amps, qubits, op, matrix, st);
    case 4: return launch_reg_m<T, 4>(amps, qubits, op, matrix, st);
    default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------- m = 5 and 6, complex128

constexpr int kMmaThreads = 256;
constexpr int kMmaBufs = 3;

struct MmaDense {
    const double2* matrix;   // transposed unitary: row b holds U(a, b) for a = 0 .. 2^m - 1
    uint64_t items;          // tiles
    uint32_t outer_mask;     // index bits enumerated by the tile number
    uint32_t tile_mask;      // index bits of the tile, ascending = local bits
    int32_t tile_bits;
    int32_t ntiles;          // groups of 8 columns per tile
    int32_t q[6], ql[6];     // the gate's qubits: index bits and local bits
    int32_t c[3], cl[3];     // the lowest three column bits: index bits and local bits
    uint32_t load_off[16];   // index bits of local index 256 i
    uint32_t nt_off[16];     // index bits of column 8 i
    uint32_t nt_slot[16];    // swizzled byte offset of column 8 i
};

// Slot of local index j: the low three bits (16-byte columns of a 128-byte row) XORed with the
// higher ones.  Linear over XOR, so offsets of disjoint bits combine.
__host__ __device__ __forceinline__ uint32_t mma_slot(uint32_t j) {
    return (j ^ (((j >> 3) ^ (j >> 6) ^ (j >> 9)) & 7u)) << 4;
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

__device__ __forceinline__ double lds_f64(uint32_t at) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at));
    return v;
}

template <int M>
__global__ void __launch_bounds__(kMmaThreads, M == 5 ? 2 : 1) k_dense_mma(double2* __restrict__ s,
                                                              const __grid_constant__ MmaDense P) {
    constexpr int D = 1 << M, KS = 2 * D / 4;          // steps of 4 real inputs (two amplitudes)
    constexpr int ROWW = 2 * D / 16, COLW = 8 / ROWW;  // warps along the 2 D real rows, and column groups
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t rw = warp % ROWW, cw = warp / ROWW;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t buf_bytes = 16u << P.tile_bits;

    // A fragments: real row 2 a + p, real column 2 b + r of [[re, -im], [im, re]] per entry of U
    double A[2][KS];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        const uint32_t row = 16 * rw + 8 * mt + (lane >> 2), a = row >> 1, p = row & 1;
        const uint32_t r = lane & 1;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            const double2 u = P.matrix[(size_t)(2 * k + ((lane & 3) >> 1)) * D + a];
            A[mt][k] = p == r ? u.x : p ? u.y : -u.y;
        }
    }
    // this lane's fragment address: columns by lane / 4, the low bit of b by bit 1, re / im by bit 0
    uint32_t lane_slot = (lane & 1) * 8;
    if (lane & 2) lane_slot ^= mma_slot(1u << P.ql[0]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if ((lane >> (2 + i)) & 1) lane_slot ^= mma_slot(1u << P.cl[i]);
    // byte offsets of step k: its bits are bits 1.. of b
    uint32_t lo[8], hi[KS / 8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        lo[k] = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if ((k >> i) & 1) lo[k] ^= mma_slot(1u << P.ql[1 + i]);
    }
#pragma unroll
    for (int k = 0; k < KS / 8; ++k) {
        hi[k] = 0;
#pragma unroll
        for (int i = 0; i < M - 4; ++i)
            if ((k >> i) & 1) hi[k] ^= mma_slot(1u << P.ql[4 + i]);
    }
    // index bits of this lane's results: row pair, then column 2 (lane % 4) + p
    const uint32_t odd = (lane >> 2) & 1;
    uint32_t out_lane = 0;
    {
        const uint32_t a = 8 * rw + (lane >> 3);
#pragma unroll
        for (int i = 0; i < M; ++i)
            if ((a >> i) & 1) out_lane |= 1u << P.q[i];
        const uint32_t col = 2 * (lane & 3) + odd;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if ((col >> i) & 1) out_lane |= 1u << P.c[i];
    }
    const uint32_t load_lane = deposit(t, P.tile_mask), load_slot = mma_slot(t);
    const int loads = 1 << (P.tile_bits - 8);

    const uint64_t step = gridDim.x;
    // tile starts (index bits) of the next load and of the current tile, advanced by masked additions
    const uint32_t step_at = deposit((uint32_t)step, P.outer_mask);
    uint32_t tile_at = deposit(blockIdx.x, P.outer_mask), load_at = tile_at;
    auto issue = [&](uint64_t item, uint32_t buf) {
        if (item < P.items) {
            const double2* src = s + (load_at | load_lane);
            load_at = deposit_add(load_at, step_at, P.outer_mask);
            const uint32_t dst = ring + buf * buf_bytes;
            for (int i = 0; i < loads; ++i)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (load_slot ^ mma_slot(256u * i))),
                             "l"(src + P.load_off[i]) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    issue(blockIdx.x, 0);
    issue(blockIdx.x + step, 1);
    uint32_t cur = 0;
    for (uint64_t item = blockIdx.x; item < P.items; item += step) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // the tile is here for every thread, and the buffer two tiles ahead is free
        issue(item + 2 * step, cur == 0 ? 2 : cur - 1);
        const uint32_t tile = ring + cur * buf_bytes;
        double2* out = s + (tile_at | out_lane);
        tile_at = deposit_add(tile_at, step_at, P.outer_mask);
        for (int n0 = 4 * cw; n0 < P.ntiles; n0 += 4 * COLW) {
            double acc[2][4][2];
            uint32_t from[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                from[u] = lane_slot ^ P.nt_slot[min(n0 + u, P.ntiles - 1)];
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) acc[mt][u][0] = acc[mt][u][1] = 0.0;
            }
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                const uint32_t at = lo[k & 7] ^ hi[k >> 3];
                double b[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) b[u] = lds_f64(tile + (from[u] ^ at));
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) mma_f64(acc[mt][u], A[mt][k], b[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    // even rows hold two real parts, odd rows their imaginary parts: each keeps one
                    // column and swaps the other for its missing half
                    const double give = odd ? acc[mt][u][0] : acc[mt][u][1];
                    const double got = __shfl_xor_sync(0xffffffffu, give, 4);
                    const double2 v = odd ? make_double2(got, acc[mt][u][1]) : make_double2(acc[mt][u][0], got);
                    if (n0 + u < P.ntiles) out[P.nt_off[n0 + u] | (mt ? 1u << P.q[2] : 0u)] = v;
                }
        }
        cur = cur == 2 ? 0 : cur + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int M>
cudaError_t launch_mma_m(void* amps, const MmaDense& P, int sm_count, cudaStream_t st) {
    static const cudaError_t configured =  // once per process, thread-safe
        cudaFuncSetAttribute(k_dense_mma<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaBufs * (16 << 12));
    if (configured != cudaSuccess) return configured;
    const unsigned grid = (unsigned)std::min<uint64_t>(P.items, (uint64_t)std::max(1, sm_count) * (M == 5 ? 2 : 1));
    k_dense_mma<M><<<grid, kMmaThreads, kMmaBufs * (16u << P.tile_bits), st>>>(reinterpret_cast<double2*>(amps), P);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dense_reg(void* amps, int qubits, int precision, const DenseOp& op, const double* matrix,
                             cudaStream_t st) {
    return precision == QM_FP32 ? launch_reg<float>(amps, qubits, op, matrix, st)
                                : launch_reg<double>(amps, qubits, op, matrix, st);
}

cudaError_t launch_dense_mma(void* amps, int qubits, const DenseOp& op, const double2* matrix, int sm_count,
                             cudaStream_t st) {
    if (op.m < 5 || op.m > 6 || qubits < 9) return cudaErrorInvalidValue;
    MmaDense P{};
    P.matrix = matrix;
    // tiles of 4096 amplitudes; 2048 at m = 5, whose two blocks per SM share the shared memory, and
    // where those leave an SM fewer than eight tiles
    int tb = std::min(op.m == 5 ? 11 : 12, qubits);
    if (tb == 12 && (1ull << (qubits - 12)) < 8ull * (uint64_t)std::max(1, sm_count)) tb = 11;
    uint32_t qmask = 0;
    for (int i = 0; i < op.m; ++i) qmask |= 1u << op.q[i];
    // the columns are the lowest other bits
    uint32_t cmask = 0;
    int c[12], nc = 0;
    for (int b = 0; b < qubits && nc < tb - op.m; ++b)
        if (!((qmask >> b) & 1u)) {
            cmask |= 1u << b;
            c[nc++] = b;
        }
    P.tile_mask = qmask | cmask;
    P.outer_mask = (qubits >= 32 ? 0xffffffffu : (1u << qubits) - 1u) & ~P.tile_mask;
    P.items = 1ull << (qubits - tb);
    P.tile_bits = tb;
    P.ntiles = 1 << (nc - 3);
    auto local = [&](int b) { return __builtin_popcount(P.tile_mask & ((1u << b) - 1u)); };
    for (int i = 0; i < op.m; ++i) {
        P.q[i] = op.q[i];
        P.ql[i] = local(op.q[i]);
    }
    for (int i = 0; i < 3; ++i) {
        P.c[i] = c[i];
        P.cl[i] = local(c[i]);
    }
    uint32_t bit_of[12];
    for (int b = 0, l = 0; b < qubits; ++b)
        if ((P.tile_mask >> b) & 1u) bit_of[l++] = 1u << b;
    for (int i = 0; i < 16; ++i) {
        for (int k = 0; 8 + k < tb; ++k)
            if ((i >> k) & 1) P.load_off[i] |= bit_of[8 + k];
        for (int k = 0; 3 + k < nc; ++k)
            if ((i >> k) & 1) {
                P.nt_off[i] |= 1u << c[3 + k];
                P.nt_slot[i] ^= mma_slot(1u << local(c[3 + k]));
            }
    }
    return op.m == 5 ? launch_mma_m<5>(amps, P, sm_count, st) : launch_mma_m<6>(amps, P, sm_count, st);
}

}  // namespace qm
