// qm_pauli_sum.cu -- Pauli-sum expectation of one resident state (sm_100a).
//
// The host loop of StateVector.ExpectationValue / ExpectationEnergy (StateVector.Observations.cs:
// 107-141, StateVector.Energy.cs:10-46) for a whole term list, in a few reads of the state.
//
// A pass covers a tile of 12 qubits (all of them below 12): 256 threads hold a tile's 4096
// amplitudes, 16 each, and the block works through many tiles before it writes one row of sums.
// - Terms that flip one to four qubits.  A stage puts four tile qubits on the register index, so a
//   flip inside them pairs registers of one thread: no partner loads, the eight products are two
//   operations each, and a term adds eight more to sum its signed pairs (its Z signs on the register
//   bits are three factors, on outer bits one).  A Hermitian term takes the same real part from j and
//   j ^ F, so half the pairs are visited and the sum doubled; a term whose phase does not match its
//   signs sums to zero.  Between stages the tile is read again from shared memory (16-byte slots
//   XORed with higher index bits, free of bank conflicts); a stage on the four highest tile qubits
//   uses the registers as loaded.  Each thread keeps a running sum per term in shared memory, so a
//   warp reduces once per twelve tiles and not once per tile and term.
// - Diagonal terms.  Signs on tile qubits only: every thread sums its 16 probabilities over its
//   tiles, and one Walsh-Hadamard transform per block at the end gives every such term.  Signs on
//   outer qubits too: the tile's signed mass for each distinct tile part is written per tile, and
//   k_outer_terms sums those with the signs of the tile index.  Many of them, and lists of nothing else,
//   are left to the tiled kernel (plan_pauli_sum has the rule).
// Products and sums are FP64 for both precisions (complex64 amplitudes widen when they are loaded).
// No value goes through more plain additions than in a reduction of every tile by itself (19 for a
// flip's pairs: 7 in a thread, 5 in a warp, 7 over warps; 12 in a tile's transform).  A running sum is
// closed after twelve tiles (3 + 11 + 3 additions, 11 for a probability) and what follows carries its
// rounding errors along.  Left plain until the block's end, a sum over its 222 tiles at 28 qubits was
// 4 % faster.
//
// Bound: 28 qubits complex128, XXZ chain of 109 terms: three passes of 0.67 ms of HBM, 1.0 ms of FP64,
// about 2 ms of shared-memory wavefronts; 16 warps per SM wait on shared loads between them.  With
// pairs read from shared memory and a warp reduction per term and tile the same call took 23.3 ms,
// 8.4 of them to add up 2^18 rows; 5.7 ms now (10 qubits: 57 to 46 us).  Two blocks per SM set the pass's
// 22 running sums (the 11 bonds of a 12-qubit tile); 11-qubit tiles need a fourth pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "qm_device.cuh"
#include "qm_internal.h"

namespace qm {

namespace {

constexpr int kRegs = 16;       // amplitudes per thread
constexpr int kMaxTile = 12;    // tile qubits
constexpr int kThreads = 1 << (kMaxTile - 4);
constexpr int kEntries = 11;    // pairs of running sums per thread (terms that flip qubits) and pass: two blocks per SM
constexpr int kMaxParts = 16;   // distinct tile parts of diagonal terms with outer signs, per pass
constexpr int kOuterRows = 16;  // partial rows of k_outer_terms at most
constexpr uint32_t kFoldTiles = 12;  // tiles of a block between two compensated additions

struct SumEntry {           // one or two terms with one flip mask, both real parts or both imaginary
    double sign[2][3];      // +-1 of the pair index's bits
    int32_t kind;           // flip in register bits (1..15), + 16 for imaginary parts
    int32_t both;
    uint32_t thread_mask[2];  // Z signs on the thread index of the entry's stage
    uint32_t outer_mask[2];   // Z signs outside the tile
    int32_t negate[2];
    int32_t column[2];
    int32_t pad[2];
};
struct SumStage {
    int32_t reg[4];         // tile-local bits of the register index, ascending
    int32_t entry, entries;
    int32_t pad[2];
};
struct SumPart {            // a tile part of diagonal signs
    double sign[4];         // +-1 of the register bits (the load layout's)
    uint32_t thread_mask;
    int32_t index;          // row of the per-tile masses
};
struct SumLocal {           // a diagonal term inside the tile
    double factor;
    uint32_t mask;          // tile-local bits
    int32_t column;
};
struct SumOuter {           // a diagonal term with signs outside the tile
    double factor;
    uint32_t mask;          // bits of the tile index
    int32_t part, column, pad;
};
struct SumPass {
    uint32_t tile_mask, outer_mask;
    int32_t stage, stages, entry, entries, part, parts;
    int32_t direct;         // whether the first stage is the load layout
    uint32_t reg_at[4];     // index bits of the load layout's register bits
    uint32_t step_at;       // from a block's tile to its next: index bits of the grid size
    int32_t pad[2];
};
static_assert(sizeof(SumEntry) == 96 && sizeof(SumPart) == 40 && sizeof(SumStage) == 32 && sizeof(SumPass) == 64,
              "device layout");

// Programs up to this size travel as kernel parameters, which saves small states a copy.
constexpr int kInlineProgram = 3584;

struct SumLaunch {
    const unsigned char* program;  // in device memory, or null: inline_program
    int32_t at[6];                 // passes, stages, entries, parts, locals, outers
    int32_t pass, local_count;     // first pass of the launch; diagonal terms inside the tile of pass 0
    int32_t zero_rows;             // whether pass 0 clears its rows for the launches that follow
    int32_t k, columns;
    uint32_t tiles;
    double* tile_masses;           // [part][tiles]
    double* partials;              // [rows][columns]
    double2* folds;                // [grid][kRegs][threads]: probabilities of more than kFoldTiles tiles
    __align__(16) unsigned char inline_program[kInlineProgram];
    template <typename V>
    __device__ __forceinline__ const V* list(int i) const {
        return reinterpret_cast<const V*>((program ? program : inline_program) + at[i]);
    }
};

// 16-byte slot of tile-local index j; linear over XOR.
__device__ __forceinline__ uint32_t slot_of(uint32_t j) { return j ^ (((j >> 3) ^ (j >> 6) ^ (j >> 9)) & 7u); }

__device__ __forceinline__ double signed_if(double v, uint32_t parity) {
    return __hiloint2double(__double2hiint(v) ^ (int)(parity << 31), __double2loint(v));
}

__device__ __forceinline__ double warp_total(double v) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    return v;
}

__device__ __forceinline__ double signed_sum(const double (&v)[8], double s0, double s1, double s2) {
    const double a = fma(s0, v[1], v[0]), b = fma(s0, v[3], v[2]), c = fma(s0, v[5], v[4]), d = fma(s0, v[7], v[6]);
    return fma(s2, fma(s1, d, c), fma(s1, b, a));
}

// Products of the pairs (i, i ^ MASK), i without MASK's highest bit: real or imaginary parts of
// conj(x[i ^ MASK]) x[i].
template <int MASK, bool IM>
__device__ __forceinline__ void pair_products(const double2 (&x)[kRegs], double (&v)[8]) {
    constexpr int PIVOT = MASK >= 8 ? 8 : MASK >= 4 ? 4 : MASK >= 2 ? 2 : 1;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = (r & (PIVOT - 1)) | ((r & ~(PIVOT - 1)) << 1);
        v[r] = IM ? x[i ^ MASK].x * x[i].y - x[i ^ MASK].y * x[i].x : x[i ^ MASK].x * x[i].x + x[i ^ MASK].y * x[i].y;
    }
}

// The entries of one stage added to this thread's running sums.  Everything an entry reads from shared
// memory is asked for ahead of its products.  A thread's own sign is the same in every tile, so it is
// left to the block's last sum; `outer` holds each term's sign in this tile.
__device__ __forceinline__ void run_stage(const double2 (&x)[kRegs], int first, int count, const SumEntry* entries,
                                          const double2* outer, double* acc, uint32_t stride) {
    int kind = entries[first].kind;
#pragma unroll 1
    for (int k = first; k < first + count; ++k) {
        const SumEntry& e = entries[k];
        double* a0 = acc + (size_t)(2 * k) * stride;
        double* a1 = a0 + stride;
        const double s00 = e.sign[0][0], s01 = e.sign[0][1], s02 = e.sign[0][2];
        const double s10 = e.sign[1][0], s11 = e.sign[1][1], s12 = e.sign[1][2];
        const double2 o = outer[k];
        const double was0 = *a0, was1 = *a1;
        const int now = kind;
        if (k + 1 < first + count) kind = entries[k + 1].kind;
        double v[8];
        switch (now) {
#define QM_PAIR(m)                                       \
    case m: pair_products<m, false>(x, v); break;        \
    case m + 16: pair_products<m, true>(x, v); break;
            QM_PAIR(1) QM_PAIR(2) QM_PAIR(3) QM_PAIR(4) QM_PAIR(5) QM_PAIR(6) QM_PAIR(7) QM_PAIR(8)
            QM_PAIR(9) QM_PAIR(10) QM_PAIR(11) QM_PAIR(12) QM_PAIR(13) QM_PAIR(14)
        case 15: pair_products<15, false>(x, v); break;
        default: pair_products<15, true>(x, v); break;
#undef QM_PAIR
        }
        *a0 = fma(o.x, signed_sum(v, s00, s01, s02), was0);
        *a1 = fma(o.y, signed_sum(v, s10, s11, s12), was1);
    }
}

__host__ __device__ constexpr size_t program_bytes() {
    return sizeof(SumPass) + kEntries * (sizeof(SumStage) + sizeof(SumEntry) + sizeof(double2) + 2 * sizeof(KSum)) +
           kMaxParts * (sizeof(SumPart) + 8 * sizeof(double));
}

// x + y and x - y of two sums that carry their rounding errors in .y.
__device__ __forceinline__ void butterfly(double2& x, double2& y) {
    const double s = x.x + y.x, sb = s - x.x, se = (x.x - (s - sb)) + (y.x - sb);
    const double d = x.x - y.x, db = d - x.x, de = (x.x - (d - db)) - (y.x + db);
    const double a = x.y, b = y.y;
    x = make_double2(s, se + (a + b));
    y = make_double2(d, de + (a - b));
}

// Shared memory: [tile: 2^k double2][pass program][warp sums of parts][totals][outer signs][running sums]
template <typename T, bool DIAG>
__global__ void __launch_bounds__(kThreads, 2) k_pauli_sum(const typename Vec2<T>::type* __restrict__ s,
                                                           const __grid_constant__ SumLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5, warps = nt >> 5;
    const int k = L.k;
    double2* tile = reinterpret_cast<double2*>(smem);
    SumPass* pass = reinterpret_cast<SumPass*>(smem + (sizeof(double2) << k));
    const SumPass* src = L.list<SumPass>(0) + L.pass + blockIdx.y;
    double* row = L.partials + (size_t)blockIdx.x * L.columns;
    if (DIAG && L.zero_rows)  // columns that no term writes are zero
        for (int i = t; i < L.columns; i += nt) row[i] = 0.0;
    if (t < sizeof(SumPass) / 4) reinterpret_cast<uint32_t*>(pass)[t] = reinterpret_cast<const uint32_t*>(src)[t];
    __syncthreads();
    SumStage* stages = reinterpret_cast<SumStage*>(pass + 1);
    SumEntry* entries = reinterpret_cast<SumEntry*>(stages + pass->stages);
    double2* outer_sign = reinterpret_cast<double2*>(entries + pass->entries);  // [entries], of the current tile
    SumPart* parts = reinterpret_cast<SumPart*>(outer_sign + pass->entries);
    double* warp_part = reinterpret_cast<double*>(parts + pass->parts);  // [parts][8]
    KSum* totals = reinterpret_cast<KSum*>(warp_part + 8 * pass->parts);  // [2 entries]
    double* sums = reinterpret_cast<double*>(totals + 2 * pass->entries);  // [2 entries][nt]
    auto copy = [&](void* dst, const void* from, size_t bytes) {
        for (uint32_t i = t; i < bytes / 4; i += nt)
            reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(from)[i];
    };
    copy(stages, L.list<SumStage>(1) + pass->stage, sizeof(SumStage) * pass->stages);
    copy(entries, L.list<SumEntry>(2) + pass->entry, sizeof(SumEntry) * pass->entries);
    copy(parts, L.list<SumPart>(3) + pass->part, sizeof(SumPart) * pass->parts);
    double* acc = sums + t;
    for (int i = 0; i < 2 * pass->entries; ++i) acc[(size_t)i * nt] = 0.0;
    if (t < 2u * pass->entries) totals[t] = KSum{0.0, 0.0};
    if (DIAG)
        for (uint32_t i = t; i < 8u * pass->parts; i += nt) warp_part[i] = 0.0;  // tiles of fewer than eight warps
    __syncthreads();

    // the load layout: threads on the lowest k - 4 tile bits, registers on the four highest
    const uint32_t thread_at = deposit(t, pass->tile_mask);
    uint32_t outer = deposit(blockIdx.x, pass->outer_mask);
    double prob[DIAG ? kRegs : 1];
#pragma unroll
    for (int i = 0; i < (DIAG ? kRegs : 1); ++i) prob[i] = 0.0;

    uint32_t done = 0;  // tiles of this block
    // the threads' running sums into the block's compensated totals, each sum by one warp
    auto fold = [&]() {
        for (uint32_t i = warp; i < 2u * pass->entries; i += warps) {
            const uint32_t mask = entries[i >> 1].thread_mask[i & 1];
            double v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t c = lane + 32 * j;
                v[j] = 0.0;
                if (c < nt) {
                    v[j] = signed_if(sums[(size_t)i * nt + c], (uint32_t)__popc(c & mask) & 1u);
                    sums[(size_t)i * nt + c] = 0.0;
                }
            }
            KSum w{((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])), 0.0};
            for (int d = 16; d > 0; d >>= 1) w.merge(shfl_down_ksum(w, d));
            if (lane == 0) totals[i].merge(w);
        }
    };
    for (uint32_t item = blockIdx.x; item < L.tiles; item += gridDim.x) {
        double2 x[kRegs];
#pragma unroll
        for (int i = 0; i < kRegs; ++i) {
            uint32_t g = outer | thread_at;
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if ((i >> m) & 1) g |= pass->reg_at[m];
            const Cx<T> v = load_amp<T>(s, g);
            x[i] = make_double2((double)v.re, (double)v.im);
        }
        if (pass->stages > 0) {
#pragma unroll
            for (int i = 0; i < kRegs; ++i) tile[slot_of(t + nt * i)] = x[i];
        }
        if (DIAG) {
            double p[kRegs];
#pragma unroll
            for (int i = 0; i < kRegs; ++i) {
                p[i] = x[i].x * x[i].x + x[i].y * x[i].y;
                prob[i] += p[i];
            }
            for (int d = 0; d < pass->parts; ++d) {
                const SumPart& part = parts[d];
                const double s3 = part.sign[3];
                double lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) lo[i] = fma(s3, p[i + 8], p[i]);
                const uint32_t parity = (uint32_t)__popc(t & part.thread_mask) & 1u;
                const double w = warp_total(signed_if(signed_sum(lo, part.sign[0], part.sign[1], part.sign[2]), parity));
                if (lane == 0) warp_part[8 * d + warp] = w;
            }
        }
        if (t < 2u * pass->entries)
            reinterpret_cast<double*>(outer_sign)[t] = (__popc(outer & entries[t >> 1].outer_mask[t & 1]) & 1) ? -1.0 : 1.0;
        __syncthreads();  // the tile, the warps' parts and the signs are in shared memory
        if (DIAG && t < (uint32_t)pass->parts) {
            const double* w = warp_part + 8 * t;
            L.tile_masses[(size_t)parts[t].index * L.tiles + item] =
                ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
        }
#pragma unroll 1
        for (int st = 0; st < pass->stages; ++st) {
            const SumStage& stage = stages[st];
            if (st > 0 || !pass->direct) {
                uint32_t base = t, slot[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    base = insert_zero(base, stage.reg[m]);
                    slot[m] = slot_of(1u << stage.reg[m]);
                }
                const uint32_t at = slot_of(base);
#pragma unroll
                for (int i = 0; i < kRegs; ++i) {
                    uint32_t a = at;
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if ((i >> m) & 1) a ^= slot[m];
                    x[i] = tile[a];
                }
            }
            run_stage(x, stage.entry, stage.entries, entries, outer_sign, acc, nt);
        }
        __syncthreads();  // every read of the tile is done
        outer = deposit_add(outer, pass->step_at, pass->outer_mask);
        if (++done % kFoldTiles == 0 && item + gridDim.x < L.tiles) {
            fold();
            if (DIAG && L.pass + blockIdx.y == 0) {
                double2* folds = L.folds + ((size_t)blockIdx.x * kRegs * nt + t);
#pragma unroll
                for (int i = 0; i < kRegs; ++i) {
                    const double2 f = done > kFoldTiles ? folds[nt * i] : make_double2(0.0, 0.0);
                    KSum sum{f.x, f.y};
                    sum.add(prob[i]);
                    folds[nt * i] = make_double2(sum.s, sum.c);
                    prob[i] = 0.0;
                }
            }
            __syncthreads();
        }
    }

    // one row of sums per block; a pair's two members contribute the same
    fold();
    for (uint32_t i = warp; i < 2u * pass->entries; i += warps) {
        const SumEntry& e = entries[i >> 1];
        if ((i & 1) && !e.both) continue;
        if (lane == 0) row[e.column[i & 1]] = e.negate[i & 1] ? -2.0 * totals[i].value() : 2.0 * totals[i].value();
    }
    if (DIAG && L.pass + blockIdx.y == 0) {
        // Walsh-Hadamard transform of the summed probabilities over the tile's bits: with the rounding
        // errors of a block's sums over several tiles, plainly for one tile
        const SumLocal* locals = L.list<SumLocal>(4);
        if (L.tiles > gridDim.x) {
            const double2* folds = L.folds + ((size_t)blockIdx.x * kRegs * nt + t);
#pragma unroll
            for (int i = 0; i < kRegs; ++i) {
                KSum sum{prob[i], 0.0};
                if (done > kFoldTiles) {
                    const double2 f = folds[nt * i];
                    sum = KSum{f.x, f.y};
                    sum.add(prob[i]);
                }
                tile[t + nt * i] = make_double2(sum.s, sum.c);
            }
            __syncthreads();
#pragma unroll 1
            for (int m = 0; m < k; ++m) {
#pragma unroll 1
                for (uint32_t i = t; i < (kRegs / 2) * nt; i += nt) {
                    const uint32_t j = insert_zero(i, m);
                    butterfly(tile[j], tile[j | (1u << m)]);
                }
                __syncthreads();
            }
            for (int i = t; i < L.local_count; i += nt)
                row[locals[i].column] = locals[i].factor * (tile[locals[i].mask].x + tile[locals[i].mask].y);
            return;
        }
        double* w = reinterpret_cast<double*>(smem);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < kRegs; ++i)
                if (!((i >> m) & 1)) {
                    const double a = prob[i], b = prob[i | (1 << m)];
                    prob[i] = a + b;
                    prob[i | (1 << m)] = a - b;
                }
#pragma unroll
        for (int i = 0; i < kRegs; ++i) w[t + nt * i] = prob[i];
        __syncthreads();
        for (int m = 0; m < k - 4; ++m) {
            for (uint32_t i = t; i < (kRegs / 2) * nt; i += nt) {
                const uint32_t j = insert_zero(i, m);
                const double a = w[j], b = w[j | (1u << m)];
                w[j] = a + b;
                w[j | (1u << m)] = a - b;
            }
            __syncthreads();
        }
        for (int i = t; i < L.local_count; i += nt) row[locals[i].column] = locals[i].factor * w[locals[i].mask];
    }
}

// Diagonal terms with signs outside the tile: the tiles' signed masses summed with the signs of the
// tile index, one column per blockIdx.x, one row per blockIdx.y.
__global__ void __launch_bounds__(256) k_outer_terms(const __grid_constant__ SumLaunch L) {
    __shared__ KSum red[8];
    const SumOuter o = L.list<SumOuter>(5)[blockIdx.x];
    const double* m = L.tile_masses + (size_t)o.part * L.tiles;
    KSum acc{0, 0};
    for (uint32_t i = blockIdx.y * 256 + threadIdx.x; i < L.tiles; i += 256 * gridDim.y)
        acc.add(signed_if(m[i], (uint32_t)__popc(i & o.mask) & 1u));
    acc = block_reduce_ksum(acc, red);
    if (threadIdx.x == 0) L.partials[(size_t)blockIdx.y * L.columns + o.column] = o.factor * acc.value();
}

template <typename T, bool DIAG>
cudaError_t launch_passes(const void* amps, const SumLaunch& L, int entries, unsigned grid, int passes, cudaStream_t st) {
    static const cudaError_t configured =  // once per process, thread-safe
        cudaFuncSetAttribute(k_pauli_sum<T, DIAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, 113 * 1024);
    if (configured != cudaSuccess) return configured;
    const int nt = 1 << (L.k - 4);
    // DIAG ends with a transform of 2^k doubles in the tile
    const size_t smem = (sizeof(double2) << L.k) + program_bytes() + sizeof(double2) * (size_t)entries * nt;
    k_pauli_sum<T, DIAG><<<dim3(grid, (unsigned)passes), nt, smem, st>>>(
        reinterpret_cast<const typename Vec2<T>::type*>(amps), L);
    return cudaGetLastError();
}

template <typename V>
size_t append(std::vector<unsigned char>& out, const std::vector<V>& v) {
    const size_t at = (out.size() + 15) & ~size_t(15);
    out.resize(at + sizeof(V) * v.size());
    if (!v.empty()) std::memcpy(out.data() + at, v.data(), sizeof(V) * v.size());
    return at;
}

double unit(bool negative) { return negative ? -1.0 : 1.0; }

}  // namespace

void plan_pauli_sum(int qubits, int precision, const qm_pauli_term* terms, int count, int sm_count, PauliSumPlan& plan) {
    plan = PauliSumPlan();
    const int k = std::min(kMaxTile, qubits), regs_at = k - 4;
    const int low = precision == QM_FP32 ? 4 : 3;  // 128-byte runs
    const uint32_t all = (1u << qubits) - 1u, first_tile = (1u << k) - 1u;
    plan.k = k;
    plan.qubits = qubits;
    plan.columns = count + 1;
    plan.tiles = 1u << (qubits - k);
    plan.grid = std::min<uint32_t>(plan.tiles, 2u * (uint32_t)std::max(1, sm_count));

    uint32_t flips = 0, signs = 0;
    for (int i = 0; i < count; ++i) {
        flips |= terms[i].flip_mask;
        signs |= terms[i].sign_mask;
    }
    if (flips == 0 && (signs & ~first_tile) && plan.tiles <= 1024) return;  // the rule stands below
    std::vector<SumPass> passes;
    std::vector<SumStage> stages;
    std::vector<SumEntry> entries;
    std::vector<SumPart> parts;
    std::vector<SumLocal> locals;
    std::vector<SumOuter> outers;

    std::vector<int> pending;
    std::vector<uint32_t> part_masks;
    std::vector<int32_t> part_of((size_t)1 << k, -1);  // of a tile part
    locals.push_back(SumLocal{1.0, 0u, count});  // the Born mass
    for (int i = 0; i < count; ++i) {
        const qm_pauli_term& t = terms[i];
        const int phase = t.y_count & 3;
        const bool negate = phase == 1 || phase == 2;
        if (t.flip_mask == 0) {
            if (phase & 1) {  // the imaginary part of a probability: zero
                plan.zeros = true;
                continue;
            }
            const uint32_t local = t.sign_mask & first_tile, outer = t.sign_mask & ~first_tile;
            if (outer == 0) {
                locals.push_back(SumLocal{unit(negate), local, i});
                continue;
            }
            if (part_of[local] < 0) {
                part_of[local] = (int32_t)part_masks.size();
                part_masks.push_back(local);
            }
            outers.push_back(SumOuter{unit(negate), outer >> k, part_of[local], i, 0});
            continue;
        }
        const bool cancels = ((__builtin_popcount(t.flip_mask & t.sign_mask) ^ phase) & 1) != 0;  // pair by pair: zero
        if (cancels) plan.zeros = true;
        else if (__builtin_popcount(t.flip_mask) > 4) plan.wide.push_back(i);
        else pending.push_back(i);
    }
    // Diagonal terms with outer signs cost a warp reduction per distinct tile part and tile here, and a read
    // of the state per kMaxParts of them; the tiled kernel (qm_expect.cu) takes 256 terms from one
    // transform per tile, at a row of sums per tile and, beside flips, a read and a wait of its own.
    // It takes diagonal lists of states of up to 22 qubits, longer ones of larger states and long ones
    // beside flips.  Random Z strings alone (complex128, sums here / tiled): 16 of them 37 / 34 us at 18
    // qubits, 73 / 58 at 22, 97 / 85 at 23, 148 / 139 at 24, 8 of them 111 / 135 at 24, 256 of them 205 / 54
    // at 18 and 1736 / 301 at 24.  Beside as many flips: 16 of them 65 / 93 us at 20 qubits, 410 / 465 at
    // 24; 32 of them 84 / 95 and 590 / 519; 128 of them 68 / 102 at 16, 167 / 114 at 18 and 217 / 159 at 20.
    const int distinct = (int)part_masks.size();
    if (flips == 0 && distinct > kMaxParts) return;
    if (plan.tiles >= 64 && distinct > 2 * kMaxParts) {
        for (const SumOuter& o : outers) plan.wide.push_back(o.column);
        outers.clear();
        part_masks.clear();
    }
    // neighbouring flips side by side, so that a tile and a stage take as many as they can
    std::stable_sort(pending.begin(), pending.end(), [&](int x, int y) {
        const int hx = 31 - __builtin_clz(terms[x].flip_mask), hy = 31 - __builtin_clz(terms[y].flip_mask);
        if (hx != hy) return hx < hy;
        if (terms[x].flip_mask != terms[y].flip_mask) return terms[x].flip_mask < terms[y].flip_mask;
        return (terms[x].y_count & 1) < (terms[y].y_count & 1);
    });

    size_t part = 0;
    while (passes.empty() || !pending.empty() || part < part_masks.size()) {
        // the diagonal passes are first, on the lowest qubits
        const bool diag = passes.empty() || part < part_masks.size();
        std::vector<int> mine, rest;
        uint32_t Q = diag ? first_tile : (1u << std::min(low, k)) - 1u;
        int pairs = 0;
        bool half = false;
        uint64_t last_kind = 0;
        for (size_t j = 0; j < pending.size(); ++j) {
            const int i = pending[j];
            const uint32_t nq = Q | terms[i].flip_mask;
            // a new pair of sums, or the second half of the last one (terms of one flip and part are neighbours)
            const uint64_t kind = ((uint64_t)terms[i].flip_mask << 1) | (uint64_t)(terms[i].y_count & 1);
            const bool opens = !half || kind != last_kind;
            if (pairs == kEntries && opens) {  // full: so is the pass for all terms behind
                rest.insert(rest.end(), pending.begin() + (std::ptrdiff_t)j, pending.end());
                break;
            }
            if (__builtin_popcount(nq) <= k) {
                Q = nq;
                mine.push_back(i);
                pairs += opens ? 1 : 0;
                half = opens;
                last_kind = kind;
            } else {
                rest.push_back(i);
            }
        }
        for (int q = 0; q < qubits && __builtin_popcount(Q) < k; ++q) Q |= 1u << q;
        pending.swap(rest);
        auto local = [&](uint32_t mask) {
            uint32_t l = 0;
            for (int q = 0, b = 0; q < qubits; ++q)
                if ((Q >> q) & 1u) l |= ((mask >> q) & 1u) << b++;
            return l;
        };
        SumPass p{};
        p.tile_mask = Q;
        p.outer_mask = all & ~Q;
        for (int q = 0, b = 0; q < qubits; ++q)
            if ((Q >> q) & 1u) {
                if (b >= regs_at) p.reg_at[b - regs_at] = 1u << q;
                ++b;
            }
        for (int q = 0, b = 0; q < qubits; ++q)
            if ((p.outer_mask >> q) & 1u) p.step_at |= ((plan.grid >> b++) & 1u) << q;
        p.stage = (int32_t)stages.size();
        p.entry = (int32_t)entries.size();
        p.part = (int32_t)parts.size();
        // stages: register layouts of four tile bits, each taking every flip it can
        int direct = -1;
        std::vector<char> done(mine.size(), 0);
        for (size_t a = 0; a < mine.size(); ++a) {
            if (done[a]) continue;
            uint32_t layout = 0;
            std::vector<size_t> held;
            for (size_t b = a; b < mine.size(); ++b) {
                const uint32_t l = layout | local(terms[mine[b]].flip_mask);
                if (done[b] || __builtin_popcount(l) > 4) continue;
                layout = l;
                held.push_back(b);
                done[b] = 1;
            }
            for (int b = k - 1; b >= 0 && __builtin_popcount(layout) < 4; --b) layout |= 1u << b;
            SumStage st{};
            for (int b = 0, m = 0; b < k; ++b)
                if ((layout >> b) & 1u) st.reg[m++] = b;
            if (layout == (15u << regs_at)) direct = (int32_t)stages.size();
            st.entry = (int32_t)entries.size() - p.entry;
            // held terms of one flip and part are neighbours: they pair up in order
            for (size_t h = 0; h < held.size();) {
                const qm_pauli_term& first = terms[mine[held[h]]];
                SumEntry e{};
                for (int m = 0; m < 4; ++m)
                    if ((local(first.flip_mask) >> st.reg[m]) & 1u) e.kind |= 1 << m;
                const int pivot = 31 - __builtin_clz((unsigned)e.kind);
                if (first.y_count & 1) e.kind |= 16;
                for (int n = 0; n < 2 && h < held.size(); ++n, ++h) {
                    const qm_pauli_term& t = terms[mine[held[h]]];
                    if (t.flip_mask != first.flip_mask || ((t.y_count ^ first.y_count) & 1)) break;
                    const int phase = t.y_count & 3;
                    const uint32_t sl = local(t.sign_mask & Q);
                    for (int b = 0, m = 0; m < 4; ++m)
                        if (m != pivot) e.sign[n][b++] = unit((sl >> st.reg[m]) & 1u);
                    for (int b = 0, r = 0; b < k; ++b)
                        if (!((layout >> b) & 1u)) e.thread_mask[n] |= ((sl >> b) & 1u) << r++;
                    e.outer_mask[n] = t.sign_mask & ~Q;
                    e.negate[n] = phase == 1 || phase == 2;
                    e.column[n] = mine[held[h]];
                    e.both = n;
                }
                entries.push_back(e);
            }
            st.entries = (int32_t)entries.size() - p.entry - st.entry;
            stages.push_back(st);
        }
        if (direct >= 0) {  // runs first, on the registers as loaded
            std::swap(stages[(size_t)p.stage], stages[(size_t)direct]);
            p.direct = 1;
        }
        if (diag) {
            ++plan.diagonal_passes;
            for (int n = 0; n < kMaxParts && part < part_masks.size(); ++n, ++part) {
                SumPart o{};
                for (int m = 0; m < 4; ++m) o.sign[m] = unit((part_masks[part] >> (regs_at + m)) & 1u);
                o.thread_mask = part_masks[part] & ((1u << regs_at) - 1u);
                o.index = (int32_t)part;
                parts.push_back(o);
            }
        }
        p.stages = (int32_t)stages.size() - p.stage;
        p.entries = (int32_t)entries.size() - p.entry;
        p.parts = (int32_t)parts.size() - p.part;
        plan.max_entries = std::max(plan.max_entries, (int)p.entries);
        passes.push_back(p);
    }
    plan.passes = (int)passes.size();
    plan.parts = (int)part_masks.size();
    plan.locals = (int)locals.size();
    plan.outers = (int)outers.size();
    plan.at[0] = append(plan.program, passes);
    plan.at[1] = append(plan.program, stages);
    plan.at[2] = append(plan.program, entries);
    plan.at[3] = append(plan.program, parts);
    plan.at[4] = append(plan.program, locals);
    plan.at[5] = append(plan.program, outers);
}

size_t pauli_sum_folds(const PauliSumPlan& plan) {
    const bool long_runs = (uint64_t)plan.tiles > (uint64_t)kFoldTiles * plan.grid;
    return long_runs ? sizeof(double2) * ((size_t)plan.grid << plan.k) : 0;
}

bool pauli_sum_inline(const PauliSumPlan& plan) { return plan.program.size() <= (size_t)kInlineProgram; }

cudaError_t launch_pauli_sum(const void* amps, int precision, const PauliSumPlan& plan, const void* program,
                             double* tile_masses, double* partials, double2* folds, cudaStream_t st) {
    SumLaunch L;
    L.program = static_cast<const unsigned char*>(program);
    if (!program) std::memcpy(L.inline_program, plan.program.data(), plan.program.size());
    for (int i = 0; i < 6; ++i) L.at[i] = (int32_t)plan.at[i];
    L.k = plan.k;
    L.columns = plan.columns;
    L.tiles = plan.tiles;
    L.tile_masses = tile_masses;
    L.partials = partials;
    L.folds = folds;
    cudaError_t e = cudaSuccess;
    L.pass = 0;
    L.local_count = plan.locals;
    L.zero_rows = 1;
    auto launch = [&](bool diag, int passes) {
        if (diag)
            return precision == QM_FP32 ? launch_passes<float, true>(amps, L, plan.max_entries, plan.grid, passes, st)
                                        : launch_passes<double, true>(amps, L, plan.max_entries, plan.grid, passes, st);
        return precision == QM_FP32 ? launch_passes<float, false>(amps, L, plan.max_entries, plan.grid, passes, st)
                                    : launch_passes<double, false>(amps, L, plan.max_entries, plan.grid, passes, st);
    };
    const bool written = !plan.zeros && plan.wide.empty() && plan.grid <= kOuterRows;
    if (written && plan.passes <= 65535) {
        // few tiles and a writer for every column and row: one launch, whose passes run side by side
        L.zero_rows = 0;
        e = launch(true, plan.passes);
    } else {
        for (; e == cudaSuccess && L.pass < plan.diagonal_passes; ++L.pass) {
            e = launch(true, 1);
            L.zero_rows = 0;
        }
        for (; e == cudaSuccess && L.pass < plan.passes; L.pass += 65535)
            e = launch(false, std::min(65535, plan.passes - L.pass));
    }
    if (e == cudaSuccess && plan.outers > 0) {
        k_outer_terms<<<dim3((unsigned)plan.outers, std::min<uint32_t>(plan.grid, kOuterRows)), 256, 0, st>>>(L);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace qm
