// y[m, n] = sum_k x[m, k] W[n, k] for a decode step's tokens (up to 8 NT rows of x, bf16): every weight byte is read once, so HBM bounds it, and for small matrices the
// latency of a launch's head and tail.  Shared by both libraries; the step behind the Linear is a template parameter.
//
// A CTA (one per SM) owns whole rows of W -- `rows` of them, a multiple of 8 with N / rows close to the number of SMs -- for all of K, so no sum crosses a CTA: there is
// nothing to exchange and nobody to wait for at the end.  A producer thread keeps a ring of stages full by TMA: [rows x 64] blocks of W (128B-swizzled), `blocks` of them
// along k so that a stage is 14 to 32 KB whatever `rows` is (47 from 17 tokens on; less where K has not so many, and one block where K is no multiple of 64), and the same columns of x.  The weights of the whole first ring are requested before the wait for the predecessor (nobody writes
// weights), x after it.  Two teams of eight warps take the stages in turn (one stage's latencies lie under the other's) and multiply on mma.sync (m16n8k16: 16 rows of W x 8 tokens):
// warp w of a team takes row tile w % tiles and every (8 / tiles)-th pair of slices of 16 columns; the sums meet in shared memory, in a fixed order.
//
// Why not tiles of 128 rows cut along k (gemm_streamk.cuh): with N / 128 = 16 .. 48 tiles for 148 SMs three or four CTAs finish a tile together, and the exchange through
// memory is 6 to 10 us at the end of every launch.  Why not the weights straight into registers (row_linear_kernel below, which small matrices keep): a fragment's lanes read 64
// bytes of each of 8 rows, 8 tag lookups an instruction, 4 to 5 TB/s, and x comes out of L2 in every step.
// What bounds it from 17 tokens on is mma.sync itself (7 tiles x 4 slices x 4 groups of tokens of a 13 KB stage take some 700 clocks, memory 600): 32 tokens 28672 x 5120 57 us, 24 tokens
// 57, 8 tokens of that shape 49.  More warps or two row tiles a warp made it slower.
// us a Linear in a chain of them, stored / added to the fp32 stream, that kernel and this one: 8 tokens 16384 x 2048 17.0 / 16.4, 13.7 / 13.4; 2048 x 8192 10.3 / 10.1, 8.7 / 8.5;
// 16 tokens 28672 x 4096 61 / 57, 45 / 44.  Behind other kernels, whose ends its first ring covers, it gains more: a
// step of 8 layers of width 2048, 8 sequences, 698 and 529.  With one team of warps 28672 x 4096 took 47.6 us instead of 40, with a ring of 100 KB 43.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_info.cuh"

namespace stream_linear {

constexpr int TEAM = 8, TEAMS = 2, WARPS = TEAM * TEAMS, THREADS = 32 * (WARPS + 1), MAX_ROWS = 16 * TEAM, SUM_PITCH = 16 * WARPS + 4 /* a warp's stores meet no bank twice */;
constexpr int MAX_STAGES = 24;
static_assert(MAX_STAGES % TEAMS == 0, "a slot is always the same team's");
constexpr int RING_BYTES = 180 * 1024;

struct Shape {
    int M, N, K;
    int rows, blocks, stages;
    int tiles;  // row tiles of 16, rounded up to a power of two
    int flat;   // 1: K is no multiple of 64, blocks are taken one by one (the columns past K read as zeros)
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) { asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory"); }
__device__ __forceinline__ void bar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory"); }
// Waits a bounded time; false: gave up
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(smem_addr(b)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst), "l"(map), "r"(smem_addr(bar)), "r"(c0),
                 "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&v)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Epi: `Ahead fetch(m, n, two)` reads what the step needs beside the sums (requested while the weights stream), `finish(m, n, v0, v1, two, ahead)` takes the sums of rows n
// (even) and n + 1 of W (two: n + 1 < N).
template <int NT, class Epi>
__global__ void __launch_bounds__(THREADS, 1) stream_linear_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Shape s, const Epi epi) {
    extern __shared__ unsigned char raw[];
    unsigned char* const ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t w_bytes = (uint32_t)s.rows * 128u * s.blocks, x_bytes = NT * 1024u * s.blocks, stage_bytes = w_bytes + x_bytes;
    float* const sums = reinterpret_cast<float*>(ring + (size_t)s.stages * stage_bytes);  // [8 NT tokens][SUM_PITCH]
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int units = (s.N + s.rows - 1) / s.rows, kbs = (s.K + 63) / 64, per_unit = (kbs + s.blocks - 1) / s.blocks;
    const int tiles_used = (s.rows + 15) / 16, groups = TEAM / s.tiles;
    if (threadIdx.x == 0) {
        for (int i = 0; i < s.stages; ++i) {
            bar_init(&full[i], 1);
            bar_init(&empty[i], (uint32_t)(tiles_used * groups));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == WARPS) {
        if (lane == 0) {
            const int mine = ((int)blockIdx.x < units ? (units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0), total = mine * per_unit;
            int w_unit = blockIdx.x, w_kb = 0, x_kb = 0;
            auto weights = [&](int slot) {
                load_box(smem_addr(ring + slot * stage_bytes), &map_w, &full[slot], s.flat ? w_kb * 64 : 0, s.flat ? 0 : w_kb, w_unit * s.rows);
                w_kb += s.blocks;
                if (w_kb >= kbs) w_kb = 0, w_unit += gridDim.x;
            };
            auto tokens = [&](int slot) {
                load_box(smem_addr(ring + slot * stage_bytes + w_bytes), &map_x, &full[slot], s.flat ? x_kb * 64 : 0, s.flat ? 0 : x_kb, 0);
                x_kb += s.blocks;
                if (x_kb >= kbs) x_kb = 0;
            };
            const int head = min(total, s.stages);
            for (int i = 0; i < head; ++i) {
                bar_expect(&full[i], stage_bytes);
                weights(i);
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int i = 0; i < head; ++i) tokens(i);
            int slot = 0, par = 0;
            for (int it = head; it < total; ++it) {
                if (!bar_wait(&empty[slot], par)) break;
                bar_expect(&full[slot], stage_bytes);
                weights(slot);
                tokens(slot);
                if (++slot == s.stages) slot = 0, par ^= 1;
            }
        }
        return;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int PAIRS = MAX_ROWS / 2 * 8 * NT / (32 * WARPS);
    const int tile = warp & (s.tiles - 1), group = warp % TEAM / s.tiles, half = s.rows / 2;
    bool turn = warp / TEAM == 0;  // the next stage is this team's
    const bool works = tile < tiles_used;
    // this lane's rows of the fragments: of W row 16 tile + lane % 16, columns 8 (lane / 16) ..; of x token lane % 8, columns 8 (lane / 8) ..  A row's blocks follow one another, 128
    // bytes each; their number is odd, so that eight rows' blocks are XORed with eight different numbers and the loads meet no bank twice.
    const uint32_t w_line = (tile * 16 + (lane & 15)) * (uint32_t)s.blocks, w_c = lane >> 4;
    const uint32_t x_line = (lane & 7) * (uint32_t)s.blocks, x_c = lane >> 3;
    const int slices = 4 * s.blocks;
    int slot = 0, par = 0;
    bool alive = true;
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
        typename Epi::Ahead ahead[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const int p = threadIdx.x + i * 32 * WARPS, m = p / half, n = unit * s.rows + p % half * 2;
            if (m < s.M && n < s.N) ahead[i] = epi.fetch(m, n, n + 1 < s.N);
        }
        float c[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
        for (int ks = 0; ks < per_unit; ++ks, turn = !turn) {
            if (works && turn) {
                if (alive && !bar_wait(&full[slot], par)) alive = false;
                __syncwarp();
                const uint32_t st = smem_addr(ring + slot * stage_bytes);
                // two neighbouring slices a turn (their columns of x are one instruction)
#pragma unroll 2
                for (int j = 2 * group; j < slices; j += 2 * groups) {
                    const uint32_t blk = j >> 2, half_blk = (j & 2) * 2;  // k-block, and 16-byte column 0 or 4 of its rows
                    uint32_t a0[4], a1[4];
                    const uint32_t wl = w_line + blk, xl = x_line + blk;
                    ldmatrix4(a0, st + wl * 128u + (((half_blk + w_c) ^ (wl & 7)) << 4));
                    ldmatrix4(a1, st + wl * 128u + (((half_blk + 2 + w_c) ^ (wl & 7)) << 4));
#pragma unroll
                    for (int t = 0; t < NT; ++t) {  // (8 tokens further is a multiple of 8 lines further)
                        uint32_t b[4];
                        ldmatrix4(b, st + w_bytes + (xl + t * 8 * (uint32_t)s.blocks) * 128u + (((half_blk + x_c) ^ (xl & 7)) << 4));
                        mma(c[t], a0, b[0], b[1]);
                        mma(c[t], a1, b[2], b[3]);
                    }
                }
                __syncwarp();
                if (lane == 0) bar_arrive(&empty[slot]);
            }
            if (++slot == s.stages) slot = 0, par ^= 1;
        }
        if (!alive)
#pragma unroll
            for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = __int_as_float(0x7fffffff);
        const int r = warp * 16 + (lane >> 2), col = (lane & 3) * 2;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            sums[(t * 8 + col) * SUM_PITCH + r] = c[t][0];
            sums[(t * 8 + col + 1) * SUM_PITCH + r] = c[t][1];
            sums[(t * 8 + col) * SUM_PITCH + r + 8] = c[t][2];
            sums[(t * 8 + col + 1) * SUM_PITCH + r + 8] = c[t][3];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * WARPS) : "memory");
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
            const int p = threadIdx.x + i * 32 * WARPS, m = p / half, row = p % half * 2, n = unit * s.rows + row;
            if (m < s.M && n < s.N) {
                float v0 = 0.f, v1 = 0.f;
                for (int g = 0; g < groups * TEAMS; ++g) {
                    const float2 v = *reinterpret_cast<const float2*>(sums + m * SUM_PITCH + g * s.tiles * 16 + row);
                    v0 += v.x;
                    v1 += v.y;
                }
                epi.finish(m, n, v0, v1, n + 1 < s.N, ahead[i]);
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * WARPS) : "memory");  // the sums have been read
    }
}

// The same for matrices of few rows, the weights straight into registers: a CTA of eight warps per 16 rows of W, which split K; a lane takes 16 contiguous bytes of two rows and of
// a token's x per step (the k order inside a step is permuted alike for both, which a dot product does not notice).  The weights of the first AHEAD steps -- all of them up to K = 2048 -- are
// requested before the wait for the predecessor, and two CTAs fit an SM beside the predecessor's: there is no ring to fill, and a launch's head and tail
// are shorter.  Needs K % 8 == 0 and 16-byte aligned rows.
constexpr int ROWS_WARPS = 8, ROWS_AHEAD = 8;
__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* p) {  // read once: not kept in L1
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
template <int NT, class Epi>
__global__ void __launch_bounds__(ROWS_WARPS * 32, 2) row_linear_kernel(const __nv_bfloat16* X, int64_t pitch, const __nv_bfloat16* W, int M, int N, int K, const Epi epi) {
    __shared__ float part[ROWS_WARPS][16][8 * NT + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int n0 = blockIdx.x * 16, k0 = warp * 32 + tig * 8;
    constexpr int STEP = ROWS_WARPS * 32;
    const __nv_bfloat16* wa = W + (size_t)min(n0 + gid, N - 1) * K + k0;
    const __nv_bfloat16* wb = W + (size_t)min(n0 + gid + 8, N - 1) * K + k0;
    uint4 va[ROWS_AHEAD], vb[ROWS_AHEAD];
    const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < ROWS_AHEAD; ++u) {
        const bool ok = k0 + u * STEP < K;
        va[u] = ok ? load_weights(wa + u * STEP) : zero;
        vb[u] = ok ? load_weights(wb + u * STEP) : zero;
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int em = threadIdx.x % (8 * NT), er = threadIdx.x / (8 * NT) * 2, en = n0 + er;  // this thread's pair of results
    const bool ends = threadIdx.x < 64 * NT && em < M && en < N;
    typename Epi::Ahead ahead;
    if (ends) ahead = epi.fetch(em, en, en + 1 < N);
    float c[NT][4];
    const __nv_bfloat16* xr[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
        xr[t] = X + (size_t)min(t * 8 + gid, M - 1) * pitch + k0;  // rows past the end repeat the last one: their sums go nowhere
    }
    const int steps = (K + STEP - 1) / STEP;
    for (int i = 0; i < steps; i += ROWS_AHEAD) {
#pragma unroll
        for (int u = 0; u < ROWS_AHEAD; ++u) {
            const int k = (i + u) * STEP;
            uint4 vx[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) vx[t] = k0 + k < K ? *reinterpret_cast<const uint4*>(xr[t] + k) : zero;
            const uint32_t a0[4] = {va[u].x, vb[u].x, va[u].y, vb[u].y}, a1[4] = {va[u].z, vb[u].z, va[u].w, vb[u].w};
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                mma(c[t], a0, vx[t].x, vx[t].y);
                mma(c[t], a1, vx[t].z, vx[t].w);
            }
            const bool more = k0 + k + ROWS_AHEAD * STEP < K;
            va[u] = more ? load_weights(wa + k + ROWS_AHEAD * STEP) : zero;
            vb[u] = more ? load_weights(wb + k + ROWS_AHEAD * STEP) : zero;
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        part[warp][gid][t * 8 + tig * 2] = c[t][0];
        part[warp][gid][t * 8 + tig * 2 + 1] = c[t][1];
        part[warp][gid + 8][t * 8 + tig * 2] = c[t][2];
        part[warp][gid + 8][t * 8 + tig * 2 + 1] = c[t][3];
    }
    __syncthreads();
    if (ends) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int w = 0; w < ROWS_WARPS; ++w) {
            s0 += part[w][er][em];
            s1 += part[w][er + 1][em];
        }
        epi.finish(em, en, s0, s1, en + 1 < N, ahead);
    }
}

// ---- host ----
typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                           CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline Encode encode() {  // the driver's entry point through the runtime: no link against libcuda
    static const Encode fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult found;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(ptr) : nullptr;
    }();
    return fn;
}
// [rows, K] bf16, `pitch` elements between rows, as blocks of 64 columns: boxes of box_rows rows of `blocks` blocks
inline bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t pitch, int box_rows, int blocks, bool flat) {
    const cuuint64_t dims[3] = {flat ? (cuuint64_t)K : 64u, flat ? 1u : (cuuint64_t)(K / 64), (cuuint64_t)rows}, strides[2] = {flat ? (cuuint64_t)pitch * 2 : 128u, (cuuint64_t)pitch * 2};
    const cuuint32_t box[3] = {64u, (cuuint32_t)blocks, (cuuint32_t)box_rows}, unit[3] = {1u, 1u, 1u};
    return encode()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// a launch that may begin before its predecessor in the stream has ended (MB200_PDL)
template <class Kernel, class... Args>
inline cudaError_t launch_serial(Kernel kernel, int ctas, int threads, size_t smem, cudaStream_t st, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = device_info::pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Which of the two, up to 16 rows of x: the one without a ring where the ring would take k-blocks one by one, and for small matrices.  us in a chain of Linears / behind a row norm, 8 rows of x, here
// and there: K = 1000 and 4096 rows 3.0 / 4.7, 5.7 / 6.7; 8192 5.7 / 7.7, 7.1 / 8.3; 16384 10.5, 9.3; 1024 x 64 1.7 / 3.4, 2.6 / 3.5; 1024 x 1024 2.2 / 3.8, 3.2 / 4.3; 2048 x 2048 3.0 / 4.9, 4.0 / 5.6.  Larger ones
// gain in such a chain (4096 x 4096 8.1, 8.5) and lose in a model's step, where the ring fills while other kernels end (two layers of the 7B shape, 8 sequences 283, 272;
// with 4096 x 14336 here too 335; eight layers of width 2048, 2048 x 2048 and 3072 x 2048 here: one sequence 431, 442, eight 502, 495).  From 9 rows of x on: behind a norm 2048 x 256 4.6, 3.9.
inline bool rows_better(int M, int N, int K, int64_t pitch) {
    if (K % 64 != 0 || pitch % 64 != 0) return N <= (M <= 8 && K >= 512 ? 8192 : 4096);
    return M <= 8 && N <= 4096 && K <= (M <= 4 ? 2048 : 1024);
}

template <int NT>
inline Shape shape_of(int M, int N, int K, int64_t pitch, int sms) {
    Shape s;
    s.M = M, s.N = N, s.K = K;
    s.flat = K % 64 != 0 || pitch % 64 != 0;  // (a map's strides are multiples of one another)
    int passes = 1;  // as few as their rows fit the warps' tiles
    do s.rows = ((N + sms * passes - 1) / (sms * passes) + 7) / 8 * 8;
    while (s.rows > MAX_ROWS && ++passes);
    s.tiles = 1;
    while (s.tiles * 16 < s.rows) s.tiles *= 2;
    const int kbs = (K + 63) / 64;
    s.blocks = 1;
    while (!s.flat && s.blocks + 2 <= kbs && s.blocks < 7 && (s.blocks + 2) * (s.rows + 8 * NT) * 128 <= (NT > 2 ? 47 : 32) * 1024) s.blocks += 2;
    s.stages = RING_BYTES / ((s.rows + 8 * NT) * 128 * s.blocks);
    if (s.stages > MAX_STAGES) s.stages = MAX_STAGES;
    s.stages = s.stages / TEAMS * TEAMS;  // a slot is always the same team's: its waits follow every phase of the slot's barriers
    return s;
}

// x rows `pitch` elements apart; K % 8 == 0, pitch % 8 == 0, both 16-byte aligned.  false: no tensor maps here
template <int NT, class Epi>
inline bool launch(const void* x, int64_t pitch, const void* w, int M, int N, int K, const Epi& epi, cudaStream_t st, cudaError_t& e) {
    e = cudaSuccess;
    const int sms = device_info::sm_count();
    if constexpr (NT <= 2)
        if (rows_better(M, N, K, pitch)) {
            e = launch_serial(row_linear_kernel<NT, Epi>, (N + 15) / 16, ROWS_WARPS * 32, 0, st, static_cast<const __nv_bfloat16*>(x), pitch, static_cast<const __nv_bfloat16*>(w), M, N, K, epi);
            return true;
        }
    if (sms == 0 || !encode()) return false;
    const Shape s = shape_of<NT>(M, N, K, pitch, sms);
    CUtensorMap map_x, map_w;
    if (!make_map(&map_x, x, M, K, pitch, 8 * NT, s.blocks, s.flat) || !make_map(&map_w, w, N, K, K, s.rows, s.blocks, s.flat)) return false;
    const int units = (N + s.rows - 1) / s.rows;
    // (a fragment of the last tile may reach past the stage's rows of W, into what follows them: its sums go nowhere)
    const size_t smem = 1024 + (size_t)s.stages * (s.rows + 8 * NT) * 128 * s.blocks + sizeof(float) * 8 * NT * SUM_PITCH;
    auto kernel = stream_linear_kernel<NT, Epi>;
    e = device_info::allow_shared<stream_linear_kernel<NT, Epi>>(RING_BYTES + 1024 + (int)sizeof(float) * 8 * NT * SUM_PITCH);
    if (e) return true;
    e = launch_serial(kernel, units < sms ? units : sms, THREADS, smem, st, map_x, map_w, s, epi);
    return true;
}

}  // namespace stream_linear
