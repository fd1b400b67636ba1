// C[M, N] = A[M, K] . W[N, K]^T, everything float32: the projections of the true 32-bit path.  Both operands are K-major as
// stored and 16-byte aligned with K % 4 == 0 and, for more than 8 rows, K >= 192 (gemm_simt.cu takes the rest).
//
// few rows (M <= 8, decode steps): bound by reading W once from HBM; two kernels.  K >= 1,536 (save for some lengths, see the end): a CTA per SM streams an even share
//   of W's rows through rings in shared memory (TMA copies of 2 KB, 96 KB in flight an SM, which start before the kernel ahead has
//   ended); its eight warps split K.  Less: a warp owns four rows of W and a part of K, four 2 KB pieces in flight in registers.
//   In both a warp's lanes lie along K, 16 bytes each; sums over lanes are taken by a transposing butterfly, those over
//   warps through shared memory, in a fixed order.  Relative error (2-norm, against 64 bits) 1.0e-7 to
//   1.6e-7.
//   4 rows against [16384, 2048] 25.5 us (5.3 TB/s), [2048, 8192] 14.1, [128256, 2048] 177 (5.9 TB/s), [2048, 2048] 5.4; 30.0, 17.0,
//   194 and 6.4 with the registers' kernel; 210, 557 and 1,161 us for the first three when a 64 x 64 tile per CTA walked K
//   alone.  One row: 23.3, 13.5, 151 (7.0 TB/s) and 3.8.  What is left with 4 and 8 rows is the multiply-adds and the sums at the end of a block of rows, two warps a
//   scheduler.
//
// more rows: bound by arithmetic, and the CUDA cores' multiply-adds give 75 TFLOP/s at most (64 x 128 register tiles: 28 to 45
//   measured).  So each number, times 2^16, is cut into three bfloat16 whose sum it is exactly, each rounded to nearest, and the
//   tensor cores multiply the parts: six of the nine products.  The three that are left out are below 2^-25 of the whole
//   (twice) and 2^-34, and as often above zero as below.  The leading products are added up in tensor memory over 128 positions of K only
//   and then in registers, rounded to nearest; the small ones have two accumulators of their own, that of a second-order product
//   beside that of a third-order one: the tokens' parts lie one behind the other, so one instruction takes a part of W against two
//   of them and reads it from shared memory once.  Relative errors (2-norm, against 64 bits, times 10^-8) beside those of one multiply-add
//   after the other (gemm_simt.cu), 300 rows:
//     K                           64     128     192     256    2048    8192   14336
//     N(0, 1) . N(0, 0.02)      7.5/14  12/20   11/25   13/29  13/81  15/162  16/215
//     |N(0, 1)| . |N(0, 1)|     9.3/12  18/17   15/19   18/25  17/70  17/140  17/178
//     a large product first      16/19  28/27   27/32   27/36  21/79  15/105
//   From 192 on they are the smaller ones whatever the numbers, so there the line lies.  (What remains is mostly that the tensor cores
//   cut what they add up instead of rounding it: the mean error is -0.9 to -1.6e-7 of the result, towards zero.)  The factor keeps the parts
//   of the smallest numbers (1e-42 against 1e30: 9e-8) above the smallest bfloat16.  Cut to the leading bits without it, the parts
//   cost 1 to 2 % less time; products of K = 4 were off by 7e-8 (multiply-adds 4e-8), and numbers below 2^-110 lost bits or vanished.
//   Eight warps fetch W two or three stages ahead (registers that a third warp group hands over hold
//   it), cut it and store the parts as tiles of 128-byte-swizzled shared memory, while one warp issues the products of the stage
//   before; the same eight drain the accumulators.  From 33 rows on the tokens are cut once, by a kernel in front, into three planes
//   that arrive by TMA; for fewer the eight warps cut them too, which saves a launch.  Tiles that are too few for 148 SMs are cut
//   along K over a cluster of up to eight CTAs that add up through distributed shared memory.  Numbers of 2^111 and more and those that are not
//   finite have no such parts: the sums that one enters, and no others, are taken again with plain multiply-adds (300 rows against [16384, 2048]
//   with one infinite token 239 us, without 138).
//   300 rows against [16384, 2048] 127 us (158 TFLOP/s), [2048, 8192] 77, [128256, 2048] 940; 204, 125 and 1,404 us with the tokens cut
//   by every CTA again, W one stage ahead and six products a step (shared memory carried 270 KB a stage: 180 read by the
//   products, 92 stored); 866, 828 and 6,397 us with multiply-adds.  64 rows against [16384, 2048] 41.3 and 50.9 us, [3072, 2048] 16.2
//   and 16.4.
//
// In both, the order in which a row's products are added depends on the shapes (the number of rows among them: a row's bits may
// change where a batch grows from 8 to 9 rows, from 32 to 33, or K is cut otherwise), never on the other rows' contents.
#include "common.cuh"
#include <cuda.h>

namespace {

constexpr int kSMs = 148;

// ---------------------------------------------------------------------------------------------- few rows
constexpr int RV = 4;            // rows of W per warp
constexpr int WARPS = 8;

__device__ __forceinline__ float4 load_stream(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// lane i of the warp gets the sum over all lanes of v[i % N] (N a power of two up to 32): halves of the values change
// lanes at every step, so N values cost about N shuffles
template <int N>
__device__ __forceinline__ float transposed_sum(float (&v)[N]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = N / 2; o >= 1; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if (i < o) {
                const float give = upper ? v[i] : v[i + o], keep = upper ? v[i + o] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
    }
    float s = v[0];
#pragma unroll
    for (int o = N; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// DEPTH: pieces of 128 K positions in flight per warp
template <int MT, int DEPTH>
__global__ void __launch_bounds__(WARPS * 32, 2) gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                                                                      int M, int N, int K, int ksplit) {
    __shared__ float part[WARPS][MT * RV];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = blockIdx.x * (WARPS / ksplit) + warp / ksplit, ks = warp % ksplit;
    const int n0 = group * RV;
    const int pieces = (K + 127) >> 7;
    const float* w[RV];
#pragma unroll
    for (int r = 0; r < RV; ++r) w[r] = W + (size_t)min(n0 + r, N - 1) * K + lane * 4;
    const bool live = n0 < N;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 buf[DEPTH][RV];
    auto fetch = [&](int d, int piece) {
        const bool in = live && piece < pieces && piece * 128 + lane * 4 < K;
#pragma unroll
        for (int r = 0; r < RV; ++r) buf[d][r] = in ? load_stream(w[r] + (size_t)piece * 128) : zero;
    };
    // (W is nobody's output: its first pieces travel while the kernel before this one ends)
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) fetch(d, ks + d * ksplit);
    grid_dependency_wait();
    grid_launch_dependents();
    float acc[MT * RV];
#pragma unroll
    for (int i = 0; i < MT * RV; ++i) acc[i] = 0.f;
    const float* a = A + lane * 4;
    for (int p0 = ks; p0 < pieces; p0 += DEPTH * ksplit) {
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
            const int piece = p0 + d * ksplit;
            if (piece < pieces) {
                const bool in = piece * 128 + lane * 4 < K;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float4 x = in ? *reinterpret_cast<const float4*>(a + (size_t)min(m, M - 1) * K + (size_t)piece * 128) : zero;
#pragma unroll
                    for (int r = 0; r < RV; ++r) {
                        float& s = acc[m * RV + r];
                        s = fmaf(x.x, buf[d][r].x, s);
                        s = fmaf(x.y, buf[d][r].y, s);
                        s = fmaf(x.z, buf[d][r].z, s);
                        s = fmaf(x.w, buf[d][r].w, s);
                    }
                }
                fetch(d, piece + DEPTH * ksplit);
            }
        }
    }
    const float sum = transposed_sum<MT * RV>(acc);
    if (lane < MT * RV) part[warp][lane] = sum;
    __syncthreads();
    if (ks == 0 && live && lane < MT * RV) {
        float s = part[warp][lane];
        for (int q = 1; q < ksplit; ++q) s += part[warp + q][lane];
        const int m = lane / RV, n = n0 + lane % RV;
        if (m < M && n < N) C[(size_t)m * N + n] = s;
    }
}

template <int MT>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, cudaStream_t s) {
    // as many warps as keep every SM's memory pipeline full, but at least two pieces of K each
    const int groups = (N + RV - 1) / RV, pieces = (K + 127) / 128;
    int ksplit = 1;
    while (ksplit < WARPS && groups * ksplit < kSMs * 16 && pieces >= 4 * ksplit) ksplit *= 2;
    const int per = WARPS / ksplit;
    const cudaError_t e = tl_launch(gemm_f32_rows_kernel<MT, MT <= 4 ? 4 : 3>, dim3((groups + per - 1) / per), dim3(WARPS * 32), 0, s, A, W, C, M, N, K, ksplit);
    return e == cudaSuccess ? TL_OK : (int)e;
}

// ---------------------------------------------------------------------------------------------- more rows
constexpr int BP = 128;                    // rows of W per CTA: the 128 rows of a tcgen05.mma
constexpr int BK = 64;                     // K per stage: 64 bfloat16, one 128-byte swizzle row
constexpr int CHUNK = 2;                   // stages whose leading products are added up in tensor memory
constexpr int CONVERTERS = 8;              // warps
// A third warp group holds the issuing warp and hands its registers to the converters: the launch gives 168 a thread (with nine
// warps it would give no more, three of them being on one scheduler).
constexpr int THREADS = (CONVERTERS + 4) * 32;
constexpr int REGS_LAUNCH = 168;
constexpr unsigned long long WAIT_LIMIT_NS = 2000ull * 1000ull * 1000ull;
constexpr int SETTLE_POLLS = 1 << 20;      // tens of milliseconds
enum : int { ERR_MMA_WAIT = 122, ERR_CONVERTER_WAIT = 123 /* for a free stage or for a sum */, ERR_PLANES_WAIT = 125 };

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// A role that ends, given up or not, first waits (without a look at the others) for the copies and products that it has under way:
// shared and tensor memory must not be another CTA's while they land.
__device__ __forceinline__ void settle(unsigned long long* bar, unsigned parity) {
    unsigned ok = 0;
    for (int i = 0; i < SETTLE_POLLS && ok == 0; ++i)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    __syncwarp();
}
// by a whole warp: false (for all its lanes) once the limit has passed or another role has given up
__device__ __forceinline__ bool warp_wait(unsigned long long* bar, unsigned parity, volatile int* abort_flag, unsigned long long limit_ns = WAIT_LIMIT_NS) {
    bool ok = mbar_try_wait(bar, parity);
    if (!ok) {
        const unsigned long long t0 = global_ns();
        for (unsigned i = 1; !ok; ++i) {
            ok = mbar_try_wait(bar, parity);
            if (!ok && (i & 255u) == 0u && (*abort_flag || global_ns() - t0 > limit_ns)) break;
        }
    }
    return __all_sync(0xffffffffu, ok);
}
// by one thread of a role whose wait ended so: the first one's reason is what the host reads, the others stopped because of it
__device__ __forceinline__ void give_up(int* abort_flag, int* status, int code) {
    if (atomicExch(abort_flag, 1) == 0) atomicExch(status, code);
}

// shared-memory matrix descriptor: K-major tile, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ unsigned long long umma_desc(unsigned addr) {
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (unsigned long long)(1024u >> 4) << 32 | (unsigned long long)1u << 46 | (unsigned long long)2u << 61;
}
// both for a whole warp in step, of which one elected lane issues
__device__ __forceinline__ void umma_bf16(unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p, e;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// eight columns of this thread's lane of tensor memory
__device__ __forceinline__ void tmem_load8(unsigned addr, unsigned (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr));
}

// ---------------------------------------------------------------------------------------------- few rows, large weights
// A CTA per SM owns an even share of W's rows, a warp an eighth of K.  The warp copies its part of two rows at a time (2 KB, one
// TMA instruction) into a ring of six in shared memory and reads what arrived while the others travel; the ring runs on through
// the CTA's blocks of RB rows, over whose ends only the warps' sums meet.  So the copies never drain between one row and the
// next, a part of A is read once for RB rows, and the first 96 KB of an SM's weights travel while the kernel before ends.
constexpr int PK = 256;            // K positions of a piece
constexpr int RING = 6;
constexpr unsigned PIECE = 2 * PK * 4;
enum : int { ERR_STREAM_WAIT = 124 };

// a warp's copies under way, from place `at` of its ring (whose next phase is `phase`) up to place `end`; there is one at least
__device__ __forceinline__ void settle_ring(unsigned long long* full, int at, unsigned phase, int end) {
    for (int left = end > at ? end - at : end - at + RING; left > 0; --left) {
        settle(&full[at], phase);
        if (++at == RING) at = 0, phase ^= 1u;
    }
}

__device__ __forceinline__ void copy_piece(const CUtensorMap* map, unsigned char* to, unsigned long long* full, int k, int row) {
    const unsigned bar = smem_u32(full);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(PIECE) : "memory");
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(to)), "l"(map), "r"(bar), "r"(k), "r"(row) : "memory");
}

template <int MT, int RB>
__global__ void __launch_bounds__(WARPS * 32, MT <= 2 ? 2 : 1) gemm_f32_stream_kernel(const __grid_constant__ CUtensorMap map_w, const float* __restrict__ A,
                                                                        float* __restrict__ C, int* status, int M, int N, int K) {
    extern __shared__ __align__(128) unsigned char ring_all[];
    __shared__ __align__(8) unsigned long long full[WARPS][RING];
    __shared__ float part[2][WARPS][MT * RB];
    __shared__ int abort_flag;
    constexpr int NV = MT * RB, VPL = NV > 32 ? NV / 32 : 1;        // sums of a block; per lane
    static_assert(NV <= 32 || NV % 32 == 0, "whole warps of sums");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (int)((long long)N * blockIdx.x / gridDim.x), r1 = (int)((long long)N * (blockIdx.x + 1) / gridDim.x);
    const int pieces = (K + PK - 1) / PK, p0 = pieces * warp / WARPS, p1 = pieces * (warp + 1) / WARPS;
    const int n_blocks = (r1 - r0 + RB - 1) / RB;
    unsigned char* ring = ring_all + warp * RING * PIECE;
    if (threadIdx.x == 0) abort_flag = 0;
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < RING; ++i) mbar_init(&full[warp][i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    volatile int* aborted = &abort_flag;

    // what is to be copied next: pair `pr` of block `pb` at piece `pp`, into place `ps` of the ring
    int pb = p0 < p1 ? 0 : n_blocks, pp = p0, pr = 0, ps = 0;
    auto issue = [&]() {
        if (pb >= n_blocks) return;
        if (lane == 0) copy_piece(&map_w, ring + ps * PIECE, &full[warp][ps], pp * PK, r0 + pb * RB + 2 * pr);
        ps = ps + 1 == RING ? 0 : ps + 1;
        if (++pr == (min(RB, r1 - r0 - pb * RB) + 1) / 2) {
            pr = 0;
            if (++pp == p1) pp = p0, ++pb;
        }
    };
    // (W is nobody's output)
#pragma unroll
    for (int i = 0; i < RING; ++i) issue();
    grid_dependency_wait();
    grid_launch_dependents();

    int at = 0, lost = -1;            // lost: the place, and its phase, whose copy was not waited for to the end
    unsigned phase = 0;
    bool ok = true;
    float4 x[MT][2];
    for (int b = 0; b < n_blocks; ++b) {
        const int rows = min(RB, r1 - r0 - b * RB);
        float acc[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = 0.f;
        for (int pc = p0; pc < p1; ++pc) {
            if (b == 0 || p1 - p0 > 1)          // (a warp whose part of A is one piece keeps it)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = pc * PK + h * 128 + lane * 4;
                    x[m][h] = k < K ? *reinterpret_cast<const float4*>(A + (size_t)min(m, M - 1) * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
            for (int g = 0; g < RB / 2; ++g) {
                if (2 * g < rows) {
                    ok = ok && warp_wait(&full[warp][at], phase, aborted);
                    if (ok) {
                        const float4* w = reinterpret_cast<const float4*>(ring + at * PIECE) + lane;
                        float4 y[2][2];
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int h = 0; h < 2; ++h) y[r][h] = w[r * (PK / 4) + h * 32];
#pragma unroll
                        for (int m = 0; m < MT; ++m)
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                float& s = acc[m * RB + 2 * g + r];
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    s = fmaf(x[m][h].x, y[r][h].x, s);
                                    s = fmaf(x[m][h].y, y[r][h].y, s);
                                    s = fmaf(x[m][h].z, y[r][h].z, s);
                                    s = fmaf(x[m][h].w, y[r][h].w, s);
                                }
                            }
                        __syncwarp();              // all lanes have read the place before it is filled again
                        issue();
                    } else if (lost < 0) {
                        lost = at + (int)phase * RING;
                    }
                    if (++at == RING) at = 0, phase ^= 1u;
                }
            }
        }
        if (!ok && lane == 0) give_up(&abort_flag, status, ERR_STREAM_WAIT);
        if (NV <= 32) {
            constexpr int NS = NV <= 32 ? NV : 32;
            const float s = transposed_sum<NS>(reinterpret_cast<float (&)[NS]>(acc));
            if (lane < NS) part[b & 1][warp][lane] = s;
        } else {
#pragma unroll
            for (int v = 0; v < VPL; ++v) {
                float some[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) some[i] = acc[(v * 32 + i) % NV];
                const float s = transposed_sum<32>(some);
                part[b & 1][warp][(v * 32 + lane) % NV] = s;
            }
        }
        __syncthreads();          // (two sets of sums: those of the block before may still be read)
        if (threadIdx.x < NV) {
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < WARPS; ++q) s += part[b & 1][q][threadIdx.x];
            const int m = threadIdx.x / RB, r = threadIdx.x % RB;
            if (m < M && r < rows && *aborted == 0) C[(size_t)m * N + r0 + b * RB + r] = s;
        }
    }
    if (!ok) settle_ring(full[warp], lost % RING, (unsigned)(lost / RING), ps);
}

// What a warp of the kernel above does when a wait runs out, with a wait that nothing ends: it fills its ring, gives up after
// limit_ns, lets its copies land, and writes out what they brought (RING pieces, [2 RING, PK] of W).  A second warp waits for the
// same and ends when the first one has given up.
__global__ void __launch_bounds__(64) give_up_selftest_kernel(const __grid_constant__ CUtensorMap map_w, float* __restrict__ out, int* status, unsigned long long limit_ns) {
    __shared__ __align__(128) unsigned char ring[RING * PIECE];
    __shared__ __align__(8) unsigned long long full[RING], never;
    __shared__ int abort_flag;
    const int lane = threadIdx.x & 31;
    grid_dependency_wait();
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(&never, 1);
        for (int i = 0; i < RING; ++i) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < RING; ++i) copy_piece(&map_w, ring + i * PIECE, &full[i], 0, 2 * i);
    }
    __syncthreads();
    const bool first = threadIdx.x < 32;
    const bool ok = warp_wait(&never, 0, &abort_flag, first ? limit_ns : WAIT_LIMIT_NS);
    if (!ok && lane == 0) give_up(&abort_flag, status, first ? ERR_STREAM_WAIT : ERR_PLANES_WAIT);
    if (first) {
        if (!ok) settle_ring(full, 0, 0, 0);
        for (int i = lane; i < RING * 2 * PK; i += 32) out[i] = reinterpret_cast<const float*>(ring)[i];
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

bool map_pieces(CUtensorMap* map, const float* W, int N, int K) {
    EncodeTiledFn fn = encode_tiled();
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {PK, 2}, elem[2] = {1, 1};
    return fn != nullptr && fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MT, int RB>
int launch_stream(const float* A, const float* W, float* C, int* status, int M, int N, int K, cudaStream_t s) {
    constexpr int SMEM = WARPS * RING * PIECE;
    auto kernel = gemm_f32_stream_kernel<MT, RB>;
    static bool raised = false;
    if (!raised) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        raised = true;
    }
    CUtensorMap map;
    if (!map_pieces(&map, W, N, K)) return TL_BAD_SIZE;
    const int ctas = (N + 1) / 2 < kSMs ? (N + 1) / 2 : kSMs;
    return (int)tl_launch(kernel, dim3(ctas), dim3(WARPS * 32), SMEM, s, map, A, C, status, M, N, K);
}

// sixteen of them with one wait
__device__ __forceinline__ void tmem_load16(unsigned addr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr));
}
// acc[0 .. N) += N columns of this thread's lane
template <int N>
__device__ __forceinline__ void add_columns(float (&acc)[N], unsigned addr) {
    constexpr int BIG = N / 16 * 16;
#pragma unroll
    for (int j = 0; j < BIG; j += 16) {
        unsigned r[16];
        tmem_load16(addr + (unsigned)j, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[j + e] += __uint_as_float(r[e]);
    }
    if (BIG < N) {
        unsigned r[8];
        tmem_load8(addr + (unsigned)BIG, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[(BIG + e) % N] += __uint_as_float(r[e]);
    }
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four numbers, each times 2^16, as three bfloat16: v 2^16 == hi + mid + lo exactly, each part the one before's remainder rounded
// to nearest (|mid| <= 2^-8, |lo| <= 2^-17 of the power of two below |v|; what is left after mid has 7 bits at most).  With the factor
// the last bit of the smallest number there is (2^-149) is the last bit of the smallest bfloat16 (2^-133).  A number of
// 2^111 and more, or one that is infinite or NaN, has an infinite or NaN part.
constexpr float CUT_SCALE = 65536.f, CUT_UNSCALE = 1.f / (65536.f * 65536.f);
struct Parts { uint2 hi, mid, lo; };
__device__ __forceinline__ float2 minus2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ unsigned round2(float2 v) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ float2 rest2(float2 v, unsigned r) { return minus2(v, make_float2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u))); }
__device__ __forceinline__ Parts split4(const float4& v) {
    Parts p;
    float2 x = __fmul2_rn(make_float2(v.x, v.y), make_float2(CUT_SCALE, CUT_SCALE)), y = __fmul2_rn(make_float2(v.z, v.w), make_float2(CUT_SCALE, CUT_SCALE));
    p.hi = make_uint2(round2(x), round2(y));
    x = rest2(x, p.hi.x), y = rest2(y, p.hi.y);
    p.mid = make_uint2(round2(x), round2(y));
    x = rest2(x, p.mid.x), y = rest2(y, p.mid.y);
    p.lo = make_uint2(round2(x), round2(y));
    return p;
}

// Products a . w of K numbers with plain multiply-adds for up to eight rows w (the lowest bits set in `rows`), by a whole warp in
// step: 16 bytes a lane, over once all of them are NaN.  Lane r gets row r's; the others keep `mine`.
__device__ __forceinline__ float plain_products(const float* __restrict__ a, const float* __restrict__ W, int K, unsigned rows, float mine) {
    const int lane = threadIdx.x & 31;
    int r[8];
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        r[i] = rows != 0 ? __ffs(rows) - 1 : r[0];
        rows &= rows - 1;
        s[i] = 0.f;
    }
    for (int k = 0; k < K; k += 128) {
        const int at = k + lane * 4;
        bool nan = true;
        if (at < K) {
            const float4 x = *reinterpret_cast<const float4*>(a + at);
            float4 y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = *reinterpret_cast<const float4*>(W + (size_t)r[i] * K + at);
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = fmaf(x.w, y[i].w, fmaf(x.z, y[i].z, fmaf(x.y, y[i].y, fmaf(x.x, y[i].x, s[i]))));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) nan = __any_sync(0xffffffffu, s[i] != s[i]) && nan;
        if (nan) break;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float sum = warp_sum(s[i]);
        if (lane == r[i]) mine = sum;
    }
    return mine;
}
__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

// BQ: tokens per CTA at most (the launch says how many, a multiple of 16); AHEAD: stages of W (and of tokens that are not cut
// beforehand) in registers
template <int BQ, int AHEAD>
struct Shape {
    static constexpr bool PLANES = BQ > 32;
    static constexpr unsigned W_PART = BP * BK * 2, STAGE = 3 * (W_PART + BQ * BK * 2);
    static constexpr unsigned SUMS = BQ * BP * 4;
    static constexpr unsigned SMEM = (2 * STAGE > SUMS ? 2 * STAGE : SUMS) + 1024;
    // what the converters get and what the others keep: three stages of W take more of the former (else 24 bytes are spilled), the
    // products of long tiles of tokens more of the latter (32 bytes, 4 % of the time)
    static constexpr int REGS_CONVERT = AHEAD > 2 ? 224 : 216, REGS_REST = AHEAD > 2 ? 56 : 72;
    static_assert(2 * REGS_CONVERT + REGS_REST <= 3 * REGS_LAUNCH, "registers are traded, not made");
    static constexpr unsigned COLS = BQ > 64 ? 512 : BQ == 64 ? 256 : BQ == 32 ? 128 : 64;      // four accumulators, a power of two
};

template <int BQ, int AHEAD>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_parts_kernel(const __grid_constant__ CUtensorMap map_planes, const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                                                                    int* status, int M, int N, int K, int bq, int token_tiles, int ksplit) {
    using S = Shape<BQ, AHEAD>;
    constexpr bool PLANES = S::PLANES;
    constexpr int WL = BP / 16, AL = PLANES ? 1 : BQ / 16, HALF = BQ / 2;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
    __shared__ __align__(8) unsigned long long full_bar[2], empty_bar[2], sum_full[2], sum_empty[2];
    __shared__ unsigned tmem_slot;
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % ksplit, tile = blockIdx.x / ksplit;
    const int m0 = (tile % token_tiles) * bq, n0 = (tile / token_tiles) * BP;      // the tiles that read a slab of W follow one another
    const int blocks_all = (K + BK - 1) / BK;
    const int first = (int)((long long)blocks_all * rank / ksplit), blocks = (int)((long long)blocks_all * (rank + 1) / ksplit) - first;
    const int chunks = (blocks + CHUNK - 1) / CHUNK;
    volatile int* aborted = &abort_flag;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full_bar[s], CONVERTERS + (PLANES ? 1 : 0));
            mbar_init(&empty_bar[s], 1);
            mbar_init(&sum_full[s], 1);
            mbar_init(&sum_empty[s], CONVERTERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == CONVERTERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(S::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = tmem_slot;
    bool ok = true;

    if (warp < CONVERTERS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::REGS_CONVERT));
        float acc[HALF];
#pragma unroll
        for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
        const int quarter = warp & 3, half = warp >> 2;                    // a converter's share of the accumulators
        const unsigned lanes = (unsigned)(quarter * 32) << 16;
        // rows warp * 2 + lane / 16 + 16 i of both tiles, 16 bytes at lane % 16 along K
        const int r0 = warp * 2 + (lane >> 4), kl = (lane & 15) * 4;
        const float *wp = W + (size_t)(n0 + r0) * K + kl, *ap = A + (size_t)(m0 + r0) * K + kl;
        const int w_rows = N - n0 - r0, a_rows = min(M - m0, bq) - r0;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 wb[AHEAD][WL], ab[AHEAD][AL];
        auto w_at = [&](int i, int b) {
            const int k = (first + b) * BK;
            return (b < blocks && 16 * i < w_rows && k + kl < K) ? load_stream(wp + (size_t)(16 * i) * K + k) : zero;
        };
        auto a_at = [&](int i, int b) {
            const int k = (first + b) * BK;
            return (b < blocks && 16 * i < a_rows && k + kl < K) ? *reinterpret_cast<const float4*>(ap + (size_t)(16 * i) * K + k) : zero;
        };
#pragma unroll
        for (int d = 0; d < AHEAD; ++d)
#pragma unroll
            for (int i = 0; i < WL; ++i) wb[d][i] = w_at(i, d);
        grid_dependency_wait();
        grid_launch_dependents();
#pragma unroll
        for (int d = 0; d < AHEAD; ++d)
#pragma unroll
            for (int i = 0; i < AL; ++i)
                if (!PLANES) ab[d][i] = a_at(i, d);
        unsigned char* put = tiles + r0 * 128 + ((((lane & 15) >> 1) ^ (r0 & 7)) << 4) + (lane & 1) * 8;
        int drained = 0;
        auto drain = [&]() {
            const int c = drained++;
            ok = ok && warp_wait(&sum_full[c & 1], (c >> 1) & 1, aborted);
            if (!ok) return;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add_columns<HALF>(acc, tmem + lanes + (unsigned)((c & 1) * BQ + half * HALF));
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[c & 1]);
        };
        for (int b0 = 0; b0 < blocks && ok; b0 += AHEAD) {
#pragma unroll
            for (int d = 0; d < AHEAD; ++d) {
                const int b = b0 + d;
                if (b >= blocks || !ok) break;
                const int s = b & 1;
                if (b >= 2) ok = warp_wait(&empty_bar[s], ((b >> 1) - 1) & 1, aborted);
                if (!ok) break;
                unsigned char* to = put + s * S::STAGE;
#pragma unroll
                for (int i = 0; i < WL; ++i) {
                    const Parts q = split4(wb[d][i]);
                    *reinterpret_cast<uint2*>(to + i * 2048) = q.hi;
                    *reinterpret_cast<uint2*>(to + i * 2048 + S::W_PART) = q.mid;
                    *reinterpret_cast<uint2*>(to + i * 2048 + 2 * S::W_PART) = q.lo;
                    wb[d][i] = w_at(i, b + AHEAD);
                }
#pragma unroll
                for (int i = 0; i < (PLANES ? 0 : AL); ++i) {
                    if (16 * i < bq) {
                        const Parts q = split4(ab[d][i]);
                        *reinterpret_cast<uint2*>(to + i * 2048 + 3 * S::W_PART) = q.hi;
                        *reinterpret_cast<uint2*>(to + i * 2048 + 3 * S::W_PART + bq * 128) = q.mid;
                        *reinterpret_cast<uint2*>(to + i * 2048 + 3 * S::W_PART + bq * 256) = q.lo;
                    }
                    ab[d][i] = a_at(i, b + AHEAD);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_bar[s]);
                if ((b % CHUNK) == CHUNK - 1 && b >= 2 * CHUNK - 1) drain();
            }
        }
        while (ok && drained < chunks) drain();
        if (ok && blocks > 0) {
            // the small products, added up over the whole range; the last chunk's signal covers them
            add_columns<HALF>(acc, tmem + lanes + (unsigned)(2 * BQ + bq + half * HALF));
            add_columns<HALF>(acc, tmem + lanes + (unsigned)(2 * BQ + half * HALF));
        }
        if (!ok && lane == 0) give_up(&abort_flag, status, ERR_CONVERTER_WAIT);
        asm volatile("tcgen05.fence::before_thread_sync;\nbar.sync 0;" ::: "memory");         // every role is done
        const bool good = abort_flag == 0;
        const int row = quarter * 32 + lane, n = n0 + row;
        float odd = 0.f;              // NaN if one of this thread's results is infinite or NaN
        int t0 = half * HALF, t1 = min(min(bq, M - m0), t0 + HALF), dt = 1;      // its tokens
        if (ksplit == 1) {
            float o[4] = {0.f, 0.f, 0.f, 0.f};        // (four short chains, and no look at which of them count: those are looked at again)
#pragma unroll
            for (int j = 0; j < HALF; ++j) o[j & 3] = fmaf(acc[j], 0.f, o[j & 3]);
            odd = (o[0] + o[1]) + (o[2] + o[3]);
            if (good && n < N) {
#pragma unroll
                for (int j = 0; j < HALF; ++j) {
                    if (t0 + j < t1) C[(size_t)(m0 + t0 + j) * N + n] = acc[j] * CUT_UNSCALE;
                }
            }
        } else {
            // The cluster's CTAs hold sums over their parts of K: each leaves its own in its shared memory (the stages are
            // done with) and adds up every ksplit-th token's from all, in the order of the parts.  A CTA that gave up takes
            // part in the barriers and leaves NaN.
            float* sums = reinterpret_cast<float*>(tiles);                 // [token][row]
#pragma unroll
            for (int j = 0; j < HALF; ++j) sums[(half * HALF + j) * BP + row] = good ? acc[j] : __int_as_float(0x7fffffff);
            cluster_sync();
            t0 = rank + half * ksplit, t1 = min(bq, M - m0), dt = 2 * ksplit;
            if (n < N) {
                for (int t = t0; t < t1; t += dt) {
                    float v[8], s = 0.f;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        if (q < ksplit) {
                            unsigned there;
                            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(&sums[t * BP + row])), "r"(q));
                            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[q]) : "r"(there) : "memory");
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) if (q < ksplit) s += v[q];
                    C[(size_t)(m0 + t) * N + n] = s * CUT_UNSCALE;
                    odd = fmaf(s, 0.f, odd);
                }
            }
            cluster_sync();          // nobody leaves while another still reads its shared memory
        }
        // An operand that is not finite makes every sum that it enters NaN (inf * 0 between its parts, where the product itself
        // may be infinite), and a sum may have overflowed on its way.  Such a result is taken again with plain multiply-adds, by
        // the whole warp; the others keep their bits.
        if (good && __any_sync(0xffffffffu, odd != odd)) {
            for (int t = t0; t < t1; t += dt) {
                const float* a = A + (size_t)(m0 + t) * K;
                float* c = C + (size_t)(m0 + t) * N + n;
                float v = n < N ? *c : 0.f;
                unsigned again = __ballot_sync(0xffffffffu, !is_finite(v));
                if (again == 0) continue;
                while (again != 0) {
                    v = plain_products(a, W + (size_t)(n0 + quarter * 32) * K, K, again, v);
#pragma unroll
                    for (int i = 0; i < 8; ++i) again &= again - 1;
                }
                if (n < N) *c = v;
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::REGS_REST));
        if (warp == CONVERTERS) {
            // ---- tensor-core issuer: the whole warp in step, one elected lane issuing
            // The parts of the tokens lie one behind the other, and so do the accumulators of the products of the second and third
            // order: a part of W meets two of them in one instruction, which reads it from shared memory once.
            const unsigned one = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(bq >> 3) << 17) | ((unsigned)(BP >> 4) << 24);
            const unsigned pair = one + ((unsigned)(bq >> 3) << 17);
            int b = 0;
            for (; b < blocks; ++b) {
                const int s = b & 1, c = b / CHUNK;
                ok = warp_wait(&full_bar[s], (b >> 1) & 1, aborted);
                if (ok && b % CHUNK == 0 && c >= 2) ok = warp_wait(&sum_empty[c & 1], ((c >> 1) - 1) & 1, aborted);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned wt = smem_u32(tiles) + s * S::STAGE, at = wt + 3 * S::W_PART;
                const unsigned lead = tmem + (unsigned)((c & 1) * BQ), mid = tmem + 2 * BQ, low = mid + bq;
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) {
                    const unsigned long long w0 = umma_desc(wt + k * 32), w1 = umma_desc(wt + S::W_PART + k * 32), w2 = umma_desc(wt + 2 * S::W_PART + k * 32);
                    const unsigned long long a0 = umma_desc(at + k * 32), a1 = umma_desc(at + bq * 128 + k * 32);
                    umma_bf16(mid, w0, a1, pair, b > 0 || k > 0);          // w0 a1 | w0 a2
                    umma_bf16(mid, w1, a0, pair, true);                    // w1 a0 | w1 a1
                    umma_bf16(low, w2, a0, one, true);
                    umma_bf16(lead, w0, a0, one, b % CHUNK > 0 || k > 0);
                }
                umma_commit(&empty_bar[s]);
                if (b % CHUNK == CHUNK - 1 || b == blocks - 1) umma_commit(&sum_full[c & 1]);
            }
            if (!ok && lane == 0) give_up(&abort_flag, status, ERR_MMA_WAIT);
            if (b > 0) settle(&empty_bar[(b - 1) & 1], ((b - 1) >> 1) & 1);       // its last products
        }
        if (PLANES && warp == CONVERTERS + 1) {
            // ---- the tokens' parts, cut beforehand: [bq x 64] boxes of the three planes, one behind the other.  (Rows past
            // the last token are another plane's or the zero fill; their sums are not stored.)
            grid_dependency_wait();
            int b = 0;
            for (; b < blocks; ++b) {
                const int s = b & 1;
                if (b >= 2) ok = warp_wait(&empty_bar[s], ((b >> 1) - 1) & 1, aborted);
                if (!ok) break;
                if (lane == 0) {
                    const unsigned bar = smem_u32(&full_bar[s]), to = smem_u32(tiles) + s * S::STAGE + 3 * S::W_PART;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((unsigned)(3 * bq * 128)) : "memory");
                    for (int q = 0; q < 3; ++q)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                                     ::"r"(to + q * bq * 128), "l"(&map_planes), "r"(bar), "r"((first + b) * BK), "r"(q * M + m0) : "memory");
                }
                __syncwarp();
            }
            if (!ok && lane == 0) give_up(&abort_flag, status, ERR_PLANES_WAIT);
            // its last copies; converters that have given up never signal these stages: then it waits as long as copies may take
            for (int q = b > 2 ? b - 2 : 0; q < b; ++q) settle(&full_bar[q & 1], (q >> 1) & 1);
        }
        asm volatile("tcgen05.fence::before_thread_sync;\nbar.sync 0;" ::: "memory");
        if (ksplit > 1) {
            cluster_sync();
            cluster_sync();
        }
    }
    __syncthreads();
    if (warp == CONVERTERS) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS) : "memory");
    }
}

// A [M, K] cut into three planes [M, KP] of bfloat16, KP = K rounded up to 8 (a tensor map's rows are multiples of 16 bytes)
__global__ void __launch_bounds__(256) cut_planes_kernel(const float* __restrict__ A, __nv_bfloat16* __restrict__ planes, int M, int K, int KP) {
    grid_launch_dependents();
    grid_dependency_wait();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    const int per_row = KP / 8, m = (int)(i / per_row), k = (int)(i % per_row) * 8;
    if (m >= M) return;
    const float4 u = *reinterpret_cast<const float4*>(A + (size_t)m * K + k);
    const float4 v = k + 4 < K ? *reinterpret_cast<const float4*>(A + (size_t)m * K + k + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    const Parts p = split4(u), q = split4(v);
    __nv_bfloat16* to = planes + (size_t)m * KP + k;
    const size_t plane = (size_t)M * KP;
    *reinterpret_cast<uint4*>(to) = make_uint4(p.hi.x, p.hi.y, q.hi.x, q.hi.y);
    *reinterpret_cast<uint4*>(to + plane) = make_uint4(p.mid.x, p.mid.y, q.mid.x, q.mid.y);
    *reinterpret_cast<uint4*>(to + 2 * plane) = make_uint4(p.lo.x, p.lo.y, q.lo.x, q.lo.y);
}

template <int BQ, int AHEAD>
int launch_parts(const float* A, const float* W, float* C, void* planes, int* status, int M, int N, int K, cudaStream_t s) {
    using S = Shape<BQ, AHEAD>;
    const int token_tiles = (M + BQ - 1) / BQ;
    const int bq = ((M + token_tiles - 1) / token_tiles + 15) / 16 * 16;       // tiles of equal size
    const long long tiles = (long long)token_tiles * ((N + BP - 1) / BP);
    auto kernel = gemm_f32_parts_kernel<BQ, AHEAD>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    // how many clusters of q CTAs the GPU holds at a time: fewer than SMs / q, since a cluster stays inside a group of 16 to
    // 18 SMs.  Asked for once (threads that ask at the same time write the same numbers).
    static int fit[9];
    if (fit[1] == 0) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        cfg.numAttrs = 1;
        for (int q = 8; q >= 1 && e == cudaSuccess; --q) {
            cfg.gridDim = dim3(q);
            attr[0].val.clusterDim.x = q;
            int n = 0;
            e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
            fit[q] = n < 1 ? 1 : n;
        }
        if (e != cudaSuccess) return (int)e;
    }
    // K is cut so that the tiles' parts come in as few and as short rounds as can be; a part has four stages at least
    const int blocks = (K + BK - 1) / BK;
    int ksplit = 1;
    long long best = 1LL << 62;
    for (int q = 1; q <= 8 && (q == 1 || blocks / q >= 4); ++q) {
        const long long cost = (tiles + fit[q] - 1) / fit[q] * ((blocks + q - 1) / q + (q > 1 ? 3 : 2));
        if (cost < best) best = cost, ksplit = q;
    }
    if (tiles * ksplit > 0x7fffffffLL) return TL_BAD_SIZE;
    cfg.gridDim = dim3((unsigned)(tiles * ksplit));
    attr[0].val.clusterDim.x = ksplit;
    cfg.numAttrs = 2;
    CUtensorMap map = {};
    if (S::PLANES) {
        const int KP = (K + 7) / 8 * 8;
        const cudaError_t e = tl_launch(cut_planes_kernel, dim3((unsigned)(((long long)M * KP / 8 + 255) / 256)), dim3(256), 0, s, A, (__nv_bfloat16*)planes, M, K, KP);
        if (e != cudaSuccess) return (int)e;
        EncodeTiledFn fn = encode_tiled();
        const cuuint64_t dims[2] = {(cuuint64_t)KP, (cuuint64_t)M * 3}, strides[1] = {(cuuint64_t)KP * 2};
        const cuuint32_t box[2] = {BK, (cuuint32_t)bq}, elem[2] = {1, 1};
        if (fn == nullptr || fn(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, planes, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return TL_BAD_SIZE;
    }
    return (int)cudaLaunchKernelEx(&cfg, kernel, map, A, W, C, status, M, N, K, bq, token_tiles, ksplit);
}

}  // namespace

// (a short product of many rows is less exact in parts than in multiply-adds: see the top)
extern "C" int tl_gemm_f32_supports(const void* A, const void* W, int M, int K) {
    return K >= (M > 8 ? 192 : 4) && K % 4 == 0 && aligned16(A) && aligned16(W) ? 1 : 0;
}

// W: 12 rows of 256 numbers on 16 bytes; out receives them; status is set.
extern "C" int tl_gemm_f32_give_up_selftest(const void* W, void* out, int* status, unsigned long long limit_ns, void* stream) {
    CUtensorMap map;
    if (!aligned16(W) || !map_pieces(&map, (const float*)W, 2 * RING, PK)) return TL_BAD_ALIGN;
    return (int)tl_launch(give_up_selftest_kernel, dim3(1), dim3(64), 0, (cudaStream_t)stream, map, (float*)out, status, limit_ns);
}

// Bytes of scratch (16-byte aligned) that tl_gemm_f32 needs for M rows of K numbers.
extern "C" long long tl_gemm_f32_scratch(int M, int K) { return M > 32 ? 6LL * M * ((K + 7) / 8 * 8) : 0; }

// status: one int that is set to a non-zero code if a wait ran out.
extern "C" int tl_gemm_f32(const void* A, const void* W, void* C, void* scratch, int M, int N, int K, int* status, void* stream) {
    if (M <= 0 || N <= 0) return TL_OK;
    if (!tl_gemm_f32_supports(A, W, M, K) || status == nullptr) return TL_BAD_ALIGN;
    if (M > 32 && (scratch == nullptr || !aligned16(scratch))) return TL_BAD_ALIGN;
    cudaStream_t s = (cudaStream_t)stream;
    const float *a = (const float*)A, *w = (const float*)W;
    float* c = (float*)C;
    // A warp of the streaming kernel owns an eighth of K in pieces of 256.  Below 1,536 half of the warps have nothing to do (4 rows
    // against [3072, 1024] 6.3 us, 5.7 in the other kernel; against [3072, 1536] 6.5 and 7.4).  With nine to twelve pieces some
    // warps have two and the others, which wait for them, one: a CTA with many rows to go through loses more by that than the
    // rings gain (4 rows against [16384, 2304] 42.3 and 32.7, [16384, 3072] 47.0 and 41.8, [9216, 3072] 27.6 and 24.3; the other way round
    // [5120, 3072] 16.7 and 20.0, [3072, 2304] 10.1 and 10.4, [16384, 3328] 46.9 and 45.1 with 4 rows, 40.2 and 42.8 with one; 1 and
    // 8 rows lie alike).
    const int pieces = (K + PK - 1) / PK;
    if (M <= 8 && K >= 1536 && !(pieces > 8 && pieces <= 12 && N >= 8192)) {
        if (M == 1) return launch_stream<1, 16>(a, w, c, status, M, N, K, s);
        if (M == 2) return launch_stream<2, 16>(a, w, c, status, M, N, K, s);
        if (M <= 4) return launch_stream<4, 16>(a, w, c, status, M, N, K, s);
        return launch_stream<8, 8>(a, w, c, status, M, N, K, s);
    }
    if (M == 1) return launch_rows<1>(a, w, c, M, N, K, s);
    if (M == 2) return launch_rows<2>(a, w, c, M, N, K, s);
    if (M <= 4) return launch_rows<4>(a, w, c, M, N, K, s);
    if (M <= 8) return launch_rows<8>(a, w, c, M, N, K, s);
    if (M <= 16) return launch_parts<16, 2>(a, w, c, scratch, status, M, N, K, s);
    if (M <= 32) return launch_parts<32, 2>(a, w, c, scratch, status, M, N, K, s);
    if (M <= 64) return launch_parts<64, 3>(a, w, c, scratch, status, M, N, K, s);
    return launch_parts<128, 2>(a, w, c, scratch, status, M, N, K, s);
}
