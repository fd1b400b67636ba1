// Decode attention over paged bfloat16 keys and values with TMA-fed tiles (head_dim 64 or 128).
//
// For steps where every request brings so few tokens that its rows (token x query heads of one kv
// group) fit one 16-row tensor-core tile: single decoded tokens above all.  Same contract and
// the same arithmetic as the kernels in attention_mma.cu (float32 scores, running maximum and
// sum, accumulators; probabilities multiplied as value + remainder), but the tiles are moved by
// the TMA unit instead of by every thread: the decode step is bound by streaming K and V once
// from HBM, and issuing 16-byte copies from all threads cost more instructions than the math.
//
// A request's keys may be cut into several pieces (whole tiles, as many pieces as the host plans for the
// longest context there could be; a shorter request has shorter pieces, or fewer).  Warp 4 of a CTA is the
// producer: for every 64-key tile it looks up the pages, and issues cp.async.bulk.tensor copies (no
// multicast) of [page rows x 64 elements] boxes into 128-byte-swizzled shared memory, completing on an
// mbarrier per stage.  Warps 0-3 share the rows and each takes 16 keys of every tile; they hand a stage back
// through a second mbarrier.  A piece leaves float32 partials; the pieces of a request are added up in order.
//
// Two ways to hand the pieces out, each a kernel.  A CTA to a piece, and merge_partials_kernel adds up (the weights of the
// product that follows stream in meanwhile).  Or, where there are many more pieces than CTAs fit (many requests; most
// pieces are short or empty then), as many CTAs as fit take even shares of the pieces, found on the device from the requests'
// lengths; the producer runs ahead across the borders of pieces and requests, and the CTA that is last to finish with a
// request adds its pieces up (a counter per request and kv head).  The sums are the same bit for bit; where the line between
// the two lies, and what both take on either side of it, stands at make_plan.  What bounds both is the latency of a tile: 24 requests
// of 130 to 1,900 tokens read 50 MB in 14 us.
//
// The products are taken transposed: scores^T = K Q^T and out^T = V^T P^T, so that the 16 rows of
// a tensor-core tile are keys (or value columns), all of them real, and the few query rows (four
// for a group of four heads) sit in the 8-wide direction.  With the queries as the 16 rows, three
// quarters of every product were padding, and instruction issue, not memory, set the pace.  The
// probabilities change sides between the two products (result columns -> operand columns),
// which is one movmatrix per 8 x 8 block.
// Every mbarrier wait is bounded in time; on a time-out the CTA records a code in the status
// word and writes no results from there on.  With shares it still goes through its pieces: the other CTAs
// of a request count on it, and whoever is last learns from the count that a part is missing.
#include "common.cuh"
#include <cuda.h>
#include <limits.h>
#include <math.h>
#include <map>
#include <mutex>
#include <tuple>

namespace {

constexpr int BN = 64;                  // keys per tile
constexpr int NCW = 4;                  // consumer warps
constexpr int NTHREADS = (NCW + 1) * 32;
constexpr int MIN_SPLIT = 128;
constexpr int MERGE_MAX_SPLITS = 64;    // pieces of one request's keys, at most
constexpr int FAILED_PART = 1 << 16;    // what a CTA that gave up adds to a counter beside its 1
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;
constexpr unsigned long long WAIT_NS = 2000ull * 1000ull * 1000ull;
enum : int { ERR_PRODUCER_WAIT = 211, ERR_CONSUMER_WAIT = 212, ERR_COUNT = 213 };

struct DecodeParams {
    const __nv_bfloat16* q;
    __nv_bfloat16* out;
    const int* block_table;
    const int* q_start;
    const int* kv_len;
    float* part_o;   // a CTA to a piece: [T * H, n_splits, head_dim]; shares: [n_seqs * units, n_splits, rows, head_dim]
    float* part_ml;  // the same with 2 in the place of head_dim: maximum (natural-log scale) and sum
    int* status;
    int table_stride;
    int n_heads, n_kv_heads, page_size, page_shift, box_rows;
    int total_rows;             // rows of the page tensor: a copy that starts there reads only the zero fill
    int group, ng, n_gchunks;
    int max_tokens;             // tokens of a request
    int n_splits;
    int window;
    int streamed;               // the call reads more keys and values than L2 holds: their copies are marked to leave it first
    float scale_log2;
};
// With the two tensor maps a launch's arguments are 384 bytes.  What only the shares need is kept out of them: with 408 the very same
// kernel took longer (24 requests of 130 to 1,900 tokens, heads of 64, 14.25 us where 384 take 13.6; 20 requests, heads of
// 128, 19.3 and 18.9; 16 of 600, heads of 64, 7.0 and 7.2 the other way round).
static_assert(sizeof(DecodeParams) == 128, "the arguments of a launch with the tensor maps: 384 bytes");
struct ShareParams : DecodeParams {
    int* counters;              // [n_seqs * units], zero between launches
    int n_seqs, units;          // requests; kv heads x chunks of a group's heads
    int rows;                   // rows of a tile in use: max_tokens * ng
    unsigned long long limit_ns;    // self-test only: how long a wait may take
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
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
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, const volatile int* failed, unsigned long long limit_ns = WAIT_NS) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (unsigned i = 1;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 0u) {
            unsigned long long t1;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
            if (*failed || t1 - t0 > limit_ns) return false;
        }
    }
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
// the same with the mark "first to leave L2": keys and values that are read once and are more than L2 holds
__device__ __forceinline__ void tma_load_2d_streamed(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y) {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(pol) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2(float x) {     // 2^x, one instruction; 2^-inf = 0
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
// byte offset of (row, 16-byte chunk c of a 128-byte row) inside a 128-byte-swizzled [rows x 128 B] tile
__device__ __forceinline__ unsigned swz(int row, int c) { return (unsigned)(row * 128 + ((c ^ (row & 7)) << 4)); }

__device__ __forceinline__ unsigned movmatrix_trans(unsigned a) {     // 8 x 8 bfloat16 block, transposed across the warp
    unsigned d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NCW * 32) : "memory"); }

// What a launch reads of one request's keys.
struct Span {
    int lo, hi;      // visible keys lo .. hi - 1 (of any of its tokens)
    int base;        // position of its first new token
    int first;       // the row of that token
    int n_tokens;    // 0: the request brings none
    int piece;       // keys of a piece: whole tiles, or all of them
    int pieces;      // how many of them have keys (at least one)
};
__device__ __forceinline__ Span span_of(const DecodeParams& p, int b) {
    Span s;
    s.first = p.q_start[b];
    const int ql = p.q_start[b + 1] - s.first;
    s.base = p.kv_len[b] - ql;
    s.n_tokens = max(0, min(ql, p.max_tokens));
    s.lo = p.window > 0 ? max(0, s.base - p.window + 1) : 0;
    s.hi = s.base + s.n_tokens;
    const int len = max(s.hi - s.lo, 0);
    s.piece = p.n_splits > 1 ? max(((len + p.n_splits - 1) / p.n_splits + BN - 1) / BN * BN, BN) : max(len, 1);
    s.pieces = p.n_splits > 1 ? max((len + s.piece - 1) / s.piece, 1) : 1;
    return s;
}

// The pieces a CTA works on, one after the other (every warp walks on its own).
struct Walk {
    int b, unit, split;  // request; kv head and chunk of its heads; piece
    Span span;
    int lo, hi;          // keys of the piece
    int start, tiles;    // its tiles: the first starts on a box (page) boundary; keys below lo are masked
    int at, end;         // shares: places on the line of pieces, of the piece and where the share ends
    int first_split;     // shares: the first piece of this (request, unit) in the share
};
__device__ __forceinline__ void walk_piece(const DecodeParams& p, Walk& w) {
    w.lo = w.span.lo + w.split * w.span.piece;
    w.hi = min(w.span.hi, w.lo + w.span.piece);
    w.start = w.lo & ~(p.box_rows - 1);
    w.tiles = w.hi > w.start ? (w.hi - w.start + BN - 1) / BN : 0;
}
// What a piece is worth on the line, in tiles: the queries, the four warps' results and the parts take as long as two or
// (more than 8 rows) three tiles.  By its tiles alone a share of many short pieces took far longer than one of few long ones:
// 64 requests of 130 to 1,900 tokens, 32 / 8 heads of 128, 63 us where pieces by themselves take 52 and shares by this measure 50;
// 128 / 8 heads 163, 93 and 89.
template <int NT> __device__ __forceinline__ int worth(const Span& s) { return s.piece / BN + (NT == 1 ? 2 : 3); }
// On to the next piece of the line; false: it belongs to the next share, or there is none.
template <int NT> __device__ __forceinline__ bool walk_next(const ShareParams& p, Walk& w) {
    w.at += worth<NT>(w.span);
    if (++w.split == w.span.pieces) {
        w.split = 0;
        if (++w.unit == p.units) {
            w.unit = 0;
            do {
                if (++w.b >= p.n_seqs) return false;
                w.span = span_of(p, w.b);
            } while (w.span.n_tokens == 0);
        }
        w.first_split = 0;
    }
    if (w.at >= w.end) return false;
    walk_piece(p, w);
    return true;
}
// The first piece of this CTA's share.  All pieces of a request's first unit, of its second and so on, then the next
// request's, lie on one line, a piece as long as it is worth; a share is every piece that starts in an equal
// part of the line.  false: there is none.
template <int NT> __device__ __forceinline__ bool walk_share(const ShareParams& p, Walk& w, int lane) {
    int total = 0;
    for (int b = lane; b < p.n_seqs; b += 32) {
        const Span s = span_of(p, b);
        if (s.n_tokens > 0) total += s.pieces * worth<NT>(s);
    }
    total = __reduce_add_sync(0xffffffffu, total);
    const int share = (total * p.units + (int)gridDim.x - 1) / (int)gridDim.x;
    const int begin = blockIdx.x * share;
    w.end = begin + share;
    if (begin >= total * p.units) return false;
    int before = 0;                                     // worth (of one unit) of the requests before this block of 32
    for (int b0 = 0; b0 < p.n_seqs; b0 += 32) {
        int t = 0;
        if (b0 + lane < p.n_seqs) {
            const Span s = span_of(p, b0 + lane);
            if (s.n_tokens > 0) t = s.pieces * worth<NT>(s);
        }
        int upto = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned here = __ballot_sync(0xffffffffu, (before + upto) * p.units > begin);
        if (here) {
            const int src = __ffs(here) - 1;            // the first request that reaches beyond the share's start
            w.b = b0 + src;
            w.span = span_of(p, w.b);
            const int request = (before + __shfl_sync(0xffffffffu, upto - t, src)) * p.units;
            const int wide = worth<NT>(w.span), all = w.span.pieces * wide;
            w.unit = (begin - request) / all;
            w.split = (begin - request - w.unit * all) / wide;
            w.at = request + w.unit * all + w.split * wide;
            w.first_split = w.split;
            if (w.at == begin) {
                walk_piece(p, w);
                return true;
            }
            // the piece that the share's start falls into belongs to the share before
            const int u = w.unit;
            const int b = w.b;
            const bool got = walk_next<NT>(p, w);
            if (w.b == b && w.unit == u) w.first_split = w.split;
            return got;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// ---- what the two kernels below have in common.  HD: head size; NT: 8-row blocks of query rows (1: up to 8 rows, 2: up to 16)

// A tile's keys and values on their way: a box per page (or per 64 rows of a larger page) and 64-element column block.  The whole
// producer warp issues it, a lane to a box: the page lookups go side by side.
template <int HD>
__device__ __forceinline__ void issue_tile(const DecodeParams& p, const CUtensorMap& map_k, const CUtensorMap& map_v, unsigned char* kt,
                                           unsigned long long* bar, const int* table, int kvh, int k0, int k_hi, int lane) {
    constexpr int HALVES = HD / 64;                     // 64-element (128-byte) column blocks of a row
    constexpr unsigned HALF_BYTES = BN * 128, KV_BYTES = HALVES * HALF_BYTES;
    if (lane == 0) mbar_expect_tx(bar, 2 * KV_BYTES);
    __syncwarp();
    for (int c = lane; c < BN / p.box_rows; c += 32) {
        const int kpos = k0 + c * p.box_rows;
        // boxes past the last key start outside the tensor: the copy writes the zero fill, so
        // that what is multiplied by probability 0 there is finite
        int row = p.total_rows;
        if (kpos < k_hi) {
            const int page = table[kpos >> p.page_shift];
            if (tl_check_page(page))                           // (debug builds: a bad page reads as the zero fill)
                row = (page * p.n_kv_heads + kvh) * p.page_size + (kpos & (p.page_size - 1));
        }
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
            unsigned char* dst = kt + h * HALF_BYTES + c * p.box_rows * 128;
            if (p.streamed) {
                tma_load_2d_streamed(dst, &map_k, bar, h * 64, row);
                tma_load_2d_streamed(dst + KV_BYTES, &map_v, bar, h * 64, row);
            } else {
                tma_load_2d(dst, &map_k, bar, h * 64, row);
                tma_load_2d(dst + KV_BYTES, &map_v, bar, h * 64, row);
            }
        }
    }
    __syncwarp();
}

// The consumers' queries into shared memory, [8 NT][HD + 8] (zero rows where there are none).
template <int HD, int NT>
__device__ __forceinline__ void fetch_queries(const DecodeParams& p, __nv_bfloat16* Qs, int first, int head0, int ng, int n_rows) {
    for (int c = threadIdx.x; c < 8 * NT * (HD / 8); c += NCW * 32) {
        const int rr = c / (HD / 8), part = c - rr * (HD / 8);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (rr < n_rows)
            v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(first + rr / ng) * p.n_heads + head0 + rr % ng) * HD + part * 8);
        *reinterpret_cast<uint4*>(Qs + rr * (HD + 8) + part * 8) = v;
    }
}

// What a consumer thread keeps of a piece.  Its two query rows of every 8-row block are 2t and 2t + 1: of the scores^T
// tile it holds keys g and g + 8 for them, of the out^T tile value columns g and g + 8.
template <int HD, int NT>
struct Consumer {
    static constexpr int KSTEPS = HD / 16;
    static constexpr unsigned HALF_BYTES = BN * 128, KV_BYTES = HD / 64 * HALF_BYTES;
    static constexpr int OPITCH = HD + 4;               // of the results in shared memory: rows two apart fall on different banks
    unsigned qf[NT][KSTEPS][2];                         // Q^T as the 8-wide operand: columns 2t, 2t + 1 (and + 8) of row g
    float m[NT][2], l[NT][2], o[NT][KSTEPS][4];
    int qpos[NT][2], warp_qmax, warp_qmin;
    int g, t, key_off;
    unsigned k_lane_off, v_lane_off;

    __device__ __forceinline__ void place(int warp, int lane) {
        const int mi = lane >> 3;
        g = lane >> 2;
        t = lane & 3;
        key_off = warp * 16;
        // this lane's row and first chunk inside a tile: K as the 16-row operand [keys x 16 columns],
        // V through a transposing load as [16 columns x keys]
        const int k_row = key_off + (lane & 7) + ((mi & 1) ? 8 : 0);
        const int v_row = key_off + (lane & 7) + ((mi & 2) ? 8 : 0);
        k_lane_off = swz(k_row, (mi & 2) ? 1 : 0);
        v_lane_off = swz(v_row, mi & 1);
    }
    __device__ __forceinline__ void take_queries(const __nv_bfloat16* Qs, int lane) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int kd2 = 0; kd2 < KSTEPS / 2; ++kd2) {
                unsigned r[4];
                ldmatrix_x4(r, smem_u32(Qs + (nt * 8 + (lane & 7)) * (HD + 8) + (kd2 * 4 + (lane >> 3)) * 8));
                qf[nt][2 * kd2][0] = r[0]; qf[nt][2 * kd2][1] = r[1];
                qf[nt][2 * kd2 + 1][0] = r[2]; qf[nt][2 * kd2 + 1][1] = r[3];
            }
    }
    __device__ __forceinline__ void begin(int base, int ng, int n_rows) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            m[nt][0] = m[nt][1] = -INFINITY;
            l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
            for (int i = 0; i < KSTEPS; ++i) o[nt][i][0] = o[nt][i][1] = o[nt][i][2] = o[nt][i][3] = 0.f;
        }
        int qmax = -1, qmin = INT_MAX;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int rr = nt * 8 + 2 * t + j;
                const int qp = rr < n_rows ? base + rr / ng : -1;
                qpos[nt][j] = qp;
                qmax = max(qmax, qp);
                if (qp >= 0) qmin = min(qmin, qp);
            }
        warp_qmax = __reduce_max_sync(0xffffffffu, qmax);
        warp_qmin = __reduce_min_sync(0xffffffffu, qmin);
    }
    // the warp's 16 keys of the tile at kt, which begins with key k0; keys lo .. hi - 1 are the piece's
    __device__ __forceinline__ void tile(const DecodeParams& p, unsigned kt, int k0, int lo, int hi) {
        const int share_lo = k0 + key_off;
        if (share_lo > warp_qmax || share_lo + 16 <= lo) return;
        // rows are 128 bytes and tiles 1024-byte aligned, so bits 4-6 of a row's address are the
        // swizzled chunk: xor-ing a constant chunk number in is all it takes to move along a row
        const unsigned ka = kt + k_lane_off, va = kt + KV_BYTES + v_lane_off;
        float sc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
        for (int kd = 0; kd < KSTEPS; ++kd) {
            unsigned kf[4];
            ldmatrix_x4(kf, (ka ^ (unsigned)(((kd * 2) & 7) << 4)) + (kd / 4) * HALF_BYTES);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma_bf16(sc[nt], kf, qf[nt][kd][0], qf[nt][kd][1]);
        }
        const bool all_visible = share_lo >= lo && share_lo + 16 <= hi && share_lo + 15 <= warp_qmin &&
                                 (p.window <= 0 || share_lo > warp_qmax - p.window);
        if (!all_visible) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int qp = qpos[nt][e & 1];
                    const int kpos = share_lo + g + 8 * (e >> 1);
                    const bool vis = kpos >= lo && kpos < hi && kpos <= qp && (p.window <= 0 || kpos > qp - p.window);
                    if (!vis) sc[nt][e] = -INFINITY;
                }
        }
        unsigned ph[NT][2], pl[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float m_safe[2], alpha[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float mx = fmaxf(sc[nt][j], sc[nt][j + 2]);            // over the 16 keys: the lanes that share t
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float m_new = fmaxf(m[nt][j], mx * p.scale_log2);   // maxima live on the base-2 scale
                m_safe[j] = (m_new == -INFINITY) ? 0.f : m_new;           // no key seen yet: keep exponents finite
                alpha[j] = ex2(m[nt][j] - m_safe[j]);
                m[nt][j] = m_new;
                l[nt][j] *= alpha[j];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float pv = ex2(fmaf(sc[nt][e], p.scale_log2, -m_safe[e & 1]));
                sc[nt][e] = pv;
                l[nt][e & 1] += pv;
            }
            if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
                for (int d = 0; d < KSTEPS; ++d) {
                    o[nt][d][0] *= alpha[0]; o[nt][d][1] *= alpha[1];
                    o[nt][d][2] *= alpha[0]; o[nt][d][3] *= alpha[1];
                }
            }
            // probabilities as value + remainder in bfloat16 (the product keeps 16 bits of them),
            // moved from result layout [key g][rows 2t, 2t+1] to operand layout [keys 2t, 2t+1][row g]
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float a = sc[nt][2 * h], c = sc[nt][2 * h + 1];
                const __nv_bfloat162 hi2 = __floats2bfloat162_rn(a, c);
                const float2 back = __bfloat1622float2(hi2);
                ph[nt][h] = movmatrix_trans(*reinterpret_cast<const unsigned*>(&hi2));
                pl[nt][h] = movmatrix_trans(pack_bf16(a - back.x, c - back.y));
            }
        }
#pragma unroll
        for (int dp = 0; dp < KSTEPS; ++dp) {
            unsigned vf[4];
            ldmatrix_x4_trans(vf, (va ^ (unsigned)(((dp * 2) & 7) << 4)) + (dp / 4) * HALF_BYTES);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                mma_bf16(o[nt][dp], vf, ph[nt][0], ph[nt][1]);
                mma_bf16(o[nt][dp], vf, pl[nt][0], pl[nt][1]);
            }
        }
    }
    __device__ __forceinline__ void end() {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                l[nt][j] += __shfl_xor_sync(0xffffffffu, l[nt][j], 4);
                l[nt][j] += __shfl_xor_sync(0xffffffffu, l[nt][j], 8);
                l[nt][j] += __shfl_xor_sync(0xffffffffu, l[nt][j], 16);
            }
    }
    // the warp's results: Om [NCW][om_rows][OPITCH], Mm and Lm [NCW][8 NT]
    __device__ __forceinline__ void leave(float* Om, float* Mm, float* Lm, int warp, int om_rows, int n_rows) const {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int rr = nt * 8 + 2 * t + j;
                if (rr < n_rows) {
#pragma unroll
                    for (int dp = 0; dp < KSTEPS; ++dp) {
                        Om[(warp * om_rows + rr) * OPITCH + dp * 16 + g] = o[nt][dp][j];
                        Om[(warp * om_rows + rr) * OPITCH + dp * 16 + g + 8] = o[nt][dp][j + 2];
                    }
                    if (g == 0) {
                        Mm[warp * 8 * NT + rr] = m[nt][j];
                        Lm[warp * 8 * NT + rr] = l[nt][j];
                    }
                }
            }
    }
    // the four warps' results of row rr, columns d .. d + 3, added up: sums, and the maximum (base-2 scale) and sum of the weights
    static __device__ __forceinline__ float4 add_up(const float* Om, const float* Mm, const float* Lm, int om_rows, int rr, int d, float& M, float& den) {
        M = -INFINITY;
#pragma unroll
        for (int v = 0; v < NCW; ++v) M = fmaxf(M, Mm[v * 8 * NT + rr]);
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        den = 0.f;
#pragma unroll
        for (int v = 0; v < NCW; ++v) {
            const float mv = Mm[v * 8 * NT + rr], lv = Lm[v * 8 * NT + rr];
            if (mv == -INFINITY) continue;
            const float f = exp2f(mv - M);
            const float4 o4 = *reinterpret_cast<const float4*>(Om + (v * om_rows + rr) * OPITCH + d);
            num.x = fmaf(f, o4.x, num.x); num.y = fmaf(f, o4.y, num.y);
            num.z = fmaf(f, o4.z, num.z); num.w = fmaf(f, o4.w, num.w);
            den = fmaf(f, lv, den);
        }
        return num;
    }
};
__device__ __forceinline__ void store_row(__nv_bfloat16* out, float4 num, float den) {
    const float inv = den > 0.f ? 1.f / den : 0.f;
    uint2 w2;
    w2.x = pack_bf16(num.x * inv, num.y * inv);
    w2.y = pack_bf16(num.z * inv, num.w * inv);
    *reinterpret_cast<uint2*>(out) = w2;
}
__device__ __forceinline__ float natural(float M) { return M == -INFINITY ? -INFINITY : M * LN2; }     // a maximum on the natural-log scale

template <int STAGES>
__device__ __forceinline__ void set_up_barriers(unsigned long long* full_bar, unsigned long long* empty_bar) {
    for (int s = 0; s < STAGES; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], NCW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// The first in the CTA whose wait runs out reports (one that only stopped with another's has nothing to say).
__device__ __forceinline__ void report(int* failed_flag, int* status, int code) {
    if (atomicExch(failed_flag, 1) == 0) atomicExch(status, code);
}
// The wait of a whole warp: false for all lanes if it ran out for any.
__device__ __forceinline__ bool warp_wait(unsigned long long* bar, unsigned parity, int* failed_flag, int* status, int code, int lane,
                                          unsigned long long limit_ns) {
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, failed_flag, limit_ns))) return true;
    if (lane == 0) report(failed_flag, status, code);
    return false;
}

// ---- a CTA to a piece (blockIdx: request z, unit y, piece x); merge_partials_kernel follows where there are several.
// The CTA's one barrier stands right behind the set-up, so that the queries are fetched while the producer looks the first pages
// up (behind the first tiles and the queries: 4 requests of 2,000 tokens and 4 new ones each, 32 / 8 heads of 128, 19.5 us, this
// order 18.4; one request of 333 5.3 and 5.0).  It is a kernel of its own because the loops of the shares cost it: 24 requests of 130 to 1,900,
// heads of 64, 14.8 us in one body with them, 14.3 here; 4 of 5,000 to 7,900, 24 / 8 heads of 128, 20.9 and 20.6.
template <int HD, int STAGES, int NT>
__global__ void __launch_bounds__(NTHREADS, NT == 1 ? 3 : 2) attention_decode_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                                  const __grid_constant__ CUtensorMap map_v,
                                                                                  const DecodeParams p) {
    using C = Consumer<HD, NT>;
    constexpr unsigned STAGE_BYTES = 2 * C::KV_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(tiles + STAGES * STAGE_BYTES);
    // (the four warps' results lie where the tiles were)
    float* Om = reinterpret_cast<float*>(tiles);
    float* Mm = Om + NCW * 8 * NT * C::OPITCH;
    float* Lm = Mm + NCW * 8 * NT;
    __shared__ __align__(8) unsigned long long full_bar[STAGES];
    __shared__ __align__(8) unsigned long long empty_bar[STAGES];
    __shared__ int failed_flag, gave_up;

    grid_launch_dependents();
    // What follows, down to the dependency wait, reads nothing that the kernels just before this one
    // write: the step's index data were uploaded before its first kernel, and keys and values of
    // positions before the step's own tokens were written by earlier steps.  Under programmatic
    // dependent launch this part runs while the predecessor is still at work.
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.z, split = blockIdx.x;
    const Span span = span_of(p, b);
    if (span.n_tokens == 0) return;
    const int kvh = blockIdx.y / p.n_gchunks;
    const int g0 = (blockIdx.y - kvh * p.n_gchunks) * p.ng;
    const int ng = min(p.ng, p.group - g0);
    const int k_lo = span.lo + split * span.piece, k_hi = min(span.hi, k_lo + span.piece);
    const int k_start = k_lo & ~(p.box_rows - 1);      // copies start on a box (page) boundary; keys below k_lo are masked
    const int n_tiles = k_hi > k_start ? (k_hi - k_start + BN - 1) / BN : 0;
    if (tid == NCW * 32) {
        failed_flag = 0;
        set_up_barriers<STAGES>(full_bar, empty_bar);
    }
    __syncthreads();

    if (warp == NCW) {
        const int* table = p.block_table + (size_t)b * p.table_stride;
        auto issue = [&](int it) {
            issue_tile<HD>(p, map_k, map_v, tiles + (it % STAGES) * STAGE_BYTES, &full_bar[it % STAGES], table, kvh, k_start + it * BN, k_hi, lane);
        };
        // tiles that end before the step's first new position can go now; a tile that may hold a key
        // written by the predecessor (only the last tile of the last piece can) waits for it
        int it = 0;
        for (; it < STAGES && it < n_tiles && k_start + (it + 1) * BN <= span.base; ++it) issue(it);
        grid_dependency_wait();
        for (; it < STAGES && it < n_tiles; ++it) issue(it);
        for (; it < n_tiles; ++it) {
            if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[it % STAGES], ((it / STAGES) - 1) & 1, &failed_flag))) {
                if (lane == 0) report(&failed_flag, p.status, ERR_PRODUCER_WAIT);
                break;
            }
            issue(it);
        }
        // (nothing that is still on its way may land in shared memory that is no longer this CTA's)
        int never = 0;
        for (int k = max(0, it - STAGES); k < it; ++k) mbar_wait(&full_bar[k % STAGES], (k / STAGES) & 1, &never);
        return;
    }

    // ---- consumers: the same rows, 16 keys of every tile each
    grid_dependency_wait();
    const int n_rows = span.n_tokens * ng, head0 = kvh * p.group + g0;
    fetch_queries<HD, NT>(p, Qs, span.first, head0, ng, n_rows);
    consumers_sync();
    C c;
    c.place(warp, lane);
    c.begin(span.base, ng, n_rows);
    c.take_queries(Qs, lane);
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
        const int s = it % STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], (it / STAGES) & 1, &failed_flag));
        if (!ok) break;
        c.tile(p, smem_u32(tiles + s * STAGE_BYTES), k_start + it * BN, k_lo, k_hi);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);     // this warp is done with the stage
    }
    if (!ok && lane == 0) report(&failed_flag, p.status, ERR_CONSUMER_WAIT);
    c.end();
    // ---- the four warps' results, through shared memory (the stages are done with; one thread reads for all whether
    // the CTA gave up, so that all take the same way; rows that are nobody's hold zeros)
    consumers_sync();
    c.leave(Om, Mm, Lm, warp, 8 * NT, 8 * NT);
    if (tid == 0) gave_up = *(volatile int*)&failed_flag;
    consumers_sync();
    if (gave_up) return;
    for (int idx = tid; idx < n_rows * (HD / 4); idx += NCW * 32) {      // four columns of a row per turn
        const int rr = idx / (HD / 4), d = (idx - rr * (HD / 4)) * 4;
        float M, den;
        const float4 num = C::add_up(Om, Mm, Lm, 8 * NT, rr, d, M, den);
        const size_t row = (size_t)(span.first + rr / ng) * p.n_heads + head0 + rr % ng;
        if (p.n_splits == 1) {
            store_row(p.out + row * HD + d, num, den);
        } else {
            *reinterpret_cast<float4*>(p.part_o + (row * p.n_splits + split) * HD + d) = num;
            if (d == 0) {
                p.part_ml[(row * p.n_splits + split) * 2] = natural(M);
                p.part_ml[(row * p.n_splits + split) * 2 + 1] = den;
            }
        }
    }
}

// ---- shares: a CTA takes the pieces of its share one after the other, and the last one adds a request's up.
// SELFTEST: every third CTA never hands back its first stage, so that its producer's wait for room runs out
template <int HD, int STAGES, int NT, bool SELFTEST = false>
__global__ void __launch_bounds__(NTHREADS, NT == 1 ? 3 : 2) attention_decode_shares_kernel(const __grid_constant__ CUtensorMap map_k,
                                                                                         const __grid_constant__ CUtensorMap map_v,
                                                                                         const ShareParams p) {
    using C = Consumer<HD, NT>;
    constexpr unsigned STAGE_BYTES = 2 * C::KV_BYTES;
    constexpr int NROWS = 8 * NT;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~uintptr_t(1023));
    // behind the stages, in the same place one after the other: the queries [NROWS][HD + 8], the four warps' results
    // [NCW][rows][OPITCH] and the weights of the pieces [rows][MERGE_MAX_SPLITS]
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(tiles + STAGES * STAGE_BYTES);
    float* Om = reinterpret_cast<float*>(tiles + STAGES * STAGE_BYTES);
    __shared__ float Mm[NCW * NROWS], Lm[NCW * NROWS];
    __shared__ __align__(8) unsigned long long full_bar[STAGES];
    __shared__ __align__(8) unsigned long long empty_bar[STAGES];
    __shared__ int failed_flag;
    __shared__ int arrived, gave_up;

    grid_launch_dependents();
    // (down to the dependency wait nothing is read that the kernels just before this one write: see above)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long limit_ns = SELFTEST ? p.limit_ns : WAIT_NS;
    Walk w;
    if (!walk_share<NT>(p, w, lane)) return;            // (the same for all warps)
    if (tid == NCW * 32) {
        failed_flag = 0;
        set_up_barriers<STAGES>(full_bar, empty_bar);
    }
    __syncthreads();

    if (warp == NCW) {
        bool waited = false;
        int it = 0;
        bool ok = true;
        do {
            const int kvh = w.unit / p.n_gchunks;
            const int* table = p.block_table + (size_t)w.b * p.table_stride;
            for (int i = 0; i < w.tiles && ok; ++i, ++it) {
                const int s = it % STAGES;
                const int k0 = w.start + i * BN;
                // tiles go at once, up to one that may hold a key written by the predecessor
                if (!waited && k0 + BN > w.span.base) {
                    grid_dependency_wait();
                    waited = true;
                }
                if (it >= STAGES && !warp_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, &failed_flag, p.status, ERR_PRODUCER_WAIT, lane, limit_ns)) {
                    ok = false;
                    break;
                }
                issue_tile<HD>(p, map_k, map_v, tiles + s * STAGE_BYTES, &full_bar[s], table, kvh, k0, w.hi, lane);
            }
        } while (ok && walk_next<NT>(p, w));
        if (!waited) grid_dependency_wait();
        // (nothing that is still on its way may land in shared memory that is no longer this CTA's)
        int never = 0;
        for (int k = max(0, it - STAGES); k < it; ++k) mbar_wait(&full_bar[k % STAGES], (k / STAGES) & 1, &never, limit_ns);
        return;
    }

    // ---- consumers: the same rows, 16 keys of every tile each
    grid_dependency_wait();
    C c;
    c.place(warp, lane);
    bool ok = true, fresh = true;
    int it = 0;
    do {
        const int kvh = w.unit / p.n_gchunks;
        const int g0 = (w.unit - kvh * p.n_gchunks) * p.ng;
        const int ng = min(p.ng, p.group - g0);
        const int n_rows = w.span.n_tokens * ng, head0 = kvh * p.group + g0;
        // the next pieces of a request find the queries in registers
        if (fresh) {
            fetch_queries<HD, NT>(p, Qs, w.span.first, head0, ng, n_rows);
            consumers_sync();
            c.take_queries(Qs, lane);
        }
        c.begin(w.span.base, ng, n_rows);
        for (int i = 0; i < w.tiles; ++i, ++it) {
            const int s = it % STAGES;
            if (!ok || !warp_wait(&full_bar[s], (it / STAGES) & 1, &failed_flag, p.status, ERR_CONSUMER_WAIT, lane, limit_ns)) {
                ok = false;
                break;
            }
            c.tile(p, smem_u32(tiles + s * STAGE_BYTES), w.start + i * BN, w.lo, w.hi);
            __syncwarp();
            if (lane == 0 && !(SELFTEST && it == 0 && blockIdx.x % 3 == 1)) mbar_arrive(&empty_bar[s]);     // this warp is done with the stage
        }
        c.end();

        // ---- the four warps' results, through shared memory (all have read the queries and the tiles)
        consumers_sync();
        c.leave(Om, Mm, Lm, warp, p.rows, n_rows);
        // (the producer may give up at any moment: one thread reads the flag for all, so that all take the same way
        // through the barriers below; what this piece is made of has arrived by now, or a consumer has set the flag)
        if (tid == 0) gave_up = *(volatile int*)&failed_flag;
        consumers_sync();
        const bool sound = gave_up == 0;
        const int parts = w.span.pieces;
        if (sound) {
            for (int idx = tid; idx < n_rows * (HD / 4); idx += NCW * 32) {      // four columns of a row per turn
                const int rr = idx / (HD / 4), d = (idx - rr * (HD / 4)) * 4;
                float M, den;
                const float4 num = C::add_up(Om, Mm, Lm, p.rows, rr, d, M, den);
                if (parts == 1) {
                    store_row(p.out + ((size_t)(w.span.first + rr / ng) * p.n_heads + head0 + rr % ng) * HD + d, num, den);
                } else {
                    const size_t place = (((size_t)w.b * p.units + w.unit) * p.n_splits + w.split) * p.rows + rr;
                    __stcg(reinterpret_cast<float4*>(p.part_o + place * HD + d), num);
                    if (d == 0) __stcg(reinterpret_cast<float2*>(p.part_ml + place * 2), make_float2(natural(M), den));
                }
            }
        }
        // ---- whoever is last with a request's pieces adds them up (in order, as merge_partials_kernel does)
        if (parts > 1 && (w.split + 1 == parts || w.at + worth<NT>(w.span) >= w.end)) {
            consumers_sync();
            const int mine = w.split + 1 - w.first_split;
            int seen = mine;
            if (mine < parts) {
                int* counter = p.counters + (size_t)w.b * p.units + w.unit;
                if (tid == 0) {
                    // (release what the barrier has gathered of all threads' stores, acquire what the others released)
                    const int add = sound ? mine : mine + FAILED_PART;
                    int before;
                    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;" : "=r"(before) : "l"(counter), "r"(add) : "memory");
                    arrived = before + add;
                    const int pieces = arrived & (FAILED_PART - 1);
                    if (pieces >= parts) *counter = 0;
                    if (pieces > parts) atomicExch(p.status, ERR_COUNT);      // (another call counts in the same place)
                }
                consumers_sync();
                seen = arrived;
            } else if (!sound) {
                seen = FAILED_PART;
            }
            if (seen == parts) {
                float* weight = Om;                                          // [rows][MERGE_MAX_SPLITS]
                const size_t place0 = ((size_t)w.b * p.units + w.unit) * p.n_splits * p.rows;
                for (int rr = warp; rr < n_rows; rr += NCW) {
                    float2 ml[MERGE_MAX_SPLITS / 32];
                    float M = -INFINITY, den = 0.f;
#pragma unroll
                    for (int i = 0; i < MERGE_MAX_SPLITS / 32; ++i) {
                        const int c1 = i * 32 + lane;
                        ml[i] = make_float2(-INFINITY, 0.f);
                        if (c1 < parts) ml[i] = __ldcg(reinterpret_cast<const float2*>(p.part_ml + (place0 + (size_t)c1 * p.rows + rr) * 2));
                        M = fmaxf(M, ml[i].x);
                    }
                    M = warp_max(M);
#pragma unroll
                    for (int i = 0; i < MERGE_MAX_SPLITS / 32; ++i) {
                        const int c1 = i * 32 + lane;
                        const float f = ml[i].x == -INFINITY ? 0.f : __expf(ml[i].x - M);
                        if (c1 < parts) weight[rr * MERGE_MAX_SPLITS + c1] = f;
                        den = fmaf(f, ml[i].y, den);
                    }
                    den = warp_sum(den);
                    if (lane == 0) Lm[rr] = den;
                }
                consumers_sync();
                for (int idx = tid; idx < n_rows * (HD / 4); idx += NCW * 32) {
                    const int rr = idx / (HD / 4), d = (idx - rr * (HD / 4)) * 4;
                    float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
                    for (int c1 = 0; c1 < parts; ++c1) {
                        const float f = weight[rr * MERGE_MAX_SPLITS + c1];
                        const float4 o4 = __ldcg(reinterpret_cast<const float4*>(p.part_o + (place0 + (size_t)c1 * p.rows + rr) * HD + d));
                        num.x = fmaf(f, o4.x, num.x); num.y = fmaf(f, o4.y, num.y);
                        num.z = fmaf(f, o4.z, num.z); num.w = fmaf(f, o4.w, num.w);
                    }
                    store_row(p.out + ((size_t)(w.span.first + rr / ng) * p.n_heads + head0 + rr % ng) * HD + d, num, Lm[rr]);
                }
            }
        }
        fresh = w.split + 1 == parts;
        consumers_sync();            // the place behind the stages is the next piece's
    } while (walk_next<NT>(p, w));
}

// out[row, d] = sum_i e^{m_i - M} o_i[d] / sum_i e^{m_i - M} l_i,  M = max_i m_i: the weights are
// computed once per row (lanes over splits), then every thread sums its lanes over the splits in order
__global__ void merge_partials_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                      __nv_bfloat16* __restrict__ out, int n_splits, int head_dim) {
    __shared__ float wgt[MERGE_MAX_SPLITS];
    __shared__ float red;
    grid_launch_dependents();
    grid_dependency_wait();
    const size_t row = blockIdx.x;
    const float* ml = part_ml + row * n_splits * 2;
    if (threadIdx.x < 32) {
        float M = -INFINITY;
        for (int i = threadIdx.x; i < n_splits; i += 32) M = fmaxf(M, ml[2 * i]);
        M = warp_max(M);
        float den = 0.f;
        for (int i = threadIdx.x; i < n_splits; i += 32) {
            const float mi = ml[2 * i];
            const float w = (mi == -INFINITY) ? 0.f : __expf(mi - M);
            wgt[i] = w;
            den = fmaf(w, ml[2 * i + 1], den);
        }
        den = warp_sum(den);
        if (threadIdx.x == 0) red = den;
    }
    __syncthreads();
    const float inv = red > 0.f ? 1.f / red : 0.f;
    for (int d = threadIdx.x; d < head_dim; d += blockDim.x) {
        float num = 0.f;
        for (int i = 0; i < n_splits; ++i) num = fmaf(wgt[i], part_o[(row * n_splits + i) * head_dim + d], num);
        out[row * head_dim + d] = __float2bfloat16_rn(num * inv);
    }
}

// ---- host side ---------------------------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// the page tensor as rows of head_dim elements; box = box_rows x 64 elements, 128-byte swizzle.
// Maps are kept per (pointer, rows, head_dim, box): the page tensors live as long as the engine.
int page_map(CUtensorMap* out, const void* base, long long rows, int head_dim, int box_rows) {
    static std::map<std::tuple<const void*, long long, int, int>, CUtensorMap> cache;
    static std::mutex lock;
    std::lock_guard<std::mutex> guard(lock);
    auto key = std::make_tuple(base, rows, head_dim, box_rows);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return TL_OK;
    }
    EncodeTiledFn fn = encode_tiled();
    if (fn == nullptr) return TL_BAD_SIZE;
    cuuint64_t dims[2] = {(cuuint64_t)head_dim, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)head_dim * 2};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUtensorMap m;
    CUresult rc = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return TL_BAD_SIZE;
    if (cache.size() > 4096) cache.clear();
    cache[key] = m;
    *out = m;
    return TL_OK;
}

template <int HD> constexpr int stages_for() { return HD == 128 ? 2 : 3; }
template <int HD> constexpr size_t smem_for() {
    return (size_t)stages_for<HD>() * 2 * (HD / 64) * BN * 128 + 16 * (HD + 8) * 2 + 1024;
}

// with shares: the warps' results lie behind the stages (`rows`: rows of a tile in use)
template <int HD> constexpr size_t smem_shares(int rows) {
    const size_t queries = (size_t)(rows <= 8 ? 8 : 16) * (HD + 8) * 2, results = (size_t)NCW * rows * (HD + 4) * 4;
    return (size_t)stages_for<HD>() * 2 * (HD / 64) * BN * 128 + (queries > results ? queries : results) + 1024;
}
static_assert(NCW * (64 + 4) >= MERGE_MAX_SPLITS, "the pieces' weights lie where the warps' results were");

template <int HD, int NT> int shares_per_sm(int rows) {
    static int known[17] = {};                     // (threads that come here at the same time write the same)
    if (known[rows] == 0) {
        auto kern = attention_decode_shares_kernel<HD, stages_for<HD>(), NT>;
        int n = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_shares<HD>(8 * NT)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, NTHREADS, smem_shares<HD>(rows)) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = 1;
        }
        known[rows] = n;
    }
    return known[rows];
}

struct Plan {
    int ng, n_gchunks, tpw, n_q_tiles, n_splits;
    int shares;        // CTAs that take shares of the pieces; 0: a CTA to a piece
};

bool takes(int n_heads, int n_kv_heads, int head_dim, int page_size, int max_q_len) {
    if (head_dim != 64 && head_dim != 128) return false;
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return false;
    if (page_size < 1 || (page_size & (page_size - 1)) != 0) return false;           // a power of two
    const int group = n_heads / n_kv_heads;
    const int ng = group < 16 ? group : 16;
    return max_q_len >= 1 && max_q_len <= 16 / ng;
}

// with a CTA to a piece
int ctas_per_sm(int head_dim) {
    const int fit = (int)((size_t)224 * 1024 / ((head_dim == 128 ? smem_for<128>() : smem_for<64>()) + 1024));
    return fit > 6 ? 6 : fit;
}

Plan make_plan(int n_seqs, int n_heads, int n_kv_heads, int head_dim, int max_q_len, int max_kv_len, int allow_split) {
    Plan pl;
    const int group = n_heads / n_kv_heads;
    pl.ng = group < 16 ? group : 16;
    pl.n_gchunks = (group + pl.ng - 1) / pl.ng;
    pl.tpw = 16 / pl.ng;
    pl.n_q_tiles = (max_q_len + pl.tpw - 1) / pl.tpw;
    pl.n_splits = 1;
    if (allow_split > 1) {                       // a given number of splits (tests and measurements)
        pl.n_splits = allow_split < MERGE_MAX_SPLITS ? allow_split : MERGE_MAX_SPLITS;
    } else if (allow_split && max_kv_len >= 2 * MIN_SPLIT) {
        // CTAs run in waves; with s splits a CTA does 1/s of the keys.  Pick the s that makes
        // (waves / s), the time in units of one unsplit CTA, smallest.  While everything fits one
        // wave, more splits cost next to nothing (a CTA walks its tiles one after the other, so few
        // CTAs with long walks leave most of the memory system idle: one request of 8,192 keys
        // takes 21.8 us in 8 splits and 11.2 us in 32); beyond one wave each split is charged
        // for its partial results and the merge.
        const long long slots = 148LL * ctas_per_sm(head_dim);
        const long long base = (long long)pl.n_q_tiles * n_kv_heads * pl.n_gchunks * n_seqs;
        int most = max_kv_len / MIN_SPLIT;
        if (most > MERGE_MAX_SPLITS) most = MERGE_MAX_SPLITS;
        double best = 1e30;
        for (int sp = 1; sp <= most; ++sp) {
            const long long waves = (base * sp + slots - 1) / slots;
            const double cost = (double)waves / sp + (waves == 1 ? 0.0005 : 0.01) * sp;
            if (cost < best - 1e-9) {
                best = cost;
                pl.n_splits = sp;
            }
        }
    }
    // Shares pay where a share is made of many pieces, most of them short (planned for the longest context there could be):
    // then the launch of a CTA to a piece costs more than the pieces.  With few pieces to a share they come out uneven.
    // Shares to pieces by themselves, contexts all of 320 / of 40 to 600 / of 130 to 1,900 / all of 2,048 tokens, us:
    //   32 / 8 heads of 128, 40 requests, 2.9 pieces a share:  17.2  17.6  38.0  56.2  to  17.1  18.0  32.6  55.1
    //                        28           3.5                  14.4  14.4  29.3  41.9      17.1  18.3  28.2  43.3
    //                        64           6.9                  22.8  22.5  49.7  84.2      28.6  30.0  51.8  86.5
    //                  64,   96           5.2                  21.1  22.1  44.7  74.5      21.4  23.0  40.9  69.2
    //                        64           9.2                  18.8  19.3  33.2  49.3      25.1  25.7  37.0  53.4
    //   128 / 8 heads of 128 (more than 8 rows: more work to a tile), and of 64:
    //                  64,   48           3.9                  23.3  26.0  41.7  55.5      25.2  27.2  40.4  54.9
    //                  128,  40           4.3                  32.7  35.0  54.7  82.7      34.0  35.4  54.4  80.4
    //                        28           5.3                  26.9  34.4  49.4  66.8      33.4  35.1  48.1  64.1
    //                        64           10.4                 53.1  53.4  89.3  125.6     63.4  65.3  92.8  127.5
    // With heads of 128 and 5 to 8 rows the warps' results, which shares keep beside the stages, leave room for two CTAs an SM
    // instead of three (64 requests, 64 / 8 heads, all of 320, of 40 to 600, all of 2,048: 34.0  37.9  100.1 to 33.9  35.3  90.7): they stay pieces.
    pl.shares = 0;
    const long long pieces = (long long)n_kv_heads * pl.n_gchunks * n_seqs * pl.n_splits;
    if (allow_split == 1 && pl.n_splits > 1 && pieces > 148LL * ctas_per_sm(head_dim)) {
        const int rows = max_q_len * pl.ng;
        const int ctas = 148 * (head_dim == 128 ? (rows <= 8 ? shares_per_sm<128, 1>(rows) : shares_per_sm<128, 2>(rows))
                                                : (rows <= 8 ? shares_per_sm<64, 1>(rows) : shares_per_sm<64, 2>(rows)));
        if (pieces > (long long)(rows <= 8 ? 6 : 4) * ctas && !(head_dim == 128 && rows > 4 && rows <= 8)) pl.shares = ctas;
    }
    return pl;
}

// A self-test of the waits: shares of 148 CTAs (a first stage that is not handed back stops each third of them once it
// has more tiles than stages), heads of 64, up to 8 rows.
int launch_selftest(const CUtensorMap& mk, const CUtensorMap& mv, const ShareParams& p, cudaStream_t s) {
    auto kern = attention_decode_shares_kernel<64, stages_for<64>(), 1, true>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_shares<64>(8));
    if (e != cudaSuccess) return (int)e;
    return (int)tl_launch(kern, dim3(148), dim3(NTHREADS), smem_shares<64>(p.rows), s, mk, mv, p);
}

template <int HD, int NT>
int launch(const CUtensorMap& mk, const CUtensorMap& mv, const ShareParams& p, const Plan& pl, cudaStream_t s) {
    if (pl.shares > 0)          // (shares_per_sm has raised the limit on shared memory)
        return (int)tl_launch(attention_decode_shares_kernel<HD, stages_for<HD>(), NT>, dim3(pl.shares), dim3(NTHREADS), smem_shares<HD>(p.rows), s, mk, mv, p);
    constexpr size_t smem = smem_for<HD>();
    auto kern = attention_decode_kernel<HD, stages_for<HD>(), NT>;
    static bool raised = false;
    if (!raised) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        raised = true;
    }
    return (int)tl_launch(kern, dim3(pl.n_splits, p.units, p.n_seqs), dim3(NTHREADS), smem, s, mk, mv, (const DecodeParams&)p);
}

}  // namespace

// 1 if this kernel takes the step: head_dim 64 or 128, a page size that is a power of two, and
// every request's rows (tokens x heads of a kv group) within one 16-row tile.
extern "C" int tl_attention_decode_supports(int n_heads, int n_kv_heads, int head_dim, int page_size, int max_q_len) {
    return takes(n_heads, n_kv_heads, head_dim, page_size, max_q_len) ? 1 : 0;
}

// Which capture the stream takes part in: 0 where it is in none, else a number that no other capture has.
extern "C" int tl_stream_capture_id(void* stream, unsigned long long* id) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    *id = 0;
    const cudaError_t e = cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, id);
    if (e != cudaSuccess) return (int)e;
    if (status != cudaStreamCaptureStatusActive) *id = 0;
    return TL_OK;
}

// What a call needs beside its operands: n_splits pieces of a request's keys, workspace_floats of scratch, and
// n_counters ints that are zero (and are zero again when the call has run); no call that may run at the same time may have
// either.  With counters there is one launch, else there are two when n_splits is over 1.
extern "C" int tl_attention_decode_plan(int n_tokens, int n_seqs, int n_heads, int n_kv_heads, int head_dim,
                                        int max_q_len, int max_kv_len, int allow_split,
                                        int* n_splits, long long* workspace_floats, long long* n_counters) {
    if (!takes(n_heads, n_kv_heads, head_dim, 16, max_q_len)) return TL_BAD_SIZE;
    const Plan pl = make_plan(n_seqs, n_heads, n_kv_heads, head_dim, max_q_len, max_kv_len, allow_split);
    const long long units = (long long)n_kv_heads * pl.n_gchunks * n_seqs;
    *n_splits = pl.n_splits;
    *workspace_floats = pl.n_splits <= 1 ? 0 : (pl.shares > 0 ? units * max_q_len * pl.ng : (long long)n_tokens * n_heads) * pl.n_splits * (head_dim + 2);
    *n_counters = pl.shares > 0 ? units : 0;
    return TL_OK;
}

// limit_ns: 0, or the limit of the self-test's waits
static int attention_decode(const void* q, const void* k_pages, const void* v_pages, void* out,
                            const int* block_table, int table_stride, const int* q_start,
                            const int* kv_len, float* workspace, int* counters, int* status, int n_tokens, int n_seqs,
                            int n_heads, int n_kv_heads, int head_dim, int page_size, long long n_pages,
                            int max_q_len, int max_kv_len, int window, float scale, int allow_split,
                            unsigned long long limit_ns, void* stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return TL_OK;
    if (!takes(n_heads, n_kv_heads, head_dim, page_size, max_q_len) || max_kv_len <= 0 || n_pages <= 0) return TL_BAD_SIZE;
    if (n_pages * n_kv_heads * page_size >= (1LL << 31)) return TL_BAD_SIZE;
    if (!aligned16(q) || !aligned16(k_pages) || !aligned16(v_pages) || !aligned16(out) || status == nullptr) return TL_BAD_ALIGN;
    const Plan pl = make_plan(n_seqs, n_heads, n_kv_heads, head_dim, max_q_len, max_kv_len, allow_split);
    if (pl.n_splits > 1 && (workspace == nullptr || !aligned16(workspace))) return TL_BAD_SIZE;
    if (pl.shares > 0 && counters == nullptr) return TL_BAD_SIZE;
    if (n_seqs > 65535 || (long long)n_kv_heads * pl.n_gchunks > 65535) return TL_BAD_SIZE;

    ShareParams p;
    p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out;
    p.block_table = block_table; p.q_start = q_start; p.kv_len = kv_len; p.table_stride = table_stride;
    p.status = status; p.counters = counters;
    p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.page_size = page_size;
    p.page_shift = 0;
    while ((1 << p.page_shift) < page_size) ++p.page_shift;
    p.box_rows = page_size < BN ? page_size : BN;
    p.total_rows = (int)(n_pages * n_kv_heads * page_size);
    p.group = n_heads / n_kv_heads; p.ng = pl.ng; p.n_gchunks = pl.n_gchunks; p.units = n_kv_heads * pl.n_gchunks;
    p.n_seqs = n_seqs; p.max_tokens = max_q_len; p.rows = max_q_len * pl.ng;
    p.window = window > 0 ? window : 0;
    {
        // (an upper bound of what the call reads: every request's keys and values up to the longest context)
        const double kv_bytes = 2.0 * n_seqs * (double)max_kv_len * n_kv_heads * head_dim * 2;
        // (measured: with 64 requests of 2,048 tokens a step is 2.5 % shorter with the mark, with 32 requests 1 %,
        // with 8 requests of 2,048 tokens, whose keys and values L2 holds, 1 % longer; no difference elsewhere)
        p.streamed = kv_bytes > 96e6 ? 1 : 0;
    }
    p.n_splits = pl.n_splits;
    p.scale_log2 = scale * LOG2E;
    p.limit_ns = limit_ns;
    p.part_o = workspace;
    p.part_ml = workspace ? workspace + (pl.shares > 0 ? (size_t)n_seqs * p.units * p.rows : (size_t)n_tokens * n_heads) * pl.n_splits * head_dim : nullptr;

    const long long rows = n_pages * n_kv_heads * page_size;
    CUtensorMap mk, mv;
    int rc = page_map(&mk, k_pages, rows, head_dim, p.box_rows);
    if (rc != TL_OK) return rc;
    rc = page_map(&mv, v_pages, rows, head_dim, p.box_rows);
    if (rc != TL_OK) return rc;

    cudaStream_t s = (cudaStream_t)stream;
    if (limit_ns != 0) return pl.shares > 0 && head_dim == 64 && p.rows <= 8 ? launch_selftest(mk, mv, p, s) : TL_BAD_SIZE;
    // query rows a CTA can meet: one 8-row block is enough for them, or two
    if (p.rows <= 8)
        rc = head_dim == 128 ? launch<128, 1>(mk, mv, p, pl, s) : launch<64, 1>(mk, mv, p, pl, s);
    else
        rc = head_dim == 128 ? launch<128, 2>(mk, mv, p, pl, s) : launch<64, 2>(mk, mv, p, pl, s);
    if (rc != TL_OK) return rc;
    if (pl.n_splits > 1 && pl.shares == 0) {
        cudaError_t e = tl_launch(merge_partials_kernel, dim3((unsigned)n_tokens * (unsigned)n_heads),
                                  dim3(head_dim >= 128 ? 128u : 64u), 0, s, (const float*)p.part_o, (const float*)p.part_ml,
                                  p.out, pl.n_splits, head_dim);
        if (e != cudaSuccess) return (int)e;
    }
    return TL_OK;
}

// Same arguments as tl_paged_attention_mma; n_pages is the first extent of the page tensors.
extern "C" int tl_paged_attention_decode(const void* q, const void* k_pages, const void* v_pages, void* out,
                                         const int* block_table, int table_stride, const int* q_start,
                                         const int* kv_len, float* workspace, int* counters, int* status, int n_tokens, int n_seqs,
                                         int n_heads, int n_kv_heads, int head_dim, int page_size, long long n_pages,
                                         int max_q_len, int max_kv_len, int window, float scale, int allow_split,
                                         void* stream) {
    return attention_decode(q, k_pages, v_pages, out, block_table, table_stride, q_start, kv_len, workspace, counters, status, n_tokens,
                            n_seqs, n_heads, n_kv_heads, head_dim, page_size, n_pages, max_q_len, max_kv_len, window, scale, allow_split,
                            0, stream);
}

// The same call as a self-test of the bounded waits (shares, heads of 64, at most 8 rows): a third of the CTAs wait for room that
// nobody makes, give up after limit_ns and set status; the rest of the results are those of the call.
extern "C" int tl_attention_decode_give_up_selftest(const void* q, const void* k_pages, const void* v_pages, void* out,
                                                    const int* block_table, int table_stride, const int* q_start,
                                                    const int* kv_len, float* workspace, int* counters, int* status, int n_tokens, int n_seqs,
                                                    int n_heads, int n_kv_heads, int head_dim, int page_size, long long n_pages,
                                                    int max_q_len, int max_kv_len, int window, float scale, unsigned long long limit_ns,
                                                    void* stream) {
    if (limit_ns == 0) return TL_BAD_SIZE;
    return attention_decode(q, k_pages, v_pages, out, block_table, table_stride, q_start, kv_len, workspace, counters, status, n_tokens,
                            n_seqs, n_heads, n_kv_heads, head_dim, page_size, n_pages, max_q_len, max_kv_len, window, scale, 1, limit_ns, stream);
}
