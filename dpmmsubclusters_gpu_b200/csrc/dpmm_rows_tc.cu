// dpmm_rows_tc.cu -- tensor-core passes over the points in label order (gathered rows): the sub-cluster
// labels (cudaKernel.cu create_subclusters_labels, :1299-1398).
//
// Form.  One persistent CTA per SM walks the chunks (points of one cluster, dpmm_kernels.cu k_segments)
// blockIdx.x, + gridDim.x, .. in tiles of 128 points; its warps take the steps of a tile as roles that hand
// over through bounded mbarriers, so that the gather of one tile, the products of another and the
// draws of a third run at the same time:
//   warps 0-15   loaders, two groups of 8 (tile n goes to group n % 2): the rows of the group's next tile are
//                in flight in registers while the last one is split into BF16 hi + lo and stored as the A operand
//   warps 16-23  two groups of 4: TMEM accumulator -> r -> draw, a thread per point, no exchange
//   warps 24-25  issue the tcgen05.mma, alternate tiles each: while one waits for its operands, the products
//                that the other has queued run
//   warp 26      copies the cluster's B operand and biases per chunk (two buffers)
// Why: the block-synchronous form before (256 threads, two CTAs per SM: gather, split, barrier, products,
// barrier, drain, barrier, draw) left the memory idle while a tile was drained and drawn.
#include <algorithm>

#include "dpmm_tc.cuh"

namespace dpmm {
namespace tc {

constexpr int RW_LOADERS = 16, RW_DRAINS = 8;             // warps, in two groups each
constexpr int RW_MMA = RW_LOADERS + RW_DRAINS, RW_MMAS = 2, RW_COPY = RW_MMA + RW_MMAS;
constexpr int RW_ROWS = BM / (RW_LOADERS / 2);            // rows per loader warp and tile
constexpr int RW_THREADS = 32 * (RW_COPY + 1);
constexpr int RW_ACC = 4;                                 // accumulators in TMEM

// A operand of one tile of 128 gathered rows: K-major, 128-byte swizzle.  DP = 64: an image of hi (a row is 64
// BF16) then one of lo; DP = 32: one image whose rows are [32 hi | 32 lo].  B operands use the same rows.
template <int DP>
struct RowOperand {
    static constexpr uint32_t A = DP == 64 ? A_TILE : A_BYTES;
    // byte offset of features 4 c4 .. 4 c4 + 3 of a row
    __device__ static uint32_t hi(int row, int c4) { return sw128_offset(row, c4 * 4); }
    __device__ static uint32_t lo(int row, int c4) { return DP == 64 ? A_BYTES + sw128_offset(row, c4 * 4) : sw128_offset(row, 32 + c4 * 4); }
};

// D (+)= hi hi + lo hi + hi lo of a tile's A at sa and B at sb (N rows; its lo image, DP = 64, N x 128 B further on)
template <int DP>
__device__ __forceinline__ void issue_split3(uint32_t td, uint32_t sa, uint32_t sb, int n)
{
    const uint32_t idesc = bf16_idesc(n);
    constexpr int KS = DP / 16;
    const uint64_t ah = sw128_desc(sa), bh = sw128_desc(sb);
    const uint64_t al = DP == 64 ? sw128_desc(sa + A_BYTES) : ah + 4;
    const uint64_t bl = DP == 64 ? sw128_desc(sb + (uint32_t)n * 128) : bh + 4;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) umma_bf16_n(td, ah + 2 * ks, bh + 2 * ks, idesc, ks != 0 ? 1u : 0u);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) umma_bf16_n(td, al + 2 * ks, bh + 2 * ks, idesc, 1u);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) umma_bf16_n(td, ah + 2 * ks, bl + 2 * ks, idesc, 1u);
}

__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint2 v)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}

// the tiles of this CTA's chunks in order; the next chunk's entry is loaded one chunk ahead
struct TileCursor {
    const int32_t* chunk;
    int nch, q, k, start, len, t0, nk, nstart, nlen;
    __device__ __forceinline__ void fetch(int at)
    {
        if (at < nch) {
            nk = __ldg(chunk + 3 * at);
            nstart = __ldg(chunk + 3 * at + 1);
            nlen = __ldg(chunk + 3 * at + 2);
        }
    }
    __device__ __forceinline__ TileCursor(const int32_t* c, int n) : chunk(c), nch(n), q(blockIdx.x), t0(0)
    {
        nk = nstart = nlen = 0;
        fetch(q);
        take();
    }
    __device__ __forceinline__ void take()
    {
        k = nk;
        start = nstart;
        len = nlen;
        fetch(q + (int)gridDim.x);
    }
    __device__ __forceinline__ bool valid() const { return q < nch; }
    __device__ __forceinline__ bool last_tile() const { return t0 + BM >= len; }
    __device__ __forceinline__ void advance()
    {
        t0 += BM;
        if (t0 >= len) {
            q += (int)gridDim.x;
            t0 = 0;
            take();
        }
    }
};

// A role's waits: bounded; on expiry (or after another role's) the error word is set and the role stops.  A
// group of warps waits through its first warp: that one polls, the others sleep in a named barrier (a poll
// of every warp took half of the issue slots: 6000 -> 3000 instructions a tile), and the outcome is the
// group's (stat: two words, used in turn, so that the next outcome cannot overtake a reader).
struct GroupWait {
    int32_t* err;
    volatile int* stat;
    int id, threads, warp, turn;
    __device__ __forceinline__ bool operator()(uint64_t* bar, uint32_t parity, int code)
    {
        turn ^= 1;
        if (warp == 0 && (threadIdx.x & 31) == 0) {
            const bool ok = mbar_wait_blocking(bar, parity, err);
            if (!ok) atomicCAS(err, 0, code);
            stat[turn] = ok;
        }
        asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
        return stat[turn] != 0;
    }
};

__device__ __forceinline__ bool thread_wait(uint64_t* bar, uint32_t parity, int32_t* err, int code)
{
    if (mbar_wait_blocking(bar, parity, err)) return true;
    atomicCAS(err, 0, code);
    return false;
}

// Loader group g (8 warps; warp w of the group takes rows RW_ROWS w .. of a tile): tiles g, g + 2, .. of the CTA
// into the A ring.  A warp instruction loads whole rows (LPR lanes of 16 bytes each); the permutation
// entries of a tile sit one per lane, a tile ahead of the rows.
template <int DP, int SLOTS>
__device__ __forceinline__ void load_tiles(const float* __restrict__ x, const int32_t* __restrict__ perm, TileCursor cur,
                                           int g, int w, uint8_t* sA, uint64_t* full, uint64_t* empty, GroupWait wait)
{
    using O = RowOperand<DP>;
    constexpr int LPR = DP / 4, RPI = 32 / LPR, ITEMS = RW_ROWS / RPI;   // lanes per row, rows per instruction
    const int lane = threadIdx.x & 31, c4 = lane % LPR, sub = lane / LPR;
    int pq = 0;
    float4 pf[ITEMS];
    const float4* xc = reinterpret_cast<const float4*>(x) + c4;
    // rows past the chunk repeat its last one: their products stay in accumulator rows that nobody reads, and
    // no load waits on a condition
    auto load_perm = [&]() {
        pq = __ldg(perm + cur.start + min(cur.t0 + RW_ROWS * w + (lane & (RW_ROWS - 1)), cur.len - 1));
        cur.advance();
        if (cur.valid()) cur.advance();
    };
    auto load_rows = [&]() {   // the shuffles before the loads: in turn, each load waited for the one before
        int p[ITEMS];
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) p[u] = __shfl_sync(0xffffffffu, pq, RPI * u + sub);
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) pf[u] = __ldg(xc + (size_t)p[u] * LPR);
    };
    // operand offsets of row RW_ROWS w + RPI u + sub: the swizzle XORs the row (mod 8) into the 16-byte piece, and
    // RPI u and sub share no bit, so items 8 / RPI apart differ by whole atoms and the others by one XOR
    constexpr int PER = 8 / RPI;
    uint32_t off[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) off[u] = O::hi(RW_ROWS * w + RPI * u + sub, c4);
    constexpr uint32_t LO = DP == 64 ? A_BYTES : 0, LOX = DP == 64 ? 0 : 64;   // lo: another image / the row's other half
    if (g == 1 && cur.valid()) cur.advance();
    bool rows = cur.valid();
    if (!rows) return;
    load_perm();
    load_rows();
    bool more = cur.valid();
    if (more) load_perm();
    for (int n = g; rows; n += 2) {
        const int s = n % SLOTS;
        if (!wait(empty + s, (uint32_t)(((n / SLOTS) & 1) ^ 1), ERR_TIMEOUT_EMPTY)) return;
        const uint32_t dst = smem_u32(sA) + (uint32_t)s * O::A;
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
            uint2 hi, lo;
            bf16_split4(pf[u].x, pf[u].y, pf[u].z, pf[u].w, hi, lo);
            const uint32_t at = dst + off[u % PER] + 1024 * (u / PER);
            st_shared_v2(at, hi);
            st_shared_v2((at ^ LOX) + LO, lo);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(full + s);
        rows = more;
        if (rows) load_rows();
        more = more && cur.valid();
        if (more) load_perm();
    }
}

// ------------------------------------------------------------------------- sub-labels
// r_s = c_s - |z_s - b_s|^2 / 2 of both sub-clusters from z = [W_l | W_r]^T x, then log lr_weights, the 2-way
// softmax and the two-category alias draw (cudaKernel.cu:352-372).
// Bound: HBM (the rows once, 256 B a point at D = 64).  Measured: 1e7 points at D = 64 1107 -> 684 us, 1e6 at D = 32
// 123 -> 51 us; what is left is the drain (128 accumulator columns a point against the products and the
// gather on the same shared memory: 383 us with neither gather nor drain)
template <int DP>
struct SubSmem {
    // even numbers of slots and accumulators: each then belongs to one group and one issuer, which see all of
    // its phases (a waiter that skips a phase could take an old one for its own)
    static constexpr int SLOTS = 4;
    static_assert(SLOTS % 2 == 0 && RW_ACC % 2 == 0, "a slot has one owner");
    static constexpr uint32_t B = DP == 64 ? 32768 : 8192;               // [W_l | W_r], 2 DP rows
    static constexpr size_t a = 0;
    static constexpr size_t b = a + (size_t)SLOTS * RowOperand<DP>::A;   // two buffers
    static constexpr size_t bias = b + 2 * (size_t)B;                    // two buffers of 2 DP floats
    static constexpr size_t bar = bias + 2 * (size_t)(2 * DP) * 4;
    static constexpr int FULL = 0, EMPTY = FULL + SLOTS, TFULL = EMPTY + SLOTS, TEMPTY = TFULL + RW_ACC,
                         BFULL = TEMPTY + RW_ACC, BEMPTY = BFULL + 2, NBAR = BEMPTY + 2;
    static constexpr size_t total = bar + NBAR * 8 + 40 + 1024;          // + tmem slot, group outcomes, alignment slack
    static constexpr uint32_t COLS = RW_ACC * 2 * DP;                    // TMEM columns
};

template <int DP>
__global__ void __launch_bounds__(RW_THREADS, 1) k_sub_labels_tc(
    const float* __restrict__ x, const int32_t* __restrict__ perm, const int32_t* __restrict__ chunk,
    const int32_t* __restrict__ nchunks, const uint8_t* __restrict__ Bsub, const float* __restrict__ bvec,
    const float* __restrict__ cvec, const float* __restrict__ lrw, RngArgs rng, int32_t* __restrict__ sub,
    float* __restrict__ r_out, int32_t* __restrict__ err, int stall)
{
    using L = SubSmem<DP>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
    volatile int* stat = reinterpret_cast<volatile int*>(tmem_slot + 2);   // outcome words of the four groups
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = *nchunks;
    if ((int)blockIdx.x >= nch) return;
    if (tid == 0) {
        for (int s = 0; s < L::SLOTS; ++s) {
            mbar_init(bars + L::FULL + s, RW_LOADERS / 2);
            mbar_init(bars + L::EMPTY + s, 1);
        }
        for (int a = 0; a < RW_ACC; ++a) {
            mbar_init(bars + L::TFULL + a, 1);
            mbar_init(bars + L::TEMPTY + a, RW_DRAINS / 2);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bars + L::BFULL + b, 1);
            mbar_init(bars + L::BEMPTY + b, RW_MMAS + RW_DRAINS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == RW_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(L::COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    TileCursor cur(chunk, nch);

    if (warp < RW_LOADERS) {
        const int g = warp / (RW_LOADERS / 2), w = warp - g * (RW_LOADERS / 2);
        load_tiles<DP, L::SLOTS>(x, perm, cur, g, w, smem + L::a, bars + L::FULL, bars + L::EMPTY,
                                 GroupWait{err, stat + 2 * g, 1 + g, 16 * RW_LOADERS, w, 0});
    } else if (warp < RW_MMA) {
        const int quarter = warp & 3, g = (warp - RW_LOADERS) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        GroupWait wait{err, stat + 4 + 2 * g, 3 + g, 16 * RW_DRAINS, (warp - RW_LOADERS) & 3, 0};
        float cl = 0.f, cr = 0.f, wl = 0.f, wr = 0.f;
        bool ok = true;
        for (int n = 0, b = 0; cur.valid() && ok; ++n, cur.advance()) {
            if (cur.t0 == 0) {
                cl = __ldg(cvec + 3 * cur.k + 1);
                cr = __ldg(cvec + 3 * cur.k + 2);
                wl = __ldg(lrw + 2 * cur.k);
                wr = __ldg(lrw + 2 * cur.k + 1);
                ok = wait(bars + L::BFULL + (b & 1), (uint32_t)((b >> 1) & 1), ERR_TIMEOUT_BFULL);
                if (!ok) break;
            }
            if ((n & 1) == g) {
                const bool live = cur.t0 + row < cur.len;
                const int pt = live ? __ldg(perm + cur.start + cur.t0 + row) : 0;
                const int a = n % RW_ACC;
                ok = wait(bars + L::TFULL + a, (uint32_t)((n / RW_ACC) & 1), ERR_TIMEOUT_TFULL);
                if (!ok) break;
                tc_fence_after();
                const float* bias = reinterpret_cast<const float*>(smem + L::bias) + (b & 1) * 2 * DP;
                const uint64_t minus = pack2(-1.f, -1.f);
                float r[2];
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    uint64_t q01 = 0, q23 = 0;   // four sums of squares, two per instruction
#pragma unroll
                    for (int h = 0; h < DP / 32; ++h) {
                        uint32_t v[32];
                        tmem_ld32(tmem_base + lane_addr + (uint32_t)(a * 2 * DP + side * DP + 32 * h), v);
                        const ulonglong2* b4 = reinterpret_cast<const ulonglong2*>(bias + side * DP + 32 * h);
#pragma unroll
                        for (int j4 = 0; j4 < 8; ++j4) {
                            const ulonglong2 bb = b4[j4];
                            const uint64_t z01 = fma2(bb.x, minus, pack2(__uint_as_float(v[4 * j4]), __uint_as_float(v[4 * j4 + 1])));
                            const uint64_t z23 = fma2(bb.y, minus, pack2(__uint_as_float(v[4 * j4 + 2]), __uint_as_float(v[4 * j4 + 3])));
                            q01 = fma2(z01, z01, q01);
                            q23 = fma2(z23, z23, q23);
                        }
                    }
                    float q0, q1, q2, q3;
                    unpack2(q01, q0, q1);
                    unpack2(q23, q2, q3);
                    r[side] = (side ? cr : cl) - 0.5f * ((q0 + q1) + (q2 + q3));
                }
                tc_fence_before();
                warp_arrive(bars + L::TEMPTY + a);
                if (live) {
                    float rl = r[0], rr = r[1];
                    if (r_out) { r_out[2 * (size_t)pt] = rl; r_out[2 * (size_t)pt + 1] = rr; }
                    rl += wl;
                    rr += wr;
                    float u1, u2;
                    draw_uniform2(rng, pt, u1, u2);
                    sub[pt] = draw_sub_label(rl, rr, u1, u2);
                }
            }
            if (cur.last_tile()) {
                warp_arrive(bars + L::BEMPTY + (b & 1));
                ++b;
            }
        }
    } else if (warp < RW_COPY) {
        if (lane == 0 && !stall) {   // stall (test seam): no product is issued, the waits for them run out
            const int m = warp - RW_MMA;
            int n = 0, issued = 0;
            for (int b = 0; cur.valid(); ++n, cur.advance()) {
                if (cur.t0 == 0 && !thread_wait(bars + L::BFULL + (b & 1), (uint32_t)((b >> 1) & 1), err, ERR_TIMEOUT_BFULL))
                    break;   // (every chunk's, whether or not a tile of it is this issuer's)
                if ((n & 1) == m) {
                    const int s = n % L::SLOTS, a = n % RW_ACC;
                    if (!thread_wait(bars + L::FULL + s, (uint32_t)((n / L::SLOTS) & 1), err, ERR_TIMEOUT_FULL)) break;
                    if (!thread_wait(bars + L::TEMPTY + a, (uint32_t)(((n / RW_ACC) & 1) ^ 1), err, ERR_TIMEOUT_TEMPTY)) break;
                    tc_fence_after();
                    issue_split3<DP>(tmem_base + (uint32_t)(a * 2 * DP),
                                     smem_u32(smem + L::a + (size_t)s * RowOperand<DP>::A),
                                     smem_u32(smem + L::b + (size_t)(b & 1) * L::B), 2 * DP);
                    umma_commit(bars + L::EMPTY + s);
                    umma_commit(bars + L::TFULL + a);
                    issued = n + 1;
                }
                if (cur.last_tile()) {
                    umma_commit(bars + L::BEMPTY + (b & 1));   // (of nothing, if this issuer had no tile of the chunk)
                    ++b;
                }
            }
            // nothing in flight when the tensor memory is freed
            if (issued > 0)
                mbar_wait_bounded(bars + L::TFULL + (issued - 1) % RW_ACC, (uint32_t)(((issued - 1) / RW_ACC) & 1), nullptr);
        }
    } else if (warp == RW_COPY && lane == 0) {
        int b = 0;
        for (int q = blockIdx.x; q < nch; q += gridDim.x, ++b) {
            if (b >= 2 && !thread_wait(bars + L::BEMPTY + (b & 1), (uint32_t)(((b >> 1) - 1) & 1), err, ERR_TIMEOUT_BEMPTY)) break;
            const int k = __ldg(chunk + 3 * q);
            uint64_t* full = bars + L::BFULL + (b & 1);
            mbar_arrive_expect_tx(full, L::B + 2 * DP * 4);
            bulk_copy_g2s(smem + L::b + (size_t)(b & 1) * L::B, Bsub + (size_t)k * L::B, L::B, full);
            bulk_copy_g2s(smem + L::bias + (size_t)(b & 1) * 2 * DP * 4, bvec + (size_t)(3 * k + 1) * DP, 2 * DP * 4, full);
        }
        // every copy has landed before shared memory is released
        for (int p = b > 2 ? b - 2 : 0; p < b; ++p) mbar_wait_bounded(bars + L::BFULL + (p & 1), (uint32_t)((p >> 1) & 1), nullptr);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == RW_MMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(L::COLS));
    }
}

// B operand at DP = 32: per cluster 64 rows (l 0..31, r 32..63) of [32 hi | 32 lo], 8 KB
__global__ void k_pack_sub32(const float* __restrict__ Wt, int K, uint8_t* __restrict__ Bsub)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;   // (cluster, row, piece of 8)
    if (e >= K * 64 * 4) return;
    const int k = e / 256, n = (e / 4) % 64, c8 = e % 4;
    const float* src = Wt + ((size_t)(3 * k + 1 + n / 32) * 32 + n % 32) * 32 + c8 * 8;
    uint2 h0, l0, h1, l1;
    bf16_split4(src[0], src[1], src[2], src[3], h0, l0);
    bf16_split4(src[4], src[5], src[6], src[7], h1, l1);
    uint8_t* dst = Bsub + (size_t)k * 8192;
    *reinterpret_cast<uint4*>(dst + RowOperand<32>::hi(n, 2 * c8)) = make_uint4(h0.x, h0.y, h1.x, h1.y);
    *reinterpret_cast<uint4*>(dst + RowOperand<32>::lo(n, 2 * c8)) = make_uint4(l0.x, l0.y, l1.x, l1.y);
}

}  // namespace tc

bool tc_sub_supported(const dpmm_ctx* c)
{
    return c->prior == DPMM_PRIOR_GAUSSIAN && c->d_Bsub != nullptr && (c->Dp == 32 || c->Dp == 64) &&
           c->ll_mode != DPMM_LL_FP32;
}

dpmm_status pack_sub32_params(dpmm_ctx* c, int K)
{
    tc::k_pack_sub32<<<(K * 256 + 255) / 256, 256, 0, c->stream>>>(c->d_Wt, K, c->d_Bsub32);
    DPMM_LAUNCHED();
    return DPMM_OK;
}

template <int DP>
static dpmm_status launch_sub_labels_tc_t(dpmm_ctx* c, RngArgs r, float* d_rout, int32_t* err)
{
    auto kern = tc::k_sub_labels_tc<DP>;
    static_assert(tc::SubSmem<DP>::total <= tc::kTcSmemCap, "shared memory");
    DPMM_TRY(allow_smem(kern, tc::SubSmem<DP>::total));
    kern<<<std::min(c->num_sms, c->max_chunks), tc::RW_THREADS, tc::SubSmem<DP>::total, c->stream>>>(
        c->d_x, c->d_perm, c->d_chunk, c->d_nchunks, DP == 32 ? c->d_Bsub32 : c->d_Bsub, c->d_b, c->d_c, c->d_lrw, r,
        c->d_sub, d_rout, err, c->stall_tc_mma);
    DPMM_LAUNCHED();
    return DPMM_OK;
}

dpmm_status launch_sub_labels_tc(dpmm_ctx* c, RngArgs r, float* d_rout, bool defer_check)
{
    int32_t* err = c->d_aux + 5;
    DPMM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int32_t), c->stream));
    if (c->Dp == 64) DPMM_TRY(launch_sub_labels_tc_t<64>(c, r, d_rout, err));
    else DPMM_TRY(launch_sub_labels_tc_t<32>(c, r, d_rout, err));
    if (defer_check) {
        c->sub_err_pending = true;
        return DPMM_OK;
    }
    int32_t h_err = 0;
    DPMM_CUDA_TRY(cudaMemcpyAsync(&h_err, err, sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream));
    DPMM_CUDA_TRY(cudaStreamSynchronize(c->stream));
    if (h_err) return fail(DPMM_ERR_TIMEOUT, "tensor-core sub-label kernel: bounded wait expired (code " +
                                                 std::to_string(h_err) + ")");
    return DPMM_OK;
}

}  // namespace dpmm
