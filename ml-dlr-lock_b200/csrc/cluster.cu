// Large-batch ("prefill") DLR-Net forward on thread-block clusters with tcgen05
// tensor cores and tensor memory.
//
// Work split.  A cluster of CS = d / W CTAs (W = 512 or 256 columns) walks all L
// layers for one tile of 128 token rows; CTA `rank` owns columns [W*rank,
// W*rank+W) of the model width for BOTH contractions of a layer (K-stripe of the
// V contraction, N-stripe of the U contraction - the reference's cooperative
// scheme, kernels/kernels/cuda/cooperative.cu:10-16, moved from global memory to
// distributed shared memory).  Per layer (dlr_lock/model.py:96-100 on folded
// weights, kernels/README.md:5-7):
//
//   V:  z_part[128 x r]  = h[128 x W] . V'[:, stripe]^T       tcgen05.mma, A from TMEM
//   X:  z = sum over the cluster of z_part, sumsq likewise    DSMEM reduce-scatter by rows
//       s = silu(z * rsqrt(sumsq/d + eps)) as bf16            DSMEM all-gather
//   U:  dh[128 x W]      = s[128 x r] . U'[stripe, :]^T       tcgen05.mma, A and B from smem
//       h += dh ; sumsq_part = sum h^2                        fused epilogue out of TMEM
//
// On-chip residency.  W/2 tensor-memory columns hold the activation stripe
// (128 x W) as packed bf16 for the whole stack - it is the A operand of the V
// contraction straight from TMEM.  The activation is re-rounded to bf16 once per
// layer, like every fused kernel of the reference (fp32 accumulation inside a
// layer).  Partial z travels between CTAs as bf16 (summed in fp32): it is
// rounded to bf16 right after the sum anyway, and the end-to-end error is
// unchanged by it.
//
// What bounds it: the chain V -> exchange -> U -> epilogue of a layer, not a
// throughput.  So U of layer l and V of layer l + 1 run interleaved over chunks of
// 64 columns: a chunk that the epilogue has updated goes to the V contraction while
// the next ones are still being worked on (z has an accumulator of its own beside
// those of dh), and behind the last chunk's epilogue only its own four
// instructions are left of V.  The epilogue is 16 warps in two groups of 8, each
// with the chunks of one parity: a chunk's chain (wait, tensor-memory load, add,
// store, signal) is latency, which the other group fills.
// Measured on a B200 (us; V after U, 8 epilogue warps and a stripe of 512 / this form): d = 1024, r = 32, 4096 rows
// 662 / 454; d = 4096, r = 128, 1000 rows 1100 / 1066, where the two hops of the exchange (28 KB each per CTA) take
// 5 k of a layer's 12.5 k cycles.
//
// Exchange mechanics.  Every remote write is an asynchronous store
// (st.async ... shared::cluster) whose bytes are counted on the RECEIVER's
// mbarrier, so no fences or remote arrivals are needed: a row's partial z
// (bf16) and its partial sum of squares go straight from the accumulators to
// the row's owner; the owner's s rows go to every CTA of the cluster, written
// directly in the core-matrix layout the MMA reads (8 rows x 16 bytes
// contiguous, no swizzle), which also makes each warp's stores contiguous.
//
// Roles.  Warp 0 streams weight tiles with TMA into two deep rings (U' and V')
// and never waits for activations; warp 1 issues U, warp 2 issues V; warps 4-19
// (four threads per row) run exchange and epilogue.  All waits are bounded
// mbarrier waits; a wait that gives up records a status word and every role
// drains to a common exit.
#include <atomic>
#include <cstdlib>
#include <cstring>

#include "cluster.h"
#include "ptx.cuh"

namespace dlr {

namespace {

constexpr int kRows = 128;
constexpr int kCW = 64;              // columns per chunk
constexpr int kMaxStages = 16;       // per ring
constexpr int kEpiWarps = 16;
constexpr int kEpi = 32 * kEpiWarps; // epilogue threads
constexpr int kThreads = 128 + kEpi;
constexpr int kProfWords = 8;       // cycle counters per CTA (debug)

struct ClusterParams {
    const __nv_bfloat16* x;
    __nv_bfloat16* y;
    int M, d, L;
    float eps, inv_d;
    int* status;
    int* mirror;                // host copy of the status word, or null
    unsigned int spin_limit;
    int stages;                 // per ring
    int num_tiles;
    unsigned long long* prof;   // optional per-CTA phase cycle counters (debug), or null
};

template <int R, int CS, int W>
struct CCfg {
    static constexpr int NCH = W / kCW;            // chunks per stripe
    static constexpr int KW = R < 64 ? R : 64;     // K columns per U' box
    static constexpr int UK = R / KW;              // U' boxes per chunk
    // tensor-memory columns: packed bf16 activation [0, W/2) | z (R columns) | as many dh accumulators as fit
    static constexpr uint32_t H_COL = 0, Z_COL = W / 2, ACC_COL = W / 2 + R;
    static constexpr int FIT = (512 - W / 2 - R) / kCW;
    static constexpr int NB = FIT < NCH ? FIT : NCH;
    static constexpr int S_BYTES = kRows * R * 2;  // s tile (A operand of the U contraction)
    static constexpr int NCK = R / 8;              // 16-byte K chunks per row
    static constexpr int S_GROUP_BYTES = NCK * 128;          // one 8-row group of the s tile
    static constexpr int R_GROUP_BYTES = (NCK + 1) * 128;    // same plus 16 bytes a row: four partial sums of squares
    static constexpr int RECV_BYTES = (kRows / 8) * R_GROUP_BYTES;
    static constexpr int STAGE_BYTES = R * 128;              // a chunk of V' (R rows x 64 K columns) or of U' (64 rows x R)
    static constexpr int U_BOX_BYTES = kCW * KW * 2;
    static constexpr uint32_t U_LAYOUT = KW == 64 ? 2u : 4u; // descriptor layout type (128- / 64-byte swizzle)
    static constexpr uint32_t U_SBO = 8 * KW * 2;            // bytes between 8-row groups of a U' box
    static constexpr int FIXED_BYTES = S_BYTES + RECV_BYTES + 1024 /*barriers*/ + 1024 /*alignment*/;
    // The owner's share of z: rows_own rows, in pieces of 16 bytes, or of 8 where that leaves threads idle.
    static constexpr int ROWS_OWN = kRows / CS;
    static constexpr int PIECE = ROWS_OWN * NCK >= kEpi ? 16 : 8;
    static constexpr int PIECES = ROWS_OWN * R * 2 / PIECE;
    static constexpr int PER_GROUP = 8 * NCK * 16 / PIECE;   // pieces per 8-row group
    static_assert(ROWS_OWN % 8 == 0 && NCH % 2 == 0 && NB >= 2 && R <= 128, "split");
};

#define DLR_CLK() (p.prof ? clock64() : 0ll)

struct Bars {
    uint64_t v_full[kMaxStages], v_empty[kMaxStages];
    uint64_t u_full[kMaxStages], u_empty[kMaxStages];
    uint64_t z_full;         // V-MMA warp -> epilogue: the partial z is complete
    uint64_t recv_full;      // peers -> owner: all partials and sums of squares landed (byte count)
    uint64_t s_full;         // peers -> U-MMA warp: the whole s tile landed (byte count)
    uint64_t dh_full[4];     // U-MMA warp -> the chunk's epilogue group: a dh chunk is in accumulator b
    uint64_t acc_empty[4];   // the 8 warps of that group -> U-MMA warp: accumulator b drained
    uint64_t h_ready[8];     // per chunk, the 8 warps of its group -> V-MMA warp: the chunk is updated in tensor memory
    uint64_t drain[2];       // all tensor-core work of an MMA warp is complete (waited for before leaving)
    uint32_t tmem_slot;
    int abort_flag;
};
static_assert(sizeof(Bars) <= 1024, "barrier block");

template <int R, int CS, int W>
__global__ void __launch_bounds__(kThreads, 1)
dlr_cluster_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmU,
                   ClusterParams p) {
    using C = CCfg<R, CS, W>;
    constexpr int NCH = C::NCH, NB = C::NB, rows_own = C::ROWS_OWN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t S = uint32_t(p.stages);
    uint8_t* vring = smem;
    uint8_t* uring = vring + size_t(S) * C::STAGE_BYTES;
    uint8_t* sbuf = uring + size_t(S) * C::STAGE_BYTES;   // s tile, core-matrix layout
    uint8_t* recv = sbuf + C::S_BYTES;                    // [source][8-row group][chunk][row in group] x 16 B
    Bars* bars = reinterpret_cast<Bars*>(recv + C::RECV_BYTES);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0);
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int cluster_id = blockIdx.x / CS;
    const int num_clusters = gridDim.x / CS;
    const int stripe0 = int(rank) * W;
    const uint32_t flag_s = smem_u32(&bars->abort_flag);
    const uint32_t limit = p.spin_limit >= 4 ? p.spin_limit >> 2 : 1u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(smem_u32(&bars->v_full[s]), 1);
            mbar_init(smem_u32(&bars->v_empty[s]), 1);
            mbar_init(smem_u32(&bars->u_full[s]), 1);
            mbar_init(smem_u32(&bars->u_empty[s]), 1);
        }
        for (int b = 0; b < 4; ++b) {
            mbar_init(smem_u32(&bars->dh_full[b]), 1);
            mbar_init(smem_u32(&bars->acc_empty[b]), kEpiWarps / 2);
        }
        for (int c = 0; c < 8; ++c) mbar_init(smem_u32(&bars->h_ready[c]), kEpiWarps / 2);
        mbar_init(smem_u32(&bars->z_full), 1);
        mbar_init(smem_u32(&bars->recv_full), 1);   // the local arrive that arms the byte count
        mbar_init(smem_u32(&bars->s_full), 1);
        mbar_init(smem_u32(&bars->drain[0]), 1);
        mbar_init(smem_u32(&bars->drain[1]), 1);
        bars->abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmU);
    }
    if (warp == 3) {
        tmem_alloc(smem_u32(&bars->tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive_release();
    cluster_wait_acquire();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_slot;
    const uint32_t vring_s = smem_u32(vring), uring_s = smem_u32(uring);
    const uint32_t sbuf_s = smem_u32(sbuf);
    const uint32_t recv_s = smem_u32(recv);

    int err = 0;
    int err_layer = 0;
    auto wait_cta = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(smem_u32(bar), parity, flag_s, limit); };
    auto wait_cluster = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp_cluster(smem_u32(bar), parity, flag_s, limit); };

    if (warp == 0) {
        // =============================== TMA producer ===============================
        // in the order of use: V' of layer 0, then chunk by chunk U' of a layer and V' of the next
        {
            RingPos up, vp;
            uint32_t nu = 0, nv = 0;
            auto ask_v = [&](int l, int c) {
                if (!wait_cta(&bars->v_empty[vp.st], vp.ph ^ 1u)) { err = DLRB200_ERR_TIMEOUT_COPY; err_layer = l; return; }
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&bars->v_full[vp.st]);
                    mbar_arrive_expect_tx(bar, C::STAGE_BYTES);
                    tma_load_2d(vring_s + vp.st * C::STAGE_BYTES, &tmV, stripe0 + kCW * c, l * R, bar);
                }
                __syncwarp();
                vp.step(S);
                ++nv;
            };
            auto ask_u = [&](int l, int c) {
                if (!wait_cta(&bars->u_empty[up.st], up.ph ^ 1u)) { err = DLRB200_ERR_TIMEOUT_COPY; err_layer = l; return; }
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&bars->u_full[up.st]);
                    mbar_arrive_expect_tx(bar, C::STAGE_BYTES);
#pragma unroll
                    for (int k = 0; k < C::UK; ++k)
                        tma_load_2d(uring_s + up.st * C::STAGE_BYTES + k * C::U_BOX_BYTES, &tmU, k * C::KW, l * p.d + stripe0 + kCW * c, bar);
                }
                __syncwarp();
                up.step(S);
                ++nu;
            };
            for (int tile = cluster_id; tile < p.num_tiles && !err; tile += num_clusters) {
                for (int c = 0; c < NCH && !err; ++c) ask_v(0, c);
                for (int l = 0; l < p.L && !err; ++l)
                    for (int c = 0; c < NCH && !err; ++c) {
                        ask_u(l, c);
                        if (l + 1 < p.L && !err) ask_v(l + 1, c);
                    }
            }
            // the copies asked for land in this CTA's rings: wait (bounded) for the last of every stage before leaving
            for (uint32_t back = 1; back <= S; ++back) {
                if (back <= nv) mbar_wait(smem_u32(&bars->v_full[(nv - back) % S]), ((nv - back) / S) & 1u, kDrainPolls);
                if (back <= nu) mbar_wait(smem_u32(&bars->u_full[(nu - back) % S]), ((nu - back) / S) & 1u, kDrainPolls);
            }
        }
    } else if (warp == 1) {
        // =============================== U-MMA warp ================================
        {
            constexpr uint32_t idesc_u = umma_idesc_bf16(128, kCW);
            RingPos up, ap;                      // weights, accumulators
            uint32_t c_s = 0;
            for (int tile = cluster_id; tile < p.num_tiles && !err; tile += num_clusters) {
                for (int l = 0; l < p.L && !err; ++l) {
                    err_layer = l;
                    if (!wait_cluster(&bars->s_full, c_s & 1u)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                    ++c_s;
                    fence_async_smem();          // the peers' stores, before the tensor core reads them
                    for (int c = 0; c < NCH; ++c) {
                        // the weights land early: wait for them first, off the critical path
                        if (!wait_cta(&bars->u_full[up.st], up.ph)) { err = DLRB200_ERR_TIMEOUT_COPY; break; }
                        if (!wait_cta(&bars->acc_empty[ap.st], ap.ph ^ 1u)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                        tc_fence_after();
                        const uint32_t acc = tmem_base + C::ACC_COL + ap.st * uint32_t(kCW);
                        const uint32_t ub = uring_s + up.st * C::STAGE_BYTES;
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < R / 16; ++k) {
                                // K step k of the s tile: two 16-byte chunks, 128 bytes apart
                                const uint64_t adesc = umma_desc_nosw(sbuf_s + uint32_t(k) * 256u, 128u, C::S_GROUP_BYTES);
                                const uint64_t bdesc = umma_desc(ub + uint32_t(k / (C::KW / 16)) * C::U_BOX_BYTES, C::U_LAYOUT, C::U_SBO) +
                                                       uint64_t(2 * (k % (C::KW / 16)));
                                umma_ss(acc, adesc, bdesc, idesc_u, k ? 1u : 0u);
                            }
                            umma_commit(smem_u32(&bars->u_empty[up.st]));
                            umma_commit(smem_u32(&bars->dh_full[ap.st]));
                        }
                        __syncwarp();
                        up.step(S);
                        ap.step(NB);
                    }
                }
            }
            if (elect_one()) umma_commit(smem_u32(&bars->drain[0]));
            __syncwarp();
            mbar_wait(smem_u32(&bars->drain[0]), 0, kDrainPolls);
        }
    } else if (warp == 2) {
        // =============================== V-MMA warp ================================
        {
            constexpr uint32_t idesc_v = umma_idesc_bf16(128, R);
            RingPos vp;
            uint32_t c_h = 0;
            for (int tile = cluster_id; tile < p.num_tiles && !err; tile += num_clusters) {
                for (int l = 0; l < p.L && !err; ++l, ++c_h) {
                    err_layer = l;
                    for (int c = 0; c < NCH; ++c) {
                        if (!wait_cta(&bars->v_full[vp.st], vp.ph)) { err = DLRB200_ERR_TIMEOUT_COPY; break; }
                        if (!wait_cta(&bars->h_ready[c], c_h & 1u)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                        tc_fence_after();
                        const uint64_t bdesc = umma_desc(vring_s + vp.st * C::STAGE_BYTES, 2u, 1024u);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < kCW / 16; ++k)
                                umma_ts(tmem_base + C::Z_COL, tmem_base + C::H_COL + uint32_t(c * (kCW / 2) + k * 8), bdesc + uint64_t(2 * k),
                                        idesc_v, (c | k) ? 1u : 0u);
                            umma_commit(smem_u32(&bars->v_empty[vp.st]));
                        }
                        __syncwarp();
                        vp.step(S);
                    }
                    if (err) break;
                    if (elect_one()) umma_commit(smem_u32(&bars->z_full));
                    __syncwarp();
                }
            }
            if (elect_one()) umma_commit(smem_u32(&bars->drain[1]));
            __syncwarp();
            mbar_wait(smem_u32(&bars->drain[1]), 0, kDrainPolls);
        }
    } else if (warp >= 4) {
        // =============================== epilogue warps =============================
        // Four threads per row: thread (row er, quarter cq) owns a quarter of the columns of z, and half hc of every
        // chunk of parity g.  Warp w reads tensor-memory lanes 32 * (w % 4) .. + 31.
        const int et = int(threadIdx.x) - 128;       // 0..511
        const int q = warp & 3;
        const int cq = (warp - 4) >> 2;
        const int g = cq >> 1, hc = cq & 1;
        const int er = 32 * q + lane;                // row of the tile
        const uint32_t tl = tmem_base + (uint32_t(32 * q) << 16);
        const int owner = er / rows_own;
        const int lr = er % rows_own;
        constexpr int groups_own = rows_own / 8;     // 8-row groups per owner
        constexpr uint32_t src_bytes = uint32_t(groups_own) * C::R_GROUP_BYTES;   // one source's block in recv
        constexpr int NZ = R / 4;                    // columns of z per thread
        // this row's slot in its owner's receive buffer
        const uint32_t dst = mapa(recv_s + uint32_t(rank) * src_bytes + uint32_t(lr >> 3) * C::R_GROUP_BYTES + uint32_t(lr & 7) * 16u,
                                  uint32_t(owner));
        const uint32_t rbar = mapa(smem_u32(&bars->recv_full), uint32_t(owner));
        uint32_t c_l = 0;                            // layers
        RingPos ap;                                  // accumulator of this group's next chunk
        ap.advance(uint32_t(g), NB);
        long long e[5] = {0, 0, 0, 0, 0};

        for (int tile = cluster_id; tile < p.num_tiles && !err; tile += num_clusters) {
            const int grow = tile * kRows + er;
            const bool valid = grow < p.M;
            const size_t at = size_t(valid ? grow : 0) * p.d + stripe0 + 32 * hc;
            float ssq0 = 0.f, ssq1 = 0.f;
            // ---- input stripe -> tensor memory (packed bf16), partial sum of squares
#pragma unroll
            for (int i = 0; i < NCH / 2; ++i) {
                const int c = 2 * i + g;
                uint32_t v[16];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint4 a = make_uint4(0u, 0u, 0u, 0u);
                    if (valid) a = __ldg(reinterpret_cast<const uint4*>(p.x + at + kCW * c) + j);
                    v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = a.z; v[4 * j + 3] = a.w;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float lo = bf16lo_to_f(v[j]), hi = bf16hi_to_f(v[j]);
                    fma_f32x2(ssq0, ssq1, lo, hi, lo, hi, ssq0, ssq1);
                }
                tmem_st16(tl + C::H_COL + uint32_t(c * (kCW / 2) + 16 * hc), v);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->h_ready[c]));
            }

            for (int l = 0; l < p.L && !err; ++l, ++c_l) {
                err_layer = l;
                const uint32_t lpar = c_l & 1u;
                const long long t0 = DLR_CLK();
                // ---- partial z of this row -> bf16 -> the row's owner
                if (!wait_cta(&bars->z_full, lpar)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                tc_fence_after();
                const long long t1 = DLR_CLK();
                if (et == 0) mbar_arrive_expect_tx(smem_u32(&bars->recv_full), C::RECV_BYTES);   // arm this layer's receive
                st_async_b32(dst + uint32_t(C::NCK * 128 + cq * 4), __float_as_uint(ssq0 + ssq1), rbar);
                {
                    uint32_t zv[NZ];
                    const uint32_t zcol = tl + C::Z_COL + uint32_t(NZ * cq);
                    if constexpr (NZ == 32) tmem_ld32(zcol, zv);
                    else if constexpr (NZ == 16) tmem_ld16(zcol, zv);
                    else tmem_ld8(zcol, zv);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < NZ / 8; ++j) {
                        uint32_t pk[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            pk[i] = pack_bf16x2(__uint_as_float(zv[8 * j + 2 * i]), __uint_as_float(zv[8 * j + 2 * i + 1]));
                        st_async_v4(dst + uint32_t(NZ * cq / 8 + j) * 128u, pk[0], pk[1], pk[2], pk[3], rbar);
                    }
                }
                tc_fence_before();      // (z has been read: the V contraction that overwrites it waits for this layer's s)
                const long long t2 = DLR_CLK();

                // ---- owner: sum the CS partials of its rows, normalise, SiLU, all-gather
                if (!wait_cluster(&bars->recv_full, lpar)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                const long long t3 = DLR_CLK();
                if (et == 0) mbar_arrive_expect_tx(smem_u32(&bars->s_full), C::S_BYTES);      // arm this layer's s tile
#pragma unroll
                for (int it = 0; it * kEpi < C::PIECES; ++it) {
                    const int i = et + kEpi * it;
                    constexpr int SUB = 16 / C::PIECE, NV = C::PIECE / 2;     // pieces per 16 bytes, values per piece
                    if (C::PIECES % kEpi != 0 && i >= C::PIECES) break;
                    const int sub = i % SUB;
                    const int r8 = (i / SUB) & 7;
                    const int c = (i / (8 * SUB)) % C::NCK;
                    const int gl = i / C::PER_GROUP;      // 8-row group inside this owner's rows
                    const uint8_t* base = recv + size_t(gl) * C::R_GROUP_BYTES + r8 * 16;
                    float tot = 0.f;
                    float a[NV];
#pragma unroll
                    for (int j = 0; j < NV; ++j) a[j] = 0.f;
#pragma unroll
                    for (int src = 0; src < CS; ++src) {
                        const uint8_t* bp = base + size_t(src) * src_bytes;
                        const float4 qq = *reinterpret_cast<const float4*>(bp + C::NCK * 128);
                        tot += (qq.x + qq.y) + (qq.z + qq.w);
                        uint32_t u[NV / 2];
                        if constexpr (NV == 8) {
                            const uint4 w4 = *reinterpret_cast<const uint4*>(bp + c * 128);
                            u[0] = w4.x; u[1] = w4.y; u[2] = w4.z; u[3] = w4.w;
                        } else {
                            const uint2 w2 = *reinterpret_cast<const uint2*>(bp + c * 128 + sub * 8);
                            u[0] = w2.x; u[1] = w2.y;
                        }
#pragma unroll
                        for (int j = 0; j < NV / 2; ++j) { a[2 * j] += bf16lo_to_f(u[j]); a[2 * j + 1] += bf16hi_to_f(u[j]); }
                    }
                    const float rstd = rsqrtf(tot * p.inv_d + p.eps);
                    uint32_t o[NV / 2];
#pragma unroll
                    for (int j = 0; j < NV / 2; ++j) o[j] = pack_bf16x2(silu_f(a[2 * j] * rstd), silu_f(a[2 * j + 1] * rstd));
                    // row (rank*rows_own + 8*gl + r8) of the s tile, chunk c, in every CTA of the cluster
                    const uint32_t so = sbuf_s + uint32_t(int(rank) * groups_own + gl) * C::S_GROUP_BYTES + uint32_t(c) * 128u +
                                        uint32_t(r8) * 16u + uint32_t(sub) * 8u;
#pragma unroll
                    for (int dc = 0; dc < CS; ++dc) {
                        const uint32_t to = mapa(so, uint32_t(dc)), bar = mapa(smem_u32(&bars->s_full), uint32_t(dc));
                        if constexpr (NV == 8) st_async_v4(to, o[0], o[1], o[2], o[3], bar);
                        else st_async_v2(to, o[0], o[1], bar);
                    }
                }
                const long long t4 = DLR_CLK();

                // ---- fused epilogue of the U contraction: h += dh, new sum of squares
                ssq0 = ssq1 = 0.f;
#pragma unroll 1
                for (int c = g; c < NCH; c += 2) {
                    const uint32_t b = ap.st;
                    if (!wait_cta(&bars->dh_full[b], ap.ph)) { err = DLRB200_ERR_TIMEOUT_BARRIER; break; }
                    ap.advance(2, NB);
                    tc_fence_after();
                    const uint32_t hcol = tl + C::H_COL + uint32_t(c * (kCW / 2) + 16 * hc);
                    uint32_t dh[32], hp[16];
                    tmem_ld32(tl + C::ACC_COL + b * uint32_t(kCW) + uint32_t(32 * hc), dh);
                    tmem_ld16(hcol, hp);
                    tmem_wait_ld();
                    // the dh values are in registers: the accumulator can take another chunk
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[b]));
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float lo, hi;
                        add_f32x2(lo, hi, bf16lo_to_f(hp[j]), bf16hi_to_f(hp[j]), __uint_as_float(dh[2 * j]), __uint_as_float(dh[2 * j + 1]));
                        fma_f32x2(ssq0, ssq1, lo, hi, lo, hi, ssq0, ssq1);
                        hp[j] = pack_bf16x2(lo, hi);
                    }
                    if (l + 1 < p.L) {
                        tmem_st16(hcol, hp);
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&bars->h_ready[c]));
                    } else if (valid) {
                        uint4* yo = reinterpret_cast<uint4*>(p.y + at + kCW * c);
#pragma unroll
                        for (int j = 0; j < 4; ++j) yo[j] = make_uint4(hp[4 * j], hp[4 * j + 1], hp[4 * j + 2], hp[4 * j + 3]);
                    }
                }
                e[0] += t1 - t0; e[1] += t2 - t1; e[2] += t3 - t2; e[3] += t4 - t3; e[4] += DLR_CLK() - t4;
            }
        }
        if (p.prof && et == 0)
            for (int k = 0; k < 5; ++k) p.prof[blockIdx.x * kProfWords + k] = (unsigned long long)e[k];
    }

    if (err) {
        *reinterpret_cast<volatile int*>(&bars->abort_flag) = 1;
        report_status(p.status, p.mirror, err | (err_layer << 8));
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    // no CTA may leave while a peer can still write into its shared memory
    cluster_arrive_release();
    cluster_wait_acquire();
    if (warp == 3) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

struct CArgs {
    void* enc;
    const void* x;
    void* y;
    const void* Vp;
    const void* Up;
    int M, d, L;
    float eps;
    int* status;
    cudaStream_t stream;
    int num_sms, smem_optin;
    unsigned int spin_limit;
    unsigned long long* prof;
};

constexpr int kMaxDevices = 64;

template <int R, int CS, int W>
struct CLaunch {
    using C = CCfg<R, CS, W>;
    int stages = 0, smem = 0;

    explicit CLaunch(int smem_optin) {
        stages = (smem_optin - C::FIXED_BYTES) / (2 * C::STAGE_BYTES);
        if (stages > kMaxStages) stages = kMaxStages;
        smem = 2 * stages * C::STAGE_BYTES + C::FIXED_BYTES;
    }

    void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int clusters, cudaStream_t stream) const {
        memset(&cfg, 0, sizeof(cfg));
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CS;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(kThreads);
        cfg.gridDim = dim3(CS * clusters);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }

    // Clusters that can be resident at once on the current device (asked for once per device: the query and the opt-in to
    // large shared memory take longer than a launch), or -1.
    int max_clusters(int num_sms) const {
        static std::atomic<int> known[kMaxDevices];          // 0: not known yet
        int dev = 0;
        if (stages < 2 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
        int n = known[dev].load(std::memory_order_acquire);
        if (n != 0) return n;
        auto kern = dlr_cluster_kernel<R, CS, W>;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cfg, attr, num_sms / CS, nullptr);
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            return -1;                                       // (not kept: it may have failed for a passing reason)
        }
        known[dev].store(n, std::memory_order_release);
        return n;
    }

    // waves of 128-row tiles, or 0
    int waves(int M, int num_sms) const {
        const int mc = max_clusters(num_sms), tiles = (M + kRows - 1) / kRows;
        return mc < 1 ? 0 : (tiles + mc - 1) / mc;
    }

    int run(const CArgs& a, dlrb200_plan* plan_only) const {
        const int mc = max_clusters(a.num_sms);
        if (mc < 1) return DLRB200_ERR_OCCUPANCY;
        const int num_tiles = (a.M + kRows - 1) / kRows;
        const int clusters = num_tiles < mc ? num_tiles : mc;
        if (plan_only) {
            plan_only->path = DLRB200_PATH_CLUSTER;
            plan_only->grid = CS * clusters;
            plan_only->cluster = CS;
            plan_only->stripe_cols = W;
            plan_only->rows_per_pass = kRows;
            plan_only->passes = (num_tiles + clusters - 1) / clusters;   // waves of row tiles
            plan_only->stages = 2 * stages;
            plan_only->smem_bytes = size_t(smem);
            return DLRB200_OK;
        }
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cfg, attr, clusters, a.stream);
        ClusterParams p;
        p.x = static_cast<const __nv_bfloat16*>(a.x);
        p.y = static_cast<__nv_bfloat16*>(a.y);
        p.M = a.M; p.d = a.d; p.L = a.L; p.eps = a.eps; p.inv_d = 1.0f / float(a.d);
        p.status = a.status;
        p.mirror = status_mirror(a.status);
        p.spin_limit = a.spin_limit;
        p.stages = stages;
        p.num_tiles = num_tiles;
        p.prof = a.prof;
        CUtensorMap tmV, tmU;
        if (!encode_2d_bf16(a.enc, &tmV, a.Vp, uint64_t(a.d), uint64_t(a.L) * R, kCW, R, 128) ||
            !encode_2d_bf16(a.enc, &tmU, a.Up, uint64_t(R), uint64_t(a.L) * a.d, C::KW, kCW, C::KW * 2))
            return DLRB200_ERR_CUDA;
        const cudaError_t ce = cudaLaunchKernelEx(&cfg, dlr_cluster_kernel<R, CS, W>, tmV, tmU, p);
        return ce == cudaSuccess ? DLRB200_OK : DLRB200_ERR_CUDA;
    }
};

// Microseconds per layer and wave of tiles, measured on a B200 with every cluster of the wave at work.
constexpr double layer_us(int r, int w) {
    return w == 256 ? (r >= 128 ? 5.9 : (r >= 64 ? 3.9 : 3.2)) : (r >= 128 ? 7.5 : (r >= 64 ? 5.2 : 4.1));
}

// A stripe of 512 columns per CTA, or of 256 where a cluster of twice the CTAs is still portable (8) and its shorter layers
// outweigh the waves it may need more.  Measured (us, 512 / 256): d = 1024, r = 32: 4096 rows 567 / 454, 4608 rows (the
// first that need two waves of clusters of 4) 567 / 885; d = 2048, r = 64: 1000 rows 734 / 554, 2000 rows 735 / 1096.
// DLRB200_CLUSTER_STRIPE=256 or 512 overrides the choice.
template <int R, int CS>
int pick_stripe(const CArgs& a, dlrb200_plan* plan_only, double* us) {
    const CLaunch<R, CS, 512> wide(a.smem_optin);
    const int ww = wide.waves(a.M, a.num_sms);
    const double tw = ww ? ww * layer_us(R, 512) * a.L : 1e30;
    if constexpr (CS <= 4) {
        const CLaunch<R, 2 * CS, 256> narrow(a.smem_optin);
        const int wn = narrow.waves(a.M, a.num_sms);
        const double tn = wn ? wn * layer_us(R, 256) * a.L : 1e30;
        int forced = 0;
        if (const char* e = std::getenv("DLRB200_CLUSTER_STRIPE")) forced = std::atoi(e);
        if (forced ? (forced == 256 && wn) : tn < tw) {
            if (us) *us = tn;
            return narrow.run(a, plan_only);
        }
    }
    if (us) *us = tw;
    return wide.run(a, plan_only);
}

// (r, d / 512) pairs that are built
bool combo_ok(int r, int cs) {
    if (!(cs == 1 || cs == 2 || cs == 4 || cs == 8)) return false;
    if (!(r == 32 || r == 64 || r == 128)) return false;
    return r >= 16 * cs;
}

int dispatch(const CArgs& a, int r, dlrb200_plan* plan_only, double* us) {
#define DLR_CASE(RR, CC) \
    if (r == RR && a.d == CC * 512) return pick_stripe<RR, CC>(a, plan_only, us);
    DLR_CASE(32, 1)
    DLR_CASE(32, 2)
    DLR_CASE(64, 1)
    DLR_CASE(64, 2)
    DLR_CASE(64, 4)
    DLR_CASE(128, 1)
    DLR_CASE(128, 2)
    DLR_CASE(128, 4)
    DLR_CASE(128, 8)
#undef DLR_CASE
    return DLRB200_ERR_UNSUPPORTED_SHAPE;
}

// Debug aid: with DLRB200_PROFILE=1 in the environment every CTA writes cycle counts at offset 256 of the workspace.  First
// epilogue thread: wait for z, send, wait for partials, reduce and send s, U epilogue.
constexpr size_t kProfBytes = 256 + size_t(256) * kProfWords * 8;

bool profiling() {
    const char* v = std::getenv("DLRB200_PROFILE");
    return v && *v && *v != '0';
}

}  // namespace

bool cluster_supported(int d, int r, int L) {
    (void)L;
    return d % 512 == 0 && combo_ok(r, d / 512);
}

size_t cluster_workspace_bytes(int, int, int, int) { return profiling() ? kProfBytes : 0; }

int cluster_plan(int M, int d, int r, int L, int num_sms, int smem_optin, dlrb200_plan* plan, double* us) {
    const size_t ws = plan->workspace_bytes;
    CArgs a{};
    a.M = M; a.d = d; a.L = L; a.num_sms = num_sms; a.smem_optin = smem_optin;
    const int rc = dispatch(a, r, plan, us);
    plan->workspace_bytes = ws;
    return rc;
}

int cluster_forward(void* encode_fn_ptr, const void* x, void* y, const void* Vp, const void* Up, int M, int d, int r,
                    int L, float eps, void* workspace, int* status_dev, cudaStream_t stream, int num_sms,
                    int smem_optin, unsigned int spin_limit) {
    unsigned long long* prof = nullptr;
    if (profiling() && workspace) {
        if (cudaMemsetAsync(workspace, 0, kProfBytes, stream) != cudaSuccess) return DLRB200_ERR_CUDA;
        prof = reinterpret_cast<unsigned long long*>(static_cast<uint8_t*>(workspace) + 256);
    }
    const CArgs a{encode_fn_ptr, x, y, Vp, Up, M, d, L, eps, status_dev, stream, num_sms, smem_optin, spin_limit, prof};
    return dispatch(a, r, nullptr, nullptr);
}

}  // namespace dlr
