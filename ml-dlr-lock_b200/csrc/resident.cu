// Small-batch DLR-Net forward, resident clusters: a cluster of CS = d / W CTAs keeps a few token rows (8 per
// "token tile", up to NT tiles) in registers for all L layers, streams the weights past them, and exchanges once or
// twice per layer through distributed shared memory.  Clusters share nothing but the weights (through L2).
//
// CTA `rank` owns columns [W * rank, W * rank + W) of the model width for both contractions of a layer (K-stripe =
// N-stripe, as in kernels/kernels/cuda/cooperative.cu:10-16).  Per layer (dlr_lock/model.py:96-100 on folded weights):
//   V   z_part[r x rows] = V'[:, stripe] . h[stripe]     mma.sync, weights as the 16-row operand; a V warp takes 16 (or
//                                                        twice 16) rows of V' and the whole stripe as K: finished sums
//   X   z = sum over the CTAs, s = silu(z / rms)         in distributed shared memory, st.async, see below
//   U   h[stripe] += U'[stripe, :] . s                   a U warp its own columns; h stays in the accumulator layout in
//                                                        registers (fp32) and turns into the next layer's B fragments
//                                                        with movmatrix
//
// What bounds it: the chain of L dependent layers (d = 1024, one row: about 1500 cycles a layer), and at d >= 4096 also the
// shared-memory port: a layer's 128 KB of weights per CTA go in (TMA) and out (ldmatrix) at 128 bytes per clock, 2048
// cycles.  So whatever a layer does not have to wait for is off the chain: V and U warps are different warps, so that each
// has its weight fragments in registers before the values they meet arrive; the weights are requested by a warp of its
// own; there is one block barrier per layer; waits look at a barrier with one instruction loop (ptx.cuh).  A local step
// costs what its instructions' latencies add up to (LDS 28, ldmatrix 43, shuffle 29, mma.sync 24, block barrier 40,
// a look at a barrier 60 cycles), so every step dropped counts.
//
// The exchange.  One store hop costs 150 to 250 cycles and distributed shared memory moves about 25 bytes per clock and SM
// (measured), so what travels decides the form:
//   BC  (rank 32, one token tile)  every CTA sends its partial z to all CTAs and each adds all of them up: one hop,
//       r x rows x 4 bytes to every peer, plus one more block barrier.  115 us against 136 for RS at d = 1024, 8 rows
//   RS  (everything else)  z's columns are dealt out, r / CS per CTA: the partials go to the owner (hop one), the owner
//       adds them in rank order, applies 1/rms and SiLU and sends its bf16 slice of s to everybody (hop two).  161 us
//       against 184 for BC at d = 2048, 4 rows
// Both are byte-counted st.async on the receiver's mbarrier: no fences.  Sums are fp32 in a fixed order: repeatable.
//
// Operands.  h and s are rounded to bf16 where they meet the weights, as in the striped kernels.  TERMS is the form for calls
// that run in fp32 throughout otherwise (decode_cluster.cu): a value goes into the tensor core as three bf16 terms of 8 bits
// each, which add up to it exactly.  A cluster has two rows there and a token tile eight columns, so the terms (column 4 row +
// term) cost no further mma.sync: what they cost is adding up the columns (one shuffle for two words) and taking h and s
// apart.  Two terms of a row are the two columns a lane holds of an accumulator, the third is in the lane beside it.  Error
// against 64 bits, output rounding included: d = 1024, 64 rows 1.6574e-3, 6e-5 to 9e-5 of the values on the other side of a
// tie, both as decode_cluster.cu (rounded operands: 1.7133e-3, 0.18); d = 2048, 28 rows 1.6673e-3 (1.7225e-3).  Time (us,
// terms / decode_cluster.cu): d = 1024, 8 rows 110 / 294; d = 2048, 28 rows 165 / 406 (a call of the other form with as many
// rows: 6 % and 12 % less).
//
// Measured on a B200 against the best kernel before it (us): d = 1024 (clusters of 4), 1 / 8 / 264 rows: 100 / 110 / 124
// against 281 / 295 / 751; d = 2048 (8), 4 / 64 / 333 rows: 140 / 162 / 390 against 333 / 767 / 886; d = 4096 (16), 1 / 16 /
// 64 rows: 222 / 236 / 357 against 323 / 521 / 1092; d = 5120 (16), 12 / 64 / 112 rows: 648 / 735 / 870 against 828 / 2350 /
// 5555.
//
// All waits are bounded; a wait that gives up records a status word, the CTA leaves its loop at the next block barrier,
// and the cluster leaves together.
#include <atomic>
#include <cstring>

#include "cluster.h"
#include "ptx.cuh"
#include "resident.h"

namespace dlr {

namespace {

struct RParams {
    const __nv_bfloat16* x;
    __nv_bfloat16* y;
    int M, d, L;
    int rows_per_cluster;
    float eps, inv_d;
    int* status;
    int* mirror;                // host copy of the status word, or null
    unsigned int spin_limit;
};

// NU warps own the columns of the stripe (U contraction, activations, exchange), NVW warps the rows of V'.
// TERMS: the form with operands of 24 bits (see the top of the file).
template <int R, int W, int NU, int NT, bool BC, int CS, bool TERMS>
struct RCfg {
    static constexpr int MT_V = R / 16, MT_U = W / 16;
    static constexpr int NVW = MT_V <= 4 ? MT_V : (R == 128 ? 4 : 8);
    static constexpr int VM = MT_V / NVW;                // 16-row tiles of V' per V warp
    static constexpr int UM = MT_U / NU;                 // 16-column tiles of the stripe per U warp
    static constexpr int KS_V = W / 16, KS_U = R / 16;
    static constexpr bool PREF = NT <= 2 && KS_V <= 16 && UM * KS_U <= 16;   // fragments of U' and of one V' tile fit in registers
    static constexpr int CWARPS = NU + NVW;
    static constexpr int THREADS = 32 * (CWARPS + 1);    // + the producer warp
    static constexpr int MP = 8 * NT;                    // padded rows
    static constexpr int NPAIR = MP / 2;
    static constexpr int KW = R < 64 ? R : 64;           // K columns per U' tile
    static constexpr int V_BOX = R * 128;                // bytes of one V' tile: R rows x 64 columns
    static constexpr int VBOXES = W / 64;                // tiles per layer
    static constexpr int VB = V_BOX * VBOXES <= 32768 ? VBOXES : (V_BOX >= 32768 ? 1 : 32768 / V_BOX);   // tiles per V' stage
    static constexpr int V_STAGE = VB * V_BOX;
    static constexpr int U_STAGE = W * KW * 2;           // one U' tile: W rows x KW columns
    static constexpr int NVS = VBOXES / VB, NUS = R / KW;   // stages per layer
    static constexpr int CH = NT * VM >= 4 ? 1 : 4 / (NT * VM);      // independent accumulators per tile of V' and token tile
    static constexpr int SS = R + 8;                     // bf16 row stride of s
    static constexpr int HB_BYTES = KS_V * NT * 32 * 8;  // bf16 activations as B fragments [ks / 2][nt][lane][ks & 1]
    static constexpr int SB_BYTES = MP * SS * 2;
    // partial sums of squares, [row][warp * 8 + g]; the row stride keeps a warp's stores (4 row pairs x 8) apart
    // (TERMS: two rows, [row][warp * 16 + 2 g + half])
    static constexpr int QN = TERMS ? NU * 16 : (NU * 8 + 31) / 32 * 32;
    static constexpr int QS = QN + 4;
    static constexpr int MAX_ROWS = TERMS ? 2 : MP;      // rows per cluster
    static constexpr int SSP_BYTES = QS * MAX_ROWS * 4;
    // The partitions of z.  RS: owner slices of SW columns, [source][row pair][column][2] with a source stride that is
    // 16 words off a multiple of 32 (two sources are read at once).  BC: [source][tile][token tile][lane][4], TERMS
    // [source][tile][lane].
    static constexpr int SW = R / CS;                    // columns of z per owner (RS)
    static constexpr int SRC_F = BC ? MT_V * NT * (TERMS ? 32 : 128) : NPAIR * SW * 2 + 16;   // floats of one source's block
    static constexpr int RECV_F = (BC ? 2 : 1) * CS * SRC_F;
    static constexpr int FIXED_BYTES = HB_BYTES + SB_BYTES + SSP_BYTES + RECV_F * 4 + 2 * CS * MP * 4 + 1024 /*barriers*/ + 1024 /*alignment*/;
    static_assert(VM <= 2, "tiles of V' per warp");
    static_assert(!TERMS || (NT == 1 && VM == 1 && UM == 2 && PREF && QN % 64 == 0), "a pair of lanes deals out 2 words of z and 4 of dh");
    static_assert(VBOXES % VB == 0 && MT_V % NVW == 0 && MT_U % NU == 0, "whole tiles");
};

constexpr int kMaxRing = 24;

struct RBars {
    uint64_t v_full[kMaxRing], v_empty[kMaxRing];
    uint64_t u_full[kMaxRing], u_empty[kMaxRing];
    uint64_t rbar[2];          // partial z and sums of squares have arrived (bytes); BC: by parity of the layer
    uint64_t sbar;             // RS: s has arrived (bytes)
    int fail[2];               // by parity of the layer: a warp gave up before this layer's block barrier
    int abort_flag;
};
static_assert(sizeof(RBars) <= 1024, "barrier block");

// Sums over two neighbouring lanes, dealt out: the even one gets that of a, the odd one that of b.
__device__ __forceinline__ float pair_deal(float a, float b, bool odd) {
    return (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
}

// What is left of v after its k leading terms of 8 bits each (k < 3): rounded to bf16, term k of v.
__device__ __forceinline__ float after_terms(float v, int k) {
    const float r1 = v - __bfloat162float(__float2bfloat16_rn(v));
    const float r2 = r1 - __bfloat162float(__float2bfloat16_rn(r1));
    return k == 0 ? v : (k == 1 ? r1 : r2);
}

// 8 x 8 transposition of packed 16-bit values across a warp
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(a));
    return r;
}

__device__ __forceinline__ void bar_id(int id, int n) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

template <int R, int W, int NU, int NT, bool BC, int CS, bool TERMS>
__global__ void __launch_bounds__(RCfg<R, W, NU, NT, BC, CS, TERMS>::THREADS, 1)
dlr_resident_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmU, RParams p, int SV, int SU) {
    using C = RCfg<R, W, NU, NT, BC, CS, TERMS>;
    constexpr int SW = C::SW, SRC_F = C::SRC_F, MP = C::MP;
    constexpr int UTHREADS = 32 * NU, ATHREADS = 32 * C::CWARPS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* vring = smem;
    uint8_t* uring = vring + size_t(SV) * C::V_STAGE;
    uint8_t* hb = uring + size_t(SU) * C::U_STAGE;
    uint8_t* sb = hb + C::HB_BYTES;
    float* ssp = reinterpret_cast<float*>(sb + C::SB_BYTES);
    float* recv = ssp + C::SSP_BYTES / 4;
    float* recvq = recv + C::RECV_F;                   // [2][source][row]
    RBars* bars = reinterpret_cast<RBars*>(recvq + 2 * CS * MP);
    volatile int* abort_flag = &bars->abort_flag;
    volatile int* fail = bars->fail;

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;             // position in an mma fragment
    const uint32_t rank = cluster_ctarank();
    const int stripe0 = int(rank) * W;
    const int row0 = (int(blockIdx.x) / CS) * p.rows_per_cluster;
    const int rows = (p.M - row0) < p.rows_per_cluster ? (p.M - row0) : p.rows_per_cluster;
    const int pairs = (rows + 1) >> 1;
    const uint32_t vring_s = smem_u32(vring), uring_s = smem_u32(uring), sb_s = smem_u32(sb), recv_s = smem_u32(recv), recvq_s = smem_u32(recvq);

    if (tid == 0) {
        for (int s = 0; s < SV; ++s) {
            mbar_init(smem_u32(&bars->v_full[s]), 1);
            mbar_init(smem_u32(&bars->v_empty[s]), C::NVW);
        }
        for (int s = 0; s < SU; ++s) {
            mbar_init(smem_u32(&bars->u_full[s]), 1);
            mbar_init(smem_u32(&bars->u_empty[s]), NU);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bars->rbar[b]), 1);
        }
        mbar_init(smem_u32(&bars->sbar), 1);
        fail[0] = fail[1] = 0;
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmU);
    }
    // operand rows past the batch never receive s; sums of squares of warps there are not
    for (int i = tid; i < C::SSP_BYTES / 4; i += C::THREADS) ssp[i] = 0.f;
    for (int i = tid; i < C::SB_BYTES / 4; i += C::THREADS) reinterpret_cast<uint32_t*>(sb)[i] = 0u;
    if constexpr (TERMS)                                     // (columns 6 and 7 of the token tile)
        for (int i = tid; i < C::HB_BYTES / 4; i += C::THREADS) reinterpret_cast<uint32_t*>(hb)[i] = 0u;
    __syncthreads();
    // the peers' barriers must exist before anyone sends to them
    cluster_arrive_release();
    cluster_wait_acquire();

    int err = 0;               // why this warp gave up
    const uint32_t flag_s = smem_u32(&bars->abort_flag);
    auto wait_for = [&](uint32_t bar, uint32_t parity, int code, bool remote) {          // whole warps
        const bool ok = remote ? mbar_wait_warp_cluster(bar, parity, flag_s, p.spin_limit) : mbar_wait_warp(bar, parity, flag_s, p.spin_limit);
        err = ok ? err : code;
    };
    auto wait_free = [&](uint64_t& bar, uint32_t parity) {                               // the producer's lane
        if (!mbar_wait_lane(smem_u32(&bar), parity, flag_s, p.spin_limit)) err = DLRB200_ERR_TIMEOUT_COPY;
        return err == 0;
    };

    // ---- weight rings: one thread asks for the tiles, in the order they are used
    RingPos vq, uq;            // producer's positions
    int vl = 0, vi = 0, ul = 0, ui = 0;                 // layer and stage in it asked for next
    auto ask_v = [&]() {
        if (vl >= p.L) return;
        if (!wait_free(bars->v_empty[vq.st], vq.ph ^ 1u)) return;
        const uint32_t bar = smem_u32(&bars->v_full[vq.st]), dst = vring_s + vq.st * C::V_STAGE;
        mbar_arrive_expect_tx(bar, C::V_STAGE);
#pragma unroll
        for (int b = 0; b < C::VB; ++b)
            tma_load_2d(dst + uint32_t(b) * C::V_BOX, &tmV, stripe0 + 64 * (vi * C::VB + b), vl * R, bar);
        vq.step(uint32_t(SV));
        if (++vi == C::NVS) { vi = 0; ++vl; }
    };
    auto ask_u = [&]() {
        if (ul >= p.L) return;
        if (!wait_free(bars->u_empty[uq.st], uq.ph ^ 1u)) return;
        const uint32_t bar = smem_u32(&bars->u_full[uq.st]), dst = uring_s + uq.st * C::U_STAGE;
        mbar_arrive_expect_tx(bar, C::U_STAGE);
        constexpr int UBR = W > 256 ? W / 2 : W;        // a box has at most 256 rows
#pragma unroll
        for (int b = 0; b < W / UBR; ++b)
            tma_load_2d(dst + uint32_t(b) * (UBR * C::KW * 2), &tmU, ui * C::KW, ul * p.d + stripe0 + b * UBR, bar);
        uq.step(uint32_t(SU));
        if (++ui == C::NUS) { ui = 0; ++ul; }
    };
    // copies already asked for still land in this CTA's shared memory: wait for the last one of every stage
    auto drain_copies = [&]() {
        int nv = vl * C::NVS + vi, nu = ul * C::NUS + ui;
        for (int k = 0; k < SV && nv > 0; ++k) { --nv; mbar_wait(smem_u32(&bars->v_full[nv % SV]), uint32_t(nv / SV) & 1u, kDrainPolls); }
        for (int k = 0; k < SU && nu > 0; ++k) { --nu; mbar_wait(smem_u32(&bars->u_full[nu % SU]), uint32_t(nu / SU) & 1u, kDrainPolls); }
    };
    // a layer's block barrier; says whether a warp had given up before it
    auto layer_barrier = [&](int l) -> bool {
        if (err) { fail[l & 1] = 1; *abort_flag = 1; }
        bar_id(1, ATHREADS);
        return fail[l & 1] != 0;
    };
    const uint32_t a_row = uint32_t((lane & 7) + ((lane >> 3) & 1) * 8), a_col = uint32_t(lane >> 4) * 16u;   // ldmatrix addresses

    int l = 0;
    if (warp >= NU && warp < C::CWARPS) {
        // =============================== V warps ====================================
        const int vw = warp - NU;
        RingPos rp, rq;
        uint32_t voff[4];                                // k step k % 4 of a tile
#pragma unroll
        for (int k = 0; k < 4; ++k) voff[k] = (16u * uint32_t(vw) + a_row) * 128u + ((uint32_t(k) * 32u + a_col) ^ ((a_row & 7u) << 4));
        // (TERMS: the fragments of the second row's columns lie two by two the other way round, so that the stores of a
        // column of both rows go to different banks)
        const int hb_lane = TERMS ? lane ^ ((lane >> 4) << 2) : lane;
        uint32_t va[C::PREF ? C::KS_V : 1][4];
        auto stage_done = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->v_empty[rp.st]));
            rp.step(uint32_t(SV));
        };
        auto prefetch_v = [&]() {
            if constexpr (C::PREF) {
#pragma unroll
                for (int s = 0; s < C::NVS; ++s) {
                    RingPos& at = C::VM == 1 ? rp : rq;      // (with more tiles per warp the stage is released after the layer)
                    wait_for(smem_u32(&bars->v_full[at.st]), at.ph, DLRB200_ERR_TIMEOUT_COPY, false);
                    __syncwarp();
                    const uint32_t base = vring_s + at.st * C::V_STAGE;
#pragma unroll
                    for (int k = 0; k < 4 * C::VB; ++k) {
                        constexpr int KS = C::PREF ? C::KS_V : 1;
                        uint32_t(&a)[4] = va[(4 * C::VB * s + k) % KS];
                        ldmatrix_x4(base + voff[k % 4] + uint32_t(k / 4) * C::V_BOX, a[0], a[1], a[2], a[3]);
                    }
                    if constexpr (C::VM == 1) stage_done();
                    else rq.step(uint32_t(SV));
                }
            }
        };
        // where this warp's partial z goes: BC the same block in every CTA, RS the owners of its two halves
        uint32_t peer_recv[BC ? CS : 2 * C::VM], peer_bar[BC ? CS : 2 * C::VM];
        if constexpr (BC) {
            const int word = TERMS ? vw * 32 + lane : (vw * NT * 32 + lane) * 4;
#pragma unroll
            for (int k = 0; k < CS; ++k) {
                peer_recv[k] = mapa(recv_s + uint32_t(int(rank) * SRC_F + word) * 4u, uint32_t(k));
                peer_bar[k] = mapa(smem_u32(&bars->rbar[0]), uint32_t(k));
            }
        } else if constexpr (TERMS) {
            const int col = 16 * vw + 8 * (t & 1) + g;
            peer_recv[0] = mapa(recv_s + uint32_t(int(rank) * SRC_F + (col % SW) * 2 + (t >> 1)) * 4u, uint32_t(col / SW));
            peer_bar[0] = mapa(smem_u32(&bars->rbar[0]), uint32_t(col / SW));
        } else {
#pragma unroll
            for (int i = 0; i < 2 * C::VM; ++i) {
                const int col = 16 * (vw + C::NVW * (i / 2)) + 8 * (i & 1) + g;
                peer_recv[i] = mapa(recv_s + uint32_t(int(rank) * SRC_F + (t * SW + col % SW) * 2) * 4u, uint32_t(col / SW));
                peer_bar[i] = mapa(smem_u32(&bars->rbar[0]), uint32_t(col / SW));
            }
        }
        prefetch_v();
#pragma unroll 1
        for (l = 0; l < p.L; ++l) {
            const uint32_t par = BC ? uint32_t(l & 1) : 0u;
            const bool stop = layer_barrier(l);
            float zc[C::VM][NT][C::CH][4];
#pragma unroll
            for (int a = 0; a < C::VM; ++a)
#pragma unroll
                for (int b = 0; b < NT; ++b)
#pragma unroll
                    for (int c = 0; c < C::CH; ++c) zc[a][b][c][0] = zc[a][b][c][1] = zc[a][b][c][2] = zc[a][b][c][3] = 0.f;
            if constexpr (C::PREF) {
                // The stages have landed (the first tile of V' is in registers).  A second tile is fetched one pair of K
                // steps ahead of its use: loaded when it is needed, every step would cost the load's latency.
                uint32_t c[C::VM > 1 ? 2 : 1][2][4];
                uint32_t bases[C::NVS];
                {
                    RingPos at = rp;
#pragma unroll
                    for (int s = 0; s < C::NVS; ++s, at.step(uint32_t(SV))) bases[s] = vring_s + at.st * C::V_STAGE;
                }
                auto fetch = [&](int k2) {
                    if constexpr (C::VM > 1) {
                        const int kk = k2 % (2 * C::VB);
                        const uint32_t at = bases[k2 / (2 * C::VB)] + uint32_t(kk / 2) * C::V_BOX + uint32_t(C::NVW) * 2048u;
                        uint32_t(&c0)[4] = c[k2 & 1][0];
                        uint32_t(&c1)[4] = c[k2 & 1][1];
                        ldmatrix_x4(at + voff[(2 * kk) % 4], c0[0], c0[1], c0[2], c0[3]);
                        ldmatrix_x4(at + voff[(2 * kk + 1) % 4], c1[0], c1[1], c1[2], c1[3]);
                    }
                };
                fetch(0);
#pragma unroll
                for (int k2 = 0; k2 < C::KS_V / 2; ++k2) {
                    constexpr int KS = C::PREF ? C::KS_V : 1;
                    const uint32_t(&a0)[4] = va[(2 * k2) % KS];
                    const uint32_t(&a1)[4] = va[(2 * k2 + 1) % KS];
                    if (k2 + 1 < C::KS_V / 2) fetch(k2 + 1);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const uint4 b = *reinterpret_cast<const uint4*>(hb + ((k2 * NT + nt) * 32 + hb_lane) * 16);
                        mma_bf16_16816(zc[0][nt][(2 * k2) % C::CH], a0[0], a0[1], a0[2], a0[3], b.x, b.y);
                        mma_bf16_16816(zc[0][nt][(2 * k2 + 1) % C::CH], a1[0], a1[1], a1[2], a1[3], b.z, b.w);
                        if constexpr (C::VM > 1) {
                            const uint32_t(&c0)[4] = c[k2 & 1][0];
                            const uint32_t(&c1)[4] = c[k2 & 1][1];
                            mma_bf16_16816(zc[1][nt][(2 * k2) % C::CH], c0[0], c0[1], c0[2], c0[3], b.x, b.y);
                            mma_bf16_16816(zc[1][nt][(2 * k2 + 1) % C::CH], c1[0], c1[1], c1[2], c1[3], b.z, b.w);
                        }
                    }
                }
                if constexpr (C::VM > 1)
                    for (int s = 0; s < C::NVS; ++s) stage_done();
            } else {
#pragma unroll 1
                for (int s = 0; s < C::NVS; ++s) {
                    wait_for(smem_u32(&bars->v_full[rp.st]), rp.ph, DLRB200_ERR_TIMEOUT_COPY, false);
                    __syncwarp();
                    const uint32_t base = vring_s + rp.st * C::V_STAGE;
#pragma unroll
                    for (int k2 = 0; k2 < 2 * C::VB; ++k2) {
                        uint4 b[NT];
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
                            b[nt] = *reinterpret_cast<const uint4*>(hb + (((2 * C::VB * s + k2) * NT + nt) * 32 + lane) * 16);
#pragma unroll
                        for (int vm = 0; vm < C::VM; ++vm) {
                            uint32_t a0[4], a1[4];
                            const uint32_t at = base + uint32_t(k2 / 2) * C::V_BOX + uint32_t(vm * C::NVW) * 2048u;
                            ldmatrix_x4(at + voff[(2 * k2) % 4], a0[0], a0[1], a0[2], a0[3]);
                            ldmatrix_x4(at + voff[(2 * k2 + 1) % 4], a1[0], a1[1], a1[2], a1[3]);
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) {
                                mma_bf16_16816(zc[vm][nt][(2 * k2) % C::CH], a0[0], a0[1], a0[2], a0[3], b[nt].x, b[nt].y);
                                mma_bf16_16816(zc[vm][nt][(2 * k2 + 1) % C::CH], a1[0], a1[1], a1[2], a1[3], b[nt].z, b[nt].w);
                            }
                        }
                    }
                    stage_done();
                }
            }
            if constexpr (C::PREF && R >= 128) asm volatile("barrier.cta.arrive 3, %0;" ::"n"(ATHREADS) : "memory");
            // ---- hop one: z columns 16 mt + g (+8), rows 8 nt + 2t, + 1
#pragma unroll
            for (int vm = 0; vm < C::VM; ++vm)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float z[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        z[c] = zc[vm][nt][0][c];
#pragma unroll
                        for (int k = 1; k < C::CH; ++k) z[c] += zc[vm][nt][k][c];
                    }
                    if constexpr (TERMS) {
                        // add up the terms: two in this lane, two in the one beside it; row t / 2, column 8 (t % 2) + g is left
                        const uint32_t word = __float_as_uint(pair_deal(z[0] + z[1], z[2] + z[3], t & 1));
#pragma unroll
                        for (int k = 0; k < (BC ? CS : 1); ++k)
                            st_async_b32(peer_recv[k] + (BC ? par * uint32_t(CS * SRC_F * 4) : 0u), word, peer_bar[k] + (BC ? 8u * par : 0u));
                    } else if (8 * nt + 2 * t < rows) {
                        if constexpr (BC) {
#pragma unroll
                            for (int k = 0; k < CS; ++k)
                                st_async_v4(peer_recv[k] + par * uint32_t(CS * SRC_F * 4) + uint32_t(nt) * 512u, __float_as_uint(z[0]), __float_as_uint(z[1]),
                                            __float_as_uint(z[2]), __float_as_uint(z[3]), peer_bar[k] + 8u * par);
                        } else {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh)
                                st_async_v2(peer_recv[2 * vm + hh] + uint32_t(nt * 4 * SW * 8), __float_as_uint(z[2 * hh]), __float_as_uint(z[2 * hh + 1]),
                                            peer_bar[2 * vm + hh]);
                        }
                    }
                }
            if (stop) break;
            if (l + 1 < p.L) prefetch_v();
        }
    } else if (warp >= C::CWARPS) {
        // =============================== producer warp ==============================
        if (lane == 0) {
            // in the order of use, as far ahead as the rings go
            for (l = 0; l < p.L && !err; ++l) {
                for (int s = 0; s < C::NVS; ++s) ask_v();
                for (int s = 0; s < C::NUS; ++s) ask_u();
            }
            // (whatever the others do: they may give up after this, with copies still on their way)
            drain_copies();
        }
    } else {
        // =============================== U warps ====================================
        // columns stripe0 + 16 u + g (+8), rows 8 nt + 2t, + 1 of this cluster's rows; TERMS: h[i][0][0] only, columns
        // stripe0 + 16 u + 8 (t % 2) + g of row t / 2
        float h[C::UM][NT][4];
        // (read with the input, which takes as long)
        const int failed_before = *reinterpret_cast<volatile int*>(p.status);
        const int row_t = t >> 1, col_t = stripe0 + 32 * warp + 8 * (t & 1) + g;
        if constexpr (TERMS) {
#pragma unroll
            for (int i = 0; i < 2; ++i) h[i][0][0] = row_t < rows ? __bfloat162float(p.x[size_t(row0 + row_t) * p.d + col_t + 16 * i]) : 0.f;
        } else {
#pragma unroll
            for (int i = 0; i < C::UM; ++i)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int row = 8 * nt + 2 * t + (c & 1);
                        const int col = stripe0 + 16 * (warp * C::UM + i) + g + 8 * (c >> 1);
                        h[i][nt][c] = row < rows ? __bfloat162float(p.x[size_t(row0 + row) * p.d + col]) : 0.f;
                    }
        }
        // activations (bf16, as B fragments) and sums of squares for the next layer
        auto publish = [&]() {
            if constexpr (TERMS) {
                float v[2] = {h[0][0][0], h[1][0][0]};
                ssp[row_t * C::QS + warp * 16 + 2 * g + (t & 1)] = v[0] * v[0] + v[1] * v[1];
                // B fragments: K row 16 i + 8 (t % 2) + g of this warp's 32, column 4 row + term of the token tile (see hb_lane)
                uint8_t* at = hb + warp * 512 + (g >> 1) * 16 + 4 * (t & 1) + 2 * (g & 1);
#pragma unroll
                for (int k = 0; k < 3; ++k)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const __nv_bfloat16 b = __float2bfloat16_rn(v[i]);
                        *reinterpret_cast<__nv_bfloat16*>(at + 64 * (row_t ? 4 + (k ^ 1) : k) + 8 * i) = b;
                        v[i] -= __bfloat162float(b);
                    }
            } else {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float q0 = 0.f, q1 = 0.f;
#pragma unroll
                    for (int i = 0; i < C::UM; ++i) {
                        const float* a = h[i][nt];
                        q0 += a[0] * a[0] + a[2] * a[2];
                        q1 += a[1] * a[1] + a[3] * a[3];
                    }
                    ssp[(8 * nt + 2 * t) * C::QS + warp * 8 + g] = q0;
                    ssp[(8 * nt + 2 * t + 1) * C::QS + warp * 8 + g] = q1;
#pragma unroll
                    for (int i = 0; i < C::UM; i += 2) {
                        const int ks = warp * C::UM + i;
                        uint4 b;
                        b.x = movmatrix_trans(pack_bf16x2(h[i][nt][0], h[i][nt][1]));
                        b.y = movmatrix_trans(pack_bf16x2(h[i][nt][2], h[i][nt][3]));
                        if constexpr (C::UM % 2 == 0) {
                            b.z = movmatrix_trans(pack_bf16x2(h[(i + 1) % C::UM][nt][0], h[(i + 1) % C::UM][nt][1]));
                            b.w = movmatrix_trans(pack_bf16x2(h[(i + 1) % C::UM][nt][2], h[(i + 1) % C::UM][nt][3]));
                            *reinterpret_cast<uint4*>(hb + ((ks / 2 * NT + nt) * 32 + lane) * 16) = b;
                        } else {
                            static_assert(C::UM == 1 || C::UM % 2 == 0, "column tiles per warp");
                            *reinterpret_cast<uint2*>(hb + ((ks / 2 * NT + nt) * 32 + lane) * 16 + (ks & 1) * 8) = make_uint2(b.x, b.y);
                        }
                    }
                }
            }
        };
        RingPos rp;
        uint32_t uoff[C::KW / 16];
#pragma unroll
        for (int k = 0; k < C::KW / 16; ++k)
            uoff[k] = (16u * uint32_t(warp * C::UM) + a_row) * (C::KW * 2) +
                      ((uint32_t(k) * 32u + a_col) ^ (C::KW == 64 ? (a_row & 7u) << 4 : ((a_row >> 1) & 3u) << 4));
        uint32_t ua[C::PREF ? C::UM * C::KS_U : 1][4];
        auto stage_done = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->u_empty[rp.st]));
            rp.step(uint32_t(SU));
        };
        const uint32_t sbar_s = smem_u32(&bars->sbar);
        const uint32_t z_bytes = BC ? (TERMS ? uint32_t(CS * R * 8) : uint32_t(CS * C::MT_V * 8 * 16) * uint32_t(pairs)) : uint32_t(CS * SW * 8) * uint32_t(pairs);
        const uint32_t q_dst = mapa(recvq_s + uint32_t(int(rank) * MP) * 4u, uint32_t(lane % CS));      // lane -> peer
        const uint32_t q_bar = mapa(smem_u32(&bars->rbar[0]), uint32_t(lane % CS));
        const uint32_t sb_b = sb_s + uint32_t((lane & 7) * C::SS + (lane >> 3) * 8) * 2u;      // ldmatrix of s
        // RS: lane -> (column of the owner's slice, share of the sources), then -> (row of the pair, two columns, peers)
        constexpr int NPART = BC ? 1 : 32 / SW, PER = CS / NPART;
        const int zl = lane % SW, part = lane / SW;
        uint32_t to_peer[PER];                             // what to add to an address here for the same in a peer
#pragma unroll
        for (int k = 0; k < PER; ++k) to_peer[k] = mapa(sb_s, uint32_t(k * NPART + part)) - sb_s;
        publish();
        // the status word was set before this launch (or by another cluster of it): give up before the first layer, whose block
        // barrier tells the whole CTA
        if (__any_sync(0xffffffffu, failed_before != 0)) err = DLRB200_ERR_TIMEOUT_BARRIER;

#pragma unroll 1
        for (l = 0; l < p.L; ++l) {
            const uint32_t par = BC ? uint32_t(l & 1) : 0u;
            const uint32_t rph = (BC ? uint32_t(l) >> 1 : uint32_t(l)) & 1u;
            const uint32_t rbar_s = smem_u32(&bars->rbar[0]) + 8u * par;
            // activations and sums of squares of all warps are in shared memory after this
            const bool stop = layer_barrier(l);
            // ---- sums of squares: a row per warp, lane -> every eighth 16 bytes of its NU * 8 partial sums, then -> peer
#pragma unroll
            for (int row = warp; row < C::MAX_ROWS; row += NU) {
                if (row < rows) {
                    constexpr int QL = TERMS ? 16 : 8;           // lanes with different words
                    float q = 0.f;
#pragma unroll
                    for (int i = 0; i < C::QN / (4 * QL); ++i) {
                        const float4 f = *reinterpret_cast<const float4*>(ssp + row * C::QS + 4 * QL * i + 4 * (lane % QL));
                        q += (f.x + f.y) + (f.z + f.w);
                    }
#pragma unroll
                    for (int o = 1; o < QL; o <<= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                    if (lane < CS) st_async_b32(q_dst + uint32_t((int(par) * CS * MP + row) * 4), __float_as_uint(q), q_bar + 8u * par);
                }
            }
            if (warp == NU - 1 && lane == 0) {
                mbar_arrive_expect_tx(rbar_s, z_bytes + uint32_t(CS * 4 * rows));
                if (!BC) mbar_arrive_expect_tx(sbar_s, uint32_t(rows * R * 2) * (TERMS ? 3u : 1u));
            }
            __syncwarp();
            // ---- this layer's U' fragments, while the V warps work and the partials travel
            if constexpr (C::PREF) {
                // (wide layers: not before the V warps are done, whose loads would queue behind these in the one port)
                if constexpr (R >= 128) bar_id(3, ATHREADS);
#pragma unroll
                for (int s = 0; s < C::NUS; ++s) {
                    wait_for(smem_u32(&bars->u_full[rp.st]), rp.ph, DLRB200_ERR_TIMEOUT_COPY, false);
                    __syncwarp();
                    const uint32_t base = uring_s + rp.st * C::U_STAGE;
#pragma unroll
                    for (int k = 0; k < C::KW / 16; ++k)
#pragma unroll
                        for (int i = 0; i < C::UM; ++i) {
                            constexpr int NF = C::PREF ? C::UM * C::KS_U : 1;
                            uint32_t(&a)[4] = ua[(i * C::KS_U + s * (C::KW / 16) + k) % NF];
                            ldmatrix_x4(base + uoff[k] + uint32_t(i) * (16 * C::KW * 2), a[0], a[1], a[2], a[3]);
                        }
                    stage_done();
                }
            }
            wait_for(rbar_s, rph, DLRB200_ERR_TIMEOUT_BARRIER, true);
            if constexpr (BC) {
                // ---- every CTA: add up all partials of z; thread -> the same word of every source's block
                static_assert(NT == 1 || !BC, "one token tile");
                // (TERMS: one word of z per lane of a tile, every term of s stored by other warps)
                constexpr int WORDS = SRC_F, ITS = TERMS ? 1 : (WORDS + UTHREADS - 1) / UTHREADS;
                static_assert(!TERMS || (WORDS % 32 == 0 && 3 * WORDS <= UTHREADS), "a thread per word and term");
                const int c = tid & 3, ln = TERMS ? lane : (tid >> 2) & 31;
                const int row = TERMS ? row_t : 2 * (ln & 3) + (c & 1), term = TERMS ? tid / WORDS : 0;
                float q = 0.f;
#pragma unroll
                for (int k = 0; k < CS; ++k) q += recvq[(int(par) * CS + k) * MP + row];
                const float rstd = rsqrtf(q * p.inv_d + p.eps);
#pragma unroll
                for (int it = 0; it < ITS; ++it) {
                    const int e = TERMS ? tid % WORDS : tid + it * UTHREADS;
                    if (row < rows && (TERMS ? term < 3 : e < WORDS)) {
                        float z = 0.f;
#pragma unroll
                        for (int k = 0; k < CS; ++k) z += recv[(int(par) * CS + k) * SRC_F + e];
                        const float s = silu_f(z * rstd);
                        if constexpr (TERMS)
                            reinterpret_cast<__nv_bfloat16*>(sb)[(4 * row + term) * C::SS + 16 * (e >> 5) + 8 * (t & 1) + g] = __float2bfloat16_rn(after_terms(s, term));
                        else
                            reinterpret_cast<__nv_bfloat16*>(sb)[row * C::SS + 16 * (e >> 7) + (ln >> 2) + 8 * (c >> 1)] = __float2bfloat16_rn(s);
                    }
                }
                bar_id(2, UTHREADS);                         // s is complete
            } else {
                // ---- owner: SW columns of z, one row pair per warp
                static_assert(BC || SW == 8 || SW == 16, "owner slices");
                float rstd[(C::NPAIR + NU - 1) / NU][2];
#pragma unroll
                for (int it = 0; it * NU < C::NPAIR; ++it) {
                    const int pr = it * NU + (NU - 1 - warp);      // (the first warps have a row's sum of squares to do)
                    float q0 = 0.f, q1 = 0.f;
                    if (pr < pairs)
#pragma unroll
                        for (int k = 0; k < CS; ++k) {
                            const float2 qq = *reinterpret_cast<const float2*>(recvq + k * MP + 2 * pr);
                            q0 += qq.x; q1 += qq.y;
                        }
                    rstd[it][0] = rsqrtf(q0 * p.inv_d + p.eps);
                    rstd[it][1] = rsqrtf(q1 * p.inv_d + p.eps);
                }
#pragma unroll
                for (int it = 0; it * NU < C::NPAIR; ++it) {
                    const int pr = it * NU + (NU - 1 - warp);      // (the first warps have a row's sum of squares to do)
                    if (pr < pairs) {
                        float z0 = 0.f, z1 = 0.f;
#pragma unroll
                        for (int k = 0; k < PER; ++k) {
                            const float2 zz = *reinterpret_cast<const float2*>(recv + (k * NPART + part) * SRC_F + (pr * SW + zl) * 2);
                            z0 += zz.x; z1 += zz.y;
                        }
#pragma unroll
                        for (int o = SW; o < 32; o <<= 1) {
                            z0 += __shfl_xor_sync(0xffffffffu, z0, o);
                            z1 += __shfl_xor_sync(0xffffffffu, z1, o);
                        }
                        // two columns of one row per lane: even lanes the first row of the pair, odd lanes the second
                        if constexpr (TERMS) {
                            const float s0 = silu_f(z0 * rstd[it][0]), s1 = silu_f(z1 * rstd[it][1]);
                            const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? s0 : s1, 1);
                            float a = (lane & 1) ? other : s0, b = (lane & 1) ? s1 : other;
                            if ((lane & 1) < rows) {
                                const uint32_t dst = sb_s + uint32_t((lane & 1) * 4 * C::SS + int(rank) * SW + (zl & ~1)) * 2u;
#pragma unroll
                                for (int term = 0; term < 3; ++term) {
                                    const uint32_t v = pack_bf16x2(a, b);
                                    a -= bf16lo_to_f(v);
                                    b -= bf16hi_to_f(v);
#pragma unroll
                                    for (int k = 0; k < PER; ++k)
                                        st_async_b32(dst + uint32_t(term * C::SS) * 2u + to_peer[k], v, sbar_s + to_peer[k]);
                                }
                            }
                            continue;
                        }
                        const uint32_t mine = pack_bf16x2(silu_f(z0 * rstd[it][0]), silu_f(z1 * rstd[it][1]));
                        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
                        const uint32_t v = (lane & 1) ? __byte_perm(other, mine, 0x7632) : __byte_perm(mine, other, 0x5410);
                        const int row = 2 * pr + (lane & 1);
                        // ---- hop two: s to everybody
                        if (row < rows) {
                            const uint32_t dst = sb_s + uint32_t(row * C::SS + int(rank) * SW + (zl & ~1)) * 2u;
#pragma unroll
                            for (int k = 0; k < PER; ++k)
                                st_async_b32(dst + to_peer[k], v, sbar_s + to_peer[k]);
                        }
                    }
                }
                wait_for(sbar_s, uint32_t(l) & 1u, DLRB200_ERR_TIMEOUT_BARRIER, true);
            }

            // ---- U: this warp's columns of h
            constexpr int UCH = C::PREF ? 2 : 1;
            float uc[C::UM][NT][UCH][4];
#pragma unroll
            for (int i = 0; i < C::UM; ++i)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int k = 0; k < UCH; ++k) uc[i][nt][k][0] = uc[i][nt][k][1] = uc[i][nt][k][2] = uc[i][nt][k][3] = 0.f;
            if constexpr (C::PREF) {
#pragma unroll
                for (int k2 = 0; k2 < C::KS_U / 2; ++k2)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        constexpr int NF = C::PREF ? C::UM * C::KS_U : 1;
                        uint32_t b[4];
                        ldmatrix_x4(sb_b + uint32_t(8 * nt * C::SS + 32 * k2) * 2u, b[0], b[1], b[2], b[3]);
#pragma unroll
                        for (int i = 0; i < C::UM; ++i) {
                            const uint32_t(&a0)[4] = ua[(i * C::KS_U + 2 * k2) % NF];
                            const uint32_t(&a1)[4] = ua[(i * C::KS_U + 2 * k2 + 1) % NF];
                            mma_bf16_16816(uc[i][nt][0], a0[0], a0[1], a0[2], a0[3], b[0], b[1]);
                            mma_bf16_16816(uc[i][nt][UCH - 1], a1[0], a1[1], a1[2], a1[3], b[2], b[3]);
                        }
                    }
            } else {
#pragma unroll 1
                for (int s = 0; s < C::NUS; ++s) {
                    wait_for(smem_u32(&bars->u_full[rp.st]), rp.ph, DLRB200_ERR_TIMEOUT_COPY, false);
                    __syncwarp();
                    const uint32_t base = uring_s + rp.st * C::U_STAGE;
#pragma unroll
                    for (int k2 = 0; k2 < C::KW / 32; ++k2) {
                        uint32_t a[C::UM][2][4];
#pragma unroll
                        for (int i = 0; i < C::UM; ++i)
#pragma unroll
                            for (int k = 0; k < 2; ++k)
                                ldmatrix_x4(base + uoff[2 * k2 + k] + uint32_t(i) * (16 * C::KW * 2), a[i][k][0], a[i][k][1], a[i][k][2], a[i][k][3]);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            uint32_t b[4];
                            ldmatrix_x4(sb_b + uint32_t(8 * nt * C::SS + s * C::KW + 32 * k2) * 2u, b[0], b[1], b[2], b[3]);
#pragma unroll
                            for (int i = 0; i < C::UM; ++i) {
                                mma_bf16_16816(uc[i][nt][0], a[i][0][0], a[i][0][1], a[i][0][2], a[i][0][3], b[0], b[1]);
                                mma_bf16_16816(uc[i][nt][0], a[i][1][0], a[i][1][1], a[i][1][2], a[i][1][3], b[2], b[3]);
                            }
                        }
                    }
                    stage_done();
                }
            }
            if constexpr (TERMS) {
                // add up the terms of dh as those of z
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float dh[2];
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh)
                        dh[hh] = (uc[i][0][0][2 * hh] + uc[i][0][0][2 * hh + 1]) + (uc[i][0][UCH - 1][2 * hh] + uc[i][0][UCH - 1][2 * hh + 1]);
                    h[i][0][0] += pair_deal(dh[0], dh[1], t & 1);
                }
            } else {
#pragma unroll
                for (int i = 0; i < C::UM; ++i)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int c = 0; c < 4; ++c) h[i][nt][c] += UCH == 2 ? uc[i][nt][0][c] + uc[i][nt][UCH - 1][c] : uc[i][nt][0][c];
            }
            if (stop) break;
            if (l + 1 < p.L) publish();
        }
        if (l >= p.L && !err) {
            if constexpr (TERMS) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (row_t < rows) p.y[size_t(row0 + row_t) * p.d + col_t + 16 * i] = __float2bfloat16_rn(h[i][0][0]);
            } else {
#pragma unroll
                for (int i = 0; i < C::UM; ++i)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const int row = 8 * nt + 2 * t + (c & 1);
                            const int col = stripe0 + 16 * (warp * C::UM + i) + g + 8 * (c >> 1);
                            if (row < rows) p.y[size_t(row0 + row) * p.d + col] = __float2bfloat16_rn(h[i][nt][c]);
                        }
            }
        }
    }
    if (err) {
        *abort_flag = 1;
        report_status(p.status, p.mirror, err | ((l & 0xffff) << 8));
    }
    __syncwarp();
    __syncthreads();
    // no CTA may leave while a peer can still send into its shared memory
    cluster_arrive_release();
    cluster_wait_acquire();
}

struct RArgs {
    void* enc;
    const void* x;
    void* y;
    const void* Vp;
    const void* Up;
    int M, d, L;
    float eps;
    int* status;
    cudaStream_t stream;
    int smem_optin;
    unsigned int spin_limit;
    bool terms;                 // operands of 24 bits
};

// How a call would be cut up: token tiles per cluster, rows per cluster, clusters at once, estimated time.
struct RShape {
    int nt = 0, rows = 0, clusters = 0, waves = 0, stages = 0, cs = 0, w = 0;
    size_t smem = 0;
    double us = 1e30;
};

constexpr int kMaxDevices = 64;

template <int R, int W, int NU, int NT, bool BC, int CS, bool TERMS = false>
struct RLaunch {
    using C = RCfg<R, W, NU, NT, BC, CS, TERMS>;
    int SV = 0, SU = 0, smem = 0;

    // Both rings as deep as fits, alike in layers.  The fragments of a layer are taken before the layer: with prefetching a
    // ring holds a whole layer at least.
    explicit RLaunch(int smem_optin) {
        const int budget = smem_optin - C::FIXED_BYTES;
        for (;;) {
            const bool v_next = (SV + 1) * C::NUS <= (SU + 1) * C::NVS;        // the ring that is behind, in layers
            if (v_next ? SV == kMaxRing : SU == kMaxRing) break;
            if ((SV + (v_next ? 1 : 0)) * C::V_STAGE + (SU + (v_next ? 0 : 1)) * C::U_STAGE > budget) break;
            if (v_next) ++SV; else ++SU;
        }
        if (SV >= (C::PREF ? C::NVS : 1) && SU >= (C::PREF ? C::NUS : 1)) smem = SV * C::V_STAGE + SU * C::U_STAGE + C::FIXED_BYTES;
    }

    void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int clusters, cudaStream_t stream) const {
        memset(&cfg, 0, sizeof(cfg));
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CS;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.blockDim = dim3(C::THREADS);
        cfg.gridDim = dim3(CS * clusters);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }

    // Clusters that can be resident at once on the current device (asked for once per device: the query and the opt-in to
    // large shared memory take longer than a launch), or -1.
    int max_clusters() const {
        static std::atomic<int> known[kMaxDevices];          // 0: not known yet
        int dev = 0;
        if (!smem || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
        int n = known[dev].load(std::memory_order_acquire);
        if (n != 0) return n;
        auto kern = dlr_resident_kernel<R, W, NU, NT, BC, CS, TERMS>;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cfg, attr, 1, nullptr);
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
            (CS > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            return -1;                                       // (not kept: it may have failed for a passing reason)
        }
        known[dev].store(n, std::memory_order_release);
        return n;
    }

    // Rows go to as many clusters as can be resident, two at least (a pair of rows is what the exchange moves): at d = 4096,
    // 16 rows take 237 us on six clusters and 262 us on two.
    void consider(int M, int L, double us_per_layer, RShape& best) const {
        const int mc = max_clusters();
        if (mc < 1) return;
        int rows = (M + mc - 1) / mc;
        rows = rows < 2 ? 2 : (rows + 1) & ~1;
        if (rows > C::MAX_ROWS) rows = C::MAX_ROWS;
        const int clusters = (M + rows - 1) / rows, waves = (clusters + mc - 1) / mc;
        const double us = double(waves) * L * us_per_layer;
        if (us < best.us) {
            best.nt = NT; best.rows = rows; best.clusters = clusters; best.waves = waves; best.us = us;
            best.stages = SV + SU; best.cs = CS; best.w = W; best.smem = size_t(smem);
        }
    }

    int launch(const RArgs& a, const RShape& sh) const {
        if (max_clusters() < 1) return DLRB200_ERR_OCCUPANCY;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cfg, attr, sh.clusters, a.stream);
        RParams p;
        p.x = static_cast<const __nv_bfloat16*>(a.x);
        p.y = static_cast<__nv_bfloat16*>(a.y);
        p.M = a.M; p.d = a.d; p.L = a.L;
        p.rows_per_cluster = sh.rows;
        p.eps = a.eps; p.inv_d = 1.0f / float(a.d);
        p.status = a.status;
        p.mirror = status_mirror(a.status);
        p.spin_limit = a.spin_limit > 8 ? a.spin_limit >> 3 : 1;
        CUtensorMap tmV, tmU;
        if (!encode_2d_bf16(a.enc, &tmV, a.Vp, uint64_t(a.d), uint64_t(a.L) * R, 64, R, 128) ||
            !encode_2d_bf16(a.enc, &tmU, a.Up, uint64_t(R), uint64_t(a.L) * a.d, C::KW, W > 256 ? W / 2 : W, C::KW * 2))
            return DLRB200_ERR_CUDA;
        const cudaError_t ce = cudaLaunchKernelEx(&cfg, dlr_resident_kernel<R, W, NU, NT, BC, CS, TERMS>, tmV, tmU, p, SV, SU);
        return ce == cudaSuccess ? DLRB200_OK : DLRB200_ERR_CUDA;
    }
};

// One shape of net: three kernels (8, 16 or 32 rows per cluster) with their time per layer, microseconds, measured on a
// B200 with every resident cluster at work; and the one with operands of 24 bits (two rows per cluster, time tt) where there is
// one.
template <int R, int W, int NU, int CS, bool BC>
int shape_call(const RArgs& a, double t1, double t2, double t4, double tt, RShape& best, bool launch) {
    if (a.terms) {
        if constexpr (R <= 64) {
            const RLaunch<R, W, NU, 1, BC, CS, true> k(a.smem_optin);
            k.consider(a.M, a.L, tt, best);
            if (best.nt == 0) return DLRB200_ERR_UNSUPPORTED_SHAPE;
            return launch ? k.launch(a, best) : DLRB200_OK;
        }
        return DLRB200_ERR_UNSUPPORTED_SHAPE;
    }
    const RLaunch<R, W, NU, 1, BC, CS> k1(a.smem_optin);
    const RLaunch<R, W, NU, 2, false, CS> k2(a.smem_optin);
    const RLaunch<R, W, NU, 4, false, CS> k4(a.smem_optin);
    k1.consider(a.M, a.L, t1, best);
    if (a.M > 8) k2.consider(a.M, a.L, t2, best);
    if (a.M > 16) k4.consider(a.M, a.L, t4, best);
    if (best.nt == 0) return DLRB200_ERR_UNSUPPORTED_SHAPE;
    if (!launch) return DLRB200_OK;
    return best.nt == 1 ? k1.launch(a, best) : (best.nt == 2 ? k2.launch(a, best) : k4.launch(a, best));
}

int dispatch_resident(const RArgs& a, int r, RShape& best, bool launch) {
    if (r == 32 && a.d == 1024) return shape_call<32, 256, 8, 4, true>(a, 0.84, 1.26, 2.19, 0.83, best, launch);
    if (r == 64 && a.d == 2048) return shape_call<64, 256, 8, 8, false>(a, 1.20, 1.82, 2.95, 1.16, best, launch);
    if (r == 128 && a.d == 4096) return shape_call<128, 256, 8, 16, false>(a, 1.80, 2.78, 4.74, 0.0, best, launch);
    if (r == 256 && a.d == 5120) return shape_call<256, 320, 10, 16, false>(a, 4.60, 5.84, 10.9, 0.0, best, launch);
    return DLRB200_ERR_UNSUPPORTED_SHAPE;
}

}  // namespace

bool resident_supported(int d, int r) {
    return (r == 32 && d == 1024) || (r == 64 && d == 2048) || (r == 128 && d == 4096) || (r == 256 && d == 5120);
}

double resident_estimate_us(int M, int d, int r, int L, bool terms, int smem_optin, dlrb200_plan* plan) {
    RArgs a{};
    a.M = M; a.d = d; a.L = L; a.smem_optin = smem_optin; a.terms = terms;
    RShape sh;
    if (dispatch_resident(a, r, sh, false) != DLRB200_OK) return 1e30;
    if (plan) {
        plan->path = DLRB200_PATH_RESIDENT;
        plan->grid = sh.cs * sh.clusters;
        plan->cluster = sh.cs;
        plan->stripe_cols = sh.w;
        plan->rows_per_pass = sh.rows;
        plan->passes = sh.waves;
        plan->stages = sh.stages;
        plan->smem_bytes = sh.smem;
    }
    return sh.us;
}

int resident_forward(void* enc, const void* x, void* y, const void* Vp, const void* Up, int M, int d, int r, int L,
                     float eps, bool terms, int* status_dev, cudaStream_t stream, int smem_optin, unsigned int spin_limit) {
    RArgs a{enc, x, y, Vp, Up, M, d, L, eps, status_dev, stream, smem_optin, spin_limit, terms};
    RShape sh;
    return dispatch_resident(a, r, sh, true);
}

}  // namespace dlr
