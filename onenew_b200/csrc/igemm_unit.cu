// igemm_unit.cu -- the contraction for launches of about one wave: D = A * B^T with ONE work unit per CTA.
//
// The persistent kernel of igemm.cu is built for throughput: a CTA fills an SM (200 KB of shared memory, up to all
// of tensor memory), so the next launch's blocks cannot be placed beside it, its epilogue drains through TMA stores,
// and a K split needs a second kernel.  A launch with few tiles is a chain of latencies instead: wait for the
// previous kernel, first operand load, a few K blocks, drain, retire.  One image of ResNet-50 is 54 such launches
// (6 - 9 us each with the persistent kernel, whose floor by bytes is 0.2 - 0.7 us).  Here:
//   * 98 KB of shared memory and 64 tensor-memory columns per CTA, two CTAs per SM: the next launch is set up
//     (barriers, tensor memory, table, WEIGHT tiles already on their way) while this one still runs;
//   * a K split is a cluster of 2, 4 or 8 CTAs: every CTA writes each slice of its partial tile into the shared memory of
//     the CTA that finishes that slice, which adds the slices in rank order -- no scratch planes, no second kernel, one
//     bulk copy per slice and peer, the same sums whatever the scheduling;
//   * the epilogue runs on all eight warps and writes whole row pieces with plain stores; its form is a template
//     parameter, because in a launch that runs every instruction once, time follows the code that has to be fetched;
//   * fp32 operands of the drop-in calls are read where they lie and rounded to tf32 in shared memory (`raw`), which
//     saves the packing kernels and their passes over memory.
// Replaces, in the reference, the same code as igemm.cu does (device/x86/Conv/conv.c:300-415, Gemm/gemm.c:9-79,
// MatMul/mat_mul.c:10-101).
#include "igemm_unit.cuh"

#include <cuda_bf16.h>
#include <string.h>

#include <atomic>

#include "act.cuh"
#include "ctx.h"
#include "h16.cuh"
#include "launch.cuh"
#include "round_tf32.cuh"
#include "sm100_prims.cuh"

namespace one {

namespace {

constexpr int BN = UNIT_BN;
constexpr int THREADS = 256;
constexpr int A_ROWS = 128;
constexpr uint32_t PATCH = 32 * 128;   // a 32 x 32 block of fp32 / int32 partial sums
constexpr int NBLK = 4 * BN / 32;      // such blocks in a tile: one per warp
static_assert(NBLK == THREADS / 32, "one block per warp");
// Forms of the epilogue: row-major fp32 / 16-bit / quantised int8 in aligned groups of four columns, or fp32 of any shape
enum { EPI_F32 = 0, EPI_16 = 1, EPI_S8 = 2, EPI_ANY = 3 };

// Bulk copy from this CTA's shared memory to a peer's; `dst` and `bar` are cluster-window addresses in the peer.
__device__ __forceinline__ void bulk_to_peer(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Two fp32 sums in one instruction (each rounded to nearest, as the scalar add).
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) { return (uint64_t)lo | ((uint64_t)hi << 32); }
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ float cvt_tf32(float v)   // nearest, ties away: the value round_to_tf32 gives (one instruction instead of four)
{
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}
template <int KIND> __device__ __forceinline__ uint32_t add_partial(uint32_t a, uint32_t b)
{
    if constexpr (KIND == KIND_I8) return a + b;
    else return __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
}
// The activations other than ReLU and the table, out of line (see the note on code size above).
__device__ __noinline__ float rare_act(float v, int act, float p0, float p1) { return apply_act(v, act, p0, p1, nullptr); }
// N accumulator cells to activated values, in the reference's order of operations.
template <int KIND, int N>
__device__ __forceinline__ void finish(float (&t)[N], const uint32_t (&raw)[N], const float (&b)[N], const float (&k)[N], const IgemmParams &p, const float *slut)
{
#pragma unroll
    for (int e = 0; e < N; ++e) {
        if constexpr (KIND == KIND_I8) t[e] = __fmul_rn(__fadd_rn(__fmul_rn(__int2float_rn((int)raw[e]), p.in_scale), b[e]), k[e]);
        else t[e] = __fadd_rn(__uint_as_float(raw[e]), b[e]);
    }
    if (p.act == 1) {
#pragma unroll
        for (int e = 0; e < N; ++e) t[e] = t[e] > 0.f ? t[e] : 0.f;
    } else if (p.act == 3) {
#pragma unroll
        for (int e = 0; e < N; ++e) t[e] = silu_table(t[e], slut);
    } else if (p.act != 0) {
#pragma unroll
        for (int e = 0; e < N; ++e) t[e] = rare_act(t[e], p.act, p.act_p0, p.act_p1);
    }
}

}  // namespace

// Operand ring, which the finished tile's 32 KB pass through afterwards (every MMA has completed by then), and beside it
// the 32 KB a cluster's slices arrive in (peers write there while this CTA may still be multiplying).
__host__ __device__ constexpr uint32_t unit_ring_bytes(int stages, int slab_bytes, int splits)
{
    const uint32_t ring = (uint32_t)stages * (A_ROWS + BN) * (uint32_t)slab_bytes, room = ring < NBLK * PATCH ? NBLK * PATCH : ring;
    return splits > 1 ? room + NBLK * PATCH : room;
}
static size_t unit_smem_bytes(int stages, int slab_bytes, int splits, bool lut)
{
    return unit_ring_bytes(stages, slab_bytes, splits) + (lut ? 8192 * 4 : 0) + 256 /* barriers */ + 1024 /* alignment */;
}

// RAW: the fp32 operands of a drop-in call, rounded by warps 2 - 7 on their way to the tensor core.
template <int KIND, bool RAW, int EPI, int S>
__global__ void __launch_bounds__(THREADS, 2)
unit_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const IgemmParams p, const UnitParams u, const int stages)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t a_slab = A_ROWS * (uint32_t)p.slab_bytes, b_slab = BN * (uint32_t)p.slab_bytes, stage_bytes = a_slab + b_slab;
    const uint32_t ring = unit_ring_bytes(stages, p.slab_bytes, S);
    const bool has_lut = p.act == 3;
    float *slut = reinterpret_cast<float *>(smem + ring);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + ring + (has_lut ? 8192 * 4 : 0));
    // barriers: full[4], empty[4], ready[4] (operands rounded), acc, slices of a cluster
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * UNIT_MAX_STAGES + 2);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + UNIT_MAX_STAGES), ready0 = smem_u32(bars + 2 * UNIT_MAX_STAGES);
    const uint32_t acc_bar = smem_u32(bars + 3 * UNIT_MAX_STAGES), slice_bar = acc_bar + 8;
    const uint32_t sbase = smem_u32(smem);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = S > 1 ? (int)(blockIdx.x % (unsigned)S) : 0;      // a cluster's CTAs are consecutive
    const int tile = (int)(blockIdx.x / (unsigned)S);
    const int n_tiles = (p.N + BN - 1) / BN, m_tiles = (p.M + A_ROWS - 1) / A_ROWS;
    const int bz = tile / (n_tiles * m_tiles), tin = tile - bz * n_tiles * m_tiles;
    const int m0 = (tin / n_tiles) * A_ROWS, n0 = (tin % n_tiles) * BN;
    const int kb0 = (int)((long long)p.num_kb * rank / S), kb1 = (int)((long long)p.num_kb * (rank + 1) / S);   // never empty: S <= num_kb
    const int nkb = kb1 - kb0;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        if (!RAW || u.a_ld == 0) tma_prefetch_desc(&tmA);
        if (!RAW || u.b_ld == 0) tma_prefetch_desc(&tmB);
        for (int s = 0; s < stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
            if (RAW) mbar_init(ready0 + 8 * s, 6);   // one arrival per rounding warp
        }
        mbar_init(acc_bar, 1);
        mbar_init(slice_bar, 1);
        fence_mbar_init();
        // what the cluster will send: this CTA's slice of every block of the tile that lies inside the matrix, from each CTA
        if (S > 1) mbar_arrive_expect_tx(slice_bar, (uint32_t)(min(4, (p.M - m0 + 31) >> 5) * min(BN / 32, (p.N - n0 + 31) >> 5)) * PATCH);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), BN);
        tmem_relinquish();
    }
    if (has_lut)   // staged before the wait: a prepared operator's, or a drop-in call's (see FirstLaunchPlain)
        for (int i = threadIdx.x; i < 2048; i += THREADS) reinterpret_cast<float4 *>(slut)[i] = __ldg(reinterpret_cast<const float4 *>(p.lut) + i);
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // (waited for before the first write to a peer)
    tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
    // The next launch may be placed from here on (this CTA holds its tensor memory, so a successor that needs what is
    // left cannot stand in its way).
    if (p.pdl) pdl_launch_dependents();

    // This lane's place in the epilogue and its per-column constants, loaded before the wait when they are weights (a cold
    // miss costs more than the rest of the epilogue)
    constexpr int PER = 32 / S;                                      // rows of a block this CTA finishes
    constexpr bool ROWS = EPI != EPI_ANY;                            // row-major output, whole 4-column groups, aligned
    const int quarter = warp & 3, c0 = (warp >> 2) * 32;
    const int chunk = lane & 7, rsub = lane >> 3;
    const int col = n0 + c0 + chunk * 4, nvalid = p.N - col;        // this lane's four columns in a row-major output
    const bool f16 = p.out_mode == OUT_F16;
    alignas(16) float cst_[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // Plain loads here and below: what an earlier kernel of the stream may have written is read after the wait, and a read-only
    // load, __ldg, is not ordered by it -- one behind a conditional wait was seen to run ahead of it.
    const float *bias = reinterpret_cast<const float *>(p.bias);
    auto load_constants = [&]() {
        if (ROWS && nvalid > 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (bias) cst_[e] = bias[col + e];
                if (KIND == KIND_I8) cst_[4 + e] = p.coeff[col + e];
            }
        }
    };
    if (u.b_const) load_constants();

    const bool tma_a = !RAW || u.a_ld == 0, tma_b = !RAW || u.b_ld == 0;
    const uint32_t tx = (tma_a ? a_slab : 0u) + (tma_b ? b_slab : 0u);
    int issued = 0;   // stages whose loads were issued
    // The role loops keep ring slot and phase as running values: a division costs a lone warp 100 - 150 clocks, and three of
    // them per K block, not the tensor memory accelerator, set the pace (420 ns a block).
    auto load_b = [&](uint32_t dst, uint32_t bar, int i) {
        if (p.batched) tma_load_3d(dst + a_slab, &tmB, bar, (kb0 + i) * p.slab_elems, n0, bz);
        else tma_load_2d(dst + a_slab, &tmB, bar, (kb0 + i) * p.slab_elems, n0);
    };
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        const int first = nkb < stages ? nkb : stages;
        const bool early_b = u.b_const && tma_b;
        if (tx && lane == 0) {
            for (int i = 0; i < first; ++i) {
                mbar_arrive_expect_tx(full0 + 8 * i, tx);
                if (early_b) load_b(sbase + i * stage_bytes, full0 + 8 * i, i);
            }
        }
        __syncwarp();
        // base pixel of the tile, filter tap and channel slab of this range's first K block (im2col mode)
        int cw = 0, ch = 0, cn = 0, cs = 0, kw = 0, kh = 0;
        if (p.a_im2col) {
            const int hw = p.OH * p.OW;
            cn = m0 / hw;
            const int rem = m0 - cn * hw, oh = rem / p.OW, ow = rem - oh * p.OW;
            cw = ow * p.stride_w - p.pad_l;
            ch = oh * p.stride_h - p.pad_t;
            cs = kb0 % p.c_slabs;
            kw = (kb0 / p.c_slabs) % p.KW;
            kh = (kb0 / p.c_slabs) / p.KW;
        }
        if (p.pdl) pdl_wait();
        uint32_t dst = sbase, bar = full0, phase = 1;   // of the next K block: its slot, the slot's barrier, the phase its `empty` must have passed
        int xa = kb0 * p.slab_elems;
        for (int i = 0; tx && i < nkb; ++i) {
            if (i >= stages) {
                if (!mbar_wait(bar - full0 + empty0, phase, abort_flag)) {
                    if (lane == 0) atomicOr(p.status, ST_TIMEOUT_PRODUCER);
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_arrive_expect_tx(bar, tx);
            }
            if (lane == 0) {
                if (tma_a) {
                    if (p.a_im2col) tma_load_im2col_4d(dst, &tmA, bar, cs * p.slab_elems, cw, ch, cn, (uint16_t)(kw * p.dil_w), (uint16_t)kh);
                    else if (p.batched) tma_load_3d(dst, &tmA, bar, xa, m0, bz);
                    else tma_load_2d(dst, &tmA, bar, xa, m0);
                }
                if (tma_b && !(early_b && i < first)) load_b(dst, bar, i);
            }
            xa += p.slab_elems;
            dst += stage_bytes;
            bar += 8;
            if (bar == full0 + 8 * stages) {
                dst = sbase;
                bar = full0;
                phase ^= 1;
            }
            if (p.a_im2col && ++cs == p.c_slabs) {
                cs = 0;
                if (++kw == p.KW) {
                    kw = 0;
                    ++kh;
                }
            }
            ++issued;
            __syncwarp();
        }
    } else {
        if (p.pdl) pdl_wait();
    }
    if (!u.b_const) load_constants();   // (behind the first loads: ahead of them they cost Gemm 256 x 2048 x 1000 0.3 us of 35)
    if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        const uint32_t idesc = make_idesc<KIND>(A_ROWS, BN) & ((KIND == KIND_BF16 && p.ab_f16) ? ~((7u << 7) | (7u << 10)) : ~0u);
        const int steps = p.slab_bytes >> 5;
        const uint64_t da0 = make_smem_desc(sbase, p.slab_bytes), db0 = make_smem_desc(sbase + a_slab, p.slab_bytes);
        uint32_t slot = 0, phase = 0;
        for (int i = 0; i < nkb; ++i) {
            if (!mbar_wait((RAW ? ready0 : full0) + 8 * slot, phase, abort_flag)) {
                if (lane == 0) atomicOr(p.status, ST_TIMEOUT_MMA);
                ok = false;
                break;
            }
            if (lane == 0) {
                const uint64_t o = (uint64_t)((slot * stage_bytes) >> 4), da = da0 + o, db = db0 + o;
                tc_mma<KIND>(tmem_base, da, db, idesc, (uint32_t)(i != 0));
                if (steps == 4) {
                    tc_mma<KIND>(tmem_base, da + 2, db + 2, idesc, 1u);
                    tc_mma<KIND>(tmem_base, da + 4, db + 4, idesc, 1u);
                    tc_mma<KIND>(tmem_base, da + 6, db + 6, idesc, 1u);
                } else if (steps == 2) {
                    tc_mma<KIND>(tmem_base, da + 2, db + 2, idesc, 1u);
                }
                if (i + 1 == nkb) tc_commit(acc_bar);
                else tc_commit(empty0 + 8 * slot);
            }
            if (++slot == (uint32_t)stages) {
                slot = 0;
                phase ^= 1;
            }
            __syncwarp();
        }
    }
    if constexpr (RAW) {
        if (warp >= 2) {
            // ------------------------------------------------------------ rounding (and plain loads), 192 threads
            // 16-byte pieces of the K-major tiles: piece c of row r lies at c ^ (r & 7) within a 128-byte row (narrower
            // rows: the corresponding swizzle), so an in-place pass needs no addresses but the linear ones.
            const int t = threadIdx.x - 64;
            auto rnd4 = [](uint4 v) {
                return make_uint4(__float_as_uint(round_to_tf32(__uint_as_float(v.x))), __float_as_uint(round_to_tf32(__uint_as_float(v.y))),
                                  __float_as_uint(round_to_tf32(__uint_as_float(v.z))), __float_as_uint(round_to_tf32(__uint_as_float(v.w))));
            };
            const int cpr = p.slab_bytes >> 4;                                     // pieces per row: 2, 4 or 8
            auto slot_of = [&](int r, int c) { return p.slab_bytes == 128 ? c ^ (r & 7) : (p.slab_bytes == 64 ? c ^ ((r >> 1) & 3) : c ^ ((r >> 2) & 1)); };
            auto fetch = [&](const float *base, int mode, long long pitch, int row, int rows, int k) -> uint4 {
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const bool in = row < rows && k + e < u.K;
                    v[e] = in ? *(mode == 2 ? base + (long long)(k + e) * pitch + row : base + (long long)row * pitch + k + e) : 0.f;
                }
                return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
            };
            // A plainly loaded B tile is fetched into registers one K block ahead: its latency runs under the current block.
            // Lanes run along the rows for a [K][rows] operand and along K for K-major rows: coalesced either way.
            constexpr int BPIECES = (BN * 8 + 191) / 192;
            uint4 bnext[BPIECES];
            const int cshift = 31 - __clz(cpr);
            auto piece_b = [&](int j, int &r, int &c) {
                r = u.b_ld == 2 ? j % BN : j >> cshift;
                c = u.b_ld == 2 ? j / BN : j & (cpr - 1);
            };
            auto fetch_b = [&](int i) {
                const float *base = u.b + (long long)bz * u.b_bstride;
#pragma unroll
                for (int q = 0; q < BPIECES; ++q) {
                    int r, c;
                    piece_b(t + 192 * q, r, c);
                    if (t + 192 * q < BN * cpr) bnext[q] = fetch(base, u.b_ld, u.b_pitch, n0 + r, p.N, (kb0 + i) * p.slab_elems + 4 * c);
                }
            };
            if (u.b_ld) fetch_b(0);
            uint32_t s = 0, phase = 0;   // ring slot, and the phase of its `full`
            for (int i = 0; i < nkb && ok; ++i) {
                uint8_t *st = smem + s * stage_bytes;
                const int k0 = (kb0 + i) * p.slab_elems;
                if ((u.a_ld || u.b_ld) && i >= stages && !mbar_wait(empty0 + 8 * s, phase ^ 1, abort_flag)) ok = false;
                if (ok && u.a_ld) {
                    const float *base = u.a + (long long)bz * u.a_bstride;
#pragma unroll 3
                    for (int j = t; j < A_ROWS * cpr; j += 192) {
                        const int r = j >> cshift, c = j & (cpr - 1);
                        *reinterpret_cast<uint4 *>(st + r * p.slab_bytes + (slot_of(r, c) << 4)) = rnd4(fetch(base, 1, u.a_pitch, m0 + r, p.M, k0 + 4 * c));
                    }
                }
                if (ok && u.b_ld) {
#pragma unroll
                    for (int q = 0; q < BPIECES; ++q) {
                        int r, c;
                        piece_b(t + 192 * q, r, c);
                        if (t + 192 * q < BN * cpr) *reinterpret_cast<uint4 *>(st + a_slab + r * p.slab_bytes + (slot_of(r, c) << 4)) = rnd4(bnext[q]);
                    }
                    if (i + 1 < nkb) fetch_b(i + 1);
                }
                if (ok && tx) {
                    if (!mbar_wait(full0 + 8 * s, phase, abort_flag)) ok = false;
                    else {
                        const uint32_t lo = tma_a ? 0u : a_slab, hi = tma_b ? stage_bytes : a_slab;
                        for (uint32_t o = lo + 16u * t; o < hi; o += 4u * 16u * 192u) {   // four pieces in flight
                            uint4 v[4];
#pragma unroll
                            for (uint32_t e = 0; e < 4; ++e)
                                if (o + e * 3072u < hi) v[e] = *reinterpret_cast<uint4 *>(st + o + e * 3072u);
#pragma unroll
                            for (uint32_t e = 0; e < 4; ++e)
                                if (o + e * 3072u < hi) *reinterpret_cast<uint4 *>(st + o + e * 3072u) = rnd4(v[e]);
                        }
                    }
                }
                if (!ok) {
                    if (lane == 0) atomicOr(p.status, ST_TIMEOUT_MMA);
                    break;
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(ready0 + 8 * s);
                if (++s == (uint32_t)stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            __syncwarp();
        }
    }

    // ---------------------------------------------------------------- epilogue: all eight warps, block (quarter, column block) each
    const uint64_t *cst = reinterpret_cast<const uint64_t *>(cst_);
    uint2 res16[8 / S];
    uint4 res32[8 / S];
    const int row_first = m0 + quarter * 32 + rank * PER + rsub;     // first of the rows this lane finishes (every fourth of the CTA's slice)
    const long long off0 = (long long)row_first * p.ldo + col, step = 4 * p.ldo;
    if constexpr (ROWS && EPI != EPI_S8) {
        if (nvalid > 0 && p.residual) {   // on its way while the K blocks are multiplied
#pragma unroll
            for (int i = 0; i < 8 / S; ++i) {
                if (row_first + i * 4 >= p.M) continue;
                if (EPI == EPI_16) res16[i] = *reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(p.residual) + off0 + i * step);
                else res32[i] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint32_t *>(p.residual) + off0 + i * step);
            }
        }
    }
    bool got = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0, abort_flag));
    // Block w of the tile passes through shared memory (the ring is free: every MMA of the tile has completed) as 32 rows
    // of 128 bytes, 16-byte piece c of row x at c ^ (x & 7).  A cluster deals the rows out in S slices, CTA z finishes
    // slice z: each warp sends every slice of its partial block to its owner, [source CTA][block][row of the slice].
    uint8_t *patch = smem + warp * PATCH;
    uint8_t *tbuf = smem + (S > 1 ? ring - NBLK * PATCH : 0u);
    if constexpr (S > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // the peers have started: their shared memory may be written
    const bool inside = m0 + quarter * 32 < p.M && n0 + c0 < p.N;
    if (got && inside) {
        uint32_t r[32];
        tc_fence_after_sync();
        tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) reinterpret_cast<uint4 *>(patch)[lane * 8 + (j ^ (lane & 7))] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        if constexpr (S > 1) {
            fence_proxy_async();
            __syncwarp();
            if (lane < S)
                bulk_to_peer(mapa_shared(smem_u32(tbuf) + (uint32_t)((rank * NBLK + warp) * PER) * 128u, lane), smem_u32(patch) + (uint32_t)(lane * PER) * 128u, PER * 128u,
                             mapa_shared(slice_bar, lane));
        }
    }
    if constexpr (S > 1) {
        got = __all_sync(0xffffffffu, mbar_wait(slice_bar, 0, abort_flag)) && got;
        // Every copy to this CTA has landed.  (Waited for at the end: a CTA stays until its own copies have been read.)
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    } else {
        __syncwarp();
    }
    if (!got && lane == 0) atomicOr(p.status, ST_TIMEOUT_EPILOGUE);
    float vmax = 0.f, vmin = 0.f;   // extremes of what is written as fp16
    if (got && inside) {
        if constexpr (ROWS) {
            if (nvalid > 0) {
                const uint8_t *src = tbuf + (warp * PER + rsub) * 128;
#pragma unroll
                for (int i = 0; i < 8 / S; ++i) {
                    const int rs = i * 4 + rsub, pc = (chunk ^ ((rank * PER + rs) & 7)) << 4;
                    uint64_t t[2];
                    {
                        uint4 raw[S];   // all in flight
#pragma unroll
                        for (int z = 0; z < S; ++z) raw[z] = *reinterpret_cast<const uint4 *>(src + z * (NBLK * PER * 128) + i * 512 + pc);
                        if constexpr (KIND == KIND_I8) {
                            int q[4] = {(int)raw[0].x, (int)raw[0].y, (int)raw[0].z, (int)raw[0].w};
#pragma unroll
                            for (int z = 1; z < S; ++z) { q[0] += (int)raw[z].x; q[1] += (int)raw[z].y; q[2] += (int)raw[z].z; q[3] += (int)raw[z].w; }
                            float f[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) f[e] = __fmul_rn(__fadd_rn(__fmul_rn(__int2float_rn(q[e]), p.in_scale), cst_[e]), cst_[4 + e]);
                            t[0] = pack2(__float_as_uint(f[0]), __float_as_uint(f[1]));
                            t[1] = pack2(__float_as_uint(f[2]), __float_as_uint(f[3]));
                        } else {
                            t[0] = pack2(raw[0].x, raw[0].y);
                            t[1] = pack2(raw[0].z, raw[0].w);
#pragma unroll
                            for (int z = 1; z < S; ++z) { t[0] = add2(t[0], pack2(raw[z].x, raw[z].y)); t[1] = add2(t[1], pack2(raw[z].z, raw[z].w)); }
                            t[0] = add2(t[0], cst[0]);
                            t[1] = add2(t[1], cst[1]);
                        }
                    }
                    float f[4] = {lo2(t[0]), hi2(t[0]), lo2(t[1]), hi2(t[1])};
                    if (p.act == 3) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) f[e] = silu_table(f[e], slut);
                    } else if (p.act > 1) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) f[e] = rare_act(f[e], p.act, p.act_p0, p.act_p1);
                    }
                    const bool has_res = EPI != EPI_S8 && p.residual;
                    const bool relu_last = has_res ? p.res_relu != 0 : p.act == 1;
                    if (has_res) {
                        if (p.act == 1) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) f[e] = fmaxf(f[e], 0.f);
                        }
                        if (EPI == EPI_16) {
                            const float2 lo = h16_unpack2(res16[i].x, f16), hi = h16_unpack2(res16[i].y, f16);
                            f[0] = __fadd_rn(f[0], lo.x); f[1] = __fadd_rn(f[1], lo.y); f[2] = __fadd_rn(f[2], hi.x); f[3] = __fadd_rn(f[3], hi.y);
                        } else {
                            f[0] = __fadd_rn(f[0], __uint_as_float(res32[i].x)); f[1] = __fadd_rn(f[1], __uint_as_float(res32[i].y));
                            f[2] = __fadd_rn(f[2], __uint_as_float(res32[i].z)); f[3] = __fadd_rn(f[3], __uint_as_float(res32[i].w));
                        }
                    }
                    if (relu_last) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) f[e] = fmaxf(f[e], 0.f);   // (a NaN becomes 0, as in v > 0 ? v : 0)
                    }
                    const bool in = row_first + i * 4 < p.M;
                    const long long off = off0 + i * step;
                    if constexpr (EPI == EPI_S8) {
                        uint32_t w = 0;
#pragma unroll
                        for (int e = 0; e < 4; ++e) w |= ((uint32_t)quant_s8(f[e], p.q_inv_scale) & 0xff) << (8 * e);
                        if (in) *reinterpret_cast<uint32_t *>(p.out_q + off) = w;
                    } else if constexpr (EPI == EPI_16) {
                        const uint2 w = f16 ? make_uint2(h16_pack2(f[0], f[1], true), h16_pack2(f[2], f[3], true)) : make_uint2(h16_pack2(f[0], f[1], false), h16_pack2(f[2], f[3], false));
                        if (in) {
                            vmax = fmaxf(fmaxf(vmax, fmaxf(f[0], f[1])), fmaxf(f[2], f[3]));
                            vmin = fminf(fminf(vmin, fminf(f[0], f[1])), fminf(f[2], f[3]));
                            *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(p.out) + off) = w;
                        }
                    } else {
                        if (p.round_tf32) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) f[e] = cvt_tf32(f[e]);
                        }
                        if (in) *reinterpret_cast<float4 *>(reinterpret_cast<float *>(p.out) + off) = make_float4(f[0], f[1], f[2], f[3]);
                    }
                }
            }
        } else {
            // fp32 output of any shape, element by element.  The reference layout of a convolution ([M / hw][N][hw]): lanes
            // run along the rows of the slice, so a store covers consecutive pixels of a channel; a row-major output of
            // ragged width: along the columns.
#pragma unroll 4
            for (int j = 0; j < PER; ++j) {
                const int rs = u.nchw_hw ? lane % PER : j, cc = u.nchw_hw ? j * S + lane / PER : lane;
                const int rr = rank * PER + rs, m = m0 + quarter * 32 + rr, n = n0 + c0 + cc;
                const uint8_t *src = tbuf + (warp * PER + rs) * 128 + (((cc >> 2) ^ (rr & 7)) << 4) + (cc & 3) * 4;
                uint32_t raw[1] = {*reinterpret_cast<const uint32_t *>(src)};
#pragma unroll
                for (int z = 1; z < S; ++z) raw[0] = add_partial<KIND>(raw[0], *reinterpret_cast<const uint32_t *>(src + z * (NBLK * PER * 128)));
                if (m >= p.M || n >= p.N) continue;
                const float b[1] = {bias ? bias[n] : 0.f}, k[1] = {KIND == KIND_I8 ? p.coeff[n] : 0.f};
                float t[1];
                finish<KIND, 1>(t, raw, b, k, p, slut);
                long long off;
                if (u.nchw_hw) {
                    const int img = m / u.nchw_hw;
                    off = ((long long)img * p.N + n) * u.nchw_hw + (m - img * u.nchw_hw);
                } else {
                    off = (long long)bz * p.out_batch_stride + (long long)m * p.ldo + n;
                }
                reinterpret_cast<float *>(p.out)[off] = p.round_tf32 ? cvt_tf32(t[0]) : t[0];
            }
        }
    }
    if (f16 && __any_sync(0xffffffffu, vmax > F16_MAX || vmin < -F16_MAX) && lane == 0) atomicOr(p.status, ST_RANGE_F16);
    if constexpr (S > 1) {
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    // ---------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag && warp == 0) {   // a role gave up: loads in flight must land before the shared memory is given back
        int dummy = 0;
        for (int i = issued > stages ? issued - stages : 0; i < issued; ++i)
            if (!mbar_wait(full0 + 8 * (i % stages), (uint32_t)((i / stages) & 1), &dummy)) {
                if (lane == 0) atomicOr(p.status, ST_TIMEOUT_DRAIN);
                break;
            }
    }
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, BN);
    }
}

template <int KIND, bool RAW, int EPI, int S>
static cudaError_t launch_unit_split(const CUtensorMap &tmA, const CUtensorMap &tmB, IgemmParams p, const UnitParams &u, cudaStream_t stream)
{
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(unit_kernel<KIND, RAW, EPI, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)unit_smem_bytes(UNIT_MAX_STAGES, 128, S, true));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
    }
    const long long tiles = (long long)((p.M + A_ROWS - 1) / A_ROWS) * ((p.N + BN - 1) / BN) * (p.batched ? p.batch : 1);
    if (tiles <= 0 || tiles * S > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const bool lut = p.act == 3;
    const int stages = (lut || S > 1) ? 3 : UNIT_MAX_STAGES;   // two CTAs fit an SM (not with the table AND a cluster's slices)
    p.pdl = get_pdl();
    return launch_ex(unit_kernel<KIND, RAW, EPI, S>, dim3((unsigned)(tiles * S)), dim3(THREADS), unit_smem_bytes(stages, p.slab_bytes, S, lut), stream, p.pdl != 0,
                     S, tmA, tmB, p, u, stages);
}

template <int KIND, bool RAW, int EPI>
static cudaError_t launch_unit_one(const CUtensorMap &tmA, const CUtensorMap &tmB, const IgemmParams &p, const UnitParams &u, cudaStream_t stream)
{
    switch (u.splits) {
    case 1: return launch_unit_split<KIND, RAW, EPI, 1>(tmA, tmB, p, u, stream);
    case 2: return launch_unit_split<KIND, RAW, EPI, 2>(tmA, tmB, p, u, stream);
    case 4: return launch_unit_split<KIND, RAW, EPI, 4>(tmA, tmB, p, u, stream);
    case 8: return launch_unit_split<KIND, RAW, EPI, 8>(tmA, tmB, p, u, stream);
    default: return cudaErrorInvalidValue;
    }
}

int unit_epilogue(int kind, const IgemmParams &p, const UnitParams &u)
{
    if (p.act == 3 && (reinterpret_cast<uintptr_t>(p.lut) & 15)) return -1;
    const bool vec = !p.batched && (p.N % 4) == 0 && (p.ldo % 4) == 0 && !u.nchw_hw &&
                     (((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual) | reinterpret_cast<uintptr_t>(p.out_q)) & 15) == 0);
    if (p.out_q) return (vec && !p.out && !p.residual) ? EPI_S8 : -1;
    if (!p.out) return -1;
    if (out_is_16(p.out_mode)) return (vec && kind != KIND_I8) ? EPI_16 : -1;
    if (p.out_mode != OUT_F32) return -1;
    return vec ? EPI_F32 : (p.residual ? -1 : EPI_ANY);
}

cudaError_t launch_unit(int kind, const CUtensorMap &tmA, const CUtensorMap &tmB, const IgemmParams &p0, const UnitParams &u, cudaStream_t stream)
{
    if (u.splits < 1 || u.splits > p0.num_kb) return cudaErrorInvalidValue;
    if (u.raw && kind != KIND_TF32) return cudaErrorInvalidValue;
    IgemmParams p = p0;
    cudaError_t e;
    if (kind == KIND_F16) p.ab_f16 = 1;
    const int epi = unit_epilogue(kind, p, u);
    if (epi < 0) return cudaErrorInvalidValue;
#define ONE_UNIT(K, R, E) e = launch_unit_one<K, R, E>(tmA, tmB, p, u, stream)
    if (u.raw) {
        if (epi == EPI_F32) ONE_UNIT(KIND_TF32, true, EPI_F32);
        else if (epi == EPI_ANY) ONE_UNIT(KIND_TF32, true, EPI_ANY);
        else return cudaErrorInvalidValue;
    } else if (kind == KIND_TF32) {
        if (epi == EPI_F32) ONE_UNIT(KIND_TF32, false, EPI_F32);
        else if (epi == EPI_16) ONE_UNIT(KIND_TF32, false, EPI_16);
        else if (epi == EPI_S8) ONE_UNIT(KIND_TF32, false, EPI_S8);
        else ONE_UNIT(KIND_TF32, false, EPI_ANY);
    } else if (kind == KIND_I8) {
        if (epi == EPI_S8) ONE_UNIT(KIND_I8, false, EPI_S8);
        else if (epi == EPI_F32) ONE_UNIT(KIND_I8, false, EPI_F32);
        else ONE_UNIT(KIND_I8, false, EPI_ANY);
    } else {
        if (epi == EPI_16) ONE_UNIT(KIND_BF16, false, EPI_16);
        else if (epi == EPI_F32) ONE_UNIT(KIND_BF16, false, EPI_F32);
        else if (epi == EPI_S8) ONE_UNIT(KIND_BF16, false, EPI_S8);
        else ONE_UNIT(KIND_BF16, false, EPI_ANY);
    }
#undef ONE_UNIT
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace one
