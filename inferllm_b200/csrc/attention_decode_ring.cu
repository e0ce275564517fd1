// Attention of single tokens over long paged caches, bfloat16, as a stream: K and V tiles come
// through a ring of shared-memory stages filled by TMA, and the query heads that share a KV head
// are the rows of one warp-level MMA tile.
//
// A block owns one (token, kv head, split).  Its keys are the 64-key tiles  first + split,
// first + split + n_splits, ...  of the token's range, so that the blocks of a token have equal
// work whatever its length is (the grid is sized for the longest sequence the cache allows and
// does not change from step to step).  One thread issues, per tile, cp.async.bulk.tensor loads of
// [64 keys x 64 channels] boxes of K and V straight from the page that holds them (128-byte
// swizzle; a tile never crosses a page because pages are multiples of 64 positions) into a ring of
// 3 (head size 128) or 6 (head size 64) stages, arming a "full" mbarrier per stage with the byte
// count (the last tile comes in boxes of 16 keys, as many as hold a visible key).  Four consumer warps wait for it; warp w takes keys 16w..16w+15 of every tile:
// S = Q K^T with m16n8k16 MMAs (rows = the G query heads, zero rows above), scaling, masking and
// the running softmax in float32, P V again on MMAs, then an arrive on the stage's "empty"
// barrier.  Nothing but the ring is synchronised inside the loop.  At the end the four warps are
// merged through shared memory in ascending order; with one split the block writes the finished
// heads, otherwise a partial (acc, max, sum) per (token, head, split) that a second kernel adds in
// ascending order of the split.  The result never depends on timing.
// Keys outside [p - window + 1, p] get weight exactly 0 and their V rows are cleared in shared
// memory before the product (a page may still hold another sequence's values there).
// In its second form (FUSE, illm_attention_decode_ring_rope) the kernel also does the position
// encoding and the cache write of the step (what rope_kv.cu does, src/kern/naive/naive.cpp:389-414
// and src/core/op.cpp:414-416 in the reference): the consumer warps rotate the query heads on
// their way into shared memory, and in the block that owns the token's last tile a sixth warp makes
// the token's new K row (rotated) and V row, writes them to the cache page and hands them through
// shared memory to the consumer warp that owns their place in that tile.  The TMA thread starts
// at once: it needs neither.
// Two further forms: the query heads of a group beyond 16 over several blocks that walk the same keys (RdExtras::alias), and the two
// maps of a differential head as two rows (DIFF).
// Formulas: src/kern/naive/naive.cpp:576-604 (scores with key head h / G), :531-553 (mask),
// :209-240 (softmax), :634-662 (values); the reference's GPU code loops over the heads with one
// library call each (src/kern/gpu/kernel_gpu.cu:688-756).
// Every wait on an mbarrier is bounded: after the limit the thread raises the error word and
// goes on, so a fault in the pipeline ends the kernel instead of hanging the GPU.
#include <math.h>

#include "tc_common.cuh"

#define RD_BN 64                        // keys per tile
#define RD_CONSUMERS 4
#define RD_THREADS ((RD_CONSUMERS + 1) * 32)
#define RD_MAX_SPLITS 32

namespace {

__device__ __forceinline__ void rd_ldm(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void rd_ldm_t(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void rd_mma(float* c, const unsigned* a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the two bfloat16 of a register as float32
__device__ __forceinline__ float rd_low(unsigned v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float rd_high(unsigned v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ unsigned rd_pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ void rd_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Byte offset of the 16-byte chunk c (8 channels) of key row r inside a K or V tile: boxes of 64
// channels, 8 KB each, rows of 128 bytes, the chunk index XORed with the row (128-byte swizzle).
__device__ __forceinline__ unsigned rd_tile_off(int r, int c) {
    return (unsigned)((c >> 3) * (RD_BN * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4));
}
template <int D> __device__ __forceinline__ int rd_qswz(int r, int c) { return r * D + ((c ^ (r & 7)) << 3); }

}  // namespace

// The position encoding and the cache write done by this kernel itself (FUSE): the packed projection
// [T, (nh + 2 nkv) d] comes unrotated, in bfloat16 or as the float32 K slices of a split matrix
// product, and the kernel does what rope_kv.cu does for one token: it rotates the query heads on
// their way into shared memory, and the block that owns the token's last tile rotates the new K row,
// writes it and the V row to the cache page and puts them into the tile it has just loaded.  The
// arithmetic and the rounding are those of rope_kv.cu.
struct RdRope {
    const float* partials;     // K slices [splits][T][width], or nullptr: the bfloat16 projection is read
    int splits;
    long long split_stride;
    const float2* cs;          // cos/sin table [positions][rot / 2]
    int rot, table_positions;
    bf16* kc;                  // the cache entry, for the write of the new row
    bf16* vc;
    int write_kv;
    int* err;                  // the step's error word: 2 no page, 3 position outside the table
};

// 8 channels (chunk c) of head slot `slot` of token t, position-encoded if the chunk is rotated
template <int D>
__device__ __forceinline__ void rd_encoded_chunk(const RdRope& rp, const bf16* __restrict__ qkv, size_t row_off, int slot,
                                                 int c, int p, float* out) {
    auto fetch = [&](int cc, float* o8) {
        const size_t off = row_off + (size_t)slot * D + cc * 8;
        if (rp.partials) {
#pragma unroll
            for (int k = 0; k < 8; k++) o8[k] = 0.f;
            const float* pz = rp.partials + off;
            int z = 0;
            for (; z + 4 <= rp.splits; z += 4) {          // four slices in flight, added in order
                float p8[4][8];
#pragma unroll
                for (int u = 0; u < 4; u++) load8(pz + (size_t)(z + u) * rp.split_stride, p8[u]);
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int k = 0; k < 8; k++) o8[k] += p8[u][k];
            }
            if (z + 2 <= rp.splits) {
                float p8[2][8];
                load8(pz + (size_t)z * rp.split_stride, p8[0]);
                load8(pz + (size_t)(z + 1) * rp.split_stride, p8[1]);
#pragma unroll
                for (int k = 0; k < 8; k++) o8[k] += p8[0][k];
#pragma unroll
                for (int k = 0; k < 8; k++) o8[k] += p8[1][k];
                z += 2;
            }
            if (z < rp.splits) {
                float p8[8];
                load8(pz + (size_t)z * rp.split_stride, p8);
#pragma unroll
                for (int k = 0; k < 8; k++) o8[k] += p8[k];
            }
        } else {
            load8(qkv + off, o8);
        }
    };
    const int hc = rp.rot >> 4;            // chunks per rotated half
    if (c < 2 * hc) {
        const int cp = c < hc ? c : c - hc;
        float a[8], b[8];
        fetch(cp, a);
        fetch(cp + hc, b);
        const float2* cst = rp.cs + (size_t)p * (rp.rot >> 1) + cp * 8;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 cc = cst[k];
            out[k] = c < hc ? a[k] * cc.x - b[k] * cc.y : a[k] * cc.y + b[k] * cc.x;
        }
    } else {
        fetch(c, out);
    }
}

// What mixers beyond the plain attention add: `sinks` (float32 [nh]: one more term exp(sink) of the
// softmax denominator, without a value), `gate` (float32, gate[t * gate_stride + h]: the head's output
// is multiplied by its sigmoid; with gate_wide gate[t * gate_stride + h * D + c], one per channel), `softcap` (> 0: the scaled
// scores s become softcap * tanh(s / softcap); softcap_x is 2 scale log2(e) / softcap).  TERMS: the softmax weights enter the product with V as so many
// bfloat16 terms (P1 = P rounded, P2 = P - P1 rounded, P3 = P - P1 - P2): 8, 16 or all 24 bits of their mantissa.  With three the
// heads are 9e-8 to 3.4e-7 of their norm from float64 before their last rounding, on CUDA cores in float32 1.3e-7 to 5.9e-7 (with two
// 6.5e-7 to 2.2e-6); 64 tokens of 32 heads at 2,000 keys 105.5 -> 109.6 us for it, one token of 32 heads as before.
// DIFF: differential attention.  A query row holds [q_1, q_2], a key row [k_1, k_2]; row 2 h + m of a block's products is map m of
// query head h, so that one walk over the keys serves both maps.  nh counts maps.
struct RdExtras {
    const float* sinks;
    const float* gate;
    int gate_stride;
    int gate_wide;
    float softcap, softcap_x;
    // alias > 1: every KV head of the cache is walked by so many blocks side by side, each for its own share of the head's query
    // heads (a group beyond the 16 rows of a block's products; the rows come from L2 from the second on).  0 counts as 1.
    int alias;
};

// num / den of a head with the sink's term added (m and the sink in units of log2) and the gate applied
__device__ __forceinline__ float rd_finish(float num, float den, float m, const RdExtras& ex, int t, int h, int d, int c) {
    if (ex.sinks) {
        const float s2 = ex.sinks[h] * 1.4426950408889634f;
        if (s2 <= m) {
            den += exp2f(s2 - m);
        } else {
            const float w = exp2f(m - s2);
            den = den * w + 1.0f;
            num *= w;
        }
    }
    float r = num / den;
    if (ex.gate) r *= 1.0f / (1.0f + expf(-ex.gate[(size_t)t * ex.gate_stride + (ex.gate_wide ? (size_t)h * d + c : h)]));
    return r;
}

// (Two blocks an SM are what the ring leaves room for.  Without that bound the compiler held head size 64 to 96 registers, with a spill in
// the fused form: 8 sequences of 32 heads at 4,000 keys 40.9 us, now 37.2 with 118.)
template <int D, bool FUSE, int TERMS, bool DIFF>
__global__ void __launch_bounds__(RD_THREADS + 32, 2)
attention_decode_ring_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                             const __grid_constant__ CUtensorMap map_k16, const __grid_constant__ CUtensorMap map_v16,
                             const bf16* __restrict__ q, int q_stride, const int* __restrict__ block_table,
                             int max_pages, const int* __restrict__ token_pos, const int* __restrict__ token_seq,
                             float* __restrict__ part_acc, float* __restrict__ part_ml, bf16* __restrict__ out,
                             int n_splits, int nh, int nkv, int G, int page_size, int span, float scale_log2e,
                             int* __restrict__ err, const RdRope rp, const RdExtras ex) {
    constexpr int STAGES = 384 / D;
    constexpr int CH = D / 8, KS = D / 16, NT_D = D / 8;
    constexpr unsigned TILE_BYTES = RD_BN * D * 2;            // a K tile, or a V tile
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * STAGES + 1];
    __shared__ __align__(16) bf16 new_row_s[2 * D];         // FUSE: the token's new K row, then its V row

    const unsigned raw = tc_smem_u32(smem_raw);
    const unsigned base = (raw + 1023u) & ~1023u;             // the swizzle's period
    unsigned char* gbase = smem_raw + (base - raw);
    bf16* Qs = reinterpret_cast<bf16*>(gbase + (size_t)STAGES * 2 * TILE_BYTES);   // [16][D]
    const unsigned full0 = tc_smem_u32(&bars[0]), empty0 = tc_smem_u32(&bars[STAGES]);
    const unsigned row_ready = tc_smem_u32(&bars[2 * STAGES]);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int split = blockIdx.x, hk = blockIdx.y, t = blockIdx.z;
    int p = 0, seq = 0;
    if (FUSE) p = token_pos[t], seq = token_seq[t];           // on their way while the barriers are made
    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, RD_CONSUMERS);
        }
        mbar_init(row_ready, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();          // the barriers exist; from here the warps go their own ways
    // Programmatic dependent launch.  What the step's sequences hold (positions, page tables) and
    // the K and V of earlier positions were written before this step began, so in the fused form
    // the TMA thread does not wait for the previous kernel (the Q/K/V product): its first tiles are
    // on their way while that kernel drains.  Everything that reads the projection or writes global
    // memory waits.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!FUSE) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        p = token_pos[t], seq = token_seq[t];
    }
    const int lo = first_visible(p, span);
    const int tile_lo = lo / RD_BN, tile_hi = p / RD_BN;
    const int n_tiles = tile_hi - tile_lo + 1;
    const int n_my = split < n_tiles ? (n_tiles - split + n_splits - 1) / n_splits : 0;
    if (n_my == 0) {
        // no keys for this split: the merge kernel skips partials whose maximum is -inf
        if (FUSE) asm volatile("griddepcontrol.wait;" ::: "memory");
        if (tid < G) {
            const size_t o = ((size_t)t * nh + hk * G + tid) * n_splits + split;
            part_ml[o * 2] = -INFINITY;
            part_ml[o * 2 + 1] = 0.f;
        }
        return;
    }

    int p_tab = p;                                    // the position, kept inside the cos/sin table
    if (FUSE && rp.rot > 0 && p >= rp.table_positions) {
        if (tid == 0) atomicExch(rp.err, 3);
        p_tab = rp.table_positions - 1;
    }
    // FUSE: the block that owns the token's last tile also makes the token's new K and V rows
    const bool new_row_here = FUSE && rp.write_kv && split == (tile_hi - tile_lo) % n_splits;

    if (warp == RD_CONSUMERS + 1) {
        // ---- (FUSE) the helper warp: lane < CH makes a chunk of the new K row (rotated), the next CH
        // lanes a chunk of the V row; they go to the cache page and to shared memory, from where the
        // consumer warp that owns the row's place in the last tile takes them
        if (new_row_here) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (lane < 2 * CH) {
                const bool is_k = lane < CH;
                const int c = is_k ? lane : lane - CH;
                float f[8];
                if (is_k) {
                    rd_encoded_chunk<D>(rp, q, (size_t)t * q_stride, nh + hk, c, p_tab, f);
                } else {
                    RdRope plain = rp;
                    plain.rot = 0;
                    rd_encoded_chunk<D>(plain, q, (size_t)t * q_stride, nh + nkv + hk, c, p_tab, f);
                }
                uint4 v;
                __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
                for (int k = 0; k < 4; k++) h2[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
                *reinterpret_cast<uint4*>(new_row_s + (is_k ? 0 : D) + c * 8) = v;
                const int page = block_table[(size_t)seq * max_pages + p / page_size];
                if (page < 0) {
                    atomicExch(rp.err, 2);
                } else {
                    bf16* dst = (is_k ? rp.kc : rp.vc) + (((size_t)page * nkv + hk) * page_size + (p % page_size)) * D + c * 8;
                    *reinterpret_cast<uint4*>(dst) = v;
                }
            }
            __syncwarp();
            if (lane == 0) rd_arrive(row_ready);
        }
        return;
    }
    if (warp == RD_CONSUMERS) {
        // ---- producer
        if (lane == 0) {
            const int* bt = block_table + (size_t)seq * max_pages;
            bool alive = true;
            for (int i = 0; i < n_my && alive; i++) {
                const int s = i % STAGES;
                if (i >= STAGES) {
                    alive = mbar_wait(empty0 + 8 * s, ((i / STAGES) - 1) & 1, err, TC_ERR_TIMEOUT_DECODE);
                    if (!alive) break;
                }
                const int key0 = (tile_lo + split + i * n_splits) * RD_BN;
                const int page = bt[key0 / page_size];
                const int row = (page * nkv + (!FUSE && ex.alias > 1 ? hk / ex.alias : hk)) * page_size + key0 % page_size;
                const unsigned kdst = base + (unsigned)s * 2 * TILE_BYTES, vdst = kdst + TILE_BYTES;
                // The last tile's keys in boxes of 16, one group per consumer warp that has a visible key: whole tiles read a tenth more
                // at contexts of 64 to 430 keys.  (64 tokens of 32 heads there: 62 us a layer, 52 with this, the merge of the warps
                // for the heads alone and the positions loaded ahead; 5.5 TB/s.  Rings of two stages, three blocks an SM: 61, and up
                // to 8 % slower at 600 to 4,000 keys.)
                const int groups = (p - key0) / 16 + 1;
                if (groups < RD_BN / 16) {
                    mbar_expect_tx(full0 + 8 * s, (unsigned)groups * (2 * TILE_BYTES / (RD_BN / 16)));
#pragma unroll
                    for (int hx = 0; hx < D / 64; hx++)
                        for (int u = 0; u < groups; u++) {
                            tma_load_2d(kdst + hx * (RD_BN * 128) + u * (16 * 128), &map_k16, hx * 64, row + u * 16, full0 + 8 * s);
                            tma_load_2d(vdst + hx * (RD_BN * 128) + u * (16 * 128), &map_v16, hx * 64, row + u * 16, full0 + 8 * s);
                        }
                    continue;
                }
                mbar_expect_tx(full0 + 8 * s, 2 * TILE_BYTES);
#pragma unroll
                for (int hx = 0; hx < D / 64; hx++) {
                    tma_load_2d(kdst + hx * (RD_BN * 128), &map_k, hx * 64, row, full0 + 8 * s);
                    tma_load_2d(vdst + hx * (RD_BN * 128), &map_v, hx * 64, row, full0 + 8 * s);
                }
            }
        }
        return;
    }

    // ---- consumers.  Q: the G heads of this kv head as rows 0..G-1, zero rows above
    if (FUSE) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = tid; i < 16 * CH; i += RD_CONSUMERS * 32) {
        const int r = i / CH, c = i % CH;
        if (FUSE && r < G) {
            float f[8];
            rd_encoded_chunk<D>(rp, q, (size_t)t * q_stride, hk * G + r, c, p_tab, f);
            store8(Qs + rd_qswz<D>(r, c), f);
        } else {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (DIFF) {
                if (r < G && (c >= CH / 2) == ((r & 1) != 0)) v = *reinterpret_cast<const uint4*>(q + (size_t)t * q_stride + (size_t)(hk * (G / 2) + (r >> 1)) * D + c * 8);
            } else if (r < G) {
                v = *reinterpret_cast<const uint4*>(q + (size_t)t * q_stride + (size_t)(hk * G + r) * D + c * 8);
            }
            *reinterpret_cast<uint4*>(Qs + rd_qswz<D>(r, c)) = v;
        }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(RD_CONSUMERS * 32) : "memory");
    // warp w owns keys 16w .. 16w+15 of every tile
    const int g = lane >> 2, t4 = lane & 3, mtx = lane >> 3;
    unsigned qf[KS][4];
#pragma unroll
    for (int ks = 0; ks < KS; ks++)
        rd_ldm(qf[ks][0], qf[ks][1], qf[ks][2], qf[ks][3],
               tc_smem_u32(Qs + rd_qswz<D>((mtx & 1) * 8 + (lane & 7), ks * 2 + (mtx >> 1))));

    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    float o[NT_D][4];
#pragma unroll
    for (int i = 0; i < NT_D; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

    bool alive = true;
    for (int i = 0; i < n_my && alive; i++) {
        const int s = i % STAGES;
        // lanes leave the polling loop one by one: together again before the warp-wide instructions
        alive = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (i / STAGES) & 1, err, TC_ERR_TIMEOUT_DECODE));
        if (!alive) break;
        const int key0 = (tile_lo + split + i * n_splits) * RD_BN + warp * 16;
        if (new_row_here && i == n_my - 1 && warp == ((p & (RD_BN - 1)) >> 4)) {
            // the tile came from the cache before the row of position p was there (or while it was
            // being written): this warp, the only reader of that row, puts in what the helper warp made
            alive = __all_sync(0xffffffffu, mbar_wait(row_ready, 0, err, TC_ERR_TIMEOUT_DECODE));
            if (lane < 2 * CH) {
                const int c = lane < CH ? lane : lane - CH;
                unsigned char* tile = gbase + (size_t)s * 2 * TILE_BYTES + (lane < CH ? 0 : TILE_BYTES);
                *reinterpret_cast<uint4*>(tile + rd_tile_off(p & (RD_BN - 1), c)) =
                    *reinterpret_cast<const uint4*>(new_row_s + (lane < CH ? 0 : D) + c * 8);
            }
            __syncwarp();
        }
        if (key0 <= p && key0 + 15 >= lo) {
            const unsigned kbase = base + (unsigned)s * 2 * TILE_BYTES, vbase = kbase + TILE_BYTES;
            // two accumulator sets shorten the chain of dependent MMAs; with DIFF one for each map's channels, of which a row takes its
            // own (its zeros for the other map's channels are not to meet an infinite key there)
            float sa[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            float sb[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            const int krow = warp * 16 + (mtx >> 1) * 8 + (lane & 7);
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                unsigned b0, b1, b2, b3;
                rd_ldm(b0, b1, b2, b3, kbase + rd_tile_off(krow, ks * 2 + (mtx & 1)));
                if (DIFF ? ks >= KS / 2 : (ks & 1) != 0) {
                    rd_mma(sb[0], qf[ks], b0, b1);
                    rd_mma(sb[1], qf[ks], b2, b3);
                } else {
                    rd_mma(sa[0], qf[ks], b0, b1);
                    rd_mma(sa[1], qf[ks], b2, b3);
                }
            }
            float sc[2][4];
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int nt = 0; nt < 2; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int key = key0 + nt * 8 + t4 * 2 + (e & 1);
                    float v = (!DIFF ? sa[nt][e] + sb[nt][e] : g & 1 ? sb[nt][e] : sa[nt][e]) * scale_log2e;
                    if (TERMS > 1 && ex.softcap > 0.f) v = 1.4426950408889634f * soft_cap_fast(sa[nt][e] + sb[nt][e], ex.softcap, ex.softcap_x);
                    if (key > p || key < lo) v = -INFINITY;
                    sc[nt][e] = v;
                    mx[e >> 1] = fmaxf(mx[e >> 1], v);
                }
            float alpha[2], mref[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
                mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
                const float m_new = fmaxf(m_run[e], mx[e]);      // finite: the warp has a valid key
                // (or infinite keys, whose scores of minus infinity have weight 0 as on CUDA cores)
                mref[e] = TERMS > 2 && m_new == -INFINITY ? 0.f : m_new;
                alpha[e] = fast_exp2(m_run[e] - mref[e]);        // 0 the first time (m_run = -inf)
                m_run[e] = m_new;
                l_run[e] *= alpha[e];
            }
            unsigned pf[4], pl[4], pt[4];
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                const float p0 = fast_exp2(sc[nt][0] - mref[0]), p1 = fast_exp2(sc[nt][1] - mref[0]);
                const float p2 = fast_exp2(sc[nt][2] - mref[1]), p3 = fast_exp2(sc[nt][3] - mref[1]);
                l_run[0] += p0 + p1;
                l_run[1] += p2 + p3;
                pf[nt * 2] = rd_pack(p0, p1);
                pf[nt * 2 + 1] = rd_pack(p2, p3);
                if (TERMS > 1) {     // what the rounding took away (exact differences), and what the rounding of that took
                    const float r0 = p0 - rd_low(pf[nt * 2]), r1 = p1 - rd_high(pf[nt * 2]), r2 = p2 - rd_low(pf[nt * 2 + 1]), r3 = p3 - rd_high(pf[nt * 2 + 1]);
                    pl[nt * 2] = rd_pack(r0, r1);
                    pl[nt * 2 + 1] = rd_pack(r2, r3);
                    if (TERMS > 2) {
                        pt[nt * 2] = rd_pack(r0 - rd_low(pl[nt * 2]), r1 - rd_high(pl[nt * 2]));
                        pt[nt * 2 + 1] = rd_pack(r2 - rd_low(pl[nt * 2 + 1]), r3 - rd_high(pl[nt * 2 + 1]));
                    }
                }
            }
            if (key0 + 15 > p || key0 < lo) {
                // a tile at the edge of the range: V rows of hidden keys may hold anything (another
                // sequence's old values), and 0 x NaN would not be 0, so they are cleared
                unsigned char* vgen = gbase + (size_t)s * 2 * TILE_BYTES + TILE_BYTES;
                for (int j = lane; j < 16 * CH; j += 32) {
                    const int r = j / CH, c = j % CH;
                    if (key0 + r > p || key0 + r < lo)
                        *reinterpret_cast<uint4*>(vgen + rd_tile_off(warp * 16 + r, c)) = make_uint4(0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // before TMA refills the stage
                __syncwarp();
            }
            const int vrow = warp * 16 + (mtx & 1) * 8 + (lane & 7);
#pragma unroll
            for (int np = 0; np < NT_D / 2; np++) {
                unsigned b0, b1, b2, b3;
                rd_ldm_t(b0, b1, b2, b3, vbase + rd_tile_off(vrow, np * 2 + (mtx >> 1)));
                if (TERMS > 2) {
                    // the 16 keys' sum from zero, the smallest terms first, and onto the running sum in float32: the tensor cores cut
                    // off what does not fit an accumulator, which with the running sum in it is lost in one direction key by key
                    float v0[4] = {0.f, 0.f, 0.f, 0.f}, v1[4] = {0.f, 0.f, 0.f, 0.f};
                    rd_mma(v0, pt, b0, b1);
                    rd_mma(v1, pt, b2, b3);
                    rd_mma(v0, pl, b0, b1);
                    rd_mma(v1, pl, b2, b3);
                    rd_mma(v0, pf, b0, b1);
                    rd_mma(v1, pf, b2, b3);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        o[np * 2][e] = fmaf(o[np * 2][e], alpha[e >> 1], v0[e]);
                        o[np * 2 + 1][e] = fmaf(o[np * 2 + 1][e], alpha[e >> 1], v1[e]);
                    }
                    continue;
                }
                o[np * 2][0] *= alpha[0];
                o[np * 2][1] *= alpha[0];
                o[np * 2][2] *= alpha[1];
                o[np * 2][3] *= alpha[1];
                o[np * 2 + 1][0] *= alpha[0];
                o[np * 2 + 1][1] *= alpha[0];
                o[np * 2 + 1][2] *= alpha[1];
                o[np * 2 + 1][3] *= alpha[1];
                rd_mma(o[np * 2], pf, b0, b1);
                rd_mma(o[np * 2 + 1], pf, b2, b3);
                if (TERMS > 1) {
                    rd_mma(o[np * 2], pl, b0, b1);
                    rd_mma(o[np * 2 + 1], pl, b2, b3);
                }
            }
        }
        __syncwarp();
        if (lane == 0) rd_arrive(empty0 + 8 * s);
    }
#pragma unroll
    for (int e = 0; e < 2; e++) {
        l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 1);
        l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 2);
    }

    // ---- merge the warps (ascending) through the ring's memory: every load has landed and been read
    asm volatile("bar.sync 1, %0;" ::"n"(RD_CONSUMERS * 32) : "memory");
    float* mrg = reinterpret_cast<float*>(gbase);            // [RD_CONSUMERS][16][D + 2]
    constexpr int ROW = D + 2;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int r = g + e * 8;
        if (r >= G) continue;
        float* dst = mrg + ((size_t)warp * 16 + r) * ROW;
#pragma unroll
        for (int i = 0; i < NT_D; i++) *reinterpret_cast<float2*>(dst + i * 8 + t4 * 2) = make_float2(o[i][e * 2], o[i][e * 2 + 1]);
        if (t4 == 0) {
            dst[D] = m_run[e];
            dst[D + 1] = l_run[e];
        }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(RD_CONSUMERS * 32) : "memory");
    for (int idx = tid; idx < G * D; idx += RD_CONSUMERS * 32) {
        const int r = idx / D, c = idx - r * D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < RD_CONSUMERS; w++) M = fmaxf(M, mrg[((size_t)w * 16 + r) * ROW + D]);
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < RD_CONSUMERS; w++) {
            const float mw = mrg[((size_t)w * 16 + r) * ROW + D];
            const float wgt = (mw == -INFINITY) ? 0.f : fast_exp2(mw - M);
            num += mrg[((size_t)w * 16 + r) * ROW + c] * wgt;
            den += mrg[((size_t)w * 16 + r) * ROW + D + 1] * wgt;
        }
        const size_t head = (size_t)t * nh + hk * G + r;
        if (n_splits == 1 && out) {
            out[head * D + c] = __float2bfloat16_rn(rd_finish(num, den, M, ex, t, hk * G + r, D, c));
        } else {
            const size_t oidx = head * n_splits + split;
            part_acc[oidx * D + c] = num;
            if (c == 0) {
                part_ml[oidx * 2] = M;
                part_ml[oidx * 2 + 1] = den;
            }
        }
    }
}

// The weight of a head's share s (lane s of every warp, at most 32 shares; 0 for a share without keys, whose sums were not written)
// and, returned, the largest maximum.  All shares' words are one load, where a thread that goes through them waits for each round.
__device__ __forceinline__ float rd_share_weights(const float* __restrict__ part_ml, size_t o, int n_splits, float& w, float& l) {
    const int lane = threadIdx.x & 31;
    float2 ml = make_float2(-INFINITY, 0.f);
    if (lane < n_splits) ml = make_float2(part_ml[(o + lane) * 2], part_ml[(o + lane) * 2 + 1]);      // (any address)
    float M = ml.x;
#pragma unroll
    for (int k = 16; k; k >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, k));
    w = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - M);
    l = ml.y;
    return M;
}
// sum of w acc and of w l over the shares, ascending, shares of weight 0 left out; eight rows' loads in flight
template <int D>
__device__ __forceinline__ void rd_add_shares(const float* __restrict__ acc, int n_splits, float w, float l, float& num, float& den) {
    num = den = 0.f;
    for (int s0 = 0; s0 < n_splits; s0 += 8) {
        float v[8], ws[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            ws[k] = __shfl_sync(0xffffffffu, w, (s0 + k) & 31);
            v[k] = s0 + k < n_splits && ws[k] != 0.f ? acc[(size_t)(s0 + k) * D] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            den += __shfl_sync(0xffffffffu, l, (s0 + k) & 31) * (s0 + k < n_splits ? ws[k] : 0.f);
            num += v[k] * ws[k];
        }
    }
}

// (One sequence of 32 heads: 2.4 -> 1.9 us; with the two maps of differential heads 5.8 -> 2.9.)
// out[t, h, :] = sum over splits (ascending) of acc * 2^(m - M) / sum of l * 2^(m - M); splits
// without keys carry m = -inf and are skipped.
template <int D>
__global__ void attention_decode_ring_merge_kernel(const float* __restrict__ part_acc,
                                                   const float* __restrict__ part_ml, bf16* __restrict__ out,
                                                   int n_splits, int nh, const RdExtras ex) {
    pdl_grid_sync();
    const int h = blockIdx.x, t = blockIdx.y, c = threadIdx.x;
    const size_t o = ((size_t)t * nh + h) * n_splits;
    float w, l, num, den;
    const float M = rd_share_weights(part_ml, o, n_splits, w, l);
    rd_add_shares<D>(part_acc + o * D + c, n_splits, w, l, num, den);
    out[((size_t)t * nh + h) * D + c] = __float2bfloat16_rn(rd_finish(num, den, M, ex, t, h, D, c));
}

// ---- host side

typedef CUresult (*RdEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static RdEncodeTiledFn rd_encode_fn() {
    static RdEncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (RdEncodeTiledFn)p;
    }
    return fn;
}

// one cache entry seen as a bfloat16 matrix [rows = pages * kv heads * page_size, d]; boxes of [box_rows, 64]
static int rd_make_map(CUtensorMap* map, const void* ptr, long long rows, int d, int box_rows) {
    RdEncodeTiledFn fn = rd_encode_fn();
    if (!fn) return ILLM_ERR_BAD_ARG;
    cuuint64_t dims[2] = {(cuuint64_t)d, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)d * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : ILLM_ERR_BAD_ARG;
}

template <int D>
static int rd_launch(const void* q, int q_stride, const void* kc, const void* vc, long long n_pages,
                     const int* block_table, int max_pages, const int* token_pos, const int* token_seq,
                     float* part_acc, float* part_ml, void* out, int T, int nh, int nkv, int page_size, int window,
                     float scale, int n_splits, int* err, cudaStream_t s, const RdRope* rope, const RdExtras* extras, int terms, bool diff) {
    CUtensorMap mk, mv, mk16, mv16;
    int rc;
    const long long rows = n_pages * nkv * page_size;
    if ((rc = rd_make_map(&mk, kc, rows, D, RD_BN)) != 0 || (rc = rd_make_map(&mv, vc, rows, D, RD_BN)) != 0) return rc;
    if ((rc = rd_make_map(&mk16, kc, rows, D, 16)) != 0 || (rc = rd_make_map(&mv16, vc, rows, D, 16)) != 0) return rc;
    constexpr int STAGES = 384 / D;
    const size_t smem = (size_t)STAGES * 2 * RD_BN * D * 2 + (size_t)16 * D * 2 + 1024;
    RdRope rp = {};
    if (rope) rp = *rope;
    RdExtras ex = {};
    if (extras) ex = *extras;
    if (rope && (terms > 1 || extras)) return ILLM_ERR_BAD_ARG;      // the fused form is the plain attention's
    const int groups = nkv * (ex.alias > 1 ? ex.alias : 1);
    auto launch = [&](auto kern) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        illm_launch(kern, dim3(n_splits, groups, T), dim3(rope ? RD_THREADS + 32 : RD_THREADS), smem, s, mk, mv, mk16, mv16, (const bf16*)q, q_stride,
                    block_table, max_pages, token_pos, token_seq, part_acc, part_ml, (bf16*)out, n_splits, nh, nkv,
                    nh / groups, page_size, window, scale * 1.4426950408889634f, err, rp, ex);
        return illm_launch_status();
    };
    if (diff) {
        if constexpr (D == 128) rc = launch(attention_decode_ring_kernel<D, false, 3, true>);
        else return ILLM_ERR_BAD_ARG;
    } else {
        rc = rope         ? launch(attention_decode_ring_kernel<D, true, 1, false>)
             : terms == 1 ? launch(attention_decode_ring_kernel<D, false, 1, false>)
             : terms == 2 ? launch(attention_decode_ring_kernel<D, false, 2, false>)
                          : launch(attention_decode_ring_kernel<D, false, 3, false>);
    }
    if (rc != 0 || n_splits == 1 || !out) return rc;        // no out: the shares are the caller's to put together
    illm_launch(attention_decode_ring_merge_kernel<D>, dim3(nh, T), dim3(D), 0, s, (const float*)part_acc,
                (const float*)part_ml, (bf16*)out, n_splits, nh, ex);
    return illm_launch_status();
}

static int rd_run(const void* q, int q_stride, const void* kc, const void* vc, long long n_pages,
                  const int* block_table, int max_pages, const int* token_pos, const int* token_seq, float* part_acc,
                  float* part_ml, void* out, int T, int nh, int nkv, int d, int page_size, int window, float scale,
                  int n_splits, int* err, void* stream, const RdRope* rope, const RdExtras* extras = nullptr, int terms = 1, bool diff = false) {
    if (T <= 0) return 0;
    const int alias = extras && extras->alias > 1 ? extras->alias : 1;
    if (nkv <= 0 || nh % (nkv * alias) || nh / (nkv * alias) > 16 || T > 65535 || nkv * alias > 65535 || (q_stride & 7) || page_size % RD_BN ||
        n_splits < 1 || n_splits > RD_MAX_SPLITS || ((uintptr_t)kc & 15) || ((uintptr_t)vc & 15) ||
        n_pages * nkv * page_size > 0x7fffffffLL || ((n_splits > 1 || !out) && (part_acc == nullptr || part_ml == nullptr)))
        return ILLM_ERR_BAD_ARG;
    if (!(rope && rope->partials) && (q == nullptr || ((uintptr_t)q & 15))) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (d == 128)
        return rd_launch<128>(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc,
                              part_ml, out, T, nh, nkv, page_size, window, scale, n_splits, err, s, rope, extras, terms, diff);
    if (d == 64)
        return rd_launch<64>(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc,
                             part_ml, out, T, nh, nkv, page_size, window, scale, n_splits, err, s, rope, extras, terms, diff);
    return ILLM_ERR_BAD_ARG;
}

// q: the packed projection [T, q_stride] whose first nh*d columns are the query heads; kc, vc: one
// cache entry [n_pages, nkv, page_size, d] with page_size a multiple of 64.  Scratch (unused with
// one split): part_acc float [T, nh, n_splits, d], part_ml float [T, nh, n_splits, 2].
extern "C" int illm_attention_decode_ring(const void* q, int q_stride, const void* kc, const void* vc,
                                          long long n_pages, const int* block_table, int max_pages,
                                          const int* token_pos, const int* token_seq, float* part_acc,
                                          float* part_ml, void* out, int T, int nh, int nkv, int d, int page_size,
                                          int window, float scale, int n_splits, int* err, void* stream) {
    return rd_run(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc, part_ml, out, T,
                  nh, nkv, d, page_size, window, scale, n_splits, err, stream, nullptr);
}

extern "C" int illm_attention_decode_ring_shared(const void* q, int q_stride, const void* kc, const void* vc, long long n_pages, const int* block_table,
                                                 int max_pages, const int* token_pos, const int* token_seq, float* part_acc, float* part_ml, void* out, int T,
                                                 int nh, int nkv, int d, int page_size, int window, float scale, int n_splits, int* err, int wide_p,
                                                 const float* sinks, const float* gate, int gate_stride, int gate_wide, float softcap, int alias, void* stream);

// The same with sinks, gates (either may be nullptr), a soft cap (0: none; needs wide_p) and, with wide_p, two-term softmax
// weights; `window` is a span (first_visible): a window, or chunks if it is negative.
extern "C" int illm_attention_decode_ring_ex(const void* q, int q_stride, const void* kc, const void* vc,
                                             long long n_pages, const int* block_table, int max_pages,
                                             const int* token_pos, const int* token_seq, float* part_acc,
                                             float* part_ml, void* out, int T, int nh, int nkv, int d, int page_size,
                                             int window, float scale, int n_splits, int* err, int wide_p, const float* sinks,
                                             const float* gate, int gate_stride, int gate_wide, float softcap, void* stream) {
    if (softcap > 0.f && !wide_p) return ILLM_ERR_BAD_ARG;
    return illm_attention_decode_ring_shared(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc, part_ml, out, T, nh, nkv, d,
                                             page_size, window, scale, n_splits, err, wide_p, sinks, gate, gate_stride, gate_wide, softcap, 1, stream);
}

// The same with a KV head's query heads over `alias` blocks (groups of more than 16 query heads).  With wide_p their weights enter in
// three terms: such groups ran in float32 on CUDA cores before (attention_maps.cu), and keep its precision.
extern "C" int illm_attention_decode_ring_shared(const void* q, int q_stride, const void* kc, const void* vc, long long n_pages, const int* block_table,
                                                 int max_pages, const int* token_pos, const int* token_seq, float* part_acc, float* part_ml, void* out, int T,
                                                 int nh, int nkv, int d, int page_size, int window, float scale, int n_splits, int* err, int wide_p,
                                                 const float* sinks, const float* gate, int gate_stride, int gate_wide, float softcap, int alias, void* stream) {
    if (softcap > 0.f && !wide_p) return ILLM_ERR_BAD_ARG;
    RdExtras ex{sinks, gate, gate_stride, gate_wide, softcap, softcap > 0.f ? 2.0f * scale * 1.4426950408889634f / softcap : 0.f, alias};
    return rd_run(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc, part_ml, out, T,
                  nh, nkv, d, page_size, window, scale, n_splits, err, stream, nullptr, &ex, !wide_p ? 1 : alias > 1 ? 3 : 2);
}

// The same with the position encoding and the cache write inside: `qkv` is the unrotated packed
// projection [T, (nh + 2 nkv) d] in bfloat16, or nullptr with `partials`, its `splits` float32 K
// slices [splits][T][(nh + 2 nkv) d].  cos_sin: float32 [table_positions][rot / 2][2] (rot = 0: no
// rotation).  write_kv = 0: the cache already holds this token's K and V (a layer that reads another
// layer's entry).  step_err: the step's error word (2: a sequence without a page for its position,
// 3: a position outside the table).  Needs rot % 16 == 0.
extern "C" int illm_attention_decode_ring_rope(const void* qkv, const float* partials, int splits,
                                               long long split_stride, const float* cos_sin, int rot,
                                               int table_positions, int write_kv, void* kc, void* vc,
                                               long long n_pages, const int* block_table, int max_pages,
                                               const int* token_pos, const int* token_seq, float* part_acc,
                                               float* part_ml, void* out, int T, int nh, int nkv, int d,
                                               int page_size, int window, float scale, int n_splits, int* err,
                                               int* step_err, void* stream) {
    if (rot < 0 || rot > d || (rot & 15) || (rot > 0 && cos_sin == nullptr) || step_err == nullptr ||
        (partials != nullptr && splits < 1))
        return ILLM_ERR_BAD_ARG;
    RdRope rp = {partials, splits, split_stride, (const float2*)cos_sin, rot, table_positions, (bf16*)kc, (bf16*)vc,
                 write_kv, step_err};
    return rd_run(qkv, (nh + 2 * nkv) * d, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc,
                  part_ml, out, T, nh, nkv, d, page_size, window, scale, n_splits, err, stream, &rp);
}

// The shares of both maps of a (token, head) put together in the order of the blocks, o = a_1 - lambda a_2, the head's unit norm and the
// factor.  A block per (token, head), a thread per map and value channel.
template <int D>
__global__ void __launch_bounds__(2 * D) attention_diff_ring_merge_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_ml, bf16* __restrict__ out,
                                                                          int n_splits, int nh, float lambda, float eps, float out_scale) {
    pdl_grid_sync();
    __shared__ float scratch[32], second[D];
    const int h = blockIdx.x, t = blockIdx.y, m = threadIdx.x / D, c = threadIdx.x % D;
    const size_t o = (((size_t)t * nh + h) * 2 + m) * n_splits;
    float w, l, num, den;
    rd_share_weights(part_ml, o, n_splits, w, l);
    rd_add_shares<D>(part_acc + o * D + c, n_splits, w, l, num, den);
    if (m == 1) second[c] = num / den;
    __syncthreads();
    const float v = m == 0 ? fmaf(-lambda, second[c], num / den) : 0.f;
    const float ss = block_sum(v * v, scratch);
    if (m == 0) out[((size_t)t * nh + h) * D + c] = __float2bfloat16_rn(v * (out_scale / sqrtf(ss / (float)D + eps)));
}

// Differential attention of single tokens: q [T, q_stride] with head h's [q_1, q_2] (2 x 64 channels) at column h * 128, pages of key
// rows [k_1, k_2] and value rows of 128; scratch part_acc float [T, nh, 2, n_splits, 128], part_ml float [T, nh, 2, n_splits, 2].
// (On CUDA cores, attention_maps.cu, one token of 32 heads over 1,800 keys took 19 us and its merge 6.3; here 6.9 and 2.9.)
extern "C" int illm_attention_diff_ring_supported(int nh, int nkv, int d, int dv, int page_size) {
    return d == 64 && dv == 128 && nkv > 0 && nh % nkv == 0 && nh / nkv <= 8 && page_size > 0 && page_size % RD_BN == 0;
}
extern "C" int illm_attention_diff_ring(const void* q, int q_stride, const void* kc, const void* vc, long long n_pages, const int* block_table, int max_pages,
                                        const int* token_pos, const int* token_seq, float* part_acc, float* part_ml, void* out, int T, int nh, int nkv, int d, int dv,
                                        int page_size, int window, float scale, int n_splits, float lambda, float eps, float out_scale, int* err, void* stream) {
    if (T <= 0) return 0;
    if (!illm_attention_diff_ring_supported(nh, nkv, d, dv, page_size) || !out) return ILLM_ERR_BAD_ARG;
    RdExtras ex{nullptr, nullptr, 0, 0, 0.f, 0.f, 1};
    const int rc = rd_run(q, q_stride, kc, vc, n_pages, block_table, max_pages, token_pos, token_seq, part_acc, part_ml, nullptr, T, 2 * nh, nkv, 128, page_size,
                          window, scale, n_splits, err, stream, nullptr, &ex, 3, true);
    if (rc) return rc;
    illm_launch(attention_diff_ring_merge_kernel<128>, dim3(nh, T), dim3(256), 0, (cudaStream_t)stream, (const float*)part_acc, (const float*)part_ml, (bf16*)out,
                n_splits, nh, lambda, eps, out_scale);
    return illm_launch_status();
}
