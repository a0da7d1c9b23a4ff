// All layers of a small decode step in one persistent kernel (sm_100a): up to eight tokens, one per
// request, through a stack of layers  h += attention(rmsnorm(h)); h += feed_forward(rmsnorm(h))
// with grouped-query attention over a paged cache, NeoX rotation of whole heads and a silu gate.
//
// What bounds such a step is the chain of dependent passes a layer is made of, not the weights: as
// kernels, even with programmatic launch, a hand-over costs 1.0 to 1.9 us and a product's body starts
// on a cold pipeline.  Here one CTA per SM stays resident for the whole step (a cooperative launch).
// Each of its 16 warps owns a list of weight pieces, known from the shapes alone, and a ring in shared
// memory that TMA fills ahead of the product: weights of later phases and of the next layer arrive
// while a phase waits for the one before it.  Five phases a layer, a barrier over the grid between them:
//   1  norm, q/k/v product, bias, rotation, cache write
//   2  attention, a request's keys split over CTAs
//   3  merge of the key splits, output projection, added into the stream
//   4  norm, gate and up product, silu(gate) * up
//   5  down projection, added into the stream
// A layer of 0.5B sizes takes 22 to 25 us at one to eight tokens (23 to 28 as kernels, 4.5 for the weights alone): per phase
// some 1,100 cycles for the barrier's fence, 800 for the wait of the last CTA, 1,500 to 4,500 for the operand (a trip to L2 and
// the work on it), 800 to 1,500 for the product, 600 to 1,600 for what becomes of its sums.  us a pass of perf/cases.py,
// layer by layer and here: decode_05b_1 4,857 and 4,618, decode_05b_8 5,902 and 5,471, decode_7b_4 12,859 and 11,785.
// Products run on mma.sync m16n8k16 with the weights as the 16-row operand and 8 tokens as the other:
// a warp multiplies straight from its ring, without the tensor-memory round trip of tcgen05 (which for a
// handful of tokens took 70 to 110 ns per 128 x 16 x 16 instruction); the math is a
// few tenths of a microsecond a phase either way.  A piece is two groups of eight weight rows (the
// two halves of a rotated head, gate and up rows of the same outputs, or neighbours) by 64 or 128
// columns, so that both values an epilogue combines end up in one tile of 16 rows.  Sums over a tile's
// pieces go through shared memory in the order of the pieces.
// The stream is kept as layer by layer: an fp32 base plus the 64-bit fixed-point accumulator of common.cuh, into
// which phases 3 and 5 add with integer atomics, so that the result does not depend on their order.  Phases 1 and 4
// read base + accumulator; behind them, while the barrier is waited for, the sum becomes the other base, and once all
// have read it the accumulator is cleared.  Only what one sublayer adds is ever in fixed point: infinities, NaN and
// numbers of any size in an embedding reach the logits.  The norm's factor 1 / sqrt(mean square + eps) is applied to
// a product's sums, its weight to the operand.
// (src/alofa/kernels/cpu/scalar.mojo:93-231, 283-470 for the formulas; src/alofa/model/arch/qwen.mojo:1367-1510
// for the order of a layer.)
//
// Every wait is bounded: after the limit the status word is raised, every CTA skips what is left, waits
// for its own copies in flight and returns.
#include <stddef.h>
#include <string.h>

#include "common.cuh"
#include "tma.cuh"

constexpr int WARPS = 16;
constexpr int THREADS = 32 * WARPS;
constexpr int PACE = 3;                  // pieces a paced warp asks for ahead of a product
constexpr int GRANULE = 16;              // keys a warp takes at a time
constexpr int MAX_TOKENS = 8;             // the columns of a product: two groups of them were slower than layer by layer (9 to 16 tokens of 0.5B sizes 3 %, of 1.5B sizes 17 %)
constexpr int MAX_TILES = 64;             // of 16 rows a CTA and phase
constexpr uint32_t BARRIER_LIMIT = 1u << 21;  // polls of the grid barrier, about a second
enum { P_QKV = 0, P_OUT = 1, P_GATE = 2, P_DOWN = 3 };

struct LayerVectors {
  const float* gamma_mixer;
  const float* gamma_ff;
  const float* qkv_bias;  // or null
  bf16* k;                // [slots, kv heads, HD]
  bf16* v;
  float eps_mixer, eps_ff;
};
struct alignas(64) StackLayer {  // of the table of layers
  CUtensorMap maps[4];  // q/k/v, output, gate and up, down: boxes of 8 rows x 2 x `chunks` x 64 columns
  LayerVectors vectors;
  int pad[4];
};
static_assert(sizeof(StackLayer) % 64 == 0, "tensor maps need 64-byte alignment");
// The table is a kernel parameter, as the maps of every other kernel are: in global memory that the host writes, each map would want a
// fence of the tensor-map proxy in every CTA first, 100 ns a map (decode_05b_1 of perf/cases.py 4,661 us a pass that way, 4,620 this).
// Parameters have 32,764 bytes: a deeper model goes in launches of so many layers.
constexpr int MAX_LAYERS = 48;
struct StackTable {
  StackLayer layers[MAX_LAYERS];
};

struct PhasePlan {
  int tiles, slices;  // tiles of 16 rows, slices of `chunks` * 64 columns
  int kg, rg;         // 0: tiles dealt whole over the CTAs; else CTAs as kg ranges of slices x rg ranges of tiles
};

struct StackArgs {
  int n_layers;
  int added;                 // whether `acc` holds something already (a launch that goes on where another stopped)
  int tokens, hidden, heads, kv_heads, group, inter;
  int page, table_stride;
  int chunks, slots;         // 64-column chunks of a piece, pieces in a warp's ring
  int paced;                 // a warp asks for a few pieces ahead of each product, not for all it can behind it
  int x_stride;              // bytes of an operand row in shared memory
  int qkv_tiles;             // of a CTA, at most
  int x_bytes, work_bytes;   // operand rows; operand, sums and attention together
  float scale;               // of the scores, times log2(e)
  float per_group, per_cta;  // 1 / group, 1 / CTAs: quotients of small numbers by a product
  PhasePlan plan[4];
  float* base;               // [tokens, hidden]: the stream, before phase 1 (and at the end) without what `acc` holds
  float* base_ff;            // the same before phase 4, without what `acc_ff` holds
  long long* acc;            // [tokens, hidden]: what the last feed-forward added; zero before unless `added`
  long long* acc_ff;         // what the attention added; zero before and afterwards
  const int* positions;
  const int* block_table;    // [tokens, table_stride]
  const int* slot_map;       // [tokens]
  const float* rope;         // [positions, HD / 2, 2]
  bf16* q;                   // [tokens, heads * HD]
  float* part_o;             // [CTAs, 8, HD]
  float* part_ml;            // [CTAs, 8, 2]
  bf16* act;                 // [CTAs][tiles][tokens][8]: a CTA writes lines of its own (lines that eight CTAs wrote took a fence three times as long)
  int act_stride;            // numbers from CTA to CTA
  unsigned* barrier;
  int* status;
};

// ---- wrappers ---------------------------------------------------------------------------------------------
// A piece: both groups of rows at once, marked to leave L2 first: a weight is read once a step, what the phases hand over stays
// (four requests of the 7B shape, us a pass of four steps without and with the mark: 12,590 and 12,120).
__device__ __forceinline__ void tma_load_piece(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row, int chunk) {
  asm volatile(
      "{\n\t.reg .b64 p;\n\tcreatepolicy.fractional.L2::evict_first.b64 p, 1.0;\n\t"
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %3, %5}], [%2], p;\n\t}" ::"r"(dst), "l"(map), "r"(bar),
      "r"(0), "r"(row), "r"(chunk)
      : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t transposed(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Where a maximum of scores starts.  Scores of minus infinity (keys or queries out of bfloat16's range) then weigh nothing also where a
// granule, a warp or a split has no others: 2^(-inf - LOWEST) is 0, the difference of two such maxima 0.
constexpr float LOWEST = -3.402823466e38f;
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}

// ---- a CTA's share of a phase -------------------------------------------------------------------------------
struct Share {
  int tile0, tile_step, tiles;  // local tile i is tile0 + i * tile_step
  int slice0, slices;
  int pieces, warps;            // tiles * slices, dealt to so many warps: warp w has pieces [w * pieces / warps, (w + 1) * pieces / warps)
  int shift, head_rows; // a tile's rows: 8 from (tile >> shift) * head_rows + (tile & mask) * 8, and 8 as far on as the map's second group is
};

struct alignas(16) Loader {  // a warp's next piece and its place in the list of them, how many it has asked for
  int row, chunk, layer, phase;
  int piece, end, tile, slice;
  int slices, asked, pad[2];
};
struct Part {  // of a phase, for one warp: its pieces, and tile and slice of the first
  short first, end, tile, slice;
};

struct Small {  // of shared memory
  Share share[4];
  Part part[4][WARPS];
  alignas(16) Loader loader[WARPS];
  unsigned char first_warp[4][MAX_TILES], last_warp[4][MAX_TILES];  // of the warps with pieces of a tile
  float square[WARPS];       // each warp's sum of squares in a norm
  float factor[MAX_TOKENS];  // 1 / sqrt(mean square + eps)
  int position[MAX_TOKENS];
  int slot[MAX_TOKENS];
  int item0[MAX_TOKENS];     // attention: a token's first item, its key splits
  int splits[MAX_TOKENS];
  int per_split, item_token, item_group, item_first, item_last;  // granules of keys a split has at most; this CTA's item
  int first_row[WARPS];      // of the cache: where the warp's first granule lies
  alignas(16) float wm[WARPS][8];  // attention: each warp's maxima and sums, by head
  alignas(16) float wl[WARPS][8];
  alignas(8) LayerVectors layer[2];  // of this layer and the next
  int abort_flag;
};

static_assert(sizeof(Small) % 16 == 0 && offsetof(Small, loader) % 16 == 0 && offsetof(Small, wm) % 16 == 0 && offsetof(Small, wl) % 16 == 0 && offsetof(Small, layer) % 8 == 0, "vector loads");

// Where a piece lies in its weight.
__device__ __forceinline__ void place_piece(Loader& ld, const Share& s, int chunks) {
  const int tile = s.tile0 + ld.tile * s.tile_step;
  ld.row = (tile >> s.shift) * s.head_rows + (tile & ((1 << s.shift) - 1)) * 8;
  ld.chunk = (s.slice0 + ld.slice) * chunks;
}
// The next phase in which a warp has pieces.
__device__ __forceinline__ void next_phase(Loader& ld, const Small& sm, int warp, int n_layers, int chunks) {
  do {
    if (++ld.phase == 4) {
      ld.phase = 0;
      if (++ld.layer >= n_layers) return;
    }
    const Part p = sm.part[ld.phase][warp];
    ld.piece = p.first;
    ld.end = p.end;
    ld.tile = p.tile;
    ld.slice = p.slice;
  } while (ld.piece >= ld.end);
  ld.slices = sm.share[ld.phase].slices;
  place_piece(ld, sm.share[ld.phase], chunks);
}

// A register that only some paths write counts as held from the start of the loop over layers to its end; that is why what a
// load may leave out is set to zero first.
template <int HD>
__global__ void __launch_bounds__(THREADS, 1) decode_stack_kernel(const __grid_constant__ StackArgs a, const __grid_constant__ StackTable table) {
  constexpr int TP = MAX_TOKENS, C32 = HD / 32;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t piece_bytes = 2048u * a.chunks;
  unsigned char* ring = smem_raw;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + (size_t)WARPS * a.slots * piece_bytes);
  unsigned char* work = reinterpret_cast<unsigned char*>(bars + WARPS * a.slots);
  float* sums = reinterpret_cast<float*>(work + a.x_bytes);
  float* osm = reinterpret_cast<float*>(work);
  float2* turn = reinterpret_cast<float2*>(work + a.work_bytes);          // [tokens, HD / 2]
  float* gamma_s = reinterpret_cast<float*>(turn + a.tokens * (HD / 2));  // the next norm's weight
  float* bias_s = gamma_s + a.hidden;                                     // of this CTA's q/k/v tiles, 16 a tile
  Small& sm = *reinterpret_cast<Small*>(bias_s + 16 * a.qkv_tiles);

  // Read anew in every phase: all of a phase's indices are the same in each layer, and kept over the loop over layers they
  // would take twice the registers there are.
  int tid, lane, warp, j, r, cta;
  auto place_thread = [&]() {
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
    lane = tid & 31;
    warp = tid >> 5;
    j = lane & 3;
    r = lane >> 2;
  };
  place_thread();
  const int ctas = gridDim.x;
  const int T = a.tokens, H = a.hidden, group = a.group;
  volatile int* abort_flag = &sm.abort_flag;

  // ---- set-up -------------------------------------------------------------------------------------------
  if (tid < 4) {
    const PhasePlan p = a.plan[tid];
    Share s;
    s.tile0 = s.tile_step = s.tiles = s.slice0 = s.slices = 0;
    if (p.kg == 0) {
      const int c = tid == P_GATE ? ctas - 1 - cta : cta;  // the CTAs with a tile more differ between the phases
      s.tile0 = c;
      s.tile_step = ctas;
      s.tiles = c < p.tiles ? (p.tiles - 1 - c) / ctas + 1 : 0;
      s.slices = p.slices;
    } else if (cta < p.kg * p.rg) {
      const int k = cta % p.kg, g = cta / p.kg;
      s.tile0 = g * p.tiles / p.rg;
      s.tiles = (g + 1) * p.tiles / p.rg - s.tile0;
      s.tile_step = 1;
      s.slice0 = k * p.slices / p.kg;
      s.slices = (k + 1) * p.slices / p.kg - s.slice0;
    }
    s.pieces = s.tiles * s.slices;
    s.warps = min(WARPS, s.pieces);  // each of them has a piece
    s.shift = tid == P_QKV ? (HD == 128 ? 3 : 2) : tid == P_GATE ? 30 : 0;
    s.head_rows = tid == P_QKV ? HD : 16;
    sm.share[tid] = s;
  }
  if (tid < (int)(sizeof(LayerVectors) / 4)) reinterpret_cast<int*>(&sm.layer[0])[tid] = reinterpret_cast<const int*>(&table.layers[0].vectors)[tid];
  if (tid == 0) sm.abort_flag = 0;
  if (tid < WARPS * a.slots) mbar_init(bars + tid, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (tid < T) {
    sm.position[tid] = a.positions[tid];
    sm.slot[tid] = a.slot_map[tid];
  }
  unsigned sense = 0;
  if (tid == 0) {
    unsigned now;
    asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(now) : "l"(a.barrier) : "memory");
    sense = now & 0x80000000u;
  }
  __syncthreads();

  if (tid < 4 * MAX_TILES) {
    const Share& s = sm.share[tid / MAX_TILES];
    const int i = tid % MAX_TILES;
    if (i < s.tiles) {
      sm.first_warp[tid / MAX_TILES][i] = (unsigned char)((s.warps * (i * s.slices + 1) - 1) / s.pieces);
      sm.last_warp[tid / MAX_TILES][i] = (unsigned char)((s.warps * (i + 1) * s.slices - 1) / s.pieces);
    }
  } else if (tid < 4 * MAX_TILES + 4 * WARPS) {
    const int phase = (tid - 4 * MAX_TILES) / WARPS, w = (tid - 4 * MAX_TILES) % WARPS;
    const Share& s = sm.share[phase];
    Part p = {0, 0, 0, 0};
    if (w < s.warps) {
      p.first = (short)(w * s.pieces / s.warps);
      p.end = (short)((w + 1) * s.pieces / s.warps);
      p.tile = (short)(p.first / s.slices);
      p.slice = (short)(p.first - p.tile * s.slices);
    }
    sm.part[phase][w] = p;
  }
  int t_bits = 0;  // tokens in items of an epilogue go up to a power of two
  while ((1 << t_bits) < T) ++t_bits;
  const int t_mask = (1 << t_bits) - 1;
  __syncthreads();

  // A warp's ring of pieces.
  uint64_t* my_bars = bars + warp * a.slots;
  const uint32_t my_ring = smem_u32(ring) + (uint32_t)(my_bars - bars) * piece_bytes;
  int slot = 0;  // the next piece's place in this warp's ring
  uint32_t parity = 0;
  int taken = 0;        // pieces multiplied
  int empty = a.slots;  // places of the ring that nothing is on its way to, the last of them before `slot`
  if (lane == 0) {
    Loader ld = {};
    ld.phase = -1;
    next_phase(ld, sm, warp, a.n_layers, a.chunks);
    sm.loader[warp] = ld;
  }
  // Asks for the next pieces of this warp's list, one for each empty place.
  auto refill = [&](int most) {
    const int ask = min(most, empty);
    if (lane == 0) {
      Loader ld = sm.loader[warp];
      int into = slot - empty;
      if (into < 0) into += a.slots;
#pragma unroll 1
      for (int k = 0; k < ask && ld.layer < a.n_layers; ++k) {
        mbar_expect_tx(my_bars + into, piece_bytes);
        tma_load_piece(my_ring + (uint32_t)into * piece_bytes, &table.layers[ld.layer].maps[ld.phase], smem_u32(my_bars + into), ld.row, ld.chunk);
        ++ld.asked;
        if (++ld.piece == ld.end) {
          next_phase(ld, sm, warp, a.n_layers, a.chunks);
        } else if (++ld.slice == ld.slices) {
          ld.slice = 0;
          ++ld.tile;
          place_piece(ld, sm.share[ld.phase], a.chunks);
        } else {
          ld.chunk += a.chunks;
        }
        if (++into == a.slots) into = 0;
      }
      sm.loader[warp] = ld;
    }
    empty -= ask;
  };
  refill(a.slots);

  // The attention item of this CTA: the keys of (request, KV head) pairs go in splits of as many granules as
  // make all items resident together, no fewer than one per warp.
  for (int i = tid; i < T * (HD / 2); i += THREADS) turn[i] = reinterpret_cast<const float2*>(a.rope)[(size_t)sm.position[i / (HD / 2)] * (HD / 2) + i % (HD / 2)];
  if (tid == 0) sm.per_split = 1 << 30;
  __syncthreads();
  {
    int total = 0;
    for (int t = 0; t < T; ++t) total += sm.position[t] / GRANULE + 1;
    for (int per = max(WARPS, (total * a.kv_heads + ctas - 1) / ctas) + tid;; per += THREADS) {  // one split a pair always fits: ends
      int items = 0;
      for (int t = 0; t < T; ++t) items += (sm.position[t] / GRANULE + per) / per;
      const int fits = items * a.kv_heads <= ctas;
      if (fits) atomicMin(&sm.per_split, per);
      if (__syncthreads_or(fits)) break;
    }
  }
  if (tid == 0) {
    const int per = sm.per_split;
    int at = 0;
    sm.item_token = -1;
    sm.item_group = sm.item_first = sm.item_last = 0;
    for (int t = 0; t < T; ++t) {
      const int granules = sm.position[t] / GRANULE + 1, n = (granules + per - 1) / per;
      sm.item0[t] = at;
      sm.splits[t] = n;
      if (cta >= at && cta < at + n * a.kv_heads) {
        const int sp = (cta - at) % n;
        sm.item_token = t;
        sm.item_group = (cta - at) / n;
        // even shares: the splits of a request differ by a granule at most
        sm.item_first = (int)((long long)sp * granules / n);
        sm.item_last = (int)((long long)(sp + 1) * granules / n);
      }
      at += n * a.kv_heads;
    }
  }
  __syncthreads();
  auto row_of = [&](int granule) {  // of the cache: where a granule's first key lies
    const int key0 = granule * GRANULE;
    return __ldg(a.block_table + (size_t)sm.item_token * a.table_stride + key0 / a.page) * a.page + key0 % a.page;
  };
  if (lane == 0 && sm.item_first + warp < sm.item_last) sm.first_row[warp] = row_of(sm.item_first + warp);

  // ---- the grid barrier -----------------------------------------------------------------------------------
  // A word whose top bit turns with each completed barrier: CTA 0 adds 2^31 less the others' ones.
  auto arrive = [&]() {
    __syncthreads();
    if (tid == 0 && !*abort_flag) {
      const unsigned add = cta == 0 ? 0x80000000u - (unsigned)(ctas - 1) : 1u;
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(a.barrier), "r"(add) : "memory");
    }
  };
  auto wait = [&]() -> bool {  // false: give up
    if (tid == 0 && !*abort_flag) {
      sense ^= 0x80000000u;
      uint32_t i = 0;
#pragma unroll 1
      for (; i < BARRIER_LIMIT; ++i) {
        unsigned now;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(a.barrier) : "memory");
        if ((now & 0x80000000u) == sense) break;
        if ((i & 1023u) == 1023u && *reinterpret_cast<volatile int*>(a.status) == 2) i = BARRIER_LIMIT;
      }
      if (i >= BARRIER_LIMIT) *abort_flag = 1;
    }
    __syncthreads();
    return *abort_flag == 0;
  };

  // ---- parts of phases ----------------------------------------------------------------------------------------
  // Vectors into shared memory, by all warps but the one that waits at the barrier: the next norm's weight, the next q/k/v
  // tiles' bias.
  auto stage = [&](const float* gamma, const float* bias) {
    if (warp == 0) return;
#pragma unroll 1
    for (int i = tid - 32; i < H / 4; i += THREADS - 32) reinterpret_cast<float4*>(gamma_s)[i] = __ldg(reinterpret_cast<const float4*>(gamma) + i);
    if (bias) {
      const Share& s = sm.share[P_QKV];
#pragma unroll 1
      for (int i = tid - 32; i < 16 * s.tiles; i += THREADS - 32) {
        const int at = s.tile0 + (i >> 4) * s.tile_step;
        bias_s[i] = __ldg(bias + (at >> s.shift) * HD + (at & ((1 << s.shift) - 1)) * 8 + (i & 7) + (i & 8 ? HD / 2 : 0));
      }
    }
  };

  // A paced warp asks for its next pieces while the operand's loads are on their way: asked for behind the barrier, as many as
  // the ring has room for, they hold up the fences of the CTAs behind (4,100 cycles after gate and up, 1,100 to 1,500 this way; 0.5B
  // sizes, one and eight requests, us a pass of eight steps when both were measured: 5,031 and 5,658 that way, 4,747 and 5,430 with three
  // a phase).
  bool asked = false;
  auto ahead = [&]() {
    if (!asked && a.paced) refill(PACE);
    asked = true;
  };

  // The stream with what a sublayer added, for the next norm: between the arrival at a barrier and its end, by all warps but the one
  // that waits there.
  auto settle = [&](float* to, const float* base, const long long* acc, bool added) {
#pragma unroll 1
    for (int i = ((warp - 1) * ctas + cta) * 32 + lane; warp > 0 && i < T * H; i += (WARPS - 1) * ctas * 32) to[i] = stream_add(__ldcg(base + i), added ? __ldcg(acc + i) : 0);
  };
  auto clear = [&](long long* acc) {  // the numbers that this thread settled, once all have read them
#pragma unroll 1
    for (int i = ((warp - 1) * ctas + cta) * 32 + lane; warp > 0 && i < T * H; i += (WARPS - 1) * ctas * 32) acc[i] = 0;
  };

  // The rows of the stream times the norm's weight as bfloat16 into shared memory, and each row's factor.  (`added`: before the first
  // norm of a step nothing was.)
  auto normed_rows = [&](float eps, const float* base, const long long* acc, bool added) {
    const int per_row = WARPS >> t_bits, t = warp >> (4 - t_bits), part = warp & (per_row - 1);
    float square = 0.f;
    if (t < T) {
      const float2* b2 = reinterpret_cast<const float2*>(base + (size_t)t * H);
      const longlong2* a2 = reinterpret_cast<const longlong2*>(acc + (size_t)t * H);
      const float2* g2 = reinterpret_cast<const float2*>(gamma_s);
      unsigned char* row = work + (size_t)t * a.x_stride;
      const int n2 = H / 2, step = 32 * per_row;
#pragma unroll 1
      for (int w0 = part * 32; w0 < n2; w0 += 8 * step) {  // H is a multiple of 64: whole warps have an element or none
        longlong2 q[8];
        float2 b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          q[u] = make_longlong2(0, 0);
          b[u] = make_float2(0.f, 0.f);
          if (w0 + u * step < n2) {
            b[u] = __ldcg(b2 + w0 + u * step + lane);
            if (added) q[u] = __ldcg(a2 + w0 + u * step + lane);
          }
        }
        ahead();
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (w0 + u * step >= n2) break;
          const int i = w0 + u * step + lane;
          const float x = stream_add(b[u].x, q[u].x), y = stream_add(b[u].y, q[u].y);
          const float2 g = g2[i];
          square += x * x + y * y;
          *reinterpret_cast<uint32_t*>(row + 4 * i) = pack2(x * g.x, y * g.y);
        }
      }
    }
    square = warp_sum(square);
    if (lane == 0) sm.square[warp] = square;
    __syncthreads();
    if (tid < T) {
      float s = 0.f;
#pragma unroll 1
      for (int p = 0; p < per_row; ++p) s += sm.square[tid * per_row + p];
      sm.factor[tid] = rsqrtf(s / (float)H + eps);
    }
  };

  // This warp's pieces of a phase times the operand rows in `work`; the sums of each tile it touched into `sums`.
  auto multiply = [&](const Share& s, int phase) {
    const Part part = sm.part[phase][warp];
    if (part.first >= part.end) return;
    if (empty == a.slots) refill(a.slots);
    const int slices = s.slices;
    int tile = part.tile, slice = part.slice;
    float c[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[0][i] = c[1][i] = 0.f;
    const uint32_t x_lane = smem_u32(work) + min(lane & 7, T - 1) * a.x_stride + (lane >> 3) * 16;  // rows past the last: a sum that nobody reads
    const uint32_t w_half = ((lane >> 3) & 1) * 1024 + (lane & 7) * 128, w_k = lane >> 4, w_x = lane & 7;
#pragma unroll 1
    for (int left = part.end - part.first - 1; left >= 0; --left) {
      if (!__all_sync(0xffffffffu, mbar_wait(my_bars + slot, parity, abort_flag))) return;
      uint32_t w_at = my_ring + (uint32_t)slot * piece_bytes + w_half, x_at = slice * a.chunks * 128;
#pragma unroll 1
      for (int ch = 0; ch < a.chunks; ++ch, w_at += 2048, x_at += 128) {
        uint32_t b[2][4], w[4][4];
        ldsm4(b[0], x_lane + x_at);
        ldsm4(b[1], x_lane + x_at + 64);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) ldsm4(w[ks], w_at + ((((uint32_t)ks * 2 + w_k) ^ w_x) << 4));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma16816(c[ks & 1], w[ks][0], w[ks][1], w[ks][2], w[ks][3], b[ks >> 1][(ks & 1) * 2], b[ks >> 1][(ks & 1) * 2 + 1]);
      }
      __syncwarp();
      ++taken;
      ++empty;
      if (++slot == a.slots) {
        slot = 0;
        parity ^= 1;
      }
      if (left > a.slots - empty) refill(a.slots);  // this phase has pieces that nobody asked for yet; else behind the barrier
      if (++slice == slices || left == 0) {
        float* dst = sums + ((warp + tile) * 16 + r) * TP + 2 * j;
        *reinterpret_cast<float2*>(dst) = make_float2(c[0][0] + c[1][0], c[0][1] + c[1][1]);
        *reinterpret_cast<float2*>(dst + 8 * TP) = make_float2(c[0][2] + c[1][2], c[0][3] + c[1][3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) c[0][i] = c[1][i] = 0.f;
        slice = 0;
        ++tile;
      }
    }
  };

  stage(sm.layer[0].gamma_mixer, sm.layer[0].qkv_bias);
  __syncthreads();
#pragma unroll 1
  for (int layer = 0; layer < a.n_layers; ++layer) {
    const LayerVectors& L = sm.layer[layer & 1];
    const LayerVectors& N = sm.layer[(layer + 1) & 1];
    if (layer + 1 < a.n_layers) {
      const LayerVectors& next = table.layers[layer + 1].vectors;
      if (tid < (int)(sizeof(LayerVectors) / 4)) reinterpret_cast<int*>(&sm.layer[(layer + 1) & 1])[tid] = reinterpret_cast<const int*>(&next)[tid];
      if (cta == ctas - 1) {  // the next layer's vectors into L2
        for (int i = tid * 32; i < H; i += THREADS * 32) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next.gamma_mixer + i));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next.gamma_ff + i));
        }
        if (next.qkv_bias)
          for (int i = tid * 32; i < (a.heads + 2 * a.kv_heads) * HD; i += THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(next.qkv_bias + i));
      }
    }
#pragma unroll 1  // one copy of the product's loop, whose instructions then stay in the cache
    for (int phase = 0; phase < 4; ++phase) {
      place_thread();
      const Share& s = sm.share[phase];
      if (s.tiles) {
        asked = false;
        // the operand
        if (phase == P_QKV || phase == P_GATE) {
          const bool mixer = phase == P_QKV;
          normed_rows(mixer ? L.eps_mixer : L.eps_ff, mixer ? a.base : a.base_ff, mixer ? a.acc : a.acc_ff, !mixer || layer > 0 || a.added);
        } else {
          const int per_row = WARPS >> t_bits, t = warp >> (4 - t_bits), first = (warp & (per_row - 1)) * 32 + lane, step = 32 * per_row;
          const int cols = s.slices * a.chunks * 64, col0 = s.slice0 * a.chunks * 64;
          unsigned char* row = work + (size_t)t * a.x_stride;
          if (t >= T) {
          } else if (phase == P_OUT) {  // the merge of the key splits, even and odd ones by neighbouring lanes
            const int n = sm.splits[t], half = lane & 1;
#pragma unroll 1
            for (int i = first; i < cols / 2; i += step) {
              const int c = (i >> 1) * 4, head = (col0 + c) / HD, d = (col0 + c) % HD, g = (int)((head + 0.5f) * a.per_group);
              const size_t at = (size_t)(sm.item0[t] + g * n) * 8 + (head - g * group);
              float top = LOWEST, sum = 0.f;
              float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
              for (int p0 = half; p0 < n; p0 += 10) {
                float2 ml[5];
                float4 o[5];
#pragma unroll
                for (int u = 0; u < 5; ++u) {
                  ml[u] = make_float2(-INFINITY, 0.f);
                  o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                  if (p0 + 2 * u < n) {
                    const size_t p = at + (size_t)(p0 + 2 * u) * 8;
                    ml[u] = __ldcg(reinterpret_cast<const float2*>(a.part_ml) + p);
                    o[u] = __ldcg(reinterpret_cast<const float4*>(a.part_o + p * HD + d));
                  }
                }
                float up = top;
#pragma unroll
                for (int u = 0; u < 5; ++u) up = fmaxf(up, ml[u].x);
                const float f = exp2_fast(top - up);
                top = up;
                sum *= f;
                v.x *= f;
                v.y *= f;
                v.z *= f;
                v.w *= f;
#pragma unroll
                for (int u = 0; u < 5; ++u) {
                  if (p0 - half + 2 * u >= n) break;
                  const float w = exp2_fast(ml[u].x - up);
                  sum += w * ml[u].y;
                  v.x += w * o[u].x;
                  v.y += w * o[u].y;
                  v.z += w * o[u].z;
                  v.w += w * o[u].w;
                }
              }
              // the neighbour's half (cols / 2 is a multiple of 32: whole warps get here)
              const float top2 = __shfl_xor_sync(0xffffffffu, top, 1), up = fmaxf(top, top2), f = exp2_fast(top - up);
              sum *= f;
              v.x *= f;
              v.y *= f;
              v.z *= f;
              v.w *= f;
              sum += __shfl_xor_sync(0xffffffffu, sum, 1);
              v.x += __shfl_xor_sync(0xffffffffu, v.x, 1);
              v.y += __shfl_xor_sync(0xffffffffu, v.y, 1);
              v.z += __shfl_xor_sync(0xffffffffu, v.z, 1);
              v.w += __shfl_xor_sync(0xffffffffu, v.w, 1);
              const float q = 1.0f / sum;
              if (half == 0) *reinterpret_cast<uint2*>(row + 2 * c) = make_uint2(pack2(v.x * q, v.y * q), pack2(v.z * q, v.w * q));
            }
          } else {
            const int n = cols / 8, tile0 = col0 / 8;
#pragma unroll 1
            for (int i0 = first; i0 < n; i0 += 4 * step) {
              uint4 v[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                v[u] = make_uint4(0u, 0u, 0u, 0u);
                if (i0 - lane + u * step >= n) continue;
                const int tile = tile0 + i0 + u * step, k = (int)((tile + 0.5f) * a.per_cta), c = tile - k * ctas;  // of the gate product: its CTA, and which of that one's
                if (i0 + u * step < n) v[u] = __ldcg(reinterpret_cast<const uint4*>(a.act + (size_t)c * a.act_stride) + k * T + t);
              }
              ahead();
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (i0 + u * step < n) *reinterpret_cast<uint4*>(row + 16 * (i0 + u * step)) = v[u];
            }
          }
          __syncthreads();
        }
        if (phase != P_OUT) ahead();  // a warp that had nothing to load
        multiply(s, phase);
        __syncthreads();
        // what becomes of the sums
        const int rows = phase == P_QKV || phase == P_GATE ? 3 : 4, items = s.tiles << (rows + t_bits);  // 8 pairs of rows a tile, or 16 rows
#pragma unroll 1
        for (int i = tid; i - lane < items; i += THREADS) {  // whole warps: eight lanes put their numbers together
          const int e = i & ((1 << rows) - 1), t = (i >> rows) & t_mask, tile = i >> (rows + t_bits);
          const bool live = i < items && t < T;
          float x = 0.f, y = 0.f;
          int at = 0;
          if (live) {
            const int first = sm.first_warp[phase][tile], last = sm.last_warp[phase][tile];
            const float* from = sums + ((first + tile) * 16 + e) * TP + t;
            at = s.tile0 + tile * s.tile_step;
#pragma unroll 1
            for (int w = first; w <= last; ++w, from += 16 * TP) {
              x += from[0];
              if (rows == 3) y += from[8 * TP];
            }
            if (rows == 4)  // into the stream
              atomicAdd(reinterpret_cast<unsigned long long*>(phase == P_OUT ? a.acc_ff : a.acc) + (size_t)t * H + at * 16 + e, (unsigned long long)__float2ll_rn(x * STREAM_SCALE));
          }
          if (rows == 4) continue;
          bf16* dst = nullptr;
          if (live) {
            x *= sm.factor[t];
            y *= sm.factor[t];
            if (phase == P_GATE) {
              x = silu_times(x, y);
              dst = a.act + (size_t)s.tile0 * a.act_stride + (tile * T + t) * 8;
            } else {
              const int head = at >> s.shift, d = (at & ((1 << s.shift) - 1)) * 8 + e, kv = head - a.heads;
              if (L.qkv_bias) {
                x += bias_s[tile * 16 + e];
                y += bias_s[tile * 16 + 8 + e];
              }
              if (head < a.heads + a.kv_heads) {
                const float2 cs = turn[t * (HD / 2) + d];
                const float u = x * cs.x - y * cs.y;
                y = y * cs.x + x * cs.y;
                x = u;
              }
              if (kv < 0) dst = a.q + ((size_t)t * a.heads + head) * HD + d;
              else if (sm.slot[t] >= 0) dst = (kv < a.kv_heads ? L.k + ((size_t)sm.slot[t] * a.kv_heads + kv) * HD : L.v + ((size_t)sm.slot[t] * a.kv_heads + kv - a.kv_heads) * HD) + d;
            }
          }
          // 16 bytes a store: the fence behind them is the shorter
          uint4 v;
          v.x = pack2(x, __shfl_down_sync(0xffffffffu, x, 1));
          v.y = __shfl_down_sync(0xffffffffu, v.x, 2);
          v.z = __shfl_down_sync(0xffffffffu, v.x, 4);
          v.w = __shfl_down_sync(0xffffffffu, v.y, 4);
          if (dst && e == 0) *reinterpret_cast<uint4*>(dst) = v;
          if (phase == P_GATE) continue;
          v.x = pack2(y, __shfl_down_sync(0xffffffffu, y, 1));
          v.y = __shfl_down_sync(0xffffffffu, v.x, 2);
          v.z = __shfl_down_sync(0xffffffffu, v.x, 4);
          v.w = __shfl_down_sync(0xffffffffu, v.y, 4);
          if (dst && e == 0) *reinterpret_cast<uint4*>(dst + HD / 2) = v;
        }
      }
      if (phase == P_DOWN && layer + 1 == a.n_layers) break;
      arrive();
      if (phase != P_QKV) {
        if (!a.paced) refill(a.slots);
        if (phase == P_OUT) stage(L.gamma_ff, nullptr);
        if (phase == P_GATE) settle(a.base, a.base_ff, a.acc_ff, true);
        if (phase == P_DOWN) stage(N.gamma_mixer, N.qkv_bias);
        if (!wait()) goto leave;
        if (phase == P_GATE) clear(a.acc_ff);
        continue;
      }

      // ---- attention ------------------------------------------------------------------------------------------
      // Scores are K Q^T (16 keys x 8 heads) and outputs V^T P^T (HD x 8 heads), so that a group of up to eight heads
      // fills the 8-wide operand.  The order of the head's dimensions inside the products is free: a thread reads 16
      // bytes of a key's row and uses them as the operand's registers of two k-steps.
      {
        const int it_token = sm.item_token, it_group = sm.item_group, it_last = sm.item_last;
        const int my_first = sm.item_first + warp;  // this warp's granules: my_first, my_first + WARPS, ...
        const int it_pos = it_token >= 0 ? sm.position[it_token] : 0, last_granule = it_pos / GRANULE;
        const bool has_keys = my_first < it_last;
        uint4 kr[C32][2] = {}, vr[C32][2] = {};
        auto load_rows = [&](uint4 (&to)[C32][2], const bf16* cache, int row0) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const size_t at = ((size_t)(row0 + r + 8 * h) * a.kv_heads + it_group) * HD + 8 * j;
#pragma unroll
            for (int c = 0; c < C32; ++c) to[c][h] = __ldcg(reinterpret_cast<const uint4*>(cache + at + 32 * c));
          }
        };
        // the first keys are on their way before the barrier; the row that phase 1 may be writing is read again after it
        if (has_keys) {
          load_rows(kr, L.k, sm.first_row[warp]);
          if (HD <= 64) {
            load_rows(vr, L.v, sm.first_row[warp]);
          } else {  // keys, values, outputs: more than the registers hold
            asm volatile("prefetch.global.L2 [%0];" ::"l"(L.v + ((size_t)(sm.first_row[warp] + (lane & 15)) * a.kv_heads + it_group) * HD + (lane >> 4) * 64));
          }
        }
        if (!a.paced) refill(a.slots);
        settle(a.base_ff, a.base, a.acc, layer > 0 || a.added);
        if (!wait()) goto leave;
        if (layer > 0 || a.added) clear(a.acc);
        if (it_token >= 0) {
          float m0 = LOWEST, m1 = LOWEST, l0 = 0.f, l1 = 0.f;  // of heads 2j and 2j + 1 of the group
          float o[HD / 16][4];
#pragma unroll
          for (int i = 0; i < HD / 16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
          if (has_keys) {
#pragma unroll 1
            for (int granule = my_first; granule < it_last; granule += WARPS) {
              const int key = granule * GRANULE + r;
              uint4 qr[C32];
#pragma unroll
              for (int c = 0; c < C32; ++c) qr[c] = __ldcg(reinterpret_cast<const uint4*>(a.q + ((size_t)it_token * a.heads + it_group * group + min(r, group - 1)) * HD + 32 * c + 8 * j));
              int row0 = sm.first_row[warp];
              if (granule != my_first) {
                row0 = row_of(granule);
                load_rows(kr, L.k, row0);
                if (HD <= 64) load_rows(vr, L.v, row0);
              } else if (granule == last_granule) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                  if (key + 8 * h == it_pos) {
                    const size_t at = ((size_t)(row0 + r + 8 * h) * a.kv_heads + it_group) * HD + 8 * j;
#pragma unroll
                    for (int c = 0; c < C32; ++c) {
                      kr[c][h] = __ldcg(reinterpret_cast<const uint4*>(L.k + at + 32 * c));
                      if (HD <= 64) vr[c][h] = __ldcg(reinterpret_cast<const uint4*>(L.v + at + 32 * c));
                    }
                  }
              }
              float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
              for (int c = 0; c < C32; ++c) {
                mma16816(s, kr[c][0].x, kr[c][1].x, kr[c][0].y, kr[c][1].y, qr[c].x, qr[c].y);
                mma16816(s, kr[c][0].z, kr[c][1].z, kr[c][0].w, kr[c][1].w, qr[c].z, qr[c].w);
              }
              if (HD > 64) load_rows(vr, L.v, row0);
#pragma unroll
              for (int i = 0; i < 4; ++i) s[i] *= a.scale;
              if (granule == last_granule) {  // keys behind the query's position are another request's leavings
                if (key > it_pos) s[0] = s[1] = -INFINITY;
                if (key + 8 > it_pos) s[2] = s[3] = -INFINITY;
#pragma unroll
                for (int c = 0; c < C32; ++c) {
                  if (key > it_pos) vr[c][0] = make_uint4(0u, 0u, 0u, 0u);
                  if (key + 8 > it_pos) vr[c][1] = make_uint4(0u, 0u, 0u, 0u);
                }
              }
              float n0 = fmaxf(s[0], s[2]), n1 = fmaxf(s[1], s[3]);
#pragma unroll
              for (int x = 4; x < 32; x *= 2) {
                n0 = fmaxf(n0, __shfl_xor_sync(0xffffffffu, n0, x));
                n1 = fmaxf(n1, __shfl_xor_sync(0xffffffffu, n1, x));
              }
              n0 = fmaxf(n0, m0);
              n1 = fmaxf(n1, m1);
              const float f0 = exp2_fast(m0 - n0), f1 = exp2_fast(m1 - n1);
              m0 = n0;
              m1 = n1;
              s[0] = exp2_fast(s[0] - n0);
              s[1] = exp2_fast(s[1] - n1);
              s[2] = exp2_fast(s[2] - n0);
              s[3] = exp2_fast(s[3] - n1);
              l0 = l0 * f0 + s[0] + s[2];
              l1 = l1 * f1 + s[1] + s[3];
              const uint32_t p0 = transposed(pack2(s[0], s[1])), p1 = transposed(pack2(s[2], s[3]));
#pragma unroll
              for (int i = 0; i < HD / 16; ++i) {
                o[i][0] *= f0;
                o[i][1] *= f1;
                o[i][2] *= f0;
                o[i][3] *= f1;
              }
#pragma unroll
              for (int c = 0; c < C32; ++c) {
                mma16816(o[2 * c], transposed(vr[c][0].x), transposed(vr[c][0].y), transposed(vr[c][1].x), transposed(vr[c][1].y), p0, p1);
                mma16816(o[2 * c + 1], transposed(vr[c][0].z), transposed(vr[c][0].w), transposed(vr[c][1].z), transposed(vr[c][1].w), p0, p1);
              }
            }
#pragma unroll
            for (int x = 4; x < 32; x *= 2) {
              l0 += __shfl_xor_sync(0xffffffffu, l0, x);
              l1 += __shfl_xor_sync(0xffffffffu, l1, x);
            }
          }
          // The warps' outputs are merged through shared memory: the second half of the warps into the first by pairs, then all
          // of these at once, each with its own maximum.
          const int used = min(WARPS, it_last - sm.item_first);  // warps with keys
          constexpr int SETS = WARPS / 2, ROW = HD + 1;
          auto place = [&](int i, int half) { return 32 * (i >> 1) + 8 * (r >> 1) + 2 * (2 * (i & 1) + half) + (r & 1); };
          float* set = osm + (warp & (SETS - 1)) * 8 * ROW + 2 * j * ROW;
          if (warp >= SETS && warp < used) {
#pragma unroll
            for (int i = 0; i < HD / 16; ++i) {
              set[place(i, 0)] = o[i][0];
              set[ROW + place(i, 0)] = o[i][1];
              set[place(i, 1)] = o[i][2];
              set[ROW + place(i, 1)] = o[i][3];
            }
            if (r == 0) {
              *reinterpret_cast<float2*>(&sm.wm[warp][2 * j]) = make_float2(m0, m1);
              *reinterpret_cast<float2*>(&sm.wl[warp][2 * j]) = make_float2(l0, l1);
            }
          }
          if (used > SETS) __syncthreads();
          if (warp < SETS && warp < used) {  // a warp's own set is read and written by that warp alone
            if (warp + SETS < used) {
              const float2 m = *reinterpret_cast<const float2*>(&sm.wm[warp + SETS][2 * j]), l = *reinterpret_cast<const float2*>(&sm.wl[warp + SETS][2 * j]);
              const float n0 = fmaxf(m0, m.x), n1 = fmaxf(m1, m.y);
              const float f0 = exp2_fast(m0 - n0), f1 = exp2_fast(m1 - n1), g0 = exp2_fast(m.x - n0), g1 = exp2_fast(m.y - n1);
              m0 = n0;
              m1 = n1;
              l0 = l0 * f0 + l.x * g0;
              l1 = l1 * f1 + l.y * g1;
#pragma unroll
              for (int i = 0; i < HD / 16; ++i) {
                o[i][0] = o[i][0] * f0 + set[place(i, 0)] * g0;
                o[i][1] = o[i][1] * f1 + set[ROW + place(i, 0)] * g1;
                o[i][2] = o[i][2] * f0 + set[place(i, 1)] * g0;
                o[i][3] = o[i][3] * f1 + set[ROW + place(i, 1)] * g1;
              }
            }
#pragma unroll
            for (int i = 0; i < HD / 16; ++i) {
              set[place(i, 0)] = o[i][0];
              set[ROW + place(i, 0)] = o[i][1];
              set[place(i, 1)] = o[i][2];
              set[ROW + place(i, 1)] = o[i][3];
            }
            if (r == 0) {
              *reinterpret_cast<float2*>(&sm.wm[warp][2 * j]) = make_float2(m0, m1);
              *reinterpret_cast<float2*>(&sm.wl[warp][2 * j]) = make_float2(l0, l1);
            }
          }
          __syncthreads();
          const int sets = min(SETS, used);
#pragma unroll 1
          for (int i = tid; i < group * HD; i += THREADS) {
            const int h = i / HD, d = i % HD;
            float m[SETS], top = sm.wm[0][h], v = 0.f, sum = 0.f;
#pragma unroll
            for (int w = 0; w < SETS; ++w) {
              m[w] = -INFINITY;
              if (w < sets) m[w] = sm.wm[w][h];
              top = fmaxf(top, m[w]);
            }
#pragma unroll
            for (int w = 0; w < SETS; ++w)
              if (w < sets) {
                const float f = exp2_fast(m[w] - top);
                v += osm[(w * 8 + h) * ROW + d] * f;
                sum += sm.wl[w][h] * f;
              }
            a.part_o[((size_t)cta * 8 + h) * HD + d] = v;
            if (d == 0) *reinterpret_cast<float2*>(a.part_ml + ((size_t)cta * 8 + h) * 2) = make_float2(top, sum);
          }
        }
        arrive();
        if (!wait()) goto leave;
      }
    }
  }
leave:

  // Copies still in flight (after a wait that ran out) land before this CTA leaves.
  __syncwarp();
#pragma unroll 1
  for (int left = sm.loader[warp].asked - taken; left > 0; --left) {
#pragma unroll 1
    for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try_wait(my_bars + slot, parity); ++i) {
    }
    if (++slot == a.slots) {
      slot = 0;
      parity ^= 1;
    }
  }
  __syncthreads();
  if (tid == 0 && *abort_flag) *reinterpret_cast<volatile int*>(a.status) = 2;
}

// ---------------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------------
namespace {

// A [rows, 64 * n] bf16 row-major matrix as boxes of 8 rows, 8 rows `second` further on, and `chunks` x 64 columns; 128-byte swizzle.
bool make_piece_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t second, int chunks) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {64, (cuuint64_t)(rows - second), 2, (cuuint64_t)(cols / 64)};
  cuuint64_t strides[3] = {(cuuint64_t)cols * 2, (cuuint64_t)(second * cols * 2), 128};
  cuuint32_t box[4] = {64, 8, 2, (cuuint32_t)chunks};
  cuuint32_t elem[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int SMEM_LIMIT = 232448;  // bytes a CTA may have

// Sizes that the kernel is written for (whether their shares and rings fit is plan_stack's to say).
bool sizes_fit(int tokens, int hidden, int heads, int kv_heads, int head_dim, int inter) {
  if (tokens < 1 || tokens > MAX_TOKENS || hidden < 64 || hidden % 64 || inter < 64 || inter % 64 || kv_heads < 1 || heads < 1 || heads % kv_heads || heads / kv_heads > 8) return false;
  // (far more than fits; below it no product of sizes leaves 32 bits)
  return (head_dim == 64 || head_dim == 128) && hidden <= 1 << 16 && inter <= 1 << 19 && heads <= 1 << 10;
}

typedef void (*StackKernel)(const StackArgs, const StackTable);
StackKernel kernel_of(int head_dim) {
  return head_dim == 64 ? (StackKernel)decode_stack_kernel<64> : head_dim == 128 ? (StackKernel)decode_stack_kernel<128> : nullptr;
}

// Ranges of slices and tiles over the CTAs for a projection whose parts are added into the stream: the fewest bytes for the
// busiest CTA, its operand (`operand` bytes a token and column) and its atomic adds (as if 16 bytes each) counted beside its weights.
void split_plan(PhasePlan* p, int ctas, int chunks, int tokens, int operand, int x_limit) {
  long long best = -1;
  for (int kg = 1; kg <= p->slices && kg <= ctas; ++kg) {
    const int rg = ctas / kg < p->tiles ? ctas / kg : p->tiles;
    const long long tiles = (p->tiles + rg - 1) / rg, slices = (p->slices + kg - 1) / kg, cols = slices * chunks * 64;
    if (cols > x_limit || tiles > 24) continue;
    const long long cost = tiles * slices * 2048 * chunks + cols * tokens * operand + tiles * 16 * tokens * 16 + (long long)kg * 32 * p->tiles;
    if (best < 0 || cost < best) {
      best = cost;
      p->kg = kg;
      p->rg = rg;
    }
  }
}

// Everything of the launch that goes by the sizes: the shares, shared memory, the ring.  0: the kernel does not take them.
size_t plan_stack(StackArgs* a, int head_dim, int ctas) {
  const int T = a->tokens, H = a->hidden, q_dim = a->heads * head_dim, F = a->inter;
  a->chunks = (H / 64) % 2 || (q_dim / 64) % 2 || (F / 64) % 2 ? 1 : 2;
  const int cols = a->chunks * 64;
  a->plan[P_QKV] = {(q_dim + 2 * a->kv_heads * head_dim) / 16, H / cols, 0, 0};
  a->plan[P_GATE] = {F / 8, H / cols, 0, 0};
  a->plan[P_OUT] = {H / 16, q_dim / cols, 0, 0};
  a->plan[P_DOWN] = {H / 16, F / cols, 0, 0};
  const int x_limit = H > 512 ? H : 512;  // columns of an operand row
  split_plan(&a->plan[P_OUT], ctas, a->chunks, T, 4 * 8, x_limit);
  split_plan(&a->plan[P_DOWN], ctas, a->chunks, T, 2, x_limit);
  if (!a->plan[P_OUT].kg || !a->plan[P_DOWN].kg) return 0;
  int most = 0, wide = H;
  for (int p = 0; p < 4; ++p) {
    const PhasePlan& s = a->plan[p];
    const int tiles = s.kg ? (s.tiles + s.rg - 1) / s.rg : (s.tiles + ctas - 1) / ctas;
    most = tiles > most ? tiles : most;
    if (s.kg) {
      const int w = (s.slices + s.kg - 1) / s.kg * cols;
      wide = w > wide ? w : wide;
    }
  }
  if (most > MAX_TILES) return 0;
  for (int p = 0; p < 4; ++p) {  // pieces of a CTA are counted in 16 bits
    const PhasePlan& s = a->plan[p];
    const int tiles = s.kg ? (s.tiles + s.rg - 1) / s.rg : (s.tiles + ctas - 1) / ctas, slices = s.kg ? (s.slices + s.kg - 1) / s.kg : s.slices;
    if ((long long)tiles * slices > 32767) return 0;
  }
  a->act_stride = ((a->plan[P_GATE].tiles + ctas - 1) / ctas * T * 8 + 63) / 64 * 64;
  a->x_stride = 2 * wide + 16;
  a->x_bytes = T * a->x_stride;
  a->qkv_tiles = (a->plan[P_QKV].tiles + ctas - 1) / ctas;
  const int sums = (most + WARPS) * 16 * MAX_TOKENS * 4, merge = WARPS / 2 * 8 * (head_dim + 1) * 4;
  a->work_bytes = a->x_bytes + sums > merge ? a->x_bytes + sums : merge;
  a->work_bytes = (a->work_bytes + 15) / 16 * 16;
  const size_t rest = (size_t)a->work_bytes + (size_t)T * head_dim * 4 + (size_t)H * 4 + 64 * (size_t)a->qkv_tiles + sizeof(Small) + 64;
  const size_t limit = SMEM_LIMIT, piece = (size_t)WARPS * (2048 * a->chunks + 8);
  if (rest + 2 * piece > limit) return 0;
  a->slots = (int)((limit - rest) / piece);
  if (a->slots > 8) a->slots = 8;
  long long all = 0;
  for (int p = 0; p < 4; ++p) all += (long long)a->plan[p].tiles * a->plan[p].slices;
  // a ring that holds half a layer or more keeps up at that pace; larger models are bound by their weights (7B sizes: a layer is 24
  // rings) and ask for all they can as soon as they can
  a->paced = all <= 2 * (long long)ctas * WARPS * a->slots;
  return rest + a->slots * piece;
}

}  // namespace

ALOFA_API int alofa_decode_stack_layer_bytes() { return (int)sizeof(StackLayer); }

// What plan_stack decides, for a look from outside: out[0..15] the phases' tiles, slices, ranges of slices and of tiles, then chunks,
// pieces in a ring, an operand row's bytes, the operand's and the work area's, all shared memory, whether it is paced.  0: sizes the kernel does not take.
ALOFA_API int alofa_decode_stack_plan(int tokens, int hidden, int heads, int kv_heads, int head_dim, int inter, int ctas, int* out) {
  memset(out, 0, 23 * sizeof(int));
  if (ctas < 1 || !sizes_fit(tokens, hidden, heads, kv_heads, head_dim, inter)) return 0;
  StackArgs a = {};
  a.tokens = tokens;
  a.hidden = hidden;
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.group = heads / kv_heads;
  a.inter = inter;
  const size_t smem = plan_stack(&a, head_dim, ctas);
  memcpy(out, a.plan, sizeof(a.plan));
  const int rest[7] = {a.chunks, a.slots, a.x_stride, a.x_bytes, a.work_bytes, (int)smem, a.paced};
  memcpy(out + 16, rest, sizeof(rest));
  return smem > 0;
}

// How many CTAs run a step of these sizes: one per SM, all resident together; 0 where the kernel does not take them.
ALOFA_API int alofa_decode_stack_ctas(int tokens, int hidden, int heads, int kv_heads, int head_dim, int inter, int page) {
  if (!sizes_fit(tokens, hidden, heads, kv_heads, head_dim, inter) || page % GRANULE || page < GRANULE) return 0;
  StackKernel kernel = kernel_of(head_dim);
  int device, sms, coop;
  if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop)
    return 0;
  if (tokens * kv_heads > sms) return 0;
  StackArgs a = {};
  a.tokens = tokens;
  a.hidden = hidden;
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.group = heads / kv_heads;
  a.inter = inter;
  const size_t smem = plan_stack(&a, head_dim, sms);
  if (!smem || cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess) return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, THREADS, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  return sms;
}

// Fills one layer's entry of the table that a launch takes (host memory).
ALOFA_API int alofa_decode_stack_layer(void* entry, const void* qkv, const void* out, const void* gate_up, const void* down, const float* gamma_mixer,
                                       const float* gamma_ff, const float* qkv_bias, void* k, void* v, float eps_mixer, float eps_ff, int hidden, int heads,
                                       int kv_heads, int head_dim, int inter) {
  if (!entry || !qkv || !out || !gate_up || !down || !gamma_mixer || !gamma_ff || !k || !v || !sizes_fit(1, hidden, heads, kv_heads, head_dim, inter)) return ALOFA_ERR_ARGUMENT;
  StackLayer L;
  memset(&L, 0, sizeof(L));
  const int q_dim = heads * head_dim, chunks = (hidden / 64) % 2 || (q_dim / 64) % 2 || (inter / 64) % 2 ? 1 : 2;
  if (((uintptr_t)qkv | (uintptr_t)out | (uintptr_t)gate_up | (uintptr_t)down | (uintptr_t)gamma_mixer | (uintptr_t)gamma_ff | (uintptr_t)k | (uintptr_t)v) & 15) return ALOFA_ERR_ARGUMENT;
  if (!make_piece_map(&L.maps[P_QKV], qkv, q_dim + 2 * kv_heads * head_dim, hidden, head_dim / 2, chunks) || !make_piece_map(&L.maps[P_OUT], out, hidden, q_dim, 8, chunks) ||
      !make_piece_map(&L.maps[P_GATE], gate_up, 2 * (uint64_t)inter, hidden, inter, chunks) || !make_piece_map(&L.maps[P_DOWN], down, hidden, inter, 8, chunks))
    return ALOFA_ERR_LAUNCH;
  L.vectors.gamma_mixer = gamma_mixer;
  L.vectors.gamma_ff = gamma_ff;
  L.vectors.qkv_bias = qkv_bias;
  L.vectors.k = (bf16*)k;
  L.vectors.v = (bf16*)v;
  L.vectors.eps_mixer = eps_mixer;
  L.vectors.eps_ff = eps_ff;
  memcpy(entry, &L, sizeof(L));
  return ALOFA_OK;
}

// `layers`: the entries of alofa_decode_stack_layer one after the other, in host memory.
ALOFA_API int alofa_decode_stack(const void* layers, int n_layers, int ctas, int tokens, int hidden, int heads, int kv_heads, int head_dim, int inter, int page,
                                 int table_stride, float scale, float* base, float* base_ff, long long* acc, long long* acc_ff, const int* positions, const int* block_table,
                                 const int* slot_map, const float* rope, void* q, float* part_o, float* part_ml, void* act, unsigned* barrier, int* status,
                                 cudaStream_t stream) {
  StackKernel kernel = kernel_of(head_dim);
  if (!sizes_fit(tokens, hidden, heads, kv_heads, head_dim, inter) || page % GRANULE || page < GRANULE || n_layers < 1 || table_stride < 1 || ctas < 1 || tokens * kv_heads > ctas) return ALOFA_ERR_ARGUMENT;
  StackArgs a = {};
  a.tokens = tokens;
  a.hidden = hidden;
  a.heads = heads;
  a.kv_heads = kv_heads;
  a.group = heads / kv_heads;
  a.inter = inter;
  a.page = page;
  a.table_stride = table_stride;
  a.scale = scale * 1.4426950408889634f;
  a.base = base;
  a.base_ff = base_ff;
  a.acc = acc;
  a.acc_ff = acc_ff;
  a.positions = positions;
  a.block_table = block_table;
  a.slot_map = slot_map;
  a.rope = rope;
  a.q = (bf16*)q;
  a.part_o = part_o;
  a.part_ml = part_ml;
  a.act = (bf16*)act;
  a.barrier = barrier;
  a.status = status;
  a.per_group = 1.0f / (float)a.group;
  a.per_cta = 1.0f / (float)ctas;
  const size_t smem = plan_stack(&a, head_dim, ctas);
  if (!smem) return ALOFA_ERR_ARGUMENT;
  // always the most there is: a size of its own for each step could come between another thread's setting and its launch
  if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess) return ALOFA_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  for (int first = 0; first < n_layers; first += MAX_LAYERS) {
    StackTable table;
    a.n_layers = n_layers - first < MAX_LAYERS ? n_layers - first : MAX_LAYERS;
    a.added = first > 0;
    memcpy(&table, (const char*)layers + first * sizeof(StackLayer), a.n_layers * sizeof(StackLayer));
    memset((char*)&table + a.n_layers * sizeof(StackLayer), 0, sizeof(table) - a.n_layers * sizeof(StackLayer));
    if (cudaLaunchKernelEx(&cfg, kernel, a, table) != cudaSuccess) {
      cudaGetLastError();
      return ALOFA_ERR_LAUNCH;
    }
  }
  return ALOFA_OK;
}
