// b2_keyed.cuh — one pass for keys that do not pack into 64 bits (a STRING column, floats, wide composites): a row's key is
// looked up in a dictionary, and its values are folded into accumulators that the key's id addresses.
//
// Serves what compute_mapping_indices.cuh:92-151 and compute_shared_memory_aggs.cu:260-353 do with a set of row indices whose
// probes compare whole rows.  Against a table of row indices (k_aggregate<KM_ROWS>):
//   * a probe compares a 30-bit tag and a length in the cell, then one 32-byte entry, and never the row that brought the key
//     (longer strings aside);
//   * a CTA holds accumulators in shared memory for up to `slots` ids, one probe each: the first id to come by takes the slot (its id
//     modulo `slots`), so that a frequent one has its place in nearly every CTA; the others are global words, dense by id.  (Slots for
//     the lowest ids, those that arrived first, left frequent ones out: all CTAs start at once, and what came by among the first
//     190K rows is in no particular order.  11M Zipf rows over 1000 strings, twelve cells: 4 to 17 ms per call
//     with those, 0.92 with these);
//   * whoever takes an id takes the place of its string in the result's chars with the same atomic, so that the STRING column of
//     the result needs no scan, and writes the accumulators' identities, so that nothing is initialised for ids that are not
//     there;
//   * a finished id is an output row: nothing is compacted.
// What bounds it is latency: a row is looked up behind the one before it, 950 instructions per row and warp with STRING and with
// 96-bit keys, L2 31 and 53 % busy, 44 and 42 % of the stalls for loads.
// (L2 takes the lanes of one atomic that meet in a sector as one request, but sharing a row's words out among lanes cost more
// instructions than it saved: 4M rows, 30K groups, six cells 344 -> 386 us per call.  Prefetching the next tile: no difference.)
// 1M rows over 50K strings, count / min / max / sum of INT32: 311 -> 131 us per call.  640 threads, two CTAs per SM: beside 512 x 2
// (64 registers, no spills) and 384 x 3, with slots for the lowest ids, 8M rows / 1000 strings 278, 311 and 297 us; with 5 x 256 the accumulators of a thousand
// groups lie half outside of shared memory, whose few lines of L2 then queue (16M rows, 1000 groups 1164 us, 627 with 2 x 640).
#pragma once
#include "b2_kernels.cuh"

namespace b2 {

constexpr int KEYED_BLOCK = 640;
constexpr int KEYED_CTAS  = 2;    // per SM
constexpr int KEYED_ROWS  = 4;    // rows per thread and tile at most
constexpr int KEYED_SLOTS = 2048; // per CTA at most
constexpr int KEYED_CHARS = 38;   // bits of the number of chars in the counter of ids: no device holds 2^38 bytes
constexpr u64 KEYED_CHARS_MASK = (1ull << KEYED_CHARS) - 1ull;
static_assert(KEYED_CHARS + 26 == 64, "ids of 26 bits");

struct DKeyed {
  DDict dict;          // (pool_cap: ids there can be)
  u64* more;           // [pool_cap] the key's fixed-width part beside a string (nullptr: a string alone, or no string)
  i64* char_at;        // strings: [pool_cap] first output byte
  u64* acc;            // [pool_cap][ncells] accumulators, in the form of keyed_addend
  int string;          // key column that is the string, -1: none
  int slots;           // ids whose accumulators a CTA has room for in shared memory
  int each;            // rows per thread and tile
  int smem;            // bytes of those accumulators
  int zeros;           // every accumulator starts from zero (keyed_none)
  DDictKeys form;      // where a key's fixed-width part lies
  unsigned short cell_at[MAX_CELLS];  // byte offset / 16 of every cell's array in shared memory
};

// cells empty, control block zero
__global__ void __launch_bounds__(256) k_keyed_init(u64* __restrict__ cells, i64 cap, DCtrl* ctrl)
{
  grid_dependents_launch();
  if (blockIdx.x == 0) for (u32 i = threadIdx.x; i < (u32)(sizeof(DCtrl) / 4); i += blockDim.x) ((u32*)ctrl)[i] = 0;
  for (i64 i = ((i64)blockIdx.x * blockDim.x + threadIdx.x) * 2; i < cap; i += (i64)gridDim.x * blockDim.x * 2)
    *(ulonglong2*)(cells + i) = make_ulonglong2(EMPTY, EMPTY);  // (cap is a power of two)
}

// Accumulators are of three kinds — sums and counts, sums of doubles, maxima of order-preserving images (complements for a
// minimum) — each of which starts from zero and is updated by one instruction.  (With a case for every operator and row the kernel
// did not fit the instruction cache: 28 % of the stalls.)
enum KeyedAdds : unsigned char { KA_INT, KA_FLOAT, KA_MAX, KA_OTHER };
__host__ __device__ __forceinline__ int keyed_adds(int op)
{
  switch (op) {
    case OP_SUM_I: case OP_SSQ_I: case OP_CNT_V: case OP_CNT_A: case OP_SUM_HI: case OP_SUM_LO: case OP_SUM_HIU: return KA_INT;
    case OP_SUM_F: case OP_SSQ_F: return KA_FLOAT;
    case OP_MIN_I: case OP_MIN_U: case OP_MIN_F: case OP_MAX_I: case OP_MAX_U: case OP_MAX_F: return KA_MAX;
    default: return KA_OTHER;  // (not served)
  }
}
__device__ __forceinline__ u64 keyed_flip(int op)
{
  return (op == OP_MIN_I || op == OP_MAX_I ? 1ull << 63 : 0ull) ^ (op == OP_MIN_I || op == OP_MIN_U || op == OP_MIN_F ? ~0ull : 0ull);
}
// what a value adds to its cell's accumulator
__device__ __forceinline__ u64 keyed_addend(int op, int adds, u64 v)
{
  if (adds == KA_MAX) return (op == OP_MIN_F || op == OP_MAX_F ? f64_ordered(v) : v) ^ keyed_flip(op);
  if (adds == KA_FLOAT) {
    const double d = __longlong_as_double((i64)v);
    return op == OP_SUM_F ? v : (u64)__double_as_longlong(d * d);
  }
  return op == OP_SUM_I ? v : op == OP_CNT_V || op == OP_CNT_A ? 1ull : sum_addend(op, v);
}
// (as reductions of global memory: through a pointer out of a parameter's structure the compiler makes generic atomics, which
// return what nobody asked for)
__device__ __forceinline__ void keyed_update(u64* p, int adds, u64 x)
{
  const u64 a = __cvta_generic_to_global(p);
  if (adds == KA_INT) asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" :: "l"(a), "l"(x) : "memory");
  else if (adds == KA_FLOAT) asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" :: "l"(a), "d"(__longlong_as_double((i64)x)) : "memory");
  else asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" :: "l"(a), "l"(x) : "memory");
}
// What an accumulator starts from: nothing, or, where shared memory keeps the cell as a 32-bit image and no value is null, what the
// image's zero stands for (the group then has a value, and none lies further out).
__device__ __forceinline__ u64 keyed_none(const DPlan& P, const DForms& F, int c)
{
  const bool narrow = F.count_of[c] < 0 && (F.form[c] == CF_MIN32 || F.form[c] == CF_MAX32);
  return narrow ? unorder32(F.kind[P.cells[c].col], F.form[c] == CF_MIN32 ? 0xFFFFFFFFu : 0u) ^ keyed_flip(P.cells[c].op) : 0ull;
}

// a key's fixed-width columns, side by side; null flags behind them
__device__ __forceinline__ void keyed_bits(const DPlan& P, const DKeyed& K, i64 row, u64 (&w)[4])
{
  for (int i = 0; i < P.nkeys; ++i) {
    const DKeyCol& kc = P.keys[i];
    const int null_at = K.form.null_at[i];
    u64 x;
    int bit;
    if (null_at != 255 && !bit_valid(kc.mask, kc.offset + row)) { x = 1; bit = null_at; }
    else if (i == K.string) continue;
    else { x = canonical_bits(kc, kc.offset + row); bit = 8 * (int)K.form.at[i]; }
#pragma unroll
    for (int q = 0; q < 4; ++q) if ((bit >> 6) == q) w[q] |= x << (bit & 63);
  }
}

// STRINGS: the key is a string column, with MORE beside up to 64 bits of other columns and null flags.  ctrl->out_cursor: ids in
// the upper 26 bits, chars of their strings below.
template <bool STRINGS, bool MORE>
__global__ void __launch_bounds__(KEYED_BLOCK, KEYED_CTAS)
k_keyed(const __grid_constant__ DPlan P, const __grid_constant__ DForms F, const __grid_constant__ DKeyed K, DCtrl* ctrl)
{
  extern __shared__ __align__(16) unsigned char keyed_smem[];
  __shared__ u32 s_ids[KEYED_ROWS][KEYED_BLOCK];
  __shared__ u32 s_owner[KEYED_SLOTS];  // 1 + the id that has the slot, 0: none
  __shared__ u32 s_stop;
  const int tid = threadIdx.x, S = K.slots;
  const DDict& D = K.dict;
  grid_dependents_launch();  // (k_report)
  if (tid == 0) s_stop = 0;
  for (int i = tid * 16; i < K.smem; i += KEYED_BLOCK * 16) *(ulonglong2*)(keyed_smem + i) = make_ulonglong2(0, 0);
  for (int i = tid; i < S; i += KEYED_BLOCK) s_owner[i] = 0;
  __syncthreads();
  grid_dependency_wait();  // (the cells are empty from here on)
  const u32 smem_a = (u32)__cvta_generic_to_shared(keyed_smem);
  const int each = K.each;
  const i64 tile_rows = (i64)KEYED_BLOCK * each;

  for (i64 base = (i64)blockIdx.x * tile_rows; base < P.nrows; base += (i64)gridDim.x * tile_rows) {
    // (a warp leaves as one: its lanes part in the probes and need not read the flag at the same time)
    if (__any_sync(0xFFFFFFFFu, *(volatile u32*)&s_stop != 0u)) break;
    // ---- keys -> ids, row by row
    u32 live = 0;
#pragma unroll
    for (int j = 0; j < KEYED_ROWS; ++j) {
      const i64 row = base + (i64)j * KEYED_BLOCK + tid;
      if (j < each && row < P.nrows && row_active(P, row)) live |= 1u << j;
    }
    i64 begin = 0, next_len = 0;
    auto offsets = [&](int j) {
      if (!STRINGS || j >= each || !((live >> j) & 1u)) return;
      const DKeyCol& c = P.keys[K.string];
      const i64 at = c.offset + base + (i64)j * KEYED_BLOCK + tid;
      begin = str_offset(c, at);
      next_len = MORE && c.mask && !bit_valid(c.mask, at) ? 0 : str_offset(c, at + 1) - begin;  // (a null is an empty string and its flag)
    };
    offsets(0);
#pragma unroll 1
    for (int j = 0; j < each; ++j) {
      const i64 row = base + (i64)j * KEYED_BLOCK + tid;
      const unsigned char* p = STRINGS ? P.keys[K.string].data + begin : nullptr;
      const i64 len = STRINGS ? next_len : 8 * K.form.words;
      offsets(j + 1);
      u32 id = ~0u;
      if ((live >> j) & 1u) {
        u64 w[4] = {0, 0, 0, 0}, more = 0, h;
        if (STRINGS) {
          if (MORE) {
            u64 x[4] = {0, 0, 0, 0};
            keyed_bits(P, K, row, x);
            more = x[0];
          }
          dict_load(p, len, w);
          h = dict_hash(w, 4, ((u64)len << 56) ^ (MORE ? mix64(more) : 0ull));
          if (len > DICT_INLINE) h = hash_bytes(p + DICT_INLINE, len - DICT_INLINE, h);
        } else {
          keyed_bits(P, K, row, w);
          h = dict_hash(w, K.form.words, 0);
        }
        const i64 s = dict_find_insert(P, D, w, len, row, h, ctrl,
          [&](u32 who, int lead) -> u64 {
            // ids and chars of the lanes that claim together, in one atomic
            const u32 lane = tid & 31u;
            const u64 mine = (1ull << KEYED_CHARS) | (STRINGS ? (u64)len : 0ull);
            u64 before = 0, all = 0;
            for (u32 m = who; m; m &= m - 1u) {
              const int l = __ffs((int)m) - 1;
              const u64 x = __shfl_sync(who, mine, l);
              if (l < (int)lane) before += x;
              all += x;
            }
            u64 first = 0;
            if ((int)lane == lead) first = atomicAdd(&ctrl->out_cursor, all);
            const u64 got = __shfl_sync(who, first, lead) + before, id = got >> KEYED_CHARS;
            if (id < (u64)D.pool_cap) {
              if (STRINGS) K.char_at[id] = (i64)(got & KEYED_CHARS_MASK);
              if (MORE) K.more[id] = more;
              for (int c = 0; c < P.ncells; ++c) K.acc[id * (u64)P.ncells + c] = K.zeros ? 0ull : keyed_none(P, F, c);
            }
            return id;
          },
          [&](u64 id) { return !MORE || __ldcg(K.more + id) == more; },
          [&] {},
          [&](int probe) { return (probe & 7) == 7 && *(volatile u32*)&ctrl->overflow != 0u; });
        if (s >= 0) id = (u32)s;
      }
      s_ids[j][tid] = id;  // (read by this thread only)
    }
    __syncwarp();
    // ---- the values: the operator is decoded once for the thread's rows
    u32 at[KEYED_ROWS], act = 0, shared = 0;  // (`shared`: rows whose place is a slot, the others' is their id)
#pragma unroll
    for (int j = 0; j < KEYED_ROWS; ++j) {
      at[j] = j < each ? s_ids[j][tid] : ~0u;
      if (at[j] == ~0u) continue;
      act |= 1u << j;
      const u32 slot = at[j] < (u32)S ? at[j] : at[j] % (u32)S;
      u32 owner = *(volatile u32*)&s_owner[slot];
      if (owner == 0) {
        owner = atomicCAS(&s_owner[slot], 0u, at[j] + 1u);
        if (owner == 0) owner = at[j] + 1u;
      }
      if (owner == at[j] + 1u) { at[j] = slot; shared |= 1u << j; }
    }
    int cur = -1;
    u32 vn = 0;
    u64 v[KEYED_ROWS] = {};
    for (int c = 0; c < P.ncells; ++c) {
      const int op = P.cells[c].op, col = P.cells[c].col;
      if (op != OP_CNT_A && col != cur) {
        cur = col;
        const DValCol& vc = P.vals[col];
        vn = 0;
#pragma unroll
        for (int j = 0; j < KEYED_ROWS; ++j) {
          const i64 row = base + (i64)j * KEYED_BLOCK + tid;
          if (((act >> j) & 1u) && value_valid(vc, row)) vn |= 1u << j;
          v[j] = ((act >> j) & 1u) && F.kind[col] != RK_NONE ? load_value(vc, row) : 0ull;
        }
      }
      const u32 use = op == OP_CNT_A ? act : vn, here = use & shared, far = use & ~shared;
      const int adds = keyed_adds(op), form = F.form[c];
      unsigned char* const cell = keyed_smem + 16u * K.cell_at[c];
      const u32 cell_a = smem_a + 16u * K.cell_at[c];
      u64 x[KEYED_ROWS];
#pragma unroll
      for (int j = 0; j < KEYED_ROWS; ++j) x[j] = keyed_addend(op, adds, v[j]);
      if (here) {
        if (form == CF_COUNT) {
#pragma unroll
          for (int j = 0; j < KEYED_ROWS; ++j) fx_red_if(cell_a + 4u * at[j], 1u, here & (1u << j));
        } else if (form == CF_SUM) {
#pragma unroll
          for (int j = 0; j < KEYED_ROWS; ++j) {
            const u32 old = fx_atom_if(cell_a + 4u * at[j], (u32)x[j], here & (1u << j));
            const u32 up = (u32)(x[j] >> 32) + (old > ~(u32)x[j] ? 1u : 0u);
            fx_red_if(cell_a + 4u * ((u32)S + at[j]), up, (here & (1u << j)) ? up : 0u);
          }
        } else if (form != CF_64) {
          const u32 flip = form == CF_MIN32 ? ~0u : 0u;
#pragma unroll
          for (int j = 0; j < KEYED_ROWS; ++j) fx_max_if(cell_a + 4u * at[j], order32(F.kind[col], v[j]) ^ flip, here & (1u << j));
        } else {
#pragma unroll
          for (int j = 0; j < KEYED_ROWS; ++j) {
            if (!((here >> j) & 1u)) continue;
            u64* const p = (u64*)cell + at[j];
            if (adds == KA_FLOAT) atomicAdd((double*)p, __longlong_as_double((i64)x[j]));
            else if (x[j] > *(volatile u64*)p) atomicMax(p, x[j]);  // (64-bit atomics of shared memory are compare-and-swap loops)
          }
        }
      }
      if (far) {
#pragma unroll
        for (int j = 0; j < KEYED_ROWS; ++j)
          if ((far >> j) & 1u) keyed_update(K.acc + (u64)at[j] * (u64)P.ncells + c, adds, x[j]);
      }
    }
    if (tid == 0 && *(volatile u32*)&ctrl->overflow) *(volatile u32*)&s_stop = 1;  // (no barrier: the others see it a tile later)
  }

  // ---- what this CTA holds joins the global accumulators (the CTAs start at different slots)
  __syncthreads();
  if (s_stop) return;
  const u32 rot = (u32)(((u64)blockIdx.x * 2654435761ull) % (u64)S);
  for (u32 i0 = tid; i0 < (u32)S; i0 += KEYED_BLOCK) {
    const u32 i = i0 + rot < (u32)S ? i0 + rot : i0 + rot - (u32)S;
    if (s_owner[i] == 0) continue;
    const u64 id = s_owner[i] - 1u;
    for (int c = 0; c < P.ncells; ++c) {
      const int op = P.cells[c].op;
      const unsigned char* at = keyed_smem + 16u * K.cell_at[c];
      u64 a;
      switch (F.form[c]) {
        case CF_64: a = ((const u64*)at)[i]; break;
        case CF_COUNT: a = ((const u32*)at)[i]; break;
        case CF_SUM: a = ((u64)((const u32*)at)[S + i] << 32) | ((const u32*)at)[i]; break;
        default: {
          const u32 word = ((const u32*)at)[i];
          const bool met = F.count_of[c] >= 0 ? ((const u32*)(keyed_smem + 16u * K.cell_at[F.count_of[c]]))[i] != 0u : word != 0u;
          a = met ? unorder32(F.kind[P.cells[c].col], word ^ (F.form[c] == CF_MIN32 ? ~0u : 0u)) ^ keyed_flip(op) : 0ull;
        }
      }
      if (a) keyed_update(K.acc + id * (u64)P.ncells + c, keyed_adds(op), a);
    }
  }
}

// ids -> output rows: results, key columns, strings.  `total`: chars of the result.
template <typename OffT>
__global__ void __launch_bounds__(256) k_keyed_finish(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O, const __grid_constant__ DKeyed K,
                                                      i64 ngroups, i64 total, OffT* __restrict__ out_offs, unsigned char* __restrict__ chars,
                                                      DCtrl* ctrl, const DReport report)
{
  const int* const rows = K.dict.first_row;
  if (K.string >= 0) {  // four lanes per string, 8 bytes per lane and step
    const DKeyCol& c = P.keys[K.string];
    const int sub = threadIdx.x & 3;
    for (i64 g = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 2; g <= ngroups; g += ((i64)gridDim.x * blockDim.x) >> 2) {
      const i64 at = g < ngroups ? K.char_at[g] : total;
      if (sub == 0) out_offs[g] = (OffT)at;
      if (g == ngroups) break;
      const i64 len = (g + 1 < ngroups ? K.char_at[g + 1] : total) - at;
      if (len == 0) continue;
      const unsigned char* src = c.data + str_offset(c, c.offset + rows[g]);
      unsigned char* dst = chars + at;
      for (i64 b = (i64)sub * 8; b < len; b += 32) {
        const int nb = (int)(len - b < 8 ? len - b : 8);
        u64 v = load_bytes8(src + b, nb);
        for (int i = 0; i < nb; ++i) { dst[b + i] = (unsigned char)v; v >>= 8; }
      }
    }
  }
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x) {
    const i64 row = rows[g];
    for (int k = 0; k < P.nkeys; ++k) {
      const DKeyCol& c = P.keys[k];
      const bool null = O.kmask[k] && !bit_valid(c.mask, c.offset + row);
      if (null) clear_bit(O.kmask[k], g, O.null_counts + MAX_OUTS + k);
      if (k == K.string) continue;
      store_int(O.kdata[k], g, c.width == 1 ? VC_U8 : c.width == 2 ? VC_U16 : c.width == 4 ? VC_U32 : VC_U64,
                null ? 0ull : load_fixed_bits(c.data, c.offset + row, c.width));
    }
    write_group(P, O, (u64)(u32)row, [&](int c) { return K.acc[(u64)g * (u64)P.ncells + c] ^ keyed_flip(P.cells[c].op); }, g, O.null_counts);
  }
  report_ctrl(ctrl, report);
}

}  // namespace b2
