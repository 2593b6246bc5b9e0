// b2_partition.cuh — the high-cardinality path: radix partition of the rows by key hash into
// buckets whose groups fit a shared-memory table, then one shared-memory aggregate per bucket.
//
// Replaces the global-memory branch of the reference (compute_global_memory_aggs.cuh:74-187: one
// probe of a global cuco set + one global atomic per row and aggregation) for inputs with millions of
// groups.  There every row costs a random read-modify-write of a 32-byte sector per accumulator; here
// the rows are moved twice at most, sequentially, and every atomic is a shared-memory atomic:
//
//   k_rp_count      one pass over the key columns: rows per level-1 digit, and whether the keys can be told by 32-bit words, or
//                   (hashed keys, the number of groups not known) the HyperLogLog registers
//   k_rp_scatter    rows -> records {key, values, validity}, written to the region of their level-1 digit
//                   (structure-of-arrays record buffer; CTA-local counting per tile, one global cursor
//                   reservation per digit and tile)
//   k_rp_count2 /   second level inside every level-1 partition (only when one level leaves more
//   k_rp_scatter2   groups per bucket than a shared-memory table holds)
//   k_rp_direct     key words: one CTA per bucket at a time, accumulators addressed by the word, groups written to the
//                   output columns (or to the list)
//   k_rp_aggregate  hashed keys: one CTA per bucket at a time: open-addressing table in shared memory, the
//                   bucket's records folded with shared-memory atomics, the finished groups appended
//                   to a compact record list (structure-of-arrays)
//   k_finalize_records  record list -> output columns (the finishers of k_finalize)
//
// Packed keys only (all key columns fixed-width non-float, at most 64 bits together).
#pragma once
#include "b2_kernels.cuh"

namespace b2 {

constexpr int RP_BLOCK    = 1024;                // threads per CTA of the counting kernel with a hot set (one CTA per SM)
constexpr int RPC_BLOCK   = 512;                 // ... without (three)
// The scatter kernels run as two 512-thread CTAs per SM (each stages a 4096-row tile in ~90 KB of shared
// memory) that overlap each other's barriers and memory round trips.
constexpr int RPS_BLOCK   = 512;
constexpr int RP_ROWS     = 8;                   // rows per thread per tile: two groups of 4 consecutive rows
constexpr int RP_TILE     = RPS_BLOCK * RP_ROWS; // 4096 rows
constexpr int RP_BITS_TOP = 10;                  // resolution of the first histogram
constexpr int RP_MAX_BITS = 9;                   // widest digit of one level (512 destinations)
constexpr u64 RP_SALT     = 0x9FB21C651E98DF25ull;
constexpr int RPA_BLOCK   = 512;                 // threads per CTA of the bucket aggregate (2 CTAs per SM)
constexpr int RPA_BATCH   = 4;                   // records per thread whose loads are issued together

__device__ __forceinline__ u64 rp_hash(u64 key) { return mix64(key ^ RP_SALT); }

// packed keys + activity of 4 consecutive rows starting at row0 (`nv` of them exist)
__device__ __forceinline__ void rp_keys4(const DPlan& P, i64 row0, int nv, u64 (&kk)[4], u32& act)
{
  act = nv >= 4 ? 0xFu : (nv > 0 ? (1u << nv) - 1u : 0u);
  if (nv == 4 && (P.flags & PF_VEC_KEYS)) {
    packed_keys4(P, row0, kk, act);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      kk[j] = 0;
      if (!((act >> j) & 1u)) continue;
      if (!row_active(P, row0 + j)) { act &= ~(1u << j); continue; }
      kk[j] = pack_key(P, row0 + j);
    }
  }
}

// ------------------------------------------------------------------------------ key words
// Where the keys of a call span few values for its rows (ids, categories, dictionary codes: at most two rows' worth of values
// per row), a key is told by one 32-bit word: its position in the box of its columns' values, counted from sampled smallest
// values, in mixed radix.  The low 18 bits of the position are spread over all 2^18 values by a multiplication, turned by
// the bits above them (a bijection: runs of neighbouring ids, strides and blocks meet all digits equally often).  The digits
// of both levels are the top bits of those 18, and what is left of the word — the bits above, the lowest bits — numbers the
// keys of one bucket without a gap, so that
//   * a record's key takes 4 bytes instead of 8, and no digit needs a hash of it again;
//   * a bucket's accumulators are addressed by the word directly: no keys in shared memory, no probing (500M rows, 10^8 ids:
//     the bucket aggregate with a hash table of 32-bit keys issued 404 instructions per record and warp).
// The counting pass notes whether every key lies in the box and how far it reaches; if not, or if the box turns out too
// large, it runs again over hashed 64-bit keys.
constexpr int WORD_KEYS = 2;      // key columns of a word
constexpr int WORD_LOW  = 18;     // = 2 * RP_MAX_BITS
constexpr u32 WORD_MASK = (1u << WORD_LOW) - 1u;
constexpr u32 WORD_LIMIT = 1u << 31;  // words stay below
constexpr u32 WORD_SPREAD = 162013u, WORD_TURN = 197887u;  // odd, near 2^18 / golden ratio and 2^18 / plastic number
constexpr u32 inverse_mod_2_32(u32 a) { u32 x = a; for (int i = 0; i < 5; ++i) x *= 2u - a * x; return x; }
constexpr u32 WORD_GATHER = inverse_mod_2_32(WORD_SPREAD);
static_assert(WORD_SPREAD * WORD_GATHER == 1u, "inverse");
struct DWord {
  int n;              // key columns; 0: no words
  u32 radix;          // two columns: values of the first one (its null included)
  u32 nul;            // bit k: column k's position 0 stands for null, its values follow
  u64 lo[WORD_KEYS];  // value at the first position, modulo 2^64
};
__device__ __forceinline__ u32 word_place(u32 w)
{
  const u32 x = w * WORD_SPREAD + (w >> WORD_LOW) * WORD_TURN;
  return (w & ~WORD_MASK) | (x & WORD_MASK);
}
__device__ __forceinline__ u32 word_unplace(u32 w)
{
  const u32 x = (w - (w >> WORD_LOW) * WORD_TURN) * WORD_GATHER;
  return (w & ~WORD_MASK) | (x & WORD_MASK);
}
// the finalizer of MurmurHash3, a bijection
__device__ __forceinline__ u32 mix32(u32 h)
{
  h ^= h >> 16; h *= 0x85ebca6bu; h ^= h >> 13; h *= 0xc2b2ae35u; h ^= h >> 16;
  return h;
}
// Position of a packed key; `bad`: it does not lie in the box of the first column.  `most`: the last column's position,
// nulls left out (the caller looks whether the word, which is taken modulo 2^32, can have been exceeded).
__device__ __forceinline__ u32 word_of_key(const DPlan& P, const DWord& W, u64 key, u32& bad, u32& most)
{
  u32 w = 0;
  for (int k = 0; k < W.n; ++k) {
    const DKeyCol& c = P.keys[k];
    const u32 nul = (W.nul >> k) & 1u;
    u32 f = 0;
    if (!(c.nullbit >= 0 && ((key >> c.nullbit) & 1ull))) {
      const u64 d = (u64)key_field(c, key) - W.lo[k];
      f = (u32)d;
      bad |= (u32)(d >> 32);
      if (k + 1 < W.n) bad |= f >= W.radix - nul ? 1u : 0u;
      else most = max(most, f);
      f += nul;
    }
    w += k == 0 ? f : f * W.radix;
  }
  return w;
}
__device__ __forceinline__ u64 word_key(const DPlan& P, const DWord& W, u32 placed)
{
  const u32 w = word_unplace(placed);
  u64 key = 0;
  for (int k = 0; k < W.n; ++k) {
    const DKeyCol& c = P.keys[k];
    const u32 f = W.n == 1 ? w : k == 0 ? w % W.radix : w / W.radix, nul = (W.nul >> k) & 1u;
    if (nul && f == 0) { key |= 1ull << c.nullbit; continue; }
    const u64 v = (u64)(f - nul) + W.lo[k];
    key |= (c.width == 8 ? v : v & ((1ull << (8 * c.width)) - 1ull)) << c.shift;
  }
  return key;
}
// positions + activity of 4 consecutive rows from row0 on (`nv` of them exist)
__device__ __forceinline__ void rp_words4(const DPlan& P, const DWord& W, i64 row0, int nv, u32 (&w)[4], u32& act, u32& bad, u32& most)
{
  act = nv >= 4 ? 0xFu : (nv > 0 ? (1u << nv) - 1u : 0u);
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = 0;
  if (nv < 4 || !(P.flags & PF_VEC_KEYS)) {
#pragma unroll 1
    for (int j = 0; j < nv; ++j) {
      if (!row_active(P, row0 + j)) { act &= ~(1u << j); continue; }
      const u32 x = word_of_key(P, W, pack_key(P, row0 + j), bad, most);
      if (j == 0) w[0] = x; else if (j == 1) w[1] = x; else if (j == 2) w[2] = x; else w[3] = x;
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < WORD_KEYS; ++k) {
    if (k >= W.n) break;
    const DKeyCol& c = P.keys[k];
    const unsigned char* src = c.data + (c.offset + row0) * c.width;
    u32 f[4], far[4] = {0, 0, 0, 0};
    if (c.width == 8) {
      const ulonglong2 a = __ldg((const ulonglong2*)src), b = __ldg((const ulonglong2*)src + 1);
      const u64 x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
      for (int j = 0; j < 4; ++j) { const u64 d = x[j] - W.lo[k]; f[j] = (u32)d; far[j] = (u32)(d >> 32); }
    } else if (c.width == 4) {
      const uint4 q = __ldg((const uint4*)src);  // (modulo 2^32: a value below the first one is far above the box)
      f[0] = q.x - (u32)W.lo[k]; f[1] = q.y - (u32)W.lo[k]; f[2] = q.z - (u32)W.lo[k]; f[3] = q.w - (u32)W.lo[k];
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        f[j] = (u32)key_field(c, load_fixed_bits(c.data, c.offset + row0 + j, c.width) << c.shift) - (u32)W.lo[k];
    }
    u32 vn = 0xFu;
    if (c.mask) {
      vn = valid_nibble(c.mask, c.offset + row0, 4);
      if (!P.include_nulls) act &= vn;  // EXCLUDE: a null key drops the row
    }
    const u32 nul = (W.nul >> k) & 1u, live = act & vn, room = W.radix - nul;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (live == 0xFu || ((live >> j) & 1u)) {
        bad |= far[j];
        if (k + 1 < W.n) bad |= f[j] >= room ? 1u : 0u;
        else most = max(most, f[j]);
      }
      if (nul) f[j] = ((vn >> j) & 1u) ? f[j] + 1u : 0u;
      w[j] = k == 0 ? f[j] : w[j] + f[j] * W.radix;
    }
  }
  for (int i = 0; i < P.nfilters; ++i) act &= valid_nibble(P.filters[i], P.filter_offsets[i] + row0, 4);
}

// ------------------------------------------------------------------------------ hot keys (skewed inputs)
// A key that holds a visible share of the rows would put all its records into one bucket and serialise them
// on one shared-memory slot.  For aggregates whose cells are Σx / n / Σx² of one float column the hottest
// keys are therefore taken out before the rows are partitioned:
//   k_hot_sample   256K evenly spaced rows -> occurrences per key (a global counting table), and the
//                  largest magnitude among the sampled values (places the fixed-point windows)
//   k_hot_hist /   the keys seen most often (at most HOT_MAX, at least 3 times each), one dense id per key
//   k_hot_select
//   k_hot_place    the hot set: buckets of HOT_WAYS hash tags and ids, the most frequent keys placed first
//   k_rp_count<..., HOT>  folds the rows of hot keys into per-CTA fixed-point accumulators (fx_add: native 32-bit
//                  shared-memory atomics, which keep their rate on hot addresses) and counts only the other rows into
//                  the digit histogram; k_rp_scatter skips hot rows
//   k_rp_append_hot  the hot keys' finished cells -> the group list
// Hot and cold keys are disjoint, so the list is the union of both parts.
constexpr int HOT_SAMPLES    = 1 << 18;
constexpr int HOT_COUNT_SLOTS = 1 << 19;  // counting table of the sampler
constexpr int HOT_MAX        = 3072;      // keys in the hot set (what shared memory holds of their accumulators)
constexpr int HOT_BUCKETS    = 4096;      // of HOT_WAYS keys each; a key whose bucket is full is not hot (about 6 % of 3072
constexpr int HOT_WAYS       = 2;         // keys, the least frequent ones)
constexpr u32 HOT_MIN_COUNT  = 3;         // occurrences among the samples that make a key hot
constexpr u32 HOT_TOP_COUNT  = PART_TOP_COUNT;  // occurrences of the most frequent key among 1024 rows that speak for a hot set
constexpr int HOT_ACC_WORDS  = 4;         // global accumulators per hot key: n, Σx, Σx², seen

struct DHot {
  u64* keys;        // [HOT_MAX] by id
  u32* counts;      // [HOT_MAX] occurrences among the samples
  u32* table;       // [HOT_BUCKETS][HOT_WAYS] hot_tag | id of the key, all ones = free
  u32* info;        // [0] number of hot keys, [1] 1 + largest biased exponent among the sampled values, [2] sum of their
                    // biased exponents, [3] their number, [4, 260) keys per occurrence count (k_hot_hist)
  u64* acc;         // [HOT_MAX][HOT_ACC_WORDS] finished accumulators (filled by k_rp_count)
  u32* row_mask;    // one bit per row: the row's key is hot (written by k_rp_count, read by k_rp_scatter)
};

// A key is known by its hash (a bijection): 12 bits of it are the bucket, 20 bits the tag, the upper 32 bits are compared.
// (A key word's hash has 32 bits: bucket and tag tell it.)
__device__ __forceinline__ u32 hot_bucket(u64 h) { return (u32)h & (u32)(HOT_BUCKETS - 1); }
__device__ __forceinline__ u32 hot_tag(u64 h) { return (u32)h & ~(u32)(HOT_BUCKETS - 1); }
static_assert(HOT_BUCKETS == 4096 && HOT_MAX < 4095, "bucket and id in 12 bits, id 4095 is free");

// Id of a hot key, or HOT_MAX.  No loop and no branch: one 8-byte read of the bucket, one compare.  (Probing a half-full table
// of keys, every lane waited for the longest chain of its warp.)  Of two keys with one tag in a bucket only the first is
// ever found; the other one's rows are cold rows like any.  `table`, `upper`: shared addresses of the buckets and of the
// upper halves of the hashes by id.
__device__ __forceinline__ u32 hot_find(const uint2* table, const u32* upper, u64 h)
{
  const uint2 t = table[hot_bucket(h)];
  const u32 d0 = t.x - hot_tag(h), d1 = t.y - hot_tag(h);   // below 4096: the tags are equal, the difference is the id
  const u32 id = min(min(d0, d1), (u32)HOT_MAX);            // (both match: a free way, or the second of two equal tags)
  return id < (u32)HOT_MAX && upper[id] == (u32)(h >> 32) ? id : (u32)HOT_MAX;
}

__device__ __forceinline__ u32 hot_find(const uint2* table, u32 h)
{
  const uint2 t = table[h & (u32)(HOT_BUCKETS - 1)];
  const u32 tag = h & ~(u32)(HOT_BUCKETS - 1);
  return min(min(t.x - tag, t.y - tag), (u32)HOT_MAX);
}

// (`ckeys` = nullptr: the magnitudes only)
__global__ void __launch_bounds__(256) k_hot_sample(const __grid_constant__ DPlan P, u64* __restrict__ ckeys,
                                                    u32* __restrict__ ccnt, u32* __restrict__ info)
{
  const i64 nsamp  = P.nrows < HOT_SAMPLES ? P.nrows : HOT_SAMPLES;
  const i64 stride = P.nrows / (nsamp > 0 ? nsamp : 1);
  u32 emax = 0, esum = 0, ecount = 0;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < nsamp; i += (i64)gridDim.x * blockDim.x) {
    const i64 row = i * stride + (stride > 1 ? (i64)(((u64)i * 7919ull) % (u64)stride) : 0);
    if (!row_active(P, row)) continue;
    const u64 key = ckeys ? pack_key(P, row) : EMPTY;
    if (key != EMPTY) {
      u32 idx = (u32)(rp_hash(key) >> 20) & (HOT_COUNT_SLOTS - 1);
      for (int p = 0; p < 64; ++p) {  // (a sample that finds no slot in 64 probes is dropped: it is only a sample)
        u64 k = ckeys[idx];
        if (k == EMPTY) {
          k = atomicCAS(ckeys + idx, EMPTY, key);
          if (k == EMPTY) k = key;
        }
        if (k == key) { atomicAdd(ccnt + idx, 1u); break; }
        idx = (idx + 1u) & (HOT_COUNT_SLOTS - 1);
      }
    }
    if (value_valid(P.vals[0], row)) {
      const u32 e = (u32)((load_value(P.vals[0], row) >> 52) & 0x7FFu);
      if (e != 0x7FFu && e + 1u > emax) emax = e + 1u;
      if (e != 0x7FFu && e != 0u) { esum += e; ++ecount; }
    }
  }
  emax = __reduce_max_sync(0xFFFFFFFFu, emax);
  esum = __reduce_add_sync(0xFFFFFFFFu, esum);      // (at most 2^18 samples of 11 bits)
  ecount = __reduce_add_sync(0xFFFFFFFFu, ecount);
  if ((threadIdx.x & 31) == 0 && emax) { atomicMax(info + 1, emax); atomicAdd(info + 2, esum); atomicAdd(info + 3, ecount); }
}

// keys per (clamped) occurrence count: `hist` = 256 zeroed words
__global__ void __launch_bounds__(256) k_hot_hist(const u32* __restrict__ ccnt, u32* __restrict__ hist)
{
  __shared__ u32 s_hist[256];
  s_hist[threadIdx.x] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < HOT_COUNT_SLOTS; i += gridDim.x * blockDim.x) {
    const u32 c = ccnt[i];
    if (c >= HOT_MIN_COUNT) atomicAdd(&s_hist[c < 255u ? c : 255u], 1u);
  }
  __syncthreads();
  if (s_hist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], s_hist[threadIdx.x]);
}

// `hot.info[0]` (the id counter, then the number of hot keys) arrives zero.  Every CTA derives the same threshold from the
// histogram: the smallest count from which on at most HOT_MAX keys qualify.
__global__ void __launch_bounds__(256) k_hot_select(const u64* __restrict__ ckeys, const u32* __restrict__ ccnt,
                                                    const u32* __restrict__ hist, DHot hot)
{
  __shared__ u32 s_min;
  if (threadIdx.x == 0) {
    u32 total = 0, t = 256;
    while (t > HOT_MIN_COUNT && total + hist[t - 1] <= (u32)HOT_MAX) { --t; total += hist[t]; }
    s_min = t;
  }
  __syncthreads();
  const u32 tmin = s_min;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < HOT_COUNT_SLOTS; i += gridDim.x * blockDim.x) {
    const u32 c = ccnt[i];
    if ((c < 255u ? c : 255u) < tmin) continue;
    const u32 id = atomicAdd(hot.info, 1u);  // (at most HOT_MAX keys qualify: tmin bounds them)
    if (id >= (u32)HOT_MAX) continue;
    hot.keys[id] = ckeys[i];
    hot.counts[id] = c;
  }
}

// One CTA: the hot keys into their buckets, by falling powers of two of their counts, so that it is the least frequent
// ones that find a bucket full.  `hot.table` arrives filled with ones.
__global__ void __launch_bounds__(1024) k_hot_place(const __grid_constant__ DPlan P, const __grid_constant__ DWord W, DHot hot)
{
  __shared__ u32 s_fill[HOT_BUCKETS];
  const int n = (int)min(hot.info[0], (u32)HOT_MAX);
  for (int i = threadIdx.x; i < HOT_BUCKETS; i += blockDim.x) s_fill[i] = 0;
  for (int top = 31; top >= 0; --top) {
    __syncthreads();
    for (int id = threadIdx.x; id < n; id += blockDim.x) {
      if (31 - __clz((int)hot.counts[id]) != top) continue;
      u32 bad = 0, most = 0;
      const u64 h = W.n > 0 ? mix32(word_of_key(P, W, hot.keys[id], bad, most)) : rp_hash(hot.keys[id]);
      if (bad) continue;
      const u32 b = hot_bucket(h), way = atomicAdd(&s_fill[b], 1u);
      if (way >= (u32)HOT_WAYS) continue;
      hot.table[b * HOT_WAYS + way] = hot_tag(h) | (u32)id;
    }
  }
}

// ------------------------------------------------------------------------------ level-1 histogram (+ HyperLogLog)
// With HOT the kernel also carries the hot set (dynamic shared memory: buckets, then per hot key its hash's upper half, an
// addend count, the words of Σx and of Σx², and a "seen" bit): rows of hot keys are folded here and left out
// of the histogram.  P.cells are Σx / n / Σx² of value column 0 in that case.
constexpr int HOT_STRIDE = HOT_MAX + 1;  // words between the words of one key: odd, so that they lie in different banks
constexpr size_t rp_count_hot_smem()
{
  return (size_t)HOT_BUCKETS * HOT_WAYS * 4 + (size_t)HOT_MAX * 4 + (size_t)HOT_STRIDE * (4 + 8 * FX_WORDS) + HOT_MAX / 8;
}

// the values of 4 consecutive rows in carried form; `vec`: the column's data takes 16-byte loads at multiples of 4 rows
__device__ __forceinline__ void load_floats4(const DValCol& c, i64 row0, int nv, bool vec, u64 (&v)[4])
{
  if (vec && nv == 4) {
    if (c.vclass == VC_F64) {
      const ulonglong2 a = __ldg((const ulonglong2*)(c.data + (c.offset + row0) * 8)), b = __ldg((const ulonglong2*)(c.data + (c.offset + row0) * 8) + 1);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else {
      const float4 a = __ldg((const float4*)(c.data + (c.offset + row0) * 4));
      v[0] = (u64)__double_as_longlong((double)a.x); v[1] = (u64)__double_as_longlong((double)a.y);
      v[2] = (u64)__double_as_longlong((double)a.z); v[3] = (u64)__double_as_longlong((double)a.w);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = j < nv ? load_value(c, row0 + j) : 0ull;
}

// What the counting pass is asked to find besides: whether the key words can be used, and whether 64-bit value columns can be
// told by 32 bits.
constexpr int RANGE_VALS = 2;
struct DRanges {
  u32* out;             // zeroed; [0] a key lies outside the box, [1] the last key column's highest position,
                        // [2 + 2i] a value of column col[i] is no sign-extended 32-bit number, [3 + 2i] no zero-extended one
  int nvals;
  int col[RANGE_VALS];
  u32 vec;              // bit i: column i of the list takes 16-byte loads at multiples of 4 rows
};
constexpr int RANGE_WORDS = 2 + 2 * RANGE_VALS;

// WORDS: keys as words (`W`); their digit is the top of their low 18 bits.  WITH_HLL: the registers of the estimator (not
// with words: the box bounds the groups).  The loop is bound by instruction issue (103 per row and warp over one 64-bit
// key column with hashes and registers).
template <bool WORDS, bool WITH_HLL, bool HOT>
__global__ void __launch_bounds__(HOT ? RP_BLOCK : RPC_BLOCK, HOT ? 1 : 3)
k_rp_count(const __grid_constant__ DPlan P, const __grid_constant__ DWord W, u64* __restrict__ hist, u32* __restrict__ hll, const DHot hot, const DRanges ranges)
{
  extern __shared__ __align__(16) unsigned char rp_hot_smem[];
  __shared__ u32 s_hist[1 << RP_BITS_TOP];
  __shared__ u32 s_regs[WITH_HLL ? HLL_REGS : 1];
  uint2* htab = (uint2*)rp_hot_smem;                      // [HOT_BUCKETS] of HOT_WAYS keys
  u32* hup  = (u32*)(htab + HOT_BUCKETS);                 // [HOT_MAX]
  u32* hcnt = hup + HOT_MAX;                              // [HOT_STRIDE]
  u32* hlx  = hcnt + HOT_STRIDE;                          // [FX_WORDS][HOT_STRIDE]
  u32* hlq  = hlx + FX_WORDS * HOT_STRIDE;                // [FX_WORDS][HOT_STRIDE]
  u32* hseen = hlq + FX_WORDS * HOT_STRIDE;               // [HOT_MAX / 32]
  int nh = 0, bx = FX_NEVER, bq = FX_NEVER;
  for (int i = threadIdx.x; i < (1 << RP_BITS_TOP); i += blockDim.x) s_hist[i] = 0;
  if (WITH_HLL) for (int i = threadIdx.x; i < HLL_REGS; i += blockDim.x) s_regs[i] = 0;
  if (HOT) {
    nh = (int)min(hot.info[0], (u32)HOT_MAX);
    if (hot.info[3]) {
      const int mean = (int)(hot.info[2] / hot.info[3]), emax = (int)hot.info[1] - 1;
      bx = fx_base(mean, emax);
      bq = fx_base_sq(mean, emax);
    }
    if (nh > 0) {
      if (!WORDS) for (int i = threadIdx.x; i < HOT_MAX; i += blockDim.x) hup[i] = i < nh ? (u32)(rp_hash(hot.keys[i]) >> 32) : 0u;
      for (int i = threadIdx.x; i < HOT_BUCKETS; i += blockDim.x) htab[i] = ((const uint2*)hot.table)[i];
      for (int i = threadIdx.x; i < HOT_STRIDE * (1 + 2 * FX_WORDS) + HOT_MAX / 32; i += blockDim.x) hcnt[i] = 0;
    }
  }
  __syncthreads();
  int c_sum = -1, c_cnt = -1, c_ssq = -1;
  if (HOT)
    for (int c = 0; c < P.ncells; ++c) {
      if (P.cells[c].op == OP_SUM_F) c_sum = c;
      if (P.cells[c].op == OP_CNT_V) c_cnt = c;
      if (P.cells[c].op == OP_SSQ_F) c_ssq = c;
    }
  const u32 hist_a = (u32)__cvta_generic_to_shared(s_hist);
  const u32 hcnt_a = (u32)__cvta_generic_to_shared(hcnt), hlx_a = (u32)__cvta_generic_to_shared(hlx), hlq_a = (u32)__cvta_generic_to_shared(hlq);
  const bool vec = HOT && (((u64)P.vals[0].data + (u64)P.vals[0].offset * (P.vals[0].vclass == VC_F64 ? 8u : 4u)) & 15u) == 0u;
  const i64 nquads = (P.nrows + 3) / 4;
  u32 bad = 0, most = 0, no_s32[RANGE_VALS] = {}, no_u32[RANGE_VALS] = {};
  // (whole warps stay in the loop — a lane beyond the last quad has no rows — because the hot-row mask of
  // 8 consecutive quads is put together with shuffles)
  for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q - (threadIdx.x & 31) < nquads; q += (i64)gridDim.x * blockDim.x) {
    u64 kk[4], xx[4] = {0, 0, 0, 0};
    u32 ww[4];
    u32 act, vn = 0;
    const int nv = (int)max((i64)0, min((i64)4, P.nrows - q * 4));
    if (HOT && nh > 0 && nv > 0) {
      load_floats4(P.vals[0], q * 4, nv, vec, xx);
      vn = P.vals[0].mask ? valid_nibble(P.vals[0].mask, P.vals[0].offset + q * 4, nv) : 0xFu;
    }
    if (WORDS && !HOT) {
#pragma unroll
      for (int i = 0; i < RANGE_VALS; ++i) {
        if (i >= ranges.nvals || nv <= 0) continue;
        const DValCol& c = P.vals[ranges.col[i]];
        const u32 ok = c.mask ? valid_nibble(c.mask, c.offset + q * 4, nv) : 0xFu;
        u64 x[4];
        if (((ranges.vec >> i) & 1u) && nv == 4) {
          const ulonglong2* src = (const ulonglong2*)(c.data + (c.offset + q * 4) * 8);
          const ulonglong2 a = __ldg(src), b = __ldg(src + 1);
          x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = j < nv ? load_value(c, q * 4 + j) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (c.mask && !((ok >> j) & 1u)) x[j] = 0;
          const u32 hi = (u32)(x[j] >> 32);
          no_u32[i] |= hi;
          no_s32[i] |= hi ^ (u32)((int)(u32)x[j] >> 31);
        }
      }
    }
    if (WORDS) rp_words4(P, W, q * 4, nv, ww, act, bad, most);
    else rp_keys4(P, q * 4, nv, kk, act);
    u32 hotm = 0, raise = 0;  // rows of hot keys; rows that raise an estimator register
    u32 id[4], ranks[4], regs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u64 h = WORDS ? 0ull : rp_hash(kk[j]);
      id[j] = HOT_MAX;
      if (HOT && nh > 0) {
        id[j] = WORDS ? hot_find(htab, mix32(ww[j])) : hot_find(htab, hup, h);
        if (id[j] != (u32)HOT_MAX) hotm |= 1u << j;
      }
      const u32 cold = act & ~hotm & (1u << j);
      const u32 digit = WORDS ? (word_place(ww[j]) & WORD_MASK) >> (WORD_LOW - RP_BITS_TOP) : (u32)(h >> (64 - RP_BITS_TOP));
      fx_red_if(hist_a + 4u * digit, 1u, cold);
      if (WITH_HLL) {
        regs[j]  = (u32)h & (u32)(HLL_REGS - 1);
        ranks[j] = (u32)__clz((int)(h >> 32)) + 1u;
        if (cold && s_regs[regs[j]] < ranks[j]) raise |= 1u << j;
      }
    }
    if (WITH_HLL && raise) {
#pragma unroll
      for (int j = 0; j < 4; ++j) if ((raise >> j) & 1u) atomicMax(&s_regs[regs[j]], ranks[j]);
    }
    if (HOT && nh > 0) {
      hotm &= act;
      // bit r of word w of the row mask = row 32 w + r: this quad's four bits sit at 4 (q mod 8) of word q / 8
      u32 w = hotm << (4 * (threadIdx.x & 7));
      w |= __shfl_xor_sync(0xFFFFFFFFu, w, 1);
      w |= __shfl_xor_sync(0xFFFFFFFFu, w, 2);
      w |= __shfl_xor_sync(0xFFFFFFFFu, w, 4);
      if ((threadIdx.x & 7) == 0 && q < nquads) hot.row_mask[q >> 3] = w;
      if (hotm & ~vn) {  // a key without a value still makes a group
#pragma unroll
        for (int j = 0; j < 4; ++j) if (((hotm & ~vn) >> j) & 1u) atomicOr(&hseen[id[j] >> 5], 1u << (id[j] & 31u));
      }
      const u32 take = hotm & vn;
      u32 at[4], full = 0, unfit = 0;
      u64 qq[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (((fx_atom_if(hcnt_a + 4u * id[j], 1u, take & (1u << j)) + 1u) & (FX_FLUSH - 1u)) == 0u) full |= 1u << j;
        at[j] = hlx_a + 4u * id[j];
        const double d = __longlong_as_double((i64)xx[j]);
        qq[j] = (u64)__double_as_longlong(d * d);
      }
      if (c_sum >= 0) unfit = fx_add4<true>(xx, bx, at, take, 4u * HOT_STRIDE);
      if (c_ssq >= 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) at[j] += hlq_a - hlx_a;
        unfit |= fx_add4<false>(qq, bq, at, take, 4u * HOT_STRIDE) << 4;
      }
      if (unfit | full) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          const u32 i = j == 0 ? id[0] : j == 1 ? id[1] : j == 2 ? id[2] : id[3];
          u64* acc = hot.acc + (size_t)i * HOT_ACC_WORDS;
          const double d = __longlong_as_double((i64)(j == 0 ? xx[0] : j == 1 ? xx[1] : j == 2 ? xx[2] : xx[3]));
          if ((unfit >> j) & 1u) atomicAdd((double*)(acc + 1), d);  // outside the window: straight to the fp64 accumulators
          if ((unfit >> j) & 16u) atomicAdd((double*)(acc + 2), d * d);
          if (!((full >> j) & 1u)) continue;
          if (c_sum >= 0) atomicAdd((double*)(acc + 1), fx_take(hlx, HOT_STRIDE, (int)i, bx));
          if (c_ssq >= 0) atomicAdd((double*)(acc + 2), fx_take(hlq, HOT_STRIDE, (int)i, bq));
        }
      }
    }
  }
  if (WORDS) {
    bad = __reduce_or_sync(0xFFFFFFFFu, bad);
    most = __reduce_max_sync(0xFFFFFFFFu, most);
    if ((threadIdx.x & 31) == 0) { if (bad) atomicOr(ranges.out, 1u); if (most) atomicMax(ranges.out + 1, most); }
#pragma unroll
    for (int i = 0; i < RANGE_VALS; ++i) {
      if (HOT || i >= ranges.nvals) continue;
      const u32 a = __reduce_or_sync(0xFFFFFFFFu, no_s32[i]), b = __reduce_or_sync(0xFFFFFFFFu, no_u32[i]);
      if ((threadIdx.x & 31) == 0) { if (a) atomicOr(ranges.out + 2 + 2 * i, 1u); if (b) atomicOr(ranges.out + 3 + 2 * i, 1u); }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (1 << RP_BITS_TOP); i += blockDim.x)
    if (s_hist[i]) atomicAdd(&hist[i], (u64)s_hist[i]);
  if (WITH_HLL)
    for (int i = threadIdx.x; i < HLL_REGS; i += blockDim.x)
      if (s_regs[i]) atomicMax(&hll[i], s_regs[i]);
  if (HOT && nh > 0) {
    // CTAs start at different ids so that they do not all hit the same accumulators at once
    const int rot = (int)(((u64)blockIdx.x * 2654435761ull) % (u64)nh);
    for (int i0 = threadIdx.x; i0 < nh; i0 += blockDim.x) {
      const int id = i0 + rot < nh ? i0 + rot : i0 + rot - nh;
      u64* acc = hot.acc + (size_t)id * HOT_ACC_WORDS;
      const u32 n = hcnt[id];
      if (n) {
        atomicAdd(acc, (u64)n);
        if (c_sum >= 0) atomicAdd((double*)(acc + 1), fx_take(hlx, HOT_STRIDE, id, bx));
        if (c_ssq >= 0) atomicAdd((double*)(acc + 2), fx_take(hlq, HOT_STRIDE, id, bq));
      }
      if (((hseen[id >> 5] >> (id & 31)) & 1u) && acc[3] == 0) acc[3] = 1;
    }
  }
}

// the hot keys' finished cells join the groups of the buckets (one thread per id): the list, or the output columns
template <bool LIST>
__global__ void k_rp_append_hot(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O, const DHot hot, u64* __restrict__ out, i64 out_cap, DCtrl* ctrl)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int)min(hot.info[0], (u32)HOT_MAX)) return;
  const u64 key = hot.keys[i];
  const u64* acc = hot.acc + (size_t)i * HOT_ACC_WORDS;
  if (acc[0] == 0 && acc[3] == 0) return;  // not placed in its bucket: a cold key
  const u64 g = atomicAdd(&ctrl->out_cursor, 1ull);
  if (g >= (u64)out_cap) { ctrl->overflow = 1; return; }
  auto cell = [&](int c) { const int op = P.cells[c].op; return op == OP_CNT_V ? acc[0] : op == OP_SUM_F ? acc[1] : acc[2]; };
  if (LIST) {
    out[g] = key;
    for (int c = 0; c < P.ncells; ++c) out[(i64)(1 + c) * out_cap + g] = cell(c);
  } else {
    write_group(P, O, key, cell, (i64)g, O.null_counts);
  }
}

// ------------------------------------------------------------------------------ records
// A record buffer is structure-of-arrays: the key of record i, then one array per value column that some accumulator reads.
// Every byte of a record is written and read again by each level and read by the bucket aggregate, and the shared-memory
// pipe carries it twice per level (staging), so records are as narrow as their contents allow:
//   * a key is 8 bytes, or 4 as a key word (placed: word_place).  The validity bits of the values go into the top bits of a
//     key word where they fit, else into an array of 16-bit words;
//   * a value that its 32 low bits tell (types of up to 4 bytes; 64-bit integers whose column holds no other) takes 4
//     bytes, one that only its validity is asked of takes none (RecKind).
// 500M INT64 keys below 10^8 with INT64 values below 2^31 move as 8 bytes instead of 16.
struct DRecords {
  unsigned char* key;                // u32 or u64 words
  unsigned short* valid;             // validity bits by value column; nullptr: in the key words, or every value is valid
  unsigned char* val[MAX_VALS];
  unsigned char kind[MAX_VALS];      // RecKind
  int nvals;
  int valid_at;                      // bit of value column 0's validity in the key word, -1: not there
  u32 key_mask;                      // the key's bits of a key word
};
static_assert(MAX_VALS <= 16, "validity bits of a record");

template <bool WORDS> struct RpKey { using T = u64; };
template <> struct RpKey<true> { using T = u32; };
// digit of a record (`shift`: see DScatter)
__device__ __forceinline__ u32 rp_digit(u64 key, int shift) { return (u32)(rp_hash(key) >> shift); }
__device__ __forceinline__ u32 rp_digit(u32 word, int shift) { return word >> shift; }

// value of an input row as a record stores it
__device__ __forceinline__ u64 stored_value(const DValCol& c, int kind, i64 row)
{
  if (kind == RK_F32) return (u64)__ldg((const u32*)c.data + c.offset + row);
  return load_value(c, row);  // (its low 32 bits where the record keeps 32)
}

struct DScatter {
  DRecords dst;
  DWord word;
  u64* cursors;  // [partitions] next free record of every destination (start offsets, advanced)
  int shift;     // digit = (rp_hash >> shift) & (fan - 1), of a key word (word >> shift) & (fan - 1)
  int fan;       // destinations per source partition (a power of two, <= 1 << RP_MAX_BITS)
};

// Both scatter levels sort a tile by digit in shared memory before writing it: every thread learns
// its records' ranks inside their digits (shared-memory atomics), the digits' runs are reserved with one
// global atomic each, the records are placed run by run in a staging array, and the staging array is
// copied out in order — consecutive threads write consecutive records of a run.  (Written straight from
// registers, every 8-byte word was an L2 write request of its own — 106 M requests for 60 M rows — and
// the level-1 pass crawled at 0.6 TB/s with DRAM 14 % busy.)  The key and the first stored value column are staged
// together, further columns one after the other through the value array, every thread keeping its records' positions.
template <typename K>
struct RpTile {
  K* keys;     // [RP_TILE] staged keys
  u64* vals;   // [RP_TILE] staged values of one column
  u32* hist;   // [fan] records per digit, then cleared
  u32* off;    // [fan + 1] first staging position of every digit
  u32* base;   // [fan] first global record of every digit's run, less its staging position (modulo 2^32; rows stay below 2^31)
  unsigned short* dig;  // [RP_TILE] digit of every staged record (key words tell theirs)
};
__host__ __device__ constexpr size_t rp_tile_smem(int fan, bool words) { return (size_t)RP_TILE * (8 + (words ? 4 : 8 + 2)) + (size_t)fan * 12 + 64; }

template <typename K>
__device__ __forceinline__ RpTile<K> rp_tile_carve(unsigned char* smem, int fan)
{
  RpTile<K> t;
  t.vals = (u64*)smem;
  t.keys = (K*)(t.vals + RP_TILE);
  t.hist = (u32*)(t.keys + RP_TILE);
  t.off  = t.hist + fan;
  t.base = t.off + fan + 1;
  t.dig  = (unsigned short*)(t.base + fan);
  return t;
}

// after phase A (hist filled): staging offsets by an exclusive scan over the digits, one global
// reservation per digit with records, counters cleared.  `fan` <= blockDim.x.  Begins and ends with a barrier; behind its
// first barrier no thread reads the previous tile's staging arrays any more.
template <typename K>
__device__ __forceinline__ void rp_tile_plan(const RpTile<K>& t, u64* cursors, int fan)
{
  __shared__ u32 s_warp[RPS_BLOCK / 32];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u32 c = (int)threadIdx.x < fan ? t.hist[threadIdx.x] : 0u;
  u32 first = 0;
  if (c) first = (u32)atomicAdd(&cursors[threadIdx.x], (u64)c);
  u32 v = c;
  for (int d = 1; d < 32; d <<= 1) { const u32 x = __shfl_up_sync(0xFFFFFFFFu, v, d); if (lane >= d) v += x; }
  if (lane == 31) s_warp[wid] = v;
  __syncthreads();
  u32 w = lane < RPS_BLOCK / 32 ? s_warp[lane] : 0u;
  if (lane >= wid) w = 0;
  const u32 before = __reduce_add_sync(0xFFFFFFFFu, w);
  if ((int)threadIdx.x < fan) {
    const u32 excl = before + v - c;
    t.off[threadIdx.x] = excl;
    t.hist[threadIdx.x] = 0;
    t.base[threadIdx.x] = first - excl;
    if ((int)threadIdx.x == fan - 1) t.off[fan] = excl + c;
  }
  __syncthreads();
}

// FULL in what follows: every record of the tile exists and takes part, so that nothing is asked about single ones.  For key
// words only: with 64-bit keys the two variants in one kernel spill 412 to 540 bytes per thread, and level 1 / level 2 of 90M rows
// took 1011 / 943 us instead of 785 / 714.

// A tile's records into the staging arrays, and their places there (pos[j]: the digit in the upper, the rank in the lower 16
// bits).  `flagged`: bit 15 of the staged digit says that the record's one value is null.
template <bool FULL, typename K>
__device__ __forceinline__ void rp_stage_keys(const RpTile<K>& t, const K (&kk)[RP_ROWS], u32 (&pos)[RP_ROWS], u32 act, u32 vok)
{
#pragma unroll
  for (int j = 0; j < RP_ROWS; ++j) {
    if (!FULL && !((act >> j) & 1u)) continue;
    const u32 d = pos[j] >> 16;
    pos[j] = t.off[d] + (pos[j] & 0xFFFFu);
    t.keys[pos[j]] = kk[j];
    if (sizeof(K) == 8) t.dig[pos[j]] = (unsigned short)(d | (((vok >> j) & 1u) ? 0u : 0x8000u));  // (digits stay below 2^RP_MAX_BITS)
  }
}
// my records' values into the staging array (32-bit ones as 32-bit words)
template <bool FULL, typename K>
__device__ __forceinline__ void rp_stage_values(const RpTile<K>& t, int kind, const u64 (&v)[RP_ROWS], const u32 (&pos)[RP_ROWS], u32 act)
{
  if (kind == RK_64) {
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) if (FULL || ((act >> j) & 1u)) t.vals[pos[j]] = v[j];
  } else {
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) if (FULL || ((act >> j) & 1u)) ((u32*)t.vals)[pos[j]] = (u32)v[j];
  }
}
// where the staged record at position p goes
template <typename K>
__device__ __forceinline__ u32 rp_target(const RpTile<K>& t, const DScatter& D, u32 p)
{
  if constexpr (sizeof(K) == 8) return t.base[t.dig[p] & 0x7FFFu] + p;
  else return t.base[(t.keys[p] >> D.shift) & ((u32)D.fan - 1u)] + p;
}
// the staged values to their places (with the keys, or behind them)
template <bool FULL, bool KEYS, typename V, typename K>
__device__ __forceinline__ void rp_copy(const RpTile<K>& t, const DScatter& D, V* __restrict__ dst, u32 n, bool flagged)
{
#pragma unroll
  for (int i = 0; i < RP_ROWS; ++i) {
    const u32 p = threadIdx.x + (u32)i * RPS_BLOCK;
    if (!FULL && p >= n) break;
    const u32 at = rp_target(t, D, p);
    if (KEYS) {
      ((K*)D.dst.key)[at] = t.keys[p];
      if (flagged) D.dst.valid[at] = (unsigned short)((t.dig[p] >> 15) ^ 1u);
    }
    if (sizeof(V) != 1) dst[at] = sizeof(V) == 8 ? (V)t.vals[p] : (V)((const u32*)t.vals)[p];
  }
}
template <bool FULL, bool KEYS, typename K>
__device__ __forceinline__ void rp_copy_column(const RpTile<K>& t, const DScatter& D, int col, u32 n, bool flagged)
{
  if (KEYS && col >= D.dst.nvals) rp_copy<FULL, KEYS>(t, D, (unsigned char*)nullptr, n, flagged);  // (keys alone)
  else if (D.dst.kind[col] == RK_64) rp_copy<FULL, KEYS>(t, D, (u64*)D.dst.val[col], n, flagged);
  else rp_copy<FULL, KEYS>(t, D, (u32*)D.dst.val[col], n, flagged);
}
__device__ __forceinline__ int rp_next_col(const DRecords& R, int col)
{
  while (col < R.nvals && R.kind[col] == RK_NONE) ++col;
  return col;
}
// What follows a tile's first column: staged keys and values `vv` of column col0 are copied out, then the further columns and
// the validity words one after the other through the value array.  `load(col, v)`, `load_valid(v)`: this thread's records'.
template <bool FULL, typename K, typename Load, typename LoadValid>
__device__ __forceinline__ void rp_place(const RpTile<K>& t, const DScatter& D, int col0, bool flagged, const K (&kk)[RP_ROWS], u64 (&vv)[RP_ROWS],
                                         u32 (&pos)[RP_ROWS], u32 act, u32 vok, Load&& load, LoadValid&& load_valid)
{
  const DRecords& R = D.dst;
  rp_stage_keys<FULL>(t, kk, pos, act, vok);
  if (col0 < R.nvals) rp_stage_values<FULL>(t, R.kind[col0], vv, pos, act);
  __syncthreads();
  const u32 n = FULL ? (u32)RP_TILE : t.off[D.fan];
  rp_copy_column<FULL, true>(t, D, col0, n, flagged);
  for (int col = rp_next_col(R, col0 + 1); col < R.nvals; col = rp_next_col(R, col + 1)) {
    load(col, vv);
    __syncthreads();
    rp_stage_values<FULL>(t, R.kind[col], vv, pos, act);
    __syncthreads();
    rp_copy_column<FULL, false>(t, D, col, n, false);
  }
  if (R.valid && !flagged) {
    load_valid(vv);
    __syncthreads();
    rp_stage_values<FULL>(t, RK_U32, vv, pos, act);
    __syncthreads();
    rp_copy<FULL, false>(t, D, R.valid, n, false);
  }
}

// first of the 4 consecutive rows of group g of this thread
constexpr int RP_GROUPS = RP_ROWS / 4;
__device__ __forceinline__ i64 rp_row0(i64 tile, int g) { return tile * RP_TILE + (i64)g * (RP_TILE / RP_GROUPS) + (i64)threadIdx.x * 4; }

// values of this thread's rows, 4 at a time where the column's alignment allows it (`vec`)
__device__ __forceinline__ void rp_load_values(const DPlan& P, int col, int kind, bool vec, i64 tile, u64 (&v)[RP_ROWS])
{
  const DValCol& c = P.vals[col];
#pragma unroll
  for (int g = 0; g < RP_GROUPS; ++g) {
    const i64 row0 = rp_row0(tile, g);
    if (vec && row0 + 4 <= P.nrows) {
      if (c.vclass == VC_F32 || c.vclass == VC_I32 || c.vclass == VC_U32) {
        const uint4 q = __ldg((const uint4*)(c.data + (c.offset + row0) * 4));
        v[4 * g] = q.x; v[4 * g + 1] = q.y; v[4 * g + 2] = q.z; v[4 * g + 3] = q.w;
      } else {
        const ulonglong2* src = (const ulonglong2*)(c.data + (c.offset + row0) * 8);
        const ulonglong2 a = __ldg(src), b = __ldg(src + 1);
        v[4 * g] = a.x; v[4 * g + 1] = a.y; v[4 * g + 2] = b.x; v[4 * g + 3] = b.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[4 * g + j] = row0 + j < P.nrows ? stored_value(c, kind, row0 + j) : 0ull;
    }
  }
}

// level 1: input rows -> records in the region of their digit
// (`hot_rows`: one bit per row, set for the rows whose keys k_rp_count folded already — they are left out here;
// `vec_cols`: value columns of 4- or 8-byte elements that take 16-byte loads at multiples of 4 rows;
// `every_row`: no row is left out for a filter, a null key or a hot one)
template <bool WORDS, bool FULL>
__device__ __forceinline__ void rp_scatter_tile(const DPlan& P, const DScatter& D, const RpTile<typename RpKey<WORDS>::T>& t, i64 tile,
                                                const u32* __restrict__ hot_rows, u32 vec_cols, int col0, bool flagged)
{
  using K = typename RpKey<WORDS>::T;
  const DRecords& R = D.dst;
  const u32 dmask = (u32)D.fan - 1u;
  K kk[RP_ROWS];
  u64 vv[RP_ROWS];
  u32 pos[RP_ROWS];
  u32 act = 0, vok = 0xFFFFFFFFu;
  // keys (and values of the first column), digits, ranks inside the tile
  if (col0 < R.nvals) rp_load_values(P, col0, R.kind[col0], (vec_cols >> col0) & 1u, tile, vv);
#pragma unroll
  for (int g = 0; g < RP_GROUPS; ++g) {
    const i64 row0 = rp_row0(tile, g);
    const int nv = FULL ? 4 : (int)max((i64)0, min((i64)4, P.nrows - row0));
    u32 a4;
    if constexpr (WORDS) {
      u32 w4[4], bad = 0, most = 0;
      rp_words4(P, D.word, row0, nv, w4, a4, bad, most);
#pragma unroll
      for (int j = 0; j < 4; ++j) kk[4 * g + j] = word_place(w4[j]);
    } else {
      u64 k4[4];
      rp_keys4(P, row0, nv, k4, a4);
#pragma unroll
      for (int j = 0; j < 4; ++j) kk[4 * g + j] = k4[j];
    }
    if (hot_rows && nv > 0) a4 &= ~(__ldg(hot_rows + (row0 >> 5)) >> (row0 & 31));  // (row0 is a multiple of 4)
    act |= a4 << (4 * g);
    if (flagged && nv > 0) vok = (vok & ~(0xFu << (4 * g))) | (valid_nibble(P.vals[0].mask, P.vals[0].offset + row0, nv) << (4 * g));
  }
#pragma unroll
  for (int j = 0; j < RP_ROWS; ++j) {
    if (!FULL && !((act >> j) & 1u)) continue;
    const u32 d = rp_digit(kk[j], D.shift) & dmask;
    pos[j] = (d << 16) | atomicAdd(&t.hist[d], 1u);  // (a tile holds 4096 rows: the rank fits 16 bits)
  }
  if constexpr (WORDS) {
    if (R.valid_at >= 0) {
#pragma unroll
      for (int g = 0; g < RP_GROUPS; ++g) {
        const i64 row0 = rp_row0(tile, g);
        if (!FULL && row0 >= P.nrows) continue;
        for (int v = 0; v < R.nvals; ++v) {
          const u32 nib = P.vals[v].mask ? valid_nibble(P.vals[v].mask, P.vals[v].offset + row0, (int)min((i64)4, P.nrows - row0)) : 0xFu;
#pragma unroll
          for (int j = 0; j < 4; ++j) kk[4 * g + j] |= ((nib >> j) & 1u) << (R.valid_at + v);
        }
      }
    }
  }
  rp_tile_plan(t, D.cursors, D.fan);
  rp_place<FULL>(t, D, col0, flagged, kk, vv, pos, act, vok,
                 [&](int col, u64 (&v)[RP_ROWS]) { rp_load_values(P, col, R.kind[col], (vec_cols >> col) & 1u, tile, v); },
                 [&](u64 (&v)[RP_ROWS]) {
#pragma unroll
                   for (int j = 0; j < RP_ROWS; ++j) {
                     const i64 row = rp_row0(tile, j >> 2) + (j & 3);
                     v[j] = 0;
                     if (FULL || ((act >> j) & 1u)) for (int i = 0; i < R.nvals; ++i) v[j] |= (u64)value_valid(P.vals[i], row) << i;
                   }
                 });
}

template <bool WORDS>
__global__ void __launch_bounds__(RPS_BLOCK, 2) k_rp_scatter(const __grid_constant__ DPlan P, const __grid_constant__ DScatter D,
                                                          const u32* __restrict__ hot_rows, u32 vec_cols, bool every_row)
{
  using K = typename RpKey<WORDS>::T;
  extern __shared__ __align__(16) unsigned char rp_stage[];
  const RpTile<K> t = rp_tile_carve<K>(rp_stage, D.fan);
  const bool flagged = !WORDS && D.dst.valid && D.dst.nvals == 1;  // one value column: its validity travels beside the staged digit
  for (int i = threadIdx.x; i < D.fan; i += blockDim.x) t.hist[i] = 0;
  __syncthreads();
  const i64 ntiles = (P.nrows + RP_TILE - 1) / RP_TILE;
  const int col0 = rp_next_col(D.dst, 0);
  for (i64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (WORDS && every_row && (tile + 1) * RP_TILE <= P.nrows) rp_scatter_tile<WORDS, true>(P, D, t, tile, nullptr, vec_cols, col0, flagged);
    else rp_scatter_tile<WORDS, false>(P, D, t, tile, hot_rows, vec_cols, col0, flagged);
  }
}

// Level 2 works on the tiles of the level-1 partitions: tile t belongs to the partition p with
// tile_start[p] <= t < tile_start[p + 1] and covers records [start[p] + j * RP_TILE, ...) of it.  A CTA takes consecutive
// tiles, so that it stays inside a few partitions.
struct DLevel2 {
  DRecords src;
  const u64* src_start;   // [parts + 1] first record of every source partition
  const u64* src_end;     // [parts] one past its last record (the advanced level-1 cursors)
  const u32* tile_start;  // [parts + 1] first tile of every source partition
  int parts;
};

__device__ __forceinline__ int rp_partition_of_tile(const u32* tile_start, int parts, u32 tile)
{
  int lo = 0, hi = parts;  // tile_start[lo] <= tile < tile_start[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(tile_start + mid) <= tile) lo = mid; else hi = mid;
  }
  return lo;
}

// rows per (source partition, level-2 digit)
template <bool WORDS>
__global__ void __launch_bounds__(RPS_BLOCK, 4) k_rp_count2(const __grid_constant__ DLevel2 L, int shift, int fan, u64* __restrict__ hist2)
{
  using K = typename RpKey<WORDS>::T;
  __shared__ u32 s_hist[1 << RP_MAX_BITS];
  for (int i = threadIdx.x; i < fan; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  const u32 ntiles = __ldg(L.tile_start + L.parts);
  const u32 dmask = (u32)fan - 1u;
  const u32 per = (ntiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per, last = min(ntiles, first + per);
  for (u32 tile = first; tile < last;) {
    // the rest of this CTA's tiles inside one partition: one run of records
    const int p = rp_partition_of_tile(L.tile_start, L.parts, tile);
    const u32 t0 = __ldg(L.tile_start + p), t1 = min(last, __ldg(L.tile_start + p + 1));
    const i64 lo = (i64)L.src_start[p] + (i64)(tile - t0) * RP_TILE;
    const i64 hi = min((i64)L.src_end[p], (i64)L.src_start[p] + (i64)(t1 - t0) * RP_TILE);
    for (i64 base = lo; base < hi; base += RP_TILE) {
      const int have = (int)min((i64)RP_TILE, hi - base) - (int)threadIdx.x;  // record j exists: j * RPS_BLOCK < have
      const K* src = (const K*)L.src.key + base + threadIdx.x;
      K k[RP_ROWS];
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) k[j] = j * RPS_BLOCK < have ? __ldg(src + j * RPS_BLOCK) : (K)0;
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) if (j * RPS_BLOCK < have) atomicAdd(&s_hist[rp_digit(k[j], shift) & dmask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < fan; d += blockDim.x) {
      const u32 c = s_hist[d];
      s_hist[d] = 0;
      if (c) atomicAdd(&hist2[(i64)p * fan + d], (u64)c);
    }
    __syncthreads();
    tile = t1;
  }
}

template <bool WORDS, bool FULL>
__device__ __forceinline__ void rp_scatter2_tile(const DRecords& S, const DScatter& D, const RpTile<typename RpKey<WORDS>::T>& t, i64 lo, int records,
                                                 u64* cursors, int col0, bool flagged)
{
  using K = typename RpKey<WORDS>::T;
  const DRecords& R = D.dst;
  const u32 dmask = (u32)D.fan - 1u;
  const int have = records - (int)threadIdx.x;  // record j exists: j * RPS_BLOCK < have
  K kk[RP_ROWS];
  u64 vv[RP_ROWS];
  u32 pos[RP_ROWS];
  u32 act = 0, vok = 0xFFFFFFFFu;
  auto load_values = [&](int col, u64 (&v)[RP_ROWS]) {
    if (R.kind[col] == RK_64) {
      const u64* src = (const u64*)S.val[col] + lo + threadIdx.x;
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) v[j] = FULL || j * RPS_BLOCK < have ? __ldg(src + j * RPS_BLOCK) : 0ull;
    } else {
      const u32* src = (const u32*)S.val[col] + lo + threadIdx.x;
#pragma unroll
      for (int j = 0; j < RP_ROWS; ++j) v[j] = FULL || j * RPS_BLOCK < have ? (u64)__ldg(src + j * RPS_BLOCK) : 0ull;
    }
  };
  const K* src = (const K*)S.key + lo + threadIdx.x;
#pragma unroll
  for (int j = 0; j < RP_ROWS; ++j) {
    kk[j] = 0;
    if (!FULL && j * RPS_BLOCK >= have) continue;
    act |= 1u << j;
    kk[j] = __ldg(src + j * RPS_BLOCK);
    if (flagged && !(__ldg(S.valid + lo + j * RPS_BLOCK + threadIdx.x) & 1u)) vok &= ~(1u << j);
  }
  if (col0 < R.nvals) load_values(col0, vv);
#pragma unroll
  for (int j = 0; j < RP_ROWS; ++j) {
    if (!FULL && !((act >> j) & 1u)) continue;
    const u32 d = rp_digit(kk[j], D.shift) & dmask;
    pos[j] = (d << 16) | atomicAdd(&t.hist[d], 1u);
  }
  rp_tile_plan(t, cursors, D.fan);
  rp_place<FULL>(t, D, col0, flagged, kk, vv, pos, act, vok, load_values, [&](u64 (&v)[RP_ROWS]) {
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) v[j] = FULL || j * RPS_BLOCK < have ? (u64)__ldg(S.valid + lo + j * RPS_BLOCK + threadIdx.x) : 0ull;
  });
}

// The next tile's records on their way into L2 while this one is sorted: the loads that a tile begins with then wait for L2, not
// for DRAM (4 to 8 % of this kernel; in front of level 1, whose tiles lie apart, it cost as much as it gave).  `bytes` from `p`
// on, a line per thread.
__device__ __forceinline__ void rp_prefetch(const unsigned char* p, i64 bytes)
{
  for (i64 at = (i64)threadIdx.x * 128; at < bytes; at += (i64)RPS_BLOCK * 128) prefetch_l2(p + at);
}

template <bool WORDS>
__global__ void __launch_bounds__(RPS_BLOCK, 2) k_rp_scatter2(const __grid_constant__ DLevel2 L, const __grid_constant__ DScatter D)
{
  using K = typename RpKey<WORDS>::T;
  extern __shared__ __align__(16) unsigned char rp_stage[];
  const RpTile<K> t = rp_tile_carve<K>(rp_stage, D.fan);
  for (int i = threadIdx.x; i < D.fan; i += blockDim.x) t.hist[i] = 0;
  __syncthreads();
  const u32 ntiles = __ldg(L.tile_start + L.parts);
  const int col0 = rp_next_col(D.dst, 0);
  const bool flagged = !WORDS && D.dst.valid && D.dst.nvals == 1;
  const u32 per = (ntiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per, last = min(ntiles, first + per);
  int p = first < last ? rp_partition_of_tile(L.tile_start, L.parts, first) : 0;
  for (u32 tile = first; tile < last; ++tile) {
    while (tile >= __ldg(L.tile_start + p + 1)) ++p;
    const i64 lo = (i64)L.src_start[p] + (i64)(tile - __ldg(L.tile_start + p)) * RP_TILE;
    const int records = (int)min((i64)RP_TILE, (i64)L.src_end[p] - lo);
    u64* cursors = D.cursors + (i64)p * D.fan;
    if (lo + 2 * RP_TILE <= (i64)L.src_end[p]) {  // (the next tile of this partition)
      rp_prefetch(L.src.key + (lo + RP_TILE) * (i64)sizeof(K), RP_TILE * (i64)sizeof(K));
      if (col0 < D.dst.nvals) {
        const int w = D.dst.kind[col0] == RK_64 ? 8 : 4;
        rp_prefetch(L.src.val[col0] + (lo + RP_TILE) * w, (i64)RP_TILE * w);
      }
    }
    if (WORDS && records == RP_TILE) rp_scatter2_tile<WORDS, true>(L.src, D, t, lo, records, cursors, col0, flagged);
    else rp_scatter2_tile<WORDS, false>(L.src, D, t, lo, records, cursors, col0, flagged);
  }
}

// first record of every level-1 partition by the top-level histogram (`fold` of its digits each), as starts and as cursors.  One CTA
// of at least `fan` threads.  (Two copies of what the host had added up cost 15 us per call.)
__global__ void __launch_bounds__(1 << RP_MAX_BITS) k_rp_starts(const u64* __restrict__ hist, int fold, int fan, u64* __restrict__ start, u64* __restrict__ cursor)
{
  __shared__ u64 s_sum[1 << RP_MAX_BITS];
  const int d = (int)threadIdx.x;
  u64 mine = 0;
  if (d < fan) for (int j = 0; j < fold; ++j) mine += hist[d * fold + j];
  s_sum[d] = mine;
  __syncthreads();
  for (int step = 1; step < (int)blockDim.x; step <<= 1) {
    const u64 t = d >= step ? s_sum[d - step] : 0ull;
    __syncthreads();
    s_sum[d] += t;
    __syncthreads();
  }
  if (d < fan) { start[d] = s_sum[d] - mine; cursor[d] = s_sum[d] - mine; }
  if (d == fan - 1) start[fan] = s_sum[d];
}

// tiles per source partition from its record count (one thread per partition), then scanned on the device
__global__ void k_rp_tiles(const u64* __restrict__ start, const u64* __restrict__ end, int parts, u32* __restrict__ tile_start)
{
  // single CTA: exclusive scan of ceil(count / RP_TILE)
  __shared__ u32 s_sum[1024];
  u32 mine = 0;
  const int per = (parts + (int)blockDim.x - 1) / (int)blockDim.x;
  const int lo = threadIdx.x * per, hi = min(parts, lo + per);
  for (int p = lo; p < hi; ++p) mine += (u32)((end[p] - start[p] + RP_TILE - 1) / RP_TILE);
  s_sum[threadIdx.x] = mine;
  __syncthreads();
  for (int d = 1; d < (int)blockDim.x; d <<= 1) {
    const u32 t = threadIdx.x >= (u32)d ? s_sum[threadIdx.x - d] : 0u;
    __syncthreads();
    s_sum[threadIdx.x] += t;
    __syncthreads();
  }
  u32 run = s_sum[threadIdx.x] - mine;
  for (int p = lo; p < hi; ++p) {
    tile_start[p] = run;
    run += (u32)((end[p] - start[p] + RP_TILE - 1) / RP_TILE);
  }
  if (threadIdx.x == blockDim.x - 1) tile_start[parts] = s_sum[threadIdx.x];
}

// ------------------------------------------------------------------------------ bucket aggregate
struct DBuckets {
  DRecords src;
  DWord word;
  const u64* start;  // [buckets] first record of every bucket
  const u64* end;    // [buckets] one past its last record
  i64 nbuckets;
  int slots;         // slots of a bucket's shared-memory table.  Hashed 64-bit keys: a power of two; slot `slots` holds the key
                     // whose bits equal EMPTY.  Key words: a multiple of 2^low_bits
  int low_bits;      // key words: WORD_LOW less the digits' bits
  u64* out;          // finished groups, structure-of-arrays: word w of group g at out[w * out_cap + g]; word 0 = key
  i64 out_cap;
  u64* next_bucket;  // work counter
  int index_at;                        // byte offset of the claim-order index (hashed) or of the "seen" bits (words) in shared memory
  int cell_at[MAX_CELLS];              // ... of every cell's array (not FIXED)
  unsigned char form[MAX_CELLS];       // CellForm
  signed char count_of[MAX_CELLS];     // CF_MIN32 / CF_MAX32: the cell that counts the column's values, -1: no value is null
  int present;                         // key words: a cell whose count tells that a slot is used, -1: none
  int seen_col;                        // ... the value column whose null values leave that count alone (their rows set the
                                       // slot's bit), -1: there is none (or, without `present`, every row sets its bit)
};

// values of 4 records, RPA_BLOCK apart, in their carried form; record j exists where j * RPA_BLOCK < have (FULL: all do)
template <bool FULL>
__device__ __forceinline__ void rec_values4(const DRecords& R, int col, i64 first, int have, u64 (&v)[4])
{
#define B2_VALUES(T, EXPR)                                                                         \
  {                                                                                                \
    const T* src = (const T*)R.val[col] + first;                                                   \
    _Pragma("unroll") for (int j = 0; j < 4; ++j) {                                                \
      const T x = FULL || j * RPA_BLOCK < have ? __ldg(src + j * RPA_BLOCK) : (T)0;                \
      v[j] = EXPR;                                                                                 \
    }                                                                                              \
    break;                                                                                         \
  }
  switch (R.kind[col]) {
    case RK_64: B2_VALUES(u64, x)
    case RK_F32: B2_VALUES(u32, float_carried(x))
    case RK_S32: B2_VALUES(int, (u64)(i64)x)
    case RK_U32: B2_VALUES(u32, (u64)x)
    default: break;
  }
#undef B2_VALUES
}

// FIXED (the cells are Σx / n / Σx² of one float column): a slot keeps its sums as fixed point (fx_add) plus one
// fp64 cell each for what does not fit the window (and for the periodic flushes), and its count as 32 bits: five to nine
// native 32-bit atomics per record (the count, two or three words of each sum and rarely its top word) instead of three
// 64-bit ones, which shared memory only does as compare-and-swap loops.  `hot_info`: DHot::info, the magnitudes among the
// sampled values.
constexpr int RPA_FIXED_SLOT_BYTES = 8 + 8 + 4 + 8 * FX_WORDS;  // beside the key and the claim-order index
constexpr int RPA_INDEX_BYTES = 2;  // per slot: the claim-order index

template <bool FIXED>
__global__ void __launch_bounds__(RPA_BLOCK, 2) k_rp_aggregate(const __grid_constant__ DPlan P, const __grid_constant__ DBuckets B, DCtrl* ctrl,
                                                            const u32* __restrict__ hot_info)
{
  using K = u64;
  constexpr K NONE = EMPTY;
  extern __shared__ __align__(16) unsigned char rp_smem[];
  __shared__ i64 s_bucket;
  __shared__ u32 s_count, s_fail, s_special;
  __shared__ u64 s_outbase;
  const int S  = B.slots;
  const int NS = S + 1;
  K* skeys    = (K*)rp_smem;     // [NS]
  // FIXED: [NS] fp64 Σx beside the fixed point, [NS] the same for Σx², [NS] counts, words of Σx, words of Σx²
  double* fex = (double*)(skeys + NS);
  double* feq = fex + NS;
  u32* fcnt   = (u32*)(feq + NS);
  u32* flx    = fcnt + NS;
  u32* flq    = flx + FX_WORDS * NS;
  const u32 fcnt_a = (u32)__cvta_generic_to_shared(fcnt), flx_a = (u32)__cvta_generic_to_shared(flx), flq_a = (u32)__cvta_generic_to_shared(flq);
  // slots in the order they were claimed: the finished groups are written in that order, consecutive
  // threads to consecutive list entries, without scanning the table for occupied slots
  unsigned short* sidx = (unsigned short*)(rp_smem + B.index_at);
  int fx_bx = FX_NEVER, fx_bq = FX_NEVER, c_sum = -1, c_cnt = -1, c_ssq = -1;
  if (FIXED) {
    if (hot_info[3]) {
      const int mean = (int)(hot_info[2] / hot_info[3]), emax = (int)hot_info[1] - 1;
      fx_bx = fx_base(mean, emax);
      fx_bq = fx_base_sq(mean, emax);
    }
    for (int c = 0; c < P.ncells; ++c) {
      if (P.cells[c].op == OP_SUM_F) c_sum = c;
      if (P.cells[c].op == OP_CNT_V) c_cnt = c;
      if (P.cells[c].op == OP_SSQ_F) c_ssq = c;
    }
  }
  const u32 smask = (u32)S - 1u;
  // a bucket whose groups fill the table beyond this gives up (the caller falls back to the global table)
  const u32 fill_limit = (u32)S - (u32)(S >> 3);
  // the first two value columns of the records are loaded together with the keys
  const int col0 = rp_next_col(B.src, 0), col1 = rp_next_col(B.src, col0 + 1);
  i64 next = 0;  // (thread 0) the bucket after this one, asked for ahead of its use
  if (threadIdx.x == 0) next = (i64)atomicAdd(B.next_bucket, 1ull);

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      s_bucket = next; s_count = 0; s_fail = 0; s_special = 0;
      if (next < B.nbuckets) next = (i64)atomicAdd(B.next_bucket, 1ull);
    }
    __syncthreads();
    const i64 b = s_bucket;
    if (b >= B.nbuckets) break;
    const i64 lo = (i64)B.start[b], hi = (i64)B.end[b];
    if (hi <= lo) continue;
    // clear the table
    for (int i = threadIdx.x; i < NS; i += blockDim.x) skeys[i] = NONE;
    if (FIXED) {
      for (int i = threadIdx.x; i < 2 * NS; i += blockDim.x) fex[i] = 0.0;                        // fex, feq
      for (int i = threadIdx.x; i < (1 + 2 * FX_WORDS) * NS; i += blockDim.x) fcnt[i] = 0;        // fcnt, flx, flq
    } else {
      for (int c = 0; c < P.ncells; ++c) {
        if (B.form[c] == CF_64) {
          const u64 id = cell_identity(P.cells[c].op);
          u64* cell = (u64*)(rp_smem + B.cell_at[c]);
          for (int i = threadIdx.x; i < NS; i += blockDim.x) cell[i] = id;
        } else {
          u32* cell = (u32*)(rp_smem + B.cell_at[c]);
          const u32 id = B.form[c] == CF_MIN32 ? 0xFFFFFFFFu : 0u;
          const int words = B.form[c] == CF_SUM ? 2 * NS : NS;
          for (int i = threadIdx.x; i < words; i += blockDim.x) cell[i] = id;
        }
      }
    }
    __syncthreads();
    // fold the records, RPA_BATCH per thread at a time: all loads of a batch are issued before the first
    // probe, so that a batch costs one DRAM round trip instead of one per record and word
    for (i64 base = lo; base < hi; base += (i64)RPA_BATCH * blockDim.x) {
      K keys[RPA_BATCH];
      u64 vals[RPA_BATCH] = {}, vals1[RPA_BATCH] = {};
      u32 vbits[RPA_BATCH];
      const i64 first = base + threadIdx.x;
      const int have = (int)min(hi - base, (i64)RPA_BATCH * RPA_BLOCK) - (int)threadIdx.x;  // record j exists: j * RPA_BLOCK < have
      const K* src = (const K*)B.src.key + first;
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) keys[j] = j * RPA_BLOCK < have ? __ldg(src + j * RPA_BLOCK) : 0ull;
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) vbits[j] = B.src.valid && j * RPA_BLOCK < have ? (u32)__ldg(B.src.valid + first + j * RPA_BLOCK) : ~0u;
      if (col0 < B.src.nvals) rec_values4<false>(B.src, col0, first, have, vals);
      if (!FIXED && col1 < B.src.nvals) rec_values4<false>(B.src, col1, first, have, vals1);
      // Slots of the batch's records.  The home slots of all of them are read together; what is not settled by that is probed
      // for in ONE loop, every lane taking its own records in turn: the warp goes round as often as its busiest lane has
      // probes to do, not as often as the longest chain of each record's 32 lanes.
      int slots[RPA_BATCH];
      u32 home[RPA_BATCH], left = 0;
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) {
        home[j] = (u32)rp_hash(keys[j]) & smask;
        slots[j] = -1;
        if (j * RPA_BLOCK >= have) continue;
        if (keys[j] == NONE) { slots[j] = S; s_special = 1; }
        else if (*(volatile K*)(skeys + home[j]) == keys[j]) slots[j] = (int)home[j];
        else left |= 1u << j;
      }
      static_assert(RPA_BATCH == 4, "selects below");
      auto pick = [&](const auto (&a)[RPA_BATCH], u32 bit) { return bit == 1u ? a[0] : bit == 2u ? a[1] : bit == 4u ? a[2] : a[3]; };
      u32 bit = left & (0u - left), idx = pick(home, bit), steps = 0;
      K key = pick(keys, bit);
      while (left) {
        K k = *(volatile K*)(skeys + idx);
        bool full = steps > smask;  // (claims that raced past the limit may have filled the table: a key then meets no free slot)
        if (k == NONE) {
          full = *(volatile u32*)&s_count >= fill_limit;
          if (!full) {
            k = atomicCAS(skeys + idx, NONE, key);
            if (k == NONE) { sidx[atomicAdd(&s_count, 1u)] = (unsigned short)idx; k = key; }
          }
        }
        if (k == key || full) {
          if (full) s_fail = 1;
          else if (bit == 1u) slots[0] = (int)idx;
          else if (bit == 2u) slots[1] = (int)idx;
          else if (bit == 4u) slots[2] = (int)idx;
          else slots[3] = (int)idx;
          left &= left - 1u;
          bit = left & (0u - left);
          idx = pick(home, bit);
          key = pick(keys, bit);
          steps = 0;
        } else {
          idx = (idx + 1u) & smask;
          ++steps;
        }
      }
      // The lanes left the loop at different iterations: bring them back together, then go
      // through the accumulators cell by cell — the operator is decoded once per cell and batch (not
      // once per record), and each update is ONE predicated atomic for the whole warp.  (Diverged,
      // each lane's atomics were issued on their own: 11.5 of 32 lanes active on average.)
      __syncwarp();
      if (FIXED) {
        static_assert(RPA_BATCH == 4, "fx_add4");
        u32 at[4], take = 0, full = 0, unfit = 0;
        u64 qq[4];
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) {
          if (slots[j] >= 0 && (vbits[j] & 1u)) take |= 1u << j;
          if (((fx_atom_if(fcnt_a + 4u * (u32)slots[j], 1u, take & (1u << j)) + 1u) & (FX_FLUSH - 1u)) == 0u) full |= 1u << j;
          at[j] = flx_a + 4u * (u32)slots[j];
          const double d = __longlong_as_double((i64)vals[j]);
          qq[j] = (u64)__double_as_longlong(d * d);
        }
        if (c_sum >= 0) unfit = fx_add4<true>(vals, fx_bx, at, take, 4u * (u32)NS);
        if (c_ssq >= 0) {
#pragma unroll
          for (int j = 0; j < RPA_BATCH; ++j) at[j] += flq_a - flx_a;
          unfit |= fx_add4<false>(qq, fx_bq, at, take, 4u * (u32)NS) << 4;
        }
        if (unfit | full) {
#pragma unroll 1
          for (int j = 0; j < RPA_BATCH; ++j) {
            const int s = j == 0 ? slots[0] : j == 1 ? slots[1] : j == 2 ? slots[2] : slots[3];
            const double d = __longlong_as_double((i64)(j == 0 ? vals[0] : j == 1 ? vals[1] : j == 2 ? vals[2] : vals[3]));
            if ((unfit >> j) & 1u) atomicAdd(fex + s, d);
            if ((unfit >> j) & 16u) atomicAdd(feq + s, d * d);
            if (!((full >> j) & 1u)) continue;
            if (c_sum >= 0) atomicAdd(fex + s, fx_take(flx, NS, s, fx_bx));
            if (c_ssq >= 0) atomicAdd(feq + s, fx_take(flq, NS, s, fx_bq));
          }
        }
      }
      int cur = col0;
      for (int c = 0; !FIXED && c < P.ncells; ++c) {
        const int op = P.cells[c].op, col = P.cells[c].col;
        if (op != OP_CNT_A && op != OP_CNT_V && col != cur) {  // (the cells of a value column are adjacent)
          cur = col;
          if (col == col1) {
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) vals[j] = vals1[j];
          } else {
            rec_values4<false>(B.src, col, first, have, vals);
          }
        }
        u32 ok = 0;  // records of the batch that update this cell
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j)
          if (slots[j] >= 0 && (op == OP_CNT_A || ((vbits[j] >> col) & 1u))) ok |= 1u << j;
        unsigned char* cell = rp_smem + B.cell_at[c];
        const u32 cell_a = (u32)__cvta_generic_to_shared(cell);
        switch (B.form[c]) {
          case CF_COUNT:
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) fx_red_if(cell_a + 4u * (u32)slots[j], 1u, ok & (1u << j));
            break;
          case CF_SUM: {
            u64 x[RPA_BATCH];
            u32 old[RPA_BATCH];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) {
              x[j] = sum_addend(op, vals[j]);
              old[j] = fx_atom_if(cell_a + 4u * (u32)slots[j], (u32)x[j], ok & (1u << j));
            }
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) {
              const u32 up = (u32)(x[j] >> 32) + (old[j] > ~(u32)x[j] ? 1u : 0u);
              fx_red_if(cell_a + 4u * (u32)(NS + slots[j]), up, (ok & (1u << j)) ? up : 0u);
            }
            break;
          }
          case CF_MIN32: case CF_MAX32: {
            const int kind = B.src.kind[col];
            const bool least = B.form[c] == CF_MIN32;
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) {
              if (!((ok >> j) & 1u)) continue;
              const u32 o = order32(kind, vals[j]);
              if (least) atomicMin((u32*)cell + slots[j], o); else atomicMax((u32*)cell + slots[j], o);
            }
            break;
          }
          default: {
            u64* where[RPA_BATCH];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) where[j] = (u64*)cell + (slots[j] >= 0 ? slots[j] : 0);
            cell_update_shared<RPA_BATCH>(where, op, vals, ok);
          }
        }
      }
    }
    __syncthreads();
    if (s_fail) { if (threadIdx.x == 0) ctrl->overflow = 1; continue; }
    // compact the occupied slots into the group list
    const u32 ngroups = s_count + s_special;
    if (threadIdx.x == 0) {
      s_outbase = atomicAdd(&ctrl->out_cursor, (u64)ngroups);
      if (s_outbase + ngroups > (u64)B.out_cap) ctrl->overflow = 1;
    }
    __syncthreads();
    if (s_outbase + ngroups > (u64)B.out_cap) continue;
    for (u32 pos = threadIdx.x; pos < ngroups; pos += blockDim.x) {
      const int i = pos < s_count ? (int)sidx[pos] : S;  // (the special slot, if used, comes last)
      const i64 g = (i64)s_outbase + pos;
      B.out[g] = i < S ? skeys[i] : EMPTY;
      if (FIXED) {
        if (c_cnt >= 0) B.out[(i64)(1 + c_cnt) * B.out_cap + g] = (u64)fcnt[i];
        if (c_sum >= 0) B.out[(i64)(1 + c_sum) * B.out_cap + g] = (u64)__double_as_longlong(fex[i] + fx_take(flx, NS, i, fx_bx));
        if (c_ssq >= 0) B.out[(i64)(1 + c_ssq) * B.out_cap + g] = (u64)__double_as_longlong(feq[i] + fx_take(flq, NS, i, fx_bq));
      } else {
        for (int c = 0; c < P.ncells; ++c) {
          const unsigned char* cell = rp_smem + B.cell_at[c];
          u64 v;
          switch (B.form[c]) {
            case CF_64: v = ((const u64*)cell)[i]; break;
            case CF_COUNT: v = ((const u32*)cell)[i]; break;
            case CF_SUM: v = ((u64)((const u32*)cell)[NS + i] << 32) | ((const u32*)cell)[i]; break;
            default: {
              // (a group without a valid value keeps the identity, whatever image that word is of)
              const int n = B.count_of[c];
              const bool any = n < 0 || ((const u32*)(rp_smem + B.cell_at[n]))[i] != 0u;
              v = any ? unorder32(B.src.kind[P.cells[c].col], ((const u32*)cell)[i]) : cell_identity(P.cells[c].op);
            }
          }
          B.out[(i64)(1 + c) * B.out_cap + g] = v;
        }
      }
    }
  }
}

// The same for records with key words: the accumulators of a bucket are addressed by what its digits leave of the word, so
// there are no keys in shared memory and nothing is probed for.  Arrays start at multiples of 16 bytes.
__device__ __forceinline__ void fill_shared(unsigned char* p, u64 v, int bytes)
{
  for (int i = (int)threadIdx.x * 16; i < bytes; i += (int)blockDim.x * 16) *(ulonglong2*)(p + i) = make_ulonglong2(v, v);
}

// Two 32-bit adds per record for a count and an integer sum, one for a minimum or maximum of a narrow value.  What a cell asks
// for is decoded once per batch of 4 records and thread.  LIST: the groups go to a list (partial aggregates that travel), else
// straight into the output columns: 10^8 groups with four results of 8 bytes saved a list of 4 GB, written and read.
template <bool FIXED, bool LIST>
__global__ void __launch_bounds__(RPA_BLOCK, 2) k_rp_direct(const __grid_constant__ DPlan P, const __grid_constant__ DBuckets B, DCtrl* ctrl,
                                                         const u32* __restrict__ hot_info, const __grid_constant__ DOutPlan O)
{
  extern __shared__ __align__(16) unsigned char rp_smem[];
  __shared__ i64 s_bucket;
  __shared__ u32 s_total;
  __shared__ u64 s_outbase;
  const int S = B.slots;
  // FIXED: [S] fp64 Σx beside the fixed point, [S] the same for Σx², [S] counts, words of Σx, words of Σx²
  double* fex = (double*)rp_smem;
  double* feq = fex + S;
  u32* fcnt   = (u32*)(feq + S);
  u32* flx    = fcnt + S;
  u32* flq    = flx + FX_WORDS * S;
  const u32 fcnt_a = (u32)__cvta_generic_to_shared(fcnt), flx_a = (u32)__cvta_generic_to_shared(flx), flq_a = (u32)__cvta_generic_to_shared(flq);
  const u32 smem_a = (u32)__cvta_generic_to_shared(rp_smem);
  u32* const seen = (u32*)(rp_smem + B.index_at);
  const int seen_bytes = (S + 127) / 128 * 16;
  int fx_bx = FX_NEVER, fx_bq = FX_NEVER, c_sum = -1, c_cnt = -1, c_ssq = -1;
  if (FIXED) {
    if (hot_info[3]) {
      const int mean = (int)(hot_info[2] / hot_info[3]), emax = (int)hot_info[1] - 1;
      fx_bx = fx_base(mean, emax);
      fx_bq = fx_base_sq(mean, emax);
    }
    for (int c = 0; c < P.ncells; ++c) {
      if (P.cells[c].op == OP_SUM_F) c_sum = c;
      if (P.cells[c].op == OP_CNT_V) c_cnt = c;
      if (P.cells[c].op == OP_SSQ_F) c_ssq = c;
    }
  }
  const u32 low_mask = (1u << B.low_bits) - 1u;
  const int down = WORD_LOW - B.low_bits;
  const u32 high_mask = (B.src.key_mask >> down) & ~low_mask;
  const bool in_word = B.src.valid_at >= 0, nullable = in_word || B.src.valid;
  const bool sees_all = !FIXED && B.present < 0, sees = sees_all || B.seen_col >= 0;
  const int col0 = rp_next_col(B.src, 0), col1 = rp_next_col(B.src, col0 + 1);
  const u32 wid = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  i64 next = 0;  // (thread 0) the bucket after this one, asked for ahead of its use
  if (threadIdx.x == 0) next = (i64)atomicAdd(B.next_bucket, 1ull);

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      s_bucket = next; s_total = 0;
      if (next < B.nbuckets) next = (i64)atomicAdd(B.next_bucket, 1ull);
    }
    __syncthreads();
    const i64 b = s_bucket;
    if (b >= B.nbuckets) break;
    const i64 lo = (i64)B.start[b], hi = (i64)B.end[b];
    if (hi <= lo) continue;
    if (FIXED) {
      fill_shared(rp_smem, 0, B.index_at + seen_bytes);
    } else {
      for (int c = 0; c < P.ncells; ++c) {
        const int form = B.form[c], bytes = (S * cell_form_bytes(form) + 15) / 16 * 16;
        fill_shared(rp_smem + B.cell_at[c], form == CF_64 ? cell_identity(P.cells[c].op) : form == CF_MIN32 ? ~0ull : 0ull, bytes);
      }
      fill_shared((unsigned char*)seen, 0, seen_bytes);
    }
    // each batch loads the keys and first values of the next one before it works (the bucket's first ones on their way while
    // the table is cleared)
    u32 wn[RPA_BATCH];
    u64 vn[RPA_BATCH];
    const int records = (int)(hi - lo);
    auto load = [&](int at) {
      const int have = records - at - (int)threadIdx.x;
      const u32* src = (const u32*)B.src.key + lo + at + threadIdx.x;
      if (at + RPA_BATCH * RPA_BLOCK <= records) {
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) wn[j] = __ldg(src + j * RPA_BLOCK);
        if (col0 < B.src.nvals) rec_values4<true>(B.src, col0, lo + at + threadIdx.x, have, vn);
      } else {
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) wn[j] = j * RPA_BLOCK < have ? __ldg(src + j * RPA_BLOCK) : 0u;
        if (col0 < B.src.nvals) rec_values4<false>(B.src, col0, lo + at + threadIdx.x, have, vn);
      }
    };
#pragma unroll
    for (int j = 0; j < RPA_BATCH; ++j) vn[j] = 0;
    load(0);
    __syncthreads();
    // FULL: every record of the batch exists and no value is null
    auto batch = [&](auto full_tag, int at) {
      constexpr bool FULL = decltype(full_tag)::value;
      u32 slots[RPA_BATCH], vbits[RPA_BATCH], act = 0;
      u64 vals[RPA_BATCH], vals1[RPA_BATCH] = {};
      const int have = records - at - (int)threadIdx.x;
      const i64 first = lo + at + threadIdx.x;
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) {
        if (FULL || j * RPA_BLOCK < have) act |= 1u << j;
        slots[j] = ((wn[j] >> down) & high_mask) | (wn[j] & low_mask);
        vbits[j] = !FULL && in_word ? wn[j] >> B.src.valid_at : ~0u;
        vals[j] = vn[j];
      }
      if (!FULL && B.src.valid) {
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) if (j * RPA_BLOCK < have) vbits[j] = __ldg(B.src.valid + first + j * RPA_BLOCK);
      }
      if (!FIXED && col1 < B.src.nvals) rec_values4<FULL>(B.src, col1, first, have, vals1);
      load(at + RPA_BATCH * RPA_BLOCK);
      if (FULL ? sees_all : sees) {
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j)
          if (((act >> j) & 1u) && (sees_all || !((vbits[j] >> B.seen_col) & 1u)) && !((seen[slots[j] >> 5] >> (slots[j] & 31u)) & 1u))
            atomicOr(&seen[slots[j] >> 5], 1u << (slots[j] & 31u));
      }
      if (FIXED) {
        static_assert(RPA_BATCH == 4, "fx_add4");
        u32 to[4], take = act, full = 0, unfit = 0;
        u64 qq[4];
        if (!FULL && nullable) {
#pragma unroll
          for (int j = 0; j < RPA_BATCH; ++j) if (!(vbits[j] & 1u)) take &= ~(1u << j);
        }
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) {
          if (((fx_atom_if(fcnt_a + 4u * slots[j], 1u, take & (1u << j)) + 1u) & (FX_FLUSH - 1u)) == 0u) full |= 1u << j;
          to[j] = flx_a + 4u * slots[j];
          const double d = __longlong_as_double((i64)vals[j]);
          qq[j] = (u64)__double_as_longlong(d * d);
        }
        if (c_sum >= 0) unfit = fx_add4<true>(vals, fx_bx, to, take, 4u * (u32)S);
        if (c_ssq >= 0) {
#pragma unroll
          for (int j = 0; j < RPA_BATCH; ++j) to[j] += flq_a - flx_a;
          unfit |= fx_add4<false>(qq, fx_bq, to, take, 4u * (u32)S) << 4;
        }
        if (unfit | full) {
#pragma unroll 1
          for (int j = 0; j < RPA_BATCH; ++j) {
            const int s = (int)(j == 0 ? slots[0] : j == 1 ? slots[1] : j == 2 ? slots[2] : slots[3]);
            const double d = __longlong_as_double((i64)(j == 0 ? vals[0] : j == 1 ? vals[1] : j == 2 ? vals[2] : vals[3]));
            if ((unfit >> j) & 1u) atomicAdd(fex + s, d);
            if ((unfit >> j) & 16u) atomicAdd(feq + s, d * d);
            if (!((full >> j) & 1u)) continue;
            if (c_sum >= 0) atomicAdd(fex + s, fx_take(flx, S, s, fx_bx));
            if (c_ssq >= 0) atomicAdd(feq + s, fx_take(flq, S, s, fx_bq));
          }
        }
        return;
      }
      int cur = col0;
      for (int c = 0; c < P.ncells; ++c) {
        const int op = P.cells[c].op, col = P.cells[c].col, form = B.form[c];
        if (op != OP_CNT_A && op != OP_CNT_V && col != cur) {  // (the cells of a value column are adjacent)
          cur = col;
          if (col == col1) {
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) vals[j] = vals1[j];
          } else {
            rec_values4<FULL>(B.src, col, first, have, vals);
          }
        }
        u32 ok = act;  // records of the batch that update this cell
        if (!FULL && nullable && op != OP_CNT_A) {
#pragma unroll
          for (int j = 0; j < RPA_BATCH; ++j) if (!((vbits[j] >> col) & 1u)) ok &= ~(1u << j);
        }
        const u32 cell_a = smem_a + (u32)B.cell_at[c];
        auto use = [&](int j) { return FULL ? 1u : ok & (1u << j); };
        switch (form) {
          case CF_COUNT:
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) fx_red_if(cell_a + 4u * slots[j], 1u, use(j));
            break;
          case CF_SUM: {
            u64 x[RPA_BATCH];
            u32 old[RPA_BATCH];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) {
              x[j] = op == OP_SUM_I ? vals[j] : sum_addend(op, vals[j]);
              old[j] = fx_atom_if(cell_a + 4u * slots[j], (u32)x[j], use(j));
            }
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) {
              const u32 up = (u32)(x[j] >> 32) + (old[j] > ~(u32)x[j] ? 1u : 0u);
              fx_red_if(cell_a + 4u * ((u32)S + slots[j]), up, use(j) ? up : 0u);
            }
            break;
          }
          case CF_MIN32: {
            const int kind = B.src.kind[col];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) fx_min_if(cell_a + 4u * slots[j], order32(kind, vals[j]), use(j));
            break;
          }
          case CF_MAX32: {
            const int kind = B.src.kind[col];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) fx_max_if(cell_a + 4u * slots[j], order32(kind, vals[j]), use(j));
            break;
          }
          default: {
            u64* where[RPA_BATCH];
#pragma unroll
            for (int j = 0; j < RPA_BATCH; ++j) where[j] = (u64*)(rp_smem + B.cell_at[c]) + slots[j];
            cell_update_shared<RPA_BATCH>(where, op, vals, FULL ? 0xFu : ok);
          }
        }
      }
    };
    for (int at = 0; at < records; at += RPA_BATCH * RPA_BLOCK) {
      if (!nullable && at + RPA_BATCH * RPA_BLOCK <= records) batch(std::true_type{}, at);
      else batch(std::false_type{}, at);
    }
    __syncthreads();
    // the used slots: every warp counts those of its slots, then writes them run by run
    const u32* counts = FIXED ? fcnt : (const u32*)(rp_smem + (B.present >= 0 ? B.cell_at[B.present] : 0));
    auto used = [&](int i) {
      return i < S && (((FIXED || B.present >= 0) && counts[i] != 0u) || (sees && ((seen[i >> 5] >> (i & 31)) & 1u)));
    };
    u32 mine = 0;
    for (int i0 = (int)wid * 32; i0 < S; i0 += RPA_BLOCK) mine += __popc(__ballot_sync(0xFFFFFFFFu, used(i0 + (int)lane)));
    u32 at = 0;
    if (lane == 0 && mine) at = atomicAdd(&s_total, mine);
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    __syncthreads();
    if (threadIdx.x == 0) {
      s_outbase = atomicAdd(&ctrl->out_cursor, (u64)s_total);
      if (s_outbase + s_total > (u64)B.out_cap) ctrl->overflow = 1;
    }
    __syncthreads();
    if (s_outbase + s_total > (u64)B.out_cap) continue;
    for (int i0 = (int)wid * 32; i0 < S; i0 += RPA_BLOCK) {
      const int i = i0 + (int)lane;
      const bool mine_used = used(i);
      const u32 who = __ballot_sync(0xFFFFFFFFu, mine_used);
      const i64 g = (i64)s_outbase + at + __popc(who & ((1u << lane) - 1u));
      at += __popc(who);
      if (!mine_used) continue;
      const u64 key = word_key(P, B.word, (((u32)i >> B.low_bits) << WORD_LOW) | ((u32)b << B.low_bits) | ((u32)i & low_mask));
      if (FIXED) {  // (emptied once, whatever number of results asks for the sums)
        if (c_sum >= 0) fex[i] += fx_take(flx, S, i, fx_bx);
        if (c_ssq >= 0) feq[i] += fx_take(flq, S, i, fx_bq);
      }
      auto cell = [&](int c) -> u64 {
        if (FIXED) return c == c_cnt ? (u64)fcnt[i] : (u64)__double_as_longlong(c == c_sum ? fex[i] : feq[i]);
        const unsigned char* at = rp_smem + B.cell_at[c];
        switch (B.form[c]) {
          case CF_64: return ((const u64*)at)[i];
          case CF_COUNT: return ((const u32*)at)[i];
          case CF_SUM: return ((u64)((const u32*)at)[S + i] << 32) | ((const u32*)at)[i];
          default: break;
        }
        // (a group without a valid value keeps the identity, whatever image that word is of)
        const int n = B.count_of[c];
        const bool any = n < 0 || ((const u32*)(rp_smem + B.cell_at[n]))[i] != 0u;
        return any ? unorder32(B.src.kind[P.cells[c].col], ((const u32*)at)[i]) : cell_identity(P.cells[c].op);
      };
      if (LIST) {
        B.out[g] = key;
        for (int c = 0; c < P.ncells; ++c) B.out[(i64)(1 + c) * B.out_cap + g] = cell(c);
      } else {
        write_group(P, O, key, cell, g, O.null_counts);
      }
    }
  }
}

// group list -> output columns
__global__ void __launch_bounds__(256) k_finalize_records(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O,
                                                          const u64* __restrict__ groups, i64 cap, i64 ngroups)
{
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x)
    write_group(P, O, groups[g], [&](int c) { return groups[(i64)(1 + c) * cap + g]; }, g, O.null_counts);
}

}  // namespace b2
