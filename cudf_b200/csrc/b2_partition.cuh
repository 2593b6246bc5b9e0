// b2_partition.cuh — the high-cardinality path: radix partition of the rows by key hash into
// buckets whose groups fit a shared-memory table, then one shared-memory aggregate per bucket.
//
// Replaces the global-memory branch of the reference (compute_global_memory_aggs.cuh:74-187: one
// probe of a global cuco set + one global atomic per row and aggregation) for inputs with millions of
// groups.  There every row costs a random read-modify-write of a 32-byte sector per accumulator; here
// the rows are moved twice at most, sequentially, and every atomic is a shared-memory atomic:
//
//   k_rp_count      one pass over the key columns: rows per level-1 digit (the top 10 bits of the key
//                   hash) and, when the number of groups is not known, the HyperLogLog registers
//   k_rp_scatter    rows -> records {key, value words, 16 validity bits}, written to the region of their
//                   level-1 digit (structure-of-arrays record buffer; CTA-local counting per tile,
//                   one global cursor reservation per digit and tile)
//   k_rp_count2 /   second level inside every level-1 partition (only when one level leaves more
//   k_rp_scatter2   groups per bucket than a shared-memory table holds)
//   k_rp_aggregate  one CTA per bucket at a time: open-addressing table in shared memory, the
//                   bucket's records folded with shared-memory atomics, the finished groups appended
//                   to a compact record list (structure-of-arrays)
//   k_finalize_records  record list -> output columns (the finishers of k_finalize)
//
// Packed keys only (all key columns fixed-width non-float, at most 64 bits together).
#pragma once
#include "b2_kernels.cuh"

namespace b2 {

constexpr int RP_BLOCK    = 1024;                // threads per CTA of the counting kernels
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
constexpr u32 HOT_TOP_COUNT  = 4;         // occurrences of the most frequent key among 1024 rows that speak for a hot set
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
__global__ void __launch_bounds__(1024) k_hot_place(DHot hot)
{
  __shared__ u32 s_fill[HOT_BUCKETS];
  const int n = (int)min(hot.info[0], (u32)HOT_MAX);
  for (int i = threadIdx.x; i < HOT_BUCKETS; i += blockDim.x) s_fill[i] = 0;
  for (int top = 31; top >= 0; --top) {
    __syncthreads();
    for (int id = threadIdx.x; id < n; id += blockDim.x) {
      if (31 - __clz((int)hot.counts[id]) != top) continue;
      const u64 h = rp_hash(hot.keys[id]);
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

template <bool WITH_HLL, bool HOT>
__global__ void __launch_bounds__(RP_BLOCK, 1) k_rp_count(const __grid_constant__ DPlan P, u64* __restrict__ hist,
                                                       u32* __restrict__ hll, const DHot hot)
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
      for (int i = threadIdx.x; i < HOT_MAX; i += blockDim.x) hup[i] = i < nh ? (u32)(rp_hash(hot.keys[i]) >> 32) : 0u;
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
  // (whole warps stay in the loop — a lane beyond the last quad has no rows — because the hot-row mask of
  // 8 consecutive quads is put together with shuffles)
  for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q - (threadIdx.x & 31) < nquads; q += (i64)gridDim.x * blockDim.x) {
    u64 kk[4], xx[4] = {0, 0, 0, 0};
    u32 act, vn = 0;
    const int nv = (int)max((i64)0, min((i64)4, P.nrows - q * 4));
    if (HOT && nh > 0 && nv > 0) {
      load_floats4(P.vals[0], q * 4, nv, vec, xx);
      vn = P.vals[0].mask ? valid_nibble(P.vals[0].mask, P.vals[0].offset + q * 4, nv) : 0xFu;
    }
    rp_keys4(P, q * 4, nv, kk, act);
    u32 hotm = 0, raise = 0;  // rows of hot keys; rows that raise an estimator register
    u32 id[4], ranks[4], regs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const u64 h = rp_hash(kk[j]);
      id[j] = HOT_MAX;
      if (HOT && nh > 0) {
        id[j] = hot_find(htab, hup, h);
        if (id[j] != (u32)HOT_MAX) hotm |= 1u << j;
      }
      const u32 cold = act & ~hotm & (1u << j);
      fx_red_if(hist_a + 4u * (u32)(h >> (64 - RP_BITS_TOP)), 1u, cold);
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

// the hot keys' finished cells join the group list (one thread per id)
__global__ void k_rp_append_hot(const __grid_constant__ DPlan P, const DHot hot, u64* __restrict__ out, i64 out_cap, DCtrl* ctrl)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int)min(hot.info[0], (u32)HOT_MAX)) return;
  const u64 key = hot.keys[i];
  const u64* acc = hot.acc + (size_t)i * HOT_ACC_WORDS;
  if (acc[0] == 0 && acc[3] == 0) return;  // not placed in its bucket: a cold key
  const u64 g = atomicAdd(&ctrl->out_cursor, 1ull);
  if (g >= (u64)out_cap) { ctrl->overflow = 1; return; }
  out[g] = key;
  for (int c = 0; c < P.ncells; ++c) {
    const int op = P.cells[c].op;
    out[(i64)(1 + c) * out_cap + g] = op == OP_CNT_V ? acc[0] : op == OP_SUM_F ? acc[1] : acc[2];
  }
}

// ------------------------------------------------------------------------------ records
// A record buffer holds `cap` records, structure-of-arrays: word w of record i at rec[w * cap + i].
// Word 0 is the packed key, words 1..nvals the value columns in their 64-bit carried form
// (load_value).  If any value column is nullable, the validity bits of the values lie in an array of 16-bit words
// (a 64-bit word for them was a third of a record of one value, and both levels move it twice).
struct DRecords {
  u64* rec;
  i64 cap;
  int words;              // 1 + value columns
  unsigned short* valid;  // [cap], nullptr = every value is valid
};
static_assert(MAX_VALS <= 16, "validity bits of a record");

struct DScatter {
  DRecords dst;
  u64* cursors;  // [partitions] next free record of every destination (start offsets, advanced)
  int shift;     // digit = (hash >> shift) & (fan - 1)
  int fan;       // destinations per source partition (a power of two, <= 1 << RP_MAX_BITS)
};

// Both scatter levels sort a tile by digit in shared memory before writing it: every thread learns
// its records' ranks inside their digits (shared-memory atomics), the digits' runs are reserved with one
// global atomic each, the records are placed run by run in a staging array, and the staging array is
// copied out in order — consecutive threads write consecutive records of a run.  (Written straight from
// registers, every 8-byte word was an L2 write request of its own — 106 M requests for 60 M rows — and
// the level-1 pass crawled at 0.6 TB/s with DRAM 14 % busy.)
struct RpTile {
  u32* hist;   // [fan] records per digit, then cleared
  u32* off;    // [fan + 1] first staging position of every digit
  u64* base;   // [fan] first global record of every digit's run
  u64* keys;   // [RP_TILE] staged keys
  u64* vals;   // [RP_TILE] staged values (records of two words)
  unsigned short* dig;  // [RP_TILE] digit of every staged record
  unsigned short* src;  // [RP_TILE] position of the record inside the source tile (records of other shapes)
};
__host__ __device__ constexpr size_t rp_tile_smem(int fan) { return (size_t)fan * 4 + (size_t)(fan + 1) * 4 + (size_t)fan * 8 + (size_t)RP_TILE * (8 + 8 + 2 + 2) + 64; }

__device__ __forceinline__ RpTile rp_tile_carve(unsigned char* smem, int fan)
{
  RpTile t;
  t.keys = (u64*)smem;
  t.vals = t.keys + RP_TILE;
  t.base = t.vals + RP_TILE;
  t.hist = (u32*)(t.base + fan);
  t.off  = t.hist + fan;
  t.dig  = (unsigned short*)(t.off + fan + 1);
  t.src  = t.dig + RP_TILE;
  return t;
}

// after phase A (hist filled): staging offsets by an exclusive scan over the digits, one global
// reservation per digit with records, counters cleared.  `fan` <= blockDim.x.  Ends with a barrier.
__device__ __forceinline__ void rp_tile_plan(const RpTile& t, u64* cursors, int fan)
{
  __shared__ u32 s_warp[RPS_BLOCK / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u32 c = (int)threadIdx.x < fan ? t.hist[threadIdx.x] : 0u;
  u32 v = c;
  for (int d = 1; d < 32; d <<= 1) { const u32 x = __shfl_up_sync(0xFFFFFFFFu, v, d); if (lane >= d) v += x; }
  if (lane == 31) s_warp[wid] = v;
  __syncthreads();
  if (wid == 0) {
    u32 w = lane < RPS_BLOCK / 32 ? s_warp[lane] : 0u;
    for (int d = 1; d < 32; d <<= 1) { const u32 x = __shfl_up_sync(0xFFFFFFFFu, w, d); if (lane >= d) w += x; }
    if (lane < RPS_BLOCK / 32) s_warp[lane] = w;
  }
  __syncthreads();
  if ((int)threadIdx.x < fan) {
    const u32 excl = (wid ? s_warp[wid - 1] : 0u) + v - c;
    t.off[threadIdx.x] = excl;
    t.hist[threadIdx.x] = 0;
    if (c) t.base[threadIdx.x] = atomicAdd(&cursors[threadIdx.x], (u64)c);
    if ((int)threadIdx.x == fan - 1) t.off[fan] = excl + c;
  }
  __syncthreads();
}

// level 1: input rows -> records in the region of their digit
// (`hot_rows`: one bit per row, set for the rows whose keys k_rp_count folded already — they are left out here)
__global__ void __launch_bounds__(RPS_BLOCK, 2) k_rp_scatter(const __grid_constant__ DPlan P, const DScatter D,
                                                          const u32* __restrict__ hot_rows)
{
  extern __shared__ __align__(16) unsigned char rp_stage[];
  const RpTile t = rp_tile_carve(rp_stage, D.fan);
  // one value column is the common case: its values are loaded together with the keys and staged with them
  // (a null value as a flag beside the staged digit); other shapes stage the key and the row, and gather the
  // value words at copy-out
  const bool one = P.nvals == 1;
  const bool nullable = one && D.dst.valid;
  for (int i = threadIdx.x; i < D.fan; i += blockDim.x) t.hist[i] = 0;
  __syncthreads();
  const i64 ntiles = (P.nrows + RP_TILE - 1) / RP_TILE;
  const u32 dmask = (u32)D.fan - 1u;
  for (i64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const i64 tile0 = tile * RP_TILE;
    u64 kk[RP_ROWS], vv[RP_ROWS];
    u32 rank[RP_ROWS];
    u32 act = 0, vok = 0xFFFFFFFFu;
    // phase A: keys (and values), digits, ranks inside the tile
#pragma unroll
    for (int g = 0; g < RP_ROWS / 4; ++g) {
      const i64 row0 = tile0 + (i64)g * (RP_TILE / (RP_ROWS / 4)) + (i64)threadIdx.x * 4;
      const int nv = (int)max((i64)0, min((i64)4, P.nrows - row0));
      u64 k4[4];
      u32 a4;
      rp_keys4(P, row0, nv, k4, a4);
      if (hot_rows && nv > 0) a4 &= ~(__ldg(hot_rows + (row0 >> 5)) >> (row0 & 31));  // (row0 is a multiple of 4)
      act |= a4 << (4 * g);
      if (nullable && nv > 0) vok = (vok & ~(0xFu << (4 * g))) | (valid_nibble(P.vals[0].mask, P.vals[0].offset + row0, nv) << (4 * g));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        kk[4 * g + j] = k4[j];
        vv[4 * g + j] = (one && j < nv) ? load_value(P.vals[0], row0 + j) : 0ull;
      }
    }
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      rank[j] = 0;
      if ((act >> j) & 1u) {
        const u32 d = (u32)(rp_hash(kk[j]) >> D.shift) & dmask;
        rank[j] = (d << 16) | atomicAdd(&t.hist[d], 1u);  // a tile holds 4096 rows: the rank fits 16 bits
      }
    }
    __syncthreads();
    rp_tile_plan(t, D.cursors, D.fan);
    // phase C: place the records run by run
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      if (!((act >> j) & 1u)) continue;
      const u32 d = rank[j] >> 16;
      const u32 pos = t.off[d] + (rank[j] & 0xFFFFu);
      t.keys[pos] = kk[j];
      t.dig[pos]  = (unsigned short)(d | (((vok >> j) & 1u) ? 0u : 0x8000u));  // (digits stay below 2^RP_MAX_BITS)
      if (one) t.vals[pos] = vv[j];
      else t.src[pos] = (unsigned short)((j >> 2) * (RP_TILE / (RP_ROWS / 4)) + (int)threadIdx.x * 4 + (j & 3));
    }
    __syncthreads();
    // phase D: copy out in staging order
    const u32 ntile = t.off[D.fan];
    for (u32 pos = threadIdx.x; pos < ntile; pos += blockDim.x) {
      const u32 dg = t.dig[pos], d = dg & 0x7FFFu;
      const i64 at = (i64)t.base[d] + (i64)(pos - t.off[d]);
      D.dst.rec[at] = t.keys[pos];
      if (one) {
        D.dst.rec[D.dst.cap + at] = t.vals[pos];
        if (nullable) D.dst.valid[at] = (unsigned short)((dg >> 15) ^ 1u);
      } else {
        const i64 row = tile0 + t.src[pos];
        u32 vbits = 0;
        for (int v = 0; v < P.nvals; ++v) {
          const DValCol& vc = P.vals[v];
          const bool ok = value_valid(vc, row);
          vbits |= (u32)ok << v;
          D.dst.rec[(i64)(1 + v) * D.dst.cap + at] = ok ? load_value(vc, row) : 0ull;
        }
        if (D.dst.valid) D.dst.valid[at] = (unsigned short)vbits;
      }
    }
    __syncthreads();  // the staging arrays are rewritten by the next tile
  }
}

// Level 2 works on the tiles of the level-1 partitions: tile t belongs to the partition p with
// tile_start[p] <= t < tile_start[p + 1] and covers records [start[p] + j * RP_TILE, ...) of it.
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
__global__ void __launch_bounds__(RP_BLOCK, 1) k_rp_count2(const DLevel2 L, int shift, int fan, u64* __restrict__ hist2)
{
  __shared__ u32 s_hist[1 << RP_MAX_BITS];
  for (int i = threadIdx.x; i < fan; i += blockDim.x) s_hist[i] = 0;
  __syncthreads();
  const u32 ntiles = __ldg(L.tile_start + L.parts);
  const u32 dmask = (u32)fan - 1u;
  for (u32 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int p = rp_partition_of_tile(L.tile_start, L.parts, tile);
    const i64 lo = (i64)L.src_start[p] + (i64)(tile - __ldg(L.tile_start + p)) * RP_TILE;
    const i64 hi = min((i64)L.src_end[p], lo + RP_TILE);
    for (i64 i = lo + threadIdx.x; i < hi; i += blockDim.x)
      atomicAdd(&s_hist[(u32)(rp_hash(__ldg(L.src.rec + i)) >> shift) & dmask], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < fan; d += blockDim.x) {
      const u32 c = s_hist[d];
      s_hist[d] = 0;
      if (c) atomicAdd(&hist2[(i64)p * fan + d], (u64)c);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(RPS_BLOCK, 2) k_rp_scatter2(const DLevel2 L, const DScatter D)
{
  extern __shared__ __align__(16) unsigned char rp_stage[];
  const RpTile t = rp_tile_carve(rp_stage, D.fan);
  for (int i = threadIdx.x; i < D.fan; i += blockDim.x) t.hist[i] = 0;
  __syncthreads();
  const u32 ntiles = __ldg(L.tile_start + L.parts);
  const u32 dmask = (u32)D.fan - 1u;
  // key + one value (+ its validity): the value is loaded and staged with the key, the validity as a
  // flag beside the staged digit; records of other shapes are copied word by word from their source position
  const bool staged = L.src.words == 2, nullable = staged && L.src.valid;
  for (u32 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int p = rp_partition_of_tile(L.tile_start, L.parts, tile);
    const i64 lo = (i64)L.src_start[p] + (i64)(tile - __ldg(L.tile_start + p)) * RP_TILE;
    const i64 hi = min((i64)L.src_end[p], lo + RP_TILE);
    u64 kk[RP_ROWS], vv[RP_ROWS];
    u32 rank[RP_ROWS];
    u32 vok = 0xFFFFFFFFu;
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      const i64 i = lo + (i64)j * RPS_BLOCK + threadIdx.x;
      kk[j] = 0; vv[j] = 0;
      if (i < hi) {
        kk[j] = __ldg(L.src.rec + i);
        if (staged) vv[j] = __ldg(L.src.rec + L.src.cap + i);
        if (nullable && !(__ldg(L.src.valid + i) & 1u)) vok &= ~(1u << j);
      }
    }
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      const i64 i = lo + (i64)j * RPS_BLOCK + threadIdx.x;
      rank[j] = 0xFFFFFFFFu;
      if (i < hi) {
        const u32 d = (u32)(rp_hash(kk[j]) >> D.shift) & dmask;
        rank[j] = (d << 16) | atomicAdd(&t.hist[d], 1u);
      }
    }
    __syncthreads();
    rp_tile_plan(t, D.cursors + (i64)p * D.fan, D.fan);
#pragma unroll
    for (int j = 0; j < RP_ROWS; ++j) {
      if (rank[j] == 0xFFFFFFFFu) continue;
      const u32 d = rank[j] >> 16;
      const u32 pos = t.off[d] + (rank[j] & 0xFFFFu);
      t.keys[pos] = kk[j];
      t.dig[pos]  = (unsigned short)(d | (((vok >> j) & 1u) ? 0u : 0x8000u));
      if (staged) t.vals[pos] = vv[j];
      else t.src[pos] = (unsigned short)(j * RPS_BLOCK + (int)threadIdx.x);
    }
    __syncthreads();
    const u32 ntile = t.off[D.fan];
    for (u32 pos = threadIdx.x; pos < ntile; pos += blockDim.x) {
      const u32 dg = t.dig[pos], d = dg & 0x7FFFu;
      const i64 at = (i64)t.base[d] + (i64)(pos - t.off[d]);
      D.dst.rec[at] = t.keys[pos];
      if (staged) {
        D.dst.rec[D.dst.cap + at] = t.vals[pos];
        if (nullable) D.dst.valid[at] = (unsigned short)((dg >> 15) ^ 1u);
      } else {
        const i64 i = lo + t.src[pos];
        for (int w = 1; w < L.src.words; ++w) D.dst.rec[(i64)w * D.dst.cap + at] = __ldg(L.src.rec + (i64)w * L.src.cap + i);
        if (L.src.valid) D.dst.valid[at] = __ldg(L.src.valid + i);
      }
    }
    __syncthreads();
  }
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
  const u64* start;  // [buckets] first record of every bucket
  const u64* end;    // [buckets] one past its last record
  i64 nbuckets;
  int slots;         // shared-memory table slots (a power of two); slot `slots` holds the key whose bits equal EMPTY
  u64* out;          // finished groups, structure-of-arrays: word w of group g at out[w * out_cap + g]; word 0 = key
  i64 out_cap;
  u64* next_bucket;  // work counter
};

// FIXED (the cells are Σx / n / Σx² of one float column): a slot keeps its sums as fixed point (fx_add) plus one
// fp64 cell each for what does not fit the window (and for the periodic flushes), and its count as 32 bits: five to nine
// native 32-bit atomics per record (the count, two or three words of each sum and rarely its top word) instead of three
// 64-bit ones, which shared memory only does as compare-and-swap loops.  `hot_info`: DHot::info, the magnitudes among the
// sampled values.
constexpr int RPA_FIXED_SLOT_BYTES = 8 + 8 + 8 + 4 + 8 * FX_WORDS;
constexpr int RPA_INDEX_BYTES = 2;  // per slot: the claim-order index

template <bool FIXED>
__global__ void __launch_bounds__(RPA_BLOCK, 2) k_rp_aggregate(const __grid_constant__ DPlan P, const DBuckets B, DCtrl* ctrl,
                                                            const u32* __restrict__ hot_info)
{
  extern __shared__ __align__(16) unsigned char rp_smem[];
  __shared__ i64 s_bucket;
  __shared__ u32 s_count, s_fail, s_special;
  __shared__ u64 s_outbase;
  const int S  = B.slots;
  const int NS = S + 1;
  u64* skeys  = (u64*)rp_smem;   // [NS]
  u64* scells = skeys + NS;      // [ncells][NS]
  // FIXED: [NS] fp64 Σx beside the fixed point, [NS] the same for Σx², [NS] counts, words of Σx, words of Σx²
  double* fex = (double*)scells;
  double* feq = fex + NS;
  u32* fcnt   = (u32*)(feq + NS);
  u32* flx    = fcnt + NS;
  u32* flq    = flx + FX_WORDS * NS;
  const u32 fcnt_a = (u32)__cvta_generic_to_shared(fcnt), flx_a = (u32)__cvta_generic_to_shared(flx), flq_a = (u32)__cvta_generic_to_shared(flq);
  // slots in the order they were claimed: the finished groups are written in that order, consecutive
  // threads to consecutive list entries, without scanning the table for occupied slots
  unsigned short* sidx = FIXED ? (unsigned short*)(flq + FX_WORDS * NS) : (unsigned short*)(scells + (size_t)P.ncells * NS);
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
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u32 smask = (u32)S - 1u;
  // a bucket whose groups fill the table beyond this gives up (the caller falls back to the global table)
  const u32 fill_limit = (u32)S - (u32)(S >> 3);

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) { s_bucket = (i64)atomicAdd(B.next_bucket, 1ull); s_count = 0; s_fail = 0; s_special = 0; }
    __syncthreads();
    const i64 b = s_bucket;
    if (b >= B.nbuckets) break;
    const i64 lo = (i64)B.start[b], hi = (i64)B.end[b];
    if (hi <= lo) continue;
    // clear the table
    for (int i = threadIdx.x; i < NS; i += blockDim.x) skeys[i] = EMPTY;
    if (FIXED) {
      for (int i = threadIdx.x; i < 2 * NS; i += blockDim.x) scells[i] = 0;                       // fex, feq
      for (int i = threadIdx.x; i < (1 + 2 * FX_WORDS) * NS; i += blockDim.x) fcnt[i] = 0;        // fcnt, flx, flq
    } else {
      for (int c = 0; c < P.ncells; ++c) {
        const u64 id = cell_identity(P.cells[c].op);
        for (int i = threadIdx.x; i < NS; i += blockDim.x) scells[(size_t)c * NS + i] = id;
      }
    }
    __syncthreads();
    // fold the records, RPA_BATCH per thread at a time: all loads of a batch are issued before the first
    // probe, so that a batch costs one DRAM round trip instead of one per record and word
    for (i64 base = lo; base < hi; base += (i64)RPA_BATCH * blockDim.x) {
      u64 keys[RPA_BATCH], vals[RPA_BATCH];
      u32 vbits[RPA_BATCH];
      const bool one_col = B.src.words == 2;  // a single value column: prefetch it too
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) {
        const i64 i = base + (i64)j * blockDim.x + threadIdx.x;
        keys[j] = 0; vbits[j] = ~0u; vals[j] = 0;
        if (i < hi) {
          keys[j] = __ldg(B.src.rec + i);
          if (B.src.valid) vbits[j] = __ldg(B.src.valid + i);
          if (one_col) vals[j] = __ldg(B.src.rec + B.src.cap + i);
        }
      }
      // slots of the batch's records
      int slots[RPA_BATCH];
#pragma unroll
      for (int j = 0; j < RPA_BATCH; ++j) {
        const i64 i = base + (i64)j * blockDim.x + threadIdx.x;
        const u64 key = keys[j];
        int slot = -1;
        if (i < hi) {
          if (key == EMPTY) {
            slot = S;
            s_special = 1;
          } else {
            u32 idx = (u32)rp_hash(key) & smask;
            for (int p = 0; p < S; ++p) {
              u64 k = *(volatile u64*)(skeys + idx);
              if (k == EMPTY) {
                if (*(volatile u32*)&s_count >= fill_limit) break;
                k = atomicCAS(skeys + idx, EMPTY, key);
                if (k == EMPTY) { sidx[atomicAdd(&s_count, 1u)] = (unsigned short)idx; k = key; }
              }
              if (k == key) { slot = (int)idx; break; }
              idx = (idx + 1u) & smask;
            }
          }
          if (slot < 0) s_fail = 1;
        }
        slots[j] = slot;
      }
      // The lanes left the probe loops at different iterations: bring them back together, then go
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
      int cur = one_col ? 0 : -1;
      for (int c = 0; !FIXED && c < P.ncells; ++c) {
        const int op = P.cells[c].op, col = P.cells[c].col;
        if (op != OP_CNT_A && col != cur) {  // (the cells of a value column are adjacent)
          cur = col;
#pragma unroll
          for (int j = 0; j < RPA_BATCH; ++j) {
            const i64 i = base + (i64)j * blockDim.x + threadIdx.x;
            vals[j] = i < hi ? __ldg(B.src.rec + (i64)(1 + col) * B.src.cap + i) : 0ull;
          }
        }
        u64* cell = scells + (size_t)c * NS;
        u32 ok = 0;  // records of the batch that update this cell
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j)
          if (slots[j] >= 0 && (op == OP_CNT_A || ((vbits[j] >> col) & 1u))) ok |= 1u << j;
        u64* where[RPA_BATCH];
#pragma unroll
        for (int j = 0; j < RPA_BATCH; ++j) where[j] = cell + (slots[j] >= 0 ? slots[j] : 0);
        cell_update_shared<RPA_BATCH>(where, op, vals, ok);
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
        for (int c = 0; c < P.ncells; ++c) B.out[(i64)(1 + c) * B.out_cap + g] = scells[(size_t)c * NS + i];
      }
    }
  }
}

// group list -> output columns
__global__ void __launch_bounds__(256) k_finalize_records(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O,
                                                          const u64* __restrict__ groups, i64 cap, i64 ngroups)
{
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x)
    write_group(P, O, groups[g], groups + cap + g, cap, g, O.null_counts);
}

}  // namespace b2
