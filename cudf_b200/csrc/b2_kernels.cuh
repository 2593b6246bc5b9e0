// b2_kernels.cuh — the CUDA kernels of the groupby engine (sm_100a).
//
//   k_table_init     identity-fills a table with linear 16-byte stores (replaces the per-column
//                    thrust::fill of cpp/src/aggregation/aggregation.cu:87-97 and the cuco slot memset)
//   k_aggregate      ONE fused pass over keys + values + bitmasks: a per-CTA shared-memory table
//                    (direct-indexed key box sampled in the kernel, or a 2-probe hashed cache) in
//                    front of the global-memory table
//                    (replaces mapping_indices_kernel + single_pass_shmem_aggs_kernel +
//                    the global-memory functors: cpp/src/groupby/hash/compute_mapping_indices.cuh:92-151,
//                    compute_shared_memory_aggs.cu:260-353, single_pass_functors.cuh:86-157)
//   k_hll            HyperLogLog pass over the key columns: sizes the table after the small
//                    speculative one overflowed (the reference sizes by rows: compute_groupby.cu:93-102)
//   k_finalize       compaction of occupied slots + key decode + compound finalisers + result
//                    null masks in one pass (replaces retrieve_all, key gather, binary DIV,
//                    m2/var/std tabulate and null-count kernels: output_utils.cu:139-224,
//                    hash_compound_agg_finalizer.cu:93-186, common/m2_var_std.cu:49-59,160-187)
//   k_gather_fixed, k_string_lengths, k_scan_*, k_string_copy
//                    key gather for row-keyed tables (fixed width and strings)
//   k_pack_* / k_merge / k_merge_chunks
//                    hash partition of partial records by owner and merge of partial records
//                    (cpp/src/partitioning/partitioning.cu:120-337, streaming_groupby/merge.cu:91-142)
//   k_partition_count / k_partition_scatter, k_mask_to_bytes / k_bytes_to_mask
//                    row-level hash partition of a table (cudf::hash_partition) and the validity
//                    conversions a row exchange needs
#pragma once
#include "b2_device.cuh"
#include <type_traits>

namespace b2 {

constexpr int AGG_BLOCK      = 1024;  // threads per CTA of the fused kernel (one CTA per SM)
constexpr int LEAN_ROWS      = 4;     // rows per thread per tile of k_aggregate_lean (1024 threads; 512 measured
                                      // 1.6x slower: too few warps to cover the shared-memory atomics' latency)
constexpr int AGG_ROWS       = 4;     // rows per thread per tile
// The shared-memory table is a cache: a key that finds neither itself nor a free slot within
// SMEM_PROBES slots of its home goes to the global table, and the CTA's merge adds both parts up.
// A short limit keeps warps converged: with 48 probes and a 75 % fill every lookup of an uncached key
// walked a long cluster while the other 31 lanes waited (125M Zipf rows: 21.7 ms; limit 2: 8.0 ms).
constexpr int SMEM_PROBES    = 2;
constexpr double SMEM_FILL   = 0.9;   // the table takes no new keys beyond this fill
constexpr int GMEM_PROBES    = 2048;  // probe limit of the global table before "overflow"
constexpr u32 F32_SPILL_AT   = 1024;  // packed {f32 sum, u32 n} cells spill to fp64 at this count
constexpr int SLOT_NONE      = -1;
constexpr u32 CACHE_TOP_COUNT = 8;    // of 1024 sampled keys: a key with so many holds about 1 % of the rows

enum SmemLayout : int { SL_NONE = 0, SL_GENERIC = 1, SL_F32MEAN = 2 };

// ------------------------------------------------------------------------------ float sums as fixed point
// 64-bit shared-memory atomics (fp64 adds among them) run as compare-and-swap loops: 21 clocks per warp over 8192 slots,
// 87 over 64, against 3.9 for a native 32-bit add whether lanes meet or not.  The partitioned path therefore keeps Σx and
// Σx² of a float column as FX_WORDS words of 32 bits per slot: one two's complement integer of 128 bits in units of
// 2^(B - 1075).  A value's 53-bit mantissa, shifted to its place, covers three consecutive words; each is added with one
// native atomic and the carry, which the returned old word tells, goes into the next (the sign of a negative value and a
// last carry meet in the word above and mostly cancel).  Nothing is rounded until a slot is emptied (fx_take).  Every
// FX_FLUSH-th addend of a slot empties it.  B comes from the magnitudes of sampled rows (fx_base): a value whose bits do
// not fit the window of FX_MAX_SHIFT binades (zero fits; denormals, infinities and NaN do not) is added to an fp64 cell
// instead, so the result does not depend on the sample — only the speed does.  (Six words of 18-bit pieces that needed no carries took four adds and twice the arithmetic per value.)
constexpr int FX_WORDS     = 4;
constexpr int FX_MAX_SHIFT = 57;
constexpr int FX_TYPICAL   = 37;    // place of the sampled values' mean exponent: a mantissa that starts at bits 32 .. 43 ends
                                    // inside its second word, so five binades on either side need two atomics, not three
constexpr int FX_HEADROOM  = 4;     // the window reaches at least 2^4 above the sampled maximum
// Addends of a slot between flushes.  A contribution stays below 2^(53 + FX_MAX_SHIFT), so 2^17 of them fit.  The thread
// that takes a multiple of FX_FLUSH empties the slot before it adds anything else: beyond FX_FLUSH a slot can only
// collect what the other warps add while that many warps (at most 32 of a CTA) are stalled in front of their flush.
constexpr u32 FX_FLUSH     = 1024;
constexpr int FX_NEVER     = 1 << 20;  // window base with which no value fits (nothing was sampled)

// p[0..2] becomes -p (96 bits) where `ext` is all ones, stays where it is zero
__device__ __forceinline__ void fx_sign(u32 (&p)[3], u32 ext)
{
#pragma unroll
  for (int i = 0; i < 3; ++i) p[i] ^= ext;
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %3, %3;\n addc.cc.u32 %0, %0, 0;\n addc.cc.u32 %1, %1, 0;\n addc.u32 %2, %2, 0;\n}"
      : "+r"(p[0]), "+r"(p[1]), "+r"(p[2]) : "r"(ext));
}
__device__ __forceinline__ u32 fx_atom(u32 saddr, u32 v)
{
  u32 old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(saddr), "r"(v) : "memory");
  return old;
}
// ... where `cond` is not zero, as one predicated instruction (else 0)
__device__ __forceinline__ u32 fx_atom_if(u32 saddr, u32 v, u32 cond)
{
  u32 old;
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.u32 %0, 0;\n @p atom.shared.add.u32 %0, [%1], %2;\n}"
               : "=r"(old) : "r"(saddr), "r"(v), "r"(cond) : "memory");
  return old;
}
__device__ __forceinline__ void fx_red_if(u32 saddr, u32 v, u32 cond)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p red.shared.add.u32 [%0], %1;\n}" ::"r"(saddr), "r"(v), "r"(cond) : "memory");
}
__device__ __forceinline__ u32 lds_u32(u32 saddr)
{
  u32 v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr) : "memory");
  return v;
}
__device__ __forceinline__ u64 lds_u64(u32 saddr)
{
  u64 v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(saddr) : "memory");
  return v;
}
__device__ __forceinline__ void fx_min_if(u32 saddr, u32 v, u32 cond)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p red.shared.min.u32 [%0], %1;\n}" ::"r"(saddr), "r"(v), "r"(cond) : "memory");
}
__device__ __forceinline__ void fx_max_if(u32 saddr, u32 v, u32 cond)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p red.shared.max.u32 [%0], %1;\n}" ::"r"(saddr), "r"(v), "r"(cond) : "memory");
}
// the carry of old + p[0] (p[1], p[2]) goes into the words above
__device__ __forceinline__ void fx_carry0(u32 old, u32 (&p)[3], u32& ext)
{
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %3, %4;\n addc.cc.u32 %0, %0, 0;\n addc.cc.u32 %1, %1, 0;\n addc.u32 %2, %2, 0;\n}"
      : "+r"(p[1]), "+r"(p[2]), "+r"(ext) : "r"(old), "r"(p[0]));
}
__device__ __forceinline__ void fx_carry1(u32 old, u32 (&p)[3], u32& ext)
{
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %2, %3;\n addc.cc.u32 %0, %0, 0;\n addc.u32 %1, %1, 0;\n}"
      : "+r"(p[2]), "+r"(ext) : "r"(old), "r"(p[1]));
}
__device__ __forceinline__ void fx_carry2(u32 old, const u32 (&p)[3], u32& ext)
{
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %1, %2;\n addc.u32 %0, %0, 0;\n}" : "+r"(ext) : "r"(old), "r"(p[2]));
}
// The window base for values of the biased exponents `mean` (typical) to `emax`.  Kept inside 1 .. 1980: then neither zero
// or a denormal (exponent 0) nor an infinity or NaN (2047) ever lies in a window.
__device__ __forceinline__ int fx_base(int mean, int emax)
{
  const int b = max(mean - FX_TYPICAL, emax + FX_HEADROOM - FX_MAX_SHIFT);
  return b < 1 || b > 1980 ? FX_NEVER : b;
}
// the same for their squares
__device__ __forceinline__ int fx_base_sq(int mean, int emax) { return fx_base(2 * mean - 1023, 2 * emax - 1022 + FX_HEADROOM); }
// Adds the doubles v[j] of the rows in `take` to the words at shared address a[j] (word step `st` bytes), four rows at a
// time, word by word, so that a warp waits for one round trip per word.  The atomics are predicated, not branched around
// (with a branch per row and word the counting pass of 100M rows issued 323 instructions per row and warp), and no dummy
// atomics are issued for the rows that do not take part (the shared-memory pipe is the next bound: those cost 10 %).
// Returns the rows whose value does not fit.
template <bool SIGNED>
__device__ __forceinline__ u32 fx_add4(const u64 (&v)[4], int B, const u32 (&a)[4], u32 take, u32 st)
{
  u32 p[4][3], ext[4], at[4], old[4], unfit = 0, last = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const u32 lo = (u32)v[j], hi = (u32)(v[j] >> 32), s = ((hi >> 20) & 0x7FFu) - (u32)B;
    const u32 m = (hi & 0xFFFFFu) | 0x100000u;
    if (s > (u32)FX_MAX_SHIFT) {
      if ((lo | (hi + hi)) != 0u) unfit |= 1u << j;
    } else {
      last |= 1u << j;
    }
    at[j] = a[j] + ((s & 32u) ? st : 0u);
    p[j][0] = __funnelshift_l(0u, lo, s);
    p[j][1] = __funnelshift_l(lo, m, s);
    p[j][2] = __funnelshift_l(m, 0u, s);
    ext[j] = 0;
    if (SIGNED) { ext[j] = (u32)((int)hi >> 31); fx_sign(p[j], ext[j]); }
  }
  unfit &= take;
  take &= last;
#pragma unroll
  for (int j = 0; j < 4; ++j) old[j] = fx_atom_if(at[j], p[j][0], take & (1u << j));
#pragma unroll
  for (int j = 0; j < 4; ++j) { fx_carry0(old[j], p[j], ext[j]); old[j] = fx_atom_if(at[j] + st, p[j][1], take & (1u << j)); }
#pragma unroll
  for (int j = 0; j < 4; ++j) { fx_carry1(old[j], p[j], ext[j]); old[j] = fx_atom_if(at[j] + 2 * st, p[j][2], (take & (1u << j)) ? p[j][2] : 0u); }
  // the word above: the sign and the last carry, which mostly cancel (a value that starts in the second word has none)
  last = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    fx_carry2(old[j], p[j], ext[j]);
    if (ext[j] != 0u && at[j] == a[j]) last |= 1u << j;
  }
  last &= take;
  if (last) {
#pragma unroll
    for (int j = 0; j < 4; ++j) if ((last >> j) & 1u) fx_atom(at[j] + 3 * st, ext[j]);
  }
  return unfit;
}
// empties the words of one slot and returns their value (word i at words[i * ns + slot])
__device__ __noinline__ double fx_take(u32* words, int ns, int slot, int B)
{
  u32 w[FX_WORDS];
#pragma unroll
  for (int i = 0; i < FX_WORDS; ++i) w[i] = atomicExch(words + (size_t)i * ns + slot, 0u);
  u64 lo = ((u64)w[1] << 32) | w[0], hi = ((u64)w[3] << 32) | w[2];
  const bool neg = (hi >> 63) != 0;
  if (neg) { lo = 0ull - lo; hi = ~hi + (lo == 0 ? 1ull : 0ull); }
  if ((lo | hi) == 0) return 0.0;
  const double a = fma((double)hi, 18446744073709551616.0, (double)lo);
  return ldexp(neg ? -a : a, B - 1075);
}

// The lean kernel's windows (b2_lean.cuh): binades from the lowest place of a mantissa to the highest, and how far above the
// sampled maximum they reach.
constexpr int PK_HEADROOM = 1, PK_WIDE_HEADROOM = 2;
__host__ __device__ constexpr int pk_span(bool v8, bool wide) { return v8 ? (wide ? 46 : 14) : (wide ? 43 : 11); }
// With more of 1024 sampled values below the narrow window the wide one is taken.  A listed row costs 0.2 ns (100M FLOAT32
// rows, 1.4 % of them listed: 270 us), the word more per row 0.75 ms per 10^9 rows (265 -> 340 us for 100M) and the second
// launch 60 us: 0.4 % of 100M rows, 4 % of 10M, and at most half of what the lists hold.
__host__ __device__ __forceinline__ u32 pk_spread_limit(i64 nrows)
{
  const i64 n = 400000000ll / (nrows + 1);
  return (u32)(n < 4 ? 4 : n > 64 ? 64 : n);
}

// ------------------------------------------------------------------------------ programmatic dependent launch
// A kernel launched with the attribute starts while its predecessor still runs; what it reads of the predecessor's
// results it reads behind the wait (which also covers everything earlier on the stream).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Called by all threads of all CTAs when they are done.
__device__ __forceinline__ void report_ctrl(DCtrl* ctrl, const DReport& R)
{
  if (!R.flag) return;
  __shared__ u32 s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // (what the CTA wrote before the barrier, to the control block among it, is seen by whoever sees the ticket)
    s_last = atomicAdd(&ctrl->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  for (u32 i = threadIdx.x; i < (u32)(sizeof(DCtrl) / 4); i += blockDim.x) ((volatile u32*)R.copy)[i] = __ldcg((const u32*)ctrl + i);
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->ticket = 0;
    __threadfence_system();
    *(volatile u64*)R.flag = R.number;
  }
}

// The same as a kernel of its own, for kernels that end with atomics of global memory under way: a fence waits for them in every
// CTA (batches of 3.4M rows over 64K groups: 113 us per launch of k_aggregate with report_ctrl at its end, 82 without; 1362 us
// for nine batches with, 1170 with this kernel behind it; 1254 with a copy command and a synchronisation).  Launched as a
// dependent of the kernel in front, which lets it start while that one still runs: what it reads, it reads behind the wait.
__global__ void __launch_bounds__(256) k_report(const DCtrl* ctrl, const DReport R)
{
  grid_dependency_wait();
  for (u32 i = threadIdx.x; i < (u32)(sizeof(DCtrl) / 4); i += blockDim.x) ((volatile u32*)R.copy)[i] = __ldcg((const u32*)ctrl + i);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    *(volatile u64*)R.flag = R.number;
  }
}

// The same for words of any kind: up to three arrays side by side.
struct DWords { const u32* src[3]; u32 words[3]; };
__global__ void __launch_bounds__(1024) k_report_words(const DWords W, u32* dst, u64* flag, u64 number)
{
  for (int a = 0; a < 3; ++a) {
    for (u32 i = threadIdx.x; i < W.words[a]; i += blockDim.x) ((volatile u32*)dst)[i] = __ldcg(W.src[a] + i);
    dst += W.words[a];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    *(volatile u64*)flag = number;
  }
}

// ------------------------------------------------------------------------------ table init
// Groups from which on a table is not filled because the rows are better partitioned (0: never), for keys in general and for keys
// that span at most two values per row.
struct DPartitionFrom { u32 sparse = 0, dense = 0; };
constexpr u32 PART_TOP_COUNT = 4;  // occurrences of the most frequent key among SAMPLE_ROWS that speak against partitions

__device__ __forceinline__ void sample_dense_box(const DPlan& P, u32 cap_slots, bool count_keys, u64 claim_limit, DDense* out, DPartitionFrom from = DPartitionFrom{});

// Must be launched with TABLE_INIT_BLOCK threads per CTA.  With `cap_dense` > 0 the last CTA also
// samples the key box of the fused kernels that follow on the stream (sample_dense_box) into the
// control block: one CTA's 1024 reads here instead of the same 1024 reads by every CTA of the fused
// kernel (148 CTAs queueing on the same sectors cost 6.5 us of that kernel). 
constexpr int TABLE_INIT_BLOCK = 256;
constexpr int SAMPLE_ROWS = 1024;
__global__ void __launch_bounds__(TABLE_INIT_BLOCK)
k_table_init(u64* __restrict__ tbl, i64 nslots, const __grid_constant__ DPlan P, DCtrl* ctrl, u64 claim_limit,
             u64 dense_slots = 0, u32 cap_dense = 0, int count_keys = 0, u32* __restrict__ odd = nullptr, int odd_words = 0, DPartitionFrom from = DPartitionFrom{})
{
  grid_dependents_launch();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < odd_words; i += gridDim.x * blockDim.x) odd[i] = 0;  // (LeanRare::odd)
  // (row keys have no box, but the repeated keys of the sample are counted all the same)
  const bool sampling = ctrl && (cap_dense > 0 || (P.key_mode == KM_ROWS && count_keys && P.nrows >= SAMPLE_ROWS));
  if (ctrl && blockIdx.x == 0 && threadIdx.x < sizeof(DCtrl) / 4) {
    // a fresh control block: all zero except the claim limit (and the key box, which the sampling CTA writes)
    u32 v = 0;
    if (threadIdx.x == offsetof(DCtrl, claim_limit) / 4) v = (u32)claim_limit;
    if (threadIdx.x == offsetof(DCtrl, claim_limit) / 4 + 1) v = (u32)(claim_limit >> 32);
    if (threadIdx.x == offsetof(DCtrl, dense_slots) / 4) v = (u32)dense_slots;
    const bool in_box = threadIdx.x >= offsetof(DCtrl, dense) / 4 && threadIdx.x < (offsetof(DCtrl, dense) + sizeof(DDense)) / 4;
    if (!(sampling && in_box)) ((u32*)ctrl)[threadIdx.x] = v;
  }
  if (sampling && blockIdx.x == gridDim.x - 1) sample_dense_box(P, cap_dense, count_keys != 0, count_keys == 1 ? claim_limit : ~0ull >> 1, &ctrl->dense, from);
  // the table is written as one linear run of 8-byte words, two per thread and step (16-byte stores):
  // word w belongs to cell (w mod stride) of slot (w div stride); cell 0 is the key
  __shared__ u64 s_init[MAX_CELLS + 1];
  const u32 stride = (u32)P.stride;
  if (threadIdx.x <= (u32)P.ncells) s_init[threadIdx.x] = threadIdx.x == 0 ? EMPTY : cell_identity(P.cells[threadIdx.x - 1].op);
  __syncthreads();
  const i64 nwords = nslots * (i64)stride;
  const i64 aos    = (nslots - (i64)dense_slots) * (i64)stride;  // words of the hashed region + special slot
  const i64 span   = (i64)blockDim.x * 2;
  for (i64 base = (i64)blockIdx.x * span; base < nwords; base += (i64)gridDim.x * span) {
    const u32 c0 = (u32)(base % stride);  // same for the whole CTA: one 64-bit division per step
    const i64 w  = base + 2 * (i64)threadIdx.x;
    const u32 c  = (c0 + 2u * threadIdx.x) % stride;
    const u32 c1 = c + 1u == stride ? 0u : c + 1u;
    if (w >= nwords) continue;
    // the dense region is structure-of-arrays: word r of it belongs to cell r / dense_slots
    // (the index is clamped so that a load the compiler hoists above the select stays in bounds)
    const u64 dz = dense_slots ? dense_slots : 1;
    u64 q0 = (u64)(w - aos) / dz, q1 = (u64)(w + 1 - aos) / dz;
    q0 = q0 < stride ? q0 : 0;
    q1 = q1 < stride ? q1 : 0;
    const u64 v0 = w < aos ? s_init[c] : s_init[q0];
    if (w + 1 < nwords) {
      const u64 v1 = w + 1 < aos ? s_init[c1] : s_init[q1];
      *(ulonglong2*)(tbl + w) = make_ulonglong2(v0, v1);
    } else {
      tbl[w] = v0;
    }
  }
}

// ------------------------------------------------------------------------------ probing
// Long probe chains: every 8th probe looks at the overflow flag and gives up when it is set (the table
// is over its claim limit and this attempt will be discarded); every 64th probe also publishes this
// CTA's unreported claims, so that a table that fills up within the first wave of tiles — before any
// CTA reaches its per-tile bookkeeping — is noticed.
__device__ __forceinline__ bool probe_gave_up(int p, DCtrl* ctrl, int* s_new)
{
  if ((p & 7) != 7) return false;
  if ((p & 63) == 63) {
    const int c = atomicExch(s_new, 0);
    if (c) {
      const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)c) + (u64)c;
      if (tot > ctrl->claim_limit) ctrl->overflow = 1;
    }
  }
  return *(volatile u32*)&ctrl->overflow != 0;
}

// Whether a CTA's hashed cache of `slots` slots pays for `rows` rows over about `groups` groups (no frequent keys): its
// slots have to meet their keys again, and most rows' keys have to have one.
__host__ __device__ __forceinline__ bool cache_pays(i64 rows, u32 groups, int slots)
{
  return rows / 2 >= (i64)groups && (i64)groups <= 2 * (i64)slots;
}

// the same from a sample: 0 groups = nothing is known
__host__ __device__ __forceinline__ bool cache_pays_for(i64 rows, u32 est_groups, u32 top_count, int slots)
{
  return est_groups == 0 || top_count >= CACHE_TOP_COUNT || cache_pays(rows, est_groups, slots);
}
// groups by the collisions among n sampled keys: n samples of G equally frequent keys are n - n^2 / 2G distinct ones
__device__ __forceinline__ u32 groups_of_sample(u32 taken, u32 distinct)
{
  const u32 twice = taken - distinct;
  return twice == 0 ? ~0u : (u32)((u64)taken * taken / (2 * twice));
}

// a CTA's bit of DCtrl::cache_ctas
__device__ __forceinline__ void note_cache(DCtrl* ctrl, bool pays)
{
  u32* const word = ctrl->cache_ctas + (blockIdx.x >> 5);
  const u32 bit = 1u << (blockIdx.x & 31);
  if (pays) atomicOr(word, bit); else atomicAnd(word, ~bit);
}

// cache_pays_for by up to 1024 rows of this CTA, spread over its tiles.  `scratch`: BATCH_SAMPLE_BYTES of shared memory.
// Called by all AGG_BLOCK threads.
// k_aggregate: rows for the table of a state; k_state_sample ran in front; the rows that a launch without a cache left over
constexpr int BATCH_ROWS = 1, BATCH_SAMPLED = 2, BATCH_REST = 4;
constexpr int BATCH_SAMPLE_BYTES = 2 * AGG_BLOCK * 12;
__device__ __forceinline__ bool cache_pays_here(const DPlan& P, u64* scratch, int slots)
{
  __shared__ u32 s_distinct, s_taken, s_top;
  u64* keys = scratch;
  u32* counts = (u32*)(scratch + 2 * AGG_BLOCK);
  const int tid = threadIdx.x;
  for (int i = tid; i < 2 * AGG_BLOCK; i += AGG_BLOCK) { keys[i] = EMPTY; counts[i] = 0; }
  if (tid == 0) { s_distinct = 0; s_taken = 0; s_top = 0; }
  __syncthreads();
  const i64 tile_rows = (i64)AGG_BLOCK * AGG_ROWS, tiles = (P.nrows + tile_rows - 1) / tile_rows;
  const i64 mine = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;  // tiles of this CTA (at least one)
  const i64 row = ((i64)blockIdx.x + (tid % mine) * gridDim.x) * tile_rows + (i64)tid * AGG_ROWS;
  if (row < P.nrows && row_active(P, row)) {
    const u64 key = pack_key(P, row);
    if (key != EMPTY) {
      u32 at = (u32)(mix64(key) >> 40) & (2 * AGG_BLOCK - 1);
      for (;;) {  // ends: half of the slots stay free
        const u64 old = atomicCAS(&keys[at], EMPTY, key);
        if (old == EMPTY) atomicAdd(&s_distinct, 1u);
        if (old == EMPTY || old == key) break;
        at = (at + 1) & (2 * AGG_BLOCK - 1);
      }
      atomicMax(&s_top, atomicAdd(&counts[at], 1u) + 1u);
      atomicAdd(&s_taken, 1u);
    }
  }
  __syncthreads();
  // (a CTA with next to no rows needs none)
  const bool pays = s_taken >= 64 && cache_pays_for(P.nrows / gridDim.x, groups_of_sample(s_taken, s_distinct), s_top, slots);
  __syncthreads();
  return pays;
}

// Global table, packed keys.  Returns the slot index, or -1 after setting ctrl->overflow.
__device__ __forceinline__ i64 gmem_find_insert_packed(u64* tbl, i64 cap, int stride, u64 key, u64 h,
                                                       DCtrl* ctrl, int* s_new)
{
  if (key == EMPTY) {
    if (ctrl->special_used == 0) ctrl->special_used = 1;
    return cap;
  }
  i64 idx = (i64)reduce64(h, (u64)cap);
  for (int p = 0; p < GMEM_PROBES; ++p) {
    u64* kp = tbl + idx * stride;
    u64 k   = *(volatile u64*)kp;
    if (k == key) return idx;
    if (k == EMPTY) {
      const u64 old = atomicCAS(kp, EMPTY, key);
      if (old == EMPTY) { atomicAdd(s_new, 1); return idx; }
      if (old == key) return idx;
    }
    if (probe_gave_up(p, ctrl, s_new)) return -1;
    if (++idx == cap) idx = 0;
  }
  ctrl->overflow = 1;
  return -1;
}

// Same, when the key cell of the home slot `idx` was already loaded (`k`): the loads of several rows
// are issued together so that their DRAM latencies overlap, then each row finishes here.
__device__ __forceinline__ i64 gmem_finish_packed(u64* tbl, i64 cap, int stride, u64 key, i64 idx, u64 k,
                                                  DCtrl* ctrl, int* s_new)
{
  for (int p = 0; p < GMEM_PROBES; ++p) {
    u64* kp = tbl + idx * stride;
    if (p > 0) k = *(volatile u64*)kp;
    if (k == key) return idx;
    if (k == EMPTY) {
      const u64 old = atomicCAS(kp, EMPTY, key);
      if (old == EMPTY) { atomicAdd(s_new, 1); return idx; }
      if (old == key) return idx;
    }
    if (probe_gave_up(p, ctrl, s_new)) return -1;
    if (++idx == cap) idx = 0;
  }
  ctrl->overflow = 1;
  return -1;
}

// Global table, row keys: key cell = (tag << 32) | representative row.
__device__ __forceinline__ i64 gmem_find_insert_rows(const DPlan& P, u64* tbl, i64 cap, int stride, i64 row,
                                                     u64 h, DCtrl* ctrl, int* s_new)
{
  const u64 tag  = h & 0xFFFFFFFF00000000ull;
  const u64 mine = tag | (u64)(u32)row;
  i64 idx        = (i64)reduce64(h, (u64)cap);
  for (int p = 0; p < GMEM_PROBES; ++p) {
    u64* kp = tbl + idx * stride;
    u64 k   = *(volatile u64*)kp;
    if (k == EMPTY) {
      k = atomicCAS(kp, EMPTY, mine);
      if (k == EMPTY) { atomicAdd(s_new, 1); return idx; }
    }
    if ((k & 0xFFFFFFFF00000000ull) == tag && rows_equal(P, row, (i64)(u32)k)) return idx;
    if (probe_gave_up(p, ctrl, s_new)) return -1;
    if (++idx == cap) idx = 0;
  }
  ctrl->overflow = 1;
  return -1;
}

// Shared-memory table (S slots + the special slot at index S).  Returns -1 when the key is not
// cached and may not be inserted (table closed) — the caller then goes to the global table.
template <int KM>
__device__ __forceinline__ int smem_find_insert(const DPlan& P, u64* skeys, int S, int fill_limit, int* s_fill,
                                                u64 key, u64 h, i64 row)
{
  if (KM == KM_PACKED && key == EMPTY) {
    if (skeys[S] == EMPTY) skeys[S] = 0;
    return S;
  }
  const u64 tag  = h & 0xFFFFFFFF00000000ull;
  const u64 mine = (KM == KM_PACKED) ? key : (tag | (u64)(u32)row);
  int idx        = (int)reduce32((u32)(h >> 11), (u32)S);
  for (int p = 0; p < SMEM_PROBES; ++p) {
    u64 k = *(volatile u64*)(skeys + idx);
    if (k == EMPTY) {
      if (*(volatile int*)s_fill >= fill_limit) return -1;
      k = atomicCAS(skeys + idx, EMPTY, mine);
      if (k == EMPTY) { atomicAdd(s_fill, 1); return idx; }
    }
    if (KM == KM_PACKED) {
      if (k == key) return idx;
    } else {
      if ((k & 0xFFFFFFFF00000000ull) == tag && rows_equal(P, row, (i64)(u32)k)) return idx;
    }
    if (++idx == S) idx = 0;
  }
  return -1;
}

// ------------------------------------------------------------------------------ dense key box
// ordered value of key column k inside a packed key
__device__ __forceinline__ i64 key_field(const DKeyCol& c, u64 key)
{
  u64 v = key >> c.shift;
  if (c.width < 8) {
    const int sh = 64 - 8 * c.width;
    v <<= sh;
    v = c.is_signed ? (u64)((i64)v >> sh) : (v >> sh);
  }
  return (i64)v;
}

// slot of a packed key inside the sampled box, -1 when the key lies outside it
__device__ __forceinline__ int dense_index(const DPlan& P, const DDense& D, u64 key)
{
  u32 idx = 0;
  for (int k = 0; k < P.nkeys; ++k) {
    const DKeyCol& c = P.keys[k];
    u64 f;
    if (c.nullbit >= 0 && ((key >> c.nullbit) & 1ull)) {
      f = D.range[k] - 1;
    } else {
      f = (u64)(key_field(c, key) - D.min[k]);
      if (f >= D.range[k] - (c.nullbit >= 0 ? 1ull : 0ull)) return -1;
    }
    idx += (u32)f * D.mult[k];
  }
  return (int)idx;
}

// inverse of dense_index
__device__ __forceinline__ u64 dense_key(const DPlan& P, const DDense& D, u32 idx)
{
  u64 key = 0;
  for (int k = 0; k < P.nkeys; ++k) {
    const DKeyCol& c = P.keys[k];
    const u64 f = (u64)((idx / D.mult[k]) % (u32)D.range[k]);  // ranges fit 32 bits (their product does)
    if (c.nullbit >= 0 && f == D.range[k] - 1) {
      key |= 1ull << c.nullbit;
    } else {
      const u64 v = (u64)((i64)f + D.min[k]);
      key |= (c.width == 8 ? v : (v & ((1ull << (8 * c.width)) - 1ull))) << c.shift;
    }
  }
  return key;
}

__device__ __forceinline__ void prefetch_l2(const void* p)
{
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// One CTA (the last one of k_table_init) looks at 1024 evenly spaced rows and derives the dense key
// box, or disables it when the box would not fit `cap_slots` shared-memory slots.  The fused kernels
// read the box from the control block, so there is no host round trip.  Keys outside the box are
// still aggregated correctly, through the global table.  Must be called
// by all TABLE_INIT_BLOCK threads of the CTA.
constexpr int SAMPLE_PER_THREAD = SAMPLE_ROWS / 256;
constexpr int SAMPLE_COLS = 2;  // key columns whose loads are in flight together
__device__ __forceinline__ void sample_dense_box(const DPlan& P, u32 cap_slots, bool count_keys, u64 claim_limit, DDense* out, DPartitionFrom from)
{
  __shared__ i64 s_min[MAX_KEYS], s_max[MAX_KEYS];
  __shared__ u32 s_vexp, s_spread, s_distinct, s_top, s_taken;
  __shared__ u64 s_keys[2 * SAMPLE_ROWS];
  __shared__ u32 s_counts[2 * SAMPLE_ROWS];
  if (count_keys) for (int i = threadIdx.x; i < 2 * SAMPLE_ROWS; i += blockDim.x) { s_keys[i] = EMPTY; s_counts[i] = 0; }
  if (threadIdx.x < MAX_KEYS) { s_min[threadIdx.x] = 0x7FFFFFFFFFFFFFFFll; s_max[threadIdx.x] = (i64)0x8000000000000000ull; }
  if (threadIdx.x == 0) { s_vexp = 0; s_spread = 0; s_distinct = 0; s_top = 0; s_taken = 0; }
  __syncthreads();
  const i64 nsamp  = P.nrows < SAMPLE_ROWS ? P.nrows : SAMPLE_ROWS;
  const i64 stride = P.nrows / (nsamp > 0 ? nsamp : 1);
  auto count_key = [&](u64 key) {  // occurrences per key, in a table twice the sample's size
    if (key == EMPTY) return;
    u32 at = (u32)(mix64(key) >> 40) & (2 * SAMPLE_ROWS - 1);
    for (;;) {  // ends: half of the slots stay free
      const u64 old = atomicCAS(&s_keys[at], EMPTY, key);
      if (old == EMPTY) atomicAdd(&s_distinct, 1u);
      if (old == EMPTY || old == key) break;
      at = (at + 1) & (2 * SAMPLE_ROWS - 1);
    }
    atomicMax(&s_top, atomicAdd(&s_counts[at], 1u) + 1u);
    atomicAdd(&s_taken, 1u);
  };
  if (P.key_mode == KM_ROWS) {
    if (count_keys) {
      for (i64 i = threadIdx.x; i < nsamp; i += blockDim.x) {
        const i64 row = i * stride + (stride > 1 ? (i64)(((u64)i * 7919ull) % (u64)stride) : 0);
        if (row_active(P, row)) count_key(hash_row(P, row));  // (the row's hash stands for its key)
      }
    }
  } else if (P.key_mode == KM_PACKED) {
    i64 rows[SAMPLE_PER_THREAD];
    u32 ok = 0;  // bit j: sample j of this thread takes part
#pragma unroll
    for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
      const i64 i = (i64)threadIdx.x + (i64)j * blockDim.x;
      rows[j] = i < nsamp ? i * stride + (stride > 1 ? (i64)(((u64)i * 7919ull) % (u64)stride) : 0) : 0;
      if (i < nsamp) ok |= 1u << j;
    }
    u32 first_filter[SAMPLE_PER_THREAD] = {~0u, ~0u, ~0u, ~0u};  // (looked at behind the loads of the columns)
    static_assert(SAMPLE_PER_THREAD == 4, "first_filter");
    if (P.nfilters > 0) {
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
        first_filter[j] = __ldg(P.filters[0] + ((P.filter_offsets[0] + rows[j]) >> 5)) >> ((P.filter_offsets[0] + rows[j]) & 31);
    }
    for (int f = 1; f < P.nfilters; ++f) {
      u32 w[SAMPLE_PER_THREAD];
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j) w[j] = __ldg(P.filters[f] + ((P.filter_offsets[f] + rows[j]) >> 5));
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
        if (!((w[j] >> ((P.filter_offsets[f] + rows[j]) & 31)) & 1u)) ok &= ~(1u << j);
    }
    // The loads of up to SAMPLE_COLS key columns (their values and masks) and of the values' exponents are issued
    // together: the sampler sits between the launch and the first row of the fused kernel, and what it costs is DRAM
    // round trips (column by column it took 8 us with one key column, 11.5 us with two).
    u32 ex[SAMPLE_PER_THREAD] = {}, exok[SAMPLE_PER_THREAD] = {};
    if (P.flags & PF_VEXP) {
      const DValCol& vc = P.vals[P.cells[0].col];
      const bool v8 = vc.vclass == VC_F64;
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
        ex[j] = v8 ? __ldg((const u32*)vc.data + 2 * (vc.offset + rows[j]) + 1) >> 20 : __ldg((const u32*)vc.data + vc.offset + rows[j]) >> 23;
        exok[j] = vc.mask ? __ldg(vc.mask + ((vc.offset + rows[j]) >> 5)) >> ((vc.offset + rows[j]) & 31) : 1u;
      }
    }
    u64 keys[SAMPLE_PER_THREAD] = {};
    for (int k0 = 0; k0 < P.nkeys; k0 += SAMPLE_COLS) {
      u64 bits[SAMPLE_COLS][SAMPLE_PER_THREAD];
      u32 w[SAMPLE_COLS][SAMPLE_PER_THREAD];
#pragma unroll
      for (int i = 0; i < SAMPLE_COLS; ++i) {
        if (k0 + i >= P.nkeys) continue;
        const DKeyCol& c = P.keys[k0 + i];
#pragma unroll
        for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
          bits[i][j] = load_fixed_bits(c.data, c.offset + rows[j], c.width);
          w[i][j]    = c.mask ? __ldg(c.mask + ((c.offset + rows[j]) >> 5)) >> ((c.offset + rows[j]) & 31) : 1u;
        }
      }
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
        if (!(first_filter[j] & 1u)) ok &= ~(1u << j);
      if (!P.include_nulls) {  // EXCLUDE: a null key drops the row (for the columns looked at so far: a row kept too long only widens a box)
#pragma unroll
        for (int i = 0; i < SAMPLE_COLS; ++i)
#pragma unroll
          for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
            if (k0 + i < P.nkeys && !(w[i][j] & 1u)) ok &= ~(1u << j);
      }
#pragma unroll
      for (int i = 0; i < SAMPLE_COLS; ++i) {
        if (k0 + i >= P.nkeys) continue;
        const DKeyCol& c = P.keys[k0 + i];
        const int sh = 64 - 8 * c.width;
        i64 lo = 0x7FFFFFFFFFFFFFFFll, hi = (i64)0x8000000000000000ull;
#pragma unroll
        for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
          keys[j] |= (c.nullbit >= 0 && !(w[i][j] & 1u)) ? 1ull << c.nullbit : bits[i][j] << c.shift;
#pragma unroll
        for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
          if (!((ok >> j) & 1u) || !(w[i][j] & 1u)) continue;
          const i64 v = c.is_signed ? ((i64)(bits[i][j] << sh) >> sh) : (i64)bits[i][j];
          lo = v < lo ? v : lo;
          hi = v > hi ? v : hi;
        }
        for (int d = 16; d > 0; d >>= 1) {
          const i64 ol = __shfl_xor_sync(0xFFFFFFFFu, lo, d), oh = __shfl_xor_sync(0xFFFFFFFFu, hi, d);
          lo = ol < lo ? ol : lo;
          hi = oh > hi ? oh : hi;
        }
        if ((threadIdx.x & 31) == 0 && lo <= hi) { atomicMin(&s_min[k0 + i], lo); atomicMax(&s_max[k0 + i], hi); }
      }
    }
    if (count_keys) {
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j)
        if ((ok >> j) & 1u) count_key(keys[j]);
    }
    if (P.flags & PF_VEXP) {
      // the largest exponent among the sampled values places the window of the fixed point
      // (zeros, denormals, infinities and NaN say nothing about it; a null's payload is not looked at)
      const u32 top = P.vals[P.cells[0].col].vclass == VC_F64 ? 0x7FFu : 0xFFu;
      u32 emax = 0;
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
        const u32 e = ex[j] & top;
        if (((ok >> j) & 1u) && (exok[j] & 1u) && e != 0u && e != top && e + 1u > emax) emax = e + 1u;
      }
      emax = __reduce_max_sync(0xFFFFFFFFu, emax);
      if ((threadIdx.x & 31) == 0 && emax) atomicMax(&s_vexp, emax);
      __syncthreads();
      const bool v8 = P.vals[P.cells[0].col].vclass == VC_F64;
      const int least = (int)s_vexp - 1 + PK_HEADROOM - pk_span(v8, false);
      u32 below = 0;
#pragma unroll
      for (int j = 0; j < SAMPLE_PER_THREAD; ++j) {
        const u32 e = ex[j] & top;
        if (((ok >> j) & 1u) && (exok[j] & 1u) && e != 0u && (int)e < least) ++below;
      }
      below = __reduce_add_sync(0xFFFFFFFFu, below);
      if ((threadIdx.x & 31) == 0 && below) atomicAdd(&s_spread, below);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    DDense& D = *out;
    D.enabled = 0;
    D.total   = 0;
    D.copies  = 1;
    D.sampled = 0;
    D.vexp    = s_vexp;
    D.wide    = s_spread > pk_spread_limit(P.nrows) ? 1u : 0u;
    D.est_groups = count_keys && s_taken >= SAMPLE_ROWS / 2 ? groups_of_sample(s_taken, s_distinct) : 0u;
    D.top_count  = s_top;
    D.too_many   = min((u64)D.est_groups, (u64)P.nrows) > 2 * claim_limit ? 1u : 0u;
    bool ok   = P.key_mode == KM_PACKED && nsamp >= SAMPLE_ROWS && cap_slots > 0;
    for (int pass = 0; pass < 2 && ok && !D.enabled; ++pass) {  // pass 0: padded box, pass 1: tight box
      u64 total = 1;
      bool fits = true;
      for (int k = 0; k < P.nkeys && fits; ++k) {
        i64 lo = s_min[k], hi = s_max[k];
        if (lo > hi) { lo = 0; hi = 0; }
        const u64 span = (u64)(hi - lo);
        if (span >= (u64)cap_slots) { fits = false; break; }
        const u64 pad = pass == 0 ? (span / 8 + 1 < 64 ? span / 8 + 1 : 64) : 0;
        // Only values that the column's type has: the lean kernel compares 4-byte keys modulo 2^32, and with a box that
        // reached below 0 of a UINT32 column it met 0xFFFFFFFF inside a box that dense_index says it lies outside of.
        const int bits = 8 * P.keys[k].width;
        const bool wide = bits == 64, sgn = P.keys[k].is_signed != 0;
        const i64 least = wide ? (i64)0x8000000000000000ull : sgn ? -(1ll << (bits - 1)) : 0;
        const i64 most  = wide ? 0x7FFFFFFFFFFFFFFFll : sgn ? (1ll << (bits - 1)) - 1 : (1ll << bits) - 1;
        const u64 below = min(pad, (u64)lo - (u64)least), above = min(pad, (u64)most - (u64)hi);
        D.min[k]   = lo - (i64)below;
        D.range[k] = span + 1 + below + above + (P.keys[k].nullbit >= 0 ? 1 : 0);
        D.mult[k]  = (u32)total;
        total *= D.range[k];
        if (total > (u64)cap_slots) fits = false;
      }
      if (fits) {
        D.enabled = 1;
        D.total   = (u32)total;
        const u32 r = cap_slots / (u32)total;
        D.copies  = r < 1 ? 1u : (r > 32u ? 32u : r);
      }
    }
    if (!D.enabled) {  // what was seen, for whoever plans with it
      for (int k = 0; k < P.nkeys; ++k) { D.min[k] = s_min[k]; D.range[k] = s_min[k] <= s_max[k] ? (u64)(s_max[k] - s_min[k]) : 0ull; }
      D.sampled = P.key_mode == KM_PACKED && nsamp >= SAMPLE_ROWS ? 1u : 0u;
      // (an attempt on a table that turns out too small costs 100 us and more, partitions in place of a table that would have done
      // some 50: 1.5 times what it holds decides there)
      if (D.sampled && from.sparse && min((u64)D.est_groups, (u64)P.nrows) > claim_limit + claim_limit / 2) D.too_many = 1;
      if (D.sampled && D.est_groups && s_top < PART_TOP_COUNT) {
        const u64 most = 2ull * (u64)P.nrows;
        u64 values = P.nkeys <= 2 ? 1 : most + 1;
        for (int k = 0; k < P.nkeys && values <= most; ++k) values = D.range[k] < most ? values * (D.range[k] + 1) : most + 1;
        const u32 limit = values <= most ? from.dense : from.sparse;
        if (limit && min((u64)D.est_groups, (u64)P.nrows) >= limit) D.too_many = 1;
      }
    }
  }
  __syncthreads();
}

// For a batch of a state whose cells are Σ and n of one float column: do its keys span a box of at most `cap_lean` slots?
// Such a batch is left to the lean kernel, whose sums are exact until they are merged.  One CTA of TABLE_INIT_BLOCK threads.
__global__ void __launch_bounds__(TABLE_INIT_BLOCK) k_state_sample(const __grid_constant__ DPlan P, DCtrl* ctrl, u32 cap_lean)
{
  __shared__ DDense s_box;
  sample_dense_box(P, cap_lean, false, ~0ull >> 1, &s_box);
  if (threadIdx.x == 0) ctrl->lean_box = s_box.enabled ? 1u : 0u;
}

// the sample on its own
__global__ void __launch_bounds__(TABLE_INIT_BLOCK) k_key_sample(const __grid_constant__ DPlan P, DDense* out, u32 cap_box)
{
  __shared__ u32 s_runs;
  if (threadIdx.x == 0) s_runs = 0;
  sample_dense_box(P, cap_box, true, ~0ull >> 1, out);
  const i64 nsamp = P.nrows < SAMPLE_ROWS ? P.nrows : SAMPLE_ROWS, stride = P.nrows / (nsamp > 0 ? nsamp : 1);
  u32 runs = 0;
  for (i64 i = threadIdx.x; i < nsamp; i += blockDim.x) {
    const i64 row = i * stride + (stride > 1 ? (i64)(((u64)i * 7919ull) % (u64)stride) : 0);
    bool same = row + 1 < P.nrows;
    for (int k = 0; k < P.nkeys && same; ++k) {
      const DKeyCol& c = P.keys[k];
      const bool a = !c.mask || bit_valid(c.mask, c.offset + row), b = !c.mask || bit_valid(c.mask, c.offset + row + 1);
      same = a == b && (!a || load_fixed_bits(c.data, c.offset + row, c.width) == load_fixed_bits(c.data, c.offset + row + 1, c.width));
    }
    runs += same;
  }
  runs = __reduce_add_sync(0xFFFFFFFFu, runs);
  if ((threadIdx.x & 31) == 0 && runs) atomicAdd(&s_runs, runs);
  __syncthreads();
  if (threadIdx.x == 0) out->runs = s_runs;
}

// shared-memory atomics on 32-bit shared addresses (native on sm_100a; measured at ~73 % of the
// HBM roofline for one float add + one count add per row into a direct-indexed table)
__device__ __forceinline__ void sred_add_f32(u32 saddr, float v)
{
  asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(saddr), "f"(v) : "memory");
}
__device__ __forceinline__ u32 satom_add_u32(u32 saddr, u32 v)
{
  u32 old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(saddr), "r"(v) : "memory");
  return old;
}
// 4 validity bits at a position that is a multiple of 4
__device__ __forceinline__ u32 nibble_aligned(const u32* mask, u32 pos)
{
  return (__ldg(mask + (pos >> 5)) >> (pos & 31u)) & 0xFu;
}

// ------------------------------------------------------------------------------ fused aggregate
// ONE pass over keys + values + bitmasks.  Each thread takes 4 consecutive rows per tile (16-byte
// vector loads when the columns allow, validity read as 4-bit nibbles of the mask words).  Each CTA
// owns a shared-memory table in front of the global table:
//   dense mode  : slot = position of the key in the sampled key box (sample_dense_box), accumulators
//                 only, no probing;
//   hashed mode : open addressing with linear probing on the 64-bit key cell, first come first
//                 cached until `fill_limit`; a CTA whose cache stops paying off turns it off.
// Rows whose key is not in shared memory go to the global table with global atomics.  At the end
// every CTA merges its table into the global one.  There is no barrier inside the row loop.
__device__ __forceinline__ u64 global_timer_ns()
{
  u64 t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

}  // namespace b2
#include "b2_box.cuh"  // the pass over a sampled key box
namespace b2 {

template <int KM, int LAYOUT>
__global__ void __launch_bounds__(AGG_BLOCK, 1)
k_aggregate(const __grid_constant__ DPlan P, const __grid_constant__ DForms F, u64* __restrict__ tbl, i64 cap, DCtrl* ctrl, int S_hash, int fill_limit,
            u32 cap_dense, u32 region_slots, int batch)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int s_fill, s_new, s_cache_on, s_abort, s_hit, s_miss;
  __shared__ DDense s_dense;

  grid_dependents_launch();  // (k_report)
  const int stride = P.stride;
  const int tid    = threadIdx.x;
  const i64 dense_slots = (i64)region_slots;  // structure-of-arrays slots behind the special slot
  const bool timekeeper = blockIdx.x == 0 && tid == 0;
  const u64 t_start = timekeeper ? global_timer_ns() : 0;
  if ((batch & BATCH_SAMPLED) && ctrl->lean_box) return;  // (left to the lean kernel, see k_state_sample)
  if ((batch & BATCH_REST) && !((ctrl->cache_ctas[blockIdx.x >> 5] >> (blockIdx.x & 31)) & 1u)) return;
  const bool sampled = LAYOUT != SL_NONE && (KM == KM_ROWS || cap_dense > 0);
  if (sampled) {
    // the key box sampled by k_table_init, which precedes this kernel on the stream
    for (int i = tid; i < (int)(sizeof(DDense) / 4); i += blockDim.x) ((u32*)&s_dense)[i] = ((const u32*)&ctrl->dense)[i];
  } else if (tid == 0) {
    s_dense.enabled = 0;
  }
  // A batch of a state: what the table's first batch looked like says nothing about it.  The kernel without a cache (its L1
  // is larger and its row loop shorter: 1M rows, 100K groups, three cells 38 us, with the cache present but off 55) looks at
  // 1024 rows of every CTA and leaves those of a CTA that needs one to a second launch (BATCH_REST); with a cache every CTA
  // notes at its end whether the cache paid.
  if (KM == KM_PACKED && batch) {
    if constexpr (KM == KM_PACKED && LAYOUT == SL_NONE) {
      __shared__ u64 s_sample[BATCH_SAMPLE_BYTES / 8];
      const bool pays = cache_pays_here(P, s_sample, S_hash);
      if (tid == 0) note_cache(ctrl, pays);
      if (pays) return;
    } else {
      __syncthreads();
      if (tid == 0) s_dense.est_groups = s_dense.too_many = 0;  // (unknown)
    }
  }
  if (tid == 0) { s_fill = 0; s_new = 0; s_cache_on = (LAYOUT != SL_NONE); s_abort = 0; s_hit = 0; s_miss = 0; }
  __syncthreads();
  if (timekeeper) { ctrl->t_phase[0] = t_start; ctrl->t_phase[1] = global_timer_ns(); }
  if (sampled && s_dense.too_many) {  // a table that would overflow is not filled first
    if (tid == 0) ctrl->overflow = 1;
    return;
  }
  if constexpr (KM == KM_PACKED && LAYOUT == SL_GENERIC) {
    if (s_dense.enabled) {
      box_aggregate(P, F, tbl, cap, ctrl, dense_slots, s_dense, smem_raw, &s_new, &s_abort, timekeeper);
      if (tid == 0) {
        if (s_new) {
          const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)s_new) + (u64)s_new;
          if (tot > ctrl->claim_limit) ctrl->overflow = 1;
        }
        if (timekeeper) ctrl->t_phase[4] = global_timer_ns();
        if (batch) note_cache(ctrl, true);
      }
      return;
    }
  }
  const bool dense = LAYOUT == SL_F32MEAN && KM == KM_PACKED && s_dense.enabled;  // (the compact slots: also addressed by the box)
  const int S      = dense ? (int)s_dense.total : S_hash;  // slots (hashed mode: + the special slot at S)
  const int NS     = dense ? S * (int)s_dense.copies : S + 1;  // allocated slots per array
  // dense mode: this warp's replica of the table
  const u32 copy_off = dense ? (u32)((threadIdx.x >> 5) % s_dense.copies) * (u32)S : 0u;
  // global slot of dense-box position i: the dense region behind the special slot (the one key whose
  // bits equal EMPTY cannot mark a key cell as used and goes to the special slot instead)
  auto dense_gslot = [&](u32 i) -> i64 { return dense_key(P, s_dense, i) == EMPTY ? cap : cap + 1 + (i64)i; };

  // Hashed mode: a cache pays when its slots meet their keys again — few groups for the rows of a CTA, or keys so
  // frequent that their rows would queue at one global slot.  Otherwise it only postpones the global atomics to the
  // merge (1M rows, 100K groups: 63 us with it, 27 without).
  const bool cached = LAYOUT != SL_NONE && (dense || !sampled || cache_pays_for(P.nrows / gridDim.x, s_dense.est_groups, s_dense.top_count, S_hash));

  // shared-memory arrays
  u64* skeys  = (u64*)smem_raw;                            // hashed mode only: [NS]
  u64* scells = dense ? (u64*)smem_raw : skeys + NS;       // SL_GENERIC: [ncells][NS]
  float* ssum = (float*)scells;                            // SL_F32MEAN: [NS] fp32 partial sums
  u32* scnt   = (u32*)(ssum + NS);                         // SL_F32MEAN: [NS] counts
  u32* socc   = (u32*)(scells + (size_t)(LAYOUT == SL_F32MEAN ? 1 : P.ncells) * NS);  // dense mode: occupancy bits
  if (cached) {
    if (!dense) for (int i = tid; i < NS; i += blockDim.x) skeys[i] = EMPTY;
    if (LAYOUT == SL_GENERIC) {
      for (int c = 0; c < P.ncells; ++c) {
        const u64 id = cell_identity(P.cells[c].op);
        for (int i = tid; i < NS; i += blockDim.x) scells[(size_t)c * NS + i] = id;
      }
    } else {
      for (int i = tid; i < NS; i += blockDim.x) scells[i] = 0;  // {sum, count} arrays together
    }
    if (dense) for (int i = tid; i < (NS + 31) / 32; i += blockDim.x) socc[i] = 0;
  }
  __syncthreads();
  if (timekeeper) ctrl->t_phase[2] = global_timer_ns();

  u32 my_hit = 0, my_miss = 0, tot_hit = 0, tot_miss = 0;
  const i64 rows_done = 0;

  const i64 tile_rows = (i64)blockDim.x * AGG_ROWS;
  const i64 ntiles    = (P.nrows - rows_done + tile_rows - 1) / tile_rows;

  // A warp leaves as one: a tile has synchronisations of the whole warp, and its lanes need not read the flag at the same time.
  // (Asked at the end of a tile for packed keys, at its start for row keys: 110M rows, 111 sparse keys, min / max / mean 1268 us
  // and 1293, without asking together 1260; 4M rows over FLOAT64 keys, sum / count 198 and 193.)
  auto leave = [&] { return __any_sync(0xFFFFFFFFu, *(volatile int*)&s_abort != 0) != 0; };
  bool stop = false;
  for (i64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (KM == KM_PACKED ? stop : leave()) break;
    const i64 row0 = rows_done + tile * tile_rows + (i64)tid * AGG_ROWS;
    const int nv   = (int)max((i64)0, min((i64)AGG_ROWS, P.nrows - row0));
    const bool cache_on = cached && (dense || *(volatile int*)&s_cache_on);

    // ---- loads first, all independent of each other, so that one DRAM round trip covers the tile
    const bool full = nv == AGG_ROWS;
    const bool vec  = KM == KM_PACKED && full && (P.flags & PF_VEC_KEYS);
    u32 act = nv > 0 ? ((1u << nv) - 1u) : 0u;
    int sl[AGG_ROWS];
    u64 kk[AGG_ROWS];
    u32 di[AGG_ROWS];   // dense mode: slot inside the key box
    u32 dout = 0;       // dense mode: rows whose key lies outside the box
#pragma unroll
    for (int j = 0; j < AGG_ROWS; ++j) { sl[j] = SLOT_NONE; kk[j] = 0; di[j] = copy_off; }
    float fx[AGG_ROWS] = {0.f, 0.f, 0.f, 0.f};  // SL_F32MEAN: the values
    u32 fvn = 0xFu;                              // SL_F32MEAN: their validity
    if (LAYOUT == SL_F32MEAN && full && (P.flags & PF_VEC_VAL0)) {
      const DValCol& vc = P.vals[P.cells[0].col];
      const float4 q = __ldg((const float4*)((const float*)vc.data + vc.offset + row0));
      fx[0] = q.x; fx[1] = q.y; fx[2] = q.z; fx[3] = q.w;
      if (vc.mask) fvn = valid_nibble(vc.mask, vc.offset + row0, nv);
    }
    if (vec) {
      for (int k = 0; k < P.nkeys; ++k) {
        const DKeyCol& c = P.keys[k];
        const unsigned char* src = c.data + (c.offset + row0) * c.width;
        u64 f[AGG_ROWS];
        if (c.width == 4) {
          const uint4 q = __ldg((const uint4*)src);
          f[0] = q.x; f[1] = q.y; f[2] = q.z; f[3] = q.w;
        } else if (c.width == 8) {
          const ulonglong2 q0 = __ldg((const ulonglong2*)src), q1 = __ldg((const ulonglong2*)src + 1);
          f[0] = q0.x; f[1] = q0.y; f[2] = q1.x; f[3] = q1.y;
        } else if (c.width == 2) {
          const uint2 q = __ldg((const uint2*)src);
          f[0] = q.x & 0xFFFFu; f[1] = q.x >> 16; f[2] = q.y & 0xFFFFu; f[3] = q.y >> 16;
        } else {
          const u32 q = __ldg((const u32*)src);
          f[0] = q & 0xFFu; f[1] = (q >> 8) & 0xFFu; f[2] = (q >> 16) & 0xFFu; f[3] = q >> 24;
        }
        u32 vn = 0xFu;
        if (c.mask) {
          vn = valid_nibble(c.mask, c.offset + row0, nv);
          if (!P.include_nulls) act &= vn;  // EXCLUDE: a null key drops the row
        }
        const int sh = 64 - 8 * c.width;
#pragma unroll
        for (int j = 0; j < AGG_ROWS; ++j) {
          const bool isnull = c.nullbit >= 0 && !((vn >> j) & 1u);
          kk[j] |= isnull ? (1ull << c.nullbit) : (f[j] << c.shift);
          if (dense) {
            const i64 ov = c.is_signed ? ((i64)(f[j] << sh) >> sh) : (i64)f[j];
            u64 d = (u64)(ov - s_dense.min[k]);
            const u64 lim = s_dense.range[k] - (c.nullbit >= 0 ? 1ull : 0ull);
            if (isnull) d = lim;
            else if (d >= lim) dout |= 1u << j;
            di[j] += (u32)d * s_dense.mult[k];
          }
        }
      }
    } else if (act && !P.include_nulls) {
      for (int k = 0; k < P.nkeys; ++k)
        if (P.keys[k].mask) act &= valid_nibble(P.keys[k].mask, P.keys[k].offset + row0, nv);
    }
    if (act)
      for (int f = 0; f < P.nfilters; ++f) act &= valid_nibble(P.filters[f], P.filter_offsets[f] + row0, nv);

    // ---- phase A: keys -> slots
    if (act) {
      if (!vec) {
#pragma unroll
        for (int j = 0; j < AGG_ROWS; ++j)
          if ((act >> j) & 1u) {
            kk[j] = (KM == KM_PACKED) ? pack_key(P, row0 + j) : hash_row(P, row0 + j);
            if (dense) {
              const int s = dense_index(P, s_dense, kk[j]);
              if (s < 0) dout |= 1u << j; else di[j] = copy_off + (u32)s;
            }
          }
      }
      // shared-memory table first
      u32 miss = 0;
      u64 hh[AGG_ROWS];
#pragma unroll
      for (int j = 0; j < AGG_ROWS; ++j) {
        hh[j] = 0;
        if (!((act >> j) & 1u)) continue;
        int s = -1;
        if (dense) {
          if (!((dout >> j) & 1u)) {
            s = (int)di[j];
            if (!((socc[s >> 5] >> (s & 31)) & 1u)) atomicOr(&socc[s >> 5], 1u << (s & 31));
          }
        } else {
          hh[j] = (KM == KM_PACKED) ? mix64(kk[j]) : kk[j];
          if (cache_on) s = smem_find_insert<KM>(P, skeys, S, fill_limit, &s_fill, kk[j], hh[j], row0 + j);
        }
        if (s >= 0) {
          sl[j] = s;
          ++my_hit;
        } else {
          if (dense) hh[j] = mix64(kk[j]);
          miss |= 1u << j;
          ++my_miss;
        }
      }
      // then the global table: the home slots of all my missing rows are loaded together (their
      // DRAM latencies overlap), then each row finishes its probe sequence
      if (miss) {
        if (KM == KM_PACKED) {
          i64 gi[AGG_ROWS];
          u64 gk[AGG_ROWS];
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) {
            gi[j] = (i64)reduce64(hh[j], (u64)cap);
            gk[j] = 0;
            if (((miss >> j) & 1u) && kk[j] != EMPTY) gk[j] = *(volatile u64*)(tbl + gi[j] * stride);
          }
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) {
            if (!((miss >> j) & 1u)) continue;
            i64 g;
            if (kk[j] == EMPTY) {
              if (ctrl->special_used == 0) ctrl->special_used = 1;
              g = cap;
            } else {
              g = gmem_finish_packed(tbl, cap, stride, kk[j], gi[j], gk[j], ctrl, &s_new);
            }
            if (g >= 0) sl[j] = -2 - (int)g;
          }
        } else {
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) {
            if (!((miss >> j) & 1u)) continue;
            const i64 g = gmem_find_insert_rows(P, tbl, cap, stride, row0 + j, hh[j], ctrl, &s_new);
            if (g >= 0) sl[j] = -2 - (int)g;
          }
        }
      }
    }
    __syncwarp();  // reconverge after the divergent probe loops before the accumulate phase

    // ---- phase B: fold the values
    if (LAYOUT == SL_F32MEAN) {
      // cells: [0] = Σx of a FLOAT32 column, [1] = n of the same column
      const DValCol& vc = P.vals[P.cells[0].col];
      if (act) {
        u32 vn = act;
        float x[AGG_ROWS];
        if (full && (P.flags & PF_VEC_VAL0)) {
          vn &= fvn;
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) x[j] = fx[j];
        } else {
          if (vc.mask) vn &= valid_nibble(vc.mask, vc.offset + row0, nv);
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) x[j] = ((vn >> j) & 1u) ? __ldg((const float*)vc.data + vc.offset + row0 + j) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < AGG_ROWS; ++j) {
          if (sl[j] == SLOT_NONE || !((vn >> j) & 1u)) continue;
          if (sl[j] >= 0) {
            atomicAdd(ssum + sl[j], x[j]);
            const u32 old = atomicAdd(scnt + sl[j], 1u);
            if (((old + 1u) & (F32_SPILL_AT - 1u)) == 0u) {
              // every F32_SPILL_AT-th addend moves the fp32 partial of this key to the fp64 global
              // cell, so that no fp32 sum ever holds many more addends than that
              const float part = atomicExch(ssum + sl[j], 0.f);
              i64 g;
              if (dense) {
                g = dense_gslot((u32)sl[j] - copy_off);
              } else {
                const u64 key = sl[j] == S ? EMPTY : skeys[sl[j]];
                g = gmem_find_insert_packed(tbl, cap, stride, key, mix64(key), ctrl, &s_new);
              }
              if (g >= 0) atomicAdd((double*)slot_ref(tbl, cap, stride, dense_slots, g).cells, (double)part);
            }
          } else {
            u64* slot = tbl + (i64)(-2 - sl[j]) * stride;
            atomicAdd((double*)(slot + 1), (double)x[j]);
            atomicAdd(slot + 2, 1ull);
          }
        }
      }
    } else {
      int cur_col = -1;
      u64 v[AGG_ROWS];
      u32 vn = 0;
      for (int c = 0; c < P.ncells; ++c) {
        const int op  = P.cells[c].op;
        const int col = P.cells[c].col;
        if (op != OP_CNT_A && col != cur_col) {
          cur_col = col;
          const DValCol& vc = P.vals[col];
          vn = act;
          if (vn && vc.mask) vn &= valid_nibble(vc.mask, vc.offset + row0, nv);
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) v[j] = ((vn >> j) & 1u) && sl[j] != SLOT_NONE ? load_value(vc, row0 + j) : 0;
        }
        const u32 use = (op == OP_CNT_A) ? act : vn;
        u64* where[AGG_ROWS];
        u32 in_shared = 0;
#pragma unroll
        for (int j = 0; j < AGG_ROWS; ++j) {
          const bool sh = LAYOUT == SL_GENERIC && sl[j] >= 0;
          where[j] = scells + (size_t)c * NS + (sh ? sl[j] : 0);
          if (sh) in_shared |= 1u << j;
        }
        if (LAYOUT == SL_GENERIC) cell_update_shared<AGG_ROWS>(where, op, v, use & in_shared);
        if (use & ~in_shared) {
#pragma unroll
          for (int j = 0; j < AGG_ROWS; ++j) {
            if (sl[j] == SLOT_NONE || !(((use & ~in_shared) >> j) & 1u)) continue;
            if (is_arg_op(op)) arg_update(tbl + (i64)(-2 - sl[j]) * stride + 1 + c, op, P.vals[col], row0 + j);  // (global table only)
            else {
              const SlotRef slot = slot_ref(tbl, cap, stride, dense_slots, (i64)(-2 - sl[j]));
              cell_update(slot.cells + (i64)c * slot.step, op, v[j]);
            }
          }
        }
      }
    }

    if (KM == KM_PACKED) stop = leave();
    // ---- bookkeeping by one lane per CTA, no barrier: claims, overflow, cache pay-off
    if (cached && !dense) {
      const u32 wh = __reduce_add_sync(0xFFFFFFFFu, my_hit), wm = __reduce_add_sync(0xFFFFFFFFu, my_miss);
      if ((tid & 31) == 0) { if (wh) atomicAdd(&s_hit, (int)wh); if (wm) atomicAdd(&s_miss, (int)wm); }
      tot_hit += my_hit; tot_miss += my_miss;
      my_hit = 0; my_miss = 0;
    }
    if (tid == 0) {
      const int c = atomicExch(&s_new, 0);
      if (c) {
        const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)c) + (u64)c;
        if (tot > ctrl->claim_limit) ctrl->overflow = 1;
      }
      if (*(volatile u32*)&ctrl->overflow) s_abort = 1;
      if (cached && !dense && s_cache_on && s_fill >= fill_limit) {
        const int h = atomicExch(&s_hit, 0), m = atomicExch(&s_miss, 0);
        if (m > 3 * h && m > 1024) s_cache_on = 0;
      }
    }
  }

  // ---- statistics: rows folded in shared memory / sent to the global table
  tot_hit  = __reduce_add_sync(0xFFFFFFFFu, tot_hit + my_hit);
  tot_miss = __reduce_add_sync(0xFFFFFFFFu, tot_miss + my_miss);
  if ((tid & 31) == 0) {
    if (tot_hit) atomicAdd(&ctrl->stat_smem_rows, (u64)tot_hit);
    if (tot_miss) atomicAdd(&ctrl->stat_gmem_rows, (u64)tot_miss);
  }

  // ---- merge this CTA's table into the global table
  __syncthreads();
  if (timekeeper) ctrl->t_phase[3] = global_timer_ns();
  if (cached && !s_abort) {
    // CTAs start their merge at different slots so that they do not all hit the same global cells at once
    const int NM  = dense ? S : NS;  // dense mode: one pass over box positions, replicas reduced on the fly
    const int rot = (int)(((u64)blockIdx.x * 2654435761ull) % (u64)NM);
    int dense_new = 0;  // dense-region key cells this thread was the first to claim
    if (dense) {
      // Dense mode: the replicas of a box position are reduced in registers, then ONE merge into the
      // dense region of the global table: no hashing, consecutive threads -> consecutive words of the
      // structure-of-arrays region.  The key cell is claimed with an unconditional exchange (every
      // CTA writes the same key there).  Four positions per step: their exchanges and reductions are
      // all issued before the first returned key is looked at, so a step waits for one L2 round trip
      // instead of four (one position per step: 21 us for 15.9K positions).
      constexpr int MB = 4;
      const int copies = (int)s_dense.copies;
      for (int base = tid; base < NM; base += MB * (int)blockDim.x) {
        u64 olds[MB];
#pragma unroll
        for (int u = 0; u < MB; ++u) {
          olds[u] = 0;  // anything but EMPTY: "not newly claimed"
          const int i0 = base + u * (int)blockDim.x;
          if (i0 >= NM) continue;
          const int i = i0 + rot < NM ? i0 + rot : i0 + rot - NM;
          bool present = false;
          for (int r = 0; r < copies; ++r) {
            const int q = r * S + i;
            present = present || ((socc[q >> 5] >> (q & 31)) & 1u) || scnt[q] != 0u;
          }
          if (!present) continue;
          const u64 key = dense_key(P, s_dense, (u32)i);
          i64 g;
          if (key == EMPTY) {
            g = cap;
            if (ctrl->special_used == 0) ctrl->special_used = 1;
          } else {
            g = cap + 1 + (i64)i;
          }
          const SlotRef slot = slot_ref(tbl, cap, stride, dense_slots, g);
          if (key != EMPTY) olds[u] = atomicExch(slot.key, key);
          double sum = 0.0;
          u64 n = 0;
          for (int r = 0; r < copies; ++r) { sum += (double)ssum[r * S + i]; n += scnt[r * S + i]; }
          if (n) { atomicAdd((double*)slot.cells, sum); atomicAdd(slot.cells + slot.step, n); }
        }
#pragma unroll
        for (int u = 0; u < MB; ++u) dense_new += olds[u] == EMPTY ? 1 : 0;
      }
    }
    for (int i0 = tid; !dense && i0 < NM; i0 += blockDim.x) {
      const int i = i0 + rot < NM ? i0 + rot : i0 + rot - NM;
      u64 key = skeys[i];
      if (key == EMPTY) continue;
      if (i == S) key = EMPTY;  // the special slot holds the key whose bits equal EMPTY
      i64 g;
      if (KM == KM_PACKED) {
        g = gmem_find_insert_packed(tbl, cap, stride, key, mix64(key), ctrl, &s_new);
      } else {
        const i64 row = (i64)(u32)key;
        g = gmem_find_insert_rows(P, tbl, cap, stride, row, hash_row(P, row), ctrl, &s_new);
      }
      if (g < 0) continue;
      u64* slot = tbl + g * stride;
      if (LAYOUT == SL_F32MEAN) {
        const u32 n = scnt[i];
        if (n) {
          atomicAdd((double*)(slot + 1), (double)ssum[i]);
          atomicAdd(slot + 2, (u64)n);
        }
      } else {
        for (int c = 0; c < P.ncells; ++c) {
          const int op = P.cells[c].op;
          const u64 a  = scells[(size_t)c * NS + i];
          if (a != cell_identity(op)) cell_merge(slot + 1 + c, op, a);
        }
      }
    }
    if (dense_new) atomicAdd(&s_new, dense_new);
  }
  __syncthreads();
  if (tid == 0) {
    if (s_new) {
      const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)s_new) + (u64)s_new;
      if (tot > ctrl->claim_limit) ctrl->overflow = 1;
    }
    if (timekeeper) ctrl->t_phase[4] = global_timer_ns();
    if (KM == KM_PACKED && LAYOUT != SL_NONE && batch) note_cache(ctrl, 2 * (i64)s_fill * gridDim.x <= P.nrows);
  }
}

// ------------------------------------------------------------------------------ cardinality estimate
// HyperLogLog over the keys of all participating rows (one streaming pass over the key columns):
// 2^13 registers, each the largest "leading zeros + 1" seen among the hashes that select it.  The host
// turns the registers into a distinct-count estimate (±~1 %) that sizes the table after the small
// speculative table overflowed — instead of growing it by trial and error.
constexpr int HLL_BITS = 13;  // 8192 registers (32 KB of static shared memory), standard error 1.15 %
constexpr int HLL_REGS = 1 << HLL_BITS;

// packed keys of 4 consecutive rows through one vector load per key column (requires PF_VEC_KEYS and
// a full group of 4 rows); clears the bits of dropped rows in `act`
__device__ __forceinline__ void packed_keys4(const DPlan& P, i64 row0, u64 (&kk)[4], u32& act)
{
#pragma unroll
  for (int j = 0; j < 4; ++j) kk[j] = 0;
  for (int k = 0; k < P.nkeys; ++k) {
    const DKeyCol& c = P.keys[k];
    const unsigned char* src = c.data + (c.offset + row0) * c.width;
    u64 f[4];
    if (c.width == 4) {
      const uint4 q = __ldg((const uint4*)src);
      f[0] = q.x; f[1] = q.y; f[2] = q.z; f[3] = q.w;
    } else if (c.width == 8) {
      const ulonglong2 q0 = __ldg((const ulonglong2*)src), q1 = __ldg((const ulonglong2*)src + 1);
      f[0] = q0.x; f[1] = q0.y; f[2] = q1.x; f[3] = q1.y;
    } else if (c.width == 2) {
      const uint2 q = __ldg((const uint2*)src);
      f[0] = q.x & 0xFFFFu; f[1] = q.x >> 16; f[2] = q.y & 0xFFFFu; f[3] = q.y >> 16;
    } else {
      const u32 q = __ldg((const u32*)src);
      f[0] = q & 0xFFu; f[1] = (q >> 8) & 0xFFu; f[2] = (q >> 16) & 0xFFu; f[3] = q >> 24;
    }
    u32 vn = 0xFu;
    if (c.mask) {
      vn = valid_nibble(c.mask, c.offset + row0, 4);
      if (!P.include_nulls) act &= vn;  // EXCLUDE: a null key drops the row
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool isnull = c.nullbit >= 0 && !((vn >> j) & 1u);
      kk[j] |= isnull ? (1ull << c.nullbit) : (f[j] << c.shift);
    }
  }
  for (int f = 0; f < P.nfilters; ++f) act &= valid_nibble(P.filters[f], P.filter_offsets[f] + row0, 4);
}

__global__ void __launch_bounds__(1024) k_hll(const __grid_constant__ DPlan P, u32* __restrict__ regs)
{
  __shared__ u32 s_regs[HLL_REGS];
  for (int i = threadIdx.x; i < HLL_REGS; i += blockDim.x) s_regs[i] = 0;
  __syncthreads();
  auto fold = [&](u64 h) {
    const u32 idx  = (u32)(h >> (64 - HLL_BITS));
    const u32 rank = (u32)__clzll((i64)((h << HLL_BITS) | (1ull << (HLL_BITS - 1)))) + 1u;
    if (s_regs[idx] < rank) atomicMax(&s_regs[idx], rank);
  };
  const i64 nquads = (P.key_mode == KM_PACKED && (P.flags & PF_VEC_KEYS)) ? P.nrows / 4 : 0;
  for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < nquads; q += (i64)gridDim.x * blockDim.x) {
    u64 kk[4];
    u32 act = 0xFu;
    packed_keys4(P, q * 4, kk, act);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if ((act >> j) & 1u) fold(mix64(kk[j] ^ 0x5bd1e9955bd1e995ull));
  }
  for (i64 row = nquads * 4 + (i64)blockIdx.x * blockDim.x + threadIdx.x; row < P.nrows; row += (i64)gridDim.x * blockDim.x) {
    if (!row_active(P, row)) continue;
    fold((P.key_mode == KM_PACKED) ? mix64(pack_key(P, row) ^ 0x5bd1e9955bd1e995ull) : hash_row(P, row));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HLL_REGS; i += blockDim.x)
    if (s_regs[i]) atomicMax(&regs[i], s_regs[i]);
}

// ------------------------------------------------------------------------------ string keys -> dictionary ids
// A STRING key column is replaced by the id of its string in a dictionary, so that (id, other keys) packs into
// one 64-bit key cell and the packed-key paths serve the aggregate.  The dictionary is an open-addressing
// table of 8-byte cells {hash tag(30) | clamped length(8) | id(26)} plus, per id, the first 32 bytes of the
// string in a dense pool (ids are handed out in order of arrival: the pool of a column with few distinct
// strings is a few contiguous megabytes that stay in L2, where the first rows' own strings — scattered over
// the column — do not) and the first row that held it (for the bytes beyond 32, and for the output).  A probe
// that finds its tag and length compares against the pool entry.  `P` holds the one string column as its only
// key.  ids[P.keys[0].offset + row] = id (0 for a null row: its null bit or its exclusion decides, not the
// payload).  Warps stop at one of their next tiles once the table or the pool is over its limit.
constexpr int DICT_BLOCK  = 256;
constexpr int DICT_CTAS   = 6;   // per SM
constexpr int DICT_TRIES  = 1 << 16;  // looks at a claimed cell, a read of L2 and up to 80 ns of sleep each, before the attempt is given up
                                      // as if the table were full (the next one has a larger table, or row keys serve the call)
constexpr int DICT_ROWS   = 4;   // rows per thread and tile, strided by the block so that loads coalesce

struct DDict {
  u64* cells;      // [cap], EMPTY = free
  i64 cap;
  u64* pool;       // [pool_cap][4]
  int* first_row;  // [pool_cap]
  i64 pool_cap;    // <= 2^26 - 2
};

// Fixed-width key columns that do not pack into 64 bits (floats, wide composites) have a dictionary of their own kind: one id
// per combination of their values, whose canonical bits — side by side in up to DICT_INLINE bytes, with a bit per nullable
// column where nulls form groups — take the string's place.  `words` is zero for strings.
struct DDictKeys {
  int words;                        // 8-byte words in use
  unsigned char at[MAX_KEYS];       // byte of every column's value (a multiple of its width)
  unsigned char null_at[MAX_KEYS];  // bit of its null flag, 255: none
};

// How many groups do rows of unpacked keys make?  One CTA hashes ROW_SAMPLES evenly spaced rows into a shared-memory table and
// tells the host in null_counts[0] the rows taken, in [1] the distinct hashes, in [2] the rows whose next row has the same key.
constexpr int ROW_SAMPLES = 2048, ROW_SAMPLE_SLOTS = 2 * ROW_SAMPLES;  // (two rows per thread: with 8192 rows the CTA took 60 us)
__global__ void __launch_bounds__(1024) k_row_sample(const __grid_constant__ DPlan P, const DReport R)
{
  extern __shared__ __align__(16) u64 rs_slots[];  // [ROW_SAMPLE_SLOTS]
  __shared__ u32 s_taken, s_distinct, s_runs;
  for (int i = threadIdx.x; i < ROW_SAMPLE_SLOTS; i += blockDim.x) rs_slots[i] = EMPTY;
  if (threadIdx.x == 0) { s_taken = 0; s_distinct = 0; s_runs = 0; }
  __syncthreads();
  const i64 step = P.nrows / ROW_SAMPLES;  // (at least one: the caller has more rows)
  u32 taken = 0, distinct = 0, runs = 0;
#pragma unroll 2
  for (int i = threadIdx.x; i < ROW_SAMPLES; i += blockDim.x) {
    const i64 row = i * step + (i64)(((u64)i * 7919ull) % (u64)step);
    if (!row_active(P, row)) continue;
    const u64 h = hash_row(P, row) & ~1ull;  // (never EMPTY)
    ++taken;
    if (row + 1 < P.nrows && row_active(P, row + 1) && (hash_row(P, row + 1) & ~1ull) == h) ++runs;
    u32 at = (u32)(h >> 20) & (ROW_SAMPLE_SLOTS - 1);
    for (;;) {  // ends: half of the slots stay free
      const u64 old = atomicCAS(&rs_slots[at], EMPTY, h);
      if (old == EMPTY) ++distinct;
      if (old == EMPTY || old == h) break;
      at = (at + 1) & (ROW_SAMPLE_SLOTS - 1);
    }
  }
  atomicAdd(&s_taken, taken);
  atomicAdd(&s_distinct, distinct);
  atomicAdd(&s_runs, runs);
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile u32* const out = R.copy->null_counts;
    out[0] = s_taken;
    out[1] = s_distinct;
    out[2] = s_runs;
    __threadfence_system();
    *(volatile u64*)R.flag = R.number;
  }
}

// Loads through L1, where a few frequent keys are met again and again (3.3M rows over 51 FLOAT64 keys: 390 us per call with every
// look at a cell going to the same few lines of L2).  L1 may hold what a word was before another SM wrote it.  A cell that
// looks free or unpublished is looked at again in L2.  An entry that matches is taken at its word: L1 is filled by sectors of 32
// bytes, an entry is exactly one, and nobody reads it before its id is published, so that a sector from before it was written is
// never there.  (Beside smaller or unaligned entries it could be; L1 is empty when a kernel starts.)
constexpr int L1_SECTOR = 32;
static_assert(DICT_INLINE == L1_SECTOR, "an entry of the pool is one sector");
__device__ __forceinline__ u64 load_l1(const u64* p)
{
  u64 v;
  asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ ulonglong2 load_l1(const ulonglong2* p)
{
  ulonglong2 v;
  asm volatile("ld.global.ca.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

// id of the string [p, p + len) of row `row`, inserting it when new; -1 after an overflow
// (`w` = the string's first DICT_INLINE bytes, zero padded).  take(who, lead): an id for each of the lanes `who`, which claim
// together, the first of them `lead`, and what goes with it where it is below the pool's capacity; more_equal(id): whether what goes
// with it is this key's; noted(): an id was published; gave_up(probe): the attempt is over.
template <typename Take, typename MoreEqual, typename Noted, typename GaveUp>
__device__ __forceinline__ i64 dict_find_insert(const DPlan& P, const DDict& D, const u64 (&w)[4], i64 len, i64 row, u64 h, DCtrl* ctrl,
                                                Take&& take, MoreEqual&& more_equal, Noted&& noted, GaveUp&& gave_up)
{
  const u64 head = dict_head(h, len);
  i64 idx = (i64)(h & (u64)(D.cap - 1));  // (a power of two; the tag is the other end of the hash)
  for (int probe = 0; probe < GMEM_PROBES; ++probe) {
    u64* const cell = D.cells + idx;
    u64 k = load_l1(cell);
    if ((k & DICT_ID_MASK) == DICT_ID_MASK) k = *(volatile u64*)cell;  // (EMPTY among them)
    if (k == EMPTY) {
      // The cell is claimed first, under an id that is none; then one id is taken, the entry written, the id published.  (With
      // ids taken in front of the claim, the threads that met the same new string at the same time each took one: 1M rows over
      // 50K strings used up 230K ids, at 1 ns each for the one address.)  The lanes that claim together take their ids together.
      k = atomicCAS(cell, EMPTY, head | DICT_ID_MASK);
      if (k == EMPTY) {
        const u32 who = __activemask();
        const u64 id = take(who, __ffs(who) - 1);
        if (id >= (u64)D.pool_cap) { ctrl->overflow = 1; return -1; }  // (whoever waits for the cell sees the flag)
        u64* e = D.pool + id * 4;
        e[0] = w[0]; e[1] = w[1]; e[2] = w[2]; e[3] = w[3];
        D.first_row[id] = (int)row;
        __threadfence();
        *(volatile u64*)cell = head | id;
        noted();
        return (i64)id;
      }
    }
    if (((k ^ head) & ~DICT_ID_MASK) == 0) {  // same tag and (clamped) length
      for (int tries = 0; (k & DICT_ID_MASK) == DICT_ID_MASK; ++tries) {  // claimed, not published yet
        if (tries >= DICT_TRIES || *(volatile u32*)&ctrl->overflow) { ctrl->overflow = 1; return -1; }
        __nanosleep(40);
        k = *(volatile u64*)cell;
      }
      const u64 id = k & DICT_ID_MASK;
      const ulonglong2* e = (const ulonglong2*)(D.pool + id * 4);
      auto matches = [&](const ulonglong2& a, const ulonglong2& b) { return a.x == w[0] && a.y == w[1] && b.x == w[2] && b.y == w[3]; };
      const bool same_l1 = matches(load_l1(e), load_l1(e + 1));
      bool same = same_l1 || matches(__ldcg(e), __ldcg(e + 1));  // (a mismatch is rare enough to be sure of)
      if (same && len > DICT_INLINE) same = rows_equal(P, row, (i64)__ldcg(D.first_row + id));
      if (same) same = more_equal(id);
      if (same) return (i64)id;
    }
    if (gave_up(probe)) return -1;
    if (++idx == D.cap) idx = 0;
  }
  ctrl->overflow = 1;
  return -1;
}

// The first DICT_INLINE bytes of the string [p, p + len), zero padded: five aligned 8-byte words at most, none of them without a
// wanted byte, all in flight together.
__device__ __forceinline__ void dict_load(const unsigned char* p, i64 len, u64 (&w)[4])
{
  const int take = dict_kept(len);
  const u32 off = (u32)(u64)p & 7u, sh = 8u * off;
  const u64* a = (const u64*)(p - off);
  u64 x[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) x[i] = 8 * i < take + (int)off && take > 0 ? __ldg(a + i) : 0ull;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    u64 v = x[i] >> sh;
    if (sh) v |= x[i + 1] << (64u - sh);
    const int left = take - 8 * i;
    w[i] = left >= 8 ? v : left > 0 ? v & ((1ull << (8 * left)) - 1ull) : 0ull;
  }
}
// hash of up to four words (a multiplication and a fold per word) and a number
__device__ __forceinline__ u64 dict_hash(const u64 (&w)[4], int words, u64 more)
{
  u64 h = 0x243F6A8885A308D3ull ^ more;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i < words) { h = (h ^ w[i]) * 0x9E3779B97F4A7C15ull; h ^= h >> 32; }
  return mix64(h);
}

// `live_rows` (keys of fixed width): a bit per row, set where the row takes part
template <bool STRINGS>
__global__ void __launch_bounds__(DICT_BLOCK, DICT_CTAS) k_dict_encode(const __grid_constant__ DPlan P, const DDict D, const __grid_constant__ DDictKeys W, DCtrl* ctrl,
                                                            u32* __restrict__ ids, u32* __restrict__ live_rows)
{
  __shared__ int s_new;
  __shared__ u32 s_stop;
  if (threadIdx.x == 0) { s_new = 0; s_stop = 0; }
  __syncthreads();
  const DKeyCol& c = P.keys[0];
  constexpr i64 TILE = (i64)DICT_BLOCK * DICT_ROWS;
  for (i64 base = (i64)blockIdx.x * TILE; base < P.nrows; base += (i64)gridDim.x * TILE) {
    // (a warp leaves as one: its lanes part in the probes below and need not read the flag at the same time, and the ballot wants
    // them all)
    if (__any_sync(0xFFFFFFFFu, *(volatile u32*)&s_stop != 0u)) break;
    // hash and probe row by row; the next row's offsets are on their way meanwhile
    u32 live = 0;
#pragma unroll
    for (int j = 0; j < DICT_ROWS; ++j) {
      const i64 row = base + (i64)j * DICT_BLOCK + threadIdx.x;
      const bool in = row < P.nrows && (STRINGS ? !(c.mask && !bit_valid(c.mask, c.offset + row)) : row_active(P, row));
      if (in) live |= 1u << j;
      if (!STRINGS && live_rows) {
        const u32 word = __ballot_sync(0xFFFFFFFFu, in);
        if ((threadIdx.x & 31) == 0 && row < P.nrows) live_rows[row >> 5] = word;
      }
    }
    i64 begin = 0;
    int next_bytes = 0;
    auto offsets = [&](int j) {
      const i64 at = c.offset + base + (i64)j * DICT_BLOCK + threadIdx.x;
      if (STRINGS && j < DICT_ROWS && ((live >> j) & 1u)) { begin = str_offset(c, at); next_bytes = dict_length(str_offset(c, at + 1) - begin); }
    };
    offsets(0);
#pragma unroll 1
    for (int j = 0; j < DICT_ROWS; ++j) {
      const i64 row = base + (i64)j * DICT_BLOCK + threadIdx.x;
      if (row >= P.nrows) continue;
      const unsigned char* p = c.data + begin;
      const int bytes = next_bytes;
      offsets(j + 1);
      u32 id = 0;
      if ((live >> j) & 1u) {
        u64 w[4] = {0, 0, 0, 0};
        u64 h;
        i64 n;
        if (STRINGS) {
          // (every lane takes the same four steps whatever its string's length; longer strings hash their rest)
          n = bytes;
          dict_load(p, n, w);
          h = dict_hash(w, 4, (u64)n << 56);
          if (n > DICT_INLINE) h = hash_bytes(p + DICT_INLINE, n - DICT_INLINE, h);
        } else {
          for (int i = 0; i < P.nkeys; ++i) {
            const DKeyCol& kc = P.keys[i];
            const int null_at = W.null_at[i];
            u64 x;
            int bit;
            if (null_at != 255 && !bit_valid(kc.mask, kc.offset + row)) { x = 1; bit = null_at; }
            else { x = canonical_bits(kc, kc.offset + row); bit = 8 * (int)W.at[i]; }
#pragma unroll
            for (int q = 0; q < 4; ++q) if ((bit >> 6) == q) w[q] |= x << (bit & 63);
          }
          n = 8 * W.words;
          h = dict_hash(w, W.words, 0);
        }
        const i64 s = dict_find_insert(P, D, w, n, row, h, ctrl,
          [&](u32 who, int lead) -> u64 {
            const u32 lane = threadIdx.x & 31u;
            u64 first = 0;
            if ((int)lane == lead) first = atomicAdd(&ctrl->out_cursor, (u64)__popc(who));
            return __shfl_sync(who, first, lead) + __popc(who & ((1u << lane) - 1u));
          },
          [](u64) { return true; }, [&] { atomicAdd(&s_new, 1); }, [&](int probe) { return probe_gave_up(probe, ctrl, &s_new); });
        if (s >= 0) id = (u32)s;
      }
      ids[(STRINGS ? c.offset : 0) + row] = id;
    }
    if (threadIdx.x == 0) {  // (no barrier: the others see the flag a tile later)
      const int n = atomicExch(&s_new, 0);
      if (n) {
        const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)n) + (u64)n;
        if (tot > ctrl->claim_limit) ctrl->overflow = 1;
      }
      if (*(volatile u32*)&ctrl->overflow) *(volatile u32*)&s_stop = 1;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) {
    const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)s_new) + (u64)s_new;
    if (tot > ctrl->claim_limit) ctrl->overflow = 1;
  }
}

// ids of the finished groups -> the first rows that held their strings (-1 for a null key)
__global__ void k_dict_rows(const u32* __restrict__ ids, const u32* __restrict__ id_mask, const int* __restrict__ first_row,
                            i64 ngroups, int* __restrict__ rows)
{
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x)
    rows[g] = (id_mask && !bit_valid(id_mask, g)) ? -1 : first_row[ids[g]];
}

// ------------------------------------------------------------------------------ dictionary values
// DICTIONARY32 value columns (cpp/include/cudf/detail/aggregation/device_aggregators.cuh:189-220: the reference
// looks the key up at every update): values[i] = keys[indices[i]] written out once, so that the aggregate passes
// see a plain column of the keys' type.  Null rows (their index may be anything) are written as zero.
struct DDictDecode {
  const unsigned char* indices; int index_width; int index_signed; i64 index_offset;  // element offset of row 0
  const unsigned char* keys; i64 keys_offset; i64 nkeys; int width;
  const u32* mask; i64 mask_offset;  // the dictionary column's validity (nullptr = all valid)
  unsigned char* dst;                // element 0 of the decoded rows
};
__global__ void __launch_bounds__(256) k_dict_decode(const DDictDecode D, i64 n)
{
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    u64 v = 0;
    if (!D.mask || bit_valid(D.mask, D.mask_offset + i)) {
      const u64 raw = load_fixed_bits(D.indices, D.index_offset + i, D.index_width);
      const int sh  = 64 - 8 * D.index_width;
      const i64 idx = D.index_signed ? ((i64)(raw << sh) >> sh) : (i64)raw;
      if (idx >= 0 && idx < D.nkeys) v = load_fixed_bits(D.keys, D.keys_offset + idx, D.width);
    }
    switch (D.width) {
      case 1: D.dst[i] = (unsigned char)v; break;
      case 2: ((unsigned short*)D.dst)[i] = (unsigned short)v; break;
      case 4: ((u32*)D.dst)[i] = (u32)v; break;
      default: ((u64*)D.dst)[i] = v; break;
    }
  }
}

__global__ void __launch_bounds__(256) k_iota(int* __restrict__ p, i64 n)
{
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) p[i] = (int)i;
}

// ------------------------------------------------------------------------------ finalize
enum OutKind : int {
  OK_COUNT = 0,  // int32 from a count cell
  OK_INT,        // integer cell (Σ, Σx², Π, min, max of integers) stored in the result width
  OK_FLT,        // double cell (Σ, Σx², Π of floats) stored as FLOAT32/FLOAT64
  OK_MINMAX_F,   // ordered-encoded double cell
  OK_MEAN, OK_M2, OK_VAR, OK_STD,
  OK_ARG,        // ARGMIN / ARGMAX: the row held by the cell as INT32, null when none
  OK_STRARG,     // MIN / MAX of strings: the row (or -1) into a scratch array the host gathers the strings by
  OK_SUMOVF,     // SUM_OVERFLOW: the sum in the source type into `data`, "the exact sum does not fit it" into `data2`
  OK_SUM128      // SUM of DECIMAL128: 16-byte elements from the four exact-sum cells c_a .. c_a + 3
};

struct DOutCol {
  void* data;
  void* data2;    // OK_SUMOVF: the BOOL8 overflow child
  u32* mask;      // nullptr = result not nullable
  int kind;       // OutKind
  int rclass;     // ValClass of the result element type
  int c_a;        // primary cell (Σx for MEAN/M2/VAR/STD)
  int c_b;        // Σx² for M2/VAR/STD
  int c_cnt;      // count cell deciding validity, -1 = always valid
  int ddof;
  int src_float;  // the Σ cells hold doubles
  int null_slot;  // index into null_counts
};

constexpr int MAX_OUTS = 64;

struct DOutPlan {
  int nouts;
  int pad;
  DOutCol outs[MAX_OUTS];
  void* kdata[MAX_KEYS];   // packed mode: decoded key columns
  u32* kmask[MAX_KEYS];
  int* rep_rows;           // row-key mode: representative row per group (nullptr: they are there already)
  u32* null_counts;        // [MAX_OUTS + MAX_KEYS]
  i64 max_groups;          // > 0: the output columns hold this many rows; groups beyond them are not written
                           // (the host compares the cursor with it afterwards)
};

__device__ __forceinline__ void store_int(void* data, i64 g, int rclass, u64 v)
{
  switch (rclass) {
    case VC_I8: case VC_U8: case VC_BOOL: ((unsigned char*)data)[g] = (unsigned char)v; break;
    case VC_I16: case VC_U16: ((unsigned short*)data)[g] = (unsigned short)v; break;
    case VC_I32: case VC_U32: ((u32*)data)[g] = (u32)v; break;
    default: ((u64*)data)[g] = v; break;
  }
}
__device__ __forceinline__ void store_flt(void* data, i64 g, int rclass, double v)
{
  if (rclass == VC_F32) ((float*)data)[g] = (float)v;
  else ((double*)data)[g] = v;
}
__device__ __forceinline__ void clear_bit(u32* mask, i64 g, u32* counter)
{
  atomicAnd(mask + (g >> 5), ~(1u << (g & 31)));
  atomicAdd(counter, 1u);
}

// The sum of a DECIMAL128 column from its four exact cells {Σ(lo & 0xFFFFFFFF), Σ(lo >> 32), Σ(hi & 0xFFFFFFFF),
// Σ(hi >> 32, signed)} (each exact below 2^31 rows): the low and high words of the sum
// modulo 2^128, and whether the exact sum leaves the 128-bit range.
__device__ __forceinline__ bool sum128(u64 c0, u64 c1, u64 c2, u64 c3, u64& lo, u64& hi)
{
  const unsigned __int128 a = (unsigned __int128)c0 + ((unsigned __int128)c1 << 32);                  // < 2^96
  const __int128 b = (__int128)c2 + (__int128)(i64)c3 * ((__int128)1 << 32) + (__int128)(u64)(a >> 64);
  lo = (u64)a;
  hi = (u64)b;
  return b < -((__int128)1 << 63) || b > (((__int128)1 << 63) - 1);
}

// One finished group -> output row g: key columns decoded from the key cell (packed keys) or the
// representative row noted (row keys), then every requested aggregation from the accumulator cells
// (`cell(c)`): COUNT as INT32, MEAN = Σx / n, M2 = Σx² − (Σx)²/n, VAR = M2 / (n − ddof),
// STD = sqrt(VAR); results without a valid input are nulled and counted.
template <typename Cells>
__device__ __forceinline__ void write_group(const DPlan& P, const DOutPlan& O, u64 key, const Cells& cell, i64 g,
                                            u32* null_counts)
{
  if (P.key_mode == KM_PACKED) {
    for (int k = 0; k < P.nkeys; ++k) {
      const DKeyCol& c = P.keys[k];
      if (c.nullbit >= 0 && ((key >> c.nullbit) & 1ull)) {
        clear_bit(O.kmask[k], g, null_counts + MAX_OUTS + k);
        store_int(O.kdata[k], g, c.width == 1 ? VC_U8 : c.width == 2 ? VC_U16 : c.width == 4 ? VC_U32 : VC_U64, 0);
      } else {
        const u64 v = (c.width == 8) ? (key >> c.shift) : ((key >> c.shift) & ((1ull << (8 * c.width)) - 1ull));
        store_int(O.kdata[k], g, c.width == 1 ? VC_U8 : c.width == 2 ? VC_U16 : c.width == 4 ? VC_U32 : VC_U64, v);
      }
    }
  } else if (O.rep_rows) {
    O.rep_rows[g] = (int)(u32)key;
  }
  for (int o = 0; o < O.nouts; ++o) {
    const DOutCol& oc = O.outs[o];
    const i64 n = oc.c_cnt >= 0 ? (i64)cell(oc.c_cnt) : 1;
    bool valid  = n > 0;
    switch (oc.kind) {
      case OK_COUNT: ((int*)oc.data)[g] = (int)cell(oc.c_a); valid = true; break;
      case OK_INT: store_int(oc.data, g, oc.rclass, valid ? cell(oc.c_a) : 0); break;
      case OK_FLT: store_flt(oc.data, g, oc.rclass, valid ? __longlong_as_double((i64)cell(oc.c_a)) : 0.0); break;
      case OK_MINMAX_F:
        store_flt(oc.data, g, oc.rclass, valid ? __longlong_as_double((i64)f64_unordered(cell(oc.c_a))) : 0.0);
        break;
      case OK_ARG: case OK_STRARG: {
        const u64 r = cell(oc.c_a);
        valid = r != ARG_NONE;
        ((int*)oc.data)[g] = valid ? (int)r : (oc.kind == OK_ARG ? 0 : -1);
        break;
      }
      case OK_SUMOVF: {
        // The exact sum is Σ(v >> 32) · 2^32 + Σ(v & 0xFFFFFFFF) for a 64-bit source (cells c_a, c_b), the one
        // int64 cell otherwise.  The reference raises the flag when an add wraps in the source type
        // (cpp/include/cudf/detail/aggregation/device_aggregators.cuh:136-160), which depends on the order the
        // rows arrive in; "the exact sum does not fit" is what every order gives when a group's values share a
        // sign, and what the order that alternates signs gives otherwise.
        bool ovf = false;
        u64 sum  = 0;
        if (oc.rclass == VC_U64X2) {  // DECIMAL128
          u64 lo = 0, hi = 0;
          if (valid) ovf = sum128(cell(oc.c_a), cell(oc.c_a + 1), cell(oc.c_a + 2), cell(oc.c_a + 3), lo, hi);
          ((u64*)oc.data)[2 * g] = lo;
          ((u64*)oc.data)[2 * g + 1] = hi;
          ((unsigned char*)oc.data2)[g] = ovf ? 1 : 0;
          break;
        }
        if (valid) {
          if (oc.c_b >= 0) {
            const u64 lo = cell(oc.c_b);
            const i64 t  = (i64)cell(oc.c_a) + (i64)(lo >> 32);
            ovf = t < -2147483648ll || t > 2147483647ll;
            sum = ((u64)t << 32) | (lo & 0xFFFFFFFFull);
          } else {
            const i64 v    = (i64)cell(oc.c_a);
            const int bits = oc.rclass == VC_I8 ? 8 : oc.rclass == VC_I16 ? 16 : 32;
            ovf = v < -(1ll << (bits - 1)) || v > (1ll << (bits - 1)) - 1;
            sum = (u64)v;
          }
        }
        store_int(oc.data, g, oc.rclass, sum);
        ((unsigned char*)oc.data2)[g] = ovf ? 1 : 0;
        break;
      }
      case OK_SUM128: {
        u64 lo = 0, hi = 0;
        if (valid) sum128(cell(oc.c_a), cell(oc.c_a + 1), cell(oc.c_a + 2), cell(oc.c_a + 3), lo, hi);
        ((u64*)oc.data)[2 * g] = lo;
        ((u64*)oc.data)[2 * g + 1] = hi;
        break;
      }
      case OK_MEAN: {
        if (oc.rclass != VC_F64) {  // durations: integer division in the source type
          store_int(oc.data, g, oc.rclass, valid ? (u64)((i64)cell(oc.c_a) / n) : 0);
          break;
        }
        const double s = oc.src_float ? __longlong_as_double((i64)cell(oc.c_a)) : (double)(i64)cell(oc.c_a);
        ((double*)oc.data)[g] = valid ? s / (double)n : 0.0;
        break;
      }
      default: {  // M2, VAR, STD
        double m2 = 0.0;
        if (n > 0) {
          const double s  = oc.src_float ? __longlong_as_double((i64)cell(oc.c_a)) : (double)(i64)cell(oc.c_a);
          const double ss = oc.src_float ? __longlong_as_double((i64)cell(oc.c_b)) : (double)(i64)cell(oc.c_b);
          m2 = ss - s * s / (double)n;
        }
        if (oc.kind == OK_M2) { ((double*)oc.data)[g] = m2; valid = true; break; }
        const i64 df = n - oc.ddof;
        valid        = n > 0 && df > 0;
        const double var = valid ? m2 / (double)df : 0.0;
        ((double*)oc.data)[g] = (oc.kind == OK_VAR) ? var : sqrt(var);
        break;
      }
    }
    if (!valid && oc.mask) clear_bit(oc.mask, g, null_counts + oc.null_slot);
  }
}

constexpr int FIN_BLOCK = 256;
constexpr int FIN_ITEMS = 8;  // slots per thread per chunk (1 for small tables, which otherwise fill few SMs)

// Occupied slots are compacted chunk by chunk: a CTA counts the occupied slots of its chunk
// (FIN_BLOCK x FIN_ITEMS slots), reserves that many output rows with ONE atomic on the cursor, and its
// threads write their groups at the reserved positions.  (One reservation per warp and 32 slots made
// the single cursor the bottleneck of large tables: 6M atomics on one address for 200M slots.)
template <int ITEMS>
__global__ void __launch_bounds__(FIN_BLOCK) k_finalize(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O,
                                                        const u64* __restrict__ tbl, i64 cap, DCtrl* ctrl, const DReport report)
{
  __shared__ u32 s_wcount[FIN_BLOCK / 32];
  __shared__ u32 s_ballot[FIN_BLOCK / 32][ITEMS];
  __shared__ u64 s_base;
  const int stride = P.stride;
  const i64 dense  = (i64)ctrl->dense_slots;
  const i64 nslots = cap + 1 + dense;
  const bool by_count = (P.flags & PF_VEXP) != 0;  // k_aggregate_lean: a group of the dense region may be known by its n only
  const i64 chunk  = (i64)FIN_BLOCK * ITEMS;
  const i64 nchunks = (nslots + chunk - 1) / chunk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (i64 ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    u32 wtotal = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const i64 s = ch * chunk + (i64)j * FIN_BLOCK + threadIdx.x;
      bool occ = false;
      if (s < nslots && s != cap) {
        const SlotRef ref = slot_ref(const_cast<u64*>(tbl), cap, stride, dense, s);
        occ = *ref.key != EMPTY || (by_count && s > cap && ref.cells[ref.step] != 0ull);
      } else if (s == cap) occ = ctrl->special_used != 0;
      const u32 m = __ballot_sync(0xFFFFFFFFu, occ);
      if (lane == 0) s_ballot[wid][j] = m;
      wtotal += __popc(m);
    }
    if (lane == 0) s_wcount[wid] = wtotal;
    __syncthreads();
    if (threadIdx.x == 0) {
      u32 tot = 0;
      for (int w = 0; w < FIN_BLOCK / 32; ++w) { const u32 c = s_wcount[w]; s_wcount[w] = tot; tot += c; }
      s_base = tot ? atomicAdd(&ctrl->out_cursor, (u64)tot) : 0ull;
    }
    __syncthreads();
    u64 next = s_base + s_wcount[wid];  // first output row of this warp's groups
#pragma unroll 1
    for (int j = 0; j < ITEMS; ++j) {
      const u32 m = s_ballot[wid][j];
      const i64 g = (i64)next + __popc(m & ((1u << lane) - 1u));
      next += __popc(m);
      if (!((m >> lane) & 1u)) continue;
      if (O.max_groups > 0 && g >= O.max_groups) continue;
      const i64 s = ch * chunk + (i64)j * FIN_BLOCK + threadIdx.x;
      const SlotRef ref = slot_ref(const_cast<u64*>(tbl), cap, stride, dense, s);
      u64 key = s == cap ? EMPTY : *ref.key;
      if (key == EMPTY && s > cap) key = dense_key(P, ctrl->dense, (u32)(s - cap - 1));
      write_group(P, O, key, [&](int c) { return ref.cells[(i64)c * ref.step]; }, g, O.null_counts);
    }
    __syncthreads();  // the shared arrays are rewritten by the next chunk
  }
  report_ctrl(ctrl, report);
}

// ------------------------------------------------------------------------------ small inputs
// A whole aggregate call in one CTA: table in shared memory (`S` slots, at least a third of them free whatever the
// keys), rows, compaction, results.  With few rows the call costs what its launches and their latencies cost: through
// k_table_init, k_aggregate and k_finalize 1000 rows took 23 us on the device and a memset per nullable column; this
// takes one launch and writes what the host has to learn into its memory.
constexpr int SMALL_BLOCK = 1024;
struct DSmallResult {  // in pinned host memory
  u32 groups;
  u32 null_counts[MAX_OUTS + MAX_KEYS];
};
// `compensate`: Σ of FLOAT64 is kept as two doubles, what each addition rounds off (known from the value that the atomic
// returns) in the second.  For Σ and n of one FLOAT64 column from SAMPLE_ROWS rows on, which the lean kernel would add up
// exactly (4095 rows of 0.1 in one group: 6e-14 relative with one double; 4096 rows take 3 us longer).
// (Without the 1 the compiler keeps to 32 registers and spills: 2730 rows over FLOAT64 keys 112 us instead of 106.)
template <int KM>
__global__ void __launch_bounds__(SMALL_BLOCK, 1) k_small(const __grid_constant__ DPlan P, const __grid_constant__ DOutPlan O, int S,
                                                       int compensate, DSmallResult* result, const DReport report)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ u32 s_nulls[MAX_OUTS + MAX_KEYS], s_warp[SMALL_BLOCK / 32], s_base;
  u64* skeys  = (u64*)smem_raw;    // [S + 1]
  u64* scells = skeys + S + 1;     // [ncells][S + 1]
  double* slow = (double*)(scells + (size_t)P.ncells * (S + 1));  // [S + 1] if `compensate`: the low parts of Σ
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, NS = S + 1;
  for (int i = tid; i < NS; i += blockDim.x) skeys[i] = EMPTY;
  for (int c = 0; c < P.ncells; ++c) {
    const u64 id = cell_identity(P.cells[c].op);
    for (int i = tid; i < NS; i += blockDim.x) scells[(size_t)c * NS + i] = id;
  }
  if (compensate) for (int i = tid; i < NS; i += blockDim.x) slow[i] = 0.0;
  if (tid < MAX_OUTS + MAX_KEYS) s_nulls[tid] = 0;
  if (tid == 0) s_base = 0;
  // result masks start all valid
  const int words = (int)((P.nrows + 511) / 512) * 16;  // (64-byte padded)
  for (int o = 0; o < O.nouts; ++o)
    if (O.outs[o].mask) for (int i = tid; i < words; i += blockDim.x) O.outs[o].mask[i] = 0xFFFFFFFFu;
  for (int k = 0; k < P.nkeys; ++k)
    if (O.kmask[k]) for (int i = tid; i < words; i += blockDim.x) O.kmask[k][i] = 0xFFFFFFFFu;
  __syncthreads();
  for (i64 row = tid; row < P.nrows; row += blockDim.x) {
    if (!row_active(P, row)) continue;
    const u64 key = KM == KM_PACKED ? pack_key(P, row) : hash_row(P, row);
    const u64 h   = KM == KM_PACKED ? mix64(key) : key;
    const u64 tag = h & 0xFFFFFFFF00000000ull, mine = KM == KM_PACKED ? key : (tag | (u64)(u32)row);
    int slot = S;
    if (KM == KM_PACKED && key == EMPTY) {
      skeys[S] = 0;  // (in use)
    } else {
      slot = (int)reduce32((u32)(h >> 11), (u32)S);
      for (;;) {  // ends: more slots than rows
        u64 k = *(volatile u64*)(skeys + slot);
        if (k == EMPTY) {
          k = atomicCAS(skeys + slot, EMPTY, mine);
          if (k == EMPTY) break;
        }
        if (KM == KM_PACKED ? k == key : ((k & 0xFFFFFFFF00000000ull) == tag && rows_equal(P, row, (i64)(u32)k))) break;
        if (++slot == S) slot = 0;
      }
    }
    int cur = -1;
    u64 v[1] = {0};
    u32 ok = 0;
    for (int c = 0; c < P.ncells; ++c) {
      const int op = P.cells[c].op, col = P.cells[c].col;
      if (op != OP_CNT_A && col != cur) {
        cur = col;
        ok = value_valid(P.vals[col], row) ? 1u : 0u;
        if (ok) v[0] = load_value(P.vals[col], row);
      }
      u64* const cell[1] = {scells + (size_t)c * NS + slot};
      if (is_arg_op(op)) { if (ok) arg_update(cell[0], op, P.vals[col], row); }
      else if (compensate && op == OP_SUM_F) {
        if (ok) {
          const double x = __longlong_as_double((i64)v[0]), old = atomicAdd((double*)cell[0], x);
          const double sum = __dadd_rn(old, x), part = __dsub_rn(sum, old);
          const double lost = __dadd_rn(__dsub_rn(old, __dsub_rn(sum, part)), __dsub_rn(x, part));
          if (lost != 0.0 && isfinite(sum)) atomicAdd(slow + slot, lost);
        }
      } else cell_update_shared<1>(cell, op, v, op == OP_CNT_A ? 1u : ok);
    }
  }
  __syncthreads();
  // occupied slots -> consecutive result rows
  for (int i0 = 0; i0 < NS; i0 += blockDim.x) {
    const int i = i0 + tid;
    const u64 key = i < NS ? skeys[i] : EMPTY;
    const u32 m = __ballot_sync(0xFFFFFFFFu, key != EMPTY);
    if (lane == 0) s_warp[wid] = __popc(m);
    __syncthreads();
    if (wid == 0) {
      const u32 c = s_warp[lane];
      u32 x = c;
      for (int d = 1; d < 32; d <<= 1) { const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, d); if (lane >= d) x += y; }
      const u32 base = s_base;
      s_warp[lane] = base + x - c;
      __syncwarp();
      if (lane == 31) s_base = base + x;
    }
    __syncthreads();
    if (compensate && key != EMPTY)
      for (int c = 0; c < P.ncells; ++c)
        if (P.cells[c].op == OP_SUM_F) *(double*)(scells + (size_t)c * NS + i) += slow[i];
    if (key != EMPTY)
      write_group(P, O, i == S ? EMPTY : key, [&](int c) { return scells[(size_t)c * NS + i]; }, (i64)(s_warp[wid] + __popc(m & ((1u << lane) - 1u))), s_nulls);
    __syncthreads();
  }
  if (tid == 0) result->groups = s_base;
  if (tid < MAX_OUTS + MAX_KEYS) result->null_counts[tid] = s_nulls[tid];
  __syncthreads();  // (the only CTA)
  if (tid == 0) {
    __threadfence_system();
    *(volatile u64*)report.flag = report.number;
  }
}

// all-valid masks of several result columns at once
struct DFillMasks { int n; u32* mask[MAX_OUTS + MAX_KEYS]; int words[MAX_OUTS + MAX_KEYS]; };
__global__ void __launch_bounds__(256) k_fill_masks(const __grid_constant__ DFillMasks F)
{
  u32* m = F.mask[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < F.words[blockIdx.y]; i += gridDim.x * blockDim.x) m[i] = 0xFFFFFFFFu;
}

// ------------------------------------------------------------------------------ finishers over partial columns
// Partial aggregates that travel as columns (string / float / wide keys between ranks and batches: Σx, n, Σx²
// per group) are finished here: mean, M2, variance, standard deviation, counts as INT32 — the formulas of
// write_group (cpp/src/groupby/hash/hash_compound_agg_finalizer.cu:93-186, common/m2_var_std.cu:57) — and the
// validity of a result from n.
struct DFinish {
  int kind;        // FK_* below
  int ddof;
  int rclass;      // ValClass of the result
  int int_mean;    // mean by integer division in the source type (durations)
  DValCol sum, cnt, ssq;
  void* out;
  u32* out_mask;   // nullptr = not nullable
  u32* null_count;
};
enum FinishKind : int { FK_COUNT = 0, FK_MEAN, FK_M2, FK_VAR, FK_STD, FK_VALID_ONLY };

__device__ __forceinline__ double carried_as_double(const DValCol& c, u64 v)
{
  if (c.vclass == VC_F32 || c.vclass == VC_F64) return __longlong_as_double((i64)v);
  if (c.vclass == VC_U64) return (double)v;
  return (double)(i64)v;
}

__global__ void k_finish_partial(const DFinish F, i64 n)
{
  const u32 lane = threadIdx.x & 31u;
  const i64 nround = (n + 31) / 32 * 32;
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < nround; g += (i64)gridDim.x * blockDim.x) {
    bool valid = false;
    if (g < n) {
      const i64 c = (i64)load_value(F.cnt, g);
      valid = c > 0;
      switch (F.kind) {
        case FK_COUNT: store_int(F.out, g, F.rclass, (u64)c); valid = true; break;
        case FK_MEAN: {
          const u64 sv = load_value(F.sum, g);
          if (F.int_mean) store_int(F.out, g, F.rclass, (u64)((i64)sv / (c > 0 ? c : 1)));
          else store_flt(F.out, g, F.rclass, carried_as_double(F.sum, sv) / (double)(c > 0 ? c : 1));
          break;
        }
        case FK_M2: case FK_VAR: case FK_STD: {
          const double s = carried_as_double(F.sum, load_value(F.sum, g)), ss = carried_as_double(F.ssq, load_value(F.ssq, g));
          const double m2 = c > 0 ? ss - s * s / (double)c : 0.0;
          if (F.kind == FK_M2) { store_flt(F.out, g, F.rclass, m2); valid = true; break; }
          const i64 df = c - F.ddof;
          valid = c > 0 && df > 0;
          const double var = valid ? m2 / (double)df : 0.0;
          store_flt(F.out, g, F.rclass, F.kind == FK_VAR ? var : sqrt(var));
          break;
        }
        default: break;  // FK_VALID_ONLY: the mask alone
      }
    }
    if (F.out_mask) {
      const u32 word = __ballot_sync(0xFFFFFFFFu, valid);
      if (lane == 0) {
        F.out_mask[g >> 5] = word;
        const i64 here = n - g < 32 ? n - g : 32;  // rows of this word
        const u32 nulls = (u32)here - (u32)__popc(word);
        if (nulls && F.null_count) atomicAdd(F.null_count, nulls);
      }
    }
  }
}

// ------------------------------------------------------------------------------ key gather (row keys)
struct DGather {
  const unsigned char* src; const u32* src_mask; i64 src_offset; int width;
  unsigned char* dst; u32* dst_mask; u32* null_counter;
};

__global__ void k_gather_fixed(DGather G, const int* __restrict__ rows, i64 ngroups)
{
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x) {
    const i64 idx = G.src_offset + rows[g];
    if (G.src_mask && !bit_valid(G.src_mask, idx)) {
      if (G.dst_mask) clear_bit(G.dst_mask, g, G.null_counter);
      for (int b = 0; b < G.width; ++b) G.dst[g * G.width + b] = 0;
    } else {
      for (int b = 0; b < G.width; ++b) G.dst[g * G.width + b] = G.src[idx * G.width + b];
    }
  }
}

// string lengths of the representative rows (0 for a null), then offsets by scan, then the bytes
__global__ void k_string_lengths(DKeyCol c, const int* __restrict__ rows, i64 ngroups, i64* __restrict__ lens,
                                 u32* dst_mask, u32* null_counter)
{
  for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += (i64)gridDim.x * blockDim.x) {
    const i64 idx = c.offset + rows[g];
    i64 len = 0;
    if (rows[g] < 0) {
      // no row (a string MIN / MAX of a group without a valid value: nulled by the finisher already)
    } else if (c.mask && !bit_valid(c.mask, idx)) {
      if (dst_mask) clear_bit(dst_mask, g, null_counter);
    } else {
      len = str_offset(c, idx + 1) - str_offset(c, idx);
    }
    lens[g] = len;
  }
}

// single-CTA exclusive scan over n int64 (n = number of groups; one pass, 1024 threads)
__global__ void __launch_bounds__(1024) k_exclusive_scan(const i64* __restrict__ in, i64* __restrict__ out, i64 n)
{
  __shared__ i64 s_warp[32];
  __shared__ i64 s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (i64 base = 0; base < n; base += blockDim.x) {
    const i64 i = base + threadIdx.x;
    const i64 x = i < n ? in[i] : 0;
    i64 v = x;
    for (int d = 1; d < 32; d <<= 1) { const i64 t = __shfl_up_sync(0xFFFFFFFFu, v, d); if (lane >= d) v += t; }
    if (lane == 31) s_warp[wid] = v;
    __syncthreads();
    if (wid == 0) {
      i64 wv = s_warp[lane];
      for (int d = 1; d < 32; d <<= 1) { const i64 t = __shfl_up_sync(0xFFFFFFFFu, wv, d); if (lane >= d) wv += t; }
      s_warp[lane] = wv;
    }
    __syncthreads();
    const i64 prefix = s_carry + (wid ? s_warp[wid - 1] : 0) + (v - x);
    if (i < n) out[i] = prefix;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry += s_warp[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = s_carry;
}

// exclusive scan of many elements in three steps: per-block totals, scan of the totals (one CTA),
// per-block scan with the block's base added
constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 4;  // elements per thread
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_block_totals(const i64* __restrict__ in, i64 n, i64* __restrict__ totals)
{
  __shared__ i64 s_warp[32];
  const i64 base = (i64)blockIdx.x * SCAN_BLOCK * SCAN_ITEMS;
  i64 v = 0;
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    const i64 i = base + (i64)threadIdx.x * SCAN_ITEMS + j;
    if (i < n) v += in[i];
  }
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    i64 w = s_warp[threadIdx.x];
    for (int d = 16; d > 0; d >>= 1) w += __shfl_xor_sync(0xFFFFFFFFu, w, d);
    if (threadIdx.x == 0) totals[blockIdx.x] = w;
  }
}
__global__ void __launch_bounds__(SCAN_BLOCK)
k_scan_apply(const i64* __restrict__ in, i64 n, const i64* __restrict__ block_bases, i64* __restrict__ out)
{
  __shared__ i64 s_warp[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i64 base = (i64)blockIdx.x * SCAN_BLOCK * SCAN_ITEMS;
  i64 x[SCAN_ITEMS], mine = 0;
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    const i64 i = base + (i64)threadIdx.x * SCAN_ITEMS + j;
    x[j] = i < n ? in[i] : 0;
    mine += x[j];
  }
  i64 v = mine;
  for (int d = 1; d < 32; d <<= 1) { const i64 t = __shfl_up_sync(0xFFFFFFFFu, v, d); if (lane >= d) v += t; }
  if (lane == 31) s_warp[wid] = v;
  __syncthreads();
  if (wid == 0) {
    i64 w = s_warp[lane];
    for (int d = 1; d < 32; d <<= 1) { const i64 t = __shfl_up_sync(0xFFFFFFFFu, w, d); if (lane >= d) w += t; }
    s_warp[lane] = w;
  }
  __syncthreads();
  i64 run = block_bases[blockIdx.x] + (wid ? s_warp[wid - 1] : 0) + (v - mine);
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    const i64 i = base + (i64)threadIdx.x * SCAN_ITEMS + j;
    if (i < n) out[i] = run;
    run += x[j];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == SCAN_BLOCK - 1) out[n] = run;
}

template <typename OffT>
__global__ void k_string_copy(DKeyCol c, const int* __restrict__ rows, i64 ngroups, const i64* __restrict__ offs,
                              OffT* __restrict__ out_offs, unsigned char* __restrict__ chars)
{
  // four lanes per string, 8 bytes per lane and step (key strings are short: a warp per string left most of
  // its lanes idle); the source is read as aligned words, the destination written byte by byte
  const int sub = threadIdx.x & 3;
  const i64 s0 = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  const i64 ns = ((i64)gridDim.x * blockDim.x) >> 2;
  for (i64 g = s0; g <= ngroups; g += ns) {
    if (sub == 0) out_offs[g] = (OffT)offs[g];
    if (g == ngroups) break;
    const i64 len = offs[g + 1] - offs[g];
    if (len == 0) continue;
    const i64 idx = c.offset + rows[g];
    const unsigned char* src = c.data + str_offset(c, idx);
    unsigned char* dst = chars + offs[g];
    for (i64 b = (i64)sub * 8; b < len; b += 32) {
      const int nb = (int)(len - b < 8 ? len - b : 8);
      u64 v = load_bytes8(src + b, nb);
      for (int i = 0; i < nb; ++i) { dst[b + i] = (unsigned char)v; v >>= 8; }
    }
  }
}

// ------------------------------------------------------------------------------ partial records
// owner partition of every occupied slot: counts, then scatter into destination-major order
// Lanes of a warp headed for the same destination add to its counter ONCE (with few destinations
// every lane of a CTA would otherwise hit the same two or eight shared-memory words).  Returns this
// lane's position among the destination's records as counted by `counter`, or nothing useful for
// lanes with `dest` = NO_DEST.  Must be called by all 32 lanes.
constexpr u32 NO_DEST = 0xFFFFFFFFu;
__device__ __forceinline__ u64 warp_add_by_dest(u64* counters, u32 dest)
{
  const u32 lane  = threadIdx.x & 31u;
  const u32 peers = __match_any_sync(0xFFFFFFFFu, dest);
  const int lead  = __ffs(peers) - 1;
  u64 base = 0;
  if (dest != NO_DEST && (int)lane == lead) base = atomicAdd(&counters[dest], (u64)__popc(peers));
  base = __shfl_sync(0xFFFFFFFFu, base, lead);
  return base + (u64)__popc(peers & ((1u << lane) - 1u));
}

__global__ void k_pack_count(const u64* __restrict__ tbl, i64 cap, int stride, int nparts, const DCtrl* ctrl,
                             u64* __restrict__ counts)
{
  extern __shared__ u64 s_cnt[];
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) s_cnt[p] = 0;
  __syncthreads();
  const i64 last = cap + (i64)ctrl->dense_slots;
  const u32 lane = threadIdx.x & 31u;
  for (i64 s0 = (i64)blockIdx.x * blockDim.x + (threadIdx.x - lane); s0 <= last; s0 += (i64)gridDim.x * blockDim.x) {
    const i64 s = s0 + lane;
    u32 dest = NO_DEST;
    if (s <= last) {
      const u64 key = s != cap ? *slot_ref(const_cast<u64*>(tbl), cap, stride, last - cap, s).key : EMPTY;
      const bool occ = s != cap ? key != EMPTY : ctrl->special_used != 0;
      if (occ) dest = owner_of(mix64(key), (u32)nparts);
    }
    warp_add_by_dest(s_cnt, dest);
  }
  __syncthreads();
  for (int p = threadIdx.x; p < nparts; p += blockDim.x)
    if (s_cnt[p]) atomicAdd(&counts[p], s_cnt[p]);
}

// Scatter of the occupied slots into destination-major order.  Each CTA owns a contiguous range of
// slots: it counts its records per destination in shared memory, reserves its output ranges with ONE
// global atomic per destination, then scatters with shared-memory cursors (one global atomic per
// record on a handful of addresses serialised: 3.5 ms for 5.4M records).
__global__ void __launch_bounds__(256)
k_pack_scatter(const u64* __restrict__ tbl, i64 cap, int stride, int nparts, const DCtrl* ctrl,
               u64* __restrict__ cursors /* start offsets, advanced */, u64* __restrict__ out)
{
  extern __shared__ u64 s_pack[];  // [nparts] counts, then [nparts] bases
  u64* s_cnt  = s_pack;
  u64* s_base = s_pack + nparts;
  const i64 last  = cap + (i64)ctrl->dense_slots;
  const i64 per   = (last + 1 + gridDim.x - 1) / gridDim.x;
  const i64 lo    = (i64)blockIdx.x * per;
  const i64 hi    = min(last + 1, lo + per);
  const u32 lane  = threadIdx.x & 31u;
  auto dest_of = [&](i64 s, u64& key) -> u32 {
    if (s >= hi) return NO_DEST;
    key = s != cap ? *slot_ref(const_cast<u64*>(tbl), cap, stride, last - cap, s).key : EMPTY;
    const bool occ = s != cap ? key != EMPTY : ctrl->special_used != 0;
    return occ ? owner_of(mix64(key), (u32)nparts) : NO_DEST;
  };
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) s_cnt[p] = 0;
  __syncthreads();
  for (i64 s0 = lo + (threadIdx.x - lane); s0 < hi; s0 += blockDim.x) {
    u64 key = 0;
    warp_add_by_dest(s_cnt, dest_of(s0 + lane, key));
  }
  __syncthreads();
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) {
    s_base[p] = s_cnt[p] ? atomicAdd(&cursors[p], s_cnt[p]) : 0;
    s_cnt[p]  = 0;
  }
  __syncthreads();
  for (i64 s0 = lo + (threadIdx.x - lane); s0 < hi; s0 += blockDim.x) {
    const i64 s = s0 + lane;
    u64 key = 0;
    const u32 p = dest_of(s, key);
    const u64 r = warp_add_by_dest(s_cnt, p);
    if (p == NO_DEST) continue;
    const u64 pos = s_base[p] + r;
    u64* dst = out + pos * stride;
    const SlotRef src = slot_ref(const_cast<u64*>(tbl), cap, stride, last - cap, s);
    dst[0] = key;
    for (int c = 1; c < stride; ++c) dst[c] = src.cells[(i64)(c - 1) * src.step];
  }
}

// The same for a state that holds its groups as a list (structure-of-arrays: word w of group g at
// groups[w * gcap + g]) — what the partitioned path leaves: CTA-contiguous ranges of the list, one global
// reservation per destination and CTA, records written in destination-major order.
__global__ void __launch_bounds__(256)
k_pack_list(const u64* __restrict__ groups, i64 gcap, i64 ngroups, int stride, int nparts, u64* __restrict__ cursors,
            u64* __restrict__ out /* nullptr: only count into `cursors` */)
{
  extern __shared__ u64 s_pack[];  // [nparts] counts, then [nparts] bases
  u64* s_cnt  = s_pack;
  u64* s_base = s_pack + nparts;
  const i64 per  = (ngroups + gridDim.x - 1) / gridDim.x;
  const i64 lo   = (i64)blockIdx.x * per;
  const i64 hi   = min(ngroups, lo + per);
  const u32 lane = threadIdx.x & 31u;
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) s_cnt[p] = 0;
  __syncthreads();
  for (i64 g0 = lo + (threadIdx.x - lane); g0 < hi; g0 += blockDim.x) {
    const i64 g = g0 + lane;
    warp_add_by_dest(s_cnt, g < hi ? owner_of(mix64(groups[g]), (u32)nparts) : NO_DEST);
  }
  __syncthreads();
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) {
    s_base[p] = s_cnt[p] ? atomicAdd(&cursors[p], s_cnt[p]) : 0;
    s_cnt[p]  = 0;
  }
  if (!out) return;
  __syncthreads();
  for (i64 g0 = lo + (threadIdx.x - lane); g0 < hi; g0 += blockDim.x) {
    const i64 g = g0 + lane;
    const u64 key = g < hi ? groups[g] : 0;
    const u32 p = g < hi ? owner_of(mix64(key), (u32)nparts) : NO_DEST;
    const u64 r = warp_add_by_dest(s_cnt, p);
    if (p == NO_DEST) continue;
    u64* dst = out + (s_base[p] + r) * stride;
    dst[0] = key;
    for (int c = 1; c < stride; ++c) dst[c] = groups[(i64)c * gcap + g];
  }
}

// Slot of a packed key in a table that may hold a dense region (a table filled by the fused kernel in
// dense mode keeps the in-box keys there): in-box keys are addressed directly, the rest is hashed, so
// that a key never ends up in both regions.
__device__ __forceinline__ i64 table_slot_packed(const DPlan& P, u64* tbl, i64 cap, int stride, u64 key, DCtrl* ctrl,
                                                 int* s_new)
{
  if (ctrl->dense_slots != 0 && ctrl->dense.enabled && key != EMPTY) {
    const int di = dense_index(P, ctrl->dense, key);
    if (di >= 0) {
      const i64 g = cap + 1 + (i64)di;
      u64* kp = slot_ref(tbl, cap, stride, (i64)ctrl->dense_slots, g).key;
      if (*(volatile u64*)kp == EMPTY && atomicCAS(kp, EMPTY, key) == EMPTY) atomicAdd(s_new, 1);
      return g;
    }
  }
  return gmem_find_insert_packed(tbl, cap, stride, key, mix64(key), ctrl, s_new);
}

// fixed-size chunks: chunk d = { count, overflow, records[chunk_records] }.  One launch: every occupied
// slot takes the next position of its destination's chunk (records beyond the chunk's capacity are not
// written); the last CTA to finish writes the headers — the counts, or, when any destination
// overflowed, the overflow mark in EVERY chunk, so that every receiver learns of it.
// `cursors` ([nparts] counters + one ticket word) must arrive zeroed.
// A table that overflowed or that a kernel could not finish marks every chunk like an overflow (the control block need not
// have been read back; the receivers then make all ranks repeat the exchange with exact sizes, and this rank continues its
// aggregate first).  `lean_attempt`: so does a lean fused kernel that declined its input (no key box).
__global__ void __launch_bounds__(256)
k_pack_chunks(const u64* __restrict__ tbl, i64 cap, int stride, int nparts, const DCtrl* ctrl, u64* __restrict__ cursors,
              u64* __restrict__ out, i64 chunk_records, int lean_attempt)
{
  __shared__ int s_last;
  const i64 chunk_words = 2 + chunk_records * stride;
  const i64 last = cap + (i64)ctrl->dense_slots;
  const u32 lane = threadIdx.x & 31u;
  for (i64 s0 = (i64)blockIdx.x * blockDim.x + (threadIdx.x - lane); s0 <= last; s0 += (i64)gridDim.x * blockDim.x) {
    const i64 s = s0 + lane;
    u32 dest = NO_DEST;
    u64 key = 0;
    SlotRef src{nullptr, nullptr, 0};
    if (s <= last) {
      src = slot_ref(const_cast<u64*>(tbl), cap, stride, last - cap, s);
      key = s != cap ? *src.key : EMPTY;
      const bool occ = s != cap ? key != EMPTY : ctrl->special_used != 0;
      if (occ) dest = owner_of(mix64(key), (u32)nparts);
    }
    const u64 pos = warp_add_by_dest(cursors, dest);  // lanes of one destination reserve together
    if (dest == NO_DEST || pos >= (u64)chunk_records) continue;
    u64* dst = out + (i64)dest * chunk_words + 2 + (i64)pos * stride;
    dst[0] = key;
    for (int c = 1; c < stride; ++c) dst[c] = src.cells[(i64)(c - 1) * src.step];
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&cursors[nparts], 1ull) == (u64)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  __shared__ int s_over;
  if (threadIdx.x == 0) s_over = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < nparts; p += blockDim.x)
    if (__ldcg(&cursors[p]) > (u64)chunk_records) s_over = 1;
  __syncthreads();
  bool over = s_over != 0;
  if (ctrl->overflow != 0 || ctrl->error != 0) over = true;
  if (lean_attempt && (ctrl->dense.enabled == 0 || ctrl->dense.wide != 0)) over = true;  // (the kernel declined: there is nothing in the table)
  for (int p = threadIdx.x; p < nparts; p += blockDim.x) {
    out[(i64)p * chunk_words]     = over ? 0ull : __ldcg(&cursors[p]);
    out[(i64)p * chunk_words + 1] = over ? 1ull : 0ull;
  }
}

__global__ void __launch_bounds__(256)
k_merge_chunks(const __grid_constant__ DPlan P, u64* __restrict__ tbl, i64 cap, DCtrl* ctrl,
               const u64* __restrict__ chunks, int nchunks, i64 chunk_records)
{
  __shared__ int s_new;
  if (threadIdx.x == 0) s_new = 0;
  __syncthreads();
  const int stride = P.stride;
  const i64 chunk_words = 2 + chunk_records * stride;
  const i64 total = (i64)nchunks * chunk_records;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (i64)gridDim.x * blockDim.x) {
    const i64 c = i / chunk_records, r = i - c * chunk_records;
    const u64* chunk = chunks + c * chunk_words;
    if (r == 0 && chunk[1] != 0) atomicMax(&ctrl->chunk_overflow, chunk[1]);  // 1 = too many records, 2 = the sender failed
    if ((u64)r >= chunk[0] || chunk[1] != 0) continue;
    const u64* rec = chunk + 2 + r * stride;
    const u64 key  = rec[0];
    const i64 g    = table_slot_packed(P, tbl, cap, stride, key, ctrl, &s_new);
    if (g < 0) continue;
    const SlotRef slot = slot_ref(tbl, cap, stride, (i64)ctrl->dense_slots, g);
    for (int k = 0; k < P.ncells; ++k) {
      const int op = P.cells[k].op;
      const u64 a  = rec[1 + k];
      if (a != cell_identity(op)) cell_merge(slot.cells + (i64)k * slot.step, op, a);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) {
    const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)s_new) + (u64)s_new;
    if (tot > ctrl->claim_limit) ctrl->overflow = 1;
  }
}

// merge packed partial records into a table (packed keys)
__global__ void __launch_bounds__(256)
k_merge(const __grid_constant__ DPlan P, u64* __restrict__ tbl, i64 cap, DCtrl* ctrl, const u64* __restrict__ recs,
        i64 nrecs)
{
  __shared__ int s_new;
  if (threadIdx.x == 0) s_new = 0;
  __syncthreads();
  const int stride = P.stride;
  for (i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x; r < nrecs; r += (i64)gridDim.x * blockDim.x) {
    const u64* rec = recs + r * stride;
    const u64 key  = rec[0];
    const i64 g    = table_slot_packed(P, tbl, cap, stride, key, ctrl, &s_new);
    if (g < 0) continue;
    const SlotRef slot = slot_ref(tbl, cap, stride, (i64)ctrl->dense_slots, g);
    for (int c = 0; c < P.ncells; ++c) {
      const int op = P.cells[c].op;
      const u64 a  = rec[1 + c];
      if (a != cell_identity(op)) cell_merge(slot.cells + (i64)c * slot.step, op, a);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_new) {
    const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)s_new) + (u64)s_new;
    if (tot > ctrl->claim_limit) ctrl->overflow = 1;
  }
}


// ------------------------------------------------------------------------------ row hash partition
// cudf::hash_partition (cpp/src/partitioning/partitioning.cu:120-337,569-750): partition of a row =
// row hash % partitions, the hash being the reference's (ref_row_hash: MurmurHash3_x86_32 + hash_combine,
// or the identity hash).  Three steps: rows per (partition, CTA) -> exclusive scan on the device -> the rows of
// every fixed-width column to their positions, and, for STRING columns, the permutation "output position ->
// input row" and a gather by it (the reference's general path gathers too, :750; its shared-memory fast path is
// limited to fixed-width tables and 1024 partitions, :253-337).  Rows keep their input order inside a (partition, CTA) run
// only up to the order of the shared-memory atomics: the order inside a partition is unspecified.
constexpr int PART_BLOCK    = 512;
constexpr int MAX_PART_COLS = 32;

struct DPartPlan {
  int nparts;
  int hash_kind;   // RefHash
  u32 seed;
  int counters_in_global;  // per-CTA partition counters live in global memory (more partitions than shared memory holds)
  i64 rows_per_cta;
};

constexpr int PART_ROWS = 4;  // rows per thread and step of the two kernels, their loads in flight together
// Partitions of the PART_ROWS rows r0 + u * step (NO_DEST from `hi` on).  Column by column, the loads of an integer column
// first: behind the type switch of ref_element_hash every row's load would wait for the previous row's hash.
__device__ __forceinline__ void row_partitions(const DPlan& P, const DPartPlan& Q, i64 r0, i64 step, i64 hi, u32 (&p)[PART_ROWS])
{
  u32 h[PART_ROWS];
  for (int k = 0; k < P.nkeys; ++k) {
    const DKeyCol& c = P.keys[k];
    u32 e[PART_ROWS];
    if (!c.mask && (c.width == 8 || c.width == 4) && c.vclass != VC_F32 && c.vclass != VC_F64 && c.vclass != VC_STRING) {
      u64 v[PART_ROWS];
      if (c.width == 8) {
#pragma unroll
        for (int u = 0; u < PART_ROWS; ++u) v[u] = r0 + u * step < hi ? __ldg((const u64*)c.data + c.offset + r0 + u * step) : 0ull;
#pragma unroll
        for (int u = 0; u < PART_ROWS; ++u) e[u] = Q.hash_kind == RH_IDENTITY ? (u32)v[u] : murmur3_x86_32_value(v[u], 8, Q.seed);
      } else {
#pragma unroll
        for (int u = 0; u < PART_ROWS; ++u) v[u] = r0 + u * step < hi ? __ldg((const u32*)c.data + c.offset + r0 + u * step) : 0u;
#pragma unroll
        for (int u = 0; u < PART_ROWS; ++u) e[u] = Q.hash_kind == RH_IDENTITY ? (u32)v[u] : murmur3_x86_32_value(v[u], 4, Q.seed);
      }
    } else {
#pragma unroll
      for (int u = 0; u < PART_ROWS; ++u) e[u] = r0 + u * step < hi ? ref_element_hash(c, r0 + u * step, Q.hash_kind, Q.seed) : 0u;
    }
#pragma unroll
    for (int u = 0; u < PART_ROWS; ++u) h[u] = k == 0 ? e[u] : hash_combine32(h[u], e[u]);
  }
  const u32 n = (u32)Q.nparts;
#pragma unroll
  for (int u = 0; u < PART_ROWS; ++u) p[u] = r0 + u * step >= hi ? NO_DEST : (n & (n - 1u)) == 0u ? (h[u] & (n - 1u)) : h[u] % n;
}

// counts[p * gridDim.x + cta] = rows of this CTA's slice that go to partition p (partition-major, so that
// one exclusive scan over the array gives every (partition, CTA) run its start)
__global__ void __launch_bounds__(PART_BLOCK)
k_partition_count(const __grid_constant__ DPlan P, const DPartPlan Q, i64* __restrict__ counts, u32* __restrict__ cta_scratch)
{
  extern __shared__ u32 s_hist[];
  const bool in_global = Q.counters_in_global != 0;
  u32* hist = in_global ? cta_scratch + (size_t)blockIdx.x * Q.nparts : s_hist;  // (global slices arrive zeroed)
  if (!in_global) for (int p = threadIdx.x; p < Q.nparts; p += blockDim.x) hist[p] = 0;
  __syncthreads();
  const i64 lo = (i64)blockIdx.x * Q.rows_per_cta;
  const i64 hi = min(P.nrows, lo + Q.rows_per_cta);
  // (plain atomics on shared counters: 32-bit words are added natively, at one rate whether lanes meet or not, and finding
  // the lanes that meet — __match_any_sync — took longer than the adds: 636 us for 100M INT64 keys with it, 277 without)
  const u32 lane = threadIdx.x & 31u;
  for (i64 r0 = lo + (threadIdx.x - lane); r0 < hi; r0 += PART_ROWS * (i64)blockDim.x) {
    u32 p[PART_ROWS];
    row_partitions(P, Q, r0 + lane, blockDim.x, hi, p);
#pragma unroll
    for (int u = 0; u < PART_ROWS; ++u) {
      if (in_global) {
        const u32 peers = __match_any_sync(0xFFFFFFFFu, p[u]);
        if (p[u] != NO_DEST && (int)lane == __ffs(peers) - 1) atomicAdd(&hist[p[u]], (u32)__popc(peers));
      } else if (p[u] != NO_DEST) {
        atomicAdd(&hist[p[u]], 1u);
      }
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < Q.nparts; p += blockDim.x) counts[(size_t)p * gridDim.x + blockIdx.x] = (i64)hist[p];
}

// offsets[p] = start of partition p (its first (partition, CTA) run), offsets[nparts] = the row count
__global__ void k_partition_offsets(const i64* __restrict__ starts, int nparts, int grid, i64* __restrict__ offsets)
{
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p <= nparts; p += gridDim.x * blockDim.x)
    offsets[p] = starts[(size_t)p * grid];  // (p == nparts reads the scan's closing total)
}

// Fixed-width columns are moved by the kernel that places the rows: it reads them in row order (coalesced) and writes each
// row to its output position — the rows of one partition inside a warp go to consecutive positions — instead of being
// gathered through the permutation afterwards, which reads every sector of a source column once per partition that has a
// row in it (100M rows of INT64, nullable FLOAT64 and two INT32 columns into 8 partitions: placing 2.5 ms and gathering
// 1.0 ms; now 1.2 ms for both).  A null mask arrives filled with ones; a null row clears its bit.
struct DDirectCols {
  int n;
  int width[MAX_PART_COLS];
  const unsigned char* src[MAX_PART_COLS];  // first element of the view
  unsigned char* dst[MAX_PART_COLS];
  const u32* mask[MAX_PART_COLS];           // nullptr: no nulls
  i64 mask_offset[MAX_PART_COLS];
  u32* dst_mask[MAX_PART_COLS];
};

template <typename T>
__device__ __forceinline__ void move_rows(const unsigned char* src, unsigned char* dst, i64 r, i64 step, const u32 (&d)[PART_ROWS])
{
  T v[PART_ROWS];
#pragma unroll
  for (int u = 0; u < PART_ROWS; ++u) if (d[u] != NO_DEST) v[u] = __ldg((const T*)src + r + u * step);
#pragma unroll
  for (int u = 0; u < PART_ROWS; ++u) if (d[u] != NO_DEST) ((T*)dst)[d[u]] = v[u];
}

// perm[output position] = input row (when `perm` is given), and the direct columns moved.  Row counts stay below 2^31, so
// positions are 32-bit words; a CTA's next position per partition lies in shared memory (or, with many partitions, as an
// offset from its start in a global slice that arrives zeroed).
__global__ void __launch_bounds__(PART_BLOCK)
k_partition_perm(const __grid_constant__ DPlan P, const DPartPlan Q, const i64* __restrict__ starts, u32* __restrict__ cta_scratch,
                 int* __restrict__ perm, const __grid_constant__ DDirectCols D)
{
  extern __shared__ u32 s_cur[];
  const bool in_global = Q.counters_in_global != 0;
  u32* cur = in_global ? cta_scratch + (size_t)blockIdx.x * Q.nparts : s_cur;
  if (!in_global) for (int p = threadIdx.x; p < Q.nparts; p += blockDim.x) cur[p] = (u32)starts[(size_t)p * gridDim.x + blockIdx.x];
  if (blockIdx.x == 0 && threadIdx.x < D.n && D.dst_mask[threadIdx.x] && (P.nrows & 31))  // the bits behind the last row
    atomicAnd(D.dst_mask[threadIdx.x] + (P.nrows >> 5), (1u << (P.nrows & 31)) - 1u);
  __syncthreads();
  const i64 lo = (i64)blockIdx.x * Q.rows_per_cta;
  const i64 hi = min(P.nrows, lo + Q.rows_per_cta);
  const i64 step = blockDim.x;
  const u32 lane = threadIdx.x & 31u;
  for (i64 r0 = lo + (threadIdx.x - lane); r0 < hi; r0 += PART_ROWS * step) {
    const i64 r = r0 + lane;
    u32 p[PART_ROWS], d[PART_ROWS];
    row_partitions(P, Q, r, step, hi, p);
#pragma unroll
    for (int u = 0; u < PART_ROWS; ++u) {
      d[u] = NO_DEST;
      if (in_global) {
        const u32 peers = __match_any_sync(0xFFFFFFFFu, p[u]);
        const int lead  = __ffs(peers) - 1;
        u32 base = 0;
        if (p[u] != NO_DEST && (int)lane == lead) base = (u32)starts[(size_t)p[u] * gridDim.x + blockIdx.x] + atomicAdd(&cur[p[u]], (u32)__popc(peers));
        base = __shfl_sync(0xFFFFFFFFu, base, lead);
        if (p[u] != NO_DEST) d[u] = base + __popc(peers & ((1u << lane) - 1u));
      } else if (p[u] != NO_DEST) {
        d[u] = atomicAdd(&cur[p[u]], 1u);
      }
    }
    if (perm) {
#pragma unroll
      for (int u = 0; u < PART_ROWS; ++u) if (d[u] != NO_DEST) perm[d[u]] = (int)(r + u * step);
    }
    for (int c = 0; c < D.n; ++c) {
      switch (D.width[c]) {
        case 8: move_rows<u64>(D.src[c], D.dst[c], r, step, d); break;
        case 4: move_rows<u32>(D.src[c], D.dst[c], r, step, d); break;
        case 2: move_rows<unsigned short>(D.src[c], D.dst[c], r, step, d); break;
        default: move_rows<unsigned char>(D.src[c], D.dst[c], r, step, d); break;
      }
      if (!D.mask[c]) continue;
      u32 nulls = 0;
#pragma unroll
      for (int u = 0; u < PART_ROWS; ++u) if (d[u] != NO_DEST && !bit_valid(D.mask[c], D.mask_offset[c] + r + u * step)) nulls |= 1u << u;
      if (nulls) {
#pragma unroll
        for (int u = 0; u < PART_ROWS; ++u) if ((nulls >> u) & 1u) atomicAnd(D.dst_mask[c] + (d[u] >> 5), ~(1u << (d[u] & 31u)));
      }
    }
  }
}

// The same for 9 to PT_BLOCK partitions (50M rows of three columns into 16 / 64 / 200: 1253 / 2299 / 2522 us without, 684 / 723 /
// 894 us with; into 8 partitions it loses, 100M rows with a mask 1274 us against 1167): a tile of rows is sorted by partition in
// shared memory, column by column, and written run by run, consecutive threads writing consecutive rows of a run.  (Written from the registers that hold the
// rows in input order, a warp's 32 rows make a short run per partition and column; with 200 partitions a sector per row.)
// Two staging arrays take turns, so that a column costs one barrier.
constexpr int PT_BLOCK = PART_BLOCK;
constexpr int PT_MIN_PARTS = 9, PT_MIN_PARTS_SMALL = 24;  // from PT_MIN_ROWS rows on, below
constexpr i64 PT_MIN_ROWS = 1 << 22;
constexpr int PT_ROWS  = 2 * PART_ROWS;      // rows per thread and tile
constexpr int PT_TILE  = PT_BLOCK * PT_ROWS;
__host__ __device__ constexpr size_t pt_smem(int nparts) { return (size_t)PT_TILE * (2 * 8 + 4) + (size_t)nparts * 16; }

template <typename T>
__device__ __forceinline__ void pt_move(const T (&v)[PT_ROWS], unsigned char* stage, T* __restrict__ dst, const u32* s_at, const u32 (&pos)[PT_ROWS], int have, u32 n)
{
  T* st = (T*)stage;
#pragma unroll
  for (int j = 0; j < PT_ROWS; ++j) if (j * PT_BLOCK < have) st[pos[j]] = v[j];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PT_ROWS; ++i) {
    const u32 q = threadIdx.x + (u32)i * PT_BLOCK;
    if (q < n) dst[s_at[q]] = st[q];
  }
}
template <typename T>
__device__ __forceinline__ void pt_column(const unsigned char* src, unsigned char* stage, unsigned char* dst, const u32* s_at, const u32 (&pos)[PT_ROWS], i64 r, int have, u32 n)
{
  T v[PT_ROWS];
#pragma unroll
  for (int j = 0; j < PT_ROWS; ++j) v[j] = j * PT_BLOCK < have ? __ldg((const T*)src + r + j * PT_BLOCK) : (T)0;
  pt_move<T>(v, stage, (T*)dst, s_at, pos, have, n);
}

__global__ void __launch_bounds__(PT_BLOCK, 2)
k_partition_tiles(const __grid_constant__ DPlan P, const DPartPlan Q, const i64* __restrict__ starts, int* __restrict__ perm, const __grid_constant__ DDirectCols D)
{
  extern __shared__ __align__(16) unsigned char pt_smem_raw[];
  __shared__ u32 s_warp[PT_BLOCK / 32];
  unsigned char* const stage = pt_smem_raw;                     // two arrays of PT_TILE elements
  u32* const s_at = (u32*)(pt_smem_raw + (size_t)PT_TILE * 16); // [PT_TILE] where the staged row goes
  const int np = Q.nparts;
  u32 *hist = s_at + PT_TILE, *off = hist + np, *base = off + np, *cur = base + np;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int p = tid; p < np; p += PT_BLOCK) { cur[p] = (u32)starts[(size_t)p * gridDim.x + blockIdx.x]; hist[p] = 0; }
  if (blockIdx.x == 0 && tid < D.n && D.dst_mask[tid] && (P.nrows & 31))  // the bits behind the last row
    atomicAnd(D.dst_mask[tid] + (P.nrows >> 5), (1u << (P.nrows & 31)) - 1u);
  __syncthreads();
  const i64 lo = (i64)blockIdx.x * Q.rows_per_cta, hi = min(P.nrows, lo + Q.rows_per_cta);
  u32 turn = 0;
  for (i64 t0 = lo; t0 < hi; t0 += PT_TILE) {
    const i64 r = t0 + tid;
    const u32 n = (u32)min((i64)PT_TILE, hi - t0);
    const int have = (int)n - tid;  // row j exists: j * PT_BLOCK < have
    u32 pos[PT_ROWS], part[PT_ROWS];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      u32 p4[PART_ROWS];
      row_partitions(P, Q, r + h * PART_ROWS * PT_BLOCK, PT_BLOCK, hi, p4);
#pragma unroll
      for (int u = 0; u < PART_ROWS; ++u) part[h * PART_ROWS + u] = p4[u];
    }
#pragma unroll
    for (int j = 0; j < PT_ROWS; ++j) pos[j] = j * PT_BLOCK < have ? atomicAdd(&hist[part[j]], 1u) : 0u;
    __syncthreads();
    // exclusive scan over the partitions (at most one per thread)
    const u32 c = tid < np ? hist[tid] : 0u;
    u32 v = c;
    for (int d = 1; d < 32; d <<= 1) { const u32 x = __shfl_up_sync(0xFFFFFFFFu, v, d); if (lane >= d) v += x; }
    if (lane == 31) s_warp[wid] = v;
    __syncthreads();
    const u32 before = __reduce_add_sync(0xFFFFFFFFu, lane < wid ? s_warp[lane] : 0u);
    if (tid < np) {
      const u32 excl = before + v - c, at = cur[tid];
      off[tid] = excl;
      base[tid] = at - excl;  // (modulo 2^32)
      cur[tid] = at + c;
      hist[tid] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PT_ROWS; ++j) {
      if (j * PT_BLOCK >= have) continue;
      pos[j] += off[part[j]];
      s_at[pos[j]] = base[part[j]] + pos[j];
    }
    auto next_stage = [&] { turn ^= 1u; return stage + (size_t)turn * PT_TILE * 8; };
    if (perm) {
      u32 v4[PT_ROWS];
#pragma unroll
      for (int j = 0; j < PT_ROWS; ++j) v4[j] = (u32)(r + j * PT_BLOCK);
      pt_move<u32>(v4, next_stage(), (u32*)perm, s_at, pos, have, n);
    }
    for (int col = 0; col < D.n; ++col) {
      unsigned char* st = next_stage();
      switch (D.width[col]) {
        case 8: pt_column<u64>(D.src[col], st, D.dst[col], s_at, pos, r, have, n); break;
        case 4: pt_column<u32>(D.src[col], st, D.dst[col], s_at, pos, r, have, n); break;
        case 2: pt_column<unsigned short>(D.src[col], st, D.dst[col], s_at, pos, r, have, n); break;
        default: pt_column<unsigned char>(D.src[col], st, D.dst[col], s_at, pos, r, have, n); break;
      }
      if (!D.mask[col]) continue;
      u32 nulls = 0;
#pragma unroll
      for (int j = 0; j < PT_ROWS; ++j) if (j * PT_BLOCK < have && !bit_valid(D.mask[col], D.mask_offset[col] + r + j * PT_BLOCK)) nulls |= 1u << j;
      if (nulls) {
#pragma unroll
        for (int j = 0; j < PT_ROWS; ++j)
          if ((nulls >> j) & 1u) { const u32 d = s_at[pos[j]]; atomicAnd(D.dst_mask[col] + (d >> 5), ~(1u << (d & 31u))); }
      }
    }
    __syncthreads();  // (tables without a column of fixed width and without a permutation: the next tile rewrites s_at)
  }
}

// validity bitmask <-> one byte per row (a row exchange moves validity as bytes: partitions start at
// arbitrary bit positions)
__global__ void k_mask_to_bytes(const u32* __restrict__ mask, i64 offset, i64 n, unsigned char* __restrict__ out)
{
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    out[i] = bit_valid(mask, offset + i) ? 1 : 0;
}
__global__ void k_bytes_to_mask(const unsigned char* __restrict__ bytes, i64 n, u32* __restrict__ mask, u32* null_count)
{
  const i64 nwords = (n + 31) / 32;
  const int lane = threadIdx.x & 31;
  const i64 warp0 = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
  u32 nulls = 0;
  for (i64 w = warp0; w < nwords; w += nwarps) {
    const i64 i = w * 32 + lane;
    const bool v = i < n && bytes[i] != 0;
    const u32 word = __ballot_sync(0xFFFFFFFFu, v);
    if (lane == 0) {
      mask[w] = word;
      const int valid_bits = (int)min((i64)32, n - w * 32);
      nulls += (u32)(valid_bits - __popc(word));
    }
  }
  if (lane == 0 && nulls) atomicAdd(null_count, nulls);
}

}  // namespace b2
