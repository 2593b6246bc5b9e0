// b2_lean.cuh — the lean instantiation of the fused aggregate pass: "Σ and n of one FLOAT32 or FLOAT64
// column" (a mean) over 1..3 fixed-width key columns whose sampled key box fits shared memory.
//
//   k_aggregate_lean<NK, K8, STAGED, KEY_MASKS, V8, WIDE>
//     replaces mapping_indices_kernel + single_pass_shmem_aggs_kernel for this shape
//     (cpp/src/groupby/hash/compute_mapping_indices.cuh:92-151, compute_shared_memory_aggs.cu:260-353).
//
// It is a kernel of its own, not a branch of k_aggregate, so that its register allocation is decided
// by its row loop alone: everything rare (keys outside the sampled box, values outside the window, the ragged
// end of the input) happens behind it.  One CTA per SM, 4 consecutive rows per thread per tile.
//
// Accumulators.  Σ and n of a slot are ONE integer of 64 (FLOAT32) or 96 bits (FLOAT64), kept as 2 or 3 words of
// 32 bits: n in the top 14 bits, below it Σ of the values as fixed point, each value biased so that its
// contribution is positive (the count field then never borrows).  A row adds its contribution word by word, the
// carry of each word taken from the value the atomic returns.  Why: shared memory adds 32-bit integers natively
// (measured on a B200, random slots: 3.9 clocks per warp and atomic, whether lanes meet or not), while an fp32 add
// is a compare-and-swap loop (12.6 clocks over 8192 slots, 45 over 64) and so is an fp64 add (21 / 87).  Per 32
// rows: {fp32 add, count} 16.0 clocks, two carried words 7.1; four 18-bit pieces and a count 17.3, three carried
// words 10.5.  The sums are exact until a slot is emptied into the fp64 cell of the global table.
// The window of the fixed point follows from the largest exponent the key-box sampler saw: 12 (FLOAT32) or 15 (FLOAT64)
// binades from twice the sampled maximum down hold every mantissa bit.  With WIDE a slot has a word more and the window 44
// or 47 binades: where more than a few of the sampled values lie below the narrow one (pk_spread_limit) the kernel leaves
// the input alone and the host launches the wide one on the same table.  (100M log-normal values of sigma 3, 64 groups:
// FLOAT32 0.34 ms, FLOAT64 0.42 per call; 17.7 and 15.9 when each value outside the narrow window was added to the global
// table by itself, 0.37 and 0.51 with {fp32 add, count} slots and 18-bit pieces.)
// A row whose key lies outside the box or whose value lies outside the window goes to a list in global memory that its CTA
// works off behind the merge, the values in windows below and above (lean_rare_rows), so the result does not depend on the
// sample: FLOAT64 sums stay exact up to the roundings of flushes and merges over 109 binades and more.  Infinities and NaN
// count as zero here and go into the global cell once per group and kind.  The row loop contains no function call: with the
// rare rows handled on the spot the C2 pass (100M rows) took 0.32 ms instead of 0.21, most of it registers moved around
// calls that were hardly ever made.
//
//   STAGED = false : tiles go global -> registers with 16-byte ld.global.nc, the next tile's vectors
//                    are loaded into a second register set while the current tile is folded;
//   STAGED = true  : one producer warp streams key / value / validity tiles into a shared-memory
//                    ring with cp.async.bulk (no multicast, no tensor map: the columns are flat)
//                    completing on an mbarrier per stage; 31 consumer warps read the tiles from
//                    shared memory.  Every wait is bounded; a wait that runs out sets ctrl->error.
//
// The key box comes from the control block: the sampler runs in k_table_init, which precedes this
// kernel on the stream.  If the box did not fit, the kernel returns at once and the host, which sees that in the
// control block it reads anyway, starts over with the generic k_aggregate.
#pragma once
#include "b2_kernels.cuh"

namespace b2 {

constexpr int LEAN_STAGED_CONSUMERS = 992;  // 31 consumer warps; warp 31 is the producer
constexpr int LEAN_STAGES           = 2;
constexpr int LEAN_MASK_BYTES       = 512;  // validity bytes of one staged tile, padded
constexpr int LEAN_WAIT_TRIES       = 1 << 20;
constexpr u32 LEAN_GAVE_UP          = 2;    // DCtrl::error: the box and the window left out more rows than a list holds

// ------------------------------------------------------------------------------ mbarrier / bulk copy
__device__ __forceinline__ void mbar_init(u32 bar, u32 count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(u32 bar, u32 bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(u32 bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(u32 bar, u32 parity)
{
  u32 ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// bounded: false when the phase did not complete within LEAN_WAIT_TRIES attempts
__device__ __forceinline__ bool mbar_wait(u32 bar, u32 parity)
{
  for (int i = 0; i < LEAN_WAIT_TRIES; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// 16 bytes of a staged tile.  Volatile: the bytes change when the stage has been given back, and a plain load may be issued
// again later where its value is needed once more (rows that do not fit the box or the window were folded with the next
// tile's keys and values).
__device__ __forceinline__ uint4 lds_once(u32 saddr)
{
  uint4 v;
  asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr) : "memory");
  return v;
}
// flat global -> shared copy of `bytes` (a multiple of 16; both addresses 16-byte aligned) that
// reports its bytes to `bar`
__device__ __forceinline__ void bulk_g2s(u32 dst, const void* src, u32 bytes, u32 bar)
{
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// ------------------------------------------------------------------------------ rare paths
struct LeanRare {  // what the rare paths need: this CTA's table and the global one (in shared memory: beside a table of
                   // this size L1 holds next to nothing, and a copy in local memory cost an L2 round trip per use)
  u32* words;   // word i of slot s at words[i * nsp + s]
  int nsp, trash;  // trash: the slot of rows that are not folded
  double unit;  // value of 1 in the fixed point
  int* s_new;
  u64* tbl; i64 cap; i64 region; int stride; int special_pos;
  DCtrl* ctrl; const DDense* box;
  u32* odd;     // one byte per box position: its cell has +infinity (1), -infinity (2), NaN (4)
};

// reports this CTA's unreported slot claims of the hashed region
__device__ __forceinline__ void lean_report_claims(const LeanRare& L)
{
  const int c = atomicExch(L.s_new, 0);
  if (c) {
    const u64 tot = atomicAdd(&L.ctrl->nclaimed, (u64)c) + (u64)c;
    if (tot > L.ctrl->claim_limit) L.ctrl->overflow = 1;
  }
}

// global slot of box position `pos`
__device__ __forceinline__ SlotRef lean_box_slot(const LeanRare& L, u32 pos)
{
  const i64 g = (int)pos == L.special_pos ? L.cap : L.cap + 1 + (i64)pos;
  return slot_ref(L.tbl, L.cap, L.stride, L.region, g);
}

// a row that cannot be folded in shared memory: its key lies outside the sampled box (global hashed
// region), or it belongs to the ragged end of the input (in-box keys go to the dense region directly)
__device__ __noinline__ void lean_slow_row(const DPlan& P, const LeanRare& L, i64 row, bool check_active)
{
  if (check_active && !row_active(P, row)) return;
  if (*(volatile u32*)&L.ctrl->overflow) return;  // this attempt will be discarded
  const u64 key = pack_key(P, row);
  const int di  = key != EMPTY ? dense_index(P, *L.box, key) : -1;
  SlotRef ref;
  if (di >= 0) {
    ref = lean_box_slot(L, (u32)di);
    if ((int)di == L.special_pos) L.ctrl->special_used = 1;
    else if (*(volatile u64*)ref.key == EMPTY && atomicExch(ref.key, key) == EMPTY) { atomicAdd(L.s_new, 1); lean_report_claims(L); }
  } else {
    const i64 g = gmem_find_insert_packed(L.tbl, L.cap, L.stride, key, mix64(key), L.ctrl, L.s_new);
    lean_report_claims(L);
    if (g < 0) return;
    ref = slot_ref(L.tbl, L.cap, L.stride, L.region, g);
  }
  const DValCol& vc = P.vals[P.cells[0].col];
  if (value_valid(vc, row)) {
    const double x = vc.vclass == VC_F64 ? __ldg((const double*)vc.data + vc.offset + row)
                                         : (double)__ldg((const float*)vc.data + vc.offset + row);
    atomicAdd((double*)ref.cells, x);
    atomicAdd(ref.cells + ref.step, 1ull);
  }
}

// ------------------------------------------------------------------------------ packed accumulators
constexpr int PK_COUNT_SHIFT = 18;           // n sits at bit 18 of the top word
// FLOAT32: 24 mantissa bits + 11 = contributions below 2^35 in magnitude, + 43 below 2^67; FLOAT64: 53 + 14 = 67, 53 + 46 = 99
constexpr u32 PK_BIAS        = 1u << 3;      // 2^35 (2^67, 2^99) in the top word: every contribution becomes positive
// Addends of a slot between flushes.  A thread that meets a slot with PK_FLUSH of them empties it before it adds anything
// else, so each of the 1024 threads adds at most the four rows of one group beyond that: 5120.
constexpr u32 PK_FLUSH       = 1024;
// The top word of an empty slot: the PK_FLUSH-th addend turns its sign bit on.  (2^32 - PK_TOP) >> 18 = 9216 addends
// fit before it wraps.
constexpr u32 PK_TOP         = 0x80000000u - (PK_FLUSH << PK_COUNT_SHIFT);

// The window of one launch, from 1 + the largest sampled biased exponent (`vexp`, 0 = nothing was sampled), `b` = the
// biased exponent of the values whose mantissa lies at bit 0.  Adding 1.5 * 2^52 units to a number leaves its count of
// units in the low bits of the sum: a FLOAT32 value is widened and added once, of a FLOAT64 value the high part (multiples
// of 2^32 units; before that, WIDE, those of 2^64) is split off first and what is left is added then; all additions are exact
// for a value that fits.
// The magnitude bounds lo <= |x| < hi (bit patterns; the high words of doubles) tell whether it does.  With no usable
// window nothing but zero fits.
struct PkWindow { double m_top, m_high, m_low; u32 lo2, hi; };  // lo2: 2 * (lower bound) - 1
template <bool V8, bool WIDE>
__device__ __forceinline__ PkWindow pk_window(u32 vexp, double& unit)
{
  constexpr int span = pk_span(V8, WIDE);
  int b = (int)vexp - 1 + (WIDE ? PK_WIDE_HEADROOM : PK_HEADROOM) - span;
  b = max(b, V8 ? 64 : 1);
  unit = 0.0;
  if (vexp == 0 || b > (V8 ? 1980 : 254)) return PkWindow{0.0, 0.0, 0.0, 0xFFFFFFFEu, 0u};
  unit = ldexp(1.0, b - (V8 ? 1075 : 150));
  const int shift = V8 ? 20 : 23;
  const double m = 1.5 * unit * 4503599627370496.0;
  return PkWindow{m * 18446744073709551616.0, m * 4294967296.0, m, ((u32)b << (shift + 1)) - 1u,
                  (u32)min(b + span + 1, V8 ? 0x7FF : 0xFF) << shift};
}
// Contribution of one value that fits: {count 1, bias, fixed point} as 64 or 96 bits.
__device__ __forceinline__ void pk_split(u32 x, const PkWindow& W, u32 (&w)[2])
{
  const double d = (double)__uint_as_float(x) + W.m_low;
  w[0] = (u32)__double2loint(d);
  w[1] = (u32)__double2hiint(d) + (((1u << PK_COUNT_SHIFT) + PK_BIAS) - (u32)__double2hiint(W.m_low));
}
__device__ __forceinline__ void pk_split(double x, const PkWindow& W, u32 (&w)[3])
{
  const double d1 = x + W.m_high, d2 = (x - (d1 - W.m_high)) + W.m_low;
  w[0] = (u32)__double2loint(d2);
  const u32 low_sign = (u32)__double2hiint(d2) - (u32)__double2hiint(W.m_low);   // 0 or -1
  // {high part + low_sign} in 64 bits, the constant of the top word on it
  asm("{\n add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, %3;\n}" : "=r"(w[1]), "=r"(w[2])
      : "r"((u32)__double2loint(d1)), "r"(low_sign), "r"((u32)__double2hiint(d1)));
  w[2] += ((1u << PK_COUNT_SHIFT) + PK_BIAS) - (u32)__double2hiint(W.m_high);
}
__device__ __forceinline__ void pk_split(double x, const PkWindow& W, u32 (&w)[4])
{
  const double d1 = x + W.m_top, r1 = x - (d1 - W.m_top), d2 = r1 + W.m_high, d3 = (r1 - (d2 - W.m_high)) + W.m_low;
  w[0] = (u32)__double2loint(d3);
  const u32 low_sign = (u32)__double2hiint(d3) - (u32)__double2hiint(W.m_low);    // 0 or -1
  const u32 mid_sign = (u32)__double2hiint(d2) - (u32)__double2hiint(W.m_high);   // 0 or -1
  w[1] = (u32)__double2loint(d2);
  w[2] = (u32)__double2loint(d1);
  w[3] = (u32)__double2hiint(d1) + (((1u << PK_COUNT_SHIFT) + PK_BIAS) - (u32)__double2hiint(W.m_top));
  asm("{\n add.cc.u32 %0, %0, %3;\n addc.cc.u32 %1, %1, %3;\n addc.u32 %2, %2, %3;\n}" : "+r"(w[1]), "+r"(w[2]), "+r"(w[3]) : "r"(low_sign));
  asm("{\n add.cc.u32 %0, %0, %2;\n addc.u32 %1, %1, %2;\n}" : "+r"(w[2]), "+r"(w[3]) : "r"(mid_sign));
}
// 2 |x| - 1 as an unsigned number: zero becomes the largest one, so that min(...) >= lo2 says "zero or >= the lower bound".
// (FLOAT64: of the high word; a nonzero low word under a zero high word — a denormal — does not pass for zero)
__device__ __forceinline__ u32 pk_low(u32 x) { return x + x - 1u; }
__device__ __forceinline__ u32 pk_low(u32 lo, u32 hi)
{
  u32 r;
  asm("{\n .reg .u32 t;\n add.cc.u32 t, %1, 0xFFFFFFFF;\n addc.u32 %0, %2, 0xFFFFFFFF;\n}" : "=r"(r) : "r"(lo), "r"(hi + hi));
  return r;
}
__device__ __forceinline__ u32 umin4(u32 a, u32 b, u32 c, u32 d) { return min(min(a, b), min(c, d)); }
__device__ __forceinline__ u32 umax4(u32 a, u32 b, u32 c, u32 d) { return max(max(a, b), max(c, d)); }
// n and Σ of slots: Σ = high * 2^(32 (WORDS - 2) or 32) + mid * 2^32 + low units, added up over slots before it is rounded
struct PkSum { i64 n, high; u64 mid, low; };
template <int WORDS>
__device__ __forceinline__ void pk_decode(const u32* w, PkSum& t)
{
  const u32 top = w[WORDS - 1] - PK_TOP;
  const i64 n = (i64)(top >> PK_COUNT_SHIFT);
  const u32 field = top & ((1u << PK_COUNT_SHIFT) - 1u);
  t.n += n;
  t.low += w[0];
  if (WORDS == 2) t.high += (i64)field - n * (i64)PK_BIAS;
  else t.high += (i64)(((u64)field << 32) | w[WORDS - 2]) - n * ((i64)PK_BIAS << 32);
  if (WORDS == 4) t.mid += w[1];
}
template <int WORDS>
__device__ __forceinline__ double pk_value(const PkSum& t, double unit)
{
  if (WORDS < 4) {  // (|high| and low below 2^53: one rounding; unit is a power of two)
    return fma((double)(t.high + (i64)(t.low >> 32)), 4294967296.0, (double)(t.low & 0xFFFFFFFFull)) * unit;
  }
  const u64 mid = t.mid + (t.low >> 32);
  u64 lo = (mid << 32) | (t.low & 0xFFFFFFFFull), hi = (u64)t.high + (mid >> 32);
  const bool neg = (hi >> 63) != 0;  // by magnitude, so that a small sum of either sign loses nothing
  if (neg) { lo = 0ull - lo; hi = ~hi + (lo == 0 ? 1ull : 0ull); }
  const double a = fma((double)hi, 18446744073709551616.0, (double)lo) * unit;
  return neg ? -a : a;
}
// Adds a contribution to the words at shared address `a` (word step `st` bytes), the carries from the words that the atomics
// return; what the top word was.
template <int WORDS>
__device__ __forceinline__ u32 pk_add(u32 a, u32 st, u32 (&w)[WORDS])
{
  u32 old = 0;
#pragma unroll
  for (int k = 0; k < WORDS; ++k) {
    old = satom_add_u32(a + (u32)k * st, w[k]);
    u64 c = ((u64)old + w[k]) >> 32;
#pragma unroll
    for (int i = k + 1; i < WORDS; ++i) { c += w[i]; w[i] = (u32)c; c >>= 32; }
  }
  return old;
}
// empties the slot whose word i lies at words[i * step]
template <int WORDS>
__device__ __forceinline__ PkSum pk_take(u32* words, int step)
{
  u32 w[WORDS];
#pragma unroll
  for (int i = 0; i < WORDS; ++i) w[i] = atomicExch(words + (size_t)i * step, i == WORDS - 1 ? PK_TOP : 0u);
  PkSum t{0, 0, 0, 0};
  pk_decode<WORDS>(w, t);
  return t;
}

// thread-block clusters
__device__ __forceinline__ u32 cluster_size() { u32 n; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n)); return n; }
__device__ __forceinline__ u32 cluster_rank() { u32 r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_barrier()
{
  asm volatile("barrier.cluster.arrive;\n barrier.cluster.wait;" ::: "memory");
}
__device__ __forceinline__ u32 cluster_map(u32 saddr, u32 rank)
{
  u32 a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
__device__ __forceinline__ u32 cluster_load(u32 addr)
{
  u32 v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ u32 cluster_load_u8(u32 addr)
{
  u32 v;
  asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// ------------------------------------------------------------------------------ the listed rows
// Rows whose key lies outside the box go to the hashed region.  A value outside the window belongs to a window of 47 binades
// below or above it, for which the CTA's shared memory, free by now, is set up once more (the positions in slices where they
// do not fit at once), so that its group's sum is rounded once per CTA and not once per value.  What fits none (denormal
// doubles) is added to the group's global cell.  Called by all threads of the CTA.
template <bool V8, bool WIDE>
__device__ __noinline__ void lean_rare_rows(const DPlan& P, const LeanRare& L, const u32* list, u32 count, unsigned char* smem, u32 smem_bytes)
{
  __shared__ u32 s_sides;
  constexpr int WORDS = 4, SPAN = pk_span(true, true);
  // the main window in biased exponents of doubles (FLOAT32 values are widened)
  const int shift = V8 ? 0 : 1023 - 127;
  int least = (int)L.box->vexp - 1 + (WIDE ? PK_WIDE_HEADROOM : PK_HEADROOM) - pk_span(V8, WIDE);
  least = max(least, V8 ? 64 : 1);
  const int base[2] = {max(least + shift - 1 - SPAN, 64), min(least + shift + pk_span(V8, WIDE) + 1, 1980)};
  auto value_of = [&](u32 row) -> double {
    const DValCol& vc = P.vals[P.cells[0].col];
    return V8 ? __ldg((const double*)vc.data + vc.offset + row) : (double)__ldg((const float*)vc.data + vc.offset + row);
  };
  auto side_of = [&](double x) -> int {  // 0 / 1: the window below / above; -1: none
    const int e = (int)((u32)__double2hiint(x) >> 20) & 0x7FF;
    if (e == 0 || e == 0x7FF) return -1;
    if (e >= base[1] && e <= base[1] + SPAN && e > least + shift) return 1;
    return e >= base[0] && e <= base[0] + SPAN ? 0 : -1;
  };
  if (threadIdx.x == 0) s_sides = 0;
  __syncthreads();
  for (u32 i = threadIdx.x; i < count; i += blockDim.x) {
    const u32 row = list[i];
    const u64 key = pack_key(P, row);
    const int side = key != EMPTY || L.special_pos >= 0 ? side_of(value_of(row)) : -1;
    if (side < 0 || dense_index(P, *L.box, key) < 0) lean_slow_row(P, L, (i64)row, false);
    else if (!((*(volatile u32*)&s_sides >> side) & 1u)) atomicOr(&s_sides, 1u << side);
  }
  __syncthreads();
  const int S = (int)L.box->total, slice = min(S, (int)(smem_bytes / (4u * WORDS)));
  u32* words = (u32*)smem;  // [WORDS][slice]
  const u32 words_a = (u32)__cvta_generic_to_shared(words), step = 4u * (u32)slice;
  for (int side = 0; side < 2; ++side) {
    if (!((s_sides >> side) & 1u)) continue;
    const double unit = ldexp(1.0, base[side] - 1075), m = 1.5 * unit * 4503599627370496.0;
    const PkWindow W{m * 18446744073709551616.0, m * 4294967296.0, m, 0u, 0u};
    for (int first = 0; first < S; first += slice) {
      for (int i = threadIdx.x; i < WORDS * slice; i += blockDim.x) words[i] = i >= (WORDS - 1) * slice ? PK_TOP : 0u;
      __syncthreads();
      auto put = [&](int at, const PkSum& t) {
        const SlotRef ref = lean_box_slot(L, (u32)(first + at));
        if (first + at == L.special_pos) L.ctrl->special_used = 1;
        atomicAdd((double*)ref.cells, pk_value<WORDS>(t, unit));
        atomicAdd(ref.cells + ref.step, (u64)t.n);
      };
      for (u32 i = threadIdx.x; i < count; i += blockDim.x) {
        const u32 row = list[i];
        const double x = value_of(row);
        if (side_of(x) != side) continue;
        const u64 key = pack_key(P, row);
        const int at = (key != EMPTY || L.special_pos >= 0 ? dense_index(P, *L.box, key) : -1) - first;
        if (at < 0 || at >= slice || first + at >= S) continue;
        u32 w[WORDS];
        pk_split(x, W, w);
        if ((int)pk_add<WORDS>(words_a + 4u * (u32)at, step, w) < 0) put(at, pk_take<WORDS>(words + at, slice));
      }
      __syncthreads();
      for (int at = threadIdx.x; at < slice && first + at < S; at += blockDim.x) {
        const PkSum t = pk_take<WORDS>(words + at, slice);
        if (t.n != 0) put(at, t);
      }
      __syncthreads();
    }
  }
}

// ------------------------------------------------------------------------------ the kernel
template <int NK, bool K8, bool STAGED, bool KEY_MASKS, bool V8, bool WIDE>
__global__ void __launch_bounds__(1024, 1)
k_aggregate_lean(const __grid_constant__ DPlan P, u64* __restrict__ tbl, i64 cap, DCtrl* ctrl, u32 region_slots, u32 smem_bytes,
                 u32 max_slots, u32* __restrict__ rare_lists, u32 rare_cap, u32* __restrict__ odd)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ DDense s_dense;
  __shared__ LeanRare L;
  __shared__ int s_new;
  __shared__ u32 s_rare;  // rows in this CTA's list
  __shared__ __align__(8) u64 s_bars[2 * LEAN_STAGES];

  const int tid = threadIdx.x;
  const DValCol& vc = P.vals[P.cells[0].col];
  const bool filt_is_val = P.nfilters == 1 && P.filters[0] == vc.mask && P.filter_offsets[0] == vc.offset;
  const bool nullocc = vc.mask && !filt_is_val; // rows with a null value take part: they make their group exist
  constexpr int WORDS = (V8 ? 3 : 2) + (WIDE ? 1 : 0);  // 32-bit words of one slot
  constexpr u32 VB = V8 ? 8u : 4u;              // bytes of one value
  // bytes of key column k: a constant when no column is 8 bytes wide, so the offsets below fold away
  auto kwidth = [&](int k) -> u32 { return K8 ? (u32)P.keys[k].width : 4u; };

  // ---- what does not need the key box, done while k_table_init in front of this kernel still samples it: the
  // barriers, the first tiles of the ring, a zeroed table.
  // Shared memory: [ring | words [WORDS][NSP] | socc [NSP]].  A stage: [key column 0 | .. | key column NK-1 | value
  // column | validity bytes of the value column].  The host only selects STAGED when there are no key masks and the
  // only row filter (if any) is the value column's own mask.
  constexpr u32 TR = LEAN_STAGED_CONSUMERS * LEAN_ROWS;
  const u32 nstaged = STAGED ? (u32)(P.nrows / TR) : 0u;  // full tiles; the rows behind them are read straight from global memory
  const u32 ragged_quads = STAGED ? (u32)(P.nrows - (i64)nstaged * TR) / LEAN_ROWS : 0u;
  u32 col_off[NK + 1];
  u32 off = 0;
#pragma unroll
  for (int k = 0; k < NK; ++k) { col_off[k] = off; off += TR * kwidth(k); }
  col_off[NK] = off;
  const u32 mask_off = off + TR * VB;
  const u32 stage_bytes = mask_off + LEAN_MASK_BYTES;
  const u32 ring_bytes = STAGED ? LEAN_STAGES * stage_bytes : 0u;
  const u32 bar0 = (u32)__cvta_generic_to_shared(s_bars);
  const u32 stage_a = (u32)__cvta_generic_to_shared(smem_raw);
  auto issue_tile = [&](u32 tile, u32 s) {  // one lane issues every copy
    const u32 dst = stage_a + s * stage_bytes;
    const u64 r0  = (u64)tile * TR;
    const u32 full = bar0 + 8u * s;
    mbar_expect_tx(full, mask_off + (vc.mask ? TR / 8u : 0u));
#pragma unroll
    for (int k = 0; k < NK; ++k)
      bulk_g2s(dst + col_off[k], P.keys[k].data + ((u64)P.keys[k].offset + r0) * kwidth(k), TR * kwidth(k), full);
    bulk_g2s(dst + col_off[NK], vc.data + ((u64)vc.offset + r0) * VB, TR * VB, full);
    if (vc.mask) bulk_g2s(dst + mask_off, (const unsigned char*)vc.mask + (((u64)vc.offset + r0) >> 3), TR / 8u, full);
  };
  u32 issued = 0;  // tiles this thread has requested (the producer lane only)
  if (STAGED && tid == LEAN_STAGED_CONSUMERS) {
    for (int s = 0; s < LEAN_STAGES; ++s) {
      mbar_init(bar0 + 8u * s, 1);                                              // "full": the producer's expect_tx
      mbar_init(bar0 + 8u * (LEAN_STAGES + s), LEAN_STAGED_CONSUMERS / 32);     // "empty": one arrival per consumer warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (u32 tile = blockIdx.x; tile < nstaged && issued < (u32)LEAN_STAGES; tile += gridDim.x, ++issued) issue_tile(tile, issued);
  }
  {
    const u32 nquads = (smem_bytes - ring_bytes) / 16u;
    for (u32 i = tid; i < nquads; i += blockDim.x) ((uint4*)(smem_raw + ring_bytes))[i] = make_uint4(0, 0, 0, 0);
  }
  // the copies in flight must land before this CTA's shared memory is released
  auto drain = [&]() {
    for (u32 s = 0; s < (u32)LEAN_STAGES && s < issued; ++s) {
      const u32 last = issued - 1 - ((issued - 1 - s) % LEAN_STAGES);  // last request that used stage s
      mbar_wait(bar0 + 8u * s, (last / LEAN_STAGES) & 1u);
    }
  };

  // ---- the key box
  grid_dependency_wait();
  for (int i = tid; i < (int)(sizeof(DDense) / 4); i += blockDim.x) ((u32*)&s_dense)[i] = ((const u32*)&ctrl->dense)[i];
  if (tid == 0) { s_new = 0; s_rare = 0; }
  __syncthreads();
  if (!s_dense.enabled || (!WIDE && s_dense.wide)) {  // the generic kernel takes the input, or the wide one
    if (STAGED && tid == LEAN_STAGED_CONSUMERS) drain();
    return;
  }
  const int stride  = P.stride;
  const int S       = (int)s_dense.total;
  const int copies  = min((int)s_dense.copies, (int)(max_slots / (u32)S));
  const int NS      = S * copies;
  const int NSP     = (NS + 1 + 3) & ~3;  // + the slot of rows that are not folded; arrays padded to 16 bytes
  const u32 copy_off = (u32)((tid >> 5) % copies) * (u32)S;
  u32* words = (u32*)(smem_raw + ring_bytes);                   // [WORDS][NSP]
  unsigned char* socc = (unsigned char*)(words + WORDS * NSP);  // [NSP] if nullocc: groups seen through a null value
  double unit;
  const PkWindow W = pk_window<V8, WIDE>(s_dense.vexp, unit);  // the window of the fixed point
  for (int i = tid; i < NSP; i += blockDim.x) words[(WORDS - 1) * NSP + i] = PK_TOP;
  const u32 words_a = (u32)__cvta_generic_to_shared(words), word_step = 4u * (u32)NSP;
  const u32 trash_a = words_a + 4u * (u32)NS, home_a = words_a + 4u * copy_off;
  if (tid == 0) {
    // position of the key whose bits equal EMPTY inside the box (it lives in the special slot), or -1
    int bits = 0;
    for (int k = 0; k < P.nkeys; ++k) bits += 8 * P.keys[k].width + (P.keys[k].nullbit >= 0 ? 1 : 0);
    const int special_pos = bits == 64 ? dense_index(P, s_dense, EMPTY) : -1;
    L = LeanRare{words, NSP, NS, unit, &s_new, tbl, cap, (i64)region_slots, stride, special_pos, ctrl, &s_dense, odd};
  }

  // the key box in registers: the shared-memory atomics below clobber memory for the compiler, so
  // anything left in s_dense would be re-read from shared memory in every tile
  using box_t = typename std::conditional<K8, u64, u32>::type;  // 32 bits when every key column is 4 bytes wide
  box_t bmin[NK], blim[NK];
  u32 bmul[NK];
  bool bnull[NK], bexcl[NK], bw4[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const DKeyCol& c = P.keys[k];
    // KEY_MASKS = false: no key column carries a mask, so nothing about nulls survives compilation
    bnull[k] = KEY_MASKS && c.nullbit >= 0;
    bexcl[k] = KEY_MASKS && c.mask && !P.include_nulls;
    bw4[k]   = !K8 || c.width == 4;
    bmin[k]  = (box_t)s_dense.min[k];
    blim[k]  = (box_t)(s_dense.range[k] - (bnull[k] ? 1ull : 0ull));
    bmul[k]  = 4u * s_dense.mult[k];  // (in bytes of a word array)
  }

  __syncthreads();

  // Empties the slots of the last group whose addend count has reached PK_FLUSH into the fp64 and count cells of the
  // global table.  The words are exchanged one by one: whatever other threads add in between (a carry among it) is
  // found by the next flush or by the merge — decoding is linear in the words.  Called when the next group's loads have
  // been issued, so that the warp does not wait for what the atomics return.
  u32 addr[4] = {trash_a, trash_a, trash_a, trash_a}, full = 0;
  auto flush_full = [&]() {
    if ((int)full >= 0) return;
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const u32 slot = ((j == 0 ? addr[0] : j == 1 ? addr[1] : j == 2 ? addr[2] : addr[3]) - words_a) >> 2;
      if ((int)*(volatile u32*)(L.words + (WORDS - 1) * L.nsp + slot) >= 0) continue;
      const PkSum t = pk_take<WORDS>(L.words + slot, L.nsp);
      if ((int)slot == L.trash) continue;
      const SlotRef ref = lean_box_slot(L, slot - copy_off);
      atomicAdd((double*)ref.cells, pk_value<WORDS>(t, L.unit));
      atomicAdd(ref.cells + ref.step, (u64)t.n);
      if ((int)(slot - copy_off) == L.special_pos) L.ctrl->special_used = 1;
    }
  };

  // Folds one group of 4 consecutive rows starting at row r0 (the values: four floats in qa, or — V8 — four doubles
  // in qa and qb).  Straight-line code: a row that is not folded (filtered, null value, rare) adds its contribution to
  // the trash slot instead of branching around the atomics, and what can be wrong with the four rows — a key outside
  // the box, a value outside the window — is tested for once, over their minimum and maximum.
  u32* const my_list = rare_lists + (size_t)blockIdx.x * rare_cap;
  auto fold = [&](i64 r0, const uint4 (&ka)[NK], const uint4 (&kb)[NK], const u32 (&kn)[NK], const uint4& qa, const uint4& qb,
                  u32 vn, u32 act) {
    auto key_of = [&](int k, int j, bool& inside) -> u32 {  // position of row j's key in column k's range
      u32 x;
      if (bw4[k]) {
        x = (j == 0 ? ka[k].x : j == 1 ? ka[k].y : j == 2 ? ka[k].z : ka[k].w) - (u32)bmin[k];
        inside = x < (u32)blim[k];
      } else {
        const u32 lo = j == 0 ? ka[k].x : j == 1 ? ka[k].z : j == 2 ? kb[k].x : kb[k].z;
        const u32 hi = j == 0 ? ka[k].y : j == 1 ? ka[k].w : j == 2 ? kb[k].y : kb[k].w;
        const u64 y = (((u64)hi << 32) | lo) - (u64)bmin[k];
        x = (u32)y;
        inside = y < (u64)blim[k];
      }
      if (KEY_MASKS && bnull[k] && !((kn[k] >> j) & 1u)) { x = (u32)blim[k]; inside = true; }
      return x;
    };
    // values: a null's payload counts as zero
    u32 xlo[4], xhi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool val = ((vn >> j) & 1u) != 0u;
      if (V8) {
        xlo[j] = val ? (j == 0 ? qa.x : j == 1 ? qa.z : j == 2 ? qb.x : qb.z) : 0u;
        xhi[j] = val ? (j == 0 ? qa.y : j == 1 ? qa.w : j == 2 ? qb.y : qb.w) : 0u;
      } else {
        xlo[j] = 0;
        xhi[j] = val ? (j == 0 ? qa.x : j == 1 ? qa.y : j == 2 ? qa.z : qa.w) : 0u;
      }
    }
    const u32 vmax = umax4(xhi[0] & 0x7FFFFFFFu, xhi[1] & 0x7FFFFFFFu, xhi[2] & 0x7FFFFFFFu, xhi[3] & 0x7FFFFFFFu);
    auto low_of = [&](int j) { return V8 ? pk_low(xlo[j], xhi[j]) : pk_low(xhi[j]); };
    const u32 vmin = umin4(low_of(0), low_of(1), low_of(2), low_of(3));
    bool fine = vmin >= W.lo2 && (vmax < W.hi || vmax == 0u);
    if (KEY_MASKS) {
#pragma unroll
      for (int k = 0; k < NK; ++k) if (bexcl[k]) act &= kn[k];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) addr[j] = home_a;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      u32 x[4];
      bool inside[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { x[j] = key_of(k, j, inside[j]); addr[j] += x[j] * bmul[k]; }
      if (bw4[k] && !(KEY_MASKS && bnull[k])) fine = fine && umax4(x[0], x[1], x[2], x[3]) < (u32)blim[k];
      else fine = fine && inside[0] && inside[1] && inside[2] && inside[3];
    }
    u32 take = act & vn;
    if (!fine) {
      // which of the rows it is, and why
      u32 live = act;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        bool in = true;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          bool inside;
          key_of(k, j, inside);
          in = in && inside;
        }
        const u32 m = xhi[j] & 0x7FFFFFFFu;
        const bool fits = low_of(j) >= W.lo2 && (m < W.hi || m == 0u);
        if (in && fits) continue;
        const bool on = (act >> j) & 1u;
        if (in && m >= (V8 ? 0x7FF00000u : 0x7F800000u)) {
          // an infinity or NaN: folded as zero; the first one of its kind goes into its group's global cell
          if (on) {
            const bool nan = V8 ? (m > 0x7FF00000u || xlo[j] != 0u) : m > 0x7F800000u;
            const u32 pos = ((addr[j] - words_a) >> 2) - copy_off, bit = (nan ? 4u : (int)xhi[j] < 0 ? 2u : 1u) << ((pos & 3u) * 8u);
            u32* const word = L.odd + (pos >> 2);
            if (!(*word & bit) && !(atomicOr(word, bit) & bit)) {
              double x;
              if constexpr (V8) x = __hiloint2double((int)xhi[j], (int)xlo[j]);
              else x = (double)__uint_as_float(xhi[j]);
              atomicAdd((double*)lean_box_slot(L, pos).cells, x);
            }
          }
        } else {
          take &= ~(1u << j);
          live &= ~(1u << j);
          if (on) {
            const u32 at = atomicAdd(&s_rare, 1u);
            if (at < rare_cap) my_list[at] = (u32)r0 + (u32)j;
          }
        }
        if (V8) xlo[j] = 0;
        xhi[j] = 0;
      }
      act = live;
    }
    if (nullocc) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (((act & ~vn) >> j) & 1u) socc[(addr[j] - words_a) >> 2] = 1;
    }
    u32 w[4][WORDS];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!((take >> j) & 1u)) addr[j] = trash_a;
      if constexpr (V8) pk_split(__hiloint2double((int)xhi[j], (int)xlo[j]), W, w[j]);
      else if constexpr (WIDE) pk_split((double)__uint_as_float(xhi[j]), W, w[j]);
      else pk_split(xhi[j], W, w[j]);
    }
    // word by word over the four rows, so that a warp waits for one round trip per word, not one per row and word; where
    // old + w overflowed, the carry enters the words above
    u32 old[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) old[j] = satom_add_u32(addr[j], w[j][0]);
    if constexpr (WORDS == 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        asm("{\n .reg .u32 t;\n add.cc.u32 t, %3, %4;\n addc.cc.u32 %0, %0, 0;\n addc.cc.u32 %1, %1, 0;\n addc.u32 %2, %2, 0;\n}"
            : "+r"(w[j][1]), "+r"(w[j][2]), "+r"(w[j][3]) : "r"(old[j]), "r"(w[j][0]));
        old[j] = satom_add_u32(addr[j] + word_step, w[j][1]);
      }
    }
    if constexpr (WORDS >= 3) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        asm("{\n .reg .u32 t;\n add.cc.u32 t, %2, %3;\n addc.cc.u32 %0, %0, 0;\n addc.u32 %1, %1, 0;\n}"
            : "+r"(w[j][WORDS - 2]), "+r"(w[j][WORDS - 1]) : "r"(old[j]), "r"(w[j][WORDS - 3]));
        old[j] = satom_add_u32(addr[j] + (WORDS - 2) * word_step, w[j][WORDS - 2]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      asm("{\n .reg .u32 t;\n add.cc.u32 t, %1, %2;\n addc.u32 %0, %0, 0;\n}" : "+r"(w[j][WORDS - 1]) : "r"(old[j]), "r"(w[j][WORDS - 2]));
      old[j] = satom_add_u32(addr[j] + (WORDS - 1) * word_step, w[j][WORDS - 1]);
    }
    full = old[0] | old[1] | old[2] | old[3];
  };

  if (!STAGED) {
    // ---- tiles from global memory into registers
    const u32 tile_rows = 1024u * LEAN_ROWS;
    const u32 nfull     = (u32)(P.nrows / tile_rows);
    auto load_tile = [&](u32 tile, uint4& qa, uint4& qb, u32& vn, u32& act, uint4 (&ka)[NK], uint4 (&kb)[NK], u32 (&kn)[NK]) {
      const u32 r0 = tile * tile_rows + (u32)tid * LEAN_ROWS;
      const u32 ve = (u32)vc.offset + r0;
      const uint4* vp = (const uint4*)(vc.data + (u64)ve * VB);
      qa = __ldg(vp);
      if (V8) qb = __ldg(vp + 1);
      else qb = make_uint4(0, 0, 0, 0);
      vn = vc.mask ? nibble_aligned(vc.mask, ve) : 0xFu;
      act = 0xFu;
      if (filt_is_val) act = vn;
      else for (int f = 0; f < P.nfilters; ++f) act &= nibble_aligned(P.filters[f], (u32)P.filter_offsets[f] + r0);
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const DKeyCol& c = P.keys[k];
        const u32 e = (u32)c.offset + r0;
        kn[k] = (KEY_MASKS && c.mask) ? nibble_aligned(c.mask, e) : 0xFu;
        const uint4* kp = (const uint4*)(c.data + (u64)e * kwidth(k));
        ka[k] = __ldg(kp);
        if (K8 && c.width == 8) kb[k] = __ldg(kp + 1);
        else kb[k] = make_uint4(0, 0, 0, 0);
      }
    };
    uint4 qa, qb, nqa, nqb;
    u32 vn = 0, act = 0, nvn = 0, nact = 0;
    uint4 ka[NK], kb[NK], nka[NK], nkb[NK];
    u32 kn[NK], nkn[NK];
    // Register prefetch of the next tile pays off with 4-byte keys; with 8-byte key columns the second
    // set of vector registers costs more than it hides, and the tile after is requested into L2 instead
    constexpr bool PREFETCH = !K8 && !V8 && NK == 1 && !KEY_MASKS;
    if (PREFETCH && blockIdx.x < nfull) load_tile(blockIdx.x, qa, qb, vn, act, ka, kb, kn);
    for (u32 tile = blockIdx.x; tile < nfull; tile += gridDim.x) {
      const u32 next = tile + gridDim.x;
      if (!PREFETCH) {
        load_tile(tile, qa, qb, vn, act, ka, kb, kn);
        if (next < nfull) {
          const u32 fr0 = next * tile_rows + (u32)tid * LEAN_ROWS;
          prefetch_l2(vc.data + (u64)((u32)vc.offset + fr0) * VB);
#pragma unroll
          for (int k = 0; k < NK; ++k) prefetch_l2(P.keys[k].data + (u64)((u32)P.keys[k].offset + fr0) * kwidth(k));
        }
      }
      if (PREFETCH && next < nfull) load_tile(next, nqa, nqb, nvn, nact, nka, nkb, nkn);
      flush_full();
      fold((i64)tile * tile_rows + (i64)tid * LEAN_ROWS, ka, kb, kn, qa, qb, vn, act);
      if (PREFETCH) {
        qa = nqa; qb = nqb; vn = nvn; act = nact;
#pragma unroll
        for (int k = 0; k < NK; ++k) { ka[k] = nka[k]; kb[k] = nkb[k]; kn[k] = nkn[k]; }
      }
    }
  } else {
    // ---- tiles through the shared-memory ring
    bool failed = false;
    if (tid >= LEAN_STAGED_CONSUMERS) {
      if (tid == LEAN_STAGED_CONSUMERS) {
        for (u32 tile = blockIdx.x + issued * gridDim.x; tile < nstaged; tile += gridDim.x, ++issued) {
          const u32 s = issued % LEAN_STAGES, round = issued / LEAN_STAGES;
          if (round > 0 && !mbar_wait(bar0 + 8u * (LEAN_STAGES + s), (round - 1) & 1u)) { failed = true; break; }
          issue_tile(tile, s);
        }
        if (failed) drain();
      }
    } else {
      u32 it = 0;
      for (u32 tile = blockIdx.x; tile < nstaged + (ragged_quads ? 1u : 0u); tile += gridDim.x, ++it) {
        const u32 s = it % LEAN_STAGES, round = it / LEAN_STAGES;
        const bool ragged = tile == nstaged;
        if (ragged && (u32)tid >= ragged_quads) break;
        if (!ragged && !mbar_wait(bar0 + 8u * s, round & 1u)) { failed = true; break; }
        const u32 st = stage_a + s * stage_bytes;
        const u32 e = (u32)tid * LEAN_ROWS;  // element inside the tile
        uint4 ka[NK], kb[NK], qa, qb = make_uint4(0, 0, 0, 0);
        u32 kn[NK], vn = 0xFu;
#pragma unroll
        for (int k = 0; k < NK; ++k) { kn[k] = 0xFu; kb[k] = make_uint4(0, 0, 0, 0); }
        if (!ragged) {
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const u32 at = st + col_off[k] + e * kwidth(k);
            ka[k] = lds_once(at);
            if (K8 && P.keys[k].width == 8) kb[k] = lds_once(at + 16u);
          }
          qa = lds_once(st + col_off[NK] + e * VB);
          if (V8) qb = lds_once(st + col_off[NK] + e * VB + 16u);
          if (vc.mask) vn = *(volatile const u32*)(smem_raw + s * stage_bytes + mask_off + (e >> 5) * 4u);
        } else {
          const u64 row = (u64)tile * TR + e;
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const uint4* kp = (const uint4*)(P.keys[k].data + ((u64)P.keys[k].offset + row) * kwidth(k));
            ka[k] = __ldg(kp);
            if (K8 && P.keys[k].width == 8) kb[k] = __ldg(kp + 1);
          }
          const uint4* vp = (const uint4*)(vc.data + ((u64)vc.offset + row) * VB);
          qa = __ldg(vp);
          if (V8) qb = __ldg(vp + 1);
          if (vc.mask) vn = __ldg(vc.mask + (((u64)vc.offset + row) >> 5));   // (tiles start at multiples of 32 rows)
        }
        if (vc.mask) vn = (vn >> (e & 31u)) & 0xFu;
        const u32 act = filt_is_val ? vn : 0xFu;
        flush_full();
        if (!ragged) {
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(bar0 + 8u * (LEAN_STAGES + s));  // the stage's data is in registers
        }
        fold((i64)tile * TR + e, ka, kb, kn, qa, qb, vn, act);
      }
    }
    if (failed) ctrl->error = 1;
  }
  flush_full();

  // ---- the last rows of the input, which fill no group of four (register tiles: no tile), row by row
  const i64 rows_done = STAGED ? P.nrows / LEAN_ROWS * LEAN_ROWS : P.nrows / (1024 * LEAN_ROWS) * (1024 * LEAN_ROWS);
  for (i64 r = rows_done + (i64)blockIdx.x * blockDim.x + tid; r < P.nrows; r += (i64)gridDim.x * blockDim.x)
    lean_slow_row(P, L, r, true);
  // ---- merge into the dense region of the global table.  The CTAs of a cluster share the box positions and read each
  // other's tables: the replicas of a position are added up as integers in registers, then Σ and n are added to the
  // global cells with one reduction each that returns nothing (consecutive threads, consecutive words).  A group's key
  // follows from its position, so its cell stays unwritten where n says that the group exists (k_finalize, k_dense_settle).
  // (One merge per CTA with a key store per position took 28 us for 148 x 10000 positions: the L2 atomic units bound it.)
  cluster_barrier();  // (also the CTA's own barrier)
  {
    const int S = (int)s_dense.total, copies = min((int)s_dense.copies, (int)(max_slots / s_dense.total)), NSP = (S * copies + 1 + 3) & ~3;
    const int special_pos = L.special_pos;
    const u32 words_a = (u32)__cvta_generic_to_shared(smem_raw + ring_bytes), socc_a = words_a + 4u * (u32)(WORDS * NSP);
    const double unit = L.unit;
    const u32 csize = cluster_size(), crank = cluster_rank();
    const int per = (S + (int)csize - 1) / (int)csize, lo = (int)crank * per, hi = min(S, lo + per);
    const int span = hi - lo;
    const int rot = span > 0 ? (int)(((u64)blockIdx.x * 2654435761ull) % (u64)span) : 0;
    for (int i0 = tid; i0 < span; i0 += blockDim.x) {
      const int i = lo + (i0 + rot < span ? i0 + rot : i0 + rot - span);
      PkSum t{0, 0, 0, 0};
      bool present = false;
      for (int r = 0; r < copies; ++r) {
        const int q = r * S + i;
        u32 w[4][WORDS], seen[4];
#pragma unroll
        for (u32 c = 0; c < 4; ++c) {  // (the loads of up to four tables are in flight together)
          if (c >= csize) break;
          const u32 from = cluster_map(words_a, c) + 4u * (u32)q;
#pragma unroll
          for (int k = 0; k < WORDS; ++k) w[c][k] = cluster_load(from + 4u * (u32)(k * NSP));
          seen[c] = nullocc ? cluster_load_u8(cluster_map(socc_a, c) + (u32)q) : 0u;
        }
#pragma unroll
        for (u32 c = 0; c < 4; ++c) {
          if (c >= csize) break;
          u32 any = seen[c] | (w[c][WORDS - 1] - PK_TOP);
#pragma unroll
          for (int k = 0; k < WORDS - 1; ++k) any |= w[c][k];
          present = present || any != 0u;
          pk_decode<WORDS>(w[c], t);
        }
      }
      if (!present) continue;
      const double sum = pk_value<WORDS>(t, unit);
      const SlotRef ref = lean_box_slot(L, (u32)i);
      if (i == special_pos) { if (ctrl->special_used == 0) ctrl->special_used = 1; }
      else if (t.n == 0 && atomicExch(ref.key, dense_key(P, s_dense, (u32)i)) == EMPTY) atomicAdd(&s_new, 1);
      if (sum != 0.0) atomicAdd((double*)ref.cells, sum);
      if (t.n) atomicAdd(ref.cells + ref.step, (u64)t.n);
    }
  }
  cluster_barrier();  // the tables stay readable until every CTA of the cluster is done
  if (s_rare != 0 && s_rare <= rare_cap) lean_rare_rows<V8, WIDE>(P, L, my_list, s_rare, smem_raw, smem_bytes);
  else if (s_rare != 0 && tid == 0) ctrl->error = LEAN_GAVE_UP;  // more than a list holds: the attempt is discarded
  __syncthreads();
  if (tid == 0) lean_report_claims(L);
}

// Key cells of the groups of a dense region whose n says that they exist, and their number, for the readers that go by
// key cells (partial records, merges); k_finalize does not need it.
__global__ void __launch_bounds__(256) k_dense_settle(const __grid_constant__ DPlan P, u64* __restrict__ tbl, i64 cap, DCtrl* ctrl)
{
  if (!ctrl->dense.enabled) return;
  const i64 region = (i64)ctrl->dense_slots;
  int mine = 0;
  for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < ctrl->dense.total; i += gridDim.x * blockDim.x) {
    const SlotRef ref = slot_ref(tbl, cap, P.stride, region, cap + 1 + (i64)i);
    if (*ref.key != EMPTY || ref.cells[ref.step] == 0ull) continue;  // (groups with a key cell have been counted)
    *ref.key = dense_key(P, ctrl->dense, i);
    ++mine;
  }
  mine = __reduce_add_sync(0xFFFFFFFFu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&ctrl->nclaimed, (u64)mine);
}

}  // namespace b2
