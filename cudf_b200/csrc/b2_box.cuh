// b2_box.cuh — the fused pass over a sampled key box (dense mode of k_aggregate): every cell of a CTA's shared-memory table
// is addressed by the key's position in the box.
//
// What bounds it is the shared-memory pipe (an atomic or a read per row and cell, 4 to 5 clocks per warp) and the
// instructions around it, so cells are kept in the forms of cell_form (native 32-bit atomics instead of 64-bit
// compare-and-swap loops), updates are predicated instead of branched around, and what a row needs only now and then (a key
// outside the box) lies behind one test per thread and tile.
#pragma once
#include "b2_kernels.cuh"

namespace b2 {

constexpr int BOX_KEYS = 2;  // key columns whose positions come from one vector load per column

// What the pass knows about cells and columns besides the plan (decided by the host)
struct DForms {
  unsigned char form[MAX_CELLS];     // CellForm
  signed char count_of[MAX_CELLS];   // CF_MIN32 / CF_MAX32: the cell that counts the column's values, -1: no value is null
  unsigned char kind[MAX_VALS];      // RecKind by the column's type; RK_NONE: no cell reads its values
  signed char first_col, second_col; // columns whose values are loaded together with the keys (-1 = none)
  signed char present;               // a cell that counts every row of its slot (-1: occupancy bits tell the used slots)
  u32 vec;                           // bit v: value column v takes 16-byte loads at multiples of 4 rows
  // Every cell is a sum, a count, a minimum or a maximum: by value column its cell of each (-1: none), the cell that counts rows.
  // The row loop then has no operator to decode.
  unsigned char plain;
  signed char sum[MAX_VALS], count[MAX_VALS], least[MAX_VALS], most[MAX_VALS], rows;
};

// keys outside the box: the global table
__device__ __noinline__ void box_outside(const DPlan& P, u64* tbl, i64 cap, DCtrl* ctrl, int* s_new, i64 row)
{
  const u64 key = pack_key(P, row);
  const i64 g = gmem_find_insert_packed(tbl, cap, P.stride, key, mix64(key), ctrl, s_new);
  if (g < 0) return;
  u64* cells = tbl + g * P.stride + 1;
  for (int c = 0; c < P.ncells; ++c) {
    const int op = P.cells[c].op;
    const DValCol& vc = P.vals[P.cells[c].col];
    if (op == OP_CNT_A) { atomicAdd(cells + c, 1ull); continue; }
    if (value_valid(vc, row)) cell_update(cells + c, op, load_value(vc, row));
  }
}

// 4 values from row0 on, in their carried form
__device__ __forceinline__ void box_values(const DValCol& c, int kind, bool vec, i64 row0, int nv, u64 (&v)[4])
{
  if (vec && nv == 4) {
    if (c.vclass == VC_I64 || c.vclass == VC_U64 || c.vclass == VC_F64) {
      const ulonglong2* src = (const ulonglong2*)(c.data + (c.offset + row0) * 8);
      const ulonglong2 a = __ldg(src), b = __ldg(src + 1);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
      return;
    }
    const uint4 q = __ldg((const uint4*)(c.data + (c.offset + row0) * 4));
    const u32 w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = kind == RK_S32 ? (u64)(i64)(int)w[j] : kind == RK_U32 ? (u64)w[j] : float_carried(w[j]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = j < nv ? load_value(c, row0 + j) : 0ull;
}

// Four rows into the cells of one column.  FLOAT: the values are doubles; NARROW: 32 bits tell a value (its minimum and maximum are
// kept as images, order32).  `sum` ...: shared addresses of the cells' arrays, ~0 = none.  A minimum or maximum is looked at first,
// and only a value that improves on it is an atomic: after a slot's first rows few do.  50M rows, 64 groups, sum / min / max / mean of
// INT64: kernel 339 -> 280 us (call 405 -> 340), with a case for every operator and a replica of the extremes per warp before.
template <bool FLOAT, bool NARROW>
__device__ __forceinline__ void box_fold(int kind, u32 sum, u32 count, u32 least, u32 most, bool is_signed, u32 NS, const u64 (&v)[4], const u32 (&at)[4], u32 use)
{
  constexpr u32 NONE = ~0u;
  if (count != NONE) {
#pragma unroll
    for (int j = 0; j < 4; ++j) fx_red_if(count + 4u * at[j], 1u, use & (1u << j));
  }
  if (sum != NONE) {
    if (FLOAT) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((use >> j) & 1u) atomicAdd((double*)__cvta_shared_to_generic(sum + 8u * at[j]), __longlong_as_double((i64)v[j]));
    } else {
      u32 old[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) old[j] = fx_atom_if(sum + 4u * at[j], (u32)v[j], use & (1u << j));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const u32 up = (u32)(v[j] >> 32) + (old[j] > ~(u32)v[j] ? 1u : 0u);
        fx_red_if(sum + 4u * (NS + at[j]), up, (use & (1u << j)) ? up : 0u);
      }
    }
  }
  if (least == NONE && most == NONE) return;
  if (NARROW) {
    u32 o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = order32(kind, v[j]);
    if (least != NONE) {
      u32 c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) c[j] = lds_u32(least + 4u * at[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) fx_min_if(least + 4u * at[j], o[j], (use & (1u << j)) && o[j] < c[j] ? 1u : 0u);
    }
    if (most != NONE) {
      u32 c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) c[j] = lds_u32(most + 4u * at[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) fx_max_if(most + 4u * at[j], o[j], (use & (1u << j)) && o[j] > c[j] ? 1u : 0u);
    }
    return;
  }
  // 64 bits: cells as in the global table, signed integers or unsigned images
  const u64 flip = !FLOAT && is_signed ? 1ull << 63 : 0ull;
  u64 x[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = FLOAT ? f64_ordered(v[j]) : v[j];
  auto extreme = [&](u32 cell, bool low) {
    u64 c[4];
    u32 better = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = lds_u64(cell + 8u * at[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (low ? (x[j] ^ flip) < (c[j] ^ flip) : (x[j] ^ flip) > (c[j] ^ flip)) better |= 1u << j;
    better &= use;
    if (better) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!((better >> j) & 1u)) continue;
        u64* const p = (u64*)__cvta_shared_to_generic(cell + 8u * at[j]);
        if (flip) { if (low) atomicMin((i64*)p, (i64)x[j]); else atomicMax((i64*)p, (i64)x[j]); }
        else { if (low) atomicMin(p, x[j]); else atomicMax(p, x[j]); }
      }
    }
  };
  if (least != NONE) extreme(least, true);
  if (most != NONE) extreme(most, false);
}

// The whole pass of one CTA: clear, fold the rows of its tiles, merge into the dense region of the global table.  Called by all
// threads; `box` and `s_new`, `s_abort` lie in shared memory.
__device__ __forceinline__ void box_aggregate(const DPlan& P, const DForms& F, u64* tbl, i64 cap, DCtrl* ctrl, i64 dense_slots,
                                              const DDense& box, unsigned char* smem, int* s_new, int* s_abort, bool timekeeper)
{
  __shared__ u32 s_at[MAX_CELLS];  // byte offsets of the cells' arrays
  __shared__ u32 s_occ;            // ... of the occupancy bits
  const int tid = threadIdx.x, stride = P.stride;
  const u32 S = box.total, copies = box.copies, NS = S * copies;
  if (tid == 0) {
    u32 at = 0;
    for (int c = 0; c < P.ncells; ++c) if (cell_form_bytes(F.form[c]) == 8) { s_at[c] = at; at += 8 * NS; }
    for (int c = 0; c < P.ncells; ++c) if (cell_form_bytes(F.form[c]) == 4) { s_at[c] = at; at += 4 * NS; }
    s_occ = at;
  }
  __syncthreads();
  for (int c = 0; c < P.ncells; ++c) {
    if (F.form[c] == CF_64) {
      const u64 id = cell_identity(P.cells[c].op);
      for (u32 i = tid; i < NS; i += blockDim.x) ((u64*)(smem + s_at[c]))[i] = id;
    } else {
      const u32 id = F.form[c] == CF_MIN32 ? 0xFFFFFFFFu : 0u, words = F.form[c] == CF_SUM ? 2 * NS : NS;
      for (u32 i = tid; i < words; i += blockDim.x) ((u32*)(smem + s_at[c]))[i] = id;
    }
  }
  u32* const socc = (u32*)(smem + s_occ);
  const bool bits = F.present < 0;  // no cell tells which slots are in use
  if (bits) for (u32 i = tid; i < (NS + 31) / 32; i += blockDim.x) socc[i] = 0;
  __syncthreads();
  if (timekeeper) ctrl->t_phase[2] = global_timer_ns();

  const u32 copy_off = (u32)((tid >> 5) % copies) * S;
  const u32 smem_a = (u32)__cvta_generic_to_shared(smem);
  const bool fast = (P.flags & PF_VEC_KEYS) && P.nkeys <= BOX_KEYS;
  const i64 tile_rows = (i64)blockDim.x * AGG_ROWS, ntiles = (P.nrows + tile_rows - 1) / tile_rows;
  const int first_col = F.first_col, second_col = F.second_col;
  u32 inside = 0, outside = 0;
  static_assert(AGG_ROWS == 4, "rows of a thread and tile");

  for (i64 tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (*(volatile int*)s_abort) break;
    const i64 row0 = tile * tile_rows + (i64)tid * AGG_ROWS;
    const int nv   = (int)max((i64)0, min((i64)AGG_ROWS, P.nrows - row0));
    u32 act = nv > 0 ? (1u << nv) - 1u : 0u, out = 0;
    u32 at[4] = {copy_off, copy_off, copy_off, copy_off};
    // all loads first
    u64 v0[4] = {}, v1[4] = {};
    if (first_col >= 0) box_values(P.vals[first_col], F.kind[first_col], (F.vec >> first_col) & 1u, row0, nv, v0);
    if (second_col >= 0) box_values(P.vals[second_col], F.kind[second_col], (F.vec >> second_col) & 1u, row0, nv, v1);
    if (fast && nv == 4) {
#pragma unroll
      for (int k = 0; k < BOX_KEYS; ++k) {
        if (k >= P.nkeys) break;
        const DKeyCol& c = P.keys[k];
        const unsigned char* src = c.data + (c.offset + row0) * c.width;
        const u32 lim = (u32)box.range[k] - (c.nullbit >= 0 ? 1u : 0u), mult = box.mult[k];
        u32 vn = 0xFu, d[4], in = 0;
        if (c.width == 8) {
          const ulonglong2 a = __ldg((const ulonglong2*)src), b = __ldg((const ulonglong2*)src + 1);
          const u64 x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const u64 y = x[j] - (u64)box.min[k];
            d[j] = (u32)y;
            if (y < (u64)lim) in |= 1u << j;
          }
        } else {
          u32 x[4];
          if (c.width == 4) {
            const uint4 q = __ldg((const uint4*)src);
            x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
          } else {
            u32 w0, w1;
            if (c.width == 2) { const uint2 q = __ldg((const uint2*)src); w0 = q.x; w1 = q.y; }
            else { const u32 q = __ldg((const u32*)src); w0 = __byte_perm(q, 0, 0x4140); w1 = __byte_perm(q, 0, 0x4342); }
            x[0] = w0 & 0xFFFFu; x[1] = w0 >> 16; x[2] = w1 & 0xFFFFu; x[3] = w1 >> 16;
            const int sh = 32 - 8 * c.width;
#pragma unroll
            for (int j = 0; j < 4; ++j) if (c.is_signed) x[j] = (u32)((int)(x[j] << sh) >> sh);
          }
          // (modulo 2^32: a box never reaches beyond the values that its column's type has)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            d[j] = x[j] - (u32)box.min[k];
            if (d[j] < lim) in |= 1u << j;
          }
        }
        if (c.mask) {
          vn = valid_nibble(c.mask, c.offset + row0, 4);
          if (!P.include_nulls) act &= vn;  // EXCLUDE: a null key drops the row
          else {
#pragma unroll
            for (int j = 0; j < 4; ++j) if (!((vn >> j) & 1u)) d[j] = lim;
            in |= ~vn;
          }
        }
        out |= ~in;
#pragma unroll
        for (int j = 0; j < 4; ++j) at[j] += d[j] * mult;
      }
      for (int f = 0; f < P.nfilters; ++f) act &= valid_nibble(P.filters[f], P.filter_offsets[f] + row0, 4);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!((act >> j) & 1u)) continue;
        if (!row_active(P, row0 + j)) { act &= ~(1u << j); continue; }
        const int d = dense_index(P, box, pack_key(P, row0 + j));
        if (d < 0) out |= 1u << j; else at[j] += (u32)d;
      }
    }
    out &= act;
    if (out) {
#pragma unroll 1
      for (int j = 0; j < 4; ++j) if ((out >> j) & 1u) box_outside(P, tbl, cap, ctrl, s_new, row0 + j);
      outside += __popc(out);
      act &= ~out;
    }
    inside += __popc(act);
    if (bits) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (((act >> j) & 1u) && !((socc[at[j] >> 5] >> (at[j] & 31u)) & 1u)) atomicOr(&socc[at[j] >> 5], 1u << (at[j] & 31u));
    }
    if (F.plain) {
      // ---- column by column
      if (act != 0xFu) {  // (cells are looked at for every row: those of a row that takes no part are any of this CTA's)
#pragma unroll
        for (int j = 0; j < 4; ++j) if (!((act >> j) & 1u)) at[j] = copy_off;
      }
      auto where = [&](int c) { return c < 0 ? ~0u : smem_a + s_at[c]; };
      if (F.rows >= 0) {
        const u32 base = where(F.rows);
#pragma unroll
        for (int j = 0; j < 4; ++j) fx_red_if(base + 4u * at[j], 1u, act & (1u << j));
      }
      for (int col = 0; col < P.nvals; ++col) {
        const int kind = F.kind[col];
        const u32 sum = where(F.sum[col]), count = where(F.count[col]);
        // (minima and maxima in the first replica alone: the fewer there are the fewer values improve on one, and reads of one
        // address do not queue; with a replica per warp 64 groups' values did so 4 times in a tile of a warp)
        const u32 back = copy_off * (kind == RK_64 ? 8u : 4u);
        const u32 least = F.least[col] < 0 ? ~0u : where(F.least[col]) - back, most = F.most[col] < 0 ? ~0u : where(F.most[col]) - back;
        const DValCol& vc = P.vals[col];
        u32 use = act;
        if (vc.mask && nv > 0) use &= valid_nibble(vc.mask, vc.offset + row0, nv);
        if (kind == RK_NONE) {
          if (count != ~0u) {
#pragma unroll
            for (int j = 0; j < 4; ++j) fx_red_if(count + 4u * at[j], 1u, use & (1u << j));
          }
          continue;
        }
        u64 v[4];
        if (col == first_col) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = v0[j];
        } else if (col == second_col) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = v1[j];
        } else {
          box_values(vc, kind, (F.vec >> col) & 1u, row0, nv, v);
        }
        const int k = (kind == RK_F32 || vc.vclass == VC_F64 ? 2 : 0) + (kind == RK_64 ? 0 : 1);
        if (k == 0) box_fold<false, false>(kind, sum, count, least, most, vc.vclass == VC_I64, NS, v, at, use);
        else if (k == 1) box_fold<false, true>(kind, sum, count, least, most, true, NS, v, at, use);
        else if (k == 2) box_fold<true, false>(kind, sum, count, least, most, false, NS, v, at, use);
        else box_fold<true, true>(kind, sum, count, least, most, false, NS, v, at, use);
      }
    }
    // ---- the cells, one after the other: the operator is decoded once for four rows
    int cur = -1;
    u32 vn = 0;
    u64 v[4] = {};
    for (int c = 0; !F.plain && c < P.ncells; ++c) {
      const int op = P.cells[c].op, col = P.cells[c].col, form = F.form[c];
      if (op != OP_CNT_A && col != cur) {
        cur = col;
        const DValCol& vc = P.vals[col];
        vn = act;
        if (vc.mask && nv > 0) vn &= valid_nibble(vc.mask, vc.offset + row0, nv);
        if (col == first_col) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = v0[j];
        } else if (col == second_col) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = v1[j];
        } else if (F.kind[col] != RK_NONE) {
          box_values(vc, F.kind[col], (F.vec >> col) & 1u, row0, nv, v);
        }
      }
      const u32 use = op == OP_CNT_A ? act : vn;
      const u32 base = smem_a + s_at[c];
      switch (form) {
        case CF_COUNT:
#pragma unroll
          for (int j = 0; j < 4; ++j) fx_red_if(base + 4u * at[j], 1u, use & (1u << j));
          break;
        case CF_SUM: {
          u32 old[4];
          if (op != OP_SUM_I) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = sum_addend(op, v[j]);
            cur = -1;  // (the next cell takes the values anew)
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) old[j] = fx_atom_if(base + 4u * at[j], (u32)v[j], use & (1u << j));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const u32 up = (u32)(v[j] >> 32) + (old[j] > ~(u32)v[j] ? 1u : 0u);
            fx_red_if(base + 4u * (NS + at[j]), up, (use & (1u << j)) ? up : 0u);
          }
          break;
        }
        case CF_MIN32:
#pragma unroll
          for (int j = 0; j < 4; ++j) fx_min_if(base + 4u * at[j], order32(F.kind[col], v[j]), use & (1u << j));
          break;
        case CF_MAX32:
#pragma unroll
          for (int j = 0; j < 4; ++j) fx_max_if(base + 4u * at[j], order32(F.kind[col], v[j]), use & (1u << j));
          break;
        default: {
          u64* where[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) where[j] = (u64*)(smem + s_at[c]) + at[j];
          cell_update_shared<4>(where, op, v, use);
        }
      }
    }
    if (tid == 0) {
      const int n = atomicExch(s_new, 0);
      if (n) {
        const u64 tot = atomicAdd(&ctrl->nclaimed, (u64)n) + (u64)n;
        if (tot > ctrl->claim_limit) ctrl->overflow = 1;
      }
      if (*(volatile u32*)&ctrl->overflow) *s_abort = 1;
    }
  }

  inside  = __reduce_add_sync(0xFFFFFFFFu, inside);
  outside = __reduce_add_sync(0xFFFFFFFFu, outside);
  if ((tid & 31) == 0) {
    if (inside) atomicAdd(&ctrl->stat_smem_rows, (u64)inside);
    if (outside) atomicAdd(&ctrl->stat_gmem_rows, (u64)outside);
  }

  // ---- merge: the replicas of a box position are reduced in registers, then ONE merge into the dense region of the global
  // table: no hashing, consecutive threads -> consecutive words of the structure-of-arrays region.  The key cell is claimed
  // with an unconditional exchange (every CTA writes the same key there; the one key whose bits equal EMPTY cannot mark a key
  // cell as used and goes to the special slot instead).  Four positions per step: their exchanges are all issued before the
  // first returned key is looked at, so a step waits for one L2 round trip instead of four (one position per step: 21 us for
  // 15.9K positions).  CTAs start at different positions so that they do not all meet at the same cells.
  __syncthreads();
  if (timekeeper) ctrl->t_phase[3] = global_timer_ns();
  if (*s_abort) return;
  constexpr int MB = 4;
  const u32 rot = (u32)(((u64)blockIdx.x * 2654435761ull) % (u64)S);
  int fresh = 0;  // key cells this thread was the first to claim
  // Few positions with many replicas: a warp per position, a lane per replica, reduced by shuffles.  A thread that adds them up one
  // after the other takes 0.1 us per replica and cell whatever the positions, a warp the longer the more positions it has (1M rows, four
  // cells, 32 replicas, us per call with threads / with warps: 10 groups 75 / 67, 32 76 / 73, 48 77 / 73, 64 77 / 79, 80 77 / 83).
  if (copies > 1 && copies <= 32 && S <= 2 * copies) {
    const u32 lane = tid & 31u, warps = blockDim.x >> 5;
    for (u32 i0 = tid >> 5; i0 < S; i0 += warps) {
      const u32 i = i0 + rot < S ? i0 + rot : i0 + rot - S, q = lane * S + i;
      const bool mine = lane < copies;
      const bool used = mine && (bits ? ((socc[q >> 5] >> (q & 31u)) & 1u) != 0u : ((const u32*)(smem + s_at[F.present]))[q] != 0u);
      if (!__any_sync(0xFFFFFFFFu, used)) continue;
      const u64 key = dense_key(P, box, i);
      const SlotRef slot = slot_ref(tbl, cap, stride, dense_slots, key == EMPTY ? cap : cap + 1 + (i64)i);
      if (lane == 0) {
        if (key == EMPTY) { if (ctrl->special_used == 0) ctrl->special_used = 1; }
        else if (atomicExch(slot.key, key) == EMPTY) ++fresh;
      }
      for (int c = 0; c < P.ncells; ++c) {
        const int op = P.cells[c].op;
        const unsigned char* cell = smem + s_at[c];
        const u64 id = cell_identity(op);
        u64 a = id;
        if (F.form[c] == CF_MIN32 || F.form[c] == CF_MAX32) {  // (in images, as below)
          const bool least = F.form[c] == CF_MIN32;
          const u32 w = mine ? ((const u32*)cell)[q] : least ? 0xFFFFFFFFu : 0u;
          const bool any = F.count_of[c] < 0 || (mine && ((const u32*)(smem + s_at[F.count_of[c]]))[q] != 0u);
          const u32 all = least ? __reduce_min_sync(0xFFFFFFFFu, w) : __reduce_max_sync(0xFFFFFFFFu, w);
          if (__any_sync(0xFFFFFFFFu, any)) a = unorder32(F.kind[P.cells[c].col], all);
        } else {
          if (mine) a = F.form[c] == CF_64 ? ((const u64*)cell)[q] : F.form[c] == CF_COUNT ? (u64)((const u32*)cell)[q] :
                        ((u64)((const u32*)cell)[NS + q] << 32) + ((const u32*)cell)[q];
#pragma unroll 1
          for (int d = 16; d > 0; d >>= 1) a = cell_combine(op, a, __shfl_xor_sync(0xFFFFFFFFu, a, d));
        }
        if (lane == 0 && a != id) cell_merge(slot.cells + (i64)c * slot.step, op, a);
      }
    }
    if (fresh) atomicAdd(s_new, fresh);
    __syncthreads();
    return;
  }
  for (u32 base = tid; base < S; base += MB * blockDim.x) {
    u64 olds[MB];
#pragma unroll
    for (int u = 0; u < MB; ++u) {
      olds[u] = 0;  // anything but EMPTY: "not newly claimed"
      const u32 i0 = base + u * blockDim.x;
      if (i0 >= S) continue;
      const u32 i = i0 + rot < S ? i0 + rot : i0 + rot - S;
      bool present = false;
      for (u32 q = i; q < NS; q += S)
        present = present || (bits ? ((socc[q >> 5] >> (q & 31u)) & 1u) != 0u : ((const u32*)(smem + s_at[F.present]))[q] != 0u);
      if (!present) continue;
      const u64 key = dense_key(P, box, i);
      if (key == EMPTY && ctrl->special_used == 0) ctrl->special_used = 1;
      const SlotRef slot = slot_ref(tbl, cap, stride, dense_slots, key == EMPTY ? cap : cap + 1 + (i64)i);
      if (key != EMPTY) olds[u] = atomicExch(slot.key, key);
      for (int c = 0; c < P.ncells; ++c) {
        const int op = P.cells[c].op;
        const unsigned char* cell = smem + s_at[c];
        const u64 id = cell_identity(op);
        u64 a = 0;
        switch (F.form[c]) {
          case CF_64: a = id; for (u32 q = i; q < NS; q += S) a = cell_combine(op, a, ((const u64*)cell)[q]); break;
          case CF_COUNT: for (u32 q = i; q < NS; q += S) a += ((const u32*)cell)[q]; break;
          case CF_SUM: for (u32 q = i; q < NS; q += S) a += ((u64)((const u32*)cell)[NS + q] << 32) + ((const u32*)cell)[q]; break;
          default: {
            const bool least = F.form[c] == CF_MIN32;
            u32 w = least ? 0xFFFFFFFFu : 0u, n = F.count_of[c] < 0 ? 1u : 0u;
            for (u32 q = i; q < NS; q += S) {
              const u32 x = ((const u32*)cell)[q];
              w = least ? min(w, x) : max(w, x);
              if (F.count_of[c] >= 0) n |= ((const u32*)(smem + s_at[F.count_of[c]]))[q];
            }
            a = n ? unorder32(F.kind[P.cells[c].col], w) : id;  // (no valid value: the identity, whatever image that word is of)
          }
        }
        if (a != id) cell_merge(slot.cells + (i64)c * slot.step, op, a);
      }
    }
#pragma unroll
    for (int u = 0; u < MB; ++u) fresh += olds[u] == EMPTY ? 1 : 0;
  }
  if (fresh) atomicAdd(s_new, fresh);
  __syncthreads();
}

}  // namespace b2
