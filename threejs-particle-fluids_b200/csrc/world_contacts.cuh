// Particle-particle contacts (src/core/contact/generate.ts, solve.ts,
// ContactBuffer.ts; scheduled by loop.ts:180-242, 347-417).
//
// The reference appends pairs to one buffer through an atomic counter, so
// its pair order (and, past maxContacts, which pairs it drops) is whatever
// order the threads reach the counter. Here every emitting slot keeps its own
// partner list (column-major, entry m of slot k at m * n + k, at most
// kMaxContacts), and a per-scene prefix over the slots numbers the pairs in
// slot order: the first max_contacts pairs of that order are solved. Each
// pair's multipliers and normal belong to one lane of its emitting
// slot, and the position and velocity corrections are fixed-point sums, so
// the results do not depend on which side of a pair emits it (swapping the
// pair negates every vector exactly) nor on the order of the atomic adds.
#pragma once

#include "world_kernels.cuh"

namespace pf {

// ContactBuffer.ts:16: multipliers are kept in ticks of 2^-20 kg m.
constexpr float kLambdaScale = 1048576.0f;
constexpr float kLambdaInv = 1.0f / 1048576.0f;
// generate.ts:20
constexpr double kContactRadiusExpansion = 1.1;

// f32 -> i32 toward zero, saturating (the shader's toInt()).
__device__ __forceinline__ int lam_ticks(float v) { return __float2int_rz(v * kLambdaScale); }

// Exclusive prefix of v over the block (blockDim.x a multiple of 32, at most
// 1024); *total receives the block's sum. `ws` holds 32 words.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* ws, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += o;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t t = lane < nw ? ws[lane] : 0u;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, t, d);
      if (lane >= d) t += o;
    }
    ws[lane] = t;  // inclusive prefix of the warp totals
  }
  __syncthreads();
  const uint32_t before = warp ? ws[warp - 1] : 0u;
  *total = ws[nw - 1];
  __syncthreads();  // ws is reused by the caller
  return before + inc - v;
}

// The contact passes give a slot several lanes: a few pairs a slot, each a
// chain of dependent loads, leave most of the chip idle with a thread per
// slot. kConLanes lanes look for a slot's partners, kPairLanes work on its
// pairs.
constexpr uint32_t kConLanes = 4;
constexpr uint32_t kConBlock = kConLanes * kConGroup;  // threads: a block numbers the pairs of one group
static_assert(kConGroup == 32, "numbered in one warp");
constexpr uint32_t kPairLanes = 4;

// generate.ts:53-88: each slot outside the noSelfContacts ranges walks the 27
// cells around its predicted position and keeps every partner closer than
// 2r * 1.1, outside its non-zero collision group, not both pinned; a pair of
// two emitting slots is kept by the lower slot. The block also forms the
// slots' prefix inside its group of 32 slots, and the group's sums.
//
// Bound by the latency of the walk (cell range, position, id, group): the
// nine rows' ranges are loaded together, then each lane's first candidate of
// every row, then the ids of the near ones and their groups. Rows of more
// than kConLanes candidates go on with loads of their own. Hits are numbered
// by ballot in row order, so a slot's list is the one a single thread's walk
// finds. Without a noSelfContacts range in the world (kQuiet false) every
// partner emits, so a slot keeps only those after it: the rows from its own
// on. 50,000 particles in a pile: 29.6 us with a thread per slot; 23.9, 23.5
// and 32.8 with 2, 4 and 8 lanes over nine rows, 14.2, 12.4 and 17.3 over five.
template <bool kQuiet>
__global__ void __launch_bounds__(kConBlock) k_con_gen(WorldView V, uint32_t sub) {
  pdl_begin();
  constexpr int kRow0 = kQuiet ? 0 : 4;
  __shared__ uint32_t found[kConGroup];
  const uint32_t lane = threadIdx.x % kConLanes;
  const uint32_t k = blockIdx.x * kConGroup + threadIdx.x / kConLanes;  // the grid covers n exactly
  const uint32_t shift = threadIdx.x % 32 - lane;  // the slot's lanes in a ballot
  const size_t n = V.n;
  const DevScene& S = scene_at(V, k);
  const uint32_t id = V.ids[k];
  const bool act = S.contact && sub < S.substeps && id < S.seg_start + S.cap && !V.cquiet[id];
  uint32_t rs[9], re[9];
#pragma unroll
  for (int r = kRow0; r < 9; ++r) rs[r] = re[r] = 0;
  f3 xi = mk(0.0f, 0.0f, 0.0f);
  float wi = 0.0f;
  uint32_t gi = 0;
  if (act) {
    const float4 xi4 = V.cur.xs[k];
    xi = xyz(xi4);
    wi = xi4.w;
    gi = V.cgroup[id];
    int32_t cx, cy, cz;
    local_cell(S, xi, &cx, &cy, &cz, nullptr);
    const int32_t x0 = max(cx - 1, 0), x1 = min(cx + 1, (int32_t)S.dims[0] - 1);
#pragma unroll
    for (int r = kRow0; r < 9; ++r) {
      const int32_t z = cz + r / 3 - 1, y = cy + r % 3 - 1;
      if (z < 0 || z >= (int32_t)S.dims[2] || y < 0 || y >= (int32_t)S.dims[1]) continue;
      const uint32_t row = S.cell_base + S.dims[0] * ((uint32_t)y + S.dims[1] * (uint32_t)z);
      rs[r] = V.cstart[row + x0];
      re[r] = V.cstart[row + x1] + V.ccount[row + x1];
    }
    if (!kQuiet) rs[4] = max(rs[4], k + 1);
  }
  const float cand2 = S.c_cand2;
  const uint32_t lim = S.seg_start + S.cap;
  const auto near = [&](uint32_t j, const float4& xj) {
    const f3 d = xi - xyz(xj);
    return !(dot(d, d) >= cand2) && j != k && !(wi <= 0.0f && xj.w <= 0.0f);
  };
  uint32_t jd[9];  // the first candidates' ids, lim where there is none or it is too far
  {
    float4 xj[9];
#pragma unroll
    for (int r = kRow0; r < 9; ++r)
      if (rs[r] + lane < re[r]) xj[r] = V.cur.xs[rs[r] + lane];
#pragma unroll
    for (int r = kRow0; r < 9; ++r) {
      const uint32_t j = rs[r] + lane;
      jd[r] = j < re[r] && near(j, xj[r]) ? V.ids[j] : lim;
    }
  }
  uint32_t keep = 0;
#pragma unroll
  for (int r = kRow0; r < 9; ++r)
    if (jd[r] < lim && (rs[r] + lane > k || (kQuiet && V.cquiet[jd[r]])) && (gi == 0u || gi != V.cgroup[jd[r]]))
      keep |= 1u << r;
  uint32_t cnt = 0;
  const auto append = [&](bool hit, uint32_t j) {
    const uint32_t b = (__ballot_sync(0xffffffffu, hit) >> shift) & ((1u << kConLanes) - 1u);
    if (hit) {
      const uint32_t m = cnt + __popc(b & ((1u << lane) - 1u));
      if (m < kMaxContacts) {
        V.con_nbr[m * n + k] = j;
        V.con_lam[m * n + k] = make_int2(0, 0);
      }
    }
    cnt += __popc(b);
  };
  uint32_t more = 0;
#pragma unroll
  for (int r = kRow0; r < 9; ++r)
    if (rs[r] + kConLanes < re[r]) more |= 1u << r;
  const uint32_t any_keep = __reduce_or_sync(0xffffffffu, keep), any_more = __reduce_or_sync(0xffffffffu, more);
#pragma unroll
  for (int r = kRow0; r < 9; ++r) {
    if (any_keep >> r & 1u) append(keep >> r & 1u, rs[r] + lane);
    if (!(any_more >> r & 1u)) continue;
    uint32_t j = rs[r] + kConLanes + lane;
    while (__any_sync(0xffffffffu, j < re[r])) {
      bool hit = false;
      if (j < re[r] && near(j, V.cur.xs[j])) {
        const uint32_t q = V.ids[j];
        hit = q < lim && (j > k || (kQuiet && V.cquiet[q])) && (gi == 0u || gi != V.cgroup[q]);
      }
      append(hit, j);
      j += kConLanes;
    }
  }
  if (lane == 0) {
    found[threadIdx.x / kConLanes] = cnt;
    V.con_cnt[k] = cnt;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const uint32_t v = found[threadIdx.x];
  uint32_t inc = v;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
    if (threadIdx.x >= d) inc += o;
  }
  V.con_pre[blockIdx.x * kConGroup + threadIdx.x] = inc - v;
  const uint32_t dropped = __reduce_add_sync(0xffffffffu, v > kMaxContacts ? v - kMaxContacts : 0u);
  if (threadIdx.x == 31) {
    V.con_sum[blockIdx.x] = inc;
    V.con_drop[blockIdx.x] = dropped;
  }
}

// The groups' first pair index inside their scene (one block per scene, a
// thread per eight groups), and the scene's pair count of this substep
// (ContactBuffer.counter).
__global__ void __launch_bounds__(1024) k_con_scan(WorldView V, uint32_t sub) {
  pdl_begin();
  __shared__ uint32_t ws[32];
  static_assert(kSegAlign == 8 * kConGroup, "segments hold whole eights of groups");
  const DevScene& S = V.scenes[blockIdx.x];
  if (!S.contact || sub >= S.substeps) return;
  const uint32_t c0 = S.seg_start / kSegAlign, c1 = S.seg_end / kSegAlign;
  const uint4* sums = reinterpret_cast<const uint4*>(V.con_sum);
  const uint4* drops = reinterpret_cast<const uint4*>(V.con_drop);
  uint4* offs = reinterpret_cast<uint4*>(V.con_off);
  uint32_t carry = 0, drop = 0;
  for (uint32_t base = c0; base < c1; base += blockDim.x) {
    const uint32_t c = base + threadIdx.x;
    uint4 a = make_uint4(0, 0, 0, 0), b = a, da = a, db = a;
    if (c < c1) {
      a = sums[2 * c];
      b = sums[2 * c + 1];
      da = drops[2 * c];
      db = drops[2 * c + 1];
    }
    uint32_t t, td;
    uint32_t at = carry + block_exclusive(a.x + a.y + a.z + a.w + b.x + b.y + b.z + b.w, ws, &t);
    (void)block_exclusive(da.x + da.y + da.z + da.w + db.x + db.y + db.z + db.w, ws, &td);
    if (c < c1) {
      const uint4 p = make_uint4(at, at + a.x, at + a.x + a.y, at + a.x + a.y + a.z);
      at = p.w + a.w;
      offs[2 * c] = p;
      offs[2 * c + 1] = make_uint4(at, at + b.x, at + b.x + b.y, at + b.x + b.y + b.z);
    }
    carry += t;
    drop += td;
  }
  if (threadIdx.x == 0) V.con_stat[blockIdx.x] = make_uint2(carry, drop);
}

// Entry m of slot k is solved when it was stored and falls inside the
// scene's first max_contacts pairs.
__device__ __forceinline__ uint32_t con_live(const WorldView& V, const DevScene& S, uint32_t k) {
  const uint32_t cnt = min(V.con_cnt[k], kMaxContacts);
  const uint32_t first = V.con_off[k / kConGroup] + V.con_pre[k];
  return first >= S.max_contacts ? 0u : min(cnt, S.max_contacts - first);
}

// The pair passes: kPairLanes lanes per slot, lane l on entries l, l +
// kPairLanes and so on of its list. A pair's multipliers and normal belong to
// its lane; the slot's own share of the corrections is summed as ticks in
// registers (whole numbers, so in any order the same) and added once. The
// solve of a pile of 50,000: 12.2 us with a thread per slot that adds every
// pair's both sides, 8.2, 6.8 and 6.9 with 2, 4 and 8 lanes.
struct PairSum {
  uint32_t x = 0, y = 0, z = 0;
  __device__ __forceinline__ void add(f3 v, float scale) {
    x += (uint32_t)to_ticks(v.x, scale);
    y += (uint32_t)to_ticks(v.y, scale);
    z += (uint32_t)to_ticks(v.z, scale);
  }
  // to be reached by every lane of the warp
  __device__ __forceinline__ void flush(int4* acc, uint32_t slot) {
#pragma unroll
    for (uint32_t d = 1; d < kPairLanes; d <<= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, d);
      y += __shfl_xor_sync(0xffffffffu, y, d);
      z += __shfl_xor_sync(0xffffffffu, z, d);
    }
    if (threadIdx.x % kPairLanes != 0 || !(x | y | z)) return;
    int* p = reinterpret_cast<int*>(acc + slot);
    atomicAdd(p + 0, (int)x);
    atomicAdd(p + 1, (int)y);
    atomicAdd(p + 2, (int)z);
  }
};
// The slot of this thread in a launch of n * kPairLanes threads.
__device__ __forceinline__ uint32_t pair_slot() {
  return blockIdx.x * (kBlock / kPairLanes) + threadIdx.x / kPairLanes;
}

// solve.ts:115-150: pairs that overlap at the start of the substep are
// separated, the change going to both the committed and the predicted
// positions (applied by k_con_apply2).
__global__ void __launch_bounds__(kBlock) k_con_stab(WorldView V, uint32_t sub) {
  pdl_begin();
  const uint32_t k = pair_slot(), lane = threadIdx.x % kPairLanes;  // the grid covers n exactly
  const DevScene& S = scene_at(V, k);
  const uint32_t live = S.contact && sub < S.substeps ? con_live(V, S, k) : 0u;
  PairSum own;
  const float4 xk = V.cur.x[k];
  const size_t n = V.n;
  for (uint32_t m = lane; m < live; m += kPairLanes) {
    const uint32_t j = V.con_nbr[m * n + k];
    const float4 xj = V.cur.x[j];
    const f3 off = xyz(xk) - xyz(xj);
    const float d = len(off);
    const float ws = xk.w + xj.w;
    if (d <= 1e-8f || d >= S.c_dist || ws <= 0.0f) continue;
    const f3 nrm = off / d;
    const float dl = (S.c_dist - d) / ws;
    own.add(nrm * (xk.w * dl), S.pos_scale);
    acc_add(V.acc_con, j, neg(nrm * (xj.w * dl)), S.pos_scale);
  }
  own.flush(V.acc_con, k);
}

// accumulator.ts:101-131 over [positions, predictedPositions] (loop.ts:393).
__global__ void __launch_bounds__(kBlock) k_con_apply2(WorldView V, uint32_t sub) {
  pdl_begin();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= V.n) return;
  const uint32_t s = scene_index(V, k);
  const DevScene& S = V.scenes[s];
  if (!S.contact || sub >= S.substeps) return;
  const int4 t = V.acc_con[k];
  if (!(t.x | t.y | t.z)) return;
  V.acc_con[k] = make_int4(0, 0, 0, 0);
  bool sat = false;
  const f3 c = ticks_change(t.x, t.y, t.z, S.pos_inv, &sat);
  const float4 x = V.cur.x[k], xs = V.cur.xs[k];
  V.cur.x[k] = with_w(xyz(x) + c, x.w);
  V.cur.xs[k] = with_w(xyz(xs) + c, xs.w);
  if (sat) atomicOr(V.flags + s * kNumFlags + FLAG_POS, 1u);
}

// solve.ts:34-104: non-penetration along the pair's normal and static
// friction inside the cone lambda_t <= mu_s lambda_n, scattered into the
// position sums that the collider pass applies.
__global__ void __launch_bounds__(kBlock) k_con_solve(WorldView V, uint32_t sub, uint32_t it) {
  pdl_begin();
  const uint32_t k = pair_slot(), lane = threadIdx.x % kPairLanes;  // the grid covers n exactly
  const DevScene& S = scene_at(V, k);
  const uint32_t live = S.contact && sub < S.substeps && it < S.iterations ? con_live(V, S, k) : 0u;
  PairSum own;
  const float4 pk = V.cur.xs[k];
  const f3 xk = xyz(pk), dk = xk - xyz(V.cur.x[k]);
  const float wk = pk.w;
  const size_t n = V.n;
  for (uint32_t m = lane; m < live; m += kPairLanes) {
    const size_t e = m * n + k;
    const uint32_t j = V.con_nbr[e];
    const float4 pj = V.cur.xs[j];
    const f3 off = xk - xyz(pj);
    const float d = len(off);
    const float wj = pj.w, ws = wk + wj;
    if (d <= 1e-8f || d >= S.c_dist || ws <= 0.0f) continue;
    const f3 nrm = off / d;
    const float dln = (S.c_dist - d) / ws;
    int2 L = V.con_lam[e];
    L.x += lam_ticks(dln);
    V.con_nrm[e] = with_w(nrm, 0.0f);
    const f3 slip = dk - (xyz(pj) - xyz(V.cur.x[j]));
    const f3 tang = slip - nrm * dot(slip, nrm);
    const float tl = len(tang);
    const float ln = (float)L.x * kLambdaInv, lt = (float)L.y * kLambdaInv;
    const float dlt = tl / ws;
    const bool sticks = tl > 1e-10f && dlt <= S.c_mus * ln - lt;
    const f3 ni = nrm * (wk * dln), nj = neg(nrm * (wj * dln));
    own.add(sticks ? ni + neg(tang * (wk / ws)) : ni, S.pos_scale);
    acc_add(V.acc_con, j, sticks ? nj + tang * (wj / ws) : nj, S.pos_scale);
    L.y += lam_ticks(sticks ? dlt : 0.0f);
    V.con_lam[e] = L;
  }
  own.flush(V.acc_con, k);
}

// solve.ts:158-189: kinetic friction, the tangential relative velocity
// reduced by at most mu_k lambda_n / dt, into the velocity sums that the
// friction pass applies.
__global__ void __launch_bounds__(kBlock) k_con_friction(WorldView V, uint32_t sub) {
  pdl_begin();
  const uint32_t k = pair_slot(), lane = threadIdx.x % kPairLanes;  // the grid covers n exactly
  const DevScene& S = scene_at(V, k);
  const uint32_t live = S.contact && sub < S.substeps ? con_live(V, S, k) : 0u;
  PairSum own;
  const float wk = V.cur.x[k].w;
  const f3 vk = xyz(V.cur.v[k]);
  const size_t n = V.n;
  for (uint32_t m = lane; m < live; m += kPairLanes) {
    const size_t e = m * n + k;
    const uint32_t j = V.con_nbr[e];
    const float wj = V.cur.x[j].w, ws = wk + wj;
    const float ln = (float)V.con_lam[e].x * kLambdaInv;
    if (ws <= 0.0f || ln <= 0.0f) continue;
    const f3 nrm = xyz(V.con_nrm[e]);
    const f3 v = vk - xyz(V.cur.v[j]);
    const f3 vt = v - nrm * dot(nrm, v);
    const float vtl = len(vt);
    if (vtl < 1e-6f) continue;
    const float change = fminf(S.c_muk * ln * ws / S.dt, vtl);
    const f3 imp = neg((vt / vtl) * change) / ws;
    own.add(imp * wk, S.vel_scale);
    acc_add(V.acc_con, j, neg(imp * wj), S.vel_scale);
  }
  own.flush(V.acc_con, k);
}

}  // namespace pf
