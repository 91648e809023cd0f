// Barnes-Hut forces and potentials on the GPU octree.
//
// Monopoles (barnes-hut.cc:76-159): every node keeps the positive charge sum
// and the |negative| charge sum with their charge centres; leaves sum their
// particles, internal nodes merge their children in octant order (one launch:
// the thread whose child arrives last at a node merges it).
//
// Walk (barnes-hut.cc:183-269): a warp takes 32 consecutive targets in tree
// order and walks one shared stack of nodes to open. Each entry carries the
// mask of lanes that open that node; the node's children are tested there and
// then. A lane accepts an internal node when (2h)^2 < theta^2 |x - c|^2 (the
// reference's test, evaluated in FP64 without contraction, so the
// accepted-node set of every target is the reference's); accepting lanes add
// the two monopoles, for the others the child goes on the stack. Leaves are
// summed directly, skipping the target itself and q = 0 sources. Pairs closer than 1e-30 m^2 are skipped
// (barnes-hut.cc:33-41). All arithmetic is FP64 (leaf sums FP32 in the
// tensor precision mode, below); inverse distances are reciprocal square
// roots where the reference divides by sqrt (an ulp-level difference).
//
// The walk is bound by the latency of the node loads, not by its arithmetic,
// so the records of a node's children (128 bytes each) lie side by side and
// the warp copies them into shared memory with two loads per opened node: one
// memory latency per up to eight tests. (A node popped and read at a time:
// 3.75 ms at 524,309 particles, theta = 0.7, with its loads one after the
// other, 3.0 ms with them together, FP64 pipe at 36 and 42 %.) A block is two
// warps, since walks differ in length.
#include <algorithm>
#include <vector>

#include "amk_internal.cuh"

namespace amk {
namespace {

constexpr int kWalkWarps = 2;
constexpr int kStack = 176;  // >= 1 + 7 * 21 + 8 nodes to open

__device__ __forceinline__ double dot_rn(double a, double b, double c) {
  // ((0 + a*a) + b*b) + c*c without contraction (the reference's Real3 dot)
  return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
}

// Another block's store, read past this SM's L1.
__device__ __forceinline__ double4 load_cg(const double4* p) {
  const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// BH node charges: pos = (Q+, centre+), neg = (|Q-|, centre-). One launch from
// the leaves to the root: a thread per leaf sums its particles, then the thread
// whose child arrives last at a parent merges the children in octant order;
// no thread waits for another. A launch per level over all nodes took 120 us
// (524k particles, 11 levels), this 67 us.
__global__ void bh_monopole_kernel(const Octree t, int* __restrict__ arrived, double4* __restrict__ pos,
                                   double4* __restrict__ neg) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= t.n_nodes) return;
  if (!t.meta[id].y) return;
  const int2 r = t.range[id];
  double qp = 0.0, qn = 0.0, mp[3] = {0.0, 0.0, 0.0}, mn[3] = {0.0, 0.0, 0.0};
  for (int k = r.x; k < r.y; ++k) {
    const double4 s = t.src[k];
    if (s.w > 0.0) {
      qp += s.w;
      mp[0] = __dadd_rn(mp[0], __dmul_rn(s.x, s.w));
      mp[1] = __dadd_rn(mp[1], __dmul_rn(s.y, s.w));
      mp[2] = __dadd_rn(mp[2], __dmul_rn(s.z, s.w));
    } else if (s.w < 0.0) {
      qn += -s.w;
      mn[0] = __dadd_rn(mn[0], __dmul_rn(s.x, -s.w));
      mn[1] = __dadd_rn(mn[1], __dmul_rn(s.y, -s.w));
      mn[2] = __dadd_rn(mn[2], __dmul_rn(s.z, -s.w));
    }
  }
  const double4 c = t.center[id];
  pos[id] = qp > 0.0 ? make_double4(mp[0] * (1.0 / qp), mp[1] * (1.0 / qp), mp[2] * (1.0 / qp), qp)
                     : make_double4(c.x, c.y, c.z, 0.0);
  neg[id] = qn > 0.0 ? make_double4(mn[0] * (1.0 / qn), mn[1] * (1.0 / qn), mn[2] * (1.0 / qn), qn)
                     : make_double4(c.x, c.y, c.z, 0.0);
  for (int par = t.parent[id]; par >= 0; par = t.parent[par]) {
    const int4* cp = reinterpret_cast<const int4*>(t.child + 8 * static_cast<size_t>(par));
    const int4 c0 = cp[0], c1 = cp[1];
    const int ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    int children = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o) children += ch[o] >= 0;
    __threadfence();  // this node's charges, before its arrival
    if (atomicAdd(&arrived[par], 1) != children - 1) return;
    __threadfence();
    double4 a[8], b[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      a[o] = b[o] = make_double4(0.0, 0.0, 0.0, 0.0);
      if (ch[o] >= 0) {
        a[o] = load_cg(&pos[ch[o]]);
        b[o] = load_cg(&neg[ch[o]]);
      }
    }
    qp = qn = 0.0;
    mp[0] = mp[1] = mp[2] = mn[0] = mn[1] = mn[2] = 0.0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      if (a[o].w > 0.0) {
        qp += a[o].w;
        mp[0] = __dadd_rn(mp[0], __dmul_rn(a[o].x, a[o].w));
        mp[1] = __dadd_rn(mp[1], __dmul_rn(a[o].y, a[o].w));
        mp[2] = __dadd_rn(mp[2], __dmul_rn(a[o].z, a[o].w));
      }
      if (b[o].w > 0.0) {
        qn += b[o].w;
        mn[0] = __dadd_rn(mn[0], __dmul_rn(b[o].x, b[o].w));
        mn[1] = __dadd_rn(mn[1], __dmul_rn(b[o].y, b[o].w));
        mn[2] = __dadd_rn(mn[2], __dmul_rn(b[o].z, b[o].w));
      }
    }
    const double4 pc = t.center[par];
    pos[par] = qp > 0.0 ? make_double4(mp[0] * (1.0 / qp), mp[1] * (1.0 / qp), mp[2] * (1.0 / qp), qp)
                        : make_double4(pc.x, pc.y, pc.z, 0.0);
    neg[par] = qn > 0.0 ? make_double4(mn[0] * (1.0 / qn), mn[1] * (1.0 / qn), mn[2] * (1.0 / qn), qn)
                        : make_double4(pc.x, pc.y, pc.z, 0.0);
  }
}

// What the walk reads of a node.
struct __align__(128) BhRec {
  double4 c;    // centre, half edge
  double4 pos;  // positive charge centre and sum
  double4 neg;  // |negative| charge centre and sum
  int4 info;    // internal: first child's record, children, 0; leaf: particles [x, y), 1
  int4 pad;
};
static_assert(sizeof(BhRec) == 128, "eight 16-byte pieces");

__global__ void bh_child_count_kernel(const Octree t, int* __restrict__ n_child) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= t.n_nodes) return;
  const int4* c = reinterpret_cast<const int4*>(t.child + 8 * static_cast<size_t>(id));
  const int4 a = c[0], b = c[1];
  n_child[id] = (a.x >= 0) + (a.y >= 0) + (a.z >= 0) + (a.w >= 0) + (b.x >= 0) + (b.y >= 0) + (b.z >= 0) + (b.w >= 0);
}

// Records grouped by parent: the children of node p (octant order) at
// first[p], first[p] + 1, ...; the root's record is the last one. Eight
// threads per parent.
__global__ void bh_record_kernel(const Octree t, const int* __restrict__ n_child, const int* __restrict__ first,
                                 const double4* __restrict__ pos, const double4* __restrict__ neg,
                                 BhRec* __restrict__ rec) {
  const long x = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  const long p = x >> 3;
  const int o = static_cast<int>(x & 7), lane = threadIdx.x & 31;
  const int id = p < t.n_nodes ? t.child[x] : -1;
  const unsigned has = __ballot_sync(0xffffffffu, id >= 0);
  long at = 0;
  if (id >= 0) {
    const unsigned mine = (has >> (lane & 24)) & 0xffu;
    at = first[p] + __popc(mine & ((1u << o) - 1u));
  }
  auto put = [&](int node, long slot) {
    const int2 r = t.range[node];
    BhRec* d = rec + slot;
    d->c = t.center[node];
    d->pos = pos[node];
    d->neg = neg[node];
    d->info = t.meta[node].y ? make_int4(r.x, r.y, 1, 0) : make_int4(first[node], n_child[node], 0, 0);
  };
  if (id >= 0) put(id, at);
  if (x == 0) put(0, t.n_nodes - 1);
}

// 1 / r of a pair, 0 below the minimum distance and (kWide: a root cube of more
// than 1e150 m) where r^2 overflowed: the pull of a finite particle that far
// away rounds to nothing, and rsqrt_f64 has no value for infinity. The second
// test costs the walk 0.8 %, so other trees go without it.
template <bool kWide>
__device__ __forceinline__ double inverse_distance(double d2, bool skip) {
  return skip || d2 < kMinSquaredDistance || (kWide && isinf(d2)) ? 0.0 : rsqrt_f64(d2);
}

// AddPointCharge, barnes-hut.cc:20-28, without the factor k q_t:
// f += r q_s / r^3; pairs without an inverse distance (and `skip`) add 0.
template <bool kWide>
__device__ __forceinline__ void add_point(double rx, double ry, double rz, double d2, double sq, bool skip,
                                          double* f) {
  const double inv = inverse_distance<kWide>(d2, skip);
  const double w = sq * (inv * inv * inv);
  f[0] += rx * w;
  f[1] += ry * w;
  f[2] += rz * w;
}

template <bool kWide>
__device__ __forceinline__ void add_phi(double d2, double sq, bool skip, double* phi) {
  *phi += sq * inverse_distance<kWide>(d2, skip);
}

// Leaf sums in FP32 (the tensor precision mode): sources as double-float
// pairs x = hi + lo (hi = float(x), lo = float(x - hi)) relative to the
// tree frame; a pair's difference (x_i,hi - x_j,hi) + (x_i,lo - x_j,lo) is
// exact to FP32 rounding of |r| for particles of neighbouring cells
// (Sterbenz), the per-leaf sums of q_j r / r^3 are FP32 and are added to the
// FP64 accumulators once per leaf. The opening test and the node monopoles
// stay FP64, so the accepted-node sets are the reference's.
struct BhF32 {
  const float4* hi;  // (x, y, z, q) hi parts, q as float
  const float4* lo;  // lo parts
  double qs;         // charges were divided by this before the float conversion
};

__global__ void bh_stage_kernel(const Octree t, double qs, float4* __restrict__ hi, float4* __restrict__ lo) {
  const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (k >= t.m) return;
  const double4 s = t.src[k];
  const float hx = static_cast<float>(s.x), hy = static_cast<float>(s.y), hz = static_cast<float>(s.z);
  hi[k] = make_float4(hx, hy, hz, static_cast<float>(s.w / qs));
  lo[k] = make_float4(static_cast<float>(s.x - hx), static_cast<float>(s.y - hy), static_cast<float>(s.z - hz), 0.f);
}

template <bool kPhi, bool kF32, bool kWide>
__global__ void __launch_bounds__(32 * kWalkWarps)
bh_walk_kernel(const Octree t, const BhRec* __restrict__ rec, double theta2, BhF32 f32, double* __restrict__ out,
               int* __restrict__ status) {
  __shared__ BhRec s_rec[kWalkWarps][8];
  __shared__ int s_first[kWalkWarps][kStack];
  __shared__ int s_count[kWalkWarps][kStack];
  __shared__ unsigned s_mask[kWalkWarps][kStack];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long k = (static_cast<long>(blockIdx.x) * kWalkWarps + w) * 32 + lane;
  const bool valid = k < t.m;
  double4 me = make_double4(0.0, 0.0, 0.0, 0.0);
  if (valid) me = t.src[k];
  // ComputeForce returns 0 for q = 0 (barnes-hut.cc:169); potentials walk anyway
  const bool want = valid && (kPhi || me.w != 0.0);
  const unsigned lanes = __ballot_sync(0xffffffffu, want);
  double f[3] = {0.0, 0.0, 0.0};
  double phi = 0.0;
  int sp = 0;
  if (lanes) {
    if (lane == 0) {
      s_first[w][0] = static_cast<int>(t.n_nodes) - 1;  // the root's record
      s_count[w][0] = 1;
      s_mask[w][0] = lanes;
    }
    sp = 1;
  }
  const BhRec* child = s_rec[w];
  while (sp > 0) {
    __syncwarp();  // the last node's records have been read, its pushes are complete
    --sp;
    const int first = s_first[w][sp], n = s_count[w][sp];
    const unsigned mask = s_mask[w][sp];
    const bool act = (mask >> lane) & 1u;
    const float4* from = reinterpret_cast<const float4*>(rec + first);
    float4* to = reinterpret_cast<float4*>(s_rec[w]);
    if (lane < 8 * n) to[lane] = from[lane];
    if (lane + 32 < 8 * n) to[lane + 32] = from[lane + 32];
    __syncwarp();
    for (int o = 0; o < n; ++o) {
      const int4 in = child[o].info;
      const double pw = child[o].pos.w, nw = child[o].neg.w;
      if (pw == 0.0 && nw == 0.0) continue;  // barnes-hut.cc:186
      if (in.z) {
        if (kF32) {
          if (act) {
            // sum over the leaf of (q_j / qs) r / r^3 (or / r) in FP32
            const float4 mh = f32.hi[k], ml = f32.lo[k];
            const float min_sq = 1e-30f;  // kMinSquaredDistance (m^2), a normal float
            float ax = 0.f, ay = 0.f, az = 0.f, ap = 0.f;
            for (int j = in.x; j < in.y; ++j) {
              const float4 s = f32.hi[j], q = f32.lo[j];
              const float rx = fmaf(s.x, -1.f, mh.x) + fmaf(q.x, -1.f, ml.x);
              const float ry = fmaf(s.y, -1.f, mh.y) + fmaf(q.y, -1.f, ml.y);
              const float rz = fmaf(s.z, -1.f, mh.z) + fmaf(q.z, -1.f, ml.z);
              const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
              // the target itself (r = 0), closer pairs and neutral sources add zero
              const float inv = (j != k && r2 >= min_sq) ? rsqrtf(r2) : 0.f;
              const float qr = s.w * inv;
              if (kPhi) {
                ap += qr;
              } else {
                const float wt = qr * (inv * inv);
                ax = fmaf(rx, wt, ax);
                ay = fmaf(ry, wt, ay);
                az = fmaf(rz, wt, az);
              }
            }
            if (kPhi) {
              phi += f32.qs * static_cast<double>(ap);
            } else {
              f[0] += f32.qs * static_cast<double>(ax);
              f[1] += f32.qs * static_cast<double>(ay);
              f[2] += f32.qs * static_cast<double>(az);
            }
          }
        } else if (act) {
#pragma unroll 4
          for (int j = in.x; j < in.y; ++j) {
            const double4 s = t.src[j];
            const double rx = me.x - s.x, ry = me.y - s.y, rz = me.z - s.z;
            const double d2 = dot_rn(rx, ry, rz);
            if (kPhi)
              add_phi<kWide>(d2, s.w, j == k, &phi);
            else
              add_point<kWide>(rx, ry, rz, d2, s.w, j == k, f);
          }
        }
        continue;
      }
      const double4 c = child[o].c;
      const double dx = me.x - c.x, dy = me.y - c.y, dz = me.z - c.z;
      const double d2 = dot_rn(dx, dy, dz);
      const double width = 2.0 * c.w;
      const bool accept = act && (__dmul_rn(width, width) < __dmul_rn(theta2, d2));
      const unsigned acc = __ballot_sync(0xffffffffu, accept);
      if (accept) {
        if (pw > 0.0) {
          const double4 pq = child[o].pos;
          const double rx = me.x - pq.x, ry = me.y - pq.y, rz = me.z - pq.z;
          const double r2 = dot_rn(rx, ry, rz);
          if (kPhi)
            add_phi<kWide>(r2, pw, false, &phi);
          else
            add_point<kWide>(rx, ry, rz, r2, pw, false, f);
        }
        if (nw > 0.0) {
          const double4 nq = child[o].neg;
          const double rx = me.x - nq.x, ry = me.y - nq.y, rz = me.z - nq.z;
          const double r2 = dot_rn(rx, ry, rz);
          if (kPhi)
            add_phi<kWide>(r2, -nw, false, &phi);
          else
            add_point<kWide>(rx, ry, rz, r2, -nw, false, f);
        }
      }
      const unsigned open = mask & ~acc;
      if (open) {
        if (sp >= kStack) {  // cannot happen for depth <= 21; guarded anyway
          if (lane == 0) atomicExch(status, 1);
          sp = 0;
          break;
        }
        if (lane == 0) {
          s_first[w][sp] = in.x;
          s_count[w][sp] = in.y;
          s_mask[w][sp] = open;
        }
        ++sp;
      }
    }
  }
  if (valid) {
    if (kPhi) {
      out[k] = phi;
    } else {
      const double sc = kCoulombConstant * me.w;
      out[3 * k + 0] = sc * f[0];
      out[3 * k + 1] = sc * f[1];
      out[3 * k + 2] = sc * f[2];
    }
  }
}

__global__ void bh_scatter_kernel(const Octree t, const double* __restrict__ fo, const double* __restrict__ po,
                                  View v) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= t.m) return;
  const long i = t.order[k];
  if (fo) {
    v.fx[i] = fo[3 * k + 0];
    v.fy[i] = fo[3 * k + 1];
    v.fz[i] = fo[3 * k + 2];
  }
  if (po && v.phi) v.phi[i] = po[k];
}

__global__ void zero_outputs_kernel(View v, bool forces) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= v.n) return;
  if (forces) {
    v.fx[i] = 0.0;
    v.fy[i] = 0.0;
    v.fz[i] = 0.0;
  }
  if (v.phi) v.phi[i] = 0.0;
}

int bh_monopoles(amk_ctx* c, const Octree& t, double4** pos_out, double4** neg_out) {
  int rc = AMK_OK;
  double4* pos = slot<double4>(c, kSlotBhPos, t.n_nodes, &rc);
  AMK_TRY(rc);
  double4* neg = slot<double4>(c, kSlotBhNeg, t.n_nodes, &rc);
  AMK_TRY(rc);
  int* arrived = slot<int>(c, kSlotBhArrived, t.n_nodes, &rc);
  AMK_TRY(rc);
  AMK_CUDA_TRY(cudaMemsetAsync(arrived, 0, static_cast<size_t>(t.n_nodes) * sizeof(int), c->stream));
  bh_monopole_kernel<<<static_cast<unsigned>((t.n_nodes + 127) / 128), 128, 0, c->stream>>>(t, arrived, pos, neg);
  AMK_TRY(check_launch(c, "bh_monopole_kernel"));
  *pos_out = pos;
  *neg_out = neg;
  return AMK_OK;
}

}  // namespace

int barnes_hut_forces(amk_ctx* c, const View& v, double theta, long leaf_capacity) {
  const long n = v.n;
  if (n == 0) return AMK_OK;
  zero_outputs_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, c->stream>>>(v, true);
  AMK_TRY(check_launch(c, "zero_outputs_kernel"));
  Octree t;
  AMK_TRY(phase_begin(c, AMK_PHASE_TREE));
  AMK_TRY(build_octree(c, v, static_cast<int>(std::min<long>(leaf_capacity, 1 << 20)), 0, &t));
  if (t.m == 0) return phase_end(c, AMK_PHASE_TREE);
  double4 *pos = nullptr, *neg = nullptr;
  AMK_TRY(bh_monopoles(c, t, &pos, &neg));
  AMK_TRY(phase_end(c, AMK_PHASE_TREE));
  int rc = AMK_OK;
  double* fo = slot<double>(c, kSlotWalkOut, 3 * static_cast<size_t>(t.m), &rc);
  AMK_TRY(rc);
  double* po = v.phi ? slot<double>(c, kSlotFmmWork5, static_cast<size_t>(t.m), &rc) : nullptr;
  AMK_TRY(rc);
  int* status = slot<int>(c, kSlotStatus, 8, &rc) + 4;
  AMK_TRY(rc);
  AMK_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), c->stream));
  BhRec* rec = slot<BhRec>(c, kSlotBhRec, t.n_nodes, &rc);
  AMK_TRY(rc);
  int* n_child = slot<int>(c, kSlotTreeCount, t.n_nodes, &rc);  // tree build scratch, free again
  AMK_TRY(rc);
  int* first = slot<int>(c, kSlotTreeBase, t.n_nodes + 1, &rc);
  AMK_TRY(rc);
  bh_child_count_kernel<<<static_cast<unsigned>((t.n_nodes + 255) / 256), 256, 0, c->stream>>>(t, n_child);
  AMK_TRY(check_launch(c, "bh_child_count_kernel"));
  AMK_TRY(exclusive_scan_int(c, n_child, t.n_nodes, first, first + t.n_nodes));
  bh_record_kernel<<<static_cast<unsigned>((8 * t.n_nodes + 255) / 256), 256, 0, c->stream>>>(t, n_child, first, pos,
                                                                                             neg, rec);
  AMK_TRY(check_launch(c, "bh_record_kernel"));
  const unsigned blocks = static_cast<unsigned>((t.m + 32 * kWalkWarps - 1) / (32 * kWalkWarps));
  const double theta2 = theta * theta;  // squared_theta_, barnes-hut.cc:36
  const bool f32 = c->fmm_precision == AMK_FMM_TENSOR;
  BhF32 fs{nullptr, nullptr, kElementaryCharge};
  if (f32) {  // sources as double-float pairs, charges in units of e
    float4* stage = slot<float4>(c, kSlotP2PStage, 2 * static_cast<size_t>(t.m), &rc);
    AMK_TRY(rc);
    bh_stage_kernel<<<static_cast<unsigned>((t.m + 255) / 256), 256, 0, c->stream>>>(t, fs.qs, stage, stage + t.m);
    AMK_TRY(check_launch(c, "bh_stage_kernel"));
    fs.hi = stage;
    fs.lo = stage + t.m;
  }
  AMK_TRY(phase_begin(c, AMK_PHASE_BH_WALK));
  auto walk = [&](auto kernel, double* out) -> int {
    kernel<<<blocks, 32 * kWalkWarps, 0, c->stream>>>(t, rec, theta2, fs, out, status);
    return check_launch(c, "bh_walk_kernel");
  };
  if (f32)
    AMK_TRY(walk(t.wide ? bh_walk_kernel<false, true, true> : bh_walk_kernel<false, true, false>, fo));
  else
    AMK_TRY(walk(t.wide ? bh_walk_kernel<false, false, true> : bh_walk_kernel<false, false, false>, fo));
  if (po) {
    if (f32)
      AMK_TRY(walk(t.wide ? bh_walk_kernel<true, true, true> : bh_walk_kernel<true, true, false>, po));
    else
      AMK_TRY(walk(t.wide ? bh_walk_kernel<true, false, true> : bh_walk_kernel<true, false, false>, po));
  }
  AMK_TRY(phase_end(c, AMK_PHASE_BH_WALK));
  bh_scatter_kernel<<<static_cast<unsigned>((t.m + 255) / 256), 256, 0, c->stream>>>(t, fo, po, v);
  AMK_TRY(check_launch(c, "bh_scatter_kernel"));
  int st = 0;
  AMK_CUDA_TRY(cudaMemcpyAsync(&st, status, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  if (st) return fail(AMK_ERR_LIMIT, "Barnes-Hut walk stack exceeded %d entries", kStack);
  return AMK_OK;
}

}  // namespace amk

using namespace amk;

// Tree introspection for tests: node arrays in the reference's layout
// (BarnesHutTree::Node, barnes-hut.h:49-61).
extern "C" long amk_bh_tree_dump(amk_ctx* c, long n, const double* x, const double* y, const double* z,
                                 const double* q, long leaf_capacity, long max_nodes, double* node_f64,
                                 long* node_i64) {
  if (!c || n < 0) return fail(AMK_ERR_INVALID, "bad argument");
  if (n == 0) return 0;
  View v;
  AMK_TRY(load_aux_view(c, n, x, y, z, q, &v));
  Octree t;
  AMK_TRY(build_octree(c, v, static_cast<int>(leaf_capacity), 0, &t));
  if (t.n_nodes > max_nodes) return fail(AMK_ERR_LIMIT, "tree has %ld nodes, buffer holds %ld", t.n_nodes, max_nodes);
  double4 *pos = nullptr, *neg = nullptr;
  AMK_TRY(bh_monopoles(c, t, &pos, &neg));
  const long nn = t.n_nodes;
  std::vector<double4> hc(nn), hp(nn), hn(nn);
  std::vector<int> hch(8 * nn);
  std::vector<int2> hr(nn);
  std::vector<uchar2> hm(nn);
  AMK_CUDA_TRY(cudaMemcpyAsync(hc.data(), t.center, nn * sizeof(double4), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(hp.data(), pos, nn * sizeof(double4), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(hn.data(), neg, nn * sizeof(double4), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(hch.data(), t.child, 8 * nn * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(hr.data(), t.range, nn * sizeof(int2), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(hm.data(), t.meta, nn * sizeof(uchar2), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  for (long k = 0; k < nn; ++k) {
    double* f = node_f64 + 12 * k;
    f[0] = hc[k].x;
    f[1] = hc[k].y;
    f[2] = hc[k].z;
    f[3] = hc[k].w;
    f[4] = hp[k].w;
    f[5] = hn[k].w;
    f[6] = hp[k].x;
    f[7] = hp[k].y;
    f[8] = hp[k].z;
    f[9] = hn[k].x;
    f[10] = hn[k].y;
    f[11] = hn[k].z;
    long* g = node_i64 + 11 * k;
    for (int o = 0; o < 8; ++o) g[o] = hch[8 * k + o];
    g[8] = hr[k].x;
    g[9] = hr[k].y;
    g[10] = hm[k].y;
  }
  return nn;
}
