// Pairs closer than a radius, and the two behaviours that walk them:
//   * the cutoff direct sum of ComputeStandardCoulombForces
//     (interaction/coulomb_interaction.cc:23-80) with the shifted-cutoff pair
//     energy of ComputeStandardEnergy (analysis/energy_analysis.cc:16-43);
//   * the annihilation contact search of AnnihilationInteraction::Run
//     (interaction/annihilation.cc:21-61), made deterministic: candidate
//     directed contacts (owner -> partner) with a Philox draw below p are
//     matched greedily in ascending (owner id, partner id) order, which is
//     the result of visiting owners one at a time in id order. The greedy
//     matching is computed in parallel by repeatedly selecting every contact
//     that has the smallest priority at both of its endpoints.
// Pair geometry is FP64 with contraction-free arithmetic so that contact
// decisions are bit-identical to a scalar FP64 evaluation.
//
// Up to kBruteMax particles every pair is tested (one launch, no list). Above
// it the particles are binned into cells no smaller than the radius: a dense
// grid over their bounding box, x fastest, so that the 27 neighbour cells of a
// particle are nine contiguous runs of the sorted records, or, where the box is
// too large for that (a sparse cloud, particles far from the others), hashed
// cells. A counting sort with four counters per particle builds either (count,
// scan, scatter; a counter's members ordered by particle index, so sums have a
// fixed order).
// The allocation-free solver keeps its Morton-sorted keys: its static scratch
// has no room for the grid's counters.
#include <algorithm>

#include "amk_internal.cuh"
#include "bbox.cuh"
#include "contacts.cuh"
#include "philox.cuh"

namespace amk {
namespace {

constexpr uint64_t kDeadKey = ~0ull;
constexpr int kCellBits = 21;
constexpr double kCellMax = 2097150.0;  // 2^21 - 2

__device__ __forceinline__ bool usable(const View& v, long i) {
  return (v.alive == nullptr || v.alive[i]) && isfinite(v.x[i]) && isfinite(v.y[i]) && isfinite(v.z[i]);
}

__global__ void __launch_bounds__(kBboxThreads) bbox_kernel(View v, unsigned long long* bb) {
  bbox_block(v, [&](long i) { return usable(v, i); }, bb);
}

struct Grid {
  double ox, oy, oz, inv_cs;
  uint32_t nmax;  // largest valid cell coordinate
};

__device__ __forceinline__ Grid grid_from(const unsigned long long* bb, double radius) {
  Grid g;
  const double lo0 = double_from_order_bits(bb[0]), lo1 = double_from_order_bits(bb[1]), lo2 = double_from_order_bits(bb[2]);
  const double hi0 = -double_from_order_bits(bb[3]), hi1 = -double_from_order_bits(bb[4]), hi2 = -double_from_order_bits(bb[5]);
  double ext = fmax(hi0 - lo0, fmax(hi1 - lo1, hi2 - lo2));
  if (!(ext >= 0.0)) ext = 0.0;  // no live particle
  double cs = radius * (1.0 + 1e-9);
  cs = fmax(cs, ext / kCellMax);
  if (!(cs > 0.0)) cs = 1.0;
  g.ox = isfinite(lo0) ? lo0 : 0.0;
  g.oy = isfinite(lo1) ? lo1 : 0.0;
  g.oz = isfinite(lo2) ? lo2 : 0.0;
  g.inv_cs = 1.0 / cs;
  g.nmax = (1u << kCellBits) - 1u;
  return g;
}

__device__ __forceinline__ void cell_of(const Grid& g, double x, double y, double z, int c[3]) {
  c[0] = static_cast<int>(fmin(floor((x - g.ox) * g.inv_cs), static_cast<double>(g.nmax)));
  c[1] = static_cast<int>(fmin(floor((y - g.oy) * g.inv_cs), static_cast<double>(g.nmax)));
  c[2] = static_cast<int>(fmin(floor((z - g.oz) * g.inv_cs), static_cast<double>(g.nmax)));
  c[0] = max(c[0], 0);
  c[1] = max(c[1], 0);
  c[2] = max(c[2], 0);
}

__global__ void cell_key_kernel(View v, const unsigned long long* bb, double radius, uint64_t* keys,
                                uint32_t* vals) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= v.n) return;
  vals[i] = static_cast<uint32_t>(i);
  if (!usable(v, i)) {
    keys[i] = kDeadKey;
    return;
  }
  const Grid g = grid_from(bb, radius);
  int c[3];
  cell_of(g, v.x[i], v.y[i], v.z[i], c);
  keys[i] = morton3_21(c[0], c[1], c[2]);
}

__device__ __forceinline__ long lower_bound(const uint64_t* keys, long n, uint64_t k) {
  long lo = 0, hi = n;
  while (lo < hi) {
    const long mid = (lo + hi) >> 1;
    if (keys[mid] < k)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ double dist2_exact(double rx, double ry, double rz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(rx, rx), __dmul_rn(ry, ry)), __dmul_rn(rz, rz));
}

// Allocation-free solver: one thread per particle of the Morton-sorted keys.
__global__ void __launch_bounds__(128)
cutoff_kernel(View v, const unsigned long long* bb, double rc, const uint64_t* __restrict__ skeys,
              const uint32_t* __restrict__ sidx) {
  const long s = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (s >= v.n) return;
  const long i = sidx[s];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  const double qi = v.q[i];
  if (skeys[s] != kDeadKey && qi != 0.0) {
    const Grid g = grid_from(bb, rc);
    const double xi = v.x[i], yi = v.y[i], zi = v.z[i];
    int c[3];
    cell_of(g, xi, yi, zi, c);
    const double rc2 = rc * rc;
    for (int dz = -1; dz <= 1; ++dz) {
      const int cz = c[2] + dz;
      if (cz < 0 || cz > static_cast<int>(g.nmax)) continue;
      for (int dy = -1; dy <= 1; ++dy) {
        const int cy = c[1] + dy;
        if (cy < 0 || cy > static_cast<int>(g.nmax)) continue;
        for (int dx = -1; dx <= 1; ++dx) {
          const int cx = c[0] + dx;
          if (cx < 0 || cx > static_cast<int>(g.nmax)) continue;
          const uint64_t key = morton3_21(cx, cy, cz);
          for (long k = lower_bound(skeys, v.n, key); k < v.n && skeys[k] == key; ++k) {
            const long j = sidx[k];
            if (j == i) continue;
            const double qj = v.q[j];
            if (qj == 0.0) continue;
            const double rx = xi - v.x[j], ry = yi - v.y[j], rz = zi - v.z[j];
            const double d2 = dist2_exact(rx, ry, rz);
            if (d2 < kMinSquaredDistance) continue;
            if (d2 < rc2) {  // coulomb_interaction.cc:60-73
              const double dist = sqrt(d2);
              const double mag = kCoulombConstant * qi * qj / d2;
              const double w = mag / dist;
              fx += rx * w;
              fy += ry * w;
              fz += rz * w;
            }
          }
        }
      }
    }
  }
  v.fx[i] = fx;
  v.fy[i] = fy;
  v.fz[i] = fz;
}

__global__ void zero_forces_kernel(View v) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= v.n) return;
  v.fx[i] = 0.0;
  v.fy[i] = 0.0;
  v.fz[i] = 0.0;
}

// ---------------------------------------------------------------- all pairs
// Small sets: every pair, kBruteLanes lanes per target over the sources
// staged in shared memory 256 at a time; the lanes' sums are added by a
// shuffle tree (a fixed order).
constexpr int kBruteLanes = 32;
constexpr int kBruteThreads = 256;
constexpr int kBruteTile = 256;
// Pairs are tested all against all up to this many particles. us per step of
// a mixed cloud (cutoff + push + cooling + annihilation), all pairs / grid,
// with 1, 20 and 200 neighbours inside the cutoff: 200 particles 24/24/25 and
// 72/83/80, 1,024 39/42/42 and 86/108/143, 2,048 87/94/95 and 166/190/234,
// 4,096 159/154/136 and 183/204/254, 6,000 362/327/220 and 187/210/267. (With
// radix-sorted Morton cells and a binary search per neighbour cell: 340 us at
// 200 particles, 880 us at 100,000, of which the two 8-pass sorts were 600;
// the grid takes 220 us there.)
constexpr long kBruteMax = 4096;

inline unsigned brute_grid(long n, int threads) {
  const long per = threads / kBruteLanes;
  return static_cast<unsigned>((n + per - 1) / per);
}

// One pair of the cutoff sum: field and (kEnergy) shifted potential of a
// charge qj at distance^2 d2 (coulomb_interaction.cc:60-73,
// energy_analysis.cc:30-40), without k q_i.
template <bool kEnergy>
__device__ __forceinline__ void cutoff_pair(double rx, double ry, double rz, double qj, double rc2, double inv_rc,
                                            double f[3], double& e) {
  const double d2 = dist2_exact(rx, ry, rz);
  if (d2 > rc2 || d2 < kMinSquaredDistance) return;
  const double inv = rsqrt(d2);
  if (kEnergy) e += qj * (inv - inv_rc);
  if (d2 < rc2) {
    const double w = qj * (inv * inv * inv);
    f[0] += rx * w;
    f[1] += ry * w;
    f[2] += rz * w;
  }
}

template <bool kEnergy>
__device__ __forceinline__ void cutoff_store(const View& v, long i, double qi, const double f[3], double e,
                                             double* __restrict__ epart) {
  const double c = kCoulombConstant * qi;
  v.fx[i] = c * f[0];
  v.fy[i] = c * f[1];
  v.fz[i] = c * f[2];
  if (kEnergy) epart[i] = qi * e;
}

template <bool kEnergy>
__global__ void __launch_bounds__(kBruteThreads)
cutoff_brute_kernel(View v, double rc, double* __restrict__ epart) {
  __shared__ double4 tile[kBruteTile];
  const int sub = threadIdx.x % kBruteLanes;
  const long i = (blockIdx.x * static_cast<long>(kBruteThreads) + threadIdx.x) / kBruteLanes;
  const bool live = i < v.n && usable(v, i) && v.q[i] != 0.0;
  const double xi = live ? v.x[i] : 0.0, yi = live ? v.y[i] : 0.0, zi = live ? v.z[i] : 0.0;
  const double rc2 = rc * rc, inv_rc = 1.0 / rc;
  double f[3] = {0.0, 0.0, 0.0}, e = 0.0;
  for (long j0 = 0; j0 < v.n; j0 += kBruteTile) {
    __syncthreads();
    const long j = j0 + threadIdx.x;
    tile[threadIdx.x] = j < v.n && usable(v, j) ? make_double4(v.x[j], v.y[j], v.z[j], v.q[j])
                                                : make_double4(0.0, 0.0, 0.0, 0.0);
    __syncthreads();
    const int cnt = static_cast<int>(min(static_cast<long>(kBruteTile), v.n - j0));
    if (live)
      for (int k = sub; k < cnt; k += kBruteLanes) {
        const double4 s = tile[k];
        if (j0 + k == i || s.w == 0.0) continue;
        cutoff_pair<kEnergy>(xi - s.x, yi - s.y, zi - s.z, s.w, rc2, inv_rc, f, e);
      }
  }
#pragma unroll
  for (int o = kBruteLanes / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
    if (kEnergy) e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if (sub == 0 && i < v.n) cutoff_store<kEnergy>(v, i, live ? v.q[i] : 0.0, f, e, epart);
}

// ---------------------------------------------------------------- contacts
__device__ __forceinline__ bool has_partner(int s) {
  return s == AMK_POSITRON || s == AMK_ELECTRON || s == AMK_PROTON || s == AMK_ANTIPROTON;
}
__device__ __forceinline__ int partner_of(int s) {
  return s == AMK_POSITRON ? AMK_ELECTRON : s == AMK_ELECTRON ? AMK_POSITRON : s == AMK_PROTON ? AMK_ANTIPROTON : AMK_PROTON;
}

struct ContactRule {
  double rc2, prob;
  uint32_t seed;
  uint64_t step;
};

// The directed contact i -> j of two partners at distance^2 d2: kept when it
// is inside the radius and its Philox draw is below the probability.
__device__ __forceinline__ void contact_pair(const ContactRule& R, double d2, uint32_t i, uint32_t j, uint32_t id_i,
                                             uint32_t id_j, Contact* __restrict__ out, unsigned long long* count,
                                             long cap) {
  if (!(d2 < R.rc2)) return;
  const Philox4 w = philox4x32(R.seed, kTagAnnihilation, id_i, id_j, static_cast<uint32_t>(R.step),
                               static_cast<uint32_t>(R.step >> 32));
  if (!(u01(w.w[0]) < R.prob)) return;
  const unsigned long long at = atomicAdd(count, 1ull);
  if (static_cast<long>(at) < cap) {
    Contact e;
    e.a = i;
    e.b = j;
    e.prio = (static_cast<uint64_t>(id_i) << 32) | id_j;
    out[at] = e;
  }
}

// Words of kSlotAnnAux: [0] contacts found, [1] finished blocks of the fused
// kernel, [2] particles marked, [3] sticky "did not converge".
constexpr int kFusedThreads = 1024;
// Up to this many particles the contact search and the matching are one
// launch whose last block matches, with room for every possible contact
// (n^2 / 2 of 16 bytes), so that nothing is read back between steps.
constexpr long kFusedMax = 1024;

template <int kThreads, bool kFused>
__global__ void __launch_bounds__(kThreads)
contact_brute_kernel(View v, const uint8_t* __restrict__ species, const uint32_t* __restrict__ ids, ContactRule R,
                     Contact* __restrict__ out, unsigned long long* words, long cap, unsigned long long* best,
                     uint8_t* matched, uint8_t* live_e) {
  __shared__ double tx[kBruteTile], ty[kBruteTile], tz[kBruteTile];
  __shared__ int ts[kBruteTile];
  __shared__ uint32_t tid_s[kBruteTile];
  __shared__ bool s_last;
  const int sub = threadIdx.x % kBruteLanes;
  const long i = (blockIdx.x * static_cast<long>(kThreads) + threadIdx.x) / kBruteLanes;
  const bool live = i < v.n && usable(v, i) && has_partner(species[i]);
  const int want = live ? partner_of(species[i]) : -2;
  const double xi = live ? v.x[i] : 0.0, yi = live ? v.y[i] : 0.0, zi = live ? v.z[i] : 0.0;
  const uint32_t id_i = live ? ids[i] : 0u;
  for (long j0 = 0; j0 < v.n; j0 += kBruteTile) {
    __syncthreads();
    if (threadIdx.x < kBruteTile) {
      const long j = j0 + threadIdx.x;
      const bool ok = j < v.n && usable(v, j);
      tx[threadIdx.x] = ok ? v.x[j] : 0.0;
      ty[threadIdx.x] = ok ? v.y[j] : 0.0;
      tz[threadIdx.x] = ok ? v.z[j] : 0.0;
      ts[threadIdx.x] = ok ? species[j] : -1;
      tid_s[threadIdx.x] = ok ? ids[j] : 0u;
    }
    __syncthreads();
    const int cnt = static_cast<int>(min(static_cast<long>(kBruteTile), v.n - j0));
    if (live)
      for (int k = sub; k < cnt; k += kBruteLanes)
        if (ts[k] == want)
          contact_pair(R, dist2_exact(xi - tx[k], yi - ty[k], zi - tz[k]), static_cast<uint32_t>(i),
                       static_cast<uint32_t>(j0 + k), id_i, tid_s[k], out, words, cap);
  }
  if (!kFused) return;
  // the last block to finish matches; the words are ready for the next call
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(words + 1, 1ull) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const long m = static_cast<long>(*static_cast<volatile unsigned long long*>(words));
  unsigned long long marked = 0;
  bool open = false;
  if (m > 0) {
    for (long k = threadIdx.x; k < m; k += kThreads) {
      live_e[k] = 1;
      matched[out[k].a] = 0;
      matched[out[k].b] = 0;
    }
    open = match_rounds(out, m, best, matched, live_e, v.alive, &marked);
  }
  if (threadIdx.x == 0) {
    words[2] = marked;
    if (open) words[3] = 1;
    words[0] = words[1] = 0;
  }
}

// ---------------------------------------------------------------- cells
// Dense: the cells of the box, x fastest. Hashed: cells of twice the radius,
// blocks of 16 x 16 x 16 of them hashed onto the same counters (a block's cells
// side by side), so that cells cost nothing where no particle is and their
// width does not depend on the box.
struct CellGrid {
  double o[3], inv_cs;
  int dim[3];
  int species;  // bit s: a live particle of species s
  int hashed;
};

constexpr long kGridCellsPer = 4;          // cells per particle at most
constexpr long kGridCellsMax = 1L << 25;
inline long grid_cell_cap(long n) { return std::min(kGridCellsMax, std::max(4096L, kGridCellsPer * n)); }

// Cutoff (species null): live charged particles. Contacts: live particles
// whose partner species is alive.
__device__ __forceinline__ bool takes_part(const View& v, const uint8_t* __restrict__ species, int alive_species,
                                           long i) {
  if (!usable(v, i)) return false;
  if (!species) return v.q[i] != 0.0;
  return has_partner(species[i]) && ((alive_species >> partner_of(species[i])) & 1);
}

__device__ __forceinline__ void grid_cell(const CellGrid& g, double x, double y, double z, int c[3]) {
  const double p[3] = {x, y, z};
#pragma unroll
  for (int d = 0; d < 3; ++d)
    c[d] = max(0, static_cast<int>(fmin(floor((p[d] - g.o[d]) * g.inv_cs), static_cast<double>(g.dim[d] - 1))));
}

constexpr int kBlockBits = 4, kBlockEdge = 1 << kBlockBits;

__device__ __forceinline__ int cell_entry(const CellGrid& g, int n_cells, int x, int y, int z) {
  if (!g.hashed) return (z * g.dim[1] + y) * g.dim[0] + x;
  const uint64_t block = static_cast<uint64_t>(x >> kBlockBits) | (static_cast<uint64_t>(y >> kBlockBits) << 21) |
                         (static_cast<uint64_t>(z >> kBlockBits) << 42);
  const uint32_t h = static_cast<uint32_t>((block * 0x9E3779B97F4A7C15ull) >> 32);  // Fibonacci hashing
  const uint32_t b = __umulhi(h, static_cast<uint32_t>(n_cells) >> (3 * kBlockBits));
  constexpr int m = kBlockEdge - 1;
  return static_cast<int>(((((b << kBlockBits) | (z & m)) << kBlockBits | (y & m)) << kBlockBits) | (x & m));
}

// Hashed cells are this many radii wide, and taken where the dense ones would be
// wider. us per cutoff evaluation of a ball, dense / hashed: 100,003 particles
// with 0.02, 0.1, 0.25, 0.5 and 12 neighbours inside the radius 67/60, 67/63,
// 67/67, 67/73, 89/147 (the dense cells are 2 radii wide at 0.25), 1,000,003
// 251/205, 252/212, 254/223, 256/238, 384/738. Cells of one radius: 259 at 0.02,
// 461 at 12 (1,000,003). Blocks of 4^3 and 8^3 instead of 16^3: 216 and 210 at
// 0.02, 782 and 766 at 12: a particle's neighbour cells lie closer together the
// larger the blocks are.
// With a dense grid alone one particle 0.01 m away from 100,003 within 2e-4 m took
// a step from 223 to 17,600 us, and one 1 m away from a million one of 735 us to
// 2.4 s; now 284 and 1,031.
constexpr double kHashWidth = 2.0;
static_assert(kBruteMax * kGridCellsPer >= 1L << (3 * kBlockBits), "a grid's counters hold a block");

// Box of the usable particles; the last block turns it into the grid.
// bb: six box words, the species mask (~0 preset: complemented bits are
// cleared) and the count of finished blocks (preset ~0).
__global__ void __launch_bounds__(kBboxThreads)
grid_setup_kernel(View v, const uint8_t* __restrict__ species, double radius, long cell_cap, unsigned long long* bb,
                  CellGrid* __restrict__ grid) {
  unsigned mask = 0;
  bbox_block(
      v,
      [&](long i) {
        const bool ok = usable(v, i);
        if (ok && species) mask |= 1u << species[i];
        return ok;
      },
      bb);
  mask = __reduce_or_sync(0xffffffffu, mask);
  if ((threadIdx.x & 31) == 0 && mask) atomicAnd(&bb[6], ~static_cast<unsigned long long>(mask));
  __threadfence();
  __syncthreads();
  if (threadIdx.x != 0 || atomicAdd(&bb[7], 1ull) + 2 != gridDim.x) return;
  __threadfence();
  volatile unsigned long long* vb = bb;
  CellGrid g;
  double ext[3];
  bool fin = true;
  for (int d = 0; d < 3; ++d) {
    const double lo = double_from_order_bits(vb[d]), hi = -double_from_order_bits(vb[3 + d]);
    ext[d] = hi - lo;
    g.o[d] = isfinite(lo) ? lo : 0.0;
    fin = fin && ext[d] >= 0.0 && isfinite(ext[d]);
  }
  // At most 2^21 cells along an axis: a cell coordinate is computed to 2^-52 of
  // itself, so two of them err by less than the 1e-9 that a cell is wider than
  // the radius, and partners are never two cells apart.
  const double finest = fmax(radius * (1.0 + 1e-9), fmax(ext[0], fmax(ext[1], ext[2])) / kCellMax);
  double cs = finest;
  double cells = INFINITY, dim[3] = {1.0, 1.0, 1.0};
  for (int it = 0; fin && it < 256; ++it) {  // cells no smaller than the radius, at most cell_cap of them
    for (int d = 0; d < 3; ++d) dim[d] = floor(ext[d] / cs) + 1.0;
    cells = dim[0] * dim[1] * dim[2];
    if (cells <= static_cast<double>(cell_cap)) break;
    cs *= fmax(1.05, fmin(cbrt(cells / static_cast<double>(cell_cap)), 1e6));
  }
  const bool ok = fin && cells <= static_cast<double>(cell_cap);
  g.hashed = fin && !(cs <= kHashWidth * finest);
  if (g.hashed) cs = kHashWidth * finest;
  g.inv_cs = ok || g.hashed ? 1.0 / cs : 0.0;
  for (int d = 0; d < 3; ++d) g.dim[d] = g.hashed ? 1 << kCellBits : ok ? static_cast<int>(dim[d]) : 1;
  g.species = static_cast<int>(~vb[6] & 0xffull);
  *grid = g;
}

// cell[i] = counter of particle i's cell, -1 when it takes no part; rank[i] = a
// place among the counter's members. Cutoff: the particles that take no part
// get their zero force here.
template <bool kEnergy>
__global__ void grid_count_kernel(View v, const uint8_t* __restrict__ species, const CellGrid* __restrict__ grid,
                                  int n_cells, int* __restrict__ cell, int* __restrict__ rank, int* __restrict__ count,
                                  double* __restrict__ epart) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i >= v.n) return;
  const CellGrid g = *grid;
  if (!takes_part(v, species, g.species, i)) {
    cell[i] = -1;
    if (!species) {
      const double f[3] = {0.0, 0.0, 0.0};
      cutoff_store<kEnergy>(v, i, 0.0, f, 0.0, epart);
    }
    return;
  }
  int c[3];
  grid_cell(g, v.x[i], v.y[i], v.z[i], c);
  const int id = cell_entry(g, n_cells, c[0], c[1], c[2]);
  cell[i] = id;
  rank[i] = atomicAdd(&count[id], 1);
}

__global__ void grid_scatter_kernel(long n, const int* __restrict__ cell, const int* __restrict__ rank,
                                    const int* __restrict__ start, int* __restrict__ member) {
  const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (i < n && cell[i] >= 0) member[start[cell[i]] + rank[i]] = static_cast<int>(i);
}

// The records in cell order, a counter's members in ascending particle index:
// position and charge (cutoff) or position and {id, species} (contacts).
__global__ void grid_record_kernel(View v, const uint8_t* __restrict__ species, const uint32_t* __restrict__ ids,
                                   const int* __restrict__ cell, const int* __restrict__ start, const int* __restrict__ m,
                                   const int* __restrict__ member, double4* __restrict__ rec, int* __restrict__ index) {
  const long p = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  if (p >= *m) return;
  const int i = member[p], b = start[cell[i]], e = start[cell[i] + 1];
  int r = 0;
  for (int k = b; k < e; ++k) r += member[k] < i ? 1 : 0;
  const double w = species ? __longlong_as_double(static_cast<long long>(
                                 (static_cast<unsigned long long>(ids[i]) << 8) | species[i]))
                           : v.q[i];
  rec[b + r] = make_double4(v.x[i], v.y[i], v.z[i], w);
  index[b + r] = i;
}

// Calls f(k) for the records k of the 27 cells around a position: nine runs of
// the dense cells; of the hashed ones those that the sphere of the radius
// touches, a block's cells of a row as one run. (Three cells in a row differ in
// their place in a block, so no counter is read twice; the particles of other
// blocks that share one are out of reach.)
template <typename F>
__device__ __forceinline__ void neighbours(const CellGrid& g, int n_cells, const int* __restrict__ start, double radius,
                                           double x, double y, double z, F f) {
  int c[3];
  grid_cell(g, x, y, z, c);
  if (!g.hashed) {
    const int x0 = max(c[0] - 1, 0), x1 = min(c[0] + 1, g.dim[0] - 1);
    for (int cz = max(c[2] - 1, 0); cz <= min(c[2] + 1, g.dim[2] - 1); ++cz)
      for (int cy = max(c[1] - 1, 0); cy <= min(c[1] + 1, g.dim[1] - 1); ++cy) {
        const int row = (cz * g.dim[1] + cy) * g.dim[0];
        const int end = start[row + x1 + 1];
        for (int k = start[row + x0]; k < end; ++k) f(k);
      }
    return;
  }
  // a partner's coordinates differ by less than this (rounding of the
  // differences, of the squares and of the bounds included)
  const double r = radius * (1.0 + 1e-9);
  const double ex = r + 4.5e-16 * fabs(x), ey = r + 4.5e-16 * fabs(y), ez = r + 4.5e-16 * fabs(z);
  int lo[3], hi[3];
  grid_cell(g, x - ex, y - ey, z - ez, lo);
  grid_cell(g, x + ex, y + ey, z + ez, hi);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = max(lo[d], c[d] - 1);
    hi[d] = min(hi[d], c[d] + 1);
  }
  for (int cz = lo[2]; cz <= hi[2]; ++cz)
    for (int cy = lo[1]; cy <= hi[1]; ++cy)
      for (int cx = lo[0]; cx <= hi[0];) {
        const int last = min(hi[0], cx | (kBlockEdge - 1));
        const int id = cell_entry(g, n_cells, cx, cy, cz), end = start[id + last - cx + 1];
        for (int k = start[id]; k < end; ++k) f(k);
        cx = last + 1;
      }
}

template <bool kEnergy>
__global__ void __launch_bounds__(128)
cutoff_grid_kernel(View v, const CellGrid* __restrict__ grid, int n_cells, double rc, const int* __restrict__ start,
                   const double4* __restrict__ rec, const int* __restrict__ index, double* __restrict__ epart) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= start[n_cells]) return;
  const double4 me = rec[p];
  const double rc2 = rc * rc, inv_rc = 1.0 / rc;
  double f[3] = {0.0, 0.0, 0.0}, e = 0.0;
  neighbours(*grid, n_cells, start, rc, me.x, me.y, me.z, [&](int k) {
    const double4 s = rec[k];
    if (k != p) cutoff_pair<kEnergy>(me.x - s.x, me.y - s.y, me.z - s.z, s.w, rc2, inv_rc, f, e);
  });
  cutoff_store<kEnergy>(v, index[p], me.w, f, e, epart);
}

__global__ void __launch_bounds__(128)
contact_grid_kernel(const CellGrid* __restrict__ grid, int n_cells, double radius, ContactRule R,
                    const int* __restrict__ start, const double4* __restrict__ rec, const int* __restrict__ index,
                    Contact* __restrict__ out, unsigned long long* count, long cap) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= start[n_cells]) return;
  const double4 me = rec[p];
  const unsigned long long own = static_cast<unsigned long long>(__double_as_longlong(me.w));
  const unsigned want = static_cast<unsigned>(partner_of(static_cast<int>(own & 0xff)));
  neighbours(*grid, n_cells, start, radius, me.x, me.y, me.z, [&](int k) {
    const double4 s = rec[k];
    const unsigned long long st = static_cast<unsigned long long>(__double_as_longlong(s.w));
    if ((st & 0xff) != want) return;
    contact_pair(R, dist2_exact(me.x - s.x, me.y - s.y, me.z - s.z), static_cast<uint32_t>(index[p]),
                 static_cast<uint32_t>(index[k]), static_cast<uint32_t>(own >> 8), static_cast<uint32_t>(st >> 8),
                 out, count, cap);
  });
}

struct CellList {
  CellGrid* grid;
  int n_cells;
  int* start;      // per cell, and the member count after the last one
  double4* rec;
  int* index;
};

// species null: the cutoff's list (zero forces written for the others).
int build_cell_list(amk_ctx* c, const View& v, double radius, const uint8_t* species, const uint32_t* ids,
                    double* epart, CellList* out) {
  int rc = AMK_OK;
  const long n = v.n, cells = grid_cell_cap(n);
  unsigned long long* bb = slot<unsigned long long>(c, kSlotCellStart, 8 + (sizeof(CellGrid) + 7) / 8, &rc);
  AMK_TRY(rc);
  CellGrid* grid = reinterpret_cast<CellGrid*>(bb + 8);
  int* cell = slot<int>(c, kSlotKeysA, 2 * static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  int* rank = cell + n;
  int* start = slot<int>(c, kSlotKeysB, static_cast<size_t>(cells) + 1, &rc);
  AMK_TRY(rc);
  int* member = slot<int>(c, kSlotValsA, static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  int* index = slot<int>(c, kSlotValsB, static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  double4* rec = slot<double4>(c, kSlotSorted1, static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  const int n_cells = static_cast<int>(cells);
  const unsigned gn = static_cast<unsigned>((n + 255) / 256);
  AMK_TRY(phase_begin(c, AMK_PHASE_SORT));
  AMK_CUDA_TRY(cudaMemsetAsync(bb, 0xFF, 8 * sizeof(unsigned long long), c->stream));
  AMK_CUDA_TRY(cudaMemsetAsync(start, 0, static_cast<size_t>(cells) * sizeof(int), c->stream));
  grid_setup_kernel<<<bbox_grid(n), kBboxThreads, 0, c->stream>>>(v, species, radius, cells, bb, grid);
  AMK_TRY(check_launch(c, "grid_setup_kernel"));
  if (epart)
    grid_count_kernel<true><<<gn, 256, 0, c->stream>>>(v, species, grid, n_cells, cell, rank, start, epart);
  else
    grid_count_kernel<false><<<gn, 256, 0, c->stream>>>(v, species, grid, n_cells, cell, rank, start, nullptr);
  AMK_TRY(check_launch(c, "grid_count_kernel"));
  AMK_TRY(exclusive_scan_int(c, start, cells, start, start + cells));
  grid_scatter_kernel<<<gn, 256, 0, c->stream>>>(n, cell, rank, start, member);
  AMK_TRY(check_launch(c, "grid_scatter_kernel"));
  grid_record_kernel<<<gn, 256, 0, c->stream>>>(v, species, ids, cell, start, start + cells, member, rec, index);
  AMK_TRY(check_launch(c, "grid_record_kernel"));
  AMK_TRY(phase_end(c, AMK_PHASE_SORT));
  out->grid = grid;
  out->n_cells = n_cells;
  out->start = start;
  out->rec = rec;
  out->index = index;
  return AMK_OK;
}

}  // namespace

int cutoff_forces(amk_ctx* c, const View& v, double cutoff, double* energy_out) {
  if (energy_out) *energy_out = 0.0;
  const long n = v.n;
  if (n == 0) return AMK_OK;
  if (!(cutoff > 0.0)) {  // coulomb_interaction.cc:33-37
    zero_forces_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, c->stream>>>(v);
    return check_launch(c, "zero_forces_kernel");
  }
  int rc = AMK_OK;
  double* epart = nullptr;
  if (energy_out) {
    epart = slot<double>(c, kSlotAuxState2, static_cast<size_t>(n) + 8, &rc);
    AMK_TRY(rc);
  }
  if (n <= kBruteMax) {
    AMK_TRY(phase_begin(c, AMK_PHASE_CUTOFF));
    const unsigned grid = brute_grid(n, kBruteThreads);
    if (epart)
      cutoff_brute_kernel<true><<<grid, kBruteThreads, 0, c->stream>>>(v, cutoff, epart);
    else
      cutoff_brute_kernel<false><<<grid, kBruteThreads, 0, c->stream>>>(v, cutoff, nullptr);
    AMK_TRY(check_launch(c, "cutoff_brute_kernel"));
    AMK_TRY(phase_end(c, AMK_PHASE_CUTOFF));
  } else {
    CellList cl;
    AMK_TRY(build_cell_list(c, v, cutoff, nullptr, nullptr, epart, &cl));
    AMK_TRY(phase_begin(c, AMK_PHASE_CUTOFF));
    const unsigned grid = static_cast<unsigned>((n + 127) / 128);
    if (epart)
      cutoff_grid_kernel<true><<<grid, 128, 0, c->stream>>>(v, cl.grid, cl.n_cells, cutoff, cl.start, cl.rec, cl.index,
                                                            epart);
    else
      cutoff_grid_kernel<false><<<grid, 128, 0, c->stream>>>(v, cl.grid, cl.n_cells, cutoff, cl.start, cl.rec, cl.index,
                                                             nullptr);
    AMK_TRY(check_launch(c, "cutoff_grid_kernel"));
    AMK_TRY(phase_end(c, AMK_PHASE_CUTOFF));
  }
  if (energy_out) {
    double* res = slot<double>(c, kSlotAuxState4, 8, &rc);
    AMK_TRY(rc);
    AMK_TRY(reduce_sum(c, epart, n, res));
    double h = 0.0;
    AMK_CUDA_TRY(cudaMemcpyAsync(&h, res, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
    *energy_out = 0.5 * kCoulombConstant * h;  // each pair counted from both ends
  }
  return AMK_OK;
}

// Buffers of a matching over the contacts of n particles.
static int match_buffers(amk_ctx* c, long n, long m, unsigned long long** best, uint8_t** flags) {
  int rc = AMK_OK;
  // two per-particle priority arrays, then the matching state
  *best = slot<unsigned long long>(c, kSlotAnnBest, 2 * static_cast<size_t>(n) + sizeof(MatchState) / 8 + 1, &rc);
  AMK_TRY(rc);
  *flags = slot<uint8_t>(c, kSlotAuxState1, static_cast<size_t>(n) + static_cast<size_t>(m) + 16, &rc);
  return rc;
}

int annihilate_check(amk_ctx* c, long* marked) {
  if (!c->ann_pending) return AMK_OK;
  c->ann_pending = false;
  int rc = AMK_OK;
  unsigned long long* words = slot<unsigned long long>(c, kSlotAnnAux, 8, &rc);
  AMK_TRY(rc);
  unsigned long long res[2] = {0, 0};
  AMK_CUDA_TRY(cudaMemcpyAsync(res, words + 2, sizeof(res), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  if (res[1]) {
    c->ann_words_clear = false;
    return fail(AMK_ERR_TIMEOUT, "annihilation matching did not converge");
  }
  if (marked) *marked = static_cast<long>(res[0]);
  return AMK_OK;
}

int annihilate_view(amk_ctx* c, const View& v, const uint8_t* species, const uint32_t* ids, double radius,
                    double probability, uint32_t seed, uint64_t step_index, long* marked) {
  if (marked) *marked = 0;
  if (!(radius > 0.0) || v.n == 0) return AMK_OK;  // annihilation.cc:34-35
  const ContactRule R{radius * radius, probability, seed, step_index};
  int rc = AMK_OK;
  unsigned long long* words = slot<unsigned long long>(c, kSlotAnnAux, 8, &rc);
  AMK_TRY(rc);
  unsigned long long* best = nullptr;
  uint8_t* flags = nullptr;
  if (v.n <= kFusedMax && match_grid_min() >= kMatchGridMin) {
    const long cap = v.n * v.n / 2 + 1;  // directed contacts of a two-species set: at most 2 (n/2)^2
    Contact* edges = slot<Contact>(c, kSlotAnnEdges, static_cast<size_t>(cap), &rc);
    AMK_TRY(rc);
    AMK_TRY(match_buffers(c, v.n, cap, &best, &flags));
    if (!c->ann_words_clear) {
      AMK_CUDA_TRY(cudaMemsetAsync(words, 0, 4 * sizeof(unsigned long long), c->stream));
      c->ann_words_clear = true;
    }
    contact_brute_kernel<kFusedThreads, true><<<brute_grid(v.n, kFusedThreads), kFusedThreads, 0, c->stream>>>(
        v, species, ids, R, edges, words, cap, best, flags, flags + v.n);
    AMK_TRY(check_launch(c, "contact_brute_kernel"));
    c->ann_pending = true;
    return marked ? annihilate_check(c, marked) : AMK_OK;
  }
  AMK_TRY(annihilate_check(c, nullptr));  // the words are about to be reused
  c->ann_words_clear = false;
  CellList cl{};
  if (v.n > kBruteMax) AMK_TRY(build_cell_list(c, v, radius, species, ids, nullptr, &cl));
  long cap = std::max<long>(1024, v.n / 16);
  for (int attempt = 0; attempt < 3; ++attempt) {
    Contact* edges = slot<Contact>(c, kSlotAnnEdges, static_cast<size_t>(cap), &rc);
    AMK_TRY(rc);
    AMK_CUDA_TRY(cudaMemsetAsync(words, 0, 4 * sizeof(unsigned long long), c->stream));
    if (v.n <= kBruteMax)
      contact_brute_kernel<kBruteThreads, false><<<brute_grid(v.n, kBruteThreads), kBruteThreads, 0, c->stream>>>(
          v, species, ids, R, edges, words, cap, nullptr, nullptr, nullptr);
    else
      contact_grid_kernel<<<static_cast<unsigned>((v.n + 127) / 128), 128, 0, c->stream>>>(
          cl.grid, cl.n_cells, radius, R, cl.start, cl.rec, cl.index, edges, words, cap);
    AMK_TRY(check_launch(c, "contact kernel"));
    unsigned long long m = 0;
    AMK_CUDA_TRY(cudaMemcpyAsync(&m, words, sizeof(m), cudaMemcpyDeviceToHost, c->stream));
    AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
    if (static_cast<long>(m) > cap) {
      cap = static_cast<long>(m) + 1024;
      continue;
    }
    if (m == 0) break;
    AMK_TRY(match_buffers(c, v.n, static_cast<long>(m), &best, &flags));
    AMK_TRY(queue_matching(c, c->stream, edges, static_cast<long>(m), nullptr, best, best + v.n, flags, flags + v.n,
                           v.alive, reinterpret_cast<MatchState*>(best + 2 * v.n), words + 2));
    unsigned long long res[2] = {0, 0};
    AMK_CUDA_TRY(cudaMemcpyAsync(res, words + 2, sizeof(res), cudaMemcpyDeviceToHost, c->stream));
    AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
    if (res[1]) return fail(AMK_ERR_TIMEOUT, "annihilation matching did not converge");
    if (marked) *marked = static_cast<long>(res[0]);
    break;
  }
  return AMK_OK;
}

int annihilate_step(amk_ctx* c, uint64_t step_index, long* marked) {
  if (marked) *marked = 0;
  const amk_params& p = c->p;
  if (!(p.contact_radius > 0.0)) return AMK_OK;  // annihilation.cc:34-35
  AMK_TRY(phase_begin(c, AMK_PHASE_ANNIHILATION));
  AMK_TRY(annihilate_view(c, main_view(c), c->species.as<uint8_t>(), c->ids.as<uint32_t>(), p.contact_radius,
                          p.annihilation_probability, static_cast<uint32_t>(p.seed), step_index, marked));
  AMK_TRY(phase_end(c, AMK_PHASE_ANNIHILATION));
  return AMK_OK;
}

}  // namespace amk

// ======================================================================
// Allocation-free cutoff solver.
//
// Some callers cannot let a library allocate device memory: a host code
// whose device memory is already owned by its own pool allocator (a
// library cudaMalloc could fail there, or fragment the pool), or a
// per-step loop that cannot take the implicit device-wide synchronisation
// of cudaMalloc/cudaFree. For them this variant of the cutoff solver keeps
// all of its scratch (cell keys, sort buffers, histograms: about 2.4 MB)
// in one file-scope device array sized for kNoAllocMaxParticles. Every GPU
// that loads this library holds that array until the process exits.
//
// Set-up: the first call on a device (with that device current) looks up
// the array's device address with cudaGetSymbolAddress and caches it; make
// that first call during set-up, before any stream capture. Later calls
// allocate nothing and call no allocating routine.
//
// Every call uses the same array and it keeps the last call's contents:
// only the bounding-box words must start cleared and they are reset at the
// start of each call. Calls that overlap on the GPU (different streams, or
// different host threads without ordering) race on the array.
// ======================================================================
#include <mutex>

namespace amk {
namespace {

constexpr long kNoAllocMaxParticles = 65536;
constexpr long kNoAllocSortTile = 4096;  // the sort's tile (256 threads x 16)
// radix_sort_pairs_buffers scans its digit histogram (256 counters per tile)
// with one CTA, which handles at most 65,536 counters
static_assert(256 * ((kNoAllocMaxParticles + kNoAllocSortTile - 1) / kNoAllocSortTile) <= 65536,
              "the allocation-free sort's histogram exceeds the one-CTA scan");
constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t kNaBbox = 0;
constexpr size_t kNaKeys = align256(kNaBbox + 8 * sizeof(unsigned long long));
constexpr size_t kNaVals = align256(kNaKeys + kNoAllocMaxParticles * sizeof(uint64_t));
constexpr size_t kNaSKeys = align256(kNaVals + kNoAllocMaxParticles * sizeof(uint32_t));
constexpr size_t kNaSIdx = align256(kNaSKeys + kNoAllocMaxParticles * sizeof(uint64_t));
constexpr size_t kNaTKeys = align256(kNaSIdx + kNoAllocMaxParticles * sizeof(uint32_t));
constexpr size_t kNaTVals = align256(kNaTKeys + kNoAllocMaxParticles * sizeof(uint64_t));
constexpr size_t kNaHist = align256(kNaTVals + kNoAllocMaxParticles * sizeof(uint32_t));
constexpr size_t kNaBytes =
    align256(kNaHist + 256 * ((kNoAllocMaxParticles + kNoAllocSortTile - 1) / kNoAllocSortTile) * sizeof(uint32_t));

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_addr[kNoAllocMaxDevices] = {};

}  // namespace

cudaError_t radix_sort_pairs_buffers(cudaStream_t stream, const uint64_t* keys_in, const uint32_t* vals_in,
                                     uint64_t* keys_out, uint32_t* vals_out, uint64_t* ktmp, uint32_t* vtmp,
                                     uint32_t* hist, long n, int key_bits);

}  // namespace amk

extern "C" int amk_coulomb_standard_noalloc(const double* x, const double* y, const double* z, const double* q,
                                            const uint8_t* alive, long n, double cutoff_radius, double* fx,
                                            double* fy, double* fz, void* stream) {
  using namespace amk;
  if (n < 0) return fail(AMK_ERR_INVALID, "amk_coulomb_standard_noalloc: n < 0");
  if (n > kNoAllocMaxParticles)
    return fail(AMK_ERR_LIMIT,
                "amk_coulomb_standard_noalloc: %ld particles exceed the allocation-free maximum of %ld", n,
                kNoAllocMaxParticles);
  if (n == 0) return AMK_OK;
  if (!x || !y || !z || !q || !fx || !fy || !fz) return fail(AMK_ERR_INVALID, "amk_coulomb_standard_noalloc: null array");
  int dev = 0;
  AMK_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(AMK_ERR_LIMIT, "device %d beyond the supported range", dev);
  unsigned char* base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || p == nullptr)
        return fail(AMK_ERR_CUDA, "cudaGetSymbolAddress of the allocation-free scratch failed: %s",
                    cudaGetErrorString(e));
      g_noalloc_addr[dev] = static_cast<unsigned char*>(p);
    }
    base = g_noalloc_addr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  View v;
  v.n = n;
  v.x = const_cast<double*>(x);
  v.y = const_cast<double*>(y);
  v.z = const_cast<double*>(z);
  v.q = const_cast<double*>(q);
  v.alive = const_cast<uint8_t*>(alive);
  v.fx = fx;
  v.fy = fy;
  v.fz = fz;
  const unsigned blocks = static_cast<unsigned>((n + 255) / 256);
  if (!(cutoff_radius > 0.0)) {  // coulomb_interaction.cc:33-37
    zero_forces_kernel<<<blocks, 256, 0, s>>>(v);
    AMK_CUDA_TRY(cudaGetLastError());
    return AMK_OK;
  }
  if (n <= kBruteMax) {  // needs no scratch
    cutoff_brute_kernel<false><<<brute_grid(n, kBruteThreads), kBruteThreads, 0, s>>>(v, cutoff_radius, nullptr);
    AMK_CUDA_TRY(cudaGetLastError());
    return AMK_OK;
  }
  unsigned long long* bb = reinterpret_cast<unsigned long long*>(base + kNaBbox);
  uint64_t* keys = reinterpret_cast<uint64_t*>(base + kNaKeys);
  uint32_t* vals = reinterpret_cast<uint32_t*>(base + kNaVals);
  uint64_t* skeys = reinterpret_cast<uint64_t*>(base + kNaSKeys);
  uint32_t* sidx = reinterpret_cast<uint32_t*>(base + kNaSIdx);
  uint64_t* ktmp = reinterpret_cast<uint64_t*>(base + kNaTKeys);
  uint32_t* vtmp = reinterpret_cast<uint32_t*>(base + kNaTVals);
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + kNaHist);
  AMK_CUDA_TRY(cudaMemsetAsync(bb, 0xFF, 6 * sizeof(unsigned long long), s));
  bbox_kernel<<<bbox_grid(n), kBboxThreads, 0, s>>>(v, bb);
  cell_key_kernel<<<blocks, 256, 0, s>>>(v, bb, cutoff_radius, keys, vals);
  AMK_CUDA_TRY(cudaGetLastError());
  AMK_CUDA_TRY(radix_sort_pairs_buffers(s, keys, vals, skeys, sidx, ktmp, vtmp, hist, n, 64));
  cutoff_kernel<<<static_cast<unsigned>((n + 127) / 128), 128, 0, s>>>(v, bb, cutoff_radius, skeys, sidx);
  AMK_CUDA_TRY(cudaGetLastError());
  return AMK_OK;
}
