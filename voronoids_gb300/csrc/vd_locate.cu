// Point location queries on a finished tree: the conflict region of a query
// point, i.e. the simplices whose circumsphere strictly contains it
// (`locate`, src/delaunay_tree.rs:33-58 with find_all_neighbors :60-75).
//
// A visibility walk from the finest location hint of the set towards the
// simplex that contains the point, then a breadth-first search over face
// neighbours with the exact conflict test: a warp per query with lists in
// shared memory, small ones and then large ones, and a block per query with
// lists as long as the tree for what outgrows both.  The query takes the role of
// the newest vertex (largest id), so a point exactly on a circumsphere is
// outside: the reference's strict `dist < r`.  The conflict region is
// connected, so the search finds all of it.
#include <cuda_runtime.h>

#include <algorithm>

#include "vd_common.cuh"

namespace vd {
namespace {

__device__ __forceinline__ int g4(const int4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

__device__ __forceinline__ void load_simp(const DevTree& T, int s, int4& v, int4& n) {
  const int4* p = reinterpret_cast<const int4*>(T.simp + s);
  v = p[0];
  n = p[1];
}

template <int D>
__device__ __forceinline__ int hint_cell(const SetGeo& g, const vdp::VPt& p, int level) {
  const int side = 1 << level;
  const double c[3] = {p.x, p.y, p.z};
  int idx = 0;
  for (int k = D - 1; k >= 0; --k) {
    int i = (int)((c[k] - g.org[k]) * g.scale * side);
    i = i < 0 ? 0 : (i >= side ? side - 1 : i);
    idx = idx * side + i;
  }
  const int off = D == 3 ? ((1 << (3 * level)) - 1) / 7 : ((1 << (2 * level)) - 1) / 3;
  return g.hint_off + off + idx;
}

// Open-addressing set of HS ids (-1 empty) in shared memory.
template <int HS>
__device__ __forceinline__ bool hset_has(const int* hk, int key) {
  unsigned h = ((unsigned)key * 2654435761u) & (HS - 1);
  for (int probe = 0; probe < HS; ++probe, h = (h + 1) & (HS - 1)) {
    const int k = *((volatile const int*)&hk[h]);
    if (k == key) return true;
    if (k == -1) return false;
  }
  return false;
}
template <int HS>
__device__ __forceinline__ bool hset_add(int* hk, int key) {
  unsigned h = ((unsigned)key * 2654435761u) & (HS - 1);
  for (int probe = 0; probe < HS; ++probe, h = (h + 1) & (HS - 1)) {
    const int old = atomicCAS(&hk[h], -1, key);
    if (old == -1) return true;
    if (old == key) return false;
  }
  return false;
}

// 1 if the query p (record fp) is in conflict with simplex s (vertices v), -1 if
// not; with `sphere` alone 0 where the stored sphere (3D) cannot decide.
template <int D>
__device__ __forceinline__ int query_side(const DevTree& T, int s, const int4& v, const vdp::VPt& p, const vdp::FPt& fp,
                                          bool sphere, vdp::Tally& tl, int& perr) {
  constexpr int NV = D + 1;
  if (D == 3) {
    const float4 c = *reinterpret_cast<const float4*>(T.sph + s);
    const int side = vdp::sphere_side<D>(vdp::Sph{c.x, c.y, c.z, c.w}, fp);
    if (side != 0) return side;
  }
  if (sphere) return 0;
  vdp::FPt fv[NV];
  int key[NV];
  for (int j = 0; j < NV; ++j) {
    key[j] = g4(v, j);
    fv[j] = T.ptf[key[j]];
  }
  auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
    for (int j = 0; j < NV; ++j) v64[j] = T.pts[key[j]];
    p64 = p;
  };
  const int qkey = 0x7fffffff;  // newer than every vertex
  return vdp::in_conflict_hl<D>(fv, key, fp, qkey, tl, perr, load64) ? 1 : -1;
}

template <int D>
__device__ __forceinline__ void load_query(const double* q, int i, vdp::VPt& p, vdp::FPt& fp) {
  p = vdp::VPt{q[(long long)i * D], q[(long long)i * D + 1], D == 3 ? q[(long long)i * D + 2] : 0.0, 0.0};
  fp = vdp::split_point(p.x, p.y, p.z);
}

// Warp form: a warp per query, region lists in shared memory.  The walk stops
// at the first simplex whose stored sphere (3D) certainly holds the point: the
// conflict region is connected, so any of its simplices will do to start from.
// The region is searched in waves of 32 (simplex, face) items, as in the
// insertion rounds.  Bound by the chain of dependent gathers of one query
// (walk, then about six waves), with every query of a call in flight: the
// kernel takes about 0.1 ms for 4,096 queries in a 100,000-point tree.
//
// Queries are 0 .. n - 1, or list[0 .. n) where a list is given.  res[i] =
// (count, first) of query i: count -1 outside the super simplex, -2 when the
// region outgrew the lists (`first` is then a simplex of the region); its
// sorted ranks are out[first ..].  *total counts the ranks of all queries, which
// may exceed cap_out; with out null only the counts are made.
//
// WIDE: the lists are 192 simplices in 3D and 64 in 2D, with 16 warps on an
// SM; the wide form, for the queries that outgrow these, has 1,024 and six warps.
template <int D, bool WIDE>
struct LocWarp {
  static constexpr int WARPS = WIDE ? 1 : 4, BLOCKS = WIDE ? 6 : 4;
  static constexpr int CAP = WIDE ? 1024 : (D == 3 ? 192 : 64), HS = WIDE ? 4096 : (D == 3 ? 512 : 128);
  int4 cn[CAP];
  int hk[HS];  // id set of the region, then its ranks while they are sorted
  int cav[CAP];
};

template <int D, bool WIDE>
__global__ void __launch_bounds__(32 * LocWarp<D, WIDE>::WARPS, LocWarp<D, WIDE>::BLOCKS)
    k_locate_warp(DevTree T, const double* q, const int* list, int n_list, const int* rank, int* out, int cap_out,
                  int2* res, int* total) {
  using Warp = LocWarp<D, WIDE>;
  constexpr int NV = D + 1, CAP = Warp::CAP, HS = Warp::HS;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ Warp sm[Warp::WARPS];
  Warp& W = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  vdp::Tally tl = {0, 0, 0, 0};
  int perr = 0;
  const SetGeo& g = T.sets[0];
  for (int j0 = blockIdx.x * Warp::WARPS + (threadIdx.x >> 5); j0 < n_list; j0 += gridDim.x * Warp::WARPS) {
    const int i = list ? list[j0] : j0;
    vdp::VPt p;
    vdp::FPt fp;
    load_query<D>(q, i, p, fp);
    auto exit_of = [&](const int4& v) {
      vdp::FPt fv[NV];
      for (int j = 0; j < NV; ++j) fv[j] = T.ptf[g4(v, j)];
      auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
        for (int j = 0; j < NV; ++j) v64[j] = T.pts[g4(v, j)];
        p64 = p;
      };
      return vdp::exit_face_hl<D>(fv, fp, (1u << NV) - 1, tl, perr, load64);
    };
    auto conflict = [&](int s, const int4& v, bool sphere) { return query_side<D>(T, s, v, p, fp, sphere, tl, perr); };
    int cur = -1;
    for (int l = g.hint_levels; l >= 0 && cur < 0; --l) cur = T.hint[hint_cell<D>(g, p, l)];
    if (cur < 0 || bad_simp(T, cur)) cur = g.root;
    int4 v, nn;
    load_simp(T, cur, v, nn);
    for (int k = 0; k < 64 && v.x < 0 && nn.x >= 0; ++k) {  // dead slot: into its star
      cur = nn.x >> 2;
      if (bad_simp(T, cur)) break;
      load_simp(T, cur, v, nn);
    }
    if (v.x < 0 || bad_simp(T, cur)) {
      if (lane == 0) {
        set_error(T.ctr, E_INTERNAL);
        res[i] = make_int2(0, 0);
      }
      continue;
    }
    // outside the super simplex: the walk below may stop before it finds out
    if (exit_of(make_int4(g.sup[0], g.sup[1], g.sup[2], g.sup[3])) >= 0) {
      if (lane == 0) res[i] = make_int2(-1, 0);
      continue;
    }
    bool hit = false;
    for (int step = 0; step < (1 << 16); ++step) {
      if (conflict(cur, v, true) > 0) {
        hit = true;
        break;
      }
      const int f = exit_of(v);
      if (f < 0) break;
      const int code = g4(nn, f);
      if (code < 0 || bad_simp(T, code >> 2)) break;
      cur = code >> 2;
      load_simp(T, cur, v, nn);
    }
    // the containing simplex is in the region unless the point is one of its
    // vertices
    if (!hit) hit = conflict(cur, v, false) > 0;
    int n = 0;
    if (hit) {
      for (int k = lane; k < HS; k += 32) W.hk[k] = -1;
      __syncwarp();
      if (lane == 0) {
        W.cav[0] = cur;
        W.cn[0] = nn;
        hset_add<HS>(W.hk, cur);
      }
      __syncwarp();
      n = 1;
      for (int head = 0; head < n * NV && n <= CAP;) {
        const int it = head + lane, avail = n * NV;
        const int k = it / NV, f = it - k * NV;
        int nb = -1;
        if (it < avail) nb = reinterpret_cast<const int*>(W.cn + k)[f];
        nb = nb < 0 ? -1 : nb >> 2;
        bool add = false;
        int4 bv, bn;
        if (nb >= 0 && !bad_simp(T, nb) && !hset_has<HS>(W.hk, nb)) {
          load_simp(T, nb, bv, bn);
          if (conflict(nb, bv, false) > 0) add = hset_add<HS>(W.hk, nb);
        }
        __syncwarp();
        const unsigned m = __ballot_sync(FULL, add);
        const int at = n + __popc(m & below);
        if (add && at < CAP) {
          W.cav[at] = nb;
          W.cn[at] = bn;
        }
        __syncwarp();
        n += __popc(m);
        head = min(head + 32, avail);
      }
    }
    int first = 0;
    if (n > CAP) {
      n = -2;
      first = cur;
    } else if (n > 0 && out) {
      if (lane == 0) first = atomicAdd(total, n);
      first = __shfl_sync(FULL, first, 0);
      // the ranks (numbering of the simplex export), sorted
      int P = 32;
      while (P < n) P <<= 1;
      for (int k = lane; k < P; k += 32) W.hk[k] = k < n ? rank[W.cav[k]] : 0x7fffffff;
      __syncwarp();
      for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          for (int a = lane; a < P; a += 32) {
            const int b = a ^ j;
            if (b <= a) continue;
            const int x = W.hk[a], y = W.hk[b];
            if ((x > y) == ((a & k) == 0)) {
              W.hk[a] = y;
              W.hk[b] = x;
            }
          }
          __syncwarp();
        }
      if ((long long)first + n <= cap_out)
        for (int k = lane; k < n; k += 32) out[first + k] = W.hk[k];
      __syncwarp();
    } else if (n > 0 && lane == 0) {
      atomicAdd(total, n);
    }
    if (lane == 0) res[i] = make_int2(n, first);
  }
  if (perr) set_error(T.ctr, E_PRECISION);
}

// Block form: a block per query list[b], which starts at res[list[b]].y (a simplex of
// its region).  The region's simplices are a set of bits over the slots and a
// list, both of the block's own and as long as the tree, so no region is too
// large; the bits are zero on entry and on return.  Waves take every (simplex,
// face) item found so far, kLocThreads at a time.  lists[b * cap ..] receives the
// region as ranks (rank given) in no order, cnt[b] its size.
constexpr int kLocThreads = 256;
template <int D>
__global__ void __launch_bounds__(kLocThreads) k_locate_block(DevTree T, const double* q, const int* list, const int2* res,
                                                              const int* rank, int* lists, long long cap, unsigned* bits,
                                                              long long words, int* cnt) {
  constexpr int NV = D + 1;
  __shared__ int s_n;
  const int b = blockIdx.x, i = list[b];
  int* L = lists + b * cap;
  unsigned* B = bits + b * words;
  vdp::Tally tl = {0, 0, 0, 0};
  int perr = 0;
  vdp::VPt p;
  vdp::FPt fp;
  load_query<D>(q, i, p, fp);
  const int start = res[i].y;
  if (bad_simp(T, start)) {
    if (threadIdx.x == 0) {
      set_error(T.ctr, E_INTERNAL);
      cnt[b] = 0;
    }
    return;
  }
  if (threadIdx.x == 0) {
    s_n = 1;
    L[0] = start;
    atomicOr(B + (start >> 5), 1u << (start & 31));
  }
  for (long long head = 0;;) {
    __syncthreads();
    const long long avail = (long long)s_n * NV;
    __syncthreads();
    if (head >= avail) break;
    for (long long it = head + threadIdx.x; it < avail; it += kLocThreads) {
      const int k = (int)(it / NV), f = (int)(it - (long long)k * NV);
      const int code = reinterpret_cast<const int*>(T.simp + L[k])[4 + f];
      const int nb = code >> 2;
      if (code < 0 || bad_simp(T, nb) || (__ldcg(B + (nb >> 5)) >> (nb & 31) & 1u)) continue;
      int4 v, n;
      load_simp(T, nb, v, n);
      if (query_side<D>(T, nb, v, p, fp, false, tl, perr) < 0) continue;
      if (atomicOr(B + (nb >> 5), 1u << (nb & 31)) >> (nb & 31) & 1u) continue;  // another thread has it
      const int at = atomicAdd(&s_n, 1);
      if (at < cap) L[at] = nb;
    }
    head = avail;
  }
  const int n = (int)min((long long)s_n, cap);  // a region has at most the tree's simplices
  if (threadIdx.x == 0) {
    if (s_n > cap) set_error(T.ctr, E_INTERNAL);
    cnt[b] = n;
  }
  for (int k = threadIdx.x; k < n; k += kLocThreads) {
    const int s = L[k];
    B[s >> 5] = 0u;  // every set bit of the word belongs to this region
    if (rank) L[k] = rank[s];
  }
  if (perr) set_error(T.ctr, E_PRECISION);
}

__global__ void k_live_flags(DevTree T, int nsimp, int* flags) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsimp; s += gridDim.x * blockDim.x)
    flags[s] = T.simp[s].v[0] >= 0 ? 1 : 0;
}

// Circumsphere of every live simplex, in the order of the simplex export
// (rank), for the dictionary view of the reference (PySimplex.center and
// .radius, src/lib.rs:32-59).  FP64 closed form relative to vertex 0:
// 3D c = p0 + (|a|^2 (b x c) + |b|^2 (c x a) + |c|^2 (a x b)) / (2 a.(b x c)),
// 2D the same in the plane.  These are floating-point values (the reference's
// own are too, src/geometry.rs:2-56); the triangulation never uses them.
template <int D>
__global__ void k_circum(DevTree T, int nsimp, const int* rank, double* centers, double* radii) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsimp; s += gridDim.x * blockDim.x) {
    const int4 v = reinterpret_cast<const int4*>(T.simp + s)[0];
    if (v.x < 0) continue;
    const int o = rank[s];
    const vdp::VPt p0 = T.pts[v.x], p1 = T.pts[v.y], p2 = T.pts[v.z];
    double cx, cy, cz = 0.0;
    if (D == 3) {
      const vdp::VPt p3 = T.pts[v.w];
      const double ax = p1.x - p0.x, ay = p1.y - p0.y, az = p1.z - p0.z;
      const double bx = p2.x - p0.x, by = p2.y - p0.y, bz = p2.z - p0.z;
      const double qx = p3.x - p0.x, qy = p3.y - p0.y, qz = p3.z - p0.z;
      const double a2 = ax * ax + ay * ay + az * az, b2 = bx * bx + by * by + bz * bz, q2 = qx * qx + qy * qy + qz * qz;
      const double bcx = by * qz - bz * qy, bcy = bz * qx - bx * qz, bcz = bx * qy - by * qx;
      const double cax = qy * az - qz * ay, cay = qz * ax - qx * az, caz = qx * ay - qy * ax;
      const double abx = ay * bz - az * by, aby = az * bx - ax * bz, abz = ax * by - ay * bx;
      const double den = 2.0 * (ax * bcx + ay * bcy + az * bcz);
      cx = (a2 * bcx + b2 * cax + q2 * abx) / den;
      cy = (a2 * bcy + b2 * cay + q2 * aby) / den;
      cz = (a2 * bcz + b2 * caz + q2 * abz) / den;
    } else {
      const double ax = p1.x - p0.x, ay = p1.y - p0.y, bx = p2.x - p0.x, by = p2.y - p0.y;
      const double a2 = ax * ax + ay * ay, b2 = bx * bx + by * by;
      const double den = 2.0 * (ax * by - ay * bx);
      cx = (by * a2 - ay * b2) / den;
      cy = (ax * b2 - bx * a2) / den;
    }
    centers[3LL * o] = p0.x + cx;
    centers[3LL * o + 1] = p0.y + cy;
    centers[3LL * o + 2] = D == 3 ? p0.z + cz : 0.0;
    radii[o] = sqrt(cx * cx + cy * cy + cz * cz);
  }
}

}  // namespace

void launch_circum(const DevTree& T, const Launch& L, int dim, int nsimp, const int* rank, double* centers,
                   double* radii) {
  note_launches(1);
  if (dim == 3)
    k_circum<3><<<L.blocks, 256, 0, L.stream>>>(T, nsimp, rank, centers, radii);
  else
    k_circum<2><<<L.blocks, 256, 0, L.stream>>>(T, nsimp, rank, centers, radii);
}

namespace {
template <int D, bool WIDE>
void locate_warp(const DevTree& T, const Launch& L, const double* d_q, const int* list, int n, const int* rank, int* out,
                 int cap_out, int2* res, int* total) {
  constexpr int W = LocWarp<D, WIDE>::WARPS;
  const int blocks = std::max(1, std::min((n + W - 1) / W, L.blocks));
  k_locate_warp<D, WIDE><<<blocks, 32 * W, 0, L.stream>>>(T, d_q, list, n, rank, out, cap_out, res, total);
}
}  // namespace

void launch_locate_warp(const DevTree& T, const Launch& L, int dim, bool wide, const double* d_q, const int* list, int n,
                        const int* rank, int* out, int cap_out, int2* res, int* total) {
  note_launches(1);
  cudaMemsetAsync(total, 0, sizeof(int), L.stream);
  if (dim == 3) {
    if (wide) locate_warp<3, true>(T, L, d_q, list, n, rank, out, cap_out, res, total);
    else locate_warp<3, false>(T, L, d_q, list, n, rank, out, cap_out, res, total);
  } else {
    if (wide) locate_warp<2, true>(T, L, d_q, list, n, rank, out, cap_out, res, total);
    else locate_warp<2, false>(T, L, d_q, list, n, rank, out, cap_out, res, total);
  }
}

void launch_locate_block(const DevTree& T, const Launch& L, int dim, const double* d_q, const int* list, int n,
                         const int2* res, const int* rank, int* lists, int64_t cap, unsigned* bits, int64_t words,
                         int* cnt) {
  note_launches(1);
  if (dim == 3)
    k_locate_block<3><<<n, kLocThreads, 0, L.stream>>>(T, d_q, list, res, rank, lists, cap, bits, words, cnt);
  else
    k_locate_block<2><<<n, kLocThreads, 0, L.stream>>>(T, d_q, list, res, rank, lists, cap, bits, words, cnt);
}

void launch_live_rank(const DevTree& T, const Launch& L, int nsimp, int* flags, int* rank, int* tmp) {
  note_launches(1);
  k_live_flags<<<L.blocks, 256, 0, L.stream>>>(T, nsimp, flags);
  scan_ints(flags, rank, nsimp, tmp, L.stream);
}

}  // namespace vd
