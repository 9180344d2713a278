// Point location queries on a finished tree: the conflict region of a query
// point, i.e. the simplices whose circumsphere strictly contains it
// (`locate`, src/delaunay_tree.rs:33-58 with find_all_neighbors :60-75).
//
// A visibility walk from the finest location hint of the set towards the
// simplex that contains the point, then a breadth-first search over face
// neighbours with the exact conflict test: a warp per query, or a thread per
// query where a region outgrows the warp's lists.  The query takes the role of
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

// Warp form: a warp per query, region lists in shared memory.  The walk stops
// at the first simplex whose stored sphere (3D) certainly holds the point: the
// conflict region is connected, so any of its simplices will do to start from.
// The region is searched in waves of 32 (simplex, face) items, as in the
// insertion rounds.  Bound by the chain of dependent gathers of one query
// (walk, then about six waves), with every query of a call in flight; the
// thread form below did a region's 50 tests one after another (4,096 queries in
// a 100,000-point tree: 1.2 ms a call, this form about 0.1 ms).
//
// res[i] = (count, first) of query i: count -1 outside the super simplex, -2
// when the region outgrew the lists (the caller then uses the thread form); its
// sorted ranks are out[first ..].  res[nq].x counts the ranks of all queries,
// which may exceed cap_out; with out null only the counts are made.
constexpr int kLocWarps = 4;
template <int D>
struct LocWarp {
  static constexpr int CAP = D == 3 ? 192 : 64, HS = D == 3 ? 512 : 128;
  int4 cn[CAP];
  int hk[HS];  // id set of the region, then its ranks while they are sorted
  int cav[CAP];
};

template <int D>
__global__ void __launch_bounds__(32 * kLocWarps, 4) k_locate_warp(DevTree T, const double* q, int nq, const int* rank,
                                                                  int* out, int cap_out, int2* res) {
  constexpr int NV = D + 1, CAP = LocWarp<D>::CAP, HS = LocWarp<D>::HS;
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ LocWarp<D> sm[kLocWarps];
  LocWarp<D>& W = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int qkey = 0x7fffffff;  // newer than every vertex
  vdp::Tally tl = {0, 0, 0, 0};
  int perr = 0;
  const SetGeo& g = T.sets[0];
  for (int i = blockIdx.x * kLocWarps + (threadIdx.x >> 5); i < nq; i += gridDim.x * kLocWarps) {
    const vdp::VPt p{q[(long long)i * D], q[(long long)i * D + 1], D == 3 ? q[(long long)i * D + 2] : 0.0, 0.0};
    const vdp::FPt fp = vdp::split_point(p.x, p.y, p.z);
    auto verts = [&](const int4& v, vdp::FPt* fv) {
      for (int j = 0; j < NV; ++j) fv[j] = T.ptf[g4(v, j)];
    };
    auto exit_of = [&](const int4& v) {
      vdp::FPt fv[NV];
      verts(v, fv);
      auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
        for (int j = 0; j < NV; ++j) v64[j] = T.pts[g4(v, j)];
        p64 = p;
      };
      return vdp::exit_face_hl<D>(fv, fp, (1u << NV) - 1, tl, perr, load64);
    };
    // 1 in conflict, -1 not; with `sphere` alone 0 where it cannot decide
    auto conflict = [&](int s, const int4& v, bool sphere) {
      if (D == 3) {
        const float4 c = *reinterpret_cast<const float4*>(T.sph + s);
        const int side = vdp::sphere_side<D>(vdp::Sph{c.x, c.y, c.z, c.w}, fp);
        if (side != 0) return side;
      }
      if (sphere) return 0;
      vdp::FPt fv[NV];
      int key[NV];
      verts(v, fv);
      for (int j = 0; j < NV; ++j) key[j] = g4(v, j);
      auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
        for (int j = 0; j < NV; ++j) v64[j] = T.pts[key[j]];
        p64 = p;
      };
      return vdp::in_conflict_hl<D>(fv, key, fp, qkey, tl, perr, load64) ? 1 : -1;
    };
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
    } else if (n > 0 && out) {
      if (lane == 0) first = atomicAdd(&res[nq].x, n);
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
      atomicAdd(&res[nq].x, n);
    }
    if (lane == 0) res[i] = make_int2(n, first);
  }
  if (perr) set_error(T.ctr, E_PRECISION);
}

template <int D>
__global__ void k_locate(DevTree T, const double* q, int nq, int cap_per, const int* rank, int* out, int* counts) {
  constexpr int NV = D + 1;
  const int qkey = 0x7fffffff;  // newer than every vertex
  vdp::Tally tl = {0, 0, 0, 0};
  int perr = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
    const vdp::VPt p{q[(long long)i * D], q[(long long)i * D + 1], D == 3 ? q[(long long)i * D + 2] : 0.0, 0.0};
    const vdp::FPt fp = vdp::split_point(p.x, p.y, p.z);
    const SetGeo& g = T.sets[0];
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
    int* o = out + (long long)i * cap_per;
    if (v.x < 0 || bad_simp(T, cur)) {
      set_error(T.ctr, E_INTERNAL);
      counts[i] = 0;
      continue;
    }
    // visibility walk
    bool outside = false;
    for (int step = 0; step < (1 << 16); ++step) {
      vdp::FPt fv[NV];
      for (int j = 0; j < NV; ++j) fv[j] = T.ptf[g4(v, j)];
      auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
        for (int j = 0; j < NV; ++j) v64[j] = T.pts[g4(v, j)];
        p64 = p;
      };
      const int f = vdp::exit_face_hl<D>(fv, fp, (1u << NV) - 1, tl, perr, load64);
      if (f < 0) break;
      const int code = g4(nn, f);
      if (code < 0 || bad_simp(T, code >> 2)) {
        outside = code < 0;
        break;
      }
      cur = code >> 2;
      load_simp(T, cur, v, nn);
    }
    if (outside) {
      counts[i] = -1;
      continue;
    }
    // breadth-first search of the conflict region (the containing simplex
    // is in it unless the point is one of its vertices)
    int cnt = 0;
    auto conflict = [&](int s, const int4& sv) {
      vdp::FPt fv[NV];
      int key[NV];
      for (int j = 0; j < NV; ++j) {
        key[j] = g4(sv, j);
        fv[j] = T.ptf[key[j]];
      }
      auto load64 = [&](vdp::VPt* v64, vdp::VPt& p64) {
        for (int j = 0; j < NV; ++j) v64[j] = T.pts[key[j]];
        p64 = p;
      };
      return vdp::in_conflict_hl<D>(fv, key, fp, qkey, tl, perr, load64);
    };
    if (conflict(cur, v)) {
      if (cap_per > 0) o[0] = cur;
      cnt = 1;
    }
    for (int h = 0; h < cnt && h < cap_per; ++h) {
      int4 cv, cn;
      load_simp(T, o[h], cv, cn);
      for (int f = 0; f < NV; ++f) {
        const int code = g4(cn, f);
        if (code < 0) continue;
        const int nb = code >> 2;
        if (bad_simp(T, nb)) continue;
        bool seen = false;
        for (int k = 0; k < cnt && k < cap_per && !seen; ++k) seen = o[k] == nb;
        if (seen) continue;
        int4 bv, bn;
        load_simp(T, nb, bv, bn);
        if (!conflict(nb, bv)) continue;
        if (cnt < cap_per) o[cnt] = nb;
        ++cnt;
      }
    }
    for (int k = 0; k < cnt && k < cap_per; ++k) o[k] = rank[o[k]];  // numbering of the simplex export
    counts[i] = cnt;
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

void launch_locate(const DevTree& T, const Launch& L, int dim, const double* d_q, int nq, int cap_per,
                   const int* rank, int* out, int* counts) {
  note_launches(1);
  const int blocks = std::max(1, std::min((nq + 127) / 128, L.blocks * 2));
  if (dim == 3)
    k_locate<3><<<blocks, 128, 0, L.stream>>>(T, d_q, nq, cap_per, rank, out, counts);
  else
    k_locate<2><<<blocks, 128, 0, L.stream>>>(T, d_q, nq, cap_per, rank, out, counts);
}

void launch_locate_warp(const DevTree& T, const Launch& L, int dim, const double* d_q, int nq, const int* rank, int* out,
                        int cap_out, int2* res) {
  note_launches(1);
  cudaMemsetAsync(res + nq, 0, sizeof(int2), L.stream);
  const int blocks = std::max(1, std::min((nq + kLocWarps - 1) / kLocWarps, L.blocks));
  if (dim == 3)
    k_locate_warp<3><<<blocks, 32 * kLocWarps, 0, L.stream>>>(T, d_q, nq, rank, out, cap_out, res);
  else
    k_locate_warp<2><<<blocks, 32 * kLocWarps, 0, L.stream>>>(T, d_q, nq, rank, out, cap_out, res);
}

void launch_live_rank(const DevTree& T, const Launch& L, int nsimp, int* flags, int* rank, int* tmp) {
  note_launches(1);
  k_live_flags<<<L.blocks, 256, 0, L.stream>>>(T, nsimp, flags);
  scan_ints(flags, rank, nsimp, tmp, L.stream);
}

}  // namespace vd
