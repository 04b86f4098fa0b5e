// Mesh pass of the exact cell-tet form: the part of a finished cell that lies
// in the mesh, without building the pieces cell ^ tet.
//
// The volume and first moment of cell ^ mesh are sums over its boundary: over
// each face of the cell, the part inside the mesh; over each boundary
// triangle of the mesh, the part inside the cell.  Split into signed tets
// from an apex (the apex, the foot of the apex on a face, a piece of one of
// the face's edges), only lines are left:
//   * the cell's edges, each as far as it lies in the mesh.  A tet cuts a
//     length off an edge (an interval of four plane tests); the lengths of
//     all the tets add up on the lane that holds the edge.  Where two tets
//     share a face, that face and its lines give opposite terms and drop out;
//   * for each open triangle (a tet face that no other tet shares from its
//     other side), the polygon triangle ^ cell: its edges on the cell's faces
//     and on its own sides.
// Summing det(F1 - F0, a, b) / 6 over the pieces [a, b] of every line of two
// faces (feet F0, F1) gives the volume, and (F + a + b) / 4 of each signed tet
// the moment.  The sums are kept in pairs of floats from one batch of tets to
// the next, and where terms cancel (much of the cell outside the mesh) they are
// taken again from the barycentre found: against 64 bits, root mean square, the
// volumes of shares 0.01 to 0.1 of a cell 7.5e-7 -> 3.3e-7 off (clipped by each
// tet 3.8e-7), of shares above a half 7.7e-8 -> 5.5e-8 (8.1e-8); an iteration
// costs 2% more for it.
//
// Consistency.  A tet face is one plane for both its tets: its three vertices
// in mesh order make it, so an edge's interval ends where the next tet's
// begins, bit for bit, also where the edge grazes the face or lies in it
// within rounding.  Points that two lines share are made once: where an edge
// of the cell meets a triangle (on the edge), where a side of a triangle meets
// a face of the cell (on the side).  Lines are kept as their point nearest
// the site and a unit direction, so that a long edge of an open cell is as
// exact near the site as a short one.  Where that is not enough (an edge and a
// triangle's side within rounding of each other, a face in a triangle's plane)
// the lines of a face or a triangle no longer close, which one more sum over
// the pieces tells (face_mark): the cell is given back and clipped by each tet.
//
// One warp per site: lanes take candidate tets, then (tet, edge) pairs, then
// faces.  Bound by latency (issuing on 65% of cycles, five blocks of four warps
// per SM; stalls on fixed latencies and on the tets' records from L2).  Loops
// are kept rolled: at 70 KB of code half the stalls were instruction fetches
// and the pass took 2.0 ms where it took 1.4 at 50 KB (1.5 with the checks and
// sums above).  A boundary cell (at 1M torus sites 36 edges, 20 tets, 6 open
// triangles) needs no vertices of its pieces, whose inner faces only cancel.
// Measured per Lloyd iteration, 1M sites in 1.96M tets: 15.0 -> 5.9 ms from random
// sites and 4.6 -> 1.9 ms once relaxed (the one-warp pass before, now that pass
// without its tets and this one).
#pragma once

#include "clip_warp.cuh"

namespace vgb {

constexpr int MESH_WARPS = 4;
// A cell of at most 64 vertices (three faces meet in each) has at most 34
// faces and 96 edges.
constexpr int MESH_FACES = 34, MESH_EDGES = 96;
static_assert(MESH_EDGES == 3 * MESH_VERTS / 2 && MESH_FACES == MESH_VERTS / 2 + 2, "a simple polytope");
constexpr int MESH_TETS = 16;  // tets in hand
constexpr int MESH_IDS = 4 + MAX_SITE_K + 12 + MESH_EXT;  // plane ids a stored cell may use
constexpr int MESH_ID_WORDS = (MESH_IDS + 31) / 32;
// A cell whose terms exceed this many times their sum keeps a sliver of
// itself in the mesh (one in a thousand of the boundary cells of random sites,
// the site mostly outside): the terms' rounding, 1e-7 of a cell, would show in
// it, so a pass that follows clips it by each tet.
constexpr float MESH_RATIO = 64.f;
// Above this many times (a quarter of the cell or less in the mesh, mostly) the
// sum is taken again from the barycentre of what the first sum found: shares of
// 0.01 to 0.1 of a cell, volumes rms 7.1e-7 -> 3.3e-7 off, barycentres 2.6e-7 ->
// 0.6e-7 of a cell's size; at 8 instead of 4 the barycentres of shares up to a
// half are 1.3 times as far off, for 0.5% of an iteration.
constexpr float MESH_NEAR = 4.f;
// So it does with a cell whose faces' lines leave more than these parts of its
// radius and of all their lengths open: the ends of pieces are rounded to 1e-7
// of the radius each, their sum to as much of what it went through.
// Where three planes nearly share a line and that line nearly lies in one of the
// mesh's planes (sites of a lattice along the mesh's axes), the sides that
// rounding gives a point of an edge and of a triangle may disagree, and a piece
// is lost, or counted twice.
constexpr float MESH_CLOSED = 2e-5f, MESH_WAY = 5e-7f;
#ifndef VGB_MESH_MIN_BLOCKS
#define VGB_MESH_MIN_BLOCKS 5
#endif

constexpr unsigned EDGE_BACK = 0x80000000u;

struct MeshSmem {
  float4 plane[MESH_FACES];  // the cell's faces, site-relative
  union {
    struct {
      unsigned char loc[MESH_ID_WORDS * 32];  // plane id -> face
    };
    float4 tp[MESH_TETS][4];  // the face planes of the tets in hand, in mesh order
  };
  union {
    unsigned char twin[MESH_FACES * MESH_FACES];  // (p, q) -> vertex, while the edges are made
    float4 slot[2][MESH_FACES];  // a triangle's plane across each face: first and second point
  };
  // the cell's edges: point nearest the site and direction, with the smaller
  // and the larger end parameter; the terms of a unit of its length (volume in w)
  float4 epos[MESH_EDGES], edir[MESH_EDGES], eterm[MESH_EDGES];
  unsigned edge[MESH_EDGES];  // faces p, q and end vertices of each (EDGE_BACK: its end lies before its start)
  float eopen[MESH_EDGES];    // what a unit of its length leaves open (face_mark)
  float3 vert[MESH_VERTS];    // the cell's vertices
  float4 side[3][2];  // a triangle's sides: point and direction, end parameters in w
  float at[3][MESH_FACES];  // where each face meets them
  int tidx[MESH_TETS];  // tets in hand: their record, and what is known of them
  unsigned char tinf[MESH_TETS], thit[MESH_TETS];
  int queue[2 * WARP];  // tets whose sphere meets the cell's
  int rng[2][WARP];     // the rows in hand: first tet, tets of the rows before
  unsigned cnt[WC_N];
  unsigned here[WC_N], spare[WC_N];  // of the site in hand; of its second sum (not counted)
  unsigned tr2[MESH_TETS];           // tet-cell method: how far each tet's piece reaches (squared, float bits),
  unsigned char tfar[MESH_TETS];     // and the tets that reach far enough to matter
};

// dot product ending in + c, the same rounding in every kernel
__device__ __forceinline__ float fma3(float ax, float ay, float az, float bx, float by, float bz, float c) {
  return __fmaf_rn(ax, bx, __fmaf_rn(ay, by, __fmaf_rn(az, bz, c)));
}
__device__ __forceinline__ float eval4(float4 P, float3 x) { return fma3(P.x, P.y, P.z, x.x, x.y, x.z, P.w); }
__device__ __forceinline__ float3 cross_rn(float3 a, float3 b) {
  return make_float3(cross_term(a.y, b.z, a.z, b.y), cross_term(a.z, b.x, a.x, b.z), cross_term(a.x, b.y, a.y, b.x));
}
__device__ __forceinline__ float dot_rn(float3 a, float3 b) { return dot3_rn(a.x, a.y, a.z, b.x, b.y, b.z); }
__device__ __forceinline__ float3 sub_rn(float3 a, float3 b) {
  return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 along(float3 p, float t, float3 u) {
  return make_float3(__fmaf_rn(t, u.x, p.x), __fmaf_rn(t, u.y, p.y), __fmaf_rn(t, u.z, p.z));
}
__device__ __forceinline__ float3 xyz(float4 v) { return make_float3(v.x, v.y, v.z); }

// Where the line p + t u meets plane P, and whether the plane's positive side
// lies ahead.  A line in the plane's direction meets it at -inf or +inf,
// with "ahead": then every point of it is on the positive side (P >= 0) or
// none is.  (The 1e-37 decides the line in the plane: positive side.)
__device__ __forceinline__ float line_at(float4 P, float3 p, float3 u, bool& ahead) {
  const float d = fma3(P.x, P.y, P.z, p.x, p.y, p.z, P.w);
  const float du = fma3(P.x, P.y, P.z, u.x, u.y, u.z, 0.f);
  ahead = du >= 0.f;
  return __fdividef(__fsub_rn(-1e-37f, d), du);
}

// Signed tets of the piece [a, b] on the line of faces 0 and 1 (feet F0, F1;
// all relative to the apex, the site at first; ab = a + b).  A lane's terms of a
// batch of tets are added up plainly, the batches with their rounding kept.
struct MeshSum {
  float v = 0.f, x = 0.f, y = 0.f, z = 0.f, mag = 0.f, open = 0.f, way = 0.f;
  // compensated: what the batches of tets before this one gave
  float hv = 0.f, hx = 0.f, hy = 0.f, hz = 0.f, lv = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
  __device__ __forceinline__ void add(float k, float mx, float my, float mz) {
    v = __fadd_rn(v, k);
    mag = __fadd_rn(mag, fabsf(k));
    x = __fadd_rn(x, mx);
    y = __fadd_rn(y, my);
    z = __fadd_rn(z, mz);
  }
  __device__ __forceinline__ void add(float k, float3 F, float3 ab) {
    add(k, __fmul_rn(k, __fadd_rn(F.x, ab.x)), __fmul_rn(k, __fadd_rn(F.y, ab.y)), __fmul_rn(k, __fadd_rn(F.z, ab.z)));
  }
  __device__ __forceinline__ void close(float o) {
    open = __fadd_rn(open, o);
    way = __fadd_rn(way, fabsf(o));
  }
  __device__ __forceinline__ void flush() {
    comp_add(hv, lv, v);
    comp_add(hx, lx, x);
    comp_add(hy, ly, y);
    comp_add(hz, lz, z);
    v = x = y = z = 0.f;
  }
  // over the warp (one loop, not unrolled: unrolled a quantity at a time these
  // sums are 5 KB of code)
  __device__ __forceinline__ void reduce() {
#pragma unroll 1
    for (int o = WARP / 2; o > 0; o >>= 1) {
      auto pair = [o](float& h, float& l) {
        const float x = __shfl_xor_sync(FULL, h, o), y = __shfl_xor_sync(FULL, l, o);
        comp_add(h, l, x);
        l += y;
      };
      pair(hv, lv);
      pair(hx, lx);
      pair(hy, ly);
      pair(hz, lz);
      mag += __shfl_xor_sync(FULL, mag, o);
      open += __shfl_xor_sync(FULL, open, o);
      way += __shfl_xor_sync(FULL, way, o);
    }
  }
};
// Around each face of a cell, and around each triangle, the pieces of its lines
// close: their vectors sum to nothing.  One sum checks them all, each piece by
// its product with a vector of its face (hashed, components within 1).
__device__ __forceinline__ float3 face_mark(unsigned f) {
  const unsigned h = (f + 1u) * 0x9e3779b1u, i = h * 0x85ebca6bu, j = i * 0xc2b2ae35u;
  return make_float3(__uint_as_float(0x40000000u | (h >> 9)) - 3.f, __uint_as_float(0x40000000u | (i >> 9)) - 3.f,
                     __uint_as_float(0x40000000u | (j >> 9)) - 3.f);
}

// Foot of the apex X on plane P, relative to X.
__device__ __forceinline__ float3 foot_of(float4 P, float3 X) {
  const float nn = dot3_rn(P.x, P.y, P.z, P.x, P.y, P.z);
  const float l = __fdividef(-eval4(P, X), nn);
  return make_float3(__fmul_rn(l, P.x), __fmul_rn(l, P.y), __fmul_rn(l, P.z));
}

// Largest / smallest of one float per lane (one instruction each).
__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float redux_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// The segment [P, Q] as a line (point nearest the origin, unit direction,
// end parameters).
struct Line {
  float3 p, u;
  float a, b;
};
__device__ __forceinline__ Line line_of(float3 P, float3 Q) {
  Line L;
  const float3 d = sub_rn(Q, P);
  const float dd = dot_rn(d, d), r0 = rsqrtf(dd);
  const float il = __fmul_rn(r0, __fmaf_rn(__fmul_rn(-0.5f * dd, r0), r0, 1.5f));  // (one Newton step)
  L.u = make_float3(__fmul_rn(d.x, il), __fmul_rn(d.y, il), __fmul_rn(d.z, il));
  L.a = dot_rn(P, L.u);
  L.b = dot_rn(Q, L.u);
  L.p = along(P, -L.a, L.u);
  return L;
}

// info word of a tet record (its 13th float's bits): open faces 0-3 (by the
// vertex they leave out, in mesh order), 4: mesh order is an even permutation
// of a positively oriented tet, 5: not positively oriented (meets nothing)
constexpr unsigned REC_EVEN = 16u, REC_SKIP = 32u;
// the side of its canonical plane i the tet lies on (true: positive)
__device__ __forceinline__ bool face_side(unsigned info, int i) { return ((info >> 4) & 1u) == (unsigned)(i & 1); }

// REF (reference form): a site's sum is over the tets it is a candidate of
// (one of the tet_k nearest sites of their centroid), and the face between
// such a tet and one it is no candidate of is open.  PAIRS (tet-cell method): the
// counter of misses is of its pieces, not of cells.
template <bool BATCHED, bool REF, bool PAIRS = false>
__global__ void __launch_bounds__(MESH_WARPS * WARP, VGB_MESH_MIN_BLOCKS) k_cell_mesh(
    const float4* __restrict__ sites, const unsigned* __restrict__ knn, const ProbDesc* __restrict__ probs,
    const int* __restrict__ site_prob, const ProbDesc lone, const float4* __restrict__ rec,
    const int* __restrict__ tet_cell_start, const float4* __restrict__ tet_sph, const float* __restrict__ reach,
    const unsigned* __restrict__ reach_max_bits, dmom4* __restrict__ mom, unsigned long long* __restrict__ stats,
    unsigned* __restrict__ prob_secmiss, const int* __restrict__ in_list, const int* __restrict__ in_count,
    int* __restrict__ work, int* __restrict__ out_list, int* __restrict__ out_count, const CellStore store,
    int* __restrict__ esc_list, float* __restrict__ esc_r2, int* __restrict__ esc_count,
    const int* __restrict__ site_start) {
  __shared__ MeshSmem smem_all[MESH_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  MeshSmem& S = smem_all[wib];
  if (lane < WC_N) S.cnt[lane] = 0u;
  __syncwarp();
  const int n_items = *in_count;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(work, 1);
    it = __shfl_sync(FULL, it, 0);
    if (it >= n_items) break;
    const int s = in_list[it];
    const int pidx = BATCHED ? site_prob[s] : 0;
#define PD(f) (BATCHED ? probs[pidx].f : lone.f)
    const float4 seed = sites[s];
    const int word = store.mnt[s];
    const int nt = min(word & 255, MESH_VERTS);
    unsigned flags = ((unsigned)word >> 8) & 255u;
    const int K = PD(K);
    const unsigned* const krow = knn + PD(knn_off) + (size_t)(s - PD(site_off)) * K;
    const bool miss = (flags & SITE_SECMISS) && !(flags & SITE_COMPLETED);
    const float dK2 = miss && (!REF || PAIRS) ? dist2(seed, sites[krow[K - 1]]) : FLT_MAX;
    if (lane < WC_N) S.here[lane] = 0u;

    // -----------------------------------------------------------------
    // the cell: its faces, vertices and edges
    unsigned T[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = k * WARP + lane;
      T[k] = i < nt ? store.mtri[(size_t)s * MESH_VERTS + i] : 0u;
    }
    for (int i = lane; i < MESH_ID_WORDS * 8; i += WARP) reinterpret_cast<unsigned*>(S.loc)[i] = 0u;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (k * WARP + lane < nt) {
#pragma unroll
        for (int e = 0; e < 3; ++e) S.loc[min(tri_at(T[k], e), (unsigned)(MESH_IDS - 1))] = 1;
      }
    __syncwarp();
    int nf = 0;
#pragma unroll 1
    for (int w = 0; w < MESH_ID_WORDS; ++w) {
      const int id = w * WARP + lane;
      const bool has = S.loc[id] != 0;
      const unsigned m = __ballot_sync(FULL, has);
      const int f = min(nf + __popc(m & lt_mask), MESH_FACES - 1);
      if (has) {
        S.loc[id] = (unsigned char)f;
        float4 P;
        if (id < 4 + K) {
          P = bisector_plane(seed, sites[krow[max(id - 4, 0)]]);
        } else if (id < 4 + K + 2 * BOX_PLANES) {
          P = start_plane(id - 4 - K, seed, cube_half_side(seed));
        } else {
          P = bisector_plane(seed, sites[store.faces[(size_t)s * PIECE_REC + min(id - (4 + K + 2 * BOX_PLANES), MESH_EXT - 1)]]);
        }
        S.plane[f] = P;
      }
      nf += __popc(m);
    }
    __syncwarp();
    bool bad = nf > MESH_FACES || nt < 4 ;
    nf = min(nf, MESH_FACES);
    float lm = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = k * WARP + lane;
      if (i < nt) {
        const unsigned a = S.loc[min(tri_at(T[k], 0), (unsigned)(MESH_IDS - 1))];
        const unsigned b = S.loc[min(tri_at(T[k], 1), (unsigned)(MESH_IDS - 1))];
        const unsigned c = S.loc[min(tri_at(T[k], 2), (unsigned)(MESH_IDS - 1))];
        const float3 x = vertex_of(S.plane[a], S.plane[b], S.plane[c]);
        const float r2 = norm2_rn(x);
        S.vert[i] = x;
        lm = fmaxf(lm, r2);
        T[k] = pack_tri(a, b, c);
        S.twin[a * MESH_FACES + b] = (unsigned char)i;
        S.twin[b * MESH_FACES + c] = (unsigned char)i;
        S.twin[c * MESH_FACES + a] = (unsigned char)i;
      }
    }
    const float Rc = sqrtf(warp_max_nonneg(lm));
    __syncwarp();
    // an edge is the directed pair (p, q) of one vertex and (q, p) of another
    int ne = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k * WARP >= nt) break;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const unsigned p = tri_at(T[k], e), q = tri_at(T[k], e == 2 ? 0 : e + 1);
        const bool has = k * WARP + lane < nt && p < q;
        const unsigned m = __ballot_sync(FULL, has);
        const int pos = ne + __popc(m & lt_mask);
        if (has && pos < MESH_EDGES)
          S.edge[pos] = p | (q << 8) | ((unsigned)(k * WARP + lane) << 16) |
                        ((unsigned)(S.twin[q * MESH_FACES + p] & (MESH_VERTS - 1)) << 24);
        ne += __popc(m);
      }
    }
    bad |= ne > MESH_EDGES || ne < 6;
    ne = max(min(ne, MESH_EDGES), 1);
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < ne; i += WARP) {
      const unsigned E = S.edge[i];
      const float4 P = S.plane[E & 0xffu], Q = S.plane[(E >> 8) & 0xffu];
      const float3 D = cross_rn(xyz(Q), xyz(P));  // from the end whose vertex holds (p, q)
      const float dd = dot_rn(D, D);
      const float3 a = cross_rn(xyz(P), D), b = cross_rn(D, xyz(Q));
      const float i2 = __fdividef(-1.f, dd), i1 = rsqrtf(dd);
      const float3 u = make_float3(__fmul_rn(D.x, i1), __fmul_rn(D.y, i1), __fmul_rn(D.z, i1));
      const float3 p = make_float3(__fmul_rn(i2, __fmaf_rn(Q.w, a.x, __fmul_rn(P.w, b.x))),
                                   __fmul_rn(i2, __fmaf_rn(Q.w, a.y, __fmul_rn(P.w, b.y))),
                                   __fmul_rn(i2, __fmaf_rn(Q.w, a.z, __fmul_rn(P.w, b.z))));
      // Where planes nearly share a line, rounding may place a vertex beyond
      // its neighbour: an edge from its end back to its start, whose terms
      // count against those of the edges that reach too far
      const float t0 = dot_rn(S.vert[(E >> 16) & 0xffu], u), t1 = dot_rn(S.vert[E >> 24], u);
      S.epos[i] = make_float4(p.x, p.y, p.z, fminf(t0, t1));
      S.edir[i] = make_float4(u.x, u.y, u.z, fmaxf(t0, t1));
      const float sg = t1 < t0 ? -1.f : 1.f;
      S.eopen[i] = __fmul_rn(sg, dot_rn(u, sub_rn(face_mark((E >> 8) & 0xffu), face_mark(E & 0xffu))));
      if (sg < 0.f) S.edge[i] = E | EDGE_BACK;
    }
    __syncwarp();

    // -----------------------------------------------------------------
    // the tets
    float3 X = make_float3(0.f, 0.f, 0.f);  // apex
    float pr2 = 0.f;
    double moment = 0.0;  // lanes 0-3: volume and first moment
    bool open = false;    // its faces' lines do not close
    bool beyond = false;  // sites beyond the K nearest may cut what is in the mesh
    const int dim = PD(dim), cbase = PD(cell_off);
    const float rt = REF ? __uint_as_float(reach_max_bits[1]) : PD(rt_max);
    const float R = __fadd_rn(fminf(__fmaf_rn(rt, 1.001f, Rc), __uint_as_float(reach_max_bits[pidx])), 0.01f);
    // is the site a candidate of the tet? (the search's order: distance, then id)
    auto candidate = [&](int q) {
      const float2 z = store.last[q];
      const float d2 = dist2(tet_sph[q], seed);
      return d2 < z.x || (d2 == z.x && site_id(seed) <= __float_as_int(z.y));
    };
    const float h = 1000.f / (float)dim;
    // (the cell of a coordinate up to its rounding, well below the margins)
    const float per = __fmul_rn((float)dim, 1e-3f);
    auto cell_at = [&](float x) { return min(max((int)floorf(__fmul_rn(x, per)), 0), dim - 1); };
    const int j0 = cell_at(seed.y - R), k0 = cell_at(seed.z - R);
    const int nj = cell_at(seed.y + R) - j0 + 1;
    const int nrow = nj * (cell_at(seed.z + R) - k0 + 1);
    const float per_row = __fdividef(1.f, (float)nj);
#pragma unroll 1
    for (bool again = false; !bad;) {
      MeshSum sum;
      float far2 = 0.f;
      unsigned* const here = again ? S.spare : S.here;
      int skew = 0;  // ends of crossing edges, less the faces' slots they took
      // a piece [a, b] of an edge: k = det(F1 - F0, p, u) (b - a), and the
      // moment k1 (F1 + a + b) - k0 (F0 + a + b), all relative to X
#pragma unroll 1
      for (int i = lane; i < ne; i += WARP) {
        const unsigned E = S.edge[i];
        const float3 F0 = foot_of(S.plane[E & 0xffu], X), F1 = foot_of(S.plane[(E >> 8) & 0xffu], X);
        const float3 p = sub_rn(xyz(S.epos[i]), X), cr = cross_rn(p, xyz(S.edir[i]));
        const float sg = (E & EDGE_BACK) ? -1.f : 1.f;
        const float k0 = __fmul_rn(sg, dot_rn(F0, cr)), k1 = __fmul_rn(sg, dot_rn(F1, cr)), k = __fsub_rn(k1, k0);
        const float k2 = 2.f * k;
        S.eterm[i] = make_float4(__fmaf_rn(k2, p.x, cross_term(k1, F1.x, k0, F0.x)),
                                 __fmaf_rn(k2, p.y, cross_term(k1, F1.y, k0, F0.y)),
                                 __fmaf_rn(k2, p.z, cross_term(k1, F1.z, k0, F0.z)), k);
      }
      __syncwarp();
      int nq = 0, row0 = 0, f0 = 0, total = 0, incl = 0;
      bool more = true;
      while (more || nq > 0) {
        // candidates to the queue: rows of centroid cells, 32 rows at a time,
        // each cut to the ball of radius R, then 32 tets at a time
        while (more && nq < WARP) {
          if (f0 >= total) {
            if (row0 >= nrow) {
              more = false;
              break;
            }
            const int r = row0 + lane;
            int len = 0, rb = 0;
            if (r < nrow) {
              const int rk = (int)__fmul_rn((float)r + 0.5f, per_row), k = k0 + rk, j = j0 + r - rk * nj;
              // (the cells at the ends of the grid also hold what lies beyond)
              const float m = 0.01f;
              float lo = j == 0 ? -FLT_MAX : __fmaf_rn((float)j, h, -m);
              float hi = j == dim - 1 ? FLT_MAX : __fmaf_rn((float)(j + 1), h, m);
              const float dy = fmaxf(fmaxf(lo - seed.y, seed.y - hi), 0.f);
              lo = k == 0 ? -FLT_MAX : __fmaf_rn((float)k, h, -m);
              hi = k == dim - 1 ? FLT_MAX : __fmaf_rn((float)(k + 1), h, m);
              const float dz = fmaxf(fmaxf(lo - seed.z, seed.z - hi), 0.f);
              const float left = __fmaf_rn(__fmul_rn(R, R), 1.0001f, -__fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
              if (left >= 0.f) {
                const float w = __fmaf_rn(left, rsqrtf(fmaxf(left, 1e-12f)), m);
                const int row = cbase + dim * (j + dim * k);
                rb = tet_cell_start[row + cell_at(seed.x - w)];
                len = tet_cell_start[row + cell_at(seed.x + w) + 1] - rb;
              }
            }
            row0 += WARP;
            incl = len;
#pragma unroll
            for (int o = 1; o < WARP; o <<= 1) {
              const int y = __shfl_up_sync(FULL, incl, o);
              if (lane >= o) incl += y;
            }
            total = __shfl_sync(FULL, incl, WARP - 1);
            f0 = 0;
            __syncwarp();
            S.rng[0][lane] = rb;
            S.rng[1][lane] = incl - len;
            __syncwarp();
            continue;
          }
          const int f = f0 + lane;
          int lo = 0;  // the row holding f
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            const int v = __shfl_sync(FULL, incl, lo + step - 1);
            if (v <= f) lo += step;
          }
          const int idx = S.rng[0][lo] + f - S.rng[1][lo];
          bool meets = false;
          if (f < total) {
            // bounding spheres (the cell lies within Rc of its site), and the
            // tet's reach: beyond it every point of the tet has a nearer site
            const float4 sp = tet_sph[idx];
            const float ex = sp.x - seed.x, ey = sp.y - seed.y, ez = sp.z - seed.z;
            const float d2 = dot3_rn(ex, ey, ez, ex, ey, ez), ds = __fmaf_rn(__fadd_rn(Rc, sp.w), 1.0001f, 1e-3f);
            meets = d2 <= __fmul_rn(ds, ds);
            if (meets) {
              if (REF) {
                meets = candidate(idx);
              } else {
                const float dr = __fmaf_rn(reach[idx], 1.0001f, 1e-2f);
                meets = d2 <= __fmul_rn(dr, dr);
              }
            }
          }
          const unsigned m = __ballot_sync(FULL, meets);
          if (meets) S.queue[nq + __popc(m & lt_mask)] = idx;
          nq += __popc(m);
          if (!REF && lane == 0) here[WC_CAND] += (unsigned)min(WARP, total - f0);
          f0 += WARP;
        }
        if (nq == 0) break;
        __syncwarp();
        // 32 of them (the rest of the queue at the end), one per lane: a tet
        // with all four corners strictly outside one face cannot meet the cell
        const int take = min(nq, WARP);
        const int idx = lane < take ? S.queue[lane] : 0;
        bool alive = lane < take;
        float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
        unsigned info = 0u;
        if (alive) {
          const float4* q = rec + 4 * (size_t)idx;
          r0 = q[0];
          r1 = q[1];
          r2 = q[2];
          info = __float_as_uint(q[3].x);
          alive = !(info & REC_SKIP);
        }
        const float3 A0 = make_float3(r0.x, r0.y, r0.z), A1 = make_float3(r0.w, r1.x, r1.y),
                     A2 = make_float3(r1.z, r1.w, r2.x), A3 = make_float3(r2.y, r2.z, r2.w);
        const float3 sd = make_float3(seed.x, seed.y, seed.z);
        const float3 c0 = sub_rn(A0, sd), c1 = sub_rn(A1, sd), c2 = sub_rn(A2, sd), c3 = sub_rn(A3, sd);
        unsigned tests = 0u;
#pragma unroll 2
        for (int f = 0; f < nf; ++f) {
          if (!__any_sync(FULL, alive)) break;
          tests += alive;
          const float4 P = S.plane[f];
          const float e = fmaxf(fmaxf(eval4(P, c0), eval4(P, c1)), fmaxf(eval4(P, c2), eval4(P, c3)));
          alive &= !(e < 0.f);
        }
        const unsigned tested = __reduce_add_sync(FULL, tests);
        const unsigned am = __ballot_sync(FULL, alive);
        const int nb = min(__popc(am), MESH_TETS), place = __popc(am & lt_mask);
        // the rest of the queue to its front, then what is more than can be
        // held (those are looked at again)
        const int rest = nq - take;
        const int move = lane < rest ? S.queue[take + lane] : 0;
        __syncwarp();
        if (lane < rest) S.queue[lane] = move;
        if (alive && place >= MESH_TETS) S.queue[rest + place - MESH_TETS] = idx;
        alive &= place < MESH_TETS;
        nq = rest + __popc(am) - nb;
        if (lane == 0) {
          here[WC_CLIPPED] += (unsigned)nb;
          here[WC_CULLTESTS] += tested;
          here[WC_CONFLICT] += (unsigned)(8 * ne * nb);
        }
        if (alive) {
          const int pos = place;
          auto face = [&](int i, float3 a, float3 b, float3 c, float3 ca) {
            const float3 n = cross_rn(sub_rn(b, a), sub_rn(c, a));
            S.tp[pos][i] = make_float4(n.x, n.y, n.z, -dot_rn(n, ca));
          };
          face(0, A1, A2, A3, c1);
          face(1, A0, A2, A3, c0);
          face(2, A0, A1, A3, c0);
          face(3, A0, A1, A2, c0);
          unsigned far = 0u;
          if (miss && (!REF || PAIRS)) {
            const float m2 = fmaxf(fmaxf(dot_rn(c0, c0), dot_rn(c1, c1)), fmaxf(dot_rn(c2, c2), dot_rn(c3, c3)));
            far = !(dK2 > __fmaf_rn(4.f * m2, 1.0001f, 1e-4f)) ? 64u : 0u;
          }
          S.tidx[pos] = idx;
          if (REF) {
            const int4 nb4 = store.beside[idx];
            if (nb4.x >= 0 && !candidate(nb4.x)) info |= 1u;
            if (nb4.y >= 0 && !candidate(nb4.y)) info |= 2u;
            if (nb4.z >= 0 && !candidate(nb4.z)) info |= 4u;
            if (nb4.w >= 0 && !candidate(nb4.w)) info |= 8u;
          }
          S.tinf[pos] = (unsigned char)((info & 31u) | far);
          S.thit[pos] = 0;
          if (PAIRS) S.tr2[pos] = 0u;
        }
        __syncwarp();

        // what each tet holds of each edge, a pair per lane
        {
          int b = lane / ne, e = lane - b * ne;
          const int db = WARP / ne, de = WARP - db * ne;
#pragma unroll 1
          for (int w = lane; w < nb * ne; w += WARP) {
            const float4 ep = S.epos[e], eu = S.edir[e];
            const float3 p = xyz(ep), u = xyz(eu);
            const unsigned inf = S.tinf[b];
            const bool even = (inf & REC_EVEN) != 0u;  // sides: -, +, -, + of an even tet
            float lo = ep.w, hi = eu.w;
            bool up;
            float t = line_at(S.tp[b][0], p, u, up);
            if (up != even) lo = fmaxf(lo, t); else hi = fminf(hi, t);
            t = line_at(S.tp[b][1], p, u, up);
            if (up == even) lo = fmaxf(lo, t); else hi = fminf(hi, t);
            t = line_at(S.tp[b][2], p, u, up);
            if (up != even) lo = fmaxf(lo, t); else hi = fminf(hi, t);
            t = line_at(S.tp[b][3], p, u, up);
            if (up == even) lo = fmaxf(lo, t); else hi = fminf(hi, t);
            if (hi > lo) {
              const float4 T4 = S.eterm[e];
              const float d = __fsub_rn(hi, lo), m = __fadd_rn(hi, lo), k = __fmul_rn(T4.w, d), km = __fmul_rn(k, m);
              sum.add(k, __fmaf_rn(km, u.x, __fmul_rn(d, T4.x)), __fmaf_rn(km, u.y, __fmul_rn(d, T4.y)),
                      __fmaf_rn(km, u.z, __fmul_rn(d, T4.z)));
              sum.close(__fmul_rn(d, S.eopen[e]));
              const float r2 = __fadd_rn(dot_rn(p, p), fmaxf(lo * lo, hi * hi));
              far2 = fmaxf(far2, r2);
              S.thit[b] = 1;
              if (PAIRS && (inf & 64u)) atomicMax(S.tr2 + b, __float_as_uint(r2));
            }
            b += db;
            e += de;
            if (e >= ne) {
              e -= ne;
              ++b;
            }
          }
        }
        __syncwarp();
        const float3 site = make_float3(seed.x, seed.y, seed.z);
        // the part of edge e (0-5) of tet b inside the cell: how far it reaches
        // (squared, below zero where there is none)
        auto tet_edge = [&](int b, int e) {
          const float4* q = rec + 4 * (size_t)S.tidx[b];
          const float4 r0 = q[0], r1 = q[1], r2 = q[2];
          const float3 c0 = make_float3(r0.x, r0.y, r0.z), c1 = make_float3(r0.w, r1.x, r1.y),
                       c2 = make_float3(r1.z, r1.w, r2.x), c3 = make_float3(r2.y, r2.z, r2.w);
          const float3 P = e < 3 ? c0 : e < 5 ? c1 : c2, Q = e == 0 ? c1 : (e == 1 || e == 3) ? c2 : c3;
          const Line L = line_of(sub_rn(P, site), sub_rn(Q, site));
          float lo = L.a, hi = L.b;
#pragma unroll 2
          for (int f = 0; f < nf; ++f) {
            bool up;
            const float t = line_at(S.plane[f], L.p, L.u, up);
            if (up) lo = fmaxf(lo, t); else hi = fminf(hi, t);
          }
          return hi > lo ? __fadd_rn(dot_rn(L.p, L.p), fmaxf(lo * lo, hi * hi)) : -1.f;
        };
        if (PAIRS && miss) {
          // the pieces that reach beyond half the K-th neighbour's distance (of
          // tets that do, alone)
          const unsigned reach = __ballot_sync(FULL, lane < nb && (S.tinf[lane & (MESH_TETS - 1)] & 64u) != 0u);
          if ((reach >> lane) & 1u) S.tfar[__popc(reach & lt_mask)] = (unsigned char)lane;
          __syncwarp();
#pragma unroll 1
          for (int w = lane; w < 6 * __popc(reach); w += WARP) {
            const int b = S.tfar[w / 6];
            const float r2 = tet_edge(b, w % 6);
            if (r2 >= 0.f) {
              S.thit[b] = 1;
              atomicMax(S.tr2 + b, __float_as_uint(r2));
            }
          }
          __syncwarp();
          const unsigned beyond_k = __ballot_sync(
              FULL, ((reach >> lane) & 1u) && S.thit[lane & (MESH_TETS - 1)] != 0 &&
                        !(dK2 > 4.f * __uint_as_float(S.tr2[lane & (MESH_TETS - 1)])));
          if (lane == 0) here[WC_SECMISS] += (unsigned)__popc(beyond_k);
        }
        const unsigned hits = __ballot_sync(FULL, lane < nb && S.thit[lane & (MESH_TETS - 1)] != 0);
        const unsigned farm = REF ? 0u : __ballot_sync(FULL, lane < nb && (S.tinf[lane & (MESH_TETS - 1)] & 64u) != 0u);
        unsigned open = __ballot_sync(FULL, lane < nb && (S.tinf[lane & (MESH_TETS - 1)] & 15u) != 0u);
        if (lane == 0) {
          here[WC_CONTRIB] += (unsigned)__popc(hits);
          here[WC_EMPTY] += (unsigned)(nb - __popc(hits));
        }
        // the tets reaching beyond half the K-th neighbour's distance, of a
        // cell its K neighbours left open: how far their pieces reach (the
        // tets' edges, one per lane; the cell's edges are in far2)
        if ((farm >> lane) & 1u) S.thit[__popc(farm & lt_mask)] = (unsigned char)lane;
        __syncwarp();
#pragma unroll 1
        for (int w = lane; w < 6 * __popc(farm); w += WARP) far2 = fmaxf(far2, tet_edge(S.thit[w / 6], w % 6));

        for (; open != 0u; open &= open - 1u) {
          const int b = __ffs(open) - 1;
          const unsigned inf = S.tinf[b];
          // its corners in mesh order, for its open faces
          const float4* q = rec + 4 * (size_t)S.tidx[b];
          const float4 r0 = q[0], r1 = q[1], r2 = q[2];
          const float3 c[4] = {sub_rn(make_float3(r0.x, r0.y, r0.z), site), sub_rn(make_float3(r0.w, r1.x, r1.y), site),
                               sub_rn(make_float3(r1.z, r1.w, r2.x), site), sub_rn(make_float3(r2.y, r2.z, r2.w), site)};
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            if (!((inf >> i) & 1u)) continue;
            // triangle (t0, t1, t2): face i, in mesh order
            const float3 t0 = i == 0 ? c[1] : c[0], t1 = i <= 1 ? c[2] : c[1], t2 = i <= 2 ? c[3] : c[2];
            bool out = false;
#pragma unroll 1
            for (int f = lane; f < nf; f += WARP) {
              const float4 P = S.plane[f];
              out |= fmaxf(fmaxf(eval4(P, t0), eval4(P, t1)), eval4(P, t2)) < 0.f;
              S.slot[0][f].w = 0.f;
              S.slot[1][f].w = 0.f;
            }
            if (__any_sync(FULL, out)) continue;
            __syncwarp();
            const float4 PT = S.tp[b][i];
            const bool side = face_side(inf, i);
            // the cell's edges across its plane: where each face's line with
            // it begins and ends.  The side of each vertex is decided once for
            // all its edges, so that a face has as many beginnings as ends (the
            // box that bounds an open cell has edges that lie in mesh planes):
            // one of each or none, else (skew) a slot is taken twice and the cell
            // given back
            const unsigned up0 = __ballot_sync(FULL, lane < nt && eval4(PT, S.vert[lane]) >= 0.f);
            const unsigned up1 = __ballot_sync(FULL, lane + WARP < nt && eval4(PT, S.vert[lane + WARP]) >= 0.f);
            auto above = [&](unsigned v) { return ((v < WARP ? up0 : up1) >> (v & 31u)) & 1u; };
#pragma unroll 1
            for (int e = lane; e < ne; e += WARP) {
              const unsigned E = S.edge[e];
              const bool end = above((E >> 24) & 63u) != 0u;
              if (end != (above((E >> 16) & 0xffu) != 0u)) {
                const float4 ep = S.epos[e], eu = S.edir[e];
                bool up;
                const float t = line_at(PT, xyz(ep), xyz(eu), up);
                const float3 x = along(xyz(ep), fminf(fmaxf(t, ep.w), eu.w), xyz(eu));
                const int in = end == side ? 0 : 1;
                S.slot[in][E & 0xffu] = make_float4(x.x, x.y, x.z, 1.f);
                S.slot[1 - in][(E >> 8) & 0xffu] = make_float4(x.x, x.y, x.z, 1.f);
                skew += 2;
              }
            }
            // its sides: 0 (t1, t2), 1 (t0, t2), 2 (t0, t1), a line each on
            // lanes 0-2
            if (lane < 3) {
              const Line L = line_of(lane == 0 ? t1 : t0, lane == 2 ? t1 : t2);
              S.side[lane][0] = make_float4(L.p.x, L.p.y, L.p.z, L.a);
              S.side[lane][1] = make_float4(L.u.x, L.u.y, L.u.z, L.b);
            }
            const float3 FT = foot_of(PT, X), mark = face_mark(MESH_FACES + 4 * b + i);
            __syncwarp();
            float lo = 1.f, hi = -1.f;  // lanes 0-2: the side's part inside the cell
#pragma unroll 1
            for (int k = 0; k < 3; ++k) {
              const float4 Lp = S.side[k][0], Lu = S.side[k][1];
              float l = Lp.w, h = Lu.w;
#pragma unroll 1
              for (int f = lane; f < nf; f += WARP) {
                bool up;
                const float w = line_at(S.plane[f], xyz(Lp), xyz(Lu), up);
                if (up) l = fmaxf(l, w); else h = fminf(h, w);
                S.at[k][f] = w;
              }
              l = redux_max(l);
              h = redux_min(h);
              if (lane == k) lo = l, hi = h;
            }
            // its plane across each face, cut by the sides
#pragma unroll 1
            for (int f = lane; f < nf; f += WARP) {
              const float4 a4 = S.slot[0][f], b4 = S.slot[1][f];
              skew -= (a4.w != 0.f) + (b4.w != 0.f);
              if (a4.w != 0.f && b4.w != 0.f) {
                float3 a = xyz(a4), bb = xyz(b4);
                bool keep = true;
#pragma unroll 1
                for (int k = 0; k < 3; ++k) {
                  // the side's other plane: the tet's face that leaves out its
                  // opposite corner
                  const int o = k < i ? k : k + 1;
                  const float4 PS = S.tp[b][o];
                  const bool pos = face_side(inf, o);
                  const float va = eval4(PS, a), vb = eval4(PS, bb);
                  const bool oa = pos ? va < 0.f : va > 0.f, ob = pos ? vb < 0.f : vb > 0.f;
                  keep &= !(oa && ob);
                  if (oa != ob) {
                    const float3 y = along(xyz(S.side[k][0]), S.at[k][f], xyz(S.side[k][1]));
                    if (oa) a = y; else bb = y;
                  }
                }
                if (keep) {
                  const float3 aX = sub_rn(a, X), bX = sub_rn(bb, X);
                  const float3 cr = cross_rn(aX, bX), ab = make_float3(__fadd_rn(aX.x, bX.x), __fadd_rn(aX.y, bX.y), __fadd_rn(aX.z, bX.z));
                  const float3 F = foot_of(S.plane[f], X);
                  sum.add(dot_rn(F, cr), F, ab);
                  sum.close(dot_rn(sub_rn(bb, a), sub_rn(face_mark(f), mark)));
                  sum.add(-dot_rn(FT, cr), FT, ab);
                }
              }
            }
            // the sides inside the cell, walked around the inward normal
            if (hi > lo) {
              const float3 p = xyz(S.side[lane][0]), u = xyz(S.side[lane][1]);
              const float3 a = along(p, lo, u), bb = along(p, hi, u), aX = sub_rn(a, X), bX = sub_rn(bb, X);
              const float3 cr = cross_rn(aX, bX), ab = make_float3(__fadd_rn(aX.x, bX.x), __fadd_rn(aX.y, bX.y), __fadd_rn(aX.z, bX.z));
              const float k6 = dot_rn(FT, cr);
              sum.add((side == (lane != 1)) ? -k6 : k6, FT, ab);
              const float op = dot_rn(sub_rn(bb, a), mark);
              sum.close((side == (lane != 1)) ? -op : op);
            }
            __syncwarp();
          }
        }
        __syncwarp();
        sum.flush();
      }
      sum.reduce();
      const float v6 = sum.hv + sum.lv, mag = sum.mag;
      pr2 = warp_max_nonneg(far2);
      // exact where it meets the mesh when that lies within half the K-th
      // neighbour's distance; else completed by the completion pass (and open as
      // long as tets out of the true cell's reach are left out)
      beyond = esc_list && miss && !(dK2 > __fmaf_rn(4.f * pr2, 1.0001f, 1e-4f));
      // much of the cell outside the mesh, and its terms cancel: again from the
      // barycentre of what is inside
      if (!again && !beyond && mag > MESH_NEAR * v6 && mag <= MESH_RATIO * v6) {
        const float w = __fdividef(0.25f, v6);
        X = make_float3(__fmul_rn(sum.hx, w), __fmul_rn(sum.hy, w), __fmul_rn(sum.hz, w));
        again = true;
        continue;
      }
      // (a component a lane: the pairs to double cost one sequence of FP64, of
      // which an SM does two a cycle)
      const float h = lane == 0 ? sum.hv : lane == 1 ? sum.hx : lane == 2 ? sum.hy : sum.hz;
      const float l = lane == 0 ? sum.lv : lane == 1 ? sum.lx : lane == 2 ? sum.ly : sum.lz;
      moment = ((double)h + (double)l) * (lane == 0 ? 1.0 / 6.0 : 1.0 / 24.0);
      if (again) {
        const double vol = __shfl_sync(FULL, moment, 0);
        if (lane > 0) moment += vol * (double)(lane == 1 ? X.x : lane == 2 ? X.y : X.z);
      }
      bad = !isfinite(sum.hv) || !isfinite(sum.hx) || !isfinite(sum.hy) || !isfinite(sum.hz);
      // large terms for a small sum: a sliver, or a cell that only touches the
      // mesh (or no number at all)
      bad |= !(mag <= MESH_RATIO * v6 || mag == 0.f);
      const float tol = __fmaf_rn(MESH_CLOSED, pr2 > 0.f ? sqrtf(pr2) : Rc, MESH_WAY * sum.way);
      open = !(fabsf(sum.open) <= tol) || __reduce_add_sync(FULL, skew) != 0;
      break;
    }
    bad |= open && !beyond;
    if (bad) {
      // degenerate, or a sliver: the pass that follows clips a copy of the cell by
      // each tet (at 128 vertices; of a completed cell at 256)
      if (lane == 0) {
        out_list[atomicAdd(out_count, 1)] = s;
        if (!(flags & SITE_COMPLETED)) S.cnt[WC_REDO]++;
        store.nt[s] = 0;
        if (store.flags) store.flags[s] = (unsigned char)(flags | SITE_HANDED | SITE_REDO);
      }
      __syncwarp();
      continue;
    }
    if (lane < 4) reinterpret_cast<double*>(mom + s)[lane] = moment;
    // (counted now that the site is done here; a cell that is given back is
    // counted by the pass that takes it)
    if (lane == 0) {
      const unsigned nc = REF ? (unsigned)(site_start[s + 1] - site_start[s]) : S.here[WC_CAND];
      S.here[WC_CAND] = nc;
      S.here[WC_CULLED] = nc - min(S.here[WC_CLIPPED], nc);
    }
    __syncwarp();
    if (lane < WC_N) S.cnt[lane] += S.here[lane];
    __syncwarp();
    if (lane == 0) {
      unsigned f = flags | SITE_HANDED;
      if (beyond) {
        // (a bound below zero: these moments are not to be kept)
        esc_list[atomicAdd(esc_count, 1)] = s;
        esc_r2[s] = open ? -pr2 : pr2;
        f |= SITE_UNRESOLVED;
      }
      if (miss) {
        if (!PAIRS) S.cnt[WC_SECMISS]++;
        if (prob_secmiss) atomicAdd(prob_secmiss + pidx, 1u);
      }
      if (flags & SITE_COMPLETED) S.cnt[WC_COMPLETED]++;
      if (store.flags) store.flags[s] = (unsigned char)f;
    }
    __syncwarp();
#undef PD
  }
  if (stats && lane < WC_N && S.cnt[lane]) atomicAdd(stats + stat_slot(lane), (unsigned long long)S.cnt[lane]);
}

}  // namespace vgb
