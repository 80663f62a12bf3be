// Mesh-mesh contact generation (MeshMeshContactGenerator,
// src/Contact/ContactGenerator/MeshMeshContactGenerator.cpp:7-119, with the
// signed distance of src/CollisionObject/Mesh.cpp:124-166).
//
// The reference seeds its search with the triangle pairs FCL reports as
// intersecting, takes the seed triangles' vertices, queries the other mesh's
// signed distance (libigl, pseudonormal sign) and keeps the vertices inside:
// position = the vertex, depth = -distance, normal = the other mesh's vertex
// normals interpolated at the closest point, from the lower body to the
// higher.  Here, for all pairs of a query at once (one launch each):
//   1. mesh_world_kernel: world vertices and box of both meshes;
//   2. mesh_cull_kernel: the triangles of either mesh that meet the other's box;
//   3. mesh_pairs_kernel: every pair of those whose boxes overlap gets a
//      separating-axis test (both normals, nine edge-edge cross products, six
//      in-plane edge normals; closed triangles); the vertices of overlapping
//      pairs are the seeds;
//   4. mesh_sdf_kernel: one warp per seed, the lanes splitting the other mesh's
//      triangles (closest point by Voronoi regions, Ericson 5.1.5), the closest
//      triangle the first of least squared distance (a fixed-order warp
//      reduction), the sign from the angle-weighted pseudonormal of the closest
//      feature (Baerentzen and Aanaes 2005): face, edge or vertex by which
//      barycentric coordinates are below 1e-12;
//   5. mesh_merge_kernel: the inside vertices, the first mesh's in index order
//      then the second's, sorted and merged as every pair's points are
//      (merge_points), frames and lever arms.
// Testing every triangle pair of the two meshes (transforming both triangles
// each time), six launches per pair and one thread merging took 7.5 ms for the 31
// pairs of a chain of 1,140-triangle links; what is left is bound by launches,
// the allocation and the copies.
// The reference's breadth-first growth from the seed vertices walks an
// adjacency map holding triangle-local corner numbers (Mesh.cpp:66-74), so it
// can only revisit vertices 0-2; the seed vertices alone are kept here.
// Mesh normals are built once per mesh on the host (pdc_mesh_create), as
// Mesh.cpp:56-63 builds them: face normals of (v1 - v0) x (v2 - v0), vertex
// normals angle-weighted, edge normals the uniform sum of the two faces'.
#pragma once
#include "pdc_collide.cuh"

struct pdc_mesh {
    int device = 0;
    int nv = 0, nf = 0, ne = 0;
    double* V = nullptr;   // [nv][3] body frame
    int* F = nullptr;      // [nf][3]
    double* fn = nullptr;  // [nf][3] face normals
    double* vn = nullptr;  // [nv][3] vertex normals
    double* en = nullptr;  // [ne][3] edge normals
    int* emap = nullptr;   // [nf][3] edge opposite each corner
};

namespace pdc {

constexpr double kPseudoEps = 1e-12;

struct MeshDev {
    int nv, nf;
    const double* V;
    const int* F;
    const double* fn;
    const double* vn;
    const double* en;
    const int* emap;
    double R[9];  // body -> world rotation
    d3 c;         // body position
};

__device__ __forceinline__ d3 ldv(const double* p, int i) { return d3{p[3 * i], p[3 * i + 1], p[3 * i + 2]}; }
__device__ __forceinline__ d3 rot(const double* R, d3 v) {
    return d3{R[0] * v.x + R[1] * v.y + R[2] * v.z, R[3] * v.x + R[4] * v.y + R[5] * v.z,
              R[6] * v.x + R[7] * v.y + R[8] * v.z};
}
__device__ __forceinline__ d3 rot_t(const double* R, d3 v) {
    return d3{R[0] * v.x + R[3] * v.y + R[6] * v.z, R[1] * v.x + R[4] * v.y + R[7] * v.z,
              R[2] * v.x + R[5] * v.y + R[8] * v.z};
}
__device__ __forceinline__ d3 world_vertex(const MeshDev& M, int i) { return add3(rot(M.R, ldv(M.V, i)), M.c); }

// Closest point to p on triangle abc and its barycentric coordinates.
__device__ inline d3 closest_on_triangle(d3 p, d3 a, d3 b, d3 c, double* bary) {
    const d3 ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a);
    const double d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    if (d1 <= 0 && d2 <= 0) { bary[0] = 1; bary[1] = 0; bary[2] = 0; return a; }
    const d3 bp = sub3(p, b);
    const double d3_ = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3_ >= 0 && d4 <= d3_) { bary[0] = 0; bary[1] = 1; bary[2] = 0; return b; }
    const double vc = d1 * d4 - d3_ * d2;
    if (vc <= 0 && d1 >= 0 && d3_ <= 0) {
        const double t = d1 / (d1 - d3_);
        bary[0] = 1.0 - t; bary[1] = t; bary[2] = 0;
        return add3(a, scl3(t, ab));
    }
    const d3 cp = sub3(p, c);
    const double d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0 && d5 <= d6) { bary[0] = 0; bary[1] = 0; bary[2] = 1; return c; }
    const double vb = d5 * d2 - d1 * d6;
    if (vb <= 0 && d2 >= 0 && d6 <= 0) {
        const double t = d2 / (d2 - d6);
        bary[0] = 1.0 - t; bary[1] = 0; bary[2] = t;
        return add3(a, scl3(t, ac));
    }
    const double va = d3_ * d6 - d5 * d4;
    if (va <= 0 && (d4 - d3_) >= 0 && (d5 - d6) >= 0) {
        const double t = (d4 - d3_) / ((d4 - d3_) + (d5 - d6));
        bary[0] = 0; bary[1] = 1.0 - t; bary[2] = t;
        return add3(b, scl3(t, sub3(c, b)));
    }
    const double den = 1.0 / (va + vb + vc);
    const double v = vb * den, w = vc * den;
    bary[0] = 1.0 - v - w; bary[1] = v; bary[2] = w;
    return add3(add3(a, scl3(v, ab)), scl3(w, ac));
}

// True if some axis separates triangles P and Q (world vertices).
__device__ inline bool tri_separated(const d3* P, const d3* Q) {
    const d3 ep[3] = {sub3(P[1], P[0]), sub3(P[2], P[1]), sub3(P[0], P[2])};
    const d3 eq[3] = {sub3(Q[1], Q[0]), sub3(Q[2], Q[1]), sub3(Q[0], Q[2])};
    const d3 n1 = cross3(ep[0], scl3(-1.0, ep[2])), n2 = cross3(eq[0], scl3(-1.0, eq[2]));
    for (int k = 0; k < 17; ++k) {
        d3 L;
        if (k == 0) L = n1;
        else if (k == 1) L = n2;
        else if (k < 11) L = cross3(ep[(k - 2) / 3], eq[(k - 2) % 3]);
        else if (k < 14) L = cross3(n1, ep[k - 11]);
        else L = cross3(n2, eq[k - 14]);
        if (dot3(L, L) < 1e-30) continue;
        double pmin = 1e300, pmax = -1e300, qmin = 1e300, qmax = -1e300;
        for (int i = 0; i < 3; ++i) {
            const double a = dot3(P[i], L), b = dot3(Q[i], L);
            pmin = fmin(pmin, a); pmax = fmax(pmax, a);
            qmin = fmin(qmin, b); qmax = fmax(qmax, b);
        }
        if (pmax < qmin || qmax < pmin) return true;
    }
    return false;
}

// One mesh pair of a query: both meshes, and where its part of the scratch
// begins (ints, doubles, output rows).
struct MeshPair {
    MeshDev m[2];
    long long i0;    // zeroed ints: 8 counters, triangle flags of both, seed and inside flags of all vertices
    long long j0;    // other ints: candidate triangles of both, seeds of both, order of the inside vertices
    long long d0;    // doubles: 12 of boxes, then per vertex world position, contact position, normal, depth
    long long row0;  // first row of the pair's merged contacts
};
struct MeshScratch {
    const MeshPair* pairs;
    const int* first;  // [pairs + 1] first block of each pair in the kernels whose blocks the pairs share
    int n_pairs;
    int* zi;
    int* wi;
    double* wd;
    int* counts;  // [pairs] merged contacts
    double *pos, *nrm, *dep, *frame, *arm;  // [rows]
};
// The scratch of one pair (side 0 = a's part first, side 1 = b's behind it).
struct PairView {
    const MeshPair& P;
    int nf0, nv0, nv;
    int *count, *flag, *seed, *inside, *cand, *list, *order;
    double *box, *world, *vpos, *vnrm, *vdep;
    int block, blocks;  // this block among the pair's, where the pairs share the blocks
    __device__ explicit PairView(const MeshScratch& S) : PairView(S, owner(S)) {
        const int k = (int)(&P - S.pairs);
        block = (int)blockIdx.x - S.first[k];
        blocks = S.first[k + 1] - S.first[k];
    }
    __device__ static int owner(const MeshScratch& S) {
        int lo = 0, hi = S.n_pairs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (S.first[mid] <= (int)blockIdx.x) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    }
    __device__ PairView(const MeshScratch& S, int k) : P(S.pairs[k]), block(0), blocks(1) {
        nf0 = P.m[0].nf;
        nv0 = P.m[0].nv;
        nv = nv0 + P.m[1].nv;
        const int nf = nf0 + P.m[1].nf;
        count = S.zi + P.i0;
        flag = count + 8;
        seed = flag + nf;
        inside = seed + nv;
        cand = S.wi + P.j0;
        list = cand + nf;
        order = list + nv;
        box = S.wd + P.d0;
        world = box + 12;
        vpos = world + 3LL * nv;
        vnrm = vpos + 3LL * nv;
        vdep = vnrm + 3LL * nv;
    }
    __device__ __forceinline__ int tri0(int side) const { return side ? nf0 : 0; }
    __device__ __forceinline__ int vert0(int side) const { return side ? nv0 : 0; }
    __device__ __forceinline__ void triangle(int side, int f, d3* t) const {
        const int* F = P.m[side].F + 3 * f;
        for (int k = 0; k < 3; ++k) t[k] = ldv(world, vert0(side) + F[k]);
    }
};
__device__ __forceinline__ void tri_box(const d3* t, double* lo, double* hi) {
    lo[0] = fmin(fmin(t[0].x, t[1].x), t[2].x); hi[0] = fmax(fmax(t[0].x, t[1].x), t[2].x);
    lo[1] = fmin(fmin(t[0].y, t[1].y), t[2].y); hi[1] = fmax(fmax(t[0].y, t[1].y), t[2].y);
    lo[2] = fmin(fmin(t[0].z, t[1].z), t[2].z); hi[2] = fmax(fmax(t[0].z, t[1].z), t[2].z);
}

// World vertices of one mesh of a pair and their box, one block (pair, then side).
__global__ void __launch_bounds__(512) mesh_world_kernel(const MeshScratch S) {
    __shared__ double red[6][16];
    const PairView V(S, blockIdx.x >> 1);
    const int side = blockIdx.x & 1;
    const MeshDev& M = V.P.m[side];
    double b[6] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY};  // lo, -hi
    for (int v = threadIdx.x; v < M.nv; v += blockDim.x) {
        const d3 w = world_vertex(M, v);
        st3(V.world + 3LL * (V.vert0(side) + v), w);
        b[0] = fmin(b[0], w.x); b[1] = fmin(b[1], w.y); b[2] = fmin(b[2], w.z);
        b[3] = fmin(b[3], -w.x); b[4] = fmin(b[4], -w.y); b[5] = fmin(b[5], -w.z);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        for (int o = 16; o > 0; o >>= 1) b[k] = fmin(b[k], __shfl_xor_sync(0xffffffffu, b[k], o));
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = b[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double x = INFINITY;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x = fmin(x, red[threadIdx.x][w]);
        V.box[6 * side + threadIdx.x] = threadIdx.x < 3 ? x : -x;
    }
}

// Triangles of either mesh whose box meets the other mesh's box: no other can
// overlap one of the other mesh's triangles.
__global__ void __launch_bounds__(256) mesh_cull_kernel(const MeshScratch S) {
    const PairView V(S);
    for (int side = 0; side < 2; ++side) {
        const double* o = V.box + 6 * (1 - side);
        for (int f = V.block * blockDim.x + threadIdx.x; f < V.P.m[side].nf; f += V.blocks * blockDim.x) {
            d3 t[3];
            double lo[3], hi[3];
            V.triangle(side, f, t);
            tri_box(t, lo, hi);
            if (hi[0] < o[0] || o[3] < lo[0] || hi[1] < o[1] || o[4] < lo[1] || hi[2] < o[2] || o[5] < lo[2]) continue;
            V.cand[V.tri0(side) + atomicAdd(&V.count[side], 1)] = f;
        }
    }
}

// Candidate triangle pairs whose boxes overlap and that no axis separates: both
// triangles flagged, and their vertices listed as seeds (once each).
__global__ void __launch_bounds__(256) mesh_pairs_kernel(const MeshScratch S) {
    const PairView V(S);
    const int ca = V.count[0], cb = V.count[1];
    const long long total = (long long)ca * cb;
    for (long long q = V.block * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)V.blocks * blockDim.x) {
        const int f[2] = {V.cand[q / cb], V.cand[V.nf0 + q % cb]};
        d3 P[3], Q[3];
        V.triangle(0, f[0], P);
        V.triangle(1, f[1], Q);
        double pl[3], ph[3], ql[3], qh[3];
        tri_box(P, pl, ph);
        tri_box(Q, ql, qh);
        if (ph[0] < ql[0] || qh[0] < pl[0] || ph[1] < ql[1] || qh[1] < pl[1] || ph[2] < ql[2] || qh[2] < pl[2])
            continue;
        if (tri_separated(P, Q)) continue;
        for (int side = 0; side < 2; ++side) {
            if (atomicExch(&V.flag[V.tri0(side) + f[side]], 1)) continue;
            for (int k = 0; k < 3; ++k) {
                const int v = V.P.m[side].F[3 * f[side] + k];
                if (!atomicExch(&V.seed[V.vert0(side) + v], 1))
                    V.list[V.vert0(side) + atomicAdd(&V.count[2 + side], 1)] = v;
            }
        }
    }
}

// Signed distance of every seed vertex to the other mesh M, a warp per vertex
// (the lanes split M's triangles; the closest is the first of least squared
// distance).  Inside vertices get their world position, depth and contact
// normal (M's interpolated vertex normal, from the lower body to the higher:
// minus b's outward normal for a's vertices).
__global__ void __launch_bounds__(256) mesh_sdf_kernel(const MeshScratch S) {
    const PairView V(S);
    const int lane = threadIdx.x & 31;
    const int warps = (V.blocks * blockDim.x) >> 5;
    const int na = V.count[2], n = na + V.count[3];
    for (int q = (V.block * blockDim.x + threadIdx.x) >> 5; q < n; q += warps) {
        const int side = q < na ? 0 : 1;
        const int v = V.vert0(side) + V.list[V.vert0(side) + q - (side ? na : 0)];
        const MeshDev& M = V.P.m[1 - side];
        const double sign = side ? 1.0 : -1.0;
        const d3 w = ldv(V.world, v);
        const d3 p = rot_t(M.R, sub3(w, M.c));
        double best = INFINITY;
        int bf = 0x7fffffff;
        for (int f = lane; f < M.nf; f += 32) {
            double bary[3];
            const d3 c = closest_on_triangle(p, ldv(M.V, M.F[3 * f]), ldv(M.V, M.F[3 * f + 1]),
                                             ldv(M.V, M.F[3 * f + 2]), bary);
            const d3 d = sub3(p, c);
            const double d2 = dot3(d, d);
            if (d2 < best) {
                best = d2;
                bf = f;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int of = __shfl_xor_sync(0xffffffffu, bf, o);
            if (ob < best || (ob == best && of < bf)) {
                best = ob;
                bf = of;
            }
        }
        if (lane == 0 && bf < M.nf) {
            double b[3];
            const int* tri = M.F + 3 * bf;
            const d3 c = closest_on_triangle(p, ldv(M.V, tri[0]), ldv(M.V, tri[1]), ldv(M.V, tri[2]), b);
            const int nsmall = (b[0] <= kPseudoEps) + (b[1] <= kPseudoEps) + (b[2] <= kPseudoEps);
            d3 pn;
            if (nsmall == 2) {  // a vertex: the corner whose coordinate is not small
                const int k = b[0] > kPseudoEps ? 0 : (b[1] > kPseudoEps ? 1 : 2);
                pn = ldv(M.vn, tri[k]);
            } else if (nsmall == 1) {  // an edge: the one opposite the small coordinate
                const int k = b[0] <= kPseudoEps ? 0 : (b[1] <= kPseudoEps ? 1 : 2);
                pn = ldv(M.en, M.emap[3 * bf + k]);
            } else {
                pn = ldv(M.fn, bf);
            }
            const double dist = (dot3(sub3(p, c), pn) >= 0 ? 1.0 : -1.0) * sqrt(best);
            if (dist < 0) {
                const d3 n3 = add3(add3(scl3(b[0], ldv(M.vn, tri[0])), scl3(b[1], ldv(M.vn, tri[1]))),
                                   scl3(b[2], ldv(M.vn, tri[2])));
                const double nn = sqrt(dot3(n3, n3));
                const d3 nu = nn > 0 ? d3{n3.x / nn, n3.y / nn, n3.z / nn} : n3;
                st3(V.vpos + 3LL * v, w);
                st3(V.vnrm + 3LL * v, scl3(sign, rot(M.R, nu)));
                V.vdep[v] = -dist;
                V.inside[v] = 1;
            }
        }
    }
}

// Block-wide exclusive scan of one value per thread (256 threads); returns the total.
__device__ __forceinline__ int block_scan256(int x, int* excl) {
    __shared__ int part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) part[warp] = s;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < 8; ++w) {
        before += w < warp ? part[w] : 0;
        total += part[w];
    }
    __syncthreads();
    *excl = before + s - x;
    return total;
}

// One block per pair: the inside vertices (a's in index order, then b's) in the
// order of merge_points (ranks on the position grid, ties in that order), runs of
// near points merged by one thread each, then frames and lever arms.  One
// thread walking all vertices and sorting took most of a query.
__global__ void __launch_bounds__(256) mesh_merge_kernel(const MeshScratch S) {
    const PairView V(S, blockIdx.x);
    const int tid = threadIdx.x;
    int m = 0, e;
    for (int base = 0; base < V.nv; base += 256) {  // indices of the inside vertices, into the seeds' list
        const int v = base + tid, in = v < V.nv ? V.inside[v] : 0;
        const int t = block_scan256(in, &e);
        if (in) V.list[m + e] = v;
        m += t;
    }
    __syncthreads();
    for (int i = tid; i < m; i += 256) {
        const d3 p = ldv(V.vpos, V.list[i]);
        const double x = grid_key(p.x), y = grid_key(p.y), z = grid_key(p.z);
        int rank = 0;
        for (int j = 0; j < m; ++j) {
            const d3 o = ldv(V.vpos, V.list[j]);
            const double ox = grid_key(o.x), oy = grid_key(o.y), oz = grid_key(o.z);
            const bool less = ox != x ? ox < x : (oy != y ? oy < y : oz < z);
            const bool tie = ox == x && oy == y && oz == z;
            rank += less || (tie && j < i);
        }
        V.order[rank] = V.list[i];
    }
    __syncthreads();
    const d3 ca = V.P.m[0].c, cb = V.P.m[1].c;
    int done = 0;
    for (int base = 0; base < m; base += 256) {
        const int i = base + tid;
        auto starts = [&](int k) {  // point k begins a run of near points
            if (k == 0) return true;
            const d3 d = sub3(ldv(V.vpos, V.order[k]), ldv(V.vpos, V.order[k - 1]));
            return dot3(d, d) > 1e-8;
        };
        const bool first = i < m && starts(i);
        const int t = block_scan256(first ? 1 : 0, &e);
        if (first) {
            const int v = V.order[i];
            d3 nrm = ldv(V.vnrm, v);
            double depth = V.vdep[v];
            int j = i + 1;
            for (; j < m && !starts(j); ++j) {
                nrm = add3(nrm, ldv(V.vnrm, V.order[j]));
                depth = fmin(V.vdep[V.order[j]], depth);
            }
            if (j - i > 1) {
                const double nn = sqrt(dot3(nrm, nrm));
                nrm = (nn > 0) ? scl3(1.0 / nn, nrm) : nrm;
            }
            const long long r = V.P.row0 + done + e;
            const d3 p = ldv(V.vpos, v);
            st3(S.pos + 3 * r, p);
            st3(S.nrm + 3 * r, nrm);
            S.dep[r] = fabs(depth);
            frame_from_normal(nrm, S.frame + 9 * r);
            st3(S.arm + 6 * r, sub3(p, ca));
            st3(S.arm + 6 * r + 3, sub3(p, cb));
        }
        done += t;
    }
    if (tid == 0) S.counts[blockIdx.x] = done;
}

// Pair k's merged contacts (rows of its own region, region k starting at row
// row0[k]) copied to rows off_k .. off_k + n_k - 1 of the packed output, off_k
// the sum of the counts of pairs 0 .. k-1, rows at or past `cap` dropped.
__global__ void mesh_gather_kernel(int n_pairs, const int* counts, const long long* row0, const double* r_pos,
                                   const double* r_nrm, const double* r_dep, const double* r_frame,
                                   const double* r_arm, int cap, double* o_pos, double* o_nrm, double* o_dep,
                                   double* o_frame, double* o_arm) {
    __shared__ long long off;
    const int k = blockIdx.x;
    if (k >= n_pairs) return;
    if (threadIdx.x == 0) {
        long long o = 0;
        for (int p = 0; p < k; ++p) o += counts[p];
        off = o;
    }
    __syncthreads();
    if (off >= cap) return;
    const long long n = min((long long)counts[k], (long long)cap - off);
    const long long src = row0[k];
    for (long long r = threadIdx.x; r < n; r += blockDim.x) {
        const long long a = src + r, d = off + r;
        for (int c = 0; c < 3; ++c) {
            o_pos[3 * d + c] = r_pos[3 * a + c];
            o_nrm[3 * d + c] = r_nrm[3 * a + c];
        }
        o_dep[d] = r_dep[a];
        for (int c = 0; c < 9; ++c) o_frame[9 * d + c] = r_frame[9 * a + c];
        for (int c = 0; c < 6; ++c) o_arm[6 * d + c] = r_arm[6 * a + c];
    }
}

}  // namespace pdc

// ---------------------------------------------------------------------------
// Host side: mesh creation (normals, Mesh.cpp:56-63) and the pair query.
namespace {
struct HostV3 {
    double x, y, z;
};
inline HostV3 hsub(HostV3 a, HostV3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
inline HostV3 hcross(HostV3 a, HostV3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
inline double hdot(HostV3 a, HostV3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline HostV3 hnorm(HostV3 a) {
    const double n = std::sqrt(hdot(a, a));
    return n > 0 ? HostV3{a.x / n, a.y / n, a.z / n} : a;
}
struct DevScratch {  // device buffers of one call, freed on every path
    std::vector<void*> ptrs;
    ~DevScratch() {
        for (void* p : ptrs) cudaFree(p);
    }
    template <class T>
    cudaError_t get(T** p, size_t n) {
        cudaError_t e = dev_malloc(p, std::max<size_t>(n, 1) * sizeof(T));
        if (e == cudaSuccess) ptrs.push_back(*p);
        return e;
    }
};
void host_quat_to_R(const double* q, double* R) {  // the expression order of pdc::quat_to_R
    const double x = q[0], y = q[1], z = q[2], w = q[3];
    const double tx = 2 * x, ty = 2 * y, tz = 2 * z;
    const double twx = tx * w, twy = ty * w, twz = tz * w;
    const double txx = tx * x, txy = ty * x, txz = tz * x;
    const double tyy = ty * y, tyz = tz * y, tzz = tz * z;
    R[0] = 1 - (tyy + tzz); R[1] = txy - twz;       R[2] = txz + twy;
    R[3] = txy + twz;       R[4] = 1 - (txx + tzz); R[5] = tyz - twx;
    R[6] = txz - twy;       R[7] = tyz + twx;       R[8] = 1 - (txx + tyy);
}
}  // namespace

extern "C" void pdc_mesh_destroy(pdc_mesh* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    cudaFree(m->V);
    cudaFree(m->F);
    cudaFree(m->fn);
    cudaFree(m->vn);
    cudaFree(m->en);
    cudaFree(m->emap);
    delete m;
}

extern "C" int pdc_mesh_create(int32_t n_verts, const double* verts, int32_t n_tris, const int32_t* tris,
                               pdc_mesh** out) {
    pdc_solver* s = nullptr;
    if (!out || !verts || !tris || n_verts < 3 || n_tris < 1)
        return fail(s, PDC_EINVAL, "pdc_mesh_create: null argument or fewer than 3 vertices / 1 triangle");
    *out = nullptr;
    for (long long k = 0; k < 3LL * n_tris; ++k)
        if (tris[k] < 0 || tris[k] >= n_verts) return fail(s, PDC_EINVAL, "pdc_mesh_create: vertex index out of range");
    const int nv = n_verts, nf = n_tris;
    auto V = [&](int i) { return HostV3{verts[3 * i], verts[3 * i + 1], verts[3 * i + 2]}; };
    std::vector<double> fn(3 * nf), vn(3 * nv, 0.0), en;
    std::vector<int> emap(3 * nf);
    for (int f = 0; f < nf; ++f) {
        const HostV3 a = V(tris[3 * f]), b = V(tris[3 * f + 1]), c = V(tris[3 * f + 2]);
        const HostV3 n = hnorm(hcross(hsub(b, a), hsub(c, a)));
        fn[3 * f] = n.x; fn[3 * f + 1] = n.y; fn[3 * f + 2] = n.z;
    }
    // edges numbered in order of first appearance over (face, corner)
    {
        std::vector<std::pair<long long, int>> all(3 * nf);
        for (int f = 0; f < nf; ++f)
            for (int k = 0; k < 3; ++k) {
                const long long i = tris[3 * f + (k + 1) % 3], j = tris[3 * f + (k + 2) % 3];
                all[3 * f + k] = {std::min(i, j) * (long long)nv + std::max(i, j), 3 * f + k};
            }
        std::vector<std::pair<long long, int>> sorted = all;
        std::sort(sorted.begin(), sorted.end());
        // first occurrence of each key -> its rank by first occurrence
        std::vector<int> first_of(3 * nf);
        for (size_t q = 0; q < sorted.size();) {
            size_t r = q;
            while (r < sorted.size() && sorted[r].first == sorted[q].first) ++r;
            for (size_t t = q; t < r; ++t) first_of[sorted[t].second] = sorted[q].second;
            q = r;
        }
        std::vector<int> id(3 * nf, -1);
        int ne = 0;
        for (int q = 0; q < 3 * nf; ++q) {
            const int fo = first_of[q];
            if (id[fo] < 0) id[fo] = ne++;
            emap[q] = id[fo];
        }
        en.assign(3 * ne, 0.0);
    }
    for (int f = 0; f < nf; ++f)
        for (int k = 0; k < 3; ++k) {
            const HostV3 p = V(tris[3 * f + k]);
            const HostV3 e1 = hnorm(hsub(V(tris[3 * f + (k + 1) % 3]), p));
            const HostV3 e2 = hnorm(hsub(V(tris[3 * f + (k + 2) % 3]), p));
            const double ang = std::acos(std::max(-1.0, std::min(1.0, hdot(e1, e2))));
            for (int r = 0; r < 3; ++r) vn[3 * tris[3 * f + k] + r] += ang * fn[3 * f + r];
            for (int r = 0; r < 3; ++r) en[3 * emap[3 * f + k] + r] += fn[3 * f + r];
        }
    for (size_t i = 0; i < vn.size(); i += 3) {
        const HostV3 n = hnorm(HostV3{vn[i], vn[i + 1], vn[i + 2]});
        vn[i] = n.x; vn[i + 1] = n.y; vn[i + 2] = n.z;
    }
    for (size_t i = 0; i < en.size(); i += 3) {
        const HostV3 n = hnorm(HostV3{en[i], en[i + 1], en[i + 2]});
        en[i] = n.x; en[i + 1] = n.y; en[i + 2] = n.z;
    }
    pdc_mesh* m = new pdc_mesh();
    CK(cudaGetDevice(&m->device), "cudaGetDevice");
    m->nv = nv;
    m->nf = nf;
    m->ne = (int)(en.size() / 3);
    cudaError_t e = dev_malloc(&m->V, 3 * sizeof(double) * nv);
    if (e == cudaSuccess) e = dev_malloc(&m->F, 3 * sizeof(int) * nf);
    if (e == cudaSuccess) e = dev_malloc(&m->fn, 3 * sizeof(double) * nf);
    if (e == cudaSuccess) e = dev_malloc(&m->vn, 3 * sizeof(double) * nv);
    if (e == cudaSuccess) e = dev_malloc(&m->en, sizeof(double) * std::max<size_t>(en.size(), 1));
    if (e == cudaSuccess) e = dev_malloc(&m->emap, 3 * sizeof(int) * nf);
    if (e == cudaSuccess) e = cudaMemcpy(m->V, verts, 3 * sizeof(double) * nv, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->F, tris, 3 * sizeof(int) * nf, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->fn, fn.data(), fn.size() * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->vn, vn.data(), vn.size() * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->en, en.data(), en.size() * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(m->emap, emap.data(), emap.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        pdc_mesh_destroy(m);
        return cuda_fail(s, e, "pdc_mesh_create");
    }
    *out = m;
    return PDC_OK;
}

// Contacts of n_pairs pairs (arguments checked): one set of launches for all of
// them, one device allocation, packed rows into the host arrays.
static int mesh_query(int32_t n_pairs, const pdc_mesh* const* a, const double* poses_a, const pdc_mesh* const* b,
                      const double* poses_b, int32_t max_points, double* pos, double* normal, double* depth,
                      double* frame, double* arm, int32_t* counts, long long* total_out, const char* who) {
    pdc_solver* s = nullptr;
    CK(cudaSetDevice(a[0]->device), "cudaSetDevice");
    auto dev = [](const pdc_mesh* m, const double* pose) {
        pdc::MeshDev d;
        d.nv = m->nv; d.nf = m->nf;
        d.V = m->V; d.F = m->F; d.fn = m->fn; d.vn = m->vn; d.en = m->en; d.emap = m->emap;
        host_quat_to_R(pose + 3, d.R);
        d.c = pdc::d3{pose[0], pose[1], pose[2]};
        return d;
    };
    std::vector<pdc::MeshPair> pairs(n_pairs);
    std::vector<long long> row0(n_pairs);
    std::vector<int> first(n_pairs + 1);
    long long ni = 0, nj = 0, nd = 0, nrows = 0;
    double work = 0;  // triangle pairs
    for (int k = 0; k < n_pairs; ++k) {
        const long long nv = (long long)a[k]->nv + b[k]->nv, nf = (long long)a[k]->nf + b[k]->nf;
        pdc::MeshPair& P = pairs[k];
        P.m[0] = dev(a[k], poses_a + 7LL * k);
        P.m[1] = dev(b[k], poses_b + 7LL * k);
        P.i0 = ni; ni += 8 + nf + 2 * nv;
        P.j0 = nj; nj += nf + 2 * nv;
        P.d0 = nd; nd += 12 + 10 * nv;
        P.row0 = row0[k] = nrows; nrows += nv;  // a pair merges at most its inside vertices
        work += (double)a[k]->nf * b[k]->nf;
    }
    // Blocks: enough to fill the GPU, shared by the pairs in proportion to their
    // triangle pairs.  (With as many for each pair, a pair of 20,000-triangle meshes
    // among 200 pairs of 480-triangle ones ran on 12 blocks: 74 ms instead of 4.5, where
    // it takes 4.3 alone.)
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, a[0]->device);
    first[0] = 0;
    for (int k = 0; k < n_pairs; ++k) {
        const double w = (double)a[k]->nf * b[k]->nf;
        first[k + 1] = first[k] + (int)std::max(1.0, std::ceil(std::min(w / 256, 16.0 * sms * w / work)));
    }
    const long long cap = std::max<long long>(1, std::min<long long>(max_points, nrows));
    Arena A;
    pdc::MeshScratch S;
    pdc::MeshPair* d_pairs = nullptr;
    long long* d_row0 = nullptr;
    int* d_first = nullptr;
    double* out = nullptr;
    auto carve_query = [&](Arena& q) {
        q.reset();
        d_pairs = q.take<pdc::MeshPair>(n_pairs);
        d_row0 = q.take<long long>(n_pairs);
        d_first = q.take<int>(n_pairs + 1);
        S.pairs = d_pairs;
        S.first = d_first;
        S.n_pairs = n_pairs;
        S.zi = q.take<int>(ni);
        S.wi = q.take<int>(nj);
        S.wd = q.take<double>(nd);
        S.counts = q.take<int>(n_pairs);
        S.pos = q.take<double>(22 * nrows);
        S.nrm = S.pos + 3 * nrows;
        S.dep = S.nrm + 3 * nrows;
        S.frame = S.dep + nrows;
        S.arm = S.frame + 9 * nrows;
        out = q.take<double>(22 * cap);
        return q.off + 256;
    };
    const size_t need = carve_query(A);
    DevScratch sc;
    char* mem = nullptr;
    const cudaError_t e = sc.get(&mem, need);
    if (e != cudaSuccess) return cuda_fail(s, e, who);
    A.base = mem;
    carve_query(A);
    CK(cudaMemcpyAsync(d_pairs, pairs.data(), sizeof(pdc::MeshPair) * n_pairs, cudaMemcpyHostToDevice), "H2D pairs");
    CK(cudaMemcpyAsync(d_row0, row0.data(), sizeof(long long) * n_pairs, cudaMemcpyHostToDevice), "H2D rows");
    CK(cudaMemcpyAsync(d_first, first.data(), sizeof(int) * (n_pairs + 1), cudaMemcpyHostToDevice), "H2D blocks");
    CK(cudaMemsetAsync(S.zi, 0, sizeof(int) * ni), "memset");
    pdc::mesh_world_kernel<<<2 * n_pairs, 512>>>(S);
    pdc::mesh_cull_kernel<<<first[n_pairs], 256>>>(S);
    pdc::mesh_pairs_kernel<<<first[n_pairs], 256>>>(S);
    pdc::mesh_sdf_kernel<<<first[n_pairs], 256>>>(S);
    pdc::mesh_merge_kernel<<<n_pairs, 256>>>(S);
    double *o_nrm = out + 3 * cap, *o_dep = o_nrm + 3 * cap, *o_frame = o_dep + cap, *o_arm = o_frame + 9 * cap;
    pdc::mesh_gather_kernel<<<n_pairs, 128>>>(n_pairs, S.counts, d_row0, S.pos, S.nrm, S.dep, S.frame, S.arm,
                                              (int)cap, out, o_nrm, o_dep, o_frame, o_arm);
    CK(cudaGetLastError(), "launch mesh kernels");
    CK(cudaMemcpy(counts, S.counts, sizeof(int32_t) * n_pairs, cudaMemcpyDeviceToHost), "D2H counts");
    long long total = 0;
    for (int k = 0; k < n_pairs; ++k) total += counts[k];
    const long long w = std::min<long long>(total, max_points);
    if (w > 0) {
        CK(cudaMemcpyAsync(pos, out, 3 * sizeof(double) * w, cudaMemcpyDeviceToHost), "D2H contacts");
        CK(cudaMemcpyAsync(normal, o_nrm, 3 * sizeof(double) * w, cudaMemcpyDeviceToHost), "D2H contacts");
        CK(cudaMemcpyAsync(depth, o_dep, sizeof(double) * w, cudaMemcpyDeviceToHost), "D2H contacts");
        CK(cudaMemcpyAsync(frame, o_frame, 9 * sizeof(double) * w, cudaMemcpyDeviceToHost), "D2H contacts");
        CK(cudaMemcpy(arm, o_arm, 6 * sizeof(double) * w, cudaMemcpyDeviceToHost), "D2H contacts");
    }
    *total_out = total;
    return PDC_OK;
}

extern "C" int pdc_mesh_contacts(const pdc_mesh* a, const double pose_a[7], const pdc_mesh* b,
                                 const double pose_b[7], int32_t max_points, double* pos, double* normal,
                                 double* depth, double* frame, double* arm, int32_t* n_points) {
    pdc_solver* s = nullptr;
    if (!a || !b || !pose_a || !pose_b || !n_points || max_points < 0 ||
        (max_points > 0 && (!pos || !normal || !depth || !frame || !arm)))
        return fail(s, PDC_EINVAL, "pdc_mesh_contacts: null argument");
    if (a->device != b->device) return fail(s, PDC_EINVAL, "pdc_mesh_contacts: meshes on different devices");
    int32_t count = 0;
    long long total = 0;
    const int rc = mesh_query(1, &a, pose_a, &b, pose_b, max_points, pos, normal, depth, frame, arm, &count, &total,
                              "pdc_mesh_contacts: scratch");
    if (rc == PDC_OK) *n_points = count;
    return rc;
}

extern "C" int pdc_mesh_contacts_pairs(int32_t n_pairs, const pdc_mesh* const* a, const double* poses_a,
                                       const pdc_mesh* const* b, const double* poses_b, int32_t max_points,
                                       double* pos, double* normal, double* depth, double* frame, double* arm,
                                       int32_t* counts, int32_t* n_points) {
    pdc_solver* s = nullptr;
    if (n_pairs < 0 || max_points < 0 || !n_points ||
        (n_pairs > 0 && (!a || !b || !poses_a || !poses_b || !counts)) ||
        (max_points > 0 && (!pos || !normal || !depth || !frame || !arm)))
        return fail(s, PDC_EINVAL, "pdc_mesh_contacts_pairs: null or negative argument");
    *n_points = 0;
    if (n_pairs == 0) return PDC_OK;
    for (int k = 0; k < n_pairs; ++k) {
        if (!a[k] || !b[k]) return fail(s, PDC_EINVAL, "pdc_mesh_contacts_pairs: null mesh");
        if (a[k]->device != a[0]->device || b[k]->device != a[0]->device)
            return fail(s, PDC_EINVAL, "pdc_mesh_contacts_pairs: meshes on different devices");
    }
    long long total = 0;
    const int rc = mesh_query(n_pairs, a, poses_a, b, poses_b, max_points, pos, normal, depth, frame, arm, counts,
                              &total, "pdc_mesh_contacts_pairs: scratch");
    if (rc == PDC_OK) *n_points = (int32_t)std::min<long long>(total, 0x7fffffffLL);
    return rc;
}
