// Device preprocessing of a cloth's constraint inputs: the unique edges of a
// triangle mesh with their rest lengths, the bend pairs with theirs, and the
// per-vertex inverse masses from triangle areas, the per-element steps of the
// reference's input pipeline (xpbd_core.py:715-747 edges and bends, 862-881
// masses) that dominate the cost of building large cloths.  Greedy colouring
// stays on the host (xpbd_prep.cu): first-fit in constraint order is
// sequential by definition; so do the hidden tethers (a k-d tree query whose
// tie-breaking between equidistant pins a device argmin would not repeat).
//
// Results are bit-identical to the cloth builders' numpy restatement:
// * edges are the distinct (min, max) endpoint pairs of every triangle side
//   in lexicographic order (np.unique over rows): a CSR of the sides keyed by
//   the lower endpoint (count, scan, scatter), each row sorted and walked
//   over its repeats;
// * rest length = max(|x_b - x_a|, eps) in float32 with the sum of squares
//   taken x, y, z in order (np.linalg.norm over a row of three);
// * bend pairs as xpbd_gb300_bend_pairs writes them (below), rest lengths
//   as for edges;
// * mass = float64 sum of float32 shares max(area * density, eps) / 3 in
//   np.add.at order (corner 0 of every triangle in index order, then corner
//   1, then 2): a CSR of the corners keyed by vertex with entries
//   corner * T + t, sorted;
//   area = 0.5 |(x1 - x0) x (x2 - x0)| in float32; inverse mass 1 / mass
//   (mass 1 where nothing was added), 0 for hard-pinned vertices.
//
// The kernels are a small part of a call (0.2 of 2.4 ms for a 500 x 500 grid
// when every list had its own count, scan and scatter: 33 launches); the rest
// was the host's: 21 allocations and their frees (1.0 ms), a check of the
// triangle indices (0.6 ms) and the downloads into new pages.  So the two
// CSRs that depend on the mesh alone (sides, corners) are built together over
// 2 V rows, the two that depend on the rows (edges, bend pairs) likewise, the
// index check rides on the first pass over the triangles, and everything
// lives in one allocation: 12 launches, and with the caller's arrays shrunk in
// place instead of copied, 3.81 -> 0.67 ms for the Python call.  What is left
// is the transfer of 19 MB into pages that the caller has just been given.
#include <algorithm>
#include <cstdint>
#include <string>

#include "xpbd_solver.cuh"

#define XG_EXPORT extern "C" __attribute__((visibility("default")))

namespace xg {
namespace {

constexpr int kPrepThreads = 256;

inline int blocks_of(long long n) { return (int)((n + kPrepThreads - 1) / kPrepThreads); }

__device__ __forceinline__ bool in_mesh(int i, int V) { return i >= 0 && i < V; }

// Triangle t: sides counted at their lower endpoints (count[0, V)), corners at
// their vertices (count[V, 2V)), and the triangle's share of its corners'
// masses, max(area * density, eps) / 3 in float32.  A triangle with an index
// outside the mesh is left out of everything and reported: `bad` ends as
// 3 T - (first such index's place), 0 when there is none.
__global__ void __launch_bounds__(kPrepThreads) k_prep_triangles(const int* tris, int T, const float* pos, int V, float density,
                                                                 float eps, int* count, float* share, int* bad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int i[3] = {tris[3 * t], tris[3 * t + 1], tris[3 * t + 2]};
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (!in_mesh(i[j], V)) {
            atomicMax(bad, 3 * (T - t) - j);
            return;
        }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        atomicAdd(&count[min(i[j], i[(j + 1) % 3])], 1);
        atomicAdd(&count[V + i[j]], 1);
    }
    const float* p0 = pos + 3ll * i[0];
    const float* p1 = pos + 3ll * i[1];
    const float* p2 = pos + 3ll * i[2];
    const float ux = p1[0] - p0[0], uy = p1[1] - p0[1], uz = p1[2] - p0[2];
    const float vx = p2[0] - p0[0], vy = p2[1] - p0[1], vz = p2[2] - p0[2];
    const float cx = uy * vz - uz * vy, cy = uz * vx - ux * vz, cz = ux * vy - uy * vx;
    const float area = 0.5f * sqrtf((cx * cx + cy * cy) + cz * cz);
    share[t] = fmaxf(area * density, eps) / 3.0f;
}

// Sides as (upper endpoint << 32 | side index s = 3 t + j), so that a sorted
// row lists every edge's sides in triangle order; corners as corner * T + t,
// so that a sorted row is np.add.at's order.  The corners' rows follow the
// sides' in `cursor` and start at cursor - (number of sides).
__global__ void __launch_bounds__(kPrepThreads) k_prep_scatter(const int* tris, int T, int V, int* cursor, const int* start,
                                                               long long* sides, int* corners) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int i[3] = {tris[3 * t], tris[3 * t + 1], tris[3 * t + 2]};
    if (!in_mesh(i[0], V) || !in_mesh(i[1], V) || !in_mesh(i[2], V)) return;
    const int corner0 = start[V];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int a = i[j], b = i[(j + 1) % 3];
        sides[atomicAdd(&cursor[min(a, b)], 1)] = ((long long)max(a, b) << 32) | (long long)(3 * t + j);
        corners[atomicAdd(&cursor[V + a], 1) - corner0] = (int)((long long)j * T + t);
    }
}

// Sort one CSR row in place (insertion sort: rows are a vertex's incident
// sides or corners, a handful of entries on a manifold mesh).
template <class T>
__device__ __forceinline__ void sort_row(T* r, int n) {
    for (int i = 1; i < n; ++i) {
        const T key = r[i];
        int j = i - 1;
        while (j >= 0 && r[j] > key) {
            r[j + 1] = r[j];
            --j;
        }
        r[j + 1] = key;
    }
}

// Thread x < V: vertex x's side row sorted, its edges counted (count[x]) and
// its bend pairs listed (xpbd_core.py:730-747): the first side of an edge
// gives the reference opposite vertex; each later side whose opposite vertex
// differs yields the pair (min, max) of the two opposite vertices, written
// into the row's own slots (at most one per side) and counted at the lower
// one (count[V + p]).  Thread V + v: vertex v's inverse mass.
__global__ void __launch_bounds__(kPrepThreads) k_prep_rows(const int* start, long long* sides, int* corners, const int* tris,
                                                            int T, int V, const float* share, const unsigned char* hard,
                                                            int* count, int* pair_p, int* pair_q, int* row_pairs, float* inv) {
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= 2 * V) return;
    if (at >= V) {
        const int v = at - V;
        int* r = corners + (start[V + v] - start[V]);
        const int n = start[V + v + 1] - start[V + v];
        sort_row(r, n);
        double mass = 0.0;
        for (int i = 0; i < n; ++i) mass += (double)share[r[i] % T];
        if (mass <= 0.0) mass = 1.0;
        inv[v] = (hard && hard[v]) ? 0.0f : (float)(1.0 / mass);
        return;
    }
    const int row = start[at], n = start[at + 1] - row;
    long long* r = sides + row;
    sort_row(r, n);
    int edges = 0, m = 0, last = -1, first_opp = 0;
    for (int i = 0; i < n; ++i) {
        const int y = (int)(r[i] >> 32);
        if (!pair_p) {
            edges += y != last;
            last = y;
            continue;
        }
        const int s = (int)(r[i] & 0xffffffffll);
        const int opp = tris[3 * (s / 3) + (s % 3 + 2) % 3];
        if (y != last) {
            ++edges;
            last = y;
            first_opp = opp;
        } else if (opp != first_opp) {
            const int p = min(first_opp, opp);
            pair_p[row + m] = p;
            pair_q[row + m] = max(first_opp, opp);
            ++m;
            atomicAdd(&count[V + p], 1);
        }
    }
    count[at] = edges;
    if (pair_p) row_pairs[at] = m;
}

__device__ __forceinline__ float rest_length(const float* pos, int a, int b, float eps) {
    const float* p = pos + 3ll * a;
    const float* q = pos + 3ll * b;
    const float dx = q[0] - p[0], dy = q[1] - p[1], dz = q[2] - p[2];
    return fmaxf(sqrtf((dx * dx + dy * dy) + dz * dz), eps);
}

// Vertex x's edges with their rest lengths, and its bend pairs' upper
// vertices into the rows of their lower ones (which follow the edges' in
// `cursor`, and start at cursor - (number of edges)).
__global__ void __launch_bounds__(kPrepThreads) k_prep_edges(const int* start, const long long* sides, const int* edge_start,
                                                             const float* pos, int V, float eps, int2* edges, float* rest,
                                                             int* cursor, const int* pair_p, const int* pair_q,
                                                             const int* row_pairs, int* pairs) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= V) return;
    const int row = start[x], n = start[x + 1] - row;
    int e = edge_start[x], last = -1;
    for (int i = 0; i < n; ++i) {
        const int y = (int)(sides[row + i] >> 32);
        if (y == last) continue;
        last = y;
        edges[e] = make_int2(x, y);
        rest[e++] = rest_length(pos, x, y, eps);
    }
    if (!pair_p) return;
    const int pair0 = edge_start[V];
    for (int i = 0, m = row_pairs[x]; i < m; ++i)
        pairs[atomicAdd(&cursor[V + pair_p[row + i]], 1) - pair0] = pair_q[row + i];
}

// Row a of the bend pairs: sorted, distinct upper vertices at its front, counted.
__global__ void __launch_bounds__(kPrepThreads) k_prep_pair_rows(const int* edge_start, int* pairs, int V, int* distinct) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= V) return;
    const int n = edge_start[V + a + 1] - edge_start[V + a];
    int* r = pairs + (edge_start[V + a] - edge_start[V]);
    sort_row(r, n);
    int u = 0;
    for (int i = 0; i < n; ++i)
        if (u == 0 || r[i] != r[u - 1]) r[u++] = r[i];
    distinct[a] = u;
}

__global__ void __launch_bounds__(kPrepThreads) k_prep_bends(const int* edge_start, const int* pairs, const int* bend_start,
                                                             const float* pos, int V, float eps, int2* bends, float* rest) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= V) return;
    const int* r = pairs + (edge_start[V + a] - edge_start[V]);
    const int b0 = bend_start[a], n = bend_start[a + 1] - b0;
    for (int i = 0; i < n; ++i) {
        bends[b0 + i] = make_int2(a, r[i]);
        rest[b0 + i] = rest_length(pos, a, r[i], eps);
    }
}

// Places in one allocation, each on a 256-byte boundary.
struct Arena {
    size_t size = 0;
    size_t take(size_t bytes) {
        const size_t at = size;
        size += (std::max<size_t>(bytes, 1) + 255) & ~(size_t)255;
        return at;
    }
};

}  // namespace
}  // namespace xg

using namespace xg;

// Edges, rest lengths, inverse masses and (when `bends` is given) bend pairs
// with their rest lengths of a cloth from its rest positions (V x 3 float),
// triangles (T x 3 int, indices in [0, V)), density and hard pin mask (V
// bytes, non-zero = pinned; may be null).  `edges` / `bends` hold room for
// 3T pairs, `edge_rest` / `bend_rest` for 3T floats, `inv_mass` for V
// floats; *bend_count receives the bend count.  Returns the number of edges,
// or -1 (ssbl_last_error() says why).
XG_EXPORT int xpbd_gb300_prepare_cloth_device(const float* positions, int vertex_count, const int* triangles,
                                              int triangle_count, float density, float eps, const unsigned char* hard,
                                              int* edges, float* edge_rest, float* inv_mass, int* bends,
                                              float* bend_rest, int* bend_count) {
    if (bend_count) *bend_count = 0;
    if (bends && (!bend_rest || !bend_count)) {
        set_last_error("invalid cloth preprocessing request");
        return -1;
    }
    const int V = vertex_count, T = triangle_count;
    if (V < 0 || T < 0 || (V > 0 && (!positions || !inv_mass)) || (T > 0 && (!triangles || !edges || !edge_rest)) ||
        3ll * T > (1ll << 30) || V > (1 << 30) - 4096) {
        set_last_error("invalid cloth preprocessing request");
        return -1;
    }
    // the first index outside the mesh, or 3 T
    auto first_bad = [&]() {
        long long i = 0;
        while (i < 3ll * T && triangles[i] >= 0 && triangles[i] < V) ++i;
        return i;
    };
    auto bad_index = [&](long long i) {
        set_last_error("triangle index " + std::to_string(triangles[i]) + " outside the " + std::to_string(V) + " vertices");
        return -1;
    };
    if (V == 0) return T > 0 ? bad_index(0) : 0;
    cudaStream_t st = nullptr;
    char* mem = nullptr;
    auto finish = [&](int result, const char* what) {
        if (what) {
            set_last_error(std::string("cloth preprocessing: ") + what + ": " + cudaGetErrorString(cudaGetLastError()));
            const long long i = first_bad();  // a mesh that is no mesh is that first of all
            if (i < 3ll * T) bad_index(i);
        }
        if (st) cudaStreamSynchronize(st);
        if (mem) cudaFree(mem);
        if (st) cudaStreamDestroy(st);
        return what ? -1 : result;
    };
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return finish(0, "stream");
    const size_t S = 3 * (size_t)T, N = (size_t)V;
    Arena A;
    const size_t o_pos = A.take(12 * N), o_tris = A.take(4 * S), o_hard = A.take(hard ? N : 0);
    // row counts of the sides and corners, then of the edges and bend pairs; the index check's result
    const size_t o_count = A.take(4 * (4 * N + 1)), o_start = A.take(4 * (2 * N + 1)), o_estart = A.take(4 * (2 * N + 1));
    const size_t o_sums = A.take(4 * (2 * N / 4096 + 2)), o_sides = A.take(8 * S), o_corners = A.take(4 * S);
    const size_t o_share = A.take(4 * (size_t)T), o_inv = A.take(4 * N), o_edges = A.take(8 * S), o_rest = A.take(4 * S);
    const size_t P = bends ? S : 0, R = bends ? N : 0;
    const size_t o_pp = A.take(4 * P), o_pq = A.take(4 * P), o_rowp = A.take(4 * R), o_pairs = A.take(4 * P);
    const size_t o_distinct = A.take(4 * R), o_bstart = A.take(4 * (R + 1)), o_bedges = A.take(8 * P), o_brest = A.take(4 * P);
    if (cudaMalloc(reinterpret_cast<void**>(&mem), A.size) != cudaSuccess) {
        mem = nullptr;
        return finish(0, "device allocation");
    }
    auto ints = [&](size_t o) { return reinterpret_cast<int*>(mem + o); };
    auto floats = [&](size_t o) { return reinterpret_cast<float*>(mem + o); };
    float *d_pos = floats(o_pos), *d_rest = floats(o_rest), *d_share = floats(o_share), *d_inv = floats(o_inv);
    unsigned char* d_hard = hard ? reinterpret_cast<unsigned char*>(mem + o_hard) : nullptr;
    int *d_tris = ints(o_tris), *d_count = ints(o_count), *d_start = ints(o_start), *d_estart = ints(o_estart);
    int *d_sums = ints(o_sums), *d_corners = ints(o_corners), *d_count2 = d_count + 2 * N, *d_bad = d_count + 4 * N;
    int *d_pp = bends ? ints(o_pp) : nullptr, *d_pq = ints(o_pq), *d_rowp = ints(o_rowp), *d_pairs = ints(o_pairs);
    int *d_distinct = ints(o_distinct), *d_bstart = ints(o_bstart);
    long long* d_sides = reinterpret_cast<long long*>(mem + o_sides);
    int2 *d_edges = reinterpret_cast<int2*>(mem + o_edges), *d_bedges = reinterpret_cast<int2*>(mem + o_bedges);
    float* d_brest = floats(o_brest);
    const bool up = cudaMemcpyAsync(d_pos, positions, 12 * N, cudaMemcpyHostToDevice, st) == cudaSuccess &&
                    (T == 0 || cudaMemcpyAsync(d_tris, triangles, 4 * S, cudaMemcpyHostToDevice, st) == cudaSuccess) &&
                    (!hard || cudaMemcpyAsync(d_hard, hard, N, cudaMemcpyHostToDevice, st) == cudaSuccess) &&
                    cudaMemsetAsync(d_count, 0, 4 * (4 * N + 1), st) == cudaSuccess;
    if (!up) return finish(0, "upload");
    if (T > 0) k_prep_triangles<<<blocks_of(T), kPrepThreads, 0, st>>>(d_tris, T, d_pos, V, density, eps, d_count, d_share, d_bad);
    scan_bucket_counts(d_count, d_start, 2 * V, d_sums, st);  // the counts become the scatter's cursors
    if (T > 0) k_prep_scatter<<<blocks_of(T), kPrepThreads, 0, st>>>(d_tris, T, V, d_count, d_start, d_sides, d_corners);
    k_prep_rows<<<blocks_of(2ll * V), kPrepThreads, 0, st>>>(d_start, d_sides, d_corners, d_tris, std::max(T, 1), V, d_share, d_hard,
                                                            d_count2, d_pp, d_pq, d_rowp, d_inv);
    scan_bucket_counts(d_count2, d_estart, 2 * V, d_sums, st);
    k_prep_edges<<<blocks_of(V), kPrepThreads, 0, st>>>(d_start, d_sides, d_estart, d_pos, V, eps, d_edges, d_rest, d_count2, d_pp,
                                                        d_pq, d_rowp, d_pairs);
    if (bends) {
        k_prep_pair_rows<<<blocks_of(V), kPrepThreads, 0, st>>>(d_estart, d_pairs, V, d_distinct);
        scan_bucket_counts(d_distinct, d_bstart, V, d_sums, st);
        k_prep_bends<<<blocks_of(V), kPrepThreads, 0, st>>>(d_estart, d_pairs, d_bstart, d_pos, V, eps, d_bedges, d_brest);
    }
    int E = 0, NB = 0, bad = 0;
    if (cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(&E, d_estart + V, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        (bends && cudaMemcpyAsync(&NB, d_bstart + V, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return finish(0, "edge build");
    if (bad > 0) {
        finish(0, nullptr);
        return bad_index(3ll * T - bad);
    }
    if (bend_count) *bend_count = NB;
    const bool ok = (NB == 0 || (cudaMemcpyAsync(bends, d_bedges, 8 * (size_t)NB, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
                                 cudaMemcpyAsync(bend_rest, d_brest, 4 * (size_t)NB, cudaMemcpyDeviceToHost, st) == cudaSuccess)) &&
                    (E == 0 || (cudaMemcpyAsync(edges, d_edges, 8 * (size_t)E, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
                                cudaMemcpyAsync(edge_rest, d_rest, 4 * (size_t)E, cudaMemcpyDeviceToHost, st) == cudaSuccess)) &&
                    cudaMemcpyAsync(inv_mass, d_inv, 4 * N, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
                    cudaStreamSynchronize(st) == cudaSuccess && cudaGetLastError() == cudaSuccess;
    if (!ok) return finish(0, "download");
    return finish(E, nullptr);
}
