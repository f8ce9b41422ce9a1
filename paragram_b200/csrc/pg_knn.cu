// pg_knn.cu -- k nearest neighbours of every point on the build's LBVH.
//
// The reference queries cuBQL for each point's K + 1 nearest points and drops
// the point itself (pwr_bvh.cu:159-215); it warm-starts every cell with them
// (voronoi_ultra.cu:205-227). Here the query runs on the LBVH of pg_build
// (pg_lbvh.cu): one thread per sorted slot (neighbouring threads query
// neighbouring points, so their traversals share nodes in L1/L2), upwards from
// the point's own leaf, the k best kept sorted by (squared distance, original
// index). Distances are the unweighted Euclidean ones in FP32 (like the
// reference's, also for power diagrams), each product and sum rounded separately so that a CPU restatement
// in float32 reproduces them and their ties exactly. A point's copies at the
// same position are neighbours like any other point; only its own index is
// excluded. The cell-per-lane pass clips its cells by the result first; pg_knn
// exports it, and the Python layer can pass it to a build as initial guesses,
// which is the reference's warm start.
#include <algorithm>
#include <string>

#include "../../include/paragram_b200.h"
#include "pg_common.cuh"
#include "pg_kernels.cuh"
#include "pg_lane.cuh"

namespace pg
{

constexpr int kKnnMax = 32;   // largest k
constexpr int kKnnStack = 96; // pending subtrees; the descent pushes one per tree level

__global__ void k_knn_single_cloud(int *cloud_off, int n)
{
    cloud_off[0] = 0;
    cloud_off[1] = n;
}

__device__ __forceinline__ float sq_dist(float4 a, float4 b)
{
    float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// Lower bound of the squared distance from q to the box (lo, hi), slightly rounded down.
__device__ __forceinline__ float box_sq_dist(float4 q, float lx, float ly, float lz, float hx, float hy, float hz)
{
    float dx = fmaxf(fmaxf(lx - q.x, q.x - hx), 0.0f);
    float dy = fmaxf(fmaxf(ly - q.y, q.y - hy), 0.0f);
    float dz = fmaxf(fmaxf(lz - q.z, q.z - hz), 0.0f);
    return (dx * dx + dy * dy + dz * dz) * (1.0f - 1e-5f);
}

// The K nearest other points of sorted slots [begin, end), nearest first. Starts at the point's own leaf and
// climbs to the cloud's root, searching each sibling subtree within the K-th distance so far. The list lives in
// registers as (distance bits, id) keys, unrolled: with a dynamically indexed array, which lives in local
// memory, and a descent from the root, 8 neighbours of 1M clustered points took 1.81 ms; 1.28 here,
// bound by the ALU (64-bit compares and selects of the insertions).
// ROWS (the cell pass): ids are sorted slots, written to the cells' rows (-1 beyond the cloud's points, -2 when
// the descent outgrew its stack). Else (pg_knn): ids are original indices, the first k of the list written.
template <int K, bool ROWS>
__global__ void __launch_bounds__(128) k_knn(int64_t begin, int64_t end, const float4 *__restrict__ pts,
                                             const int *__restrict__ oid, const float4 *__restrict__ rec,
                                             const int *__restrict__ rparent, const int *__restrict__ pleaf,
                                             const int *__restrict__ cloud_off, int num_clouds,
                                             const int *__restrict__ cloud_root, int *__restrict__ out, int k,
                                             int *err, LaneChoice choice)
{
    if (ROWS && choice.declined())
        return;
    const int64_t ii = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool alive = ii < end;
    const int i = (int)(alive ? ii : end - 1);
    const float4 q = pts[i];
    const int root = cloud_root[cloud_of(cloud_off, num_clouds, i)];
    auto dist = [&](float4 p) -> float { return ROWS ? lane_sq_dist(q, p) : sq_dist(q, p); };
    unsigned long long best[K];
#pragma unroll
    for (int t = 0; t < K; ++t)
        best[t] = ~0ull;
    float worst = INFINITY;
    int stk[kKnnStack];
    int sp = 0;
    int e = -1; // entry (parent << 1 | side) of the path node whose subtree is done
    int leaf = alive ? root : 0; // (a cloud of one leaf has no records)
    bool full = false;
    if (alive && root >= 0)
    {
        e = pleaf[i];
        const float4 r3 = rec[4 * (size_t)(e >> 1) + 3];
        leaf = __float_as_int((e & 1) ? r3.y : r3.x);
    }
    for (;;)
    {
        // the next leaf within the K-th distance: pending subtrees, then the next sibling up the path
        while (alive && leaf >= 0)
        {
            int ent;
            if (sp > 0)
                ent = stk[--sp];
            else if (e >= 0)
            {
                ent = e ^ 1;
                e = (e >> 1) == root ? -1 : rparent[e >> 1];
            }
            else
            {
                alive = false;
                break;
            }
            const float4 *r = rec + 4 * (size_t)(ent >> 1);
            const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
            const float key = (ent & 1) ? box_sq_dist(q, r1.z, r1.w, r2.x, r2.y, r2.z, r2.w)
                                        : box_sq_dist(q, r0.x, r0.y, r0.z, r0.w, r1.x, r1.y);
            if (key > worst)
                continue;
            const int ref = __float_as_int((ent & 1) ? r3.y : r3.x);
            if (ref < 0)
            {
                leaf = ref;
                break;
            }
            const float4 *c = rec + 4 * (size_t)ref;
            const float4 c0 = c[0], c1 = c[1], c2 = c[2];
            const float k0 = box_sq_dist(q, c0.x, c0.y, c0.z, c0.w, c1.x, c1.y);
            const float k1 = box_sq_dist(q, c1.z, c1.w, c2.x, c2.y, c2.z, c2.w);
            const int far = k1 >= k0 ? 1 : 0; // the nearer child is popped first
            if (sp + 2 > kKnnStack)
            {
                full = true; // the list may lack points: the cell is left to the warp-per-cell pass
                continue;
            }
            if ((far ? k1 : k0) <= worst)
                stk[sp++] = (ref << 1) | far;
            if ((far ? k0 : k1) <= worst)
                stk[sp++] = (ref << 1) | (far ^ 1);
        }
        __syncwarp();
        if (__ballot_sync(0xFFFFFFFFu, alive) == 0u)
            break;
        if (alive)
        {
            const int first = leaf_first(leaf), count = leaf_count(leaf);
            leaf = 0;
            unsigned todo = 0u;
            for (int p = 0; p < count; ++p)
                if (first + p != i && dist(pts[first + p]) <= worst)
                    todo |= 1u << p;
            for (; todo != 0u; todo &= todo - 1u)
            {
                const int j = first + __ffs(todo) - 1;
                const unsigned long long key =
                    ((unsigned long long)__float_as_uint(dist(pts[j])) << 32) | (unsigned)(ROWS ? j : oid[j]);
                bool below = key < best[K - 1];
#pragma unroll
                for (int t = K - 1; t > 0; --t)
                {
                    const bool prev = key < best[t - 1];
                    best[t] = prev ? best[t - 1] : (below ? key : best[t]);
                    below = prev;
                }
                best[0] = below ? key : best[0];
            }
            worst = best[K - 1] == ~0ull ? INFINITY : __uint_as_float((unsigned)(best[K - 1] >> 32));
        }
        __syncwarp();
    }
    if (ii >= end)
        return;
    if (!ROWS && full)
        atomicExch(err, 3);
    int *o = out + (size_t)oid[i] * (ROWS ? kRowWidth : k);
#pragma unroll
    for (int t = 0; t < K; ++t)
        if (ROWS || t < k)
            o[t] = ROWS && full ? -2 : (best[t] == ~0ull ? -1 : (int)(unsigned)best[t]);
}

void knn_rows_launch(const Workspace &ws, int num_clouds, int64_t begin, int64_t end, const LaneChoice &choice,
                     cudaStream_t st)
{
    if (end <= begin)
        return;
    ++g_launches;
    k_knn<kLaneWarm, true><<<(unsigned)((end - begin + 127) / 128), 128, 0, st>>>(
        begin, end, ws.pts, ws.oid, ws.records, ws.rparent, ws.pleaf, ws.cloud_off, num_clouds, ws.cloud_root,
        ws.rows, kLaneWarm, nullptr, choice);
}

} // namespace pg

extern "C" int pg_knn(int64_t num_points, const float *points, int32_t k, void *workspace, size_t workspace_bytes,
                      int32_t *neighbours, void *stream)
{
    using namespace pg;
    if (num_points < 0 || num_points >= kMaxPoints)
        return set_last_error(PG_ERR_INVALID, "num_points must be in [0, 2^26)");
    if (k < 1 || k > kKnnMax)
        return set_last_error(PG_ERR_INVALID, "k must be in [1, " + std::to_string(kKnnMax) + "]");
    if (num_points == 0)
        return set_last_error(PG_OK, "");
    if (!points || !workspace || !neighbours)
        return set_last_error(PG_ERR_INVALID, "points, workspace and neighbours must not be NULL");
    if (((uintptr_t)workspace & 255u) != 0)
        return set_last_error(PG_ERR_INVALID, "workspace must be 256-byte aligned");
    const size_t need = workspace_layout(num_points, 1, nullptr, nullptr);
    if (workspace_bytes < need)
        return set_last_error(PG_ERR_INVALID, "workspace too small: need " + std::to_string(need) + " bytes");
    cudaStream_t st = (cudaStream_t)stream;
    cudaGetLastError();
    Workspace ws;
    workspace_layout(num_points, 1, (char *)workspace, &ws);
    cudaMemsetAsync(ws.counters, 0, 16 * sizeof(int), st);
    ++g_launches;
    k_knn_single_cloud<<<1, 1, 0, st>>>(ws.cloud_off, (int)num_points);
    lbvh_build(ws, num_points, 1, points, nullptr, kDefaultLeaf, st);
    ++g_launches;
    // the smallest list that holds k (its length prunes the search)
    auto run = [&](auto kern) {
        kern<<<(unsigned)((num_points + 127) / 128), 128, 0, st>>>(0, num_points, ws.pts, ws.oid, ws.records,
                                                                   ws.rparent, ws.pleaf, ws.cloud_off, 1,
                                                                   ws.cloud_root, neighbours, k, &ws.counters[2],
                                                                   LaneChoice{});
    };
    if (k <= 2)
        run(k_knn<2, false>);
    else if (k <= 4)
        run(k_knn<4, false>);
    else if (k <= 6)
        run(k_knn<6, false>);
    else if (k <= 8)
        run(k_knn<8, false>);
    else if (k <= 12)
        run(k_knn<12, false>);
    else if (k <= 16)
        run(k_knn<16, false>);
    else if (k <= 24)
        run(k_knn<24, false>);
    else
        run(k_knn<32, false>);
    int flag = 0;
    cudaMemcpyAsync(&flag, &ws.counters[2], sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return set_last_error(PG_ERR_CUDA, std::string("CUDA error: ") + cudaGetErrorString(e));
    if (flag == 2)
        return set_last_error(PG_ERR_INTERNAL, "the points do not form one BVH subtree");
    if (flag == 3)
        return set_last_error(PG_ERR_INTERNAL, "kNN descent exceeded its stack (BVH deeper than 96 levels)");
    return set_last_error(PG_OK, "");
}
