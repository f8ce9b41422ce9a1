// pg_lane.cu -- per-cell convex clipping, one cell per lane.
//
// The first pass of builds that fill the GPU (build_impl's rule). The same clipping
// and the same exact predicates as pg_cells.cu (reference counterpart:
// voronoi_ultra.cu:39-141, laguerre_ultra.cu:43-174, also one thread per cell), so
// the cells are the same; what differs is who does the work. A warp per cell issues
// every step of a cell's search once per cell (28,900 warp instructions for a cell of
// about 27 vertices, 21.8 of 32 lanes active); 32 cells per warp, kept in step, share
// them: 6,300 per cell.
//
// What keeps the lanes in step: (1) a cell is first clipped by its kLaneWarm nearest
// points (k_knn), nearly all of which cut it; (2) the points that can still
// reach it come from one search of the BVH for the warp's 32 cells, whose nodes and
// leaves every lane tests at the same time; (3) the points in reach are tested four
// at a time against the vertices, and only those that may cut (about 8 of 50) are
// kept for clipping; (4) in clipping every lane first looks for its next point that
// cuts, then all clip. Lanes that search on their own (a traversal per lane, whether
// left to diverge or scheduled step by step) ran at 4 to 10 active lanes: 45 and
// 22 ms for 500,000 clustered cells, against 21 ms for a warp per cell and 11 here.
// Eight lanes per cell: 26 ms (instruction-cache misses between the steps).
//
// Builds whose points would mostly be listed are declined as a whole (LaneChoice,
// pg_common.cuh). A cell that does not fit (more than kLaneV vertices, a reach that holds
// more than kLaneMarks points: cells at the hull, beside a far denser region, or long cells
// of surface data) is listed for the warp-per-cell pass: 3% of 5M clustered cells, 8% of
// 500,000, 22% of 60,000.
//
// Measured on one B200, first pass with its kNN query and listed cells: 2M clustered
// points 85.3 -> 37.2 ms, 500,000 21.1 -> 10.8 ms, 500,000 uniform power 21.5 -> 9.6 ms,
// jittered 80^3 power lattice 19.5 -> 5.8 ms. Bound by latency: one warp per block, 8
// blocks per SM (28 KB of shared memory each), 38% of the issue slots used.
#include <algorithm>

#include "pg_kernels.cuh"
#include "pg_lane.cuh"

namespace pg
{

constexpr int kLaneBlocks = 8; // resident one-warp blocks per SM (28 KB of shared memory each)
// Squared radius of the first search over the last near point's. 500,000 clustered cells: 2.0 14.5, 2.5 13.8,
// 3.0 14.8 ms (a smaller one leaves more cells to the second search, a larger one more points to test).
constexpr float kLaneShell = 2.5f;
constexpr float kLaneFar = 6.0f; // the largest that a cell may need after it (beyond: listed)
constexpr int kLaneMarks = 96;   // points of a search within a cell's reach

// Optional per-phase SM cycle counters, as in pg_cells.cu (compile with -DPG_PHASE_CYCLES): the clips by the
// nearest points, the search, its tests, the clips by its points, and whole cells, per cell.
#ifdef PG_PHASE_CYCLES
#define PG_LANE_T0(t) long long t = clock64()
#define PG_LANE_T1(cell, k, t)                                                                                         \
    do                                                                                                                 \
    {                                                                                                                  \
        const long long pg_now_ = clock64();                                                                           \
        (cell).cyc[k] += pg_now_ - (t);                                                                                \
        (t) = pg_now_;                                                                                                 \
    } while (0)
#else
#define PG_LANE_T0(t)
#define PG_LANE_T1(cell, k, t)
#endif

__device__ __forceinline__ float lane_box_dist(float4 s, float lx, float ly, float lz, float hx, float hy, float hz)
{
    const float dx = fmaxf(fmaxf(lx - s.x, s.x - hx), 0.0f), dy = fmaxf(fmaxf(ly - s.y, s.y - hy), 0.0f),
                dz = fmaxf(fmaxf(lz - s.z, s.z - hz), 0.0f);
    return (dx * dx + dy * dy + dz * dz) * (1.0f - 1e-5f);
}

// 32 consecutive cells of the curve order per warp at a time (persistent warps, cells from a counter).
// GUESS: the caller's initial guesses clip a cell first, in the place of its nearest points. EXPORT: geometry
// and vertices are asked for. A search radius per cell (A.hint: learned or given) bounds its first search; a
// negative one marks a cell that the model routed past this pass.
template <bool GUESS, bool EXPORT>
__global__ void __launch_bounds__(32, kLaneBlocks) k_cells_lane(CellArgs A, int *list)
{
    __shared__ LaneMem m;
    const int lane = threadIdx.x;
    if (A.choice.declined())
        return; // every cell is left to k_cells_list
    LaneCell C(m, A, lane);
    const int root = A.cloud_root[0];
    unsigned cmask[kLaneLeaves / 2];
    int cand[kLaneCut];
    for (;;)
    {
        int g = 0;
        if (lane == 0)
            g = atomicAdd(&A.counters[0], 1);
        g = __shfl_sync(kFull, g, 0);
        const int64_t gb = (A.begin & ~(int64_t)31) + (int64_t)g * 32;
        if (gb >= A.end)
            break;
        // Groups lie at multiples of 32 of the curve order and are built whole, so that a cell does not depend on
        // the range or chunk that asks for it (what its warp searches for depends on the other cells of the
        // group); cells outside the range are not written.
        const bool mine = gb + lane >= A.begin && gb + lane < A.end;
        bool act = gb + lane < A.n;
        C.init((int)(act ? gb + lane : A.n - 1));
        float hint = INFINITY; // search radius
        if (A.hint != nullptr)
        {
            const float r = A.hint[C.i];
            if (r > 0.0f && r < 1e30f)
                hint = r;
            act = act && !(r < 0.0f);
        }
        C.alive = C.alive && act;
        PG_LANE_T0(t0);
        // Its nearest points (sorted slots, nearest first, -1: none, left in the cell's row) clip a cell first,
        // then the other points within reach, in shells around it. No point farther than
        // R + sqrt(R^2 + w) can cut a cell of radius R, w the excess of the cloud's largest weight over the
        // seed's: its bisector distance (d^2 - dw) / (2 d) exceeds R.
        int nk = 0, jK = -1;
        float dK = 0.0f; // squared distance of the last of them, the scale of the search
        bool search = C.alive;
        if (GUESS)
        {
            const int g0 = A.guess_off[C.soid], g1 = A.guess_off[C.soid + 1];
            if (C.alive && g1 - g0 > kLaneCut)
                C.give_up();
            for (int k = g0; C.alive && k < g1; ++k)
            {
                const int o = A.guesses[k];
                const int j = o >= 0 && o < A.n ? A.rank[o] : -1;
                if (j >= 0 && j != C.i)
                {
                    cand[nk++] = j;
                    dK += __log2f(fmaxf(lane_sq_dist(C.s, A.pts[j]), 1e-30f));
                }
            }
            // the scale of the search: the geometric mean, which the far neighbours of a cell at the hull hardly
            // move, to about where the 16th nearest point lies (1.6 times it among uniform points)
            dK = nk > 0 ? 1.6f * exp2f(dK / (float)nk) : 0.0f;
            search = C.alive;
        }
        else
        {
            const int4 *kn = reinterpret_cast<const int4 *>(A.rows + (size_t)C.soid * kRowWidth);
#pragma unroll
            for (int t = 0; t < kLaneWarm / 4; ++t)
            {
                const int4 k4 = kn[t];
                cand[4 * t + 0] = k4.x;
                cand[4 * t + 1] = k4.y;
                cand[4 * t + 2] = k4.z;
                cand[4 * t + 3] = k4.w;
                nk += (k4.x >= 0) + (k4.y >= 0) + (k4.z >= 0) + (k4.w >= 0);
                jK = k4.w;
            }
            if (C.alive && jK == -2)
                C.give_up();
            search = C.alive && jK >= 0; // (fewer points than that: all of them are in the list)
            if (search)
                dK = lane_sq_dist(C.s, A.pts[jK]);
        }
        if (search && !(dK > 0.0f && dK < 1e30f))
        {
            C.give_up(); // no scale to search by: no guesses, or coincident points only
            search = false;
        }
        if (!C.alive)
            nk = 0;
        const float dwm = search ? fmaxf(C.box[6] - C.s.w, 0.0f) * (1.0f + 1e-6f) : 0.0f;
        float lo = GUESS ? 0.0f : dK, hi = 0.0f; // the points nearer than lo were clipped
#pragma unroll 1
        for (int shell = -1; shell < 4; ++shell)
        {
            if (shell >= 0)
            {
                search = search && C.alive;
                if (search)
                {
                    C.radius();
                    float need = C.rsafe + sqrtf(fmaf(C.rsafe, C.rsafe, dwm));
                    need = need * need * (1.0f + 4e-5f);
                    const bool base = lo < kLaneShell * dK; // within the first radius
                    if (need <= lo)
                        search = false; // every point within reach was clipped
                    else if (shell == 3 || (!base && need > kLaneFar * dK))
                    {
                        C.give_up();
                        search = false;
                    }
                    hi = base ? fminf(need, kLaneShell * dK) : need;
                    if (shell == 0)
                    {
                        const float r = hint + sqrtf(fmaf(hint, hint, dwm));
                        hi = fmaxf(fminf(hi, r * r * (1.0f + 4e-5f)), lo);
                    }
                }
                if (!__any_sync(kFull, search))
                    break;
                // Points with lo <= d^2 <= hi of every lane's cell: one search of the BVH for the warp's 32 cells.
                // Leaves within reach of some lane are listed, scanned in pairs into a bit mask per lane, and the
                // marked points tested; those that may remove a vertex of the present cell are kept.
                nk = 0;
                int sp = 0, marks = 0;
                bool over = false;
                float rr = search ? hi : -1.0f;
                // pending nodes: entry k in lane k % 32's stk0 (k < 32) or stk1
                int stk0 = root, stk1 = 0;
                auto pending = [&](int k) -> int { return __shfl_sync(kFull, k < 32 ? stk0 : stk1, k & 31); };
                sp = 1;
                while (sp > 0)
                {
                    int nl = 0;
                    while (sp > 0 && nl <= kLaneLeaves - 4)
                    {
                        // two nodes at a time: their loads overlap
                        const int two = sp > 1 ? 1 : 0;
                        const float4 *pa = A.rec + 4 * (size_t)pending(sp - 1),
                                     *pb = A.rec + 4 * (size_t)pending(sp - 1 - two);
                        const float4 a0 = pa[0], a1 = pa[1], a2 = pa[2], a3 = pa[3];
                        const float4 b0 = pb[0], b1 = pb[1], b2 = pb[2], b3 = pb[3];
                        sp -= 1 + two;
                        // (the two children of each; a lane counts those within its own reach)
                        const bool mine[4] = {lane_box_dist(C.s, a0.x, a0.y, a0.z, a0.w, a1.x, a1.y) <= rr,
                                              lane_box_dist(C.s, a1.z, a1.w, a2.x, a2.y, a2.z, a2.w) <= rr,
                                              two && lane_box_dist(C.s, b0.x, b0.y, b0.z, b0.w, b1.x, b1.y) <= rr,
                                              two && lane_box_dist(C.s, b1.z, b1.w, b2.x, b2.y, b2.z, b2.w) <= rr};
                        if (sp + 4 > kLaneStack)
                        {
                            over = true;
                            break;
                        }
                        const float f4[4] = {a3.x, a3.y, b3.x, b3.y};
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (__any_sync(kFull, mine[c]))
                            {
                                const int f = __float_as_int(f4[c]);
                                C.n_nodes += mine[c] ? 1u : 0u;
                                C.n_leaves += mine[c] && f < 0 ? 1u : 0u;
                                if (f < 0)
                                {
                                    if (lane == 0)
                                        m.lv[nl] = f;
                                    ++nl;
                                }
                                else
                                {
                                    if (lane == (sp & 31))
                                        (sp < 32 ? stk0 : stk1) = f;
                                    ++sp;
                                }
                            }
                        __syncwarp();
                    }
                    if (over)
                        break;
                    if (lane == 0)
                        m.lv[nl] = 0; // the last pair may have one leaf
                    __syncwarp();
                    const int nr = (nl + 1) >> 1;
                    auto load = [&](int k) -> float4 {
                        const int ref = m.lv[2 * k + (lane >> 4)];
                        return ref < 0 && (lane & 15) < leaf_count(ref) ? A.pts[leaf_first(ref) + (lane & 15)]
                                                                        : make_float4(INFINITY, INFINITY, INFINITY, 0.0f);
                    };
                    float4 pt = load(0);
                    for (int k = 0; k < nr; ++k)
                    {
                        m.pt[lane] = pt;
                        __syncwarp();
                        if (k + 1 < nr)
                            pt = load(k + 1);
                        unsigned mask = 0;
#pragma unroll
                        for (int p = 0; p < 32; ++p)
                        {
                            const float d = lane_sq_dist(C.s, m.pt[p]);
                            if (d >= lo && d <= rr)
                                mask |= 1u << p;
                        }
                        cmask[k] = mask;
                        marks += __popc(mask);
                        if (marks > kLaneMarks)
                        {
                            // a far denser region within reach: listed, and no longer part of the search
                            C.give_up();
                            rr = -1.0f;
                            marks = INT_MIN;
                        }
                        __syncwarp();
                    }
                    PG_LANE_T1(C, kLaneCycSearch, t0);
                    // All lanes test up to four of their points at a time; the next four are loaded meanwhile.
                    int rd = rr >= 0.0f ? 0 : nr;
                    unsigned mw = 0;
                    int jn[4];
                    float4 qn[4];
                    auto pull = [&]() {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                        {
                            while (mw == 0u && rd < nr)
                                mw = cmask[rd++];
                            jn[u] = -1;
                            if (mw != 0u)
                            {
                                const int b = __ffs(mw) - 1;
                                mw &= mw - 1u;
                                jn[u] = leaf_first(m.lv[2 * (rd - 1) + (b >> 4)]) + (b & 15);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            qn[u] = A.pts[max(jn[u], 0)];
                    };
                    pull();
                    while (__any_sync(kFull, jn[0] >= 0))
                    {
                        int j[4];
                        float4 q4[4];
                        Cand cq[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                        {
                            j[u] = jn[u];
                            q4[u] = qn[u];
                        }
                        pull();
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            cq[u] = make_cand(C.s, q4[u], j[u]);
                        const unsigned may = j[0] >= 0 ? C.may_cut4(cq) : 0u;
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (j[u] >= 0 && ((may >> u) & 1u) &&
                                !(!GUESS && shell == 0 && j[u] <= jK && lane_sq_dist(C.s, q4[u]) == dK)) // (clipped)
                            {
                                if (nk < kLaneCut)
                                    cand[nk] = j[u];
                                ++nk;
                            }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            C.n_cands += j[u] >= 0 ? 1u : 0u;
                        __syncwarp();
                    }
                    PG_LANE_T1(C, kLaneCycTests, t0);
                }
                __syncwarp();
                C.clear_dx(); // (the search's list lies there)
                if ((over && search) || nk > kLaneCut)
                    C.give_up();
                if (!C.alive)
                    nk = 0;
                lo = __uint_as_float(__float_as_uint(hi) + 1u); // the next shell begins beyond hi
            }
            __syncwarp();
            PG_LANE_T1(C, kLaneCycTests, t0);
            // clip by the listed points that cut: every lane looks for its next one, then all clip
            int jn = nk > 0 ? cand[0] : 0;
            float4 qn = A.pts[jn];
            for (int c = 0;;)
            {
                bool cut = false;
                unsigned r0 = 0, r1 = 0;
                Cand cq;
                int j = -1;
                while (c < nk && !cut)
                {
                    j = jn;
                    const float4 q = qn;
                    if (++c < nk) // (loaded beside this point's tests)
                    {
                        jn = cand[c];
                        qn = A.pts[jn];
                    }
                    if (q.x == C.s.x && q.y == C.s.y && q.z == C.s.z)
                        continue; // coincident points do not clip each other
                    if (GUESS && C.has_plane(j))
                        continue; // clipped before
                    cq = make_cand(C.s, q, j);
                    cut = C.classify(cq, j, r0, r1);
                    if (!C.alive)
                        nk = 0;
                }
                __syncwarp();
                if (__ballot_sync(kFull, cut) == 0u)
                    break;
                if (cut)
                {
                    C.update(cq, j, r0, r1);
                    if (!C.alive)
                        nk = 0;
                }
                __syncwarp();
                PG_LANE_T1(C, shell < 0 ? kLaneCycNear : kLaneCycClips, t0);
            }
        }
        __syncwarp();
        if (A.hint != nullptr && C.alive && hint < INFINITY)
        {
            C.radius();
            C.n_hit += C.rsafe <= hint ? 1u : 0u;
            C.n_miss += C.rsafe <= hint ? 0u : 1u;
        }
        if (EXPORT && act && mine)
            C.export_cell();
        __syncwarp();
        if (act && mine)
            C.output(list, &A.counters[kCountListed]);
        __syncwarp();
    }
    C.flush();
}

// Survey of a build's points: per sampled group of 32 consecutive points of the curve (a warp's cells), whether
// they lie flat, and the level of the octree cell around them (the highest bit in which the first and last key
// differ). Flat: with the eigenvalues a >= b >= c of their covariance, c (1/a + 1/b) < 0.1. Integer sums: the
// outcome does not depend on the order of the warps.
__global__ void __launch_bounds__(256) k_lane_survey(const float4 *__restrict__ pts,
                                                     const unsigned long long *__restrict__ keys, int64_t n, int groups,
                                                     int *__restrict__ counters)
{
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    int flat = 0, level = 0, level2 = 0;
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < groups; t += warps)
    {
        const int64_t i = (n / 32) * t / groups * 32;
        const float4 p = pts[i + lane];
        auto sum = [](float v) -> float {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                v += __shfl_xor_sync(kFull, v, o);
            return v;
        };
        float x = p.x - sum(p.x) * (1.0f / 32.0f), y = p.y - sum(p.y) * (1.0f / 32.0f),
              z = p.z - sum(p.z) * (1.0f / 32.0f);
        const float big = __uint_as_float(
            __reduce_max_sync(kFull, __float_as_uint(fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))))));
        const float sc = big > 0.0f ? 1.0f / big : 0.0f;
        x *= sc;
        y *= sc;
        z *= sc;
        const float xx = sum(x * x), yy = sum(y * y), zz = sum(z * z), xy = sum(x * y), xz = sum(x * z),
                    yz = sum(y * z);
        // det = abc, minors = ab + bc + ca, trace = a + b + c
        const float m0 = yy * zz - yz * yz, m1 = xx * zz - xz * xz, m2 = xx * yy - xy * xy;
        const float det = xx * m0 - xy * (xy * zz - yz * xz) + xz * (xy * yz - yy * xz), minors = m0 + m1 + m2;
        flat += det * (xx + yy + zz) < 0.1f * minors * minors ? 1 : 0;
        const unsigned long long d = keys[i] ^ keys[i + 31];
        const int l = d != 0ull ? 63 - __clzll(d) : 0;
        level += l;
        level2 += l * l;
    }
    if (lane == 0)
    {
        atomicAdd(&counters[kCountFlat], flat);
        atomicAdd(&counters[kCountLevel], level);
        atomicAdd(&counters[kCountLevelSq], level2);
    }
}

int lane_survey_launch(const Workspace &ws, int64_t n, cudaStream_t st)
{
    const int groups = (int)std::min<int64_t>(n / 32, kSurveyGroups);
    ++g_launches;
    k_lane_survey<<<kSurveyGroups / 8, 256, 0, st>>>(ws.pts, ws.keys0, n, groups, ws.counters);
    return groups;
}

void lane_launch(const CellArgs &A, int *list, int num_sms, cudaStream_t st)
{
    const int64_t need = (A.end - (A.begin & ~(int64_t)31) + 31) / 32;
    const int64_t grid = std::min<int64_t>((int64_t)num_sms * kLaneBlocks, need);
    const bool exports = A.geometry_out || A.vertices_out || A.vertex_planes_out || A.vertex_count_out;
    void (*kern)(CellArgs, int *) = A.guesses ? (exports ? k_cells_lane<true, true> : k_cells_lane<true, false>)
                                              : (exports ? k_cells_lane<false, true> : k_cells_lane<false, false>);
    ++g_launches;
    kern<<<(unsigned)std::max<int64_t>(grid, 1), 32, 0, st>>>(A, list);
}

} // namespace pg
