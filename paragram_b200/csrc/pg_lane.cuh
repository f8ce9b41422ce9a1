// pg_lane.cuh -- one lane's cell: the polytope of the cell-per-lane pass (pg_lane.cu).
//
// Shared memory is laid out [slot][lane], so that the lanes' accesses to a slot's vertex
// never share a bank. Planes are not stored but recomputed from their points, whose loads
// L1 and L2 serve, and what a search and a clip need only in turn lies in one place, so
// that 256 cells fit in an SM's shared memory.
#pragma once

#include "pg_clip.cuh"

namespace pg
{

constexpr int kLaneP = 24;      // plane slots of a cell: V vertices lie on V / 2 + 2 planes, and one more in a clip
constexpr int kLaneStack = 64;  // pending BVH nodes of a warp's search
constexpr int kLaneLeaves = 92; // leaves that a warp's search lists before they are scanned
constexpr int kLaneCut = 48;    // points of a search that may cut a cell
static_assert(kLaneP >= kLaneV / 2 + 3 && kLaneP <= 32, "a live mask has a bit for each plane");

// One warp's 32 cells (lane = column) and its search of the BVH.
struct LaneMem
{
    float4 vx[kLaneV][32];          // vertex relative to the seed; w: error radius psi
    unsigned short vt[kLaneV][32];  // its plane slots, five bits each
    int pid[kLaneP][32];            // >= 0: sorted point index; < 0: -1 - box code
    union
    {
        unsigned dx[kLaneP / 4][32]; // in a clip (else zero), per plane slot (bytes): xor of its boundary successor and predecessor
        struct
        {
            float4 pt[32];           // points of the leaf pair in work
            int lv[kLaneLeaves + 4]; // leaves within reach
        };
    };
};
static_assert(sizeof(LaneMem) + 1024 <= 228 * 1024 / 8, "eight blocks of one warp per SM");

__device__ __forceinline__ unsigned tri5(unsigned a, unsigned b, unsigned c) { return a | (b << 5) | (c << 10); }

struct LPlane
{
    float4 p; // n, h
    float e;  // bound on |h - h_exact|
};

// Plane of a candidate point (as make_cand) or of a box face (as the warp-per-cell pass's cell_init).
__device__ __forceinline__ LPlane lane_plane(int pid, float4 s, const float4 *__restrict__ pts, const float *box)
{
    LPlane r;
    if (pid >= 0)
    {
        float4 q = pts[pid];
        float nx = q.x - s.x, ny = q.y - s.y, nz = q.z - s.z;
        float n2 = __fmaf_rn(nx, nx, __fmaf_rn(ny, ny, __fmul_rn(nz, nz)));
        float dw = q.w - s.w;
        float h = 0.5f * __fsub_rn(n2, dw);
        r.p = make_float4(nx, ny, nz, h);
        r.e = 2.0f * kEps * (fabsf(h) + 3.0f * n2 + fabsf(dw));
    }
    else
    {
        int code = -1 - pid, ax = code >> 1, hi = code & 1;
        float sc = ax == 0 ? s.x : (ax == 1 ? s.y : s.z);
        float b = box[hi * 3 + ax];
        float h = hi ? __fsub_rn(b, sc) : __fsub_rn(sc, b);
        float sg = hi ? 1.0f : -1.0f;
        r.p = make_float4(ax == 0 ? sg : 0.0f, ax == 1 ? sg : 0.0f, ax == 2 ? sg : 0.0f, h);
        r.e = kEps * fabsf(h);
    }
    return r;
}

// Squared distance of two points; k_knn and the cell pass compute it alike, so that they agree exactly.
__device__ __forceinline__ float lane_sq_dist(float4 a, float4 b)
{
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
}

// phases of the cell-per-lane pass (cycle counters)
enum LaneCyc : int
{
    kLaneCycNear,
    kLaneCycSearch,
    kLaneCycTests,
    kLaneCycClips,
    kLaneCycNum,
};

struct LaneCell
{
    LaneMem &m;
    const CellArgs &A;
    const int lane;
    int i = -1, soid = 0;
    float4 s;
    const float *const box;
    bool alive = false, defer = false, empty = false;
    int nv = 0;              // vertices (slots 0 .. nv - 1)
    unsigned live = 0;       // plane slots that a vertex uses
    float rsafe = INFINITY;  // no vertex lies farther from the seed (after radius())
    // statistics
    unsigned n_tests = 0, n_nodes = 0, n_leaves = 0, n_clips = 0, n_cands = 0, n_fp64 = 0, n_exp = 0, n_v64 = 0,
             n_hit = 0, n_miss = 0;
#ifdef PG_PHASE_CYCLES
    long long cyc[kLaneCycNum] = {};
#endif

    __device__ __forceinline__ LaneCell(LaneMem &mem, const CellArgs &args, int l) : m(mem), A(args), lane(l), box(args.box)
    {
        s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        clear_dx();
    }
    __device__ __forceinline__ void clear_dx()
    {
#pragma unroll
        for (int k = 0; k < kLaneP / 4; ++k)
            m.dx[k][lane] = 0u;
    }
    __device__ __forceinline__ float4 &vxl(int v) { return m.vx[v][lane]; }
    __device__ __forceinline__ unsigned tri_of(int v) { return m.vt[v][lane]; }
    __device__ __forceinline__ int &pidl(unsigned p) { return m.pid[p][lane]; }
    __device__ __forceinline__ unsigned char &dxa(unsigned x)
    {
        return reinterpret_cast<unsigned char *>(&m.dx[x >> 2][lane])[x & 3u];
    }
    // ints in the place of the vertices (once these are no longer needed)
    __device__ __forceinline__ int &lst(int k) { return reinterpret_cast<int *>(&m.vx[k >> 2][lane])[k & 3]; }
    __device__ __forceinline__ void give_up()
    {
        defer = true;
        alive = false;
    }
    // lowest set bit of the two-word mask (r0, r1), cleared
    static __device__ __forceinline__ int take(unsigned &r0, unsigned &r1)
    {
        if (r0)
        {
            const int v = __ffs(r0) - 1;
            r0 &= r0 - 1u;
            return v;
        }
        const int v = 31 + __ffs(r1);
        r1 &= r1 - 1u;
        return v;
    }
    static __device__ __forceinline__ unsigned tri_bits(unsigned tr)
    {
        return (1u << (tr & 31u)) | (1u << ((tr >> 5) & 31u)) | (1u << (tr >> 10));
    }

    // Cell of sorted slot c of a build of one cloud: the box (planes 0..5, corners 0..7).
    __device__ __forceinline__ void init(int c)
    {
        i = c;
        s = A.pts[i];
        soid = A.oid[i];
        empty = false;
        defer = false;
        alive = true;
        rsafe = INFINITY;
        nv = 8;
        live = 0x3Fu;
        float h[6], eh[6];
#pragma unroll
        for (int k = 0; k < 6; ++k)
        {
            float sc = (k >> 1) == 0 ? s.x : ((k >> 1) == 1 ? s.y : s.z);
            float b = box[(k & 1) * 3 + (k >> 1)];
            h[k] = (k & 1) ? __fsub_rn(b, sc) : __fsub_rn(sc, b);
            eh[k] = kEps * fabsf(h[k]);
            pidl(k) = -1 - k;
        }
#pragma unroll
        for (int c8 = 0; c8 < 8; ++c8)
        {
            const int sx = c8 & 1, sy = (c8 >> 1) & 1, sz = (c8 >> 2) & 1;
            const int px = sx, py = 2 + sy, pz = 4 + sz;
            const int sign = (sx ? 1 : -1) * (sy ? 1 : -1) * (sz ? 1 : -1);
            const int p0 = sign > 0 ? px : py, p1 = sign > 0 ? py : px, p2 = pz;
            float X = sx ? h[px] : -h[px], Y = sy ? h[py] : -h[py], Z = sz ? h[pz] : -h[pz];
            float ex = (eh[px] + eh[py] + eh[pz]) * (1.0f + 1e-6f);
            float x2 = X * X + Y * Y + Z * Z;
            float xn = x2 > 0.0f ? x2 * rsqrtf(x2) * (1.0f + 4e-6f) : 0.0f;
            float psi = (2.0f * ex + 4.0f * kEps * xn) * (1.0f + 1e-6f);
            vxl(c8) = make_float4(X, Y, Z, psi);
            m.vt[c8][lane] = tri5(p0, p1, p2);
        }
    }

    // No vertex (with its error bound) lies farther from the seed than rsafe.
    __device__ __forceinline__ void radius()
    {
        float r = 0.0f;
#pragma unroll 4
        for (int v = 0; v < nv; ++v)
        {
            const float4 X = vxl(v);
            const float x2 = X.x * X.x + X.y * X.y + X.z * X.z;
            r = fmaxf(r, (x2 > 0.0f ? x2 * rsqrtf(x2) * (1.0f + 4e-6f) : 0.0f) + X.w);
        }
        rsafe = r * (1.0f + 1e-6f);
    }

    // Which of four candidates may remove a vertex (bit clear: it certainly removes none). One pass over the
    // vertices serves all four: independent chains, and a quarter of the shared-memory reads.
    __device__ __forceinline__ unsigned may_cut4(const Cand (&cq)[4])
    {
        float nrm[4], c[4];
        bool any[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            nrm[u] = cq[u].nrm * (1.0f + 2e-6f);
            c[u] = cq[u].cerr * (1.0f + 2e-6f) + 2e-6f * fabsf(cq[u].h) - cq[u].h;
            any[u] = !(cq[u].cerr < 1e30f);
        }
#pragma unroll 2
        for (int v = 0; v < nv; ++v)
        {
            const float4 X = vxl(v);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                any[u] = any[u] || __fmaf_rn(cq[u].nx, X.x,
                                             __fmaf_rn(cq[u].ny, X.y, __fmaf_rn(cq[u].nz, X.z, __fmaf_rn(nrm[u], X.w, c[u])))) > 0.0f;
        }
        n_tests += 4 * nv;
        return (any[0] ? 1u : 0u) | (any[1] ? 2u : 0u) | (any[2] ? 4u : 0u) | (any[3] ? 8u : 0u);
    }

    // The vertices that candidate j removes, as bits of (r0, r1). False: none, or the cell was given up.
    __device__ __forceinline__ bool classify(const Cand &cq, int j, unsigned &r0, unsigned &r1)
    {
        r0 = r1 = 0u;
        bool und = false;
        const float nrm = cq.nrm * (1.0f + 2e-6f), cerr = cq.cerr * (1.0f + 2e-6f);
        auto side = [&](int v) -> unsigned {
            const float4 X = vxl(v);
            const float g = __fmaf_rn(cq.nx, X.x, __fmaf_rn(cq.ny, X.y, __fmaf_rn(cq.nz, X.z, -cq.h)));
            const float b = __fmaf_rn(nrm, X.w, cerr);
            und = und || !(fabsf(g) > b);
            return g > b ? 1u : 0u;
        };
        for (int v = nv - 1; v >= 32; --v)
            r1 = r1 * 2u + side(v);
#pragma unroll 4
        for (int v = min(nv, 32) - 1; v >= 0; --v)
            r0 = r0 * 2u + side(v);
        n_tests += nv;
        if (und)
            for (int v = 0; v < nv; ++v)
            {
                int r = side_fp32(vxl(v), cq);
                if (r < 0)
                {
                    const unsigned tr = tri_of(v);
                    int used = 0;
                    r = side_exact(pidl(tr & 31u), pidl((tr >> 5) & 31u), pidl(tr >> 10), j, A.pts, A.oid, box, s,
                                   soid, &used);
                    ++n_fp64;
                    n_exp += used ? 1u : 0u;
                    if (r < 0)
                    {
                        give_up(); // the warp-per-cell pass reports it
                        return false;
                    }
                }
                if (r == 1)
                    (v < 32 ? r0 : r1) |= 1u << (v & 31);
            }
        return (r0 | r1) != 0u;
    }

    // Clip by candidate j, which removes the vertices (r0, r1).
    __device__ __forceinline__ void update(const Cand &cq, int j, unsigned r0, unsigned r1)
    {
        if (__popc(r0) + __popc(r1) == nv)
        {
            empty = true;
            alive = false;
            return;
        }
        const unsigned P = __ffs(~live) - 1;
        if (P >= (unsigned)kLaneP)
        {
            give_up(); // (not reached: see kLaneP)
            return;
        }
        ++n_clips;
        pidl(P) = j;
        // Boundary of the removed region. Every removed triangle xors, for each of its planes, the other
        // two into that plane's byte: inside the region each neighbour enters twice, so a plane on the
        // boundary keeps (successor xor predecessor) and an interior plane 0, and the cycle can be walked
        // from any one boundary edge.
        unsigned removed_planes = 0, inter = 0;
        unsigned tr0 = tri_of(r0 ? __ffs(r0) - 1 : 31 + __ffs(r1));
        unsigned mt0 = tri_bits(tr0);
        for (unsigned w0 = r0, w1 = r1; (w0 | w1) != 0u;)
        {
            const unsigned tr = tri_of(take(w0, w1));
            const unsigned a = tr & 31u, b = (tr >> 5) & 31u, c = tr >> 10;
            dxa(a) ^= b ^ c;
            dxa(b) ^= c ^ a;
            dxa(c) ^= a ^ b;
            const unsigned mt = tri_bits(tr);
            removed_planes |= mt;
            if (__popc(mt & mt0) == 2)
                inter |= mt0 & ~mt; // the edge of the first triangle opposite to this plane is interior
        }
        // a triangle with all three edges interior: take another one
        for (unsigned w0 = r0, w1 = r1; (w0 | w1) != 0u && (mt0 & ~inter) == 0u;)
        {
            tr0 = tri_of(take(w0, w1));
            mt0 = tri_bits(tr0);
            inter = 0;
            for (unsigned u0 = r0, u1 = r1; (u0 | u1) != 0u;)
            {
                const unsigned mu = tri_bits(tri_of(take(u0, u1)));
                if (__popc(mu & mt0) == 2)
                    inter |= mt0 & ~mu;
            }
        }
        unsigned x, z; // a boundary edge z -> x
        {
            const unsigned a = tr0 & 31u, b = (tr0 >> 5) & 31u, c = tr0 >> 10;
            const unsigned open = mt0 & ~inter;
            if ((open >> c) & 1u)
                z = a, x = b;
            else if ((open >> a) & 1u)
                z = b, x = c;
            else
                z = c, x = a;
        }
        // the cycle of planes along the boundary, five bits each, from x on (12 in seq0, the rest in seq1)
        const unsigned xs = x;
        unsigned boundary = 0;
        unsigned long long seq0 = 0, seq1 = 0;
        int nb = 0;
        do
        {
            const unsigned y = ((unsigned)dxa(x) ^ z) & 31u;
            dxa(x) = 0;
            boundary |= 1u << x;
            if (nb < 12)
                seq0 |= (unsigned long long)x << (5 * nb);
            else
                seq1 |= (unsigned long long)x << (5 * nb - 60);
            ++nb;
            z = x;
            x = y;
        } while (x != xs && nb < 24);
        const int nr = __popc(r0) + __popc(r1);
        if (x != xs || nv - nr + nb > kLaneV)
        {
            // out of vertex slots (or an inconsistent boundary): the warp-per-cell pass
            give_up();
            clear_dx();
            return;
        }
        // the new vertices (P, x, y) along it, in the removed slots first; the next plane is loaded beside
        // the arithmetic of the present vertex
        const float4 pP = make_float4(cq.nx, cq.ny, cq.nz, cq.h);
        unsigned ill0 = 0, ill1 = 0;
        auto next = [&](int k) -> unsigned {
            seq0 = (seq0 >> 5) | ((seq1 & 31ull) << 55);
            seq1 >>= 5;
            return k < nb ? (unsigned)seq0 & 31u : xs;
        };
        LPlane px = lane_plane(pidl(xs), s, A.pts, box);
        x = xs;
        unsigned y = next(1);
        LPlane py = lane_plane(pidl(y), s, A.pts, box);
#pragma unroll 1
        for (int k = 0; k < nb; ++k)
        {
            const unsigned w = next(k + 2);
            const LPlane pw = lane_plane(pidl(w), s, A.pts, box);
            float vr;
            float4 X = make_vertex(pP, cq.eh, px.p, px.e, py.p, py.e, vr);
            const int slot = (r0 | r1) != 0u ? take(r0, r1) : nv++;
            if (!(X.w <= kVertex64Rel * (fabsf(X.x) + fabsf(X.y) + fabsf(X.z))))
            {
                (slot < 32 ? ill0 : ill1) |= 1u << (slot & 31);
                if (!(X.w < 1e30f))
                    X = make_float4(0.0f, 0.0f, 0.0f, INFINITY); // (not NaN: such a vertex may be cut by any point)
            }
            vxl(slot) = X;
            m.vt[slot][lane] = tri5(P, x, y);
            x = y;
            y = w;
            px = py;
            py = pw;
        }
        live = (live & ~removed_planes) | boundary | (1u << P);
        // ill-conditioned in FP32: rebuilt in FP64 so that the empty sphere stays tight
        while ((ill0 | ill1) != 0u)
        {
            const int v = take(ill0, ill1);
            const float4 X = vxl(v);
            const unsigned tr = tri_of(v);
            float vr;
            const float4 Y = make_vertex64(pidl(tr & 31u), pidl((tr >> 5) & 31u), pidl(tr >> 10), A.pts, A.oid, box, s,
                                           X, 0.0f, vr);
            if (Y.w < X.w)
                vxl(v) = Y;
            ++n_v64;
        }
        // holes left by removed vertices are filled from the end
        while ((r0 | r1) != 0u)
        {
            const int hole = r1 ? 63 - __clz(r1) : 31 - __clz(r0);
            (r1 ? r1 : r0) &= ~(1u << (hole & 31));
            --nv;
            if (hole != nv)
            {
                vxl(hole) = vxl(nv);
                m.vt[hole][lane] = m.vt[nv][lane];
            }
        }
    }

    // Whether point j is one of the cell's planes.
    __device__ __forceinline__ bool has_plane(int j)
    {
        bool has = false;
        for (unsigned w = live; w != 0u; w &= w - 1u)
            has = has || pidl(__ffs(w) - 1) == j;
        return has;
    }

    // Geometry and vertex export of a finished cell, as export_cell of pg_cells.cu: the vertices whose error
    // radius exceeds 32 ulps are first solved in FP64; the volume is the signed sum of the tetrahedra (o, f_a,
    // v, u) over the directed edges v -> u of every face a, o the mean vertex and f_a the foot of its
    // perpendicular on the face. Two vertices share an edge when their triples share two planes; the edge t - u
    // of t = (a, b, c) and u = (a, c, d) runs t -> u in face a and u -> t in face c.
    __device__ __forceinline__ void export_cell()
    {
        if (defer)
            return; // the larger pass exports it
        const bool vertices = A.vertex_count_out != nullptr || A.vertices_out != nullptr || A.vertex_planes_out != nullptr;
        if (empty)
        {
            const float nan = __int_as_float(0x7fc00000);
            if (A.geometry_out != nullptr)
                A.geometry_out[soid] = make_float4(nan, nan, nan, 0.0f);
            if (A.vertex_count_out != nullptr)
                A.vertex_count_out[soid] = 0;
            return;
        }
        float ox = 0.0f, oy = 0.0f, oz = 0.0f;
#pragma unroll 1
        for (int v = 0; v < nv; ++v)
        {
            float4 X = vxl(v);
            if (!(X.w <= 32.0f * kEps * (fabsf(X.x) + fabsf(X.y) + fabsf(X.z))))
            {
                const unsigned tr = tri_of(v);
                X = vertex64_plain(pidl(tr & 31u), pidl((tr >> 5) & 31u), pidl(tr >> 10), A.pts, A.oid, box, s, X);
                vxl(v) = X;
            }
            ox += X.x;
            oy += X.y;
            oz += X.z;
            if (vertices && v < A.vertex_cap)
            {
                const size_t at = (size_t)soid * A.vertex_cap + v;
                if (A.vertices_out != nullptr)
                    A.vertices_out[at] = X;
                if (A.vertex_planes_out != nullptr)
                {
                    const unsigned tr = tri_of(v);
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                    {
                        const int id = pidl((tr >> (5 * e)) & 31u);
                        A.vertex_planes_out[at * 3 + e] = id >= 0 ? A.oid[id] : id;
                    }
                }
            }
        }
        if (A.vertex_count_out != nullptr)
            A.vertex_count_out[soid] = nv;
        if (A.geometry_out == nullptr)
            return;
        const float inv = 1.0f / (float)nv;
        ox *= inv;
        oy *= inv;
        oz *= inv;
        auto foot = [&](unsigned p) -> float3 {
            const float4 n = lane_plane(pidl(p), s, A.pts, box).p;
            const float sc =
                (n.w - (n.x * ox + n.y * oy + n.z * oz)) / (n.x * n.x + n.y * n.y + n.z * n.z);
            return make_float3(n.x * sc, n.y * sc, n.z * sc);
        };
        double S = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll 1
        for (int t = 0; t < nv; ++t)
        {
            const unsigned tr = tri_of(t), bt = tri_bits(tr);
            int e0 = -1, e1 = -1, e2 = -1; // the later vertices that share an edge with t
            for (int u = t + 1; u < nv; ++u)
                if (__popc(bt & tri_bits(tri_of(u))) == 2)
                {
                    e2 = e1;
                    e1 = e0;
                    e0 = u;
                }
            const float4 T = vxl(t);
            const float vx = T.x - ox, vy = T.y - oy, vz = T.z - oz;
            while (e0 >= 0)
            {
                const unsigned shared = bt & tri_bits(tri_of(e0));
                const unsigned p0 = tr & 31u, p1 = (tr >> 5) & 31u, p2 = tr >> 10;
                unsigned a = p1, c = p0; // b = p2
                if (!((shared >> p0) & 1u))
                    a = p2, c = p1;
                else if (!((shared >> p1) & 1u))
                    a = p0, c = p2;
                const float4 U = vxl(e0);
                const float ux = U.x - ox, uy = U.y - oy, uz = U.z - oz;
                const float rx = vy * uz - vz * uy, ry = vz * ux - vx * uz, rz = vx * uy - vy * ux;
                const float3 fa = foot(a), fc = foot(c);
                const float da = fa.x * rx + fa.y * ry + fa.z * rz, dc = -(fc.x * rx + fc.y * ry + fc.z * rz);
                S += (double)da + (double)dc;
                cx += (double)da * (fa.x + vx + ux) + (double)dc * (fc.x + vx + ux);
                cy += (double)da * (fa.y + vy + uy) + (double)dc * (fc.y + vy + uy);
                cz += (double)da * (fa.z + vz + uz) + (double)dc * (fc.z + vz + uz);
                e0 = e1;
                e1 = e2;
                e2 = -1;
            }
        }
        const double q = 0.25 / S;
        A.geometry_out[soid] =
            make_float4((float)((double)s.x + (double)ox + cx * q), (float)((double)s.y + (double)oy + cy * q),
                        (float)((double)s.z + (double)oz + cz * q), (float)(fabs(S) / 6.0));
    }

    // Row, degree and status of a finished cell, or its entry in `list` (counted in *list_n).
    __device__ __forceinline__ void output(int *list, int *list_n)
    {
        if (defer)
        {
            A.deg[soid] = 0;
            A.status[soid] = kPlaneOverflow; // placeholder until the pass over the list
            list[atomicAdd(list_n, 1)] = i;
        }
        else if (empty)
        {
            A.deg[soid] = 0;
            A.status[soid] = kEmptyCell;
        }
        else
        {
            int d = 0;
            for (unsigned w = live; w != 0u; w &= w - 1u)
            {
                const int id = pidl(__ffs(w) - 1);
                if (id < 0)
                    continue;
                const int o = A.oid[id];
                int k = d++;
                for (; k > 0 && lst(k - 1) > o; --k)
                    lst(k) = lst(k - 1);
                lst(k) = o;
            }
            int *row = A.rows + (size_t)soid * kRowWidth;
            for (int k = 0; k < d; ++k)
                row[k] = lst(k);
            A.deg[soid] = d;
            A.status[soid] = kSuccess;
        }
    }

    __device__ __forceinline__ void flush_one(unsigned v, int idx)
    {
        unsigned long long sum = v;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            sum += __shfl_xor_sync(kFull, sum, o);
        if (lane == 0 && sum != 0ull)
            atomicAdd(&A.stats[idx], sum);
    }
    __device__ __forceinline__ void flush()
    {
        flush_one(n_tests, kStatTests);
        flush_one(n_nodes, kStatNodes);
        flush_one(n_leaves, kStatLeaves);
        flush_one(n_clips, kStatClips);
        flush_one(n_cands, kStatCandidates);
        flush_one(n_fp64, kStatFp64);
        flush_one(n_exp, kStatExpansion);
        flush_one(n_v64, kStatVertex64);
        flush_one(n_hit, kStatHintHit);
        flush_one(n_miss, kStatHintMiss);
#ifdef PG_PHASE_CYCLES
        // (every lane of a warp is in the same phase: each of its cells sees these cycles)
        long long all = 0;
        for (int k = 0; k < kLaneCycNum; ++k)
            all += cyc[k];
        if (lane == 0)
        {
            atomicAdd(&A.stats[kStatCycCell], (unsigned long long)all);
            atomicAdd(&A.stats[kStatCycWarm], (unsigned long long)cyc[kLaneCycNear]);
            atomicAdd(&A.stats[kStatCycNodes], (unsigned long long)cyc[kLaneCycSearch]);
            atomicAdd(&A.stats[kStatCycLeaves], (unsigned long long)(cyc[kLaneCycTests] + cyc[kLaneCycClips]));
            atomicAdd(&A.stats[kStatCycClips], (unsigned long long)cyc[kLaneCycClips]);
        }
#endif
    }
};

} // namespace pg
