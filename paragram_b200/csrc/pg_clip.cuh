// pg_clip.cuh -- what the cell kernels share: the candidate plane, its FP32 side
// test with a rigorous error bound, the exact cascade behind it, and the vertex
// of three planes with its a-posteriori error bound.
#pragma once

#include <cfloat>
#include <climits>

#include "pg_common.cuh"
#include "pg_exact.cuh"

namespace pg
{

constexpr float kEps = 5.9604645e-8f; // 2^-24
// A vertex whose FP32 error radius exceeds this fraction of its L1 norm is rebuilt in FP64.
#ifndef PG_VERTEX64_REL
#define PG_VERTEX64_REL 3e-4f
#endif
constexpr float kVertex64Rel = PG_VERTEX64_REL;
constexpr unsigned kFull = 0xFFFFFFFFu;

struct CellArgs
{
    const float4 *pts;
    const int *oid;
    const int *rank;
    const float4 *rec;
    const float *box;        // 8 floats per cloud: reference box lo xyz, hi xyz, max weight
    const int *cloud_off;    // [clouds + 1]
    const int *cloud_root;   // [clouds]
    int num_clouds;
    int n;
    int window;
    const int *guesses;
    const int *guess_off;
    int *rows;
    int *deg;
    int *status;
    int *big_list;
    int *big_list2; // cells that outgrew the middle tier too, and their deferred-row slots
    int *big_slot2;
    int *big_rows;
    int *counters;
    unsigned long long *stats;
    int64_t begin, end;
    const int *list; // cells that the cell-per-lane pass left (sorted slots; their number in counters[kCountListed])
    LaneChoice choice;
    int64_t big_cap;
    char *huge_slabs;
    float *radius_out; // optional per-cell diagnostics (original ids)
    int4 *work_out;
    float4 *geometry_out; // optional per-cell centroid and volume (original ids)
    int vertex_cap;            // optional vertex export (original ids)
    float4 *vertices_out;
    int *vertex_planes_out;
    int *vertex_count_out;
    const float *hint; // search radius per sorted slot (learned or given), or nullptr
    const int *rparent; // record node -> entry in its parent's record
    const int *pleaf;   // sorted point -> entry of its leaf
    int fp32_only;      // undecided FP32 side tests take the FP32 sign (no exact cascade)
};

struct Cand
{
    float nx, ny, nz, h;
    float nrm;  // upper bound on |q - s|
    float cerr; // constant part of the side-test error bound
    float eh;   // bound on |h - h_exact|
    int id;     // sorted index
};

__device__ __forceinline__ Cand make_cand(float4 s, float4 q, int id)
{
    Cand c;
    c.nx = q.x - s.x;
    c.ny = q.y - s.y;
    c.nz = q.z - s.z;
    float n2 = __fmaf_rn(c.nx, c.nx, __fmaf_rn(c.ny, c.ny, __fmul_rn(c.nz, c.nz)));
    float dw = q.w - s.w;
    c.h = 0.5f * __fsub_rn(n2, dw);
    c.eh = 2.0f * kEps * (fabsf(c.h) + 3.0f * n2 + fabsf(dw));
    c.nrm = n2 * rsqrtf(n2) * (1.0f + 4e-6f); // rsqrtf: <= 2 ulp
    c.cerr = (3.0f * kEps * fabsf(c.h) + c.eh) * (1.0f + 8.0f * kEps);
    if (!(n2 > 1e-30f && n2 < 1e30f))
        c.cerr = INFINITY; // out of the filter's range: always exact
    c.id = id;
    return c;
}

// +1 removed, 0 kept, -1 undecided
__device__ __forceinline__ int side_fp32(float4 X, const Cand &q)
{
    float g = __fmaf_rn(q.nx, X.x, __fmaf_rn(q.ny, X.y, __fmaf_rn(q.nz, X.z, -q.h)));
    float b = __fmaf_rn(q.nrm, X.w, q.cerr) * (1.0f + 1e-6f);
    return g > b ? 1 : (g < -b ? 0 : -1);
}

// Source of plane `pid` (a sorted point index, or -1 - box code) of a cell
// whose cloud box is `box`.
// Sign of the FP32 side value alone (1 removed, 0 kept), for FP32-only predicates.
__device__ __forceinline__ int side_fp32_sign(float4 X, const Cand &q)
{
    float g = __fmaf_rn(q.nx, X.x, __fmaf_rn(q.ny, X.y, __fmaf_rn(q.nz, X.z, -q.h)));
    return g > 0.0f ? 1 : 0;
}

__device__ __forceinline__ exact::PlaneSrc plane_src(int pid, const float4 *__restrict__ pts,
                                                     const int *__restrict__ oid, const float *__restrict__ box)
{
    exact::PlaneSrc r;
    if (pid >= 0)
    {
        float4 p = pts[pid];
        r.x = p.x;
        r.y = p.y;
        r.z = p.z;
        r.w = p.w;
        r.box = -1;
        r.oid = oid[pid];
    }
    else
    {
        int code = -1 - pid;
        r.x = box[(code & 1) * 3 + (code >> 1)];
        r.y = r.z = r.w = 0.0f;
        r.box = code;
        r.oid = -1;
    }
    return r;
}

// Exact cascade for one undecided test. Takes plain values so that no
// per-warp state has its address taken (which would move it to local memory).
static __device__ __noinline__ int side_exact(int p0, int p1, int p2, int qid, const float4 *__restrict__ pts,
                                       const int *__restrict__ oid, const float *__restrict__ box, float4 s, int soid,
                                       int *used)
{
    exact::PlaneSrc vp[3] = {plane_src(p0, pts, oid, box), plane_src(p1, pts, oid, box), plane_src(p2, pts, oid, box)};
    exact::PlaneSrc cp = plane_src(qid, pts, oid, box);
    return exact::side_test(vp, cp, s.x, s.y, s.z, s.w, soid, used);
}

// Vertex of three planes (FP32 Cramer) with its side-test error radius psi.
__device__ __forceinline__ float4 make_vertex(float4 a, float ea, float4 b, float eb, float4 c, float ec, float &vr)
{
    float u0x = b.y * c.z - b.z * c.y, u0y = b.z * c.x - b.x * c.z, u0z = b.x * c.y - b.y * c.x;
    float u1x = c.y * a.z - c.z * a.y, u1y = c.z * a.x - c.x * a.z, u1z = c.x * a.y - c.y * a.x;
    float u2x = a.y * b.z - a.z * b.y, u2y = a.z * b.x - a.x * b.z, u2z = a.x * b.y - a.y * b.x;
    float D = a.x * u0x + a.y * u0y + a.z * u0z;
    float nx = a.w * u0x + b.w * u1x + c.w * u2x;
    float ny = a.w * u0y + b.w * u1y + c.w * u2y;
    float nz = a.w * u0z + b.w * u1z + c.w * u2z;
    // any FP32 point is acceptable here: the bound below is a-posteriori
    float rD = __frcp_rn(D);
    float X = nx * rD, Y = ny * rD, Z = nz * rD;
    float x2 = X * X + Y * Y + Z * Z;
    float xn = x2 > 0.0f ? x2 * rsqrtf(x2) * (1.0f + 4e-6f) : 0.0f;
    float la = fabsf(a.x) + fabsf(a.y) + fabsf(a.z);
    float lb = fabsf(b.x) + fabsf(b.y) + fabsf(b.z);
    float lc = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
    float ra = fabsf(__fmaf_rn(a.x, X, __fmaf_rn(a.y, Y, __fmaf_rn(a.z, Z, -a.w)))) + 4.0f * kEps * (la * xn + fabsf(a.w)) + ea;
    float rb = fabsf(__fmaf_rn(b.x, X, __fmaf_rn(b.y, Y, __fmaf_rn(b.z, Z, -b.w)))) + 4.0f * kEps * (lb * xn + fabsf(b.w)) + eb;
    float rc = fabsf(__fmaf_rn(c.x, X, __fmaf_rn(c.y, Y, __fmaf_rn(c.z, Z, -c.w)))) + 4.0f * kEps * (lc * xn + fabsf(c.w)) + ec;
    // X - X_exact = adj(A) r / D with the columns u0, u1, u2 of adj(A) and the residuals r, so
    // |X - X_exact| <= (ra |u0| + rb |u1| + rc |u2|) / |D|, each |u_i| bounded with its rounding
    // error (2 eps per product pair). Per-plane weighting keeps the bound tight for a vertex far
    // along a thin prism, whose large-offset box plane only moves it along the prism axis.
    float q0 = u0x * u0x + u0y * u0y + u0z * u0z;
    float q1 = u1x * u1x + u1y * u1y + u1z * u1z;
    float q2 = u2x * u2x + u2y * u2y + u2z * u2z;
    float U0 = (q0 > 0.0f ? q0 * rsqrtf(q0) * (1.0f + 4e-6f) : 0.0f) + 8.0f * kEps * lb * lc;
    float U1 = (q1 > 0.0f ? q1 * rsqrtf(q1) * (1.0f + 4e-6f) : 0.0f) + 8.0f * kEps * lc * la;
    float U2 = (q2 > 0.0f ? q2 * rsqrtf(q2) * (1.0f + 4e-6f) : 0.0f) + 8.0f * kEps * la * lb;
    float num = (ra * U0 + rb * U1 + rc * U2) * (1.0f + 4e-6f);
    float den = fabsf(D) - 8.0f * kEps * la * lb * lc;
    float ex = den > 0.0f ? __fdividef(num, den) * (1.0f + 4e-6f) : INFINITY;
    float psi = (2.0f * ex + 4.0f * kEps * xn) * (1.0f + 1e-6f);
    if (!(psi < 1e30f) || !(xn < 1e30f))
        psi = INFINITY;
    float r = xn + psi;
    vr = r * r * (1.0f + 1e-6f);
    return make_float4(X, Y, Z, psi);
}

// Vertex of three planes rebuilt in FP64 from the planes' sources (the FP32
// plane coefficients are themselves rounded), for a vertex whose FP32 error
// radius is large: three nearly dependent planes, e.g. two bisectors of
// near-coplanar points meeting a third along a long thin cell. Returns the FP32
// point with psi = 2 * (FP64 a-posteriori bound) + |X32 - X64| + the FP32
// side-test rounding term, or `fallback` when a plane is not exact in FP64.
static __device__ __noinline__ float4 make_vertex64(int pid0, int pid1, int pid2, const float4 *__restrict__ pts,
                                             const int *__restrict__ oid, const float *__restrict__ box, float4 s,
                                             float4 fallback, float fallback_vr, float &vr)
{
    const double u = 1.1102230246251565e-16; // 2^-53
    exact::DRow r[3];
    exact::make_drow(plane_src(pid0, pts, oid, box), s.x, s.y, s.z, s.w, r[0]);
    exact::make_drow(plane_src(pid1, pts, oid, box), s.x, s.y, s.z, s.w, r[1]);
    exact::make_drow(plane_src(pid2, pts, oid, box), s.x, s.y, s.z, s.w, r[2]);
    if (!(r[0].ok && r[1].ok && r[2].ok))
    {
        vr = fallback_vr;
        return fallback;
    }
    // plane i: a_i . X = b_i / 2 with |b_i - b_i exact| <= eb_i
    const double *a = r[0].a, *b = r[1].a, *c = r[2].a;
    double u0x = b[1] * c[2] - b[2] * c[1], u0y = b[2] * c[0] - b[0] * c[2], u0z = b[0] * c[1] - b[1] * c[0];
    double u1x = c[1] * a[2] - c[2] * a[1], u1y = c[2] * a[0] - c[0] * a[2], u1z = c[0] * a[1] - c[1] * a[0];
    double u2x = a[1] * b[2] - a[2] * b[1], u2y = a[2] * b[0] - a[0] * b[2], u2z = a[0] * b[1] - a[1] * b[0];
    double D = a[0] * u0x + a[1] * u0y + a[2] * u0z;
    double h0 = 0.5 * r[0].b, h1 = 0.5 * r[1].b, h2 = 0.5 * r[2].b;
    double X = (h0 * u0x + h1 * u1x + h2 * u2x) / D;
    double Y = (h0 * u0y + h1 * u1y + h2 * u2y) / D;
    double Z = (h0 * u0z + h1 * u1z + h2 * u2z) / D;
    double la = fabs(a[0]) + fabs(a[1]) + fabs(a[2]);
    double lb = fabs(b[0]) + fabs(b[1]) + fabs(b[2]);
    double lc = fabs(c[0]) + fabs(c[1]) + fabs(c[2]);
    double xn = sqrt(X * X + Y * Y + Z * Z) * (1.0 + 1e-14);
    double ra = fabs(fma(a[0], X, fma(a[1], Y, fma(a[2], Z, -h0)))) + 4.0 * u * (la * xn + fabs(h0)) + 0.5 * r[0].eb;
    double rb = fabs(fma(b[0], X, fma(b[1], Y, fma(b[2], Z, -h1)))) + 4.0 * u * (lb * xn + fabs(h1)) + 0.5 * r[1].eb;
    double rc = fabs(fma(c[0], X, fma(c[1], Y, fma(c[2], Z, -h2)))) + 4.0 * u * (lc * xn + fabs(h2)) + 0.5 * r[2].eb;
    double U0 = sqrt(u0x * u0x + u0y * u0y + u0z * u0z) * (1.0 + 1e-14) + 4.0 * u * lb * lc;
    double U1 = sqrt(u1x * u1x + u1y * u1y + u1z * u1z) * (1.0 + 1e-14) + 4.0 * u * lc * la;
    double U2 = sqrt(u2x * u2x + u2y * u2y + u2z * u2z) * (1.0 + 1e-14) + 4.0 * u * la * lb;
    double den = fabs(D) - 8.0 * u * la * lb * lc;
    if (!(den > 0.0) || !(xn < 1e30))
    {
        vr = fallback_vr;
        return fallback;
    }
    double ex = (ra * U0 + rb * U1 + rc * U2) / den * (1.0 + 1e-13);
    float fx = (float)X, fy = (float)Y, fz = (float)Z;
    double dx = (double)fx - X, dy = (double)fy - Y, dz = (double)fz - Z;
    double e32 = sqrt(dx * dx + dy * dy + dz * dz) * (1.0 + 1e-14);
    float x2 = fx * fx + fy * fy + fz * fz;
    float xnf = x2 > 0.0f ? x2 * rsqrtf(x2) * (1.0f + 4e-6f) : 0.0f;
    float psi = (float)((2.0 * ex + e32) * (1.0 + 1e-6)) * (1.0f + 1e-6f) + 4.0f * kEps * xnf;
    if (!(psi < fallback.w))
    {
        vr = fallback_vr;
        return fallback;
    }
    float rr = xnf + psi;
    vr = rr * rr * (1.0f + 1e-6f);
    return make_float4(fx, fy, fz, psi);
}

// The vertex of three planes solved in FP64 from the planes' sources (the
// bisector coefficients are exact differences of FP32 values), without the
// error bound of make_vertex64: a vertex of the cell geometry. Returns X
// unchanged when the planes do not give exact FP64 rows or a usable solve.
static __device__ __noinline__ float4 vertex64_plain(int pid0, int pid1, int pid2, const float4 *__restrict__ pts,
                                              const int *__restrict__ oid, const float *__restrict__ box, float4 s,
                                              float4 X)
{
    exact::DRow r[3];
    exact::make_drow(plane_src(pid0, pts, oid, box), s.x, s.y, s.z, s.w, r[0]);
    exact::make_drow(plane_src(pid1, pts, oid, box), s.x, s.y, s.z, s.w, r[1]);
    exact::make_drow(plane_src(pid2, pts, oid, box), s.x, s.y, s.z, s.w, r[2]);
    if (!(r[0].ok && r[1].ok && r[2].ok))
        return X;
    const double *a = r[0].a, *b = r[1].a, *c = r[2].a;
    double u0x = b[1] * c[2] - b[2] * c[1], u0y = b[2] * c[0] - b[0] * c[2], u0z = b[0] * c[1] - b[1] * c[0];
    double u1x = c[1] * a[2] - c[2] * a[1], u1y = c[2] * a[0] - c[0] * a[2], u1z = c[0] * a[1] - c[1] * a[0];
    double u2x = a[1] * b[2] - a[2] * b[1], u2y = a[2] * b[0] - a[0] * b[2], u2z = a[0] * b[1] - a[1] * b[0];
    double D = a[0] * u0x + a[1] * u0y + a[2] * u0z;
    if (!(fabs(D) > 0.0))
        return X;
    double q = 0.5 / D;
    double x = (r[0].b * u0x + r[1].b * u1x + r[2].b * u2x) * q;
    double y = (r[0].b * u0y + r[1].b * u1y + r[2].b * u2y) * q;
    double z = (r[0].b * u0z + r[1].b * u1z + r[2].b * u2z) * q;
    return make_float4((float)x, (float)y, (float)z, X.w);
}

} // namespace pg
