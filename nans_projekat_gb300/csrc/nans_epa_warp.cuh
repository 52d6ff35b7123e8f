// GJK and EPA with a warp per candidate pair: the forms for pairs whose chain of dependent
// iterations is what their step waits for (long GJK runs, hulls of many points, polytopes beyond the
// per-thread EPA's), and for steps with too few pairs to fill the GPU with a thread each.
//
// Each lane holds a vertex of both shapes, so a support is two warp reductions; the EPA's faces lie
// in registers, two a lane. Results equal the sequential ones bit for bit: the same operations per
// vertex, face and edge, with the reference's orders kept by birth numbers in place of the loops.
#pragma once
#include "nans_gjk.cuh"

namespace nans
{

// Maximum over the warp; NaNs never win (all NaN: NaN).
__device__ __forceinline__ float warp_max(float x)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// The support of a sphere, or of a hull of more than 32 vertices read from memory, on the whole warp. A
// call of its own: inline at four places it was a third of the pair tier's code, and a small world
// waits for the tier's instructions as much as for its data. (A sphere as the second shape, the usual
// place of one, stays inline: as a call 4,608 bodies with 512 spheres took 1 % longer.)
static __device__ __noinline__ v3 warp_side_other(const float *verts, v3 p, float radius, int off, int npts, v3 d, int lane)
{
    const unsigned full = 0xffffffffu;
    if (npts == 0)
        return sphere_support(p, radius, d);
    float best = -FLT_MAX;
    v3 lv = mk3(0.0f, 0.0f, 0.0f);
    int bi = 0x7fffffff;
#pragma unroll 1
    for (int t = lane; t < npts; t += 32)
    {
        const float *q = verts + off + 3 * t;
        const v3 v = mk3(q[0], q[1], q[2]);
        const float dist = dot3(v, d);
        if (dist > best)
        {
            best = dist;
            bi = t;
            lv = v;
        }
    }
    const float m = warp_max(best);
    if (m == -FLT_MAX)
        return mk3(0.0f, 0.0f, 0.0f);
    const int i = __reduce_min_sync(full, best == m ? bi : 0x7fffffff);
    const int src = __ffs(__ballot_sync(full, bi == i)) - 1;
    return mk3(__shfl_sync(full, lv.x, src), __shfl_sync(full, lv.y, src), __shfl_sync(full, lv.z, src));
}

// Both shapes' supports, along d and -d, on the whole warp: lane t holds vertex t of a hull of up to 32
// vertices (va, vb). The first maximum over the vertices that beat -FLT_MAX, else (0, 0, 0), as
// hull_support. The two sides' reductions run beside each other (one after the other, with the calls
// above inline: 10 steps of 777 hull scenes 2.44 ms against 2.20, 60 fused steps of 9 bodies 3.59
// against 3.46, 120 taped steps of 1,024 scenes of 33 and their adjoint 29.6 against 28.9).
__device__ __forceinline__ void pair_support(const float *verts, const Shape &A, const Shape &B, v3 va, v3 vb, v3 d,
                                             int lane, v3 &sa, v3 &sb)
{
    const unsigned full = 0xffffffffu;
    const v3 nd = -1.0f * d;
    const float da = dot3(va, d), db = dot3(vb, nd);
    const float ba = lane < A.npts && da > -FLT_MAX ? da : -FLT_MAX, bb = lane < B.npts && db > -FLT_MAX ? db : -FLT_MAX;
    const float ma = warp_max(ba), mb = warp_max(bb);
    const int ia = __ffs(__ballot_sync(full, ba == ma)) - 1, ib = __ffs(__ballot_sync(full, bb == mb)) - 1;
    sa = mk3(__shfl_sync(full, va.x, ia), __shfl_sync(full, va.y, ia), __shfl_sync(full, va.z, ia));
    sb = mk3(__shfl_sync(full, vb.x, ib), __shfl_sync(full, vb.y, ib), __shfl_sync(full, vb.z, ib));
    if (ma == -FLT_MAX)
        sa = mk3(0.0f, 0.0f, 0.0f);
    if (mb == -FLT_MAX)
        sb = mk3(0.0f, 0.0f, 0.0f);
    if (A.npts == 0 || A.npts > 32)
        sa = warp_side_other(verts, A.p, A.radius, A.off, A.npts, d, lane);
    if (B.npts == 0)
        sb = sphere_support(B.p, B.radius, nd);
    else if (B.npts > 32)
        sb = warp_side_other(verts, B.p, B.radius, B.off, B.npts, nd, lane);
}

// This lane's vertex of a shape of up to 32.
__device__ __forceinline__ v3 lane_vertex(const float *verts, const Shape &s, int lane)
{
    v3 r = mk3(0.0f, 0.0f, 0.0f);
    if (lane < s.npts && s.npts <= 32)
    {
        const float *p = verts + s.off + 3 * lane;
        r = mk3(p[0], p[1], p[2]);
    }
    return r;
}

// A face in a lane's registers: normal, distance to the origin, first vertex, the three vertices
// (6 bits each) and its birth number. Faces are only erased and appended, so the reference's list
// order is the order of the birth numbers and nothing ever moves.
struct LaneFace
{
    v3 n, a;
    float d;
    unsigned v;
    int seq;
};

// PushTriangle (code/nans.cpp:292-322): N = normalize(cross(B-A, C-A)), flipped to face away from
// the origin, and the distance |dot(N, A)|.
__device__ __forceinline__ void lane_face(LaneFace &f, v3 pa, v3 pb, v3 pc, unsigned v, int seq)
{
    v3 n = normalize3(cross3(pb - pa, pc - pa));
    if (dot3(pa, n) < 0.0f)
        n = -1.0f * n;
    f.n = n;
    f.a = pa;
    f.d = fabsf(dot3(n, pa));
    f.v = v;
    f.seq = seq;
}

constexpr int kWarpEpaVerts = 34, kWarpEpaFaces = 64, kWarpEpaEdges = 32, kWarpEpaVisible = 16;
struct WarpEpa
{
    float v[9][kWarpEpaVerts]; // P, SupA, SupB by component
    unsigned edge[kWarpEpaEdges]; // u | v << 6
};
__device__ __forceinline__ v3 warp_p(const WarpEpa &S, int i) { return mk3(S.v[0][i], S.v[1][i], S.v[2][i]); }
__device__ __forceinline__ v3 warp_sup(const WarpEpa &S, int i, int side)
{
    return mk3(S.v[3 + 3 * side][i], S.v[4 + 3 * side][i], S.v[5 + 3 * side][i]);
}

// ResolveCollision (code/nans.cpp:787-904) of one pair by the whole warp, its tetrahedron in
// vertices 0..3 of S: two faces per lane in registers, a vertex of each shape per lane. Same results
// as epa_run, or EPA_OVERFLOW for a polytope this form does not hold: more than 64 faces or 34
// vertices, a repeated or NaN vertex, a repeated horizon edge, no face left.
__device__ __forceinline__ int epa_warp(const DevWorld &w, WarpEpa &S, const Shape &A, const Shape &B, v3 va, v3 vb,
                                        int lane, v3 &out_pa, v3 &out_pb, v3 &out_n, int &iters)
{
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    iters = 0;
    {
        const v3 p = warp_p(S, lane & 3);
        bool odd = isnan(p.x) || isnan(p.y) || isnan(p.z);
        for (int j = 0; j < 4; ++j)
            odd = odd || (j < (lane & 3) && eq3(warp_p(S, j), p));
        if (__any_sync(full, odd))
            return EPA_OVERFLOW;
    }
    LaneFace f0 = {}, f1 = {};
    unsigned al0 = 0xfu, al1 = 0u; // lanes whose first / second face is in the list
    {
        // ABC, ACD, ADB, BDC (code/nans.cpp:799-802)
        const int k = lane & 3, a = k == 3 ? 1 : 0, b = k == 0 ? 1 : (k == 1 ? 2 : 3),
                  c = k == 0 ? 2 : (k == 1 ? 3 : (k == 2 ? 1 : 2));
        lane_face(f0, warp_p(S, a), warp_p(S, b), warp_p(S, c), (unsigned)(a | (b << 6) | (c << 12)), k);
    }
    int nv = 4, nseq = 4;
    for (int it = 0; it <= 64; ++it)
    {
        iters = it + 1;
        const bool in0 = (al0 >> lane) & 1u, in1 = (al1 >> lane) & 1u;
        // closest face: the first minimum in list order, NaN distances never winning, except that a
        // NaN first face stays the closest (CurrentDistance starts at face 0, strict '<')
        // (distances by their bits: no negative ones; 0 stands for a NaN)
        const bool nan0 = in0 && isnan(f0.d), nan1 = in1 && isnan(f1.d);
        unsigned k0 = in0 ? (nan0 ? 0u : __float_as_uint(f0.d)) : 0xffffffffu,
                 k1 = in1 ? (nan1 ? 0u : __float_as_uint(f1.d)) : 0xffffffffu;
        unsigned m = __reduce_min_sync(full, min(k0, k1));
        bool c0 = k0 == m, c1 = k1 == m;
        if (m == 0u && __any_sync(full, nan0 || nan1))
        {
            const int fs = __reduce_min_sync(full, min(in0 ? f0.seq : 0x7fffffff, in1 ? f1.seq : 0x7fffffff));
            c0 = nan0 && f0.seq == fs;
            c1 = nan1 && f1.seq == fs;
            if (!__any_sync(full, c0 || c1))
            {
                k0 = in0 && !nan0 ? k0 : 0xffffffffu;
                k1 = in1 && !nan1 ? k1 : 0xffffffffu;
                m = __reduce_min_sync(full, min(k0, k1));
                c0 = k0 == m;
                c1 = k1 == m;
            }
        }
        unsigned b0 = __ballot_sync(full, c0), b1 = al1 ? __ballot_sync(full, c1) : 0u;
        if (__popc(b0) + __popc(b1) > 1)
        {
            const int fs = __reduce_min_sync(full, min(c0 ? f0.seq : 0x7fffffff, c1 ? f1.seq : 0x7fffffff));
            b0 = __ballot_sync(full, c0 && f0.seq == fs);
            b1 = __ballot_sync(full, c1 && f1.seq == fs);
        }
        const int src = __ffs(b0 ? b0 : b1) - 1;
        const LaneFace &fc = b0 ? f0 : f1;
        const v3 n = mk3(__shfl_sync(full, fc.n.x, src), __shfl_sync(full, fc.n.y, src), __shfl_sync(full, fc.n.z, src));
        const float cur = __shfl_sync(full, fc.d, src);
        GV ns;
        pair_support(w.verts, A, B, va, vb, n, lane, ns.sa, ns.sb);
        ns.p = ns.sa - ns.sb;
        if (dot3(n, ns.p) - cur < 0.001f)
        {
            // Barycentric (code/nans.cpp:771-785) of N * dist on the closest face
            const unsigned v = __shfl_sync(full, fc.v, src);
            const int ia = v & 63u, ib = (v >> 6) & 63u, ic = v >> 12;
            const v3 pa = warp_p(S, ia), pb = warp_p(S, ib), pc = warp_p(S, ic);
            const v3 p = cur * n;
            const v3 v0 = pb - pa, v1 = pc - pa, v2 = p - pa;
            const float d00 = dot3(v0, v0), d01 = dot3(v0, v1), d11 = dot3(v1, v1);
            const float d20 = dot3(v2, v0), d21 = dot3(v2, v1);
            const float den = d00 * d11 - d01 * d01;
            const float bv = (d11 * d20 - d01 * d21) / den;
            const float bw = (d00 * d21 - d01 * d20) / den;
            const float bu = 1.0f - bv - bw;
            if (fabsf(bu) > 1.0f || fabsf(bv) > 1.0f || fabsf(bw) > 1.0f)
                return EPA_NONE;
            if (!isfinite(bu) || !isfinite(bv) || !isfinite(bw))
                return EPA_NONE;
            out_pa = ((bu * warp_sup(S, ia, 0)) + (bv * warp_sup(S, ib, 0))) + (bw * warp_sup(S, ic, 0));
            out_n = -1.0f * n;
            out_pb = ((bu * warp_sup(S, ia, 1)) + (bv * warp_sup(S, ib, 1))) + (bw * warp_sup(S, ic, 1));
            return EPA_CONTACT;
        }
        // faces that see the new support point (code/nans.cpp:869-891)
        const bool vis0 = in0 && dot3(f0.n, ns.p - f0.a) > 0.0f, vis1 = in1 && dot3(f1.n, ns.p - f1.a) > 0.0f;
        const unsigned bv0 = __ballot_sync(full, vis0), bv1 = al1 ? __ballot_sync(full, vis1) : 0u;
        const int nvis = __popc(bv0) + __popc(bv1);
        if (nvis == 0)
            return EPA_NONE; // no face sees the support: every later iteration repeats this one
        // distinct vertices only: then an edge is the reverse of another iff their indices say so
        bool odd = isnan(ns.p.x) || isnan(ns.p.y) || isnan(ns.p.z) || nvis > kWarpEpaVisible || nv >= kWarpEpaVerts;
        for (int j = lane; j < nv && !odd; j += 32)
            odd = eq3(warp_p(S, j), ns.p);
        if (__any_sync(full, odd))
            return EPA_OVERFLOW;
        // Horizon (PushEdge, code/nans.cpp:232-266): with all pushed edges distinct, an edge
        // survives unless its reverse was pushed. Each visible face is shown to all: a lane notes
        // which of its own faces' edges it cancels and how many visible faces precede its own.
        unsigned gone0 = 0u, gone1 = 0u;
        bool twice = false;
        const unsigned p0a = f0.v & 63u, p0b = (f0.v >> 6) & 63u, p0c = f0.v >> 12;
        const unsigned p1a = f1.v & 63u, p1b = (f1.v >> 6) & 63u, p1c = f1.v >> 12;
        const unsigned e00 = p0a | (p0b << 6), e01 = p0b | (p0c << 6), e02 = p0c | (p0a << 6);
        const unsigned e10 = p1a | (p1b << 6), e11 = p1b | (p1c << 6), e12 = p1c | (p1a << 6);
        if (nvis > 1)
        {
            const unsigned r00 = p0b | (p0a << 6), r01 = p0c | (p0b << 6), r02 = p0a | (p0c << 6);
            const unsigned r10 = p1b | (p1a << 6), r11 = p1c | (p1b << 6), r12 = p1a | (p1c << 6);
            unsigned left0 = bv0, left1 = bv1;
            while (left0 | left1)
            {
                const bool one = left0 != 0u;
                const int j = __ffs(one ? left0 : left1) - 1;
                if (one)
                    left0 &= left0 - 1u;
                else
                    left1 &= left1 - 1u;
                const unsigned v = __shfl_sync(full, one ? f0.v : f1.v, j);
                const unsigned a = v & 63u, b = (v >> 6) & 63u, c = v >> 12;
                const unsigned x = a | (b << 6), y = b | (c << 6), z = c | (a << 6);
                gone0 |= (r00 == x || r00 == y || r00 == z ? 1u : 0u) | (r01 == x || r01 == y || r01 == z ? 2u : 0u) |
                         (r02 == x || r02 == y || r02 == z ? 4u : 0u);
                const bool me0 = one && j == lane;
                if (vis0 && !me0)
                    twice = twice || e00 == x || e00 == y || e00 == z || e01 == x || e01 == y || e01 == z || e02 == x ||
                            e02 == y || e02 == z;
                if (al1)
                {
                    gone1 |= (r10 == x || r10 == y || r10 == z ? 1u : 0u) | (r11 == x || r11 == y || r11 == z ? 2u : 0u) |
                             (r12 == x || r12 == y || r12 == z ? 4u : 0u);
                    const bool me1 = !one && j == lane;
                    if (vis1 && !me1)
                        twice = twice || e10 == x || e10 == y || e10 == z || e11 == x || e11 == y || e11 == z ||
                                e12 == x || e12 == y || e12 == z;
                }
            }
            if (__any_sync(full, twice))
                return EPA_OVERFLOW;
        }
        const unsigned keep0 = vis0 ? ~gone0 & 7u : 0u, keep1 = vis1 ? ~gone1 & 7u : 0u;
        // the place of a face's edges: the surviving edges of the visible faces before it
        int at0 = 0, at1 = 0, ne = 3;
        if (nvis > 1)
        {
            ne = 0;
            unsigned left0 = bv0, left1 = bv1;
            while (left0 | left1)
            {
                const bool one = left0 != 0u;
                const int j = __ffs(one ? left0 : left1) - 1;
                if (one)
                    left0 &= left0 - 1u;
                else
                    left1 &= left1 - 1u;
                const int info = __shfl_sync(full, one ? (f0.seq << 2) | __popc(keep0) : (f1.seq << 2) | __popc(keep1), j);
                const int cnt = info & 3;
                at0 += (info >> 2) < f0.seq ? cnt : 0;
                at1 += (info >> 2) < f1.seq ? cnt : 0;
                ne += cnt;
            }
        }
        al0 &= ~bv0;
        al1 &= ~bv1;
        const int kept = __popc(al0) + __popc(al1);
        if (ne > kWarpEpaEdges || kept + ne > kWarpEpaFaces || kept + ne == 0)
            return EPA_OVERFLOW;
        if (keep0 & 1u)
            S.edge[at0++] = e00;
        if (keep0 & 2u)
            S.edge[at0++] = e01;
        if (keep0 & 4u)
            S.edge[at0] = e02;
        if (keep1 & 1u)
            S.edge[at1++] = e10;
        if (keep1 & 2u)
            S.edge[at1++] = e11;
        if (keep1 & 4u)
            S.edge[at1] = e12;
        // the new support joins the vertices
        if (lane < 9)
        {
            const float x = lane < 3 ? (lane == 0 ? ns.p.x : (lane == 1 ? ns.p.y : ns.p.z))
                                     : (lane < 6 ? (lane == 3 ? ns.sa.x : (lane == 4 ? ns.sa.y : ns.sa.z))
                                                 : (lane == 6 ? ns.sb.x : (lane == 7 ? ns.sb.y : ns.sb.z)));
            S.v[lane][nv] = x;
        }
        __syncwarp();
        // new faces (S, e.A, e.B) in edge order, into the free places in lane order
        const int free0 = 32 - __popc(al0), r0 = __popc(~al0 & below);
        const bool new0 = !((al0 >> lane) & 1u) && r0 < ne;
        if (new0)
        {
            const unsigned e = S.edge[r0];
            lane_face(f0, ns.p, warp_p(S, e & 63u), warp_p(S, e >> 6), (unsigned)nv | (e << 6), nseq + r0);
        }
        al0 |= __ballot_sync(full, new0);
        if (ne > free0)
        {
            const int r1 = free0 + __popc(~al1 & below);
            const bool new1 = !((al1 >> lane) & 1u) && r1 < ne;
            if (new1)
            {
                const unsigned e = S.edge[r1];
                lane_face(f1, ns.p, warp_p(S, e & 63u), warp_p(S, e >> 6), (unsigned)nv | (e << 6), nseq + r1);
            }
            al1 |= __ballot_sync(full, new1);
        }
        __syncwarp();
        nseq += ne;
        ++nv;
    }
    return EPA_NONE;
}

__device__ __forceinline__ bool same_bits(v3 a, v3 b)
{
    return __float_as_uint(a.x) == __float_as_uint(b.x) && __float_as_uint(a.y) == __float_as_uint(b.y) &&
           __float_as_uint(a.z) == __float_as_uint(b.z);
}

// A simplex vertex of the warp's GJK: the point in registers, its supports in slot `slot` of the
// simplex store.
struct SlotVertex
{
    v3 p;
    int slot;
};

// CheckCollision's GJK loop of one pair by the whole warp, from call `it` with the n points in
// vertices 0 .. n - 1 of S. Returns G_FOUND with the final simplex in vertices 0..3, or G_NOHIT.
//
// A call's outcome depends on the simplex alone (its direction starts at normalize(PB - PA) each
// time), so a run that comes back to an earlier simplex repeats the calls between them until the
// cap and never finds a collision: it ends at once. The lanes hold the simplices of the last 32
// calls. Of the stack workload's misses that take more than eight calls nearly half run to the
// 65-call cap, and three quarters of those repeat themselves, after 17 calls on average.
__device__ __forceinline__ int gjk_warp(const DevWorld &w, WarpEpa &S, const Shape &A, const Shape &B, v3 va, v3 vb, int n,
                                        int it, int lane)
{
    const unsigned full = 0xffffffffu;
    const v3 dir0 = normalize3(B.p - A.p);
    SlotVertex s0 = {warp_p(S, 0), 0}, s1 = {warp_p(S, 1), 1}, s2 = {warp_p(S, 2), 2}, s3 = {warp_p(S, 3), 3};
    SlotVertex h0 = {}, h1 = {}, h2 = {}, h3 = {}; // this lane's earlier simplex
    int hn = 0;
    bool found = false;
    for (; it <= 64; ++it)
    {
        const bool same = hn == n && n > 0 && same_bits(h0.p, s0.p) && (n < 2 || same_bits(h1.p, s1.p)) &&
                          (n < 3 || same_bits(h2.p, s2.p)) && (n < 4 || same_bits(h3.p, s3.p));
        if (__any_sync(full, same))
            break;
        if (lane == (it & 31))
        {
            h0 = s0;
            h1 = s1;
            h2 = s2;
            h3 = s3;
            hn = n;
        }
        v3 dir = dir0;
        if (gjk_direction(s0, s1, s2, s3, n, dir))
        {
            found = true;
            break;
        }
        if (dir_too_short(dir))
            break;
        v3 sa, sb;
        pair_support(w.verts, A, B, va, vb, dir, lane, sa, sb);
        // a slot the simplex does not use takes the new point
        unsigned used = 0u;
        if (n > 0)
            used |= 1u << s0.slot;
        if (n > 1)
            used |= 1u << s1.slot;
        if (n > 2)
            used |= 1u << s2.slot;
        const SlotVertex sv = {sa - sb, __ffs(~used) - 1};
        if (lane < 6)
            S.v[3 + lane][sv.slot] = lane < 3 ? (lane == 0 ? sa.x : (lane == 1 ? sa.y : sa.z))
                                              : (lane == 3 ? sb.x : (lane == 4 ? sb.y : sb.z));
        if (n == 0)
            s0 = sv;
        else if (n == 1)
            s1 = sv;
        else if (n == 2)
            s2 = sv;
        else
            s3 = sv;
        ++n;
        if (!(dot3(dir, sv.p) >= 0.0f))
            break;
    }
    if (!found)
        return G_NOHIT;
    __syncwarp();
    // the simplex in order: lane k moves vertex k's supports from their slot
    const SlotVertex sv = lane == 0 ? s0 : (lane == 1 ? s1 : (lane == 2 ? s2 : s3));
    const v3 sa = warp_sup(S, sv.slot, 0), sb = warp_sup(S, sv.slot, 1);
    __syncwarp();
    if (lane < 4)
    {
        S.v[0][lane] = sv.p.x;
        S.v[1][lane] = sv.p.y;
        S.v[2][lane] = sv.p.z;
        S.v[3][lane] = sa.x;
        S.v[4][lane] = sa.y;
        S.v[5][lane] = sa.z;
        S.v[6][lane] = sb.x;
        S.v[7][lane] = sb.y;
        S.v[8][lane] = sb.z;
    }
    __syncwarp();
    return G_FOUND;
}

} // namespace nans
