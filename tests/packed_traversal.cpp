// The two forms of the traversal (sol_b200/csrc/kernels/traverse.cuh: exact on
// lower and upper bounds, packed on centres and half sizes with its redo rule)
// restated on the host over core/math.h, on small scenes and rays made to meet
// their edge cases.  Prints the rays traced, those that hit and, for closest and
// any hits, those the two forms answer differently; arguments: family, rays, seed.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "core/math.h"

using namespace sol_b200;

namespace {

struct Box { float lo[3], hi[3], centre[3], half[3]; };
struct Node { Box box[2]; int ref[2]; };   // ref < 0: ~(first << 3 | count - 1)
struct Tri { Vec3 v[3]; };
struct Hit { int tri = -1; float t = 0.0f; bool redo = false; };

std::vector<Tri> tris;
std::vector<Node> nodes;

float round_up(double x) {
    const float f = (float)x;
    return (double)f < x ? std::nextafter(f, INFINITY) : f;
}

Box bounds(int first, int last) {
    Box b;
    for (int k = 0; k < 3; ++k) {
        b.lo[k] = INFINITY;
        b.hi[k] = -INFINITY;
        for (int i = first; i < last; ++i)
            for (const Vec3& v : tris[i].v) {
                b.lo[k] = std::min(b.lo[k], comp(v, k));
                b.hi[k] = std::max(b.hi[k], comp(v, k));
            }
        b.centre[k] = 0.5f * b.lo[k] + 0.5f * b.hi[k];
        const float h = round_up(std::max((double)b.hi[k] - b.centre[k], (double)b.centre[k] - b.lo[k]));
        b.half[k] = round_up((double)h * (1.0 + 16.0 / 16777216.0));
        if (!(std::fabs(b.centre[k]) + b.half[k] <= 1e13f)) { b.centre[k] = 0.0f; b.half[k] = INFINITY; }
    }
    return b;
}

int build(int first, int last) {
    if (last - first <= 3) return ~(first << 3 | (last - first - 1));
    const int me = (int)nodes.size();
    nodes.push_back({});
    const Box b = bounds(first, last);
    int axis = 0;
    for (int k = 1; k < 3; ++k)
        if (b.hi[k] - b.lo[k] > b.hi[axis] - b.lo[axis]) axis = k;
    const int mid = (first + last) / 2;
    auto key = [&](const Tri& t) { return comp(t.v[0], axis) + comp(t.v[1], axis) + comp(t.v[2], axis); };
    std::nth_element(tris.begin() + first, tris.begin() + mid, tris.begin() + last,
                     [&](const Tri& x, const Tri& y) { return key(x) < key(y); });
    Node n;
    n.ref[0] = build(first, mid);
    n.ref[1] = build(mid, last);
    n.box[0] = bounds(first, mid);
    n.box[1] = bounds(mid, last);
    nodes[me] = n;
    return me;
}

/// child_slabs and child_boxes for one box.
template <bool kExact>
bool enters(const Box& b, Vec3 org, Vec3 inv, float tmin, float tmax, float& near) {
    float n = tmin, f = tmax;
    for (int k = 0; k < 3; ++k) {
        const float o = comp(org, k), i = comp(inv, k), a = std::fabs(i);
        if (kExact) {
            const float t0 = (b.lo[k] - o) * i, t1 = (b.hi[k] - o) * i;
            n = std::fmax(n, std::fmin(t0, t1));
            f = std::fmin(f, std::fmax(t0, t1));
        } else {
            const float t = (b.centre[k] - o) * i;
            n = std::fmax(n, std::fma(b.half[k], -a, t));
            f = std::fmin(f, std::fma(b.half[k], a, t));
        }
    }
    near = n;
    return n <= f * kSlabWiden;
}

template <bool kExact, bool kAnyHit>
Hit trace(Vec3 org, Vec3 dir, float tmin, float tmax) {
    Hit h;
    h.t = tmax;
    if (!kExact && !boxes_take(dir)) { h.redo = true; return h; }
    const RayShear rs = make_shear(org, dir);
    const Vec3 inv = kExact ? safe_inverse(dir) : vec3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
    int stack[64], sp = 0, node = 0;
    while (true) {
        if (node >= 0) {
            const Node& q = nodes[node];
            float n0, n1;
            const bool h0 = enters<kExact>(q.box[0], org, inv, tmin, h.t, n0);
            const bool h1 = enters<kExact>(q.box[1], org, inv, tmin, h.t, n1);
            if (h0 && h1) {
                const bool swap = (kExact || !kAnyHit) && n1 < n0;
                stack[sp++] = q.ref[swap ? 0 : 1];
                node = q.ref[swap ? 1 : 0];
                continue;
            }
            if (h0 || h1) { node = q.ref[h0 ? 0 : 1]; continue; }
        } else {
            const int first = ~node >> 3, last = first + (~node & 7) + 1;
            for (int i = first; i < last; ++i) {
                float t, u, v;
                if (!intersect_triangle_upto(rs, tris[i].v[0], tris[i].v[1], tris[i].v[2], tmin, h.t, &t, &u, &v)) continue;
                if (t < h.t) {
                    h.tri = i;
                    h.t = t;
                    h.redo = false;
                    if (kAnyHit) return h;
                } else if (h.tri >= 0 && h.tri != i) {
                    h.redo = !kExact;
                }
            }
        }
        if (sp == 0) return h;
        node = stack[--sp];
    }
}

/// A packed traversal with its redo rule.
template <bool kAnyHit>
Hit resolved(Vec3 org, Vec3 dir, float tmin, float tmax) {
    const Hit h = trace<false, kAnyHit>(org, dir, tmin, tmax);
    return h.redo ? trace<true, false>(org, dir, tmin, tmax) : h;
}

}  // namespace

int main(int argc, char** argv) {
    if (argc != 4) return 2;
    const bool lengths = !std::strcmp(argv[1], "lengths");
    const long count = std::atol(argv[2]);
    std::mt19937_64 gen(std::strtoull(argv[3], nullptr, 10));
    auto real = [&] { return (gen() >> 11) * 0x1p-53; };
    auto pick = [&](int n) { return (int)(gen() % (uint64_t)n); };
    auto component = [](Vec3& v, int k) -> float& { return k == 0 ? v.x : k == 1 ? v.y : v.z; };
    long rays = 0, hits = 0, closest = 0, any = 0;
    for (long scene = 0; scene < (count + 1999) / 2000; ++scene) {
        auto coord = [&] { return (float)(8.0 * real() - 4.0); };
        tris.clear();
        nodes.clear();
        for (int i = 0, n = 4 + pick(60); i < n; ++i) {
            Tri t;
            for (Vec3& v : t.v) v = vec3(coord(), coord(), coord());
            tris.push_back(t);
        }
        build(0, (int)tris.size());
        for (int r = 0; r < 2000; ++r) {
            const Tri& q = tris[pick((int)tris.size())];
            double a = real(), b = real();
            if (a + b > 1.0) { a = 1.0 - a; b = 1.0 - b; }
            const Vec3 at = q.v[0] + (q.v[1] - q.v[0]) * (float)a + (q.v[2] - q.v[0]) * (float)b;
            Vec3 dir = vec3((float)(2.0 * real() - 1.0), (float)(2.0 * real() - 1.0), (float)(2.0 * real() - 1.0));
            float length = 1.0f;
            if (lengths) {
                if (pick(3) == 0) component(dir, pick(3)) *= std::ldexp(1.0f, -pick(60));
                if (pick(6) == 0) component(dir, pick(3)) *= std::ldexp(1.0f, -pick(60));
                length = std::ldexp(1.0f, pick(180) - 100);
            }
            const float dist = (float)std::exp(4.0 * real() - 2.0);
            const Vec3 org = at - dir * dist;
            dir = dir * length;
            const float tmin = pick(2) ? 0.0f : 1e-4f / length;
            const float tmax = pick(4) ? kFloatMax : (float)(2.0 * real()) * dist / length;
            const Hit e = trace<true, false>(org, dir, tmin, tmax), p = resolved<false>(org, dir, tmin, tmax);
            ++rays;
            hits += e.tri >= 0;
            closest += p.tri != e.tri || (e.tri >= 0 && p.t != e.t);
            any += (resolved<true>(org, dir, tmin, tmax).tri >= 0) != (trace<true, true>(org, dir, tmin, tmax).tri >= 0);
        }
    }
    std::printf("%ld %ld %ld %ld\n", rays, hits, closest, any);
    return 0;
}
