// raycast.cu — the particle path of the raycast depth camera on the HashGrid.
//
// Replaces, for particles, SensorRaycast.update(state, include_particles=True)
// (newton/_src/sensors/sensor_raycast.py:185-263, 272-320): the launch of
// sensor_raycast_particles_kernel (newton/_src/geometry/raycast.py:1090-1180)
// with its helpers ray_for_pixel (raycast.py:727-775) and
// ray_intersect_particle_sphere (raycast.py:123-156), and the final
// clamp_no_hits_kernel (sensor_raycast.py:18-23).
//
// Reference semantics: each pixel marches its ray from the camera in steps of
// march_step. At every sample it queries the grid (Warp's query box around
// the sample, radius search_radius) and intersects the ray with the sphere of
// every candidate, keeping the nearest hit; it stops after max_steps samples,
// beyond max_distance, or beyond the nearest hit so far. The depth is the
// minimum over the candidates of the samples taken, which does not depend on
// the order they are tested in.
//
// Three facts make most of the march unnecessary:
// 1. Every hit is at least M, the nearest computed hit over ALL spheres. A
//    ray without any computed hit leaves its pixel as it is, whatever cells
//    its march would visit. M comes from a bounding-box tree over the spheres
//    (k_ray_leaves, k_ray_upper), whose boxes are inflated by a bound on the
//    rounding of the sphere test, so it misses no computed hit.
// 2. Every sample with t <= M is taken (nothing stops the march before). So
//    when the box of such a sample holds the nearest sphere's cell, the depth
//    is M. Otherwise, and if 3 does not apply, the march is run, but only over
//    the samples whose box overlaps (modulo the grid's dims) the cells that can
//    hold a sphere hit before M + window: spheres hit later cannot stop the
//    march inside the window, and those that can are tested at these samples
//    only. A march that leaves the window without a hit is repeated with a
//    wider one, in the end the reference's whole march.
// 3. A ray whose nearest hit is not decided so has its computed hits collected
//    from the tree, up to a distance that grows until the depth is known. Up to
//    kRayList of them, only these spheres' cells matter: march_few passes over
//    the samples far from all of them in strides. (Marching over the window's
//    cells instead, and adding up t sample by sample, the image of the block at
//    640 x 480 took 1.11 ms, and 0.99 with this.)
// The march itself tests each cell once per ray: along every axis both ends
// of the query box are monotone in t, so a cell that an earlier sample tested
// and that this box still holds was in the previous box.
//
// The march alone was bound by instruction issue: most rays miss, and each
// missing ray took every sample up to max_distance through cells that the
// grid's 128 cells per axis alias onto the scene.
//
// fp32, every operation rounded as written (explicit _rn intrinsics, dot
// products ((x + y) + z)), so the depth image matches the CPU restatement
// bit for bit.
#include <algorithm>

#include "nsph_internal.cuh"

namespace nsph {

NSPH_BOUNDS_READER(raycast)
namespace {

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// float -> unsigned, increasing, 0 below every float (the bounds start at 0)
__device__ __forceinline__ unsigned ordered(float f)
{
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float unordered(unsigned u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Radius that bounds the centres of spheres whose COMPUTED test can hit,
// around the ray, at distances up to d from the camera. With u = 2^-24: proj
// is within 3u d of the dot product and its square within 7u d^2, |o|^2 within
// 3u d^2, |o|^2 - r^2 rounds by u d^2, the last difference keeps its sign, and
// the direction's squared length is within 7u of 1: 18u d^2 in all (24u is
// taken). The centre is the rounded difference o itself: the boxes are formed
// from the same differences, and rounding is monotone. The box test's own
// roundings (5u of the distance) lie inside the last factor where the radius is
// the larger part, and between 18u and 24u (1.6e-4 d) where the distance is.
// (1e-43: 71 denormals, for what the products round by below the normal range.)
__device__ __forceinline__ float reach(float r, float d)
{
    return sqrtf(fmaf(1.4306e-6f * d, d, fmaf(r, r, 1e-43f))) * 1.0001f;
}

// Whether sphere q can be hit within max_distance of the camera at all: not
// without a positive, finite radius, nor where the square of the distance
// overflows (the test's discriminant is then no number, or its root infinite).
__device__ __forceinline__ bool in_reach(float4 q, const nsph_raycast_camera& c)
{
    const float ox = q.x - c.position[0], oy = q.y - c.position[1], oz = q.z - c.position[2];
    const float d2 = dot3(ox, oy, oz, ox, oy, oz);
    if (!(q.w > 0.f && isfinite(q.w) && isfinite(d2))) return false;
    return !(sqrtf(d2) * 0.99999f - reach(q.w, sqrtf(d2)) > c.max_distance);
}

// sorted mirror (x, y, z, radius) of the grid's points, and the bounds of the
// spheres in reach: bounds[a] = max of ordered(x_a), bounds[3 + a] = max of
// ordered(-x_a), both 0 at first. (One atomic per block and bound: one per warp
// kept 500,000 spheres' pass waiting on six addresses, 24 us of 26.)
__global__ void __launch_bounds__(256) k_raycast_gather(const int* __restrict__ ids, const float* __restrict__ x,
                                 const float* __restrict__ radius, int n, const nsph_raycast_camera cam,
                                 float4* __restrict__ m, unsigned* __restrict__ bounds)
{
    launch_entry();
    __shared__ unsigned block[6][8];
    const int k = blockIdx.x * 256 + threadIdx.x;
    unsigned b[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    if (k < n) {
        const size_t i = (size_t)ids[k];
        const Row3 xi = load_row(x + 3 * i);
        const float4 q = make_float4(xi.x, xi.y, xi.z, radius[i]);
        m[k] = q;
        if (in_reach(q, cam)) {
            b[0] = ordered(q.x);
            b[1] = ordered(q.y);
            b[2] = ordered(q.z);
            b[3] = ordered(-q.x);
            b[4] = ordered(-q.y);
            b[5] = ordered(-q.z);
        }
    }
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        const unsigned v = __reduce_max_sync(0xffffffffu, b[a]);
        if ((threadIdx.x & 31) == a) block[a][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        unsigned v = 0u;
#pragma unroll
        for (int w = 0; w < 8; ++w) v = max(v, block[threadIdx.x][w]);
        if (v > bounds[threadIdx.x]) atomicMax(bounds + threadIdx.x, v);
    }
}

__device__ __forceinline__ unsigned spread8(unsigned v)  // bits 0..7 to bits 0, 3, .., 21
{
    v = (v | (v << 8)) & 0x00f00fu;
    v = (v | (v << 4)) & 0x0c30c3u;
    return (v | (v << 2)) & 0x249249u;
}

// 24-bit Morton key of each sphere inside the bounds (spheres out of reach
// last), and its position in the sorted mirror
__global__ void k_ray_keys(const float4* __restrict__ m, int n, const nsph_raycast_camera cam,
                           const unsigned* __restrict__ bounds, int* __restrict__ keys, int* __restrict__ vals)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 q = m[k];
    unsigned key = 0xffffffu;
    if (in_reach(q, cam)) {
        const float lo[3] = {-unordered(bounds[3]), -unordered(bounds[4]), -unordered(bounds[5])};
        const float x[3] = {q.x, q.y, q.z};
        float ext = 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) ext = fmaxf(ext, unordered(bounds[a]) - lo[a]);
        const float scale = ext > 0.f ? 255.f / ext : 0.f;
        key = 0u;
#pragma unroll
        for (int a = 0; a < 3; ++a) key |= spread8((unsigned)min(255, max(0, (int)((x[a] - lo[a]) * scale)))) << a;
    }
    keys[k] = (int)key;
    vals[k] = k;
}

// ---- the tree: nodes of eight consecutive children, leaves of eight spheres -----
// A node is two float4: (min of the centres, largest radius), (max of the
// centres, -); an empty one has min > max. Level 0 (the leaves) lies in its
// own array, the levels above it one after another in `upper`.
constexpr int kRayArity = 8;
constexpr int kRayLevels = 12;

struct RayTree {
    float4* leaves;
    float4* upper;
    int levels;                // level levels - 1 holds one node
    int count[kRayLevels];     // nodes per level
    int offset[kRayLevels];    // first node of a level >= 1 in `upper`
    __host__ __device__ float4* node(int level, int i) const
    {
        return level == 0 ? leaves + 2 * (size_t)i : upper + 2 * ((size_t)offset[level] + i);
    }
};

struct RayBox {
    float lo[3], hi[3], r;
};

__device__ __forceinline__ RayBox empty_box()
{
    RayBox b;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        b.lo[a] = INFINITY;
        b.hi[a] = -INFINITY;
    }
    b.r = 0.f;
    return b;
}

// union over the eight lanes of an aligned group, in every lane of it
__device__ __forceinline__ RayBox join8(RayBox b)
{
#pragma unroll
    for (int o = 1; o < kRayArity; o <<= 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            b.lo[a] = fminf(b.lo[a], __shfl_xor_sync(0xffffffffu, b.lo[a], o));
            b.hi[a] = fmaxf(b.hi[a], __shfl_xor_sync(0xffffffffu, b.hi[a], o));
        }
        b.r = fmaxf(b.r, __shfl_xor_sync(0xffffffffu, b.r, o));
    }
    return b;
}

__device__ __forceinline__ void store_box(float4* node, const RayBox& b)
{
    node[0] = make_float4(b.lo[0], b.lo[1], b.lo[2], b.r);
    node[1] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
}

// the spheres in Morton order (radius -1 out of reach) and the leaves
__global__ void __launch_bounds__(256) k_ray_leaves(const float4* __restrict__ m, const int* __restrict__ order,
                                                    int n, const nsph_raycast_camera cam, float4* __restrict__ sorted,
                                                    const __grid_constant__ RayTree tree)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    RayBox b = empty_box();
    if (k < n) {
        float4 q = m[order[k]];
        if (in_reach(q, cam)) {
            b.lo[0] = b.hi[0] = q.x;
            b.lo[1] = b.hi[1] = q.y;
            b.lo[2] = b.hi[2] = q.z;
            b.r = q.w;
        } else {
            q.w = -1.f;
        }
        sorted[k] = q;
    }
    b = join8(b);
    if (k < n && (threadIdx.x & (kRayArity - 1)) == 0) store_box(tree.node(0, k / kRayArity), b);
}

// levels 1 .. levels - 1, each from the one below
__global__ void __launch_bounds__(256) k_ray_upper(const __grid_constant__ RayTree tree, int level)
{
    launch_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // child
    RayBox b = empty_box();
    if (i < tree.count[level - 1]) {
        const float4* c = tree.node(level - 1, i);
        const float4 lo = c[0], hi = c[1];
        b = RayBox{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}, lo.w};
    }
    b = join8(b);
    if (i < tree.count[level - 1] && (threadIdx.x & (kRayArity - 1)) == 0) store_box(tree.node(level, i / kRayArity), b);
}

// the levels from `first` up, in one block (the first has at most 4,096 children)
__global__ void __launch_bounds__(1024) k_ray_top(const __grid_constant__ RayTree tree, int first)
{
    launch_entry();
    for (int level = first; level < tree.levels; ++level) {
        const int children = tree.count[level - 1];
        for (int base = 0; base < children; base += blockDim.x) {
            const int i = base + threadIdx.x;
            RayBox b = empty_box();
            if (i < children) {
                const float4* c = tree.node(level - 1, i);
                const float4 lo = c[0], hi = c[1];
                b = RayBox{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}, lo.w};
            }
            b = join8(b);
            if (i < children && (threadIdx.x & (kRayArity - 1)) == 0) store_box(tree.node(level, i / kRayArity), b);
        }
        __syncthreads();  // the next level reads this one
    }
}

struct Ray {
    float ox, oy, oz, dx, dy, dz;
};

// ray_for_pixel: pixel centre in normalised device coordinates (y up),
// scaled by tan(fov/2) and the aspect ratio, then right*x + up*y + forward
// normalised (the zero vector for a zero length)
__device__ __forceinline__ Ray ray_for_pixel(const nsph_raycast_camera& c, int px, int py)
{
    const float ndc_x =
        __fsub_rn(__fdiv_rn(__fadd_rn(__fmul_rn(2.f, (float)px), 1.f), (float)c.width), 1.f);
    const float ndc_y =
        __fsub_rn(1.f, __fdiv_rn(__fadd_rn(__fmul_rn(2.f, (float)py), 1.f), (float)c.height));
    const float cx = __fmul_rn(__fmul_rn(ndc_x, c.fov_scale), c.aspect_ratio);
    const float cy = __fmul_rn(ndc_y, c.fov_scale);
    float d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        d[k] = __fadd_rn(__fadd_rn(__fmul_rn(c.right[k], cx), __fmul_rn(c.up[k], cy)), c.direction[k]);
    const float l = __fsqrt_rn(dot3(d[0], d[1], d[2], d[0], d[1], d[2]));
#pragma unroll
    for (int k = 0; k < 3; ++k) d[k] = l > 0.f ? __fdiv_rn(d[k], l) : 0.f;
    return Ray{c.position[0], c.position[1], c.position[2], d[0], d[1], d[2]};
}

// ray_intersect_particle_sphere: the nearer non-negative root, else -1
__device__ __forceinline__ float ray_sphere(const Ray& r, float4 s)
{
    const float ox = __fsub_rn(r.ox, s.x), oy = __fsub_rn(r.oy, s.y), oz = __fsub_rn(r.oz, s.z);
    const float proj = dot3(r.dx, r.dy, r.dz, ox, oy, oz);
    const float c = __fsub_rn(dot3(ox, oy, oz, ox, oy, oz), __fmul_rn(s.w, s.w));
    const float disc = __fsub_rn(__fmul_rn(proj, proj), c);
    if (disc < 0.f) return -1.f;
    const float sq = __fsqrt_rn(disc);
    float t = __fsub_rn(-proj, sq);
    if (t < 0.f) t = __fadd_rn(-proj, sq);
    if (t < 0.f) return -1.f;
    return t;
}

// physical coordinate of virtual cell lo + i along one axis (i < dim: the
// query box spans at most dim cells): a 32-bit modulo for the first and an
// increment that wraps once at dim for the next; the general mapping when
// the run starts below the 2^20 origin (clamped cells)
struct AxisWalk {
    int first, dim, lo;
    bool general;
    __device__ __forceinline__ int at(int i) const
    {
        if (general) return phys_axis((long long)lo + i, dim);
        const int v = first + i;  // <= 2 dim - 2
        return v < dim ? v : v - dim;
    }
};

__device__ __forceinline__ AxisWalk axis_walk(int lo, int dim)
{
    AxisWalk a;
    a.dim = dim;
    a.lo = lo;
    a.general = (long long)lo + kOrigin < 0;
    a.first = a.general ? 0 : (int)((unsigned)((long long)lo + kOrigin) % (unsigned)dim);
    return a;
}

// query box of one axis as ints (Warp's bounds fit: start >= INT_MIN, and
// end <= the truncated upper bound <= INT_MAX)
__device__ __forceinline__ void box_axis(float p, float r, float inv, int dim, int& lo, int& hi)
{
    long long a, b;
    query_bounds(p, r, inv, dim, a, b);
    lo = (int)a;
    hi = (int)b;
}

// Cells that can hold a sphere hit before the window's end: a box of virtual
// cells [lo, lo + span] per axis, as physical coordinates. `all`: every cell.
// A sample farther than `half` cells from `centre` along an axis, modulo the
// grid's dims, has a box that does not meet them (two cells of slack for the
// roundings).
struct RayRegion {
    int first[3], span[3];
    float centre[3], half[3];
    bool all;
};

// Samples from the one at p on, `move` cells apart along the axis, that are
// sure to be that far: the distance modulo the dims shrinks by at most `move`
// per sample. So a march passes over the samples that cannot matter in strides.
__device__ __forceinline__ int far_samples(float p, float inv, float centre, float half, float dim, float move)
{
    const float c = p * inv, w = c - centre;
    const float e = fabsf(fmaf(-dim, rintf(w / dim), w)) - half;
    // (a sample whose cells the 2^20 origin may clamp is left to the box)
    return fabsf(c) < 1e6f && e > 0.f ? (int)fminf(e / move, 1e6f) + 1 : 0;
}

// Up to k samples on: ++s and t = t + step, k times, but not beyond the first
// t > lim nor past max_steps. Within a binade the rounded sum grows by the same
// multiple of its last place each time (from the second sum inside the binade
// on, if step lies half way between two), so all additions that stay inside it
// are one exact product.
__device__ __forceinline__ void stride(float& t, int& s, int k, float lim, float step, int max_steps)
{
    k = min(k, max_steps - s);
    while (k > 0) {
        ++s;
        t = __fadd_rn(t, step);
        if (--k == 0 || !(t <= lim)) return;
        const float before = t;
        ++s;
        t = __fadd_rn(t, step);
        if (--k == 0 || !(t <= lim)) return;
        if ((__float_as_uint(before) ^ __float_as_uint(t)) & 0x7f800000u) continue;
        const float grow = __fadd_rn(t, step) - t;
        if (!(grow > 0.f)) {
            s += k;
            return;
        }
        const float top = __uint_as_float((__float_as_uint(t) & 0x7f800000u) + 0x00800000u);
        const int j = min(k - 1, (int)fminf((fminf(top, lim) - t) / grow, 1e9f) - 2);
        if (j > 0) {
            s += j;
            t = fmaf((float)j, grow, t);
            k -= j;
        }
    }
}

// per-sample movement along the axes, in cells, and the grid's dims
struct RayMoves {
    float move[3], dim[3];
    __device__ __forceinline__ RayMoves(const GridDev& g, const Ray& r, float march_step, float max_distance,
                                        int max_steps);
};

__device__ __forceinline__ RayMoves::RayMoves(const GridDev& g, const Ray& r, float march_step, float max_distance,
                                              int max_steps)
{
    // the largest t (2^20 roundings of the sum stay below the factor), and a step with the rounding of t
    const float last = fminf(fminf(max_distance, 1.1f * march_step * (float)max_steps), 1e30f);
    const float step = march_step + 1.2e-7f * last;
    const float d[3] = {r.dx, r.dy, r.dz};
    const int dims[3] = {g.dx, g.dy, g.dz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        move[a] = fabsf(d[a]) * step * g.inv * 1.01f + 1e-3f;
        dim[a] = (float)dims[a];
    }
}

// whether the physical cells of the virtual run [lo, hi] meet those of the region's axis a
__device__ __forceinline__ bool axis_meets(const RayRegion& g, int a, int lo, int hi, int dim)
{
    if ((long long)lo + kOrigin < 0 || g.span[a] + (hi - lo) + 2 > dim) return true;
    const int p = wrap_cell(lo, dim);
    const int d = p >= g.first[a] ? p - g.first[a] : p - g.first[a] + dim;  // from the region's first to lo
    return d <= g.span[a] || dim - d <= hi - lo;
}

// the march over the samples whose box meets the region, testing each cell
// once; `best` as the buffer had it on entry. Returns whether anything was hit.
__device__ __noinline__ bool march(const GridDev& g, const float4* __restrict__ m, const Ray& r, float max_distance,
                                   float search_radius, float march_step, int max_steps, const RayRegion& region,
                                   float stop, float& best)
{
    bool hit = false;
    // previous query box, empty at first (every cell then counts as new)
    int pxl = 0, pxh = -1, pyl = 0, pyh = -1, pzl = 0, pzh = -1;
    const RayMoves mv(g, r, march_step, max_distance, max_steps);
    int s = 0;
    float t = 0.f;
    while (s < max_steps && t <= max_distance && t <= best && t <= stop) {
        if (!region.all) {
            int far = 0;
            const float p[3] = {fmaf(r.dx, t, r.ox), fmaf(r.dy, t, r.oy), fmaf(r.dz, t, r.oz)};
#pragma unroll
            for (int a = 0; a < 3; ++a)
                far = max(far, far_samples(p[a], g.inv, region.centre[a], region.half[a], mv.dim[a], mv.move[a]));
            if (far > 0) {
                stride(t, s, far, fminf(fminf(max_distance, best), stop), march_step, max_steps);
                continue;
            }
        }
        int xl, xh, yl, yh, zl, zh;
        box_axis(__fadd_rn(r.ox, __fmul_rn(r.dx, t)), search_radius, g.inv, g.dx, xl, xh);
        box_axis(__fadd_rn(r.oy, __fmul_rn(r.dy, t)), search_radius, g.inv, g.dy, yl, yh);
        box_axis(__fadd_rn(r.oz, __fmul_rn(r.dz, t)), search_radius, g.inv, g.dz, zl, zh);
        const bool meets = region.all || (axis_meets(region, 0, xl, xh, g.dx) && axis_meets(region, 1, yl, yh, g.dy) &&
                                          axis_meets(region, 2, zl, zh, g.dz));
        if (meets && (xl != pxl || xh != pxh || yl != pyl || yh != pyh || zl != pzl || zh != pzh)) {
            const AxisWalk ax = axis_walk(xl, g.dx), ay = axis_walk(yl, g.dy), az = axis_walk(zl, g.dz);
            const int nx = xh - xl + 1, ny = yh - yl + 1, nz = zh - zl + 1;
            for (int iz = 0; iz < nz; ++iz) {
                const int z = zl + iz;
                const bool zin = z >= pzl && z <= pzh;
                const int cz = az.at(iz);
                for (int iy = 0; iy < ny; ++iy) {
                    const int y = yl + iy;
                    const bool yzin = zin && y >= pyl && y <= pyh;
                    const int rowbase = cz * (g.dx * g.dy) + ay.at(iy) * g.dx;
                    for (int ix = 0; ix < nx; ++ix) {
                        const int x = xl + ix;
                        if (yzin && x >= pxl && x <= pxh) continue;  // tested by an earlier sample
                        const int2 se = __ldg(g.ranges + rowbase + ax.at(ix));
                        for (int k = se.x; k < se.y; ++k) {
                            const float4 q = __ldg(m + k);
                            if (q.w <= 0.f) continue;
                            const float th = ray_sphere(r, q);
                            if (th < 0.f) continue;
                            if (th > max_distance) continue;
                            if (th < best) {
                                best = th;
                                hit = true;
                            }
                        }
                    }
                }
            }
            pxl = xl;
            pxh = xh;
            pyl = yl;
            pyh = yh;
            pzl = zl;
            pzh = zh;
        }
        ++s;
        t = __fadd_rn(t, march_step);
    }
    return hit;
}

// A warp takes four rays, eight lanes to a ray. The walk over the tree is shared
// by the warp, depth-first and nearest child first; a lane tests one of a node's
// eight children, or of a leaf's spheres, for its ray. (With a ray per lane a warp
// went over the children one by one for 32 rays' worth of nodes: the few warps that
// see the scene's edges walked for 1.4 million cycles while the other SMs were
// idle, 9.6 % of the warps active. Depth image of 640 x 480 pixels, 515,100
// spheres: this kernel 930 -> 269 us, now bound by issue at 63 %; the whole
// update 0.99 -> 0.40 ms.)
constexpr int kRayLanes = 8;
constexpr int kRayRays = 32 / kRayLanes;
constexpr int kRayThreads = 128;
constexpr int kRayTile = 4;  // pixels along each side of a block's tile
constexpr int kRayStack = kRayLevels * kRayArity;
constexpr int kRayList = 32;
static_assert(kRayLanes == kRayArity && kRayThreads / 32 * kRayRays == kRayTile * kRayTile, "");

// over the ray's lanes
__device__ __forceinline__ unsigned ray_mask() { return 0xffu << (threadIdx.x & 24); }

// Nearest computed hit: `best` is the bound on entry; returns the sphere's
// Morton position or -1. kList: the Morton positions of all hits up to `best`
// into list (the first kRayList of them), returning their number. For the whole
// warp together; the same result in all lanes of a ray.
template <bool kList>
__device__ __forceinline__ int walk_hits(const RayTree& tree, const float4* __restrict__ sorted, int n, const Ray& r,
                                         bool live, float max_distance, float& best, int2* stack, int* list)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, c = lane & (kRayLanes - 1);
    int who = kList ? 0 : -1;
    if (!live) best = -1.f;
    // a zero component would give 0 x inf on a box face
    auto inverse = [](float d) { return 1.f / (fabsf(d) < 1e-12f ? copysignf(1e-12f, d) : d); };
    const float ix = inverse(r.dx), iy = inverse(r.dy), iz = inverse(r.dz);
    if (lane == 0) stack[0] = make_int2((int)((unsigned)(tree.levels - 1) << 28), 0);
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
        const int2 top = stack[--sp];
        __syncwarp();
        float far = fmaxf(best, __shfl_xor_sync(kAll, best, 8));
        far = fmaxf(far, __shfl_xor_sync(kAll, far, 16));
        if (__int_as_float(top.y) > far) continue;
        const int level = (int)((unsigned)top.x >> 28), child = kRayArity * (top.x & 0x0fffffff) + c;
        if (level == 0) {
            float th = -1.f;
            if (child < n) {
                const float4 q = __ldg(sorted + child);
                if (q.w > 0.f) th = ray_sphere(r, q) + 0.f;  // (no negative zero)
            }
            const bool hit = th >= 0.f && th <= max_distance && (kList ? th <= best : th < best);
            if (kList) {
                const unsigned hits = __ballot_sync(kAll, hit) & ray_mask();
                const int at = who + __popc(hits & ((1u << lane) - 1u));
                if (hit && at < kRayList) list[at] = child;
                who += __popc(hits);
                if (who > kRayList) best = -1.f;  // too many: no more of them
            } else {
                // a float that is not negative orders as its bits do
                unsigned near = hit ? __float_as_uint(th) : 0xffffffffu;
#pragma unroll
                for (int o = 1; o < kRayLanes; o <<= 1) near = min(near, __shfl_xor_sync(kAll, near, o));
                const unsigned first = __ballot_sync(kAll, hit && __float_as_uint(th) == near) & ray_mask();
                if (first) {
                    best = __uint_as_float(near);
                    who = child - c + ((__ffs((int)first) - 1) & (kRayLanes - 1));
                }
            }
            continue;
        }
        float entry = INFINITY;
        if (child < tree.count[level - 1]) {
            const float4* node = tree.node(level - 1, child);
            const float4 lo = __ldg(node), hi = __ldg(node + 1);
            if (lo.x <= hi.x) {
                // the farthest point of the box from the camera bounds the rounding of its spheres' tests
                const float fx = fmaxf(fabsf(lo.x - r.ox), fabsf(hi.x - r.ox));
                const float fy = fmaxf(fabsf(lo.y - r.oy), fabsf(hi.y - r.oy));
                const float fz = fmaxf(fabsf(lo.z - r.oz), fabsf(hi.z - r.oz));
                const float w = reach(lo.w, sqrtf(fx * fx + fy * fy + fz * fz) * 1.0001f);
                // differences first: those of the sphere test, so no centre leaves its box, however coarse the
                // coordinates; the radius then rounds by 1u of the distance, the slab's ends by 2u each
                const float ax = (lo.x - r.ox - w) * ix, bx = (hi.x - r.ox + w) * ix;
                const float ay = (lo.y - r.oy - w) * iy, by = (hi.y - r.oy + w) * iy;
                const float az = (lo.z - r.oz - w) * iz, bz = (hi.z - r.oz + w) * iz;
                const float tn = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
                const float tf = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
                // the ray's nearest point to a centre lies in the inflated
                // box; the hit may lie up to w before it (or, from inside a
                // sphere, after it)
                const float near = fmaxf(tn - w, 0.f);
                if (tn <= tf && tf >= -2.f * w && near <= best) entry = near;
            }
        }
        entry = fminf(entry, __shfl_xor_sync(kAll, entry, 8));
        entry = fminf(entry, __shfl_xor_sync(kAll, entry, 16));
        const bool take = entry < INFINITY;
        const unsigned taken = __ballot_sync(kAll, take) & 0xffu;
        int rank = 0;  // farthest first, so that the nearest is popped next
#pragma unroll
        for (int o = 1; o < kRayLanes; ++o) {
            const float other = __shfl_xor_sync(kAll, entry, o);
            rank += other < INFINITY && (other > entry || (other == entry && (c ^ o) > c));
        }
        if (take && lane < kRayLanes)
            stack[sp + rank] = make_int2((int)(((unsigned)(level - 1) << 28) | (unsigned)child), __float_as_int(entry));
        sp += __popc(taken);
        __syncwarp();
    }
    return who;
}

// The march of a ray whose computed hits up to `stop` are the spheres
// list[0 .. count), all of them: up to there, which of them a taken sample's
// box holds decides the depth, and no other candidate matters. A lane of the
// ray looks after every eighth of them. False when a cell may be clamped.
__device__ __noinline__ bool march_few(const GridDev& g, const float4* __restrict__ sorted, const int* list, int count,
                                       const Ray& r, float max_distance, float search_radius, float march_step,
                                       int max_steps, float stop, float& best)
{
    constexpr int kMine = kRayList / kRayLanes;
    const unsigned lanes = ray_mask();
    // (the box's two cells of slack hold the roundings of coordinates this small)
    bool fits = fmaxf(fmaxf(fabsf(r.ox), fabsf(r.oy)), fabsf(r.oz)) * g.inv < 1e6f;
    float hit[kMine], cell[kMine][3];
    unsigned left = 0;  // spheres no sample has tested
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
        const int at = i * kRayLanes + (threadIdx.x & (kRayLanes - 1));
        hit[i] = cell[i][0] = cell[i][1] = cell[i][2] = 0.f;
        if (at < count) {
            const float4 q = sorted[list[at]];
            left |= 1u << i;
            hit[i] = ray_sphere(r, q) + 0.f;  // (no negative zero)
            const float x[3] = {q.x, q.y, q.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float c = __fmul_rn(x[a], g.inv);
                fits &= fabsf(c) < 1e6f;
                cell[i][a] = (float)trunc_sat(c);
            }
        }
    }
    if (!__all_sync(lanes, fits)) return false;
    const RayMoves mv(g, r, march_step, max_distance, max_steps);
    const float half = 0.5f + search_radius * g.inv + 2.f;
    int s = 0;
    float t = 0.f;
    while (s < max_steps && t <= max_distance && t <= best && t <= stop && __any_sync(lanes, left != 0u)) {
        int far = 1 << 30;
        const float p[3] = {fmaf(r.dx, t, r.ox), fmaf(r.dy, t, r.oy), fmaf(r.dz, t, r.oz)};
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            int f = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a)
                f = max(f, far_samples(p[a], g.inv, cell[i][a] + 0.5f, half, mv.dim[a], mv.move[a]));
            if ((left >> i) & 1u) far = min(far, f);
        }
        far = __reduce_min_sync(lanes, far);
        if (far == 0) {
            int xl, xh, yl, yh, zl, zh;
            box_axis(__fadd_rn(r.ox, __fmul_rn(r.dx, t)), search_radius, g.inv, g.dx, xl, xh);
            box_axis(__fadd_rn(r.oy, __fmul_rn(r.dy, t)), search_radius, g.inv, g.dy, yl, yh);
            box_axis(__fadd_rn(r.oz, __fmul_rn(r.dz, t)), search_radius, g.inv, g.dz, zl, zh);
            float found = INFINITY;
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
                auto holds = [&](int lo, int hi, float c, int dim) {
                    const int pc = wrap_cell((int)c, dim);
                    for (int v = lo; v <= hi; ++v)
                        if (phys_axis(v, dim) == pc) return true;
                    return false;
                };
                if (((left >> i) & 1u) && holds(xl, xh, cell[i][0], g.dx) && holds(yl, yh, cell[i][1], g.dy) &&
                    holds(zl, zh, cell[i][2], g.dz)) {
                    left &= ~(1u << i);
                    found = fminf(found, hit[i]);
                }
            }
            __syncwarp(lanes);
            best = fminf(best, __uint_as_float(__reduce_min_sync(lanes, __float_as_uint(found))));
            far = 1;
        }
        stride(t, s, far, fminf(fminf(max_distance, best), stop), march_step, max_steps);
    }
    return true;
}

// The samples with t <= th are all taken: does the box of one of the last of
// them hold the cell of sphere q, hit at th? A lane of the ray takes a sample.
__device__ __forceinline__ bool held_before(const GridDev& g, const Ray& r, float4 q, float th, float max_distance,
                                            float search_radius, float march_step, int max_steps)
{
    const int cx = phys_axis(trunc_sat(__fmul_rn(q.x, g.inv)), g.dx),
              cy = phys_axis(trunc_sat(__fmul_rn(q.y, g.inv)), g.dy),
              cz = phys_axis(trunc_sat(__fmul_rn(q.z, g.inv)), g.dz);
    auto holds = [](int lo, int hi, int c, int dim) {
        if ((long long)lo + kOrigin < 0) return false;  // clamped cells: left to the march
        int d = c - wrap_cell(lo, dim);
        if (d < 0) d += dim;
        return d <= hi - lo;
    };
    int s = 0;
    float t = 0.f;
    const float lim = th - 6.f * march_step;
    if (t <= lim) stride(t, s, max_steps, lim, march_step, max_steps);
    for (int j = threadIdx.x & (kRayLanes - 1); j > 0; --j) {
        ++s;
        t = __fadd_rn(t, march_step);
    }
    bool held = false;
    if (s < max_steps && t <= max_distance && t <= th) {
        int xl, xh, yl, yh, zl, zh;
        box_axis(__fadd_rn(r.ox, __fmul_rn(r.dx, t)), search_radius, g.inv, g.dx, xl, xh);
        box_axis(__fadd_rn(r.oy, __fmul_rn(r.dy, t)), search_radius, g.inv, g.dy, yl, yh);
        box_axis(__fadd_rn(r.oz, __fmul_rn(r.dz, t)), search_radius, g.inv, g.dz, zl, zh);
        held = holds(xl, xh, cx, g.dx) && holds(yl, yh, cy, g.dy) && holds(zl, zh, cz, g.dz);
    }
    return __any_sync(ray_mask(), held);
}

// The march over the cells that can hold a hit up to nearest + window, with
// wider windows until the depth is known. Returns whether there is one.
__device__ __noinline__ bool march_windows(const GridDev& g, const float4* __restrict__ m, const Ray& r, float rmax,
                                           float nearest, float window, float max_distance, float search_radius,
                                           float march_step, int max_steps, float had, float& best)
{
    for (;; window *= 4.f) {
        // centres of spheres hit in [nearest, until]: within `w` of the ray's
        // points at [nearest - w, until + w]
        const float until = nearest + window;
        const float w = 1.001f * reach(rmax, until + 2.f * rmax) + 1e-5f * until;
        RayRegion region;
        region.all = !(until < max_distance && max_steps < (1 << 24) && window * g.inv < 1e6f);
        const float o[3] = {r.ox, r.oy, r.oz}, d[3] = {r.dx, r.dy, r.dz};
        const int dims[3] = {g.dx, g.dy, g.dz};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float p0 = o[a] + d[a] * (nearest - w), p1 = o[a] + d[a] * (until + w);
            const float lo = (fminf(p0, p1) - w) * g.inv, hi = (fmaxf(p0, p1) + w) * g.inv;
            const bool fits = fabsf(lo) < 1e6f && fabsf(hi) < 1e6f;
            const int vlo = fits ? (int)floorf(lo) - 1 : 0, vhi = fits ? (int)ceilf(hi) + 1 : 0;
            region.span[a] = vhi - vlo;
            region.centre[a] = 0.5f * ((float)vlo + (float)vhi + 1.f);
            region.half[a] = 0.5f * (float)(vhi - vlo + 1) + search_radius * g.inv + 2.f;
            region.first[a] = wrap_cell(vlo, dims[a]);
            region.all |= !fits;
        }
        best = had;
        const bool hit = march(g, m, r, max_distance, search_radius, march_step, max_steps, region,
                               region.all ? INFINITY : until, best);
        // a march that ended on a hit inside the window is the reference's
        if (region.all || (hit && best <= until)) return hit;
    }
}

// a warp takes a square of four pixels, a block one of kRayTile x kRayTile
__global__ void __launch_bounds__(kRayThreads) k_raycast(
    const __grid_constant__ GridDev g, const float4* __restrict__ m, const float4* __restrict__ sorted,
    const __grid_constant__ RayTree tree, int n, const __grid_constant__ nsph_raycast_camera cam, int tiles_x,
    float search_radius, float march_step, int max_steps, float* __restrict__ depth)
{
    launch_entry();
    __shared__ int2 stacks[kRayThreads / 32][kRayStack];
    __shared__ int lists[kRayThreads / 32][kRayRays][kRayList];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ray = lane / kRayLanes;
    const int px = (int)(blockIdx.x % (unsigned)tiles_x) * kRayTile + (warp & 1) * 2 + (ray & 1);
    const int py = (int)(blockIdx.x / (unsigned)tiles_x) * kRayTile + (warp >> 1) * 2 + (ray >> 1);
    const bool live = px < cam.width && py < cam.height;
    const Ray r = ray_for_pixel(cam, min(px, cam.width - 1), min(py, cam.height - 1));
    float* out = depth + (live ? (size_t)py * cam.width + px : 0);
    const float had = live ? (*out < 0.f ? cam.max_distance : *out) : 0.f;
    float best = had;
    const int who = walk_hits<false>(tree, sorted, n, r, live, cam.max_distance, best, stacks[warp], nullptr);
    const float nearest = best;
    float window = 4.f * (search_radius + march_step);
    bool open = live && who >= 0, found = false;  // open: the depth is not known yet
    if (open && held_before(g, r, sorted[who], nearest, cam.max_distance, search_radius, march_step, max_steps)) {
        found = true;
        open = false;
    }
    // then the ray's hits up to a distance, if they are few, else the march
    for (; __any_sync(0xffffffffu, open); window *= 4.f) {
        const bool all = !(nearest + window < fminf(had, cam.max_distance));
        const float until = all ? fminf(had, cam.max_distance) : nearest + window;
        float bound = until;
        const int count = walk_hits<true>(tree, sorted, n, r, open, cam.max_distance, bound, stacks[warp],
                                          lists[warp][ray]);
        __syncwarp();
        if (open) {
            best = had;
            if (count > kRayList || !march_few(g, sorted, lists[warp][ray], count, r, cam.max_distance, search_radius,
                                               march_step, max_steps, all ? INFINITY : until, best)) {
                const float rmax = tree.node(tree.levels - 1, 0)->w;
                found = march_windows(g, m, r, rmax, nearest, window, cam.max_distance, search_radius, march_step,
                                      max_steps, had, best);
                open = false;
            } else if (all || best <= until) {
                found = best < had;
                open = false;
            }
        }
    }
    if (found && (lane & (kRayLanes - 1)) == 0) *out = best;
}

__global__ void k_clamp_no_hits(float* __restrict__ depth, int count, float max_distance)
{
    launch_entry();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count && depth[i] >= max_distance) depth[i] = -1.f;
}

// the tree and the image of one call, in stream order
int raycast_enqueue(nsph_grid* grid, const float* x, const float* radius, int n, const nsph_raycast_camera& c,
                    float search_radius, float march_step, int max_steps, float* depth, cudaStream_t cs)
{
    Grid& g = grid->g;
    float4* m = grid->mirror;
    float4* sorted = grid->mirror + grid->mirror_cap;
    unsigned* bounds = g.bounds;
    NSPH_CUDA_TRY(cudaMemsetAsync(bounds, 0, 6 * sizeof(unsigned), cs));
    const int blocks_n = (n + 255) / 256;
    NSPH_CUDA_TRY(launch_dependent(k_raycast_gather, blocks_n, 256, 0, cs,
                                   g.point_ids, x, radius, n, c, m, bounds));
    NSPH_LAUNCH_CHECK("k_raycast_gather");
    // the tree: Morton order by the grid's sort buffers (free after its
    // build), then the nodes into the same buffers
    NSPH_CUDA_TRY(launch_dependent(k_ray_keys, blocks_n, 256, 0, cs,
                                   m, n, c, bounds, g.keys_a, g.vals_a));
    NSPH_LAUNCH_CHECK("k_ray_keys");
    const int st = grid_sort_keys(g, n, 24, cs);
    if (st != NSPH_OK) return st;
    RayTree tree;
    tree.leaves = reinterpret_cast<float4*>(g.keys_a);
    tree.upper = reinterpret_cast<float4*>(g.vals_a);
    tree.count[0] = (n + kRayArity - 1) / kRayArity;
    tree.offset[0] = 0;
    tree.levels = 1;
    for (int used = 0; tree.count[tree.levels - 1] > 1; ++tree.levels) {
        tree.count[tree.levels] = (tree.count[tree.levels - 1] + kRayArity - 1) / kRayArity;
        tree.offset[tree.levels] = used;
        used += tree.count[tree.levels];
    }
    NSPH_CUDA_TRY(launch_dependent(k_ray_leaves, blocks_n, 256, 0, cs,
                                   m, g.vals_b, n, c, sorted, tree));
    NSPH_LAUNCH_CHECK("k_ray_leaves");
    int level = 1;
    for (; level < tree.levels && tree.count[level - 1] > 4096; ++level) {
        NSPH_CUDA_TRY(launch_dependent(k_ray_upper, (tree.count[level - 1] + 255) / 256, 256, 0, cs,
                                       tree, level));
        NSPH_LAUNCH_CHECK("k_ray_upper");
    }
    if (level < tree.levels) {
        NSPH_CUDA_TRY(launch_dependent(k_ray_top, 1, 1024, 0, cs,
                                       tree, level));
        NSPH_LAUNCH_CHECK("k_ray_top");
    }
    const int tiles_x = (c.width + kRayTile - 1) / kRayTile, tiles_y = (c.height + kRayTile - 1) / kRayTile;
    NSPH_CUDA_TRY(launch_dependent(k_raycast, tiles_x * tiles_y, kRayThreads, 0, cs, g.view(), m, sorted, tree, n, c,
                                   tiles_x, search_radius, march_step, max_steps, depth));
    NSPH_LAUNCH_CHECK("k_raycast");
    return NSPH_OK;
}

}  // namespace
}  // namespace nsph

using namespace nsph;

extern "C" int nsph_raycast_particles(nsph_grid* grid, const float* x, const float* radius, int n,
                                      const nsph_raycast_camera* camera, float search_radius, float march_step,
                                      int max_steps, float* depth, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_raycast_particles");
    if (!grid || !camera) return fail(NSPH_ERR_INVALID_ARG, "null grid or camera");
    const nsph_raycast_camera& c = *camera;
    if (c.width < 0 || c.height < 0) return fail(NSPH_ERR_INVALID_ARG, "negative image size");
    if ((long long)c.width * c.height > 0x7fffffffLL) return fail(NSPH_ERR_INVALID_ARG, "image too large");
    if (n < 0) return fail(NSPH_ERR_INVALID_ARG, "negative particle count");
    if (!(march_step > 0.f)) return fail(NSPH_ERR_INVALID_ARG, "march_step must be positive");
    if (!(search_radius > 0.f) || !isfinite(search_radius))
        return fail(NSPH_ERR_INVALID_ARG, "search_radius must be positive and finite");
    if (max_steps < 0 || max_steps > NSPH_RAYCAST_MAX_STEPS)
        return fail(NSPH_ERR_INVALID_ARG, "max_steps must be in [0, NSPH_RAYCAST_MAX_STEPS]");
    if (c.width == 0 || c.height == 0 || n == 0 || max_steps == 0) return NSPH_OK;
    if (!x || !radius || !depth) return fail(NSPH_ERR_INVALID_ARG, "null array");
    Grid& g = grid->g;
    if (g.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the raycast needs a single-world grid");
    if (!g.built || g.num_points != n)
        return fail(NSPH_ERR_NOT_BUILT, "the grid must be built on the n particle positions first");
    DeviceGuard guard(g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    std::lock_guard<std::mutex> lock(grid->raycast_mutex);
    if (grid->mirror_cap < n) {
        cudaFree(grid->mirror);
        grid->mirror = nullptr;
        grid->mirror_cap = 0;
        NSPH_CUDA_TRY(cudaMalloc(&grid->mirror, sizeof(float4) * 2 * (size_t)g.capacity));
        grid->mirror_cap = g.capacity;
    }
    cudaStream_t cs = (cudaStream_t)stream;
    // (a captured call is ordered by whoever launches its graph)
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    NSPH_CUDA_TRY(cudaStreamIsCapturing(cs, &capture));
    const bool ordered = capture == cudaStreamCaptureStatusNone;
    if (ordered && grid->raycast_done)
        NSPH_CUDA_TRY(cudaStreamWaitEvent(cs, grid->raycast_done, 0));
    else if (ordered)
        NSPH_CUDA_TRY(cudaEventCreateWithFlags(&grid->raycast_done, cudaEventDisableTiming));
    const int st = raycast_enqueue(grid, x, radius, n, c, search_radius, march_step, max_steps, depth, cs);
    // (also behind a call that failed half way)
    if (ordered) NSPH_CUDA_TRY(cudaEventRecord(grid->raycast_done, cs));
    return st;
}

extern "C" int nsph_raycast_clamp_no_hits(float* depth, int count, float max_distance, void* stream)
{
    clear_error();
    if (count < 0) return fail(NSPH_ERR_INVALID_ARG, "negative count");
    if (count == 0) return NSPH_OK;
    if (!depth) return fail(NSPH_ERR_INVALID_ARG, "null depth");
    NSPH_CUDA_TRY(launch_dependent(k_clamp_no_hits, (count + 255) / 256, 256, 0, (cudaStream_t)stream,
                                   depth, count, max_distance));
    NSPH_LAUNCH_CHECK("k_clamp_no_hits");
    return NSPH_OK;
}
