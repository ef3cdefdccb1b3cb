// contact.cu — particle-particle contact on the HashGrid: the other
// consumers of the grid in the reference, rebuilt on this library's grid.
//
//   nsph_particle_contact_forces   eval_particle_contact + particle_force
//       (newton/_src/solvers/semi_implicit/kernels_contact.py:11-84, launched
//       by eval_particle_contact_forces, :559-579): spring-damper normal
//       force and Coulomb friction, written to f[i].
//   nsph_particle_contact_deltas   solve_particle_particle_contacts
//       (newton/_src/solvers/xpbd/kernels.py:225-289, launched at
//       newton/_src/solvers/xpbd/solver_xpbd.py:420-440): XPBD position
//       corrections, added to deltas[i].
//
// One thread per grid point, taken in sorted order (the reference's
// hash_grid_point_id(grid, tid)); each particle gathers over the candidates
// of hash_grid_query(grid, x_i, r_i + max_radius + cohesion) in Warp's
// iteration order. A first kernel copies the particles into sorted float4
// mirrors held by the grid object, m0 = (x, r) and m1 = (v, inverse mass),
// so that the candidates of a cell run are read contiguously; an inactive
// particle's radius slot holds -inf (radii of active particles are
// finite). Every fp32 operation is an explicit round-to-nearest
// intrinsic in the order the reference's expressions are written (dot
// products ((x + y) + z), no contraction), so the CPU restatement reproduces
// the results bit for bit.
#include "nsph_internal.cuh"

namespace nsph {

NSPH_BOUNDS_READER(contact)
namespace {

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// particle_force (kernels_contact.py:11-32): normal force c k_n + min(v.n, 0) k_d
// along -n, Coulomb friction min(|vt| k_f, mu |fn|) along -vt/|vt|
__device__ __forceinline__ void particle_force(float nx, float ny, float nz, float vx, float vy, float vz, float c,
                                               const nsph_contact_params& p, float& fx, float& fy, float& fz)
{
    const float vn = dot3(nx, ny, nz, vx, vy, vz);
    const float jn = __fmul_rn(c, p.k_contact);
    const float jd = __fmul_rn(fminf(vn, 0.f), p.k_damp);
    const float fn = __fadd_rn(jn, jd);
    float tx = __fsub_rn(vx, __fmul_rn(nx, vn));
    float ty = __fsub_rn(vy, __fmul_rn(ny, vn));
    float tz = __fsub_rn(vz, __fmul_rn(nz, vn));
    const float vs = __fsqrt_rn(dot3(tx, ty, tz, tx, ty, tz));
    if (vs > 0.f) {
        tx = __fdiv_rn(tx, vs);
        ty = __fdiv_rn(ty, vs);
        tz = __fdiv_rn(tz, vs);
    }
    const float ft = fminf(__fmul_rn(vs, p.k_friction), __fmul_rn(p.k_mu, fabsf(fn)));
    fx = __fsub_rn(__fmul_rn(-nx, fn), __fmul_rn(tx, ft));
    fy = __fsub_rn(__fmul_rn(-ny, fn), __fmul_rn(ty, ft));
    fz = __fsub_rn(__fmul_rn(-nz, fn), __fmul_rn(tz, ft));
}

__device__ __forceinline__ bool mirror_active(float4 m0) { return m0.w != -INFINITY; }

// sorted mirrors: m0[k] = (x, r or -inf if inactive), m1[k] = (v, inverse mass or 0)
__global__ void k_contact_gather(const int* __restrict__ ids, int n, const float* __restrict__ x,
                                 const float* __restrict__ v, const float* __restrict__ radius,
                                 const int* __restrict__ flags, const float* __restrict__ inv_mass,
                                 float4* __restrict__ m0, float4* __restrict__ m1)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const size_t i = (size_t)ids[k];
    const bool active = (flags[i] & NSPH_PARTICLE_ACTIVE) != 0;
    const Row3 xi = load_row(x + 3 * i), vi = load_row(v + 3 * i);
    m0[k] = make_float4(xi.x, xi.y, xi.z, active ? radius[i] : -INFINITY);
    m1[k] = make_float4(vi.x, vi.y, vi.z, inv_mass ? inv_mass[i] : 0.f);
}

// ---- candidates in two phases ----------------------------------------------------
// A particle touches a handful of its candidates, but the contact terms (a
// square root and several exactly rounded divisions) are ten times the cost
// of a distance. Evaluated inside the candidate loop, a warp runs them at
// every candidate slot at which any of its 32 particles has a contact, which
// is nearly all of them. So the candidates are first tested with a bound on
// the squared distance, the ones that pass wait in shared memory, and each
// thread then walks its own in order and applies the definition's test.
// kContactSlots waiting candidates per thread; a particle with more (dense
// piles) evaluates its candidates where it finds them.
constexpr int kContactThreads = 128;
constexpr int kContactSlots = 24;
// resident blocks per SM: 48 registers instead of 64 (56 for the XPBD pass), some
// 90 bytes of spills outside the candidate loop. Contact step of 1M particles
// 232 -> 219 us, XPBD step of 262k 286 -> 281; 9 blocks 227 and 280, 12 blocks
// (40 registers) 229 and 298.
constexpr int kContactBlocks = 10;

// Bound of the contact test: err <= c implies fl(d) <= reach, with err =
// fl(fl(d - r_i) - r_j) three roundings of quantities no larger than d + r_i
// + r_j + |c|; reach() adds 2^-20 (16 roundings) of each to r_i + r_j + c.
struct ContactBound {
    float base;
    __device__ __forceinline__ ContactBound(float ri, float cohesion)
        : base((ri + cohesion) + 9.5367432e-7f * (fabsf(ri) + 2.f * fabsf(cohesion)))
    {
    }
    // r2: the squared distance, dot3 of the differences. NaN distances (and
    // inactive candidates, whose radius slot is -inf) do not pass.
    __device__ __forceinline__ bool may_touch(float r2, float rj) const
    {
        const float s = fmaf(fabsf(rj), 1.9073486e-6f, base + rj);
        return s >= 0.f && r2 <= s * s * 1.000004f;
    }
};

// calls contact(k, b) for the candidates k (mirror b) of particle kk that may
// touch it, in query order, itself excluded
template <class F>
__device__ __forceinline__ void for_each_near(const GridDev& g, const float4* __restrict__ m0, int kk, float4 a,
                                              float query_radius, float cohesion, F&& contact)
{
    __shared__ int waiting[kContactSlots][kContactThreads];
    int* slot = &waiting[0][threadIdx.x];
    const ContactBound bound(a.w, cohesion);
    int cnt = 0;
    auto passes = [&](int k, float4 b) {
        const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
        return bound.may_touch(dot3(dx, dy, dz, dx, dy, dz), b.w) && k != kk;
    };
    auto test = [&](int k, float4 b) {
        slot[min(cnt, kContactSlots - 1) * kContactThreads] = k;
        cnt += passes(k, b);
    };
    // A box of at most 3 x 3 cells per plane (a cell width that covers the
    // query radius) whose rows do not wrap in x: the plane's nine ranges are
    // loaded together and its rows' runs walked as one sequence, the next
    // candidate's load ahead of each test. Walking the cells one after
    // another made the pass a chain of 27 dependent loads.
    int xl, xh, yl, yh, zl, zh;
    bool clamped = false;
    box_axis_regular(a.x, query_radius, g.inv, g.dx, xl, xh, clamped);
    box_axis_regular(a.y, query_radius, g.inv, g.dy, yl, yh, clamped);
    box_axis_regular(a.z, query_radius, g.inv, g.dz, zl, zh, clamped);
    const int nx = xh - xl + 1, ny = yh - yl + 1, nz = zh - zl + 1;
    const int cx = clamped ? 0 : wrap_cell(xl, g.dx);
    if (!clamped && nx <= 3 && ny <= 3 && cx + nx <= g.dx) {
        int cy[3];
        cy[0] = wrap_cell(yl, g.dy);
        cy[1] = cy[0] + 1 == g.dy ? 0 : cy[0] + 1;
        cy[2] = cy[1] + 1 == g.dy ? 0 : cy[1] + 1;
        int cz = wrap_cell(zl, g.dz);
        for (int iz = 0; iz < nz; ++iz) {
            int2 se[3][3];
#pragma unroll
            for (int iy = 0; iy < 3; ++iy) {
                const int2* row = g.ranges + (cz * g.dy + cy[iy]) * g.dx + cx;
#pragma unroll
                for (int ix = 0; ix < 3; ++ix) se[iy][ix] = iy < ny && ix < nx ? __ldg(row + ix) : make_int2(0, 0);
            }
            // candidate t of the plane is at t + off[row]
            int off[3], upto[3], total = 0;
#pragma unroll
            for (int iy = 0; iy < 3; ++iy) {
                int lo = 0x7fffffff, hi = 0;
#pragma unroll
                for (int ix = 0; ix < 3; ++ix) {
                    if (se[iy][ix].y > se[iy][ix].x && in_bounds(se[iy][ix].x >= 0 && se[iy][ix].y <= g.n)) {
                        lo = min(lo, se[iy][ix].x);
                        hi = max(hi, se[iy][ix].y);
                    }
                }
                off[iy] = lo - total;
                total += max(hi - lo, 0);
                upto[iy] = total;
            }
            auto at = [&](int t) { return t + (t < upto[0] ? off[0] : (t < upto[1] ? off[1] : off[2])); };
            if (total > 0) {
                int k = at(0);
                float4 b = __ldg(m0 + k);
                for (int t = 1; t < total; ++t) {
                    const int kn = at(t);
                    const float4 bn = __ldg(m0 + kn);
                    test(k, b);
                    k = kn;
                    b = bn;
                }
                test(k, b);
            }
            cz = cz + 1 == g.dz ? 0 : cz + 1;
        }
    } else {
        for_each_run(g, a.x, a.y, a.z, query_radius, [&](int lo, int hi) {
            for (int k = lo; k < hi; ++k) test(k, __ldg(m0 + k));
        });
    }
    const bool few = cnt < kContactSlots;
    if (few) {
        for (int t = 0; t < cnt; ++t) {
            const int k = slot[t * kContactThreads];
            contact(k, __ldg(m0 + k));
        }
    } else {
        for_each_run(g, a.x, a.y, a.z, query_radius, [&](int lo, int hi) {
            for (int k = lo; k < hi; ++k) {
                const float4 b = __ldg(m0 + k);
                if (passes(k, b)) contact(k, b);
            }
        });
    }
}

__global__ void __launch_bounds__(kContactThreads, kContactBlocks) k_contact_forces(GridDev g, int n, const float4* __restrict__ m0,
                                                                    const float4* __restrict__ m1,
                                                                    const nsph_contact_params p,
                                                                    float* __restrict__ f_out)
{
    launch_entry();
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= n) return;
    const float4 a = m0[kk];
    if (!mirror_active(a)) return;
    const float4 va = m1[kk];
    const float ri = a.w;
    const float qr = __fadd_rn(__fadd_rn(ri, p.max_radius), p.k_cohesion);
    float fx = 0.f, fy = 0.f, fz = 0.f;
    for_each_near(g, m0, kk, a, qr, p.k_cohesion, [&](int k, float4 b) {
        float nx = __fsub_rn(a.x, b.x);
        float ny = __fsub_rn(a.y, b.y);
        float nz = __fsub_rn(a.z, b.z);
        const float d = __fsqrt_rn(dot3(nx, ny, nz, nx, ny, nz));
        const float err = __fsub_rn(__fsub_rn(d, ri), b.w);
        if (err <= p.k_cohesion) {
            const float4 vb = __ldg(m1 + k);
            nx = __fdiv_rn(nx, d);
            ny = __fdiv_rn(ny, d);
            nz = __fdiv_rn(nz, d);
            float cx, cy, cz;
            particle_force(nx, ny, nz, __fsub_rn(va.x, vb.x), __fsub_rn(va.y, vb.y), __fsub_rn(va.z, vb.z), err, p,
                           cx, cy, cz);
            fx = __fadd_rn(fx, cx);
            fy = __fadd_rn(fy, cy);
            fz = __fadd_rn(fz, cz);
        }
    });
    const size_t i = (size_t)g.ids[kk];
    store_row(f_out + 3 * i, fx, fy, fz);
}

// the correction of solve_particle_particle_contacts (xpbd/kernels.py:225-289)
// of particle kk (mirrors a, va), before its factors w1 and relaxation
__device__ __forceinline__ void contact_delta(const GridDev& g, const float4* __restrict__ m0,
                                              const float4* __restrict__ m1, int kk, float4 a, float4 va, float k_mu,
                                              float k_cohesion, float max_radius, float dt, float& dx, float& dy,
                                              float& dz)
{
    const float ri = a.w;
    const float w1 = va.w;
    const float qr = __fadd_rn(__fadd_rn(ri, max_radius), k_cohesion);
    dx = dy = dz = 0.f;
    for_each_near(g, m0, kk, a, qr, k_cohesion, [&](int k, float4 b) {
        float nx = __fsub_rn(a.x, b.x);
        float ny = __fsub_rn(a.y, b.y);
        float nz = __fsub_rn(a.z, b.z);
        const float d = __fsqrt_rn(dot3(nx, ny, nz, nx, ny, nz));
        const float err = __fsub_rn(__fsub_rn(d, ri), b.w);
        const float4 vb = __ldg(m1 + k);
        const float denom = __fadd_rn(w1, vb.w);
        if (err <= k_cohesion && denom > 0.f) {
            nx = __fdiv_rn(nx, d);
            ny = __fdiv_rn(ny, d);
            nz = __fdiv_rn(nz, d);
            const float rx = __fsub_rn(va.x, vb.x);
            const float ry = __fsub_rn(va.y, vb.y);
            const float rz = __fsub_rn(va.z, vb.z);
            // normal
            const float lambda_n = err;
            const float dnx = __fmul_rn(nx, lambda_n), dny = __fmul_rn(ny, lambda_n), dnz = __fmul_rn(nz, lambda_n);
            // friction
            const float vn = dot3(nx, ny, nz, rx, ry, rz);
            float tx = __fsub_rn(rx, __fmul_rn(nx, vn));
            float ty = __fsub_rn(ry, __fmul_rn(ny, vn));
            float tz = __fsub_rn(rz, __fmul_rn(nz, vn));
            const float lt = __fsqrt_rn(dot3(tx, ty, tz, tx, ty, tz));
            const float lambda_f = fmaxf(__fmul_rn(k_mu, lambda_n), __fmul_rn(-lt, dt));
            if (lt > 0.f) {  // normalize(vt); the zero vector stays zero
                tx = __fdiv_rn(tx, lt);
                ty = __fdiv_rn(ty, lt);
                tz = __fdiv_rn(tz, lt);
            } else {
                tx = ty = tz = 0.f;
            }
            dx = __fadd_rn(dx, __fdiv_rn(__fsub_rn(__fmul_rn(tx, lambda_f), dnx), denom));
            dy = __fadd_rn(dy, __fdiv_rn(__fsub_rn(__fmul_rn(ty, lambda_f), dny), denom));
            dz = __fadd_rn(dz, __fdiv_rn(__fsub_rn(__fmul_rn(tz, lambda_f), dnz), denom));
        }
    });
}

// deltas[i] += delta * w1 * relaxation (one writer per particle: no atomics)
__global__ void __launch_bounds__(kContactThreads, kContactBlocks) k_contact_deltas(GridDev g, int n, const float4* __restrict__ m0,
                                                                    const float4* __restrict__ m1, float k_mu,
                                                                    float k_cohesion, float max_radius, float dt,
                                                                    float relaxation, float* __restrict__ deltas)
{
    launch_entry();
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= n) return;
    const float4 a = m0[kk];
    if (!mirror_active(a)) return;
    const float4 va = m1[kk];
    const float w1 = va.w;
    float dx, dy, dz;
    contact_delta(g, m0, m1, kk, a, va, k_mu, k_cohesion, max_radius, dt, dx, dy, dz);
    const size_t i = (size_t)g.ids[kk];
    deltas[3 * i] = __fadd_rn(deltas[3 * i], __fmul_rn(__fmul_rn(dx, w1), relaxation));
    deltas[3 * i + 1] = __fadd_rn(deltas[3 * i + 1], __fmul_rn(__fmul_rn(dy, w1), relaxation));
    deltas[3 * i + 2] = __fadd_rn(deltas[3 * i + 2], __fmul_rn(__fmul_rn(dz, w1), relaxation));
}

// ---- one XPBD iteration in one pass ----------------------------------------------
// The contact correction and apply_particle_deltas of the same particle, from
// the sorted mirrors of this iterate to the arrays and the mirrors of the next
// (the other pair): the iteration's zeroing, its gather of new mirrors and the
// round trip of the deltas through memory fall away. Each particle reads other
// particles only through the mirrors of this iterate.
struct XpbdPass {
    const float4* m0;  // this iterate: (x, r or -inf), (v, inverse mass)
    const float4* m1;
    float4* n0;        // the next one
    float4* n1;
    const float4* x0;  // sorted positions at the step's start
    float* x_out;
    float* v_out;
    float k_mu, k_cohesion, max_radius, dt, relaxation, v_max;
};

__global__ void k_xpbd_gather(const int* __restrict__ ids, int n, const float* __restrict__ x,
                              const float* __restrict__ v, const float* __restrict__ radius,
                              const int* __restrict__ flags, const float* __restrict__ inv_mass,
                              const float* __restrict__ x_orig, float4* __restrict__ m0, float4* __restrict__ m1,
                              float4* __restrict__ x0)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const size_t i = (size_t)ids[k];
    const bool active = (flags[i] & NSPH_PARTICLE_ACTIVE) != 0;
    const Row3 xi = load_row(x + 3 * i), vi = load_row(v + 3 * i), oi = load_row(x_orig + 3 * i);
    m0[k] = make_float4(xi.x, xi.y, xi.z, active ? radius[i] : -INFINITY);
    m1[k] = make_float4(vi.x, vi.y, vi.z, inv_mass[i]);
    x0[k] = make_float4(oi.x, oi.y, oi.z, 0.f);
}

__global__ void __launch_bounds__(kContactThreads, kContactBlocks) k_xpbd_pass(GridDev g, int n, const XpbdPass p,
                                                               const float* __restrict__ shape_deltas)
{
    launch_entry();
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= n) return;
    const float4 a = p.m0[kk];
    const float4 va = p.m1[kk];
    if (!mirror_active(a)) {
        p.n0[kk] = a;
        p.n1[kk] = va;
        return;
    }
    const float w1 = va.w;
    float dx, dy, dz;
    contact_delta(g, p.m0, p.m1, kk, a, va, p.k_mu, p.k_cohesion, p.max_radius, p.dt, dx, dy, dz);
    const size_t i = (size_t)__ldg(g.ids + kk);
    const float4 x0 = __ldg(p.x0 + kk);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    if (shape_deltas) {
        sx = __ldg(shape_deltas + 3 * i);
        sy = __ldg(shape_deltas + 3 * i + 1);
        sz = __ldg(shape_deltas + 3 * i + 2);
    }
    // x = x_pred + delta, v = (x - x0)/dt clamped to v_max
    const float x = __fadd_rn(a.x, __fadd_rn(sx, __fmul_rn(__fmul_rn(dx, w1), p.relaxation)));
    const float y = __fadd_rn(a.y, __fadd_rn(sy, __fmul_rn(__fmul_rn(dy, w1), p.relaxation)));
    const float z = __fadd_rn(a.z, __fadd_rn(sz, __fmul_rn(__fmul_rn(dz, w1), p.relaxation)));
    float vx = __fdiv_rn(__fsub_rn(x, x0.x), p.dt), vy = __fdiv_rn(__fsub_rn(y, x0.y), p.dt),
          vz = __fdiv_rn(__fsub_rn(z, x0.z), p.dt);
    const float m = __fsqrt_rn(dot3(vx, vy, vz, vx, vy, vz));
    if (m > p.v_max) {
        const float s = __fdiv_rn(p.v_max, m);
        vx = __fmul_rn(vx, s);
        vy = __fmul_rn(vy, s);
        vz = __fmul_rn(vz, s);
    }
    p.n0[kk] = make_float4(x, y, z, a.w);
    p.n1[kk] = make_float4(vx, vy, vz, w1);
    store_row(p.x_out + 3 * i, x, y, z);
    store_row(p.v_out + 3 * i, vx, vy, vz);
}

int check_grid(const nsph_grid* grid, int n)
{
    if (!grid) return fail(NSPH_ERR_INVALID_ARG, "null grid");
    if (grid->g.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "contacts need a single-world grid");
    if (!grid->g.built) return fail(NSPH_ERR_NOT_BUILT, "the grid has not been built");
    if (n < 0) return fail(NSPH_ERR_INVALID_ARG, "negative particle count");
    if (n != grid->g.num_points)
        return fail(NSPH_ERR_INVALID_ARG, "particle count differs from the points of the grid's last build");
    if (n > grid->mirror_cap) return fail(NSPH_ERR_CAPACITY, "grid not reserved through nsph_grid_reserve");
    return NSPH_OK;
}

}  // namespace
}  // namespace nsph

using namespace nsph;

extern "C" int nsph_particle_contact_forces(const nsph_grid* grid, const nsph_contact_params* params, int n,
                                            const float* x, const float* v, const float* radius, const int* flags,
                                            float* f_out, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_particle_contact_forces");
    int st = check_grid(grid, n);
    if (st != NSPH_OK) return st;
    if (!params) return fail(NSPH_ERR_INVALID_ARG, "null params");
    if (n == 0) return NSPH_OK;
    if (!x || !v || !radius || !flags || !f_out) return fail(NSPH_ERR_INVALID_ARG, "null array");
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    float4* m0 = grid->mirror;
    float4* m1 = grid->mirror + grid->mirror_cap;
    NSPH_CUDA_TRY(launch_dependent(k_contact_gather, (n + 255) / 256, 256, 0, cs,
                                   grid->g.point_ids, n, x, v, radius, flags, nullptr, m0, m1));
    NSPH_LAUNCH_CHECK("k_contact_gather");
    NSPH_CUDA_TRY(launch_dependent(k_contact_forces, (n + kContactThreads - 1) / kContactThreads, kContactThreads, 0, cs,
                                   grid->g.view(), n, m0, m1, *params, f_out));
    NSPH_LAUNCH_CHECK("k_contact_forces");
    return NSPH_OK;
}

extern "C" int nsph_particle_contact_deltas(const nsph_grid* grid, int n, const float* x, const float* v,
                                            const float* inv_mass, const float* radius, const int* flags, float k_mu,
                                            float k_cohesion, float max_radius, float dt, float relaxation,
                                            float* deltas, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_particle_contact_deltas");
    int st = check_grid(grid, n);
    if (st != NSPH_OK) return st;
    if (n == 0) return NSPH_OK;
    if (!x || !v || !inv_mass || !radius || !flags || !deltas) return fail(NSPH_ERR_INVALID_ARG, "null array");
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    float4* m0 = grid->mirror;
    float4* m1 = grid->mirror + grid->mirror_cap;
    NSPH_CUDA_TRY(launch_dependent(k_contact_gather, (n + 255) / 256, 256, 0, cs,
                                   grid->g.point_ids, n, x, v, radius, flags, inv_mass, m0, m1));
    NSPH_LAUNCH_CHECK("k_contact_gather");
    NSPH_CUDA_TRY(launch_dependent(k_contact_deltas, (n + kContactThreads - 1) / kContactThreads, kContactThreads, 0, cs,
                                   grid->g.view(), n, m0, m1, k_mu, k_cohesion, max_radius, dt, relaxation, deltas));
    NSPH_LAUNCH_CHECK("k_contact_deltas");
    return NSPH_OK;
}

extern "C" int nsph_xpbd_solve(const nsph_grid* grid, int n, int iterations, const float* x_orig, float* x_a, float* v_a,
                               float* x_b, float* v_b, const float* inv_mass, const float* radius, const int* flags,
                               const nsph_shape* shapes, int shape_count, const nsph_soft_contacts* contacts,
                               const nsph_soft_contact_params* soft, float k_mu, float k_cohesion, float max_radius,
                               float dt, float relaxation, float v_max, float* deltas, float* scratch, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_xpbd_solve");
    int st = check_grid(grid, n);
    if (st != NSPH_OK) return st;
    if (iterations < 0) return fail(NSPH_ERR_INVALID_ARG, "negative iteration count");
    if (n == 0 || iterations == 0) return NSPH_OK;
    if (!x_orig || !x_a || !v_a || !x_b || !v_b || !inv_mass || !radius || !flags || !scratch)
        return fail(NSPH_ERR_INVALID_ARG, "null array");
    if (x_a == x_b || v_a == v_b) return fail(NSPH_ERR_INVALID_ARG, "the two iterates share memory");
    const bool with_shapes = contacts && contacts->max > 0 && shape_count > 0;
    if (with_shapes && (!soft || !deltas)) return fail(NSPH_ERR_INVALID_ARG, "shape contacts need soft and deltas");
    DeviceGuard guard(grid->g.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    float4* m0[2] = {grid->mirror, reinterpret_cast<float4*>(scratch)};
    float4* m1[2] = {grid->mirror + grid->mirror_cap, m0[1] + n};
    float4* x0 = m0[1] + 2 * (size_t)n;
    NSPH_CUDA_TRY(launch_dependent(k_xpbd_gather, (n + 255) / 256, 256, 0, cs,
                                   grid->g.point_ids, n, x_a, v_a, radius, flags, inv_mass, x_orig, m0[0], m1[0], x0));
    NSPH_LAUNCH_CHECK("k_xpbd_gather");
    for (int t = 0; t < iterations; ++t) {
        const int from = t & 1, to = from ^ 1;
        if (with_shapes) {
            NSPH_CUDA_TRY(cudaMemsetAsync(deltas, 0, sizeof(float) * 3 * (size_t)n, cs));
            st = nsph_particle_shape_contact_deltas(shapes, shape_count, contacts, soft, from ? x_b : x_a,
                                                    from ? v_b : v_a, inv_mass, radius, flags, deltas, stream);
            if (st != NSPH_OK) return st;
        }
        const XpbdPass p{m0[from], m1[from], m0[to], m1[to], x0,
                         from ? x_a : x_b, from ? v_a : v_b, k_mu, k_cohesion, max_radius, dt, relaxation, v_max};
        NSPH_CUDA_TRY(launch_dependent(k_xpbd_pass, (n + kContactThreads - 1) / kContactThreads, kContactThreads, 0, cs,
                                       grid->g.view(), n, p,
                                       with_shapes ? deltas : nullptr));
        NSPH_LAUNCH_CHECK("k_xpbd_pass");
    }
    return NSPH_OK;
}
