// sph.cu — the WCSPH step: grid build on x_n, density/EOS pass, then the
// pressure + XSPH + integrate pass that writes x_{n+1}, v_{n+1}.
//
// The reference has no SPH solver (its particle hot path is the HashGrid
// gather of newton/_src/solvers/semi_implicit/kernels_contact.py:35-84 plus
// integrate_particles, newton/_src/solvers/solver.py:10-47); the step keeps
// that structure and replaces the contact law with published WCSPH math:
//   W      cubic spline with support h (Monaghan 1992), sigma = 8/(pi h^3)
//   rho_i  = sum_j m_j W_ij (self included)
//   p_i    = B((rho_i/rho0)^gamma - 1) clamped at 0 (Tait EOS)
//   a_i    = -sum_{j!=i} m_j (p_i/rho_i^2 + p_j/rho_j^2) grad W_ij
//   dv_i   = eps sum_{j!=i} (m_j/rho_j)(v_j - v_i) W_ij (XSPH on v_n)
// and integrates with integrate_particles' semantics (gravity and forces
// only for inv_mass > 0, |v| clamp, inactive particles keep x and v).
//
// Layout in HBM (sorted by cell, written by the last radix pass):
//   xs[k]  float4 (x, y, z, m_eff)   m_eff = -0 for inactive particles
//   vs[k]  float4 (vx, vy, vz, attr) attr = active | dynamic<<1 | gravity<<2
//   rec[k] 2 float4 (x, y, z, m_eff), (vx, vy, vz, m/rho), and
//   pr2[k] float p/rho^2             what the force passes gather of a neighbour,
//                                    written by the density pass
//   rp[k]  float2 (rho, p)           written by the density pass
// Outputs are scattered back to original particle order through point_ids.
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include <cuda_fp16.h>

#include "mlp.cuh"
#include "nsph_internal.cuh"

namespace nsph {

NSPH_BOUNDS_READER(sph)

namespace {

constexpr int kSphThreads = 256;

// the neighbour test shared with the oracle (no contraction beyond the two
// explicit FMAs): r2 = fma(dz, dz, fma(dy, dy, dx*dx))
__device__ __forceinline__ float dist2(float4 a, float4 b, float& dx, float& dy, float& dz)
{
    dx = __fsub_rn(a.x, b.x);
    dy = __fsub_rn(a.y, b.y);
    dz = __fsub_rn(a.z, b.z);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// Every fp32 operation below is written with an explicit rounding intrinsic
// (no compiler contraction), in the same order as the fp32 oracle, and each
// particle's neighbours are summed in the grid's query order, so the device
// reproduces the fp32 restatement's sums.

// W(q) = sigma * {fma((6q)q, q-1, 1) for q <= 1/2; ((2t)t)t with t = max(1-q, 0) beyond}
template <class P>
__device__ __forceinline__ float kernel_w(float q, const P& p)
{
    const float t = fmaxf(__fsub_rn(1.f, q), 0.f);
    const float nearv = __fmaf_rn(__fmul_rn(__fmul_rn(6.f, q), q), __fsub_rn(q, 1.f), 1.f);
    const float farv = __fmul_rn(__fmul_rn(__fmul_rn(2.f, t), t), t);
    return __fmul_rn(p.sigma, q <= 0.5f ? nearv : farv);
}

// (dW/dr)/r = {c_near * fma(3, q, -2) for q <= 1/2; ((c_far t) t)(1/r), t = max(1-q, 0), beyond}
template <class P>
__device__ __forceinline__ float kernel_f(float q, float inv_r, const P& p)
{
    const float t = fmaxf(__fsub_rn(1.f, q), 0.f);
    const float nearv = __fmul_rn(p.c_near, __fmaf_rn(3.f, q, -2.f));
    const float farv = __fmul_rn(__fmul_rn(__fmul_rn(p.c_far, t), t), inv_r);
    return q <= 0.5f ? nearv : farv;
}

// Square root of a squared distance, and its reciprocal, both correctly
// rounded (the bits of __fsqrt_rn and of __frcp_rn of it), from one hardware
// reciprocal square root y ~ 1/sqrt(x): Markstein's iterations (IBM J. Res.
// Dev. 34(1), 1990), whose residuals x - g g and 1 - r y are exact in one FMA.
// They need no test for special operands, which the general operations spend
// about half of their instructions on: x outside [2^-100, 2^100] (coincident
// particles apart, nothing a simulation meets) takes those, and x = 0 gives
// r = 0. Checked against them over every mantissa and exponent parity.
__device__ __forceinline__ bool plain_range(float x)  // or zero
{
    const unsigned u = __float_as_uint(x);
    return u - 0x0d800000u < 0x64000000u || u == 0u;
}

__device__ __forceinline__ float sqrt_plain(float x, float& y)
{
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float g = __fmul_rn(x, y), hy = __fmul_rn(0.5f, y);
    const float r = __fmaf_rn(__fmaf_rn(-g, g, x), hy, g);
    return x == 0.f ? 0.f : r;
}

__device__ __forceinline__ float rcp_plain(float r, float y)  // y ~ 1/r from sqrt_plain
{
    // rounded up: the last step then also meets the one mantissa (all ones)
    // for which an estimate below leads to a tie
    const float y1 = __fmaf_ru(__fmaf_rn(-r, y, 1.f), y, y);
    return __fmaf_rn(__fmaf_rn(-r, y1, 1.f), y1, y1);
}

__device__ __forceinline__ float eos(float rho, const nsph_sph_params& p)
{
    const float ratio = __fmul_rn(rho, p.inv_rho0);
    float pw = 1.f;
    for (int k = 0; k < p.eos_gamma; ++k) pw = __fmul_rn(pw, ratio);
    float pr = __fmul_rn(p.eos_b, __fsub_rn(pw, 1.f));
    if (p.clamp_pressure && pr < 0.f) pr = 0.f;
    return pr;
}

template <class P>
__device__ __forceinline__ float wterm(float r2, const P& p)
{
    float y, r;
    if (plain_range(r2))
        r = sqrt_plain(r2, y);
    else
        r = __fsqrt_rn(r2);
    return kernel_w(__fmul_rn(r, p.inv_h), p);
}

// wterm of a squared distance known to be zero or in the plain range: the
// estimate of max(x, 2^-100) is finite, and gives r = 0 for x = 0
template <class P>
__device__ __forceinline__ float wterm_near(float r2, const P& p)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(r2, 7.8886091e-31f)));
    const float g = __fmul_rn(r2, y), hy = __fmul_rn(0.5f, y);
    return kernel_w(__fmul_rn(__fmaf_rn(__fmaf_rn(-g, g, r2), hy, g), p.inv_h), p);
}

// ---- tolerance ("fast") arithmetic ---------------------------------------------
// The same kernel values with the hardware reciprocal square root instead of
// the correctly rounded square root, reciprocal and division, and with the
// compiler free to contract multiply-adds: r = r2 * rsqrt(r2), 1/r = rsqrt(r2).
// The neighbour test r2 < h2 is unchanged, so neighbour sets stay bit-exact;
// sums keep the query order. Results are within the fp64 oracle's tolerance
// (checked by the tests), not bit-exact with the fp32 oracle.
template <class P>
__device__ __forceinline__ float kernel_w_fast(float q, const P& p)
{
    const float t = 1.f - q;
    const float v = q <= 0.5f ? fmaf(6.f * q * q, q - 1.f, 1.f) : (q < 1.f ? 2.f * t * t * t : 0.f);
    return p.sigma * v;
}

template <class P>
__device__ __forceinline__ float wterm_fast(float r2, const P& p)
{
    const float r = r2 > 0.f ? r2 * rsqrtf(r2) : 0.f;
    return kernel_w_fast(r * p.inv_h, p);
}

// ---- density + EOS -----------------------------------------------------------
// What the force pass gathers of a neighbour: one 32-byte record (x, y, z, m |
// vx, vy, vz, m/rho), read by one 256-bit load, and p/rho^2. The gathers bound
// that pass (83% of the L1's wavefronts at 49% issue active): a warp's lanes
// read neighbours from about 10 lines of 16-byte or 25 lines of 32-byte
// records at a time, one wavefront per line. Two loads instead of three took
// the 1M tank's pass from 0.158 to 0.152 ms, the batched worlds' (512 worlds,
// 2.2M particles; with the shorter terms below) from 0.375 to 0.268 ms.
struct ForceRec {
    float4* rec;  // 2 per particle
    float* pr2;
    unsigned* overflow;  // or null: set when a particle's list overflowed (the segment tape)
};

struct Neighbour {
    float4 x, v;  // (x, m), (v, m/rho)
};

__device__ __forceinline__ Neighbour load_neighbour(const float4* __restrict__ rec, int j)
{
    Neighbour r;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r.x.x), "=f"(r.x.y), "=f"(r.x.z), "=f"(r.x.w), "=f"(r.v.x), "=f"(r.v.y), "=f"(r.v.z), "=f"(r.v.w)
        : "l"(rec + 2 * (size_t)j));
    return r;
}

template <bool Fast = false>
__device__ __forceinline__ void density_finish(int k, float4 xi, float4 vi, float rho, const nsph_sph_params& p,
                                               float2* __restrict__ rp, const ForceRec& fr,
                                               unsigned* __restrict__ status)
{
    const float m = xi.w;
    float pr = 0.f, mor = 0.f, pr2 = 0.f;
    if (rho > 0.f) {
        pr = eos(rho, p);
        if (Fast) {
            const float ir = __frcp_rn(rho);
            mor = m * ir;
            pr2 = pr * ir * ir;
        } else {
            mor = __fdiv_rn(m, rho);
            pr2 = __fdiv_rn(pr, __fmul_rn(rho, rho));
        }
    } else if (status) {
        atomicOr(status, (unsigned)NSPH_STATUS_ZERO_DENSITY);
    }
    rp[k] = make_float2(rho, pr);
    fr.rec[2 * (size_t)k] = xi;
    fr.rec[2 * (size_t)k + 1] = make_float4(vi.x, vi.y, vi.z, mor);
    fr.pr2[k] = pr2;
}

// ---- neighbour lists (the plain step) -----------------------------------------
// The density pass of the plain step first tests every candidate (in query
// order) and appends the sorted index of each neighbour to the particle's
// list, in groups of four: group g (slots 4g .. 4g+3) at nbr[g * n + k] as
// one int4 (group-major, so that a warp reading group g of 32 consecutive
// particles reads one contiguous 512-byte span), for the first kNbrSlots
// neighbours, and their number in ncnt[k]. A thread keeps the last four hits
// in registers and stores a full group at once (a store per four neighbours
// instead of one per neighbour). The cubic-spline terms are then evaluated
// by a second loop over the list, in the same order, so every lane of a warp
// runs the term code only for its own neighbours (evaluated inside the
// candidate loop, a warp runs it for every candidate slot at which any of
// its 32 lanes has a hit, which at a ~15% hit rate is nearly all of them).
// Readers load a whole group ahead of its use. The force pass walks the same
// list with one uniform loop and no grid traversal. A particle with more
// than kNbrSlots neighbours (dense clusters) is summed by re-testing its
// candidates, in the same order. Sums, their order and every rounding are
// those of the fp32 oracle.
constexpr int kNbrSlots = 64;
constexpr int kNbrGroups = kNbrSlots / 4;
// entries every sorted-position array that neighbor_list reads holds past
// its last particle (the candidate groups' reads past a run's end)
constexpr int kXsPad = 4;

// One candidate's hit bit pushed into `acc` from the right: the sign bit of
// fl(r2 - h2), by one funnel shift. fl(r2 - h2) is negative exactly when
// r2 < h2: an IEEE subtraction of two unequal values is never zero and its
// rounding keeps the sign, and r2 == h2 gives +0. A NaN difference (from a
// non-finite position) is the GPU's canonical NaN, whose sign bit is clear,
// as r2 < h2 is false for it. So the bits are those of the comparison, at
// one FADD and one shift per candidate instead of a compare, a select, a
// variable shift and an OR.
__device__ __forceinline__ unsigned push_hit(unsigned acc, float r2, float h2)
{
    return __funnelshift_l(__float_as_uint(__fsub_rn(r2, h2)), acc, 1);
}

// Appends neighbours to particle k's list in groups of four: the last four
// are held in registers and a full group is stored at once.
struct ListWriter {
    int4* nbr;
    int n, k;
    int cnt = 0;
    int b0 = 0, b1 = 0, b2 = 0, b3 = 0;
    __device__ __forceinline__ ListWriter(int4* nbr_, int n_, int k_) : nbr(nbr_), n(n_), k(k_) {}
    __device__ __forceinline__ void append(int j)
    {
        b0 = b1;
        b1 = b2;
        b2 = b3;
        b3 = j;
        ++cnt;
        if ((cnt & 3) == 0 && cnt <= kNbrSlots) nbr[(size_t)((cnt >> 2) - 1) * n + k] = make_int4(b0, b1, b2, b3);
    }
    // the last, partial group: its r hits are b(4-r) .. b3; the rest of it is
    // filled with the particle itself, which its readers skip
    __device__ __forceinline__ void finish()
    {
        const int r = cnt & 3;
        if (r && cnt <= kNbrSlots)
            nbr[(size_t)(cnt >> 2) * n + k] = r == 1 ? make_int4(b3, k, k, k)
                                                     : (r == 2 ? make_int4(b2, b3, k, k) : make_int4(b1, b2, b3, k));
    }
};

// The general scan of one particle by one thread: its candidates are tested
// branch-free into a bit mask per chunk of up to 32 of a run (four loads
// issued together; a run's last group reads up to three entries past the run,
// whose bits are cleared: every xs array the density passes read holds at
// least kXsPad entries past its last particle), and a chunk's hits are
// appended to the list after it. Serves the warps that tile_neighbors
// (below) does not take.
__device__ __forceinline__ int neighbor_list(const GridDev& g, const float4* __restrict__ xs,
                                             const nsph_sph_params& p, float4 xi, int4* __restrict__ nbr, int n,
                                             int k)
{
    ListWriter list(nbr, n, k);
    for_each_run(g, xi.x, xi.y, xi.z, p.h, [&](int lo, int hi) {
        for (int c0 = lo; c0 < hi; c0 += 32) {
            const int m = min(32, hi - c0);
            unsigned acc = 0u;  // candidate t of the chunk at bit mp - 1 - t
#pragma unroll 1
            for (int j = 0; j < m; j += 4) {
                float4 xj[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) xj[u] = __ldg(xs + c0 + j + u);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float dx, dy, dz;
                    acc = push_hit(acc, dist2(xi, xj[u], dx, dy, dz), p.h2);
                }
            }
            // reversed, candidate t sits at bit t; the group's reads past
            // the run (bits m .. mp - 1) are cleared
            const int mp = (m + 3) & ~3;
            unsigned bits = __brev(acc) >> (32 - mp);
            if (m < 32) bits &= (1u << m) - 1u;
            while (bits) {
                const int j = c0 + __ffs(bits) - 1;
                if (!mirror_inactive(__ldg(xs + j))) list.append(j);
                bits &= bits - 1u;
            }
        }
    });
    list.finish();
    return list.cnt;
}

// Element u (0..3, a constant after unrolling) of a list group.
__device__ __forceinline__ int group_item(const int4& gr, int u)
{
    return u == 0 ? gr.x : (u == 1 ? gr.y : (u == 2 ? gr.z : gr.w));
}

// Walk of a particle's list by whole groups: visit(j) for its neighbours in
// order. The group after the current one is loaded when the current one
// starts; the four items of a group are unrolled, so each index is a fixed
// register (no per-item select, as a reader returning one item at a time
// needs) and the visits' loads can issue together. kReadOnly: the list was
// written by an earlier kernel (read-only path); otherwise it is read back by
// the thread that wrote it (plain loads). (The items stay a function of their
// own: written into the loop, the compiler contracts the surrogate's feature
// sums another way, and its outputs differ in the last place of a feature.)
template <bool kReadOnly, class F>
__device__ __forceinline__ void for_each_listed(const int4* __restrict__ nbr, int n, int k, int cnt, F&& visit)
{
    in_bounds(cnt >= 0 && cnt <= kNbrSlots);
    const int4* a = nbr + k;
    auto load = [&](int gi) { return kReadOnly ? __ldg(a + (size_t)gi * n) : a[(size_t)gi * n]; };
    int4 cur = cnt > 0 ? load(0) : make_int4(0, 0, 0, 0);
    int4 nxt = cnt > 4 ? load(1) : make_int4(0, 0, 0, 0);
    for (int t = 0; t < cnt; t += 4) {
        const int4 gr = cur;
        cur = nxt;
        if (t + 8 < cnt) nxt = load((t >> 2) + 2);
        auto item = [&](int u) {
            if (t + u < cnt) {
                const int j = group_item(gr, u);
                visit(in_bounds(j >= 0 && j < n) ? j : 0);
            }
        };
#pragma unroll
        for (int u = 0; u < 4; ++u) item(u);
    }
}

// rho of particle k from its list (read back by the thread that wrote it,
// with plain loads), or by re-testing its candidates when the list overflowed
template <bool Fast>
__device__ __forceinline__ float density_from_list(const GridDev& g, const float4* __restrict__ xs,
                                                   const nsph_sph_params& p, float4 xi, const int4* nbr, int cnt,
                                                   int n, int k)
{
    float rho = 0.f;
    auto w = [&](float r2) { return Fast ? wterm_fast(r2, p) : wterm(r2, p); };
    if (cnt <= kNbrSlots) {
        for_each_listed<false>(nbr, n, k, cnt, [&](int j) {
            const float4 xj = __ldg(xs + j);
            float dx, dy, dz;
            rho = __fmaf_rn(xj.w, w(dist2(xi, xj, dx, dy, dz)), rho);
        });
    } else {
        for_each_candidate(g, xi.x, xi.y, xi.z, p.h, [&](int j) {
            const float4 xj = __ldg(xs + j);
            float dx, dy, dz;
            const float r2 = dist2(xi, xj, dx, dy, dz);
            if (r2 < p.h2) rho = __fmaf_rn(xj.w, w(r2), rho);
        });
    }
    return rho;
}

// The general path of one particle: list, then rho over it (a call, so that
// its registers do not count against the kernels whose rare path it is).
template <bool Fast>
__device__ __noinline__ int scan_general(const GridDev* g, const float4* xs, const nsph_sph_params* p, float4 xi,
                                         int4* nbr, int n, int k, float* rho)
{
    const int cnt = neighbor_list(*g, xs, *p, xi, nbr, n, k);
    *rho = density_from_list<Fast>(*g, xs, *p, xi, nbr, cnt, n, k);
    return cnt;
}

// ---- candidate tests on the tensor cores ----------------------------------------
// A warp takes 32 consecutive sorted particles, one per lane. Particles of
// one grid row (the same y and z cells, x cells within kTileSpan) share their
// candidates: the union of their stencils is one contiguous run of sorted
// positions per (z, y) row. Each run is tested in chunks of 32 candidates
// against all 32 particles at once, as the contraction
//   r2 - T = |a|^2 - T + |b|^2 - 2 a.b
// of fp16 coordinates relative to the group's origin in units of h
// (mma.m16n8k8, fp32 sums: eight instructions per chunk; the norms are split
// into fp16 hi + lo parts along K). The sign of r2 - T marks a possible
// neighbour: T exceeds 1 by a bound on the rounding errors, so no neighbour is
// missed. (fp16 sums, of which only half precision is specified, would save 3 of
// the 434 us of the 1M tank's step.) A chunk's marks (one 32-bit word per
// particle) wait in shared memory; then each lane walks its own marks in order,
// repeats the exact fp32 test of the definition, sums rho and appends to the
// list. Sets, order and every rounding are therefore those of the general scan.
//
// Why: per particle about 216 candidates are tested for 30 neighbours. One
// thread per particle spent three quarters of its 211 warp instructions per
// particle on the tests and the traversal; a chunk of 1,024 tests costs about
// 75 warp instructions, a third of them the matrix part, and the traversal is
// done once per group. The 1M tank's pass went from 0.291 to 0.246 ms (160 warp
// instructions per particle, 78% issue active), the 128^3 block's from 0.563
// to 0.48. What bounds it now is the walk: some 70 instructions for each of a
// warp's 38 steps. The tiles are 32 x 32 with K = 8 and live in one warp's
// registers: tcgen05's 128-row tiles would span 16 cells, of whose joint
// stencil a particle uses a sixth. 64 registers; 48 (five blocks per SM) were
// slower (0.288 ms).
constexpr int kTileWords = 20;   // words of 32 candidates between two walks (a dense stencil has 18)
constexpr int kTileSpan = 12;     // x cells between the first and the last particle of a group

// resident blocks per SM of the density passes (registers: see the kernels)
constexpr int kDensityBlocks = 4;

struct __align__(16) TileSmem {
    union {
        // B operand of a chunk's halves: word t (of k = 2t, 2t + 1) of candidate c at [t][c]. Rows of 40 words put
        // the eight lanes of a 128-bit load's phase (4 rows x 2 columns) on different banks.
        unsigned frag[2][4][40];
        int ring[8][32];          // during a walk: the lane's last neighbours, until a group of four is stored
    };
    union {
        unsigned a[4][32];     // A operand: word t of row r at [t][r]
        unsigned bits[2][32];  // sign bytes of a chunk's halves by lane
    };
    unsigned marks[kTileWords][32];  // of 32 waiting candidates, by lane; words from the last one down
    int first[kTileWords];           // the last of them
};

__device__ __forceinline__ unsigned pack_h2(float lo, float hi)
{
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ float2 unpack_h2(unsigned u)
{
    return __half22float2(*reinterpret_cast<const __half2*>(&u));
}

// D = A (16 x 8) B (8 x 8), fp16 operands and fp32 sums: d[0], d[1] = row
// lane / 4, columns 2 (lane % 4) and + 1; d[2], d[3] = row lane / 4 + 8
__device__ __forceinline__ void mma_16x8x8(float (&d)[4], unsigned a0, unsigned a1, unsigned b)
{
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}

// c moved up by two bytes, below it the signs of hi and lo: 0 where negative, 0xff
// above a hundred denormals (as integers, saturated to eight bits). Two of these
// for four products instead of three byte permutations.
__device__ __forceinline__ unsigned push_signs(unsigned c, float hi, float lo)
{
    unsigned s;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;"
        : "=r"(s)
        : "r"(__float_as_int(hi)), "r"(__float_as_int(lo)), "r"(c));
    return s;
}

// Neighbour list and rho of the warp's particles k (one per lane; lanes with
// !member have none). g, p: the lane's grid and parameters (the same in every
// lane unless kWorlds, where `world` tells them apart). Returns the lane's
// neighbour count, or -1 in every lane when the warp needs the general scan:
// clamped cells, a stencil as wide as the grid (where it wraps onto itself)
// or of more than 32 runs, or particles scattered over many rows.
template <bool Fast, bool kWorlds>
__device__ __forceinline__ int tile_neighbors(const GridDev& g, const float4* __restrict__ xs,
                                              const nsph_sph_params& p, int world, float4 xi, bool member,
                                              int4* __restrict__ nbr, int n, int k, TileSmem& sm, float& rho_out)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    rho_out = 0.f;
    // a particle without a finite position has no neighbours
    member = member && isfinite(xi.x) && isfinite(xi.y) && isfinite(xi.z);
    int bx = 0, ex = 0, by = 0, ey = 0, bz = 0, ez = 0;
    bool clamped = false;
    if (member) {
        box_axis_regular(xi.x, p.h, g.inv, g.dx, bx, ex, clamped);
        box_axis_regular(xi.y, p.h, g.inv, g.dy, by, ey, clamped);
        box_axis_regular(xi.z, p.h, g.inv, g.dz, bz, ez, clamped);
        // a box as wide as the grid meets its own image
        clamped |= ex - bx + 3 > g.dx || ey - by + 3 > g.dy || ez - bz + 3 > g.dz;
        clamped |= (ey - by + 1) * (ez - bz + 1) > 16;
    }
    if (__any_sync(kAll, clamped)) return -1;
    unsigned todo = __ballot_sync(kAll, member);
    const int k_self = min(k, n - 1);
    // Below this squared distance a candidate's cell is surely inside the box
    // (its cell and the box ends are monotone in the coordinate up to three
    // roundings each); nearer to h the cell is compared, since the definition
    // visits a cell of the box and nothing else.
    const float cells = fmaxf(fmaxf(fabsf(xi.x), fabsf(xi.y)), fabsf(xi.z)) * p.inv_h;
    const float h2_safe = p.h2 * (1.f - (cells + 2.f) * 1.9073486e-6f);  // 2^-19 per cell

    float rho = 0.f;
    int cnt = 0, stored = 0;         // neighbours, and those in stored groups
    int p0 = k, p1 = k, p2 = k;      // the cnt - stored < 4 others
    int nw = kTileWords;             // words free
    unsigned any = 0u;               // those with marks of this lane
    int total = 0;                   // this lane's waiting marks
    // The lane's candidate of a chunk's half, last first, so that bit l of a
    // ballot and of a word of marks is lane l's and words are walked from the top
    // bit down.
    const int cand = 31 - lane;

    int groups = 0;
    while (todo) {
        // ---- the next group and its runs ----
        const int lead = __ffs(todo) - 1;
        const int lbx = __shfl_sync(kAll, bx, lead), lby = __shfl_sync(kAll, by, lead);
        const int ley = __shfl_sync(kAll, ey, lead), lbz = __shfl_sync(kAll, bz, lead);
        const int lez = __shfl_sync(kAll, ez, lead);
        const int lworld = kWorlds ? __shfl_sync(kAll, world, lead) : world;
        const bool mine = ((todo >> lane) & 1u) && by == lby && ey == ley && bz == lbz && ez == lez &&
                          world == lworld && (unsigned)(bx - lbx) < (unsigned)kTileSpan;
        const unsigned in_group = __ballot_sync(kAll, mine);
        todo &= ~in_group;
        if (++groups > 12 && todo) return -1;  // scattered particles: one thread each is cheaper
        const int xe = __reduce_max_sync(kAll, mine ? ex : lbx);
        const int x0 = __reduce_min_sync(kAll, mine ? bx : lbx);
        int gdx = g.dx, gdy = g.dy, gdz = g.dz;
        float inv_h = p.inv_h;
        const int2* ranges = g.ranges;
        if (kWorlds) {
            gdx = __shfl_sync(kAll, g.dx, lead);
            gdy = __shfl_sync(kAll, g.dy, lead);
            gdz = __shfl_sync(kAll, g.dz, lead);
            inv_h = __shfl_sync(kAll, p.inv_h, lead);
            ranges = reinterpret_cast<const int2*>(
                __shfl_sync(kAll, reinterpret_cast<unsigned long long>(g.ranges), lead));
        }
        const int nx = xe - x0 + 1;
        if (nx + 2 > gdx) return -1;
        // runs: row (z, y) of the box, in two parts where x wraps
        const int ny = ley - lby + 1, rows = ny * (lez - lbz + 1);
        const int cx0 = wrap_cell(x0, gdx);
        const int wrap = min(nx, gdx - cx0);  // cells before the wrap
        const bool two = wrap < nx;
        int lo = 0x7fffffff, hi = 0;
        {
            const int row = two ? lane >> 1 : lane;
            if (row < rows) {
                const int iz = ny == 3 ? (row * 0x5556) >> 16 : row / ny, iy = row - iz * ny;
                const int cz = wrap_cell(lbz + iz, gdz), cy = wrap_cell(lby + iy, gdy);
                const bool second = two && (lane & 1);
                const int2* cell = ranges + (cz * gdy + cy) * gdx + (second ? 0 : cx0);
                const int cells_here = second ? nx - wrap : wrap;
                // from the first cell with particles to the last (an empty cell reads 0, 0)
                const int2 front = __ldg(cell), back = __ldg(cell + cells_here - 1);
                lo = front.x;
                hi = back.y;
                if (front.y == front.x || back.y == back.x) {
                    lo = 0x7fffffff;
                    hi = 0;
#pragma unroll 4
                    for (int c = 0; c < cells_here; ++c) {
                        const int2 se = __ldg(cell + c);
                        if (se.y > se.x) {
                            lo = min(lo, se.x);
                            hi = max(hi, se.y);
                        }
                    }
                }
                if (lo < hi && !in_bounds(lo >= 0 && hi <= g.n)) hi = lo;
            }
        }
        unsigned runs = __ballot_sync(kAll, lo < hi);

        // ---- the A operand: rows (-2x, -2y | -2z, 1 | 1, n_hi | n_lo, 0) ----
        const int last = 31 - __clz(in_group);
        const float ox = 0.5f * (__shfl_sync(kAll, xi.x, lead) + __shfl_sync(kAll, xi.x, last));
        const float oy = __shfl_sync(kAll, xi.y, lead), oz = __shfl_sync(kAll, xi.z, lead);
        unsigned a0, a1, a2, a3;
        {
            const float ux = mine ? (xi.x - ox) * inv_h : 0.f, uy = mine ? (xi.y - oy) * inv_h : 0.f,
                        uz = mine ? (xi.z - oz) * inv_h : 0.f;
            const unsigned hxy = pack_h2(ux, uy), hz = pack_h2(uz, 0.f);
            const float2 fxy = unpack_h2(hxy);
            const float fz = unpack_h2(hz).x;
            // the largest coordinates bound the fp16 rounding of a pair's
            // difference: |u| 2^-11 for each of the two (a neighbour lies
            // within 1 of its particle)
            const float mx = __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(fabsf(ux)))) + 1.01f;
            const float myz =
                __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(fmaxf(fabsf(uy), fabsf(uz))))) + 1.01f;
            const float d = 9.765625e-4f * sqrtf(mx * mx + 2.f * myz * myz);  // 2 x 2^-11
            const float big = mx * mx + 2.f * myz * myz;
            // (1 + d)^2 of the rounded coordinates, and for the sum, of which the
            // PTX specification promises products and additions in at least
            // single precision, in any order, subnormal operands kept or not:
            // per axis the product of a coordinate below 2^-14, at most 2^-13 of
            // the other; the norms' parts below 2^-14, 2^-13 in all; eight
            // additions of at most 5 big, 2^-23 each (4.8e-6 big); and the norms'
            // splits and the fp32 roundings of coordinates, norms and the
            // definition's test (under 1.2e-6 big)
            const float thr = (1.f + d) * (1.f + d) + 1.3e-4f * (mx + 2.f * myz + 1.f) + 8e-6f * big;
            const float n2 = fmaf(fz, fz, fmaf(fxy.y, fxy.y, fxy.x * fxy.x)) - thr;
            const float n2h = unpack_h2(pack_h2(n2, 0.f)).x;
            const unsigned w0 = pack_h2(-2.f * fxy.x, -2.f * fxy.y), w1 = pack_h2(-2.f * fz, 1.f);
            const unsigned w2 = pack_h2(1.f, n2h), w3 = pack_h2(n2 - n2h, 0.f);
            if (!(big < 4096.f)) return -1;  // cells far wider than h: the norms leave fp16's range
            __syncwarp();  // (the last chunk's sign bytes are read)
            sm.a[0][lane] = w0;
            sm.a[1][lane] = w1;
            sm.a[2][lane] = w2;
            sm.a[3][lane] = w3;
            __syncwarp();
            const unsigned* a = &sm.a[lane & 3][lane >> 2];
            a0 = a[0];
            a1 = a[8];
            a2 = a[16];
            a3 = a[24];
            __syncwarp();
        }

        // ---- chunks of 64 candidates (a dense run has about 50) ----
        sm.frag[0][3][lane] = sm.frag[1][3][lane] = 0x00003c00u;  // k = 6, 7 of B: (1, 0)
        int c0 = 0, end = 0;
        float4 q[2];
        bool more;
        auto next_chunk = [&]() {  // and issue the loads of its candidates
            c0 += 64;
            if (c0 >= end) {
                more = runs != 0u;
                if (!more) return;
                const int r = __ffs(runs) - 1;
                runs &= runs - 1u;
                c0 = __shfl_sync(kAll, lo, r);
                end = __shfl_sync(kAll, hi, r);
            }
            q[0] = __ldg(xs + min(c0 + cand, end - 1));
            q[1] = __ldg(xs + min(c0 + 32 + cand, end - 1));
        };
        q[0] = q[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        more = true;
        next_chunk();
        do {
            if (more) {
                const int at = c0, m = end - c0;
                const int halves = m > 32 ? 2 : 1;
                unsigned counted[2] = {0u, 0u};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h >= halves) break;
                    const float ux = (q[h].x - ox) * inv_h, uy = (q[h].y - oy) * inv_h, uz = (q[h].z - oz) * inv_h;
                    const unsigned hxy = pack_h2(ux, uy);
                    const float2 fxy = unpack_h2(hxy);
                    const float fz = unpack_h2(pack_h2(uz, 0.f)).x;
                    const float n2 = fmaf(fz, fz, fmaf(fxy.y, fxy.y, fxy.x * fxy.x));
                    const unsigned w1 = pack_h2(fz, n2);
                    sm.frag[h][0][lane] = hxy;
                    sm.frag[h][1][lane] = w1;
                    sm.frag[h][2][lane] = pack_h2(n2 - unpack_h2(w1).y, 1.f);
                    // past the run's end and inactive (in no list): no mark
                    counted[h] = __ballot_sync(kAll, 32 * h + cand < m && !mirror_inactive(q[h]));
                }
                next_chunk();
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h >= halves) break;
                    // column j of tile i is the candidate of lane 4 j + i
                    const uint4 b = *reinterpret_cast<const uint4*>(&sm.frag[h][lane & 3][lane & ~3]);
                    const unsigned bw[4] = {b.x, b.y, b.z, b.w};
                    // bit 4 j + i of byte g: tile i, column 2 (lane % 4) + j, row lane / 4 + 8 g; 1 where not near
                    unsigned acc = 0u;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float d01[4], d23[4];
                        mma_16x8x8(d01, a0, a1, bw[i]);
                        mma_16x8x8(d23, a2, a3, bw[i]);
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            acc |= push_signs(push_signs(0u, d23[2 + j], d23[j]), d01[2 + j], d01[j]) &
                                   (0x01010101u << (4 * j + i));
                    }
                    sm.bits[h][lane] = acc;
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h >= halves) break;
                    // this lane's row from the four lanes that hold its columns
                    const uint4 v = *reinterpret_cast<const uint4*>(&sm.bits[h][4 * (lane & 7)]);
                    const unsigned sel = 0x4040u + 0x1111u * (unsigned)(lane >> 3);
                    const unsigned y0 = __byte_perm(v.x, v.y, sel), y1 = __byte_perm(v.z, v.w, sel);
                    const unsigned marks = ~((y0 & 0xffffu) | (y1 & 0xffff0000u)) & (mine ? counted[h] : 0u);
                    --nw;
                    sm.marks[nw][lane] = marks;
                    if (lane == 0) sm.first[nw] = at + 32 * h + 31;
                    any |= (marks != 0u ? 1u : 0u) << nw;
                    total += __popc(marks);
                }
            }
            if (nw < 2 || !(more || todo)) {
                // ---- the walk over the waiting marks ----
                // without branches on the way; a lane that has run out visits
                // its own particle in vain
                const int most = __reduce_max_sync(kAll, total);
                __syncwarp();  // first[], and the last reads of frag
                auto push = [&](int j) {
                    sm.ring[cnt & 7][lane] = j;
                    ++cnt;
                };
                sm.ring[stored & 7][lane] = p0;
                sm.ring[(stored + 1) & 7][lane] = p1;
                sm.ring[(stored + 2) & 7][lane] = p2;
                unsigned cur = 0u;
                int jb = 0;
                auto pop = [&](int t) {
                    const int c = max(31 - __clz(any), 0);
                    const unsigned word = sm.marks[c][lane];
                    const int base = sm.first[c];
                    const bool dry = cur == 0u;
                    cur = dry ? word : cur;
                    jb = dry ? base : jb;
                    any = dry ? any & ~(1u << c) : any;
                    const int b = 31 - __clz(cur);
                    cur &= ~(1u << (b & 31));
                    return t < total ? jb - b : k_self;
                };
                int j = pop(0);
                float4 xj = __ldg(xs + j);
                for (int t0 = 0; t0 < most; t0 += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int t = t0 + u;
                        const int jn = pop(t + 1);
                        const float4 xn = __ldg(xs + jn);
                        float dx, dy, dz;
                        const float r2 = dist2(xi, xj, dx, dy, dz);
                        const float rho1 = __fmaf_rn(xj.w, Fast ? wterm_fast(r2, p) : wterm_near(r2, p), rho);
                        const bool valid = t < total, inside = r2 < h2_safe;
                        // near the support's edge, or closer than 2^-50: rare
                        if (valid && (!inside || __float_as_uint(r2) - 1u < 0x0d7fffffu)) {
                            const int cx = trunc_sat(__fmul_rn(xj.x, g.inv)), cy = trunc_sat(__fmul_rn(xj.y, g.inv)),
                                      cz = trunc_sat(__fmul_rn(xj.z, g.inv));
                            if (r2 < p.h2 && cx >= bx && cx <= ex && cy >= by && cy <= ey && cz >= bz && cz <= ez) {
                                push(j);
                                rho = __fmaf_rn(xj.w, Fast ? wterm_fast(r2, p) : wterm(r2, p), rho);
                            }
                        } else if (valid) {
                            rho = rho1;
                            push(j);
                        }
                        j = jn;
                        xj = xn;
                    }
                    if (cnt - stored >= 4) {  // (at most seven are in the ring)
                        const int* r = &sm.ring[stored & 7][lane];
                        if (stored < kNbrSlots)
                            nbr[(size_t)(stored >> 2) * n + k] = make_int4(r[0], r[32], r[64], r[96]);
                        stored += 4;
                    }
                }
                const int* r = &sm.ring[stored & 7][lane];
                p0 = r[0];
                p1 = r[32];
                p2 = r[64];
                __syncwarp();
                nw = kTileWords;
                total = 0;
                any = 0u;
                sm.frag[0][3][lane] = sm.frag[1][3][lane] = 0x00003c00u;
            }
        } while (more);
    }
    // the last, partial group: the rest of it is filled with the particle itself
    const int rest = cnt - stored;
    if (rest > 0 && cnt <= kNbrSlots)
        nbr[(size_t)(stored >> 2) * n + k] = make_int4(p0, rest > 1 ? p1 : k, rest > 2 ? p2 : k, k);
    rho_out = rho;
    return cnt;
}

struct ForceAcc {
    float ax, ay, az, dvx, dvy, dvz;
};

// the constants that a force term reads (of one world, or of all particles)
struct ForceConst {
    float inv_h, sigma, c_near, c_far;
    __device__ __forceinline__ explicit ForceConst(const nsph_sph_params& p)
        : inv_h(p.inv_h), sigma(p.sigma), c_near(p.c_near), c_far(p.c_far)
    {
    }
};

// Pressure and XSPH terms of one neighbour: a -= s d, dv += c u, accumulated
// in order (not of the particle itself). A coincident one has no pressure term.
struct ForceTerm {
    float s, dx, dy, dz, c, ux, uy, uz;
};

template <class P>
__device__ __forceinline__ ForceTerm force_factors(float4 xj, float4 vj, float pr2_j, float4 xi, float4 vi, float pr2_i,
                                                   const P& p)
{
    ForceTerm t;
    const float r2 = dist2(xi, xj, t.dx, t.dy, t.dz);
    float r, inv_r;
    if (plain_range(r2)) {
        float y;
        r = sqrt_plain(r2, y);
        inv_r = rcp_plain(r, y);  // (not a number for r = 0, where it is not used)
    } else {
        r = __fsqrt_rn(r2);
        inv_r = __frcp_rn(r);
    }
    const float q = __fmul_rn(r, p.inv_h);
    const float w = kernel_w(q, p);
    const float f = kernel_f(q, inv_r, p);
    t.s = r2 > 0.f ? __fmul_rn(__fmul_rn(xj.w, __fadd_rn(pr2_i, pr2_j)), f) : 0.f;
    t.c = __fmul_rn(vj.w, w);
    t.ux = __fsub_rn(vj.x, vi.x);
    t.uy = __fsub_rn(vj.y, vi.y);
    t.uz = __fsub_rn(vj.z, vi.z);
    return t;
}

template <class P>
__device__ __forceinline__ void force_term_data(float4 xj, float4 vj, float pr2_j, float4 xi, float4 vi, float pr2_i,
                                                const P& p, ForceAcc& acc)
{
    const ForceTerm t = force_factors(xj, vj, pr2_j, xi, vi, pr2_i, p);
    acc.ax = __fmaf_rn(-t.s, t.dx, acc.ax);
    acc.ay = __fmaf_rn(-t.s, t.dy, acc.ay);
    acc.az = __fmaf_rn(-t.s, t.dz, acc.az);
    acc.dvx = __fmaf_rn(t.c, t.ux, acc.dvx);
    acc.dvy = __fmaf_rn(t.c, t.uy, acc.dvy);
    acc.dvz = __fmaf_rn(t.c, t.uz, acc.dvz);
}

// force_term_data in the tolerance arithmetic (see kernel_w_fast)
template <class P>
__device__ __forceinline__ void force_term_fast(float4 xj, float4 vj, float pr2_j, float4 xi, float4 vi, float pr2_i,
                                                const P& p, ForceAcc& acc)
{
    const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    float w = p.sigma;
    if (r2 > 0.f) {
        const float ir = rsqrtf(r2);
        const float q = r2 * ir * p.inv_h;
        const float t = 1.f - q;
        w = kernel_w_fast(q, p);
        const float f = q <= 0.5f ? p.c_near * fmaf(3.f, q, -2.f) : (q < 1.f ? p.c_far * t * t * ir : 0.f);
        const float s = xj.w * (pr2_i + pr2_j) * f;
        acc.ax -= s * dx;
        acc.ay -= s * dy;
        acc.az -= s * dz;
    }
    const float c = vj.w * w;
    acc.dvx += c * (vj.x - vi.x);
    acc.dvy += c * (vj.y - vi.y);
    acc.dvz += c * (vj.z - vi.z);
}

struct StepOut {
    const float* f_ext;
    const float* inv_mass;
    const float* gravity;
    float* x_out;
    float* v_out;
    float* rho_out;
    float* p_out;
    float* a_out;
    unsigned* status;
    float4* acc_sorted;  // or null: (a, 0), (dv, 0) of sorted particle k at 2k, 2k + 1 (the segment tape)
    bool carry_v;        // write inactive particles' velocities too (unchanged; a step leaves them alone)
};

// integrate particle k (original index i) and scatter its outputs
__device__ __forceinline__ void integrate_out(size_t i, float4 xi, float4 vi, int attr, float2 rpk,
                                              const ForceAcc& acc, const nsph_sph_params& p, float dt,
                                              const StepOut& o)
{
    if (o.rho_out) o.rho_out[i] = rpk.x;
    if (o.p_out) o.p_out[i] = rpk.y;
    if (!(attr & kAttrActive)) {
        o.x_out[3 * i + 0] = xi.x;
        o.x_out[3 * i + 1] = xi.y;
        o.x_out[3 * i + 2] = xi.z;
        if (o.carry_v) {
            o.v_out[3 * i + 0] = vi.x;
            o.v_out[3 * i + 1] = vi.y;
            o.v_out[3 * i + 2] = vi.z;
        }
        if (o.a_out) o.a_out[3 * i + 0] = o.a_out[3 * i + 1] = o.a_out[3 * i + 2] = 0.f;
        return;
    }
    const float ax = acc.ax, ay = acc.ay, az = acc.az;
    if (o.a_out) {
        store_row(o.a_out + 3 * i, ax, ay, az);
    }
    float v1x = vi.x, v1y = vi.y, v1z = vi.z;
    const bool dynamic = (attr & kAttrDynamic) != 0;
    if (dynamic) {
        const int gw = attr >> kAttrGravShift;
        float fx = 0.f, fy = 0.f, fz = 0.f;
        if (o.f_ext) {
            const float w = o.inv_mass[i];
            const Row3 f = load_row(o.f_ext + 3 * i);
            fx = __fmul_rn(f.x, w);
            fy = __fmul_rn(f.y, w);
            fz = __fmul_rn(f.z, w);
        }
        const float gx = o.gravity[3 * gw + 0], gy = o.gravity[3 * gw + 1], gz = o.gravity[3 * gw + 2];
        // v1 = fma(eps, dv, fma((a + f w) + g, dt, v0))
        v1x = __fmaf_rn(p.xsph_eps, acc.dvx, __fmaf_rn(__fadd_rn(__fadd_rn(ax, fx), gx), dt, vi.x));
        v1y = __fmaf_rn(p.xsph_eps, acc.dvy, __fmaf_rn(__fadd_rn(__fadd_rn(ay, fy), gy), dt, vi.y));
        v1z = __fmaf_rn(p.xsph_eps, acc.dvz, __fmaf_rn(__fadd_rn(__fadd_rn(az, fz), gz), dt, vi.z));
    }
    const float vm = __fsqrt_rn(__fmaf_rn(v1z, v1z, __fmaf_rn(v1y, v1y, __fmul_rn(v1x, v1x))));
    if (vm > p.v_max) {
        const float s = __fdiv_rn(p.v_max, vm);
        v1x = __fmul_rn(v1x, s);
        v1y = __fmul_rn(v1y, s);
        v1z = __fmul_rn(v1z, s);
    }
    float x1x = __fmaf_rn(v1x, dt, xi.x), x1y = __fmaf_rn(v1y, dt, xi.y), x1z = __fmaf_rn(v1z, dt, xi.z);
    if (dynamic && p.use_box) {
        if (x1x < p.box_lo[0]) { x1x = p.box_lo[0]; v1x = fmaxf(v1x, 0.f); }
        if (x1x > p.box_hi[0]) { x1x = p.box_hi[0]; v1x = fminf(v1x, 0.f); }
        if (x1y < p.box_lo[1]) { x1y = p.box_lo[1]; v1y = fmaxf(v1y, 0.f); }
        if (x1y > p.box_hi[1]) { x1y = p.box_hi[1]; v1y = fminf(v1y, 0.f); }
        if (x1z < p.box_lo[2]) { x1z = p.box_lo[2]; v1z = fmaxf(v1z, 0.f); }
        if (x1z > p.box_hi[2]) { x1z = p.box_hi[2]; v1z = fminf(v1z, 0.f); }
    }
    if (o.status && !(isfinite(x1x) && isfinite(x1y) && isfinite(x1z) && isfinite(v1x) && isfinite(v1y) &&
                      isfinite(v1z)))
        atomicOr(o.status, (unsigned)NSPH_STATUS_NONFINITE_OUTPUT);
    store_row(o.x_out + 3 * i, x1x, x1y, x1z);
    store_row(o.v_out + 3 * i, v1x, v1y, v1z);
}

// ---- the density pass of a small scene: eight lanes per particle -----------------
// A tile's warp is one long chain of dependent work (50,000 cycles and more),
// which nothing hides while there are only a few warps per SM. Here the
// candidates of a particle's query box, its rows' runs one after another, are
// dealt to eight lanes in equal stretches: each tests its own into bit marks, a
// prefix sum over the lanes gives each one's place in the list, the lanes
// evaluate their neighbours' kernel values into shared memory at those places,
// and the sum over them runs in order. Same sets, order and roundings as the
// general scan, which takes a particle whose box has clamped cells, wraps in
// x, has more than 16 rows or 512 candidates, or whose list overflows.
constexpr int kOctetThreads = 128;
constexpr int kOctetParticles = kOctetThreads / 8;
// Density pass on a B200: 14 us instead of 28 at 1,000 to 4,096 particles, 21
// and 30 at 15,625, 29 and 29 at 24,389, 36 and 34 at 32,768, 157 and 70 at
// 219k (it issues three times the instructions); hence kOctetMax.
constexpr int kOctetMax = 16384;

struct OctetSmem {
    float2 terms[kNbrSlots + 1];  // (m, W) by place in the list
    int off[17];                  // candidate t of row r is at sorted position t + off[r]
    int upto[17];                 //   for t < upto[r] (the last entry ends every row)
};

template <bool Fast>
__device__ __forceinline__ int octet_neighbors(const GridDev& g, const float4* __restrict__ xs,
                                               const nsph_sph_params& p, float4 xi, bool active,
                                               int4* __restrict__ nbr, int n, int k, OctetSmem& sm, float& rho_out)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int sub = threadIdx.x & 7;
    int xl, xh, yl, yh, zl, zh;
    bool general = !active;
    box_axis_regular(xi.x, p.h, g.inv, g.dx, xl, xh, general);
    box_axis_regular(xi.y, p.h, g.inv, g.dy, yl, yh, general);
    box_axis_regular(xi.z, p.h, g.inv, g.dz, zl, zh, general);
    const int nx = xh - xl + 1, ny = yh - yl + 1;
    const int cx = general ? 0 : wrap_cell(xl, g.dx);
    general = general || cx + nx > g.dx || (long long)ny * (zh - zl + 1) > 16;
    const int rows = general ? 0 : ny * (zh - zl + 1);
    // rows sub and sub + 8: their runs, and the candidates up to each
    int lo[2] = {0, 0}, num[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = sub + 8 * h;
        if (row < rows) {
            const int iz = ny == 3 ? (row * 0x5556) >> 16 : row / ny, iy = row - iz * ny;
            const int2* cell = g.ranges + (wrap_cell(zl + iz, g.dz) * g.dy + wrap_cell(yl + iy, g.dy)) * g.dx + cx;
            int first = 0x7fffffff, end = 0;
#pragma unroll 3
            for (int c = 0; c < nx; ++c) {
                const int2 se = __ldg(cell + c);
                if (se.y > se.x && in_bounds(se.x >= 0 && se.y <= g.n)) {
                    first = min(first, se.x);
                    end = max(end, se.y);
                }
            }
            lo[h] = first;
            num[h] = max(end - first, 0);
        }
    }
    int cands = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int inc = num[h];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int y = __shfl_up_sync(kAll, inc, o, 8);
            if (sub >= o) inc += y;
        }
        const int row = sub + 8 * h;
        if (row < rows) {
            sm.off[row] = lo[h] - (cands + inc - num[h]);
            sm.upto[row] = cands + inc;
        }
        cands += __shfl_sync(kAll, inc, 7, 8);
    }
    if (sub == 0) sm.upto[rows] = 0x7fffffff;
    __syncwarp();
    const int each = (cands + 7) >> 3;  // candidates per lane
    general = general || each > 64;
    const int t0 = sub * each, t1 = general ? t0 : min(t0 + each, cands);
    // the row of candidate t0 (rows without candidates are passed over)
    int r0 = 0;
    if (t0 < t1)
        while (sm.upto[r0] <= t0) ++r0;
    unsigned marks[2] = {0u, 0u};
    {
        int r = r0, next = sm.upto[r], off = sm.off[r];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            unsigned bits = 0u;
            const int end = min(t1, t0 + 32 * (c + 1));
            for (int t = t0 + 32 * c; t < end; t += 4) {
                float4 xj[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int tu = min(t + u, end - 1);
                    if (tu >= next) {
                        do {
                            ++r;
                            next = sm.upto[r];
                        } while (tu >= next);
                        off = sm.off[r];
                    }
                    xj[u] = __ldg(xs + tu + off);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float dx, dy, dz;
                    const bool hit = dist2(xi, xj[u], dx, dy, dz) < p.h2 && !mirror_inactive(xj[u]) && t + u < end;
                    bits |= (hit ? 1u : 0u) << (t - t0 - 32 * c + u);
                }
            }
            marks[c] = bits;
        }
    }
    const int mine = __popc(marks[0]) + __popc(marks[1]);
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int y = __shfl_up_sync(kAll, inc, o, 8);
        if (sub >= o) inc += y;
    }
    const int total = __shfl_sync(kAll, inc, 7, 8);
    general = general || total > kNbrSlots;
    if (!general) {
        int at = inc - mine;
        int r = r0, next = sm.upto[r], off = sm.off[r];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            unsigned bits = marks[c];
            while (bits) {
                const int t = t0 + 32 * c + __ffs(bits) - 1;
                bits &= bits - 1u;
                if (t >= next) {
                    do {
                        ++r;
                        next = sm.upto[r];
                    } while (t >= next);
                    off = sm.off[r];
                }
                const int j = t + off;
                const float4 xj = __ldg(xs + j);
                float dx, dy, dz;
                const float r2 = dist2(xi, xj, dx, dy, dz);
                sm.terms[at] = make_float2(xj.w, Fast ? wterm_fast(r2, p) : wterm(r2, p));
                reinterpret_cast<int*>(nbr + (size_t)(at >> 2) * n + k)[at & 3] = j;
                ++at;
            }
        }
        // the rest of the last group is the particle itself
        const int pad = total + sub;
        if (sub < 3 && (total & 3) && (pad >> 2) == (total >> 2))
            reinterpret_cast<int*>(nbr + (size_t)(pad >> 2) * n + k)[pad & 3] = k;
    }
    __syncwarp();
    float rho = 0.f;
    if (!general) {
#pragma unroll 4
        for (int t = 0; t < total; ++t) {
            const float2 mw = sm.terms[t];
            rho = __fmaf_rn(mw.x, mw.y, rho);
        }
    }
    rho_out = rho;
    return general ? -1 : total;
}

// ---- the plain step's passes on neighbour lists ----------------------------------
template <bool Fast>
__global__ void __launch_bounds__(kSphThreads, kDensityBlocks) k_density_list(
    const __grid_constant__ GridDev g, const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
    const __grid_constant__ nsph_sph_params p, float2* __restrict__ rp,
    int4* __restrict__ nbr, int* __restrict__ ncnt, const ForceRec fr, unsigned* __restrict__ status)
{
    launch_entry();
    extern __shared__ TileSmem tile_smem[];
    TileSmem& sm = tile_smem[threadIdx.x >> 5];
    // whole warps: lanes past n take part as non-members
    for (int k0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); k0 < n; k0 += gridDim.x * blockDim.x) {
        const int k = k0 + (threadIdx.x & 31);
        const bool live = k < n;
        float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
        bool active = false;
        if (live) {
            xi = xs[k];
            active = (__float_as_int(vs[k].w) & kAttrActive) != 0;
        }
        float rho;
        int cnt = tile_neighbors<Fast, false>(g, xs, p, 0, xi, active, nbr, n, k, sm, rho);
        if (active) {
            if (cnt < 0) cnt = scan_general<Fast>(&g, xs, &p, xi, nbr, n, k, &rho);
            ncnt[k] = cnt;
            if (cnt > kNbrSlots && fr.overflow) atomicOr(fr.overflow, 1u);
            density_finish<Fast>(k, xi, vs[k], rho, p, rp, fr, status);
        } else if (live) {
            rp[k] = make_float2(0.f, 0.f);
            fr.rec[2 * (size_t)k] = xi;  // (marked inactive)
            ncnt[k] = 0;
        }
    }
}

template <bool Fast>
__global__ void __launch_bounds__(kOctetThreads) k_density_octet(
    const __grid_constant__ GridDev g, const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
    const __grid_constant__ nsph_sph_params p, float2* __restrict__ rp,
    int4* __restrict__ nbr, int* __restrict__ ncnt, const ForceRec fr, unsigned* __restrict__ status)
{
    launch_entry();
    __shared__ OctetSmem octets[kOctetParticles];
    const int kt = blockIdx.x * kOctetParticles + threadIdx.x / 8, k = min(kt, n - 1);
    const float4 xi = xs[k], vi = vs[k];
    const bool active = kt < n && (__float_as_int(vi.w) & kAttrActive) != 0;
    float rho;
    int cnt = octet_neighbors<Fast>(g, xs, p, xi, active, nbr, n, k, octets[threadIdx.x / 8], rho);
    if ((threadIdx.x & 7) != 0 || kt >= n) return;
    if (active) {
        if (cnt < 0) cnt = scan_general<Fast>(&g, xs, &p, xi, nbr, n, k, &rho);
        ncnt[k] = cnt;
        if (cnt > kNbrSlots && fr.overflow) atomicOr(fr.overflow, 1u);
        density_finish<Fast>(k, xi, vi, rho, p, rp, fr, status);
    } else {
        rp[k] = make_float2(0.f, 0.f);
        fr.rec[2 * (size_t)k] = xi;  // (marked inactive)
        ncnt[k] = 0;
    }
}

// pressure and XSPH sums of particle k over its list, in order, by whole
// groups (the last one is filled with the particle itself): the loads of two
// neighbours are issued together, those of the next group's indices ahead. A
// particle whose list overflowed re-tests its candidates.
template <bool Fast, class P>
__device__ __forceinline__ void force_from_list(const GridDev& g, const ForceRec& fr, const int4* __restrict__ nbr,
                                                int cnt, int n, int k, float4 xi, float4 vi, float h, float h2,
                                                const P& p, ForceAcc& acc)
{
    const float pr2_i = fr.pr2[k];
    auto term = [&](const Neighbour& o, float pr2_j) {
        if (Fast)
            force_term_fast(o.x, o.v, pr2_j, xi, vi, pr2_i, p, acc);
        else
            force_term_data(o.x, o.v, pr2_j, xi, vi, pr2_i, p, acc);
    };
    auto checked = [&](int j) { return in_bounds(j >= 0 && j < n) ? j : 0; };
    if (cnt <= kNbrSlots) {
        const int4* a = nbr + k;
        int4 next = cnt > 0 ? __ldg(a) : make_int4(k, k, k, k);
#pragma unroll 1
        for (int t = 0; t < cnt; t += 4) {
            const int4 gr = next;
            a += n;
            if (t + 4 < cnt) next = __ldg(a);
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                const int j0 = checked(group_item(gr, u)), j1 = checked(group_item(gr, u + 1));
                const Neighbour o0 = load_neighbour(fr.rec, j0);
                const float p0 = __ldg(fr.pr2 + j0);
                const Neighbour o1 = load_neighbour(fr.rec, j1);
                const float p1 = __ldg(fr.pr2 + j1);
                if (j0 != k) term(o0, p0);
                if (j1 != k) term(o1, p1);
            }
        }
    } else {
        for_each_run(g, xi.x, xi.y, xi.z, h, [&](int lo, int hi) {
            for (int j = lo; j < hi; ++j) {
                const Neighbour o = load_neighbour(fr.rec, j);
                float dx, dy, dz;
                if (dist2(xi, o.x, dx, dy, dz) < h2 && j != k && !mirror_inactive(o.x)) term(o, __ldg(fr.pr2 + j));
            }
        });
    }
}

template <bool Fast>
__global__ void __launch_bounds__(kSphThreads, 4) k_force_list(GridDev g, const float4* __restrict__ xs,
                                                               const float4* __restrict__ vs, const ForceRec fr,
                                                               const float2* __restrict__ rp, int n,
                                                               const __grid_constant__ nsph_sph_params p,
                                                               const int4* __restrict__ nbr,
                                                               const int* __restrict__ ncnt, const StepOut o)
{
    launch_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 xi = xs[k], vi = vs[k];
        const int attr = __float_as_int(vi.w);
        ForceAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (attr & kAttrActive) force_from_list<Fast>(g, fr, nbr, ncnt[k], n, k, xi, vi, p.h, p.h2, p, acc);
        if (o.acc_sorted) {  // the force sums, for the adjoint's segment tape
            o.acc_sorted[2 * (size_t)k] = make_float4(acc.ax, acc.ay, acc.az, 0.f);
            o.acc_sorted[2 * (size_t)k + 1] = make_float4(acc.dvx, acc.dvy, acc.dvz, 0.f);
        }
        integrate_out((size_t)g.ids[k], xi, vi, attr, rp[k], acc, p, p.dt, o);
    }
}

// The force pass of a small scene: four lanes per particle. Lane u of a
// particle evaluates the factors of item u of each list group; the factors
// cross through shared memory, and lanes 0 .. 2 accumulate the x, y and z sums
// of the group's four terms in order, so every rounding is k_force_list's.
// It spends about 1.4 times the instructions, but a particle's chain of
// dependent work is a third as long and there are four times the warps, which
// is what bounds scenes that do not fill the SMs. Whole step with it and
// without on a B200: 25 and 31 us at 2,197 particles, 54 and 59 at 24,389, 66
// and 64 at 32,768, 76 and 70 at 64,000 (a 64k rollout with its gradient, whose
// pair passes follow the same rule: 4.25 and 3.87 ms); hence kQuadMax.
constexpr int kQuadThreads = 256;
constexpr int kQuadMax = 24576;

__global__ void __launch_bounds__(kQuadThreads, 4) k_force_quad(const __grid_constant__ GridDev g,
                                                                const float4* __restrict__ xs,
                                                                const float4* __restrict__ vs,
                                                                const ForceRec fr, const float2* __restrict__ rp,
                                                                int n, const __grid_constant__ nsph_sph_params p,
                                                                const int4* __restrict__ nbr,
                                                                const int* __restrict__ ncnt, const StepOut o)
{
    launch_entry();
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ __align__(16) float cross[kQuadThreads / 32][2][8][32];  // [parity][factor][lane]
    const int lane = threadIdx.x & 31, u = lane & 3;
    const int kt = (blockIdx.x * kQuadThreads + threadIdx.x) >> 2;
    const int k = min(kt, n - 1);
    const float4 xi = xs[k], vi = vs[k];
    const int attr = __float_as_int(vi.w);
    const bool active = kt < n && (attr & kAttrActive);
    const int cnt = active ? ncnt[k] : 0;
    const float pr2_i = fr.pr2[k];
    const int groups = cnt <= kNbrSlots ? (cnt + 3) >> 2 : 0;  // an overflowed list: see below
    const int most = __reduce_max_sync(kAll, groups);
    const int* item = reinterpret_cast<const int*>(nbr + k) + u;
    auto load = [&](int gi) {
        const int j = gi < groups ? __ldg(item + 4 * (size_t)gi * n) : k;
        return in_bounds(j >= 0 && j < n) ? j : 0;
    };
    const int axis = min(u, 2);
    float a = 0.f, dv = 0.f;
    int j = load(0), jn = load(1);
    Neighbour oj = load_neighbour(fr.rec, j);
    float pj = __ldg(fr.pr2 + j);
    for (int gi = 0; gi < most; ++gi) {
        // the next group's data and the index after it go out first
        const int j1 = jn;
        const Neighbour on = load_neighbour(fr.rec, j1);
        const float pn = __ldg(fr.pr2 + j1);
        jn = load(gi + 2);
        const unsigned live = __ballot_sync(kAll, j != k);  // (fillers are the particle itself)
        const ForceTerm t = force_factors(oj.x, oj.v, pj, xi, vi, pr2_i, p);
        float(*c)[32] = cross[threadIdx.x >> 5][gi & 1];
        c[0][lane] = t.dx;
        c[1][lane] = t.dy;
        c[2][lane] = t.dz;
        c[3][lane] = -t.s;
        c[4][lane] = t.ux;
        c[5][lane] = t.uy;
        c[6][lane] = t.uz;
        c[7][lane] = t.c;
        __syncwarp();
        const int row = lane & ~3;
        const float4 d = *reinterpret_cast<const float4*>(&c[axis][row]);
        const float4 s = *reinterpret_cast<const float4*>(&c[3][row]);
        const float4 w = *reinterpret_cast<const float4*>(&c[4 + axis][row]);
        const float4 m = *reinterpret_cast<const float4*>(&c[7][row]);
        const unsigned in = (live >> row) & 15u;  // the group's items that are neighbours
        auto add = [&](unsigned bit, float sv, float dvv, float mv, float wv) {
            if (in & bit) {
                a = __fmaf_rn(sv, dvv, a);
                dv = __fmaf_rn(mv, wv, dv);
            }
        };
        add(1u, s.x, d.x, m.x, w.x);
        add(2u, s.y, d.y, m.y, w.y);
        add(4u, s.z, d.z, m.z, w.z);
        add(8u, s.w, d.w, m.w, w.w);
        j = j1;
        oj = on;
        pj = pn;
    }
    ForceAcc acc;
    acc.ax = a;
    acc.dvx = dv;
    acc.ay = __shfl_down_sync(kAll, a, 1, 4);
    acc.dvy = __shfl_down_sync(kAll, dv, 1, 4);
    acc.az = __shfl_down_sync(kAll, a, 2, 4);
    acc.dvz = __shfl_down_sync(kAll, dv, 2, 4);
    if (u != 0 || kt >= n) return;
    if (cnt > kNbrSlots) {
        acc = ForceAcc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        force_from_list<false>(g, fr, nbr, cnt, n, k, xi, vi, p.h, p.h2, p, acc);
    }
    if (o.acc_sorted) {  // the force sums, for the adjoint's segment tape
        o.acc_sorted[2 * (size_t)k] = make_float4(acc.ax, acc.ay, acc.az, 0.f);
        o.acc_sorted[2 * (size_t)k + 1] = make_float4(acc.dvx, acc.dvy, acc.dvz, 0.f);
    }
    integrate_out((size_t)g.ids[k], xi, vi, attr, rp[k], acc, p, p.dt, o);
}

// ---- batched worlds ------------------------------------------------------------
// One launch per pass covers every world. The kernels are persistent: a grid
// of (SMs x resident blocks) threads strides over all particles, whose work
// is similar whatever their world, so no work queue is needed. A particle's
// world (attr >> kAttrGravShift, clamped at the gather) selects its grid
// (dims, 1/cell width, cell-table offset) and its parameter block; its
// neighbours are found and summed exactly as in the single-world kernels, in
// its own world's query order.
__device__ __forceinline__ GridDev world_grid(const WorldCells& c, const int2* __restrict__ ranges,
                                              const int* __restrict__ ids, int n)
{
    return GridDev{c.dx, c.dy, c.dz, c.inv, ranges + c.off, ids, n};
}

// scan_general of a particle of world w
__device__ __noinline__ int scan_general_world(const WorldCells* wc, const nsph_sph_params* wp, const int2* ranges,
                                               const int* ids, int w, const float4* xs, float4 xi, int4* nbr, int n,
                                               int k, float* rho)
{
    const GridDev g = world_grid(wc[w], ranges, ids, n);
    const int cnt = neighbor_list(g, xs, wp[w], xi, nbr, n, k);
    *rho = density_from_list<false>(g, xs, wp[w], xi, nbr, cnt, n, k);
    return cnt;
}

__global__ void __launch_bounds__(kSphThreads, kDensityBlocks) k_density_worlds(
    const WorldCells* __restrict__ wc, const nsph_sph_params* __restrict__ wp, const int2* __restrict__ ranges,
    const int* __restrict__ ids, const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
    float2* __restrict__ rp, int4* __restrict__ nbr, int* __restrict__ ncnt,
    const ForceRec fr, unsigned* __restrict__ status)
{
    launch_entry();
    extern __shared__ TileSmem tile_smem[];
    TileSmem& sm = tile_smem[threadIdx.x >> 5];
    for (int k0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); k0 < n; k0 += gridDim.x * blockDim.x) {
        const int k = k0 + (threadIdx.x & 31);
        const bool live = k < n;
        float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
        int attr = 0;
        if (live) {
            xi = xs[k];
            attr = __float_as_int(vs[k].w);
        }
        const bool active = (attr & kAttrActive) != 0;
        const int w = attr >> kAttrGravShift;
        const nsph_sph_params p = wp[w];  // a copy: its fields stay in registers across the candidate loop
        const GridDev g = world_grid(wc[w], ranges, ids, n);
        float rho;
        int cnt = tile_neighbors<false, true>(g, xs, p, w, xi, active, nbr, n, k, sm, rho);
        if (active) {
            if (cnt < 0) cnt = scan_general_world(wc, wp, ranges, ids, w, xs, xi, nbr, n, k, &rho);
            ncnt[k] = cnt;
            density_finish(k, xi, vs[k], rho, p, rp, fr, status);
        } else if (live) {
            rp[k] = make_float2(0.f, 0.f);
            fr.rec[2 * (size_t)k] = xi;  // (marked inactive)
            ncnt[k] = 0;
        }
    }
}

__global__ void __launch_bounds__(kOctetThreads) k_density_octet_worlds(
    const WorldCells* __restrict__ wc, const nsph_sph_params* __restrict__ wp, const int2* __restrict__ ranges,
    const int* __restrict__ ids, const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
    float2* __restrict__ rp, int4* __restrict__ nbr, int* __restrict__ ncnt,
    const ForceRec fr, unsigned* __restrict__ status)
{
    launch_entry();
    __shared__ OctetSmem octets[kOctetParticles];
    const int kt = blockIdx.x * kOctetParticles + threadIdx.x / 8, k = min(kt, n - 1);
    const float4 xi = xs[k], vi = vs[k];
    const int attr = __float_as_int(vi.w), w = attr >> kAttrGravShift;
    const bool active = kt < n && (attr & kAttrActive) != 0;
    const nsph_sph_params& p = wp[w];
    const GridDev g = world_grid(wc[w], ranges, ids, n);
    float rho;
    int cnt = octet_neighbors<false>(g, xs, p, xi, active, nbr, n, k, octets[threadIdx.x / 8], rho);
    if ((threadIdx.x & 7) != 0 || kt >= n) return;
    if (active) {
        if (cnt < 0) cnt = scan_general_world(wc, wp, ranges, ids, w, xs, xi, nbr, n, k, &rho);
        ncnt[k] = cnt;
        density_finish(k, xi, vi, rho, p, rp, fr, status);
    } else {
        rp[k] = make_float2(0.f, 0.f);
        fr.rec[2 * (size_t)k] = xi;  // (marked inactive)
        ncnt[k] = 0;
    }
}

// Bounded to 64 registers: 2.39 -> 2.11 ms per pass on worlds_4096 against
// 80 at three blocks per SM (same box, back to back).
__global__ void __launch_bounds__(kSphThreads, 4) k_force_worlds(const WorldCells* __restrict__ wc,
                                                                 const nsph_sph_params* __restrict__ wp,
                                                                 const int2* __restrict__ ranges,
                                                                 const int* __restrict__ ids,
                                                                 const float4* __restrict__ xs,
                                                                 const float4* __restrict__ vs, const ForceRec fr,
                                                                 const float2* __restrict__ rp, int n, float dt,
                                                                 const int4* __restrict__ nbr,
                                                                 const int* __restrict__ ncnt, const StepOut o)
{
    launch_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 xi = xs[k], vi = vs[k];
        const int attr = __float_as_int(vi.w);
        const int w = attr >> kAttrGravShift;
        const nsph_sph_params& p = wp[w];
        const GridDev g = world_grid(wc[w], ranges, ids, n);
        ForceAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (attr & kAttrActive) force_from_list<false>(g, fr, nbr, ncnt[k], n, k, xi, vi, p.h, p.h2, ForceConst(p), acc);
        integrate_out((size_t)ids[k], xi, vi, attr, rp[k], acc, p, dt, o);
    }
}

__global__ void k_neighbors_worlds(const WorldCells* __restrict__ wc, const nsph_sph_params* __restrict__ wp,
                                   const int2* __restrict__ ranges, const int* __restrict__ ids,
                                   const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
                                   int* __restrict__ counts, const long long* __restrict__ offsets,
                                   int* __restrict__ out)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = ids[k];
    const float4 xi = xs[k];
    const int attr = __float_as_int(vs[k].w);
    long long o = out ? offsets[i] : 0;
    int c = 0;
    if (attr & kAttrActive) {
        const int w = attr >> kAttrGravShift;
        const float h = wp[w].h, h2 = wp[w].h2;
        const GridDev g = world_grid(wc[w], ranges, ids, n);
        for_each_candidate(g, xi.x, xi.y, xi.z, h, [&](int j) {
            float dx, dy, dz;
            if (dist2(xi, xs[j], dx, dy, dz) < h2 && (__float_as_int(vs[j].w) & kAttrActive)) {
                if (out) out[o++] = ids[j];
                ++c;
            }
        });
    }
    if (!out) counts[i] = c;
}

// ---- neighbour lists of the last build (parity export) ----------------------
__global__ void k_neighbors(GridDev g, const float4* __restrict__ xs, const float4* __restrict__ vs, int n,
                            nsph_sph_params p, int* __restrict__ counts, const long long* __restrict__ offsets,
                            int* __restrict__ out)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = g.ids[k];
    const float4 xi = xs[k];
    const bool active = (__float_as_int(vs[k].w) & kAttrActive) != 0;
    long long o = out ? offsets[i] : 0;
    int c = 0;
    if (active) {
        for_each_candidate(g, xi.x, xi.y, xi.z, p.h, [&](int j) {
            const float4 xj = xs[j];
            float dx, dy, dz;
            if (dist2(xi, xj, dx, dy, dz) < p.h2 && (__float_as_int(vs[j].w) & kAttrActive)) {
                if (out) out[o++] = g.ids[j];
                ++c;
            }
        });
    }
    if (!out) counts[i] = c;
}

// The part of a step's grid that its reverse reads, into the segment tape: the
// sorted ids and, only when a list of the step overflowed (its particle's
// neighbours are then found through the grid again), the cell table.
__global__ void k_tape_copy(const GridDev g, long long ncells, int n, const unsigned* __restrict__ overflow,
                            int* __restrict__ ids, int2* __restrict__ ranges)
{
    launch_entry();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long k = t; k < n; k += step) ids[k] = g.ids[k];
    if (*overflow)
        for (long long c = t; c < ncells; c += step) ranges[c] = g.ranges[c];
}

// ==========================================================================
// Adjoint of the step (reverse mode): given the adjoints of x_{n+1}, v_{n+1}
// (and optionally of rho), the adjoints of x_n, v_n, f_ext and of the EOS
// stiffness B. The neighbour set is held fixed (it is piecewise constant in
// x; W and dW/dr vanish at r = h, so the step is C1 across its changes); the
// pressure clamp, |v| clamp and box are differentiated on the side the
// forward step took, which the reverse pass recomputes bit for bit.
//
// The forward step sums pair terms into particle i only (a gather), so its
// transpose scatters into both particles of a pair. Because the neighbour
// relation is symmetric (the fp32 r2 of (i, j) and (j, i) are equal) every
// scatter is rewritten as a gather over the same neighbour lists, with no
// atomics, and each particle's adjoint is written by one thread:
//   local   G_i = adj(a_i), D_i = adj(dv_i), and the integrate reverse
//   pair    adj(p_i/rho_i^2) = sum_j F_ij (Z_ij . d_ij)
//           adj(m_i/rho_i)   = sum_j W_ij D_j . (v_i - v_j)
//           adj(x_i)        += sum_j S_ij [F Z + (F'/r)(d.Z) d]
//                              + F ((v_j - v_i) . Y_ij) d
//           adj(v_i)        -= sum_j W_ij Y_ij
//           with Z = m_i G_j - m_j G_i, Y = mor_j D_i - mor_i D_j,
//           S = p_i/rho_i^2 + p_j/rho_j^2, d = x_i - x_j, F = (dW/dr)/r
//           then adj(rho_i) through the EOS and the m/rho, p/rho^2 factors
//   density adj(x_i)        += sum_j F_ij (adj(rho_i) m_j + adj(rho_j) m_i) d_ij
// ==========================================================================

// (dF/dr)/r of F = (dW/dr)/r: near 3 c_near / (h r); far -c_far t (2/(h r^2) + t/r^3)
__device__ __forceinline__ float kernel_df_over_r(float q, float inv_r, const nsph_sph_params& p)
{
    const float t = 1.f - q;
    if (q <= 0.5f) return 3.f * p.c_near * p.inv_h * inv_r;
    if (q < 1.f) return -p.c_far * t * (2.f * p.inv_h + t * inv_r) * inv_r * inv_r;
    return 0.f;
}

// visit(j) for every neighbour j != k of sorted particle k, in query order,
// from the density pass's neighbour list (re-testing its candidates when the
// list overflowed). With kLanes = 4, lane `sub` of the particle's four visits
// item `sub` of each list group (or every fourth candidate).
template <int kLanes, class V>
__device__ __forceinline__ void for_each_neighbor(const GridDev& g, const float4* __restrict__ xs,
                                                  const int4* __restrict__ nbr, int cnt, int n, int k, int sub,
                                                  float4 xi, const nsph_sph_params& p, V&& visit)
{
    if (cnt <= kNbrSlots) {
        if constexpr (kLanes == 1) {
            for_each_listed<true>(nbr, n, k, cnt, [&](int j) {
                if (j != k) visit(j);
            });
        } else {
            const int* item = reinterpret_cast<const int*>(nbr + k) + sub;
            const size_t stride = 4 * (size_t)n;
            int next = sub < cnt ? __ldg(item) : k;
            for (int t = sub; t < cnt; t += 4) {
                const int j = in_bounds(next >= 0 && next < n) ? next : k;
                item += stride;
                if (t + 4 < cnt) next = __ldg(item);
                if (j != k) visit(j);
            }
        }
    } else {
        for_each_run(g, xi.x, xi.y, xi.z, p.h, [&](int lo, int hi) {
            for (int j = lo + sub; j < hi; j += kLanes) {
                float dx, dy, dz;
                const float4 xj = __ldg(xs + j);
                if (j != k && dist2(xi, xj, dx, dy, dz) < p.h2 && !mirror_inactive(xj)) visit(j);
            }
        });
    }
}

// the sum over a particle's lanes, in each of them (all of a warp's lanes call it)
template <int kLanes>
__device__ __forceinline__ float lanes_sum(float v)
{
#pragma unroll
    for (int o = 1; o < kLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct AdjIO {
    const float* x_out_adj;
    const float* v_out_adj;
    const float* rho_out_adj;
    float* x_in_adj;
    float* v_in_adj;
    float* f_ext_adj;
    const float* f_ext;
    const float* inv_mass;
    const float* gravity;
    float4* gd;    // sorted: adj(a), adj(dv) of particle k at 2k, 2k + 1
    float4* xv;    // sorted: the adjoints of x and v so far, at 2k, 2k + 1 (the particle arrays, in original
                   // order, are only read by the first pass and only written by the last one: adding to
                   // their scattered rows in place, where a line's rows belong to blocks on both dies,
                   // made each addition wait for the other die's L2)
    float* rho;    // sorted: adj(rho)
    float* bpart;  // per block: partial adj(B)
    const float4* acc;  // or null: the forward's sorted (a, 0), (dv, 0) (the segment tape), else recomputed
};

// reverse of integrate: recompute the forward particle update (bit for bit,
// so the clamp decisions are the forward's), then transpose it. The force
// sums a, dv are the forward's, stored (io.acc) or recomputed here.
__global__ void __launch_bounds__(kSphThreads, 2) k_adj_local(GridDev g, const float4* __restrict__ xs,
                                                              const float4* __restrict__ vs,
                                                              const ForceRec fr, int n,
                                                              const __grid_constant__ nsph_sph_params p,
                                                              const int4* __restrict__ nbr,
                                                              const int* __restrict__ ncnt, const AdjIO io)
{
    launch_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 xi = xs[k], vi = vs[k];
        const int attr = __float_as_int(vi.w);
        const size_t i = (size_t)g.ids[k];
        const Row3 xo = load_row(io.x_out_adj + 3 * i), vo = load_row(io.v_out_adj + 3 * i);
        const float xb1[3] = {xo.x, xo.y, xo.z}, vb1[3] = {vo.x, vo.y, vo.z};
        float fb[3] = {0.f, 0.f, 0.f};
        float4 gk = make_float4(0.f, 0.f, 0.f, 0.f), dk = gk;
        if (!(attr & kAttrActive)) {
            io.xv[2 * (size_t)k] = make_float4(xb1[0], xb1[1], xb1[2], 0.f);
            io.xv[2 * (size_t)k + 1] = make_float4(vb1[0], vb1[1], vb1[2], 0.f);
        } else {
            ForceAcc acc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (io.acc) {
                const float4 a = io.acc[2 * (size_t)k], d = io.acc[2 * (size_t)k + 1];
                acc = ForceAcc{a.x, a.y, a.z, d.x, d.y, d.z};
            } else {
                force_from_list<false>(g, fr, nbr, ncnt[k], n, k, xi, vi, p.h, p.h2, p, acc);
            }
            const bool dynamic = (attr & kAttrDynamic) != 0;
            float w = 0.f;
            float u[3] = {vi.x, vi.y, vi.z};
            if (dynamic) {  // the forward update of integrate_out, same rounding
                const int gw = attr >> kAttrGravShift;
                float fe[3] = {0.f, 0.f, 0.f};
                if (io.f_ext) {
                    w = io.inv_mass[i];
                    for (int c = 0; c < 3; ++c) fe[c] = __fmul_rn(io.f_ext[3 * i + c], w);
                }
                const float a[3] = {acc.ax, acc.ay, acc.az}, dv[3] = {acc.dvx, acc.dvy, acc.dvz};
                for (int c = 0; c < 3; ++c)
                    u[c] = __fmaf_rn(p.xsph_eps, dv[c],
                                     __fmaf_rn(__fadd_rn(__fadd_rn(a[c], fe[c]), io.gravity[3 * gw + c]), p.dt, u[c]));
            }
            const float vm = __fsqrt_rn(__fmaf_rn(u[2], u[2], __fmaf_rn(u[1], u[1], __fmul_rn(u[0], u[0]))));
            const bool vclamp = vm > p.v_max;
            const float s = vclamp ? __fdiv_rn(p.v_max, vm) : 1.f;
            const float xin[3] = {xi.x, xi.y, xi.z};
            float vcb[3], xpb[3];
            for (int c = 0; c < 3; ++c) {
                const float vc = vclamp ? __fmul_rn(u[c], s) : u[c];
                const float xp = __fmaf_rn(vc, p.dt, xin[c]);
                xpb[c] = xb1[c];
                vcb[c] = vb1[c];
                if (dynamic && p.use_box) {
                    if (xp < p.box_lo[c]) {  // x = lo, v = max(v, 0)
                        xpb[c] = 0.f;
                        if (vc < 0.f) vcb[c] = 0.f;
                    } else if (xp > p.box_hi[c]) {  // x = hi, v = min(v, 0)
                        xpb[c] = 0.f;
                        if (vc > 0.f) vcb[c] = 0.f;
                    }
                }
                vcb[c] += xpb[c] * p.dt;
            }
            float ub[3] = {vcb[0], vcb[1], vcb[2]};
            if (vclamp) {  // v = v_max u/|u|: adj(u) = (v_max/|u|)(adj(v) - u^ (u^ . adj(v)))
                const float inv = 1.f / vm;
                const float uh[3] = {u[0] * inv, u[1] * inv, u[2] * inv};
                const float dot = uh[0] * vcb[0] + uh[1] * vcb[1] + uh[2] * vcb[2];
                for (int c = 0; c < 3; ++c) ub[c] = s * (vcb[c] - uh[c] * dot);
            }
            io.xv[2 * (size_t)k] = make_float4(xpb[0], xpb[1], xpb[2], 0.f);
            io.xv[2 * (size_t)k + 1] = make_float4(ub[0], ub[1], ub[2], 0.f);
            if (dynamic) {
                gk = make_float4(ub[0] * p.dt, ub[1] * p.dt, ub[2] * p.dt, 0.f);
                dk = make_float4(ub[0] * p.xsph_eps, ub[1] * p.xsph_eps, ub[2] * p.xsph_eps, 0.f);
                if (io.f_ext)
                    for (int c = 0; c < 3; ++c) fb[c] = ub[c] * p.dt * w;
            }
        }
        if (io.f_ext_adj)
            for (int c = 0; c < 3; ++c) io.f_ext_adj[3 * i + c] += fb[c];
        io.gd[2 * (size_t)k] = gk;
        io.gd[2 * (size_t)k + 1] = dk;
    }
}

// sum of v over the block, valid in thread 0 (a second call needs a
// __syncthreads() in between: the shared partials are reused)
__device__ __forceinline__ float block_sum(float v)
{
    __shared__ float part[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) part[warp] = v;
    __syncthreads();
    v = 0.f;
    if (warp == 0) {
        v = lane < (int)(blockDim.x >> 5) ? part[lane] : 0.f;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;
}

// gather of the transposed pressure and XSPH terms, then adj(rho) through
// the EOS; per-block partial sums of adj(B). kLanes = 4 gives each particle
// four lanes, for scenes that do not fill the SMs with one thread each.
template <int kLanes>
__global__ void __launch_bounds__(kSphThreads, 2) k_adj_pair(GridDev g, const float4* __restrict__ xs,
                                                             const float4* __restrict__ vs,
                                                             const ForceRec fr,
                                                             const float2* __restrict__ rp, int n,
                                                             const __grid_constant__ nsph_sph_params p,
                                                             const int4* __restrict__ nbr,
                                                             const int* __restrict__ ncnt, const AdjIO io)
{
    launch_entry();
    float bsum = 0.f;
    const int sub = threadIdx.x & (kLanes - 1);
    const int step = gridDim.x * blockDim.x / kLanes;
    // whole warps: the lanes of a particle sum together
    for (int k0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / kLanes; k0 < n; k0 += step) {
        const int kt = k0 + (threadIdx.x & 31) / kLanes, k = min(kt, n - 1);
        const float4 xi = xs[k], vi = vs[k];
        const size_t i = (size_t)g.ids[k];
        const bool active = kt < n && (__float_as_int(vi.w) & kAttrActive);
        const float2 ak = make_float2(fr.rec[2 * (size_t)k + 1].w, fr.pr2[k]);  // (m/rho, p/rho^2)
        const float4 gk = io.gd[2 * (size_t)k], dk = io.gd[2 * (size_t)k + 1];
        const float mk = xi.w;
        float pr2b = 0.f, morb = 0.f;
        float xb[3] = {0.f, 0.f, 0.f}, vb[3] = {0.f, 0.f, 0.f};
        for_each_neighbor<kLanes>(g, xs, nbr, active ? ncnt[k] : 0, n, k, sub, xi, p, [&](int j) {
            const Neighbour o = load_neighbour(fr.rec, j), od = load_neighbour(io.gd, j);
            const float4 xj = o.x, vj = o.v, gj = od.x, dj = od.v;
            const float2 aj = make_float2(vj.w, __ldg(fr.pr2 + j));
            float dx, dy, dz;
            const float r2 = dist2(xi, xj, dx, dy, dz);
            const float r = __fsqrt_rn(r2);
            const float q = r * p.inv_h;
            const float w = kernel_w(q, p);
            const float yx = aj.x * dk.x - ak.x * dj.x, yy = aj.x * dk.y - ak.x * dj.y, yz = aj.x * dk.z - ak.x * dj.z;
            const float rvx = vj.x - vi.x, rvy = vj.y - vi.y, rvz = vj.z - vi.z;
            if (r2 > 0.f) {
                const float inv_r = 1.f / r;
                const float f = kernel_f(q, inv_r, p);
                const float dfr = kernel_df_over_r(q, inv_r, p);
                const float zx = mk * gj.x - xj.w * gk.x, zy = mk * gj.y - xj.w * gk.y, zz = mk * gj.z - xj.w * gk.z;
                const float zd = zx * dx + zy * dy + zz * dz;
                pr2b += f * zd;
                const float sp = ak.y + aj.y;
                const float cx = sp * dfr * zd + f * (rvx * yx + rvy * yy + rvz * yz);
                xb[0] += sp * f * zx + cx * dx;
                xb[1] += sp * f * zy + cx * dy;
                xb[2] += sp * f * zz + cx * dz;
            }
            vb[0] -= w * yx;
            vb[1] -= w * yy;
            vb[2] -= w * yz;
            morb -= w * (dj.x * rvx + dj.y * rvy + dj.z * rvz);
        });
        if constexpr (kLanes > 1) {
            pr2b = lanes_sum<kLanes>(pr2b);
            morb = lanes_sum<kLanes>(morb);
            for (int c = 0; c < 3; ++c) {
                xb[c] = lanes_sum<kLanes>(xb[c]);
                vb[c] = lanes_sum<kLanes>(vb[c]);
            }
        }
        if (sub != 0 || kt >= n) continue;
        const float4 x0 = io.xv[2 * (size_t)k], v0 = io.xv[2 * (size_t)k + 1];
        store_row(io.v_in_adj + 3 * i, active ? v0.x + vb[0] : v0.x, active ? v0.y + vb[1] : v0.y,
                  active ? v0.z + vb[2] : v0.z);
        if (!active) {
            io.rho[k] = 0.f;
            continue;
        }
        io.xv[2 * (size_t)k] = make_float4(x0.x + xb[0], x0.y + xb[1], x0.z + xb[2], 0.f);
        // adj(rho) from p/rho^2 (through the EOS) and m/rho
        const float2 rpk = rp[k];
        float rb = io.rho_out_adj ? io.rho_out_adj[i] : 0.f;
        if (rpk.x > 0.f) {
            const float rho = rpk.x, ratio = __fmul_rn(rho, p.inv_rho0);
            float pw1 = 1.f;  // ratio^(gamma-1)
            for (int e = 1; e < p.eos_gamma; ++e) pw1 = __fmul_rn(pw1, ratio);
            const float pw = p.eos_gamma > 0 ? __fmul_rn(pw1, ratio) : 1.f;
            const float praw = __fmul_rn(p.eos_b, __fsub_rn(pw, 1.f));
            const bool live = !(p.clamp_pressure && praw < 0.f);
            const float inv_rho = 1.f / rho, inv_rho2 = inv_rho * inv_rho;
            const float dp = (live && p.eos_gamma > 0) ? p.eos_b * (float)p.eos_gamma * pw1 * p.inv_rho0 : 0.f;
            rb += pr2b * (dp - 2.f * rpk.y * inv_rho) * inv_rho2 - morb * mk * inv_rho2;
            if (live) bsum += pr2b * (pw - 1.f) * inv_rho2;
        }
        io.rho[k] = rb;
    }
    bsum = block_sum(bsum);
    if (threadIdx.x == 0) io.bpart[blockIdx.x] = bsum;
}

// gather of the transposed density sum
template <int kLanes>
__global__ void __launch_bounds__(kSphThreads, 3) k_adj_density(GridDev g, const float4* __restrict__ xs,
                                                                const float4* __restrict__ vs, int n,
                                                                const __grid_constant__ nsph_sph_params p,
                                                                const int4* __restrict__ nbr,
                                                                const int* __restrict__ ncnt,
                                                                const float* __restrict__ rho_adj,
                                                                const float4* __restrict__ xv,
                                                                float* __restrict__ x_in_adj)
{
    launch_entry();
    const int sub = threadIdx.x & (kLanes - 1);
    const int step = gridDim.x * blockDim.x / kLanes;
    for (int k0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / kLanes; k0 < n; k0 += step) {
        const int kt = k0 + (threadIdx.x & 31) / kLanes, k = min(kt, n - 1);
        const bool active = kt < n && (__float_as_int(vs[k].w) & kAttrActive);
        const float4 xi = xs[k];
        const float rbk = rho_adj[k], mk = xi.w;
        float xb[3] = {0.f, 0.f, 0.f};
        for_each_neighbor<kLanes>(g, xs, nbr, active ? ncnt[k] : 0, n, k, sub, xi, p, [&](int j) {
            const float4 xj = __ldg(xs + j);
            float dx, dy, dz;
            const float r2 = dist2(xi, xj, dx, dy, dz);
            if (!(r2 > 0.f)) return;
            const float r = __fsqrt_rn(r2);
            const float c = kernel_f(r * p.inv_h, 1.f / r, p) * (rbk * xj.w + __ldg(rho_adj + j) * mk);
            xb[0] += c * dx;
            xb[1] += c * dy;
            xb[2] += c * dz;
        });
        for (int c = 0; c < 3; ++c) xb[c] = lanes_sum<kLanes>(xb[c]);
        if (sub != 0 || kt >= n) continue;
        const size_t i = (size_t)g.ids[k];
        const float4 x0 = xv[2 * (size_t)k];
        store_row(x_in_adj + 3 * i, active ? x0.x + xb[0] : x0.x, active ? x0.y + xb[1] : x0.y,
                  active ? x0.z + xb[2] : x0.z);
    }
}

// adj(B) += sum of the per-block partials, in a fixed order
__global__ void k_adj_b_reduce(const float* __restrict__ bpart, int blocks, float* __restrict__ b_adj)
{
    launch_entry();
    float v = 0.f;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) v += bpart[b];
    v = block_sum(v);
    if (threadIdx.x == 0) *b_adj += v;
}

// ==========================================================================
// Surrogate step: the plain step's build and density pass (neighbour lists),
// then one kernel (k_surrogate_fused) that gathers each particle's force
// sums and 16 neighbour features, evaluates the MLP on the tensor cores
// (mlp.cuh) and integrates with the corrected acceleration a + da. The
// feature pass alone (k_force_features_list) serves the training data. The
// features are dimensionless (lengths / h, velocities / c0, accelerations
// h / c0^2, with c0^2 = B gamma / rho0):
//   0 rho/rho0   1 rho/rho0 - 1   2-4 sum V_j W (x_j - x_i) / h
//   5-7 sum V_j W (v_j - v_i) / c0 (the XSPH sum)   8-10 a h / c0^2
//   11 sum V_j W r^2 / h^2   12 Shepard sum V_i W(0) + sum V_j W
//   13 sum V_j F (v_j - v_i).(x_i - x_j) h / c0 (velocity divergence)
//   14 p / (rho0 c0^2)   15 |a| h / c0^2
// with V_j = m_j / rho_j and F = (dW/dr)/r.
// ==========================================================================
constexpr int kFeat = kMlpIn;

struct FeatAcc {
    float sw, mx, my, mz, m2, dvg;
};

// the pressure and XSPH terms of force_term_data (same statements, so the
// same rounding) plus the feature sums
__device__ __forceinline__ void force_feature_term(float4 xj, float4 vj, float pr2_j, float4 xi, float4 vi, float pr2_i,
                                                   const nsph_sph_params& p, ForceAcc& acc, FeatAcc& fa)
{
    float dx, dy, dz;
    const float r2 = dist2(xi, xj, dx, dy, dz);
    const float r = __fsqrt_rn(r2);
    const float q = __fmul_rn(r, p.inv_h);
    const float w = kernel_w(q, p);
    float f = 0.f;
    if (r2 > 0.f) {
        f = kernel_f(q, __frcp_rn(r), p);
        const float s = __fmul_rn(__fmul_rn(xj.w, __fadd_rn(pr2_i, pr2_j)), f);
        acc.ax = __fmaf_rn(-s, dx, acc.ax);
        acc.ay = __fmaf_rn(-s, dy, acc.ay);
        acc.az = __fmaf_rn(-s, dz, acc.az);
    }
    const float c = __fmul_rn(vj.w, w);
    const float rvx = __fsub_rn(vj.x, vi.x), rvy = __fsub_rn(vj.y, vi.y), rvz = __fsub_rn(vj.z, vi.z);
    acc.dvx = __fmaf_rn(c, rvx, acc.dvx);
    acc.dvy = __fmaf_rn(c, rvy, acc.dvy);
    acc.dvz = __fmaf_rn(c, rvz, acc.dvz);
    fa.sw += c;
    fa.mx -= c * dx;
    fa.my -= c * dy;
    fa.mz -= c * dz;
    fa.m2 += c * r2;
    fa.dvg += vj.w * f * (rvx * dx + rvy * dy + rvz * dz);
}

// pressure and XSPH sums (the statements of force_term_data, so the same
// rounding) and the feature sums of particle k over its neighbour list, in
// order
__device__ __forceinline__ void force_features_from_list(const GridDev& g, const ForceRec& fr,
                                                         const int4* __restrict__ nbr, int cnt, int n, int k, float4 xi,
                                                         float4 vi, float pr2_i, const nsph_sph_params& p,
                                                         ForceAcc& acc, FeatAcc& fa)
{
    if (cnt <= kNbrSlots) {
        bool have = false;
        Neighbour po{make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        float pp = 0.f;
        for_each_listed<true>(nbr, n, k, cnt, [&](int j) {
            if (j == k) return;
            const Neighbour o = load_neighbour(fr.rec, j);
            const float pj = __ldg(fr.pr2 + j);
            if (have) force_feature_term(po.x, po.v, pp, xi, vi, pr2_i, p, acc, fa);
            po = o;
            pp = pj;
            have = true;
        });
        if (have) force_feature_term(po.x, po.v, pp, xi, vi, pr2_i, p, acc, fa);
    } else {
        for_each_run(g, xi.x, xi.y, xi.z, p.h, [&](int lo, int hi) {
            for (int j = lo; j < hi; ++j) {
                const Neighbour o = load_neighbour(fr.rec, j);
                float dx, dy, dz;
                if (dist2(xi, o.x, dx, dy, dz) < p.h2 && j != k && !mirror_inactive(o.x))
                    force_feature_term(o.x, o.v, __ldg(fr.pr2 + j), xi, vi, pr2_i, p, acc, fa);
            }
        });
    }
}

// The 16 features of sorted particle k (all zero for an inactive one) and
// its force sums; adds the particle's compression max(0, rho/rho0 - 1) and
// 1 to (csum, ccount) when it is active.
__device__ __forceinline__ void particle_features(const GridDev& g, const ForceRec& fr,
                                                  const float2* __restrict__ rp, const int4* __restrict__ nbr,
                                                  const int* __restrict__ ncnt, int n, int k, float4 xi, float4 vi,
                                                  const nsph_sph_params& p, float (&f)[kFeat], ForceAcc& acc,
                                                  float& csum, float& ccount)
{
    acc = ForceAcc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (!(__float_as_int(vi.w) & kAttrActive)) {
#pragma unroll
        for (int j = 0; j < kFeat; ++j) f[j] = 0.f;
        return;
    }
    const float c0sq = fmaxf(p.eos_b * (float)p.eos_gamma * p.inv_rho0, 1e-30f);
    const float inv_c0 = rsqrtf(c0sq);
    const float ascale = p.h / c0sq;
    const float2 ak = make_float2(fr.rec[2 * (size_t)k + 1].w, fr.pr2[k]);  // (m/rho, p/rho^2)
    FeatAcc fa{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    force_features_from_list(g, fr, nbr, ncnt[k], n, k, xi, vi, ak.y, p, acc, fa);
    const float2 rpk = rp[k];
    const float ratio = rpk.x * p.inv_rho0;
    f[0] = ratio;
    f[1] = ratio - 1.f;
    f[2] = fa.mx * p.inv_h;
    f[3] = fa.my * p.inv_h;
    f[4] = fa.mz * p.inv_h;
    f[5] = acc.dvx * inv_c0;
    f[6] = acc.dvy * inv_c0;
    f[7] = acc.dvz * inv_c0;
    f[8] = acc.ax * ascale;
    f[9] = acc.ay * ascale;
    f[10] = acc.az * ascale;
    f[11] = fa.m2 * p.inv_h * p.inv_h;
    f[12] = fa.sw + ak.x * p.sigma;
    f[13] = fa.dvg * p.h * inv_c0;
    f[14] = rpk.y * p.inv_rho0 / c0sq;
    f[15] = sqrtf(f[8] * f[8] + f[9] * f[9] + f[10] * f[10]);
    csum += fmaxf(ratio - 1.f, 0.f);
    ccount += 1.f;
}

// per sorted particle k: feat[16 k ..] and sacc[2k] = (a, 0), sacc[2k+1] =
// (dv, 0), from the neighbour lists; per block: (sum of max(0, rho/rho0 - 1),
// active count)
__global__ void __launch_bounds__(kSphThreads, 4) k_force_features_list(GridDev g, const float4* __restrict__ xs,
                                                                        const float4* __restrict__ vs,
                                                                        const ForceRec fr,
                                                                        const float2* __restrict__ rp, int n,
                                                                        const __grid_constant__ nsph_sph_params p,
                                                                        const int4* __restrict__ nbr,
                                                                        const int* __restrict__ ncnt,
                                                                        float* __restrict__ feat,
                                                                        float4* __restrict__ sacc,
                                                                        float* __restrict__ cpart)
{
    launch_entry();
    float csum = 0.f, ccount = 0.f;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 xi = xs[k], vi = vs[k];
        float f[kFeat];
        ForceAcc acc;
        particle_features(g, fr, rp, nbr, ncnt, n, k, xi, vi, p, f, acc, csum, ccount);
        float4* fo = reinterpret_cast<float4*>(feat + (size_t)k * kFeat);
#pragma unroll
        for (int j = 0; j < kFeat; j += 4) fo[j / 4] = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
        sacc[2 * (size_t)k] = make_float4(acc.ax, acc.ay, acc.az, 0.f);
        sacc[2 * (size_t)k + 1] = make_float4(acc.dvx, acc.dvy, acc.dvz, 0.f);
    }
    csum = block_sum(csum);
    __syncthreads();  // block_sum's shared partials are reused
    ccount = block_sum(ccount);
    if (threadIdx.x == 0) {
        cpart[2 * blockIdx.x] = csum;
        cpart[2 * blockIdx.x + 1] = ccount;
    }
}

// stats[0] = mean compression of this step; stats[1] = max since reset;
// stats[2] += 1; stats[3] += stats[0]
__global__ void k_compression_reduce(const float* __restrict__ cpart, int blocks, float* __restrict__ stats)
{
    launch_entry();
    float s = 0.f, c = 0.f;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) {
        s += cpart[2 * b];
        c += cpart[2 * b + 1];
    }
    s = block_sum(s);
    __syncthreads();
    c = block_sum(c);
    if (threadIdx.x == 0) {
        const float e = c > 0.f ? s / c : 0.f;
        stats[0] = e;
        stats[1] = fmaxf(stats[1], e);
        stats[2] += 1.f;
        stats[3] += e;
    }
}

// The surrogate step's force pass fused with the MLP: each CTA takes tiles
// of 128 consecutive sorted particles; every thread gathers its particle's
// pressure / XSPH sums and 16 features from the neighbour list, stages the
// normalised bf16 feature row straight into the A tile of layer 1 in shared
// memory, the tcgen05 chain runs (accumulators in TMEM), and the thread
// integrates with a + da. Features and force sums never leave the SM.
// While one CTA waits on its MMAs, the other resident CTAs gather. If an
// MMA-completion wait gives up (after wait_limit polls), the CTA issues no
// further MMAs, integrates its remaining particles without the correction
// (the plain step at this dt) and flags NSPH_STATUS_SURROGATE_TIMEOUT. Per
// CTA: (sum of max(0, rho/rho0 - 1), active count) into cpart.
__global__ void __launch_bounds__(kMlpTile, 6) k_surrogate_fused(const float* __restrict__ model, float acc_scale,
                                                                 int wait_limit, GridDev g,
                                                                 const float4* __restrict__ xs,
                                                                 const float4* __restrict__ vs,
                                                                 const ForceRec fr,
                                                                 const float2* __restrict__ rp, int n,
                                                                 const __grid_constant__ nsph_sph_params p,
                                                                 const int4* __restrict__ nbr,
                                                                 const int* __restrict__ ncnt, const StepOut o,
                                                                 float* __restrict__ cpart)
{
    launch_entry();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    MlpFwdSmem& s = *reinterpret_cast<MlpFwdSmem*>(smem_raw);
    const uint32_t tmem = mlp_cta_begin(model, s, kMlpFwdCols);
    uint32_t phase = 0;
    bool ok = true;
    float csum = 0.f, ccount = 0.f;
    const int tiles = (n + kMlpTile - 1) / kMlpTile;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int k = t * kMlpTile + threadIdx.x;
        const int kk = k < n ? k : 0;
        const float4 xi = xs[kk], vi = vs[kk];
        float f[kFeat];
        ForceAcc acc;
        if (k < n) {
            particle_features(g, fr, rp, nbr, ncnt, n, k, xi, vi, p, f, acc, csum, ccount);
        } else {
            acc = ForceAcc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < kFeat; ++j) f[j] = 0.f;
        }
        float y[kMlpOut] = {0.f, 0.f, 0.f};
        if (ok) {  // uniform across the CTA (mlp_wait makes the outcome uniform)
            mlp_stage_input(s, f);
            mlp_sync();
            ok = mlp_forward_tile(s, tmem, 0, 0, 0, phase, y, wait_limit);
        }
        if (k < n) {
            const int attr = __float_as_int(vi.w);
            if (ok && (attr & kAttrDynamic)) {
                acc.ax = __fadd_rn(acc.ax, acc_scale * mlp_denorm(s, y, 0));
                acc.ay = __fadd_rn(acc.ay, acc_scale * mlp_denorm(s, y, 1));
                acc.az = __fadd_rn(acc.az, acc_scale * mlp_denorm(s, y, 2));
            }
            integrate_out((size_t)g.ids[k], xi, vi, attr, rp[k], acc, p, p.dt, o);
        }
        __syncthreads();
    }
    if (!ok && o.status && threadIdx.x == 0) atomicOr(o.status, (unsigned)NSPH_STATUS_SURROGATE_TIMEOUT);
    csum = block_sum(csum);
    __syncthreads();
    ccount = block_sum(ccount);
    if (threadIdx.x == 0) {
        cpart[2 * blockIdx.x] = csum;
        cpart[2 * blockIdx.x + 1] = ccount;
    }
    mlp_cta_end(s, tmem, kMlpFwdCols, !ok, phase);
}

// k_surrogate_fused with kGroups tiles per CTA: groups of 128 threads share
// one copy of the weights (12 KB) and run their tiles independently (own
// input / hidden tiles, completion barrier, 64 TMEM columns, named barriers),
// so one group's MMA round trips overlap the other groups' gathers, and a CTA
// of 2 groups holds 53 KB of shared memory for 8 warps instead of 67 KB.
// Same per-particle arithmetic as k_surrogate_fused; the timeout rule
// applies per group.
template <int kGroups>
__global__ void __launch_bounds__(kGroups * kMlpTile, 6 / kGroups)
    k_surrogate_fused_groups(const float* __restrict__ model, float acc_scale, int wait_limit, GridDev g,
                             const float4* __restrict__ xs, const float4* __restrict__ vs,
                             const ForceRec fr, const float2* __restrict__ rp, int n,
                             const __grid_constant__ nsph_sph_params p, const int4* __restrict__ nbr,
                             const int* __restrict__ ncnt, const StepOut o, float* __restrict__ cpart)
{
    launch_entry();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    auto& s = *reinterpret_cast<MlpFwdGroupSmem<kGroups>*>(smem_raw);
    const int grp = threadIdx.x / kMlpTile, row = threadIdx.x % kMlpTile;
    mlp_stage_weights(model, s);
    if (threadIdx.x < kGroups) umma::mbar_init(&s.bar[threadIdx.x], 1);
    if (threadIdx.x < 32) umma::tmem_alloc(&s.tmem, kGroups * kMlpFwdCols);
    mlp_sync();
    const uint32_t tmem = s.tmem;
    uint32_t phase = 0;
    bool ok = true;
    float csum = 0.f, ccount = 0.f;
    const int tiles = (n + kMlpTile - 1) / kMlpTile;
    for (int t = blockIdx.x * kGroups + grp; t < tiles; t += gridDim.x * kGroups) {
        const int k = t * kMlpTile + row;
        const int kk = k < n ? k : 0;
        const float4 xi = xs[kk], vi = vs[kk];
        float f[kFeat];
        ForceAcc acc;
        if (k < n) {
            particle_features(g, fr, rp, nbr, ncnt, n, k, xi, vi, p, f, acc, csum, ccount);
        } else {
            acc = ForceAcc{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < kFeat; ++j) f[j] = 0.f;
        }
        float y[kMlpOut] = {0.f, 0.f, 0.f};
        if (ok) {  // uniform across the group (mlp_group_wait makes the outcome uniform)
            mlp_group_stage_input(s, grp, row, f);
            mlp_group_sync(grp);
            ok = mlp_group_forward_tile(s, grp, row, tmem, phase, y, wait_limit);
        }
        if (k < n) {
            const int attr = __float_as_int(vi.w);
            if (ok && (attr & kAttrDynamic)) {
                acc.ax = __fadd_rn(acc.ax, acc_scale * mlp_denorm(s, y, 0));
                acc.ay = __fadd_rn(acc.ay, acc_scale * mlp_denorm(s, y, 1));
                acc.az = __fadd_rn(acc.az, acc_scale * mlp_denorm(s, y, 2));
            }
            integrate_out((size_t)g.ids[k], xi, vi, attr, rp[k], acc, p, p.dt, o);
        }
    }
    if (!ok && o.status && row == 0) atomicOr(o.status, (unsigned)NSPH_STATUS_SURROGATE_TIMEOUT);
    // a group whose wait gave up waits once more (bounded) for the completion
    // it left outstanding, before the CTA frees its TMEM
    if (!ok) umma::mbar_wait(&s.bar[grp], phase, kMlpWaitLimit);
    csum = block_sum(csum);
    __syncthreads();
    ccount = block_sum(ccount);
    if (threadIdx.x == 0) {
        cpart[2 * blockIdx.x] = csum;
        cpart[2 * blockIdx.x + 1] = ccount;
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (threadIdx.x < 32) umma::tmem_dealloc(tmem, kGroups * kMlpFwdCols);
}

// sorted scratch -> original order: feat (n x 16), acc (n x 6: a, dv)
__global__ void k_scatter_features(const int* __restrict__ ids, int n, const float* __restrict__ sfeat,
                                   const float4* __restrict__ sacc, float* __restrict__ feat_out,
                                   float* __restrict__ acc_out)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const size_t i = (size_t)ids[k];
    if (feat_out)
        for (int j = 0; j < kFeat; ++j) feat_out[i * kFeat + j] = sfeat[(size_t)k * kFeat + j];
    if (acc_out) {
        const float4 a = sacc[2 * (size_t)k], dv = sacc[2 * (size_t)k + 1];
        acc_out[6 * i + 0] = a.x;
        acc_out[6 * i + 1] = a.y;
        acc_out[6 * i + 2] = a.z;
        acc_out[6 * i + 3] = dv.x;
        acc_out[6 * i + 4] = dv.y;
        acc_out[6 * i + 5] = dv.z;
    }
}

__global__ void k_scatter_rho(const int* __restrict__ ids, int n, const float2* __restrict__ rp,
                              float* __restrict__ rho_out)
{
    launch_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) rho_out[ids[k]] = rp[k].x;
}

// mismatches of sqrt_plain / rcp_plain over the mantissas of [1, 4) x 2^(2 e)
__global__ void k_root_mismatches(int e, unsigned long long* __restrict__ count)
{
    unsigned bad = 0;
    for (unsigned u = 0x3f800000u + blockIdx.x * blockDim.x + threadIdx.x; u < 0x40800000u; u += gridDim.x * blockDim.x) {
        const float x = ldexpf(__uint_as_float(u), 2 * e);
        float y;
        const float r = sqrt_plain(x, y);
        bad += !plain_range(x) || __float_as_uint(r) != __float_as_uint(__fsqrt_rn(x)) ||
               __float_as_uint(rcp_plain(r, y)) != __float_as_uint(__frcp_rn(r));
    }
    if (bad) atomicAdd(count, (unsigned long long)bad);
}

}  // namespace
}  // namespace nsph

extern "C" int nsph_debug_root_mismatches(const int* exponents, int num_exponents, unsigned long long* count)
{
    using namespace nsph;
    clear_error();
    if (!count || num_exponents < 0 || (num_exponents > 0 && !exponents))
        return fail(NSPH_ERR_INVALID_ARG, "null argument");
    unsigned long long* d = nullptr;
    NSPH_CUDA_TRY(cudaMalloc(&d, sizeof(*d)));
    cudaError_t e = cudaMemset(d, 0, sizeof(*d));
    for (int i = 0; i < num_exponents; ++i) k_root_mismatches<<<1024, 256>>>(exponents[i], d);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(count, d, sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? NSPH_OK : cuda_fail(e, "nsph_debug_root_mismatches");
}

// ==========================================================================
// C ABI: solver context
// ==========================================================================
using namespace nsph;

struct nsph_sph {
    Grid grid;
    int capacity = 0;
    float4* xs = nullptr;
    float4* vs = nullptr;
    float2* rp = nullptr;
    ForceRec fr{nullptr, nullptr, nullptr};  // the force pass's records
    int4* nbr = nullptr;       // kNbrGroups x capacity neighbour lists (group-major), every step form
    int* ncnt = nullptr;       //   neighbours per particle
    int fast = 0;              // plain step: tolerance arithmetic (nsph_sph_set_arithmetic)
    unsigned* status = nullptr;
    int last_n = 0;
    int last_launches = 0;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};  // start, built, density, end
    nsph_sph_params* wparams = nullptr;  // batched worlds: per-world parameters (device)
    int wparams_set = 0;
    int persistent_blocks = 0;           // batched worlds: blocks of the persistent passes
    int launch_threads = 0;              // neighbour passes: threads per block (0 = default)
    int launch_blocks_per_sm = -1;       // neighbour passes: persistent blocks per SM (-1 = default, 0 = one thread per particle)
    int sms = 0;
    float4* adj_gd = nullptr;            // adjoint scratch (nsph_sph_enable_adjoint), sorted: adj(a), adj(dv) at 2k, 2k + 1
    float4* adj_xv = nullptr;            //   the adjoints of x and v so far
    float* adj_rho = nullptr;            //   adj(rho)
    float* adj_bpart = nullptr;          //   per-block partial sums of adj(B)
    int adj_bcap = 0;                    //   entries of adj_bpart
    cudaEvent_t eva[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // adjoint / surrogate phases
    float* sfeat = nullptr;              // surrogate scratch (nsph_sph_enable_surrogate), sorted: 16 features
    float4* sacc = nullptr;              //   (a, 0), (dv, 0)
    float* cpart = nullptr;              //   per-block (compression sum, active count)
    int surr_ctas = 0;                   //   resident CTAs of the fused surrogate kernel (its grid)
    int surr_groups = 1;                 //   tiles of 128 particles per CTA (1: k_surrogate_fused, 2: the grouped kernel)
    int surr_wait_limit = -1;            //   polls of an MMA-completion wait (-1: kMlpWaitLimit)
    char* tape = nullptr;                // segment tape (nsph_sph_segment_adjoint): per step of a segment,
    int tape_steps = 0;                  //   the build and density outputs the step's reverse reads,
    size_t tape_step_bytes = 0;          //   tape_steps slots of tape_step_bytes, then two states
};

// One step's slot of the segment tape: the sorted mirrors, the density
// pass's outputs and neighbour lists, the grid (sorted ids, cell table) and
// the force pass's sums.
struct TapeStep {
    float4* xs;
    float4* vs;
    float2* rp;
    ForceRec fr;
    int4* nbr;
    int* ncnt;
    int* ids;
    int2* ranges;
    float4* acc;  // the force pass's (a, 0), (dv, 0) per sorted particle
};

static size_t tape_align(size_t b) { return (b + 255) & ~(size_t)255; }

static size_t tape_slot_bytes(size_t c, long long ncells)
{
    return 2 * tape_align(sizeof(float4) * c) + tape_align(sizeof(float2) * c) +
           tape_align(sizeof(float4) * 2 * c) + tape_align(sizeof(float) * c) +
           tape_align(sizeof(int4) * kNbrGroups * c) + 2 * tape_align(sizeof(int) * c) +
           tape_align(sizeof(int2) * (size_t)ncells) + tape_align(sizeof(float4) * 2 * c);
}

static TapeStep tape_slot(const nsph_sph* s, int t)
{
    const size_t c = (size_t)s->capacity;
    char* b = s->tape + (size_t)t * s->tape_step_bytes;
    TapeStep ts;
    ts.xs = reinterpret_cast<float4*>(b);
    b += tape_align(sizeof(float4) * c);
    ts.vs = reinterpret_cast<float4*>(b);
    b += tape_align(sizeof(float4) * c);
    ts.rp = reinterpret_cast<float2*>(b);
    b += tape_align(sizeof(float2) * c);
    ts.fr.rec = reinterpret_cast<float4*>(b);
    b += tape_align(sizeof(float4) * 2 * c);
    ts.fr.pr2 = reinterpret_cast<float*>(b);
    ts.fr.overflow = nullptr;
    b += tape_align(sizeof(float) * c);
    ts.nbr = reinterpret_cast<int4*>(b);
    b += tape_align(sizeof(int4) * kNbrGroups * c);
    ts.ncnt = reinterpret_cast<int*>(b);
    b += tape_align(sizeof(int) * c);
    ts.ids = reinterpret_cast<int*>(b);
    b += tape_align(sizeof(int) * c);
    ts.ranges = reinterpret_cast<int2*>(b);
    b += tape_align(sizeof(int2) * (size_t)s->grid.ncells);
    ts.acc = reinterpret_cast<float4*>(b);
    return ts;
}

// after the slots: the two recompute states (x then v, 3 x capacity floats
// each), then a word per step that tells whether a list overflowed
static unsigned* tape_overflow(const nsph_sph* s)
{
    const size_t c = (size_t)s->capacity;
    return reinterpret_cast<unsigned*>(s->tape + (size_t)s->tape_steps * s->tape_step_bytes +
                                       tape_align(sizeof(float) * 12 * c));
}

static float* tape_state(const nsph_sph* s, int which)
{
    return reinterpret_cast<float*>(s->tape + (size_t)s->tape_steps * s->tape_step_bytes) +
           (size_t)which * 6 * (size_t)s->capacity;
}

// grid of a neighbour pass: one thread per particle, or a persistent grid of
// blocks_per_sm blocks per SM striding over the particles
static void pass_launch(const nsph_sph* s, int n, bool persistent_default, int& blocks, int& threads)
{
    threads = s->launch_threads > 0 ? s->launch_threads : kSphThreads;
    const int full = (n + threads - 1) / threads;
    int bps = s->launch_blocks_per_sm;
    if (bps < 0) bps = persistent_default ? -1 : 0;
    if (bps < 0)
        blocks = std::min(full, s->persistent_blocks > 0 ? s->persistent_blocks : full);
    else if (bps == 0)
        blocks = full;
    else
        blocks = std::min(full, std::max(1, s->sms * bps));
    blocks = std::max(blocks, 1);
}

// whether the force and adjoint passes take four lanes per particle: scenes of
// at most kQuadMax particles, unless the caller set a launch shape
static bool quad_pass(const nsph_sph* s, int n)
{
    return n <= kQuadMax && s->launch_threads == 0 && s->launch_blocks_per_sm < 0;
}

// shared memory of a density pass: one TileSmem per warp
static size_t tile_smem_bytes(int threads) { return sizeof(TileSmem) * (size_t)(threads / 32); }

// whether the density pass takes eight lanes per particle, by the same rule
static bool octet_pass(const nsph_sph* s, int n)
{
    return n <= kOctetMax && s->launch_threads == 0 && s->launch_blocks_per_sm < 0;
}

// How a density pass of tiles is launched. One whose blocks are all resident
// at once (kDensityBlocks per SM) must not start early: its blocks would be
// placed while the build's last blocks still hold some of the SMs, two and
// three on one SM beside an idle one, and the pass lasts as long as its fullest
// SM. A step took 80 us with the early start and 54 without at 24k particles,
// 82 and 70 at 64k, 96 and 95 at 125k; larger passes level out over their
// blocks and gain the launch (116 and 118 us at 166k). A pass of eight lanes
// per particle is always that small (31 and 25 us at 2,197 particles).
template <class... P, class... A>
static cudaError_t launch_tiles(const nsph_sph* s, void (*kernel)(P...), int blocks, int threads, cudaStream_t cs,
                                A&&... args)
{
    return blocks <= s->sms * kDensityBlocks
               ? launch_plain(kernel, blocks, threads, tile_smem_bytes(threads), cs, std::forward<A>(args)...)
               : launch_dependent(kernel, blocks, threads, tile_smem_bytes(threads), cs, std::forward<A>(args)...);
}

// the density pass of a single-world step into the given arrays
static int density_enqueue(const nsph_sph* s, const GridDev& g, const nsph_sph_params* p, int n, bool fast,
                           const float4* xs, const float4* vs, float2* rp, int4* nbr, int* ncnt,
                           const ForceRec& fr, cudaStream_t cs, int& launches)
{
    if (octet_pass(s, n)) {
        const int blocks = (n + kOctetParticles - 1) / kOctetParticles;
        NSPH_CUDA_TRY(launch_plain(fast ? k_density_octet<true> : k_density_octet<false>, blocks, kOctetThreads,
                                   0, cs, g, xs, vs, n, *p, rp, nbr, ncnt, fr, s->status));
    } else {
        int blocks, threads;
        pass_launch(s, n, false, blocks, threads);
        NSPH_CUDA_TRY(launch_tiles(s, fast ? k_density_list<true> : k_density_list<false>, blocks, threads, cs, g, xs,
                                   vs, n, *p, rp, nbr, ncnt, fr, s->status));
    }
    ++launches;
    return NSPH_OK;
}

// Record a timing event: as an external event node while the stream is being
// captured (so a replayed graph records it), as a plain record otherwise.
static cudaError_t record_mark(cudaEvent_t ev, cudaStream_t stream)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(stream, &cap);
    if (e != cudaSuccess) return e;
    return cap == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ev, stream, cudaEventRecordExternal)
                                                : cudaEventRecord(ev, stream);
}

static void sph_free(nsph_sph* s)
{
    DeviceGuard guard(s->grid.device);
    for (cudaEvent_t& e : s->ev)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    for (cudaEvent_t& e : s->eva)
        if (e) {
            cudaEventDestroy(e);
            e = nullptr;
        }
    cudaFree(s->xs);
    cudaFree(s->vs);
    cudaFree(s->rp);
    cudaFree(s->fr.rec);
    cudaFree(s->fr.pr2);
    cudaFree(s->nbr);
    cudaFree(s->ncnt);
    cudaFree(s->wparams);
    cudaFree(s->status);
    cudaFree(s->adj_gd);
    cudaFree(s->adj_xv);
    cudaFree(s->adj_rho);
    cudaFree(s->adj_bpart);
    cudaFree(s->sfeat);
    cudaFree(s->tape);
    cudaFree(s->sacc);
    cudaFree(s->cpart);
    grid_free(s->grid);
}

static int sph_create_common(nsph_sph* s, int device, int capacity);

extern "C" int nsph_sph_create(int device, int capacity, const int grid_dims[3], nsph_sph** out)
{
    clear_error();
    if (!out || !grid_dims) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    *out = nullptr;
    if (capacity < 0) return fail(NSPH_ERR_INVALID_ARG, "negative capacity");
    nsph_sph* s = new (std::nothrow) nsph_sph();
    if (!s) return fail(NSPH_ERR_OUT_OF_MEMORY, "host allocation failed");
    int st = grid_init(s->grid, grid_dims[0], grid_dims[1], grid_dims[2], device);
    if (st == NSPH_OK) st = sph_create_common(s, device, capacity);
    if (st == NSPH_OK) {  // the plain step's kernels
        DeviceGuard guard(device);
        cudaError_t e = cudaSuccess;
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_list<false>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_force_list<false>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_force_quad);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_octet<false>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_octet<true>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_tape_copy);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_list<true>);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_force_list<true>);
        if (e != cudaSuccess) {
            cudaGetLastError();
            st = fail(NSPH_ERR_OUT_OF_MEMORY, std::string("solver allocation: ") + cudaGetErrorString(e));
        }
    }
    if (st != NSPH_OK) {
        sph_free(s);
        delete s;
        return st;
    }
    *out = s;
    return NSPH_OK;
}

extern "C" int nsph_sph_create_worlds(int device, int capacity, int world_count, const int* world_dims,
                                      nsph_sph** out)
{
    clear_error();
    if (!out || !world_dims) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    *out = nullptr;
    if (capacity < 0) return fail(NSPH_ERR_INVALID_ARG, "negative capacity");
    nsph_sph* s = new (std::nothrow) nsph_sph();
    if (!s) return fail(NSPH_ERR_OUT_OF_MEMORY, "host allocation failed");
    int st = grid_init_worlds(s->grid, world_dims, world_count, device);
    if (st == NSPH_OK) st = sph_create_common(s, device, capacity);
    if (st == NSPH_OK) {
        DeviceGuard guard(device);
        cudaError_t e = cudaMalloc(&s->wparams, sizeof(nsph_sph_params) * (size_t)world_count);
        int sms = 0, per_sm = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_force_worlds, kSphThreads, 0);
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_worlds);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_density_octet_worlds);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_neighbors_worlds);
        if (e != cudaSuccess) {
            cudaGetLastError();
            st = fail(NSPH_ERR_CUDA, std::string("worlds setup: ") + cudaGetErrorString(e));
        }
        s->persistent_blocks = std::max(1, sms * std::max(1, per_sm));
    }
    if (st != NSPH_OK) {
        sph_free(s);
        delete s;
        return st;
    }
    *out = s;
    return NSPH_OK;
}

static int sph_create_common(nsph_sph* s, int device, int capacity)
{
    if (cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        s->sms = 1;
    }
    int st = grid_reserve(s->grid, capacity);
    if (st == NSPH_OK) {
        DeviceGuard guard(device);
        const size_t c = (size_t)(capacity > 0 ? capacity : 1);
        cudaError_t e = cudaMalloc(&s->xs, sizeof(float4) * (c + kXsPad));
        if (e == cudaSuccess) e = cudaMemset(s->xs + c, 0, sizeof(float4) * kXsPad);
        if (e == cudaSuccess) e = cudaMalloc(&s->vs, sizeof(float4) * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->rp, sizeof(float2) * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->fr.rec, sizeof(float4) * 2 * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->fr.pr2, sizeof(float) * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->nbr, sizeof(int4) * kNbrGroups * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->ncnt, sizeof(int) * c);
        if (e == cudaSuccess) e = cudaMalloc(&s->status, sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemset(s->status, 0, sizeof(unsigned));
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_neighbors);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            cudaGetLastError();
            st = fail(NSPH_ERR_OUT_OF_MEMORY, std::string("solver allocation: ") + cudaGetErrorString(e));
        }
    }
    if (st == NSPH_OK) s->capacity = capacity;
    return st;
}

extern "C" int nsph_sph_destroy(nsph_sph* solver)
{
    clear_error();
    if (!solver) return NSPH_OK;
    sph_free(solver);
    delete solver;
    return NSPH_OK;
}

static int check_params(const nsph_sph_params* p)
{
    if (!p) return fail(NSPH_ERR_INVALID_ARG, "null params");
    if (!(p->h > 0.f) || !(p->h2 > 0.f) || !(p->cell_inv > 0.f) || !isfinite(p->h) || !isfinite(p->cell_inv))
        return fail(NSPH_ERR_INVALID_ARG, "h and cell width must be positive and finite");
    if (p->eos_gamma < 0 || p->eos_gamma > 16) return fail(NSPH_ERR_INVALID_ARG, "eos_gamma out of [0, 16]");
    if (!(p->rho0 > 0.f)) return fail(NSPH_ERR_INVALID_ARG, "rho0 must be positive");
    return NSPH_OK;
}

// Checks shared by the single-world step entry points (the caller has
// checked the solver handle and the parameter block).
static int check_step_inputs(const nsph_sph* s, int n, const float* x_in, const float* v_in, const float* mass,
                             const float* inv_mass, const int* flags, const float* gravity, int world_count)
{
    if (n < 0) return fail(NSPH_ERR_INVALID_ARG, "negative particle count");
    if (n > s->capacity) return fail(NSPH_ERR_CAPACITY, "more particles than the solver was created for");
    if (world_count < 1 || !gravity) return fail(NSPH_ERR_INVALID_ARG, "gravity needs world_count >= 1");
    if (n > 0 && (!x_in || !v_in || !mass || !inv_mass || !flags))
        return fail(NSPH_ERR_INVALID_ARG, "null state or model array");
    if (s->grid.world_count > 0)
        return fail(NSPH_ERR_INVALID_ARG, "solver was created for batched worlds: use nsph_sph_step_worlds");
    return NSPH_OK;
}

// Enqueue one step on validated inputs: grid build + sorted gather, density,
// force + integrate (with the phase events when enabled).
static int step_enqueue(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in, const float* v_in,
                        const float* f_ext, const float* mass, const float* inv_mass, const int* flags,
                        const int* world, const float* gravity, int world_count, float* x_out, float* v_out,
                        float* rho_out, float* p_out, float* a_out, cudaStream_t cs, int& launches,
                        bool carry_v = false)
{
    GatherArgs ga{x_in, v_in, mass, inv_mass, flags, world, world_count, s->xs, s->vs};
    if (s->ev[0]) NSPH_CUDA_TRY(record_mark(s->ev[0], cs));
    int st = grid_build(s->grid, x_in, n, p->cell_width, p->cell_inv, &ga, s->status, cs, &launches);
    if (st != NSPH_OK) return st;
    s->last_n = n;
    if (s->ev[1]) NSPH_CUDA_TRY(record_mark(s->ev[1], cs));
    if (n > 0) {
        const GridDev g = s->grid.view();
        int blocks, threads;
        st = density_enqueue(s, g, p, n, s->fast != 0, s->xs, s->vs, s->rp, s->nbr, s->ncnt, s->fr, cs, launches);
        if (st != NSPH_OK) return st;
        if (s->ev[2]) NSPH_CUDA_TRY(record_mark(s->ev[2], cs));
        pass_launch(s, n, false, blocks, threads);
        const StepOut o{f_ext, inv_mass, gravity, x_out, v_out, rho_out, p_out, a_out, s->status, nullptr, carry_v};
        if (s->fast)
            NSPH_CUDA_TRY(launch_plain(k_force_list<true>, blocks, threads, 0, cs,
                                           g, s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, o));
        else if (quad_pass(s, n))
            NSPH_CUDA_TRY(launch_dependent(k_force_quad, (4 * n + kQuadThreads - 1) / kQuadThreads, kQuadThreads, 0, cs,
                                           g, s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, o));
        else
            NSPH_CUDA_TRY(launch_plain(k_force_list<false>, blocks, threads, 0, cs,
                                           g, s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, o));
        NSPH_LAUNCH_CHECK("k_force_list");
        ++launches;
    } else if (s->ev[2]) {
        NSPH_CUDA_TRY(record_mark(s->ev[2], cs));
    }
    if (s->ev[3]) NSPH_CUDA_TRY(record_mark(s->ev[3], cs));
    return NSPH_OK;
}

extern "C" int nsph_sph_step(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in, const float* v_in,
                             const float* f_ext, const float* mass, const float* inv_mass, const int* flags,
                             const int* world, const float* gravity, int world_count, float* x_out,
                             float* v_out, float* rho_out, float* p_out, float* a_out, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_step");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x_in, v_in, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (n > 0 && (!x_out || !v_out)) return fail(NSPH_ERR_INVALID_ARG, "null state or model array");
    if (n > 0 && (x_out == x_in || v_out == v_in))
        return fail(NSPH_ERR_INVALID_ARG, "state_out must not alias state_in");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    int launches = 0;
    st = step_enqueue(s, p, n, x_in, v_in, f_ext, mass, inv_mass, flags, world, gravity, world_count, x_out, v_out,
                      rho_out, p_out, a_out, (cudaStream_t)stream, launches);
    s->last_launches = launches;
    return st;
}

// [a, a + na) and [b, b + nb) (in floats) share memory
static bool overlaps(const float* a, size_t na, const float* b, size_t nb)
{
    return a < b + nb && b < a + na;
}

extern "C" int nsph_sph_rollout(nsph_sph* s, const nsph_sph_params* p, int n, int steps, const float* x0,
                                const float* v0, const float* f_ext, const float* mass, const float* inv_mass,
                                const int* flags, const int* world, const float* gravity, int world_count,
                                float* x_traj, float* v_traj, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_rollout");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x0, v0, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (steps < 0) return fail(NSPH_ERR_INVALID_ARG, "negative step count");
    const size_t len = 3 * (size_t)n;
    if (n > 0 && steps > 0) {
        if (!x_traj || !v_traj) return fail(NSPH_ERR_INVALID_ARG, "null trajectory array");
        const size_t tot = len * (size_t)steps;
        if (overlaps(x_traj, tot, v_traj, tot) || overlaps(x0, len, x_traj, tot) || overlaps(v0, len, v_traj, tot) ||
            overlaps(x0, len, v_traj, tot) || overlaps(v0, len, x_traj, tot))
            return fail(NSPH_ERR_INVALID_ARG, "trajectory arrays overlap each other or the initial state");
    }
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    int launches = 0;
    for (int t = 0; t < steps && n > 0; ++t) {
        const float* xi = t == 0 ? x0 : x_traj + (size_t)(t - 1) * len;
        const float* vi = t == 0 ? v0 : v_traj + (size_t)(t - 1) * len;
        float* xo = x_traj + (size_t)t * len;
        float* vo = v_traj + (size_t)t * len;
        // inactive particles keep their velocity
        st = step_enqueue(s, p, n, xi, vi, f_ext, mass, inv_mass, flags, world, gravity, world_count, xo, vo, nullptr,
                          nullptr, nullptr, cs, launches, true);
        if (st != NSPH_OK) return st;
    }
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_set_world_params(nsph_sph* s, const nsph_sph_params* params, int world_count)
{
    clear_error();
    if (!s || !params) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    if (s->grid.world_count <= 0) return fail(NSPH_ERR_INVALID_ARG, "solver was not created for batched worlds");
    if (world_count != s->grid.world_count) return fail(NSPH_ERR_INVALID_ARG, "world_count differs from the solver's");
    for (int w = 0; w < world_count; ++w) {
        const int st = check_params(params + w);
        if (st != NSPH_OK) return fail(st, "world " + std::to_string(w) + ": " + nsph_last_error());
    }
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    std::vector<WorldCells> wc((size_t)world_count);
    NSPH_CUDA_TRY(cudaMemcpy(wc.data(), s->grid.worlds, sizeof(WorldCells) * world_count, cudaMemcpyDeviceToHost));
    for (int w = 0; w < world_count; ++w) wc[w].inv = params[w].cell_inv;
    NSPH_CUDA_TRY(cudaMemcpy(s->grid.worlds, wc.data(), sizeof(WorldCells) * world_count, cudaMemcpyHostToDevice));
    NSPH_CUDA_TRY(cudaMemcpy(s->wparams, params, sizeof(nsph_sph_params) * world_count, cudaMemcpyHostToDevice));
    s->wparams_set = 1;
    return NSPH_OK;
}

extern "C" int nsph_sph_step_worlds(nsph_sph* s, float dt, int n, const float* x_in, const float* v_in,
                                    const float* f_ext, const float* mass, const float* inv_mass, const int* flags,
                                    const int* world, const float* gravity, int world_count, float* x_out,
                                    float* v_out, float* rho_out, float* p_out, float* a_out, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_step_worlds");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (s->grid.world_count <= 0) return fail(NSPH_ERR_INVALID_ARG, "solver was not created for batched worlds");
    if (!s->wparams_set) return fail(NSPH_ERR_INVALID_ARG, "world parameters not set (nsph_sph_set_world_params)");
    if (!isfinite(dt)) return fail(NSPH_ERR_INVALID_ARG, "dt must be finite");
    if (n < 0) return fail(NSPH_ERR_INVALID_ARG, "negative particle count");
    if (n > s->capacity) return fail(NSPH_ERR_CAPACITY, "more particles than the solver was created for");
    if (world_count != s->grid.world_count || !gravity)
        return fail(NSPH_ERR_INVALID_ARG, "gravity must have one row per world of the solver");
    if (n > 0 && (!x_in || !v_in || !mass || !inv_mass || !flags || !x_out || !v_out))
        return fail(NSPH_ERR_INVALID_ARG, "null state or model array");
    if (n > 0 && (x_out == x_in || v_out == v_in))
        return fail(NSPH_ERR_INVALID_ARG, "state_out must not alias state_in");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    GatherArgs ga{x_in, v_in, mass, inv_mass, flags, world, world_count, s->xs, s->vs};
    int launches = 0;
    if (s->ev[0]) NSPH_CUDA_TRY(record_mark(s->ev[0], cs));
    int st = grid_build(s->grid, x_in, n, 0.f, 0.f, &ga, s->status, cs, &launches, world);
    if (st != NSPH_OK) return st;
    s->last_n = n;
    if (s->ev[1]) NSPH_CUDA_TRY(record_mark(s->ev[1], cs));
    if (n > 0) {
        int blocks, threads;
        if (octet_pass(s, n)) {
            NSPH_CUDA_TRY(launch_plain(k_density_octet_worlds, (n + kOctetParticles - 1) / kOctetParticles,
                                       kOctetThreads, 0, cs, s->grid.worlds, s->wparams, s->grid.cell_ranges,
                                       s->grid.point_ids, s->xs, s->vs, n, s->rp, s->nbr, s->ncnt, s->fr,
                                       s->status));
        } else {
            pass_launch(s, n, true, blocks, threads);
            NSPH_CUDA_TRY(launch_tiles(s, k_density_worlds, blocks, threads, cs, s->grid.worlds, s->wparams,
                                       s->grid.cell_ranges, s->grid.point_ids, s->xs, s->vs, n, s->rp, s->nbr,
                                       s->ncnt, s->fr, s->status));
        }
        ++launches;
        if (s->ev[2]) NSPH_CUDA_TRY(record_mark(s->ev[2], cs));
        pass_launch(s, n, true, blocks, threads);
        const StepOut o{f_ext, inv_mass, gravity, x_out, v_out, rho_out, p_out, a_out, s->status};
        NSPH_CUDA_TRY(launch_plain(k_force_worlds, blocks, threads, 0, cs,
                                       s->grid.worlds, s->wparams, s->grid.cell_ranges, s->grid.point_ids, s->xs, s->vs, s->fr, s->rp, n, dt, s->nbr, s->ncnt, o));
        NSPH_LAUNCH_CHECK("k_force_worlds");
        ++launches;
    } else if (s->ev[2]) {
        NSPH_CUDA_TRY(record_mark(s->ev[2], cs));
    }
    if (s->ev[3]) NSPH_CUDA_TRY(record_mark(s->ev[3], cs));
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_neighbors(const nsph_sph* s, const nsph_sph_params* p, int* counts,
                                  const long long* offsets, int* out_ids, void* stream)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (s->grid.world_count > 0) {
        if (!s->grid.built) return fail(NSPH_ERR_NOT_BUILT, "no step has run yet");
        if (out_ids ? !offsets : !counts)
            return fail(NSPH_ERR_INVALID_ARG, "counts (count call) or offsets (fill call) required");
        const int n = s->last_n;
        if (n == 0) return NSPH_OK;
        DeviceGuard guard(s->grid.device);
        if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
        NSPH_CUDA_TRY(launch_dependent(k_neighbors_worlds, (n + 127) / 128, 128, 0, (cudaStream_t)stream,
                                       s->grid.worlds, s->wparams, s->grid.cell_ranges, s->grid.point_ids, s->xs, s->vs, n, counts, offsets, out_ids));
        NSPH_LAUNCH_CHECK("k_neighbors_worlds");
        return NSPH_OK;
    }
    int st = check_params(p);
    if (st != NSPH_OK) return st;
    if (!s->grid.built) return fail(NSPH_ERR_NOT_BUILT, "no step has run yet");
    if (out_ids ? !offsets : !counts) return fail(NSPH_ERR_INVALID_ARG, "counts (count call) or offsets (fill call) required");
    const int n = s->last_n;
    if (n == 0) return NSPH_OK;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(launch_dependent(k_neighbors, (n + 127) / 128, 128, 0, (cudaStream_t)stream,
                                   s->grid.view(), s->xs, s->vs, n, *p, counts, offsets, out_ids));
    NSPH_LAUNCH_CHECK("k_neighbors");
    return NSPH_OK;
}

extern "C" int nsph_sph_get_grid_view(const nsph_sph* s, nsph_grid_view* view)
{
    clear_error();
    if (!s || !view) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    const Grid& g = s->grid;
    view->point_cells = g.point_cells;
    view->point_ids = g.point_ids;
    view->cell_starts = reinterpret_cast<const int*>(g.cell_ranges);
    view->cell_ends = reinterpret_cast<const int*>(g.cell_ranges) + 1;
    view->cell_stride = 2;
    view->num_points = g.num_points;
    view->dim_x = g.dx;
    view->dim_y = g.dy;
    view->dim_z = g.dz;
    view->cell_width = g.cell_width;
    view->cell_width_inv = g.cell_inv;
    view->built = g.built;
    return NSPH_OK;
}

extern "C" int nsph_sph_enable_phase_timing(nsph_sph* s, int enable)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    for (cudaEvent_t* set : {s->ev, s->eva}) {
        const int count = set == s->ev ? 4 : 6;
        for (int k = 0; k < count; ++k) {
            cudaEvent_t& e = set[k];
            if (enable && !e) NSPH_CUDA_TRY(cudaEventCreate(&e));
            if (!enable && e) {
                NSPH_CUDA_TRY(cudaEventDestroy(e));
                e = nullptr;
            }
        }
    }
    return NSPH_OK;
}

extern "C" int nsph_sph_phase_times(nsph_sph* s, float ms_out[3])
{
    clear_error();
    if (!s || !ms_out) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    if (!s->ev[0]) return fail(NSPH_ERR_INVALID_ARG, "phase timing is not enabled");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaEventSynchronize(s->ev[3]));
    for (int k = 0; k < 3; ++k) NSPH_CUDA_TRY(cudaEventElapsedTime(ms_out + k, s->ev[k], s->ev[k + 1]));
    return NSPH_OK;
}

extern "C" int nsph_sph_set_launch(nsph_sph* s, int threads, int blocks_per_sm)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (threads != 0 && (threads < 32 || threads > kSphThreads || (threads & 31)))
        return fail(NSPH_ERR_INVALID_ARG, "threads must be 0 or a multiple of 32 in [32, 256]");
    if (blocks_per_sm < -1 || blocks_per_sm > 64) return fail(NSPH_ERR_INVALID_ARG, "blocks_per_sm out of [-1, 64]");
    s->launch_threads = threads;
    s->launch_blocks_per_sm = blocks_per_sm;
    return NSPH_OK;
}

extern "C" int nsph_sph_last_launches(const nsph_sph* s) { return s ? s->last_launches : 0; }

extern "C" int nsph_sph_status(nsph_sph* s, unsigned int* status, void* stream)
{
    clear_error();
    if (!s || !status) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaMemcpyAsync(status, s->status, sizeof(unsigned), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    NSPH_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    return NSPH_OK;
}

extern "C" int nsph_sph_reset_status(nsph_sph* s, void* stream)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaMemsetAsync(s->status, 0, sizeof(unsigned), (cudaStream_t)stream));
    return NSPH_OK;
}

// ==========================================================================
// C ABI: adjoint of the step
// ==========================================================================
extern "C" int nsph_sph_enable_adjoint(nsph_sph* s)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (s->grid.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the adjoint supports single-world solvers only");
    if (s->adj_gd) return NSPH_OK;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    const size_t c = (size_t)(s->capacity > 0 ? s->capacity : 1);
    const int bcap = (int)((c + 31) / 32) + 1;  // blocks of a pass of >= 32 threads per block, or of 64 particles
    cudaError_t e = cudaMalloc(&s->adj_gd, sizeof(float4) * 2 * c);
    if (e == cudaSuccess) e = cudaMalloc(&s->adj_xv, sizeof(float4) * 2 * c);
    if (e == cudaSuccess) e = cudaMalloc(&s->adj_rho, sizeof(float) * c);
    if (e == cudaSuccess) e = cudaMalloc(&s->adj_bpart, sizeof(float) * (size_t)bcap);
    cudaFuncAttributes fa;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_adj_local);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_adj_pair<1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_adj_density<1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_adj_pair<4>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_adj_density<4>);
    if (e != cudaSuccess) {
        cudaGetLastError();
        cudaFree(s->adj_gd);
        cudaFree(s->adj_xv);
        cudaFree(s->adj_rho);
        cudaFree(s->adj_bpart);
        s->adj_gd = s->adj_xv = nullptr;
        s->adj_rho = s->adj_bpart = nullptr;
        return fail(NSPH_ERR_OUT_OF_MEMORY, std::string("adjoint allocation: ") + cudaGetErrorString(e));
    }
    s->adj_bcap = bcap;
    return NSPH_OK;
}

// The adjoint kernels of one step whose build and density outputs are `ts`
// (its grid seen through g). mark: record the adjoint phase events.
static int adjoint_kernels(nsph_sph* s, const nsph_sph_params* p, int n, const GridDev& g, const TapeStep& ts,
                           const AdjIO& io, float* eos_b_adj, cudaStream_t cs, int& launches, bool mark)
{
    int blocks, threads;
    pass_launch(s, n, false, blocks, threads);
    NSPH_CUDA_TRY(launch_dependent(k_adj_local, blocks, threads, 0, cs,
                                   g, ts.xs, ts.vs, ts.fr, n, *p, ts.nbr, ts.ncnt, io));
    NSPH_LAUNCH_CHECK("k_adj_local");
    if (mark && s->eva[3]) NSPH_CUDA_TRY(record_mark(s->eva[3], cs));
    const bool quad = quad_pass(s, n);
    const int pair_blocks = quad ? (4 * n + kSphThreads - 1) / kSphThreads : blocks;
    const int pair_threads = quad ? kSphThreads : threads;
    if (quad)
        NSPH_CUDA_TRY(launch_dependent(k_adj_pair<4>, pair_blocks, pair_threads, 0, cs,
                                       g, ts.xs, ts.vs, ts.fr, ts.rp, n, *p, ts.nbr, ts.ncnt, io));
    else
        NSPH_CUDA_TRY(launch_dependent(k_adj_pair<1>, pair_blocks, pair_threads, 0, cs,
                                       g, ts.xs, ts.vs, ts.fr, ts.rp, n, *p, ts.nbr, ts.ncnt, io));
    NSPH_LAUNCH_CHECK("k_adj_pair");
    if (mark && s->eva[4]) NSPH_CUDA_TRY(record_mark(s->eva[4], cs));
    if (quad)
        NSPH_CUDA_TRY(launch_dependent(k_adj_density<4>, pair_blocks, pair_threads, 0, cs,
                                       g, ts.xs, ts.vs, n, *p, ts.nbr, ts.ncnt, io.rho, io.xv, io.x_in_adj));
    else
        NSPH_CUDA_TRY(launch_dependent(k_adj_density<1>, pair_blocks, pair_threads, 0, cs,
                                       g, ts.xs, ts.vs, n, *p, ts.nbr, ts.ncnt, io.rho, io.xv, io.x_in_adj));
    NSPH_LAUNCH_CHECK("k_adj_density");
    launches += 3;
    if (eos_b_adj) {
        NSPH_CUDA_TRY(launch_dependent(k_adj_b_reduce, 1, 256, 0, cs,
                                       io.bpart, pair_blocks, eos_b_adj));
        NSPH_LAUNCH_CHECK("k_adj_b_reduce");
        ++launches;
    }
    return NSPH_OK;
}

// Enqueue the reverse of one step on validated inputs.
static int adjoint_enqueue(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in, const float* v_in,
                           const float* f_ext, const float* mass, const float* inv_mass, const int* flags,
                           const int* world, const float* gravity, int world_count, const float* x_out_adj,
                           const float* v_out_adj, const float* rho_out_adj, float* x_in_adj, float* v_in_adj,
                           float* f_ext_adj, float* eos_b_adj, cudaStream_t cs, int& launches)
{
    GatherArgs ga{x_in, v_in, mass, inv_mass, flags, world, world_count, s->xs, s->vs};
    if (s->eva[0]) NSPH_CUDA_TRY(record_mark(s->eva[0], cs));
    int st = grid_build(s->grid, x_in, n, p->cell_width, p->cell_inv, &ga, s->status, cs, &launches);
    if (st != NSPH_OK) return st;
    s->last_n = n;
    if (s->eva[1]) NSPH_CUDA_TRY(record_mark(s->eva[1], cs));
    if (n > 0) {
        const GridDev g = s->grid.view();
        st = density_enqueue(s, g, p, n, false, s->xs, s->vs, s->rp, s->nbr, s->ncnt, s->fr, cs, launches);
        if (st != NSPH_OK) return st;
        if (s->eva[2]) NSPH_CUDA_TRY(record_mark(s->eva[2], cs));
        const AdjIO io{x_out_adj, v_out_adj, rho_out_adj, x_in_adj, v_in_adj, f_ext_adj, f_ext, inv_mass, gravity,
                       s->adj_gd, s->adj_xv, s->adj_rho, s->adj_bpart};
        const TapeStep ts{s->xs, s->vs, s->rp, s->fr, s->nbr, s->ncnt, nullptr, nullptr, nullptr};
        st = adjoint_kernels(s, p, n, g, ts, io, eos_b_adj, cs, launches, true);
        if (st != NSPH_OK) return st;
    } else {
        for (int k = 2; k < 5; ++k)
            if (s->eva[k]) NSPH_CUDA_TRY(record_mark(s->eva[k], cs));
    }
    if (s->eva[5]) NSPH_CUDA_TRY(record_mark(s->eva[5], cs));
    return NSPH_OK;
}

static int check_adjoint_ready(const nsph_sph* s)
{
    if (s->grid.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the adjoint supports single-world solvers only");
    if (!s->adj_gd) return fail(NSPH_ERR_INVALID_ARG, "adjoint scratch not allocated (nsph_sph_enable_adjoint)");
    return NSPH_OK;
}

extern "C" int nsph_sph_step_adjoint(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in,
                                     const float* v_in, const float* f_ext, const float* mass, const float* inv_mass,
                                     const int* flags, const int* world, const float* gravity, int world_count,
                                     const float* x_out_adj, const float* v_out_adj, const float* rho_out_adj,
                                     float* x_in_adj, float* v_in_adj, float* f_ext_adj, float* eos_b_adj,
                                     void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_step_adjoint");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_adjoint_ready(s);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x_in, v_in, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (n > 0 && (!x_out_adj || !v_out_adj || !x_in_adj || !v_in_adj))
        return fail(NSPH_ERR_INVALID_ARG, "null adjoint array");
    if (n > 0 && ((const float*)x_in_adj == v_out_adj || (const float*)v_in_adj == x_out_adj || x_in_adj == v_in_adj))
        return fail(NSPH_ERR_INVALID_ARG, "position and velocity adjoints must not share memory");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    int launches = 0;
    st = adjoint_enqueue(s, p, n, x_in, v_in, f_ext, mass, inv_mass, flags, world, gravity, world_count, x_out_adj,
                         v_out_adj, rho_out_adj, x_in_adj, v_in_adj, f_ext_adj, eos_b_adj, (cudaStream_t)stream,
                         launches);
    s->last_launches = launches;
    return st;
}

extern "C" int nsph_sph_rollout_adjoint(nsph_sph* s, const nsph_sph_params* p, int n, int steps,
                                        const float* x_states, const float* v_states, const float* f_ext,
                                        const float* mass, const float* inv_mass, const int* flags, const int* world,
                                        const float* gravity, int world_count, float* x_adj, float* v_adj,
                                        float* f_ext_adj, float* eos_b_adj, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_rollout_adjoint");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_adjoint_ready(s);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x_states, v_states, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (steps < 0) return fail(NSPH_ERR_INVALID_ARG, "negative step count");
    const size_t len = 3 * (size_t)n;
    if (n > 0 && steps > 0) {
        if (!x_adj || !v_adj) return fail(NSPH_ERR_INVALID_ARG, "null adjoint array");
        const size_t tot = len * (size_t)steps;
        if (overlaps(x_adj, len, v_adj, len) || overlaps(x_adj, len, x_states, tot) ||
            overlaps(x_adj, len, v_states, tot) || overlaps(v_adj, len, x_states, tot) ||
            overlaps(v_adj, len, v_states, tot))
            return fail(NSPH_ERR_INVALID_ARG, "adjoint arrays overlap each other or the states");
    }
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    int launches = 0;
    for (int t = steps - 1; t >= 0 && n > 0; --t) {
        st = adjoint_enqueue(s, p, n, x_states + (size_t)t * len, v_states + (size_t)t * len, f_ext, mass, inv_mass,
                             flags, world, gravity, world_count, x_adj, v_adj, nullptr, x_adj, v_adj, f_ext_adj,
                             eos_b_adj, cs, launches);
        if (st != NSPH_OK) return st;
    }
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_reserve_segment(nsph_sph* s, int steps)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (s->grid.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the adjoint supports single-world solvers only");
    if (steps < 0) return fail(NSPH_ERR_INVALID_ARG, "negative step count");
    if (steps <= s->tape_steps) return NSPH_OK;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    const size_t c = (size_t)(s->capacity > 0 ? s->capacity : 1);
    const size_t slot = tape_slot_bytes(c, s->grid.ncells);
    const size_t bytes = slot * (size_t)steps + tape_align(sizeof(float) * 12 * c) + sizeof(unsigned) * (size_t)steps;
    char* t = nullptr;
    const cudaError_t e = cudaMalloc(&t, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(NSPH_ERR_OUT_OF_MEMORY, "segment tape of " + std::to_string(bytes) + " bytes: " +
                                                cudaGetErrorString(e));
    }
    cudaFree(s->tape);
    s->tape = t;
    s->tape_steps = steps;
    s->tape_step_bytes = slot;
    return NSPH_OK;
}

extern "C" int nsph_sph_segment_adjoint(nsph_sph* s, const nsph_sph_params* p, int n, int steps, const float* x0,
                                        const float* v0, const float* f_ext, const float* mass,
                                        const float* inv_mass, const int* flags, const int* world,
                                        const float* gravity, int world_count, float* x_adj, float* v_adj,
                                        float* f_ext_adj, float* eos_b_adj, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_segment_adjoint");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_adjoint_ready(s);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x0, v0, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (steps < 0) return fail(NSPH_ERR_INVALID_ARG, "negative step count");
    const size_t len = 3 * (size_t)n;
    if (n > 0 && steps > 0) {
        if (!x_adj || !v_adj) return fail(NSPH_ERR_INVALID_ARG, "null adjoint array");
        if (overlaps(x_adj, len, v_adj, len) || overlaps(x_adj, len, x0, len) || overlaps(x_adj, len, v0, len) ||
            overlaps(v_adj, len, x0, len) || overlaps(v_adj, len, v0, len))
            return fail(NSPH_ERR_INVALID_ARG, "adjoint arrays overlap each other or the initial state");
    }
    if (n == 0 || steps == 0) {
        s->last_launches = 0;
        return NSPH_OK;
    }
    st = nsph_sph_reserve_segment(s, steps);
    if (st != NSPH_OK) return st;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    int launches = 0;
    int blocks, threads;
    pass_launch(s, n, false, blocks, threads);
    // forward: the build, density and force passes of every step, their
    // outputs into the step's slot (the last step's new state is not used)
    NSPH_CUDA_TRY(cudaMemsetAsync(tape_overflow(s), 0, sizeof(unsigned) * (size_t)steps, cs));
    for (int t = 0; t < steps; ++t) {
        const float* xi = t == 0 ? x0 : tape_state(s, t & 1);
        const float* vi = t == 0 ? v0 : tape_state(s, t & 1) + len;
        TapeStep ts = tape_slot(s, t);
        ts.fr.overflow = tape_overflow(s) + t;
        GatherArgs ga{xi, vi, mass, inv_mass, flags, world, world_count, ts.xs, ts.vs};
        st = grid_build(s->grid, xi, n, p->cell_width, p->cell_inv, &ga, s->status, cs, &launches);
        if (st != NSPH_OK) return st;
        const GridDev g = s->grid.view();
        st = density_enqueue(s, g, p, n, false, ts.xs, ts.vs, ts.rp, ts.nbr, ts.ncnt, ts.fr, cs, launches);
        if (st != NSPH_OK) return st;
        float* xo = tape_state(s, (t + 1) & 1);
        float* vo = xo + len;
        // the sorted ids and, where a list overflowed, the cell table into the slot
        NSPH_CUDA_TRY(launch_dependent(k_tape_copy, s->sms * 2, 512, 0, cs, g, s->grid.ncells, n, ts.fr.overflow, ts.ids,
                                       ts.ranges));
        NSPH_LAUNCH_CHECK("k_tape_copy");
        ++launches;
        // inactive particles keep their velocity
        const StepOut o{f_ext, inv_mass, gravity, xo, vo, nullptr, nullptr, nullptr, s->status, ts.acc, true};
        if (quad_pass(s, n))
            NSPH_CUDA_TRY(launch_dependent(k_force_quad, (4 * n + kQuadThreads - 1) / kQuadThreads, kQuadThreads, 0, cs,
                                           g, ts.xs, ts.vs, ts.fr, ts.rp, n, *p, ts.nbr, ts.ncnt, o));
        else
            NSPH_CUDA_TRY(launch_plain(k_force_list<false>, blocks, threads, 0, cs,
                                           g, ts.xs, ts.vs, ts.fr, ts.rp, n, *p, ts.nbr, ts.ncnt, o));
        NSPH_LAUNCH_CHECK("k_force_list");
        ++launches;
    }
    // the solver's mirrors describe its grid's last build (the last step's input)
    const TapeStep last = tape_slot(s, steps - 1);
    NSPH_CUDA_TRY(cudaMemcpyAsync(s->xs, last.xs, sizeof(float4) * (size_t)n, cudaMemcpyDeviceToDevice, cs));
    NSPH_CUDA_TRY(cudaMemcpyAsync(s->vs, last.vs, sizeof(float4) * (size_t)n, cudaMemcpyDeviceToDevice, cs));
    s->last_n = n;
    // reverse, from the slots
    AdjIO io{x_adj, v_adj, nullptr, x_adj, v_adj, f_ext_adj, f_ext, inv_mass, gravity,
             s->adj_gd, s->adj_xv, s->adj_rho, s->adj_bpart, nullptr};
    for (int t = steps - 1; t >= 0; --t) {
        const TapeStep ts = tape_slot(s, t);
        io.acc = ts.acc;
        GridDev g = s->grid.view();
        g.ranges = ts.ranges;
        g.ids = ts.ids;
        // phase events: the build and density phases of a step reversed from
        // the tape are empty (the recompute ran them)
        for (int k = 0; k < 3; ++k)
            if (s->eva[k]) NSPH_CUDA_TRY(record_mark(s->eva[k], cs));
        st = adjoint_kernels(s, p, n, g, ts, io, eos_b_adj, cs, launches, true);
        if (st != NSPH_OK) return st;
        if (s->eva[5]) NSPH_CUDA_TRY(record_mark(s->eva[5], cs));
    }
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_adjoint_phase_times(nsph_sph* s, float ms_out[5])
{
    clear_error();
    if (!s || !ms_out) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    if (!s->eva[0]) return fail(NSPH_ERR_INVALID_ARG, "phase timing is not enabled");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaEventSynchronize(s->eva[5]));
    for (int k = 0; k < 5; ++k) NSPH_CUDA_TRY(cudaEventElapsedTime(ms_out + k, s->eva[k], s->eva[k + 1]));
    return NSPH_OK;
}

// ==========================================================================
// C ABI: surrogate step
// ==========================================================================
// Default launch of the fused surrogate kernel: CTAs of two 128-particle
// tiles sharing the weights, as many per SM as fit (3: registers), with the
// carveout they need. Measured on the relaxed 1M tank (same box, back to
// back): 0.273 ms per launch; one tile per CTA: 0.292 ms at 5 CTAs per SM,
// 0.319 at 4, 0.395 at 6 (which leaves about 28 KB of L1 for the gathers).
constexpr int kSurrogateCtasPerSm = 5;  // CTAs per SM when tiles_per_cta = 1
constexpr int kSurrogateGroups = 2;

// resident CTAs per SM of a fused surrogate kernel: registers (allocated per
// warp in units of 256), shared memory (plus the per-CTA reservation) and
// the SM's 512 TMEM columns; 0 on a CUDA error
template <class K>
static int surrogate_per_sm(K kernel, int threads, size_t smem, int tmem_cols, int device)
{
    cudaFuncAttributes fa;
    int smem_sm = 0, reserved = 0, regs_sm = 0;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const int warp_regs = ((fa.numRegs * 32 + 255) / 256) * 256;
    const int by_regs = regs_sm / (warp_regs * (threads / 32));
    const int by_smem = smem_sm / (int)(smem + fa.sharedSizeBytes + reserved);
    return std::min(std::min(by_regs, by_smem), kTmemCols / tmem_cols);
}

static int set_surrogate_ctas(nsph_sph* s, int ctas_per_sm, int groups)
{
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    int sms = 0, smem_sm = 0, reserved = 0;
    NSPH_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->grid.device));
    NSPH_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, s->grid.device));
    NSPH_CUDA_TRY(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, s->grid.device));
    if (groups == 0) groups = kSurrogateGroups;
    const size_t smem = groups == 2 ? sizeof(MlpFwdGroupSmem<2>) : sizeof(MlpFwdSmem);
    const int most = groups == 2 ? surrogate_per_sm(k_surrogate_fused_groups<2>, 2 * kMlpTile, smem,
                                                    2 * (int)kMlpFwdCols, s->grid.device)
                                 : surrogate_per_sm(k_surrogate_fused, kMlpTile, smem, (int)kMlpFwdCols,
                                                    s->grid.device);
    if (most <= 0 || sms <= 0 || smem_sm <= 0) return fail(NSPH_ERR_CUDA, "cannot size the surrogate grid");
    const int def = groups == 2 ? most : kSurrogateCtasPerSm;
    const int per_sm = std::max(1, std::min(ctas_per_sm == 0 ? def : ctas_per_sm, most));
    // the shared-memory carveout that holds per_sm CTAs, so that the rest of
    // the SM's unified L1 / shared storage serves the neighbour gathers
    const int need = per_sm * (int)(smem + reserved);
    const int pct = std::min(100, (need * 100 + smem_sm - 1) / smem_sm);
    if (groups == 2)
        NSPH_CUDA_TRY(
            cudaFuncSetAttribute(k_surrogate_fused_groups<2>, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
    else
        NSPH_CUDA_TRY(cudaFuncSetAttribute(k_surrogate_fused, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
    s->surr_ctas = sms * per_sm;
    s->surr_groups = groups;
    return NSPH_OK;
}

extern "C" int nsph_sph_enable_surrogate(nsph_sph* s)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (s->grid.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the surrogate supports single-world solvers only");
    if (s->sfeat) return NSPH_OK;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    const size_t c = (size_t)(s->capacity > 0 ? s->capacity : 1);
    const size_t blocks = std::max((c + 31) / 32 + 1, (size_t)4096);  // per-block partials of either pass
    cudaError_t e = cudaMalloc(&s->sfeat, sizeof(float) * kFeat * c);
    if (e == cudaSuccess) e = cudaMalloc(&s->sacc, sizeof(float4) * 2 * c);
    if (e == cudaSuccess) e = cudaMalloc(&s->cpart, sizeof(float) * 2 * blocks);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_surrogate_fused, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(MlpFwdSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_surrogate_fused_groups<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(MlpFwdGroupSmem<2>));
    if (e == cudaSuccess) {  // an upper bound on either kernel's grid, for the partials
        const int most = mlp_resident_grid(k_surrogate_fused, sizeof(MlpFwdSmem), s->grid.device);
        if (most <= 0) e = cudaErrorUnknown;
        else if (most + 1 > (int)blocks) e = cudaErrorInvalidValue;
    }
    cudaFuncAttributes fa;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_force_features_list);
    if (e != cudaSuccess) {
        cudaGetLastError();
        cudaFree(s->sfeat);
        cudaFree(s->sacc);
        cudaFree(s->cpart);
        s->sfeat = s->cpart = nullptr;
        s->sacc = nullptr;
        return fail(NSPH_ERR_OUT_OF_MEMORY, std::string("surrogate allocation: ") + cudaGetErrorString(e));
    }
    return set_surrogate_ctas(s, 0, 0);  // the default launch and its carveout
}

// grid build, density pass and (with `features`) the feature pass into the
// sorted scratch (with `mark`, records phase events 0-2 when phase timing is
// enabled: start, built, after the density pass)
static int features_enqueue(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in, const float* v_in,
                            const float* mass, const float* inv_mass, const int* flags, const int* world,
                            int world_count, cudaStream_t cs, int& launches, int& blocks, bool mark = false,
                            bool features = true)
{
    GatherArgs ga{x_in, v_in, mass, inv_mass, flags, world, world_count, s->xs, s->vs};
    if (mark && s->eva[0]) NSPH_CUDA_TRY(record_mark(s->eva[0], cs));
    int st = grid_build(s->grid, x_in, n, p->cell_width, p->cell_inv, &ga, s->status, cs, &launches);
    if (st != NSPH_OK) return st;
    s->last_n = n;
    blocks = 0;
    if (mark && s->eva[1]) NSPH_CUDA_TRY(record_mark(s->eva[1], cs));
    if (n > 0) {
        const GridDev g = s->grid.view();
        int threads;
        st = density_enqueue(s, g, p, n, false, s->xs, s->vs, s->rp, s->nbr, s->ncnt, s->fr, cs, launches);
        if (st != NSPH_OK) return st;
        if (mark && s->eva[2]) NSPH_CUDA_TRY(record_mark(s->eva[2], cs));
        pass_launch(s, n, false, blocks, threads);
        if (features) {
            NSPH_CUDA_TRY(launch_plain(k_force_features_list, blocks, threads, 0, cs,
                                           g, s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, s->sfeat, s->sacc, s->cpart));
            NSPH_LAUNCH_CHECK("k_force_features_list");
            ++launches;
        }
    } else if (mark && s->eva[2]) {
        NSPH_CUDA_TRY(record_mark(s->eva[2], cs));
    }
    return NSPH_OK;
}

static int check_surrogate_ready(const nsph_sph* s)
{
    if (s->grid.world_count > 0) return fail(NSPH_ERR_INVALID_ARG, "the surrogate supports single-world solvers only");
    if (!s->sfeat) return fail(NSPH_ERR_INVALID_ARG, "surrogate scratch not allocated (nsph_sph_enable_surrogate)");
    return NSPH_OK;
}

extern "C" int nsph_sph_features(nsph_sph* s, const nsph_sph_params* p, int n, const float* x_in, const float* v_in,
                                 const float* mass, const float* inv_mass, const int* flags, const int* world,
                                 const float* gravity, int world_count, float* feat_out, float* acc_out,
                                 float* rho_out, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_features");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_surrogate_ready(s);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x_in, v_in, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    int launches = 0, blocks = 0;
    st = features_enqueue(s, p, n, x_in, v_in, mass, inv_mass, flags, world, world_count, cs, launches, blocks);
    if (st != NSPH_OK) return st;
    if (n > 0 && (feat_out || acc_out)) {
        NSPH_CUDA_TRY(launch_dependent(k_scatter_features, (n + 255) / 256, 256, 0, cs,
                                       s->grid.point_ids, n, s->sfeat, s->sacc, feat_out, acc_out));
        NSPH_LAUNCH_CHECK("k_scatter_features");
        ++launches;
    }
    if (n > 0 && rho_out) {
        NSPH_CUDA_TRY(launch_dependent(k_scatter_rho, (n + 255) / 256, 256, 0, cs,
                                       s->grid.point_ids, n, s->rp, rho_out));
        NSPH_LAUNCH_CHECK("k_scatter_rho");
        ++launches;
    }
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_step_surrogate(nsph_sph* s, const nsph_sph_params* p, const float* model, float acc_scale,
                                       int n, const float* x_in, const float* v_in, const float* f_ext,
                                       const float* mass, const float* inv_mass, const int* flags, const int* world,
                                       const float* gravity, int world_count, float* x_out, float* v_out,
                                       float* rho_out, float* p_out, float* stats, void* stream)
{
    clear_error();
    NvtxRange nvtx_range("nsph_sph_step_surrogate");
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    int st = check_params(p);
    if (st == NSPH_OK) st = check_surrogate_ready(s);
    if (st == NSPH_OK) st = check_step_inputs(s, n, x_in, v_in, mass, inv_mass, flags, gravity, world_count);
    if (st != NSPH_OK) return st;
    if (n > 0 && (!x_out || !v_out || !model || !stats)) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    if (n > 0 && (x_out == x_in || v_out == v_in))
        return fail(NSPH_ERR_INVALID_ARG, "state_out must not alias state_in");
    if (!isfinite(acc_scale)) return fail(NSPH_ERR_INVALID_ARG, "acc_scale must be finite");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    cudaStream_t cs = (cudaStream_t)stream;
    int launches = 0, blocks = 0;
    st = features_enqueue(s, p, n, x_in, v_in, mass, inv_mass, flags, world, world_count, cs, launches, blocks,
                          true, false);
    if (st != NSPH_OK) return st;
    if (n > 0) {
        const int tiles = (n + kMlpTile - 1) / kMlpTile;
        const int wait_limit = s->surr_wait_limit >= 0 ? s->surr_wait_limit : kMlpWaitLimit;
        const StepOut o{f_ext, inv_mass, gravity, x_out, v_out, rho_out, p_out, nullptr, s->status};
        int grid;
        if (s->surr_groups == 2) {
            grid = std::min((tiles + 1) / 2, std::max(1, s->surr_ctas));
            NSPH_CUDA_TRY(launch_plain(k_surrogate_fused_groups<2>, grid, 2 * kMlpTile, sizeof(MlpFwdGroupSmem<2>), cs,
                                           model, acc_scale, wait_limit, s->grid.view(), s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, o, s->cpart));
            NSPH_LAUNCH_CHECK("k_surrogate_fused_groups");
        } else {
            grid = std::min(tiles, std::max(1, s->surr_ctas));
            NSPH_CUDA_TRY(launch_plain(k_surrogate_fused, grid, kMlpTile, sizeof(MlpFwdSmem), cs,
                                           model, acc_scale, wait_limit, s->grid.view(), s->xs, s->vs, s->fr, s->rp, n, *p, s->nbr, s->ncnt, o, s->cpart));
            NSPH_LAUNCH_CHECK("k_surrogate_fused");
        }
        if (s->eva[3]) NSPH_CUDA_TRY(record_mark(s->eva[3], cs));
        NSPH_CUDA_TRY(launch_dependent(k_compression_reduce, 1, 256, 0, cs,
                                       s->cpart, grid, stats));
        NSPH_LAUNCH_CHECK("k_compression_reduce");
        launches += 2;
    } else if (s->eva[3]) {
        NSPH_CUDA_TRY(record_mark(s->eva[3], cs));
    }
    if (s->eva[4]) NSPH_CUDA_TRY(record_mark(s->eva[4], cs));
    s->last_launches = launches;
    return NSPH_OK;
}

extern "C" int nsph_sph_set_surrogate_launch(nsph_sph* s, int ctas_per_sm, int tiles_per_cta)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (ctas_per_sm < 0 || ctas_per_sm > 64) return fail(NSPH_ERR_INVALID_ARG, "ctas_per_sm out of [0, 64]");
    if (tiles_per_cta < 0 || tiles_per_cta > 2) return fail(NSPH_ERR_INVALID_ARG, "tiles_per_cta out of [0, 2]");
    if (!s->sfeat) return fail(NSPH_ERR_INVALID_ARG, "surrogate not enabled (nsph_sph_enable_surrogate)");
    return set_surrogate_ctas(s, ctas_per_sm, tiles_per_cta);
}

extern "C" int nsph_sph_set_surrogate_wait_limit(nsph_sph* s, int polls)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (polls < -1) return fail(NSPH_ERR_INVALID_ARG, "poll count below -1");
    s->surr_wait_limit = polls;
    return NSPH_OK;
}

extern "C" int nsph_sph_set_arithmetic(nsph_sph* s, int mode)
{
    clear_error();
    if (!s) return fail(NSPH_ERR_INVALID_ARG, "null solver");
    if (mode != NSPH_ARITH_EXACT && mode != NSPH_ARITH_FAST) return fail(NSPH_ERR_INVALID_ARG, "unknown arithmetic");
    s->fast = mode == NSPH_ARITH_FAST;
    return NSPH_OK;
}

extern "C" int nsph_sph_surrogate_phase_times(nsph_sph* s, float ms_out[4])
{
    clear_error();
    if (!s || !ms_out) return fail(NSPH_ERR_INVALID_ARG, "null argument");
    if (!s->eva[0]) return fail(NSPH_ERR_INVALID_ARG, "phase timing is not enabled");
    DeviceGuard guard(s->grid.device);
    if (!guard.ok) return fail(NSPH_ERR_CUDA, "cannot select CUDA device");
    NSPH_CUDA_TRY(cudaEventSynchronize(s->eva[4]));
    for (int k = 0; k < 4; ++k) NSPH_CUDA_TRY(cudaEventElapsedTime(ms_out + k, s->eva[k], s->eva[k + 1]));
    return NSPH_OK;
}
