// The natural-order Gauss-Seidel sweep (src/ComputeSYMGS_ref.cpp:51-104) as
// one dataflow kernel per direction.
//
// What bounds it: the sweep is a chain of nx + 2 (ny-1) + 4 (nz-1) dependent
// rows (natural.cuh's fronts), each a chain of 20 FP64 adds and a division;
// one launch per front takes 11.7 us a front (104^3 step, 1444 launches: 16.8 ms,
// the host issues them), this form 0.77 us with the check and the re-laying (1.11
// ms), 0.68 in the sweeps alone, hand-offs between blocks included (0.34 within a
// block of one plane): the 104^3 reference V-cycle went from 54.8 to 3.9 ms.  Here
// a block owns a group of z planes, one thread per grid line along x, and steps
// along s = ix + 2 iy; plane lz of the group runs four steps behind plane lz - 1,
// which is the fronts' order, so one __syncthreads per front replaces a launch and
// new values pass between lines through shared memory.  Groups pipeline: the last plane of a group is read
// by the next group's block from global memory, every value being its own
// ready flag (the buffer is filled with a NaN pattern no computation returns),
// so a value costs one L2 round trip and no fence.
//
// The vectors are first re-laid as [iz][s mod nx][iy] (a permutation of the
// level, no padding), so that a step's loads and stores are contiguous over
// the lines of a plane.  The matrix is read once per level, by the kernel
// that checks it: where every row is the generated 27-point row (columns,
// count and diagonal slot in place, off-diagonals -1) the sweeps need the
// diagonal only, and sum - (-1 * x) is sum + x bit for bit; any other matrix
// leaves the flag set and takes k_nat_gs_fronts, the per-front sweep with a
// grid barrier between fronts.
#include <math_constants.h>

#include <algorithm>

#include "natural.cuh"

namespace hb {

namespace {

constexpr int kRing = 24;        // staged steps of x per line
constexpr int kHalf = kRing / 2; // steps the loop is unrolled over
constexpr int kAhead = 18;       // steps between an x copy's issue and its own step
constexpr int kRowRing = 12;     // staged steps of r and a_ii
constexpr int kRowAhead = 11;
constexpr int kLanded = 9;       // copies still in flight when a step ends
constexpr int kLag = 4;          // steps between neighbouring planes
constexpr int kFlowMaxLines = 256;  // one plane and its two neighbours fit shared memory
constexpr int kFlowSmem = 226 * 1024;
constexpr int kBS = 256;
constexpr unsigned long long kUnset = ~0ull;           // not yet computed
constexpr unsigned long long kFlowTimeoutNs = 1000000000ull;

struct FlowArgs
{
    int nx, ny, nz;
    int planes;                  // planes per group
    const double* xold;          // skewed: values before this sweep
    double* xnew;                // skewed: values of this sweep, filled with kUnset
    const double* r;             // skewed
    const double* diag;          // skewed
    const int* other;            // != 0: the matrix is not the generated stencil (nothing to do here)
    int* status;
};

__device__ __forceinline__ double ld_flag(const double* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
}

__device__ __forceinline__ void st_flag(double* p, double v)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if(b == kUnset) b = 0x7ff8000000000000ull;  // an input NaN with the flag's bits stays a NaN
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

__device__ __forceinline__ bool unset(double v) { return (unsigned long long)__double_as_longlong(v) == kUnset; }

__device__ __forceinline__ void copy8_async(double* smem, const double* gmem)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a), "l"(gmem) : "memory");
}

// One sweep.  Everything runs in coordinates mirrored for the backward sweep
// (kDir < 0), so "earlier" is always the smaller index; the sum keeps the
// natural slot order, which is the mirrored order reversed.
//
// Warps of plane p < planes: a lane is line i of plane p.  At step t it
// stands at s = t - 4 p, that is ix = s - 2 i.  Warps of p == planes: line i
// of the two halo planes -- they wait for the new values below the group and
// copy the old ones above it.  xring[plane + 1][slot][line + 1] holds -0.0 for
// points outside the grid (v + -0.0 is v), old values, and new ones once their
// row is done; the slot of plane p's step s is (s + 4 p) mod 24 = t mod 24, so
// with the loop unrolled over half the ring every slot is an immediate offset.  At
// step t the slots t - 5 .. t + 7 of a plane are read, t + 18 = t - 6 is
// being copied.  A thread keeps its 27 neighbours in registers (nine lines of
// three, the newest replacing the oldest each step) and starts the sum of
// step s + 1 with the terms that step s does not produce (forward slots 0-7,
// backward slots 0-13) while the sum of step s waits on its chain of adds.
// kPitch: ring columns of a plane (ny + 2 at most), a constant so that every
// ring access is a base register and an immediate.
template <int kDir, int kPitch, int kThreads>
__global__ void __launch_bounds__(kThreads, 1) k_nat_gs_flow(const FlowArgs a)
{
    extern __shared__ double smem[];
    __shared__ int dead;
    if(*a.other) return;
    const int nx = a.nx, ny = a.ny, nz = a.nz, np = a.planes;
    constexpr int row = kPitch, plane_sz = kRing * kPitch;
    const int nyp = (ny + 31) & ~31;
    const int p = threadIdx.x / nyp, i = threadIdx.x - p * nyp;
    const bool on = i < ny;
    const bool halo = p == np;
    const int iy = kDir > 0 ? i : ny - 1 - i;
    const int s_max = nx - 1 + 2 * (ny - 1);
    const int ngroups = (nz + np - 1) / np;
    double* rring = smem + (size_t)(np + 2) * plane_sz;  // [plane][slot][line], then the same for a_ii
    const int xs_total = (np + 2) * plane_sz;
    if(threadIdx.x == 0) dead = 0;

    for(int grp = blockIdx.x; grp < ngroups; grp += gridDim.x)
    {
        const int z0 = grp * np, nzg = min(np, nz - z0);
        __syncthreads();
        for(int k = threadIdx.x; k < xs_total; k += blockDim.x) smem[k] = -0.0;
        __syncthreads();

        // natural phase (s mod nx) of mirrored step s; it runs by +-1
        auto phase = [&](int s) {
            const int q = (kDir > 0 ? s : s_max - s) % nx;
            return q < 0 ? q + nx : q;
        };
        // offset of (phase, this line) in a plane, stepped with it
        struct Walk
        {
            int q, off;
        };
        auto walk = [&](int s) {
            const int q = phase(s);
            return Walk{q, q * ny + iy};
        };
        auto next = [&](Walk& w) {
            if(kDir > 0)
            {
                const bool wrap = w.q == nx - 1;
                w.q = wrap ? 0 : w.q + 1;
                w.off = wrap ? iy : w.off + ny;
            }
            else
            {
                const bool wrap = w.q == 0;
                w.q = wrap ? nx - 1 : w.q - 1;
                w.off = wrap ? (nx - 1) * ny + iy : w.off - ny;
            }
        };
        auto plane_base = [&](int z) { return (unsigned)(kDir > 0 ? z : nz - 1 - z) * (unsigned)(nx * ny); };
        const bool rows = on && p < nzg;                           // p < np follows from nzg <= np
        const bool copies = rows || (on && halo && z0 + np < nz);  // its own plane, or the one above the group
        const bool below = on && halo && grp > 0;
        // element index of the copied plane, or (halo) of the plane below the group
        const unsigned own = copies ? plane_base(z0 + p) : 0u;
        const unsigned under = below ? plane_base(z0 - 1) : 0u;
        double* cring = smem + (size_t)(p + 1) * plane_sz + i + 1;
        const bool cells = on && p <= np;  // lanes with a ring column of their own
        double* rr = rring + (size_t)p * kRowRing * row + i;
        const int dro = np * kRowRing * row;  // from r's ring to a_ii's

        const int t0 = -kLag;
        int ix = t0 - kLag * p - 2 * i;  // this lane's point at the current step (halo: in the plane above)
        int hx = t0 + kLag - 2 * i;      // halo: the point below the group it delivers
        Walk wc = walk(t0 - kLag * p), wr = wc, wo = wc, wh = walk(t0 + kLag);
        auto copy_x = [&](int cell, int x) {  // point x of the copied plane to ring offset cell
            if((unsigned)x < (unsigned)nx)
            {
                if(copies) copy8_async(cring + cell, a.xold + (own + wc.off));
            }
            else if(cells) cring[cell] = -0.0;
            next(wc);
        };
        auto copy_row = [&](int slot, int x) {
            if(rows && (unsigned)x < (unsigned)nx)
            {
                copy8_async(rr + slot * row, a.r + (own + wr.off));
                copy8_async(rr + dro + slot * row, a.diag + (own + wr.off));
            }
            next(wr);
        };
#pragma unroll 1
        for(int k = 0; k < kAhead; ++k)
        {
            copy_x(k * row, ix + k);
            if(k < kRowAhead) copy_row(k, ix + k);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");

        double hv[4] = {0.0, 0.0, 0.0, 0.0};  // halo: new values below the group, loaded four steps ahead
        if(below)
        {
#pragma unroll
            for(int k = 0; k < 4; ++k)
            {
                if((unsigned)(hx + k) < (unsigned)nx) hv[k] = ld_flag(a.xnew + (under + wh.off));
                next(wh);
            }
        }
        double w[9][3];  // line l = 3 (dz + 1) + (dy + 1); dx = c - 1 at [(u + c) mod 3]
#pragma unroll
        for(int l = 0; l < 9; ++l) w[l][0] = w[l][1] = w[l][2] = -0.0;
        double acc = 0.0, d = 1.0, xd = 0.0;  // the sum begun for the next step, its a_ii and a_ii x_i
        __syncthreads();

        const int steps = s_max + kLag * (nzg - 1) + 1;
        auto step_end = [&] {
            asm volatile("cp.async.commit_group;\ncp.async.wait_group %0;\n" ::"n"(kLanded) : "memory");
            asm volatile("bar.sync 0;\n" ::: "memory");
        };
        // One loop for the warps of the planes, one for the halo's: they meet
        // at the same barrier.  The step loop is unrolled over half the ring
        // (the whole ring: 0.44 us a step, instruction fetch); the halves'
        // offsets swap after each.
        int lo = 0, hi = kHalf * row;
        auto at = [&](int slot) {  // ring offset of `slot` steps past the half's first
            slot = (slot + 2 * kRing) % kRing;
            return slot < kHalf ? lo + slot * row : hi + (slot - kHalf) * row;
        };
        if(!halo)
        {
            const double* lines = smem + (size_t)p * plane_sz + i;  // plane p - 1, line i - 1
            // newest value (point dx = +1) of line l at loop step u
            auto newest = [&](int l, int u) {
                const int dz = l / 3, dy = l % 3;
                return lines[dz * plane_sz + at(u + kLag * (dz - 1) + 2 * dy - 1) + dy];
            };
            for(int t = t0; t < steps; t += kHalf)
            {
#pragma unroll
                for(int u = 0; u < kHalf; ++u)
                {
                    if(u % 4 == 0 && t + u >= steps) break;
                    if(rows)
                    {
                        const bool in = (unsigned)ix < (unsigned)nx;
                        const int c0 = u % 3, c1 = (u + 1) % 3, c2 = (u + 2) % 3;
                        const double d0 = d, xd0 = xd;
                        double sum = acc;
                        acc = rr[((u + 1) % kRowRing) * row];
                        d = rr[dro + ((u + 1) % kRowRing) * row];
                        if constexpr(kDir > 0)
                        {
                            // this step: the newest of lines 2..8, slots 8..26
#pragma unroll
                            for(int l = 2; l < 9; ++l) w[l][c2] = newest(l, u);
                            sum = __dadd_rn(sum, w[2][c2]);
#pragma unroll
                            for(int c = 0; c < 3; ++c) sum = __dadd_rn(sum, w[3][(u + c) % 3]);
                            sum = __dadd_rn(sum, w[4][c0]);
                            sum = __dsub_rn(sum, xd0);
                            sum = __dadd_rn(sum, w[4][c2]);
#pragma unroll
                            for(int l = 5; l < 9; ++l)
#pragma unroll
                                for(int c = 0; c < 3; ++c) sum = __dadd_rn(sum, w[l][(u + c) % 3]);
                            // next step: lines 0 and 1, slots 0..7
                            w[0][c0] = newest(0, u + 1);
                            w[1][c0] = newest(1, u + 1);
#pragma unroll
                            for(int l = 0; l < 2; ++l)
#pragma unroll
                                for(int c = 0; c < 3; ++c) acc = __dadd_rn(acc, w[l][(u + 1 + c) % 3]);
                            acc = __dadd_rn(acc, w[2][c1]);
                            acc = __dadd_rn(acc, w[2][c2]);
                            xd = __dmul_rn(d, w[4][c2]);
                        }
                        else
                        {
                            // this step: the own line's new value, the newest of lines 3..0, natural slots 14..26
                            sum = __dadd_rn(sum, w[4][c0]);
#pragma unroll
                            for(int l = 3; l >= 0; --l) w[l][c2] = newest(l, u);
#pragma unroll
                            for(int l = 3; l >= 0; --l)
#pragma unroll
                                for(int c = 2; c >= 0; --c) sum = __dadd_rn(sum, w[l][(u + c) % 3]);
                            // next step: lines 8..4, natural slots 0..13
#pragma unroll
                            for(int l = 8; l >= 4; --l) w[l][c0] = newest(l, u + 1);
#pragma unroll
                            for(int l = 8; l >= 5; --l)
#pragma unroll
                                for(int c = 2; c >= 0; --c) acc = __dadd_rn(acc, w[l][(u + 1 + c) % 3]);
                            acc = __dadd_rn(acc, w[4][c0]);
                            xd = __dmul_rn(d, w[4][c2]);
                            acc = __dsub_rn(acc, xd);
                        }
                        if(in)
                        {
                            sum = __dadd_rn(sum, xd0);  // remove the diagonal term of the loop
                            const double xn = __ddiv_rn(sum, d0);
                            w[4][c1] = xn;
                            cring[at(u)] = xn;
                            st_flag(a.xnew + (own + wo.off), xn);
                        }
                        next(wo);
                    }
                    copy_x(at(u + kAhead), ix + kAhead);
                    copy_row((u + kRowAhead) % kRowRing, ix + kRowAhead);
                    ++ix;
                    step_end();
                }
                const int swap = lo;
                lo = hi;
                hi = swap;
            }
        }
        else
        {
            for(int t = t0; t < steps; t += 4)
            {
#pragma unroll
                for(int u = 0; u < 4; ++u)
                {
                    if(below)
                    {
                        // delivered now, read by plane 0 at the next step
                        double v = hv[u];
                        if((unsigned)hx < (unsigned)nx)
                        {
                            if(unset(v) && !*(volatile int*)&dead)
                            {
                                const double* src = a.xnew + (under + phase(t + u + kLag) * ny + iy);
                                const unsigned long long began = global_ns();
                                long long spins = 0;
                                while(unset(v = ld_flag(src)))
                                    if(++spins > kBarrierSpins ||
                                       ((spins & 63) == 0 && global_ns() - began > kFlowTimeoutNs))
                                    {
                                        atomicExch(a.status, 1);
                                        *(volatile int*)&dead = 1;
                                        break;
                                    }
                            }
                            if(unset(v)) v = CUDART_NAN;
                        }
                        else v = -0.0;
                        smem[lo + i + 1] = v;
                        if((unsigned)(hx + 4) < (unsigned)nx) hv[u] = ld_flag(a.xnew + (under + wh.off));
                        next(wh);
                        ++hx;
                    }
                    const int ahead = lo + kAhead * row;
                    copy_x(ahead >= plane_sz ? ahead - plane_sz : ahead, ix + kAhead);
                    ++ix;
                    lo = lo + row == plane_sz ? 0 : lo + row;
                    step_end();
                }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
}

// Rows of the generated matrix: reads the matrix once (coalesced over the
// slots of kCheckRows consecutive rows) and sets *other where a row is not the
// generated one; writes the diagonal skewed.
constexpr int kCheckRows = 64;

__global__ void __launch_bounds__(kBS) k_nat_check_rows(NaturalLevel L, double* __restrict__ diag, int* other)
{
    __shared__ int s_dims[kCheckRows];  // bit 0-1 slots in x, 2-3 y, 4-5 z, 6/7/8: first x / y / z neighbour missing
    __shared__ int s_slot[kCheckRows];
    __shared__ int s_row[kCheckRows];   // skewed index
    __shared__ int s_off[kWidth];       // column offsets of an inside row
    constexpr int kInside = 3 | 3 << 2 | 3 << 4;
    const long long row0 = (long long)blockIdx.x * kCheckRows;
    const int nrows = (int)min((long long)kCheckRows, L.rows() - row0);
    const int nxy = L.nx * L.ny;
    bool bad = false;
    if(threadIdx.x >= kBS - kWidth)
    {
        const int q = threadIdx.x - (kBS - kWidth);
        s_off[q] = (q / 9 - 1) * nxy + (q / 3 % 3 - 1) * L.nx + q % 3 - 1;
    }
    if((int)threadIdx.x < nrows)
    {
        const int row = (int)row0 + threadIdx.x;
        const int iz = row / nxy, rem = row - iz * nxy, iy = rem / L.nx, ix = rem - iy * L.nx;
        const int x0 = ix == 0, y0 = iy == 0, z0 = iz == 0;
        const int cx = 3 - x0 - (ix == L.nx - 1), cy = 3 - y0 - (iy == L.ny - 1), cz = 3 - z0 - (iz == L.nz - 1);
        const int slot = ((1 - z0) * cy + (1 - y0)) * cx + (1 - x0);
        s_dims[threadIdx.x] = cx | cy << 2 | cz << 4 | x0 << 6 | y0 << 7 | z0 << 8;
        s_slot[threadIdx.x] = slot;
        s_row[threadIdx.x] = (iz * L.nx + (ix + 2 * iy) % L.nx) * L.ny + iy;
        bad = L.nnz[row] != cx * cy * cz || L.diag_slot[row] != slot;
    }
    __syncthreads();
    const size_t base = (size_t)row0 * kWidth;
    for(int e = threadIdx.x; e < nrows * kWidth; e += kBS)
    {
        const int l = e / kWidth, q = e - l * kWidth;
        const int c = ld_stream(L.ind + base + e);
        const double v = ld_stream(L.val + base + e);
        const int d = s_dims[l];
        if(d == kInside)
        {
            bad = bad || c - ((int)row0 + l) != s_off[q] || (q != 13 && v != -1.0);
            if(q == 13) diag[s_row[l]] = v;
            continue;
        }
        const int cx = d & 3, cy = d >> 2 & 3, cz = d >> 4 & 3;
        if(q >= cx * cy * cz) continue;
        const int t = q / cx, jx = q - t * cx, jz = t / cy, jy = t - jz * cy;
        const int dx = jx - 1 + (d >> 6 & 1), dy = jy - 1 + (d >> 7 & 1), dz = jz - 1 + (d >> 8 & 1);
        bad = bad || c != (int)row0 + l + dz * nxy + dy * L.nx + dx;
        if(q == s_slot[l]) diag[s_row[l]] = v;
        else bad = bad || v != -1.0;
    }
    if(__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(other, 1);
}

// Natural order [iz][iy][ix] <-> [iz][(ix + 2 iy) mod nx][iy], a 32 x 32 tile
// of a plane through shared memory per block.  The planes are the grid's x: there
// may be more than 65535 of them.
constexpr int kTile = 32;

template <bool kTo>
__global__ void __launch_bounds__(kBS) k_nat_skew(int nx, int ny, const double* __restrict__ in,
                                                  double* __restrict__ out, const int* other)
{
    __shared__ double tile[kTile][kTile + 1];
    if(!kTo && *other) return;
    const int x0 = blockIdx.y * kTile, y0 = blockIdx.z * kTile;
    const size_t plane = (size_t)blockIdx.x * nx * ny;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto natural = [&](auto f) {
        for(int j = warp; j < kTile; j += kBS / 32)
            if(y0 + j < ny && x0 + lane < nx) f(plane + (size_t)(y0 + j) * nx + x0 + lane, j, lane);
    };
    auto skewed = [&](auto f) {  // step s = ix + 2 iy over the tile, one line per lane
        for(int k = warp; k < 3 * kTile - 2; k += kBS / 32)
        {
            const int jx = k - 2 * lane;
            if(jx < 0 || jx >= kTile || x0 + jx >= nx || y0 + lane >= ny) continue;
            f(plane + (size_t)((x0 + 2 * y0 + k) % nx) * ny + y0 + lane, lane, jx);
        }
    };
    if(kTo) natural([&](size_t g, int jy, int jx) { tile[jy][jx] = in[g]; });
    else skewed([&](size_t g, int jy, int jx) { tile[jy][jx] = in[g]; });
    __syncthreads();
    if(kTo) skewed([&](size_t g, int jy, int jx) { out[g] = tile[jy][jx]; });
    else natural([&](size_t g, int jy, int jx) { out[g] = tile[jy][jx]; });
}

// The per-front sweep of any matrix within the stencil, fronts separated by
// a grid barrier (runs only where k_nat_check_rows set *other).
__global__ void __launch_bounds__(kBS) k_nat_gs_fronts(NaturalLevel L, const double* __restrict__ r, double* x,
                                                       const int* other, GridBarrier* gb, int* status)
{
    if(!*other) return;
    const int fronts = natural_fronts(L.nx, L.ny, L.nz);
    const int width = natural_front_width(L.nx);
    for(int k = 0; k < 2 * fronts; ++k)
    {
        const int t = k < fronts ? k : 2 * fronts - 1 - k;
        for(int idx = blockIdx.x * kBS + threadIdx.x; idx < L.ny * width; idx += gridDim.x * kBS)
            natural_front_row(L, t, width, idx, r, x);
        if(!grid_barrier(gb, gridDim.x, status)) return;
    }
}

struct Workspace
{
    double *x0, *x1, *x2, *r, *diag;
    GridBarrier* gb;
    int* other;
};

Workspace carve(void* ws, size_t m)
{
    double* d = static_cast<double*>(ws);
    Workspace w;
    w.x1 = d;
    w.x2 = d + m;
    w.x0 = d + 2 * m;
    w.r = d + 3 * m;
    w.diag = d + 4 * m;
    w.gb = reinterpret_cast<GridBarrier*>(d + 5 * m);
    w.other = reinterpret_cast<int*>(d + 5 * m + 1);
    return w;
}

constexpr size_t flow_smem(int pitch, int planes)
{
    return sizeof(double) * (size_t)pitch * (size_t)((planes + 2) * kRing + planes * 2 * kRowRing);
}

// Launch of one sweep: as many planes a block as its threads and shared
// memory allow (fewer hand-offs between blocks; 104^3: 3 planes).
template <int kDir, int kPitch, int kThreads>
int launch_flow(FlowArgs a, cudaStream_t s)
{
    constexpr int most = kThreads / (kPitch - 2) - 1;
    static_assert(most >= 1 && flow_smem(kPitch, most) <= kFlowSmem, "a plane, its halo and its neighbours");
    const int lanes = (a.ny + 31) / 32 * 32;
    int planes = std::min(a.nz, kThreads / lanes - 1);
    while(flow_smem(kPitch, planes) > kFlowSmem) --planes;
    a.planes = planes;
    int dev = 0, sms = 0;
    HB_CUDA(cudaGetDevice(&dev));
    HB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const auto kernel = k_nat_gs_flow<kDir, kPitch, kThreads>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFlowSmem));
    HB_CUDA(launch_coop_smem(kernel, (unsigned)std::min((a.nz + planes - 1) / planes, sms),
                             (unsigned)((planes + 1) * lanes), flow_smem(kPitch, planes), s, a));
    return 0;
}

template <int kDir>
int launch_flow(const FlowArgs& a, cudaStream_t s)
{
    if(a.ny <= 32) return launch_flow<kDir, 34, 512>(a, s);
    if(a.ny <= 64) return launch_flow<kDir, 66, 512>(a, s);
    if(a.ny <= 128) return launch_flow<kDir, 130, 512>(a, s);
    return launch_flow<kDir, kFlowMaxLines + 2, 2 * kFlowMaxLines>(a, s);
}

}  // namespace

bool nat_flow_ok(int nx, int ny, int nz)
{
    (void)nx;
    (void)nz;
    return ny <= kFlowMaxLines;
}

size_t nat_flow_workspace_bytes(long long rows) { return sizeof(double) * (5 * (size_t)rows + 2); }

int launch_nat_symgs_flow(const NaturalLevel& L, const double* r, double* x, void* workspace, bool prepared,
                          int* status, cudaStream_t s)
{
    const size_t m = (size_t)L.rows();
    const Workspace w = carve(workspace, m);
    const dim3 tiles((unsigned)L.nz, (unsigned)((L.nx + kTile - 1) / kTile), (unsigned)((L.ny + kTile - 1) / kTile));

    HB_CUDA(cudaMemsetAsync(w.x1, 0xff, 2 * m * sizeof(double), s));
    if(!prepared)
    {
        HB_CUDA(cudaMemsetAsync(w.gb, 0, sizeof(GridBarrier) + sizeof(int), s));
        k_nat_check_rows<<<(unsigned)((m + kCheckRows - 1) / kCheckRows), kBS, 0, s>>>(L, w.diag, w.other);
        HB_LAUNCHED();
        k_nat_skew<true><<<tiles, kBS, 0, s>>>(L.nx, L.ny, r, w.r, w.other);
        HB_LAUNCHED();
    }
    k_nat_skew<true><<<tiles, kBS, 0, s>>>(L.nx, L.ny, x, w.x0, w.other);
    HB_LAUNCHED();
    FlowArgs a{L.nx, L.ny, L.nz, 0, w.x0, w.x1, w.r, w.diag, w.other, status};
    HB_RETURN_IF(launch_flow<1>(a, s));
    a.xold = w.x1;
    a.xnew = w.x2;
    HB_RETURN_IF(launch_flow<-1>(a, s));
    k_nat_skew<false><<<tiles, kBS, 0, s>>>(L.nx, L.ny, w.x2, x, w.other);
    HB_LAUNCHED();
    static const int resident = resident_grid(k_nat_gs_fronts, kBS, 1 << 20);
    const int blocks = (L.ny * natural_front_width(L.nx) + kBS - 1) / kBS;
    HB_CUDA(launch_coop(k_nat_gs_fronts, (unsigned)std::min(blocks, resident), kBS, s, L, r, x, w.other, w.gb,
                        status));
    return 0;
}

}  // namespace hb
