// SymGS of a small multigrid level: the 15 dependent colour passes as one
// kernel on one thread-block cluster.
//
// What bounds them: a pass of a coarse level has a few hundred to a few
// thousand rows, so as a launch of its own it is all launch gap (1.8-2.2 us in a
// graph, 3-4 us launched one by one, 2.8-4 us with the ELL kernels' two
// dependent gathers).  Here the level's x lives in the shared memory of up to 16 CTAs, each
// owning a run of z-plane pairs (so every CTA has rows in every pass) and a
// copy of the plane below and above; a new value of a first or last plane is
// also stored into the neighbour's copy, and a cluster barrier (0.25 us) ends the
// pass.
//
// Shared x is split by the parity of (ix, iy, iz) into eight bricks with a
// one-point border of -0.0 (v + -0.0 is v), so that rows of a colour read
// consecutive words and no row tests for faces; a neighbour is the row's
// address plus an offset of its slot, the slots in ELL order as in the
// one-launch kernels: the same sums, bit for bit.
//
// A zero-guess step in a graph, one cluster against 15 launches: 16^3 FP32 18.6
// against 26.8 us, FP64 20.6 against 32.8, ELL arrays 20.5 against 45.1; 32^3 20.6
// / 30.8, 22.6 / 36.9, 26.6 / 45.2.  The whole V-cycle called through the operator
// API: 16^3 FP64 446 -> 134 us, 104^3 mixed 466 -> 334 us.
#include <algorithm>
#include <type_traits>

#include "small_level.cuh"

namespace hb {

namespace {

constexpr int kMaxCtas = 16;
// A thread has one row of each colour, so a level fits where a CTA's share of a
// pass does: 640 threads leave 96 registers (48 x 24 x 40 with 576 gains, 28.3
// against 31.3 us; two rows a thread at 40^3 lost, 40.4 against 32.8 us), the
// ELL form needs 112.
constexpr int kMaxThreads = 640, kMaxThreadsEll = 512;
constexpr int kSmallSmem = 220 * 1024;
constexpr int kOneCta = 2048;    // rows of a level up to which one CTA takes it: no cluster barrier (8^3 20.5 -> 14.5 us)
constexpr int kMostRows = 1 << 17;

// ELL slots of a row of each colour under the canonical colouring (parity
// class p -> colour 7,2,3,6,5,4,1,0): neighbour colour, then (dz, dy, dx).
struct Order
{
    signed char dx[8][27], dy[8][27], dz[8][27];
    unsigned gone[8][6];         // slots that face x-, x+, y-, y+, z-, z+ removes
    int dp[8];                   // slot of the diagonal
    int cls[8];                  // parity class of colour v (ix&1)<<2 | (iy&1)<<1 | (iz&1)
};

constexpr int colour_of(int cls) { return (int)((0x01456327u >> (4 * cls)) & 15u); }

constexpr Order make_order()
{
    Order o{};
    for(int cls = 0; cls < 8; ++cls)
    {
        const int v = colour_of(cls);
        o.cls[v] = cls;
        int k = 0;
        for(int c = 0; c < 8; ++c)
            for(int dz = -1; dz <= 1; ++dz)
                for(int dy = -1; dy <= 1; ++dy)
                    for(int dx = -1; dx <= 1; ++dx)
                    {
                        if(colour_of(cls ^ (((dx & 1) << 2) | ((dy & 1) << 1) | (dz & 1))) != c) continue;
                        o.dx[v][k] = (signed char)dx;
                        o.dy[v][k] = (signed char)dy;
                        o.dz[v][k] = (signed char)dz;
                        const int d[3] = {dx, dy, dz};
                        for(int q = 0; q < 3; ++q)
                            if(d[q] != 0) o.gone[v][2 * q + (d[q] > 0)] |= 1u << k;
                        if(dx == 0 && dy == 0 && dz == 0) o.dp[v] = k;
                        ++k;
                    }
    }
    return o;
}

__constant__ Order c_order = make_order();

template <typename T>
struct SmallArgs
{
    int nx, ny, nz, m;
    int pairs;             // z-plane pairs of the level
    int sx, sy, brick;     // extents of a parity brick in shared memory, and its size
    int off[8];            // first row of each colour
    const T* diag;
    const T* inv_diag;
    const double* r64;
    T* r;
    T* x;
    double* z64;
    const int* inj_c;      // coarse row of each row of colour 7
    T* rc;                 // coarse residual (may be null)
    Prolong<T> pro;
};

// What the ELL form reads besides.
struct EllArgs
{
    SmallEll m;
    int dcol[8][27];       // by stencil point: its column in a row of a colour, from the row's brick position
    signed char slot[8][27];  // and its slot
};

struct NoEll
{
};

// The columns as they are at set-up: stencil point t of a colour-v row at brick
// position (kx, ky, kz) is dcol[v][t] + (kz * by + ky) * bx + kx with the extents
// of the neighbour's brick.
void expected_columns(const StencilLevel& L, EllArgs* e)
{
    constexpr Order o = make_order();
    for(int v = 0; v < 8; ++v)
        for(int j = 0; j < 27; ++j)
        {
            const int cls = o.cls[v], dx = o.dx[v][j], dy = o.dy[v][j], dz = o.dz[v][j];
            const int c = colour_of(cls ^ (((dx & 1) << 2) | ((dy & 1) << 1) | (dz & 1)));
            auto shift = [](int parity, int d) { return parity + d < 0 ? -1 : (parity + d > 1 ? 1 : 0); };
            const int sx = shift((cls >> 2) & 1, dx), sy = shift((cls >> 1) & 1, dy), sz = shift(cls & 1, dz);
            const int t = (dz + 1) * 9 + (dy + 1) * 3 + dx + 1;
            e->dcol[v][t] = L.offsets[c] + (sz * L.by[c] + sy) * L.bx[c] + sx;
            e->slot[v][t] = (signed char)j;
        }
}

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ unsigned cluster_size()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// The barrier between passes, in two halves; __syncthreads where one CTA has the
// whole level.  The .aligned forms want the whole warp at one instruction, and
// what stands before them is divergent (lanes without a row, copies to a
// neighbour).
__device__ __forceinline__ void cluster_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// v into the same shared-memory cell of CTA `rank` of the cluster
__device__ __forceinline__ void store_peer(double* cell, unsigned rank, double v)
{
    unsigned a = (unsigned)__cvta_generic_to_shared(cell), p;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory");
}

__device__ __forceinline__ void store_peer(float* cell, unsigned rank, float v)
{
    unsigned a = (unsigned)__cvta_generic_to_shared(cell), p;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory");
}

__device__ __forceinline__ float mul_once(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_once(double a, double b) { return __dmul_rn(a, b); }

__device__ __forceinline__ float fma_once(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_once(double a, double b, double c) { return fma(a, b, c); }

// A row's final value of the step.
template <typename T>
__device__ __forceinline__ void finish(const SmallArgs<T>& a, int g, T v)
{
    a.x[g] = v;
    if(sizeof(T) == 4 && a.z64) a.z64[g] = (double)v;
    a.pro.add(g, v);
}

// x of a level through L2: in the passes on any matrix other CTAs write it.
struct L2Reads
{
    const double* x;
    __device__ __forceinline__ double operator[](int i) const { return __ldcg(x + i); }
};

// The row of a full step, of a zero-guess step's forward pass (offset: the
// colour's first row) or its backward pass on any matrix: k_symgs_sweep,
// k_symgs_fwd0 and k_symgs_bwd0.
template <bool kZero>
__device__ double any_row(const SmallArgs<double>& a, const SmallEll& e, int row, int offset, bool back)
{
    const int m = a.m;
    const L2Reads x{a.x};
    double sum;
    if constexpr(!kZero)
        sum = ell_row_sum(m, row, e.col, e.val, x, a.r[row], -1.0, 0, kWidth,
                          [m, row](int col) { return col >= 0 && col < m && col != row; });
    else if(!back)
        sum = ell_row_sum(m, row, e.col, e.val, x, a.r[row], -1.0, 0, offset > 0 ? e.diag_idx[row] : 0,
                          [offset](int col) { return col >= 0 && col < offset; });
    else
        sum = ell_row_sum(m, row, e.col, e.val, x, __dmul_rn(x[row], a.diag[row]), -1.0, e.diag_idx[row] + 1, kWidth,
                          [offset, m](int col) { return col >= offset && col < m; });
    return sum * a.inv_diag[row];
}

// t / n for 0 <= t < 2^20
__device__ __forceinline__ int quotient(int t, int n) { return __float2int_rd(((float)t + 0.5f) * __frcp_rn((float)n)); }

// Not 0 where row t of colour v is not the stencil's in the ELL arrays, its
// diagonal slot or (zero guess) its diagonal, or is injected elsewhere.
template <bool kZero>
__device__ __forceinline__ unsigned row_differs(const SmallArgs<double>& a, const EllArgs& ell, int v, int t)
{
    const int cls = c_order.cls[v], px = (cls >> 2) & 1, py = (cls >> 1) & 1, pz = cls & 1;
    const int bx = (a.nx - px + 1) / 2, by = (a.ny - py + 1) / 2;
    const int q = quotient(t, bx), kx = t - q * bx, kz = quotient(q, by), ky = q - kz * by;
    const int g = a.off[v] + t;
    const int ix = 2 * kx + px, iy = 2 * ky + py, iz = 2 * kz + pz;
    const unsigned* face = c_order.gone[v];
    const unsigned gone = (ix == 0 ? face[0] : 0u) | (ix == a.nx - 1 ? face[1] : 0u) | (iy == 0 ? face[2] : 0u) |
                          (iy == a.ny - 1 ? face[3] : 0u) | (iz == 0 ? face[4] : 0u) |
                          (iz == a.nz - 1 ? face[5] : 0u);
    // the row's position in the neighbours' bricks: index bit 0 dx odd, bit 1 dy odd
    int at[4];
#pragma unroll
    for(int k = 0; k < 4; ++k)
        at[k] = (kz * ((a.ny + 1 - (py ^ (k >> 1))) / 2) + ky) * ((a.nx + 1 - (px ^ (k & 1))) / 2) + kx;
    const double diag = kZero ? __ldg(a.diag + g) : 0.0;
    unsigned other = 0;
    // slots are packed: those the faces remove leave the row's last ones empty
#pragma unroll
    for(int n = 0; n < 27; ++n)
    {
        const int j = ell.slot[v][n], missing = __popc(gone & ((1u << j) - 1u));
        const bool off = gone >> j & 1u;
        const int at_e = (off ? 26 - missing : j - missing) * a.m + g;
        const unsigned c = (unsigned)__ldg(ell.m.col + at_e);
        const unsigned want = (unsigned)(at[(n % 3 != 1) + 2 * (n / 3 % 3 != 1)] + ell.dcol[v][n]);
        unsigned differs = c ^ want;
        if(n != 13 || kZero) differs |= __ldg(ell.m.val + at_e) == (n == 13 ? diag : -1.0) ? 0u : 1u;
        other |= off ? (unsigned)(c < (unsigned)a.m) : differs;
    }
    if constexpr(kZero)
    {
        const int dp = c_order.dp[v];
        other |= (unsigned)(__ldg(ell.m.diag_idx + g) ^ (dp - __popc(gone & ((1u << dp) - 1u))));
        if(a.rc && v == 7) other |= (unsigned)(__ldg(ell.m.inj_f + t) ^ g);
    }
    return other;
}

// Sets *ell.m.changed where some row differs.  A kernel of its own: a level's
// arrays are up to 21 MB, which the cluster's 16 SMs alone take 12 us to read
// (64 x 32 x 32 zero-guess step 45.1 us with the check in its prologue, 32.7 so;
// 16^3 20.5 either way).
template <bool kZero>
__global__ void __launch_bounds__(kBS)
    k_small_check(const __grid_constant__ SmallArgs<double> a, const __grid_constant__ EllArgs ell)
{
    pdl_launch_dependents();
    const int g = blockIdx.x * kBS + threadIdx.x;
    unsigned other = 0;
    if(g < a.m)
    {
        int v = 0;
        while(v < 7 && g >= a.off[v + 1]) ++v;
        other = row_differs<kZero>(a, ell, v, g - a.off[v]);
    }
    if(__syncthreads_or((int)other) && threadIdx.x == 0) atomicExch(ell.m.changed, 1);
}

// The dynamic shared memory: the x bricks, then per colour and thread the
// row's r, 1/a_ii and (zero guess) a_ii, and its cell.
template <typename T, bool kZero>
constexpr size_t bytes_per_thread = 8 * ((kZero ? 3 : 2) * sizeof(T) + 4);

// s_cell: the row's cell, or kNone; flags where its value has a copy in the CTA below or above
constexpr int kNone = -1, kToBelow = 1 << 30, kToAbove = 1 << 29, kCellMask = kToAbove - 1;

// kZero: the zero-guess step (forward pass: slots before the diagonal,
// backward: a_ii x_i and the slots after it) and, with rc given, the
// restriction of its residual; else the full step.  kEll: the step is that of
// the ELL arrays as they are now -- k_small_check has read them just before.
// Where every column, value and diagonal slot is the stencil's, the passes are
// the implicit ones (sum + x is fma(1, x, sum)); else the cluster runs them on
// the arrays, with x in global memory.  A thread has at most one row of each colour; what a pass needs of it
// besides its neighbours' x is fetched between the barrier's arrival and its
// wait.
template <typename T, bool kZero, bool kEll>
__global__ void __launch_bounds__(kEll ? kMaxThreadsEll : kMaxThreads, 1)
    k_small_symgs(const __grid_constant__ SmallArgs<T> a,
                  const __grid_constant__ std::conditional_t<kEll, EllArgs, NoEll> ell)
{
    extern __shared__ __align__(16) unsigned char small_smem[];
    const int nt = blockDim.x, tid = threadIdx.x;
    T* const xs = reinterpret_cast<T*>(small_smem);
    T* const s_r = xs + 8 * a.brick + tid;
    T* const s_inv = s_r + 8 * nt;
    T* const s_diag = s_inv + 8 * nt;  // kZero only
    int* const s_cell = reinterpret_cast<int*>(xs + 8 * a.brick + (kZero ? 24 : 16) * nt) + tid;
    __shared__ __align__(16) int s_tab[8][28];  // per colour: cell offset of each slot but the diagonal's, in order
    __shared__ int s_row0[8];                   // per colour: the CTA's first row
    __shared__ int s_dp[8];                     // per colour: the diagonal's slot
    const unsigned rank = cluster_rank(), size = cluster_size();
    const int p0 = (int)(rank * (unsigned)a.pairs / size), p1 = (int)((rank + 1) * (unsigned)a.pairs / size);
    const int np = p1 - p0;
    const int below = rank ? p0 - (int)((rank - 1) * (unsigned)a.pairs / size) : 0;  // pairs of the CTA below
    const int sxy = a.sx * a.sy;

    // parity brick and position of local point (hx, hy, hz) = (ix, iy, iz - 2 p0) + 1
    auto cell_of = [&](int hx, int hy, int hz) {
        return (((hx & 1) << 2) | ((hy & 1) << 1) | (hz & 1)) * a.brick + (hz >> 1) * sxy + (hy >> 1) * a.sx + (hx >> 1);
    };

    // this thread's row of every colour
#pragma unroll
    for(int v = 0; v < 8; ++v)
    {
        constexpr Order o = make_order();
        const int cls = o.cls[v], px = (cls >> 2) & 1, py = (cls >> 1) & 1, pz = cls & 1;
        const int bx = (a.nx - px + 1) / 2, by = (a.ny - py + 1) / 2, bz = (a.nz - pz + 1) / 2;
        const int first = a.off[v] + p0 * by * bx;
        if(tid == 0)
        {
            s_row0[v] = first;
            s_dp[v] = o.dp[v];
        }
        s_cell[v * nt] = kNone;
        if(tid >= (min(p1, bz) - p0) * by * bx) continue;
        const int q = quotient(tid, bx), kx = tid - q * bx, kp = quotient(q, by), ky = q - kp * by;
        const int g = first + tid;
        s_cell[v * nt] = cell_of(2 * kx + px + 1, 2 * ky + py + 1, 2 * kp + pz + 1) |
                         (pz == 0 && kp == 0 && rank > 0 ? kToBelow : 0) |
                         (pz == 1 && kp == np - 1 && rank + 1 < size ? kToAbove : 0);
        s_inv[v * nt] = __ldg(a.inv_diag + g);
        if(kZero) s_diag[v * nt] = __ldg(a.diag + g);
        T r;
        if(sizeof(T) == 4 && a.r64)
        {
            r = (T)__ldg(a.r64 + g);
            a.r[g] = r;
        }
        else r = __ldg(a.r + g);
        s_r[v * nt] = r;
    }
    for(int e = tid; e < 8 * a.brick; e += nt) xs[e] = T(-0.0);
    for(int e = tid; e < 8 * 28; e += nt)
    {
        const int v = e / 28, j = e - v * 28, cls = c_order.cls[v], dp = c_order.dp[v];
        const int hx = ((cls >> 2) & 1) + 1, hy = ((cls >> 1) & 1) + 1, hz = (cls & 1) + 1;
        if(j < 27 && j != dp)
            s_tab[v][j < dp ? j : j - 1] =
                cell_of(hx + c_order.dx[v][j], hy + c_order.dy[v][j], hz + c_order.dz[v][j]) - cell_of(hx, hy, hz);
        else if(j == 27) s_tab[v][26] = s_tab[v][27] = 0;
    }
    __syncthreads();
    if constexpr(!kZero)
    {
        for(int v = 0; v < 8; ++v)
        {
            const int cls = c_order.cls[v], px = (cls >> 2) & 1, py = (cls >> 1) & 1, pz = cls & 1;
            const int bx = (a.nx - px + 1) / 2, by = (a.ny - py + 1) / 2, bz = (a.nz - pz + 1) / 2;
            // own planes and the copies of the planes next to them
            const int lo = max(0, p0 - pz), hi = min(bz, p1 + 1 - pz);
            for(int t = tid; t < (hi - lo) * by * bx; t += nt)
            {
                const int q = quotient(t, bx), kx = t - q * bx, kz = quotient(q, by), ky = q - kz * by;
                xs[cell_of(2 * kx + px + 1, 2 * ky + py + 1, 2 * (lo + kz - p0) + pz + 1)] =
                    __ldcg(a.x + a.off[v] + lo * by * bx + t);
            }
        }
    }
    auto arrive = [&] {
        if(size > 1) cluster_arrive();
    };
    auto wait = [&] {
        if(size > 1) cluster_wait();
        else __syncthreads();
    };
    arrive();  // every CTA's x is in place before a neighbour stores into it

    // pass i: colours 0..7, 6..0 and, for the restriction, 7 again
    auto colour = [](int i) { return i < 8 ? i : (i < 15 ? 14 - i : 7); };
    const int passes = kZero && a.rc ? 16 : 15;
    int cell = kNone, off[28], lo = 0;  // slots from lo on take part
    T opr = T(0), opi = T(0), opd = T(0);
    auto fetch = [&](int i) {
        const int v = colour(i);
        cell = s_cell[v * nt];
        if(cell == kNone) return;
        opr = s_r[v * nt];
        opi = s_inv[v * nt];
        if(kZero) opd = s_diag[v * nt];
        lo = kZero && i >= 8 && i < 15 ? s_dp[v] : 0;
#pragma unroll
        for(int q = 0; q < 7; ++q)
        {
            const int4 o = *reinterpret_cast<const int4*>(&s_tab[v][4 * q]);
            off[4 * q] = o.x;
            off[4 * q + 1] = o.y;
            off[4 * q + 2] = o.z;
            off[4 * q + 3] = o.w;
        }
    };
    fetch(0);
    wait();
    if constexpr(kEll)
    {
        pdl_wait();
        if(__ldcg(ell.m.changed))
        {
#pragma unroll 1
            for(int i = 0; i < 15; ++i)
            {
                const int v = colour(i);
                if(s_cell[v * nt] != kNone)
                {
                    const int row = s_row0[v] + tid;
                    const double out = any_row<kZero>(a, ell.m, row, a.off[v], i >= 8);
                    a.x[row] = out;
                    if(i >= 7) a.pro.add(row, out);
                }
                arrive();
                wait();
            }
            if(rank == 0 && tid == 0) *ell.m.changed = 0;  // everyone has read it
            if constexpr(kZero)
            {
                const int nc = a.rc ? ell.m.nc : 0, m = a.m;
                for(int ic = (int)rank * nt + tid; ic < nc; ic += (int)size * nt)
                {
                    const int row = ell.m.inj_f[ic];
                    a.rc[a.inj_c[ic]] = ell_row_sum(m, row, ell.m.col, ell.m.val, L2Reads{a.x}, a.r[row], -1.0, 0,
                                                    kWidth, [m](int col) { return col >= 0 && col < m; });
                }
            }
            return;
        }
    }
#pragma unroll 1
    for(int i = 0; i < passes; ++i)
    {
        const int v = colour(i);
        T out = T(0);
        const bool row = cell != kNone;
        if(row)
        {
            T* const own = xs + (cell & kCellMask);
            const bool back = kZero && i >= 8 && i < 15;
            T sum = back ? mul_once(*own, opd) : opr;
            // All neighbours first, then their terms in slot order.  Forward
            // zero-guess: the slots after the diagonal still hold -0.0.
            T nb[26];
#pragma unroll
            for(int e = 0; e < 26; ++e) nb[e] = own[off[e]];
            if(kZero && back)
            {
#pragma unroll
                for(int e = 0; e < 26; ++e) nb[e] = e >= lo ? nb[e] : T(-0.0);
            }
#pragma unroll
            for(int e = 0; e < 26; ++e) sum = sum + nb[e];
            if(kZero && i == 15)  // the diagonal is colour 7's last slot
                a.rc[a.inj_c[s_row0[7] + tid - a.off[7]]] = fma_once(-opd, *own, sum);
            else
            {
                out = sum * opi;
                *own = out;
                // the copies of this plane in the CTAs below and above: the plane above the
                // last pair of the one, the plane below the first pair of the other (nobody
                // reads the last pass's, and the neighbour may be gone by then)
                if(i < passes - 1)
                {
                    if(cell & kToBelow) store_peer(own + below * sxy, rank - 1, out);
                    if(cell & kToAbove) store_peer(own - np * sxy, rank + 1, out);
                }
            }
        }
        // colour 7 is not visited again, the others once more
        const bool last = row && i >= 7 && i < 15;
        const int g = s_row0[v] + tid;
        if(i == passes - 1)
        {
            if(last) finish(a, g, out);
            break;
        }
        arrive();
        if(last) finish(a, g, out);
        fetch(i + 1);
        wait();
    }
}

// Largest cluster the device runs with a full shared memory: 16 (beyond the
// portable 8) where its GPCs have the SMs.
int max_ctas()
{
    static const int most = [] {
        const auto kernel = k_small_symgs<float, false, false>;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kMaxCtas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kMaxCtas);
        cfg.blockDim = dim3(kMaxThreads);
        cfg.dynamicSmemBytes = kSmallSmem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) != cudaSuccess ||
           cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
           cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess)
        {
            cudaGetLastError();
            n = 0;
        }
        return n > 0 ? kMaxCtas : 8;
    }();
    return most;
}

// Cluster shape of a level.
struct Shape
{
    int ctas, threads, per;  // per: z-plane pairs of a CTA at most
    size_t smem;
};

template <typename T>
Shape shape_of(const StencilLevel& L)
{
    Shape s{};
    const int pairs = (L.nz + 1) / 2;
    s.ctas = 1;
    if(L.m > kOneCta)
        while(s.ctas < max_ctas() && s.ctas < pairs) s.ctas *= 2;
    while(s.ctas > pairs) s.ctas /= 2;
    s.per = (pairs + s.ctas - 1) / s.ctas;
    const int rows = ((L.nx + 1) / 2) * ((L.ny + 1) / 2) * s.per;
    s.threads = (rows + 31) / 32 * 32;
    s.smem = sizeof(T) * 8 * (size_t)((L.nx + 3) / 2) * ((L.ny + 3) / 2) * (s.per + 1) +
             bytes_per_thread<T, true> * (size_t)s.threads;
    return s;
}

template <typename T>
SmallArgs<T> args_of(const StencilLevel& L)
{
    SmallArgs<T> a{};
    a.nx = L.nx;
    a.ny = L.ny;
    a.nz = L.nz;
    a.m = L.m;
    a.pairs = (L.nz + 1) / 2;
    a.sx = (L.nx + 3) / 2;
    a.sy = (L.ny + 3) / 2;
    for(int v = 0; v < 8; ++v) a.off[v] = L.offsets[v];
    return a;
}

template <typename T, bool kZero, bool kEll>
int launch_shape(const StencilLevel& L, SmallArgs<T> a, const std::conditional_t<kEll, EllArgs, NoEll>& ell,
                 cudaStream_t s)
{
    const Shape sh = shape_of<T>(L);
    a.brick = a.sx * a.sy * (sh.per + 1);
    const auto kernel = k_small_symgs<T, kZero, kEll>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem));
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)sh.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)sh.ctas);
    cfg.blockDim = dim3((unsigned)sh.threads);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if constexpr(kEll)
    {
        k_small_check<kZero><<<(a.m + kBS - 1) / kBS, kBS, 0, s>>>(a, ell);
        HB_LAUNCHED();
        cfg.numAttrs = 2;  // the passes' kernel sets itself up meanwhile
    }
    HB_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, ell));
    return 0;
}

template <typename T, bool kZero>
int launch_small(const StencilLevel& L, const SmallArgs<T>& a, const SmallEll* ell, cudaStream_t s)
{
    if constexpr(sizeof(T) == 8)
        if(ell)
        {
            EllArgs e{};
            e.m = *ell;
            expected_columns(L, &e);
            return launch_shape<T, kZero, true>(L, a, e, s);
        }
    return launch_shape<T, kZero, false>(L, a, NoEll{}, s);
}

}  // namespace

template <typename T>
bool small_level_ok(const StencilLevel& L, bool ell)
{
    if(L.ncolors != 8 || L.m > kMostRows) return false;
    for(int p = 0; p < 8; ++p)
        if(L.color_of_par[p] != colour_of(p)) return false;
    const Shape s = shape_of<T>(L);
    return s.threads <= (ell ? kMaxThreadsEll : kMaxThreads) && s.smem <= kSmallSmem;
}

template <typename T>
int launch_small_zero(const StencilLevel& L, const T* diag, const T* inv_diag, const double* r64, T* r, T* x,
                      const SmallEll* ell, const int* inj_c, T* rc, cudaStream_t s, Prolong<T> pro)
{
    SmallArgs<T> a = args_of<T>(L);
    a.diag = diag;
    a.inj_c = inj_c;
    a.rc = rc;
    a.inv_diag = inv_diag;
    a.r64 = r64;
    a.r = r;
    a.x = x;
    a.pro = pro;
    return launch_small<T, true>(L, a, ell, s);
}

template <typename T>
int launch_small_symgs(const StencilLevel& L, const T* inv_diag, const T* r, T* x, double* z64,
                       const SmallEll* ell, cudaStream_t s, Prolong<T> pro)
{
    SmallArgs<T> a = args_of<T>(L);
    a.inv_diag = inv_diag;
    a.r = const_cast<T*>(r);
    a.x = x;
    a.z64 = z64;
    a.pro = pro;
    return launch_small<T, false>(L, a, ell, s);
}

template bool small_level_ok<float>(const StencilLevel&, bool);
template bool small_level_ok<double>(const StencilLevel&, bool);
template int launch_small_zero<float>(const StencilLevel&, const float*, const float*, const double*, float*, float*,
                                      const SmallEll*, const int*, float*, cudaStream_t, Prolong<float>);
template int launch_small_zero<double>(const StencilLevel&, const double*, const double*, const double*, double*,
                                       double*, const SmallEll*, const int*, double*, cudaStream_t, Prolong<double>);
template int launch_small_symgs<float>(const StencilLevel&, const float*, const float*, float*, double*,
                                       const SmallEll*, cudaStream_t, Prolong<float>);
template int launch_small_symgs<double>(const StencilLevel&, const double*, const double*, double*, double*,
                                        const SmallEll*, cudaStream_t, Prolong<double>);

}  // namespace hb
