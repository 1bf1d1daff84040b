// The differentiable program (halo exchange, 7-point update, repeated; and its transpose) in one
// kernel per step.
//
// Between the first and the last step nobody sees the halos, so a pass does not fill them: a cell
// next to a domain's face takes the neighbour's interior cell that the exchange would have copied
// beside it, and the transpose adds, after the cell's own value, the contribution that the
// exchange's adjoint would have added from each of its images, in the same order. Every value is
// the one that the exchange kernel and the stencil kernel (stencil.cu) compute one after the
// other, with the same roundings, so results have the same bits.
// (One exception: images of halo cells that no interior cell lies beside are zeros, which a pass
// leaves out and the exchange's adjoint adds. Where that is all that is added to a cell, a zero may
// keep the minus sign that a negative alpha gave it.)
//
// The fields between two passes are the program's own, and packed: interiors only, rows on
// 32-byte boundaries, so that a thread moves 16 bytes at a time whatever the domains' extents.
//
// One step on 8 domains of 128 x 128 x 64, in us: exchange kernel + update kernel, a pass, and the
// floor (one read and one write of every cell at the HBM rate; the float32 fields fit the L2):
//   forward     float64  6.6 + 42.3   22.8   20.5     float32  5.5 + 31.2   11.7   10.2
//   transposed  float64  8.6 + 42.9   32.5   20.5     float32  7.9 + 28.1   18.1   10.2
// and on 12 uneven domains of 500 x 510 x 250 in all, float64: forward 32.1 + 261.8, 182.8, 155.7;
// transposed 37.8 + 262.8, 206.9, 155.7.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "async_copy.hpp"
#include "plan.hpp"
#include "program.hpp"
#include "staged.hpp"

namespace ghexb
{
namespace
{
template <typename T> __device__ __forceinline__ T add_rn(T a, T b);
template <typename T> __device__ __forceinline__ T sub_rn(T a, T b);
template <typename T> __device__ __forceinline__ T mul_rn(T a, T b);
template <> __device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// x + alpha * (s - 6 x), s the sum of the six neighbours (stencil.cu)
template <typename T> __device__ __forceinline__ T update(T x, T s, T alpha)
{
    return add_rn(x, mul_rn(alpha, sub_rn(s, mul_rn(T(6), x))));
}

// 16 bytes of consecutive cells
template <typename T> struct alignas(16) cells
{
    static constexpr int V = 16 / (int)sizeof(T);
    T v[V];
};

// Cell by cell. Sums of float cells two at a time (add.f32x2: the same rounding); products stay
// scalar, since a packed product is contracted with the sum that follows it, explicit roundings or
// not (of 2^20 random mul.rn.f32x2 + add.rn.f32x2 all had the bits of the fused form).
__device__ __forceinline__ float2 add_rn(float2 a, float2 b)
{
    float2 c;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(c.x), "=f"(c.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return c;
}
template <typename T> __device__ __forceinline__ cells<T> add_rn(const cells<T>& a, const cells<T>& b)
{
    cells<T> c;
    if constexpr (sizeof(T) == 4)
    {
#pragma unroll
        for (int v = 0; v < cells<T>::V; v += 2)
        {
            const float2 s = add_rn(make_float2(a.v[v], a.v[v + 1]), make_float2(b.v[v], b.v[v + 1]));
            c.v[v] = s.x, c.v[v + 1] = s.y;
        }
    }
    else
    {
#pragma unroll
        for (int v = 0; v < cells<T>::V; ++v) c.v[v] = add_rn(a.v[v], b.v[v]);
    }
    return c;
}
template <typename T> __device__ __forceinline__ cells<T> mul_rn(T f, const cells<T>& a)
{
    cells<T> c;
#pragma unroll
    for (int v = 0; v < cells<T>::V; ++v) c.v[v] = mul_rn(f, a.v[v]);
    return c;
}
// The update of a row's cells x (m of them count) between the cells l and e and the rows around:
// s - 6 x is taken as s + (-6) x, the same value.
template <typename T>
__device__ __forceinline__ cells<T> update(const cells<T>& x, T l, T e, int m, const cells<T>& up, const cells<T>& down, const cells<T>& below,
    const cells<T>& above, T alpha)
{
    constexpr int V = cells<T>::V;
    cells<T> s;
#pragma unroll
    for (int v = 0; v < V; ++v) s.v[v] = add_rn(v > 0 ? x.v[v > 0 ? v - 1 : 0] : l, v < V - 1 && v < m - 1 ? x.v[v + 1 < V ? v + 1 : v] : e);
    s = add_rn(s, up);
    s = add_rn(s, down);
    s = add_rn(s, below);
    s = add_rn(s, above);
    return add_rn(x, mul_rn(alpha, add_rn(s, mul_rn(T(-6), x))));
}
template <typename T> __device__ __forceinline__ void zero(cells<T>& a)
{
#pragma unroll
    for (int v = 0; v < cells<T>::V; ++v) a.v[v] = T(0);
}
template <typename T> __device__ __forceinline__ cells<T> zero_if(bool z, const cells<T>& a)
{
    cells<T> c;
#pragma unroll
    for (int v = 0; v < cells<T>::V; ++v) c.v[v] = z ? T(0) : a.v[v];
    return c;
}

template <typename T> __device__ __forceinline__ void not_a_number(cells<T>& a)
{
#pragma unroll
    for (int v = 0; v < cells<T>::V; ++v) a.v[v] = sizeof(T) == 8 ? (T)__longlong_as_double(0x7ff8000000000000ll) : (T)__int_as_float(0x7fc00000);
}

// the program's status word (host memory)
__device__ __forceinline__ void report(unsigned* status) { *reinterpret_cast<volatile unsigned*>(status) = 1u; }

constexpr int k_batch = 32; // domains per launch
constexpr int k_sms = 148;  // of a B200

// Passes follow one another: a pass lets the next one be launched (programmatic stream serialisation)
// when its blocks come to their last plane, so that the other's blocks start and set up their
// barriers as its own leave; they wait for the whole of it before they touch any memory but their
// arguments. 256 x 256 x 128 float32, 10 steps forward and back: 347 -> 336 us; 48 x 50 x 40: 102.7
// -> 90.5. Let go at a block's start instead, the next pass's blocks settle in whatever slots are
// free and leave some SMs with more of them than others: 330 and 101.7 us, and 64 x 200 x 60 157 us
// where it had been 148 (at the last plane: 145).
// What the pass before wrote is read by ordinary loads: it is not constant while the kernel runs, so
// neither __ldg nor a const __restrict__ pointer may name it.
__device__ __forceinline__ void follow() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void lead() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... Params, typename... Args>
cudaError_t launch_following(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t shared, cudaStream_t stream, Args&&... args)
{
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(blocks), config.blockDim = dim3(threads), config.dynamicSmemBytes = shared, config.stream = stream;
    config.attrs = &attribute, config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

// One domain of a launch; cell (0, 0, 0) is the first interior cell, strides count elements.
struct pass_domain
{
    const void* in;
    void* out;
    int32_t nx, ny, nz, halo;
    int32_t isx, isy, isz, osx, osy, osz;
    struct
    {
        const void* p; // the cells beyond the face: p[u * s0 + v * s1], (u, v) the other axes in order
        int32_t s0, s1;
    } f[6];
    uint32_t ranks, images;
    uint32_t chunks, slab, columns, groups; // chunks a row, planes a slab, columns (chunks x strips), blocks a slab
    uint32_t block0, marches; // first block; blocks that march (the others write the halo)
};
struct pass_args
{
    pass_domain d[k_batch];
    int n;
};

// A thread marches along z through a slab of planes of a column of 16 bytes of consecutive cells
// (x) by `rows` rows (y); consecutive threads take consecutive cells of a row, then the next strip
// of rows, so no thread idles but in a row's last chunk. The planes it reads (its rows, the row
// before and after them and the cells beside them) pass through a ring of its own in shared
// memory, filled by asynchronous copies k_stages - 1 planes ahead; nothing is shared between
// threads, so there is no barrier, and the rows and cells that neighbouring threads read too come
// from L1 or L2.
constexpr int k_threads = 128;
constexpr int k_rows = 2;
constexpr int k_stages = 3;
constexpr int k_resident = 5; // blocks per SM
// Planes of a slab at least: small domains take as many slabs as the chip holds blocks, so that a
// block's loads are all under way at once (48 x 50 x 40 in 8 domains, 8 steps forward and back: 4
// planes at least 90.5 us, 2 71.9, 1 64.2; 64 x 200 x 60, 10 steps: 144.9, 118.1, 118.0).
constexpr int k_min_slab = 1;
constexpr int k_halo_cells = 8; // halo cells a thread writes

// a plane in the ring of a block: rows -1 .. R of 16 bytes per thread, then the cells beside the R rows
template <typename T> struct ring
{
    static constexpr int wide = 16 * k_threads, narrow = (int)sizeof(T) * k_threads;
    static constexpr int stage = (k_rows + 2) * wide + 2 * k_rows * narrow;
    static constexpr int bytes = k_stages * stage;
};

template <int N> __device__ __forceinline__ void copy_async(uint32_t dst, const void* src, bool valid)
{
    // src-size 0 writes zeros and reads nothing
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(valid ? N : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, bool ADJOINT, bool TWICE, int THREADS>
__device__ __forceinline__ void write_halo(const pass_domain& d, T alpha, uint32_t block)
{
    const int h = d.halo, nx = d.nx, ny = d.ny, nz = d.nz;
    const uint32_t ex = nx + 2 * h, ey = ny + 2 * h;
    const uint32_t zcells = ex * ey * (2 * h), ycells = ex * (2 * h) * nz, xcells = (2 * h) * ny * nz;
    const T* in = static_cast<const T*>(d.in);
    T* __restrict__ out = static_cast<T*>(d.out);
    for (int q = 0; q < k_halo_cells; ++q)
    {
        uint32_t c = (block * k_halo_cells + q) * THREADS + threadIdx.x;
        int i, j, k;
        if (c < zcells)
        {
            const uint32_t r = c / ex, v = r / ey;
            i = (int)(c - r * ex) - h, j = (int)(r - v * ey) - h;
            k = (int)v < h ? (int)v - h : nz + (int)v - h;
        }
        else if ((c -= zcells) < ycells)
        {
            const uint32_t r = c / ex, v = r / (2 * h);
            i = (int)(c - r * ex) - h, k = (int)v;
            j = (int)(r - v * (2 * h));
            j = j < h ? j - h : ny + j - h;
        }
        else if ((c -= ycells) < xcells)
        {
            const uint32_t r = c / (2 * h), v = r / ny;
            i = (int)(c - r * (2 * h)), j = (int)(r - v * ny), k = (int)v;
            i = i < h ? i - h : nx + i - h;
        }
        else
            return;
        T y = T(0);
        if constexpr (ADJOINT)
        {
            const int region = (i < 0 ? 0 : i < nx ? 1 : 2) + 3 * (j < 0 ? 0 : j < ny ? 1 : 2) + 9 * (k < 0 ? 0 : k < nz ? 1 : 2);
            if (!((d.images >> region) & 1u)) // a halo cell that nothing was copied to keeps its gradient
            {
                const auto G = [&](int a, int b, int e) {
                    if (a < 0 || a >= nx || b < 0 || b >= ny || e < 0 || e >= nz) return T(0);
                    const T g = in[a * d.isx + b * d.isy + e * d.isz];
                    return TWICE ? mul_rn(T(2), g) : g;
                };
                T t = add_rn(G(i - 1, j, k), G(i + 1, j, k));
                t = add_rn(t, G(i, j - 1, k));
                t = add_rn(t, G(i, j + 1, k));
                t = add_rn(t, G(i, j, k - 1));
                t = add_rn(t, G(i, j, k + 1));
                y = update(T(0), t, alpha);
            }
        }
        out[i * d.osx + j * d.osy + k * d.osz] = y;
    }
}

// What the exchange's adjoint adds for an image whose neighbour has gradient g: the transposed
// update of a zero cell.
template <typename T> __device__ __forceinline__ T image(T g, T alpha) { return add_rn(T(0), mul_rn(alpha, add_rn(g, T(0)))); }

// The images of a row of cells along x and y alone: those of its cells along y (`along`: the row is
// on face y- or y+), and along x of its first cell (fi) or of the last that counts (la); *_first:
// that one comes before the one along y.
template <typename T>
__device__ __forceinline__ void add_row_images(cells<T>& y, bool along, const cells<T>& iy, bool fi, bool la, T il, T ie, bool fi_first, bool la_first,
    int m)
{
#pragma unroll
    for (int v = 0; v < cells<T>::V; ++v)
    {
        const bool at_l = v == 0 && fi, at_e = v == m - 1 && la;
        const T ix = at_l ? il : ie;
        const bool x_first = at_l ? fi_first : la_first;
        const T before = add_rn(y.v[v], ix); // the image along x first
        T a = (at_l || at_e) && x_first ? before : y.v[v];
        const T with = add_rn(a, T(iy.v[v]));
        a = along ? with : a;
        const T after = add_rn(a, ix);
        y.v[v] = (at_l || at_e) && !x_first ? after : a;
    }
}

// Adds to a row of cells the images of the faces that it touches (fr, ba: y-, y+; fi, la: x-, x+;
// bo, to: z-, z+): l, e, across, beyond are the cells beyond along x, y and z. An axis has at least two cells, so a
// cell touches at most one face of each; their images are added in the order of their ranks (7:
// no image).
template <typename T>
__device__ __forceinline__ void add_images(cells<T>& y, const pass_domain& d, bool fr, bool ba, bool fi, bool la, bool bo, bool to, int m, T l, T e,
    const cells<T>& across, const cells<T>& beyond, T alpha)
{
    constexpr int V = cells<T>::V;
    if (!(fr || ba || bo || to))
    {
        if (fi && d.f[0].p) y.v[0] = add_rn(y.v[0], image(l, alpha));
        if (la && d.f[1].p)
        {
            const T add = image(e, alpha);
            if (m == V) y.v[V - 1] = add_rn(y.v[V - 1], add);
            else
            {
#pragma unroll
                for (int v = 0; v < V - 1; ++v)
                {
                    const T sum = add_rn(y.v[v], add);
                    y.v[v] = v == m - 1 ? sum : y.v[v];
                }
            }
        }
        return;
    }
    const auto rank = [&](bool at, int f) { return at ? (int)(d.ranks >> (3 * f)) & 7 : 7; };
    const int rl = rank(fi, 0), rr = rank(la, 1);
    const int ry = fr ? rank(true, 2) : rank(ba, 3);
    const int rz = bo ? rank(true, 4) : rank(to, 5);
#pragma unroll
    for (int v = 0; v < V; ++v)
    {
        int rx = 7;
        T gx = T(0);
        if (v == 0 && rl < 7) rx = rl, gx = l;
        if (v == m - 1 && rr < 7) rx = rr, gx = e;
        const T ix = image(gx, alpha), iy = image(across.v[v], alpha), iz = image(beyond.v[v], alpha);
        T a = y.v[v];
        // three rounds: the image of the least rank left
        const bool x0 = rx < ry && rx < rz, y0 = !x0 && ry < rz;
        const int r0 = x0 ? rx : y0 ? ry : rz;
        a = r0 < 7 ? add_rn(a, x0 ? T(ix) : y0 ? T(iy) : T(iz)) : a;
        const int x1 = rx == r0 ? 7 : rx, y1 = ry == r0 ? 7 : ry, z1 = rz == r0 ? 7 : rz;
        const bool xs = x1 < y1 && x1 < z1, ys = !xs && y1 < z1;
        const int r1 = xs ? x1 : ys ? y1 : z1;
        a = r1 < 7 ? add_rn(a, xs ? T(ix) : ys ? T(iy) : T(iz)) : a;
        const bool x2 = x1 < 7 && x1 != r1, y2 = y1 < 7 && y1 != r1, z2 = z1 < 7 && z1 != r1;
        y.v[v] = x2 || y2 || z2 ? add_rn(a, x2 ? T(ix) : y2 ? T(iy) : T(iz)) : a;
    }
}

template <typename T, bool ADJOINT, bool OUT_PACKED>
__global__ void __launch_bounds__(k_threads, k_resident) pass_kernel(const __grid_constant__ pass_args args, T alpha)
{
    constexpr int V = cells<T>::V, R = k_rows;
    uint32_t b = blockIdx.x;
    int di = 0;
    while (di + 1 < args.n && b >= args.d[di + 1].block0) ++di;
    const pass_domain& d = args.d[di];
    b -= d.block0;
    follow();
    if (b >= d.marches)
    {
        if constexpr (!OUT_PACKED) write_halo<T, ADJOINT, false, k_threads>(d, alpha, b - d.marches);
        return;
    }
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const uint32_t bz = b / d.groups, t = (b - bz * d.groups) * k_threads + threadIdx.x;
    const bool live = t < d.columns; // the others only take part in the shuffles
    const uint32_t column = live ? t : d.columns - 1, strip = column / d.chunks;
    const int k0 = (int)(bz * d.slab), k1 = min(nz, k0 + (int)d.slab);
    const int i0 = (int)(column - strip * d.chunks) * V, m = min(V, nx - i0);
    const int j0 = min((int)strip * R, ny - R); // the last strip overlaps the one before (same values)
    const T* in = static_cast<const T*>(d.in);
    T* __restrict__ out = static_cast<T*>(d.out);
    const int sx = d.isx, sy = d.isy, sz = d.isz;
    const bool first = i0 == 0, last = i0 + V >= nx; // the chunk touches face x-, x+
    const int lane = threadIdx.x & 31;

    const T* const c0 = in + (i0 * sx + j0 * sy);
    // the rows before and after the strip and the cells beside it, in the column's own domain or
    // beyond a face (nullptr: zeros)
    const T *lo = c0 - sy, *hi = c0 + R * sy;
    int lo_x = sx, lo_z = sz, hi_x = sx, hi_z = sz;
    const auto face = [&](int f) { return static_cast<const T*>(d.f[f].p); };
    const bool front = j0 == 0, back = j0 + R == ny; // the strip touches face y-, y+
    if (front) lo = face(2) ? face(2) + i0 * d.f[2].s0 : nullptr, lo_x = d.f[2].s0, lo_z = d.f[2].s1;
    if (back) hi = face(3) ? face(3) + i0 * d.f[3].s0 : nullptr, hi_x = d.f[3].s0, hi_z = d.f[3].s1;
    // a neighbouring lane holds the cell beside a row but at the ends of the row and of the warp,
    // where a thread reads the cell itself: the left one, or the right one, seldom both
    struct side_cells
    {
        const T* p;
        int y, z;
    };
    const bool need_left = first || lane == 0, need_right = last || lane == 31, need_both = need_left && need_right;
    const auto left_cells = [&]() -> side_cells {
        return first ? side_cells{face(0) ? face(0) + j0 * d.f[0].s0 : nullptr, d.f[0].s0, d.f[0].s1} : side_cells{c0 - sx, sy, sz};
    };
    const auto right_cells = [&]() -> side_cells {
        return last ? side_cells{face(1) ? face(1) + j0 * d.f[1].s0 : nullptr, d.f[1].s0, d.f[1].s1} : side_cells{c0 + V * sx, sy, sz};
    };
    const side_cells side = need_left ? left_cells() : need_right ? right_cells() : side_cells{nullptr, 0, 0};

    extern __shared__ __align__(16) char shared[];
    char* const mine = shared + threadIdx.x * 16;
    char* const beside = shared + (R + 2) * ring<T>::wide + threadIdx.x * sizeof(T);
    const uint32_t mine_at = (uint32_t)__cvta_generic_to_shared(mine), beside_at = (uint32_t)__cvta_generic_to_shared(beside);
    const auto copy_cells = [&](uint32_t at, const T* p, int stride, bool valid) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            copy_async<(int)sizeof(T)>(at + v * (int)sizeof(T), valid && v < m ? p + v * stride : in, valid && v < m);
    };
    const auto issue = [&](int k, uint32_t st) { // plane k into the ring at byte st
        if (k <= k1)
        {
            if (k >= 0 && k < nz)
            {
                const T* q = c0 + k * sz;
#pragma unroll
                for (int r = 0; r < R; ++r) copy_cells(mine_at + st + (r + 1) * ring<T>::wide, q + r * sy, sx, true);
                if (k >= k0 && k < k1)
                {
                    copy_cells(mine_at + st, lo + k * lo_z, lo_x, lo != nullptr);
                    copy_cells(mine_at + st + (R + 1) * ring<T>::wide, hi + k * hi_z, hi_x, hi != nullptr);
                    if (need_left || need_right)
                    {
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            copy_async<(int)sizeof(T)>(beside_at + st + r * ring<T>::narrow, side.p ? side.p + (r * side.y + k * side.z) : in, side.p != nullptr);
                    }
                    if (need_both)
                    {
                        const side_cells s = right_cells();
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            copy_async<(int)sizeof(T)>(beside_at + st + (R + r) * ring<T>::narrow, s.p ? s.p + (r * s.y + k * s.z) : in, s.p != nullptr);
                    }
                }
            }
            else
            {
                const int f = k < 0 ? 4 : 5, s0 = d.f[f].s0, s1 = d.f[f].s1;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    copy_cells(mine_at + st + (r + 1) * ring<T>::wide, face(f) + (i0 * s0 + (j0 + r) * s1), s0, face(f) != nullptr);
            }
        }
        copy_commit();
    };
    const auto wide = [&](uint32_t st, int row) { // row -1 .. R of a plane
        return *reinterpret_cast<const cells<T>*>(mine + st + (row + 1) * ring<T>::wide);
    };
    const auto narrow = [&](uint32_t st, int q) {
        return *reinterpret_cast<const T*>(beside + st + q * ring<T>::narrow);
    };

    cells<T> below[R], cur[R], next[R];
#pragma unroll
    for (int p = 0; p < k_stages; ++p) issue(k0 - 1 + p, p * ring<T>::stage);
    copy_wait<k_stages - 2>();
#pragma unroll
    for (int r = 0; r < R; ++r) below[r] = wide(0, r), cur[r] = wide(ring<T>::stage, r);
    uint32_t here = ring<T>::stage, free_at = 0; // plane k, the plane before it
    T* o = out + (i0 * (OUT_PACKED ? 1 : d.osx) + j0 * d.osy + k0 * d.osz);
#pragma unroll 1
    for (int k = k0; k < k1; ++k)
    {
        if (k + 1 == k1) lead();
        issue(k + k_stages - 1, free_at);
        copy_wait<k_stages - 2>(); // plane k + 1 has landed
        const uint32_t up = here + ring<T>::stage == ring<T>::bytes ? 0 : here + ring<T>::stage;
#pragma unroll
        for (int r = 0; r < R; ++r) next[r] = wide(up, r);
        const cells<T> clo = wide(here, -1), chi = wide(here, R);
        // In the transpose a cell beyond a face is not a neighbour (zero) but beside an image of
        // the cell on this side.
        const bool bottom = ADJOINT && k == 0, top = ADJOINT && k == nz - 1;
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            T l = __shfl_up_sync(0xffffffffu, cur[r].v[V - 1], 1), e = __shfl_down_sync(0xffffffffu, cur[r].v[0], 1);
            const T n = narrow(here, r);
            if (need_left) l = n;
            else if (need_right) e = n;
            if (need_both) e = narrow(here, R + r);
            const T before = ADJOINT && first ? T(0) : l, after = ADJOINT && last ? T(0) : e;
            cells<T> y = update(cur[r], before, after, m, r > 0 ? cur[r > 0 ? r - 1 : 0] : zero_if(ADJOINT && front, clo),
                r < R - 1 ? cur[r + 1 < R ? r + 1 : r] : zero_if(ADJOINT && back, chi), zero_if(bottom, below[r]), zero_if(top, next[r]), alpha);
            if constexpr (ADJOINT)
                add_images<T>(y, d, r == 0 && front, r == R - 1 && back, first, last, bottom, top, m, l, e, r == 0 && front ? clo : chi, bottom ? below[r] : next[r], alpha);
            if (!live) continue;
            if constexpr (OUT_PACKED)
                *reinterpret_cast<cells<T>*>(o + r * d.osy) = y;
            else
            {
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (v < m) o[v * d.osx + r * d.osy] = y.v[v];
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) below[r] = cur[r], cur[r] = next[r];
        free_at = here, here = up;
        o += d.osz;
    }
}

// ---- packed input: tiles through the copy engine -------------------------------------------------
// A pass over a packed buffer reads a tile of rows (with the rows and chunks around it) per plane
// by one tensor-map load into a ring of k_tile_stages planes, issued by a warp of its own as the
// other warps release stages; cells beyond the domain arrive as zeros. The rows beyond faces y- and
// y+ come beside the tile by one bulk load each, the plane beyond z- or z+ through the neighbour's
// map, and the cells beyond x- and x+ by single element copies of the threads that need them. A
// thread marches along z with its column of 16 bytes by R rows, as above, and reads each plane of
// it once from shared memory; the load/store unit moves no byte into shared memory, which is what
// bounded the thread-private rings above on packed input (L1 82 % busy; a step of 27.9 / 43.3 us in
// float64, 13.7 / 23.4 us in float32, 215 / 314 us on the large grid).
//
// What bounds it now: forward, HBM (float64) and the latency of a plane's chain of roundings with
// 16 warps per SM (float32); the transpose, its images: a tile on a face adds them after the sum, a
// second chain of roundings. Measured alike or slower: 128 or 224 marching threads, 2 or 3 rows a
// thread (24.4 / 36.2 us), 5 or 6 planes, a block barrier in place of the released stages (25 / 37).
constexpr int k_tile_threads = 96, k_tile_stages = 4, k_tile_resident = 4; // marching threads, planes, blocks per SM
constexpr int k_tile_rows = 4; // rows of a thread; 2 for domains of fewer rows

struct tile_domain
{
    pass_domain d;
    uint32_t cw, strips;  // chunks and strips of a tile
    uint32_t xtiles, ytiles;
    uint32_t pitch;       // bytes of a tile row: cw + 2 chunks
    uint32_t face0, side0, stage; // byte offsets in a stage of the face rows and the cells beside, and its size
};
struct tile_args
{
    tile_domain t[k_batch];
    CUtensorMap map[k_batch][3]; // the domain's buffer, the ones of its neighbours across z- and z+
    int32_t zlo[k_batch], zhi[k_batch]; // the plane of those next to the domain, or -1 and nz of its own (zeros)
    unsigned* status;
    int n;
};

__device__ __forceinline__ void load_tile(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}

template <typename T, bool ADJOINT, bool TWICE, bool OUT_PACKED, int R>
__global__ void __launch_bounds__(k_tile_threads + 32, k_tile_resident) tile_kernel(const __grid_constant__ tile_args args, T alpha)
{
    constexpr int V = cells<T>::V, S = k_tile_stages;
    uint32_t b = blockIdx.x;
    int di = 0;
    while (di + 1 < args.n && b >= args.t[di + 1].d.block0) ++di;
    const tile_domain& g = args.t[di];
    const pass_domain& d = g.d;
    b -= d.block0;
    if (b >= d.marches)
    {
        follow();
        if constexpr (!OUT_PACKED) write_halo<T, ADJOINT, TWICE, k_tile_threads + 32>(d, alpha, b - d.marches);
        return;
    }
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const uint32_t tx = b % g.xtiles, rest = b / g.xtiles, ty = rest % g.ytiles, bz = rest / g.ytiles;
    const int k0 = (int)(bz * d.slab), k1 = min(nz, k0 + (int)d.slab);
    const int h = (int)g.strips * R;
    const int c0 = (int)min(tx * g.cw, d.chunks - g.cw), y0 = min((int)ty * h, max(0, ny - h)); // the last tiles overlap
    const uint32_t columns = g.cw * g.strips, column = min((uint32_t)threadIdx.x, columns - 1);
    const bool live = threadIdx.x < columns;
    const int s = (int)(column / g.cw), c = (int)(column - (uint32_t)s * g.cw);
    const int i0 = (c0 + c) * V, m = min(V, nx - i0), j0 = min(y0 + s * R, ny - R);
    const bool first = i0 == 0, last = i0 + V >= nx, front = j0 == 0, back = j0 + R == ny;
    const auto face = [&](int f) { return static_cast<const T*>(d.f[f].p); };

    extern __shared__ __align__(128) unsigned char dynamic[];
    unsigned char* const shared = dynamic + (128u - smem_u32(dynamic) % 128u) % 128u; // stages start on 128 bytes
    __shared__ __align__(8) uint64_t full[S], empty[S]; // a stage has landed; every warp has read it
    if (threadIdx.x == 0)
    {
#pragma unroll
        for (int q = 0; q < S; ++q) mbar_init(&full[q], 1), mbar_init(&empty[q], k_tile_threads / 32);
        mbar_init_fence();
    }
    __syncthreads();
    follow();
    // planes k0 - 1 .. k1 of the slab, numbered from 0
    const int planes = k1 - k0 + 2;
    const bool row_lo = y0 == 0 && face(2), row_hi = y0 + h >= ny && face(3);
    const bool edge_tile = row_lo || row_hi || (c0 == 0 && face(0)) || ((uint32_t)c0 + g.cw >= d.chunks && face(1)); // it touches a face with images
    const uint32_t wide = g.cw * 16u;
    const auto issue = [&](int q, int st) { // the loads of plane q into stage st
        const int k = k0 - 1 + q;
        unsigned char* dst = shared + (uint32_t)st * g.stage;
        const bool inner = q > 0 && q + 1 < planes;
        mbar_expect_tx(&full[st], g.pitch * (uint32_t)(h + 2) + (inner ? wide * ((row_lo ? 1u : 0u) + (row_hi ? 1u : 0u)) : 0u));
        const int which = k < 0 ? 1 : k == nz ? 2 : 0;
        load_tile(dst, &args.map[di][which], c0 * V - V, y0 - 1, which == 0 ? k : which == 1 ? args.zlo[di] : args.zhi[di], &full[st]);
        if (inner && row_lo) bulk_load(dst + g.face0, face(2) + (c0 * V + k * d.f[2].s1), wide, &full[st]);
        if (inner && row_hi) bulk_load(dst + g.face0 + wide, face(3) + (c0 * V + k * d.f[3].s1), wide, &full[st]);
    };
    if (threadIdx.x >= k_tile_threads) // the last warp issues the loads, as stages become free
    {
        if (threadIdx.x == k_tile_threads)
        {
            int issued = 0;
            for (; issued < planes; ++issued)
            {
                const int st = issued % S;
                if (issued >= S && !mbar_wait(&empty[st], (uint32_t)(issued / S - 1) & 1u))
                {
                    report(args.status);
                    break;
                }
                issue(issued, st);
            }
            // the block's shared memory is not given back before its last loads have landed, also where
            // the stages ran out or the other threads gave up
            for (int q = max(0, issued - S); q < issued; ++q) mbar_wait(&full[q % S], (uint32_t)(q / S) & 1u);
        }
        return;
    }
    // the cells beyond x- and x+ beside this thread's rows (only a thread with a column of its own
    // writes them: the others stand on the last column, and their warps may be planes ahead of it)
    const bool side_lo = first && face(0), side_hi = last && face(1);
    const uint32_t side = g.side0 + (uint32_t)(s * R) * (uint32_t)sizeof(T), side_other = side + (uint32_t)h * (uint32_t)sizeof(T);
    const auto issue_sides = [&](int q, int st) {
        if (live && (side_lo || side_hi) && q > 0 && q + 1 < planes)
        {
            const uint32_t at = smem_u32(shared + (uint32_t)st * g.stage);
            const int k = k0 - 1 + q;
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                if (side_lo) copy_async<(int)sizeof(T)>(at + side + r * (int)sizeof(T), face(0) + ((j0 + r) * d.f[0].s0 + k * d.f[0].s1), true);
                if (side_hi) copy_async<(int)sizeof(T)>(at + side_other + r * (int)sizeof(T), face(1) + ((j0 + r) * d.f[1].s0 + k * d.f[1].s1), true);
            }
        }
        copy_commit();
    };
    // a load did not arrive in time: nothing more is waited for, and what depends on it is not a
    // number, here and in every result computed from it
    bool failed = false;
    const auto wait = [&](int st, uint32_t parity) {
        if (!failed && !mbar_wait(&full[st], parity))
        {
            failed = true;
            report(args.status);
        }
    };
#pragma unroll
    for (int q = 0; q < S; ++q) issue_sides(q, q);
    const uint32_t at = (uint32_t)(j0 - y0 + 1) * g.pitch + (uint32_t)(c + 1) * 16u; // row 0 of the strip in a stage
    const auto read = [&](uint32_t off) {
        cells<T> v = *reinterpret_cast<const cells<T>*>(shared + off);
        if constexpr (TWICE)
        {
#pragma unroll
            for (int e = 0; e < V; ++e) v.v[e] = mul_rn(T(2), v.v[e]);
        }
        return v;
    };
    const auto read_one = [&](uint32_t off) {
        const T v = *reinterpret_cast<const T*>(shared + off);
        return TWICE ? mul_rn(T(2), v) : v;
    };
    // the rows before and after the strip and the cells beside it in a stage: the tile's own (zeros
    // beyond the domain) or, forward, what came from beyond a face
    const bool far_lo = front && row_lo, far_hi = back && row_hi;
    const uint32_t face_lo = g.face0 + (uint32_t)c * 16u, face_hi = face_lo + wide;
    const uint32_t lo_at = !ADJOINT && far_lo ? face_lo : at - g.pitch, hi_at = !ADJOINT && far_hi ? face_hi : at + R * g.pitch;
    const uint32_t left_at = !ADJOINT && side_lo ? side : at - (uint32_t)sizeof(T), left_step = !ADJOINT && side_lo ? (uint32_t)sizeof(T) : g.pitch;
    const uint32_t right_at = !ADJOINT && side_hi ? side_other : at + 16u, right_step = !ADJOINT && side_hi ? (uint32_t)sizeof(T) : g.pitch;

    cells<T> below[R], cur[R], next[R];
    wait(0, 0);
    wait(1, 0);
#pragma unroll
    for (int r = 0; r < R; ++r) below[r] = read(at + r * g.pitch), cur[r] = read(g.stage + at + r * g.pitch);
    // after the warp's reads of a stage. The copy engine's writes do not wait for reads that are
    // merely issued: in the loop the values read are used (stored) before, here the fence waits.
    const auto release = [&](int st) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(&empty[st]);
    };
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    release(0);
    int st = 1, up = 2 % S; // the stages of planes k and k + 1
    uint32_t up_parity = 2 / S;
    T* o = static_cast<T*>(d.out) + (i0 * (OUT_PACKED ? 1 : d.osx) + j0 * d.osy + k0 * d.osz);
#pragma unroll 1
    for (int k = k0; k < k1; ++k)
    {
        const int q = k - k0 + 1;
        if (k + 1 == k1) lead();
        issue_sides(q - 1 + S, st == 0 ? S - 1 : st - 1); // (a thread's own, read one plane ago)
        wait(up, up_parity);
        copy_wait<S - 1>(); // the sides of plane q
        const uint32_t here = (uint32_t)st * g.stage, above = (uint32_t)up * g.stage;
#pragma unroll
        for (int r = 0; r < R; ++r) next[r] = read(above + at + r * g.pitch);
        const cells<T> clo = read(here + lo_at), chi = read(here + hi_at);
        // In the transpose a plane beyond a face is not a neighbour but images of this plane.
        const bool bottom = ADJOINT && k == 0, top = ADJOINT && k == nz - 1;
        cells<T> beyond[R];
        if (ADJOINT && (bottom || top))
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                beyond[r] = bottom ? below[r] : next[r];
                below[r] = zero_if(bottom, below[r]), next[r] = zero_if(top, next[r]);
            }
        }
        cells<T> y[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            y[r] = update(cur[r], read_one(here + left_at + r * left_step), read_one(here + right_at + r * right_step), m,
                r > 0 ? cur[r > 0 ? r - 1 : 0] : clo, r < R - 1 ? cur[r + 1 < R ? r + 1 : r] : chi, below[r], next[r], alpha);
        if (ADJOINT && (edge_tile || bottom || top)) // the same for the whole block
        {
            // the images of a thread's rows together: their chains of roundings are long, and overlap
            T l[R], e[R];
            cells<T> across[R];
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                l[r] = side_lo ? read_one(here + side + r * (uint32_t)sizeof(T)) : T(0);
                e[r] = side_hi ? read_one(here + side_other + r * (uint32_t)sizeof(T)) : T(0);
                zero(across[r]);
                if (r == 0 && far_lo) across[r] = read(here + face_lo);
                if (r == R - 1 && far_hi) across[r] = read(here + face_hi);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                const bool lo = r == 0 && far_lo, hi = r == R - 1 && far_hi;
                if (bottom || top) add_images<T>(y[r], d, lo, hi, side_lo, side_hi, bottom, top, m, l[r], e[r], across[r], beyond[r], alpha);
                else
                {
                    cells<T> iy;
#pragma unroll
                    for (int v = 0; v < V; ++v) iy.v[v] = image(across[r].v[v], alpha);
                    const uint32_t ry = (d.ranks >> (lo ? 6 : 9)) & 7u;
                    const bool along = lo || hi;
                    add_row_images<T>(y[r], along, iy, side_lo, side_hi, image(l[r], alpha), image(e[r], alpha), !along || (d.ranks & 7u) < ry,
                        !along || ((d.ranks >> 3) & 7u) < ry, m);
                }
            }
        }
        if (failed)
        {
#pragma unroll
            for (int r = 0; r < R; ++r) not_a_number(y[r]);
        }
        if (live)
        {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if constexpr (OUT_PACKED)
                    *reinterpret_cast<cells<T>*>(o + r * d.osy) = y[r];
                else
                {
#pragma unroll
                    for (int v = 0; v < V; ++v)
                        if (v < m) o[v * d.osx + r * d.osy] = y[r].v[v];
                }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) below[r] = cur[r], cur[r] = next[r];
        o += d.osz;
        release(st);
        st = up;
        if (++up == S) up = 0, up_parity ^= 1u;
    }
    copy_wait<0>();
}

// The number of slabs a pass cuts the z axis into: the least time in planes (every slab starts
// with a few loads that nothing hides) over the waves of resident blocks. groups: blocks a slab.
int slabs_of(uint64_t groups, int nz, int per_sm)
{
    int best = 1;
    double least = 0;
    for (int s = 1; s <= std::max(1, nz / k_min_slab); ++s)
    {
        const double blocks = (double)(groups * s), resident = (double)k_sms * per_sm;
        const double waves = blocks <= resident ? 1.0 : (double)(int64_t)((blocks + resident - 1) / resident);
        const double planes = waves * ((nz + s - 1) / s + 3);
        if (s == 1 || planes < least) best = s, least = planes;
    }
    return best;
}

// What a pass reads and writes: fields in the caller's layout, or (fields null) a packed buffer.
struct pass_io
{
    const void* const* in;
    const void* source;
    void* const* out;
    void* packed;
};

int64_t in_stride(const program_domain& d, bool packed, int a) { return packed ? (a == 0 ? 1 : a == 1 ? d.row : d.plane) : d.s[a]; }
const char* in_cell(const ghexb_program_s& P, const pass_io& io, int slot) // interior cell (0, 0, 0)
{
    const program_domain& d = P.domains[slot];
    const int64_t es = P.f64 ? 8 : 4;
    return io.source ? static_cast<const char*>(io.source) + d.offset * es
                     : static_cast<const char*>(io.in[slot]) + P.halo * (d.s[0] + d.s[1] + d.s[2]) * es;
}

void fill_domain(pass_domain& a, const ghexb_program_s& P, const pass_io& io, int slot, bool adjoint)
{
    const program_domain& d = P.domains[slot];
    const int64_t es = P.f64 ? 8 : 4, h = P.halo;
    const bool packed = io.source != nullptr;
    a.in = in_cell(P, io, slot);
    a.out = io.out ? static_cast<char*>(io.out[slot]) + h * (d.s[0] + d.s[1] + d.s[2]) * es : static_cast<char*>(io.packed) + d.offset * es;
    a.nx = d.n[0], a.ny = d.n[1], a.nz = d.n[2], a.halo = P.halo;
    a.isx = (int32_t)in_stride(d, packed, 0), a.isy = (int32_t)in_stride(d, packed, 1), a.isz = (int32_t)in_stride(d, packed, 2);
    a.osx = (int32_t)(io.out ? d.s[0] : 1), a.osy = (int32_t)(io.out ? d.s[1] : d.row), a.osz = (int32_t)(io.out ? d.s[2] : d.plane);
    a.ranks = d.ranks, a.images = d.images;
    for (int f = 0; f < 6; ++f)
    {
        const int axis = f / 2, u = axis == 0 ? 1 : 0, v = axis == 2 ? 1 : 2;
        const int e = adjoint ? d.to[f] : d.from[f];
        a.f[f] = {nullptr, 0, 0};
        if (e >= 0)
        {
            // the face cells of the neighbour that face this domain
            const program_domain& nb = P.domains[e];
            const int64_t at = f % 2 == 0 ? nb.n[axis] - 1 : 0;
            a.f[f] = {in_cell(P, io, e) + at * in_stride(nb, packed, axis) * es, (int32_t)in_stride(nb, packed, u), (int32_t)in_stride(nb, packed, v)};
        }
        else if (!adjoint && !packed)
        {
            // no exchange fills this halo: the caller's own halo cells (zero after a step)
            const int64_t at = f % 2 == 0 ? -1 : d.n[axis];
            a.f[f] = {in_cell(P, io, slot) + at * d.s[axis] * es, (int32_t)d.s[u], (int32_t)d.s[v]};
        }
    }
}

// blocks of `threads` threads that write a domain's halo
uint64_t halo_blocks(const program_domain& d, int64_t h, int threads)
{
    const uint64_t all = (uint64_t)(d.n[0] + 2 * h) * (d.n[1] + 2 * h) * (d.n[2] + 2 * h);
    const uint64_t inner = (uint64_t)d.n[0] * d.n[1] * d.n[2], per = (uint64_t)threads * k_halo_cells;
    return (all - inner + per - 1) / per;
}

template <typename T, bool ADJOINT, bool OUT_PACKED>
cudaError_t launch_fields(const ghexb_program_s& P, const pass_io& io, double alpha, cudaStream_t stream)
{
    const int n = (int)P.domains.size();
    for (int b0 = 0; b0 < n; b0 += k_batch)
    {
        pass_args args;
        args.n = std::min(k_batch, n - b0);
        uint64_t groups = 0, blocks = 0;
        int nz = 1;
        for (int i = 0; i < args.n; ++i)
        {
            const program_domain& d = P.domains[b0 + i];
            pass_domain& a = args.d[i];
            fill_domain(a, P, io, b0 + i, ADJOINT);
            a.chunks = (uint32_t)((d.n[0] + cells<T>::V - 1) / cells<T>::V);
            a.columns = a.chunks * (uint32_t)((d.n[1] + k_rows - 1) / k_rows);
            a.groups = (a.columns + k_threads - 1) / k_threads;
            groups += a.groups;
            nz = std::max(nz, d.n[2]);
        }
        const int slabs = slabs_of(groups, nz, k_resident);
        for (int i = 0; i < args.n; ++i)
        {
            pass_domain& a = args.d[i];
            a.slab = (uint32_t)((a.nz + slabs - 1) / slabs);
            a.block0 = (uint32_t)blocks;
            const uint64_t marches = (uint64_t)a.groups * ((a.nz + a.slab - 1) / a.slab);
            a.marches = (uint32_t)marches;
            blocks += marches + (OUT_PACKED ? 0 : halo_blocks(P.domains[b0 + i], P.halo, k_threads));
        }
        if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
        const auto kernel = pass_kernel<T, ADJOINT, OUT_PACKED>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ring<T>::bytes);
        if (e != cudaSuccess) return e;
        e = launch_following(kernel, (unsigned)blocks, k_threads, ring<T>::bytes, stream, args, (T)alpha);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// The tile of a domain of `chunks` by `strips` columns: the one of least cost, a block's time in
// units of its threads' work plus the cells its loads move beyond its own.
void shape_tile(tile_domain& t, uint32_t chunks, uint32_t strips, int V, int rows)
{
    double least = 0;
    t.cw = 0;
    const uint32_t widest = std::min<uint32_t>(k_tile_threads, 256u / V - 2u); // a load box is at most 256 elements wide
    const uint32_t tallest = (256u - 2u) / (uint32_t)rows; // and at most 256 rows high, the ones around the tile among them
    const uint32_t few = (chunks + widest - 1) / widest;
    for (uint32_t nt = few; nt <= std::min(chunks, few + 16); ++nt)
    {
        const uint32_t cw = (chunks + nt - 1) / nt;
        const uint32_t hs = std::min(std::min((uint32_t)k_tile_threads / cw, strips), tallest);
        const double blocks = (double)((chunks + cw - 1) / cw) * ((strips + hs - 1) / hs);
        const double cost = blocks * (1.0 + (double)(cw + 2) * (hs * rows + 2) / (k_tile_threads * rows));
        if (t.cw == 0 || cost < least) t.cw = cw, t.strips = hs, least = cost;
    }
    t.xtiles = (chunks + t.cw - 1) / t.cw;
    t.ytiles = (strips + t.strips - 1) / t.strips;
}

template <typename T, bool ADJOINT, bool TWICE, bool OUT_PACKED, int R>
cudaError_t launch_tiles_r(const ghexb_program_s& P, const pass_io& io, double alpha, cudaStream_t stream)
{
    const int n = (int)P.domains.size(), V = cells<T>::V;
    const int64_t es = sizeof(T);
    for (int b0 = 0; b0 < n; b0 += k_batch)
    {
        tile_args args;
        args.n = std::min(k_batch, n - b0);
        args.status = P.status;
        uint64_t groups = 0, blocks = 0;
        uint32_t stage = 0;
        int nz = 1;
        for (int i = 0; i < args.n; ++i)
        {
            const program_domain& d = P.domains[b0 + i];
            tile_domain& t = args.t[i];
            fill_domain(t.d, P, io, b0 + i, ADJOINT);
            t.d.chunks = (uint32_t)((d.n[0] + V - 1) / V);
            shape_tile(t, t.d.chunks, (uint32_t)((d.n[1] + R - 1) / R), V, R);
            const uint32_t h = t.strips * R;
            t.pitch = (t.cw + 2) * 16u;
            t.face0 = (t.pitch * (h + 2) + 15u) / 16u * 16u;
            t.side0 = t.face0 + 2u * t.cw * 16u;
            t.stage = (t.side0 + 2u * h * (uint32_t)es + 127u) / 128u * 128u;
            stage = std::max(stage, t.stage);
            groups += (uint64_t)t.xtiles * t.ytiles;
            nz = std::max(nz, d.n[2]);
            for (int w = 0; w < 3; ++w)
            {
                const int e = w == 0 ? -1 : ADJOINT ? d.to[w + 3] : d.from[w + 3];
                const int slot = e >= 0 ? e : b0 + i; // without a neighbour: beyond the domain's own planes, zeros
                const program_domain& nb = P.domains[slot];
                const cuuint64_t dims[3] = {(cuuint64_t)nb.n[0], (cuuint64_t)nb.n[1], (cuuint64_t)nb.n[2]};
                const cuuint64_t strides[2] = {(cuuint64_t)(nb.row * es), (cuuint64_t)(nb.plane * es)};
                const cuuint32_t box[3] = {(t.cw + 2) * V, h + 2, 1};
                if (encode_tensor_map(&args.map[i][w], es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                        const_cast<char*>(in_cell(P, io, slot)), dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS)
                    return cudaErrorInvalidValue;
                if (w == 1) args.zlo[i] = e >= 0 ? nb.n[2] - 1 : -1;
                if (w == 2) args.zhi[i] = e >= 0 ? 0 : nb.n[2];
            }
        }
        const uint32_t bytes = stage * k_tile_stages + 128u;
        const int per_sm = std::max(1, std::min(k_tile_resident, (int)(227u * 1024u / (bytes + 1024u))));
        const int slabs = slabs_of(groups, nz, per_sm);
        for (int i = 0; i < args.n; ++i)
        {
            tile_domain& t = args.t[i];
            pass_domain& a = t.d;
            a.slab = (uint32_t)((a.nz + slabs - 1) / slabs);
            a.block0 = (uint32_t)blocks;
            const uint64_t marches = (uint64_t)t.xtiles * t.ytiles * ((a.nz + a.slab - 1) / a.slab);
            a.marches = (uint32_t)marches;
            blocks += marches + (OUT_PACKED ? 0 : halo_blocks(P.domains[b0 + i], P.halo, k_tile_threads + 32));
        }
        if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
        const auto kernel = tile_kernel<T, ADJOINT, TWICE, OUT_PACKED, R>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        e = launch_following(kernel, (unsigned)blocks, k_tile_threads + 32, bytes, stream, args, (T)alpha);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename T, bool ADJOINT, bool TWICE, bool OUT_PACKED>
cudaError_t launch_tiles(const ghexb_program_s& P, const pass_io& io, double alpha, cudaStream_t stream)
{
    bool rows = true;
    for (const auto& d : P.domains) rows = rows && d.n[1] >= k_tile_rows;
    return rows ? launch_tiles_r<T, ADJOINT, TWICE, OUT_PACKED, k_tile_rows>(P, io, alpha, stream)
                : launch_tiles_r<T, ADJOINT, TWICE, OUT_PACKED, k_rows>(P, io, alpha, stream);
}

template <typename T, bool ADJOINT, bool TWICE>
cudaError_t launch_passes_t(const ghexb_program_s& P, const void* const* fields, const void* source, void* const* out, void* a,
    void* b, int steps, double alpha, cudaStream_t stream)
{
    // the first pass reads the source as it is given, the later ones a packed buffer, unscaled
    cudaError_t e = cudaSuccess;
    for (int s = 0; s < steps && e == cudaSuccess; ++s)
    {
        const bool end = out && s == steps - 1;
        const pass_io io{fields, source, end ? out : nullptr, source == a ? b : a};
        if (!source) e = end ? launch_fields<T, ADJOINT, false>(P, io, alpha, stream) : launch_fields<T, ADJOINT, true>(P, io, alpha, stream);
        else if (TWICE && s == 0) e = end ? launch_tiles<T, ADJOINT, TWICE, false>(P, io, alpha, stream) : launch_tiles<T, ADJOINT, TWICE, true>(P, io, alpha, stream);
        else e = end ? launch_tiles<T, ADJOINT, false, false>(P, io, alpha, stream) : launch_tiles<T, ADJOINT, false, true>(P, io, alpha, stream);
        fields = nullptr, source = io.packed;
    }
    return e;
}

template <typename T>
cudaError_t launch_passes_any(const ghexb_program_s& P, const void* const* fields, const void* source, void* const* out, void* a,
    void* b, int steps, double alpha, bool adjoint, bool twice, cudaStream_t stream)
{
    if (!adjoint) return twice ? cudaErrorInvalidValue : launch_passes_t<T, false, false>(P, fields, source, out, a, b, steps, alpha, stream);
    return twice ? launch_passes_t<T, true, true>(P, fields, source, out, a, b, steps, alpha, stream)
                 : launch_passes_t<T, true, false>(P, fields, source, out, a, b, steps, alpha, stream);
}
} // namespace

cudaError_t launch_passes(const ghexb_program_s& P, const void* const* fields, const void* source, void* const* out, void* a,
    void* b, int steps, double alpha, bool adjoint, bool twice, cudaStream_t stream)
{
    return P.f64 ? launch_passes_any<double>(P, fields, source, out, a, b, steps, alpha, adjoint, twice, stream)
                 : launch_passes_any<float>(P, fields, source, out, a, b, steps, alpha, adjoint, twice, stream);
}

// ---- status words ------------------------------------------------------------------------------
namespace
{
struct status_words
{
    std::mutex mutex;
    std::vector<unsigned*> unused; // each one address on the host and on every device
};
status_words& statuses()
{
    static status_words& words = *new status_words; // programs may outlive the library's statics
    return words;
}
} // namespace

unsigned* take_status_word()
{
    constexpr int count = 1024;
    status_words& s = statuses();
    std::lock_guard<std::mutex> lock(s.mutex);
    if (s.unused.empty())
    {
        void* p = nullptr;
        check_cuda(cudaHostAlloc(&p, count * sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc(program status)");
        for (int i = count; i-- > 0;) s.unused.push_back(static_cast<unsigned*>(p) + i);
    }
    unsigned* word = s.unused.back();
    s.unused.pop_back();
    *word = 0;
    return word;
}

void return_status_word(unsigned* word)
{
    status_words& s = statuses();
    std::lock_guard<std::mutex> lock(s.mutex);
    s.unused.push_back(word);
}
} // namespace ghexb

ghexb_program_s::~ghexb_program_s()
{
    if (status) ghexb::return_status_word(status);
}

namespace ghexb
{
// ---- geometry ----------------------------------------------------------------------------------
void build_program(ghexb_program_s& P, const ghexb_field* fields, int nfields, int halo)
{
    const auto require = [](bool ok, const char* why) {
        if (!ok) throw error(GHEXB_ERR_INVALID, std::string("the program cannot be fused: ") + why);
    };
    require(halo >= 1, "the 7-point update needs a halo of width >= 1");
    const int n = nfields;
    P.f64 = fields[0]->dtype == GHEXB_F64;
    P.halo = halo;
    P.domains.assign(n, program_domain{});
    P.packed_elements = 0;
    const int64_t es = fields[0]->esize;
    // field slots by pattern and domain: the k-th field of a domain pairs with the k-th of its neighbours
    std::map<std::pair<const ghexb_pattern_s*, int>, std::vector<int>> slots;
    std::vector<const ghexb_pattern_s*> patterns;
    for (int s = 0; s < n; ++s)
    {
        const auto& f = *fields[s];
        require(f.pattern->kind == pattern_kind::regular && f.pattern->dim == 3 && f.ndim == 3 && f.num_components == 1, "fields of three regular dimensions only");
        require((f.dtype == GHEXB_F64 || f.dtype == GHEXB_F32) && f.dtype == fields[0]->dtype, "fields of one floating type only");
        if (std::find(patterns.begin(), patterns.end(), f.pattern) == patterns.end()) patterns.push_back(f.pattern);
        slots[{f.pattern, f.domain_index}].push_back(s);
        program_domain& d = P.domains[s];
        const auto& dom = f.pattern->domains[f.domain_index];
        int64_t span = 1, whole = 1;
        for (int a = 0; a < 3; ++a)
        {
            d.n[a] = dom.last[a] - dom.first[a] + 1;
            require(f.offsets[a] == halo && f.extents[a] == d.n[a] + 2 * halo, "fields padded by the halo on every side only");
            require(f.byte_strides[a] > 0 && f.byte_strides[a] % es == 0, "strides of whole elements only");
            d.s[a] = f.byte_strides[a] / es;
            span += (int64_t)(f.extents[a] + 2 * k_rows) * d.s[a];
            whole *= f.extents[a];
        }
        require(span < (int64_t(1) << 31) && whole < (int64_t(1) << 31), "a field of 2^31 elements");
        require(d.n[0] >= 2 && d.n[1] >= k_rows && d.n[2] >= 2, "a domain one cell thick, or of fewer rows than a strip");
        const int64_t unit = 32 / es;
        d.row = (d.n[0] + unit - 1) / unit * unit;
        d.plane = d.row * d.n[1];
        require(d.plane * d.n[2] < (int64_t(1) << 31), "a field of 2^31 elements");
        d.offset = P.packed_elements;
        P.packed_elements += (d.plane * d.n[2] + 127) / 128 * 128;
        for (int k = 0; k < 6; ++k) d.from[k] = d.to[k] = -1;
        d.ranks = 0777777u; // 7 in every place
        d.images = 0;
    }
    std::vector<int> images_added(n, 0);
    for (const auto* pattern : patterns)
        for (int di = 0; di < (int)pattern->domains.size(); ++di)
        {
            const auto it = slots.find({pattern, di});
            if (it == slots.end()) continue;
            for (const auto& entry : pattern->domains[di].recv)
            {
                const auto sit = slots.find({pattern, entry.neighbor});
                require(sit != slots.end() && sit->second.size() == it->second.size(), "a neighbour without the field");
                const auto& sources = sit->second;
                for (size_t k = 0; k < it->second.size(); ++k)
                {
                    const int slot = it->second[k], src = sources[k];
                    program_domain& d = P.domains[slot];
                    program_domain& o = P.domains[src];
                    const auto& owner = pattern->domains[entry.neighbor];
                    for (const auto& sp : entry.spaces)
                    {
                        int side[3], outside = 0, face = -1, region = 0;
                        for (int a = 0, w = 1; a < 3; ++a, w *= 3)
                        {
                            const int lo = sp.lfirst[a], hi = sp.llast[a];
                            side[a] = lo == -halo && hi == -1 ? 0 : lo == 0 && hi == d.n[a] - 1 ? 1 : lo == d.n[a] && hi == d.n[a] + halo - 1 ? 2 : -1;
                            require(side[a] >= 0, "a halo region that several domains fill, or of another width than the update's halo");
                            region += w * side[a];
                            if (side[a] != 1) ++outside, face = 2 * a + (side[a] == 2);
                        }
                        require(outside > 0 && !((d.images >> region) & 1u), "a halo region that is filled twice");
                        d.images |= 1u << region;
                        if (outside != 1) continue; // edges and corners: no cell of the update reads them
                        for (int a = 0; a < 3; ++a)
                        {
                            const int at = sp.has_src ? sp.sfirst[a] : sp.gfirst[a] - owner.first[a];
                            const int want = side[a] == 1 ? 0 : side[a] == 0 ? o.n[a] - halo : 0;
                            require(at == want && (side[a] != 1 || o.n[a] == d.n[a]), "a face that is part of its neighbour's face");
                        }
                        require(d.s[0] > 0 && o.to[face ^ 1] < 0, "a face with two images");
                        d.from[face] = src;
                        o.to[face ^ 1] = slot;
                        o.ranks = (o.ranks & ~(7u << (3 * (face ^ 1)))) | (uint32_t)images_added[src]++ << (3 * (face ^ 1));
                    }
                }
            }
        }
}

// ---- sum of squares of the interiors -------------------------------------------------------------
namespace
{
constexpr int k_sum_threads = 256, k_sum_chunks = 8; // a block adds 2048 chunks of 16 bytes
struct sum_args
{
    struct
    {
        const void* p;
        int32_t nx, ny, nz;
        uint32_t chunks, block0;
        int64_t sx, sy, sz;
        fast_div by_chunks, by_rows; // of chunks and ny, for arrays of fewer than 2^31 chunks
    } d[k_batch];
    int n;
};

__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double part[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = threadIdx.x < blockDim.x >> 5 ? part[threadIdx.x] : 0.0;
    if (threadIdx.x < 32)
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v; // of thread 0
}

// One pass over the interiors, in order of memory: bound by HBM (or L2 where the fields fit it).
template <typename T, bool PACKED>
__global__ void __launch_bounds__(k_sum_threads) sumsq_kernel(const __grid_constant__ sum_args args, double* __restrict__ partials)
{
    constexpr int V = cells<T>::V;
    uint32_t b = blockIdx.x;
    int di = 0;
    while (di + 1 < args.n && b >= args.d[di + 1].block0) ++di;
    const auto& d = args.d[di];
    b -= d.block0;
    follow();
    const uint64_t all = (uint64_t)d.chunks * d.ny * d.nz;
    const T* p = static_cast<const T*>(d.p);
    cells<T> c[k_sum_chunks];
    int m[k_sum_chunks];
#pragma unroll
    for (int q = 0; q < k_sum_chunks; ++q)
    {
        const uint64_t e = ((uint64_t)b * k_sum_chunks + q) * k_sum_threads + threadIdx.x;
        m[q] = 0;
        if (e >= all) continue;
        const uint32_t row = all >> 31 ? (uint32_t)(e / d.chunks) : d.by_chunks.div((uint32_t)e), i0 = (uint32_t)(e - (uint64_t)row * d.chunks) * V;
        const uint32_t k = d.by_rows.div(row), j = row - k * d.ny;
        m[q] = min(V, d.nx - (int)i0);
        if constexpr (PACKED)
        {
            union
            {
                int4 w;
                cells<T> c;
            } u;
            u.w = *reinterpret_cast<const int4*>(p + (i0 + j * d.sy + k * d.sz));
            c[q] = u.c;
        }
        else
        {
#pragma unroll
            for (int v = 0; v < V; ++v) c[q].v[v] = v < m[q] ? p[(int64_t)(i0 + v) * d.sx + j * d.sy + k * d.sz] : T(0);
        }
    }
    double s = 0;
#pragma unroll
    for (int q = 0; q < k_sum_chunks; ++q)
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (v < m[q]) s = __dadd_rn(s, __dmul_rn((double)c[q].v[v], (double)c[q].v[v]));
    s = block_sum(s);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

template <typename T> __global__ void __launch_bounds__(1024) sum_partials_kernel(const double* partials, uint32_t n, T* out)
{
    follow();
    double s = 0;
    for (uint32_t i = threadIdx.x; i < n; i += 1024) s = __dadd_rn(s, partials[i]);
    s = block_sum(s);
    if (threadIdx.x == 0) *out = (T)s;
}

struct grad_args
{
    struct
    {
        const void* p;
        void* out;
        int32_t ex, ey, ez;
        uint32_t block0;
        int64_t sx, sy, sz;
        fast_div by_row, by_rows; // of ex and ey, for arrays of fewer than 2^31 cells
    } d[k_batch];
    int n, halo;
};

template <typename T>
__global__ void __launch_bounds__(k_sum_threads) sumsq_grad_kernel(const __grid_constant__ grad_args args, const T* g)
{
    uint32_t b = blockIdx.x;
    int di = 0;
    while (di + 1 < args.n && b >= args.d[di + 1].block0) ++di;
    const auto& d = args.d[di];
    b -= d.block0;
    const int h = args.halo;
    follow();
    const uint64_t all = (uint64_t)d.ex * d.ey * d.ez;
    const T scale = *g;
    const T* p = static_cast<const T*>(d.p);
    T* __restrict__ out = static_cast<T*>(d.out);
    T x[k_sum_chunks];
    int64_t at[k_sum_chunks];
    bool inside[k_sum_chunks];
#pragma unroll
    for (int q = 0; q < k_sum_chunks; ++q)
    {
        const uint64_t e = ((uint64_t)b * k_sum_chunks + q) * k_sum_threads + threadIdx.x;
        at[q] = -1;
        x[q] = T(0), inside[q] = false;
        if (e >= all) continue;
        const uint32_t row = all >> 31 ? (uint32_t)(e / d.ex) : d.by_row.div((uint32_t)e);
        const int i = (int)(e - (uint64_t)row * d.ex), k = (int)d.by_rows.div(row), j = (int)(row - (uint32_t)k * d.ey);
        at[q] = (int64_t)i * d.sx + (int64_t)j * d.sy + (int64_t)k * d.sz;
        inside[q] = i >= h && i < d.ex - h && j >= h && j < d.ey - h && k >= h && k < d.ez - h;
        if (inside[q]) x[q] = p[at[q]];
    }
    // (products in a loop of their own: every load is under way before the first is waited for)
#pragma unroll
    for (int q = 0; q < k_sum_chunks; ++q)
        if (at[q] >= 0) out[at[q]] = inside[q] ? mul_rn(scale, mul_rn(T(2), x[q])) : T(0);
}

uint64_t sum_blocks(int V, const int32_t* n)
{
    const uint64_t chunks = (uint64_t)((n[0] + V - 1) / V) * n[1] * n[2], per = (uint64_t)k_sum_threads * k_sum_chunks;
    return (chunks + per - 1) / per;
}

template <typename T>
cudaError_t launch_sumsq_t(const interior* d, int n, bool packed, double* partials, void* out, cudaStream_t stream)
{
    uint64_t done = 0;
    for (int b0 = 0; b0 < n; b0 += k_batch)
    {
        sum_args args;
        args.n = std::min(k_batch, n - b0);
        uint64_t blocks = 0;
        for (int i = 0; i < args.n; ++i)
        {
            const interior& s = d[b0 + i];
            auto& a = args.d[i];
            a.p = s.p, a.nx = s.n[0], a.ny = s.n[1], a.nz = s.n[2], a.sx = s.s[0], a.sy = s.s[1], a.sz = s.s[2];
            a.chunks = (uint32_t)((s.n[0] + cells<T>::V - 1) / cells<T>::V);
            a.by_chunks = fast_div::make(a.chunks), a.by_rows = fast_div::make((uint32_t)s.n[1]);
            a.block0 = (uint32_t)blocks;
            blocks += sum_blocks(cells<T>::V, s.n);
        }
        if (done + blocks > 0x7fffffffull) return cudaErrorInvalidValue;
        const cudaError_t e = launch_following(packed ? sumsq_kernel<T, true> : sumsq_kernel<T, false>, (unsigned)blocks, k_sum_threads, 0, stream, args, partials + done);
        done += blocks;
        if (e != cudaSuccess) return e;
    }
    return launch_following(sum_partials_kernel<T>, 1, 1024, 0, stream, (const double*)partials, (uint32_t)done, static_cast<T*>(out));
}

template <typename T>
cudaError_t launch_grad_t(const interior* d, void* const* out, int n, int halo, const void* g, cudaStream_t stream)
{
    for (int b0 = 0; b0 < n; b0 += k_batch)
    {
        grad_args args;
        args.n = std::min(k_batch, n - b0), args.halo = halo;
        uint64_t blocks = 0;
        const uint64_t per = (uint64_t)k_sum_threads * k_sum_chunks;
        for (int i = 0; i < args.n; ++i)
        {
            const interior& s = d[b0 + i];
            auto& a = args.d[i];
            a.p = s.p, a.out = out[b0 + i], a.ex = s.n[0], a.ey = s.n[1], a.ez = s.n[2], a.sx = s.s[0], a.sy = s.s[1], a.sz = s.s[2];
            a.by_row = fast_div::make((uint32_t)s.n[0]), a.by_rows = fast_div::make((uint32_t)s.n[1]);
            a.block0 = (uint32_t)blocks;
            blocks += ((uint64_t)s.n[0] * s.n[1] * s.n[2] + per - 1) / per;
        }
        if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
        const cudaError_t e = launch_following(sumsq_grad_kernel<T>, (unsigned)blocks, k_sum_threads, 0, stream, args, static_cast<const T*>(g));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
} // namespace

int64_t sumsq_blocks(bool f64, const int32_t (*extents)[3], int n)
{
    uint64_t blocks = 0;
    for (int i = 0; i < n; ++i) blocks += sum_blocks(f64 ? cells<double>::V : cells<float>::V, extents[i]);
    return (int64_t)blocks;
}

cudaError_t launch_sumsq(bool f64, const interior* d, int n, bool packed, double* partials, void* out, cudaStream_t stream)
{
    return f64 ? launch_sumsq_t<double>(d, n, packed, partials, out, stream) : launch_sumsq_t<float>(d, n, packed, partials, out, stream);
}

cudaError_t launch_sumsq_grad(bool f64, const interior* d, void* const* out, int n, int halo, const void* g, cudaStream_t stream)
{
    return f64 ? launch_grad_t<double>(d, out, n, halo, g, stream) : launch_grad_t<float>(d, out, n, halo, g, stream);
}
} // namespace ghexb
