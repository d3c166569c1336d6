// qz_direct.cu -- direct solve of the head's discrete Poisson problem.
//
// The head's equation (potential_head_node.c:99-179: the 7-point Laplacian on the
// (2^L + 1)^3 solve grid with given boundary values) separates: sine transforms along
// the three axes diagonalise it.  From any potential phi the correction e with zero
// boundary that solves (6 e - sum of neighbours) / H^2 = -r, r the residual, makes phi
// the discrete solution to rounding, whatever smoother the multigrid cycles would have
// iterated with:
//   x: r of phi, sine transform   y: transform   z: transform, divide by the
//   eigenvalues, transform        y: transform   x: transform, phi += e
// Five passes that each read and write the grid once (three of FP64 transforms in L2 at
// 128^3) take the place of ten cycles of thirty dependent grid-wide phases; the
// convergence test of the cycles (poisson_error.c:290-347) is applied to the result, and
// cycles go on from it where it does not hold.  Head solve on B200, cycles and direct, us
// (events around every launch included): 16^3 head 330 and 54, 32^3 615 and 56, 64^3
// 1,124 and 63, 128^3 1,956 and 139, 256^3 10,118 and 927, 512^3 98,700 and 9,050.
//
// A sine transform of N - 1 = 2^L - 1 points is a complex Fourier transform of 2 N points
// of the odd extension, two lines at a time as real and imaginary part: a thread holds 8
// points and makes radix-8 steps (the last one radix 2, 4 or 8) in Stockham's order with
// an exchange through shared memory between steps.  Along y and z a block takes eight
// pairs of adjacent x, so that its loads are 128-byte segments; along x, pairs of rows.
#include <math.h>
#include <algorithm>
#include <vector>

#include "qz_internal.cuh"

namespace qz {

struct Cplx {
    double x, y;
};
__device__ __forceinline__ Cplx operator+(Cplx a, Cplx b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ Cplx operator-(Cplx a, Cplx b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ Cplx mul(Cplx a, double2 w)
{
    return {fma(a.x, w.x, -(a.y * w.y)), fma(a.x, w.y, a.y * w.x)};
}
__device__ __forceinline__ Cplx mul_mi(Cplx a) { return {a.y, -a.x}; } // a * (-i)

__device__ __forceinline__ void fft2(Cplx &a, Cplx &b)
{
    const Cplx t = a - b;
    a = a + b;
    b = t;
}

__device__ __forceinline__ void fft4(Cplx &a, Cplx &b, Cplx &c, Cplx &d)
{
    fft2(a, c);
    fft2(b, d);
    d = mul_mi(d);
    fft2(a, b);
    fft2(c, d);
    const Cplx t = b; // outputs in order: a, c, b, d
    b = c;
    c = t;
}

__device__ __forceinline__ void fft8(Cplx (&v)[8])
{
    const double h = 0.70710678118654752440;
#pragma unroll
    for (int q = 0; q < 4; q++)
        fft2(v[q], v[q + 4]);
    const Cplx a = v[5], b = v[7];
    v[5] = {h * (a.x + a.y), h * (a.y - a.x)};
    v[6] = mul_mi(v[6]);
    v[7] = {h * (b.y - b.x), -h * (b.x + b.y)};
    fft4(v[0], v[1], v[2], v[3]);
    fft4(v[4], v[5], v[6], v[7]);
    // v[0..3] hold the even outputs, v[4..7] the odd ones
    const Cplx o[8] = {v[0], v[4], v[1], v[5], v[2], v[6], v[3], v[7]};
#pragma unroll
    for (int q = 0; q < 8; q++)
        v[q] = o[q];
}

// One block's exchange memory: point i of pair p.  ALONGX: a pair's points together, one
// slot in nine left free (steps write with stride 8); else the pairs of a point together.
template <int LG, int P, bool ALONGX> __device__ __forceinline__ int slot(int i, int p)
{
    constexpr int L2 = 2 << LG;
    return ALONGX ? p * (L2 + L2 / 8) + i + (i >> 3) : i * P + p;
}

// Sine transform of P pairs of lines of N - 1 points, N = 2^LG: thread (p, t) holds points
// t + T q, q = 0..3, of pair p and receives outputs t + T q.  Point 0 counts as zero.
template <int LG, int P, bool ALONGX>
__device__ __forceinline__ void sine_pairs(Cplx (&z)[4], int t, int p, Cplx *buf,
                                           const double2 *__restrict__ tw)
{
    constexpr int N = 1 << LG, L2 = 2 * N, T = L2 / 8;
    Cplx v[8];
    if (t == 0)
        z[0] = {0.0, 0.0};
    __syncthreads(); // the buffer's last readers
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        v[q] = z[q];
        buf[slot<LG, P, ALONGX>(t + T * q, p)] = z[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 4; q < 8; q++)
    {
        const int i = L2 - t - T * q; // 1..N; N is the zero of the extension
        const Cplx c = buf[slot<LG, P, ALONGX>(i & (N - 1), p)];
        v[q] = i == N ? Cplx{0.0, 0.0} : Cplx{-c.x, -c.y};
    }
    fft8(v);
    int ns = 8;
#pragma unroll
    for (int s = 1; s < (LG + 3) / 3; s++)
    {
        // exchange: this step's outputs are the next one's inputs
        const int span = ns / 8; // of the step that was made
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 8; q++)
            buf[slot<LG, P, ALONGX>((t / span) * ns + (t % span) + q * span, p)] = v[q];
        __syncthreads();
        constexpr int LAST = (LG + 1) % 3; // bits of the last step when it is not radix 8
        const bool last = LAST != 0 && s == (LG + 3) / 3 - 1;
        if (!last)
        {
#pragma unroll
            for (int q = 0; q < 8; q++)
            {
                v[q] = buf[slot<LG, P, ALONGX>(t + T * q, p)];
                if (q > 0)
                    v[q] = mul(v[q], __ldg(&tw[(t % ns) * q * (L2 / 8 / ns)]));
            }
            fft8(v);
            ns *= 8;
        }
        else if (LAST == 2)
        {
#pragma unroll
            for (int b = 0; b < 2; b++)
            {
                Cplx u[4];
                const int j = t + T * b;
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    u[q] = buf[slot<LG, P, ALONGX>(j + (L2 / 4) * q, p)];
                    if (q > 0)
                        u[q] = mul(u[q], __ldg(&tw[j * q]));
                }
                fft4(u[0], u[1], u[2], u[3]);
                v[b] = u[0];
                v[b + 2] = u[1];
            }
        }
        else
        {
#pragma unroll
            for (int b = 0; b < 4; b++)
            {
                const int j = t + T * b;
                const Cplx a = buf[slot<LG, P, ALONGX>(j, p)];
                v[b] = a + mul(buf[slot<LG, P, ALONGX>(j + L2 / 2, p)], __ldg(&tw[j]));
            }
        }
    }
    // Z = 2 (b - i a) of the lines' transforms a, b
#pragma unroll
    for (int q = 0; q < 4; q++)
        z[q] = {-0.5 * v[q].y, 0.5 * v[q].x};
}

template <int LG> struct DirectShape {
    static constexpr int N = 1 << LG;
    static constexpr int P = LG >= 9 ? 4 : N / 2 < 8 ? N / 2 : 8; // pairs of a block
    static constexpr int T = N / 4;                               // threads of a pair
    static constexpr int THREADS = P * T;
    static constexpr size_t SMEM = sizeof(Cplx) * P * (2 * N + N / 4);
    // 64 registers a thread: the passes wait for their loads, so warps count
    static constexpr int BLOCKS = 1024 / THREADS < 1 ? 1 : 1024 / THREADS > 16 ? 16 : 1024 / THREADS;
};

// x passes: pairs of rows (j = 2 p, 2 p + 1) of plane k.  FORWARD: r of phi into w, else
// phi += the transform of w.
template <int LG, bool FORWARD>
__global__ void __launch_bounds__(DirectShape<LG>::THREADS, DirectShape<LG>::BLOCKS)
    k_sine_x(Grid<double> phi, Grid<double> rho, double *__restrict__ w,
             const double2 *__restrict__ tw, const int *__restrict__ done)
{
    using S = DirectShape<LG>;
    constexpr int N = S::N, T = S::T;
    extern __shared__ __align__(16) unsigned char direct_sm[];
    if (done && __ldcg(done))
        return;
    const int t = threadIdx.x % T, p = threadIdx.x / T;
    const int j = 2 * (blockIdx.x * S::P + p), k = 1 + blockIdx.y;
    double *row = w + (long)k * N * N + (long)j * N;
    const double ooh2 = (double)(N * N);
    Cplx z[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        const int i = t + T * q;
        if constexpr (FORWARD)
        {
            auto r = [&](int jj) {
                if (i == 0 || jj == 0)
                    return 0.0;
                const double *f = phi.p + phi.off + i + jj * phi.sy + k * phi.sz;
                return rho.p[rho.off + i + jj * rho.sy + k * rho.sz] +
                       ooh2 * (6.0 * f[0] - f[1] - f[-1] - f[phi.sy] - f[-phi.sy] - f[phi.sz] -
                               f[-phi.sz]);
            };
            z[q] = {r(j), r(j + 1)};
        }
        else
            z[q] = {row[i], row[N + i]};
    }
    sine_pairs<LG, S::P, true>(z, t, p, reinterpret_cast<Cplx *>(direct_sm), tw);
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        const int i = t + T * q;
        if constexpr (FORWARD)
        {
            row[i] = z[q].x;
            row[N + i] = z[q].y;
        }
        else if (i > 0)
        {
            double *f = phi.p + phi.off + i + j * phi.sy + k * phi.sz;
            if (j > 0)
                f[0] += z[q].x;
            f[phi.sy] += z[q].y;
        }
    }
}

// y passes (stride N, plane blockIdx.y) and the z pass (stride N^2, row blockIdx.y): pairs of
// adjacent x.  The z pass divides by the eigenvalues between its two transforms.
template <int LG, bool SOLVE>
__global__ void __launch_bounds__(DirectShape<LG>::THREADS, DirectShape<LG>::BLOCKS)
    k_sine_yz(double *__restrict__ w, const double2 *__restrict__ tw,
              const double *__restrict__ lam, const int *__restrict__ done)
{
    using S = DirectShape<LG>;
    constexpr int N = S::N, T = S::T, P = S::P;
    extern __shared__ __align__(16) unsigned char direct_sm[];
    if (done && __ldcg(done))
        return;
    Cplx *buf = reinterpret_cast<Cplx *>(direct_sm);
    const int p = threadIdx.x % P, t = threadIdx.x / P;
    const int i = 2 * (blockIdx.x * P + p), b = 1 + blockIdx.y;
    const long stride = SOLVE ? (long)N * N : N;
    double *at = w + i + (SOLVE ? (long)b * N : (long)b * N * N);
    Cplx z[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        // the planes and rows of coordinate 0 are never written: zeros, as in the extension
        if (t + T * q > 0)
        {
            const double2 c = *reinterpret_cast<const double2 *>(at + (t + T * q) * stride);
            z[q] = {c.x, c.y};
        }
        else
            z[q] = {0.0, 0.0};
    }
    sine_pairs<LG, P, false>(z, t, p, buf, tw);
    if constexpr (SOLVE)
    {
        // (2 / N)^3 of the three pairs of transforms, H^2 of the right-hand side
        const double c = 8.0 / ((double)N * N * N) / ((double)N * N);
        const double ly = lam[b], l0 = lam[i], l1 = lam[i + 1];
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const double lz = lam[t + T * q] + ly;
            z[q].x = i > 0 ? z[q].x * (c / (lz + l0)) : 0.0;
            z[q].y = z[q].y * (c / (lz + l1));
        }
        sine_pairs<LG, P, false>(z, t, p, buf, tw);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (t + T * q > 0)
            *reinterpret_cast<double2 *>(at + (t + T * q) * stride) = make_double2(z[q].x, z[q].y);
}

// The convergence test of the head (poisson_error.c:36-133) on the direct solution, without
// the ratio test (a second solve would change nothing), and pot_old <- pot.  Block sums in
// part; the last block to finish adds them in order and decides.
constexpr int DC_THREADS = 256;

__global__ void __launch_bounds__(DC_THREADS)
    k_direct_check(int nc, unsigned D, unsigned inv, const double *__restrict__ pot, double *__restrict__ pot_old,
                   const double *__restrict__ d, double rm, double tol, int method, double nintr,
                   double *__restrict__ part, int *__restrict__ outst, bool again)
{
    if (again && __ldcg(&outst[2]))
        return;
    __shared__ double sh[DC_THREADS / 32];
    __shared__ int sh_last;
    const unsigned D2 = D * D, k = blockIdx.y;
    const double oh2 = (double)nc * nc;
    double acc = 0.0;
    int fail = 0;
    for (unsigned q = blockIdx.x * DC_THREADS + threadIdx.x; q < D2; q += gridDim.x * DC_THREADS)
    {
        const unsigned j = __umulhi(q, inv), i = q - j * D, g = k * D2 + q;
        const double c = pot[g];
        pot_old[g] = c;
        if (i < 2 || j < 2 || k < 2 || i > (unsigned)nc || j > (unsigned)nc || k > (unsigned)nc)
            continue;
        const double r = d[g] + oh2 * (6.0 * c - pot[g + 1] - pot[g - 1] - pot[g + D] - pot[g - D] -
                                       pot[g + D2] - pot[g - D2]);
        if (method == 1)
            fail |= !(fabs(r) / rm < tol);
        else
            acc += r * r;
    }
    if (fail)
        acc = 1.0;
    auto block_sum = [&](double v) {
        for (int o = 16; o > 0; o >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0)
            sh[threadIdx.x >> 5] = v;
        __syncthreads();
        v = 0.0;
        for (int q = 0; q < DC_THREADS / 32; q++)
            v += sh[q];
        __syncthreads();
        return v;
    };
    acc = block_sum(acc);
    if (threadIdx.x == 0)
    {
        part[blockIdx.y * gridDim.x + blockIdx.x] = acc;
        __threadfence();
        sh_last = atomicAdd(&outst[3], 1) == (int)(gridDim.x * gridDim.y) - 1;
    }
    __syncthreads();
    if (!sh_last)
        return;
    __threadfence();
    double t = 0.0;
    for (int b = threadIdx.x; b < (int)(gridDim.x * gridDim.y); b += DC_THREADS)
        t += __ldcg(part + b);
    t = block_sum(t);
    if (threadIdx.x == 0)
    {
        int ok;
        if (method == 1)
            ok = t == 0.0;
        else
        {
            double err = sqrt(t / nintr) / rm;
            if (method == 2)
                err = err / (cbrt(nintr) * cbrt(nintr));
            ok = err < tol;
        }
        outst[0] = 0;
        outst[1] = ok;
        outst[2] = ok;
        outst[3] = 0;
    }
}

// ---- host ---------------------------------------------------------------------------------
// Twiddles exp(-2 pi i q / 2N), q < 2N, then the eigenvalues 2 cos(pi k / N) - 2, k < N.
// Made with the simulation and waited for there: the passes run on streams that no copy on
// the default stream precedes, and a copy from pageable memory returns before it has arrived.
bool direct_tables(qz_sim *s)
{
    const int N = 1 << s->L;
    std::vector<double> h(4 * N + N);
    const long double pi = 3.14159265358979323846264338327950288L;
    for (int q = 0; q < 2 * N; q++)
    {
        h[2 * q] = (double)cosl(pi * q / N);
        h[2 * q + 1] = (double)-sinl(pi * q / N);
    }
    for (int k = 0; k < N; k++)
    {
        const long double v = sinl(pi * k / (2 * N));
        h[4 * N + k] = (double)(-4.0L * v * v);
    }
    double *p = nullptr;
    if (!check_cuda(cudaMalloc((void **)&p, h.size() * sizeof(double)), "sine tables"))
        return false;
    s->direct_tab = p;
    return check_cuda(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(double),
                                      cudaMemcpyHostToDevice, s->stream), "sine tables") &&
           check_cuda(cudaStreamSynchronize(s->stream), "sine tables");
}

template <int LG>
static bool direct_passes(qz_sim *s, Grid<double> phi, Grid<double> rho, const int *done)
{
    using S = DirectShape<LG>;
    constexpr int N = S::N;
    static PerDevice<bool> ready;
    const bool fits = ready.get(s->device, [] {
        const void *f[] = {(const void *)k_sine_x<LG, true>, (const void *)k_sine_x<LG, false>,
                           (const void *)k_sine_yz<LG, true>, (const void *)k_sine_yz<LG, false>};
        bool ok = true;
        for (const void *k : f)
            ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)S::SMEM) == cudaSuccess;
        return ok;
    });
    if (!fits)
    {
        set_error("direct solve: the kernels' shared memory cannot be had");
        return false;
    }
    double *w = s->fine_alt_buf;
    const double2 *tw = reinterpret_cast<const double2 *>(s->direct_tab);
    const double *lam = s->direct_tab + 4 * N;
    const dim3 g(N / 2 / S::P, N - 1), b(S::THREADS);
    const double pts = (double)(N - 1) * (N - 1) * (N - 1);
    launch_shm(s, QZ_PROF_SMOOTH, 24.0 * pts, S::SMEM, k_sine_x<LG, true>, g, b, phi, rho, w, tw, done);
    launch_shm(s, QZ_PROF_SMOOTH, 16.0 * pts, S::SMEM, k_sine_yz<LG, false>, g, b, w, tw, lam, done);
    launch_shm(s, QZ_PROF_SMOOTH, 16.0 * pts, S::SMEM, k_sine_yz<LG, true>, g, b, w, tw, lam, done);
    launch_shm(s, QZ_PROF_SMOOTH, 16.0 * pts, S::SMEM, k_sine_yz<LG, false>, g, b, w, tw, lam, done);
    launch_shm(s, QZ_PROF_SMOOTH, 24.0 * pts, S::SMEM, k_sine_x<LG, false>, g, b, phi, rho, w, tw, done);
    return true;
}

// Corrects phi (a head grid) to the solution with right-hand side rho and phi's boundary
// values, unless *done (when given) is set; the head's red-black partner grid is the
// transforms' work space.
static int direct_correct_unless(qz_sim *s, double *phi, double *rho, const int *done)
{
    const Grid<double> p = head_view(s, phi), r = head_view(s, rho);
    bool ok;
    switch (s->L)
    {
    case 2: ok = direct_passes<2>(s, p, r, done); break;
    case 3: ok = direct_passes<3>(s, p, r, done); break;
    case 4: ok = direct_passes<4>(s, p, r, done); break;
    case 5: ok = direct_passes<5>(s, p, r, done); break;
    case 6: ok = direct_passes<6>(s, p, r, done); break;
    case 7: ok = direct_passes<7>(s, p, r, done); break;
    case 8: ok = direct_passes<8>(s, p, r, done); break;
    default: ok = direct_passes<9>(s, p, r, done); break;
    }
    return ok && check_cuda(cudaGetLastError(), "direct solve") ? QZ_SUCCESS : QZ_FAILURE;
}

int direct_correct(qz_sim *s, double *phi, double *rho)
{
    return direct_correct_unless(s, phi, rho, nullptr);
}

// again: only where the test did not hold so far
static int direct_check(qz_sim *s, bool again)
{
    const qz_config &c = s->cfg;
    const int nc = 1 << s->L;
    const double H = 1.0 / nc;
    const double rm = 4.0 * c.G * 3.14159265358979323846 * s->head_mass / ((double)nc * nc * nc * H * H * H);
    const double m = nc - 1;
    const unsigned D = (unsigned)s->D;
    // a plane of points a row of blocks; the partials' buffer holds 2 x QZ_CG_PART_MAX
    const unsigned bx = std::max(1u, std::min((D * D + 4 * DC_THREADS - 1) / (4 * DC_THREADS),
                                              2 * QZ_CG_PART_MAX / D));
    launch(s, QZ_PROF_CHECK, 24.0 * s->gpts, k_direct_check, dim3(bx, D), dim3(DC_THREADS), nc, D,
           div_magic(D), s->pot, s->pot_old, s->d, rm, c.tol, c.check_method, m * m * m, s->mg_part,
           s->outst, again);
    return check_cuda(cudaGetLastError(), "direct solve test") ? QZ_SUCCESS : QZ_FAILURE;
}

// The head's direct solve and its test, queued; the outcome is outst[2].  Heads of 256^3 and
// more are corrected a second time where the first result does not pass: rounding in the
// transforms of a start far from the solution (a new simulation's) leaves a residual
// that grows with N^2, of the order of the default tolerance there.
int direct_head(qz_sim *s)
{
    const int *done = s->outst + 2;
    if (direct_correct(s, s->pot, s->d) || direct_check(s, false))
        return QZ_FAILURE;
    return s->L >= 8 && (direct_correct_unless(s, s->pot, s->d, done) || direct_check(s, true))
               ? QZ_FAILURE
               : QZ_SUCCESS;
}

} // namespace qz
