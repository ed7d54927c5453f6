// uvgrid.cu -- the DFT to the uv points and its adjoint through a regular grid
// of the uv plane.
//
// The image covers N pixels a side, so its transform E(a, b) = sum_yx I[y][x]
// e^{2 pi i (a x' - b y')} (a, b in cycles per pixel, x' = x - (N-1)/2) is a
// band-limited function of (a, b): it is known everywhere from its values on a
// grid of spacing 1/M, M = 2 N, and a Kaiser-Bessel window of UG_W = 8 grid
// points a side interpolates it (a nonuniform Fourier transform of type 2;
// Dutt and Rokhlin 1993, Fessler and Sutton 2003). Dividing the image by the
// window's transform phi is folded into the grid's own twiddles. A data set
// has many more uv points than grid points inside its uv coverage (1024^2
// workload: 194,560 uv points, 60 x 119 grid points), so two small
// contractions onto the grid and 64 window products per uv point take the
// place of the N^2 nuv contraction:
//   forward   T[y][jx] = sum_x I[y][x] e^{2 pi i jx x'/M} / phi(x')          (tcgen05, or k_ug_x)
//             G[jy][jx] = sum_y T[y][jx] e^{-2 pi i jy y'/M} / phi(y')       (k_ug_rows)
//             V_k = sum over 8 x 8 grid points of G, window weights          (k_ug_interp)
//   adjoint   C[jy][jx] = sum_k c_k at the 8 x 8 grid points around k        (k_ug_spread, k_ug_gather)
//             S[y][jx] = sum_jy C[jy][jx] e^{-2 pi i jy y'/M} / phi(y')      (k_ug_cols)
//             g[y][x] = Re sum_jx S[y][jx] e^{2 pi i jx x'/M} / phi(x')      (k_ug_grad, with the gradient assembly)
// Conjugating uv points with a < 0 leaves jx >= -3, half of the plane.
//
// Accuracy. The window's own error is at most 4e-8 of the flux (FP64 model over
// the workloads' uv points and flat, random and compact images). V measures
// 7e-8 to 9e-8 relative on FP32 contexts (the direct FP32 sums 1e-7 to 4e-7),
// the gradient 3e-8 to 2e-7 (as the direct sums) from 96 pixels up; on the
// tensor paths the gradient measures 2e-6 to 4e-6 where the direct
// contractions measure 2e-6 to 2e-5 (their accumulation truncates). The
// longest FP32 chains are the x contraction's partial sums: on the tensor cores 128
// products up to 1,024 pixels and N / 8 above, on the CUDA cores from 32 folded pixels (64
// products) to all of them (N products) where the blocks fill the device without
// partial sums, as with eight trials of 1024^2; then 64 products per uv point, 32 points of a
// run and 16 columns of the gradient, and FP64 between those stages. The objectives of the trials so
// summed are within 2e-10 (FP32, 1024^2 and 1,500 uv points) and 3e-6 (tensor modes) of FP64 sums.
// Measured on a B200, one objective with its gradient (events around the
// stages, launches included): 1024^2 and 194,560 uv points 3,240 -> 147 us on the tensor
// path, 57,000 -> 157 us in FP32; 256^2 and 21,120 uv points 120 -> 80 us and 483 -> 78 us.
//
// Everything is summed in a fixed order: uv points are sorted by their grid
// cell, and the adjoint adds per-cell patches, so there are no atomics.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "gpair_internal.cuh"
#include "group.cuh"
#include "reduce.cuh"
#include "uvgrid.cuh"

#define UG_PI 3.14159265358979323846
#define UGX_T 32  // tile of the x contraction on the CUDA cores (k_ug_x): image rows, columns, folded pixels
#define UG_RPMAS ((3.14159265358979323 / 180.0) / 3600000.0)  // radians per milliarcsecond, as k_gen_twiddles

// ------------------------------------------------------------------ plan

// I0 by its series (x <= pi UG_W)
__device__ __forceinline__ double ug_bessel_i0(double x)
{
    const double t = 0.25 * x * x;
    double term = 1.0, sum = 1.0;
    for (int n = 1; n < 200; n++) {
        term *= t / ((double)n * (double)n);
        sum += term;
        if (term < 1e-17 * sum) break;
    }
    return sum;
}

// Window weights and centre phase of every sorted uv point, from (u, v) in FP64
__global__ void k_ug_points(const float2 *__restrict__ uvc, const int *__restrict__ src, const int *__restrict__ base,
                            int nuv, double pix, int N, double M, int jxf, int J, int nbx, double beta,
                            float *__restrict__ wts, float2 *__restrict__ phase)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nuv) return;
    const int k = src[p] & 0x7fffffff;
    const bool flip = src[p] < 0;
    const float2 uv = uvc[k];
    double a = UG_RPMAS * pix * (double)uv.x, b = UG_RPMAS * pix * (double)uv.y;
    a -= rint(a);
    b -= rint(b);
    if (flip) {
        a = -a;
        b = -b;
    }
    const double gx = a * M - (double)(base[p] % nbx + jxf), gy = b * M - (double)(base[p] / nbx - J);
    const double inv0 = 1.0 / ug_bessel_i0(beta);
    for (int i = 0; i < UG_W; i++) {
        const double tx = (gx - i) * (2.0 / UG_W), ty = (gy - i) * (2.0 / UG_W);
        wts[(size_t)p * (2 * UG_W) + i] = (float)(ug_bessel_i0(beta * sqrt(fmax(0.0, 1.0 - tx * tx))) * inv0);
        wts[(size_t)p * (2 * UG_W) + UG_W + i] = (float)(ug_bessel_i0(beta * sqrt(fmax(0.0, 1.0 - ty * ty))) * inv0);
    }
    double t = (a - b) * (0.5 * (double)(N - 1));
    t -= rint(t);
    double sn, cn;
    sincospi(2.0 * t, &sn, &cn);
    phase[p] = make_float2((float)cn, (float)sn);
}

// Grid twiddles over the folded image coordinate h (pixels h and N-1-h, at
// -+x'_h, x'_h = (N-1)/2 - h): (cos, sin)(2 pi j x'_h / M) / phi(x'_h), FP64 phase.
// ftab[j][h] for the columns j = jxf .. jxf + nbx - 1, ctab[h][j] for the rows j = 0 .. J
__global__ void k_ug_tables(const double *__restrict__ invphi, int N, int H, double M, int jxf, int nbx, int J,
                            float2 *__restrict__ ftab, float2 *__restrict__ ctab)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nf = (long long)nbx * H;
    int h, j;
    if (i < nf) {
        j = (int)(i / H) + jxf;
        h = (int)(i % H);
    } else {
        i -= nf;
        if (i >= (long long)H * (J + 1)) return;
        h = (int)(i / (J + 1));
        j = (int)(i % (J + 1));
    }
    double t = (double)j * (0.5 * (double)(N - 1) - (double)h) / M;
    t -= rint(t);
    double sn, cn;
    sincospi(2.0 * t, &sn, &cn);
    const double f = invphi[h];
    const float2 v = make_float2((float)(cn * f), (float)(sn * f));
    if ((long long)blockIdx.x * blockDim.x + threadIdx.x < nf) ftab[i] = v;
    else ctab[i] = v;
}

// Whether the grid's contractions are small beside the direct ones (UG_GRID_RATIO), with one partial sum
// of the gradient's dot products per 64 x 64 tile
static bool ug_small(int N, int nuv, int nbx, int J)
{
    const double direct = 2.0 * (double)N * N * (double)nuv;
    const double grid = (double)nbx * (2.0 * N + 2.0 * J + 1.0) * (double)N;
    return (long long)gp_cdiv(N, 64) * gp_cdiv((N + 1) / 2, 64) <= GP_MAX_PARTIALS && UG_GRID_RATIO * grid <= direct;
}

// The precision mode's least direct work 2 N^2 nuv for the grid (uvgrid.cuh)
static double ug_min_work(int precision)
{
    if (precision == GPAIR_PREC_FP32) return UG_MIN_WORK_FP32;
    return precision == GPAIR_PREC_SPLIT16F8 ? UG_MIN_WORK_F8 : UG_MIN_WORK_TC;
}

// The mode's direct sums 2 N nuv an image row against the grid's y contractions nbx J (uvgrid.cuh); 0: not asked
static double ug_wide_ratio(int precision)
{
    if (precision == GPAIR_PREC_FP32 || precision == GPAIR_PREC_TF32X3) return 0.0;
    return precision == GPAIR_PREC_SPLIT16 ? UG_WIDE_RATIO_TC : UG_WIDE_RATIO_F8;
}

bool gp_ug_takes(const gpair_ctx *c, int precision)
{
    if (!c->ug_able) return false;
    const double row = 2.0 * (double)c->N * (double)c->nuv;
    return row * (double)c->N >= ug_min_work(precision) &&
           row >= ug_wide_ratio(precision) * (double)c->ug_nbx * (double)c->ug_J;
}

// The points' first window points and the extent of the grid, columns ug_jxf .. ug_jxf + ug_nbx - 1 and rows -ug_J .. ug_J;
// whether some precision mode may take it (c->ug_able; not with a coordinate that is not finite). The sizes of the
// context are set.
int gp_ug_scan(gpair_ctx *c, const gpair_uv *uv)
{
    const int N = c->N, nuv = c->nuv;
    if (!uv || N < UG_MIN_WIDTH || 2.0 * (double)N * N * (double)nuv < UG_MIN_WORK_FP32) return GPAIR_OK;
    const double M = UG_OVERSAMPLING * N, pix = (double)c->pix;
    int2 *first = (int2 *)malloc(sizeof(int2) * (size_t)nuv);
    if (!first) return GPAIR_ERR_ALLOC;
    int xmin = 1 << 30, xmax = -(1 << 30), ymax = 0;
    bool ok = true;
    for (int k = 0; k < nuv && ok; k++) {
        double a = UG_RPMAS * pix * (double)uv[k].u, b = UG_RPMAS * pix * (double)uv[k].v;
        ok = isfinite(a) && isfinite(b);
        if (!ok) break;
        a -= rint(a);
        b -= rint(b);
        const bool flip = a < 0.0;
        if (flip) {
            a = -a;
            b = -b;
        }
        const int jx = (int)floor(a * M) - (UG_W / 2 - 1), jy = (int)floor(b * M) - (UG_W / 2 - 1);
        first[k] = make_int2(jx, 2 * jy + (flip ? 1 : 0));
        if (jx < xmin) xmin = jx;
        if (jx > xmax) xmax = jx;
        const int lo = -jy, hi = jy + UG_W - 1;
        if (lo > ymax) ymax = lo;
        if (hi > ymax) ymax = hi;
    }
    const int nbx = xmax - xmin + UG_W;
    if (!ok || !ug_small(N, nuv, nbx, ymax)) {
        free(first);
        return GPAIR_OK;
    }
    c->ug_first = first;
    c->ug_jxf = xmin;
    c->ug_nbx = nbx;
    c->ug_J = ymax;
    c->ug_able = 1;
    return GPAIR_OK;
}

static void ug_free_plan(gpair_ctx *c)
{
    UgState *g = (UgState *)c->ug_plan;
    if (g) {
        void *bufs[] = {g->mem, g->t_mem[0], g->t_mem[1], g->Tb[0], g->Tb[1], g->gridb};
        for (void *b : bufs)
            if (b) cudaFree(b);
        free(g);
    }
    c->ug_plan = nullptr;
    c->ug = nullptr;
}

void gp_ug_free(gpair_ctx *c)
{
    ug_free_plan(c);
    free(c->ug_first);
    c->ug_first = nullptr;
    c->ug_able = 0;
}

// 0: the CUDA cores' x contraction, 1: the tensor cores'
static int ug_class(const gpair_ctx *c) { return c->precision != GPAIR_PREC_FP32; }

// Partial sums of the x contraction of `images` images on the CUDA cores, and folded pixels in each: slices
// of whole tiles until the blocks fill two waves of 148 SMs
static int ug_x_splits(const UgState *g, int images, int *hper)
{
    const int blocks = gp_cdiv(g->N, UGX_T) * gp_cdiv(g->nbx, UGX_T) * images;
    int s = 1;
    while (s < UG_MAX_SPLITS && 2 * s * UGX_T <= g->H && blocks * s < 2 * 148) s *= 2;
    *hper = gp_cdiv(gp_cdiv(g->H, s), UGX_T) * UGX_T;
    return gp_cdiv(g->H, *hper);
}

// floats of the x contraction's sums of one image or the batch's, in the context's mode (the tensor path's
// operand stack has at least as many rows per image as the CUDA cores, N)
static size_t ug_t_floats(const gpair_ctx *c, const UgState *g, int images)
{
    int hper;
    if (!ug_class(c)) return (size_t)ug_x_splits(g, images, &hper) * images * g->N * g->ldT;
    return (size_t)ug_tc_splits(g->N) * (images > 1 ? (size_t)images * gp_tc_stack_rows(g->N) : (size_t)g->N) * g->ldT;
}

// Builds the plan of the problem that gp_ug_scan looked over, when a mode first takes it. A new context is in FP32, so a
// program that goes on to a mode with direct sums has built a plan that it does not use. An allocation costs 0.3 to
// 0.4 ms, so the plan is one, and so are the direct sums' buffers: such a context's preparation takes what it took without the
// grid (set_problem and set_precision, 256^2, split-f16/E4M3: 8,000 uv points 4.2 to 4.4 ms without the grid, 4.8 to 5.0 with an
// allocation per array, 4.3 now; 21,120 5.4, 6.0 to 6.3, 5.0 to 5.4). A context whose mode is set before the problem builds its mode's alone.
static int ug_plan(gpair_ctx *c)
{
    const int N = c->N, nuv = c->nuv, jxf = c->ug_jxf, nbx = c->ug_nbx, J = c->ug_J;
    const double M = UG_OVERSAMPLING * N;
    const int cells = nbx * (2 * J + 1);
    // counting sort by cell (stable), then runs of at most 32 points of one cell
    std::vector<int> off((size_t)cells + 1, 0), src(nuv), base(nuv), cst((size_t)cells + 1, 0);
    std::vector<int2> chunk;
    const int2 *first = c->ug_first;
    auto cell_of = [&](int k) { return ((first[k].y >> 1) + J) * nbx + (first[k].x - jxf); };
    for (int k = 0; k < nuv; k++) off[(size_t)cell_of(k) + 1]++;
    for (int q = 0; q < cells; q++) {
        cst[q] = (int)chunk.size();
        for (int s = 0; s < off[q + 1]; s += 32) {
            const int left = off[q + 1] - s;
            chunk.push_back(make_int2(off[q] + s, left < 32 ? left : 32));
        }
        off[q + 1] += off[q];
    }
    cst[cells] = (int)chunk.size();
    std::vector<int> pos(off.begin(), off.end() - 1);
    for (int k = 0; k < nuv; k++) {
        const int cell = cell_of(k);
        const int p = pos[cell]++;
        src[p] = k | ((first[k].y & 1) ? (int)0x80000000 : 0);
        base[p] = cell;
    }
    // 1 / phi over the folded coordinate: phi(x') = w sinh(z) / z / I0(beta), z^2 = beta^2 - (pi w x'/M)^2
    const int H = (N + 1) / 2;
    const double beta = UG_PI * UG_W * (1.0 - (double)N / (2.0 * M));
    double i0 = 1.0, term = 1.0;
    for (int n = 1; n < 200; n++) {
        term *= 0.25 * beta * beta / ((double)n * n);
        i0 += term;
    }
    std::vector<double> invphi(H);
    for (int h = 0; h < H; h++) {
        const double xi = UG_PI * UG_W * (0.5 * (N - 1) - h) / M;
        const double z = sqrt(beta * beta - xi * xi);
        invphi[h] = i0 * z / (UG_W * sinh(z));
    }
    UgState *g = (UgState *)calloc(1, sizeof(UgState));
    if (!g) return GPAIR_ERR_ALLOC;
    c->ug_plan = g;
    g->N = N;
    g->H = H;
    g->jxf = jxf;
    g->nbx = nbx;
    g->J = J;
    g->cells = cells;
    g->nchunk = (int)chunk.size();
    g->ldT = (2 * nbx + 3) & ~3;
    cudaStream_t st = c->stream;
    // one allocation for all, the arrays from the host first, in one copy
    const struct {
        void **p;
        size_t bytes;
        const void *host;
    } arrays[] = {{(void **)&g->src, sizeof(int) * (size_t)nuv, src.data()},
                  {(void **)&g->base, sizeof(int) * (size_t)nuv, base.data()},
                  {(void **)&g->chunk, sizeof(int2) * (size_t)g->nchunk, chunk.data()},
                  {(void **)&g->cst, sizeof(int) * ((size_t)cells + 1), cst.data()},
                  {(void **)&g->invphi, sizeof(double) * (size_t)H, invphi.data()},
                  {(void **)&g->wts, sizeof(float) * 2 * UG_W * (size_t)nuv, nullptr},
                  {(void **)&g->phase, sizeof(float2) * (size_t)nuv, nullptr},
                  {(void **)&g->ftab, sizeof(float2) * (size_t)nbx * H, nullptr},
                  {(void **)&g->ctab, sizeof(float2) * (size_t)H * (J + 1), nullptr},
                  {(void **)&g->grid, sizeof(float2) * (size_t)cells, nullptr},
                  {(void **)&g->patch, sizeof(float2) * UG_W * UG_W * (size_t)g->nchunk, nullptr},
                  {(void **)&g->cgrid, sizeof(float2) * (size_t)cells, nullptr},
                  {(void **)&g->S, sizeof(float2) * (size_t)N * nbx, nullptr},
                  {(void **)&g->T[ug_class(c)], sizeof(float) * ug_t_floats(c, g, 1), nullptr}};
    auto padded = [](size_t n) { return (n + 255) & ~(size_t)255; };
    size_t total = 0, given = 0;
    for (const auto &x : arrays) {
        total += padded(x.bytes);
        if (x.host) given = total;
    }
    GP_CUDA(c, cudaMalloc(&g->mem, total));
    std::vector<unsigned char> host(given);
    size_t at = 0;
    for (const auto &x : arrays) {
        *x.p = (unsigned char *)g->mem + at;
        if (x.host) memcpy(&host[at], x.host, x.bytes);
        at += padded(x.bytes);
    }
    GP_CUDA(c, cudaMemcpyAsync(g->mem, host.data(), given, cudaMemcpyHostToDevice, st));
    k_ug_points<<<gp_cdiv(nuv, 128), 128, 0, st>>>(c->uvc, g->src, g->base, nuv, (double)c->pix, N, M, jxf, J, nbx,
                                                   beta, g->wts, g->phase);
    GP_LAUNCH_CHECK(c);
    const long long nt = (long long)nbx * H + (long long)H * (J + 1);
    k_ug_tables<<<gp_cdiv(nt, 256), 256, 0, st>>>(g->invphi, N, H, M, jxf, nbx, J, g->ftab, g->ctab);
    GP_LAUNCH_CHECK(c);
    GP_CUDA(c, cudaStreamSynchronize(st));  // the host's arrays end here
    return GPAIR_OK;
}

int gp_ug_choose(gpair_ctx *c)
{
    c->ug = nullptr;
    if (!gp_ug_takes(c, c->precision)) return GPAIR_OK;
    if (!c->ug_plan) {
        const int rc = ug_plan(c);
        if (rc) {
            ug_free_plan(c);  // the whole plan or none
            return rc;
        }
        free(c->ug_first);
        c->ug_first = nullptr;
    }
    UgState *g = (UgState *)c->ug_plan;
    const int cls = ug_class(c);
    if (!g->T[cls]) {  // the plan was built by a mode on the other cores
        GP_CUDA(c, cudaMalloc(&g->t_mem[cls], sizeof(float) * ug_t_floats(c, g, 1)));
        g->T[cls] = (float *)g->t_mem[cls];
    }
    c->ug = c->ug_plan;
    return GPAIR_OK;
}

// ----------------------------------------- x contraction on the CUDA cores
//
// T[y][2j + c] of one image (FP32 contexts), folded over x' -> -x': the cosine
// row meets I[N-1-h] + I[h], the sine row I[N-1-h] - I[h]. A block makes 32
// image rows x 32 columns over a slice of h; the slices are partial sums that
// k_ug_rows adds.
struct UgXArgs {
    const float *img;  // image b at img + b npix
    const float2 *ftab;
    float *T;  // [split][image row][ldT]
    int N, H, nbx, ldT, splits, hper, images;
    const int *gate;
};

__global__ void __launch_bounds__(256) k_ug_x(const UgXArgs a)
{
    gp_pdl_enter();
    if (a.gate && !*a.gate) return;
    __shared__ float2 Is[UGX_T][UGX_T + 1];  // [h][y] (even, odd)
    __shared__ float2 Fs[UGX_T][UGX_T + 1];  // [h][j]
    const int N = a.N, H = a.H;
    const int y0 = blockIdx.x * UGX_T, j0 = blockIdx.y * UGX_T;
    const int split = blockIdx.z % a.splits, image = blockIdx.z / a.splits;
    const float *img = a.img + (size_t)image * N * N;
    const int hb = split * a.hper, he = min(H, hb + a.hper);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2 acc[2][2];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) acc[i][j] = make_float2(0.f, 0.f);
    for (int h0 = hb; h0 < he; h0 += UGX_T) {
        const int h = h0 + lane;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int yy = warp + 8 * r, y = y0 + yy, j = j0 + yy;
            float2 v = make_float2(0.f, 0.f), f = make_float2(0.f, 0.f);
            if (h < he && y < N) {
                const float p = __ldg(&img[(size_t)y * N + (N - 1 - h)]);
                const float m = (N - 1 - h) != h ? __ldg(&img[(size_t)y * N + h]) : 0.f;
                v = make_float2(p + m, p - m);
            }
            if (h < he && j < a.nbx) f = __ldg(&a.ftab[(size_t)j * H + h]);
            Is[lane][yy] = v;
            Fs[lane][yy] = f;
        }
        __syncthreads();
#pragma unroll 8
        for (int q = 0; q < UGX_T; q++) {
            const float2 i0 = Is[q][ty], i1 = Is[q][ty + 16], f0 = Fs[q][tx], f1 = Fs[q][tx + 16];
            acc[0][0].x = fmaf(i0.x, f0.x, acc[0][0].x);
            acc[0][0].y = fmaf(i0.y, f0.y, acc[0][0].y);
            acc[0][1].x = fmaf(i0.x, f1.x, acc[0][1].x);
            acc[0][1].y = fmaf(i0.y, f1.y, acc[0][1].y);
            acc[1][0].x = fmaf(i1.x, f0.x, acc[1][0].x);
            acc[1][0].y = fmaf(i1.y, f0.y, acc[1][0].y);
            acc[1][1].x = fmaf(i1.x, f1.x, acc[1][1].x);
            acc[1][1].y = fmaf(i1.y, f1.y, acc[1][1].y);
        }
        __syncthreads();
    }
    float *T = a.T + ((size_t)split * a.images + image) * N * a.ldT;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int y = y0 + ty + 16 * i, jj = j0 + tx + 16 * j;
            if (y < N && jj < a.nbx) *reinterpret_cast<float2 *>(&T[(size_t)y * a.ldT + 2 * jj]) = acc[i][j];
        }
}

// four doubles in 16-byte halves of shared memory
struct __align__(16) double4_a16 {
    double x, y, z, w;
};

// ------------------------------------------------------ y contraction
//
// G[+-j][jx] of C columns jx and 32 rows j per block: lane = j, the W warps take
// every W-th folded image row h (pixels h and N-1-h), whose folded T values (sum and
// difference of the two rows, partial sums added, row scales removed) wait in
// shared memory, in FP64: converted where they are used they would be converted
// by every warp, at a quarter of the FP64 rate. cos and sin serve +j and -j. Bound by
// latency: T's partial sums (all loads of a row in flight), then the row twiddles
// (H x 32 x 8 B per block). 1024^2, 60 x 119 grid points: 14.2 us (19.6 with
// conversions, loads one by one and 8 warps), 8 trials 30.4 (49).
template <int C> struct UgRowsGeo {
    static constexpr int W = C == 1 ? 16 : 8;          // warps
    static constexpr int HB = C == 1 ? 512 : 256;      // folded rows staged at once
    static constexpr int BYTES = HB * C * 32 > W * 32 * C * 32 ? HB * C * 32 : W * 32 * C * 32;
};
struct UgRowsArgs {
    const float *T;  // image b: rows b lrows .. b lrows + N - 1
    const float *rsc;  // power-of-two factor of every row (tensor path), or null
    const float2 *ctab;
    float2 *grid;  // cell e at grid[e], of trial b of a batch at grid[GP_NTR e + b]
    int N, H, gw, J, ldT, cells, splits, lrows;  // gw: grid columns
    size_t split_stride;
    const int *gate;
    GP_VGRID_FIELDS;
};

template <int C>
__device__ __forceinline__ void ug_rows_body(const UgRowsArgs &A, const GpVGrid &vg)
{
    using G = UgRowsGeo<C>;
    __shared__ __align__(16) unsigned char raw[G::BYTES];
    double4_a16(*Ts)[C] = reinterpret_cast<double4_a16(*)[C]>(raw);          // [h][column]: sum, difference
    double(*red)[32][C][4] = reinterpret_cast<double(*)[32][C][4]>(raw);     // [warp][j], once Ts has been used
    if (A.gate && !*A.gate) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ctiles = (A.gw + C - 1) / C;
    const int c0 = (vg.bx % ctiles) * C, j = (vg.bx / ctiles) * 32 + lane;
    const int image = vg.by;
    const int N = A.N, H = A.H, J1 = A.J + 1, splits = A.splits;
    const size_t row0 = (size_t)image * A.lrows;
    double acc[C][4];
#pragma unroll
    for (int q = 0; q < C; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[q][i] = 0.0;
    for (int hb = 0; hb < H; hb += G::HB) {
        const int nh = min(G::HB, H - hb);
        for (int e = threadIdx.x; e < nh * C; e += 32 * G::W) {
            const int h = hb + e / C, col = c0 + e % C;
            float2 p = make_float2(0.f, 0.f), m = make_float2(0.f, 0.f);
            if (col < A.gw) {
                const size_t rp = row0 + (N - 1 - h), rm = row0 + h;
                const bool two = rp != rm;
                float2 a[UG_MAX_SPLITS], b[UG_MAX_SPLITS];
#pragma unroll
                for (int s = 0; s < UG_MAX_SPLITS; s++) {
                    if (s >= splits) break;
                    const float *T = A.T + s * A.split_stride + 2 * col;
                    a[s] = __ldg(reinterpret_cast<const float2 *>(T + rp * A.ldT));
                    b[s] = __ldg(reinterpret_cast<const float2 *>(T + rm * A.ldT));
                }
                const float sp = A.rsc ? __ldg(&A.rsc[rp]) : 1.f, sm = A.rsc ? __ldg(&A.rsc[rm]) : 1.f;
#pragma unroll
                for (int s = 0; s < UG_MAX_SPLITS; s++) {
                    if (s >= splits) break;
                    p.x += a[s].x;
                    p.y += a[s].y;
                    m.x += b[s].x;
                    m.y += b[s].y;
                }
                p.x *= sp;
                p.y *= sp;
                m.x *= sm;
                m.y *= sm;
                if (!two) m = make_float2(0.f, 0.f);  // the middle row
            }
            double4_a16 t;
            t.x = p.x + m.x;
            t.y = p.y + m.y;
            t.z = p.x - m.x;
            t.w = p.y - m.y;
            Ts[e / C][e % C] = t;
        }
        __syncthreads();
        if (j < J1) {
            const float2 *ct = A.ctab + (size_t)hb * J1 + j;
#pragma unroll 8
            for (int h = warp; h < nh; h += G::W) {
                const float2 wf = __ldg(&ct[(size_t)h * J1]);
                const double wc = wf.x, ws = wf.y;
#pragma unroll
                for (int q = 0; q < C; q++) {
                    const double4_a16 t = Ts[h][q];
                    acc[q][0] = fma(wc, t.x, acc[q][0]);
                    acc[q][1] = fma(wc, t.y, acc[q][1]);
                    acc[q][2] = fma(ws, t.z, acc[q][2]);
                    acc[q][3] = fma(ws, t.w, acc[q][3]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < C; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) red[warp][lane][q][i] = acc[q][i];
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * C; e += 32 * G::W) {
        const int l = e / C, q = e % C, jj = (vg.bx / ctiles) * 32 + l, col = c0 + q;
        if (jj >= J1 || col >= A.gw) continue;
        double t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            t[i] = red[0][l][q][i];
#pragma unroll
            for (int w = 1; w < G::W; w++) t[i] += red[w][l][q][i];
        }
        // sum T e^{-+i theta} = (even . cos) -+ i (odd . sin)
        const int st = vg.nby > 1 ? GP_NTR : 1;
        float2 *g = A.grid + image + (size_t)col * st;
        g[(size_t)(A.J + jj) * A.gw * st] = make_float2((float)(t[0] + t[3]), (float)(t[1] - t[2]));
        g[(size_t)(A.J - jj) * A.gw * st] = make_float2((float)(t[0] - t[3]), (float)(t[1] + t[2]));
    }
}

template <int C>
__global__ void __launch_bounds__(32 * UgRowsGeo<C>::W) k_ug_rows(const UgRowsArgs a)
{
    gp_pdl_enter();
    ug_rows_body<C>(a, gp_vgrid_hw());
}

template <int C> struct UgRowsOp {
    using Args = UgRowsArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_rows_body<C>(a, v); }
};

// ------------------------------------------------------- interpolation
//
// V_k / F of one sorted uv point per thread. The points of a warp share a grid
// cell or lie in neighbouring ones, so the 64 grid loads are served by one or two
// sectors each; the window weights stream (64 B per point).
#define UGI_THREADS 128
struct UgInterpArgs {
    const float2 *grid;
    const int *src, *base;
    const float *wts;
    const float2 *phase;
    const DevScalars *sc;
    double2 *out;  // [nuv], or [nuv][GP_NTR] (trials)
    int nuv, gw, nchunk;
    const int2 *chunk;
    const int *gate;
    GP_VGRID_FIELDS;
};

__device__ __forceinline__ double2 ug_vis_out(float re, float im, float2 ph, bool conj, double invF)
{
    const double vr = (double)re * ph.x - (double)im * ph.y;
    const double vi = (double)re * ph.y + (double)im * ph.x;
    return make_double2(vr * invF, (conj ? -vi : vi) * invF);
}

__device__ __forceinline__ void ug_interp_body(const UgInterpArgs &A, const GpVGrid &vg)
{
    if (A.gate && !*A.gate) return;
    const int p = vg.bx * blockDim.x + threadIdx.x;
    if (p >= A.nuv) return;
    const float4 *w4 = reinterpret_cast<const float4 *>(A.wts + (size_t)p * (2 * UG_W));
    float w[2 * UG_W];
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<float4 *>(&w[4 * i]) = __ldg(&w4[i]);
    const float2 *g = A.grid + __ldg(&A.base[p]);
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int i = 0; i < UG_W; i++) {
        float rr = 0.f, ri = 0.f;
#pragma unroll
        for (int j = 0; j < UG_W; j++) {
            const float2 v = __ldg(&g[j]);
            rr = fmaf(w[j], v.x, rr);
            ri = fmaf(w[j], v.y, ri);
        }
        g += A.gw;
        re = fmaf(w[UG_W + i], rr, re);
        im = fmaf(w[UG_W + i], ri, im);
    }
    const int s = __ldg(&A.src[p]);
    A.out[s & 0x7fffffff] = ug_vis_out(re, im, __ldg(&A.phase[p]), s < 0, A.sc->invflux);
}

// The trials of a batch: one warp per run of at most 32 uv points of one grid cell
// (the adjoint's runs), lane = (group of 8 of its points, trial). A lane reads each
// of the cell's 64 grid values once for its 8 points (the 8 trials' values of a grid
// point lie side by side) and keeps their x weights in registers, so the
// multiply-adds bound it (1,152 a warp and run); with a thread per point and trial
// the loads of the grid values did. The sums are those of ug_interp_body.
// 194,560 points: 28 us against 46.
__device__ __forceinline__ void ug_interp_trials_body(const UgInterpArgs &A, const GpVGrid &vg)
{
    __shared__ __align__(16) float ws[UGI_THREADS / 32][2 * UG_W][32];  // the run's weights, [weight][point]
    if (A.gate && !*A.gate) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ch = vg.bx * (UGI_THREADS / 32) + warp;
    if (ch >= A.nchunk) return;  // warp-uniform
    const int2 q = __ldg(&A.chunk[ch]);
    {
        float w[2 * UG_W];
        const float4 *w4 = reinterpret_cast<const float4 *>(A.wts + (size_t)(q.x + lane) * (2 * UG_W));
#pragma unroll
        for (int i = 0; i < 4; i++)
            *reinterpret_cast<float4 *>(&w[4 * i]) = lane < q.y ? __ldg(&w4[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 2 * UG_W; i++) ws[warp][i][lane] = w[i];
    }
    __syncwarp();
    const int trial = lane & 7, p0 = lane & 24;
    float wx[UG_W][8];
#pragma unroll
    for (int j = 0; j < UG_W; j++) {
        *reinterpret_cast<float4 *>(&wx[j][0]) = *reinterpret_cast<const float4 *>(&ws[warp][j][p0]);
        *reinterpret_cast<float4 *>(&wx[j][4]) = *reinterpret_cast<const float4 *>(&ws[warp][j][p0 + 4]);
    }
    const float2 *g = A.grid + (size_t)__ldg(&A.base[q.x]) * GP_NTR + trial;
    float re[8], im[8];
#pragma unroll
    for (int n = 0; n < 8; n++) re[n] = im[n] = 0.f;
#pragma unroll 2
    for (int i = 0; i < UG_W; i++) {
        float2 v[UG_W];
#pragma unroll
        for (int j = 0; j < UG_W; j++) v[j] = __ldg(&g[j * GP_NTR]);
        g += (size_t)A.gw * GP_NTR;
        float wy[8];
        *reinterpret_cast<float4 *>(&wy[0]) = *reinterpret_cast<const float4 *>(&ws[warp][UG_W + i][p0]);
        *reinterpret_cast<float4 *>(&wy[4]) = *reinterpret_cast<const float4 *>(&ws[warp][UG_W + i][p0 + 4]);
#pragma unroll
        for (int n = 0; n < 8; n++) {
            float rr = 0.f, ri = 0.f;
#pragma unroll
            for (int j = 0; j < UG_W; j++) {
                rr = fmaf(wx[j][n], v[j].x, rr);
                ri = fmaf(wx[j][n], v[j].y, ri);
            }
            re[n] = fmaf(wy[n], rr, re[n]);
            im[n] = fmaf(wy[n], ri, im[n]);
        }
    }
    const double invF = A.sc->t_invflux[trial];
#pragma unroll
    for (int n = 0; n < 8; n++) {
        if (p0 + n < q.y) {
            const int s = __ldg(&A.src[q.x + p0 + n]);
            A.out[(size_t)(s & 0x7fffffff) * GP_NTR + trial] =
                ug_vis_out(re[n], im[n], __ldg(&A.phase[q.x + p0 + n]), s < 0, invF);
        }
    }
}

__global__ void __launch_bounds__(UGI_THREADS) k_ug_interp_trials(const UgInterpArgs a)
{
    gp_pdl_enter();
    ug_interp_trials_body(a, gp_vgrid_hw());
}

struct UgInterpTrialsOp {
    using Args = UgInterpArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_interp_trials_body(a, v); }
};

__global__ void __launch_bounds__(UGI_THREADS) k_ug_interp(const UgInterpArgs a)
{
    gp_pdl_enter();
    ug_interp_body(a, gp_vgrid_hw());
}

struct UgInterpOp {
    using Args = UgInterpArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_interp_body(a, v); }
};

// ------------------------------------------------------------ spreading
//
// One warp per run of at most 32 uv points of one grid cell: their 8 x 8 patch
// sum_k c_k wx wy, two patch points per lane, in point order. The run's weights pass
// through shared memory, loaded a point per lane: bound by the chain run -> point ->
// weight c_k, not by a load per point. 1024^2: 13.4 us, 15 with the weights read
// point by point.
#define UGS_LD 20  // floats per point in shared memory: 16 weights, padded against bank conflicts
struct UgSpreadArgs {
    const float2 *cw;
    const int *src;
    const int2 *chunk;
    const float *wts;
    const float2 *phase;
    float2 *patch;
    int nchunk;
    GP_VGRID_FIELDS;
};

__device__ __forceinline__ void ug_spread_body(const UgSpreadArgs &A, const GpVGrid &vg)
{
    __shared__ __align__(16) float ws[8][32][UGS_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ch = vg.bx * 8 + warp;
    if (ch >= A.nchunk) return;  // warp-uniform
    const int2 q = __ldg(&A.chunk[ch]);
    float2 cv = make_float2(0.f, 0.f);
    float4 w4[4];
    if (lane < q.y) {
#pragma unroll
        for (int n = 0; n < 4; n++)
            w4[n] = __ldg(reinterpret_cast<const float4 *>(A.wts + (size_t)(q.x + lane) * (2 * UG_W)) + n);
        // c_k e^{2 pi i (a - b)(N-1)/2}; a conjugated point contributes conj(c_k) (only the real part of the image is kept)
        const int s = __ldg(&A.src[q.x + lane]);
        float2 c = __ldg(&A.cw[s & 0x7fffffff]);
        if (s < 0) c.y = -c.y;
        const float2 ph = __ldg(&A.phase[q.x + lane]);
        cv = make_float2(c.x * ph.x - c.y * ph.y, c.x * ph.y + c.y * ph.x);
    }
#pragma unroll
    for (int n = 0; n < 4; n++)
        if (lane < q.y) *reinterpret_cast<float4 *>(&ws[warp][lane][4 * n]) = w4[n];
    __syncwarp();
    const float *w = ws[warp][0];
    const int i = lane >> 3, j = lane & 7;
    float2 a0 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int n = 0; n < q.y; n++) {
        const float cx = __shfl_sync(0xffffffffu, cv.x, n), cy = __shfl_sync(0xffffffffu, cv.y, n);
        const float wx = w[j];
        const float f0 = wx * w[UG_W + i], f1 = wx * w[UG_W + 4 + i];
        a0.x = fmaf(f0, cx, a0.x);
        a0.y = fmaf(f0, cy, a0.y);
        a1.x = fmaf(f1, cx, a1.x);
        a1.y = fmaf(f1, cy, a1.y);
        w += UGS_LD;
    }
    float2 *out = A.patch + (size_t)ch * (UG_W * UG_W);
    out[lane] = a0;
    out[32 + lane] = a1;
}

__global__ void __launch_bounds__(256) k_ug_spread(const UgSpreadArgs a)
{
    gp_pdl_enter();
    ug_spread_body(a, gp_vgrid_hw());
}

struct UgSpreadOp {
    using Args = UgSpreadArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_spread_body(a, v); }
};

// Grid point (jy, jx) = the patches of the cells (jy - i, jx - j) at (i, j): one
// warp per grid point, lane = (i, j mod 4), two cells a lane, FP64, in a fixed order. Few
// loads, so bound by the longest chain of them: a cell of a dense coverage has dozens of
// runs. 1024^2: 9.3 us, 20 with eight threads a grid point and eight cells each.
struct UgGatherArgs {
    const int *cst;
    const float2 *patch;
    float2 *cgrid;
    int gw, cells;
    GP_VGRID_FIELDS;
};

__device__ __forceinline__ void ug_gather_body(const UgGatherArgs &A, const GpVGrid &vg)
{
    const int q = (vg.bx * (int)blockDim.x + (int)threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (q >= A.cells) return;  // warp-uniform
    const int i = lane >> 2, jy = q / A.gw - i, jx = q % A.gw;
    double re = 0.0, im = 0.0;
    int st[2], end[2];  // runs of its two cells
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const int j = (lane & 3) + 4 * n;
        const bool ok = jy >= 0 && jx >= j;
        st[n] = ok ? __ldg(&A.cst[jy * A.gw + jx - j]) : 0;
        end[n] = ok ? __ldg(&A.cst[jy * A.gw + jx - j + 1]) : 0;
    }
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const float2 *p = A.patch + i * UG_W + (lane & 3) + 4 * n;
        for (int s = st[n]; s < end[n]; s += 8) {
            float2 v[8];  // eight loads in flight
#pragma unroll
            for (int m = 0; m < 8; m++)
                v[m] = s + m < end[n] ? __ldg(&p[(size_t)(s + m) * (UG_W * UG_W)]) : make_float2(0.f, 0.f);
#pragma unroll
            for (int m = 0; m < 8; m++) {
                re += v[m].x;
                im += v[m].y;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
    }
    if (lane == 0) A.cgrid[q] = make_float2((float)re, (float)im);
}

__global__ void __launch_bounds__(256) k_ug_gather(const UgGatherArgs a)
{
    gp_pdl_enter();
    ug_gather_body(a, gp_vgrid_hw());
}

struct UgGatherOp {
    using Args = UgGatherArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_gather_body(a, v); }
};

// ------------------------------------------------- adjoint y contraction
//
// S[y][jx] for 32 columns (lane = jx) and 8 folded image rows per block (a warp
// takes one, image rows h and N-1-h). The sums and differences of the grid rows +-j and
// the twiddles wait in shared memory in FP64 (converted once, not by every warp); the
// next UGC_J rows are loaded meanwhile. Bound by latency. 1024^2: 10.4 us (14.6 with
// two rows a warp, 64 blocks, and conversions where they are used).
#define UGC_J 32
struct UgColsArgs {
    const float2 *cgrid, *ctab;
    float2 *S;
    int N, H, gw, J;
    GP_VGRID_FIELDS;
};

__device__ __forceinline__ void ug_cols_body(const UgColsArgs &A, const GpVGrid &vg)
{
    __shared__ __align__(16) double4_a16 Cs[UGC_J][32];  // (sum, difference)
    __shared__ __align__(16) double2 Ws[8][UGC_J];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xt = (A.gw + 31) / 32;
    const int jx = (vg.bx % xt) * 32 + lane, h = (vg.bx / xt) * 8 + warp;
    const int J1 = A.J + 1;
    float2 p[UGC_J / 8], m[UGC_J / 8], w;  // the next UGC_J rows: +-j = warp, warp + 8, ..; twiddle of row h
    auto load = [&](int jb) {
#pragma unroll
        for (int n = 0; n < UGC_J / 8; n++) {
            const int j = jb + warp + 8 * n;
            const bool ok = j < J1 && jx < A.gw;
            p[n] = ok ? __ldg(&A.cgrid[(size_t)(A.J + j) * A.gw + jx]) : make_float2(0.f, 0.f);
            m[n] = ok && j ? __ldg(&A.cgrid[(size_t)(A.J - j) * A.gw + jx]) : make_float2(0.f, 0.f);
        }
        w = h < A.H && jb + lane < J1 ? __ldg(&A.ctab[(size_t)h * J1 + jb + lane]) : make_float2(0.f, 0.f);
    };
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // even (re, im), odd (re, im)
    load(0);
    for (int jb = 0; jb < J1; jb += UGC_J) {
        const int nj = min(UGC_J, J1 - jb);
#pragma unroll
        for (int n = 0; n < UGC_J / 8; n++) {
            double4_a16 t;
            t.x = p[n].x + m[n].x;
            t.y = p[n].y + m[n].y;
            t.z = p[n].x - m[n].x;
            t.w = p[n].y - m[n].y;
            Cs[warp + 8 * n][lane] = t;
        }
        Ws[warp][lane] = make_double2(w.x, w.y);
        __syncthreads();
        if (jb + UGC_J < J1) load(jb + UGC_J);
#pragma unroll 8
        for (int jj = 0; jj < nj; jj++) {
            const double4_a16 v = Cs[jj][lane];
            const double2 c = Ws[warp][jj];
            acc[0] = fma(c.x, v.x, acc[0]);
            acc[1] = fma(c.x, v.y, acc[1]);
            acc[2] = fma(c.y, v.z, acc[2]);
            acc[3] = fma(c.y, v.w, acc[3]);
        }
        __syncthreads();
    }
    if (jx >= A.gw || h >= A.H) return;
    // C[j] e^{-i theta} + C[-j] e^{i theta} = sum . cos - i difference . sin, theta -> -theta at row h
    A.S[(size_t)(A.N - 1 - h) * A.gw + jx] = make_float2((float)(acc[0] + acc[3]), (float)(acc[1] - acc[2]));
    if (h != A.N - 1 - h)
        A.S[(size_t)h * A.gw + jx] = make_float2((float)(acc[0] - acc[3]), (float)(acc[1] + acc[2]));
}

__global__ void __launch_bounds__(256) k_ug_cols(const UgColsArgs a)
{
    gp_pdl_enter();
    ug_cols_body(a, gp_vgrid_hw());
}

struct UgColsOp {
    using Args = UgColsArgs;
    static __device__ __forceinline__ void run(const Args &a, const GpVGrid &v) { ug_cols_body(a, v); }
};

// ------------------------------------------------------------ host side

// Buffers of the batched trials
int gp_ug_batch_alloc(gpair_ctx *c)
{
    UgState *g = (UgState *)c->ug;
    const int cls = ug_class(c);
    if (!g->Tb[cls]) GP_CUDA(c, cudaMalloc(&g->Tb[cls], sizeof(float) * ug_t_floats(c, g, GP_NTR)));
    if (!g->gridb) GP_CUDA(c, cudaMalloc(&g->gridb, sizeof(float2) * GP_NTR * (size_t)g->cells));
    return GPAIR_OK;
}

// x contraction on the CUDA cores: the current or trial image, or the batch's trial images
int gp_ug_x(gpair_ctx *c, const float *img, int images)
{
    UgState *g = (UgState *)c->ug;
    UgXArgs a;
    a.img = img;
    a.ftab = g->ftab;
    a.T = images > 1 ? g->Tb[0] : g->T[0];
    a.N = g->N;
    a.H = g->H;
    a.nbx = g->nbx;
    a.ldT = g->ldT;
    a.images = images;
    const int bx = gp_cdiv(g->N, UGX_T), by = gp_cdiv(g->nbx, UGX_T);
    a.splits = ug_x_splits(g, images, &a.hper);
    a.gate = images > 1 ? c->gate : nullptr;
    GP_LAUNCH(c, gp_launch(c, k_ug_x, dim3(bx, by, a.splits * images), dim3(256), 0, a));
    (images > 1 ? g->splitsb : g->splits) = a.splits;
    return GPAIR_OK;
}

// columns per block of the y contraction: one for a single image (enough blocks), four for a batch
#define UGR_COLS_BATCH 4

// rsc, lrows: row scales and rows per image of the tensor path's operand (null and N on the CUDA cores)
static UgRowsArgs ug_rows_args(gpair_ctx *c, int images, int splits, const float *rsc, int lrows, const int *gate)
{
    UgState *g = (UgState *)c->ug;
    UgRowsArgs a;
    memset(&a, 0, sizeof(a));
    a.T = images > 1 ? g->Tb[ug_class(c)] : g->T[ug_class(c)];
    a.rsc = rsc;
    a.ctab = g->ctab;
    a.grid = images > 1 ? g->gridb : g->grid;
    a.N = g->N;
    a.H = g->H;
    a.gw = g->nbx;
    a.J = g->J;
    a.ldT = g->ldT;
    a.cells = g->cells;
    a.splits = splits;
    a.lrows = lrows;
    a.split_stride = (size_t)(images > 1 ? images * lrows : g->N) * g->ldT;
    a.gate = gate;
    a.nbx = gp_cdiv(g->nbx, images > 1 ? UGR_COLS_BATCH : 1) * gp_cdiv(g->J + 1, 32);
    a.nby = images;
    return a;
}

static UgInterpArgs ug_interp_args(gpair_ctx *c, int images, const int *gate)
{
    UgState *g = (UgState *)c->ug;
    UgInterpArgs a;
    memset(&a, 0, sizeof(a));
    a.grid = images > 1 ? g->gridb : g->grid;
    a.src = g->src;
    a.base = g->base;
    a.wts = g->wts;
    a.phase = g->phase;
    a.sc = c->sc;
    a.out = images > 1 ? c->visb : c->visd;
    a.nuv = c->nuv;
    a.gw = g->nbx;
    a.chunk = g->chunk;
    a.nchunk = g->nchunk;
    a.gate = gate;
    a.nbx = images > 1 ? gp_cdiv(g->nchunk, UGI_THREADS / 32) : gp_cdiv(c->nuv, UGI_THREADS);
    a.nby = 1;
    return a;
}

static UgSpreadArgs ug_spread_args(gpair_ctx *c)
{
    UgState *g = (UgState *)c->ug;
    UgSpreadArgs a = {c->cw, g->src, g->chunk, g->wts, g->phase, g->patch, g->nchunk, gp_cdiv(g->nchunk, 8), 1};
    return a;
}

static UgGatherArgs ug_gather_args(gpair_ctx *c)
{
    UgState *g = (UgState *)c->ug;
    UgGatherArgs a = {g->cst, g->patch, g->cgrid, g->nbx, g->cells, gp_cdiv(32LL * g->cells, 256), 1};
    return a;
}

static UgColsArgs ug_cols_args(gpair_ctx *c)
{
    UgState *g = (UgState *)c->ug;
    UgColsArgs a = {g->cgrid, g->ctab, g->S, g->N, g->H, g->nbx, g->J,
                    gp_cdiv(g->nbx, 32) * gp_cdiv(g->H, 8), 1};
    return a;
}

// From T to the visibilities: V_k / F into visd (images = 1), or of every trial into visb
int gp_ug_vis(gpair_ctx *c, int images)
{
    UgState *g = (UgState *)c->ug;
    const float *rsc = nullptr;
    int lrows = g->N, splits = images > 1 ? g->splitsb : g->splits;
    if (c->precision != GPAIR_PREC_FP32) {
        int rc = gp_tc_ug_rows(c, images, &rsc, &lrows, &splits);
        if (rc) return rc;
    }
    const int *gate = images > 1 ? c->gate : nullptr;
    const UgRowsArgs r = ug_rows_args(c, images, splits, rsc, lrows, gate);
    GP_LAUNCH(c, gp_launch(c, images > 1 ? k_ug_rows<UGR_COLS_BATCH> : k_ug_rows<1>, dim3(r.nbx, r.nby),
                           dim3(32 * (images > 1 ? UgRowsGeo<UGR_COLS_BATCH>::W : UgRowsGeo<1>::W)), 0,
                           r));
    const UgInterpArgs t = ug_interp_args(c, images, gate);
    GP_LAUNCH(c, gp_launch(c, images > 1 ? k_ug_interp_trials : k_ug_interp, dim3(t.nbx, t.nby), dim3(UGI_THREADS), 0,
                           t));
    return GPAIR_OK;
}

// From the uv weights c_k to S[y][jx], the x contraction's operand (gp_grad_finalize finishes the gradient)
int gp_ug_adjoint(gpair_ctx *c)
{
    const UgSpreadArgs s = ug_spread_args(c);
    GP_LAUNCH(c, gp_launch(c, k_ug_spread, dim3(s.nbx), dim3(256), 0, s));
    const UgGatherArgs t = ug_gather_args(c);
    GP_LAUNCH(c, gp_launch(c, k_ug_gather, dim3(t.nbx), dim3(256), 0, t));
    const UgColsArgs q = ug_cols_args(c);
    GP_LAUNCH(c, gp_launch(c, k_ug_cols, dim3(q.nbx), dim3(256), 0, q));
    return GPAIR_OK;
}

// ------------------------------------------------- grouped stage launches

size_t gp_ug_stage_args_size(int stage)
{
    switch (stage) {
    case GS_UG_ROWS:
    case GS_UG_ROWS_T: return sizeof(UgRowsArgs);
    case GS_UG_INTERP:
    case GS_UG_INTERP_T: return sizeof(UgInterpArgs);
    case GS_UG_SPREAD: return sizeof(UgSpreadArgs);
    case GS_UG_GATHER: return sizeof(UgGatherArgs);
    case GS_UG_COLS: return sizeof(UgColsArgs);
    default: return 0;
    }
}

template <class A>
static int put_args(const A &a, void *out, int *nblocks)
{
    memcpy(out, &a, sizeof(A));
    *nblocks = a.nbx * a.nby;
    return GPAIR_OK;
}

int gp_ug_stage_args(gpair_ctx *c, int stage, void *out, int *nblocks)
{
    const int images = (stage == GS_UG_ROWS_T || stage == GS_UG_INTERP_T) ? GP_NTR : 1;
    switch (stage) {
    case GS_UG_ROWS:
    case GS_UG_ROWS_T: {
        const float *rsc;
        int lrows, splits, rc;
        if ((rc = gp_tc_ug_rows(c, images, &rsc, &lrows, &splits))) return rc;
        return put_args(ug_rows_args(c, images, splits, rsc, lrows, nullptr), out, nblocks);
    }
    case GS_UG_INTERP:
    case GS_UG_INTERP_T: return put_args(ug_interp_args(c, images, nullptr), out, nblocks);
    case GS_UG_SPREAD: return put_args(ug_spread_args(c), out, nblocks);
    case GS_UG_GATHER: return put_args(ug_gather_args(c), out, nblocks);
    case GS_UG_COLS: return put_args(ug_cols_args(c), out, nblocks);
    default: return GPAIR_ERR_INVALID;
    }
}

template <class Op, int THREADS>
static int group_launch(gpair_ctx *c, const void *d_args, const int *d_start, int n, int total, const int *gate)
{
    GP_LAUNCH(c, gp_launch(c, k_grouped<Op, THREADS>, dim3(total), dim3(THREADS), 0,
                           (const typename Op::Args *)d_args, d_start, n, gate));
    return GPAIR_OK;
}

int gp_ug_stage_group_launch(gpair_ctx *c, int stage, const void *d_args, const int *d_start, int n, int total,
                             const int *gate)
{
    if (total < 1 || n < 1) return GPAIR_ERR_INVALID;
    switch (stage) {
    case GS_UG_ROWS: return group_launch<UgRowsOp<1>, 32 * UgRowsGeo<1>::W>(c, d_args, d_start, n, total, gate);
    case GS_UG_ROWS_T:
        return group_launch<UgRowsOp<UGR_COLS_BATCH>, 32 * UgRowsGeo<UGR_COLS_BATCH>::W>(c, d_args, d_start, n, total,
                                                                                         gate);
    case GS_UG_INTERP: return group_launch<UgInterpOp, UGI_THREADS>(c, d_args, d_start, n, total, gate);
    case GS_UG_INTERP_T: return group_launch<UgInterpTrialsOp, UGI_THREADS>(c, d_args, d_start, n, total, gate);
    case GS_UG_SPREAD: return group_launch<UgSpreadOp, 256>(c, d_args, d_start, n, total, gate);
    case GS_UG_GATHER: return group_launch<UgGatherOp, 256>(c, d_args, d_start, n, total, gate);
    case GS_UG_COLS: return group_launch<UgColsOp, 256>(c, d_args, d_start, n, total, gate);
    default: return GPAIR_ERR_INVALID;
    }
}
