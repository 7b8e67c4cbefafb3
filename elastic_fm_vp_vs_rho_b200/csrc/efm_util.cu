// Volume utilities of the inversion loop: float64 reductions (misfit, dot products), the
// L-BFGS history shift and two-loop recursion with device-resident scalars, gradient
// smoothing + masking, and the lambda/mu/rho -> Vp/Vs/rho chain rule.
//
// Reductions are deterministic: a fixed grid of blocks writes float64 partials in block
// order and one block sums them in order, so repeated calls give identical bits.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <algorithm>
#include <initializer_list>

#include "efm_util.cuh"

namespace {

constexpr int RB = 256;  // threads per reduction block

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sh[RB / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < RB / 32) ? sh[threadIdx.x] : 0.0;
    if (wid == 0)
        for (int o = 4; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    return v;
}

// partial[blockIdx.y * gridDim.x + blockIdx.x] = sum over this block's share of segment y
// of (a-b)^2 (mode 0, also writes res = a-b) or a*b (mode 1).
__global__ void __launch_bounds__(RB)
k_partial(const float *__restrict__ a, const float *__restrict__ b, float *__restrict__ res,
          const int64_t *__restrict__ seg, int mode, double *__restrict__ partial) {
    const int64_t lo = seg[blockIdx.y], hi = seg[blockIdx.y + 1];
    double acc = 0.0;
    const int64_t stride = (int64_t)gridDim.x * RB;
    for (int64_t i = lo + (int64_t)blockIdx.x * RB + threadIdx.x; i < hi; i += stride) {
        if (mode == 0) {
            const float r = a[i] - b[i];
            res[i] = r;
            acc += (double)r * (double)r;
        } else {
            acc += (double)a[i] * (double)b[i];
        }
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) partial[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

__global__ void __launch_bounds__(RB)
k_finish(const double *__restrict__ partial, int nblk, double scale, double *__restrict__ out) {
    double acc = 0.0;
    const double *p = partial + (int64_t)blockIdx.x * nblk;
    // fixed-order strided accumulation, then a fixed-order tree
    for (int i = threadIdx.x; i < nblk; i += RB) acc += p[i];
    acc = block_sum(acc);
    if (threadIdx.x == 0) out[blockIdx.x] = scale * acc;
}

// ----------------------------------------------------------------------- L-BFGS pieces
template <int V>
struct Vec {
    float a[V];
};

template <int V>
__device__ __forceinline__ Vec<V> vload(const float *p) {
    Vec<V> r;
    if (V == 4) {
        const float4 q = *reinterpret_cast<const float4 *>(p);
        r.a[0] = q.x;
        r.a[1 % V] = q.y;
        r.a[2 % V] = q.z;
        r.a[3 % V] = q.w;
    } else {
        r.a[0] = *p;
    }
    return r;
}

template <int V>
__device__ __forceinline__ void vstore(float *p, const Vec<V> &v) {
    if (V == 4)
        *reinterpret_cast<float4 *>(p) = make_float4(v.a[0], v.a[1 % V], v.a[2 % V], v.a[3 % V]);
    else
        *p = v.a[0];
}

__global__ void k_sub(float *__restrict__ out, const float *__restrict__ a,
                      const float *__restrict__ b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a[i] - b[i];
}

// The two-loop recursion from inner products.  Its direction is a combination of g and the used
// history vectors whose coefficients follow from the products s_i.y_j (i >= j, layers newest
// first), y_i.y_j, s_i.g and y_i.g: one pass forms all of them, a small kernel runs the two loops
// on them, one pass forms the combination (49 us at 200 x 200 x 100, 8 pairs: the DRAM rate).  Each
// vector is read twice, 272 MB each time; vector by vector, every step of the recursion reads and
// writes the direction and two more vectors (1.5 GB, about 70 launches, 740 us; this way 130 us).
// Products and combination are in float64; the direction is rounded once, at the end, instead of
// after every step.  Long histories of large vectors take the vectors (by_products).
//
// The products: a warp takes groups a >= b of eight layers and runs the float64 matrix instruction
// (8 x 8 products, four cells per step) for y_a.y_b and s_a.y_b; a lane's four consecutive cells of
// one vector serve as operand in four steps, as row or as column alike.  Bound by the latency of
// its loads (fetched a step ahead; without that 109 us), then conversions and the matrix rate.  With 4 x 4 products per
// warp on the vector unit (52 conversions) the pass took 116 us at 200 x 200 x 100, this 72 us.
// Per pair of groups 64 + 64 products and, on the diagonal, 8 + 8 with g.
constexpr int GT = 144;

__host__ __device__ constexpr int gram_groups(int u) { return (u + 7) / 8; }
__host__ __device__ constexpr int gram_tiles(int u) { return gram_groups(u) * (gram_groups(u) + 1) / 2; }

__device__ __forceinline__ int gram_at(bool s, int i, int j) {  // group of i >= group of j
    const int a = i / 8, b = j / 8;
    return (a * (a + 1) / 2 + b) * GT + (s ? 64 : 0) + (i % 8) * 8 + j % 8;
}
__device__ __forceinline__ int gram_g(bool s, int i) {
    const int a = i / 8;
    return (a * (a + 1) / 2 + a) * GT + 128 + (s ? 8 : 0) + i % 8;
}

// c (8 x 8: row lane / 4, columns 2 (lane % 4) and the next) += a (row lane / 4, cell lane % 4) b
// (cell lane % 4, column lane / 4)
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

template <int V>
__device__ __forceinline__ void cells4(const float *p, int64_t i, int64_t n, float (&v)[4]) {
    if (V == 4 && i < n) {
        const Vec<V> q = vload<V>(p + i);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = q.a[k % V];
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k < n ? p[i + k] : 0.f;
    }
}

template <int V>
__global__ void __launch_bounds__(256, 3)
k_lbfgs_gram(const float *__restrict__ s1, const float *__restrict__ y1, const float *__restrict__ g, int64_t n,
             int u, double *__restrict__ partial) {
    __shared__ double sh[8][GT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int a = 0;
    while ((a + 1) * (a + 2) / 2 <= (int)blockIdx.x) ++a;
    const int b = blockIdx.x - a * (a + 1) / 2;
    // this lane's vectors (past the last one: the last one again, its products unused)
    const int64_t ra = (int64_t)min(8 * a + lane / 4, u - 1) * n, rb = (int64_t)min(8 * b + lane / 4, u - 1) * n;
    double yy[2] = {}, sy[2] = {}, yg = 0.0, sg = 0.0;
    const int64_t step = (int64_t)gridDim.y * 8 * 16;
    float now[4][4], next[4][4];  // y_a, s_a, y_b, g: this step's and the next one's cells
    auto load = [&](int64_t e, float (&f)[4][4]) {
        const int64_t i = e + 4 * (lane % 4);
        cells4<V>(y1 + ra, i, n, f[0]);
        cells4<V>(s1 + ra, i, n, f[1]);
        if (a != b) cells4<V>(y1 + rb, i, n, f[2]);
        if (a == b) cells4<V>(g, i, n, f[3]);
    };
    int64_t e = ((int64_t)blockIdx.y * 8 + warp) * 16;
    load(e, now);
    for (; e < n; e += step) {
        load(e + step, next);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double y = (double)now[0][k], s = (double)now[1][k], c = a == b ? y : (double)now[2][k];
            dmma(yy, y, c);
            dmma(sy, s, c);
            if (a == b) {
                const double q = (double)now[3][k];
                yg += y * q;
                sg += s * q;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int k = 0; k < 4; ++k) now[q][k] = next[q][k];
    }
    yg += __shfl_xor_sync(0xffffffffu, yg, 1);
    yg += __shfl_xor_sync(0xffffffffu, yg, 2);
    sg += __shfl_xor_sync(0xffffffffu, sg, 1);
    sg += __shfl_xor_sync(0xffffffffu, sg, 2);
    const int at = (lane / 4) * 8 + 2 * (lane % 4);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        sh[warp][at + k] = yy[k];
        sh[warp][64 + at + k] = sy[k];
    }
    if (lane % 4 == 0) {
        sh[warp][128 + lane / 4] = yg;
        sh[warp][136 + lane / 4] = sg;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < GT; k += 256) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += sh[w][k];
        partial[((int64_t)blockIdx.x * GT + k) * gridDim.y + blockIdx.y] = v;
    }
}

// The two loops on the products (one block).  w: [0] y1.y1  [1] s1.y1  [3] gamma  [4..4+L) sigma
// [4+L..4+2L) eps  [4+2L..4+3L) coefficients of s; those of y are -gamma eps.
__global__ void __launch_bounds__(128)
k_lbfgs_solve(const double *__restrict__ G, double *__restrict__ w, int L, int u, int used) {
    double *sigma = w + 4, *eps = w + 4 + L, *coef = w + 4 + 2 * L, *run = w + 4 + 3 * L;
    const int t = threadIdx.x;
    const double yy = G[gram_at(false, 0, 0)], sy = G[gram_at(true, 0, 0)];
    const double gamma = yy == 0.0 ? 0.0 : sy / yy;
    if (t == 0) {
        w[0] = yy;
        w[1] = sy;
        w[3] = gamma;
    }
    for (int m = t; m < used; m += 128) {
        const double d = G[gram_at(true, m, m)];
        sigma[m] = d == 0.0 ? 0.0 : 1.0 / d;
        run[m] = G[gram_g(true, m)];  // s_m . q
    }
    __syncthreads();
    for (int k = 0; k < used; ++k) {
        if (t == 0) eps[k] = sigma[k] * run[k];
        __syncthreads();
        const double e = eps[k];
        for (int m = k + 1 + t; m < used; m += 128) run[m] -= e * G[gram_at(true, m, k)];
        __syncthreads();
    }
    for (int k = t; k < used; k += 128) {  // y_k . gamma q
        double v = G[gram_g(false, k)];
        for (int j = 0; j < used; ++j) v -= eps[j] * G[j <= k ? gram_at(false, k, j) : gram_at(false, j, k)];
        run[k] = gamma * v;
    }
    __syncthreads();
    for (int k = used - 1; k >= 0; --k) {
        if (t == 0) coef[k] = eps[k] - sigma[k] * run[k];
        __syncthreads();
        const double c = coef[k];
        for (int m = t; m < k; m += 128) run[m] += c * G[gram_at(true, k, m)];
        __syncthreads();
    }
}

// r = gamma g - sum_k gamma eps_k y_k + sum_k coef_k s_k
template <int V>
__global__ void __launch_bounds__(256)
k_lbfgs_combine(const float *__restrict__ s1, const float *__restrict__ y1, const float *g, float *r,
                const double *__restrict__ w, int L, int used, int64_t n) {
    extern __shared__ double sh[];  // [used] of y, [used] of s
    const double gamma = w[3];
    for (int k = threadIdx.x; k < used; k += 256) {
        sh[k] = -gamma * w[4 + L + k];
        sh[used + k] = w[4 + 2 * L + k];
    }
    __syncthreads();
    for (int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * V; i < n; i += (int64_t)gridDim.x * 256 * V) {
        const Vec<V> vg = vload<V>(g + i);
        double acc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = gamma * (double)vg.a[v];
#pragma unroll 4
        for (int k = 0; k < used; ++k) {
            const Vec<V> vy = vload<V>(y1 + k * n + i), vs = vload<V>(s1 + k * n + i);
            const double cy = sh[k], cs = sh[used + k];
#pragma unroll
            for (int v = 0; v < V; ++v) acc[v] += cy * (double)vy.a[v] + cs * (double)vs.a[v];
        }
        Vec<V> o;
#pragma unroll
        for (int v = 0; v < V; ++v) o.a[v] = (float)acc[v];
        vstore<V>(r + i, o);
    }
}

// The recursion vector by vector, for histories whose products cost more (by_products).  The
// direction is read, changed and written once per vector.  w as in k_lbfgs_solve, [2] the last dot.
enum { LB_GAMMA, LB_SIGMA, LB_EPS };

__global__ void k_lbfgs_scalar(double *w, int L, int k, int what) {
    if (what == LB_GAMMA) w[3] = w[0] == 0.0 ? 0.0 : w[1] / w[0];
    if (what == LB_SIGMA) w[4 + k] = w[2] == 0.0 ? 0.0 : 1.0 / w[2];
    if (what == LB_EPS) w[4 + L + k] = w[4 + k] * w[2];
}

__global__ void k_lbfgs_bounds(int64_t *seg, int64_t n) {
    seg[0] = 0;
    seg[1] = n;
}

// q -= eps_k y   (first loop)
__global__ void k_lbfgs_axpy1(float *__restrict__ q, const float *__restrict__ y, const double *__restrict__ w, int L,
                              int k, int64_t n) {
    const double e = w[4 + L + k];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        q[i] = (float)((double)q[i] - e * (double)y[i]);
}

__global__ void k_lbfgs_scale(float *__restrict__ r, const double *__restrict__ w, int64_t n) {
    const double gmm = w[3];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = (float)(gmm * (double)r[i]);
}

// r += s_k (eps_k - sigma_k w[2]), w[2] = y_k . r   (second loop)
__global__ void k_lbfgs_axpy2(float *__restrict__ r, const float *__restrict__ s, const double *__restrict__ w, int L,
                              int k, int64_t n) {
    const double coef = w[4 + L + k] - w[4 + k] * w[2];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = (float)((double)r[i] + (double)s[i] * coef);
}

// ------------------------------------------------------------------- smoothing + mask
struct Gauss {
    int radius;
    float w[33];
};

__device__ __forceinline__ int reflect_idx(int i, int n) {
    // scipy.ndimage mode 'reflect': (d c b a | a b c d | d c b a)
    while (i < 0 || i >= n) {
        if (i < 0) i = -i - 1;
        if (i >= n) i = 2 * n - i - 1;
    }
    return i;
}

// One 1-D pass, S outputs per thread along the axis: each of the S + 2 radius inputs is read once and
// feeds up to S sums, in ascending order of the taps as a sum by itself would take them.  The
// volumes of the inversion grids fit in L2, so the passes run at its rate; one thread per output
// with the index arithmetic of three axes took 57 us per 200 x 200 x 100 pass (issue bound), this
// 13 us.  A line is `count` cells, `step` floats apart; `outer` sets of `inner` lines side by side.
// The block has as many threads side by side as there are lines, up to a warp's, and the rest along
// them: with always 32, planes 4 cells wide left 31 lanes of a warp idle (400 x 400 x 4: 98 us, 32 now).
template <int V>
__global__ void __launch_bounds__(256)
k_gauss_line(const float *__restrict__ in, float *__restrict__ out, int64_t inner, int count, int64_t step,
             int64_t outer, int64_t outer_step, Gauss g) {
    constexpr int S = 8;
    const int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * V;
    const int strips = (count + S - 1) / S, R = g.radius;
    if (x >= inner) return;
    for (int64_t l = (int64_t)blockIdx.y * blockDim.y + threadIdx.y; l < strips * outer;
         l += (int64_t)gridDim.y * blockDim.y) {
        const int64_t o = l / strips;
        const int c0 = (int)(l - o * strips) * S;
        const float *p = in + o * outer_step + x;
        float acc[S][V] = {};
        const int end = min(S, count - c0) + R;
        for (int i0 = -R; i0 < end; i0 += 4) {  // (what a batch reads past the last input is not used)
            Vec<V> in4[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) in4[b] = vload<V>(p + reflect_idx(c0 + i0 + b, count) * step);
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int k = 0; k < S; ++k) {
                    const int j = i0 + b - k + R;
                    if (j < 0 || j > 2 * R) continue;
#pragma unroll
                    for (int q = 0; q < V; ++q) acc[k][q] += g.w[j] * in4[b].a[q];
                }
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
            if (c0 + k >= count) break;
            Vec<V> r;
#pragma unroll
            for (int q = 0; q < V; ++q) r.a[q] = acc[k][q];
            vstore<V>(out + o * outer_step + (c0 + k) * step + x, r);
        }
    }
}

// The mask: zero z < top and the (W+2) margins of the x, y and bottom faces (:2484-2504).
struct Mask {
    int nx, ny, nz, W, top;
    __device__ __forceinline__ bool row(int y, int z) const {
        return z < top || y < W + 2 || y >= ny - W - 2 || z >= nz - W - 2;
    }
    __device__ __forceinline__ bool col(int x) const { return x < W + 2 || x >= nx - W - 2; }
};

// The pass along x, in place, and the mask: a warp per row, held in shared memory; masked rows are
// only written.
__global__ void __launch_bounds__(256) k_gauss_row_mask(float *__restrict__ vol, Mask M, Gauss g) {
    extern __shared__ float rows[];
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, R = g.radius, nx = M.nx, len = nx + 2 * R;
    float *row = rows + (threadIdx.x >> 5) * len;
    for (int64_t q = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); q < (int64_t)M.ny * M.nz;
         q += (int64_t)gridDim.x * warps) {
        const int y = (int)(q / M.nz), z = (int)(q - (int64_t)y * M.nz);
        float *p = vol + q * nx;
        if (M.row(y, z)) {
            for (int x = lane; x < nx; x += 32) p[x] = 0.f;
            continue;
        }
#pragma unroll 4
        for (int x = lane; x < nx; x += 32) row[R + x] = p[x];
        __syncwarp();
        if (lane < R) {
            row[lane] = row[R + reflect_idx(lane - R, nx)];
            row[R + nx + lane] = row[R + reflect_idx(nx + lane, nx)];
        }
        __syncwarp();
        for (int x0 = lane; x0 < nx; x0 += 128) {
            float acc[4] = {};
            for (int j = 0; j <= 2 * R; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (x0 + 32 * k < nx) acc[k] += g.w[j] * row[x0 + 32 * k + j];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int x = x0 + 32 * k;
                if (x < nx) p[x] = M.col(x) ? 0.f : acc[k];
            }
        }
        __syncwarp();
    }
}

// The mask by itself: of `vol` in place, or of a copy of `in`.
template <bool COPY>
__global__ void __launch_bounds__(256) k_mask(const float *__restrict__ in, float *__restrict__ vol, Mask M) {
    const int64_t n = (int64_t)M.nx * M.ny * M.nz;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int x = (int)(i % M.nx);
        const int64_t q = i / M.nx;
        if (M.row((int)(q / M.nz), (int)(q % M.nz)) || M.col(x))
            vol[i] = 0.f;
        else if (COPY)
            vol[i] = in[i];
    }
}

__global__ void k_chain(float *__restrict__ gl, float *__restrict__ gm, float *__restrict__ gr,
                        const float *__restrict__ vp, const float *__restrict__ vs,
                        const float *__restrict__ rho, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        // float64 arithmetic: g_mu - 2 g_lambda and the rho sum cancel strongly, and float32
        // intermediates would add rounding of the large terms to the small results
        const double l = gl[i], m = gm[i], r = rho[i], p = vp[i], s = vs[i];
        gl[i] = (float)(2.0 * r * p * l);
        gm[i] = (float)(2.0 * r * s * (m - 2.0 * l));
        gr[i] = (float)((double)gr[i] + (p * p - 2.0 * s * s) * l + s * s * m);
    }
}

// One Adam step of up to ADAM_MAX tensors (blockIdx.y), in float32 throughout and rounded where
// elementwise tensor operations would round: a launch instead of eight per tensor.
constexpr int ADAM_MAX = 16;
struct AdamArgs {
    float *p[ADAM_MAX], *m[ADAM_MAX], *v[ADAM_MAX];
    const float *g[ADAM_MAX];
    int64_t n[ADAM_MAX];
    float lr, beta1, beta2, alpha1, alpha2, eps, r1, r2;  // alpha = 1 - beta, r = 1 / (1 - beta^step)
};

__global__ void __launch_bounds__(256) k_adam(AdamArgs A) {
    const int k = blockIdx.y;
    float *const p = A.p[k], *const m = A.m[k], *const v = A.v[k];
    const float *const g = A.g[k];
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < A.n[k]; i += (int64_t)gridDim.x * 256) {
        const float a = g[i];
        const float mi = __fmaf_rn(A.alpha1, a, __fmul_rn(m[i], A.beta1));
        const float vi = __fmaf_rn(A.alpha2, __fmul_rn(a, a), __fmul_rn(v[i], A.beta2));
        m[i] = mi;
        v[i] = vi;
        const float d = __fadd_rn(__fsqrt_rn(__fmul_rn(vi, A.r2)), A.eps);
        p[i] = __fmaf_rn(-A.lr, __fdiv_rn(__fmul_rn(mi, A.r1), d), p[i]);
    }
}

int grid_for(int64_t n) {
    int64_t b = (n + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    return (int)b;
}

// Whether n floats behind each pointer can be read four at a time, layer by layer.
bool vec4_ok(std::initializer_list<const float *> p, int64_t n) {
    uintptr_t a = 0;
    for (const float *q : p) a |= (uintptr_t)q;
    return n % 4 == 0 && a % 16 == 0;
}

// Blocks per pair of groups: three waves of the device, shared by the pairs.
int gram_blocks(int T) { return std::max(8, 6 * 148 / T); }

// Whether the products of u pairs take less time than the recursion vector by vector.  A pair of
// groups costs the products 24 vectors' reads (17 on the diagonal) whatever the groups hold; the
// recursion takes seven launches and twelve reads and writes of a vector per pair of vectors, from
// L2 while a few of them fit.  us measured, products and vectors: 4 000 000 cells, 65 pairs 3627, 4313;
// 81 pairs 5717, 5401; 97 pairs 7693, 6397; rows off 16 bytes, 65 pairs 4593, 4305; 1 000 000 cells,
// 199 pairs 5688, 8987; 32 000 000 cells, 33 pairs 9954, 11483; 41 pairs 14244, 14224; 64 000 000
// cells, 1 pair 1035, 993.  Beyond MAX_PRODUCTS pairs the products' scratch would pass 90 MB.
constexpr int MAX_PRODUCTS = 1024;

bool by_products(int u, int64_t n, bool v4) {
    if (u > MAX_PRODUCTS) return false;
    const double cells = (double)n, groups = gram_groups(u), reads = 17 * groups + 12 * groups * (groups - 1);
    const double products = cells * (8.8e-7 * (v4 ? 1 : 1.2) * reads + 6.2e-7 * (2 * u + 2));
    return products <= 30 + 4.2e-6 * cells + u * std::max(37 + 7.2e-6 * cells, 25 + 1e-5 * cells);
}

}  // namespace

// ------------------------------------------------------------------------- entry points
cudaError_t efm_util_reduce(const float *a, const float *b, float *res, const int64_t *seg_dev,
                            int nseg, int mode, double scale, double *partial, int nblk,
                            double *out, cudaStream_t s) {
    dim3 g(nblk, nseg);
    k_partial<<<g, RB, 0, s>>>(a, b, res, seg_dev, mode, partial);
    k_finish<<<nseg, RB, 0, s>>>(partial, nblk, scale, out);
    return cudaGetLastError();
}

cudaError_t efm_util_lbfgs_history(float *sk, float *yk, const float *m, const float *g, int L,
                                   int64_t n, int iter, cudaStream_t s) {
    cudaError_t e;
    if (iter == 0) {
        if ((e = cudaMemcpyAsync(sk, m, n * sizeof(float), cudaMemcpyDeviceToDevice, s))) return e;
        return cudaMemcpyAsync(yk, g, n * sizeof(float), cudaMemcpyDeviceToDevice, s);
    }
    // newest difference into layer 1 after shifting layers 1..L-3 up by one (lbfgs.py:18-25)
    for (int j = L - 2; j >= 2; --j) {
        if ((e = cudaMemcpyAsync(sk + (int64_t)j * n, sk + (int64_t)(j - 1) * n, n * sizeof(float),
                                 cudaMemcpyDeviceToDevice, s)))
            return e;
        if ((e = cudaMemcpyAsync(yk + (int64_t)j * n, yk + (int64_t)(j - 1) * n, n * sizeof(float),
                                 cudaMemcpyDeviceToDevice, s)))
            return e;
    }
    if (L >= 3) {
        k_sub<<<grid_for(n), 256, 0, s>>>(sk + n, m, sk, n);
        k_sub<<<grid_for(n), 256, 0, s>>>(yk + n, g, yk, n);
    }
    if ((e = cudaMemcpyAsync(sk, m, n * sizeof(float), cudaMemcpyDeviceToDevice, s))) return e;
    if ((e = cudaMemcpyAsync(yk, g, n * sizeof(float), cudaMemcpyDeviceToDevice, s))) return e;
    return cudaGetLastError();
}

// Doubles of scratch a direction of L layers needs: per product, the blocks' parts and their sum
// (more than what the recursion by vectors uses, the parts of one dot and its bounds).
int64_t efm_util_lbfgs_scratch(int L) {
    const int64_t T = gram_tiles(std::min(L - 1, MAX_PRODUCTS));
    return T * GT + std::max<int64_t>(8 * T, 6 * 148) * GT;
}

static cudaError_t lbfgs_by_vectors(const float *s1, const float *y1, const float *g, float *r, double *w, int L,
                                    int64_t n, int used, double *scratch, cudaStream_t s) {
    const int gb = grid_for(n);
    int64_t *const seg = reinterpret_cast<int64_t *>(scratch + EFM_RED_BLOCKS);
    cudaError_t e;
    auto dot = [&](const float *a, const float *b, double *out) {
        return efm_util_reduce(a, b, nullptr, seg, 1, 1, 1.0, scratch, EFM_RED_BLOCKS, out, s);
    };
    k_lbfgs_bounds<<<1, 1, 0, s>>>(seg, n);
    if ((e = dot(y1, y1, w + 0)) || (e = dot(s1, y1, w + 1))) return e;
    k_lbfgs_scalar<<<1, 1, 0, s>>>(w, L, 0, LB_GAMMA);
    if (r != g && (e = cudaMemcpyAsync(r, g, n * sizeof(float), cudaMemcpyDeviceToDevice, s))) return e;
    for (int k = 0; k < used; ++k) {
        if ((e = dot(y1 + k * n, s1 + k * n, w + 2))) return e;
        k_lbfgs_scalar<<<1, 1, 0, s>>>(w, L, k, LB_SIGMA);
        if ((e = dot(s1 + k * n, r, w + 2))) return e;
        k_lbfgs_scalar<<<1, 1, 0, s>>>(w, L, k, LB_EPS);
        k_lbfgs_axpy1<<<gb, 256, 0, s>>>(r, y1 + k * n, w, L, k, n);
    }
    k_lbfgs_scale<<<gb, 256, 0, s>>>(r, w, n);
    for (int k = used - 1; k >= 0; --k) {
        if ((e = dot(y1 + k * n, r, w + 2))) return e;
        k_lbfgs_axpy2<<<gb, 256, 0, s>>>(r, s1 + k * n, w, L, k, n);
    }
    return cudaGetLastError();
}

cudaError_t efm_util_lbfgs_direction(const float *sk, const float *yk, const float *g, float *r,
                                     double *w, int L, int64_t n, int iter, double *scratch,
                                     cudaStream_t s) {
    const int used = iter < L ? iter : L - 1;
    const int u = used > 0 ? used : 1;  // (gamma takes the newest pair also before any is used)
    const bool v4 = vec4_ok({sk, yk, g, r}, n);
    if (!by_products(u, n, v4)) return lbfgs_by_vectors(sk + n, yk + n, g, r, w, L, n, used, scratch, s);
    const int T = gram_tiles(u);
    const int nblk = gram_blocks(T);
    const dim3 grid(T, nblk);
    if (v4)
        k_lbfgs_gram<4><<<grid, 256, 0, s>>>(sk + n, yk + n, g, n, u, scratch);
    else
        k_lbfgs_gram<1><<<grid, 256, 0, s>>>(sk + n, yk + n, g, n, u, scratch);
    double *G = scratch + (int64_t)T * GT * nblk;
    k_finish<<<T * GT, RB, 0, s>>>(scratch, nblk, 1.0, G);
    k_lbfgs_solve<<<1, 128, 0, s>>>(G, w, L, u, used);
    const int csh = 2 * used * (int)sizeof(double);
    if (v4)
        k_lbfgs_combine<4><<<grid_for(n / 4), 256, csh, s>>>(sk + n, yk + n, g, r, w, L, used, n);
    else
        k_lbfgs_combine<1><<<grid_for(n), 256, csh, s>>>(sk + n, yk + n, g, r, w, L, used, n);
    return cudaGetLastError();
}

static cudaError_t gauss_line(const float *in, float *out, int64_t inner, int count, int64_t step, int64_t outer,
                              int64_t outer_step, const Gauss &g, cudaStream_t s) {
    const int64_t lines = (count + 7) / 8 * outer;
    const bool v4 = vec4_ok({in, out}, inner) && step % 4 == 0 && outer_step % 4 == 0;
    const int64_t wide = v4 ? inner / 4 : inner;  // threads that have cells side by side
    int bx = 32;
    while (bx > 1 && bx / 2 >= wide) bx /= 2;
    const dim3 block(bx, 256 / bx);
    const dim3 grid((unsigned)((wide + bx - 1) / bx),
                    (unsigned)std::min<int64_t>((lines + block.y - 1) / block.y, 65535));
    if (v4)
        k_gauss_line<4><<<grid, block, 0, s>>>(in, out, inner, count, step, outer, outer_step, g);
    else
        k_gauss_line<1><<<grid, block, 0, s>>>(in, out, inner, count, step, outer, outer_step, g);
    return cudaGetLastError();
}

cudaError_t efm_util_smooth_mask(float *gv, float *tmp, int nx, int ny, int nz, float sigma,
                                 int W, int top, cudaStream_t s) {
    const int64_t n = (int64_t)nx * ny * nz, plane = (int64_t)nx * nz;
    const Mask M = {nx, ny, nz, W, top};
    if (!(sigma > 0.f)) {
        k_mask<false><<<grid_for(n), 256, 0, s>>>(nullptr, gv, M);
        return cudaGetLastError();
    }
    Gauss g;
    int radius = (int)(4.0 * sigma + 0.5);
    if (radius > 16) radius = 16;
    g.radius = radius;
    double wsum = 0.0, ww[33];
    for (int j = -radius; j <= radius; ++j) {
        ww[j + radius] = exp(-0.5 / ((double)sigma * sigma) * (double)j * j);
        wsum += ww[j + radius];
    }
    for (int j = 0; j < 2 * radius + 1; ++j) g.w[j] = (float)(ww[j] / wsum);
    cudaError_t e;
    if ((e = gauss_line(gv, tmp, plane, ny, plane, 1, 0, g, s))) return e;
    if ((e = gauss_line(tmp, gv, nx, nz, nx, ny, plane, g, s))) return e;
    // Along x: rows in shared memory, where a row gives a warp work and the rows give the device
    // warps; otherwise lines of neighbouring cells out of place (us for sigma 1 and 4, rows | lines:
    // 400 x 400 rows of 16 cells 76, 192 | 48, 75, of 32 85, 209 | 75, 123, of 48 97, 233 | 101, 173;
    // 100 x 100 rows of 2000 164, 343 | 239, 419, of 4000 406, 851 | 460, 815, of 8000 1198, 2636 |
    // 892, 1593; 8 x 8 rows of 500 22, 34 | 27, 32, of 2000 33, 63 | 28, 33).
    const int64_t rows = (int64_t)ny * nz;
    if (nx > 32 && nx <= 4096 && 8 * rows >= nx) {
        const int row = (nx + 2 * radius) * (int)sizeof(float), warps = std::min(8, 48 * 1024 / row);
        k_gauss_row_mask<<<grid_for(rows * 256 / warps), warps * 32, warps * row, s>>>(gv, M, g);
        return cudaGetLastError();
    }
    if ((e = gauss_line(gv, tmp, 1, nx, 1, rows, nx, g, s))) return e;
    k_mask<true><<<grid_for(n), 256, 0, s>>>(tmp, gv, M);
    return cudaGetLastError();
}

cudaError_t efm_util_chain_rule(float *gl, float *gm, float *gr, const float *vp, const float *vs,
                                const float *rho, int64_t n, cudaStream_t s) {
    k_chain<<<grid_for(n), 256, 0, s>>>(gl, gm, gr, vp, vs, rho, n);
    return cudaGetLastError();
}

cudaError_t efm_util_adam(int count, float *const *p, const float *const *g, float *const *m, float *const *v,
                          const int64_t *n, double lr, double beta1, double beta2, double eps, double c1, double c2,
                          cudaStream_t s) {
    for (int k0 = 0; k0 < count; k0 += ADAM_MAX) {
        AdamArgs A = {};
        const int k1 = std::min(count - k0, ADAM_MAX);
        int64_t most = 0;
        for (int k = 0; k < k1; ++k) {
            A.p[k] = p[k0 + k];
            A.g[k] = g[k0 + k];
            A.m[k] = m[k0 + k];
            A.v[k] = v[k0 + k];
            A.n[k] = n[k0 + k];
            most = std::max(most, A.n[k]);
        }
        A.lr = (float)lr;
        A.beta1 = (float)beta1;
        A.beta2 = (float)beta2;
        A.alpha1 = (float)(1.0 - beta1);
        A.alpha2 = (float)(1.0 - beta2);
        A.eps = (float)eps;
        A.r1 = (float)(1.0 / c1);
        A.r2 = (float)(1.0 / c2);
        k_adam<<<dim3(grid_for(most), k1), 256, 0, s>>>(A);
    }
    return cudaGetLastError();
}
