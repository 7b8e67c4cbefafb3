// Plane-streaming stress / velocity / imaging kernels: a TMA producer warp feeding shared-memory rings.
//
// A block takes chunks -- a tile of tw x th (x, z) cells over a run of y planes -- from the
// launch's counter.  Its producer warp issues, per plane, a TMA tile load of every field the
// half-step reads: fields whose x / y / z neighbours enter (boxes with just the neighbour columns
// / rows that are used) and cell-only fields.  Slot q of the ring holds the neighbour fields of
// plane p + 1 and the cell fields of plane p, so computing plane p needs slot q and the neighbour
// part of slot q - 1; what the stencil reads of plane p - 1 is this thread's own column and stays
// in registers.  A ring of D + 1 slots keeps D - 1 planes in flight while one is computed, and
// the loads of the next chunk follow the last plane of the current one without a gap.  A chunk's
// first slot brings the neighbour fields of its first plane and, in the unused cell part, the
// own-column values of the plane before.
//
// Each consumer thread computes a pair of x-neighbours: operands come as 8-byte shared-memory
// loads (the x neighbour inside the pair is already in a register), results go straight to global
// memory as 8-byte stores, so the slot is free as soon as it has been read, and addresses, tests
// and waits are shared by two cells.  Consumer warps never wait for one another: each waits for
// the plane's full barrier and arrives on its empty barrier.  Before, one thread computed two
// separate cells of a 64 x 8 tile with a block barrier per plane, 4-byte loads and TMA stores out
// of the ring.  The imaging runs the same way: as a kernel of its own with another amount of shared
// memory it also left the next stress launch, which starts while it drains, with its smaller L1
// (256 x 256 x 128 gradient step: 491 us, 465 now).
//
// us per launch, before (two cells per thread) and now: 128 x 128 x 96 forward stress 23.4, 22.0,
// velocity 23.2, 23.1; 256 x 256 x 128: 114.6, 102.3 and 115.5, 94.4 (the DRAM rate: a pass moves
// 15 volumes and the memory variables), adjoint stress + rebuild velocity 193.7, 164.7, rebuild
// stress + adjoint velocity 190.2, 167.0, imaging 127.1, 118.2; 64 x 64 x 64 forward 10.1, 6.7 and
// 12.0, 7.5 (launch and first loads).  Small grids are bound by issue and latency: about 260
// instructions per warp and plane of pairs without memory variables, 16 warps per SM.
//
// Sources are looked up once per chunk, receivers per plane from a map built on the host.
// Arithmetic, guards, CPML, sources, receivers, strips and MT strain follow efm_stencil.cu
// (kernel_Tau :59-128, kernel_Vx_Vy_Vz :133-188, kernel_Gradients_* :191-294 of
// mainPropElastic3D_MT.py); harmonic means
// use the hardware reciprocal (relative error ~1 ulp).
#include "efm_internal.cuh"
#include "efm_stream.cuh"
#include "efm_tma.cuh"

// A launch: the chunks of a stress pass (table s), then of a velocity or imaging pass (table v).
struct EfmStream {
    const EfmInst *s, *v;
    int ns, nv, cs, cv;  // table entries still active, and their chunks
    int it;
    int *counter;
    uint32_t lim;
    unsigned int *err;
};

namespace {

__device__ __forceinline__ float frcp(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// a x + b y, rounded as fma(b, y, a x): written out where a compiler is free to fuse either product,
// so that every instantiation of a plane's update rounds alike.
__device__ __forceinline__ float two_products(float a, float x, float b, float y) {
    return __fmaf_rn(b, y, __fmul_rn(a, x));
}

// The instantiations of a plane's update, picked per plane by a warp-uniform test: no memory
// variables (0), those of the x slabs (1: every plane of the tiles at the x faces), every family
// and, in the velocity, receivers (2: few planes, and the registers of all three families).
template <int V>
struct Tag {
    static constexpr int value = V;
};

constexpr int VX = 2;  // cells per thread along x

struct QV {
    float v[VX];
};

__device__ __forceinline__ QV ldv(const unsigned char *f, int i) {
    const float2 a = *reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(f) + i);
    return QV{{a.x, a.y}};
}

__device__ __forceinline__ float2 ld2(const unsigned char *f, int i) {
    return *reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(f) + i);
}

__device__ __forceinline__ float ld1(const unsigned char *f, int i) {
    return reinterpret_cast<const float *>(f)[i];
}

// two consecutive floats (8-byte aligned) of memory this launch also writes
__device__ __forceinline__ QV ldgv(const float *p) {
    QV a;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(a.v[0]), "=f"(a.v[1]) : "l"(p) : "memory");
    return a;
}

__device__ __forceinline__ void stv(float *p, const QV &a) {
    asm volatile("st.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a.v[0]), "f"(a.v[1]) : "memory");
}

__device__ __forceinline__ void st1(float *p, float a) {
    asm volatile("st.global.f32 [%0], %1;" ::"l"(p), "f"(a) : "memory");
}

// The memory variables of a pair's cells (one family, three components and a pad each) in one access:
// 32 bytes, on 32 bytes since x, nx and the slabs' offsets are even.  (By cell, every store filled
// half of each lane's sector, and with values read where they are used the second cell's load
// waited behind the first one's store; forward velocity 128 x 128 x 96, 30 layers: 38.7 us, 35.0 now.)
__device__ __forceinline__ void ld_psi(const float4 *p, float (&a)[3], float (&b)[3]) {
    float pad0, pad1;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(pad0), "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(pad1)
                 : "l"(p)
                 : "memory");
}

__device__ __forceinline__ void st_psi(float4 *p, const float (&a)[3], const float (&b)[3]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %7, %4, %5, %6, %7};" ::"l"(p), "f"(a[0]), "f"(a[1]), "f"(a[2]),
                 "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(0.f)
                 : "memory");
}

__device__ __forceinline__ void st_psi1(float4 *p, const float (&a)[3]) {
    asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(0.f)
                 : "memory");
}

// ------------------------------------------------------------------------------- the ring
// Position in the ring: slot q (of D + 1) and the one before it, its barrier (q mod D) and phase.
template <int D>
struct Cursor {
    int cs = 0, hs = 0, hp = D;
    uint32_t ph = 0;
    __device__ __forceinline__ void next() {
        hp = hs;
        hs = hs == D ? 0 : hs + 1;
        if (++cs == D) {
            cs = 0;
            ph ^= 1u;
        }
    }
};

// One chunk: a tile over the planes [ys, ye) of a stress (0), velocity (1) or imaging (2) pass; -1: no more.
struct Chunk {
    int type, x0, z0, ys, ye, col, tw, th;
};

// The block's shared memory: D + 1 ring slots, then this.  The barriers: a slot's loads have
// arrived (full), every consumer warp has read it (empty), a chunk's description is in place
// (ready: the consumers set up a chunk while its first loads travel).  Two descriptions with their
// table entries (three for the deeper ring): a chunk has at least two slots, so the producer, with
// the first slot of chunk c in hand -- the consumers have left the slot D before it -- knows that
// they have left chunk c - N.
template <int D>
struct Block {
    static constexpr int N = D / 2 + 1;
    uint64_t full[D], empty[D], ready[N];
    Chunk chunk[N];
    alignas(16) EfmInst inst[N];
    int abort;
    uint32_t lim;       // polls per wait (0: the default bound)
    unsigned int *err;  // the context's error word
    static __device__ __forceinline__ int next(int i) { return i == N - 1 ? 0 : i + 1; }
};

template <int D, int SLOT>
__device__ __forceinline__ Block<D> &block_state() {
    extern __shared__ __align__(1024) unsigned char smem[];
    return *reinterpret_cast<Block<D> *>(smem + (D + 1) * SLOT);
}

template <int SLOT>
__device__ __forceinline__ unsigned char *ring_slot(int i) {
    extern __shared__ __align__(1024) unsigned char smem[];
    return smem + i * SLOT;
}

template <int D>
__device__ __forceinline__ void give_up(Block<D> &B) {
    *(volatile int *)&B.abort = 1;
    if (B.err) atomicOr(B.err, EFM_ERR_FLAG_TIMEOUT);
}

// Wait (bounded) that also gives up once another warp of the block has given up.
template <int D>
__device__ __forceinline__ bool ring_wait(Block<D> &B, uint64_t *bar, uint32_t parity, uint32_t lim) {
    if (lim == 0) {
        for (uint32_t i = 0; i < EFM_WAIT_LIMIT; ++i) {
            if (efm_mbar_try_wait(bar, parity)) return true;
            if ((i & 255u) == 255u && *(volatile int *)&B.abort) return false;
        }
    } else {
        for (uint32_t i = 0; i < lim; ++i)
            if (efm_mbar_test_wait(bar, parity)) return true;
    }
    give_up(B);
    return false;
}

// What a consumer warp walks the ring with.
template <int D, int SLOT>
struct Ctx {
    Block<D> &B;
    uint32_t lim;
    bool lane0;
    Cursor<D> cur;
    static constexpr int START = D << 8;  // slot 0, before it slot D
    __device__ __forceinline__ Ctx(int packed)
        : B(block_state<D, SLOT>()), lim(B.lim), lane0((threadIdx.x & 31) == 0) {
        cur.cs = packed & 15;
        cur.hs = (packed >> 4) & 15;
        cur.hp = (packed >> 8) & 15;
        cur.ph = (packed >> 12) & 1;
    }
    __device__ __forceinline__ int packed() const {
        return cur.cs | cur.hs << 4 | cur.hp << 8 | (int)cur.ph << 12;
    }
    __device__ __forceinline__ const unsigned char *slot() const { return ring_slot<SLOT>(cur.hs); }
    __device__ __forceinline__ const unsigned char *prev() const { return ring_slot<SLOT>(cur.hp); }
    __device__ __forceinline__ bool wait() { return ring_wait(B, &B.full[cur.cs], cur.ph, lim); }
    // this warp is done with the slot
    __device__ __forceinline__ void release() {
        __syncwarp();
        if (lane0) efm_mbar_arrive(&B.empty[cur.cs]);
        cur.next();
    }
};

// ------------------------------------------------------------- per-thread state of a chunk
// The thread's pair (x, x + 1) at z: its place in the boxes of a plane (i0: rows of tw + 4, k0:
// rows of tw) and what applies to its cells.
enum {
    F_IN = 3,           // bit v: the stencil updates cell v (planes permitting)
    F_PX = 3 << 4,      // ... and it has x memory variables
    F_ACT = 3 << 8,     // cell v lies in the grid and the pair in the tile
    F_PZ = 1 << 12,     // the updated cells have z memory variables
    F_WX = 1 << 13,     // some lane of the warp has x memory variables
    F_WZ = 1 << 14,     // ... z memory variables
    F_PART = 1 << 15    // ... updates some but not all of its cells
};

struct Pair {
    int x, z;
    int i0, k0, hp, tw;  // hp = tw + 4
    int fl;
    __device__ __forceinline__ bool in(int v) const { return (fl >> v) & 1; }
    __device__ __forceinline__ bool px(int v) const { return (fl >> (4 + v)) & 1; }
    __device__ __forceinline__ bool act(int v) const { return (fl >> (8 + v)) & 1; }
    __device__ __forceinline__ bool any_in() const { return fl & F_IN; }
};

template <bool BOX>
__device__ __forceinline__ Pair make_pair(const EfmInst &I, const Chunk &T) {
    Pair p;
    const int nx = I.nx, nz = I.nz, W = I.W, per_row = T.tw / VX;
    int r = threadIdx.x / per_row;
    int c = VX * ((int)threadIdx.x - r * per_row);
    const bool mine = r < T.th;
    if (!mine) r = c = 0;
    p.tw = T.tw;
    p.hp = T.tw + 4;
    p.x = T.x0 + c;
    p.z = T.z0 + r;
    p.i0 = r * p.hp + c;
    p.k0 = r * T.tw + c;
    const bool row = mine && p.z < nz;
    const bool zin = row && p.z >= EFM_HS && p.z < nz - EFM_HS && !(BOX && p.z >= nz - W);
    p.fl = 0;
#pragma unroll
    for (int v = 0; v < VX; ++v) {
        const int x = p.x + v;
        const bool slab = x < W || x >= nx - W;
        const bool in = zin && x >= EFM_HS && x < nx - EFM_HS && !(BOX && slab);
        p.fl |= (in ? 1 << v : 0) | (in && slab ? 16 << v : 0) | (row && x < nx ? 256 << v : 0);
    }
    if ((p.fl & F_IN) && p.z >= nz - W) p.fl |= F_PZ;
    if (__any_sync(0xffffffffu, p.fl & F_PX)) p.fl |= F_WX;
    if (__any_sync(0xffffffffu, p.fl & F_PZ)) p.fl |= F_WZ;
    if (__any_sync(0xffffffffu, (p.fl & F_IN) != 0 && (p.fl & F_IN) != F_IN)) p.fl |= F_PART;
    return p;
}

// CPML memory variables of the pair: a 16-byte vector (three components) per cell, group 0 the
// stress pass's, 1 the velocity pass's of each slab family.  The first slab's base and 32-bit
// offsets address all three families (one allocation; the host checks the range).  x and z
// follow the planes; y is looked up on the planes of the y slabs.
struct Psi {
    float4 *base;
    int x, z, sx, sz;
    float ax[VX], bx[VX], az, bz;
};

__device__ __forceinline__ Psi psi_at(const EfmInst &I, const Pair &p, int group, int y) {
    const int nx = I.nx, ny = I.ny, nz = I.nz, W = I.W;
    Psi P;
    P.base = reinterpret_cast<float4 *>(I.psi_x);
    P.sx = nz * 2 * W;
    P.sz = W * nx;
    P.x = ((group * ny + y) * nz + p.z) * 2 * W + (p.x + VX - 1 < nx - W ? p.x : p.x - (nx - 2 * W));
    P.z = 4 * W * ny * nz + 4 * W * nz * nx + ((group * ny + y) * W + p.z - (nz - W)) * nx + p.x;
#pragma unroll
    for (int v = 0; v < VX; ++v) {
        P.ax[v] = p.px(v) ? I.cpml[p.x + v] : 0.f;
        P.bx[v] = p.px(v) ? I.cpml[nx + p.x + v] : 0.f;
    }
    P.az = p.fl & F_PZ ? I.cpml[2 * (nx + ny) + p.z] : 0.f;
    P.bz = p.fl & F_PZ ? I.cpml[2 * (nx + ny) + nz + p.z] : 0.f;
    return P;
}

__device__ __forceinline__ int psi_y(const EfmInst &I, const Pair &p, int group, int y) {
    const int nx = I.nx, ny = I.ny, nz = I.nz, W = I.W;
    return 4 * W * ny * nz + ((group * 2 * W + (y < W ? y : y - (ny - 2 * W))) * nz + p.z) * nx + p.x;
}

// Pull the next plane's memory variables into L1 (no register, no wait).
__device__ __forceinline__ void prefetch2(const float4 *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

__device__ __forceinline__ void prefetch_psi(const Pair &p, const Psi &P) {
    if (p.fl & F_PX) prefetch2(P.base + (P.x + P.sx));
    if (p.fl & F_PZ) prefetch2(P.base + (P.z + P.sz));
}

// ... and a chunk's first plane's.
__device__ __forceinline__ void prefetch_first(const EfmInst &I, const Pair &p, const Psi &P, int group, int y) {
    if (p.fl & F_PX) prefetch2(P.base + P.x);
    if (p.fl & F_PZ) prefetch2(P.base + P.z);
    if ((p.fl & F_IN) && (y < I.W || y >= I.ny - I.W)) prefetch2(P.base + psi_y(I, p, group, y));
}

// The memory variables of the pair's cells, [cell][component] by family, zero where the pair has none
// (a vector next to a slab cell's may be another cell's: it is read and not used).  Each family
// sits behind a test that is uniform over the warp (x, z) or the block (y).  Requested before the
// plane's wait, so the wait covers their latency; with YZ false only the x family, and the others
// (12 registers per pair that would spill beside the plane's operands) are read where they are
// used, from L1.  YZ is for the stress passes, where it does not spill (adjoint stress 128 x 128 x 96:
// 28.3 us, 29.3 without); in the velocity passes it does (forward velocity at that size: 31.6 us,
// 29.6 without; 256 x 256 x 128: 102.8 and 98.6; the pair with the adjoint velocity, whole
// gradient steps of 100 x 100 x 100 with 20 layers: 109.5 us and 105.6).
template <int PML, bool YZ>
struct PsiOld {
    static constexpr bool EARLY = YZ && PML == 2;
    float x[VX][3], y[EARLY ? VX : 1][3], z[EARLY ? VX : 1][3];
    __device__ __forceinline__ void load(const Pair &p, const Psi &P, bool ypml, int py) {
#pragma unroll
        for (int v = 0; v < VX; ++v) x[v][0] = x[v][1] = x[v][2] = 0.f;
        if (p.fl & F_PX) ld_psi(P.base + P.x, x[0], x[1]);
        if (EARLY) {
#pragma unroll
            for (int v = 0; v < VX; ++v) y[v][0] = y[v][1] = y[v][2] = z[v][0] = z[v][1] = z[v][2] = 0.f;
            if (ypml && (p.fl & F_IN)) ld_psi(P.base + py, y[0], y[1]);
            if (p.fl & F_PZ) ld_psi(P.base + P.z, z[0], z[1]);
        }
    }
    // where they are used: o = what was requested early, or read now for pairs that have the family
    __device__ __forceinline__ void get_y(bool c, const float4 *q, float (&o)[VX][3]) const { get(c, q, y, o); }
    __device__ __forceinline__ void get_z(bool c, const float4 *q, float (&o)[VX][3]) const { get(c, q, z, o); }
    static __device__ __forceinline__ void get(bool c, const float4 *q, const float (&early)[EARLY ? VX : 1][3],
                                               float (&o)[VX][3]) {
#pragma unroll
        for (int v = 0; v < VX; ++v)
#pragma unroll
            for (int k = 0; k < 3; ++k) o[v][k] = EARLY ? early[EARLY ? v : 0][k] : 0.f;
        if (!EARLY && c) ld_psi(q, o[0], o[1]);
    }
};

// psi <- b psi + a d for one cell's three components of a family; cells without them (c false) get zeros.
__device__ __forceinline__ void psi_step(bool c, float (&o)[3], float a, float b, float d0, float d1, float d2) {
    const float n0 = b * o[0] + a * d0, n1 = b * o[1] + a * d1, n2 = b * o[2] + a * d2;
    o[0] = c ? n0 : 0.f;
    o[1] = c ? n1 : 0.f;
    o[2] = c ? n2 : 0.f;
}

// The x slabs' new values of the pair (an odd slab width leaves pairs with one such cell).
__device__ __forceinline__ void st_psi_x(const Pair &p, float4 *q, const float (&o)[VX][3]) {
    if (p.px(0) && p.px(1))
        st_psi(q, o[0], o[1]);
    else if (p.px(0))
        st_psi1(q, o[0]);
    else if (p.px(1))
        st_psi1(q + 1, o[1]);
}

// ------------------------------------------------------------------------------ stress
// Neighbour fields: vx (x0-4, z0), vy (x0, z0), vz (x0, z0-1), 1/mu (x0, z0), each tw+4 columns
// and th+1 rows; cell fields: lambda txx tyy tzz txy txz tyz.  First slot's cell part: vy of the
// plane before the chunk.
// New stress of the pair on plane y.  h: neighbour fields of plane y, hn: of plane y + 1, cc: the
// cell fields; vym: vy of plane y - 1 (in), of plane y (out).
template <int PASS, int NT, int PML>
__device__ __forceinline__ void stress_pair(const EfmInst &I, const unsigned char *h, const unsigned char *hn,
                                            const unsigned char *cc, int it, int y, const Pair &p, bool has_src,
                                            float k, const Psi &P, bool ypml, int py, float ay, float by,
                                            PsiOld<PML, true> &O, QV &vym, float *t0, int64_t N) {
    constexpr int XZ = efm_slot_xz(NT), CF = efm_slot_c(NT);
    const int i0 = p.i0, i1 = p.i0 + p.hp;
    const QV vx = ldv(h, i0 + 4), vxz = ldv(h, i1 + 4), vxj = ldv(hn, i0 + 4);
    const float vxm = ld1(h, i0 + 3);
    const QV vy = ldv(h + XZ, i0), vyz = ldv(h + XZ, i1);
    const float vyx = ld1(h + XZ, i0 + VX);
    const QV vz = ldv(h + 2 * XZ, i1), vzm = ldv(h + 2 * XZ, i0), vzj = ldv(hn + 2 * XZ, i1);
    const float vzx = ld1(h + 2 * XZ, i1 + VX);
    const QV m0 = ldv(h + 3 * XZ, i0), mk = ldv(h + 3 * XZ, i1), mj = ldv(hn + 3 * XZ, i0);
    const QV mjk = ldv(hn + 3 * XZ, i1);
    const float mi = ld1(h + 3 * XZ, i0 + VX), mik = ld1(h + 3 * XZ, i1 + VX), mij = ld1(hn + 3 * XZ, i0 + VX);
    const QV lam4 = ldv(cc, p.k0);
    QV t[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) t[q] = ldv(cc + (1 + q) * CF, p.k0);
    QV o[6];
    float oy[VX][3], oz[VX][3];
    const bool wy = PML == 2 && ypml && p.any_in(), wz = PML == 2 && (p.fl & F_PZ);
#pragma unroll
    for (int v = 0; v < VX; ++v) {
        const float vxc = vx.v[v], vyc = vy.v[v], vzc = vz.v[v];
        const float dvx_dx = vxc - (v ? vx.v[v - 1] : vxm);
        const float dvy_dy = vyc - vym.v[v];
        const float dvz_dz = vzc - vzm.v[v];
        const float dvx_dz = vxz.v[v] - vxc;
        const float dvx_dy = vxj.v[v] - vxc;
        const float dvy_dx = (v < VX - 1 ? vy.v[v + 1] : vyx) - vyc;
        const float dvy_dz = vyz.v[v] - vyc;
        const float dvz_dx = (v < VX - 1 ? vz.v[v + 1] : vzx) - vzc;
        const float dvz_dy = vzj.v[v] - vzc;
        // harmonic 4-point averages of mu from the precomputed 1/mu (:80-89)
        const float r0 = m0.v[v], ri = v < VX - 1 ? m0.v[v + 1] : mi, rk = mk.v[v];
        const float rik = v < VX - 1 ? mk.v[v + 1] : mik;
        const float rj = mj.v[v], rjk = mjk.v[v], rij = v < VX - 1 ? mj.v[v + 1] : mij;
        const float mu0 = frcp(r0);
        const float mu_xz = 4.f * frcp(r0 + ri + rk + rik);
        const float mu_xy = 4.f * frcp(r0 + ri + rj + rij);
        const float mu_yz = 4.f * frcp(r0 + rj + rk + rjk);
        const float lam = lam4.v[v];
        const float l2m = lam + 2.f * mu0;
        float txx, tyy, tzz, txy, txz, tyz;
        if (PML == 0) {  // (the sums below without their zero terms)
            txx = t[0].v[v] + k * two_products(l2m, dvx_dx, lam, (dvy_dy + dvz_dz));
            tyy = t[1].v[v] + k * two_products(l2m, dvy_dy, lam, (dvx_dx + dvz_dz));
            tzz = t[2].v[v] + k * two_products(l2m, dvz_dz, lam, (dvx_dx + dvy_dy));
            txy = t[3].v[v] + k * mu_xy * (dvx_dy + dvy_dx);
            txz = t[4].v[v] + k * mu_xz * (dvx_dz + dvz_dx);
            tyz = t[5].v[v] + k * mu_yz * (dvy_dz + dvz_dy);
        } else {
            float pvx_x = 0.f, pvy_x = 0.f, pvz_x = 0.f, pvy_y = 0.f, pvx_y = 0.f, pvz_y = 0.f;
            float pvz_z = 0.f, pvx_z = 0.f, pvy_z = 0.f;
            if (PML == 1 || (p.fl & F_WX)) {
                psi_step(p.px(v), O.x[v], P.ax[v], P.bx[v], dvx_dx, dvy_dx, dvz_dx);
                pvx_x = O.x[v][0];
                pvy_x = O.x[v][1];
                pvz_x = O.x[v][2];
                if (v == VX - 1) st_psi_x(p, P.base + P.x, O.x);
            }
            if (PML == 2 && ypml) {
                if (v == 0) O.get_y(wy, P.base + py, oy);
                psi_step(wy, oy[v], ay, by, dvy_dy, dvx_dy, dvz_dy);
                pvy_y = oy[v][0];
                pvx_y = oy[v][1];
                pvz_y = oy[v][2];
                if (v == VX - 1 && wy) st_psi(P.base + py, oy[0], oy[1]);
            }
            if (PML == 2 && (p.fl & F_WZ)) {
                if (v == 0) O.get_z(wz, P.base + P.z, oz);
                psi_step(wz, oz[v], P.az, P.bz, dvz_dz, dvx_dz, dvy_dz);
                pvz_z = oz[v][0];
                pvx_z = oz[v][1];
                pvy_z = oz[v][2];
                if (v == VX - 1 && wz) st_psi(P.base + P.z, oz[0], oz[1]);
            }
            txx = t[0].v[v] + k * two_products(l2m, (dvx_dx + pvx_x), lam, (dvy_dy + dvz_dz + pvy_y + pvz_z));
            tyy = t[1].v[v] + k * two_products(l2m, (dvy_dy + pvy_y), lam, (dvx_dx + dvz_dz + pvx_x + pvz_z));
            tzz = t[2].v[v] + k * two_products(l2m, (dvz_dz + pvz_z), lam, (dvx_dx + dvy_dy + pvx_x + pvy_y));
            txy = t[3].v[v] + k * mu_xy * ((dvx_dy + pvx_y) + (dvy_dx + pvy_x));
            txz = t[4].v[v] + k * mu_xz * ((dvx_dz + pvx_z) + (dvz_dx + pvz_x));
            tyz = t[5].v[v] + k * mu_yz * ((dvy_dz + pvy_z) + (dvz_dy + pvz_y));
        }
        o[0].v[v] = txx;
        o[1].v[v] = tyy;
        o[2].v[v] = tzz;
        o[3].v[v] = txy;
        o[4].v[v] = txz;
        o[5].v[v] = tyz;
    }
    // few chunks hold a source: its cell's operands are read again, instead of keeping them for all
    if (has_src) {
#pragma unroll
        for (int v = 0; v < VX; ++v) {
            if (!p.in(v)) continue;
            for (int s = 0; s < I.nsrc; ++s) {
                if (p.x + v != I.sx[s] || y != I.sy[s] || p.z != I.sz[s]) continue;
                if (PASS != EFM_ADJ) {
                    const float w = I.wav[PASS == EFM_FWD ? it : I.nt - 1 - it];
                    const float sg = PASS == EFM_FWD ? 1.f : -1.f;
#pragma unroll
                    for (int q = 0; q < 6; ++q) o[q].v[v] = __fadd_rn(o[q].v[v], sg * __fmul_rn(I.mt[s][q], w));
                } else if (I.mtg != nullptr) {
                    const unsigned char *r = h + 3 * XZ, *rn = hn + 3 * XZ;
                    const float r0 = ld1(r, i0 + v), ri = ld1(r, i0 + v + 1), rk = ld1(r, i1 + v);
                    const float rik = ld1(r, i1 + v + 1), rj = ld1(rn, i0 + v), rjk = ld1(rn, i1 + v);
                    const float rij = ld1(rn, i0 + v + 1), mu0 = frcp(r0), lam = ld1(cc, p.k0 + v);
                    const float txx = o[0].v[v], tyy = o[1].v[v], tzz = o[2].v[v];
                    const float w = I.wav[I.nt - 1 - it];
                    const float f = __frcp_rn(2.f * mu0 * (3.f * lam + 2.f * mu0));
                    const float lpm2 = 2.f * (lam + mu0);
                    // one thread adds to these per step: a reduction in L2 need not wait for the old value
                    double *g = I.mtg + 6 * s;
                    atomicAdd(g + 0, (double)(w * (f * (lpm2 * txx - lam * tyy - lam * tzz))));
                    atomicAdd(g + 1, (double)(w * (f * (lpm2 * tyy - lam * txx - lam * tzz))));
                    atomicAdd(g + 2, (double)(w * (f * (lpm2 * tzz - lam * txx - lam * tyy))));
                    atomicAdd(g + 3, (double)(w * (o[3].v[v] * __frcp_rn(4.f * frcp(r0 + ri + rj + rij)))));
                    atomicAdd(g + 4, (double)(w * (o[4].v[v] * __frcp_rn(4.f * frcp(r0 + ri + rk + rik)))));
                    atomicAdd(g + 5, (double)(w * (o[5].v[v] * __frcp_rn(4.f * frcp(r0 + rj + rk + rjk)))));
                }
            }
        }
    }
    vym = vy;
    if (p.fl & F_PART) {  // a pair at the edge of the updated cells keeps the others' values
#pragma unroll
        for (int v = 0; v < VX; ++v)
#pragma unroll
            for (int q = 0; q < 6; ++q) o[q].v[v] = p.in(v) ? o[q].v[v] : t[q].v[v];
    }
    if (p.any_in()) {
#pragma unroll
        for (int q = 0; q < 6; ++q) stv(t0 + q * N, o[q]);
    }
}

template <int PASS, int NT, int D, int SLOT>
__device__ __forceinline__ int stress_chunk(int packed, int ib, int it) {
    Ctx<D, SLOT> X(packed);
    const EfmInst &I = X.B.inst[ib];
    const Chunk &T = X.B.chunk[ib];
    constexpr int HB = efm_halo_s(NT);
    const Pair p = make_pair<PASS == EFM_REV>(I, T);
    const int ylo_in = I.W, yhi_in = I.ny - I.W, plane = I.nz * I.pitch;
    const float k = I.k;
    bool has_src = false;
    for (int s = 0; s < I.nsrc; ++s)
        has_src = has_src || (I.sx[s] >= T.x0 && I.sx[s] < T.x0 + T.tw && I.sz[s] >= T.z0 &&
                              I.sz[s] < T.z0 + T.th && I.sy[s] >= T.ys && I.sy[s] < T.ye);
    const int64_t N = I.vol;
    float *t0 = I.f.t[0] + (int64_t)T.ys * plane + p.z * I.pitch + p.x;
    Psi P = psi_at(I, p, 0, T.ys);
    const int ye = T.ye;
    efm_pdl_wait();
    if (PASS != EFM_REV && T.ys >= EFM_HS) prefetch_first(I, p, P, 0, T.ys);
    if (!__all_sync(0xffffffffu, X.wait())) return -1;
    QV vym = ldv(X.slot() + HB, p.k0);
    X.release();
    for (int j = T.ys; j < ye; ++j, t0 += plane, P.x += P.sx, P.z += P.sz) {
        const bool plane_in = j >= EFM_HS && j < ylo_in + yhi_in - EFM_HS;
        const bool ypml = PASS != EFM_REV && (j < ylo_in || j >= yhi_in);
        auto update = [&](auto tag) -> bool {
            constexpr int PML = decltype(tag)::value;
            PsiOld<PML, true> O;
            float ay = 0.f, by = 0.f;
            int py = 0;
            if (PML) {
                if (PML == 2 && ypml) {
                    py = psi_y(I, p, 0, j);
                    ay = I.cpml[2 * I.nx + j];
                    by = I.cpml[2 * I.nx + I.ny + j];
                }
                O.load(p, P, ypml, py);
                if (j + 1 < ye) {
                    prefetch_psi(p, P);
                    if (PML == 2 && ypml && (p.fl & F_IN) && (j + 1 < ylo_in || j >= yhi_in))
                        prefetch2(P.base + (py + I.nz * I.nx));
                }
            }
            if (!X.wait()) return false;
            stress_pair<PASS, NT, PML>(I, X.prev(), X.slot(), X.slot() + HB, it, j, p, has_src, k, P, ypml, py, ay, by,
                                       O, vym, t0, N);
            return true;
        };
        bool mine;
        if (!plane_in) {  // (a region that reaches past the updated planes)
            mine = X.wait();
            vym = ldv(X.prev() + efm_slot_xz(NT), p.i0);
        } else {
            mine = PASS != EFM_REV && (ypml || (p.fl & F_WZ)) ? update(Tag<2>{})
                   : PASS != EFM_REV && (p.fl & F_WX)         ? update(Tag<1>{})
                                                              : update(Tag<0>{});
        }
        if (!__all_sync(0xffffffffu, mine)) return -1;
        X.release();
    }
    return X.packed();
}

// ---------------------------------------------------------------------------- velocity
// Boundary-strip slot of a box cell (xr, yr, zr from the box's corner) in one of its families
// (efm_strip_slots_v): 0 the x faces, 1 the y faces, 2 the z faces.
__device__ __forceinline__ int strip_slot(int bx, int by, int bz, int xr, int yr, int zr, int family) {
    if (family == 0) return ((xr < 2 ? xr : 4 + xr - bx) * by + yr) * bz + zr;
    if (family == 1) return 4 * by * bz + ((yr < 2 ? yr : 4 + yr - by) * bz + zr) * bx + xr;
    return 4 * by * bz + 4 * bz * bx + ((zr < 2 ? zr : 4 + zr - bz) * by + yr) * bx + xr;
}

// Neighbour fields: txx (x0, z0; tw+4 columns), tzz (th+1 rows), txy (x0-4; tw+4), txz (x0-4, z0-1;
// both), tyz (z0-1; th+1), 1/rho (x0, z0; both), tyy (cells); cell fields: vx vy vz.  First slot's
// cell part: txy and tyz of the plane before the chunk.
template <int NT>
struct VOff {
    static constexpr int X = efm_slot_x(NT), Z = efm_slot_z(NT), XZ = efm_slot_xz(NT), CF = efm_slot_c(NT);
    static constexpr int txx = 0, tzz = X, txy = X + Z, txz = 2 * X + Z, tyz = 2 * X + Z + XZ,
                         bu = 2 * X + 2 * Z + XZ, tyy = 2 * X + 2 * Z + 2 * XZ;
};

// The stress differences' operands and the buoyancies of the pair on one plane.
struct VelIn {
    QV txx, tzz, tzzk, txy, txz, txzk, tyz, tyzk, tyy, tyyj, b0, bk, bj;
    float txxi, txym, txzm, bi;
};

template <int NT>
__device__ __forceinline__ VelIn velocity_in(const Pair &p, const unsigned char *h, const unsigned char *hn) {
    using O = VOff<NT>;
    const int i0 = p.i0, i1 = p.i0 + p.hp, k0 = p.k0, k1 = p.k0 + p.tw;
    VelIn a;
    a.txx = ldv(h + O::txx, i0);
    a.txxi = ld1(h + O::txx, i0 + VX);
    a.tzz = ldv(h + O::tzz, k0);
    a.tzzk = ldv(h + O::tzz, k1);
    a.txy = ldv(h + O::txy, i0 + 4);
    a.txym = ld1(h + O::txy, i0 + 3);
    a.txz = ldv(h + O::txz, i1 + 4);
    a.txzm = ld1(h + O::txz, i1 + 3);
    a.txzk = ldv(h + O::txz, i0 + 4);
    a.tyz = ldv(h + O::tyz, k1);
    a.tyzk = ldv(h + O::tyz, k0);
    a.b0 = ldv(h + O::bu, i0);
    a.bi = ld1(h + O::bu, i0 + VX);
    a.bk = ldv(h + O::bu, i1);
    a.bj = ldv(hn + O::bu, i0);
    a.tyy = ldv(h + O::tyy, k0);
    a.tyyj = ldv(hn + O::tyy, k0);
    return a;
}

template <int PASS, int NT, int D, int SLOT, bool ILLUM>
__device__ __forceinline__ int velocity_chunk(int packed, int ib, int it) {
    using OF = VOff<NT>;
    Ctx<D, SLOT> X(packed);
    const EfmInst &I = X.B.inst[ib];
    const Chunk &T = X.B.chunk[ib];
    constexpr int HB = efm_halo_v(NT);
    const Pair p = make_pair<false>(I, T);
    const int ylo_in = I.W, yhi_in = I.ny - I.W, plane = I.nz * I.pitch;
    const float k = I.k;
    // strips: which cells lie in the box (bit v), next to an x face (4 + v) or a z face (8)
    int sf = 0;
    if (PASS == EFM_REV || (PASS == EFM_FWD && I.border != nullptr)) {
        const int bx = I.nx - 2 * I.W, bz = I.nz - I.W - 2, zr = p.z - 2;
#pragma unroll
        for (int v = 0; v < VX; ++v) {
            const int xr = p.x + v - I.W;
            if (!p.act(v) || xr < 0 || xr >= bx || zr < 0 || zr >= bz) continue;
            sf |= 1 << v;
            if (xr < 2 || xr >= bx - 2) sf |= 16 << v;
            if (zr < 2 || zr >= bz - 2) sf |= 256;
        }
    }
    const int64_t N = I.vol;
    float *v0 = I.f.vo[0] + (int64_t)T.ys * plane + p.z * I.pitch + p.x;
    const uint8_t *const recs = PASS == EFM_REV ? nullptr : I.rec_col + (int64_t)T.col * I.ny;
    Psi P = psi_at(I, p, 1, T.ys);
    uint8_t rec_now = PASS == EFM_REV ? 0 : __ldg(recs + T.ys);
    const int ye = T.ye;
    efm_pdl_wait();
    if (PASS != EFM_REV && T.ys >= EFM_HS) prefetch_first(I, p, P, 1, T.ys);
    if (!__all_sync(0xffffffffu, X.wait())) return -1;
    QV txym = ldv(X.slot() + HB, p.k0), tyzm = ldv(X.slot() + HB + OF::CF, p.k0);
    X.release();
    for (int j = T.ys; j < ye; ++j, v0 += plane, P.x += P.sx, P.z += P.sz) {
        const bool plane_in = j >= EFM_HS && j < yhi_in + ylo_in - EFM_HS;
        const bool ypml = j < ylo_in || j >= yhi_in;
        // the plane is one of the outer two of the box on either side of y (strips)
        const bool yface = !ypml && (j < ylo_in + 2 || j >= yhi_in - 2);
        bool mine;
        if (PASS == EFM_REV) {
            // reverse rebuild (-dt, no CPML) into the ping-pong partner f.vo: CPML slabs -> 0,
            // boundary strips -> the values saved at forward step nt-2-it (:1955-1960),
            // box interior -> stencil update, never-updated cells -> 0.  The strip values of
            // this plane are requested before the wait.
            int slot[VX];
            float sval[VX][3];
            const bool strips = !ypml && (sf & (yface ? 15 : (15 << 4) | 256)) != 0;
#pragma unroll
            for (int v = 0; v < VX; ++v) slot[v] = -1;
            if (strips) {
                const int W = I.W, by = I.ny - 2 * W, bx = I.nx - 2 * W, bz = I.nz - W - 2;
                const float *sv = I.border + (int64_t)(I.nt - 2 - it) * 3 * I.strip_n;
                const int64_t strip_n = I.strip_n;
#pragma unroll
                for (int v = 0; v < VX; ++v) {
                    const bool xf = sf & (16 << v);
                    if (!(sf & (1 << v)) || !(xf || yface || (sf & 256))) continue;
                    // (a cell's families hold the same values)
                    slot[v] = strip_slot(bx, by, bz, p.x + v - W, j - W, p.z - 2, xf ? 0 : yface ? 1 : 2);
                    sval[v][0] = sv[slot[v]];
                    sval[v][1] = sv[strip_n + slot[v]];
                    sval[v][2] = sv[2 * strip_n + slot[v]];
                }
            }
            mine = X.wait();
            if (mine) {
                const VelIn a = velocity_in<NT>(p, X.prev(), X.slot());
                QV old[3], o[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) old[c] = ldv(X.slot() + HB + c * OF::CF, p.k0);
#pragma unroll
                for (int v = 0; v < VX; ++v) {
                    const float dtxx_dx = (v < VX - 1 ? a.txx.v[v + 1] : a.txxi) - a.txx.v[v];
                    const float dtzz_dz = a.tzzk.v[v] - a.tzz.v[v];
                    const float dtyy_dy = a.tyyj.v[v] - a.tyy.v[v];
                    const float txyc = a.txy.v[v], txzc = a.txz.v[v], tyzc = a.tyz.v[v];
                    const float dtxy_dy = txyc - txym.v[v];
                    const float dtxy_dx = txyc - (v ? a.txy.v[v - 1] : a.txym);
                    const float dtxz_dz = txzc - a.txzk.v[v];
                    const float dtxz_dx = txzc - (v ? a.txz.v[v - 1] : a.txzm);
                    const float dtyz_dz = tyzc - a.tyzk.v[v];
                    const float dtyz_dy = tyzc - tyzm.v[v];
                    const float b0 = a.b0.v[v], bi = v < VX - 1 ? a.b0.v[v + 1] : a.bi, bk = a.bk.v[v];
                    const float bj = a.bj.v[v];
                    const float b_x = 2.f * b0 * bi * frcp(b0 + bi);
                    const float b_y = 2.f * b0 * bj * frcp(b0 + bj);
                    const float b_z = 2.f * b0 * bk * frcp(b0 + bk);
                    const float nvx = old[0].v[v] + k * b_x * (dtxx_dx + dtxy_dy + dtxz_dz);
                    const float nvy = old[1].v[v] + k * b_y * (dtxy_dx + dtyy_dy + dtyz_dz);
                    const float nvz = old[2].v[v] + k * b_z * (dtxz_dx + dtyz_dy + dtzz_dz);
                    const bool in = (sf & (1 << v)) && !ypml && plane_in && p.in(v);
                    o[0].v[v] = in ? nvx : 0.f;
                    o[1].v[v] = in ? nvy : 0.f;
                    o[2].v[v] = in ? nvz : 0.f;
                }
                if (strips) {
#pragma unroll
                    for (int v = 0; v < VX; ++v)
#pragma unroll
                        for (int c = 0; c < 3; ++c) o[c].v[v] = slot[v] >= 0 ? sval[v][c] : o[c].v[v];
                }
                txym = a.txy;
                tyzm = a.tyz;
                if (p.fl & F_ACT) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) stv(v0 + c * N, o[c]);
                }
            }
        } else {
            const bool rec_plane = rec_now != 0;
            if (j + 1 < ye) rec_now = __ldg(recs + j + 1);
            // the plane's update (see Tag)
            auto update = [&](auto tag) -> bool {
                constexpr int PML = decltype(tag)::value;
                constexpr bool REC = PML == 2;
                PsiOld<PML, false> O;
                float ay = 0.f, by_ = 0.f;
                int py = 0;
                if (PML) {
                    if (PML == 2 && ypml) {
                        py = psi_y(I, p, 1, j);
                        ay = I.cpml[2 * I.nx + j];
                        by_ = I.cpml[2 * I.nx + I.ny + j];
                    }
                    if (plane_in) O.load(p, P, ypml, py);
                    if (j + 1 < ye) {
                        prefetch_psi(p, P);
                        if (PML == 2 && ypml && (p.fl & F_IN) && (j + 1 < ylo_in || j >= yhi_in))
                            prefetch2(P.base + (py + I.nz * I.nx));
                    }
                }
                int rq[VX];
                bool more[VX];  // the cell may hold several receivers
#pragma unroll
                for (int v = 0; v < VX; ++v) {
                    rq[v] = -1;
                    more[v] = false;
                    if (REC && rec_plane && p.act(v)) rq[v] = efm_rec_first(I, p.x + v, j, p.z, &more[v]);
                }
                if (!X.wait()) return false;
                const VelIn a = velocity_in<NT>(p, X.prev(), X.slot());
                QV old[3], o[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) old[c] = ldv(X.slot() + HB + c * OF::CF, p.k0);
                float oy[VX][3], oz[VX][3];
                const bool wy = PML == 2 && ypml && p.any_in(), wz = PML == 2 && (p.fl & F_PZ);
#pragma unroll
                for (int v = 0; v < VX; ++v) {
                    const float dtxx_dx = (v < VX - 1 ? a.txx.v[v + 1] : a.txxi) - a.txx.v[v];
                    const float dtzz_dz = a.tzzk.v[v] - a.tzz.v[v];
                    const float dtyy_dy = a.tyyj.v[v] - a.tyy.v[v];
                    const float txyc = a.txy.v[v], txzc = a.txz.v[v], tyzc = a.tyz.v[v];
                    const float dtxy_dy = txyc - txym.v[v];
                    const float dtxy_dx = txyc - (v ? a.txy.v[v - 1] : a.txym);
                    const float dtxz_dz = txzc - a.txzk.v[v];
                    const float dtxz_dx = txzc - (v ? a.txz.v[v - 1] : a.txzm);
                    const float dtyz_dz = tyzc - a.tyzk.v[v];
                    const float dtyz_dy = tyzc - tyzm.v[v];
                    // harmonic 2-point buoyancy from the precomputed 1/rho (:153-159)
                    const float b0 = a.b0.v[v], bi = v < VX - 1 ? a.b0.v[v + 1] : a.bi, bk = a.bk.v[v];
                    const float bj = a.bj.v[v];
                    const float b_x = 2.f * b0 * bi * frcp(b0 + bi);
                    const float b_y = 2.f * b0 * bj * frcp(b0 + bj);
                    const float b_z = 2.f * b0 * bk * frcp(b0 + bk);
                    if (PML == 0) {  // (the sums below without their zero terms)
                        o[0].v[v] = old[0].v[v] + k * b_x * (dtxx_dx + dtxy_dy + dtxz_dz);
                        o[1].v[v] = old[1].v[v] + k * b_y * (dtxy_dx + dtyy_dy + dtyz_dz);
                        o[2].v[v] = old[2].v[v] + k * b_z * (dtxz_dx + dtyz_dy + dtzz_dz);
                        continue;
                    }
                    float q1 = 0.f, q2 = 0.f, q3 = 0.f, q4 = 0.f, q5 = 0.f, q6 = 0.f, q7 = 0.f, q8 = 0.f, q9 = 0.f;
                    if (PML && plane_in) {
                        if (PML == 1 || (p.fl & F_WX)) {
                            psi_step(p.px(v), O.x[v], P.ax[v], P.bx[v], dtxx_dx, dtxy_dx, dtxz_dx);
                            q1 = O.x[v][0];
                            q2 = O.x[v][1];
                            q3 = O.x[v][2];
                            if (v == VX - 1) st_psi_x(p, P.base + P.x, O.x);
                        }
                        if (PML == 2 && ypml) {
                            if (v == 0) O.get_y(wy, P.base + py, oy);
                            psi_step(wy, oy[v], ay, by_, dtyy_dy, dtxy_dy, dtyz_dy);
                            q4 = oy[v][0];
                            q5 = oy[v][1];
                            q6 = oy[v][2];
                            if (v == VX - 1 && wy) st_psi(P.base + py, oy[0], oy[1]);
                        }
                        if (PML == 2 && (p.fl & F_WZ)) {
                            if (v == 0) O.get_z(wz, P.base + P.z, oz);
                            psi_step(wz, oz[v], P.az, P.bz, dtzz_dz, dtxz_dz, dtyz_dz);
                            q7 = oz[v][0];
                            q8 = oz[v][1];
                            q9 = oz[v][2];
                            if (v == VX - 1 && wz) st_psi(P.base + P.z, oz[0], oz[1]);
                        }
                    }
                    o[0].v[v] = old[0].v[v] + k * b_x * ((dtxx_dx + q1) + (dtxy_dy + q5) + (dtxz_dz + q8));
                    o[1].v[v] = old[1].v[v] + k * b_y * ((dtxy_dx + q2) + (dtyy_dy + q4) + (dtyz_dz + q9));
                    o[2].v[v] = old[2].v[v] + k * b_z * ((dtxz_dx + q3) + (dtyz_dy + q6) + (dtzz_dz + q7));
                }
                txym = a.txy;
                tyzm = a.tyz;
                // cells the stencil does not update keep their values
                if (!plane_in || (p.fl & F_PART) || REC) {
#pragma unroll
                    for (int v = 0; v < VX; ++v) {
                        const bool guard = plane_in && p.in(v);
#pragma unroll
                        for (int c = 0; c < 3; ++c) o[c].v[v] = guard ? o[c].v[v] : old[c].v[v];
                    }
                }
                bool any = plane_in && p.any_in();
                if (REC && rec_plane) {
#pragma unroll
                    for (int v = 0; v < VX; ++v) {
                        if (rq[v] < 0) continue;
                        const int64_t ntr = (int64_t)I.nt * I.nrec;
                        const int c = p.x + v + I.nx * (p.z + I.nz * j);
                        if (PASS == EFM_ADJ) {
                            any = true;
                            for (int q = rq[v];;) {
                                const int64_t e = (int64_t)(I.nt - 1 - it) * I.nrec + I.rec_id[q];
                                o[0].v[v] = __fadd_rn(o[0].v[v], I.res[e]);
                                o[1].v[v] = __fadd_rn(o[1].v[v], I.res[ntr + e]);
                                o[2].v[v] = __fadd_rn(o[2].v[v], I.res[2 * ntr + e]);
                                if (!more[v] || ++q >= I.nrec || I.rec_lin[q] != c) break;
                            }
                        } else if (I.gather != nullptr) {
                            for (int q = rq[v];;) {
                                const int64_t e = (int64_t)it * I.nrec + I.rec_id[q];
                                I.gather[e] = o[0].v[v];
                                I.gather[ntr + e] = o[1].v[v];
                                I.gather[2 * ntr + e] = o[2].v[v];
                                if (!more[v] || ++q >= I.nrec || I.rec_lin[q] != c) break;
                            }
                        }
                    }
                }
                if (any) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) stv(v0 + c * N, o[c]);
                }
                if (PASS == EFM_FWD) {
                    if (ILLUM && plane_in) {
#pragma unroll
                        for (int v = 0; v < VX; ++v) {
                            const float nvx = o[0].v[v], nvy = o[1].v[v], nvz = o[2].v[v];
                            if (!p.in(v)) continue;
                            float *const e = I.illum + (p.x + v + I.nx * (p.z + I.nz * j));
                            *e = __fadd_rn(*e, __fmaf_rn(nvz, nvz, two_products(nvy, nvy, nvx, nvx)));
                        }
                    }
                    // the strips the pair's box cells belong to (sf is zero without strips)
                    if (!ypml && (sf & (yface ? 15 : (15 << 4) | 256))) {
                        const int W = I.W, by = I.ny - 2 * W, bx = I.nx - 2 * W, bz = I.nz - W - 2;
                        float *s = I.border + (int64_t)it * 3 * I.strip_n;
                        const int64_t strip_n = I.strip_n;
#pragma unroll
                        for (int f = 0; f < 3; ++f) {
                            if (!(f == 0 ? (sf & (15 << 4)) != 0 : f == 1 ? yface : (sf & 256) != 0)) continue;
#pragma unroll
                            for (int v = 0; v < VX; ++v) {
                                if (!(sf & ((f == 0 ? 16 : 1) << v))) continue;
                                float *e = s + strip_slot(bx, by, bz, p.x + v - W, j - W, p.z - 2, f);
                                st1(e, o[0].v[v]);
                                st1(e + strip_n, o[1].v[v]);
                                st1(e + 2 * strip_n, o[2].v[v]);
                            }
                        }
                    }
                }
                return true;
            };
            mine = ypml || rec_plane || (p.fl & F_WZ) ? update(Tag<2>{})
                   : p.fl & F_WX                      ? update(Tag<1>{})
                                                      : update(Tag<0>{});
        }
        if (!__all_sync(0xffffffffu, mine)) return -1;
        X.release();
    }
    return X.packed();
}

// ----------------------------------------------------------------------------- imaging
// Zero-lag imaging of a reverse step (kernel_Gradients_Rho/Lambda/Mu, :191-294): fV_present (the
// forward velocity before the rebuild step), fV (after it), the adjoint fields after the adjoint
// step, into the lambda / mu / rho gradients.  Neighbour fields: fV_present vx (x0-4, z0), vy (x0,
// z0), vz (x0, z0-2; two rows below), 1/mu (x0, z0); cell fields: fV vx vy vz, adjoint vx vy vz,
// lambda.  The adjoint stresses (in L2 from the velocity pass) and the gradients are requested
// with plain loads before the plane's wait.  First slot's cell part: fV_present vy of the two
// planes before the chunk.
template <int NT>
struct IOff {
    static constexpr int XZ = efm_slot_xz(NT), CF = efm_slot_c(NT);
    static constexpr int px = 0, py = XZ, rm = 2 * XZ, pz = 3 * XZ;
};

template <int NT, int D, int SLOT>
__device__ __forceinline__ int image_chunk(int packed, int ib) {
    using O = IOff<NT>;
    Ctx<D, SLOT> X(packed);
    const EfmInst &I = X.B.inst[ib];
    const Chunk &T = X.B.chunk[ib];
    constexpr int HB = efm_halo_i(NT), CF = O::CF;
    const Pair p = make_pair<false>(I, T);
    const int plane = I.nz * I.pitch, gplane = I.nz * I.nx;
    const int64_t N = I.vol;
    const float *bt = I.bt[0] + (int64_t)T.ys * plane + p.z * I.pitch + p.x;
    int64_t go = (int64_t)T.ys * gplane + p.z * I.nx + p.x;
    float *const g_[3] = {I.g_lam, I.g_mu, I.g_rho};
    const float idt = I.inv_dt, idx = I.inv_dx;
    const int ye = T.ye, jlo = EFM_HS, jhi = I.ny - EFM_HS;
    const int i0 = p.i0, i1 = p.i0 + p.hp, i2 = i1 + p.hp;
    efm_pdl_wait();
    if (!__all_sync(0xffffffffu, X.wait())) return -1;
    QV py1 = ldv(X.slot() + HB, p.k0), py2 = ldv(X.slot() + HB + CF, p.k0);
    X.release();
    for (int j = T.ys; j < ye; ++j, bt += plane, go += gplane) {
        const bool live = j >= jlo && j < jhi && p.any_in();
        QV b[6], g[3];
        if (live) {
#pragma unroll
            for (int q = 0; q < 6; ++q) b[q] = ldgv(bt + q * N);
#pragma unroll
            for (int q = 0; q < 3; ++q) g[q] = ldgv(g_[q] + go);
        }
        if (!__all_sync(0xffffffffu, X.wait())) return -1;
        const unsigned char *h = X.prev(), *hn = X.slot(), *cc = X.slot() + HB;
        const QV py = ldv(h + O::py, i0);
        if (live) {
            const QV px = ldv(h + O::px, i0 + 4), pxz = ldv(h + O::px, i1 + 4), pxj = ldv(hn + O::px, i0 + 4);
            const float2 pxm2 = ld2(h + O::px, i0 + 2);  // x - 2, x - 1
            const QV pyz = ldv(h + O::py, i1);
            const float pyx = ld1(h + O::py, i0 + VX);
            const QV pz = ldv(h + O::pz, i2), pzm1 = ldv(h + O::pz, i1), pzm2 = ldv(h + O::pz, i0);
            const QV pzj = ldv(hn + O::pz, i2);
            const float pzx = ld1(h + O::pz, i2 + VX);
            const QV m0 = ldv(h + O::rm, i0), mk = ldv(h + O::rm, i1);
            const QV mj = ldv(hn + O::rm, i0), mjk = ldv(hn + O::rm, i1);
            const float mi = ld1(h + O::rm, i0 + VX), mik = ld1(h + O::rm, i1 + VX), mij = ld1(hn + O::rm, i0 + VX);
            QV c[7], o[3];
#pragma unroll
            for (int q = 0; q < 7; ++q) c[q] = ldv(cc + q * CF, p.k0);
#pragma unroll
            for (int v = 0; v < VX; ++v) {
                const float pxc = px.v[v], pyc = py.v[v], pzc = pz.v[v];
                const float nvx = c[0].v[v], nvy = c[1].v[v], nvz = c[2].v[v];
                const float bvx = c[3].v[v], bvy = c[4].v[v], bvz = c[5].v[v], lam = c[6].v[v];
                const float btxx = b[0].v[v], btyy = b[1].v[v], btzz = b[2].v[v];
                const float btxy = b[3].v[v], btxz = b[4].v[v], btyz = b[5].v[v];
                const float grho = -((bvx * ((pxc - nvx) * idt)) + (bvy * ((pyc - nvy) * idt)) +
                                     (bvz * ((pzc - nvz) * idt)));
                // lambda: average of two backward differences / dx (:234-238)
                const float pxm = v ? px.v[v - 1] : pxm2.y, pym = py1.v[v], pzm = pzm1.v[v];
                const float pxmm = v == 0 ? pxm2.x : pxm2.y;
                const float dvx = two_products(0.5f * (pxm - pxmm), idx, 0.5f * (pxc - pxm), idx);
                const float dvy = two_products(0.5f * (pym - py2.v[v]), idx, 0.5f * (pyc - pym), idx);
                const float dvz = two_products(0.5f * (pzm - pzm2.v[v]), idx, 0.5f * (pzc - pzm), idx);
                const float r0 = m0.v[v], ri = v < VX - 1 ? m0.v[v + 1] : mi, rk = mk.v[v];
                const float rik = v < VX - 1 ? mk.v[v + 1] : mik;
                const float rj = mj.v[v], rjk = mjk.v[v], rij = v < VX - 1 ? mj.v[v + 1] : mij;
                const float mu0 = frcp(r0);
                const float glam = (btxx + btyy + btzz) * (dvx + dvy + dvz) * frcp(3.f * lam + 2.f * mu0);
                // mu: forward strain differences, not divided by dx (:277-291)
                const float ex = pxc - pxm, ey = pyc - pym, ez = pzc - pzm;
                const float exz = pxz.v[v] - pxc, exy = pxj.v[v] - pxc;
                const float eyx = (v < VX - 1 ? py.v[v + 1] : pyx) - pyc, eyz = pyz.v[v] - pyc;
                const float ezx = (v < VX - 1 ? pz.v[v + 1] : pzx) - pzc, ezy = pzj.v[v] - pzc;
                const float imu_xy = 0.25f * (r0 + ri + rj + rij);
                const float imu_xz = 0.25f * (r0 + ri + rk + rik);
                const float imu_yz = 0.25f * (r0 + rj + rk + rjk);
                const float f = frcp(mu0 * (3.f * lam + 2.f * mu0));
                const float lpm2 = 2.f * (lam + mu0);
                const float gmu = f * (lpm2 * btxx - lam * btyy - lam * btzz) * ex +
                                  f * (lpm2 * btyy - lam * btxx - lam * btzz) * ey +
                                  f * (lpm2 * btzz - lam * btxx - lam * btyy) * ez +
                                  imu_xy * btxy * (eyx + exy) + imu_xz * btxz * (exz + ezx) +
                                  imu_yz * btyz * (ezy + eyz);
                o[0].v[v] = g[0].v[v] + glam;
                o[1].v[v] = g[1].v[v] + gmu;
                o[2].v[v] = g[2].v[v] + grho;
            }
            if (p.fl & F_PART) {  // a pair at the edge of the updated cells keeps the other's values
#pragma unroll
                for (int v = 0; v < VX; ++v)
#pragma unroll
                    for (int q = 0; q < 3; ++q) o[q].v[v] = p.in(v) ? o[q].v[v] : g[q].v[v];
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) stv(g_[q] + go, o[q]);
        }
        py2 = py1;
        py1 = py;
        X.release();
    }
    return X.packed();
}

// ------------------------------------------------------------------------------ the loads
// One load of a slot: where the field goes, its map, the box's corner relative to the tile's and
// the plane relative to the slot's, and the box's size class.  The producer's lanes
// take one each (one lane issuing them all takes longer than a plane's computation).
enum { BOX_C, BOX_X, BOX_Z, BOX_XZ, BOX_XZ2 = 5 };  // cells; + 4 columns; + a row; both; two rows

struct LoadOp {
    int off;
    signed char map, dx, dz, dy, box;
};

struct LoadTab {
    int n[2];          // loads of a slot, of a chunk's first slot
    LoadOp op[2][12];
};

template <int NT>
struct Loads {
    static constexpr int X = efm_slot_x(NT), Z = efm_slot_z(NT), XZ = efm_slot_xz(NT), C = efm_slot_c(NT);
    static constexpr int HS = efm_halo_s(NT), HV = efm_halo_v(NT), HI = efm_halo_i(NT);
    using V = VOff<NT>;
    using M = IOff<NT>;
    static constexpr LoadTab stress() {
        return {{11, 5},
                {{{0, 0, -4, 0, 1, BOX_XZ}, {XZ, 1, 0, 0, 1, BOX_XZ}, {2 * XZ, 2, 0, -1, 1, BOX_XZ},
                  {3 * XZ, 3, 0, 0, 1, BOX_XZ}, {HS, 4, 0, 0, 0, BOX_C}, {HS + C, 5, 0, 0, 0, BOX_C},
                  {HS + 2 * C, 6, 0, 0, 0, BOX_C}, {HS + 3 * C, 7, 0, 0, 0, BOX_C}, {HS + 4 * C, 8, 0, 0, 0, BOX_C},
                  {HS + 5 * C, 9, 0, 0, 0, BOX_C}, {HS + 6 * C, 10, 0, 0, 0, BOX_C}},
                 {{0, 0, -4, 0, 1, BOX_XZ}, {XZ, 1, 0, 0, 1, BOX_XZ}, {2 * XZ, 2, 0, -1, 1, BOX_XZ},
                  {3 * XZ, 3, 0, 0, 1, BOX_XZ}, {HS, 11, 0, 0, 0, BOX_C}}}};
    }
    static constexpr LoadTab velocity() {
        return {{10, 9},
                {{{V::txx, 0, 0, 0, 1, BOX_X}, {V::tzz, 1, 0, 0, 1, BOX_Z}, {V::txy, 2, -4, 0, 1, BOX_X},
                  {V::txz, 3, -4, -1, 1, BOX_XZ}, {V::tyz, 4, 0, -1, 1, BOX_Z}, {V::bu, 5, 0, 0, 1, BOX_XZ},
                  {V::tyy, 6, 0, 0, 1, BOX_C}, {HV, 7, 0, 0, 0, BOX_C}, {HV + C, 8, 0, 0, 0, BOX_C},
                  {HV + 2 * C, 9, 0, 0, 0, BOX_C}},
                 {{V::txx, 0, 0, 0, 1, BOX_X}, {V::tzz, 1, 0, 0, 1, BOX_Z}, {V::txy, 2, -4, 0, 1, BOX_X},
                  {V::txz, 3, -4, -1, 1, BOX_XZ}, {V::tyz, 4, 0, -1, 1, BOX_Z}, {V::bu, 5, 0, 0, 1, BOX_XZ},
                  {V::tyy, 6, 0, 0, 1, BOX_C}, {HV, 10, 0, 0, 0, BOX_C}, {HV + C, 11, 0, 0, 0, BOX_C}}}};
    }
    static constexpr LoadTab image() {
        return {{11, 6},
                {{{M::px, 0, -4, 0, 1, BOX_XZ}, {M::py, 1, 0, 0, 1, BOX_XZ}, {M::pz, 2, 0, -2, 1, BOX_XZ2},
                  {M::rm, 3, 0, 0, 1, BOX_XZ}, {HI, 4, 0, 0, 0, BOX_C}, {HI + C, 5, 0, 0, 0, BOX_C},
                  {HI + 2 * C, 6, 0, 0, 0, BOX_C}, {HI + 3 * C, 7, 0, 0, 0, BOX_C}, {HI + 4 * C, 8, 0, 0, 0, BOX_C},
                  {HI + 5 * C, 9, 0, 0, 0, BOX_C}, {HI + 6 * C, 10, 0, 0, 0, BOX_C}},
                 {{M::px, 0, -4, 0, 1, BOX_XZ}, {M::py, 1, 0, 0, 1, BOX_XZ}, {M::pz, 2, 0, -2, 1, BOX_XZ2},
                  {M::rm, 3, 0, 0, 1, BOX_XZ}, {HI, 11, 0, 0, 0, BOX_C}, {HI + C, 11, 0, 0, -1, BOX_C}}}};
    }
};

__constant__ LoadTab g_loads[2][3] = {{Loads<224>::stress(), Loads<224>::velocity(), Loads<224>::image()},
                                      {Loads<96>::stress(), Loads<96>::velocity(), Loads<96>::image()}};

// This lane's loads of a chunk's slots ([1]: of the first one), and the bytes of all of them.
struct LaneLoads {
    int off[2], x[2], z[2], dy[2], map[2], bytes[2];
    bool on[2];
};

template <int NT>
__device__ __forceinline__ LaneLoads lane_loads(const Chunk &T, int lane) {
    const LoadTab &L = g_loads[NT == 96][T.type];
    LaneLoads r;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        r.on[k] = lane < L.n[k];
        const LoadOp o = L.op[k][r.on[k] ? lane : 0];
        r.off[k] = o.off;
        r.x[k] = T.x0 + o.dx;
        r.z[k] = T.z0 + o.dz;
        r.dy[k] = o.dy;
        r.map[k] = o.map;
        const int w = T.tw + (o.box & 1 ? 4 : 0), h = T.th + (o.box >> 1);  // (BOX_XZ2 >> 1 = 2 rows)
        r.bytes[k] = __reduce_add_sync(0xffffffffu, r.on[k] ? 4 * w * h : 0);
    }
    return r;
}

// ---------------------------------------------------------------------------- the producer
// Chunk `id` of an instance: tiles first, then y; the last run of planes comes second, so that
// the slower CPML planes at both ends of y start early.
__device__ __forceinline__ Chunk chunk_at(const EfmInst &I, int type, int id) {
    const int l = id - I.tile_begin;
    const int cols = I.tiles_x * I.tiles_z;
    int ty = l / cols;
    Chunk c;
    c.type = type;
    c.tw = I.tw;
    c.th = I.th;
    c.col = l - ty * cols;
    ty = ty == 0 ? 0 : ty == 1 ? I.tiles_y - 1 : ty - 1;
    const int tz = c.col / I.tiles_x;
    c.x0 = I.ox + (c.col - tz * I.tiles_x) * I.tw;
    c.z0 = I.oz + tz * I.th;
    c.ys = I.ylo + ty * I.ychunk;
    c.ye = min(I.yhi, c.ys + I.ychunk);
    return c;
}

// The producer warp: every chunk's slots in order, its lanes issuing one field each.  Block b
// starts with chunk b; the numbers of the next chunks, and their table entries, are fetched while
// the current one is loaded.  CPML chunks take longer than interior ones: dealt out in turn
// instead, the slowest block of a 256 x 256 x 128 launch ran a quarter longer than the mean.
// Every block fetches until its first number past the end, `total` fetches in all, so the last
// one resets the counter for the next launch (which waits for this grid); a call starts with the
// counter cleared, in case a wait ran out before.  Before it leaves it waits (default bound) for
// its own loads still in flight, so that none outlives the block when consumers gave up on them;
// where nothing gave up the consumers wait for the same loads, and it costs nothing.
template <int NT, int D, int SLOT, int VT>
struct Producer {
    static constexpr int PARTS = (int)((sizeof(EfmInst) / 16 + 31) / 32);
    const EfmStream &A;
    Block<D> &B;
    const int lane, total;
    int id, pend;  // the next chunk, lane 0's number after it
    int4 part[PARTS];
    Chunk T;
    const CUtensorMap *tm;

    __device__ __forceinline__ Producer(const EfmStream &A_)
        : A(A_), B(block_state<D, SLOT>()), lane(threadIdx.x & 31), total(A.cs + A.cv), id(blockIdx.x), pend(0) {}

    __device__ __forceinline__ void fetch() {
        if (lane == 0) {
            const int v = atomicAdd(A.counter, 1);
            if (v == total - 1) *(volatile int *)A.counter = 0;
            pend = (int)gridDim.x + v;
        }
    }

    // chunk id's table entry (the call's static tables)
    __device__ __forceinline__ void entry() {
        if (id >= total) return;
        const int type = id < A.cs ? 0 : VT, k = id - (type ? A.cs : 0);
        const EfmInst &I = type ? A.v[efm_find_inst(A.v, A.nv, k)] : A.s[efm_find_inst(A.s, A.ns, k)];
#pragma unroll
        for (int q = 0; q < PARTS; ++q)
            if (lane + 32 * q < (int)(sizeof(EfmInst) / 16))
                part[q] = __ldg(reinterpret_cast<const int4 *>(&I) + lane + 32 * q);
        T = chunk_at(I, type, k);
        tm = I.tmap;
    }

    // Hand the description to the consumers.
    __device__ __forceinline__ void announce(int ib) {
        int4 *o = reinterpret_cast<int4 *>(&B.inst[ib]);
#pragma unroll
        for (int q = 0; q < PARTS; ++q)
            if (lane + 32 * q < (int)(sizeof(EfmInst) / 16)) o[lane + 32 * q] = part[q];
        if (lane == 0) B.chunk[ib] = T;
        __syncwarp();
        if (lane == 0) efm_mbar_arrive(&B.ready[ib]);
    }

    // The first chunk, before the preceding kernel has finished.
    __device__ __forceinline__ void prepare() {
        entry();
        const LaneLoads ll = lane_loads<NT>(T, lane);
#pragma unroll
        for (int f = 0; f < 2; ++f)
            if (ll.on[f]) efm_prefetch_tmap(tm + ll.map[f]);
        announce(0);
    }

    __device__ __forceinline__ void run() {
        const uint32_t lim = B.lim;
        Cursor<D> c;
        int q = 0;
        bool ok = true;
        fetch();
        int ib = 0;
        while (true) {
            const LaneLoads ll = lane_loads<NT>(T, lane);
            const int ys = T.ys, ye = T.ye;
            const CUtensorMap *const m = tm;
            for (int p = ys - 1; p < ye; ++p) {
                ok = __all_sync(0xffffffffu, ring_wait(B, &B.empty[c.cs], c.ph ^ 1u, lim));
                if (!ok) break;
                const int f = p < ys;
                if (f && q) announce(ib);
                if (lane == 0) efm_mbar_expect_tx(&B.full[c.cs], ll.bytes[f]);
                __syncwarp();
                if (ll.on[f])
                    efm_tma_load_3d(ring_slot<SLOT>(c.hs) + ll.off[f], m + ll.map[f], &B.full[c.cs], ll.x[f], ll.z[f],
                                    p + ll.dy[f]);
                __syncwarp();
                if (p == min(ys, ye - 1)) {  // (the first slots are on their way)
                    id = __shfl_sync(0xffffffffu, pend, 0);
                    if (id < total) fetch();
                    entry();
                }
                c.next();
                ++q;
            }
            if (!ok) break;
            ib = B.next(ib);
            if (id >= total) {
                ok = __all_sync(0xffffffffu, ring_wait(B, &B.empty[c.cs], c.ph ^ 1u, lim));
                if (ok && lane == 0) {
                    B.chunk[ib].type = -1;
                    efm_mbar_arrive(&B.ready[ib]);
                }
                break;
            }
        }
        // whoever gave up, this warp or a consumer that has left: the newest load of every barrier
        if (lane == 0)
            for (int s = max(0, q - D); s < q; ++s) efm_mbar_wait(&B.full[s % D], (s / D) & 1, nullptr);
    }
};

// The consumers' side of one pass: the launch's chunks of type TYPE, n the number of chunks done
// before.  Returns the ring position (negative: a wait gave up).
template <int TYPE, int D, int SLOT, class F>
__device__ __forceinline__ int consume(int cur, int &n, F &&chunk) {
    constexpr int N = Block<D>::N;
    while (cur >= 0) {
        Block<D> &B = block_state<D, SLOT>();
        const int ib = n % N;
        if (!__all_sync(0xffffffffu, ring_wait(B, &B.ready[ib], (uint32_t)(n / N) & 1u, B.lim))) return -1;
        if (*(volatile int *)&B.chunk[ib].type != TYPE) return cur;
        cur = chunk(cur, ib);
        ++n;
    }
    return cur;
}

}  // namespace

// One streaming launch: stress pass PS (-1: none), then velocity pass PV (-1: none, EFM_IMG: the
// imaging).  With both,
// two independent half-steps share a grid: the gradient's adjoint chain and its reverse-time
// rebuild touch disjoint fields within a step, so (adjoint stress, rebuild velocity) and (rebuild
// stress, adjoint velocity) fill the SMs together instead of running back to back.  Each pass has
// a loop of its own: one loop over both kinds of chunks needs more registers than there are
// (spills of 200 to 500 bytes per thread, and a third more time).
template <int PS, int PV, int NT, int D, bool ILLUM>
__global__ void __launch_bounds__(NT + 32, efm_stream_blocks(NT, D)) efm_stream(const __grid_constant__ EfmStream A) {
    constexpr int SLOT = efm_slot_bytes(NT, PV == EFM_IMG);
    Block<D> &B = block_state<D, SLOT>();
    efm_pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < D; ++s) {
            efm_mbar_init(&B.full[s], 1);
            efm_mbar_init(&B.empty[s], NT / 32);
        }
        for (int s = 0; s < Block<D>::N; ++s) efm_mbar_init(&B.ready[s], 1);
        B.abort = 0;
        B.lim = A.lim;
        B.err = A.err;
        efm_fence_barrier_init();
    }
    __syncthreads();
    // what comes before efm_pdl_wait (a chunk's set-up, here and in the consumers) reads only the
    // call's static tables; the fields and the counter come after the preceding kernel has finished
    if (threadIdx.x >= NT) {
        Producer<NT, D, SLOT, PV == EFM_IMG ? 2 : 1> P(A);
        P.prepare();
        efm_pdl_wait();
        P.run();
        return;
    }
    constexpr int S = PS < 0 ? 0 : PS, V = PV < 0 || PV == EFM_IMG ? 0 : PV;
    int cur = Ctx<D, SLOT>::START, n = 0;
    if (PS >= 0)
        cur = consume<0, D, SLOT>(cur, n, [&](int c, int b) { return stress_chunk<S, NT, D, SLOT>(c, b, A.it); });
    if (PV == EFM_IMG)
        consume<2, D, SLOT>(cur, n, [&](int c, int b) { return image_chunk<NT, D, SLOT>(c, b); });
    else if (PV >= 0)
        consume<1, D, SLOT>(
            cur, n, [&](int c, int b) { return velocity_chunk<V, NT, D, SLOT, ILLUM>(c, b, A.it); });
}

// 1/mu and 1/rho for the streaming kernels (once per call; the model may change in place).
__global__ void efm_model_reciprocals(const float *__restrict__ mu, const float *__restrict__ rho,
                                      float *__restrict__ rmu, float *__restrict__ buoy, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        rmu[i] = __frcp_rn(mu[i]);
        buoy[i] = __frcp_rn(rho[i]);
    }
}


// ---------------------------------------------------------------------------- launchers
// Launch with the programmatic-serialization attribute when enabled: the kernel's prologue
// overlaps the tail of the preceding kernel (every streaming kernel waits in
// efm_pdl_wait before it reads or writes fields).  Set by each efm_forward / efm_gradient
// call from its context's option, per calling thread.
static thread_local int g_pdl = 1;

extern "C" void efm_stream_set_pdl(int enable) { g_pdl = enable != 0; }
extern "C" int efm_stream_pdl() { return g_pdl; }

// Errors surface through the launcher's cudaGetLastError(); a failed cudaLaunchKernelEx is
// recorded there too, but keep its own status for the first failure of a sequence.
static thread_local cudaError_t g_launch_err = cudaSuccess;

template <typename... KArgs, typename... Args>
static void launch_k(void (*k)(KArgs...), int grid, int threads, int smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, args...);
    if (e != cudaSuccess && g_launch_err == cudaSuccess) g_launch_err = e;
}

static cudaError_t take_launch_err() {
    const cudaError_t e = g_launch_err;
    g_launch_err = cudaSuccess;
    const cudaError_t l = cudaGetLastError();
    return e != cudaSuccess ? e : l;
}

template <int NT, int D>
constexpr int smem_bytes(bool image) {
    return (D + 1) * efm_slot_bytes(NT, image) + (int)sizeof(Block<D>);
}
static_assert(2 * (smem_bytes<224, 3>(true) + 1024) <= 228 * 1024, "two blocks of 224 consumers per SM");
static_assert(4 * (smem_bytes<96, 3>(true) + 1024) <= 228 * 1024, "four blocks of 96 consumers per SM");
static_assert(3 * (smem_bytes<96, 5>(true) + 1024) <= 228 * 1024, "three with the deeper ring");

// Blocks that fill the device.
extern "C" int efm_stream_slots(int rows, int ring) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms * efm_stream_blocks(efm_st_nt(rows), rows == 1 && ring == 6 ? 5 : 3);
}

// Kernels by stress and velocity pass; f is called with each one.
template <int NT, int D, class F>
static void each_stream(F &&f) {
    f(EFM_FWD, -1, 0, efm_stream<EFM_FWD, -1, NT, D, false>);
    f(EFM_ADJ, -1, 0, efm_stream<EFM_ADJ, -1, NT, D, false>);
    f(EFM_REV, -1, 0, efm_stream<EFM_REV, -1, NT, D, false>);
    f(-1, EFM_FWD, 0, efm_stream<-1, EFM_FWD, NT, D, false>);
    f(-1, EFM_FWD, 1, efm_stream<-1, EFM_FWD, NT, D, true>);
    f(-1, EFM_ADJ, 0, efm_stream<-1, EFM_ADJ, NT, D, false>);
    f(-1, EFM_REV, 0, efm_stream<-1, EFM_REV, NT, D, false>);
    f(-1, EFM_IMG, 0, efm_stream<-1, EFM_IMG, NT, D, false>);
    f(EFM_ADJ, EFM_REV, 0, efm_stream<EFM_ADJ, EFM_REV, NT, D, false>);
    f(EFM_REV, EFM_ADJ, 0, efm_stream<EFM_REV, EFM_ADJ, NT, D, false>);
}

template <int NT, int D>
static void launch_stream_k(int ps, int pv, int illum, int grid, const EfmStream &A, cudaStream_t s) {
    each_stream<NT, D>([&](int a, int b, int i, auto k) {
        if (a == ps && b == pv && i == illum) launch_k(k, grid, NT + 32, smem_bytes<NT, D>(pv == EFM_IMG), s, A);
    });
}

// Stress pass ps of the leading ns entries of table ts (cs chunks) and / or velocity pass pv of
// table tv's; a pass not wanted is -1 with no chunks.  illum: the forward velocity also sums the
// illumination.
extern "C" cudaError_t efm_launch_stream(int ps, int pv, int illum, int rows, int ring, const EfmInst *ts, int ns,
                                         int cs, const EfmInst *tv, int nv, int cv, int grid, int it, int *counter,
                                         unsigned int lim, unsigned int *err, cudaStream_t s) {
    const EfmStream A = {ts, tv, ns, nv, cs, cv, it, counter, lim, err};
    if (rows == 1 && ring == 6)
        launch_stream_k<96, 5>(ps, pv, illum, grid, A, s);
    else if (rows == 1)
        launch_stream_k<96, 3>(ps, pv, illum, grid, A, s);
    else
        launch_stream_k<224, 3>(ps, pv, illum, grid, A, s);
    return take_launch_err();
}

extern "C" cudaError_t efm_launch_reciprocals(const float *mu, const float *rho, float *rmu,
                                              float *buoy, int64_t n, cudaStream_t s) {
    int64_t b = (n + 255) / 256;
    if (b > 148 * 8) b = 148 * 8;
    efm_model_reciprocals<<<(int)b, 256, 0, s>>>(mu, rho, rmu, buoy, n);
    return cudaGetLastError();
}

template <int NT, int D>
static cudaError_t set_attributes() {
    cudaError_t e = cudaSuccess;
    each_stream<NT, D>([&](int, int pv, int, auto k) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<NT, D>(pv == EFM_IMG));
    });
    return e;
}

extern "C" cudaError_t efm_stream_init_attributes() {
    cudaError_t e;
    if ((e = set_attributes<96, 3>())) return e;
    if ((e = set_attributes<96, 5>())) return e;
    return set_attributes<224, 3>();
}
