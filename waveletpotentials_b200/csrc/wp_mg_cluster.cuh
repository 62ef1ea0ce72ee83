// wp_mg_cluster.cuh -- the V-cycle of the small levels in one launch of one thread-block cluster
// (included by wp_mg.cu inside its anonymous namespace).
//
// What bounds the small levels is latency: as separate launches a 32^3 level costs 6-11 us per sweep
// (under 0.3 us of L2 traffic), and the levels from 16^3 down took 35 us per cycle in one CTA, whose
// single SM does all the arithmetic.  Here up to 16 CTAs hold a level as slabs of planes in their shared
// memory, stencils included, so a sweep is a pass over shared memory and a cluster barrier:
//   - a CTA owns P consecutive z planes of a level (P a power of two, halved with the level, so a
//     coarse cell's children are its owner's) and copies the planes beside them from its neighbours'
//     shared memory before a pass reads them;
//   - below P = 1 a level is replicated: every CTA holds and computes all of it (at most a few hundred
//     cells for cubes), so its sweeps need no cluster barrier at all and its coarsest iterations run
//     in one warp;
//   - the stencils (6 or 8 floats per cell, in the order the shared memory holds them, one block per CTA)
//     are built once per handle and copied in asynchronously before the previous kernel has finished.
// A 2D level (nx, ny) is the slab problem (1, ny, nx): planes are rows along y.
//
// A handle that shares the device takes only the levels of one CTA this way, and the pack's larger levels by
// the kernels at the end of this file (see wp_mg_share_device); the persistent cycle and the persistent batch
// run the same two halves as phases of theirs.  All of them give the same bits.
// Measured (B200, per V(2,2) cycle): 32^3 ... 2^3 31 us in one launch, formerly 75 us in six; 2D 256^2 ... 2^2 50 us
// against 110 us.  Projections: 32^3 872 -> 663 us, 128^3 (FP32) 2292 -> 2000 us, 2D 256^2 1055 -> 731 us.
// The cycle's functions have two forms, CL: the cluster's CTAs of 512 threads, stencils in shared memory; else one
// 1024-thread CTA of a persistent kernel, stencils read through L1, which the kernel's other work needs large.
constexpr int kCyThreads = 512;
__host__ __device__ constexpr int cy_nt(bool cl) { return cl ? kCyThreads : 1024; }
constexpr int kCyMax = 12;           // levels of a pack
constexpr int kCyCells = 4096;       // cells of a level a CTA may hold
// floats per cell: the face coefficients y- y+ z- z+ and (3D) x- x+, then 1 / diagonal (0: inactive) and
// the restriction weight
__host__ __device__ constexpr int cy_floats(bool two_d) { return two_d ? 6 : 8; }
constexpr size_t kCySmem = 208 * 1024;

struct CyLev {
    int nx, ny, nz, nxy;
    int P;               // planes per CTA; 0: replicated
    int cap;             // cells a CTA holds: P nxy, or all
    int cf, f, v, t;     // offsets (floats) in shared memory; v and t past their lower halo plane
};
struct CyPack {
    CyLev lv[kCyMax];
    int n, ctas;
    int image;           // floats of a CTA's stencil block (a multiple of 4)
    int floats;          // shared floats in all
};

// a pack, its finest level and its stencils (one block of the image per CTA); image null: none
struct CyPlan {
    CyPack pack;
    int l0;
    float* image;
};

// Stencils of one level into every CTA's block.  V: the level (2D: nz = 1, its x axis is the pack's z).
template <bool D2>
__global__ void cy_coeff_kernel(float* __restrict__ out, CyPack C, int l, Lvl<float> V) {
    const CyLev L = C.lv[l];
    const int r = blockIdx.y;
    float* o = out + (long)r * C.image + L.cf;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.cap; i += gridDim.x * blockDim.x) {
        float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float rd = 0.f, wc = 0.f;
        const int pz = (L.P ? r * L.P : 0) + i / L.nxy, rem = i % L.nxy;
        if (pz < L.nz) {
            const int x = D2 ? pz : rem / L.ny, y = rem % L.ny, z = D2 ? 0 : pz;
            const int nx = V.nx, ny = V.ny, nz = V.nz;
            const long i3 = y + (long)x * ny + (long)z * nx * ny;
            const long iax = y + (long)x * ny + (long)z * (nx + 1) * ny;
            const long iay = y + (long)x * (ny + 1) + (long)z * nx * (ny + 1);
            float dg = 0.f;
            if (y > 0) { c[0] = V.ay[iay] * V.glo[1][y]; dg += c[0]; }
            if (y < ny - 1) { c[1] = V.ay[iay + 1] * V.ghi[1][y]; dg += c[1]; }
            constexpr int kx = D2 ? 2 : 4;  // the slab axis is x in 2D
            if (x > 0) { c[kx] = V.ax[iax] * V.glo[0][x]; dg += c[kx]; }
            if (x < nx - 1) { c[kx + 1] = V.ax[iax + ny] * V.ghi[0][x]; dg += c[kx + 1]; }
            if (!D2 && z > 0) { c[2] = V.az[i3] * V.glo[2][z]; dg += c[2]; }
            if (!D2 && z < nz - 1) { c[3] = V.az[i3 + (long)nx * ny] * V.ghi[2][z]; dg += c[3]; }
            rd = dg > (float)kEps ? 1.f / dg : 0.f;
            const int x0 = x & ~1, y0 = y & ~1, zb = z & ~1;
            const double sx = V.d[0][x0] + (x0 + 1 < nx ? V.d[0][x0 + 1] : 0.0);
            const double sy = V.d[1][y0] + (y0 + 1 < ny ? V.d[1][y0 + 1] : 0.0);
            const double sz = V.d[2][zb] + (zb + 1 < nz ? V.d[2][zb + 1] : 0.0);
            wc = (float)(V.d[2][z] / sz) * (float)(V.d[1][y] / sy * (V.d[0][x] / sx));
        }
        constexpr int nc = cy_floats(D2) - 2;
#pragma unroll
        for (int k = 0; k < nc; ++k) o[k * L.cap + i] = c[k];
        o[nc * L.cap + i] = rd;
        o[(nc + 1) * L.cap + i] = wc;
    }
}

__device__ __forceinline__ void cy_barrier() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// *p of CTA `rank` of the cluster (p: this CTA's address of the same word)
__device__ __forceinline__ uint32_t cy_map(const float* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(wptc::smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float cy_pull(const float* p, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cy_map(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float4 cy_pull4(const float* p, int rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(cy_map(p, rank))
                 : "memory");
    return v;
}

// A level as one CTA sees it, kept at the start of the dynamic shared memory.  The arrays are offsets into
// it, not pointers: a pointer read from memory is a generic one, and generic loads made every pass twice as
// long.
struct CySm {
    int nx, ny, nz, nxy, P, cap;
    int z0, n;          // first plane, cells owned
    int lo, hi;         // a neighbour owns the planes below / above
    unsigned mxy, my;   // i / nxy = umulhi(i, mxy), rem / ny = umulhi(rem, my) (0: a divisor of 1)
    int cf, f, v, t;
    const float* gcf;   // without CL: the stencils
};
constexpr int kCyHead = 256; // floats reserved for the level table
static_assert(kCyMax * sizeof(CySm) <= kCyHead * sizeof(float), "level table");
extern __shared__ __align__(16) float cy_smem[];
__device__ __forceinline__ const CySm& cy_lv(int l) { return reinterpret_cast<const CySm*>(cy_smem)[l]; }
template <bool CL>
__device__ __forceinline__ const float* cy_stencils(const CySm& S) { return CL ? cy_smem + S.cf : S.gcf; }
__device__ __forceinline__ int cy_div(int i, unsigned m) { return m ? (int)__umulhi((unsigned)i, m) : i; }

// The passes below are calls, not inlined: a cycle runs each of them once or a few times per level, so its time
// is instruction fetch as much as arithmetic.  Specialised and unrolled per level (stencils in
// registers) the same cycle took 29 us with its code in the instruction cache and 43 us without.

// Copies the neighbours' planes beside this CTA's into the halos of b (a buffer every CTA has finished
// writing).  A remote load instruction takes the SM some 40 cycles whatever its width, so planes move 16
// bytes per lane: reading them word by word inside the sweeps made a 32^3 sweep 3600 cycles.
template <bool CL>
__device__ __noinline__ void cy_halos(int l, int bo, int rank) {
    const CySm& S = cy_lv(l);
    const int nxy = S.nxy, cap = S.cap;
    const bool lo = S.lo, hi = S.hi;
    float* b = cy_smem + bo;
    if (((nxy | bo) & 3) == 0) {
#pragma unroll 1
        for (int i = 4 * threadIdx.x; i < 2 * nxy; i += 4 * cy_nt(CL)) {
            const bool up = i >= nxy;
            const int j = up ? i - nxy : i;
            if (up ? hi : lo)
                *reinterpret_cast<float4*>(up ? b + cap + j : b + j - nxy) =
                    up ? cy_pull4(b + j, rank + 1) : cy_pull4(b + cap - nxy + j, rank - 1);
        }
    } else {
#pragma unroll 1
        for (int i = threadIdx.x; i < 2 * nxy; i += cy_nt(CL)) {
            const bool up = i >= nxy;
            const int j = up ? i - nxy : i;
            if (up ? hi : lo) b[up ? cap + j : j - nxy] = up ? cy_pull(b + j, rank + 1) : cy_pull(b + cap - nxy + j, rank - 1);
        }
    }
    __syncthreads();
}

// One cell of a pass: CY_SWEEP the swept value (0 where the diagonal is 0; from zero if `zero`), CY_RESID the
// residual times the restriction weight.  k: the cell's first stencil entry, entries cap apart; u(o): the iterate o
// cells further.  Its operations are spelled out, so that the shared-memory passes and the kernels below, which
// run a level of a pack from global memory, give the same bits.
enum { CY_SWEEP = 0, CY_RESID = 1 };
template <bool D2, class U>
__device__ __forceinline__ float cy_cell(const float* k, int cap, int ny, int nxy, float f, float w, int mode, bool zero, U u) {
    constexpr int NC = cy_floats(D2) - 2;
    const float rd = k[NC * cap];
    float r = f, x = 0.f;
    if (!zero) {
        x = u(0);
        float s = __fmul_rn(k[0], u(-1) - x);
        s = fmaf(k[cap], u(1) - x, s);
        if (!D2) {
            r = fmaf(k[4 * cap], u(-ny) - x, r);
            r = fmaf(k[5 * cap], u(ny) - x, r);
        }
        s = fmaf(k[2 * cap], u(-nxy) - x, s);
        r = __fadd_rn(fmaf(k[3 * cap], u(nxy) - x, r), s);
    }
    const float o = mode == CY_SWEEP ? fmaf(__fmul_rn(w, rd), r, x) : __fmul_rn(r, k[(NC + 1) * cap]);
    return rd > 0.f ? o : 0.f;
}

// The interpolated correction of fine cell (x, y, z) from the coarse level at u (extents cnx, cny, cnz)
template <bool D2>
__device__ __forceinline__ float cy_interp(const float* u, int x, int y, int z, int cnx, int cny, int cnz, int kind) {
    const int cx = x >> 1, cy = y >> 1, cz = z >> 1, cnxy = cnx * cny;
    auto mix = [](float near, float far) { return fmaf(0.25f, far, __fmul_rn(0.75f, near)); };
    u += cz * cnxy + cx * cny;
    float o = u[cy];
    if (kind == WP_PROLONG_TRILINEAR) {
        int oy = (y & 1) ? cy + 1 : cy - 1, dz = (z & 1) ? 1 : -1, dx = (x & 1) ? 1 : -1;
        if (oy < 0 || oy >= cny) oy = cy;
        if (cz + dz < 0 || cz + dz >= cnz) dz = 0;
        if (cx + dx < 0 || cx + dx >= cnx) dx = 0;
        const float* q = u + dz * cnxy;
        o = mix(o, u[oy]);
        float p = mix(q[cy], q[oy]);
        if (!D2) {
            const float *ux = u + dx * cny, *qx = q + dx * cny;
            o = mix(o, mix(ux[cy], ux[oy]));
            p = mix(p, mix(qx[cy], qx[oy]));
        }
        o = mix(o, p);
    }
    return o;
}

// One pass over the owned cells: CY_SWEEP dst = src + w (f - A src) / diagonal (0 where the diagonal is 0; from
// zero if so < 0), CY_RESID dst = the residual times the restriction weight.  Ends with every CTA in
// step (CY_SWEEP) or this one (CY_RESID).
template <bool D2, bool CL>
__device__ __noinline__ void cy_pass(int l, int so, int dof, float w, int mode, int rank) {
    const CySm& S = cy_lv(l);
    const int cap = S.cap, nxy = S.nxy, ny = S.ny, n = S.n, P = S.P;
    const float *cf = cy_stencils<CL>(S), *f = cy_smem + S.f, *src = cy_smem + so;
    float* dst = cy_smem + dof;
    if (so >= 0 && P) cy_halos<CL>(l, so, rank);
#pragma unroll 2
    for (int i = threadIdx.x; i < n; i += cy_nt(CL))
        dst[i] = cy_cell<D2>(cf + i, cap, ny, nxy, f[i], w, mode, so < 0, [src, i](int o) { return src[i + o]; });
    if (mode == CY_SWEEP && P) cy_barrier();
    else __syncthreads();
}

// n sweeps of v (from zero: zero); v the iterate's offset, t the other buffer's
template <bool D2, bool CL>
__device__ __forceinline__ void cy_smooth(int l, int& v, int& t, int n, float w, bool zero, int rank) {
    if (zero && n == 0) cy_pass<D2, CL>(l, -1, v, 0.f, CY_SWEEP, rank);
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        cy_pass<D2, CL>(l, zero && k == 0 ? -1 : v, t, w, CY_SWEEP, rank);
        const int u = v;
        v = t;
        t = u;
    }
}

// f of level l + 1 = the sums of level l's weighted residuals r over each coarse cell's children
template <bool D2, bool CL>
__device__ __noinline__ void cy_sums(int l, int ro) {
    const CySm *S = &cy_lv(l), *C = &cy_lv(l + 1);
    float *r = cy_smem + ro, *fc = cy_smem + C->f;
    const int planes = S->n / S->nxy, z0 = S->z0, nx = S->nx, ny = S->ny, nxy = S->nxy, cnxy = C->nxy;
    const int cz0 = z0 >> 1, cz1 = (z0 + planes + 1) >> 1;  // coarse planes with children here
    // a replicated level below a distributed one: the owners' sums (of one plane of children each) are left
    // beside r and collected by every CTA after a barrier
    const bool gather = S->P && C->P == 0;
    float* out = gather ? r + S->cap : fc;
#pragma unroll 1
    for (int i = threadIdx.x; i < (planes ? cz1 - cz0 : 0) * cnxy; i += cy_nt(CL)) {
        const int pz = cy_div(i, C->mxy), rem = i - pz * cnxy, x = D2 ? 0 : cy_div(rem, C->my), y = rem - x * C->ny;
        float s = 0.f;
#pragma unroll 1
        for (int dz = 0; dz < 2; ++dz) {
            const int z = 2 * (cz0 + pz) + dz - z0;
            if (z < 0 || z >= planes) continue;
            const float* row = r + z * nxy + 2 * x * ny + 2 * y;
            const bool y1 = 2 * y + 1 < ny;
            // plane by plane, as the collected sums below: the same result for every number of CTAs
            float p = row[0] + (y1 ? row[1] : 0.f);
            if (!D2 && 2 * x + 1 < nx) p += row[ny] + (y1 ? row[ny + 1] : 0.f);
            s += p;
        }
        out[i] = s;
    }
    if (gather) {
        cy_barrier();
#pragma unroll 1
        for (int i = threadIdx.x; i < C->cap; i += cy_nt(CL)) {
            const int z = cy_div(i, C->mxy), rem = i - z * cnxy;
            float s = cy_pull(out + rem, 2 * z);
            if (2 * z + 1 < S->nz) s += cy_pull(out + rem, 2 * z + 1);
            fc[i] = s;
        }
    }
    __syncthreads();
}

// v += P vc, v of level l, vc of level l + 1
template <bool D2, bool CL>
__device__ __noinline__ void cy_prolong(int l, int vo, int vco, int kind, int rank) {
    const CySm *S = &cy_lv(l), *C = &cy_lv(l + 1);
    float* v = cy_smem + vo;
    const int cnxy = C->nxy, cny = C->ny, cnx = C->nx, cnz = C->nz;
    if (S->P && C->P) cy_halos<CL>(l + 1, vco, rank);
    const int base = vco - C->z0 * cnxy;
    const int nxy = S->nxy, ny = S->ny, z0 = S->z0, n = S->n;
#pragma unroll 2
    for (int i = threadIdx.x; i < n; i += cy_nt(CL)) {
        const int pz = cy_div(i, S->mxy), rem = i - pz * nxy, x = D2 ? 0 : cy_div(rem, S->my), y = rem - x * ny;
        v[i] += cy_interp<D2>(cy_smem + base, x, y, z0 + pz, cnx, cny, cnz, kind);
    }
    if (S->P) cy_barrier();
    else __syncthreads();
}

// A coarsest level of extents <= 2 (cubes and squares of a power of two end there): its citers sweeps from
// zero are one linear map of f.  One warp forms it (row i, column j at m[8 i + j]) in the prologue, while
// the previous kernel still runs, by sweeping the unit right-hand sides: lane l carries cell l & 7 of the
// columns 2 (l >> 3) and 2 (l >> 3) + 1.
template <bool D2, bool CL>
__device__ __noinline__ void cy_coarsest_map(int l, float* m, float w, int citers) {
    constexpr int NC = cy_floats(D2) - 2;
    const CySm* S = &cy_lv(l);
    const int lane = threadIdx.x, i = lane & 7, cap = S->cap;
    const float* cf = cy_stencils<CL>(*S);
    const int step[3] = {1, S->nxy, S->ny};
    const float rd = i < cap ? cf[NC * cap + i] : 0.f;
    float c[3] = {0.f, 0.f, 0.f};
    int src[3] = {lane, lane, lane};
#pragma unroll
    for (int k = 0; k < NC / 2; ++k) {
        // an axis of extent 2 has one neighbour per cell: the lower or the upper coefficient is 0
        const float lo = i < cap ? cf[2 * k * cap + i] : 0.f, hi = i < cap ? cf[(2 * k + 1) * cap + i] : 0.f;
        c[k] = w * rd * (lo + hi);
        if (lo != 0.f) src[k] = lane - step[k];
        else if (hi != 0.f) src[k] = lane + step[k];
    }
    const int j0 = 2 * (lane >> 3);
    const float b0 = i == j0 ? w * rd : 0.f, b1 = i == j0 + 1 ? w * rd : 0.f, keep = rd > 0.f ? 1.f - w : 0.f;
    float x0 = 0.f, x1 = 0.f;
#pragma unroll 1
    for (int it = 0; it < citers; ++it) {
        float a0 = fmaf(keep, x0, b0), a1 = fmaf(keep, x1, b1);
#pragma unroll
        for (int k = 0; k < NC / 2; ++k) {
            const float u0 = __shfl_sync(0xffffffffu, x0, src[k]), u1 = __shfl_sync(0xffffffffu, x1, src[k]);
            a0 = fmaf(c[k], u0, a0);
            a1 = fmaf(c[k], u1, a1);
        }
        x0 = a0;
        x1 = a1;
    }
    if (i < cap) {
        m[8 * i + j0] = x0;
        m[8 * i + j0 + 1] = x1;
    }
}

// citers sweeps from zero of a replicated level of at most 32 cells by one warp, a cell per lane in registers
template <bool D2, bool CL>
__device__ __noinline__ void cy_warp_sweeps(int l, float* v, float w, int citers) {
    constexpr int NC = cy_floats(D2) - 2;
    const CySm* S = &cy_lv(l);
    const int n = S->cap, i = threadIdx.x;
    const float *cf = cy_stencils<CL>(*S), *f = cy_smem + S->f;
    const int off[6] = {-1, 1, -S->nxy, S->nxy, -S->ny, S->ny};
    const float rd = i < n ? cf[NC * n + i] : 0.f;
    float c[NC], x = 0.f;
    int src[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int j = i + off[k];
        const bool in = i < n && j >= 0 && j < n;
        src[k] = in ? j : i;
        c[k] = in ? w * rd * cf[k * n + i] : 0.f;
    }
    const float b = rd > 0.f ? w * (f[i] * rd) : 0.f, keep = rd > 0.f ? 1.f - w : 0.f;
#pragma unroll 1
    for (int it = 0; it < citers; ++it) {
        float s = fmaf(keep, x, b), t = 0.f;
#pragma unroll
        for (int k = 0; k < NC; k += 2) {
            s = fmaf(c[k], __shfl_sync(0xffffffffu, x, src[k]), s);
            t = fmaf(c[k + 1], __shfl_sync(0xffffffffu, x, src[k + 1]), t);
        }
        x = s + t;
    }
    if (i < n) v[i] = x;
}

// V-cycle from level `first` of the pack: f the level's right-hand side, from v = 0 or (vin) from vin,
// into vout or (p64) added to p64.  What the previous kernel wrote is first read after wp_pdl_enter.
template <bool D2, bool CL>
__device__ __forceinline__ void cy_cycle(const CyPack& C, const float* image, int rank, int first, const float* f,
                                         const float* vin, float* vout, double* p64, int nu1, int nu2, float w, int citers,
                                         int prolong) {
    __shared__ float cmap[64];
    float* sm = cy_smem;
    CySm* S = reinterpret_cast<CySm*>(cy_smem);
    const int tid = threadIdx.x;
    // the stencils are constant: their copy starts before the previous kernel has finished
    if (CL) {
        const float* g = image + (long)rank * C.image;
        const int from = C.lv[first].cf;  // a multiple of 4
        for (int i = from / 4 + tid; i < C.image / 4; i += cy_nt(CL)) cp_async16(sm + kCyHead + 4 * i, g + 4 * i);
        cp_async_commit();
    }
    if (tid < C.n) {
        const CyLev& L = C.lv[tid];
        CySm q;
        q.nx = L.nx; q.ny = L.ny; q.nz = L.nz; q.nxy = L.nxy; q.P = L.P; q.cap = L.cap;
        q.z0 = L.P ? rank * L.P : 0;
        const int planes = L.P ? max(0, min(L.P, L.nz - q.z0)) : L.nz;
        q.n = planes * L.nxy;
        q.lo = L.P && rank > 0 && planes > 0;
        q.hi = L.P && q.z0 + L.P < L.nz;
        // exact for the indices here: i d < 2^32 (at most 2^13 cells)
        q.mxy = L.nxy > 1 ? (unsigned)((0x100000000ull + L.nxy - 1) / L.nxy) : 0u;
        q.my = L.ny > 1 ? (unsigned)((0x100000000ull + L.ny - 1) / L.ny) : 0u;
        const int at = CL ? kCyHead : kCyHead - C.image;
        q.cf = at + L.cf; q.f = at + L.f; q.v = at + L.v; q.t = at + L.t;
        q.gcf = image + L.cf;
        S[tid] = q;
    }
    __syncthreads();
    // the planes around a level's cells are read with zero coefficients only: they have to be finite
#pragma unroll 1
    for (int l = first; l < C.n; ++l) {
        const CySm& q = S[l];
#pragma unroll 1
        for (int i = tid; i < 2 * q.nxy + q.cap - q.n; i += cy_nt(CL)) {
            const int j = i < q.nxy ? i - q.nxy : q.n + i - q.nxy;
            sm[q.v + j] = 0.f;
            sm[q.t + j] = 0.f;
        }
    }
    const int last = C.n - 1;
    const bool mapped = C.lv[last].P == 0 && C.lv[last].nx <= 2 && C.lv[last].ny <= 2 && C.lv[last].nz <= 2;
    cp_async_wait<0>();
    __syncthreads();
    if (mapped && tid < 32) cy_coarsest_map<D2, CL>(last, cmap, w, citers);
    if (CL) wp_pdl_enter();
    const CySm& F = S[first];
    const long g0 = (long)F.z0 * F.nxy;
#pragma unroll 1
    for (int i = tid; i < F.n; i += cy_nt(CL)) {
        sm[F.f + i] = f[g0 + i];
        if (vin) sm[F.v + i] = vin[g0 + i];
    }
    // with an iterate, the neighbours read it in the first sweep
    if (vin && F.P) cy_barrier();
    else __syncthreads();
    unsigned flip = 0;  // bit l: level l's iterate is in t
#pragma unroll 1
    for (int l = first; l < C.n; ++l) {
        int v = S[l].v, t = S[l].t;
        const int cap = S[l].cap;
        if (l == last && mapped) {
            if (tid < cap) {
                float x = 0.f;
                for (int j = 0; j < cap; ++j) x = fmaf(cmap[8 * tid + j], sm[S[l].f + j], x);
                sm[v + tid] = x;
            }
            __syncthreads();
            break;
        }
        if (l == last && S[l].P == 0 && cap <= 32) {
            if (tid < 32) cy_warp_sweeps<D2, CL>(l, sm + v, w, citers);
            __syncthreads();
            break;
        }
        cy_smooth<D2, CL>(l, v, t, l < last ? nu1 : citers, w, !(l == first && vin), rank);
        if (v != S[l].v) flip |= 1u << l;
        if (l < last) {
            cy_pass<D2, CL>(l, v, t, w, CY_RESID, rank);
            cy_sums<D2, CL>(l, t);
        }
    }
#pragma unroll 1
    for (int l = last - 1; l >= first; --l) {
        const bool in_t = (flip >> l) & 1;
        int v = in_t ? S[l].t : S[l].v, t = in_t ? S[l].v : S[l].t;
        cy_prolong<D2, CL>(l, v, (flip >> (l + 1)) & 1 ? S[l + 1].t : S[l + 1].v, prolong, rank);
        cy_smooth<D2, CL>(l, v, t, nu2, w, false, rank);
        flip = v == S[l].t ? flip | 1u << l : flip & ~(1u << l);
    }
    // (the last pass ended in a barrier: no CTA leaves while a neighbour reads its planes)
    const float* v = sm + ((flip >> first) & 1 ? F.t : F.v);
    const int n = F.P || rank == 0 ? F.n : 0;  // a replicated first level is written by CTA 0
    if (p64)
        for (int i = tid; i < n; i += cy_nt(CL)) p64[g0 + i] += (double)v[i];
    else
        for (int i = tid; i < n; i += cy_nt(CL)) vout[g0 + i] = v[i];
}

template <bool D2>
__global__ void __launch_bounds__(kCyThreads) cycle_cluster_kernel(const __grid_constant__ CyPack C,
                                                                   const float* __restrict__ image, int first,
                                                                   const float* f, const float* vin, float* vout,
                                                                   double* p64, int nu1, int nu2, float w, int citers,
                                                                   int prolong) {
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    cy_cycle<D2, true>(C, image, (int)rank, first, f, vin, vout, p64, nu1, nu2, w, citers, prolong);
}

// The cycle of a pack of one CTA from v = 0, as a phase of a 1024-thread persistent kernel
template <bool D2>
__device__ __noinline__ void cy_one_cta(const CyPack& C, const float* image, int first, const float* f, float* vout, int nu1,
                                        int nu2, float w, int citers, int prolong) {
    cy_cycle<D2, false>(C, image, 0, first, f, nullptr, vout, nullptr, nu1, nu2, w, citers, prolong);
}

// Layout of a pack of levels (extents e[l] = {nx, ny, nz} of the slab problem) over `ctas` CTAs; false
// when it does not fit a CTA's shared memory.
// (dynamic shared bytes of its cycle with and without the stencils: floats, floats - image)
inline bool cy_layout(CyPack* C, const int (*e)[3], int n, int ctas, bool two_d) {
    if (n < 2 || n > kCyMax) return false;
    C->n = n;
    C->ctas = ctas;
    int P = 1;
    while (P * ctas < e[0][2]) P *= 2;
    long off = 0;
    for (int l = 0; l < n; ++l, P >>= 1) {
        CyLev& L = C->lv[l];
        L.nx = e[l][0];
        L.ny = e[l][1];
        L.nz = e[l][2];
        if ((long)L.nx * L.ny * L.nz > (1L << 24)) return false;
        L.nxy = L.nx * L.ny;
        L.P = ctas > 1 ? P : 0;
        L.cap = L.P ? L.P * L.nxy : L.nxy * L.nz;
        if (L.cap > kCyCells) return false;
        L.cf = (int)off;
        off += (cy_floats(two_d) * (long)L.cap + 3) / 4 * 4;
    }
    C->image = (int)off;
    for (int l = 0; l < n; ++l) {
        CyLev& L = C->lv[l];
        // (v and t on 16-byte boundaries where a plane is a multiple of one)
        L.f = (int)off;
        off = (off + L.cap + 3) / 4 * 4;
        L.v = (int)(off + L.nxy);
        off = (off + L.cap + 2L * L.nxy + 3) / 4 * 4;
        L.t = (int)(off + L.nxy);
        off = (off + L.cap + 2L * L.nxy + 3) / 4 * 4;
        if ((off + kCyHead) * sizeof(float) > kCySmem) return false;
    }
    C->floats = (int)off + kCyHead;
    return true;
}

// ---- one level of a pack from global memory, launch by launch: the cluster's arithmetic, on its stencil image
struct CyGlobal {
    const float* k;   // the level's entries in the image
    int image, cap;   // floats between the CTAs' blocks, cells of a block
    int nx, ny, nz, nxy, n;
};
__device__ __forceinline__ const float* cy_entry(const CyGlobal& G, int i) {
    const int r = i / G.cap;
    return G.k + (long)r * G.image + (i - r * G.cap);
}
// the cells beside the level's ends are read with zero coefficients only
template <bool D2>
__device__ __forceinline__ float cy_cell_global(const CyGlobal& G, const float* v, const float* f, int i, float w, int mode) {
    return cy_cell<D2>(cy_entry(G, i), G.cap, G.ny, G.nxy, f[i], w, mode, v == nullptr,
                       [&](int o) { return v[min(max(i + o, 0), G.n - 1)]; });
}
// cell i of a sweep of v (null: from zero) into dst or (p64) added to p64
template <bool D2>
__device__ __forceinline__ void cy_sweep_one(float* dst, double* p64, const float* v, const float* f, const CyGlobal& G, float w,
                                             int i) {
    const float o = cy_cell_global<D2>(G, v, f, i, w, CY_SWEEP);
    if (p64) p64[i] += (double)o;
    else dst[i] = o;
}
// coarse cell i of the restricted residual
template <bool D2>
__device__ __forceinline__ void cy_restrict_one(float* fc, const float* v, const float* f, const CyGlobal& G, int cnx, int cny,
                                                int i) {
    const int cz = i / (cnx * cny), rem = i - cz * cnx * cny, x = D2 ? 0 : 2 * (rem / cny), y = 2 * (rem % cny);
    float s = 0.f;
    // cy_sums' order
    for (int z = 2 * cz; z < min(2 * cz + 2, G.nz); ++z) {
        const int j = y + x * G.ny + z * G.nxy;
        auto pair = [&](int k) {
            const float a = cy_cell_global<D2>(G, v, f, k, 0.f, CY_RESID);
            return a + (y + 1 < G.ny ? cy_cell_global<D2>(G, v, f, k + 1, 0.f, CY_RESID) : 0.f);
        };
        float p = pair(j);
        if (!D2 && x + 1 < G.nx) p += pair(j + G.ny);
        s += p;
    }
    fc[i] = s;
}
// cell i of v += P vc
template <bool D2>
__device__ __forceinline__ void cy_prolong_one(float* v, const float* vc, const CyGlobal& G, int cnx, int cny, int cnz, int kind,
                                               int i) {
    const int z = i / G.nxy, rem = i - z * G.nxy, x = D2 ? 0 : rem / G.ny, y = rem - x * G.ny;
    v[i] += cy_interp<D2>(vc, x, y, z, cnx, cny, cnz, kind);
}
template <bool D2>
__global__ void __launch_bounds__(256) cy_sweep_kernel(float* __restrict__ dst, const float* __restrict__ v,
                                                       const float* __restrict__ f, CyGlobal G, float w) {
    wp_pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < G.n) cy_sweep_one<D2>(dst, nullptr, v, f, G, w, i);
}
template <bool D2>
__global__ void __launch_bounds__(256) cy_restrict_kernel(float* __restrict__ fc, const float* __restrict__ v,
                                                          const float* __restrict__ f, CyGlobal G, int cnx, int cny, int cn) {
    wp_pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < cn) cy_restrict_one<D2>(fc, v, f, G, cnx, cny, i);
}
template <bool D2>
__global__ void __launch_bounds__(256) cy_prolong_kernel(float* __restrict__ v, const float* __restrict__ vc, CyGlobal G,
                                                         int cnx, int cny, int cnz, int kind) {
    wp_pdl_enter();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < G.n) cy_prolong_one<D2>(v, vc, G, cnx, cny, cnz, kind, i);
}
